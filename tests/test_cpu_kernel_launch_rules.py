"""Rules for kernels that start while the kernel in front of them still runs (csrc/kernels/launch_pdl.cuh), read off the sources: a violation is a race that a
run shows rarely or never."""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KERNELS = os.path.join(ROOT, "csrc", "kernels")


def _code(path):
    """The file without its comments."""
    with open(path) as f:
        text = f.read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def _files_that_launch_early():
    files = {n: _code(os.path.join(KERNELS, n)) for n in sorted(os.listdir(KERNELS)) if n.endswith((".cu", ".cuh"))}

    def reaches(name, seen=()):
        return name == "launch_pdl.cuh" or any(reaches(i, (*seen, name)) for i in re.findall(r'#include "([^"]+)"', files.get(name, "")) if i not in seen)

    early = {n for n in files if reaches(n)}
    # ... and the headers of their own that those include
    for n in list(early):
        early |= {i for i in re.findall(r'#include "([^"/]+\.cuh)"', files[n])}
    return {n: files[n] for n in sorted(early)}


EARLY = _files_that_launch_early()


def test_the_scan_finds_the_files():
    assert {"flash_decode.cu", "gemm_host.cuh", "gemm_ops.cu", "gemm_skinny.cu", "moe.cu", "moe_experts.cuh", "quantize.cu", "quantize_common.cuh",
            "ring_attention_tc.cu"} <= set(EARLY)


@pytest.mark.parametrize("name", sorted(EARLY))
def test_no_promise_that_inputs_do_not_change_while_the_kernel_runs(name):
    """A kernel in front may write them until griddepcontrol.wait returns. `const T* __restrict__`, __ldg and ld.global.nc tell the compiler and the
    read-only path that nobody does, so loads could move in front of the wait or return what was there before."""
    found = re.findall(r"__restrict__|__ldg\b|ld\.global\.nc", EARLY[name])
    assert not found, f"{name}: {found}"
