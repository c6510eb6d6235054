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


def _body(text, head):
    """The function whose definition contains `head`, from its name to its closing brace."""
    at = text.index(head)
    i = text.index("{", text.index(")", at))
    depth, j = 1, i + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
    return text[at:j]


@pytest.mark.parametrize("path,function", [
    ("include/iris/gemm/sm100_mainloop.cuh", "void gemm_cta_main("), ("csrc/kernels/gemm_skinny.cu", " skinny_gemm_kernel(")])
def test_tensor_memory_is_allocated_between_wait_and_trigger(path, function):
    """A CTA that waits for the kernel in front holds no columns that kernel may still ask for, and the kernel behind does not start before this one
    has its columns: otherwise two kernels on one SM can wait for each other without end."""
    body = _body(_code(os.path.join(ROOT, path)), function)
    wait, alloc, trigger = (body.index(w) for w in ("pdl_wait()", "tmem_alloc", "pdl_trigger()"))
    assert wait < alloc < trigger, path


@pytest.mark.parametrize("name", ["router_topk_kernel", "moe_meta_kernel", "moe_sort_kernel", "moe_clear_kernel", "moe_prep_kernel", "moe_gather_kernel",
                                  "moe_gather_quant_kernel", "moe_reduce_kernel"])
def test_moe_kernels_trigger_behind_their_wait(name):
    """The kernel behind one of them reads tokens, weights or tables before its own wait: they are complete because this one has waited."""
    body = _body(EARLY["moe.cu"], " " + name + "(")
    assert body.index("pdl_wait()") < body.index("pdl_trigger()")


def test_attention_waits_before_anything_else():
    """The attention kernel's CTA body allocates and triggers; the kernel waits in front of it."""
    text = EARLY["ring_attention_tc.cu"]
    main, kernel = _body(text, "void attn_main_tc("), _body(text, " ring_attention_tc_kernel(")
    assert main.index("tmem_alloc") < main.index("pdl_trigger()") and "pdl_wait" not in main
    assert kernel.index("pdl_wait()") < kernel.index("attn_main_tc<")


def test_expert_kernel_allocates_before_its_trigger_behind_a_gather_that_waited():
    """It allocates in front of its wait. Nothing but its own layer's kernels can be in flight then: stage 1 is launched behind a gather, which triggers
    behind its own wait, and stage 2 behind stage 1, which triggers when it has its columns."""
    body = _body(EARLY["moe_experts.cuh"], " expert_gemm_kernel(")
    assert body.index("tmem_alloc") < body.index("pdl_trigger()")
    for name in ("moe_gather_kernel(", "moe_gather_quant_kernel("):
        gather = _body(EARLY["moe.cu"], " " + name)
        assert gather.index("pdl_wait()") < gather.index("pdl_trigger()")


def test_every_kernel_with_tensor_memory_that_starts_early_is_checked_above():
    """A source that both triggers and allocates is one of those four (gemm_cta_main's users share its body)."""
    both = {n for n, t in EARLY.items() if "pdl_trigger" in t and "tmem_alloc" in t}
    assert both == {"gemm_skinny.cu", "moe_experts.cuh", "ring_attention_tc.cu"}
