"""Rules that a run cannot show to be kept (a kernel that breaks one may still pass every numerics test, until another
kernel lands beside it on an SM), checked on the text of the kernels."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "jitllm_b200" / "csrc"


def _code(path):
    """The source without comments, line breaks kept."""
    text = re.sub(r"/\*.*?\*/", lambda m: "\n" * m.group().count("\n"), path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _function_at(text, start):
    """The body of the function whose definition starts at `start`."""
    open_at = text.index("{", start)
    depth = 0
    for i in range(open_at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[open_at:i + 1]
    raise AssertionError("unbalanced braces")


def _tensor_memory_kernels():
    for path in sorted(CSRC.glob("*.cu")):
        text = _code(path)
        for m in re.finditer(r"__global__", text):
            body = _function_at(text, m.start())
            if "tmem_alloc(" in body or "tcgen05.alloc" in body:
                name = re.search(r"(\w+_kernel)\s*\(", text[m.start():]).group(1)
                yield pytest.param(body, id=f"{path.name}:{name}")


@pytest.mark.parametrize("body", list(_tensor_memory_kernels()))
def test_dependents_are_released_after_the_tensor_memory_is_allocated(body):
    """A dependent kernel's CTA that lands on the SM of a CTA which has not allocated yet could take the tensor memory and
    then wait for that CTA's grid to finish: neither would ever go on."""
    alloc = re.search(r"tmem_alloc\(|tcgen05\.alloc", body).start()
    barrier = body.index("__syncthreads()", alloc)  # the allocating warp has passed it with its columns
    release = [m.start() for m in re.finditer(r"pdl_launch_dependents\(\)", body)]
    assert release and min(release) > barrier


ALIGNED = re.compile(r"tmem_ld16\(|tmem_st16\(|tmem_wait_st\(\)|bar\.sync ")
SPLITS = re.compile(r"lane == 0|tid == 0|mbar_poll_bounded\w*\(|mbar_spin_bounded\(|wait_pair\(|\.inside|\bcontinue;")
JOINS = re.compile(r"__syncwarp\(\)|__all_sync\([^;]*;|__any_sync\([^;]*;|__syncthreads\(\)|cluster_sync_all\(\)")


@pytest.mark.parametrize("name", ["gemm_wide.cu", "attn_prompt_tc.cu"])
def test_warps_are_whole_where_aligned_instructions_stand(name):
    """tcgen05.ld / st / wait and bar.sync are .sync.aligned: executed by a warp that is split, they are undefined. Between
    anything that can split it and the next such instruction stands something that joins it again, in the order of the text."""
    text = _code(CSRC / name)
    places = [m.start() for m in ALIGNED.finditer(text)]
    assert places
    joins = [m.end() for m in JOINS.finditer(text)]
    splits = [m.start() for m in SPLITS.finditer(text)]
    for at in places:
        split = max((s for s in splits if s < at), default=-1)
        assert split < 0 or any(split < j <= at for j in joins), text[:at].count("\n") + 1


def test_a_timeout_clears_every_arrival_counter_with_the_status_word():
    """A launch that gave up leaves its counters partly counted. The status word is therefore reset (but for its
    allocation) in one function only, and that function zeroes each device counter the context holds."""
    text = _code(CSRC / "engine.cu")
    clear = _function_at(text, text.index("cudaError_t clear_after_timeout("))
    resets = re.findall(r"cudaMemset(?:Async)?\(ctx->d_status", text)
    assert len(resets) == len(re.findall(r"cudaMemset(?:Async)?\(ctx->d_status", clear)) + 1  # jl_init
    counters = set(re.findall(r"unsigned \*(\w*count\w*) = nullptr", text))
    assert counters == {"gemm_counters", "att_count", "amax_count"}
    for name in counters:
        assert f"cudaMemsetAsync(ctx->{name}, 0," in clear, name


def test_what_is_on_its_way_is_waited_for_whatever_ended_the_kernel():
    """A launch that gave up leaves in order too: copies into a CTA's shared memory and MMAs on its tensor memory are over
    before the CTA is. The pair's first CTA, on whose barriers the activation boxes of both complete, waits for them behind
    the barrier that both pass when nothing more is issued, and the second stays until it has; the issuing warps wait for
    their last commits without looking at how the loop ended."""
    wide = _code(CSRC / "gemm_wide.cu")
    kernel = _function_at(wide, wide.index("__global__"))
    drain = kernel.index("drain_activations(")
    assert kernel.rindex("cluster_sync_all()", 0, drain) and kernel.index("cluster_sync_all()", drain) < kernel.index("tcgen05.dealloc")
    assert "if (issued > 0) wait_pair(done0" in kernel
    assert re.search(r"\n            for \(int k = i > RS \? i - RS : 0; k < i; \+\+k\) mbar_poll_bounded\(raw_full", kernel)
    attention = _code(CSRC / "attn_prompt_tc.cu")
    for done in ("k_empty", "v_empty"):
        loop = re.search(r"for \(int t = max\(\w+ - 2, 0\); ([^;]*); \+\+t\) ok = mbar_poll_bounded\(" + done, attention)
        assert loop and "ok" not in loop.group(1), done
