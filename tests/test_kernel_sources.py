"""What the kernels' sources have to say for a fault that no run shows: orderings that hold by luck on one device or another (no GPU, no compiler)."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "thintensor_b200" / "csrc"
SOURCES = sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])


def code(path: Path) -> str:
    return re.sub(r"//[^\n]*", "", path.read_text())


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_arrivals_on_another_ctas_barrier_release_what_was_written(path):
    """An arrival without a scope releases to its own CTA only, a wait without one acquires from it only: what a thread of the other CTA wrote before
    it arrived need not be there for whoever waited.  Without release only accumulators that were read are handed back."""
    text = code(path)
    assert set(re.findall(r"mbar_arrive_even_cta\(smem_u32\(&(\w+)\[", text)) <= {"acc_empty"}
    released = set(re.findall(r"mbar_release_even_cta\(smem_u32\(&(\w+)\[", text))
    for bar in released:
        # the issuer sits in the even CTA
        assert re.search(r"mbar_wait<true>\(smem_u32\(&" + bar + r"\[", text) and not re.search(r"mbar_wait\(smem_u32\(&" + bar + r"\[", text), bar
    if path.name == "tcgen05.cuh":
        assert re.search(r"void mbar_release_even_cta\(uint32_t bar\) \{\s*asm volatile\(\"mbarrier\.arrive\.release\.cluster\.shared::cluster\.b64 ", text)
        assert re.search(r"if \(CLUSTER\)\s*asm volatile\((?:(?!else).)*?mbarrier\.try_wait\.parity\.acquire\.cluster\.shared::cta\.b64 ", text, re.S)


def test_rows_cut_by_the_odd_cta_are_released_by_a_thread_that_has_seen_them():
    """In the product in parts a CTA's warps arrive at a barrier of their own CTA; one thread of the odd CTA waits for all of them before it arrives at the
    issuer's barrier."""
    text = code(CSRC / "gemm_split.cu")
    passed_on = re.search(r"rank == 1\) \{(.*?)\n        \}", text, re.S).group(1)
    assert passed_on.index("mbar_wait(smem_u32(&cut_bar") < passed_on.index("mbar_release_even_cta(smem_u32(&full_bar")
    assert text.count("mbar_release_even_cta(") == 1 and "mbar_arrive_even_cta(" not in text
    workers = text[text.index("fence_async_shared();"):]
    assert re.match(r"fence_async_shared\(\);\s*__syncwarp\(\);\s*if \(lane == 0\) mbar_arrive\(smem_u32\(rank \? &cut_bar\[i & 1\] : &full_bar\[i & 1\]\)\);", workers)


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_shared_memory_is_asked_for_on_every_launch(path):
    """What a kernel may have beyond 48 KB holds for the device that was current when it was asked for: nothing remembers for the whole process that it was."""
    text = code(path)
    for ask in re.finditer(r"cudaFuncSetAttribute|tt_allow_shared\(", text):
        function = text[text.rfind("\n}", 0, ask.start()) + 2:ask.start()]
        assert not re.search(r"\bstatic\s+(?:bool|int|size_t)\s+\w+\s*=", function), function[-400:]


def test_no_copy_is_left_on_its_way_when_a_wait_runs_out():
    """A CTA whose wait ran out ends, and its shared memory is the next one's: it fetches nothing more and waits for what it has fetched."""
    text = code(CSRC / "recurrent_chunks.cu")
    for name in ("scan_chunks_kernel", "delta_chunks_kernel"):
        kernel = text[text.index(f"\n{name}(const"):]
        kernel = kernel[:kernel.index("\n}\n")]
        for expect in re.finditer(r"mbar_expect_tx\(", kernel):
            condition = kernel[:expect.start()]
            condition = condition[condition.rindex("if (threadIdx.x"):]
            assert "in_time" in condition, condition
        # every wait that may run out sets the flag, and every barrier is waited for again at the end
        waits = set(re.findall(r"if \(in_time && !tc::mbar_wait\((\w+), chunk & 1\)\) \{ in_time = false; late = ", kernel))
        end = kernel[kernel.rindex("if (!in_time && threadIdx.x == 0)"):]
        assert len(waits) == 2 and all(f"tc::mbar_wait({bar}, " in end for bar in waits)
        assert kernel[:-len(end)].count("tc::mbar_wait(") == len(re.findall(r"in_time && !?tc::mbar_wait\(", kernel))
