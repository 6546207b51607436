"""What the tensor-core kernels' barrier waits have to keep to, read from the sources: neither undefined behaviour nor a CTA that
leaves too early can be shown by running them.

tcgen05.ld / st, shuffles and __syncwarp need all lanes of a warp at the same instruction, and mbar_wait() lets them leave, or
give up, one by one.  Only the branch of one elected thread may call it; everything else goes through mbar_wait_warp().

A role that has given up waits for the copies it has issued before the CTA frees its memory."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm-scaler_b200", "csrc")
KERNELS = sorted(f for f in os.listdir(CSRC) if f.startswith("umma_") and f.endswith(".cu"))


def _per_lane_waits(text):
    """Line numbers of mbar_wait() calls that no enclosing block's head restricts to one thread."""
    text = re.sub(r"//[^\n]*", "", text)
    heads, start, found = [], 0, []
    for m in re.finditer(r"[{};]|\bmbar_wait\(", text):
        tok = m.group()
        if tok == "{":
            heads.append(text[start:m.start()])
        elif tok == "}":
            heads.pop()
        elif tok != ";":
            if not any(re.search(r"elect_one\(\)|_selftest_kernel", h) for h in heads):
                found.append(text.count("\n", 0, m.start()) + 1)
            continue
        start = m.end()
    return found


def test_the_reader_sees_both_forms():
    assert _per_lane_waits("if (elect_one()) { while (x) { if (!mbar_wait(a)) break; } }") == []
    assert _per_lane_waits("if (lane == 0) {\n mbar_wait(a);\n}\nelse { ok = mbar_wait_warp(b); }") == [2]


@pytest.mark.parametrize("name", KERNELS)
def test_whole_warps_wait_together(name):
    with open(os.path.join(CSRC, name)) as f:
        assert _per_lane_waits(f.read()) == []


@pytest.mark.parametrize("name", KERNELS)
def test_copies_in_flight_are_waited_for(name):
    with open(os.path.join(CSRC, name)) as f:
        kernels = f.read().split("__global__ ")[1:]
    for text in kernels:
        # one drain per elected producer, one wait behind asynchronous copies that arrive on a barrier
        producers = sum(bool(re.search(r"\btma_load_2d(_pair)?\(", part)) for part in text.split("if (elect_one()) {")[1:])
        assert text.count("drain_issued(") == producers
        assert ("cp_async_arrive(" in text) == ("cp_async_wait_all()" in text)


STREAMS = ["w4_stream.cu", "w8_stream.cu"]


@pytest.mark.parametrize("name", STREAMS)
def test_streaming_kernels_wait_together_and_for_their_copies(name):
    with open(os.path.join(CSRC, name)) as f:
        source = f.read()
    assert _per_lane_waits(source) == []
    for text in source.split("__global__ ")[1:]:
        assert text.count("drain_issued(") == sum("tma_load_2d(" in part for part in text.split("if (elect_one()) {")[1:]) == 1
        assert "cp_async_arrive(" in text and "cp.async.wait_all" in text


def _unconverged_barriers(text):
    """Line numbers of aligned block barriers in front of which, since the last statement that a whole warp executes together, only
    some of its lanes did something."""
    text = re.sub(r"//[^\n]*", "", text)
    found = []
    for m in re.finditer(r'asm volatile\("bar\.sync', text):
        before = text[:m.start()]
        lanes = max((x.end() for x in re.finditer(r"\bif \((?:\w+ && )?lane (?:==|<) \w+\)", before)), default=-1)
        together = max((x.end() for x in re.finditer(r"__syncwarp\(\)|__syncthreads\(\)|_sync\(0x|mbar_wait_warp\w*\(|bar\.sync", before)), default=-1)
        if lanes > together:
            found.append(text.count("\n", 0, m.start()) + 1)
    return found


def test_the_reader_sees_lanes_on_their_own():
    assert _unconverged_barriers('if (lane == 0) a = b;\n__syncwarp();\nasm volatile("bar.sync 1, 64;");') == []
    assert _unconverged_barriers('__syncwarp();\nif (lane == 0) a = b;\nasm volatile("bar.sync 1, 64;");') == [3]


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_whole_warps_meet_at_aligned_barriers(name):
    """bar.sync is the aligned form: all lanes of a warp have to execute it together."""
    with open(os.path.join(CSRC, name)) as f:
        assert _unconverged_barriers(f.read()) == []


def _read_only_loads(text):
    """In kernels that begin while the one in front is running: places where a const __restrict__ pointer is read by a plain
    dereference, which the compiler may turn into a load by the read-only path."""
    text, found = re.sub(r"//[^\n]*", "", text), []
    for m in re.finditer(r"__global__ (.*?)\n}\n", text, re.S):
        body = m.group(1)
        if re.search(r"grid_dep_wait\(\)|dep_enter\(\)", body):
            for d in re.finditer(r"\*reinterpret_cast<const uint[24]\*>\((?!out \+|t\[|&)|\*n_valid|\bidx\[|\b[xz]r\[|\bw\[k\]", body):
                found.append(text.count("\n", 0, m.start(1) + d.start()) + 1)
    return found


def test_the_reader_sees_plain_dereferences():
    assert _read_only_loads("__global__ void f(const void* __restrict__ x) {\n  dep_enter();\n  a = *reinterpret_cast<const uint4*>(row + k);\n}\n") == [3]
    assert _read_only_loads("__global__ void f(const void* __restrict__ x) {\n  dep_enter();\n  a = ld_shared_vec(row + k);\n}\n") == []


def test_kernels_that_start_early_read_their_inputs_by_ordinary_loads():
    """The read-only path promises that nothing is written while the kernel runs, and these run while their inputs are written."""
    with open(os.path.join(CSRC, "moe_aux.cu")) as f:
        assert _read_only_loads(f.read()) == []


# Stages that warps read by ordinary loads, and that somebody overwrites after their arrival.  The loads of the tcgen05 kernels' raw
# stages feed tensor-memory stores that are waited for in front of the arrival.
READ_STAGES = {"w4_stream.cu": ["empty", "sc_empty"], "w8_stream.cu": ["empty"], "umma_w4.cu": ["sc_empty"]}


@pytest.mark.parametrize("name", sorted(READ_STAGES))
def test_a_stage_is_released_behind_its_loads(name):
    """mbar_arrive() alone lets the last loads of a stage pass the arrival; mbar_arrive_read() fences them."""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for bar in READ_STAGES[name]:
        assert len(re.findall(r"\bmbar_arrive_read\(%s \+" % bar, text)) == 1
        assert not re.search(r"\bmbar_arrive\(%s \+" % bar, text)
    with open(os.path.join(CSRC, "sm100.cuh")) as f:
        body = re.search(r"void mbar_arrive_read\(uint32_t bar\) \{(.*?)\n\}", f.read(), re.S).group(1)
    assert body.index("fence.acq_rel.cta") < body.index("__syncwarp()") < body.index("mbar_arrive(bar)")


@pytest.mark.parametrize("name", ["umma_gemm.cu", "umma_w4.cu", "umma_w4_i8.cu"])
def test_raw_stages_are_released_behind_the_stores_that_they_feed(name):
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    at = text.index("mbar_arrive(raw_empty +")
    assert max(text.rfind("lds128(", 0, at), text.rfind("lds32(", 0, at)) < text.rfind("tmem_st_wait()", 0, at)
