"""Order of the fit kernels' shared-memory accesses, on the CPU: the barriers
and accesses are read from the kernels' source in textual order and replayed
on a model of the threads that share the memory.  Two accesses of one place by
different threads are ordered when a barrier of both lies between them; the
model counts the barriers passed."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "periodsearch_gb300" / "csrc" / "ps_fit.cuh").read_text()


def body(name: str) -> str:
    """The text of function `name`, comments removed."""
    text = re.sub(r"//[^\n]*", "", SOURCE)
    at = re.search(r"\b" + name + r"\([^;{}]*\)\s*\{", text).end()
    depth, end = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return text[at:end]


@pytest.mark.parametrize("chunks", [1, 2, 3, 4])
def test_cluster_chi2_buffers(chunks):
    """chi2_fp64 of a cluster, called again and again (rejected steps): a CTA's
    stores into another CTA's model values lie a cluster barrier after that
    CTA's reads of the same buffer."""
    text = body("chi2_fp64")
    loop, tail = text.split("while (q0 < N)")[1], text.rsplit("buf ^= 1;", 1)[1]
    kinds = {"first": r"if \(first\) cgr::this_cluster\(\)\.sync\(\)",
             "every": r"if constexpr \(SPLIT\) cgr::this_cluster\(\)\.sync\(\)",
             "store": r"map_shared_rank\(ym", "read": r"double \*y = ym"}
    order = [k for _, k in sorted((m.start(), k) for k, pat in kinds.items() for m in re.finditer(pat, loop))]
    assert [order.count(k) for k in ("every", "store", "read")] == [1, 1, 1] and "chain(" in loop and "chain(" in tail
    passed = 0                  # cluster barriers
    last_read = {0: -1, 1: -1}  # barriers passed before the latest read of a buffer
    for _ in range(3):          # calls
        buf = 0
        for c in range(chunks):
            for e in order:
                if e == "store":
                    assert last_read[buf] < passed, f"chunk {c}: a store may meet the reads of buffer {buf}"
                elif e == "read":
                    last_read[buf] = passed
                elif e == "every" or c == 0:
                    if c and e == "every":
                        last_read[buf ^ 1] = passed   # the chain over the chunk before
                    passed += 1
            buf ^= 1
        last_read[buf ^ 1] = passed   # the last chain


def test_cluster_started_before_remote_access():
    """A CTA's shared memory may be reached by the others of its cluster once
    it has started: a cluster barrier comes before the first remote access (of
    an evaluation: the barrier of its first round of tiles)."""
    for text in (body("fit_kernel_split"), body("evaluate_fp64").split("auto flush_round")[1]):
        assert 0 <= text.find(".sync()") < text.index("map_shared_rank")


def test_pivot_flags_of_the_solve():
    """cholesky_solve: a step's pivot flag is read behind the barrier that ends
    the step, when warp 0 may already store the next step's: not in its place,
    and in no place before another barrier has passed."""
    loop = body("cholesky_solve").split("for (int j = 0; j + 2 < n; j += 2)")[1]
    store = re.search(r"chol_pivot_block<NT>\(([^;]*)\);", loop).group(1).split(", ", 12)[12].rsplit(",", 1)[0]
    barrier = loop.index("team_sync<NT>()")
    read = re.search(r"if \(\*(.*) == 0\) return 2;", loop[barrier:]).group(1)
    rule = re.search(r"int \*pivot_flag\(int \*flags, int j\) \{ return (.*); \}", SOURCE)

    def place(expr, jn):
        return eval(rule.group(1), {"flags": 0, "j": jn}) if rule and expr == "pivot_flag(flags, jn)" else 0

    reads = {}
    for step, jn in enumerate(range(2, 40, 2)):
        reads[step] = place(read, jn)
        assert place(store, jn) == reads[step]
        assert step == 0 or place(store, jn) != reads[step - 1]


def test_chunks_of_the_mixed_chi2_pass():
    """chi2_mixed takes a relative lightcurve whole, and its chunk loop passes
    one that does not fit never: the smallest operand region of any layout, and
    the sums of a chunk's tiles, hold the longest lightcurve that is accepted."""
    header = (Path(__file__).resolve().parent.parent / "include" / "ps_gb300.h").read_text()
    longest = int(re.search(r"#define PS_POINTS_MAX (\d+)", header).group(1))
    engine = (Path(__file__).resolve().parent.parent / "periodsearch_gb300" / "csrc" / "ps_engine.h").read_text()
    region = re.search(r"size_t readback = (.*) \* sizeof\(float\);", engine).group(1)
    assert re.search(r"kChi2Bytes = (.*) \* sizeof\(float\);", SOURCE).group(1) == region
    assert "static_assert(kChi2Points >= PS_POINTS_MAX" in SOURCE
    assert (eval(region) * 4 // 32 & ~31) >= longest
    tiles = 16 * int(re.search(r"kRedStride = (\d+);", engine).group(1))
    assert tiles * 32 >= longest
