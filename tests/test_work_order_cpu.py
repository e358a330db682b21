"""The blend's work order (csrc/fhtgs_order.h), compiled with g++ alone: the two order kernels
restated (count the decisions, scan the buckets, write each tile at its reserved place) around the
header's own places.  Whatever the decisions, every tile must be in the list exactly once, whole or
as its two halves, the periphery and quarter tiles in items of four and sixteen without a gap, and
longer buckets first.  The place of a tile depends only on the decision that was counted: the
scatter kernel takes it from memory and estimates nothing again, since an estimate that rounded
differently there would overrun a run and leave a slot with an item word of an earlier frame."""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "foveatedhtgscudabackend_b200", "csrc")
BUCKETS = 130

WRAPPER = r"""
#include <vector>
#include "fhtgs_order.h"
using namespace fhtgs;
// n tiles with their decision words and packed view/index words, written in the given order.
// totals: block items, periphery entries, quarter entries
extern "C" void order(const uint16_t* word, const uint32_t* packed, const int* sequence, int n, uint32_t* out,
                      uint32_t* runs, uint32_t* totals) {
    std::vector<uint32_t> hist(kOrderBuckets), base(kOrderBuckets), cursor(kOrderBuckets);
    for (int i = 0; i < n; ++i)
        if (word[i] != kOrderSplit) hist[order_bucket(word[i])] += order_entries(word[i]);
    uint32_t all = 0;
    for (int b = kOrderBuckets - 1; b >= 0; --b) { base[b] = all; all += hist[b]; }
    const OrderTotals t(base.data(), all);
    totals[0] = t.items(); totals[1] = t.low; totals[2] = t.quarter;
    for (int s = 0; s < n; ++s) {
        const int i = sequence[s];
        if (word[i] == kOrderSplit) continue;
        const int b = order_bucket(word[i]);
        const uint32_t at = base[b] + cursor[b];
        cursor[b] += order_entries(word[i]);
        t.put(word[i], at, packed[i], out, runs);
    }
}
"""


@pytest.fixture(scope="module")
def order(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    src = d / "order.cpp"
    src.write_text(WRAPPER)
    so = d / "liborder.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I" + CSRC, str(src), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    u16, u32, i32 = (np.ctypeslib.ndpointer(t, flags="C") for t in (np.uint16, np.uint32, np.int32))
    lib.order.argtypes = [u16, u32, i32, C.c_int, u32, u32, u32]
    return lib.order


@pytest.mark.parametrize("counts", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (3, 5, 17), (200, 0, 31),
                                    (0, 333, 16), (150, 400, 700)])
@pytest.mark.parametrize("spread", [1, 3, BUCKETS])
@pytest.mark.parametrize("split", [False, True])
def test_every_tile_once_longest_first(order, counts, spread, split):
    rng = np.random.default_rng(sum(counts) * 7 + spread)
    cls = np.repeat([2, 1, 0], counts)
    n = len(cls)
    bucket = rng.integers(BUCKETS - spread, BUCKETS, n) if spread < BUCKETS else rng.integers(0, BUCKETS, n)
    halves = (rng.random(n) < 0.4) & (cls > 0)
    alone = (rng.random(n) < 0.3) & (cls == 0)  # quarter tiles that a warp blends alone: entries of low items
    word = (np.where(alone, 1, cls) * BUCKETS + bucket + (halves << 15) + (alone << 14)).astype(np.uint16)
    gone = split & (cls == 2) & (rng.random(n) < 0.3)
    word[gone] = 0xFFFF
    index = np.concatenate([np.arange(counts[0]), np.arange(counts[1] + counts[2])]).astype(np.uint32)
    packed = (rng.integers(0, 255, n).astype(np.uint32) << 21) | index
    key = {(c == 2, int(p)): i for i, (c, p) in enumerate(zip(cls, packed))}
    out, runs, totals = (np.full(2 * n + 8, 0xFFFFFFFF, np.uint32), np.full(2 * n + 8, 0xFFFFFFFF, np.uint32),
                         np.zeros(3, np.uint32))
    order(word, packed, rng.permutation(n).astype(np.int32), n, out, runs, totals)
    n_items, n_low, n_quarter = (int(x) for x in totals)
    assert (out[n_items:] == 0xFFFFFFFF).all() and (runs[n_low + n_quarter:] == 0xFFFFFFFF).all()

    seen = []
    def tile(entry, full):
        kind, p = int(entry) >> 29, int(entry) & ((1 << 29) - 1)
        i = key[(full, p)]
        seen.append((i, kind))
        return i
    run_bucket = [bucket[tile(e, False)] for e in runs[:n_low + n_quarter]]
    for part in (run_bucket[:n_low], run_bucket[n_low:]):
        assert all(a >= b for a, b in zip(part, part[1:]))
    items, last, numbers = out[:n_items], BUCKETS, {3: [], 4: []}
    for w in items:
        kind = int(w) >> 29
        if kind < 3:
            b = bucket[tile(w, True)]
        else:
            k = int(w) & ((1 << 29) - 1)
            numbers[kind].append(k)
            b = run_bucket[4 * k] if kind == 3 else run_bucket[n_low + 16 * k]
        assert b <= last, "a longer bucket after a shorter one"
        last = b
    assert numbers[3] == list(range(-(-n_low // 4))) and numbers[4] == list(range(-(-n_quarter // 16)))
    want = [(i, k) for i in range(n) if not gone[i] for k in ((1, 2) if halves[i] else (4,) if alone[i] else (0,))]
    assert sorted(seen) == want


def test_scatter_takes_the_counted_decision():
    src = open(os.path.join(CSRC, "fhtgs_kernels.cuh")).read()
    body = re.search(r"order_scatter_kernel\(FrameParams.*?\n}\n", src, re.S).group(0)
    assert "order_decisions(" in body
    for estimate in ("item_cost(", "blend_halves(", "blend_apart(", "cost_bucket(", "half_threshold("):
        assert estimate not in body, f"the scatter kernel makes its own {estimate}...)"
