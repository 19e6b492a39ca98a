"""How the one-GPU decode step is laid out for a shape, without a GPU: its tables and buffers hold the largest share that the
cut of the matrices gives any thread block or warp."""
import ctypes as C

import numpy as np
import pytest

from exactinfer_b200 import capi, synth

F16, Q8_0, Q4_K, Q6_K = synth.F16, synth.Q8_0, synth.Q4_K, synth.Q6_K
CTAS, SMEM, WARPS = 148, 232448, 15
COST = {Q6_K: 1455, Q8_0: 481, Q4_K: 875, F16: 875}


def plan(shape, types):
    s, t, out = np.array(shape, np.int32), np.array(types, np.int32), np.zeros(25, np.int32)
    p = lambda a: a.ctypes.data_as(C.POINTER(C.c_int32))
    capi.check(capi.lib().elb_selftest_decode_plan(p(s), p(t), CTAS, SMEM, p(out)))
    return {"parts": int(out[0]), "ring": int(out[1]), "slots": int(out[2]), "kept": int(out[3]),
            "table": [int(v) for v in out[4:14]] + [int(out[24])], "slot": [int(v) for v in out[14:24]]}


def qkv_shares(shape, types):
    """tiles[i] = (units per tile, first tile and number of tiles of matrix i that every thread block gets): tile t of q, k, v in
    that order starts at the sum of the costs in front of it; block c takes what starts in [C c / G, C (c + 1) / G)."""
    E, _, H, HKV, _ = shape
    rows = [H * 128, HKV * 128, HKV * 128]
    upt = [E // (256 if t in (Q4_K, Q6_K) else 128) for t in types[:3]]
    tiles = [r // 16 for r in rows]
    at, total, G = 0, sum(COST[t] * u * n for t, u, n in zip(types, upt, tiles)), min(CTAS, sum(tiles))
    edges = np.array([total * c // G for c in range(G + 1)])
    out = []
    for t, u, n in zip(types, upt, tiles):
        start = at + COST[t] * u * np.arange(n)
        at += COST[t] * u * n
        first = np.searchsorted(start, edges[:-1], "left")
        out.append((u, first, np.searchsorted(start, edges[1:], "left") - first))
    return out


MIXED, SAME = (Q6_K, Q4_K, Q6_K, Q4_K, Q4_K, Q6_K, Q6_K), (Q4_K,) * 7


@pytest.mark.parametrize("shape,types,beyond", (
    ((2048, 6144, 96, 12, 512), MIXED, True),     # a block with tiles of k alone: more than three times k's share by count
    ((2048, 6144, 128, 16, 512), MIXED, True),
    ((2048, 6144, 160, 40, 512), SAME, False),
    ((2560, 9728, 32, 8, 151936), (Q4_K, Q4_K, Q6_K, Q4_K, Q4_K, Q6_K, Q6_K), False),
    ((5120, 25600, 64, 8, 151936), (Q4_K, Q4_K, Q6_K, Q4_K, Q4_K, Q6_K, Q6_K), False),
    ((1024, 3072, 16, 8, 151936), (F16,) * 7, False),
    ((256, 512, 2, 1, 64), (Q8_0,) * 7, False)))
def test_tables_hold_the_largest_share(shape, types, beyond):
    got = plan(shape, types)
    assert got["parts"] >= 1
    room = [b - a for a, b in zip(got["table"], got["table"][1:])]
    slot_end = got["slot"][1:3] + [got["slots"]]
    past = False
    for i, (upt, first, count) in enumerate(qkv_shares(shape, types)):
        assert room[i] >= count.max(), f"matrix {i}: {count.max()} row tiles of one thread block, room for {room[i]}"
        by_count = -(-(shape[2 if i == 0 else 3] * 8) // CTAS)
        past = past or count.max() > 3 * (by_count + 2)
        units = count[:, None] * upt * np.arange(WARPS + 1) // WARPS  # a warp's units of the block's, in tiles it touches
        touched = np.where(units[:, 1:] > units[:, :-1], (units[:, 1:] - 1) // upt - units[:, :-1] // upt + 1, 0)
        assert slot_end[i] - got["slot"][i] >= max(1, touched.max())
    assert past == beyond  # (the cases that a size from the matrix's own share would not cover)


@pytest.mark.parametrize("n_ff,layout,parts", ((9728, Q4_K, 1), (25600, Q4_K, 2), (25600, Q6_K, 2), (25600, Q8_0, 2), (25600, F16, 1),
                                               (28672, F16, 2), (57344, Q4_K, 4), (57344, F16, 4)))
def test_parts_of_a_long_feed_forward_vector(n_ff, layout, parts):
    """The lengths that the GPU tests take do make the step work in that many parts."""
    got = plan((256, n_ff, 2, 1, 640), (layout,) * 7)
    assert got["parts"] == parts and got["ring"] >= 8192


def test_shape_that_does_not_fit_is_refused():
    assert plan((256, 256 * 1009, 2, 1, 640), (F16,) * 7)["parts"] == 0  # (1009 is a prime: no equal parts)
    assert plan((2048, 6144, 256, 32, 512), SAME)["parts"] == 0           # (32768 attention outputs beside the rings)
