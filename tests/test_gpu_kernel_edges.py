"""Kernels and dispatch branches at the sizes where they can go wrong (edges of tiles, remainders, smallest and largest
of a range), through the public entry points, against the CPU oracle or the host's own arithmetic."""
import numpy as np
import pytest

import oracle_lib as ol
from exactinfer_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def elb():
    import exactinfer_b200 as e
    ok, why = e.cuda_available()
    assert ok, f"CUDA path unavailable: {why}"
    return e


# vectors shorter than the split kernel's cluster, a ragged cut over it, and one past what its registers hold
@pytest.mark.parametrize("n", (256, 256 * 9, 32768, 32768 + 256))
def test_split_of_one_vector_over_a_cluster(elb, n):
    rng = np.random.default_rng(n)
    wb = synth.rand_weight(rng, synth.Q4_K, 16, n)
    x = rng.normal(size=n).astype(np.float32)
    w = elb.Weight(synth.Q4_K, 16, n, wb)
    P, I, J = w.limb_sums(x, 4)
    limbs, _, _ = ol.split_limbs(x, 4)
    assert np.array_equal(P, ol.limb_partials(synth.Q4_K, 16, n, wb, limbs))
    wI, wJ = ol.limb_block_sums(synth.Q4_K, 16, n, wb, limbs)
    assert np.array_equal(I, wI) and np.array_equal(J, wJ)


def test_operator_scratch_is_reused_and_given_back(elb):
    """The scratch of the operator calls is kept between calls and freed with the last weight."""
    import ctypes as C
    from exactinfer_b200 import capi

    def free():
        f, t = C.c_size_t(), C.c_size_t()
        capi.check(capi.lib().elb_device_mem_info(0, C.byref(f), C.byref(t)))
        return f.value

    rng = np.random.default_rng(1)
    before = free()
    w = elb.Weight(synth.Q8_0, 64, 256, synth.rand_weight(rng, synth.Q8_0, 64, 256), planes=True)
    x = rng.normal(size=(40, 256)).astype(np.float32)
    y = w.matmul(x)
    held = free()
    for b in (40, 3, 17, 40):
        assert np.array_equal(w.matmul(x[:b]).shape, (b, 64))
    assert np.array_equal(w.matmul(x), y) and free() == held
    w.close()
    assert free() >= before


def test_operator_scratch_of_a_failed_call_is_not_kept(elb):
    """A call that fails behind a launch has not waited for it: its scratch is freed, which does, and not given to the next."""
    import ctypes as C
    from exactinfer_b200 import capi

    def free():
        f, t = C.c_size_t(), C.c_size_t()
        capi.check(capi.lib().elb_device_mem_info(0, C.byref(f), C.byref(t)))
        return f.value

    rng = np.random.default_rng(2)
    w = elb.Weight(synth.Q4_K, 64, 4096, synth.rand_weight(rng, synth.Q4_K, 64, 4096))  # no digit planes: refused behind the split
    x, y = C.c_void_p(), C.c_void_p()
    capi.check(capi.lib().elb_malloc(0, 512 * 4096 * 4, C.byref(x)))
    capi.check(capi.lib().elb_malloc(0, 512 * 64 * 4, C.byref(y)))
    capi.check(capi.lib().elb_memcpy_h2d(x, rng.normal(size=512 * 4096).astype(np.float32).ctypes.data_as(C.c_void_p), 512 * 4096 * 4))
    w.matvec(np.zeros(4096, np.float32))
    before = free()
    for _ in range(3):
        assert capi.lib().elb_matmul_dev(w._h, x, 512, y, 4) == capi.ERR_STATE
    assert free() == before  # 8 MB of limbs otherwise
    for p in (x, y):
        capi.check(capi.lib().elb_free(p))
    w.close()


def test_idle_operator_scratch_gives_way(elb):
    """Buffers, weights and models get the memory that lies idle in the operators' scratch."""
    import ctypes as C
    from exactinfer_b200 import capi

    def free():
        f, t = C.c_size_t(), C.c_size_t()
        capi.check(capi.lib().elb_device_mem_info(0, C.byref(f), C.byref(t)))
        return f.value

    MB = 1 << 20
    rng = np.random.default_rng(3)
    w = elb.Weight(synth.Q8_0, 64, 4096, synth.rand_weight(rng, synth.Q8_0, 64, 4096), planes=True)
    x = rng.normal(size=(8192, 4096)).astype(np.float32)
    spec = synth.Spec(name="small", n_layer=1, n_embd=256, n_ff=512, n_head=2, n_head_kv=1, n_vocab=512, layout="q8_0")
    tens = list(synth.generate(spec, 3))
    big = synth.rand_weight(rng, synth.Q8_0, 1024, 16384)

    def short_of_memory(left):  # the scratch holds 128 MB or more, about `left` MB are free beside it
        w.matmul(x)
        hold = C.c_void_p()
        capi.check(capi.lib().elb_malloc(0, (free() - left * MB) // (2 * MB) * (2 * MB), C.byref(hold)))
        assert free() < (left + 8) * MB
        return hold

    hold, buf = short_of_memory(40), C.c_void_p()
    capi.check(capi.lib().elb_malloc(0, 100 * MB, C.byref(buf)))
    for p in (buf, hold):
        capi.check(capi.lib().elb_free(p))
    hold = short_of_memory(40)
    elb.Weight(synth.Q8_0, 1024, 16384, big, planes=True).close()  # 17 MB, tiled 17 MB, planes 16 MB or pairs 64 MB
    capi.check(capi.lib().elb_free(hold))
    hold = short_of_memory(240)
    m = elb.Backend(spec, tens, 40000)  # 45 MB for the model's own count, and it wants 256 MB beside that
    assert np.isfinite(m.eval(np.array([1], np.int32), 0)).all()
    m.close()
    capi.check(capi.lib().elb_free(hold))
    w.close()


# vocabularies below, at and just past a chunk of the reduction (2560 logits), and of several chunks
@pytest.mark.parametrize("vocab", (64, 2559, 2560, 2561, 7681))
def test_top_tokens_at_chunk_edges(elb, vocab):
    spec = synth.Spec(name="small", n_layer=1, n_embd=256, n_ff=512, n_head=4, n_head_kv=2, n_vocab=vocab, layout="q8_0",
                      head_sigma=1e-4)
    tens = list(synth.generate(spec, vocab))
    role, layer, t, rows, n, emb = tens[0]
    emb[vocab // 2:vocab // 2 + 20] = emb[0]  # equal rows of the tied head: equal logits, the lower id comes first
    gpu = elb.Backend(spec, tens, 40, n_seq=3)
    toks = np.array([5, 9, 11], np.int32)
    for k in (1, 33, 64):
        full = gpu.eval_batch(toks, [0, 1, 2], [0, 0, 0])
        ids, vals, lse = gpu.eval_batch_top(toks, [0, 1, 2], [0, 0, 0], k=k)
        for r in range(3):
            order = np.lexsort((np.arange(vocab), -full[r].astype(np.float64)))[:k]
            assert np.array_equal(ids[r], order) and np.array_equal(vals[r], full[r][order])
            assert abs(lse[r] - ol.logsumexp(full[r])) <= 1e-12 * max(1.0, abs(lse[r]))
    gpu.close()


# rows of logits that a broken model gives: one chunk of the reduction (and a part of one) without any finite logit
@pytest.mark.parametrize("lo,hi", ((2560, 5120), (0, 2560), (7680, 7681), (100, 200)))
@pytest.mark.parametrize("what", ("nan", "-inf", "both"))
def test_log_sum_exp_with_nan_and_infinity(elb, lo, hi, what):
    spec = synth.Spec(name="small", n_layer=1, n_embd=256, n_ff=512, n_head=4, n_head_kv=2, n_vocab=7681, layout="f16", head_sigma=1e-2)
    tens = list(synth.generate(spec, 5))
    tok = np.array([6000], np.int32)

    def logits_with(inf):  # one weight of the rows is +-infinity or NaN, the others are 0
        role, layer, t, rows, n, emb = tens[0]
        half = emb.copy().view(np.uint16).reshape(rows, n)
        half[lo:hi] = 0
        half[lo:hi, 0] = 0x7E00 if what == "nan" else inf
        if what == "both":
            half[lo:hi:2, 0] = 0x7E00
        gpu = elb.Backend(spec, [(role, layer, t, rows, n, half.view(np.uint8).reshape(rows, -1))] + tens[1:], 8)
        full = gpu.eval(tok, 0)
        return (full.copy(), *gpu.eval_top(tok, 0, k=5))

    for inf in (0x7C00, 0xFC00):  # (the sign of the activation decides which of them gives -infinity)
        full, ids, vals, lse = logits_with(inf)
        if not np.isposinf(full).any():
            break
    bad = full[lo:hi]
    assert (np.isnan(bad) if what == "nan" else np.isneginf(bad) if what == "-inf" else ~np.isfinite(bad)).all()
    assert np.isfinite(np.delete(full, np.s_[lo:hi])).all()
    if what == "-inf":
        want = ol.logsumexp(full)
        assert np.isfinite(want) and abs(lse - want) <= 1e-12 * max(1.0, abs(want))
    else:
        assert np.isnan(lse)
    order = np.argsort(-np.where(np.isnan(full), -np.inf, full).astype(np.float64), kind="stable")[:5]
    assert np.array_equal(ids, order) and np.array_equal(vals, full[order])


def runs_on(gpu, barrier_kernel=False):
    """Which of the two persistent kernels a model's single steps run on (only the one-GPU kernel has exchange buffers)."""
    from exactinfer_b200 import capi
    rc = capi.lib().elb_selftest_decode_exchange(gpu._h, 0)
    return rc == (capi.ERR_STATE if barrier_kernel else capi.OK)


def decode_pair(elb, spec, seed, n_ctx, walk, barrier_kernel=False):
    """Single-token evaluations at the positions of `walk` (rows in front of them filled by prompt chunks), against the
    CPU oracle on the same cache contents; every evaluation twice, which must give the same bits."""
    tens = list(synth.generate(spec, seed))
    gpu, cpu = elb.Backend(spec, tens, n_ctx), ol.OracleModel(spec, tens, n_ctx)
    assert runs_on(gpu, barrier_kernel)
    toks = synth.lcg_tokens(n_ctx, spec.n_vocab, seed)
    filled, worst = 0, 0.0
    for pos in walk:
        if pos > filled:
            gpu.eval(toks[filled:pos], filled, want_logits=False)
            cpu.eval(toks[filled:pos], filled)
            filled = pos
        a, b = gpu.eval(toks[pos:pos + 1], pos), cpu.eval(toks[pos:pos + 1], pos)
        assert gpu.last_eval_stats()[1] == 1, "the persistent kernel must run"
        assert np.array_equal(a, gpu.eval(toks[pos:pos + 1], pos)), "deterministic"
        worst = max(worst, float(np.abs(a - b).max() / np.abs(b).max()))
        filled = max(filled, pos + 1)
    gpu.close()
    cpu.close()
    return worst


# attention splits of 60 keys: one, two, many, back to one, many again; every group size of query heads the kernel is
# compiled for; all-F16 and quantized weights; an odd number of layers
@pytest.mark.parametrize("layout,heads,kv", (("q4_k_m", 8, 4), ("f16", 6, 2), ("q8_0", 8, 1), ("q6_k", 2, 2)))
def test_decode_across_attention_splits(elb, layout, heads, kv):
    spec = synth.Spec(name="small", n_layer=3, n_embd=512, n_ff=768, n_head=heads, n_head_kv=kv, n_vocab=1111, layout=layout,
                      head_sigma=2e-5)
    assert decode_pair(elb, spec, 31, 700, (0, 59, 60, 61, 650, 3, 651, 120)) <= 2e-4


# the grid-barrier kernel, which tensor-parallel models run on, on one GPU: block formats, group sizes, split counts, a
# feed-forward activation in global memory, and a cut of q|k|v that gives a thread block many more tiles of k than its share
@pytest.mark.parametrize("layout,heads,kv,n_ff", (("q4_k_m", 8, 4, 768), ("q8_0", 8, 1, 768), ("q6_k", 2, 2, 768), ("q4_k_m", 2, 1, 25600)))
def test_barrier_decode_kernel_on_one_gpu(elb, monkeypatch, layout, heads, kv, n_ff):
    monkeypatch.setenv("ELB_DK_OLD", "1")
    spec = synth.Spec(name="small", n_layer=3, n_embd=512, n_ff=n_ff, n_head=heads, n_head_kv=kv, n_vocab=1111, layout=layout,
                      head_sigma=2e-5)
    assert decode_pair(elb, spec, 33, 700, (0, 59, 60, 61, 650, 3, 651, 120), barrier_kernel=True) <= 2e-4


# single evaluations at long and short contexts in turn, with an odd and an even number of short ones in between: what a step
# with several key splits leaves in the exchange buffers must not be taken for a later step's, whatever the number of layers
@pytest.mark.parametrize("n_layer", (1, 2, 3, 5))
def test_decode_long_and_short_contexts_in_turn(elb, n_layer):
    spec = synth.Spec(name="small", n_layer=n_layer, n_embd=512, n_ff=768, n_head=8, n_head_kv=2, n_vocab=640, layout="q8_0",
                      head_sigma=2e-5)
    tens = list(synth.generate(spec, 41))
    gpu, cpu = elb.Backend(spec, tens, 704), ol.OracleModel(spec, tens, 704)
    toks = synth.lcg_tokens(704, spec.n_vocab, 41)
    gpu.eval(toks[:700], 0, want_logits=False)
    cpu.eval(toks[:700], 0)
    walk = (650, 5, 651, 7, 8, 9, 100, 5, 699, 5, 6, 650, 59, 60, 59, 61, 58, 400)
    seen = {}
    for pos in sorted(set(walk)):  # (upwards first: a row of the cache then is what a single step writes, and stays so)
        seen[pos], want = gpu.eval(toks[pos:pos + 1], pos), cpu.eval(toks[pos:pos + 1], pos)
        assert gpu.last_eval_stats()[1] == 1, "the persistent kernel must run"
        assert np.abs(seen[pos] - want).max() <= 2e-4 * np.abs(want).max(), pos
    for _ in range(60):
        for pos in walk:
            assert np.array_equal(gpu.eval(toks[pos:pos + 1], pos), seen[pos]), pos
    gpu.close()
    cpu.close()


# keys whose score is -infinity for some query heads of a KV head and finite for the others: probability 0 for the former, the
# latter as ever. The first keys, so that a warp's first tile has nothing else; alone in a tile; and behind finite ones.
@pytest.mark.parametrize("special", ((0, 1, 2, 3), (0, 1, 2, 3, 4, 5, 6, 7, 8), (2,), (12, 13, 14, 15), (33, 34, 35, 36, 37, 38, 39)))
def test_attention_scores_of_minus_infinity(elb, special):
    spec = synth.Spec(name="small", n_layer=1, n_embd=256, n_ff=512, n_head=8, n_head_kv=1, n_vocab=512, layout="f16", head_sigma=2e-2)
    rng, tens = np.random.default_rng(8), []
    odd = 400  # the token of those keys: the only one with a value in column 7
    for role, layer, t, rows, n, data in synth.generate(spec, 51):
        if role in ("attn_q_norm", "attn_k_norm"):  # (dimension 63 is turned the least by the rotation)
            data = data.copy().view(np.float32)
            data[0, 63] = 1e10 if role == "attn_q_norm" else 1e30
            data = data.view(np.uint8)
        elif role in ("token_embd", "attn_q", "attn_k"):
            w = data.copy().view(np.float16).reshape(rows, n)
            if role == "token_embd":
                w[:, 7] = 0
                w[odd, 7] = 0.05
                w[:, 3] = 0.05
            elif role == "attn_k":  # k[63] > 0 for that token, 0 for the others
                w[63] = 0
                w[63, 7] = 0.1
            else:                   # q[63] < 0 in heads 0..3; 0 there and in its partner of the rotation in heads 4..7
                for h in range(8):
                    w[h * 128 + 63] = w[h * 128 + 127] = 0
                    w[h * 128 + 63, 3] = -0.1 if h < 4 else 0
            data = w.view(np.uint8).reshape(rows, -1)
        tens.append((role, layer, t, rows, n, data))
    n_ctx = 100
    toks = rng.integers(0, 399, n_ctx).astype(np.int32)
    toks[list(special)] = odd
    gpu, cpu = elb.Backend(spec, tens, n_ctx, n_seq=2), ol.OracleModel(spec, tens, n_ctx)
    for s in (0, 1):
        gpu.eval_batch(toks[:90], np.full(90, s), np.arange(90), want_logits=False)
    cpu.eval(toks[:90], 0)
    for pos in (45, 50, 59, 61, 89):
        want = cpu.eval(toks[pos:pos + 1], pos)
        assert np.isfinite(want).all()
        one = gpu.eval(toks[pos:pos + 1], pos)
        two = gpu.eval_batch(toks[[pos, pos]], [0, 1], [pos, pos])
        for got in (one, two[0], two[1]):
            assert np.abs(got - want).max() <= 2e-4 * np.abs(want).max(), pos
    gpu.close()
    cpu.close()


# a residual stream whose mean square is beyond the range of a float: the norm's factor is taken in double, as the CPU path does
@pytest.mark.parametrize("layout,factor", (("f16", 1e12), ("q8_0", 3e10), ("q4_k_m", 3e10)))
def test_decode_with_a_very_large_residual_stream(elb, layout, factor):
    spec = synth.Spec(name="small", n_layer=2, n_embd=256, n_ff=512, n_head=2, n_head_kv=1, n_vocab=512, layout=layout, head_sigma=2e-2)
    tens = []
    for role, layer, t, rows, n, data in synth.generate(spec, 53):
        if role == "ffn_norm":
            data = (data.copy().view(np.float32) * np.float32(factor)).view(np.uint8)
        tens.append((role, layer, t, rows, n, data))
    gpu, cpu = elb.Backend(spec, tens, 16), ol.OracleModel(spec, tens, 16)
    toks = synth.lcg_tokens(8, spec.n_vocab, 53)
    for pos in range(4):
        a, b = gpu.eval(toks[pos:pos + 1], pos), cpu.eval(toks[pos:pos + 1], pos)
        assert gpu.last_eval_stats()[1] == 1, "the persistent kernel must run"
        assert np.square(gpu.hidden().astype(np.float64)).mean() > 1e39
        assert np.abs(a - b).max() <= 2e-4 * np.abs(b).max() and np.abs(b).max() > 0
    gpu.close()
    cpu.close()


# more query heads than the built-in shapes have, q and v in a costlier format than k: one thread block gets ten row tiles of k
# alone, more than three times k's share by count
@pytest.mark.parametrize("barrier_kernel", (False, True))
def test_decode_uneven_cut_of_qkv(elb, monkeypatch, barrier_kernel):
    if barrier_kernel:
        monkeypatch.setenv("ELB_DK_OLD", "1")
    spec = synth.Spec(name="small", n_layer=2, n_embd=512, n_ff=512, n_head=96, n_head_kv=12, n_vocab=512, layout="q4_k_m",
                      head_sigma=2e-5)
    tens = []
    rng = np.random.default_rng(5)
    for role, layer, t, rows, n, data in synth.generate(spec, 37):
        want = {"attn_q": synth.Q6_K, "attn_k": synth.Q4_K, "attn_v": synth.Q6_K}.get(role, t)
        if want != t:
            data = synth.rand_weight(rng, want, rows, n)
        tens.append((role, layer, want, rows, n, data))
    toks = synth.lcg_tokens(150, spec.n_vocab, 37)
    gpu, cpu = elb.Backend(spec, tens, 160), ol.OracleModel(spec, tens, 160)
    assert runs_on(gpu, barrier_kernel)
    gpu.eval(toks[:140], 0, want_logits=False)
    cpu.eval(toks[:140], 0)
    for pos in (0, 139, 140, 141):
        a, b = gpu.eval(toks[pos:pos + 1], pos), cpu.eval(toks[pos:pos + 1], pos)
        assert gpu.last_eval_stats()[1] == 1, "the persistent kernel must run"
        assert np.abs(a - b).max() <= 2e-4 * np.abs(b).max()
        assert np.array_equal(a, gpu.eval(toks[pos:pos + 1], pos))
    gpu.close()
    cpu.close()


# the words in the exchange buffers when a step starts - of an earlier step, of another layer, anything that is not numbered
# for this step - never reach a result: garbage with plausible values between evaluations, and a numbering that starts again
# after every few steps (the 32-bit numbers of a long-lived model do), give the same bits
@pytest.mark.parametrize("layout,heads,kv,n_layer", (("q4_k_m", 8, 2, 3), ("f16", 4, 2, 2), ("q8_0", 2, 2, 1)))
def test_decode_does_not_read_old_exchange_words(elb, monkeypatch, layout, heads, kv, n_layer):
    from exactinfer_b200 import capi
    spec = synth.Spec(name="small", n_layer=n_layer, n_embd=512, n_ff=768, n_head=heads, n_head_kv=kv, n_vocab=640, layout=layout,
                      head_sigma=2e-5)
    tens = list(synth.generate(spec, 43))
    toks = synth.lcg_tokens(400, spec.n_vocab, 43)
    walk = (399, 3, 398, 120, 4, 5, 121, 397)

    def evals(gpu, fill):
        gpu.eval(toks[:399], 0, want_logits=False)
        out = []
        for pos in sorted(walk) + list(walk) * 3:
            if fill is not None:
                capi.check(capi.lib().elb_selftest_decode_exchange(gpu._h, fill))
            out.append(gpu.eval(toks[pos:pos + 1], pos).copy())
        gpu.close()
        return out

    want = evals(elb.Backend(spec, tens, 400), None)
    for fill in (0x3F, 0xBD, 0xFF, 0):  # (four equal bytes as a float: 0.747, -0.0925, NaN, 0; as a number: none that is near)
        for a, b in zip(evals(elb.Backend(spec, tens, 400), fill), want):
            assert np.array_equal(a, b), fill
    monkeypatch.setenv("ELB_DK_STEPS", "3")
    for a, b in zip(evals(elb.Backend(spec, tens, 400), None), want):
        assert np.array_equal(a, b)


# a feed-forward vector whose limbs (or fp32 values: F16) do not fit in shared memory beside the weight rings: worked off
# in two and in four parts along k, which every weight format walks with coordinates of its own (test_decode_plan_cpu.py says
# how many parts a length gives)
@pytest.mark.parametrize("layout,n_ff", (("q4_k_m", 25600), ("f16", 25600), ("q8_0", 25600), ("q6_k", 25600), ("f16", 28672), ("f16", 57344), ("q4_k_m", 57344)))
def test_decode_long_feed_forward(elb, layout, n_ff):
    spec = synth.Spec(name="small", n_layer=2, n_embd=256, n_ff=n_ff, n_head=2, n_head_kv=1, n_vocab=640, layout=layout,
                      head_sigma=2e-5)
    assert decode_pair(elb, spec, 32, 80, (0, 17, 70)) <= 2e-4


# prompt attention: query tiles that are not full, one key tile, cuts of few and of many key tiles (more partial results per
# query tile than a full batch could have), a cut with a short last chunk, more CTAs than places
@pytest.mark.parametrize("heads,kv", ((4, 2), (8, 1), (4, 4)))
@pytest.mark.parametrize("pos0,n", ((0, 2), (63, 2), (0, 65), (203, 77), (1500, 3), (1400, 130), (0, 512)))
def test_prompt_attention_cuts(elb, heads, kv, pos0, n):
    """The same tokens in one chunk and in chunks of 64, which cut the keys differently: the order of fp32 sums differs, no more."""
    spec = synth.Spec(name="small", n_layer=1, n_embd=256, n_ff=512, n_head=heads, n_head_kv=kv, n_vocab=512, layout="q8_0",
                      head_sigma=1e-4)
    tens = list(synth.generate(spec, 3))
    toks = synth.lcg_tokens(pos0 + n, spec.n_vocab)
    a, b = elb.Backend(spec, tens, 1664), elb.Backend(spec, tens, 1664)
    if pos0:
        a.eval(toks[:pos0], 0, want_logits=False)
        b.eval(toks[:pos0], 0, want_logits=False)
    got = a.eval(toks[pos0:], pos0)
    for lo in range(pos0, pos0 + n, 64):
        want = b.eval(toks[lo:min(lo + 64, pos0 + n)], lo)
    # scores, probabilities and sums carry 24 bits; fp32 sums over up to 1664 keys in another order: 2^-24 sqrt(1664) of the
    # values' size, a few such steps in a layer
    assert np.linalg.norm(got - want) <= 8 * 2.0 ** -24 * np.sqrt(1664) * np.linalg.norm(want)
    assert np.array_equal(got.view(np.uint32), a.eval(toks[pos0:], pos0).view(np.uint32))
