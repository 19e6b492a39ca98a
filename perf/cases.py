"""The work that a user of this library has it do, as timed cases over the public entry points.

Four kinds of call, over the model shapes of `synth.SPECS` (the 32B shape cut to eight layers, as the tests cut shapes):
  decode   single-token steps of one sequence behind a cached prefix (Backend.eval / Backend.eval_top)
  prefill  a prompt, or the next turn of a conversation behind a cached prefix (Backend.eval)
  batch    one step of several sequences with contexts of different lengths (Backend.eval_batch_top)
  matvec, matmul   the operator interface on device buffers (elb_matvec_dev, elb_matmul_dev)

A model is loaded once and serves many requests, so its weights do not depend on a case's seed: the seed gives the
tokens. The cached prefix is a fixed stream as well (a system prompt that every request shares): `prepare` puts it into
the KV cache and `run` writes rows behind it only, so that states of one case can share the model. Weights have mean 0 and
a spread of about 0.02 in every format, as trained ones do (in Q4_K the mins cancel the mean of the nibbles).
"""
import collections
import ctypes
import dataclasses
import math

import numpy as np
import torch

from exactinfer_b200 import Backend, Weight, synth
from exactinfer_b200.capi import check, lib

F16, Q8_0, Q4_K, Q6_K = synth.F16, synth.Q8_0, synth.Q4_K, synth.Q6_K
SHAPES = {"0.6b-f16": ("qwen3-0.6b-f16", 28), "1.7b-q8_0": ("qwen3-1.7b-q8_0", 28), "4b-q4_k_m": ("qwen3-4b-q4_k_m", 36),
          "32b-q4_k_m-8-layers": ("qwen3-32b-q4_k_m", 8)}
N_CTX = 8320                        # context of a model that serves one sequence
BATCH_SEQ, BATCH_CTX = 64, 1152     # sequences and context of a model that serves batches
KEEP = 3                            # models kept loaded


def listed():
    return [
        # a chat answer from the smallest model right after a short question: launches and latency
        {"name": "decode-0.6b-f16", "kind": "decode", "model": "0.6b-f16", "prefix": 41, "steps": 8, "top": 0},
        # the same from an 8-bit model, tokens picked on the device
        {"name": "decode-1.7b-q8_0", "kind": "decode", "model": "1.7b-q8_0", "prefix": 300, "steps": 8, "top": 1},
        # the benchmark's configuration: steps behind a 512-token prompt, full logits to the host's sampler
        {"name": "decode-4b-q4_k_m", "kind": "decode", "model": "4b-q4_k_m", "prefix": 512, "steps": 8, "top": 0},
        # long conversation / document: the KV cache is a third of a step's bytes
        {"name": "decode-4b-long-context", "kind": "decode", "model": "4b-q4_k_m", "prefix": 4375, "steps": 4, "top": 20},
        # wide matrices of the largest shape
        {"name": "decode-32b-8-layers", "kind": "decode", "model": "32b-q4_k_m-8-layers", "prefix": 1023, "steps": 8, "top": 8},
        # the benchmark's prompt
        {"name": "prefill-4b-512", "kind": "prefill", "model": "4b-q4_k_m", "prefix": 0, "tokens": 512},
        # a short next turn of a conversation, ragged length
        {"name": "prefill-0.6b-turn-77", "kind": "prefill", "model": "0.6b-f16", "prefix": 203, "tokens": 77},
        # a document: several chunks and a remainder
        {"name": "prefill-1.7b-2050", "kind": "prefill", "model": "1.7b-q8_0", "prefix": 0, "tokens": 2050},
        # a server's step with a moderate and with a full batch
        {"name": "batch-4b-16", "kind": "batch", "model": "4b-q4_k_m", "rows": 16, "ctx_lo": 64, "ctx_hi": 700, "top": 4},
        {"name": "batch-1.7b-64", "kind": "batch", "model": "1.7b-q8_0", "rows": 64, "ctx_lo": 100, "ctx_hi": 1000, "top": 1},
        # the operators alone: the 4B shape's ffn_down for one token, and a few rows of a Q6_K matrix
        {"name": "matvec-q4_k-2560x9728", "kind": "matvec", "type": Q4_K, "rows": 2560, "n": 9728, "b": 1},
        {"name": "matmul-q6_k-2560x4096x37", "kind": "matmul", "type": Q6_K, "rows": 2560, "n": 4096, "b": 37},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "batch", "op"])
    if kind == "decode":
        return {"kind": kind, "model": rng.choice(sorted(SHAPES)), "prefix": _log_int(rng, 1, 8000), "steps": rng.randint(4, 8),
                "top": rng.choice([0, 0, 1, rng.randint(2, 40)])}
    if kind == "prefill":
        model = rng.choice(sorted(SHAPES))
        most = 2050 if model[0] in "01" else 900
        return {"kind": kind, "model": model, "prefix": rng.choice([0, 0, _log_int(rng, 4, 3000)]), "tokens": _log_int(rng, 2, most)}
    if kind == "batch":
        lo = _log_int(rng, 8, 400)
        return {"kind": kind, "model": rng.choice(["0.6b-f16", "1.7b-q8_0", "4b-q4_k_m"]), "rows": _log_int(rng, 2, 64), "ctx_lo": lo,
                "ctx_hi": rng.randint(lo, 1000), "top": rng.choice([1, rng.randint(2, 40)])}
    spec = synth.SPECS[rng.choice(sorted(synth.SPECS))]
    role, (rows, n) = rng.choice(sorted(synth.layer_shapes(spec).items()))
    t = rng.choice([F16, Q8_0, Q4_K, Q6_K])
    b = rng.choice([1, _log_int(rng, 2, 512)])
    return {"kind": "matvec" if b == 1 else "matmul", "type": t, "rows": rows - rng.choice([0, 0, rng.randint(1, 200)]), "n": n, "b": b}


# ---------------------------------------------------------------- weights

def _blocks(gen, t, rows, n):
    """Random blocks of a weight as host bytes, drawn on the GPU."""
    if t == F16:
        w = torch.randn((rows, n), generator=gen, device="cuda").mul_(0.02).half().view(torch.uint8)
        return w.cpu().numpy().reshape(rows, -1)
    blk, size = synth.BLOCK[t]
    nb = n // blk
    w = torch.randint(0, 256, (rows, nb, size), generator=gen, device="cuda", dtype=torch.uint8)
    at, spread = {Q8_0: (0, 3e-4), Q4_K: (0, 1.2e-4), Q6_K: (208, 1.5e-5)}[t]
    d = torch.randn((rows, nb), generator=gen, device="cuda").mul_(spread).abs_().half()
    w[:, :, at:at + 2] = d.view(torch.uint8).reshape(rows, nb, 2)
    if t == Q4_K:  # every sub-block's min equal to its scale, dmin = 7.5 d: w = d * scale * (nibble - 7.5)
        w[:, :, 2:4] = (d * 7.5).view(torch.uint8).reshape(rows, nb, 2)
        w[:, :, 8:12] = w[:, :, 4:8]
        w[:, :, 12:16] = (w[:, :, 12:16] & 15) * 17
    return w.cpu().numpy().reshape(rows, -1)


def _tensors(spec):
    """The tensors of a model in the order of synth.generate; layers of one parity share their random blocks on the host."""
    gen = torch.Generator(device="cuda").manual_seed(20240607)
    norm = lambda n: torch.randn(n, generator=gen, device="cuda").mul_(0.01).add_(1).cpu().numpy().view(np.uint8).reshape(1, -1)
    t = spec.weight_type("token_embd", -1)
    yield "token_embd", -1, t, spec.n_vocab, spec.n_embd, _blocks(gen, t, spec.n_vocab, spec.n_embd)
    yield "output_norm", -1, synth.F32, 1, spec.n_embd, norm(spec.n_embd)
    shared = {}
    for layer in range(spec.n_layer):
        for role in ("attn_norm", "ffn_norm", "attn_q_norm", "attn_k_norm"):
            n = spec.head_dim if role[5:7] in ("q_", "k_") else spec.n_embd
            yield role, layer, synth.F32, 1, n, norm(n)
        for role, (rows, n) in synth.layer_shapes(spec).items():
            t = spec.weight_type(role, layer)
            if (role, layer % 2) not in shared:
                shared[role, layer % 2] = _blocks(gen, t, rows, n)
            yield role, layer, t, rows, n, shared[role, layer % 2]


class _Served:
    """A loaded model and what its KV cache holds."""

    def __init__(self, name, batch):
        full, layers = SHAPES[name]
        self.spec = dataclasses.replace(synth.SPECS[full], n_layer=layers)
        self.backend = Backend(self.spec, _tensors(self.spec), BATCH_CTX if batch else N_CTX, n_seq=BATCH_SEQ if batch else 0)
        torch.cuda.empty_cache()
        self.cached = None


_models = collections.OrderedDict()


def _model(name, batch):
    key = (name, batch)
    if key not in _models:
        while len(_models) >= KEEP:
            _models.popitem(last=False)
        _models[key] = _Served(name, batch)
    _models.move_to_end(key)
    return _models[key]


def _spec(case):
    full, layers = SHAPES[case["model"]]
    return dataclasses.replace(synth.SPECS[full], n_layer=layers)


# ---------------------------------------------------------------- the calls

def _contexts(case):
    """Cached tokens of each sequence of a batch: ragged, fixed by the case."""
    return np.random.default_rng(case["rows"]).integers(case["ctx_lo"], case["ctx_hi"] + 1, case["rows"]).astype(np.int32)


def _load_prefix(served, case):
    v, b = served.spec.n_vocab, served.backend
    if case["kind"] == "batch":
        key = ("batch", case["rows"], case["ctx_lo"], case["ctx_hi"])
        if served.cached != key:
            for s, n in enumerate(_contexts(case)):
                toks = synth.lcg_tokens(int(n), v, 777 + s)
                for lo in range(0, int(n), 512):
                    part = toks[lo:lo + 512]
                    b.eval_batch(part, np.full(part.size, s), np.arange(lo, lo + part.size), want_logits=False)
    else:
        key = case["prefix"]
        if served.cached != key and key:
            b.eval(synth.lcg_tokens(key, v), 0, want_logits=False)
    served.cached = key


def prepare(case, seed):
    if case["kind"] in ("matvec", "matmul"):
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        w = Weight(case["type"], case["rows"], case["n"], _blocks(gen, case["type"], case["rows"], case["n"]),
                   planes=case["kind"] == "matmul")
        x = torch.randn((case["b"], case["n"]), generator=gen, device="cuda")
        y = torch.empty((case["b"], case["rows"]), device="cuda")
        return {"case": case, "w": w, "x": x, "y": y}
    served = _model(case["model"], case["kind"] == "batch")
    _load_prefix(served, case)
    rng = np.random.default_rng(int(seed))
    count = case.get("steps") or case.get("tokens") or case.get("rows")
    state = {"case": case, "model": served.backend, "tokens": rng.integers(0, served.spec.n_vocab, count).astype(np.int32)}
    if case["kind"] == "batch":
        state["seq"], state["pos"] = np.arange(count, dtype=np.int32), _contexts(case)
    return state


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "matvec":
        check(lib().elb_matvec_dev(state["w"]._h, ctypes.c_void_p(state["x"].data_ptr()), ctypes.c_void_p(state["y"].data_ptr()), 0))
        return state["y"]
    if kind == "matmul":
        check(lib().elb_matmul_dev(state["w"]._h, ctypes.c_void_p(state["x"].data_ptr()), case["b"],
                                   ctypes.c_void_p(state["y"].data_ptr()), 0))
        return state["y"]
    model, tokens = state["model"], state["tokens"]
    if kind == "prefill":
        return model.eval(tokens, case["prefix"])
    if kind == "batch":
        return model.eval_batch_top(tokens, state["seq"], state["pos"], k=case["top"])
    if case["top"]:
        return [model.eval_top(tokens[i:i + 1], case["prefix"] + i, k=case["top"]) for i in range(case["steps"])]
    return [model.eval(tokens[i:i + 1], case["prefix"] + i) for i in range(case["steps"])]


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    if case["kind"] in ("matvec", "matmul"):
        rows, n, b = case["rows"], case["n"], case["b"]
        return {"bytes": rows * synth.row_bytes(case["type"], n) + 4 * b * (rows + n), "flops": 2 * b * rows * n}
    spec = _spec(case)
    weights = synth.decode_weight_bytes(spec)           # every matrix of every layer and the head, once
    linear = sum(r * n for r, n in synth.layer_shapes(spec).values()) * spec.n_layer   # multiply-adds of a token, head left out
    head, kv = spec.n_vocab * spec.n_embd, 8 * spec.kd * spec.n_layer                  # kv: bytes of a cached position
    attn = lambda keys: 4 * spec.qd * spec.n_layer * keys                              # flops of one query row
    if case["kind"] == "prefill":
        n, p = case["tokens"], case["prefix"]
        return {"bytes": weights + kv * (p + n) + 4 * spec.n_vocab, "flops": 2 * (linear * n + head) + attn(n * p + n * (n + 1) // 2)}
    if case["kind"] == "batch":
        keys, b = int(_contexts(case).sum()) + case["rows"], case["rows"]
        return {"bytes": weights + kv * keys + 8 * b * (1 + case["top"]), "flops": 2 * b * (linear + head) + attn(keys)}
    steps, p = case["steps"], case["prefix"]
    keys = steps * p + steps * (steps + 1) // 2
    out = 8 * (1 + case["top"]) if case["top"] else 4 * spec.n_vocab
    return {"bytes": steps * (weights + out) + kv * keys, "flops": 2 * steps * (linear + head) + attn(keys)}


def tolerance(case):
    if case["kind"] in ("matvec", "matmul"):
        return {"rel": 1e-5}   # the bar of the operator parity tests
    # 32-bit sums through 8 to 36 layers, each of which passes its rounding on: the library's own variants of a path (one
    # kernel or many, 3 or 4 limbs, fp32 or tensor-core attention) differ by up to 4e-6 here; picked ids may change places
    # where two logits are closer than that
    return {"rel": 3e-5, "differ": 0.01}
