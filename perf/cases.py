"""Workloads of the batched decode engine, as a serving host drives it: what is timed, and with what inputs.

A case names one of five uses of the public interface:

  step      one `Engine.step`: B conversations advance by one token and the host gets all logits (the scheduler that samples
            by itself; also scoring a given continuation)
  greedy    `Engine.decode_greedy` for `new` tokens without a host round trip, then one `Engine.step` on the last ids
  sample    `new` rounds of `Engine.step_sample` feeding each other, then one `Engine.step` on the last ids
  prefill   `Engine.prefill` of a prompt into an empty slot, then one `Engine.step` with the next given token
  matvec    one batch of quantized matrix-vector products through the device interface (IQ3_S q/k/v and output projections,
            Q8_0 output head), as a host that keeps its own layer loop issues them

The closing `step` returns logits that depend on all the state (KV pages, recurrent and convolution state) the pass has
written.  Models: the full 48-layer shape (hidden 2048, 512 experts, top-10, vocabulary 151936), shallower stacks of the same
layers, and the small 4-layer, 32-expert one the tests use.  Weights, contexts, tokens and sampler states come from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from qwental_b200.engine import Engine, default_cfg
from qwental_b200.gpu import Gpu
from qwental_b200.layers import Qmv
from qwental_b200.synth import row_bytes

IQ3_S, Q8_0 = 21, 8
D, INTER, VOCAB = 2048, 512, 151936
KV_TOKEN = 2 * 2 * 256 * 2       # bytes per token and attention layer: K and V, 2 heads of 256 fp16
GDN_STATE = 32 * 128 * 128 * 4   # bytes per slot and Gated DeltaNet layer
RESEED = 1024                    # tokens a slot grows by before its conversation is replaced by a fresh one of the first length

FULL = dict(layers=48, experts=512, topk=10, vocab=VOCAB)
SMALL = dict(layers=4, experts=32, topk=4, vocab=512)


def _engine_case(name, kind, model, slots=1, lo=0, hi=0, new=0, prompt=0):
    c = dict(kind=kind, slots=slots, lo=lo, hi=hi, new=new, prompt=prompt, **model)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a small model answering three short conversations: launches and host work are everything
        _engine_case("step_3slots_small", "step", SMALL, 3, 100, 900),
        # one user, full model: the latency of a token
        _engine_case("step_1slot", "step", FULL, 1, 900, 1100),
        # one user with a long document, sixteen tokens on the device
        _engine_case("greedy_1slot_long", "greedy", FULL, 1, 24000, 26000, new=15),
        # a lightly loaded server
        _engine_case("greedy_5slots", "greedy", FULL, 5, 256, 12000, new=7),
        # the benchmark's load: 16 ragged slots of 1K to 48K tokens
        _engine_case("greedy_16slots", "greedy", FULL, 16, 1024, 49152, new=7),
        # the same server with sampling
        _engine_case("sample_23slots", "sample", FULL, 23, 512, 8192, new=3),
        # a full server whose host wants every row's logits
        _engine_case("step_64slots", "step", FULL, 64, 256, 4096),
        # prompts: a chat turn, a page of text, and a long one on a quarter-depth stack
        _engine_case("prefill_45", "prefill", FULL, prompt=45),
        _engine_case("prefill_419", "prefill", FULL, prompt=419),
        _engine_case("prefill_1700_12layers", "prefill", dict(FULL, layers=12), prompt=1700),
        # a host with its own layer loop: projections and output head for a few and for many rows
        dict(name="matvec_4rows", kind="matvec", rows=4, vocab=VOCAB),
        dict(name="matvec_61rows", kind="matvec", rows=61, vocab=VOCAB),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "greedy", "sample", "prefill", "prefill", "matvec"])
    if kind == "matvec":
        return dict(kind=kind, rows=_log_int(rng, 1, 64), vocab=16 * _log_int(rng, 256, VOCAB // 16))
    layers = 4 * _log_int(rng, 1, 12)
    model = dict(FULL, layers=layers, vocab=16 * _log_int(rng, 2000, VOCAB // 16))
    if rng.random() < 0.15:
        model = dict(SMALL, vocab=16 * _log_int(rng, 32, 2000))
        layers = SMALL["layers"]
    if kind == "prefill":
        return _engine_case(None, kind, model, prompt=_log_int(rng, 5, min(3000, 419 * 48 // layers)))
    slots = _log_int(rng, 1, 64)
    lo = _log_int(rng, 40, 2000)
    most = min(48000, 150000 // slots)  # keeps the state of three such servers on one card
    hi = max(lo + 50, _log_int(rng, min(lo + 50, most), most))
    new = 0 if kind == "step" else rng.randint(2, 15 if slots <= 4 else 7 if slots <= 16 else 3)
    return _engine_case(None, kind, model, slots, lo, hi, new=new)


class _Wrap:
    """A device buffer of the framework as a torch tensor (no copy); the tensor keeps the buffer alive."""

    def __init__(self, buf, shape, typestr):
        self.buf = buf
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(buf.dev_ptr, False), version=3)


def _view(buf, shape, typestr):
    return torch.as_tensor(_Wrap(buf, shape, typestr), device="cuda")


class _Server:
    """What a serving process holds: the device, the model, its slots and the rows it is about to advance."""

    def __init__(self, case, seed):
        self.eng = self.gpu = None
        self.case = case
        rng = np.random.default_rng([seed, 1])
        B, V = case["slots"], case["vocab"]
        if case["kind"] == "prefill":
            self.ctx = []
            self.prompt = rng.integers(0, V, case["prompt"]).astype(np.int32)
            self.next = rng.integers(0, V, 1).astype(np.int32)
            top = case["prompt"] + 64
        else:
            # one length from each of B equal parts of the log range, in random order
            u = (rng.permutation(B) + rng.random(B)) / B
            self.ctx = [int(round(case["lo"] * (case["hi"] / case["lo"]) ** x)) for x in u]
            self.toks = rng.integers(0, V, B).astype(np.int32)
            self.sids = list(range(B))
            self.seeds = [int(s) for s in rng.integers(1, 1 << 60, B)]
            top = max(self.ctx) + RESEED + 64
        if case["kind"] == "sample":
            # most users sample, a few take the best token
            self.params = [(0.0, 0, 1.0) if i % 8 == 7 else (0.8, 40, 0.95) if i % 2 else (0.7, 20, 0.8) for i in range(B)]
            self.rng = rng.integers(0, 1 << 63, B).astype(np.uint64)
        pages = sum((c + RESEED + 64) // 256 + 1 for c in self.ctx) or top // 256 + 1
        cfg = default_cfg(layers=case["layers"], experts=case["experts"], topk=case["topk"], vocab=V, max_slots=B, max_ctx=top, kv_pages=pages, seed=seed)
        self.gpu = Gpu()
        self.gpu.L.qw_gpu_set_graphs(self.gpu.g, True)
        self.eng = Engine(self.gpu, cfg)
        for s in range(len(self.ctx)):
            self._start(s)

    def _start(self, s):
        self.eng.seed_slot(s, self.ctx[s], self.seeds[s])

    def make_room(self, n):
        for s, c in enumerate(self.ctx):
            if self.eng.pos(s) + n > c + RESEED:
                self._start(s)

    def __del__(self):
        if self.eng is not None:
            self.eng.close()
        if self.gpu is not None:
            self.gpu.close()


class _Matvecs:
    """(rows, inputs, format, fp32 result) of each product, its weights, activations and results on the device."""

    def __init__(self, case, seed):
        self.gpu = Gpu()
        self.gpu.L.qw_gpu_set_graphs(self.gpu.g, True)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        self.rows, self.mats, self.out = case["rows"], [], {}
        for name, N, K, fmt in _mats(case):
            rb, per = row_bytes(fmt, K), 110 if fmt == IQ3_S else 34
            W = self.gpu.buf(N * rb)
            w = _view(W, (N * rb // per, per), "|u1")
            w.copy_(torch.randint(0, 256, w.shape, generator=gen, device="cuda", dtype=torch.uint8))
            d = torch.rand(w.shape[0], generator=gen, device="cuda") * 0.019 + 0.001
            # (-128 does not occur in Q8_0 blocks)
            if fmt == Q8_0:
                w[:, 2:][w[:, 2:] == 128] = 129
            w[:, :2] = (d / (64 if fmt == IQ3_S else 1)).to(torch.float16).view(torch.uint8).view(-1, 2)
            x = self.gpu.buf(self.rows * K * 2)
            _view(x, (self.rows, K), "<f2").copy_(torch.randn(self.rows, K, generator=gen, device="cuda"))
            y = self.gpu.buf(self.rows * N * (4 if fmt == Q8_0 else 2))
            self.mats.append((Qmv(self.gpu, W, fmt, N, K, f32_out=fmt == Q8_0), x, y))
            self.out[name] = _view(y, (self.rows, N), "<f4" if fmt == Q8_0 else "<f2")
        torch.cuda.synchronize()

    def __del__(self):
        self.out, self.mats = {}, []
        self.gpu.close()


def _mats(case):
    return [("qkv", 5120, D, IQ3_S), ("o", D, 4096, IQ3_S), ("head", case["vocab"], D, Q8_0)]


def prepare(case, seed):
    return (_Matvecs if case["kind"] == "matvec" else _Server)(case, seed)


def run(s):
    if isinstance(s, _Matvecs):
        b = s.gpu.batch()
        for m, x, y in s.mats:
            m.encode(b, x, y, s.rows)
        b.end()
        return s.out
    kind, new, eng = s.case["kind"], s.case["new"], s.eng
    if kind == "prefill":
        first = eng.prefill(0, s.prompt)
        return {"prompt": first, "next": eng.step([0], s.next)[0]}
    s.make_room(new + 1)
    if kind == "step":
        return {"logits": eng.step(s.sids, s.toks)[0]}
    if kind == "greedy":
        ids, _ = eng.decode_greedy(s.sids, s.toks, new)
    else:
        ids = np.empty((new, len(s.sids)), np.int32)
        toks = s.toks
        for k in range(new):
            toks, _ = eng.step_sample(s.sids, toks, s.params, s.rng)
            ids[k] = toks
    out = {"ids": ids, "logits": eng.step(s.sids, ids[-1])[0]}
    return out if kind == "greedy" else dict(out, rng=s.rng.view(np.int64).copy())


def work(case):
    if case["kind"] == "matvec":
        r = case["rows"]
        by = sum(N * row_bytes(f, K) + r * (2 * K + N * (4 if f == Q8_0 else 2)) for _, N, K, f in _mats(case))
        return {"bytes": by, "flops": sum(2 * r * N * K for _, N, K, _ in _mats(case))}
    L, E, k, V = case["layers"], case["experts"], case["topk"], case["vocab"]
    attn = L // 4
    gdn = L - attn
    gdn_rows, qkv_rows = 12352, 9216
    dense = gdn * (gdn_rows * row_bytes(IQ3_S, D) + D * row_bytes(IQ3_S, 4096)) + attn * (qkv_rows * row_bytes(IQ3_S, D) + D * row_bytes(IQ3_S, 4096))
    expert = 2 * INTER * row_bytes(IQ3_S, D) + D * row_bytes(IQ3_S, INTER)
    head = V * row_bytes(Q8_0, D)
    params = gdn * (gdn_rows * D + D * 4096) + attn * (qkv_rows * D + D * 4096) + L * ((k + 1) * 3 * INTER * D + (E + 1) * D)

    def weights(tokens):  # dense weights, router, shared expert and the distinct experts that this many tokens choose
        return dense + L * ((E + 1) * D * 2 + expert * (1 + E * (1 - (1 - k / E) ** tokens)))

    def steps(B, ctx_sum, n):  # n steps of B slots with ctx_sum tokens of context in all
        by = n * (weights(B) + head + attn * KV_TOKEN * (ctx_sum + B) + gdn * B * GDN_STATE * 2 + B * V * 4)
        return by, n * 2 * B * (params + V * D) + n * attn * ctx_sum * 4 * 16 * 256

    if case["kind"] == "prefill":
        n = case["prompt"]
        by, fl = steps(1, n, 1)
        by += weights(n) + head + attn * KV_TOKEN * n + gdn * GDN_STATE + V * 4
        fl += 2 * n * params + 2 * V * D + attn * n * n / 2 * 4 * 16 * 256 + gdn * n * 32 * 128 * 128 * 6
        return {"bytes": by, "flops": fl}
    lo, hi, B = case["lo"], case["hi"], case["slots"]
    by, fl = steps(B, B * (hi - lo) / math.log(hi / lo), case["new"] + 1)
    return {"bytes": by, "flops": fl}


def tolerance(case):
    # The products against the fp32-order kernels of the same format: 1.4e-5 (single roundings of the fp16 results that fall the
    # other way), 1.5e-7 for the fp32 ones.
    if case["kind"] == "matvec":
        return {"rel": 6e-5}
    # The engine with its dense products in another order of summation: 3e-3 to 7e-3 after 12 layers.  A deeper stack of random
    # layers diverges where two orders pick different experts or tokens, so it has no wider bound: there an implementation has
    # to keep the orders that make a row independent of its batch.
    return {"rel": 0.028, "differ": 0.01}
