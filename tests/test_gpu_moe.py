"""GPU parity of the MoE decode layer (benchmark config 2), through the C ABI.

Router logits and the chosen expert ids must be bit-exact against the CPU oracle's canonical-order router and
top-k; the layer output must be within the reference's own tolerance (max error / max |ref| < 1e-2,
bench/moe_decode.c:181-182 -- we hold 2e-3) of the FP64 layer (tools/moe_ref.py:72-82) and agree on top-1;
each token's output must be bit-identical whether it runs alone or in a batch."""
import numpy as np
import pytest

from oracle import oracle as orc
from qwental_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from qwental_b200.gpu import Gpu
    g = Gpu()
    yield g
    g.close()


def make_layer(gpu, E, D, I, topk, seed, shared=True, e_lo=0, e_hi=None, ffn="auto"):
    from qwental_b200.layers import MoeLayer
    rng = np.random.default_rng(seed)
    h = {}
    h["Wr"] = (rng.standard_normal((E, D)) * 0.02).astype(np.float16)
    h["wsg"] = (rng.standard_normal(D) * 0.02).astype(np.float16)
    # block scales d are the stated range times a power of two per tensor so that the layer output stays O(1):
    # at the unscaled range a SwiGLU expert's output has rms ~1.5e5 and the fp16 layer output would be inf
    sD, sI = synth.d_scale_for(D), synth.d_scale_for(I)
    h["gate"] = synth.iq3s_rows(rng, E * I, D, sD).reshape(E, I, -1)
    h["up"] = synth.iq3s_rows(rng, E * I, D, sD).reshape(E, I, -1)
    h["down"] = synth.iq3s_rows(rng, E * D, I, sI).reshape(E, D, -1)
    h["sg"] = synth.iq3s_rows(rng, I, D, sD)
    h["su"] = synth.iq3s_rows(rng, I, D, sD)
    h["sd"] = synth.iq3s_rows(rng, D, I, sI)
    b = {k: gpu.buf_from(v) for k, v in h.items()}
    layer = MoeLayer(gpu, E, D, I, topk, b["Wr"], b["wsg"], b["gate"], b["up"], b["down"],
                     b["sg"] if shared else None, b["su"] if shared else None, b["sd"] if shared else None, e_lo, e_hi, ffn)
    return layer, h, b


def run_layer(gpu, layer, x, fused_route=False):
    nb = x.shape[0]
    xb, ob = gpu.buf_from(x), gpu.buf(nb * layer.D * 2).zero()
    bt = gpu.batch()
    layer.encode(bt, xb, ob, nb, fused_route=fused_route)
    bt.end()
    return ob.download(np.float16, nb * layer.D).reshape(nb, layer.D)


@pytest.mark.parametrize("ffn", ["iq3x", "fused", "split"])
@pytest.mark.parametrize("E,B", [(64, 16), (64, 1), (64, 64), (512, 16)])
def test_moe_layer_parity(gpu, E, B, ffn):
    """ffn = "iq3x": gate/up + down in one launch with H in shared memory, on expert weights re-coded once into the kernel's
    own layout (what the engine runs at these shapes); "fused": the same kernel on the raw IQ3_S blocks; "split": the
    two-launch family that serves every other shape."""
    D, I, topk = 2048, 512, 10
    layer, h, _ = make_layer(gpu, E, D, I, topk, seed=10 + E, ffn=ffn)
    x = synth.acts_fp16(np.random.default_rng(B), B, D)
    out = run_layer(gpu, layer, x)

    # 1. router logits bit-exact (canonical order), shared-gate row included
    lg = layer.read_logits(B)
    ref_lg = orc.router_canon(np.concatenate([h["Wr"], h["wsg"][None]]), x)
    assert np.array_equal(lg.view(np.uint32), ref_lg.view(np.uint32))
    # 2. expert ids bit-exact; weights to 1e-6; grouping consistent
    U, ids, w, ue, off, ent = layer.read_sel(B)
    ref_ids, ref_w = orc.topk(ref_lg[:, :E], topk)
    assert np.array_equal(ids, ref_ids)
    assert np.allclose(w[:, :topk], ref_w, rtol=2e-6, atol=1e-7)
    assert np.allclose(w[:, topk], 1 / (1 + np.exp(-ref_lg[:, E].astype(np.float64))), rtol=2e-6)
    uniq = np.unique(ref_ids)
    assert U == len(uniq) and np.array_equal(ue, uniq) and off[-1] == B * topk
    pairs = sorted((int(e >> 8), int(e & 255)) for e in ent)
    assert pairs == sorted((t, k) for t in range(B) for k in range(topk))
    for u in range(U):
        for e in ent[off[u]:off[u + 1]]:
            assert ref_ids[e >> 8, e & 255] == ue[u]
    # 3. layer output vs the FP64 layer on the same experts
    ref, ids64, gap = orc.moe_ref(x, h["Wr"], h["wsg"], h["gate"], h["up"], h["down"], h["sg"], h["su"], h["sd"], D, I, topk, ids=ids)
    err = np.abs(out.astype(np.float64) - ref).max() / np.abs(ref).max()
    assert err < 2e-3, err
    assert np.array_equal(out.astype(np.float64).argmax(1), ref.argmax(1))
    # the FP64 router picks the same set wherever its 10th/11th gap exceeds the fp32 error bound
    for t in range(B):
        if gap[t] > 1e-5:
            assert set(ids64[t]) == set(ids[t])


@pytest.mark.parametrize("ffn", ["iq3x", "fused", "split"])
def test_moe_batched_equals_alone(gpu, ffn):
    D, I, topk, E, B = 2048, 512, 10, 64, 24
    layer, h, _ = make_layer(gpu, E, D, I, topk, seed=3, ffn=ffn)
    x = synth.acts_fp16(np.random.default_rng(9), B, D)
    out = run_layer(gpu, layer, x)
    for t in (0, 7, 23):
        alone = run_layer(gpu, layer, x[t:t + 1])
        assert np.array_equal(alone[0].view(np.uint16), out[t].view(np.uint16))
    # identical tokens in one batch give identical rows (more than 8 tokens on one expert -> several column tiles)
    xs = np.repeat(x[:1], 20, axis=0)
    outs = run_layer(gpu, layer, xs)
    assert all(np.array_equal(outs[i].view(np.uint16), out[0].view(np.uint16)) for i in range(20))


@pytest.mark.parametrize("ffn", ["iq3x", "fused", "split"])
def test_moe_expert_range_partitions_the_work(gpu, ffn):
    """Expert-parallel building block: with experts restricted to [lo, hi) each part writes only its own
    (token, rank) rows; the union over a partition equals the full layer's rows bit for bit."""
    D, I, topk, E, B = 2048, 512, 10, 64, 16
    full, h, b = make_layer(gpu, E, D, I, topk, seed=5, ffn=ffn)
    x = synth.acts_fp16(np.random.default_rng(2), B, D)
    run_layer(gpu, full, x)
    pg_full = full.Pg.download(np.float32, B * (topk + 1) * D).reshape(B, topk + 1, D)
    _, ids, _, _, _, _ = full.read_sel(B)
    from qwental_b200.layers import MoeLayer
    acc = np.zeros_like(pg_full)
    for lo, hi in ((0, 32), (32, 64)):
        part = MoeLayer(gpu, E, D, I, topk, b["Wr"], b["wsg"], b["gate"], b["up"], b["down"], b["sg"], b["su"], b["sd"], lo, hi, ffn)
        run_layer(gpu, part, x)
        pg = part.Pg.download(np.float32, B * (topk + 1) * D).reshape(B, topk + 1, D)
        mine = (ids >= lo) & (ids < hi)
        assert np.all(pg[:, :topk][~mine] == 0)
        acc[:, :topk] += pg[:, :topk]
        acc[:, topk] = pg[:, topk]
    assert np.array_equal(acc.view(np.uint32), pg_full.view(np.uint32))


@pytest.mark.parametrize("B", [1, 16, 64])
def test_fused_router_select_equals_two_launches(gpu, B):
    """moe_route (router + selection in one launch, last block selects) gives the same logits, selection record and
    layer output, bit for bit, as moe_router followed by moe_select -- also when launched repeatedly (the hand-over
    counter must be left at zero)."""
    D, I, topk, E = 2048, 512, 10, 64
    layer, h, _ = make_layer(gpu, E, D, I, topk, seed=21)
    x = synth.acts_fp16(np.random.default_rng(B + 5), B, D)
    out = run_layer(gpu, layer, x)
    lg, sel = layer.read_logits(B).copy(), layer.sel.download(np.uint8, layer.sel.size).copy()
    for _ in range(3):
        layer.sel.zero()
        layer.logits.zero()
        out2 = run_layer(gpu, layer, x, fused_route=True)
        assert np.array_equal(layer.read_logits(B).view(np.uint32), lg.view(np.uint32))
        got = layer.sel.download(np.uint8, layer.sel.size)
        U, ids, w, ue, off, ent = layer.read_sel(B)
        n = 16 + 64 * 16 * 4 + 64 * 17 * 4
        ref_ids = sel[16:16 + 64 * 16 * 4].view(np.int32).reshape(64, 16)[:B, :topk]
        assert np.array_equal(ids, ref_ids)
        assert np.array_equal(got[n:n + 4 * U], sel[n:n + 4 * U]) and got[:4].view(np.uint32)[0] == sel[:4].view(np.uint32)[0]
        assert np.array_equal(out2.view(np.uint16), out.view(np.uint16))


def test_selection_with_equal_logits_takes_lowest_ids(gpu):
    """Ties in the router: equal logits resolve to the lower expert id (as the reference's stable selection,
    kernels/moe_gg.metal:118-189).  Token 0 is all zeros (every logit equal: 512 candidates, the general path of the
    selection); in the other tokens some router rows are duplicated, so winners and the cut-off come in equal pairs
    (the fast path with a few candidates more than top-k)."""
    D, I, topk, E = 2048, 512, 10, 512
    layer, h, b = make_layer(gpu, E, D, I, topk, seed=33)
    Wr = h["Wr"].copy()
    rng = np.random.default_rng(8)
    for _ in range(60):  # duplicated rows -> exactly equal logits for every token
        a, c = rng.integers(0, E, 2)
        Wr[c] = Wr[a]
    b["Wr"].upload(Wr)
    x = synth.acts_fp16(rng, 6, D)
    x[0] = 0
    for fused in (False, True):
        layer.sel.zero()
        run_layer(gpu, layer, x, fused_route=fused)
        lg = layer.read_logits(6)
        ref_lg = orc.router_canon(np.concatenate([Wr, h["wsg"][None]]), x)
        assert np.array_equal(lg.view(np.uint32), ref_lg.view(np.uint32))
        U, ids, w, ue, off, ent = layer.read_sel(6)
        ref_ids, ref_w = orc.topk(ref_lg[:, :E], topk)
        assert np.array_equal(ids[:6, :topk], ref_ids), fused
        assert list(ids[0, :topk]) == list(range(topk))
        assert np.abs(w[:6, :topk] - ref_w).max() < 1e-6


def test_iq3x_recoding_is_lossless(gpu):
    """iq3x_pack followed by the IQ3X decoder gives, bit for bit, what the CPU oracle decodes from the original IQ3_S blocks
    (the oracle itself is pinned against gguf and the reference's decoder): the re-coding keeps every weight's exact value.
    Edge blocks included: all-zero and all-one fields, largest scales, every sign pattern."""
    from qwental_b200.layers import u32
    rng = np.random.default_rng(77)
    rows, K = 256, 1024
    W = synth.iq3s_rows(rng, rows, K, 1.0).copy()
    blk = W.reshape(rows, K // 256, 110)
    blk[0, 0, 2:110] = 0          # every index 0, no signs, scale 0
    blk[1, 0, 2:110] = 255        # every index 511, all signs, scale 15
    blk[2, 1, 74:106] = 0xAA      # alternating signs
    blk[3, 2, 66:74] = 0x55       # alternating codebook high bits
    src = gpu.buf_from(W)
    dst = gpu.buf((rows // 128) * (K // 512) * 128 * 272)
    y = gpu.buf(rows * K * 4)
    bt = gpu.batch()
    bt.kernel(gpu.compile("iq3x_pack", "iq3x_pack")).buf(0, src).buf(2, dst).bytes(3, u32(1, 1, K, rows)).dispatch((1,), (256,))
    bt.kernel(gpu.compile("iq3x_dq_test", "iq3x_dq_test")).buf(0, dst).buf(1, y).bytes(2, u32(rows, K)).dispatch((1,), (128,))
    bt.end()
    got = y.download(np.float32, rows * K).reshape(rows, K)
    ref = orc.dq_rows(orc.IQ3_S, W, K)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("B", [4, 5, 15, 17, 48, 49])
def test_fused_router_at_the_edges_of_its_passes(gpu, B):
    """moe_route reads up to four tokens directly and stages more by 16, three groups in flight: the comparison above at those edges."""
    test_fused_router_select_equals_two_launches(gpu, B)


@pytest.mark.parametrize("topk,edge", [(10, 1), (4, 5), (1, 18)])
def test_half_pieces_of_few_items_give_the_same_rows(gpu, topk, edge):
    """moe_ffn halves its gate/up pieces while the tokens choose few enough experts (64 of them here) that a block gets one half piece: up to `edge`
    tokens on 148 SMs.  A row is the same from both forms."""
    D, I, E = 2048, 512, 64
    layer, h, _ = make_layer(gpu, E, D, I, topk, seed=20 + topk, ffn="iq3x")
    x = synth.acts_fp16(np.random.default_rng(topk), edge + 1, D)
    whole = run_layer(gpu, layer, x)
    ids = layer.read_sel(edge + 1)[1]
    few = run_layer(gpu, layer, x[:edge])
    assert np.array_equal(few.view(np.uint16), whole[:edge].view(np.uint16))
    ref, _, _ = orc.moe_ref(x, h["Wr"], h["wsg"], h["gate"], h["up"], h["down"], h["sg"], h["su"], h["sd"], D, I, topk, ids=ids)
    assert np.abs(few.astype(np.float64) - ref[:edge]).max() < 2e-3 * np.abs(ref).max()  # the bound of the layer test above


def wide_ffn(gpu, h, x, E, topk, lo=0, hi=None, rows=1024, say=True):
    """Pg [tokens][topk + 1][D] and the chosen experts of a prompt's piece: logits, top-k, grouping and the one-launch FFN on records of their own, with
    the weights of experts [lo, hi) alone.  rows = tokens that Pg and the scratch have room for; say: the launcher is told the number of tokens"""
    import ctypes as C
    from qwental_b200.layers import iq3x_pack, u32
    D, I, nb, hi = 2048, 512, len(x), E if hi is None else hi
    gpu.L.qw_moe_sel_wide_bytes.restype = C.c_size_t
    d = dict(E=E, EL=hi - lo, D=D, I=I, TOPK=topk, SHARED=1, WIDE=1, IQ3X=1, SELECT=0)
    k = {f: gpu.compile(f, "t_%s_%d_%d_%d" % (f, E, topk, lo), **d) for f in ("moe_route", "moe_topk_wide", "moe_group_wide", "moe_ffn")}
    up = lambda a: gpu.buf_from(a)
    gu, dn = iq3x_pack(gpu, up(h["gate"][lo:hi]), up(h["up"][lo:hi]), up(h["down"][lo:hi]), hi - lo, D, I)
    sgu, sdn = iq3x_pack(gpu, up(h["sg"]), up(h["su"]), up(h["sd"]), 1, D, I)
    sel, lg, xb = gpu.buf(gpu.L.qw_moe_sel_wide_bytes()).zero(), gpu.buf(nb * (E + 1) * 4), up(x)
    Wr, wsg = up(h["Wr"]), up(h["wsg"])
    scr, Pg = gpu.buf(8192 + rows * 16 * 2 * I * 2).zero(), gpu.buf(rows * (topk + 1) * D * 4).zero()
    b = gpu.batch()
    b.kernel(k["moe_route"]).buf(0, Wr).buf(1, wsg).buf(2, xb).buf(3, lg).bytes(14, u32(nb, lo, hi)).dispatch((1,), (1024,))
    b.kernel(k["moe_topk_wide"]).buf(0, lg).buf(1, sel).bytes(2, u32(nb, lo, hi)).dispatch((1,), (128,))
    b.kernel(k["moe_group_wide"]).buf(1, sel).bytes(2, u32(nb, lo, hi)).dispatch((1,), (512,))
    b.kernel(k["moe_ffn"]).buf(0, gu).buf(2, sgu).buf(4, xb).buf(5, sel).buf(6, dn).buf(7, sdn).buf(8, scr).buf(9, Pg).bytes(10, u32(lo))
    if say:
        b.bytes(13, u32(nb))
    b.dispatch((1,), (256,)).end()
    ids, _ = orc.topk(lg.download(np.float32, nb * (E + 1)).reshape(nb, E + 1)[:, :E], topk)
    return Pg.download(np.float32, nb * (topk + 1) * D).reshape(nb, topk + 1, D), ids


def test_wide_ffn_of_a_range_of_experts(gpu):
    """The expert FFN of a piece on a slice of the experts writes the rows of those experts (and the shared one's) and no others; the slices' rows together are
    the step kernel's, bit for bit."""
    E, topk, B = 64, 10, 150
    layer, h, _ = make_layer(gpu, E, 2048, 512, topk, seed=6, ffn="iq3x")
    x = synth.acts_fp16(np.random.default_rng(12), B, 2048)
    want = []
    for t in range(0, B, 64):
        run_layer(gpu, layer, x[t:t + 64])
        n = len(x[t:t + 64])
        want.append(layer.Pg.download(np.float32, n * (topk + 1) * 2048).reshape(n, topk + 1, 2048))
    want = np.concatenate(want)
    whole, ids = wide_ffn(gpu, h, x, E, topk)
    assert np.array_equal(whole.view(np.uint32), want.view(np.uint32))
    for lo, hi in ((0, 32), (32, 64)):
        part, _ = wide_ffn(gpu, h, x, E, topk, lo, hi)
        mine = (ids >= lo) & (ids < hi)
        assert np.all(part[:, :topk][~mine] == 0)
        assert np.array_equal(part[:, :topk][mine].view(np.uint32), want[:, :topk][mine].view(np.uint32))
        assert np.array_equal(part[:, topk].view(np.uint32), want[:, topk].view(np.uint32))


def test_wide_ffn_with_room_for_half_a_piece(gpu):
    """Pg and scratch for 512 tokens do for pieces of up to 512; more are refused, by the launcher or (where it is not told their number) by the kernel."""
    from qwental_b200.gpu import GpuError
    E, topk = 64, 2
    _, h, _ = make_layer(gpu, E, 2048, 512, topk, seed=7, ffn="iq3x")
    x = synth.acts_fp16(np.random.default_rng(3), 513, 2048)
    want, _ = wide_ffn(gpu, h, x, E, topk)
    for say in (True, False):
        got, _ = wide_ffn(gpu, h, x[:512], E, topk, rows=512, say=say)
        assert np.array_equal(got.view(np.uint32), want[:512].view(np.uint32))
    for say in (True, False):
        with pytest.raises(GpuError):
            wide_ffn(gpu, h, x, E, topk, rows=513, say=say)
    with pytest.raises(GpuError):
        wide_ffn(gpu, h, x[:100], E, topk, rows=511)


@pytest.mark.parametrize("D,nb", [(2048, 3), (2048, 64), (2048, 65), (2048, 143), (256, 4), (256, 65), (256, 200)])
def test_logits_alone_are_those_of_the_router(gpu, D, nb):
    """moe_route with SELECT defined 0, in the form for many tokens and in the other one: the canonical-order logits, bit for bit."""
    from qwental_b200.layers import u32
    E = 64
    rng = np.random.default_rng(nb)
    Wr, wsg = (rng.standard_normal((E, D)) * 0.02).astype(np.float16), (rng.standard_normal(D) * 0.02).astype(np.float16)
    x = synth.acts_fp16(rng, nb, D)
    k = gpu.compile("moe_route", "t_logits_%d" % D, E=E, D=D, TOPK=4, SELECT=0)
    b = [gpu.buf_from(a) for a in (Wr, wsg, x)] + [gpu.buf(nb * (E + 1) * 4)]
    gpu.batch().kernel(k).buf(0, b[0]).buf(1, b[1]).buf(2, b[2]).buf(3, b[3]).bytes(14, u32(nb, 0, E)).dispatch((1,), (1024,)).end()
    got = b[3].download(np.uint32, nb * (E + 1)).reshape(nb, E + 1)
    assert np.array_equal(got, orc.router_canon(np.concatenate([Wr, wsg[None]]), x).view(np.uint32))


@pytest.mark.parametrize("nb", [65, 131])
def test_combine_and_norm_of_many_rows_wherever_the_buffers_lie(gpu, nb):
    """More than 64 rows of the combine + norm go by 16-byte loads where all buffers lie at such boundaries, and column by column where one does not: the same bits."""
    import ctypes as C
    from qwental_b200.layers import u32
    D, topk = 2048, 10
    rng = np.random.default_rng(nb)
    gpu.L.qw_moe_sel_wide_bytes.restype = C.c_size_t
    k = gpu.compile("add_rmsnorm", "t_cmb_wide", CMB=1, TOPK=topk, WIDE=1, ROWS=1024)
    sel = gpu.buf(gpu.L.qw_moe_sel_wide_bytes()).zero()
    sel.upload(rng.random((nb, 17)).astype(np.float32), 16 + 64 * 16 * 4)
    h, Pg = rng.standard_normal((nb, D)).astype(np.float32), rng.standard_normal((nb, topk + 1, D)).astype(np.float32)
    w, pg = gpu.buf_from((1 + 0.1 * rng.standard_normal(D)).astype(np.float32)), gpu.buf_from(Pg)

    def run(off):
        hb, x = gpu.buf(h.nbytes + 16).upload(h, off), gpu.buf(nb * D * 2)
        gpu.batch().kernel(k).buf(0, hb, off).buf(2, w).buf(3, x).buf(5, sel).buf(6, pg).bytes(4, u32(nb, D)).dispatch((nb,), (256,)).end()
        return hb.download(np.uint32, nb * D, off), x.download(np.uint16, nb * D)

    for a, b in zip(run(0), run(4)):
        assert np.array_equal(a, b)
