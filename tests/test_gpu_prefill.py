"""Prompt processing in pieces (qw_engine_par_prefill) against the decode step fed one token at a time: logits, recurrent and
conv state and KV pages bit for bit, at prompt lengths around the edges of a piece, of the convolution's window and of a KV page."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from qwental_b200.gpu import Gpu
    g = Gpu()
    yield g
    g.close()


def state_of(e, sid):
    c = e.cfg
    n_attn = c.layers // c.attn_every
    pages = e.tap("pages", sid, np.int32)
    kv = np.stack([e.tap("kvpage", int(p), np.float16).reshape(n_attn, 2, c.kvh, 256, c.hd) for p in pages])
    kv = np.moveaxis(kv, 0, 3).reshape(n_attn, 2, c.kvh, -1, c.hd)[:, :, :, :e.pos(sid)]
    return e.tap("sstate", sid, np.uint32), e.tap("cstate", sid, np.uint32), kv.view(np.uint16)


@pytest.mark.parametrize("model", ["tiny", "wide", "wide_fma"])
def test_prefill_equals_stepping_every_token(gpu, model):
    from qwental_b200.engine import Engine, tiny_cfg, wide_cfg
    e = Engine(gpu, tiny_cfg() if model == "tiny" else wide_cfg(fma=int(model == "wide_fma")))
    try:
        lengths = {1, 2, 3, 4, 5, 63, 64, 65, 67, 128, 257} if model != "wide_fma" else {3, 66}
        text = np.random.default_rng(4).integers(0, e.cfg.vocab, max(lengths)).astype(np.int32)
        e.prefill(0, text[:1])  # slot 0 steps every token
        for n in range(1, max(lengths) + 1):
            if n > 1:
                lg, _ = e.step([0], text[n - 1:n])
            if n not in lengths:
                continue
            e.seed_slot(5, 40, n)  # the slot was in use
            got = e.prefill(5, text[:n])
            assert e.pos(5) == n
            if n > 1:
                assert np.array_equal(got.view(np.uint32), lg[0].view(np.uint32)), n
            for a, b in zip(state_of(e, 5), state_of(e, 0)):
                assert np.array_equal(a, b), n
    finally:
        e.close()


def test_recurrence_around_the_edges_of_its_buffers(gpu):
    """The recurrence stages 16 tokens at a time and adds up outputs a buffer later: one less, as many and one more than one to four buffers."""
    from qwental_b200.engine import Engine, tiny_cfg
    e = Engine(gpu, tiny_cfg())
    try:
        lengths = {15, 16, 17, 18, 31, 32, 33, 34, 47, 48, 49}
        text = np.random.default_rng(9).integers(0, e.cfg.vocab, max(lengths)).astype(np.int32)
        e.prefill(0, text[:1])  # slot 0 steps every token
        for n in range(2, max(lengths) + 1):
            lg, _ = e.step([0], text[n - 1:n])
            if n not in lengths:
                continue
            got = e.prefill(5, text[:n])
            assert np.array_equal(got.view(np.uint32), lg[0].view(np.uint32)), n
            for a, b in zip(state_of(e, 5), state_of(e, 0)):
                assert np.array_equal(a, b), n
    finally:
        e.close()


def test_wide_pieces_equal_stepping_every_token(gpu):
    """Pieces of 65 to 577 tokens (512 experts, ten per token: several items per expert and most experts chosen), at the edges of the groups of 64 rows
    inside them and of half a piece, whose rest of up to 64 tokens goes by itself."""
    from qwental_b200.engine import Engine, wide_cfg
    e = Engine(gpu, wide_cfg(experts=512, topk=10, max_slots=2))
    try:
        lengths = {65, 127, 192, 193, 255, 256, 257, 321, 511, 512, 513, 515, 550, 576, 577}
        text = np.random.default_rng(5).integers(0, e.cfg.vocab, max(lengths)).astype(np.int32)
        e.prefill(0, text[:1])  # slot 0 steps every token
        for n in range(2, max(lengths) + 1):
            lg, _ = e.step([0], text[n - 1:n])
            if n not in lengths:
                continue
            got = e.prefill(1, text[:n])
            assert np.array_equal(got.view(np.uint32), lg[0].view(np.uint32)), n
            for a, b in zip(state_of(e, 1), state_of(e, 0)):
                assert np.array_equal(a, b), n
    finally:
        e.close()


@pytest.mark.parametrize("ffn", ["fused", "split"])
def test_prompts_with_the_other_expert_kernels(gpu, ffn, monkeypatch):
    """Engines whose experts are not re-coded run prompts in pieces of 64: nearly all of 512 experts chosen, several pieces."""
    from qwental_b200.engine import Engine, wide_cfg
    monkeypatch.setenv("QW_MOE_FFN", ffn)
    e = Engine(gpu, wide_cfg(experts=512, topk=10, max_slots=2))
    try:
        text = np.random.default_rng(7).integers(0, e.cfg.vocab, 200).astype(np.int32)
        e.prefill(0, text[:1])
        for n in range(2, len(text) + 1):
            lg, _ = e.step([0], text[n - 1:n])
        got = e.prefill(1, text)
        assert np.array_equal(got.view(np.uint32), lg[0].view(np.uint32))
        for a, b in zip(state_of(e, 1), state_of(e, 0)):
            assert np.array_equal(a, b)
    finally:
        e.close()


@pytest.mark.parametrize("n,kernel,family,broken,whole", [(40, "gdn_gate", "gdn_gate", dict(DV=64), dict()), (540, "kb_embed", "kb_embed", dict(ROWS=8), dict())])
def test_a_failed_prompt_frees_its_slot(gpu, n, kernel, family, broken, whole):
    """A launch that the host refuses (a kernel specialised so that its argument check fails) in the first piece, or in the last one after a piece
    of 512 tokens has gone through: the prompt fails, its slot is free -- no step runs on what the pieces left -- and the same prompt works afterwards."""
    from qwental_b200.engine import Engine, wide_cfg
    from qwental_b200.gpu import GpuError
    e = Engine(gpu, wide_cfg(max_slots=2, kv_pages=4))
    try:
        text = np.random.default_rng(n).integers(0, e.cfg.vocab, n).astype(np.int32)
        want = e.prefill(1, text)
        e.finish(1)
        gpu.compile(family, kernel, HK=16, HV=32, **broken)
        with pytest.raises(GpuError):
            e.prefill(0, text)
        gpu.compile(family, kernel, HK=16, HV=32, **whole)
        assert e.pos(0) == -1 and e.mem() == 0
        with pytest.raises(GpuError, match="not in use"):
            e.step([0], [1])
        got = e.prefill(1, text)  # all pages are there again, and nothing of the failed launches is left
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
        assert e.pos(1) == n
    finally:
        e.close()


@pytest.mark.parametrize("n", [2, 40, 130, 600])
def test_records_after_a_prompt_are_those_of_its_last_token(gpu, n):
    """The selection record and the step's byte counts after a prompt (pieces of up to 64 tokens and wider ones keep different records on the
    device) equal those after stepping its last token; h, x and logits are that token's."""
    from qwental_b200.engine import Engine, wide_cfg
    e = Engine(gpu, wide_cfg(experts=256, topk=6, max_slots=2))
    try:
        text = np.random.default_rng(n).integers(0, e.cfg.vocab, n).astype(np.int32)

        def records():
            out = []
            for l in range(e.cfg.layers):
                r = e.tap("sel", l, np.uint8)
                U, nb, topk = (int(v) for v in r[:12].view(np.uint32))
                at = np.cumsum([16, 64 * 16 * 4, 64 * 17 * 4, 1024 * 4, 1025 * 4, 1024 * 2])
                f = lambda i, t, k: r[at[i]:].view(np.uint8)[:k * np.dtype(t).itemsize].view(t).tolist()
                out.append((U, nb, topk, f(0, np.int32, topk), f(1, np.uint32, topk + 1), f(2, np.uint32, U), f(3, np.uint32, U + 1), f(4, np.uint16, U),
                            f(5, np.uint32, U + 1)))
            b = e.step_bytes()
            return out, [getattr(b, k) for k, _ in b._fields_], [e.tap(t, 0, np.uint16).tolist() for t in ("h", "x", "logits")]
        e.prefill(0, text)
        got = records()
        e.prefill(1, text[:-1])
        e.step([1], text[-1:])
        want = records()
        assert all(r[0] == 6 and r[1] == 1 for r in want[0])
        assert got == want
    finally:
        e.close()


def test_attention_over_the_rows_of_a_piece(gpu):
    """The attention core takes 16 rows of a piece per (page, kv head): pieces around multiples of 16 rows, rows that end in every part of a tile, pages that some
    rows of a block reach and others do not, pieces behind earlier ones, and (4300 tokens) more than 16 pages, which go through the general merge."""
    from qwental_b200.engine import Engine, wide_cfg
    e = Engine(gpu, wide_cfg(layers=3, attn_every=2, max_slots=2, max_ctx=4608))
    try:
        lengths = {65, 79, 80, 81, 127, 255, 256, 257, 263, 271, 272, 300, 511, 590, 777, 1024, 1100, 1301, 2000, 4300}
        text = np.random.default_rng(17).integers(0, e.cfg.vocab, max(lengths)).astype(np.int32)
        e.prefill(0, text[:1])  # slot 0 steps every token
        for n in range(2, max(lengths) + 1):
            lg, _ = e.step([0], text[n - 1:n])
            if n not in lengths:
                continue
            got = e.prefill(1, text[:n])
            assert np.array_equal(got.view(np.uint32), lg[0].view(np.uint32)), n
            for a, b in zip(state_of(e, 1), state_of(e, 0)):
                assert np.array_equal(a, b), n
    finally:
        e.close()


def test_pieces_of_up_to_1024_tokens(gpu):
    """One piece of 577 to 1024 tokens, and what is left after 1024: one token, one of the rests that go by themselves, more."""
    from qwental_b200.engine import Engine, wide_cfg
    e = Engine(gpu, wide_cfg(experts=512, topk=10, layers=4, max_slots=2))
    try:
        lengths = {578, 1023, 1024, 1025, 1100, 1560}
        text = np.random.default_rng(15).integers(0, e.cfg.vocab, max(lengths)).astype(np.int32)
        e.prefill(0, text[:1])  # slot 0 steps every token
        for n in range(2, max(lengths) + 1):
            lg, _ = e.step([0], text[n - 1:n])
            if n not in lengths:
                continue
            got = e.prefill(1, text[:n])
            assert np.array_equal(got.view(np.uint32), lg[0].view(np.uint32)), n
            for a, b in zip(state_of(e, 1), state_of(e, 0)):
                assert np.array_equal(a, b), n
    finally:
        e.close()


@pytest.mark.parametrize("experts,topk", [(32, 15), (512, 1), (64, 2), (512, 10)])
def test_expert_items_of_a_piece(gpu, experts, topk):
    """The expert FFN of a piece takes items of up to 16 columns, two stages of 128 rows side by side: experts with hundreds of tokens (full items, a
    remainder of one column and of one tile), with one token or none, and a work list shorter than the number of blocks."""
    from qwental_b200.engine import Engine, wide_cfg
    e = Engine(gpu, wide_cfg(experts=experts, topk=topk, layers=2, attn_every=2, max_slots=2))
    try:
        lengths = {66, 129, 145, 192, 400, 512}
        text = np.random.default_rng(13).integers(0, e.cfg.vocab, max(lengths)).astype(np.int32)
        e.prefill(0, text[:1])  # slot 0 steps every token
        for n in range(2, max(lengths) + 1):
            lg, _ = e.step([0], text[n - 1:n])
            if n not in lengths:
                continue
            got = e.prefill(1, text[:n])
            assert np.array_equal(got.view(np.uint32), lg[0].view(np.uint32)), n
    finally:
        e.close()


@pytest.mark.parametrize("layers,every", [(4, 4), (5, 4), (1, 1), (3, 2)])
def test_last_layer_of_a_prompt(gpu, layers, every):
    """After the last layer's K, V and state only the prompt's last token goes on: Gated DeltaNet and attention as the last layer, one piece and several
    (the last one of a single token too), then a step on the state left behind."""
    from qwental_b200.engine import Engine, wide_cfg
    e = Engine(gpu, wide_cfg(layers=layers, attn_every=every, max_slots=2))
    try:
        lengths = {2, 64, 66, 200, 513}
        text = np.random.default_rng(11).integers(0, e.cfg.vocab, max(lengths)).astype(np.int32)
        e.prefill(0, text[:1])  # slot 0 steps every token
        for n in range(2, max(lengths) + 1):
            lg, _ = e.step([0], text[n - 1:n])
            if n not in lengths:
                continue
            got = e.prefill(1, text[:n])
            assert np.array_equal(got.view(np.uint32), lg[0].view(np.uint32)), n
            for a, b in zip(state_of(e, 1), state_of(e, 0)):
                assert np.array_equal(a, b), n
        both, _ = e.step([0, 1], [7, 7])
        assert np.array_equal(both[0].view(np.uint32), both[1].view(np.uint32))
    finally:
        e.close()


@pytest.mark.parametrize("experts", [32, 512])
def test_a_full_piece_with_the_most_choices(gpu, experts):
    """1023 and 1024 tokens with 15 experts each: every row of the FFN's H (15360 entries and the shared expert's 1024), the most items a block's share can touch (512
    experts) and experts with some 480 entries (32)."""
    from qwental_b200.engine import Engine, wide_cfg
    e = Engine(gpu, wide_cfg(experts=experts, topk=15, layers=2, attn_every=2, max_slots=2))
    try:
        text = np.random.default_rng(experts).integers(0, e.cfg.vocab, 1024).astype(np.int32)
        e.prefill(0, text[:1])  # slot 0 steps every token
        for n in range(2, 1025):
            lg, _ = e.step([0], text[n - 1:n])
            if n < 1023:
                continue
            got = e.prefill(1, text[:n])
            assert np.array_equal(got.view(np.uint32), lg[0].view(np.uint32)), n
            for a, b in zip(state_of(e, 1), state_of(e, 0)):
                assert np.array_equal(a, b), n
    finally:
        e.close()


@pytest.mark.parametrize("hk,hv", [(16, 16), (16, 48), (8, 64)])
def test_prompts_with_other_numbers_of_value_heads(gpu, hk, hv):
    """Other numbers of Gated DeltaNet heads than 16 and 32: the recurrence in more than one wave of blocks (48 and 64 value heads on 148 SMs), channels that fill the
    epilogue's blocks in part, output projections without a form for wide pieces."""
    from qwental_b200.engine import Engine, wide_cfg
    e = Engine(gpu, wide_cfg(layers=3, attn_every=2, hk=hk, hv=hv, max_slots=2))
    try:
        lengths = {2, 17, 64, 65, 130, 300}
        text = np.random.default_rng(hv).integers(0, e.cfg.vocab, max(lengths)).astype(np.int32)
        e.prefill(0, text[:1])  # slot 0 steps every token
        for n in range(2, max(lengths) + 1):
            lg, _ = e.step([0], text[n - 1:n])
            if n not in lengths:
                continue
            got = e.prefill(1, text[:n])
            assert np.array_equal(got.view(np.uint32), lg[0].view(np.uint32)), n
            for a, b in zip(state_of(e, 1), state_of(e, 0)):
                assert np.array_equal(a, b), n
    finally:
        e.close()
