"""GPU parity of the full decode step through the engine C ABI (benchmark config 4 at two reduced model sizes, so
the FP64 oracle finishes in seconds: "tiny" shrinks every dimension, "wide" keeps the full-size layer shapes and with
them the kernel variants of the benchmark model): logits within fp16 tolerance of the chained FP64 reference with top-1
agreement, chosen experts identical, batched rows bit-identical to each slot alone, chained greedy decode equal to
step-by-step decode, CUDA-graph replay equal to plain launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from qwental_b200.gpu import Gpu
    g = Gpu()
    yield g
    g.close()


@pytest.fixture(scope="module", params=["tiny", "wide"])
def eng(gpu, request):
    from qwental_b200.engine import Engine, tiny_cfg, wide_cfg
    e = Engine(gpu, tiny_cfg() if request.param == "tiny" else wide_cfg())
    yield e
    e.close()


CTX = {0: 300, 3: 5, 5: 777, 6: 255}


def seed_all(eng):
    for sid, n in CTX.items():
        eng.seed_slot(sid, n, 1000 + sid)


def test_step_logits_match_fp64_reference(eng):
    from oracle.model_ref import RefModel
    seed_all(eng)
    ref = RefModel(eng.cfg, eng)
    sids = [0, 3, 5, 6]
    toks = [7, 100, 511, 0]
    states = {s: ref.read_slot(eng, s) for s in sids}
    logits, ms = eng.step(sids, toks)
    assert ms > 0 and logits.shape == (4, eng.cfg.vocab) and np.isfinite(logits).all()
    h = eng.tap("h", 0, np.float32).reshape(4, -1)
    for i, s in enumerate(sids):
        dev_ids = [eng.tap("sel", l, np.uint8)[16:16 + 64 * 16 * 4].view(np.int32).reshape(64, 16)[i, :eng.cfg.topk] for l in range(eng.cfg.layers)]
        lg, hh, chosen = ref.step(states[s], toks[i], ids_by_layer=dev_ids)
        scale = np.abs(lg).max()
        assert np.abs(logits[i] - lg).max() < 2e-2 * scale, (s, np.abs(logits[i] - lg).max(), scale)
        assert int(logits[i].argmax()) == int(lg.argmax())
        assert eng.pos(s) == CTX[s] + 1
    # the slot state the device left behind matches the reference's (KV append, GDN state)
    for s in sids:
        after = ref.read_slot(eng, s)
        assert np.abs(after["S"] - states[s]["S"]).max() < 1e-3 * max(1.0, np.abs(states[s]["S"]).max())
        p = CTX[s]
        assert np.abs(after["kv"][:, :, :, p].astype(np.float64) - states[s]["kv"][:, :, :, p].astype(np.float64)).max() < 2e-2


def test_batched_rows_bit_identical_to_alone(eng):
    sids, toks = [0, 3, 5, 6], [11, 12, 13, 14]
    seed_all(eng)
    lb, _ = eng.step(sids, toks)
    for i, s in enumerate(sids):
        seed_all(eng)
        la, _ = eng.step([s], [toks[i]])
        assert np.array_equal(la[0].view(np.uint32), lb[i].view(np.uint32)), s
    # order of rows does not matter either
    seed_all(eng)
    lp, _ = eng.step([6, 0], [14, 11])
    assert np.array_equal(lp[0].view(np.uint32), lb[3].view(np.uint32)) and np.array_equal(lp[1].view(np.uint32), lb[0].view(np.uint32))


def test_greedy_chain_equals_stepwise_and_graph_replay(eng, gpu):
    sids, toks = [0, 5], [3, 4]
    seed_all(eng)
    ids_chain, _ = eng.decode_greedy(sids, toks, 4)
    seed_all(eng)
    cur = list(toks)
    for k in range(4):
        ids, _ = eng.step_greedy(sids, cur)
        assert np.array_equal(ids, ids_chain[k])
        cur = list(ids)
    # logits path gives the same arg-max (ties -> lowest id)
    seed_all(eng)
    lg, _ = eng.step(sids, toks)
    assert np.array_equal(lg.argmax(1).astype(np.int32), ids_chain[0])
    gpu.L.qw_gpu_set_graphs(gpu.g, True)
    try:
        seed_all(eng)
        ids_graph, _ = eng.decode_greedy(sids, toks, 4)
    finally:
        gpu.L.qw_gpu_set_graphs(gpu.g, False)
    assert np.array_equal(ids_graph, ids_chain)


def test_slot_errors_and_accounting(eng):
    from qwental_b200.gpu import GpuError
    seed_all(eng)
    with pytest.raises(GpuError):
        eng.step([0, 0], [1, 2])            # the same slot twice
    with pytest.raises(GpuError):
        eng.step([1], [1])                  # slot never seeded
    with pytest.raises(GpuError):
        eng.step([0], [eng.cfg.vocab])      # token out of range
    with pytest.raises(GpuError):
        eng.step([], [])                    # an empty batch
    with pytest.raises(GpuError):
        eng.step(list(range(65)), [0] * 65) # more rows than QW_PAR_MAX
    eng.seed_slot(7, eng.cfg.max_ctx - 1, 9)  # the last position that fits
    eng.step([7], [1])
    with pytest.raises(GpuError):
        eng.step([7], [1])                  # one more would exceed max_ctx
    eng.finish(7)
    lg, _ = eng.step([0, 3], [1, 2])        # the engine is still usable
    b = eng.step_bytes()
    c = eng.cfg
    assert b.ctx_tokens == (CTX[0] + 1) + (CTX[3] + 1)
    assert 1 <= b.unique_experts_sum <= c.layers * 2 * c.topk
    assert b.total == pytest.approx(b.moe + b.dense + b.lm_head + b.kv + b.gdn_state + b.other)
    assert eng.mem() > 0 and eng.cost(2) > 0
    assert eng.pick(busy=0b1111111) == 7
    eng.finish(3)
    assert eng.pos(3) == -1 and eng.pick(busy=0) in (1, 2, 3, 4, 7)


@pytest.mark.parametrize("attn_every", [4, 1])
def test_fresh_engines_agree_bit_for_bit(gpu, attn_every):
    """Two engines opened one after the other (so the second one's buffers hold the first one's leftovers) produce the
    same logits, bit for bit, with dependent launch on: a kernel that read its predecessor's output too early, or through a
    non-coherent path, shows up here as run-to-run noise."""
    from qwental_b200.engine import Engine, wide_cfg
    outs = []
    for _ in range(3):
        e = Engine(gpu, wide_cfg(layers=2, attn_every=attn_every))
        for sid, n in CTX.items():
            e.seed_slot(sid, n, 1000 + sid)
        lg, _ = e.step([0, 3, 5, 6], [7, 100, 511, 0])
        lg2, _ = e.step([0, 5], [1, 2])
        outs.append((lg.copy(), lg2.copy()))
        e.close()
    for a, b2 in outs[1:]:
        assert np.array_equal(a.view(np.uint32), outs[0][0].view(np.uint32))
        assert np.array_equal(b2.view(np.uint32), outs[0][1].view(np.uint32))


def test_full_batch_of_64_rows_matches_each_slot_alone(gpu):
    """The largest batch the step accepts (QW_PAR_MAX = 64 rows, contexts straddling page boundaries): a sample of its rows
    is bit-identical to the same slots stepped alone, on both model sizes' kernel variants."""
    from qwental_b200.engine import Engine, tiny_cfg, wide_cfg
    for cfg in (tiny_cfg(max_slots=64, max_ctx=1024), wide_cfg(max_slots=64, max_ctx=1024, layers=2)):
        e = Engine(gpu, cfg)
        ctx = {s: [1, 255, 256, 257, 511, 512, 700, 33][s % 8] + s for s in range(64)}

        def seed():
            for s, n in ctx.items():
                e.seed_slot(s, n, 5000 + s)
        seed()
        sids = list(range(63, -1, -1))
        toks = [(s * 37 + 11) % cfg.vocab for s in sids]
        lb, _ = e.step(sids, toks)
        assert np.isfinite(lb).all()
        for i in (0, 7, 31, 40, 63):
            seed()
            la, _ = e.step([sids[i]], [toks[i]])
            assert np.array_equal(la[0].view(np.uint32), lb[i].view(np.uint32)), (cfg.hidden, sids[i])
        e.close()


def test_benchmark_layer_shapes_match_fp64_reference(gpu):
    """Four layers of the benchmark model itself (hidden 2048, 512 experts with top-10, 151 936-token vocabulary; three
    Gated DeltaNet layers and one attention layer) against the chained FP64 reference: logits within tolerance, top-1
    equal, chosen experts taken from the device and checked to be the reference's own top-10 wherever its margin is clear."""
    from oracle.model_ref import RefModel
    from qwental_b200.engine import Engine, default_cfg
    e = Engine(gpu, default_cfg(layers=4, max_slots=4, max_ctx=2048, kv_pages=0, seed=3))
    try:
        ctx = {0: 700, 2: 255, 3: 40}
        for sid, n in ctx.items():
            e.seed_slot(sid, n, 2000 + sid)
        ref = RefModel(e.cfg, e)
        sids, toks = [3, 0, 2], [11, 150000, 77]
        states = {s: ref.read_slot(e, s) for s in sids}
        logits, _ = e.step(sids, toks)
        assert np.isfinite(logits).all()
        for i, s in enumerate(sids):
            dev_ids = [e.tap("sel", l, np.uint8)[16:16 + 64 * 16 * 4].view(np.int32).reshape(64, 16)[i, :e.cfg.topk] for l in range(e.cfg.layers)]
            lg, hh, chosen = ref.step(states[s], toks[i], ids_by_layer=dev_ids)
            scale = np.abs(lg).max()
            assert np.abs(logits[i] - lg).max() < 2e-2 * scale, (s, np.abs(logits[i] - lg).max(), scale)
            assert int(logits[i].argmax()) == int(lg.argmax())
    finally:
        e.close()


def test_prefill_is_the_decode_path_token_by_token(gpu):
    """qw_engine_par_prefill, in pieces, computes what the decode step computes token by token: prefill(p) equals prefill(p[:-1]) followed by one
    step of p[-1], bit for bit; the result does not depend on the slot; a slot that was in use is emptied first; a
    prefilled slot steps together with a seeded one exactly as it steps alone."""
    from qwental_b200.engine import Engine, tiny_cfg
    from qwental_b200.gpu import GpuError
    e = Engine(gpu, tiny_cfg())
    try:
        prompt = [5, 17, 300, 4, 4, 511, 0, 260, 33]
        full = e.prefill(1, prompt)
        assert e.pos(1) == len(prompt) and np.isfinite(full).all()
        part = e.prefill(4, prompt[:-1])
        lg, _ = e.step([4], [prompt[-1]])
        assert np.array_equal(lg[0].view(np.uint32), full.view(np.uint32))
        e.seed_slot(2, 300, 77)  # slot 2 in use with other contents: prefill starts it over
        again = e.prefill(2, prompt)
        assert np.array_equal(again.view(np.uint32), full.view(np.uint32)) and e.pos(2) == len(prompt)
        a, _ = e.step([1], [9])
        e.prefill(1, prompt)
        e.seed_slot(6, 500, 5)
        b, _ = e.step([6, 1], [3, 9])
        assert np.array_equal(b[1].view(np.uint32), a[0].view(np.uint32))
        with pytest.raises(GpuError):
            e.prefill(0, [e.cfg.vocab])
        with pytest.raises(GpuError):
            e.prefill(99, [1])
    finally:
        e.close()


def test_benchmark_engine_full_depth_batched_equals_alone_and_graph_replay(gpu):
    """The benchmark engine itself -- all 48 layers, the 16 ragged conversations bench.py steps (contexts log-uniform in
    1K..48K, the same seeds) -- needs no oracle for the reference's own guarantee (src/engine.c:7977-7986,
    tools/run.c:217-229): three rows of the 16-row step are bit-identical to the same slots stepped alone, and the step
    replayed as a CUDA graph gives the bytes of the plain launches."""
    from qwental_b200 import synth
    from qwental_b200.engine import Engine, default_cfg
    B = 16
    ctx = synth.ragged_contexts(np.random.default_rng(0), B)
    pages = int(sum((int(n) + 64 + 256) // 256 + 1 for n in ctx))
    e = Engine(gpu, default_cfg(max_slots=B, max_ctx=int(ctx.max()) + 1024, kv_pages=pages, seed=0))
    try:
        def seed(rows):
            for s in rows:
                e.seed_slot(s, int(ctx[s]), 100 + s)
        sids = np.arange(B, dtype=np.int32)
        toks = (np.arange(B, dtype=np.int32) * 7919) % e.cfg.vocab
        seed(range(B))
        lb, _ = e.step(sids, toks)
        assert np.isfinite(lb).all()
        longest, shortest = int(np.argmax(ctx)), int(np.argmin(ctx))
        for r in sorted({longest, shortest, 7}):
            seed([r])
            la, _ = e.step([r], [toks[r]])
            assert np.array_equal(la[0].view(np.uint32), lb[r].view(np.uint32)), (r, int(ctx[r]))
        gpu.L.qw_gpu_set_graphs(gpu.g, True)
        try:
            seed(range(B))
            e.step(sids, toks)        # records the graph
            seed(range(B))
            lg, _ = e.step(sids, toks)  # replays it
        finally:
            gpu.L.qw_gpu_set_graphs(gpu.g, False)
        assert np.array_equal(lg.view(np.uint32), lb.view(np.uint32))
    finally:
        e.close()


def test_step_logits_belong_to_the_caller(gpu):
    """Logits of earlier steps keep their values while they (or views of them) are held, however many; they outlive the engine."""
    from qwental_b200.engine import Engine, _HostRows, tiny_cfg
    cfg = tiny_cfg(vocab=8192)
    assert 8 * cfg.vocab * 4 >= _HostRows.SMALL > cfg.vocab * 4
    a, b = Engine(gpu, cfg), Engine(gpu, cfg)
    for e in (a, b):
        for s in range(8):
            e.seed_slot(s, 20 + s, 100 + s)
    rng = np.random.default_rng(6)
    held, want = [], []
    for k in range(8):
        rows = list(range(8)) if k % 3 else [5]
        toks = rng.integers(0, cfg.vocab, len(rows)).astype(np.int32)
        lg, _ = a.step(rows, toks)
        assert lg.flags.writeable and lg.flags.c_contiguous and lg.dtype == np.float32 and lg.shape == (len(rows), cfg.vocab)
        held.append(lg[1:] if len(rows) > 1 else lg)
        want.append(b.step(rows, toks)[0][-len(held[-1]):].copy())  # given back at once: the next step reuses its buffer
    a.close()
    for x, y in zip(held, want):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
    b.close()


def test_slot_table_is_read_ahead_only_behind_two_full_launches(gpu):
    """A step that begins with the control block's copy (par_begin) writes the slot table its GDN kernels find their state by: up to the second
    FFN launch after it they wait for the previous kernel first (the plain forms); from the third layer on, and in steps fed on the device, they
    may read ahead.  And rows that change their slots from step to step get the states of their own slots."""
    import ctypes as C
    from qwental_b200.engine import Engine, wide_cfg
    a, b = Engine(gpu, wide_cfg(layers=6)), Engine(gpu, wide_cfg(layers=6))
    try:
        def kernels(run):
            gpu.L.qw_profile_enable(gpu.g, True)
            run()
            names = [gpu.L.qw_profile_get(gpu.g, i, C.byref(C.c_double())).decode() for i in range(gpu.L.qw_profile_count(gpu.g))]
            gpu.L.qw_profile_enable(gpu.g, False)
            return names
        gdn = lambda names: [n for n in names if n.startswith(("dn_epi", "gdn_fstep"))]
        for e in (a, b):
            for s in range(8):
                e.seed_slot(s, 100 + 30 * s, 50 + s)
        plain, ahead = ["dn_epi", "gdn_fstep"], ["dn_epi_early", "gdn_fstep_early"]
        k1 = kernels(lambda: a.step([0, 1], [1, 2]))
        assert "par_begin" in k1 and gdn(k1) == 2 * plain + 3 * ahead  # layers 0, 1 | 2, 4, 5 (3 is attention)
        k2 = kernels(lambda: a.decode_greedy([2, 3], [5, 6], 2))  # what is profiled is the last batch: the step fed on the device
        assert "par_begin" not in k2 and gdn(k2) == 5 * ahead
        b.step([0, 1], [1, 2])
        b.decode_greedy([2, 3], [5, 6], 2)
        gpu.L.qw_gpu_set_graphs(gpu.g, True)
        rng = np.random.default_rng(8)
        try:
            for _ in range(40):
                rows = rng.permutation(8)[:rng.integers(1, 5)]
                toks = rng.integers(0, a.cfg.vocab, len(rows))
                la, _ = a.step(rows, toks)
                for i, s in enumerate(rows):
                    lb, _ = b.step([s], toks[i:i + 1])
                    assert np.array_equal(la[i].view(np.uint32), lb[0].view(np.uint32))
        finally:
            gpu.L.qw_gpu_set_graphs(gpu.g, False)
        for s in range(8):
            assert np.array_equal(a.tap("sstate", s, np.uint32), b.tap("sstate", s, np.uint32))
            assert np.array_equal(a.tap("cstate", s, np.uint32), b.tap("cstate", s, np.uint32))
    finally:
        a.close()
        b.close()


def test_a_rejected_step_leaves_the_last_logits_readable(gpu):
    """qw_engine_par_step gets memory for all rows with the first step of several rows.  The logits of a prompt stay where they are while such
    calls are rejected (a slot that is not in use, a slot twice, a token out of range) or fail on the device; the next good step replaces them."""
    import ctypes as C
    from qwental_b200.engine import Engine, tiny_cfg
    e = Engine(gpu, tiny_cfg())
    try:
        e.seed_slot(3, 50, 1)
        e.seed_slot(4, 60, 2)
        prompt = np.array([5, 17, 300], np.int32)
        L, V = e.L, e.cfg.vocab
        ip, i32p = C.POINTER(C.c_int), C.POINTER(C.c_int32)
        p = C.cast(L.qw_engine_par_prefill(e.e, 0, prompt.ctypes.data, 3, None), C.POINTER(C.c_float))
        want = np.ctypeslib.as_array(p, shape=(V,)).copy()

        def step(sids, toks):
            s, t = np.array(sids, np.int32), np.array(toks, np.int32)
            return L.qw_engine_par_step(e.e, s.ctypes.data_as(ip), t.ctypes.data_as(i32p), len(s), None)
        for sids, toks in (([0, 5], [1, 1]), ([3, 3], [1, 1]), ([3, 4], [1, V])):
            assert not step(sids, toks)
            assert np.array_equal(np.ctypeslib.as_array(p, shape=(V,)).view(np.uint32), want.view(np.uint32)), sids
        gpu.compile("kb_embed", "kb_embed", ROWS=1)  # two rows are refused at launch
        assert not step([3, 4], [1, 2])
        gpu.compile("kb_embed", "kb_embed")
        assert np.array_equal(np.ctypeslib.as_array(p, shape=(V,)).view(np.uint32), want.view(np.uint32))
        q = step([3, 4], [1, 2])
        both = np.ctypeslib.as_array(q, shape=(2, V)).copy()
        e.seed_slot(4, 60, 2)
        alone = step([4], [2])
        assert np.array_equal(np.ctypeslib.as_array(alone, shape=(V,)).view(np.uint32), both[1].view(np.uint32))
    finally:
        e.close()


def test_slices_of_a_buffer(gpu):
    """qw_buf_slice: the bytes of the whole, ranges of its own, freed without the whole's memory; out of range is refused."""
    import ctypes as C
    from qwental_b200.lib import QwBuf
    L, whole = gpu.L, gpu.buf_from(np.arange(4096, dtype=np.uint32))
    part = QwBuf()
    assert L.qw_buf_slice(C.byref(whole.b), 1024, 512, C.byref(part)) and part.size == 512
    got = np.empty(128, np.uint32)
    assert L.qw_buf_download(gpu.g, C.byref(part), 0, got.ctypes.data, 512) and np.array_equal(got, np.arange(256, 384))
    assert not L.qw_buf_download(gpu.g, C.byref(part), 4, got.ctypes.data, 512)
    assert L.qw_buf_zero(gpu.g, C.byref(part), 0, 512)
    L.qw_buf_free(C.byref(part))
    want = np.arange(4096, dtype=np.uint32)
    want[256:384] = 0
    assert np.array_equal(whole.download(np.uint32, 4096), want)
    for off, n in ((16384, 1), (16000, 385), (0, 16385), (0, 0), (2 ** 64 - 8, 16)):
        assert not L.qw_buf_slice(C.byref(whole.b), off, n, C.byref(part)), (off, n)


@pytest.mark.parametrize("start", [64, 65])
def test_replayed_steps_and_their_ids(gpu, start):
    """Greedy chains whose steps are submitted ahead leave their ids in alternating halves by the first row's position: chains of 1, 2 and 5
    steps from even and odd positions, recorded and replayed, against one step at a time; and again after another engine has registered the same
    kernels anew, which drops the recorded graphs."""
    from qwental_b200.engine import Engine, tiny_cfg
    a, b = Engine(gpu, tiny_cfg()), Engine(gpu, tiny_cfg())
    rows, toks = [2, 0, 1], np.array([3, 1, 2], np.int32)

    def run(e, n, ahead):
        for i, s in enumerate(rows):
            e.seed_slot(s, start + 7 * i, 90 + i)
        if ahead:
            return e.decode_greedy(rows, toks, n)[0], e.step(rows, toks)[0]
        ids, cur = [], toks
        for _ in range(n):
            cur = np.array(e.step_greedy(rows, cur)[0], np.int32)
            ids.append(cur)
        return np.array(ids), e.step(rows, toks)[0]

    try:
        want = {n: run(b, n, False) for n in (1, 2, 5)}
        gpu.L.qw_gpu_set_graphs(gpu.g, True)
        for rnd in range(3):
            for n in (1, 2, 5):
                for ahead in (True, False):
                    ids, lg = run(a, n, ahead)
                    assert np.array_equal(ids, want[n][0]) and np.array_equal(lg.view(np.uint32), want[n][1].view(np.uint32)), (rnd, n, ahead)
            if rnd == 1:
                Engine(gpu, tiny_cfg()).close()
    finally:
        gpu.L.qw_gpu_set_graphs(gpu.g, False)
        a.close()
        b.close()


def test_engines_open_with_less_memory_for_prompts(gpu):
    """What an engine cannot do without is allocated first, then the rows of a prompt's piece: 1024, or 512, or 64 where the memory is not there.  With ever less free
    memory the same prompt runs in 1, 2 and 16 pieces, to the same logits, before the engine no longer opens; and that happens no sooner than 64 rows need."""
    import torch
    from qwental_b200.engine import Engine, wide_cfg
    from qwental_b200.gpu import GpuError
    MB = 1 << 20
    free = lambda: torch.cuda.mem_get_info()[0]
    text = np.random.default_rng(2).integers(0, 512, 1024).astype(np.int32)

    def prompt():  # launches of the whole prompt, its logits, memory taken by the engine
        before = free()
        e = Engine(gpu, wide_cfg(max_slots=1))
        try:
            taken, n = before - free(), gpu.launches()
            lg = e.prefill(0, text)
            return gpu.launches() - n, lg, taken
        finally:
            e.close()

    prompt()  # (loads the kernels: what that takes is not the engine's)
    one, want, most = prompt()
    seen, left, least = [], most + 8 * MB, None
    while left > 0:
        filler = gpu.buf(free() - left)
        try:
            n, lg, _ = prompt()
        except GpuError as err:
            assert "allocation of" in str(err)
            break
        finally:
            filler.free()
        assert np.array_equal(lg.view(np.uint32), want.view(np.uint32)), left // MB
        if not seen or seen[-1] != n:
            seen.append(n)
        least = left
        left -= 20 * MB
    assert len(seen) == 3 and seen[0] == one and seen[1] < 3 * one and seen[2] > 10 * one, (one, seen)
    # 64 rows instead of 1024: 39 MB less of Pg (topk + 1 = 5 rows of 2048 fp32 per token), 33 of the FFN's scratch, 24 of projections, 25 of attention's partials, and so on
    assert most - least > 130 * MB, (most // MB, least // MB)



def ticket_calls(gpu):
    import ctypes as C
    L = gpu.L
    L.qw_batch_ticket.restype, L.qw_batch_ticket.argtypes = C.c_ulonglong, [C.c_void_p]
    L.qw_batch_replay.restype, L.qw_batch_replay.argtypes = C.c_void_p, [C.c_void_p, C.c_ulonglong]
    L.qw_gpu_set_pdl.restype, L.qw_gpu_set_pdl.argtypes = None, [C.c_void_p, C.c_bool]
    return L


def test_tickets_are_void_where_the_batch_would_be_another(gpu, monkeypatch):
    """A ticket replays its batch, and only while the recorded graph is what a new recording would give: not with graphs off, with profiling on, on another
    stream, in another launch mode (set through any device handle: the mode is the process's), after a kernel was registered anew, or once the graphs were dropped for
    others.  What is read from the environment once does not void it later."""
    from qwental_b200.gpu import Gpu
    L = ticket_calls(gpu)
    k = gpu.compile("qw_fill", "ticket_fill")
    buf = gpu.buf(1024)
    n = 256

    def fill(value, kind=5, keep=False):  # fills the buffer with a constant, then with its double
        b = gpu.batch()
        for v in (value, 2 * value):
            a = np.zeros(1, np.dtype([("seed", "<u8"), ("n", "<u8"), ("base", "<u8"), ("mode", "<u4"), ("p0", "<f4"), ("p1", "<f4"), ("pad", "<u4")]))
            a["n"], a["mode"], a["p0"] = n, kind, v
            b.kernel(k).buf(0, buf).bytes(1, a).dispatch((1,), (256,))
        L.qw_batch_submit(b.b)
        t = L.qw_batch_ticket(b.b)
        assert L.qw_batch_wait(b.b) >= 0
        b.b = None
        return t

    def replays(t):
        buf.zero()
        b = L.qw_batch_replay(gpu.g, t)
        if not b:
            return False
        assert L.qw_batch_wait(b) >= 0
        assert np.all(buf.download(np.float32, n) == 6.0)
        return True

    assert fill(3.0) == 0  # graphs are off: no ticket
    gpu.L.qw_gpu_set_graphs(gpu.g, True)
    other = Gpu()
    try:
        t = fill(3.0)
        assert t and replays(t) and replays(t) and not replays(t + 1) and not replays(0)
        for off, on in ((lambda: L.qw_gpu_set_graphs(gpu.g, False), lambda: L.qw_gpu_set_graphs(gpu.g, True)),
                        (lambda: L.qw_profile_enable(gpu.g, True), lambda: L.qw_profile_enable(gpu.g, False)),
                        (lambda: L.qw_gpu_set_stream(gpu.g, 1), lambda: L.qw_gpu_set_stream(gpu.g, 0)),
                        (lambda: L.qw_gpu_set_pdl(other.g, False), lambda: L.qw_gpu_set_pdl(other.g, True)),
                        (lambda: L.qw_gpu_set_pdl(None, False), lambda: L.qw_gpu_set_pdl(None, True))):
            off()
            try:
                assert not replays(t)
            finally:
                on()
            assert replays(t)
        monkeypatch.setenv("QW_PDL_OFF", "qw_fill")
        assert replays(t) and fill(3.0) == t
        L.qw_gpu_set_pdl(gpu.g, True)  # drops this device's graphs
        assert not replays(t)
        u = fill(3.0)
        assert u and u != t and replays(u)
        k = gpu.compile("qw_fill", "ticket_fill")
        assert not replays(u)
        u = fill(3.0)
        for i in range(256):
            assert replays(u)
            fill(100.0 + i)
        assert not replays(u) and fill(3.0) not in (0, t, u)
    finally:
        gpu.L.qw_gpu_set_graphs(gpu.g, False)
        other.close()



@pytest.mark.parametrize("graphs", [False, True])
def test_a_chain_whose_second_step_fails(gpu, graphs):
    """The step that is fed by the one before uses kernels the first one does not (the Gated DeltaNet forms that read ahead, in layers 0 and 1); one of them made to
    fail at launch, it fails while the first step runs: the call fails, the first step's ids are there, and the engine works on."""
    import ctypes as C
    from qwental_b200.engine import Engine, wide_cfg
    from qwental_b200.gpu import GpuError
    e = Engine(gpu, wide_cfg(layers=3, attn_every=3))
    gd = dict(HK=16, HV=32, DV=128, GDN_TILED=1, EARLY=1)

    def seed():
        for s in (0, 2):
            e.seed_slot(s, 70 + s, 9 + s)
    try:
        seed()
        want, _ = e.decode_greedy([0, 2], [5, 6], 3)
        gpu.L.qw_gpu_set_graphs(gpu.g, graphs)
        seed()
        out = np.full((3, 2), -7, np.int32)
        s, t = np.array([0, 2], np.int32), np.array([5, 6], np.int32)
        p = lambda a, ty: a.ctypes.data_as(C.POINTER(ty))
        gpu.compile("gdn_fstep", "gdn_fstep_early", **dict(gd, DV=64))
        assert e.L.qw_engine_par_decode_greedy(e.e, p(s, C.c_int), p(t, C.c_int32), 2, 3, p(out, C.c_int32), None) == -1
        assert "at step 1" in e.error() and np.array_equal(out[0], want[0]) and np.all(out[1:] == -7)
        with pytest.raises(GpuError):
            e.decode_greedy([0, 2], [5, 6], 2)
        gpu.compile("gdn_fstep", "gdn_fstep_early", **gd)
        seed()
        assert np.array_equal(e.decode_greedy([0, 2], [5, 6], 3)[0], want)
    finally:
        gpu.L.qw_gpu_set_graphs(gpu.g, False)
        e.close()
