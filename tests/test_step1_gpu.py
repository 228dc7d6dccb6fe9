"""A step of one sequence as one persistent launch (k_step1) against the same step as one launch per stage.

DeltaNet, experts and head add in the same order on both ways, so a model without attention has the same bits. The attention cuts its
context differently; each way is within 3e-4 of the oracle (test_kernel_edges), so they are within 6e-4 of one another (2e-3 each with
the bf16 cache, whose newest values round alike but meet a hidden state that differs in its last bits)."""
import importlib
import threading
import time

import numpy as np
import pytest

gpu = pytest.mark.gpu


@pytest.fixture(scope="module")
def E(pkg):
    return importlib.import_module("b200moe.engine")


def shape(pkg, name, layers):
    """The widths the kernel is built for: d_model / output width of the mixers / key width / head width / expert width."""
    cfg = pkg.HybridConfig.full(n_layers=layers)
    if name == "narrow":                     # mixers as wide as the model
        cfg.lin_k_heads, cfg.lin_v_heads, cfg.n_heads, cfg.head_dim, cfg.rotary_dim = 8, 16, 16, 128, 64
    if name == "half":
        cfg.d_model, cfg.expert_hidden, cfg.shared_hidden = 1024, 256, 256
        cfg.lin_k_heads, cfg.lin_v_heads, cfg.n_heads, cfg.head_dim, cfg.rotary_dim = 8, 16, 16, 128, 32
    if name != "full":
        cfg.vocab_size = 20008               # blocks' shares of the head that are no whole tiles
    return cfg


def pair(E, pkg, monkeypatch, cfg, kv, cap, keep=lambda name: True):
    from b200moe import brain
    dev = [t for t in brain.random_brain(cfg, seed=1, device="cuda:0", vary_1d=True) if keep(t[0])]
    one = E.HybridEngine.from_tensors(cfg.to_dict(), dev, max_context=cap, device=0, batch=1, kv_dtype=kv)
    monkeypatch.setenv("B2_NO_STEP1", "1")
    many = E.HybridEngine.from_tensors(cfg.to_dict(), dev, max_context=cap, device=0, batch=1, kv_dtype=kv)
    monkeypatch.delenv("B2_NO_STEP1")
    assert one.kernels_per_step() == 1 and many.kernels_per_step() > cfg.n_layers
    return one, many


@pytest.mark.parametrize("keys", [True, False])
@pytest.mark.parametrize("name", ["half", "narrow", "full", "few"])
def test_every_row_is_copied_once_and_no_copy_leaves_its_tensor(E, pkg, name, keys):
    """The layout of the persistent step, on the CPU. A brain without core engine tensors has no rows of theirs: with fewer experts than
    keys ("few") copies in their place would read past the router."""
    cfg = shape(pkg, "half" if name == "few" else name, 4)
    if name == "few":
        cfg.n_experts, cfg.core_grid = 64, (128, 128)
    plan = E.step1_plan(cfg.to_dict(), 148, keys)
    assert len(plan)
    D, C, HV, VD, SH, En = cfg.d_model, cfg.conv_dim, cfg.lin_v_heads, cfg.lin_v_heads * cfg.lin_v_dim, cfg.shared_hidden, cfg.n_experts
    q, kv = 2 * cfg.n_heads * cfg.head_dim, cfg.n_kv_heads * cfg.head_dim
    n1, n2 = cfg.core_grid if keys else (0, 0)
    # rows of a stage's matrices and bytes of a row; the tensors by the layer's pointer word, in bytes
    rows = {0: [(HV, 2 * D), (HV, 2 * D), (C, D), (VD, D)], 1: [(q, D), (kv, D), (kv, D)], 2: [(D, VD)],
            3: [(En, 2 * D), (n1, 2 * D), (n2, 2 * D), (1, 2 * D), (SH, D)], 4: [(D, SH)]}
    first_ptr = {0: 0, 1: 0, 2: 4, 3: 5, 4: 11}
    for kind, segs in rows.items():
        size = {first_ptr[kind] + i: n * rb for i, (n, rb) in enumerate(segs)}
        size.update({0: {12: 2 * C, 13: 2 * VD, 23: 8 * C, 24: 2 * HV, 25: 2 * HV, 26: 12 * C}, 1: {12: 2 * q, 13: 2 * kv, 14: 2 * kv},
                     2: {15: 2 * D}, 3: {10: SH * D, 16: 2 * SH, 17: 2 * SH, 28: 4 * En}, 4: {18: 2 * D}}[kind])
        of = plan[plan[:, 1] == kind]
        for ptr, at, n in of[:, 5:8]:
            assert at >= 0 and n > 0 and at % 16 == 0 and n % 16 == 0 and at + n <= size[ptr], (kind, ptr, at, n)
        for i, (n, rb) in enumerate(segs):
            for ptr in [first_ptr[kind] + i] + ([10] if (kind, i) == (3, 4) else []):
                got = of[(of[:, 2] == i) & (of[:, 5] == ptr) & (of[:, 8] < 0)]
                covered = np.zeros(n, np.int64)
                for _, _, _, _, _, _, at, size_, _ in got:
                    assert at % rb == 0 and size_ % rb == 0
                    covered[at // rb:(at + size_) // rb] += 1
                assert (covered == 1).all(), (kind, i, ptr)


@gpu
@pytest.mark.parametrize("name", ["half", "narrow", "full"])
def test_same_bits_without_attention(E, pkg, monkeypatch, name):
    cfg = shape(pkg, name, 3)
    one, many = pair(E, pkg, monkeypatch, cfg, E.KV_F32, 64)
    for tok in np.random.default_rng(3).integers(0, cfg.vocab_size, 6):
        a, b = (np.array(e.feed([int(tok)])) for e in (one, many))
        assert np.array_equal(a, b)
    for layer in range(cfg.n_layers):
        for a, b in zip(one.router(layer, cfg.experts_active), many.router(layer, cfg.experts_active)):
            assert np.array_equal(a, b), layer
    assert np.array_equal(one.core_counts(cfg.n_layers, cfg.n_cores), many.core_counts(cfg.n_layers, cfg.n_cores))
    one.close(); many.close()


@gpu
def test_routes_of_small_probabilities(E, pkg, monkeypatch):
    """Picks down to probabilities that are subnormal or 0, where ranks and weights hang on how the softmax is divided: the same picks and bits
    as a launch per stage."""
    cfg = shape(pkg, "half", 1)
    one, many = pair(E, pkg, monkeypatch, cfg, E.KV_F32, 64)
    rng = np.random.default_rng(0)
    for tok in range(40):
        bias = np.full(cfg.n_experts, -200, np.float32)
        top = rng.permutation(cfg.n_experts)[:12]
        bias[top] = -rng.uniform(0, 110, 12)
        bias[top[0]] = 0
        for e in (one, many):
            e.set_router_bias(0, bias)
            e.feed([tok])
        for a, b in zip(one.router(0, cfg.experts_active), many.router(0, cfg.experts_active)):
            assert np.array_equal(a, b)
    for at, value in ((slice(3, None), -np.inf), (slice(7, 8), np.inf), (slice(9, 10), np.nan)):
        bias = np.zeros(cfg.n_experts, np.float32)
        bias[at] = value
        for e in (one, many):
            e.crop(0)
            e.set_router_bias(0, bias)
            e.feed([1])
        for a, b in zip(one.router(0, cfg.experts_active), many.router(0, cfg.experts_active)):
            assert np.array_equal(a, b, equal_nan=True)
    one.close(); many.close()


@gpu
@pytest.mark.parametrize("which", ["none", "some layers"])
def test_brain_without_core_engine(E, pkg, monkeypatch, which):
    """Fewer experts than keys, and no keys: same bits as a launch per stage, and counts for the layers that have keys only."""
    cfg = shape(pkg, "half", 3)
    cfg.n_experts, cfg.core_grid = 64, (128, 128)
    one, many = pair(E, pkg, monkeypatch, cfg, E.KV_F32, 64, lambda name: not (".engine.key" in name and (which == "none" or "blocks.1." in name)))
    for tok in (5, 6, 7):
        a, b = (np.array(e.feed([tok])) for e in (one, many))
        assert np.array_equal(a, b)
    counts = one.core_counts(cfg.n_layers, cfg.n_cores)
    assert np.array_equal(counts, many.core_counts(cfg.n_layers, cfg.n_cores))
    n = 3 * cfg.cores_active
    assert counts.sum(1).tolist() == ([0, 0, 0] if which == "none" else [n, 0, n])
    one.close(); many.close()


@gpu
@pytest.mark.parametrize("kv", ["f32", "bf16"])
@pytest.mark.parametrize("name,context", [("half", 1), ("half", 15), ("half", 1184), ("narrow", 17), ("full", 16), ("full", 63),
                                          ("full", 64), ("full", 1183), ("full", 1185), ("full", 4800)])
def test_attention_slices(E, pkg, monkeypatch, name, context, kv):
    """Slices of 16 positions up to 16 x 74 (blocks per KV head), longer ones behind; page borders; a block's second pass over its slice
    (more than two tiles of keys)."""
    cfg = shape(pkg, name, 4)
    one, many = pair(E, pkg, monkeypatch, cfg, E.KV_F32 if kv == "f32" else E.KV_BF16, context + 16)
    ids = np.random.default_rng(context).integers(0, cfg.vocab_size, context)
    for e in (one, many):
        e.feed(ids[:-1] if context > 1 else ids, want_logits=False)
    tol = 6e-4 if kv == "f32" else 4e-3
    for tok in (5, 6, 7):
        a, b = (np.array(e.feed([tok])) for e in (one, many))
        assert np.isfinite(a).all() and np.abs(a - b).max() < tol
    one.close(); many.close()


@gpu
@pytest.mark.parametrize("kv", ["f32", "bf16"])
@pytest.mark.parametrize("name,context", [("full", 4142), ("full", 8434), ("full", 16900), ("half", 8300)])
def test_attention_passes(E, pkg, monkeypatch, name, context, kv):
    """A block's pass over its slice is two tiles of keys: at full width 56 positions of an fp32 cache, 114 of bf16. 4142 and 8434 cross
    74 times that within three tokens; 8434 (fp32) and 16900 have a third pass."""
    test_attention_slices(E, pkg, monkeypatch, name, context, kv)


@gpu
def test_narrow_model_keeps_its_launches(E, pkg):
    from b200moe import brain
    cfg = pkg.HybridConfig.tiny()
    e = E.HybridEngine.from_tensors(cfg.to_dict(), brain.random_brain(cfg, seed=1, device="cuda:0"), max_context=64, device=0, batch=1, kv_dtype=E.KV_F32)
    assert e.kernels_per_step() > cfg.n_layers
    e.close()


@gpu
def test_timeline(E, pkg):
    """One launch, and a row of the timeline for each of its stages: six of a DeltaNet layer, seven of attention, the head."""
    from b200moe import brain
    cfg = shape(pkg, "half", 4)
    e = E.HybridEngine.from_tensors(cfg.to_dict(), brain.random_brain(cfg, seed=1, device="cuda:0"), max_context=64, device=0, batch=1, kv_dtype=E.KV_F32)
    e.feed([1, 2, 3])
    t = e.trace_step().astype(np.int64)
    assert e.launches_per_step() == 1 and e.stages_per_step() == 3 * 6 + 7 + 1 and t.shape == (26, 16) and e.length() == 4
    delta, attn = [1, 3, 1, 1, 5, 6], [1, 7, 8, 1, 1, 5, 6]          # in-projections, mixer (and merge), out, router, gate/up, down
    assert t[:, 5].tolist() == 3 * delta + attn + [1]
    assert (t[:, 4] > t[:, 0]).all() and (np.diff(t[:, 4]) > 0).all()      # a stage ends after it began, and after the one before
    e.close()


@gpu
@pytest.mark.parametrize("polls", [1, 2, 40])
def test_waits_that_run_out(E, pkg, polls):
    """Fewer polls than a value takes to come: the step ends with an error, no wait lasts, and the engine works again after it."""
    from b200moe import brain
    cfg = shape(pkg, "half", 4)
    e = E.HybridEngine.from_tensors(cfg.to_dict(), brain.random_brain(cfg, seed=1, device="cuda:0"), max_context=1300, device=0, batch=1, kv_dtype=E.KV_F32)
    ids = np.arange(1200) % cfg.vocab_size
    e.feed(ids, want_logits=False)
    want = np.array(e.feed([7]))
    e.set_step1_polls(polls)
    errors = 0
    for _ in range(3):
        try:
            e.feed([8])
        except E.EngineError as x:
            assert "waited too long" in str(x)
            errors += 1
    assert errors == 3 or polls > 2
    e.set_step1_polls()
    assert e.crop(0) == 0
    e.feed(ids, want_logits=False)
    assert np.array_equal(np.array(e.feed([7])), want)
    e.close()


@gpu
def test_taps(E, pkg, monkeypatch):
    """A layer that is tapped twice has one place in the launch's table: steps go by launches then, and back when the taps change."""
    cfg = shape(pkg, "half", 3)
    one, many = pair(E, pkg, monkeypatch, cfg, E.KV_F32, 64)
    for layers in ([0, 2], [1, 1], [2]):
        one.set_taps(layers); many.set_taps(layers)
        assert (one.kernels_per_step() == 1) == (len(set(layers)) == len(layers))
        a, b = (np.array(e.feed([9])) for e in (one, many))
        assert np.array_equal(a, b) and np.array_equal(np.array(one.taps()), np.array(many.taps()))
    one.close(); many.close()


@gpu
@pytest.mark.parametrize("rows1,rows2", [(0, 0), (3, 0), (1, 1), (1, 3), (3, 2)])
def test_core_scores_that_are_no_numbers(E, pkg, monkeypatch, rows1, rows2):
    """Key rows of NaN, but for the first few of each table: a token's picks are different cores of the others, as many as there are, in a
    step of one sequence, of several and of a prompt."""
    from b200moe import brain
    cfg = shape(pkg, "half", 2)
    cfg.cores_active = 4
    dev = list(brain.random_brain(cfg, seed=1, device="cuda:0", vary_1d=True))
    for name, _, t in dev:
        if ".engine.key" in name:
            t[rows1 if "key1" in name else rows2:] = float("nan")
    make = lambda batch: E.HybridEngine.from_tensors(cfg.to_dict(), dev, max_context=64, device=0, batch=batch, kv_dtype=E.KV_F32)
    one, some, many = make(1), make(3), make(8)
    monkeypatch.setenv("B2_NO_STEP1", "1")
    stages = make(1)
    assert one.kernels_per_step() == 1 and stages.kernels_per_step() > 1
    allowed = np.zeros((cfg.core_grid[0], cfg.core_grid[1]), bool)
    allowed[:rows1, :rows2] = True

    def check(e, tokens):
        counts = e.core_counts(cfg.n_layers, cfg.n_cores)
        assert (counts.sum(1) == tokens * min(cfg.cores_active, rows1 * rows2)).all()
        assert counts.max() <= tokens and not counts[:, ~allowed.ravel()].any()
        e.reset_counts()

    for e in (one, stages):
        e.feed([5])
        e.feed([6])
        check(e, 2)
        e.feed(np.arange(40))
        check(e, 40)
    for e, batch in ((some, 3), (many, 8)):
        e.feed_batch(np.arange(batch))
        check(e, batch)
    for e in (one, some, many, stages):
        e.close()


@gpu
def test_another_engine_with_a_smaller_ring(E, pkg):
    """The shared memory of the launch depends on more than the widths it is built for; an engine keeps its own when another one is opened."""
    from b200moe import brain
    cfg, less = shape(pkg, "full", 2), shape(pkg, "full", 2)
    less.experts_active = 4
    dev = list(brain.random_brain(cfg, seed=1, device="cuda:0", vary_1d=True))
    a, b = (E.HybridEngine.from_tensors(c.to_dict(), dev, max_context=64, device=0, batch=1, kv_dtype=E.KV_F32) for c in (cfg, less))
    assert a.kernels_per_step() == b.kernels_per_step() == 1
    want = np.array(a.feed([7]))
    a.set_taps([0])                      # captured again
    a.crop(0)
    assert np.array_equal(np.array(a.feed([7])), want)
    b.feed([7])
    a.close(); b.close()


@gpu
def test_engines_of_several_threads(E, pkg):
    """Three engines on one device, each from its own thread: no launch may hold some SMs and wait for others."""
    from b200moe import brain
    cfg = shape(pkg, "half", 4)
    dev = list(brain.random_brain(cfg, seed=1, device="cuda:0", vary_1d=True))
    es = [E.HybridEngine.from_tensors(cfg.to_dict(), dev, max_context=512, device=0, batch=1, kv_dtype=E.KV_F32) for _ in range(3)]
    want = []
    for i, e in enumerate(es):
        want.append(np.array(e.decode_greedy([i + 1], 100)[0]))
        e.crop(0)
    got = [None] * 3

    def run(i):
        got[i] = np.array(es[i].decode_greedy([i + 1], 100)[0])

    ts = [threading.Thread(target=run, args=(i,)) for i in range(3)]
    for t in ts: t.start()
    for t in ts: t.join()
    for w, g in zip(want, got):
        assert np.array_equal(w, g)
    for e in es:
        e.close()


@gpu
def test_taps_change_beside_another_engine(E, pkg):
    """An engine captures its step anew whenever its taps change; another engine that follows its steps has nothing to do with that."""
    from b200moe import brain
    cfg = shape(pkg, "half", 4)
    dev = list(brain.random_brain(cfg, seed=1, device="cuda:0", vary_1d=True))
    a, b = (E.HybridEngine.from_tensors(cfg.to_dict(), dev, max_context=64, device=0, batch=1, kv_dtype=E.KV_F32) for _ in range(2))
    want = np.array(b.feed([3]))
    errors, done = [], threading.Event()

    def taps():
        try:
            while not done.is_set():
                a.crop(0)
                a.set_taps([0])
                a.feed([1])
                a.set_taps([1, 1])               # captured as many launches, which takes longer than one
        except E.EngineError as x:
            errors.append(x)

    t = threading.Thread(target=taps)
    t.start()
    try:
        for pause in np.random.default_rng(0).uniform(0, 3e-4, 1000):
            b.crop(0)
            assert np.array_equal(np.array(b.feed([3])), want)
            time.sleep(pause)
    finally:
        done.set()
        t.join()
    assert not errors
    a.close(); b.close()


@gpu
def test_a_step_beside_a_long_loop_has_its_turn(E, pkg):
    """One step of an engine, asked for while another one is in a greedy loop of 3000 (about 0.6 s): it comes after the few steps that the loop has
    queued, not after the loop."""
    from b200moe import brain
    cfg = shape(pkg, "half", 4)
    dev = list(brain.random_brain(cfg, seed=1, device="cuda:0", vary_1d=True))
    a, b = (E.HybridEngine.from_tensors(cfg.to_dict(), dev, max_context=3200, device=0, batch=1, kv_dtype=E.KV_F32) for _ in range(2))
    want = np.array(a.decode_greedy([1], 3000)[0])
    a.crop(0)
    got = []
    t = threading.Thread(target=lambda: got.append((np.array(a.decode_greedy([1], 3000)[0]), time.perf_counter())))
    t0 = time.perf_counter()
    t.start()
    time.sleep(0.05)
    b.feed([3])
    fed = time.perf_counter()
    t.join()
    assert np.array_equal(got[0][0], want)
    assert fed - t0 < 0.25 * (got[0][1] - t0)
    a.close(); b.close()
