"""Engines of one process, each used by a thread of its own (include/b200moe.h): while one of them captures its step anew again and again as
its taps change, and beside a persistent step, which needs every SM."""
import contextlib
import importlib
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def E(pkg):
    return importlib.import_module("b200moe.engine")


@contextlib.contextmanager
def captures(e):
    errors, done = [], threading.Event()

    def taps():
        try:
            while not done.is_set():
                e.set_taps([0])
                e.set_taps([1, 2])
        except Exception as x:
            errors.append(x)

    t = threading.Thread(target=taps)
    t.start()
    try:
        yield
    finally:
        done.set()
        t.join()
    assert not errors, errors


def test_prompts_beside_captures(E, tiny_path):
    """The kernels' limit of shared memory is one for all threads: no launch lowers it for another one's."""
    a, b = (E.HybridEngine.load(tiny_path, max_context=1024) for _ in range(2))
    lengths = (40, 333, 40, 700, 17) * 20
    want = {n: np.array(a.feed(np.arange(n))) for n in set(lengths) if a.crop(0) == 0}
    with captures(b):
        for n in lengths:
            a.crop(0)
            assert np.array_equal(np.array(a.feed(np.arange(n))), want[n])
    a.close(); b.close()


def test_opening_beside_captures(E, tiny_path):
    """Opening and closing an engine, and its first prompt, wait for what they have begun, not for the device with other threads' streams."""
    b = E.HybridEngine.load(tiny_path, max_context=64)
    want = None
    with captures(b):
        for _ in range(20):
            a = E.HybridEngine.load(tiny_path, max_context=256)
            got = np.array(a.feed(np.arange(100)))
            want = got if want is None else want
            assert np.array_equal(got, want)
            a.close()
    b.close()


def test_timeline_beside_captures(E, tiny_path):
    """The slots of a timeline go to the launches of the thread that asked for it."""
    a, b = (E.HybridEngine.load(tiny_path, max_context=256) for _ in range(2))
    with captures(b):
        rows = {a.trace_step().shape[0] for _ in range(200)}
    assert rows == {a.stages_per_step()} and a.launches_per_step() == a.stages_per_step()
    b.close(); a.close()


def test_persistent_steps_beside_prompts_and_batches(E, pkg):
    """A step that needs all SMs at once, prompts and steps of eight sequences: whatever holds SMs is waited for, and all results are as alone."""
    from b200moe import brain
    from test_step1_gpu import shape
    cfg = shape(pkg, "half", 4)
    dev = list(brain.random_brain(cfg, seed=1, device="cuda:0", vary_1d=True))
    a, b, c = (E.HybridEngine.from_tensors(cfg.to_dict(), dev, max_context=1024, device=0, batch=n, kv_dtype=E.KV_F32) for n in (1, 1, 8))
    assert a.launches_per_step() == 1 < c.launches_per_step()

    def steps():
        a.crop(0)
        return np.array(a.decode_greedy([1], 400)[0])

    def prompts():
        out = []
        for n in (40, 333, 700, 64):
            b.crop(0)
            out.append(np.array(b.feed(np.arange(n))))
        return np.stack(out)

    def batches():
        c.crop(0)
        return np.array(c.decode_greedy(np.arange(8), 60)[0])

    work = (steps, prompts, batches)
    want, got = [f() for f in work], [None] * 3

    def run(i):
        got[i] = [work[i]() for _ in range(3)]

    ts = [threading.Thread(target=run, args=(i,)) for i in range(3)]
    for t in ts: t.start()
    for t in ts: t.join()
    for w, g in zip(want, got):
        assert g is not None and all(np.array_equal(w, x) for x in g)
    a.close(); b.close(); c.close()
