"""Sequences whose weights leave a float's range (stable helices, GC-rich RNAs) fold in the log domain, several of them
together on a CTA: each the result it has alone, within float32 log-sum-exp rounding of the FP64 oracle.

Batches of one such sequence and of hundreds (one and several a CTA), of lengths alike and mixed, and among ordinary
sequences; slices of an arena that holds few of them at a time.

Tolerance: d log-sum-exps in turn on a value's longest path, at most 3 L of them, each off by half a unit of the last
place of log Z and 2^-23 of its own terms: 2 L 2^-23 max(1, log Z) in all.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hairpin(rng, arm, loop="GAAA"):
    h = "".join(rng.choice(list("ACGU"), arm))
    return h + loop + h[::-1].translate(str.maketrans("ACGU", "UGCA"))


def _random(rng, L, gc=0.5):
    return "".join(rng.choice(list("ACGU"), L, p=[(1 - gc) / 2, gc / 2, gc / 2, (1 - gc) / 2]))


def _check(engine, oracle, P, seqs, few=6):
    from contrafold_gpu_gb300.engine import Batch
    z = engine.logz(Batch(seqs))
    at = np.unique(np.linspace(0, len(seqs) - 1, few).astype(int))
    want = np.array(oracle.batch(oracle.JOB_LOGZ64, [seqs[k] for k in at], P, None))
    L = np.array([len(seqs[k]) for k in at])
    assert np.all(np.abs(z[at] - want) <= 2 * L * 2.0 ** -23 * np.maximum(1.0, np.abs(want)))
    for k in at:
        assert engine.logz(Batch([seqs[k]]))[0] == z[k]
    return z


@pytest.mark.parametrize("n", [1, 3, 457, 1000])
def test_hairpins_alike(engine, oracle, P, n):
    engine.set_mode("batched")
    engine.set_schedule("auto")
    rng = np.random.default_rng(n)
    _check(engine, oracle, P, [_hairpin(rng, 60) for _ in range(n)])


def test_gc_rich_and_mixed(engine, oracle, P):
    engine.set_mode("batched")
    engine.set_schedule("auto")
    rng = np.random.default_rng(2)
    _check(engine, oracle, P, [_random(rng, 300, 0.8) for _ in range(40)])
    seqs = [_hairpin(rng, int(rng.integers(55, 110))) if k % 3 else _random(rng, int(rng.integers(20, 300))) for k in range(2200)]
    _check(engine, oracle, P, seqs, 9)


def test_slices_of_a_small_arena(P, oracle, engine):
    """Each slice has its own list of what left the range; gradients likewise, with length classes on side streams."""
    from contrafold_gpu_gb300 import grad
    from contrafold_gpu_gb300.engine import Batch, Engine
    rng = np.random.default_rng(3)
    seqs = [_hairpin(rng, int(rng.integers(60, 100))) if k % 4 == 1 else _random(rng, int(rng.integers(20, 390)))
            for k in range(40)]
    engine.set_mode("batched")
    engine.set_schedule("auto")
    B = Batch(seqs)
    want, want64, counts = engine.logz(B), engine.logz64(B), grad.logz_grad(seqs, engine=engine)
    eng = Engine(P)
    try:
        eng.set_budget(4 << 20)      # 400 nt: 1 MB (logZ), 2.1 MB (FP64), 1.8 MB (gradients)
        assert np.array_equal(eng.logz(B), want)
        assert np.array_equal(eng.logz64(B), want64)
        got = grad.logz_grad(seqs, engine=eng)
        assert np.array_equal(got.logz, counts.logz) and np.array_equal(got.d_blob, counts.d_blob)
        assert all(np.array_equal(a, b) for a, b in zip(got.d_bonus, counts.d_bonus))
    finally:
        eng.close()


def test_length_classes(engine, oracle, P):
    """Lengths on either side of the launch classes' ends: the result each has alone, in a launch of its own, on a shared
    device, in float and in double (tolerance of test_gpu_linear.py)."""
    from contrafold_gpu_gb300.engine import Batch, Engine
    engine.set_mode("batched")
    engine.set_schedule("auto")
    rng = np.random.default_rng(4)
    seqs = [_random(rng, L) for L in (1, 95, 96, 97, 159, 160, 161, 235, 236, 300, 395, 396, 415, 512)]
    z, z64 = engine.logz(Batch(seqs)), engine.logz64(Batch(seqs[:-1]))
    want = np.array(oracle.batch(oracle.JOB_LOGZ64, seqs, P, None))
    L = np.array([len(s) for s in seqs])
    assert np.all(np.abs(z - want) <= 16 * L * 2.0 ** -24 + 2.0 ** -23 * np.abs(want))
    for k, s in enumerate(seqs):
        assert engine.logz(Batch([s]))[0] == z[k]
        if k < len(z64):
            assert engine.logz64(Batch([s]))[0] == z64[k]
    eng = Engine(P)
    try:
        eng.set_shared(True)
        assert np.array_equal(eng.logz(Batch(seqs)), z)
        assert np.array_equal(eng.logz64(Batch(seqs[:-1])), z64)
    finally:
        eng.close()
