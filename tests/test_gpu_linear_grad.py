"""Gradients as sums of products (csrc/cf_linear.cu): every table entry's count and every position's
probability against FP64 central differences of the oracle, at the sizes where the kernels' chunks, rings and
row placement change, and against the log-domain kernels at the longest length they take.

Tolerance: a probability is a product of an inside and an outside weight, each at most 16 L roundings off
(tests/test_gpu_linear.py), so a count is off by at most 48 L 2^-24 of itself, at most L events an entry; the
central difference (h = 1e-4) of a smooth log Z with L events has an error of at most L h^2 + 2 L 2^-52 / h.
"""
import numpy as np
import pytest

from contrafold_gpu_gb300 import grad, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,masked", [(1, False), (5, False), (33, True), (66, False), (129, True), (300, False),
                                      (301, True), (400, False)])
def test_counts_against_fp64_differences(engine, P, oracle, L, masked):
    rng = np.random.default_rng(900 + L)
    seq = "".join(rng.choice(list("ACGUN"), p=[.24, .24, .24, .24, .04], size=L))
    mask = (rng.random(L) < 0.1).astype(np.int8) if masked else None
    bonus = rng.normal(0, 0.5, L).astype(np.float32)
    res = grad.logz_grad([seq], None, [bonus], None if mask is None else [mask])
    blob = params.pack64(P)
    u = bonus.astype(np.float64)
    h = 1e-4
    tol = L * (48 * L * 2.0 ** -24 + h * h + 2.0 ** -51 / h)
    logz = oracle.logz64_bonus(seq, P, u, mask)
    assert abs(res.logz[0] - logz) <= 24 * L * 2.0 ** -24 + 2.0 ** -23 * abs(logz)
    # every scalar, and the largest and a few random entries of every table
    off = params.OFFSETS
    names = list(params.TABLES)
    ends = [off[n] for n in names[1:]] + [off["mb"]]
    pick = [off[s] for s in params.SCALARS]
    for n, e in zip(names, ends):
        o = off[n]
        pick += [o + int(np.argmax(np.abs(res.d_blob[0, o:e])))] + [o + int(k) for k in rng.integers(0, e - o, 2)]
    for k in pick:
        bp, bm = blob.copy(), blob.copy()
        bp[k] += h
        bm[k] -= h
        fd = (oracle.logz64_bonus(seq, P, u, mask, blob64=bp) - oracle.logz64_bonus(seq, P, u, mask, blob64=bm)) / (2 * h)
        assert abs(res.d_blob[0, k] - fd) <= tol, (k, res.d_blob[0, k], fd)
    for k in {0, L // 2, L - 1}:
        up, um = u.copy(), u.copy()
        up[k] += h
        um[k] -= h
        fd = (oracle.logz64_bonus(seq, P, up, mask) - oracle.logz64_bonus(seq, P, um, mask)) / (2 * h)
        assert abs(res.d_bonus[0][k] - fd) <= tol, (k, res.d_bonus[0][k], fd)


def test_gradients_outside_the_floats_range(engine, P):
    """Sequences whose weights leave the float's range take the log-domain kernels: the result each has alone, and
    probabilities that add up (each position is paired or not), within float32 log-sum-exp rounding."""
    hard = "G" * 150 + "AAAA" + "C" * 150
    rng = np.random.default_rng(7)
    easy = ["".join(rng.choice(list("ACGU"), size=L)) for L in (50, 200)]
    seqs = [easy[0], hard, easy[1]]
    res = grad.logz_grad(seqs)
    o = params.OFFSETS["bp"]
    for b, s in enumerate(seqs):
        alone = grad.logz_grad([s])
        assert alone.d_blob[0].tobytes() == res.d_blob[b].tobytes()
        assert alone.d_bonus[0].tobytes() == res.d_bonus[b].tobytes() and alone.logz[0] == res.logz[b]
        assert abs(res.d_bonus[b].sum() - (len(s) - 2 * res.d_blob[b, o:o + 25].sum())) < 1e-3 * len(s)


def test_gradients_do_not_depend_on_checkpoints_or_batch(engine, P):
    from contrafold_gpu_gb300.engine import Engine
    rng = np.random.default_rng(8)
    seqs = ["".join(rng.choice(list("ACGU"), size=L)) for L in (400, 401, 120, 31)]
    eng = Engine(P)
    try:
        got = []
        for every in (1, 8):
            eng.set_grad_checkpoint(every)
            r = grad.logz_grad(seqs, engine=eng)
            got.append([(r.logz[b], r.d_blob[b].tobytes(), r.d_bonus[b].tobytes()) for b in range(4)])
        assert got[0] == got[1]
        for b, s in enumerate(seqs):
            r = grad.logz_grad([s], engine=eng)
            assert (r.logz[0], r.d_blob[0].tobytes(), r.d_bonus[0].tobytes()) == got[0][b]
    finally:
        eng.close()
