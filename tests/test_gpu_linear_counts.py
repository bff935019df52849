"""Expected counts of short sequences, rare events among them, against FP64 central differences of the oracle: each to
its own size.  (test_gpu_linear_grad.py bounds them to the largest.)

Tolerance: a probability is a product of an inside and an outside weight, each at most 16 L roundings off
(tests/test_gpu_linear.py), and a count a sum of such terms of one sign, so it is off by at most 48 L 2^-24 of itself.
The difference (h = 1e-3, Richardson's step with 2 h: error 4 h^4 of a smooth log Z's fifth derivative, at most 24 of
those of an event's own count for each of L / 4 events at most) and the oracle's rounding, 32 L 2^-53 max(1, log Z) / h.
"""
import numpy as np
import pytest

from contrafold_gpu_gb300 import grad, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [18, 20, 24, 30, 45, 60, 90])
def test_counts_to_their_own_size(engine, P, oracle, L):
    rng = np.random.default_rng(1200 + L)
    seq = "".join(rng.choice(list("ACGU"), size=L))
    seq = "G" + seq[1:-1] + "C"          # a pair may close the multiloops
    res = grad.logz_grad([seq])
    blob = params.pack64(P)
    zero = np.zeros(L)
    logz = lambda b: oracle.logz64_bonus(seq, P, zero, None, blob64=b)   # noqa: E731
    off = params.OFFSETS
    pick = [off[s] for s in params.SCALARS]
    names = list(params.TABLES)
    for n, e in zip(names, [off[x] for x in names[1:]] + [off["mb"]]):
        o = off[n]
        order = o + np.argsort(-np.abs(res.d_blob[0, o:e]))
        seen = order[res.d_blob[0, order] != 0.0]
        pick += [int(k) for k in {*seen[:2], *seen[len(seen) // 2:len(seen) // 2 + 1], *seen[-2:]}]
    h = 1e-3
    for k in pick:
        def central(step):
            up, down = blob.copy(), blob.copy()
            up[k] += step
            down[k] -= step
            return (logz(up) - logz(down)) / (2 * step)
        want = (4 * central(h) - central(2 * h)) / 3
        size = max(abs(want), 1e-300)
        tol = size * (48 * L * 2.0 ** -24 + 24 * L * h ** 4) + 32 * L * 2.0 ** -53 * max(1.0, abs(logz(blob))) / h
        assert abs(res.d_blob[0, k] - want) <= tol, (k, res.d_blob[0, k], want, tol)
        assert res.d_blob[0, k] >= 0.0
