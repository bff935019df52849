"""Expected counts, rare events among them, and unpaired probabilities against FP64 central differences of the oracle:
each to its own size.  (test_gpu_linear_grad.py bounds them to the largest.)

Tolerance: a probability is a product of an inside and an outside weight, each at most 16 L roundings off
(tests/test_gpu_linear.py), and a count a sum of such terms of one sign, so it is off by at most 48 L 2^-24 of itself.
The difference (h = 1e-3, Richardson's step with 2 h: error 4 h^4 of a smooth log Z's fifth derivative, at most 24 of
those of an event's own count for each of L / 4 events at most) and the oracle's rounding, 32 L 2^-53 max(1, log Z) / h.
An unpaired probability is 1 - P, off by as much as P.
"""
import concurrent.futures as cfut

import numpy as np
import pytest

from contrafold_gpu_gb300 import grad, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [18, 20, 24, 30, 45, 60, 90, 150, 300, 301, 400])
def test_counts_to_their_own_size(engine, P, oracle, L):
    rng = np.random.default_rng(1200 + L)
    seq = "".join(rng.choice(list("ACGU"), size=L))
    seq = "G" + seq[1:-1] + "C"          # a pair may close the multiloops
    res = grad.logz_grad([seq])
    blob = params.pack64(P)
    zero = np.zeros(L)
    logz = lambda b, u=zero: oracle.logz64_bonus(seq, P, u, None, blob64=b)   # noqa: E731
    off = params.OFFSETS
    pick = [off[s] for s in params.SCALARS]
    names = list(params.TABLES)
    for n, e in zip(names, [off[x] for x in names[1:]] + [off["mb"]]):
        o = off[n]
        order = o + np.argsort(-np.abs(res.d_blob[0, o:e]))
        seen = order[res.d_blob[0, order] != 0.0]
        few = 1 if L > 200 else 2      # a long sequence's oracle takes a while
        pick += [int(k) for k in {*seen[:few], *seen[len(seen) // 2:len(seen) // 2 + 1], *seen[-few:]}]
    h = 1e-3
    rounding = 32 * L * 2.0 ** -53 * max(1.0, abs(logz(blob))) / h

    def derivative(at):
        central = lambda step: (at(step) - at(-step)) / (2 * step)   # noqa: E731
        return (4 * central(h) - central(2 * h)) / 3

    def step_blob(k, x):
        b = blob.copy()
        b[k] += x
        return b

    def step_bonus(k, x):
        u = zero.copy()
        u[k] += x
        return u

    ends = [0, 1, L // 2, L - 1]
    with cfut.ThreadPoolExecutor() as ex:   # the oracle runs outside the interpreter
        counts = list(ex.map(lambda k: derivative(lambda x: logz(step_blob(k, x))), pick))
        unpaired = list(ex.map(lambda k: derivative(lambda x: logz(blob, step_bonus(k, x))), ends))
    for k, want in zip(pick, counts):
        tol = abs(want) * (48 * L * 2.0 ** -24 + 24 * L * h ** 4) + rounding
        assert abs(res.d_blob[0, k] - want) <= tol, (k, res.d_blob[0, k], want, tol)
        assert res.d_blob[0, k] >= 0.0
    for k, want in zip(ends, unpaired):
        # 1 - P, from sums of at most L terms of P
        tol = abs(1.0 - want) * 48 * L * 2.0 ** -24 + 24 * L * h ** 4 + rounding
        assert abs(res.d_bonus[0][k] - want) <= tol, (k, res.d_bonus[0][k], want, tol)
