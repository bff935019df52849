"""The window walk of the grouped kernels (queue_rows of csrc/cf_inside.cuh, and its callers) against the latency
kernels, which list a cell's candidates instead: structures, posteriors, logZ and samples, all bitwise.

Rows of unlike fullness: full, empty (one and several in turn, before and behind full ones), of masked positions, and
windows cut by either end of the sequence."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cases():
    rng = np.random.default_rng(17)
    out = []
    for L in (7, 31, 33, 62, 64, 96, 131):
        out.append(("A" * (L // 2) + "U" * (L - L // 2), None))              # rows full or empty by the half
        out.append((("AAC" * L)[: L // 2] + ("GGU" * L)[: L - L // 2], None))
        out.append((("GU" * L)[:L], None))            # every second cell pairs
        out.append(("".join(rng.choice(list("ACGU"), L)), (rng.random(L) < 0.6).astype(np.uint8)))
        one = np.ones(L, np.uint8)
        one[[0, L // 2, L - 1]] = 0                                          # three positions left to pair
        out.append(("".join(rng.choice(list("GU"), L)), one))
    return out


@pytest.mark.parametrize("group", [1, 5])
def test_window_walk_equals_listed_candidates(P, engine, group):
    from contrafold_gpu_gb300.engine import Batch, Engine
    engine.set_mode("batched")
    engine.set_schedule("auto")
    seqs, masks = zip(*_cases())
    B = Batch(list(seqs), [m if m is not None else np.zeros(len(s), np.uint8) for s, m in zip(seqs, masks)])
    eng = Engine(P)
    try:
        eng.set_shared(True)   # a shared device keeps the grouped kernels
        eng.set_group(group)
        assert eng.mea(B, 6.0) == engine.mea(B, 6.0)
        (ma, za), (mb, zb) = eng.bpp(B), engine.bpp(B)
        assert za.tobytes() == zb.tobytes()
        for a, b in zip(ma, mb):
            assert a.tobytes() == b.tobytes()
        assert eng.sample(B, 2, seed=3) == engine.sample(B, 2, seed=3)
    finally:
        eng.close()
