"""The kernels of batches that leave most of the device idle (csrc/cf_latency.cu) against the grouped kernels,
which an engine in shared-device mode keeps: MEA structures, posteriors, their logZ and samples, all bitwise.

Lengths around what the kernels divide by (32-cell chunks, 31-row windows, eight-term blocks, eight decode parts,
256 exterior terms), masked, with unknown bases, and batches on 1, 2, 4 and 8 CTAs a sequence."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 3, 4, 5, 9, 10, 17, 31, 32, 33, 34, 40, 63, 64, 65, 66, 127, 128, 129, 130, 200, 257, 258, 259, 300]


def _batch(seed, lens):
    rng = np.random.default_rng(seed)
    seqs = ["".join(rng.choice(list("ACGUN"), p=[.24, .24, .24, .24, .04], size=int(L))) for L in lens]
    return seqs, [(rng.random(int(L)) < 0.1).astype(np.uint8) for L in lens]


@pytest.fixture(scope="module")
def grouped(P):
    from contrafold_gpu_gb300.engine import Engine
    eng = Engine(P)
    eng.set_shared(True)
    yield eng
    eng.close()


def _same(engine, grouped, seqs, masks):
    from contrafold_gpu_gb300.engine import Batch
    B = Batch(seqs, masks)
    assert engine.mea(B, 6.0) == grouped.mea(B, 6.0)
    assert engine.mea(B, 0.5) == grouped.mea(B, 0.5)
    ma, za = engine.bpp(B)
    mb, zb = grouped.bpp(B)
    assert za.tobytes() == zb.tobytes()
    for a, b in zip(ma, mb):
        assert a.tobytes() == b.tobytes()
    assert engine.sample(B, 3, seed=5) == grouped.sample(B, 3, seed=5)


@pytest.mark.parametrize("n", [1, 27, 60, 76, 130])
def test_latency_kernels_equal_grouped(engine, grouped, n):
    engine.set_mode("batched")
    engine.set_schedule("auto")
    lens = (LENGTHS * 5)[:n] if n > 1 else [300]
    seqs, masks = _batch(100 + n, lens)
    _same(engine, grouped, seqs, masks)


def test_latency_kernels_dense_pairs(engine, grouped):
    """Alternating G and U: nearly every cell pairs, so windows hold hundreds of candidates."""
    _same(engine, grouped, ["GU" * 70, "GC" * 40 + "A" * 30 + "GC" * 40], None)


def test_latency_kernels_without_room_for_terms(P, grouped):
    """A budget that holds the tables but not the latency kernels' terms folds grouped: same results."""
    from contrafold_gpu_gb300.engine import Engine
    seqs, masks = _batch(7, [300, 120])
    eng = Engine(P)
    try:
        eng.set_budget(2 << 20)
        _same(eng, grouped, seqs, masks)
    finally:
        eng.close()
