"""The Viterbi kernels (csrc/cf_viterbi.cu) against the CPU oracle's FP64 recurrence: structures, ties included.

Lengths around what the kernels divide by (32 candidates a turn, 31-row windows, 128-cell parts), masked, with unknown
bases, and batches on one CTA and on clusters of 4 and 8 CTAs a sequence."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 3, 4, 5, 6, 9, 31, 32, 33, 34, 35, 63, 64, 65, 66, 127, 128, 129, 130, 200, 257, 258]


@pytest.mark.parametrize("n", [1, 24, 60, 100])
def test_viterbi_equals_oracle(engine, oracle, P, n):
    from contrafold_gpu_gb300.engine import Batch
    engine.set_mode("batched")
    engine.set_schedule("auto")
    rng = np.random.default_rng(300 + n)
    lens = (LENGTHS * 5)[:n] if n > 1 else [258]
    seqs = ["".join(rng.choice(list("ACGUN"), p=[.24, .24, .24, .24, .04], size=L)) for L in lens]
    masks = [(rng.random(L) < (1.0 if k % 11 == 7 else 0.1)).astype(np.uint8) for k, L in enumerate(lens)]
    assert engine.mfe(Batch(seqs, masks)) == oracle.batch(oracle.JOB_MFE, seqs, P, masks)


def test_viterbi_ties(engine, oracle, P):
    """Repeats, whose equal scores leave the choice to the order of the candidates."""
    from contrafold_gpu_gb300.engine import Batch
    seqs = ["GU" * 60, "GC" * 50, "GGGAAACCC" * 14, "A" * 40 + "U" * 40, "G" * 70 + "C" * 70]
    assert engine.mfe(Batch(seqs, None)) == oracle.batch(oracle.JOB_MFE, seqs, P, None)


@pytest.mark.parametrize("lo,hi", [(0, 8), (22, 22), (15, 40), (55, 60)])
def test_viterbi_groups_equal_oracle(engine, oracle, P, lo, hi):
    """Thousands of very short sequences fold several a CTA: whole groups, a last one that is not full, lengths alike and
    mixed, with empty sequences."""
    from contrafold_gpu_gb300.engine import Batch, Engine
    rng = np.random.default_rng(40 + hi)
    lens = rng.integers(lo, hi + 1, 3421)
    seqs = ["".join(rng.choice(list("ACGUN"), p=[.24, .24, .24, .24, .04], size=L)) for L in lens]
    masks = [(rng.random(L) < 0.1).astype(np.uint8) for L in lens]
    want = oracle.batch(oracle.JOB_MFE, seqs, P, masks)
    engine.set_mode("batched")
    engine.set_schedule("auto")
    B = Batch(seqs, masks)
    assert engine.mfe(B) == want
    eng = Engine(P)
    try:
        for group in (1, 3, 8):
            eng.set_group(group)
            assert eng.mfe(B) == want
    finally:
        eng.close()
