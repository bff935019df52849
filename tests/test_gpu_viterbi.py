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
