"""Shared memory is asked for by the kernels that run and by no other: a group of sequences needs more of it than
kernels with static shared memory of their own (the Viterbi ones) could be given."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_widest_groups_of_long_sequences(engine, P):
    """32 sequences a CTA whose longest has 2,300 nt: 201,440 bytes."""
    from contrafold_gpu_gb300.engine import Batch, Engine
    rng = np.random.default_rng(5)
    B = Batch(["".join(rng.choice(list("ACGU"), L)) for L in (2300, 30)])
    engine.set_mode("batched")
    engine.set_schedule("auto")
    want = engine.logz(B)
    eng = Engine(P)
    try:
        eng.set_schedule("group")
        eng.set_group(32)
        assert np.array_equal(eng.logz(B), want)
        short = Batch([s for s in ("GGGGAAAACCCC", "GCGCAAAAGCGC")])
        assert eng.mfe(short) == engine.mfe(short)
    finally:
        eng.close()
