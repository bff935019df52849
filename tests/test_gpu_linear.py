"""logZ and FP64 logZ as sums of products (csrc/cf_linear.cu) against the FP64 oracle.

Sizes: the smallest sequences, the edges of the stencil's 128-cell and the
splits' 32-cell chunks, of the 32-diagonal ring and of the 256 exterior
threads, the longest that take the path, and one more (log-domain kernels).

Tolerance: a structure's weight is a product of at most 6 factors per position,
and each position's sums add at most 10 more roundings to it, so a scaled Z is
off by at most 16 L units of rounding (2^-24, or 2^-53) and log Z by as much,
plus the rounding of the result itself.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 5, 6, 7, 30, 31, 32, 33, 34, 35, 36, 63, 64, 65, 127, 128, 129, 130, 131, 255, 256, 257, 258,
           259, 385, 415, 416, 417]


def _batch(seed, lens, p_mask):
    rng = np.random.default_rng(seed)
    seqs = ["".join(rng.choice(list("ACGUN"), p=[.24, .24, .24, .24, .04], size=int(L))) for L in lens]
    return seqs, [(rng.random(int(L)) < p_mask).astype(np.uint8) for L in lens]


@pytest.mark.parametrize("p_mask", [0.0, 0.1])
def test_logz_against_fp64(engine, P, oracle, p_mask):
    from contrafold_gpu_gb300.engine import Batch
    lens = LENGTHS + [511, 512]
    seqs, masks = _batch(71, lens, p_mask)
    B = Batch(seqs, masks if p_mask else None)
    want = np.asarray(oracle.batch(oracle.JOB_LOGZ64, seqs, P, masks if p_mask else None))
    L = np.array(lens, np.float64)
    z = engine.logz(B).astype(np.float64)
    assert np.all(np.abs(z - want) <= 16 * L * 2.0 ** -24 + 2.0 ** -23 * np.abs(want)), np.abs(z - want) / L
    z64 = engine.logz64(B)
    short = L <= 416     # longer ones are log-sum-exp chains: as many roundings, of log Z's own size
    tol = 16 * L * 2.0 ** -53 * np.where(short, 1.0, np.maximum(1.0, np.abs(want))) + 2.0 ** -52 * np.abs(want)
    # the oracle's chains round at log Z's size too
    tol = tol + L * 2.0 ** -53 * np.maximum(1.0, np.abs(want))
    assert np.all(np.abs(z64 - want) <= tol), np.abs(z64 - want) / L


def test_logz_outside_the_floats_range(engine, P, oracle):
    """Weights that leave the range of scaled floats fold in the log domain: a finite result, the same as
    alone and in either mode, and in FP64 the oracle's."""
    from contrafold_gpu_gb300.engine import Batch
    hard = ["G" * 150 + "AAAA" + "C" * 150, "A" * 300 + "GGGGAAAACCCC" + "U" * 200, "GC" * 200]
    seqs, _ = _batch(72, [40, 200, 90], 0.0)
    mixed = [seqs[0], hard[0], seqs[1], hard[1], hard[2], seqs[2]]
    z = engine.logz(Batch(mixed))
    for s, v in zip(mixed, z):
        assert np.isfinite(v) and engine.logz(Batch([s]))[0] == v
    engine.set_mode("plain")
    assert np.array_equal(engine.logz(Batch(mixed)), z)
    engine.set_mode("batched")
    z64 = engine.logz64(Batch(mixed))
    for s, v in zip(mixed, z64):
        want = oracle.logz64(s, P)
        assert abs(v - want) <= 32 * len(s) * 2.0 ** -53 * max(1.0, abs(want))


def test_logz_follows_the_parameters(engine, P, oracle):
    """Weights are made again when the parameters change, for calls and for plans made before."""
    torch = pytest.importorskip("torch")
    from contrafold_gpu_gb300.engine import CF_JOB_LOGZ, Batch, Engine, Plan
    seqs, _ = _batch(73, [60, 100], 0.0)
    B = Batch(seqs)
    from contrafold_gpu_gb300 import params
    Q = {k: P[k] for k in params.TABLES + params.SCALARS}   # not what the engine and the oracle keep beside them
    Q["ep"] = Q["ep"] + 0.5
    eng = Engine(P)
    try:
        d = torch.from_numpy(B.buf.copy()).cuda()
        out = torch.zeros(2, dtype=torch.float32, device="cuda")
        plan = Plan(eng, CF_JOB_LOGZ, B.offsets)
        plan.set_graph(True)
        for par in (P, Q):
            eng.set_params(par)
            plan.run(d.data_ptr(), 0, out.data_ptr())
            plan.status()
            want = np.array([oracle.logz64(s, par) for s in seqs])
            assert np.max(np.abs(out.cpu().numpy() - want)) < 1e-4
            assert np.array_equal(eng.logz(B), out.cpu().numpy())
        plan.close()
    finally:
        eng.close()


def test_shared_device_same_sums(engine, P):
    """A shared device's launches have fewer threads from 236 nt up; sums and their order are the same."""
    from contrafold_gpu_gb300.engine import Batch, Engine
    rng = np.random.default_rng(23)
    B = Batch(["".join(rng.choice(list("ACGU"), L)) for L in (60, 235, 236, 257, 395, 396, 511, 512)], None)
    engine.set_mode("batched")
    eng = Engine(P)
    try:
        eng.set_shared(True)
        assert np.asarray(eng.logz(B)).tobytes() == np.asarray(engine.logz(B)).tobytes()
    finally:
        eng.close()
