"""The engine's host code over a CUDA runtime without a device (native/fake_cudart.cpp): what it refuses before a
launch, what it copies and when, and the streams it makes.  Each check is a program of its own, with the fake runtime
loaded before the library."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)

PRELUDE = """
import ctypes, os, sys
import numpy as np
fake = ctypes.CDLL(os.environ["LD_PRELOAD"])
fake.fake_stream.restype = ctypes.c_void_p
from contrafold_gpu_gb300 import params
from contrafold_gpu_gb300.engine import *
from contrafold_gpu_gb300.engine import Plan, Batch, Engine
P = params.load()
rng = np.random.default_rng(1)
def seqs(*lens):
    return ["".join(rng.choice(list("ACGU"), L)) for L in lens]
eng = Engine(P)
"""


@pytest.fixture(scope="session")
def run(tmp_path_factory):
    from contrafold_gpu_gb300 import build
    gxx = shutil.which("g++")
    try:
        cuda = os.path.dirname(os.path.dirname(build.nvcc()))
        build.build()
    except RuntimeError:
        cuda = None
    if not gxx or not cuda:
        pytest.skip("compilers not available")
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.check_call([gxx, "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(cuda, "include"), "-o", so,
                           os.path.join(HERE, "native", "fake_cudart.cpp")])

    def go(body):
        env = dict(os.environ, LD_PRELOAD=so, PYTHONPATH=REPO)
        env.pop("CONTRAFOLD_GB300_LIB", None)
        r = subprocess.run([sys.executable, "-c", PRELUDE + body], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout
    return go


def test_plan_run_refuses_null_buffers(run):
    """Plans whose sequences take the sums of products alone, the other kernels alone, or both."""
    run("""
for lens in ((20, 40), (600,), (600, 40)):
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    for job in (CF_JOB_LOGZ, CF_JOB_LOGZ64, CF_JOB_BPP, CF_JOB_MEA, CF_JOB_MFE):
        plan = Plan(eng, job, offs)
        for graph, d_seqs, d_out in ((False, 0, 4096), (False, 4096, 0), (True, 0, 4096), (True, 4096, 0)):
            plan.set_graph(graph)
            try:
                plan.run(d_seqs, 0, d_out)
            except EngineError as e:
                assert e.code == CF_EINVAL
            else:
                raise SystemExit(f"accepted: {lens}, job {job}")
assert fake.fake_launches() == 0
""")


def test_copied_parameters_live_until_the_copy(run):
    """A host-to-device copy may read its source as late as the stream's next synchronisation."""
    run("""
B = Batch(seqs(30, 40))
eng.logz(B)
eng.logz64(B)        # both sets of weights exist from here on: set_params copies them again
for k in range(3):
    Q = {k: P[k] for k in params.TABLES + params.SCALARS}
    Q["ep"] = Q["ep"] + 0.5 * k
    eng.set_params(Q)
assert fake.fake_changed_sources() == 0, fake.fake_changed_sources()
""")


def test_plan_of_sums_needs_no_room_for_other_kernels(run):
    """A budget that holds what the plan launches is enough, whatever the schedule it reports would need; one that
    does not hold the longest sequence is refused, as by the call itself."""
    run("""
B = Batch(seqs(*[120] * 64))
eng.set_schedule("group")
eng.set_group(32)
eng.set_budget(1 << 20)                  # one sequence's tables are 100 KB
eng.logz(B)
plan = Plan(eng, CF_JOB_LOGZ, B.offsets)
assert plan.schedule == "group", plan.schedule
plan.run(4096, 0, 8192)
eng.set_budget(1 << 14)
for call in (lambda: eng.logz(B), lambda: Plan(eng, CF_JOB_LOGZ, B.offsets)):
    try:
        call()
    except EngineError as e:
        assert e.code == CF_ENOMEM
    else:
        raise SystemExit("accepted")
""")


def test_gradient_result_is_a_plain_record(run):
    """Positional construction, asdict and replace; d_theta is the counts through the tying."""
    run("""
import dataclasses
from contrafold_gpu_gb300 import grad
assert [f.name for f in dataclasses.fields(grad.GradResult)] == ["logz", "d_blob", "d_theta", "d_bonus"]
r = grad.logz_grad(seqs(20, 30), engine=eng)
assert set(dataclasses.asdict(r)) == {"logz", "d_blob", "d_theta", "d_bonus"}
assert np.array_equal(r.d_theta, r.d_blob @ grad.tying_jacobian()) and r.d_theta.shape[0] == 2
assert dataclasses.replace(r, logz=None).d_theta is r.d_theta
assert grad.GradResult(1, 2, 3, 4).d_bonus == 4
""")


def test_side_streams_have_the_callers_priority(run):
    """Length classes beside the first one run at the priority of the stream that the call or the run is on."""
    run("""
offs = Batch(seqs(20, 120, 220, 380, 500)).offsets
B = Batch(seqs(20, 120, 220, 380, 500))
LEAST, GREATEST = 0, -5
def made():
    return fake.fake_streams_of(LEAST), fake.fake_streams_of(GREATEST)
least, greatest = made()
eng.logz(B)
assert made()[0] > least and made()[1] == greatest == 0
eng.set_priority(True)                   # the engine's own high-priority stream, then its side streams
least = made()[0]
own = made()[1]
eng.logz(B)
assert made()[0] == least and made()[1] > own
greatest = made()[1]
eng.logz(B)
assert made() == (least, greatest)       # kept between calls
plan = Plan(eng, CF_JOB_LOGZ, offs)
for graph in (False, True):
    plan.set_graph(graph)
    stream = fake.fake_stream(-3)
    plan.run(4096, 0, 8192, 6.0, stream)
    assert fake.fake_streams_of(-3) > 1
""")


def test_groups_of_short_mixed_batches(run):
    """Short sequences of mixed lengths fold several a CTA as soon as every CTA has a group (152 SMs here), long ones
    only where two waves of CTAs remain; no batch takes the warp-per-sequence kernel on its own."""
    run("""
def plan(n, lo, hi, job=CF_JOB_MEA):
    p = Plan(eng, job, Batch(seqs(*rng.integers(lo, hi + 1, n), lo, hi)).offsets)
    return p.schedule, p.group
eng.set_budget(1 << 30)
assert plan(2046, 15, 25) == ("group", 3)        # 608 CTAs
assert plan(10000, 20, 40) == ("group", 8)
assert plan(3000, 100, 256) == ("group", 2)
assert plan(2046, 40, 400) == ("group", 1)
assert plan(300, 15, 25) == ("group", 1)         # the latency kernels
assert plan(2046, 60, 70) == ("group", 4)        # lengths alike: one wave
""")
