"""Calls of the public API whose time is tracked, with their exact results.

A case names an entry point (`api`) and the size of one call:

  n            sequences in the call
  lo, hi       lengths, uniform over [lo, hi] (lo == hi: all alike); the same lengths for every seed
  mask         share of positions forced unpaired (0: no masks are passed)
  samples      structures drawn for each sequence (`sample`)

Bases are i.i.d. uniform over ACGU, as in the benchmark's workloads.  The model
is the bundled one, loaded once per process with its engine, as a program that
folds keeps it.
"""
import math
import os

import numpy as np
import torch

import contrafold_gpu_gb300 as cf
from contrafold_gpu_gb300 import grad, gpu

ALPHA = np.frombuffer(b"ACGU", np.uint8)
THETA_STEP = 1e-3    # gradient descent on the mean of the weighted logZ; a sequence's soft constraints are
BONUS_STEP = 0.05    # parameters of its own, whose step does not shrink with the batch
_MODEL = {}


def _model():
    if not _MODEL:
        _MODEL["P"] = cf.load()
        _MODEL["theta"] = torch.tensor(grad.raw_vector(), dtype=torch.float32)
    return _MODEL


def _case(name, api, n, lo, hi, mask=0.0, samples=0):
    return {"name": name, "api": api, "n": n, "lo": lo, "hi": hi, "mask": mask, "samples": samples}


def listed():
    return [
        # the smallest call: the partition function of one short sequence, as an interactive user asks for it
        _case("logz_one_60", "logz", 1, 60, 60),
        # the benchmark's first workload: the windows of a tiled transcript
        _case("logz_1000x128", "logz", 1000, 128, 128),
        # chemical-probing data: many transcripts of unlike lengths with forced-unpaired positions
        _case("logz_mixed_masked", "logz", 1024, 50, 500, 0.1),
        # a few long RNAs, odd length
        _case("logz_4x997", "logz", 4, 997, 997),
        # the double-precision partition function, for checking a score against another program
        _case("logz64_96x200", "logz64", 96, 200, 200),
        # one structure prediction, as the command line and a notebook make it
        _case("mea_one_150", "mea", 1, 150, 150, 0.1),
        # the benchmark's headline workload: structures of a large screen
        _case("mea_10000x200", "mea", 10000, 200, 200, 0.1),
        # structures of a few long RNAs
        _case("mea_4x801", "mea", 4, 801, 801, 0.1),
        # pair-probability matrices of a small family of unlike lengths
        _case("bpp_48_mixed", "bpp", 48, 40, 400),
        # Viterbi structures of a library of short RNAs
        _case("mfe_2048_mixed", "mfe", 2048, 60, 300, 0.1),
        # an ensemble of structures for each RNA of a set (the sampling workload's lengths)
        _case("sample_1024x25", "sample", 1024, 40, 400, 0.0, 25),
        # one training step: logZ, its gradients to the features and to the soft constraints, and the updated weights
        _case("train_512x300", "train", 512, 300, 300),
    ]


# api: (sequences, lengths, cells x sequences at most, masks, samples) of the calls people make
_RANGES = {
    "logz": ((1, 2048), (20, 1000), 5.0e7),
    "logz64": ((1, 128), (20, 400), 2.0e6),
    "mea": ((1, 8192), (20, 900), 3.0e7),
    "bpp": ((1, 60), (20, 500), 3.0e6),
    "mfe": ((1, 4096), (20, 600), 3.0e7),
    "sample": ((1, 2048), (20, 500), 2.0e7),
    "train": ((1, 512), (20, 400), 2.0e7),
}


def draw(rng):
    api = rng.choice(sorted(_RANGES))
    (n0, n1), (l0, l1), most = _RANGES[api]

    def spread(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    hi = spread(l0, l1)
    lo = hi if rng.random() < 0.5 else max(l0 // 2, int(hi * rng.uniform(0.15, 0.95)))
    # a long sequence costs its length cubed: fewer of them, so that a drawn call stays below the largest listed ones
    cost = hi * hi / 2 * max(1.0, hi / 300)
    n = spread(n0, max(n0, min(n1, int(most / cost))))
    case = _case("", api, n, lo, hi, rng.choice([0.0, 0.05, 0.1, 0.25]) if api != "logz64" else 0.0,
                 rng.choice([1, 5, 10, 40]) if api == "sample" else 0)
    del case["name"]
    return case


def _lengths(case):
    rng = np.random.default_rng([case["n"], case["lo"], case["hi"]])
    return rng.integers(case["lo"], case["hi"] + 1, case["n"])


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    m = _model()
    lens = _lengths(case)
    seqs = [ALPHA[rng.integers(0, 4, int(L))].tobytes().decode() for L in lens]
    masks = None
    if case["mask"] > 0:
        masks = [(rng.random(int(L)) < case["mask"]).astype(np.uint8) for L in lens]
    state = {"api": case["api"], "P": m["P"], "seqs": seqs, "masks": masks, "samples": case["samples"],
             "seed": int(seed)}
    if case["api"] == "train":
        # soft constraints N(0, 0.5), zero beyond a sequence's end
        bonus = np.zeros((case["n"], int(lens.max())), np.float32)
        for b, L in enumerate(lens):
            bonus[b, :L] = rng.normal(0, 0.5, int(L))
        state["theta"] = m["theta"].clone().requires_grad_(True)
        state["bonus"] = torch.from_numpy(bonus).requires_grad_(True)
        # the loss of a training step: each sequence's logZ with its own weight
        state["weight"] = torch.from_numpy(rng.uniform(0.5, 1.5, case["n"]).astype(np.float32))
    return state


def _chars(structures):
    return np.frombuffer("".join(structures).encode(), np.uint8)


def run(state):
    api, seqs, masks, P = state["api"], state["seqs"], state["masks"], state["P"]
    if api == "logz":
        return np.asarray(gpu.logZ_batch(seqs, P, masks), np.float32)   # float32 values, listed as Python floats
    if api == "logz64":
        return np.asarray(gpu.logZ64_batch(seqs, P, masks), np.float64)
    if api == "mea":
        return _chars([cf.mea(seqs[0], P, 6.0, masks and masks[0])] if len(seqs) == 1
                      else gpu.mea_batch(seqs, P, 6.0, masks))
    if api == "mfe":
        return _chars([cf.mfe(seqs[0], P, masks and masks[0])] if len(seqs) == 1 else gpu.mfe_batch(seqs, P, masks))
    if api == "bpp":
        return [cf.bpp(seqs[0], P, masks and masks[0])] if len(seqs) == 1 else gpu.bpp_batch(seqs, P, masks)
    if api == "sample":
        if state["samples"] == 1:
            return _chars(gpu.fold_tasks_gpu(seqs, masks, P, seed=state["seed"]))
        drawn = gpu.sample_batch(seqs, P, state["samples"], masks, seed=state["seed"])
        return _chars([s for per in drawn for s in per])
    theta, bonus = state["theta"], state["bonus"]
    theta.grad = bonus.grad = None
    z = grad.LogZ.apply(theta, bonus, seqs, masks)
    (z * state["weight"]).mean().backward()
    return {"logz": z.detach(), "theta": theta.detach() - THETA_STEP * theta.grad,
            "bonus": bonus.detach() - BONUS_STEP * len(seqs) * bonus.grad}


def work(case):
    """Inputs read and outputs written once, and two operations for every term of the recurrences.

    Terms: a multiloop split for each of the L^3 / 6 (i, k, j), and for each of the pairable cells (6 of 16
    base pairs, both positions free) the pairable inner pairs of its window (up to 496, shorter at small spans)."""
    lo, hi, n = case["lo"], case["hi"], case["n"]
    grid = np.unique(np.linspace(lo, hi, 9).round())
    L = grid.astype(float)
    free = 6.0 / 16.0 * (1.0 - case["mask"]) ** 2
    splits = float(np.mean(L ** 3 / 6.0))
    window = float(np.mean([free * free * sum((s[1] - d) * min(496.0, d * (d - 1) / 2.0) for d in range(int(s[1])))
                            for s in [(0, x) for x in grid]]))
    length = float(np.mean(L))
    passes = {"logz": (1, 1), "logz64": (1, 1), "mfe": (1, 1), "sample": (1, 1), "bpp": (3, 3), "mea": (4, 3),
              "train": (3, 3)}[case["api"]]
    flops = 2.0 * n * (passes[0] * splits + passes[1] * window)
    inputs = length * (2 if case["mask"] else 1)
    outputs = {"logz": 4.0, "logz64": 8.0, "mfe": length, "mea": length, "sample": length * case["samples"],
               "bpp": 8.0 * float(np.mean(L ** 2)), "train": 4.0 + 8.0 * length}[case["api"]]
    if case["api"] == "sample":   # a draw reads at least one state's value for each base pair, about L / 4 of them
        flops += n * case["samples"] * length / 2.0
    return {"bytes": n * (inputs + outputs) + (708 * 8.0 if case["api"] == "train" else 0.0), "flops": flops}


# ----------------------------------------------------------------------------------------------------------------
# Exact results: the model's sum over structures in 64 bits, as sums of products (weights are exponentials of the
# scores, scaled by exp(-RATE) per position so that nothing overflows), with its derivatives by the chain rule.
# ----------------------------------------------------------------------------------------------------------------
RATE = 0.25       # per position; the factor is taken out of log Z again
WINDOW = 30       # longest interior loop


def _features():
    path = os.path.join(os.path.dirname(cf.__file__), "data", "contrafold.params.complementary")
    with open(path) as fh:
        pairs = [line.split() for line in fh]
    return {p[0]: float(p[1]) for p in pairs if len(p) == 2}


def _tied():
    """{table: (features of each entry, shape)}: an entry's score is the sum of its features."""
    names = list(_features())
    at = {k: i for i, k in enumerate(names)}
    bases = "ACGUN"

    def entry(*keys):
        for k in keys:
            if k in at:
                return [at[k]]
        return []

    def upto(prefix, first, k):
        return [at["%s_at_least_%d" % (prefix, x)] for x in range(first, k + 1) if "%s_at_least_%d" % (prefix, x) in at]

    T = {}
    two = [(a, b) for a in bases for b in bases]
    three = [(a, b, c) for a, b in two for c in bases]
    four = [t + (d,) for t in three for d in bases]
    T["bp"] = [entry("base_pair_" + a + b, "base_pair_" + b + a) for a, b in two], (5, 5)
    T["i11"] = [entry("internal_1x1_nucleotides_" + a + b, "internal_1x1_nucleotides_" + b + a) for a, b in two], (5, 5)
    T["hc"] = [entry("helix_closing_" + a + b) for a, b in two], (5, 5)
    T["dl"] = [entry("dangle_left_" + a + b + c) for a, b, c in three], (5, 5, 5)
    T["dr"] = [entry("dangle_right_" + a + b + c) for a, b, c in three], (5, 5, 5)
    T["tm"] = [entry("terminal_mismatch_" + "".join(t)) for t in four], (5, 5, 5, 5)
    T["stack"] = [entry("helix_stacking_" + "".join(t), "helix_stacking_" + "".join(t[::-1])) for t in four], (5, 5, 5, 5)
    T["b01"] = [entry("bulge_0x1_nucleotides_" + a) for a in bases], (5,)
    T["hp"] = [upto("hairpin_length", 0, k) for k in range(31)], (31,)
    loops = []
    for l1 in range(WINDOW + 1):
        for l2 in range(WINDOW + 1):
            f = []
            if 0 < l1 + l2 <= WINDOW:
                if l1 == 0 or l2 == 0:
                    f = upto("bulge_length", 1, l1 + l2)
                else:
                    if max(l1, l2) <= 4:
                        f = entry("internal_explicit_%d_%d" % (min(l1, l2), max(l1, l2)))
                    f = f + upto("internal_length", 2, l1 + l2) + upto("internal_asymmetry", 1, min(28, abs(l1 - l2)))
                    if l1 == l2:
                        f = f + upto("internal_symmetric_length", 1, min(15, l1))
            loops.append(f)
    T["cs"] = loops, (WINDOW + 1, WINDOW + 1)
    for short, key in (("mb", "multi_base"), ("mu", "multi_unpaired"), ("mp", "multi_paired"),
                       ("eu", "external_unpaired"), ("ep", "external_paired")):
        T[short] = [entry(key)], ()
    return T


def _weights(theta):
    """{table: exp(scores)} of the raw feature values, differentiable."""
    out = {}
    for k, (entries, shape) in _tied().items():
        where = [i for i, e in enumerate(entries) for _ in e]
        which = [f for e in entries for f in e]
        flat = torch.zeros(len(entries), dtype=torch.float64, device=theta.device)
        if where:
            flat = flat.index_add(0, torch.tensor(where, device=theta.device), theta[torch.tensor(which, device=theta.device)])
        out[k] = flat.reshape(shape).exp()
    return out


class _Exact:
    """Z of a batch of sequences and its derivatives.  Matrices are [sequence, i, j] with the reference's indices:
    FC[i][j] is the inside of the pair (i, j + 1), FM1 / FM multiloop parts of positions i + 1 .. j."""

    def __init__(self, seqs, masks, theta, bonus, derivatives):
        dev = theta.device
        self.lens = torch.tensor([len(s) for s in seqs], device=dev)
        n, L = len(seqs), int(self.lens.max())
        self.n, self.L, self.N = n, L, L + 3
        code = np.full((n, self.N), 4, np.int64)
        free = np.zeros((n, self.N), bool)
        for b, s in enumerate(seqs):
            code[b, 1:len(s) + 1] = ["ACGU".index(c) for c in s]
            free[b, 1:len(s) + 1] = True if masks is None or masks[b] is None else np.asarray(masks[b])[:len(s)] == 0
        s = torch.from_numpy(code).to(dev)
        free = torch.from_numpy(free).to(dev)
        self.theta = theta.detach().clone().requires_grad_(derivatives)
        w = _weights(self.theta)
        N = self.N
        k = torch.full((n, N), math.exp(-RATE), dtype=torch.float64, device=dev)   # weight of a paired position
        if bonus is not None:
            k[:, 1:L + 1] *= torch.exp(-bonus.double().to(dev))
        self.bonus = bonus
        self.unp = math.exp(-RATE)                                                 # of an unpaired one
        canon = torch.zeros((5, 5), dtype=torch.float64, device=dev)
        for x, y in ((0, 3), (1, 2), (2, 3)):
            canon[x, y] = canon[y, x] = 1.0
        i, j = torch.arange(N, device=dev)[:, None], torch.arange(N, device=dev)[None, :]
        si, sj = s[:, :, None], s[:, None, :]
        nxt, prv = torch.roll(s, -1, 1), torch.roll(s, 1, 1)
        fit = canon[si, sj] * (free[:, :, None] & free[:, None, :]) * (i < j)
        # factors of the pair (a, b), indexed [a, b]
        self.F = {
            "pair": w["bp"][si, sj] * fit * k[:, :, None] * k[:, None, :],
            "close": w["hc"][si, sj] * w["tm"][si, sj, nxt[:, :, None], prv[:, None, :]],         # loop inside the pair
            "out": w["hc"][sj, si] * w["tm"][sj, si, nxt[:, None, :], prv[:, :, None]],           # loop outside it
            "multi": w["hc"][si, sj] * w["dl"][si, sj, nxt[:, :, None]] * w["dr"][si, sj, prv[:, None, :]]
                     * w["mp"] * w["mb"],                                                          # closes a multiloop
            "end": w["hc"][sj, si] * w["dl"][sj, si, nxt[:, None, :]] * w["dr"][sj, si, prv[:, :, None]],
            # the pair (i, j + 1) on (i + 1, j), and its one-base bulges and 1x1 loop, indexed by (i, j)
            "stack": w["stack"][s[:, :, None], nxt[:, None, :], nxt[:, :, None], s[:, None, :]],
            "b_left": w["b01"][nxt][:, :, None].expand(n, N, N), "b_right": w["b01"][s][:, None, :].expand(n, N, N),
            "one_one": w["i11"][nxt[:, :, None], s[:, None, :]],
            "cs": w["cs"], "hp": w["hp"], "mu": w["mu"], "mp": w["mp"], "eu": w["eu"], "ep": w["ep"],
        }
        self.fit = fit
        self.V = {key: v.detach().clone() for key, v in self.F.items()}
        unpaired = torch.arange(WINDOW + 1, device=dev, dtype=torch.float64)
        self.V["loop"] = self.V["cs"] * self.unp ** (unpaired[:, None] + unpaired[None, :])
        self._inside()
        if derivatives:
            self._outside()

    def diag(self, M, d, lo, count, rows=0, cols=0):
        """View of M[:, i + rows, i + d + cols] for i = lo .. lo + count - 1."""
        N = self.N
        return M.as_strided((self.n, count), (N * N, N + 1), (lo + rows) * N + lo + d + cols)

    def splits(self, M, d, lo, count, second):
        """View [n, i, s] of M[:, i, i + s] (first factor) or M[:, i + s, i + d] (second), s = 1 .. d - 1."""
        N = self.N
        if second:
            return M.as_strided((self.n, count, d - 1), (N * N, N + 1, N), (lo + 1) * N + lo + d)
        return M.as_strided((self.n, count, d - 1), (N * N, N + 1, 1), lo * N + lo + 1)

    def taps(self, M, d, lo, count, t):
        """View [n, i, l1] of the inner pairs (i + 1 + l1, j - l2), l1 + l2 = t, j = i + d, of M[a, b]."""
        N = self.N
        return M.as_strided((self.n, count, t + 1), (N * N, N + 1, N + 1), (lo + 1) * N + lo + d - t)

    def row(self, W, t):
        """View of W[l1, t - l1], l1 = 0 .. t."""
        return W.as_strided((t + 1,), (WINDOW,), t)

    def _inside(self):
        V, n, N, L, dev = self.V, self.n, self.N, self.L, self.theta.device
        zero = lambda: torch.zeros((n, N, N), dtype=torch.float64, device=dev)   # noqa: E731
        self.FC, self.FM, self.FM1, self.FM2, self.win = zero(), zero(), zero(), zero(), zero()
        self.B, self.G = zero(), zero()        # the pair (a, b) with its inside; and seen from a loop around it
        loop = V["loop"]
        for d in range(0, L - 1):
            lo, c = 1, L - 1 - d               # i = 1 .. L - 1 - d
            at = lambda M, r=0, q=0: self.diag(M, d, lo, c, r, q)   # noqa: E731, B023
            if d >= 2:
                f2 = (self.splits(self.FM1, d, lo, c, False) * self.splits(self.FM, d, lo, c, True)).sum(-1)
                at(self.FM2).copy_(f2)
                f1 = at(self.B, 1, 0) * at(V["end"], 1, 0) * V["mp"] + self.diag(self.FM1, d, lo, c, 1, 0) * V["mu"] * self.unp
                at(self.FM1).copy_(f1)
                at(self.FM).copy_(f2 + at(self.FM, 0, -1) * V["mu"] * self.unp + f1)
            window = torch.zeros((n, c), dtype=torch.float64, device=dev)
            for t in range(2, min(WINDOW, d - 2) + 1):
                wt = self.row(loop, t).clone()
                if t == 2:
                    wt[1] = 0.0
                window += self.taps(self.G, d, lo, c, t) @ wt
            if d >= 3:
                window += loop[0, 1] * at(V["b_right"]) * at(self.G, 1, -1) + loop[1, 0] * at(V["b_left"]) * at(self.G, 2, 0)
            if d >= 4:
                window += loop[1, 1] * at(V["one_one"]) * at(self.G, 2, -1)
            at(self.win).copy_(window)
            fc = at(V["close"], 0, 1) * (V["hp"][min(d, 30)] * self.unp ** d + window)
            if d >= 2:
                fc = fc + at(V["stack"]) * at(self.B, 1, 0) + at(V["multi"], 0, 1) * at(self.FM2)
            fc = fc * at(self.fit, 0, 1)
            at(self.FC).copy_(fc)
            at(self.B, 0, 1).copy_(fc * at(V["pair"], 0, 1))
            at(self.G, 0, 1).copy_(at(self.B, 0, 1) * at(V["out"], 0, 1))
        self.E = self.B * V["end"] * V["ep"]
        F5 = torch.zeros((n, N), dtype=torch.float64, device=dev)
        F5[:, 0] = 1.0
        for j in range(1, L + 1):
            F5[:, j] = F5[:, j - 1] * V["eu"] * self.unp + (F5[:, :j] * self.E[:, 1:j + 1, j]).sum(1)
        self.F5 = F5
        self.Z = F5.gather(1, self.lens[:, None])[:, 0]
        total = RATE * self.lens.double()
        if self.bonus is not None:
            total = total + self.bonus.double().to(dev).sum(1)
        self.logz = self.Z.log() + total

    def _outside(self):
        """Derivatives of log Z (summed over the batch) to every factor, in reverse order of _inside."""
        V, n, N, L, dev = self.V, self.n, self.N, self.L, self.theta.device
        zero = lambda: torch.zeros((n, N, N), dtype=torch.float64, device=dev)   # noqa: E731
        D = {k: torch.zeros((n,) + v.shape if v.dim() < 3 else v.shape, dtype=torch.float64, device=dev) for k, v in V.items()}
        dF5 = torch.zeros((n, N), dtype=torch.float64, device=dev)
        dF5.scatter_(1, self.lens[:, None], (1.0 / self.Z)[:, None])
        dE = zero()
        for j in range(L, 0, -1):
            g = dF5[:, j:j + 1]
            dF5[:, j - 1] += g[:, 0] * V["eu"] * self.unp
            D["eu"] += g[:, 0] * self.F5[:, j - 1] * self.unp
            dF5[:, :j] += g * self.E[:, 1:j + 1, j]
            dE[:, 1:j + 1, j] = g * self.F5[:, :j]
        dB, dG, dFM, dFM1 = dE * V["end"] * V["ep"], zero(), zero(), zero()
        D["end"] += dE * self.B * V["ep"]
        D["ep"] += (dE * self.B * V["end"]).sum((1, 2))
        loop = V["loop"]
        for d in range(L - 2, -1, -1):
            lo, c = 1, L - 1 - d
            at = lambda M, r=0, q=0: self.diag(M, d, lo, c, r, q)   # noqa: E731, B023
            b = at(dB, 0, 1) + at(dG, 0, 1) * at(V["out"], 0, 1)
            at(D["out"], 0, 1).add_(at(dG, 0, 1) * at(self.B, 0, 1))
            at(D["pair"], 0, 1).add_(b * at(self.FC))
            f = b * at(V["pair"], 0, 1) * at(self.fit, 0, 1)           # derivative to FC
            hp = V["hp"][min(d, 30)] * self.unp ** d
            at(D["close"], 0, 1).add_(f * (hp + at(self.win)))
            D["hp"][:, min(d, 30)] += (f * at(V["close"], 0, 1)).sum(1) * self.unp ** d
            g = f * at(V["close"], 0, 1)                               # to the window's sum
            for t in range(2, min(WINDOW, d - 2) + 1):
                wt = self.row(loop, t).clone()
                if t == 2:
                    wt[1] = 0.0
                taps = self.taps(self.G, d, lo, c, t)
                got = (g[:, :, None] * taps).sum(1)
                if t == 2:
                    got[:, 1] = 0.0
                D["cs"].as_strided((n, t + 1), ((WINDOW + 1) ** 2, WINDOW), t).add_(got * self.unp ** t)
                for l1 in range(t + 1):    # overlapping taps: one offset at a time
                    self.diag(dG, d, lo, c, 1 + l1, -(t - l1)).add_(g * wt[l1])
            for need, l1, l2, key in ((3, 0, 1, "b_right"), (3, 1, 0, "b_left"), (4, 1, 1, "one_one")):
                if d >= need:
                    inner = at(self.G, 1 + l1, -l2)
                    at(D[key]).add_(g * loop[l1, l2] * inner)
                    D["cs"][:, l1, l2] += (g * at(V[key]) * inner).sum(1) * self.unp ** (l1 + l2)
                    at(dG, 1 + l1, -l2).add_(g * loop[l1, l2] * at(V[key]))
            if d >= 2:
                at(D["stack"]).add_(f * at(self.B, 1, 0))
                at(dB, 1, 0).add_(f * at(V["stack"]))
                at(D["multi"], 0, 1).add_(f * at(self.FM2))
                m = at(dFM)
                at(dFM, 0, -1).add_(m * V["mu"] * self.unp)
                D["mu"] += (m * at(self.FM, 0, -1)).sum(1) * self.unp
                one = at(dFM1) + m
                at(dB, 1, 0).add_(one * at(V["end"], 1, 0) * V["mp"])
                at(D["end"], 1, 0).add_(one * at(self.B, 1, 0) * V["mp"])
                D["mp"] += (one * at(self.B, 1, 0) * at(V["end"], 1, 0)).sum(1)
                at(dFM1, 1, 0).add_(one * V["mu"] * self.unp)
                D["mu"] += (one * at(self.FM1, 1, 0)).sum(1) * self.unp
                two = (f * at(V["multi"], 0, 1) + m)[:, :, None]
                first, second = self.splits(self.FM1, d, lo, c, False), self.splits(self.FM, d, lo, c, True)
                self.splits(dFM1, d, lo, c, False).add_(two * second)
                self.splits(dFM, d, lo, c, True).add_(two * first)
        self.D = D
        self.P = D["pair"] * V["pair"]          # probability of the pair (a, b)

    def unpaired(self):
        p = 1.0 - self.P.sum(1) - self.P.sum(2)
        return p[:, 1:self.L + 1]

    def to_theta(self, weight):
        """d (sum of weight[b] logZ_b) / d theta."""
        per = {k: torch.tensordot(weight.to(self.theta.device).double(), self.D[k], 1) if self.F[k].dim() < 3
               else self.D[k] * weight.to(self.theta.device).double()[:, None, None] for k in self.F}
        total = sum((self.F[k] * per[k]).sum() for k in self.F)
        return torch.autograd.grad(total, self.theta)[0]


def _device():
    return torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")


def exact(case, seed):
    api, n, hi = case["api"], case["n"], case["hi"]
    if api in ("mea", "mfe", "sample"):
        return None                             # structures, not numbers
    state = prepare(case, seed)
    seqs, masks = state["seqs"], state["masks"]
    theta = torch.tensor(list(_features().values()), dtype=torch.float64, device=_device())
    per = max(1, int(2.0e7 // (hi + 3) ** 2))   # sequences whose matrices are held at once
    if -(-n // per) * hi > 12000:
        return None                             # over some 20 seconds
    parts = [slice(k, min(n, k + per)) for k in range(0, n, per)]
    some = lambda v, p: None if v is None else v[p]   # noqa: E731
    if api in ("logz", "logz64"):
        z = [_Exact(seqs[p], some(masks, p), theta, None, False).logz.cpu().numpy() for p in parts]
        return np.concatenate(z)
    if api == "bpp":
        out = []
        for p in parts:
            X = _Exact(seqs[p], some(masks, p), theta, None, True)
            M = X.P.cpu().numpy()
            out += [M[b, 1:len(s) + 1, 1:len(s) + 1] for b, s in enumerate(seqs[p])]
        return out
    theta = state["theta"].detach().double().to(_device())
    z, unp, total = [], [], 0.0
    for p in parts:
        X = _Exact(seqs[p], some(masks, p), theta, state["bonus"].detach()[p, :max(map(len, seqs[p]))], True)
        w = state["weight"][p]
        z.append(X.logz.cpu().numpy())
        total = total + X.to_theta(w).cpu().numpy()
        u = np.zeros((len(seqs[p]), state["bonus"].shape[1]))
        got = (X.unpaired() * w.to(_device()).double()[:, None]).cpu().numpy()
        for b, s in enumerate(seqs[p]):
            u[b, :len(s)] = got[b, :len(s)]
        unp.append(u)
    return {"logz": np.concatenate(z), "theta": theta.cpu().numpy() - THETA_STEP * total / n,
            "bonus": state["bonus"].detach().double().numpy() - BONUS_STEP * np.concatenate(unp)}
