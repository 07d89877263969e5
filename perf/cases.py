"""Workloads of the inference loop that are timed and compared, by name.

Three kinds of pass, the phases of one quasi-Newton round:

  sample   new couplings, then `calls` sampler calls of `nsteps` proposals
           per walker (runMCMC); whole walkers and generator states come back
  newton   the Zwanzig-reweighted Newton phase on fixed walkers (iterNewton):
           counts, then per step updateJ, regularizer, energies of dJ,
           weights, weighted bimarginals; J, dJ, bi, weights come back
  measure  one checkpoint of fixed walkers: energies, their ranks, pair
           counts, bimarginals, round statistics and the re-gauged couplings

Shapes are the ones of this repository's benchmark modes and tests: the
protein family (L=232, q=21, 2^20 walkers), the HIV protease example (L=93,
q=4, 2^18 walkers), the one-problem graph shape (L=48, q=4, 2^14 walkers),
the long family (L=512, q=21), and shapes like those of the batched problems
(L in [50, 300], q in {4, 8, 21}, odd L, walkers not a power of two).

Inputs are made on the GPU in plain torch from the seed: couplings with
fields N(0, 1) folded evenly, a background N(0, 0.05^2) and 3L contacts
N(0, 0.5^2); walkers and target sequences from mixtures of site profiles, so
that their pairs are correlated.
"""
import math

import numpy as np
import torch

from mi3gpu_b200 import MCMCGPU, GPU_node, NewtonSteps

DEVICE = 0
GAMMA, DAMPING, LAMBDA = 4e-4, 1e-3, 2e-4  # inference.infer's defaults
MSA = 8192  # sequences behind the target bimarginals


def listed():
    return [
        # smallest round's sampling: launch latency and the per-step chain
        dict(name="sample_tiny", kind="sample", L=48, q=4, N=1 << 14, nsteps=384, calls=2),
        # the real-data example's sampling phase
        dict(name="sample_hiv", kind="sample", L=93, q=4, N=1 << 18, nsteps=744, calls=1),
        # a batched problem: odd L, middle alphabet, walkers not a power of two
        dict(name="sample_mid", kind="sample", L=187, q=8, N=50688, nsteps=748, calls=1),
        # the headline workload, four sweeps of it
        dict(name="sample_protein", kind="sample", L=232, q=21, N=1 << 20, nsteps=928, calls=1),
        # long sequences: couplings larger than L2
        dict(name="sample_long", kind="sample", L=512, q=21, N=1 << 18, nsteps=512, calls=1),
        # Newton phase where launches and the per-step host read count
        dict(name="newton_tiny", kind="newton", L=48, q=4, N=1 << 14, steps=16, reg="l1z", fused=True),
        dict(name="newton_hiv", kind="newton", L=93, q=4, N=1 << 18, steps=8, reg="l1z", fused=True),
        # ragged batched problem, the unfused weight passes and l2z
        dict(name="newton_mid", kind="newton", L=151, q=8, N=66048, steps=8, reg="l2z", fused=False),
        # the headline workload's Newton phase
        dict(name="newton_protein", kind="newton", L=232, q=21, N=1 << 20, steps=3, reg="l1z", fused=True),
        # one equilibration checkpoint: small, ragged and long
        dict(name="measure_hiv", kind="measure", L=93, q=4, N=1 << 18),
        dict(name="measure_mid", kind="measure", L=101, q=21, N=99840),
        dict(name="measure_long", kind="measure", L=512, q=21, N=1 << 18),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: any length from a few sites to the long
    family, alphabets from binary to protein, walkers in steps of 512."""
    kind = rng.choice(["sample", "sample", "newton", "newton", "measure"])
    q = rng.choice([2, 3, 4, 4, 5, 6, 8, 8, 12, 16, 20, 21, 21])
    L = _log_int(rng, 12, 512)
    N = 512 * max(1, _log_int(rng, 1 << 13, 1 << 20) // 512)
    if kind == "sample":
        nsteps, calls = L * rng.choice([1, 2, 4]) + rng.randrange(0, 7), rng.choice([1, 1, 2])
        while N * nsteps * calls * L > (1 << 20) * 928 * 232 // 2:
            N = max(8192, N // 2 // 512 * 512)
            nsteps = nsteps // 2 if N == 8192 else nsteps
        return dict(kind=kind, L=L, q=q, N=N, nsteps=nsteps, calls=calls)
    while N * L * L > (1 << 20) * 232 * 232 // 2:
        N = N // 2 // 512 * 512
    if kind == "newton":
        return dict(kind=kind, L=L, q=q, N=N, steps=rng.choice([2, 3, 5]), reg=rng.choice(["l1z", "l2z", "none"]),
                    fused=rng.random() < 0.7)
    return dict(kind=kind, L=L, q=q, N=N)


# ------------------------------------------------------------------ inputs
def _pairs(L, dev):
    return torch.triu_indices(L, L, 1, device=dev)


def _inputs(case, seed):
    """Couplings (nPairs, q*q), packed walkers (words, N) and their residues
    (N, L) -- and for the counting kinds the target bimarginals."""
    dev = torch.device("cuda", DEVICE)
    L, q, N = case["L"], case["q"], case["N"]
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed) * 1000003 + 17)
    rnd = lambda *s: torch.randn(*s, device=dev, generator=g)  # noqa: E731
    h = rnd(L, q)
    i, j = _pairs(L, dev)
    P = i.numel()
    J = 0.05 * rnd(P, q, q)
    contact = torch.randperm(P, device=dev, generator=g)[: min(3 * L, P)]
    J[contact] += 0.5 * rnd(contact.numel(), q, q)
    hz = h - h.mean(1, keepdim=True)
    J += (hz[i][:, :, None] + hz[j][:, None, :]) / (L - 1)
    profiles = torch.softmax(h[None] + 0.6 * rnd(4, L, q), -1)  # P(a) ~ exp(h): the sampler's energies are -J there

    def draw_seqs(n, prof):
        comp = torch.randint(0, 4, (n,), device=dev, generator=g)
        out = torch.empty((n, L), dtype=torch.uint8, device=dev)
        cdf = prof.cumsum(-1)
        for m in range(L):
            u = torch.rand((n,), device=dev, generator=g)
            out[:, m] = (u[:, None] >= cdf[comp, m, : q - 1]).sum(1).to(torch.uint8)
        return out

    seqs = draw_seqs(N, profiles)
    J = (-J).reshape(P, q * q).contiguous()
    target = None
    if case["kind"] != "sample":
        shifted = torch.softmax(profiles.log() + 0.2 * rnd(4, L, q), -1)
        f = _pair_sums(draw_seqs(MSA, shifted), torch.ones(MSA, device=dev, dtype=torch.float64), L, q) / MSA
        target = ((f + 0.5 / MSA) / (1 + 0.5 * q * q / MSA)).float().contiguous()
    return J, seqs, target


def _pack(seqs):
    N, L = seqs.shape
    W = (L - 1) // 4 + 1
    pad = torch.zeros((N, 4 * W), dtype=torch.uint8, device=seqs.device)
    pad[:, :L] = seqs
    return pad.view(torch.int32).t().contiguous()


def _onehot(seqs, q):
    n, L = seqs.shape
    x = torch.zeros((n, L * q), dtype=torch.float64, device=seqs.device)
    x.scatter_(1, seqs.long() + torch.arange(L, device=seqs.device) * q, 1.0)
    return x


def _chunks(seqs, q):
    step = max(1, (1 << 28) // (seqs.shape[1] * q))
    for k in range(0, seqs.shape[0], step):
        yield k, _onehot(seqs[k:k + step], q)


def _pair_sums(seqs, w, L, q):
    """sum_n w_n [s_i = a][s_j = b] for i < j, (nPairs, q*q), in 64 bits."""
    acc = torch.zeros((L * q, L * q), dtype=torch.float64, device=seqs.device)
    for k, x in _chunks(seqs, q):
        acc += x.t() @ (x * w[k:k + x.shape[0], None])
    i, j = _pairs(L, seqs.device)
    return acc.view(L, q, L, q)[i, :, j, :].reshape(-1, q * q)


def _energies(J, seqs, L, q):
    """sum_{i<j} J_ij(s_i, s_j) in 64 bits."""
    i, j = _pairs(L, seqs.device)
    full = torch.zeros((L, q, L, q), dtype=torch.float64, device=seqs.device)
    full[i, :, j, :] = J.double().view(-1, q, q)
    full = full.view(L * q, L * q)
    return torch.cat([((x @ full) * x).sum(1) for _, x in _chunks(seqs, q)])


def prepare(case, seed):
    J, seqs, target = _inputs(case, seed)
    words = _pack(seqs)
    torch.cuda.synchronize()  # the device object below works on a stream of its own
    L, q, N = case["L"], case["q"], case["N"]
    gpu = MCMCGPU((torch.device("cuda", DEVICE), 0), L, q, N, 512, None, 1024, int(seed) % (1 << 31))
    node = GPU_node([gpu])
    state = dict(case=case, gpu=gpu, node=node, J=J)
    gpu.setBuf("seq main", words)
    if case["kind"] == "sample":
        node.initMCMC(case["nsteps"])
    else:
        node.initJstep()
        gpu.setBuf("bi target", target)
    gpu.setBuf("J", J)
    if case["kind"] == "newton":
        p = NewtonSteps.Param()
        p.update(bimarg=None, gamma0=GAMMA, newtonSteps=case["steps"], pcdamping=DAMPING, fracNeff=0.2, nwalkers=N,
                 reg=None if case["reg"] == "none" else case["reg"], regarg=(LAMBDA,), beta=None,
                 distribute_jstep="all", L=L, q=q, device_resident=True)
        state["param"] = p
    gpu.wait()
    return state


def run(state):
    case, gpu, node = state["case"], state["gpu"], state["node"]
    if case["kind"] == "sample":
        node.setBuf("J", state["J"])
        for _ in range(case["calls"]):
            node.runMCMC()
        return dict(seq=gpu.bufs["seq main"], rng=gpu.bufs["rngstates"])
    if case["kind"] == "newton":
        node.setBuf("J", state["J"])
        NewtonSteps.iterNewton(state["param"], None, node, _quiet, fused=case["fused"])
        b = gpu.bufs
        return dict(J=b["J"], dJ=b["dJ"], bi=b["bi"], E=b["E main"], weights=b["weights"])
    node.calcEnergies("main")
    node.rankEnergies(0)
    node.calcBicounts("main")
    node.bicounts_to_bimarg("main")
    stats = node.bimargStats("bi", "bi target", "J")[0]
    for g in node.gpus:
        g.gaugeJ("J", "dJ")
    b = gpu.bufs
    return dict(E=b["E main"], rank=b["Erank 0"], count=b["bicount"], bi=b["bi"], gauged=b["dJ"],
                stats=stats.read()[:6])


def _quiet(*a):
    pass


def work(case):
    L, q, N = case["L"], case["q"], case["N"]
    P = L * (L - 1) // 2
    table, seq = 4.0 * P * q * q, 4.0 * ((L - 1) // 4 + 1) * N
    if case["kind"] == "sample":
        n = case["nsteps"] * case["calls"]
        # per proposal 2 (L - 1) couplings added or subtracted
        return dict(bytes=table + 2 * seq + 32.0 * N + 4.0 * n, flops=2.0 * (L - 1) * N * n)
    if case["kind"] == "newton":
        # energies of J, counts, then per step energies of dJ and weighted counts
        return dict(bytes=5 * table + seq + 8.0 * N, flops=P * N * (2.0 + 2.0 * case["steps"]))
    return dict(bytes=5 * table + seq + 8.0 * N, flops=2.0 * P * N)


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"  # residues and generator words
    if case["kind"] == "newton":
        # 32-bit couplings and weights through a few steps; dJ is the small
        # difference of two bimarginals, which holds the largest error
        return dict(rel=2e-5, max=2e-3, differ=0.0)
    # energies are 32-bit sums; walkers whose energies are equal but for the
    # last bit may trade ranks
    return dict(rel=1e-5, max=1e-3, differ=0.0)


# ------------------------------------------------------------------ 64 bits
def _zero_gauge(J, q):
    J = J.view(-1, q, q)
    return J - J.mean(2, keepdim=True) - J.mean(1, keepdim=True) + J.mean((1, 2), keepdim=True)


def _exact_newton(case, J, seqs, target):
    L, q, N = case["L"], case["q"], case["N"]
    J, bt = J.double(), target.double()
    bi = _pair_sums(seqs, torch.ones(N, dtype=torch.float64, device=J.device), L, q) / N
    dJ = torch.zeros_like(J)
    ref = 0.0
    for _ in range(case["steps"]):
        dJ = dJ - GAMMA * (bt - bi) / (bi + DAMPING)
        if case["reg"] != "none":
            j0 = _zero_gauge(J + dJ, q).reshape(-1, q * q)
            pull = j0 if case["reg"] == "l2z" else torch.sign(j0)
            R = -LAMBDA * pull * GAMMA / (bi + DAMPING)
            dJ = torch.where(torch.sign(j0) != torch.sign(j0 + R), dJ - j0, dJ + R)
        E = _energies(dJ, seqs, L, q)
        w = torch.exp(ref - E)
        ref = min(0.0, float(E.min()))
        bi = _pair_sums(seqs, w, L, q)
        bi = bi / bi.sum(1, keepdim=True)
    return dict(J=J + dJ, dJ=dJ, bi=bi, E=E, weights=w)


def _exact_measure(case, J, seqs, target):
    L, q, N = case["L"], case["q"], case["N"]
    J64 = J.double()
    count = _pair_sums(seqs, torch.ones(N, dtype=torch.float64, device=J.device), L, q)
    bi = count / N
    i, j = _pairs(L, J.device)
    # fields folded evenly: zero-gauge couplings plus each site's share
    Jz = _zero_gauge(J64, q)
    row, col, mean = J64.view(-1, q, q).mean(2), J64.view(-1, q, q).mean(1), J64.mean(1)
    h = torch.zeros((L, q), dtype=torch.float64, device=J.device)
    h.index_add_(0, i, row - mean[:, None])
    h.index_add_(0, j, col - mean[:, None])
    gauged = Jz + (h[i][:, :, None] + h[j][:, None, :]) / (L - 1)
    m, t = bi.float().double(), target.double()

    def X(f):
        f = f.view(-1, q, q)
        return float((J64.view(-1, q, q) * (f - f.sum(2, keepdim=True) * f.sum(1, keepdim=True))).sum())

    top = target > 0.01
    d = (t - m).abs()
    stats = np.array([float((d * d).sum()), float(d.max()), float((d[top] / t[top]).mean()), float(top.sum()),
                      X(m), X(t)])
    return dict(E=_energies(J, seqs, L, q), rank=None, count=count, bi=bi, gauged=gauged.reshape(-1, q * q),
                stats=stats)


def exact(case, seed):
    """What run() returns, in 64 bits; None for the sampler (whole numbers)
    and where the dense one-hot products would take long."""
    if case["kind"] == "sample":
        return None
    L, q, N = case["L"], case["q"], case["N"]
    products = 2 * case["steps"] + 2 if case["kind"] == "newton" else 2
    if 2.0 * products * N * (L * q) ** 2 > 6e14:
        return None
    J, seqs, target = _inputs(case, seed)
    f = _exact_newton if case["kind"] == "newton" else _exact_measure
    return {k: None if v is None else (v.reshape(-1) if torch.is_tensor(v) else v)
            for k, v in f(case, J, seqs, target).items()}
