"""The work a user of netket_gb300 has it do, as cases that can be timed and compared.

Each case is one pass through a public entry point:

* ``sample``    ``MCState.sample()``: discarded and kept Metropolis sweeps of all chains
* ``energies``  ``kernels.local_energies_fused``: E_loc of a batch of configurations
* ``log_value`` ``MCState.log_value``: log-amplitudes of given configurations
* ``minsr``     ``ngd.minsr_update``: the natural-gradient update from tanh(theta) and E_loc
* ``qgt``       ``optimizer.qgt`` on the fly: one product S v, the unit of the default SR's CG
* ``grad``      ``MCState.expect_and_grad``: sampling, energies, statistics and gradient
* ``step``      ``VMC_SR.advance``: a whole optimisation step from given parameters

Precision is "fp64" (what ``RBM()`` and ``MCState`` give by default) or "mixed"
/ "fp32" (FP32 arithmetic, as the benchmark and the batched and serving layers
use it).  ``std`` is the spread of the RBM kernel: 0.01 is the initialiser's,
the larger values those of trained parameters, where the amplitudes differ.
"""
import math

import numpy as np
import torch

import netket_gb300 as nk
from netket_gb300 import kernels as K
from netket_gb300 import ngd


def listed():
    return [
        # the first thing anyone runs: a short TFIM chain with every default
        # (FP64, 16 chains, 1008 samples); all launches and latency
        dict(name="grad_tfim16_fp64", kind="grad", lattice="chain", size=16, alpha=1,
             precision="fp64", chains=16, length=63, std=0.01),
        # Local rule on a chain of ordinary size in the default precision
        dict(name="sample_tfim64_fp64", kind="sample", lattice="chain", size=64, alpha=2,
             precision="fp64", chains=1024, length=4, discard=5, std=0.05),
        # Exchange rule in the default precision, the 6x6 Heisenberg square
        dict(name="sample_heis36_fp64", kind="sample", lattice="square", size=6, alpha=2,
             precision="fp64", chains=1024, length=4, discard=5, std=0.1),
        # the benchmark's sampling phase: 10x10 J1-J2, 4096 chains, weights that fit an SM
        dict(name="sample_j1j2_100_mixed", kind="sample", lattice="j1j2", size=10, alpha=4,
             precision="mixed", chains=4096, length=4, discard=5, std=0.05),
        # the large configuration's sampling phase: 16x16, alpha 8, 65,536 samples
        dict(name="sample_heis256_mixed", kind="sample", lattice="square", size=16, alpha=8,
             precision="mixed", chains=16384, length=4, discard=5, std=0.01),
        # single-flip energies of a long chain (a served TFIM request) in FP64
        dict(name="energies_tfim256_fp64", kind="energies", lattice="chain", size=256, alpha=1,
             precision="fp64", n=2048, std=0.03),
        # Heisenberg energies in the default precision
        dict(name="energies_heis100_fp64", kind="energies", lattice="square", size=10, alpha=2,
             precision="fp64", n=4096, std=0.05),
        # the benchmark's local-energy phase: about 200 connected elements a sample
        dict(name="energies_j1j2_100_mixed", kind="energies", lattice="j1j2", size=10, alpha=4,
             precision="mixed", n=16384, std=0.05),
        # amplitudes of many stored configurations of a wide FP32 model
        dict(name="log_value_256_fp32", kind="log_value", lattice="square", size=16, alpha=8,
             precision="fp32", n=16384, std=0.03),
        # minSR update in the default precision, 10x10 with 4096 samples
        dict(name="minsr_100_fp64", kind="minsr", lattice="square", size=10, alpha=4,
             precision="fp64", n=4096, shift=0.01, std=0.05),
        # one CG product of the default SR()
        dict(name="qgt_100_fp64", kind="qgt", lattice="square", size=10, alpha=2,
             precision="fp64", n=4096, shift=0.01, std=0.05),
        # the benchmark: a whole minSR step of the 10x10 J1-J2 model, 16,384 samples
        dict(name="step_j1j2_100_mixed", kind="step", lattice="j1j2", size=10, alpha=4,
             precision="mixed", chains=4096, length=4, discard=5, shift=1e-4, std=0.01),
    ]


# ------------------------------------------------------------------ drawing
def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _sites(lattice, size):
    return size if lattice == "chain" else size * size


def _lattice(rng, most=16):
    if rng.random() < 0.4:
        return "chain", _log_int(rng, 8, 256 if most > 10 else 100)
    lattice = rng.choice(("square", "j1j2"))
    return lattice, rng.choice([s for s in (4, 6, 8, 10, 12, 16) if s <= most])


# Terms (hidden units evaluated, one per proposal or connected element): the
# start of the range is a few thousand, the end what the listed cases take.
_MOST_TERMS = {"fp64": 4e8, "mixed": 2e10, "fp32": 2e10}


def draw(rng):
    kind = rng.choice(("sample", "sample", "energies", "energies", "log_value", "minsr", "qgt",
                       "grad", "step"))
    std = rng.choice((0.01, 0.03, 0.05, 0.1))
    alpha = rng.choice((1, 2, 3, 4, 8))
    if kind == "sample":
        precision = rng.choice(("fp64", "mixed"))
        lattice, size = _lattice(rng)
        N = _sites(lattice, size)
        length, discard = rng.choice((1, 2, 4, 7)), rng.choice((0, 5))
        most = _MOST_TERMS[precision] / (alpha * N * N * (length + discard))
        chains = _log_int(rng, 8, int(max(8, min(16384, most))))
        return dict(kind=kind, lattice=lattice, size=size, alpha=alpha, precision=precision,
                    chains=chains, length=length, discard=discard, std=std)
    if kind == "energies":
        precision = rng.choice(("fp64", "mixed"))
        lattice, size = _lattice(rng)
        N = _sites(lattice, size)
        n = _log_int(rng, 16, int(max(16, min(32768, _MOST_TERMS[precision] / (2 * alpha * N * N)))))
        return dict(kind=kind, lattice=lattice, size=size, alpha=alpha, precision=precision, n=n,
                    std=std)
    if kind == "log_value":
        precision = rng.choice(("fp64", "fp32"))
        lattice, size = _lattice(rng)
        N = _sites(lattice, size)
        n = _log_int(rng, 1, int(min(65536, 4e9 / (alpha * N * N))))
        return dict(kind=kind, lattice=lattice, size=size, alpha=alpha, precision=precision, n=n,
                    std=std)
    if kind in ("minsr", "qgt"):
        lattice, size = _lattice(rng, 10)
        alpha = min(alpha, 4)
        n = _log_int(rng, 100, 4096)
        return dict(kind=kind, lattice=lattice, size=size, alpha=alpha, precision="fp64", n=n,
                    shift=rng.choice((0.01, 0.02)), std=std)
    if kind == "grad":
        lattice, size = rng.choice((("chain", _log_int(rng, 8, 64)), ("square", 4),
                                    ("square", 6)))
        return dict(kind=kind, lattice=lattice, size=size, alpha=min(alpha, 3),
                    precision="fp64", chains=_log_int(rng, 8, 1024), length=rng.choice((1, 4, 16)),
                    std=std)
    size = rng.choice((6, 8, 10))
    alpha = rng.choice((2, 4))
    length = rng.choice((1, 2, 4))
    most = min(16384, alpha * size ** 4) // length  # no more samples than parameters
    return dict(kind=kind, lattice=rng.choice(("square", "j1j2")), size=size, alpha=alpha,
                precision="mixed", chains=_log_int(rng, 64, most), length=length, discard=5,
                shift=rng.choice((1e-3, 1e-2)), std=0.01)


# ------------------------------------------------------------------ inputs
def _model(case):
    """(graph, hilbert, operator, sampler class) as a script sets them up."""
    s = case["size"]
    if case["lattice"] == "chain":  # transverse-field Ising, single flips
        g = nk.graph.Chain(s)
        hi = nk.hilbert.Spin(0.5, N=s)
        return g, hi, nk.operator.Ising(hi, g, h=1.0, J=-1.0), nk.sampler.MetropolisLocal
    hi = nk.hilbert.Spin(0.5, N=s * s, total_sz=0)
    if case["lattice"] == "square":
        g = nk.graph.Square(s)
        H = nk.operator.Heisenberg(hi, g, J=1.0, sign_rule=True)
    else:
        g = nk.graph.Square(s, max_neighbor_order=2)
        H = nk.operator.Heisenberg(hi, g, J=[1.0, 0.5], sign_rule=[True, False])
    return g, hi, H, nk.sampler.MetropolisExchange


def _shape(case):
    N = _sites(case["lattice"], case["size"])
    return N, case["alpha"] * N


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _parameters(case, g):
    """Flat FP64 parameters [hidden bias | kernel | visible bias]; FP32 values
    where the state computes in FP32."""
    N, M = _shape(case)
    p = torch.randn(M + N * M + N, generator=g, dtype=torch.float64, device="cuda")
    p[:M] *= case["std"]
    p[M:M + N * M] *= case["std"]
    p[M + N * M:] *= case["std"]
    return p if case["precision"] == "fp64" else p.float().double()


def _configurations(case, g):
    """(n, N) spins: any on a chain, zero magnetisation on the squares."""
    N, _ = _shape(case)
    r = torch.rand((case["n"], N), generator=g, device="cuda")
    if case["lattice"] == "chain":
        return torch.where(r < 0.5, 1, -1).to(torch.int8)
    return torch.where(r.argsort(dim=1) < N // 2, 1, -1).to(torch.int8)


def _state(case, flat, seed, chains, length, discard):
    N, M = _shape(case)
    g, hi, H, sampler = _model(case)
    kw = {} if case["lattice"] == "chain" else {"graph": g}
    dtype = torch.float32 if case["precision"] == "fp32" else torch.float64
    model = nk.models.RBM(alpha=case["alpha"], param_dtype=dtype)
    vs = nk.vqs.MCState(sampler(hi, n_chains=chains, **kw), model, n_samples=chains * length,
                        n_discard_per_chain=discard, sampler_seed=seed,
                        variables={"params": model.unflatten(flat, N, M)},
                        precision=case["precision"])
    return H, vs


def _tangent(case, g, flat):
    """tanh(theta), configurations, local energies and their mean, as an SR or
    minSR solve gets them."""
    N, M = _shape(case)
    x = _configurations(case, g)
    t = torch.tanh(x.double() @ flat[M:M + N * M].view(N, M) + flat[:M])
    e = torch.randn(case["n"], generator=g, dtype=torch.float64, device="cuda") - 0.6 * N
    return t, x, e, e.mean().reshape(1)


def prepare(case, seed):
    g = _generator(seed)
    flat = _parameters(case, g)
    kind = case["kind"]
    N, M = _shape(case)
    if kind in ("sample", "grad", "step"):
        H, vs = _state(case, flat, seed + 1, case["chains"], case["length"],
                       case.get("discard", 5))
        s = dict(kind=kind, vs=vs, H=H)
        if kind == "step":
            s["flat"] = flat
            s["driver"] = nk.driver.VMC_SR(H, nk.optimizer.Sgd(0.01), diag_shift=case["shift"],
                                           variational_state=vs, use_ntk=True)
        return s
    if kind == "energies":
        x = _configurations(case, g)
        p = flat if case["precision"] == "fp64" else flat.float()
        return dict(kind=kind, H=_model(case)[2], p=p, x=x, N=N, M=M)
    if kind == "log_value":
        _, vs = _state(case, flat, seed + 1, 16, 1, 0)
        return dict(kind=kind, vs=vs, x=_configurations(case, g))
    t, x, e, mean = _tangent(case, g, flat)
    s = dict(kind=kind, t=t, x=x, e=e, mean=mean, N=N, M=M, shift=case["shift"])
    if kind == "qgt":
        s["S"] = ngd.QGTOnTheFly(t, x, N, M, case["shift"])
        s["v"] = torch.randn(flat.numel(), generator=g, dtype=torch.float64, device="cuda")
    return s


# ------------------------------------------------------------------ one pass
def _chains(vs):
    """What a sampling call leaves behind: the samples and the chains' state."""
    st = vs.sampler_state
    return dict(samples=vs.samples, sigma=st.σ, log_prob=st.log_prob,
                n_accepted=st.n_accepted_proc)


def _stats(s):
    return dict(mean=s.mean, error_of_mean=s.error_of_mean, variance=s.variance,
                tau_corr=s.tau_corr, R_hat=s.R_hat)


def run(s):
    kind = s["kind"]
    if kind == "sample":
        s["vs"].sample()
        return _chains(s["vs"])
    if kind == "energies":
        return dict(e=K.local_energies_fused(s["H"], s["p"], s["x"], s["N"], s["M"]))
    if kind == "log_value":
        return dict(log_psi=s["vs"].log_value(s["x"]))
    if kind == "minsr":
        delta, _ = ngd.minsr_update(s["t"], s["x"], s["N"], s["M"], s["e"], s["mean"], s["shift"])
        return dict(delta=delta)
    if kind == "qgt":
        return dict(Sv=s["S"] @ s["v"])
    vs = s["vs"]
    if kind == "grad":
        vs.reset()
        stats, grad = vs.expect_and_grad(s["H"])
        return dict(stats=_stats(stats), grad=grad, **_chains(vs))
    vs.flat_parameters = s["flat"]  # a step from these parameters
    stats = s["driver"].advance(1)
    st = vs.sampler_state
    return dict(stats=_stats(stats), parameters=vs.flat_parameters, sigma=st.σ,
                n_accepted=st.n_accepted_proc)


# ------------------------------------------------------------------ what a pass cannot do without
def _n_bonds(case):
    N = _sites(case["lattice"], case["size"])
    return {"chain": N, "square": 2 * N, "j1j2": 4 * N}[case["lattice"]]


def work(case):
    """Bytes: inputs read once and outputs written once.  Flops: per hidden unit
    of an amplitude ratio two updates, an exponential, a product and a sum
    (counted as 6); contractions and factorisations as usual."""
    kind = case["kind"]
    N, M = _shape(case)
    P = M + N * M + N
    es = 8 if case["precision"] == "fp64" else 4

    def sampling():
        c, L, sweeps = case["chains"], case["length"], case["length"] + case.get("discard", 5)
        return P * es + c * L * N + 2 * c * N + 24 * c, 6.0 * c * sweeps * N * M

    def energies(n):
        ratios = N if case["lattice"] == "chain" else _n_bonds(case) / 2
        return P * es + n * N + 8 * n, n * (2.0 * N * M + 6.0 * ratios * M)

    def update(n):  # T (lower triangle), its Cholesky and two products with the Jacobian
        return (n * M * es + n * N + 8 * n + 8 * P,
                1.0 * n * n * M + n ** 3 / 3.0 + 4.0 * n * N * M)

    if kind == "sample":
        b, f = sampling()
    elif kind == "energies":
        b, f = energies(case["n"])
    elif kind == "log_value":
        b, f = P * es + case["n"] * (N + es), case["n"] * (2.0 * N * M + 4.0 * M)
    elif kind == "minsr":
        b, f = update(case["n"])
    elif kind == "qgt":
        b, f = case["n"] * (M * es + N) + 24 * P, 4.0 * case["n"] * N * M
    else:
        n = case["chains"] * case["length"]
        (b0, f0), (b1, f1) = sampling(), energies(n)
        b2, f2 = update(n) if kind == "step" else (n * M * es + 8 * P, 2.0 * n * N * M)
        b, f = b0 + b1 + b2, f0 + f1 + f2
    return dict(bytes=float(b), flops=float(f))


# ------------------------------------------------------------------ the same in 64 bits
def _log_cosh(v):
    v = v.abs()
    return v + torch.log1p(torch.exp(-2.0 * v)) - math.log(2.0)


def _bonds(case):
    """(i, j, J, off-diagonal element) of the periodic square's bonds, each once."""
    s = case["size"]
    at = np.arange(s * s).reshape(s, s)
    out = {}
    for (dr, dc), J, sign in (((0, 1), 1.0, -1.0), ((1, 0), 1.0, -1.0), ((1, 1), 0.5, 1.0),
                              ((1, -1), 0.5, 1.0)):
        if J != 1.0 and case["lattice"] != "j1j2":
            continue
        to = np.roll(at, (-dr, -dc), axis=(0, 1))
        for i, j in zip(at.ravel().tolist(), to.ravel().tolist()):
            out[(min(i, j), max(i, j))] = (J, 2.0 * J * sign)
    ij = torch.tensor(list(out), device="cuda")
    v = torch.tensor(list(out.values()), dtype=torch.float64, device="cuda")
    return ij[:, 0], ij[:, 1], v[:, 0], v[:, 1]


def _exact_energies(case, flat, x):
    N, M = _shape(case)
    b, W, a = flat[:M], flat[M:M + N * M].view(N, M), flat[M + N * M:]
    chain = case["lattice"] == "chain"
    if chain:
        nbr = torch.arange(N, device="cuda").roll(-1)
        terms = N
    else:
        bi, bj, J, off = _bonds(case)
        terms = bi.numel()
    out = []
    step = max(1, int(1.5e8 // (terms * M)))
    for x0 in x.double().split(step):
        theta = x0 @ W + b
        lc = _log_cosh(theta).sum(1)
        if chain:  # h = 1, J = -1
            diag = -(x0 * x0[:, nbr]).sum(1)
            d = -2.0 * x0
            lr = torch.stack([(_log_cosh(theta + d[:, k:k + 1] * W[k]).sum(1) - lc
                               + d[:, k] * a[k]) for k in range(N)], 1)
            out.append(diag - torch.exp(lr).sum(1))
            continue
        diag = (J * x0[:, bi] * x0[:, bj]).sum(1)
        anti = x0[:, bi] != x0[:, bj]
        r, k = anti.nonzero(as_tuple=True)
        di = -2.0 * x0[r, bi[k]]
        dW = W[bi] - W[bj]  # the spins differ: both changes have the same size
        lr = _log_cosh(theta[r] + di[:, None] * dW[k]).sum(1) - lc[r] + di * (a[bi] - a[bj])[k]
        out.append(diag.index_add(0, r, off[k] * torch.exp(lr)))
    return torch.cat(out)


def _centred_jacobian(t, x):
    xd = x.double()
    O = torch.cat([t, (xd[:, :, None] * t[:, None, :]).reshape(x.shape[0], -1), xd], 1)
    O -= O.mean(0, keepdim=True)
    O /= math.sqrt(x.shape[0])
    return O


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sample", "grad", "step"):
        return None  # needs the chains' own random stream
    g = _generator(seed)
    flat = _parameters(case, g)
    N, M = _shape(case)
    if kind in ("energies", "log_value"):
        x = _configurations(case, g)
        if kind == "energies":
            terms = case["n"] * M * (N if case["lattice"] == "chain" else _n_bonds(case) / 2)
            return dict(e=_exact_energies(case, flat, x)) if terms < 8e9 else None
        xd = x.double()
        theta = xd @ flat[M:M + N * M].view(N, M) + flat[:M]
        return dict(log_psi=_log_cosh(theta).sum(1) + xd @ flat[M + N * M:])
    t, x, e, _ = _tangent(case, g, flat)
    if case["n"] * (M + N * M + N) > 3e8:
        return None
    O = _centred_jacobian(t, x)
    if kind == "minsr":
        T = O @ O.T
        T.diagonal().add_(case["shift"])
        dv = 2.0 * (e - e.mean()) / math.sqrt(case["n"])
        aux = torch.cholesky_solve(dv[:, None], torch.linalg.cholesky(T))[:, 0]
        return dict(delta=O.T @ aux)
    v = torch.randn(flat.numel(), generator=g, dtype=torch.float64, device="cuda")
    return dict(Sv=O.T @ (O @ v) + case["shift"] * v)
