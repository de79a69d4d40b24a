"""The calls that are timed, and how: moments, gradients and the conductivity.

Each case is one call (or the two calls of a conductivity) that a program makes
through the public entry points of ``kpm_gb300``, on operators it holds as
device handles.  Sizes are those of the package's benchmark workloads and tests
and of the reference's own benchmark suite; ``draw`` spreads over the same
ranges.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "kpm.jl_gb300"))

import kpm_gb300 as kg  # noqa: E402
from kpm_gb300 import models  # noqa: E402

_DEVICE = "cuda"


# ------------------------------------------------------------------- cases
def listed():
    return [
        # A small sample's density of states from host arrays: what an
        # interactive session or a parameter scan calls thousands of times;
        # latency and launches decide.
        dict(name="dos small host", call="dos_host", lattice="square", Lx=32, Ly=32, W=2.0,
             NC=256, NR=8, precision="fp64"),
        # The 2D Anderson benchmark in double precision, cache resident.
        dict(name="dos 2d fp64", call="dos", lattice="square", Lx=64, Ly=64, W=2.0, NC=1024,
             NR=12, precision="fp64"),
        # The reference suite's first density of states (NH = 65536, NR = 8),
        # in float-float: mid-size, few columns.
        dict(name="dos square ff", call="dos", lattice="square", Lx=256, Ly=256, W=1.0,
             NC=1024, NR=8, precision="ff"),
        # The reference suite's second (NH = 262144, NR = 4), in the default
        # double precision.
        dict(name="dos square fp64", call="dos", lattice="square", Lx=512, Ly=512, W=1.0,
             NC=512, NR=4, precision="fp64"),
        # The headline workload's step: 3D Anderson L = 128 with 64 columns;
        # vectors far larger than the caches, bound by memory.
        dict(name="dos 3d ff", call="dos", lattice="cubic", Lx=128, Ly=128, W=16.5, NC=256,
             NR=64, precision="ff"),
        # Bra/ket moments (local spectral functions) of a complex operator at
        # odd sizes: odd NC, odd column count, rows of ten entries.
        dict(name="ldos haldane ff", call="ldos", lattice="haldane", Lx=101, Ly=87, W=0.5,
             NC=257, NR=27, precision="ff"),
        # The reference suite's conductivity moments (NH = 16384, NC = 64,
        # NR = 4), all double precision: a short call.
        dict(name="cond square fp64", call="cond", lattice="square", Lx=128, Ly=128, W=1.0,
             NC=64, NR=4, precision="fp64", contraction="fp64"),
        # The Haldane conductivity moments of the derivative workload in the
        # default double precision: dominated by the moment contraction.
        dict(name="cond haldane fp64", call="cond", lattice="haldane", Lx=64, Ly=64, W=0.0,
             NC=256, NR=8, precision="fp64", contraction="fp64"),
        # The large conductivity workload in its chosen form (float-float
        # recurrences, split contraction).
        dict(name="cond haldane split", call="cond", lattice="haldane", Lx=192, Ly=192, W=0.0,
             NC=512, NR=16, precision="ff", contraction="split"),
        # Disorder averaging: 256 samples of uneven size in one call.
        dict(name="ensemble ff", call="ensemble", members=256, Lmin=24, Lmax=96, sizes=7, W=2.0,
             NC=512, NR=8, precision="ff"),
        # The backward direction: gradient of a loss on the density of states
        # with respect to every matrix entry (graphene, from host arrays).
        dict(name="grad graphene", call="grad", lattice="graphene", Lx=128, Ly=128, W=1.0,
             NC=1024, NR=16, precision="fp64"),
        # The conductivity at 201 Fermi energies from a moment matrix.
        dict(name="sigma 201 energies", call="sigma", NC=512, nE=201, beta=0.0, NH=131072,
             precision="fp64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# rows x columns x recurrence steps of a drawn call, by precision: below the
# largest listed ones
_MOST = {"fp64": 1.0e9, "ff": 6.0e9}


def draw(rng):
    call = rng.choice(["dos", "dos", "dos", "dos_host", "ldos", "cond", "cond", "ensemble",
                       "grad", "sigma"])
    if call == "sigma":
        return dict(call=call, NC=_log_int(rng, 32, 512), nE=_log_int(rng, 1, 401),
                    beta=rng.choice([0.0, 0.0, 40.0]), NH=_log_int(rng, 1024, 200000),
                    precision="fp64")
    precision = "fp64" if call == "grad" else rng.choice(["fp64", "ff"])
    if call == "ensemble":
        Lmin = _log_int(rng, 8, 40)
        return dict(call=call, members=_log_int(rng, 8, 256), Lmin=Lmin,
                    Lmax=Lmin + rng.randint(0, 56), sizes=rng.randint(0, 999), W=2.0,
                    NC=2 * _log_int(rng, 32, 128), NR=_log_int(rng, 1, 16), precision=precision)
    NR = _log_int(rng, 1, {"cond": 16, "grad": 32, "dos_host": 16}.get(call, 64))
    if call == "cond":
        NC = _log_int(rng, 32, 256)
        contraction = "split" if precision == "ff" and rng.random() < 0.7 else "fp64"
        lattice = rng.choice(["square", "haldane"])
        rows = min(_log_int(rng, 512, 131072), int(2.0e10 / (NR * NC * NC)) + 64)
    else:
        NC = 2 * _log_int(rng, 32, 512) + (1 if call == "ldos" else 0)
        contraction = "fp64"
        lattice = "graphene" if call == "grad" else rng.choice(["square", "cubic", "haldane"])
        most = 4096 if call == "dos_host" else 32768 if call == "grad" else 600000
        rows = min(_log_int(rng, 512, most), int(_MOST[precision] / (NR * NC)) + 64)
    if lattice == "cubic":
        Lx = Ly = max(5, round(rows ** (1 / 3)))
    else:
        cells = rows if lattice == "square" else rows / 2
        Lx = max(6, round(math.sqrt(cells) * rng.uniform(0.7, 1.4)))
        Ly = max(6, round(cells / Lx))
    if lattice == "square":
        Ly = Lx
    return dict(call=call, lattice=lattice, Lx=Lx, Ly=Ly, W=rng.choice([0.5, 2.0, 8.0]), NC=NC,
                NR=NR, precision=precision, contraction=contraction)


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=96)
def _lattice(lattice, Lx, Ly):
    """The clean operators of a lattice: H, where its diagonal lies in H.data,
    and (for conductivities) the currents."""
    Jx = Jy = None
    if lattice == "square":
        H, Jx, Jy = models.square_anderson(Lx, currents=True)
    elif lattice == "cubic":
        H = models.cubic_anderson(Lx)
    elif lattice == "graphene":
        H = models.graphene(Lx, Ly, onsite=np.ones(2 * Lx * Ly))
    else:
        H, Jx, Jy, _ = models.haldane(Lx, Ly)
    cols = np.repeat(np.arange(H.shape[1]), np.diff(H.indptr))
    return H, np.flatnonzero(H.indices == cols), Jx, Jy


def _hamiltonian(lattice, Lx, Ly, W, rng):
    """The lattice with onsite disorder, spectrum scaled into (-1, 1) by the
    largest absolute row sum."""
    clean, diagonal, *_ = _lattice(lattice, Lx, Ly)
    H = clean.copy()
    H.data[diagonal] = W * (rng.random(diagonal.size) - 0.5)
    a = 1.02 * float(abs(H).sum(axis=0).max())
    H.data /= a
    return H, a


def _probes(NH, NR, seed):
    """Random-phase probes of unit norm, (NR, NH) on the GPU."""
    gen = torch.Generator(device=_DEVICE)
    gen.manual_seed(seed)
    phase = torch.rand((NR, NH), generator=gen, device=_DEVICE, dtype=torch.float64)
    return torch.polar(torch.full_like(phase, 1.0 / math.sqrt(NH)), phase.mul_(2 * math.pi))


def _members(case, rng):
    sizes = np.random.default_rng(case["sizes"]).integers(case["Lmin"], case["Lmax"] + 1,
                                                          case["members"])
    return [_hamiltonian("square", int(L), int(L), case["W"], rng)[0] for L in sizes]


def _inputs(case, seed):
    """Everything of a case that comes from the seed."""
    rng = np.random.default_rng(seed)
    call = case["call"]
    if call == "sigma":
        NC = case["NC"]
        # moments of a local response: they fall off away from the diagonal
        # and carry the noise of a stochastic trace
        n = np.arange(NC)
        mu = np.exp(-np.abs(n[:, None] - n) / 8.0) / (1.0 + n / 16.0)
        mu = mu + (rng.standard_normal((NC, NC)) + 1j * rng.standard_normal((NC, NC))) / math.sqrt(
            case["NH"])
        return dict(mu=np.asfortranarray(mu), Ef=np.linspace(-2.9, 2.9, case["nE"])
                    + 1e-3 * rng.random())
    if call == "ensemble":
        Hs = _members(case, rng)
        return dict(Hs=Hs, psi=torch.cat([_probes(H.shape[0], case["NR"], seed * 1000 + i)
                                          for i, H in enumerate(Hs)], dim=1))
    H, a = _hamiltonian(case["lattice"], case["Lx"], case["Ly"], case["W"], rng)
    NH = H.shape[0]
    got = dict(H=H, a=a, psi=_probes(NH, case["NR"], seed))
    if call == "ldos":
        got["bra"] = _probes(NH, case["NR"], seed + 500_000_000)
    if call == "cond":
        _, _, got["Jx"], got["Jy"] = _lattice(case["lattice"], case["Lx"], case["Ly"])
    if call == "grad":
        got["g"] = rng.standard_normal(case["NC"]) / (1.0 + np.arange(case["NC"]) / 32.0)
    return got


def prepare(case, seed):
    got = _inputs(case, seed)
    call, NC, NR = case["call"], case["NC"], case.get("NR")
    state = dict(case=case)
    if call == "sigma":
        return dict(state, **got)
    if call == "ensemble":
        op = kg.EnsembleOperator(got["Hs"])
        return dict(state, op=op, psi=got["psi"],
                    mu=torch.empty((len(op), NC, NR), dtype=torch.complex128, device=_DEVICE))
    state["op"] = kg.GB300Operator(got["H"])
    if call in ("dos_host", "grad"):
        # host arrays, column i = probe i
        state["psi"] = np.asfortranarray(got["psi"].cpu().numpy().T)
        state["g"] = got.get("g")
        return state
    state["psi"], state["bra"] = got["psi"], got.get("bra")
    if call == "cond":
        state["Ja"], state["Jb"] = kg.GB300Operator(got["Jx"]), kg.GB300Operator(got["Jy"])
    shape = (NC, NC) if call == "cond" else (NC, NR)
    state["mu"] = torch.empty(shape, dtype=torch.complex128, device=_DEVICE)
    return state


# --------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    call, NC = case["call"], case["NC"]
    precision = case["precision"]
    if call == "dos_host":
        return kg.kpm_1d(state["op"], NC, case["NR"], psi_in=state["psi"], avg_output=False,
                         precision=precision)
    if call == "dos":
        kg.kpm_1d_device(state["op"], NC, state["psi"], state["mu"], precision=precision)
        return state["mu"]
    if call == "ldos":
        kg.kpm_1d_device(state["op"], NC, state["psi"], state["mu"], psi_l_t=state["bra"],
                         precision=precision)
        return state["mu"]
    if call == "cond":
        kg.kpm_2d_device(state["op"], state["Ja"], state["Jb"], NC, state["psi"], state["psi"],
                         state["mu"], precision=precision, contraction=case["contraction"])
        return state["mu"]
    if call == "ensemble":
        kg.kpm_1d_ensemble_device(state["op"], NC, state["psi"], state["mu"],
                                  precision=precision)
        return state["mu"]
    if call == "grad":
        return kg.kpm_1d_grad(state["op"], NC, state["psi"], state["g"]).data
    return kg.kubo_bastin_cond(state["mu"], 3.3, state["Ef"], NH=case["NH"],
                               area=2.6 * case["NH"] / 2, beta=case["beta"] or math.inf)


# -------------------------------------------------------------------- work
_ROW = {"square": (5, 1), "cubic": (7, 1), "haldane": (10, 2), "graphene": (4, 1)}


def _rows(case):
    Lx, Ly = case["Lx"], case["Ly"]
    return {"square": Lx * Ly, "cubic": Lx ** 3}.get(case["lattice"], 2 * Lx * Ly)


def work(case):
    """Inputs read once, outputs written once; one multiplication or addition
    of two real numbers counts as one operation."""
    call, NC = case["call"], case["NC"]
    if call == "sigma":
        # the node sums need every moment once; 2 NC harmonics on 8 NC nodes
        Q = 8 * NC
        return dict(bytes=16 * NC * NC + 16 * case["nE"],
                    flops=8 * NC * NC + 16 * NC * Q + 4 * Q * case["nE"])
    if call == "ensemble":
        sizes = np.random.default_rng(case["sizes"]).integers(case["Lmin"], case["Lmax"] + 1,
                                                              case["members"])
        NH, nnz, parts = int((sizes ** 2).sum()), 5, 1
        out = 16 * case["members"] * NC * case["NR"]
    else:
        NH = _rows(case)
        nnz, parts = _ROW[case["lattice"]]
        out = 16 * NC * (NC if call == "cond" else case["NR"])
    NR = case["NR"]
    vector = 16 * NH * NR
    operator = NH * nnz * (8 * parts + 4)
    step = NH * NR * (4 * parts * nnz + 4)  # one step of the recurrence, complex vectors
    dot = 8 * NH * NR
    if call == "cond":
        return dict(bytes=vector + 3 * operator + out,
                    flops=3 * NC * step + 8 * NC * NC * NH * NR)
    if call == "ldos":
        return dict(bytes=2 * vector + operator + out, flops=NC * (step + dot))
    if call == "grad":
        # forward and adjoint steps, and one product per stored entry and step
        return dict(bytes=vector + operator + 16 * NH * nnz + 8 * NC,
                    flops=NC // 2 * (2 * step + 8 * NH * nnz * NR))
    return dict(bytes=vector + operator + out, flops=NC // 2 * (step + 2 * dot))


# ------------------------------------------------------------------- exact
def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(_DEVICE)


class _Rows:
    """A sparse operator (the block diagonal of several) as padded rows on the
    GPU, applied in 64 bits."""

    def __init__(self, *blocks):
        blocks = [M.tocsr() for M in blocks]
        first = np.cumsum([0] + [M.shape[0] for M in blocks])
        count = np.concatenate([np.diff(M.indptr) for M in blocks])
        n, width = count.size, int(count.max())
        slot = np.arange(count.sum()) - np.repeat(np.cumsum(count) - count, count)
        row = np.repeat(np.arange(n), count)
        col = np.zeros((width, n), dtype=np.int64)
        val = np.zeros((width, n), dtype=np.complex128)
        col[slot, row] = np.concatenate([M.indices + f for M, f in zip(blocks, first)])
        val[slot, row] = np.concatenate([M.data for M in blocks])
        self.col, self.val, self.slot, self.row = (_gpu(v) for v in (col, val, slot, row))
        self.block = _gpu(np.repeat(np.arange(len(blocks)), np.diff(first)))

    def __call__(self, x):
        y = x[self.col[0]].mul_(self.val[0][:, None])
        for c, v in zip(self.col[1:], self.val[1:]):
            y.add_(x[c].mul_(v[:, None]))
        return y

    def outer(self, grad, a, b, scale):
        """grad[k] += scale * sum_p conj(a[i, p]) b[j, p] for every slot."""
        for s in range(self.col.shape[0]):
            grad[s] += scale * (a.conj() * b[self.col[s]]).sum(1)


def _columns(t):
    return t.t().contiguous()  # (NR, NH) -> (NH, NR)


def _moments(H, psi, NC, sums):
    """Doubling moments of the columns of psi; sums(x) reduces over rows."""
    x, y = psi, H(psi)
    mu = [sums(x.conj() * x), sums(x.conj() * y)]
    for _ in range(NC // 2 - 1):
        x, y = y, H(y).mul_(2).sub_(x)
        mu.append(2 * sums(x.conj() * x) - mu[0])
        mu.append(2 * sums(x.conj() * y) - mu[1])
    return torch.stack(mu)


def _chain(H, v, n):
    """T_0 v, T_1 v, ... T_{n-1} v, one after another."""
    last, here = None, v
    for k in range(n):
        yield here
        if k == n - 1:
            return
        last, here = here, (H(here) if k == 0 else H(here).mul_(2).sub_(last))


def _exact_cond(got, NC):
    H, Jx, Jy = _Rows(got["H"]), _Rows(got["Jx"]), _Rows(got["Jy"])
    psi = _columns(got["psi"])
    left = torch.empty((NC, psi.numel()), dtype=psi.dtype, device=psi.device)
    for m, v in enumerate(_chain(H, psi, NC)):
        left[m] = v.reshape(-1)
    left = left.conj().t()
    mu = torch.empty((NC, NC), dtype=psi.dtype, device=psi.device)
    held = []
    for n, v in enumerate(_chain(H, Jx(psi), NC)):
        held.append(Jy(v).reshape(-1))
        if len(held) == 32 or n == NC - 1:
            mu[n + 1 - len(held):n + 1] = torch.stack(held) @ left
            held = []
    return mu.t() / psi.shape[1]  # (NC, NC) holding mu[n, m] at [m, n]


def _exact_grad(got, NC):
    """d/dH_k of sum_m g_m mu_m, by the adjoint recurrence, for every entry."""
    H, psi, g = _Rows(got["H"]), _columns(got["psi"]), got["g"]
    N, NR = NC // 2, psi.shape[1]
    v = list(_chain(H, psi, N + 1))
    grad = torch.zeros(H.val.shape, dtype=psi.dtype, device=psi.device)
    after = last = torch.zeros_like(psi)  # lambda_{k+1}, lambda_{k+2}
    for k in range(N, 0, -1):
        seed = torch.zeros_like(psi)
        if k < N:
            seed += 4 * g[2 * k] * v[k] + 2 * g[2 * k + 1] * v[k + 1]
        if k >= 2:
            seed += 2 * g[2 * k - 1] * v[k - 1]
        here = seed / NR + 2 * H(after) - last
        H.outer(grad, after, v[k], 2.0)
        after, last = here, after
    H.outer(grad, after, psi, 1.0)
    c1 = g[1] - g[3::2].sum()
    H.outer(grad, psi, psi, c1 / NR)
    # entries of the transposed order (H is Hermitian, its pattern symmetric):
    # stored entry (i, j) in rows is entry (i, j) of the column arrays at the
    # place of (j, i)
    rows = grad[H.slot, H.row].conj()
    M = got["H"].tocsr()
    order = np.lexsort((np.repeat(np.arange(M.shape[0]), np.diff(M.indptr)), M.indices))
    return rows[_gpu(order)].cpu().numpy()


def _exact_sigma(case, got):
    NC, beta = case["NC"], case["beta"]
    mu = _gpu(got["mu"])
    k = np.arange(NC)
    c = math.pi / (NC + 1)
    damp = ((NC + 1 - k) * np.cos(c * k) + np.sin(c * k) / math.tan(c)) / (NC + 1)
    damp = _gpu(damp * np.where(k > 0, 2.0, 1.0))
    mu = mu * damp[:, None] * damp
    Q = 8 * NC
    x = np.cos((2 * np.arange(Q, 0, -1) - 1) * math.pi / (2 * Q))
    x = _gpu(x[np.abs(x) < 1.0 - 1e-3])
    theta, s = torch.arccos(x), torch.sqrt(1 - x * x)
    n = torch.arange(NC, dtype=torch.float64, device=_DEVICE)[:, None]
    T = torch.cos(n * theta).to(mu.dtype)
    phase = torch.polar(torch.ones_like(T.real), n * theta)
    up = torch.complex((x + 0 * n), -n * s) * phase
    S = ((mu.t() @ T) * up + (mu @ T) * up.conj()).sum(0).real
    E = 3.3 * x
    Ef = _gpu(got["Ef"])[:, None]
    if beta:
        f = 1.0 / (torch.exp((E - Ef) * beta) + 1.0)
    else:
        f = ((E < Ef).double() + (E <= Ef).double()) / 2
    out = (f * (math.pi / Q / s ** 3 * S)).sum(1)
    scale = -2.0 * case["NH"] / (2.6 * case["NH"] / 2 * 3.3 * 3.3)
    return (scale * out).cpu().numpy()


def exact(case, seed):
    got = _inputs(case, seed)
    call, NC = case["call"], case["NC"]
    if call == "sigma":
        return _exact_sigma(case, got)
    if call == "cond":
        return _exact_cond(got, NC)
    if call == "grad":
        return _exact_grad(got, NC)
    psi = _columns(got["psi"])
    if call == "ensemble":
        H = _Rows(*got["Hs"])
        zero = torch.zeros((len(got["Hs"]), case["NR"]), dtype=psi.dtype, device=psi.device)
        mu = _moments(H, psi, NC, lambda x: zero.index_add(0, H.block, x))
        return mu.transpose(0, 1)
    H = _Rows(got["H"])
    if call == "ldos":
        bra = _columns(got["bra"]).conj()
        return torch.stack([(bra * v).sum(0) for v in _chain(H, psi, NC)])
    mu = _moments(H, psi, NC, lambda x: x.sum(0))
    return mu.t().cpu().numpy() if call == "dos_host" else mu
