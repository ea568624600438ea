"""The work a program gives this library, as cases that can be timed and compared.

One NRG step is: assemble the block Hamiltonians (hamiltonian_batch), diagonalise all blocks
(diag_batch_ptrs), recalculate the operators in the new basis and sweep the density matrix back
(gemm3_batch_array), accumulate spectral functions (spec_accumulate_array,
spec_accumulate_mats_array). Each case is one such call, or a whole run (QSRun), as
nrg_run.py makes them, on the size mixes of the autotuner's workloads and the benchmark:
orders 8-480 in batches of 40 (Anderson model, keep 1000), 800-4096 in batches of a dozen
(keep 4000; two-channel Kondo), and bulk batches of more than a thousand blocks.

Eigenvectors are defined up to their signs, so the diagonalisation cases go on to what an NRG
program forms from them: the density matrix U^T diag(exp(-betabar E)) U of every block (the
diagonal sectors of init_rho_FDM, c++/dmnrg.hpp:146-162), which every eigenvector enters.
"""
import math

import numpy as np
import torch

from nrgljubljana_b200._lib import GEMM3_DTYPE, HPIECE_DTYPE, SPECPAIR_DTYPE
from nrgljubljana_b200.api import (BinGrid, context, diag_batch_ptrs, gemm3_batch_array, hamiltonian_batch,
                                   spec_accumulate_array, spec_accumulate_mats_array)

BETABAR = 0.46      # the reference's default inverse temperature of the td output
FDMGT, FDMLS, FDMMATS, DMNRG = 1, 2, 3, 0
F64 = torch.float64

RUN_PARAM = """[param]
symtype=QS
model=SIAM
band=flat
discretization=Z
Lambda=2
z=1
keep={keep}
keepenergy=10
T=1e-8
ops=n_d A_d
dmnrg=true
specd=A_d-A_d
"""


def listed():
    return [
        # the first steps of every run, and the shallow ones of a sweep: a few tiny blocks
        {"name": "diag_first_steps", "kind": "diag", "nblk": 9, "nmin": 3, "nmax": 33},
        # an ordinary step of an Anderson-model run at keep 1000
        {"name": "diag_step", "kind": "diag", "nblk": 40, "nmin": 8, "nmax": 480},
        # many runs served at once: their steps' blocks merged into one batch
        {"name": "diag_merged_runs", "kind": "diag", "nblk": 300, "nmin": 8, "nmax": 1024},
        # a step of a two-channel Kondo run: a dozen blocks, the largest on the two-stage path
        {"name": "diag_large_blocks", "kind": "diag", "nblk": 12, "nmin": 300, "nmax": 4096},
        # the benchmark's throughput regime: more large blocks than the chip has SMs for
        {"name": "diag_bulk", "kind": "diag", "nblk": 1400, "nmin": 601, "nmax": 900},
        # the operators of an ordinary step over its kept states
        {"name": "recalc_step", "kind": "recalc", "nblk": 40, "nmin": 8, "nmax": 480, "kept": 0.4, "ops": 2},
        # the same over all states of a large step (the FDM pass)
        {"name": "recalc_all_states", "kind": "recalc", "nblk": 12, "nmin": 800, "nmax": 2000, "kept": 1.0, "ops": 1},
        # one step of the density-matrix sweep
        {"name": "rotate_step", "kind": "rotate", "nblk": 40, "nmin": 8, "nmax": 480, "kept": 0.4},
        # DM-NRG spectral function of an ordinary step on the default grid (1000 bins a decade)
        {"name": "spec_dmnrg_step", "kind": "dmnrg", "nblk": 40, "nmin": 8, "nmax": 480, "kept": 0.4, "bins": 1000},
        # both FDM parts of a large step on a coarse grid (10 bins a decade)
        {"name": "spec_fdm_large", "kind": "fdm", "nblk": 12, "nmin": 800, "nmax": 2000, "kept": 0.25, "bins": 10},
        # a Green's function on the Matsubara axis, an ordinary step, the default 100 points
        {"name": "spec_mats_step", "kind": "mats", "nblk": 40, "nmin": 8, "nmax": 480, "kept": 0.4, "mats": 100,
         "sign": -1},
        # a whole Anderson-model run with its DM-NRG spectral function
        {"name": "run_dmnrg", "kind": "run", "keep": 1000, "nmax": 40},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["diag", "diag", "diag", "diag", "recalc", "recalc", "rotate", "dmnrg", "fdm", "mats", "assemble",
                       "run"])
    if kind == "run":
        return {"kind": kind, "keep": log_int(150, 1000), "nmax": rng.randint(8, 40)}
    if kind == "diag":
        nmax = log_int(16, 4096)
        nmin = log_int(3, max(4, nmax * 2 // 3))
        nblk = log_int(1, 1400)
        c = {"kind": kind, "nblk": nblk, "nmin": nmin, "nmax": nmax}
        most = sum(n ** 3 for n in _orders(listed()[4]))
        # wide batches of blocks above the two-stage threshold are not drawn: a dozen is a large step
        while sum(n ** 3 for n in _orders(c)) > most / (4 if nmax > 1024 else 1):
            c["nblk"] = max(1, c["nblk"] // 2)
        return c
    nmax = log_int(24, 2000)
    nmin = log_int(4, max(5, nmax * 2 // 3))
    c = {"kind": kind, "nblk": log_int(2, 60), "nmin": nmin, "nmax": nmax}
    while sum(n * n for n in _orders(c)) > 12 * 1300 ** 2:
        c["nblk"] = max(2, c["nblk"] // 2)
        if c["nblk"] == 2:
            break
    if kind == "assemble":
        return dict(c, combs=rng.choice([4, 16]))
    c["kept"] = rng.choice([0.2, 0.37, 0.5, 1.0])
    if kind == "recalc":
        c["ops"] = rng.randint(1, 4)
    if kind in ("dmnrg", "fdm"):
        c["bins"] = rng.choice([10, 37, 100, 1000])
    if kind == "mats":
        c["mats"] = log_int(10, 300)
        c["sign"] = rng.choice([-1, 1])
        while c["nblk"] > 2 and sum(n * n for n in _orders(c)) * c["mats"] > 4e8:
            c["nblk"] = max(2, c["nblk"] // 2)
        while sum(n * n for n in _orders(c)) * c["mats"] > 4e8:
            c["nmax"] = max(24, c["nmax"] * 2 // 3)
            c["nmin"] = min(c["nmin"], c["nmax"] * 2 // 3)
    return c


# ---------------------------------------------------------------- sizes
def _orders(c):
    """The block orders: log-uniform between nmin and nmax."""
    r = c["nmax"] / c["nmin"]
    return [max(1, round(c["nmin"] * r ** ((b + 0.5) / c["nblk"]))) for b in range(c["nblk"])]


def _kept(c):
    return [max(1, int(n * c["kept"])) for n in _orders(c)]


def _parts(n, combs=4):
    """Ragged widths of a block's ancestors (a tiny block has empty ones)."""
    p = [n * i * (i + 2) // (combs * (combs + 2)) for i in range(combs + 1)]
    return [p[i + 1] - p[i] for i in range(combs)]


def _offsets(sizes):
    return [0] + np.cumsum(np.asarray(sizes, dtype=np.int64)).tolist()


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape):
    return torch.randn(shape, generator=g, dtype=F64, device="cuda")


def _stream():
    return torch.cuda.current_stream()


# ---------------------------------------------------------------- diagonalisation
def _hams(c, seed):
    """The benchmark's blocks: diag(2^{-k/2}) plus symmetric N(0, 0.1^2) couplings, upper triangle."""
    g, ns = _gen(seed), _orders(c)
    off = _offsets([n * n for n in ns])
    H = torch.empty(off[-1], dtype=F64, device="cuda")
    for b, n in enumerate(ns):
        h = _randn(g, n, n).mul_(0.1).triu_(1)
        h.diagonal().copy_(torch.pow(2.0, -torch.arange(n, dtype=F64, device="cuda") / 2.0))
        H[off[b]:off[b + 1]].view(n, n).copy_(h)
    return ns, off, H


def _prepare_diag(c, seed):
    ns, off, H = _hams(c, seed)
    voff = _offsets(ns)
    s = {"kind": "diag", "ns": ns, "H0": H, "H": torch.empty_like(H), "V": torch.empty_like(H),
         "rho": torch.empty_like(H), "E": torch.empty(voff[-1], dtype=F64, device="cuda"),
         "w": torch.empty(voff[-1], dtype=F64, device="cuda"), "ctx": context()}
    at = lambda t, o: [t.data_ptr() + 8 * int(x) for x in o[:-1]]  # noqa: E731
    s["Hp"], s["Ep"], s["Vp"] = at(s["H"], off), at(s["E"], voff), at(s["V"], off)
    rows = [(r, n, v, n, w, 0, v, n, n, n, n, n, 1, 0, 1.0)
            for n, r, v, w in zip(ns, at(s["rho"], off), s["Vp"], at(s["w"], voff))]
    s["terms"] = np.array(rows, dtype=GEMM3_DTYPE)
    return s


def _run_diag(s):
    s["H"].copy_(s["H0"])  # the call consumes its input
    info = diag_batch_ptrs(s["ns"], s["Hp"], s["Ep"], s["Vp"], ctx=s["ctx"], stream=_stream())
    torch.exp(torch.mul(s["E"] - s["E"].min(), -BETABAR, out=s["w"]), out=s["w"])
    s["rho"].zero_()
    gemm3_batch_array(s["terms"], ctx=s["ctx"], stream=_stream())
    return {"info": info, "evals": s["E"], "rho": s["rho"]}


def _exact_diag(c, seed):
    if sum(n ** 3 for n in _orders(c)) > 8e11:
        return None
    ns, off, H = _hams(c, seed)
    E, V = [], []
    for b, n in enumerate(ns):
        h = H[off[b]:off[b + 1]].view(n, n)
        e, v = torch.linalg.eigh(h, UPLO="U")
        E.append(e)
        V.append(v)
    E0 = torch.cat(E).min()
    rho = [((v * torch.exp(-BETABAR * (e - E0))) @ v.T).reshape(-1) for e, v in zip(E, V)]
    return {"info": None, "evals": torch.cat(E), "rho": torch.cat(rho)}


# ---------------------------------------------------------------- recalculation and density-matrix sweep
def _rows_basis(g, k, n):
    return _randn(g, k, n) / math.sqrt(n)


def _recalc_inputs(c, seed):
    """Subspaces b with k_b kept states of n_b, U (k x n) cut into four ancestors' columns, and
    `ops` operators between neighbouring subspaces, given in the ancestors' bases."""
    g, ns, ks = _gen(seed), _orders(c), _kept(c)
    U = [_rows_basis(g, k, n) for k, n in zip(ks, ns)]
    parts = [_parts(n) for n in ns]
    O = [[[_randn(g, parts[b][i], parts[b + 1][i]) for i in range(4)] for b in range(c["nblk"] - 1)]
         for _ in range(c["ops"])]
    return ns, ks, U, parts, O


def _prepare_recalc(c, seed):
    ns, ks, U, parts, O = _recalc_inputs(c, seed)
    sizes = [ks[b] * ks[b + 1] for _ in range(c["ops"]) for b in range(c["nblk"] - 1)]
    moff = _offsets(sizes)
    M = torch.empty(moff[-1], dtype=F64, device="cuda")
    rows, m = [], 0
    for o in range(c["ops"]):
        for b in range(c["nblk"] - 1):
            p, q = _offsets(parts[b]), _offsets(parts[b + 1])
            for i in range(4):
                r, rp = parts[b][i], parts[b + 1][i]
                if r and rp:
                    rows.append((M.data_ptr() + 8 * moff[m], ks[b + 1], U[b].data_ptr() + 8 * p[i], ns[b],
                                 O[o][b][i].data_ptr(), rp, U[b + 1].data_ptr() + 8 * q[i], ns[b + 1], ks[b], ks[b + 1],
                                 r, rp, 0, 1, 0.5 + 0.25 * i))
            m += 1
    return {"kind": "recalc", "U": U, "O": O, "M": M, "terms": np.array(rows, dtype=GEMM3_DTYPE), "ctx": context()}


def _run_gemm(s):
    s["M"].zero_()
    gemm3_batch_array(s["terms"], ctx=s["ctx"], stream=_stream())
    return s["M"]


def _exact_recalc(c, seed):
    ns, ks, U, parts, O = _recalc_inputs(c, seed)
    out = []
    for o in range(c["ops"]):
        for b in range(c["nblk"] - 1):
            p, q = _offsets(parts[b]), _offsets(parts[b + 1])
            M = torch.zeros(ks[b], ks[b + 1], dtype=F64, device="cuda")
            for i in range(4):
                M += (0.5 + 0.25 * i) * (U[b][:, p[i]:p[i + 1]] @ (O[o][b][i] @ U[b + 1][:, q[i]:q[i + 1]].T))
            out.append(M.reshape(-1))
    return torch.cat(out)


def _rotate_inputs(c, seed):
    g, ns, ks = _gen(seed), _orders(c), _kept(c)
    U = [_rows_basis(g, k, n) for k, n in zip(ks, ns)]
    rho = []
    for k in ks:
        a = _randn(g, k, k)
        rho.append((a + a.T) / (2.0 * k))
    return ns, ks, U, rho


def _prepare_rotate(c, seed):
    ns, ks, U, rho = _rotate_inputs(c, seed)
    sizes = [r * r for n in ns for r in _parts(n)]
    moff = _offsets(sizes)
    M = torch.empty(moff[-1], dtype=F64, device="cuda")
    rows, m = [], 0
    for b, n in enumerate(ns):
        p = _offsets(_parts(n))
        for i, r in enumerate(_parts(n)):
            if r:
                u = U[b].data_ptr() + 8 * p[i]
                rows.append((M.data_ptr() + 8 * moff[m], r, u, n, rho[b].data_ptr(), ks[b], u, n, r, r, ks[b], ks[b], 1, 0,
                             0.75))
            m += 1
    return {"kind": "rotate", "U": U, "rho": rho, "M": M, "terms": np.array(rows, dtype=GEMM3_DTYPE), "ctx": context()}


def _exact_rotate(c, seed):
    ns, ks, U, rho = _rotate_inputs(c, seed)
    out = []
    for b, n in enumerate(ns):
        p = _offsets(_parts(n))
        for i in range(4):
            u = U[b][:, p[i]:p[i + 1]]
            out.append((0.75 * (u.T @ rho[b] @ u)).reshape(-1))
    return torch.cat(out)


# ---------------------------------------------------------------- spectral functions
SCALE = 1e-3  # energy scale of the step


def _spec_inputs(c, seed):
    """Pairs of neighbouring subspaces: sorted energies in the step's units (the density of
    many-body levels grows with energy), two operators over all states, kept-space density matrices."""
    g, ns = _gen(seed), _orders(c)
    ks = _kept(c)
    dims = ks if c["kind"] == "dmnrg" else ns
    E = [torch.sort(torch.rand(n, generator=g, dtype=F64, device="cuda"))[0].sqrt() * (10.0 * SCALE) for n in dims]
    op = [[_randn(g, dims[b + 1], dims[b]) for b in range(c["nblk"] - 1)] for _ in range(2)]
    rho = []
    for k in ks:
        a = _randn(g, k, k)
        rho.append((a + a.T) / (2.0 * k))
    return ns, ks, dims, E, op, rho


def _spec_params(c):
    grid = BinGrid(-10.0, 2.0, c["bins"]) if "bins" in c else None
    return grid, {"dmnrg": dict(Emin=2.0 * SCALE, Emax=8.0 * SCALE), "fdm": dict(T=SCALE, wnf=1e-3)}.get(c["kind"])


def _prepare_spec(c, seed):
    ns, ks, dims, E, op, rho = _spec_inputs(c, seed)
    grid, prm = _spec_params(c)
    rows = []
    for b in range(c["nblk"] - 1):
        rows.append((E[b].data_ptr(), E[b + 1].data_ptr(), op[0][b].data_ptr(), dims[b], op[1][b].data_ptr(), dims[b],
                     rho[b].data_ptr(), ks[b], rho[b + 1].data_ptr(), ks[b + 1], dims[b], ks[b], dims[b + 1], ks[b + 1],
                     ks[b], ks[b + 1], 1.0 + 0.5 * (b % 3)))
    npt = c["mats"] if c["kind"] == "mats" else grid.nbins
    return {"kind": c["kind"], "E": E, "op": op, "rho": rho, "pairs": np.array(rows, dtype=SPECPAIR_DTYPE), "grid": grid,
            "prm": prm, "mats": c.get("mats"), "sign": c.get("sign", -1),
            "a": torch.zeros(npt, dtype=F64, device="cuda"), "b": torch.zeros(npt, dtype=F64, device="cuda"),
            "ctx": context()}


def _run_spec(s):
    s["a"].zero_()
    s["b"].zero_()
    kw = dict(ctx=s["ctx"], stream=_stream())
    if s["kind"] == "mats":
        spec_accumulate_mats_array(FDMMATS, s["pairs"], s["mats"], s["a"], s["b"], s["sign"], SCALE, 1e-3, **kw)
    elif s["kind"] == "dmnrg":
        spec_accumulate_array(DMNRG, s["pairs"], s["grid"], s["a"], s["b"], sign=-1, **s["prm"], **kw)
    else:
        for algo in (FDMGT, FDMLS):
            spec_accumulate_array(algo, s["pairs"], s["grid"], s["a"], s["b"], sign=-1, **s["prm"], **kw)
    return [s["a"], s["b"]]


def _bin(grid, E, w, pos, neg):
    """The log grid's linear split of each weight between neighbouring bins, by the sign of E."""
    E, w = E.reshape(-1), w.reshape(-1)
    x = (torch.log10(E.abs().clamp_min(1e-300)) - grid.log10emin) * grid.bins
    i = x.floor()
    rem = x - i
    lo, hi = i < 0, i >= grid.nbins - 1
    rem = torch.where(lo | hi, torch.zeros_like(rem), rem)
    i = i.clamp(0, grid.nbins - 1).long()
    j = (i + 1).clamp(max=grid.nbins - 1)
    for half, sel in ((pos, E >= 0), (neg, E < 0)):
        ww = torch.where(sel, w, torch.zeros_like(w))
        half.index_add_(0, i, (1.0 - rem) * ww)
        half.index_add_(0, j, rem * ww)


def _exact_spec(c, seed):
    ns, ks, dims, E, op, rho = _spec_inputs(c, seed)
    grid, prm = _spec_params(c)
    if c["kind"] == "mats":
        sign, T = c["sign"], SCALE
        wn = math.pi * T * (2 * torch.arange(c["mats"], dtype=F64, device="cuda") + (0 if sign == 1 else 1))
        a, b_ = torch.zeros_like(wn), torch.zeros_like(wn)
    else:
        a = torch.zeros(grid.nbins, dtype=F64, device="cuda")
        b_ = torch.zeros_like(a)
        T = SCALE
    for b in range(c["nblk"] - 1):
        o1, o2, ki, kj, f = op[0][b], op[1][b], ks[b], ks[b + 1], 1.0 + 0.5 * (b % 3)
        en = E[b + 1][:, None] - E[b][None, :]
        if c["kind"] == "dmnrg":
            w = (o2 @ rho[b].T) * o1 + (rho[b + 1] @ o1) * o2
            w = torch.where((en.abs() >= prm["Emin"]) & (en.abs() <= prm["Emax"]), w, torch.zeros_like(w))
            _bin(grid, en, f * w, a, b_)
            continue
        # FDM: weights of D x (D + K) and K x D (greater), (D + K) x D and D x K (lesser)
        sg = 1.0 if c["kind"] == "fdm" else float(-c["sign"])
        gt, ls = torch.zeros_like(en), torch.zeros_like(en)
        gt[:, ki:] = (o1 * o2)[:, ki:] * 1e-3 * torch.exp(-E[b] / T)[None, ki:]
        gt[kj:, :ki] = o1[kj:, :ki] * (o2[kj:, :ki] @ rho[b])
        ls[kj:, :] = sg * (o1 * o2)[kj:, :] * 1e-3 * torch.exp(-E[b + 1] / T)[kj:, None]
        ls[:kj, ki:] = sg * o1[:kj, ki:] * (rho[b + 1] @ o2[:kj, ki:])
        if c["kind"] == "fdm":
            _bin(grid, en, f * gt, a, b_)
            _bin(grid, en, f * ls, a, b_)
            continue
        e, w = en.reshape(-1), f * (gt + ls).reshape(-1)
        for n in range(c["mats"]):
            d = e * e + wn[n] * wn[n]
            re, im = -w * e / d, -w * wn[n] / d
            if n == 0 and c["sign"] == 1:  # the limit at E -> 0 of the discarded x discarded terms
                dd = torch.zeros_like(en, dtype=torch.bool)
                dd[kj:, ki:] = en[kj:, ki:].abs() <= 1e-8
                re = torch.where(dd.reshape(-1), -f * gt.reshape(-1) / T, re)
                im = torch.where(dd.reshape(-1), torch.zeros_like(im), im)
            a[n] += re.sum()
            b_[n] += im.sum()
    return [a, b_]


# ---------------------------------------------------------------- Hamiltonian assembly
def _assemble_inputs(c, seed):
    g, ns = _gen(seed), _orders(c)
    out = []
    for n in ns:
        w = _parts(n, c["combs"])
        p = _offsets(w)
        ps = []  # (kind, r0, c0, rows, cols, trans, src, factor, shift)
        for i, r in enumerate(w):
            if r:
                ps.append((0, p[i], p[i], r, r, 0, torch.rand(r, generator=g, dtype=F64, device="cuda"), 1.4142, 0.0))
        for i in range(c["combs"]):
            for j in (i + 1, i + c["combs"] // 4 + 1):
                if j < c["combs"] and w[i] and w[j]:
                    t = (i + j) % 2
                    src = _randn(g, w[j], w[i]) if t else _randn(g, w[i], w[j])
                    ps.append((1, p[i], p[j], w[i], w[j], t, src, 0.3 + 0.01 * j, 0.0))
        for i, r in enumerate(w):
            if r:
                ps.append((0, p[i], p[i], r, r, 0, None, 0.0, 0.1 * i))
        out.append(ps)
    return ns, out


def _prepare_assemble(c, seed):
    ns, pieces = _assemble_inputs(c, seed)
    off = _offsets([n * n for n in ns])
    H = torch.empty(off[-1], dtype=F64, device="cuda")
    rows = []
    for b, ps in enumerate(pieces):
        for kind, r0, c0, r, cc, t, src, f, sh in ps:
            ld = 0 if kind == 0 else src.shape[1]
            rows.append((b, kind, r0, c0, r, cc, t, 0, ld, 0 if src is None else src.data_ptr(), f, sh))
    return {"kind": "assemble", "ns": ns, "H": H, "keep": pieces, "Hp": [H.data_ptr() + 8 * int(o) for o in off[:-1]],
            "pieces": np.array(rows, dtype=HPIECE_DTYPE), "ctx": context()}


def _run_assemble(s):
    hamiltonian_batch(s["ns"], s["Hp"], s["pieces"], ctx=s["ctx"], stream=_stream())
    return s["H"]


def _exact_assemble(c, seed):
    ns, pieces = _assemble_inputs(c, seed)
    out = []
    for n, ps in zip(ns, pieces):
        H = torch.zeros(n, n, dtype=F64, device="cuda")
        for kind, r0, c0, r, cc, t, src, f, sh in ps:
            if kind == 0:
                H.diagonal()[r0:r0 + r] += (f * src if src is not None else 0.0) + sh
            else:
                H[r0:r0 + r, c0:c0 + cc] += f * (src.T if t else src)
        out.append(H.reshape(-1))
    return torch.cat(out)


# ---------------------------------------------------------------- whole runs
def _prepare_run(c, seed):
    from nrgljubljana_b200.datagen import siam_qs
    from nrgljubljana_b200.inputs import parse_param, read_data
    from nrgljubljana_b200.nrg_run import RunParams
    u = np.random.default_rng(seed).uniform(size=2)
    data = siam_qs(1.0, 0.1 * u[0], 0.03 + 0.02 * u[1], 2.0, c["nmax"], 1.0, "Z", ops=["n_d", "A_d"])
    return {"kind": "run", "p": RunParams.from_param(parse_param(RUN_PARAM.format(keep=c["keep"]))),
            "d": read_data(data)}


def _run_run(s):
    from nrgljubljana_b200.nrg_run import QSRun
    r = QSRun(s["p"], s["d"]).run()
    return {"td": np.array(r.td), "custom": np.array(r.custom),
            "spectra": {k: np.asarray(v) for k, v in r.spectra.items()}}


# ---------------------------------------------------------------- the five functions
_PREPARE = {"diag": _prepare_diag, "recalc": _prepare_recalc, "rotate": _prepare_rotate, "dmnrg": _prepare_spec,
            "fdm": _prepare_spec, "mats": _prepare_spec, "assemble": _prepare_assemble, "run": _prepare_run}
_RUN = {"diag": _run_diag, "recalc": _run_gemm, "rotate": _run_gemm, "dmnrg": _run_spec, "fdm": _run_spec,
        "mats": _run_spec, "assemble": _run_assemble, "run": _run_run}
_EXACT = {"diag": _exact_diag, "recalc": _exact_recalc, "rotate": _exact_rotate, "dmnrg": _exact_spec,
          "fdm": _exact_spec, "mats": _exact_spec, "assemble": _exact_assemble}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    return _EXACT[case["kind"]](case, seed) if case["kind"] in _EXACT else None


def work(case):
    k = case["kind"]
    if k == "run":  # the eigensolves: a step has about 40 blocks of a keep-dependent order up to 0.46 keep
        ns = _orders({"nblk": 40, "nmin": 8, "nmax": max(16, int(0.46 * case["keep"]))})
        f = case["nmax"] * sum(10 / 3 * n ** 3 for n in ns)
        return {"bytes": 8.0 * case["nmax"] * sum(4 * n * n for n in ns), "flops": f}
    ns = _orders(case)
    if k == "diag":  # eigenpairs (10/3 n^3) and the density matrix (2 n^3); H in, rho out
        return {"bytes": 8.0 * sum(2 * n * n + n for n in ns), "flops": sum((10 / 3 + 2) * n ** 3 for n in ns)}
    if k == "assemble":
        src = 0
        for n in ns:
            w, cb = _parts(n, case["combs"]), case["combs"]
            src += n + sum(w[i] * w[j] for i in range(cb) for j in (i + 1, i + cb // 4 + 1) if j < cb)
        return {"bytes": 8.0 * (sum(n * n for n in ns) + src), "flops": 2.0 * src}
    ks = _kept(case)
    pairs = list(zip(range(len(ns) - 1), range(1, len(ns))))
    if k == "recalc":
        fl = by = 0.0
        for a, b in pairs:
            for r, rp in zip(_parts(ns[a]), _parts(ns[b])):
                fl += case["ops"] * 2.0 * (r * rp * ks[b] + ks[a] * r * ks[b])
                by += case["ops"] * r * rp
            by += case["ops"] * ks[a] * ks[b]
        return {"bytes": 8.0 * (by + sum(x * y for x, y in zip(ks, ns))), "flops": fl}
    if k == "rotate":
        return {"bytes": 8.0 * sum(x * n + x * x + sum(r * r for r in _parts(n)) for x, n in zip(ks, ns)),
                "flops": sum(2.0 * x * x * n + sum(2.0 * r * x * r for r in _parts(n)) for x, n in zip(ks, ns))}
    d = ks if k == "dmnrg" else ns
    terms = float(sum(d[a] * d[b] for a, b in pairs))
    if k == "dmnrg":
        fl = sum(2.0 * ks[a] * ks[b] * (ks[a] + ks[b]) for a, b in pairs)
    else:  # kept x discarded blocks of the two products with the density matrices
        fl = sum(2.0 * ((ns[b] - ks[b]) * ks[a] * ks[a] + (ns[a] - ks[a]) * ks[b] * ks[b]) for a, b in pairs)
    fl += terms * (8.0 * case["mats"] if k == "mats" else 20.0)
    return {"bytes": 8.0 * (2 * terms + sum(x * x for x in ks)), "flops": fl}
