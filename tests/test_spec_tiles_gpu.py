"""Tile edges of the binning kernel (32 columns x 8..64 rows, four rows at a time) and of the
Matsubara kernel (2048 terms, four points at a time): rectangles of one row or column, a
remainder on either side, empty kept or discarded parts, operators inside larger matrices, every
weight formula, against the oracle's term loops (c++/algo_DMNRG.hpp, c++/algo_FDM.hpp,
c++/algo_FT.hpp)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# relative to the largest bin or point: FP64 sums of up to 2e4 terms in another order, each to
# 2^-53, a worst case of about 2e4 * 1e-16 * (sum of magnitudes / largest sum)
TOL = 1e-10

SHAPES = [(1, 1, 1, 1), (31, 0, 33, 33), (33, 33, 8, 0), (64, 32, 65, 1), (97, 40, 129, 70), (1, 0, 70, 3), (70, 69, 1, 1)]


@pytest.fixture(scope="module")
def nb():
    import nrgljubljana_b200 as m
    m.context()
    return m


def pair(rng, shape, degenerate=False):
    """One subspace pair; the operators are views of wider matrices (odd leading dimension)."""
    import torch
    ni, ki, nj, kj = shape
    Ei, Ej = np.sort(rng.uniform(0.0, 2.0, ni)), np.sort(rng.uniform(0.0, 2.0, nj))
    if degenerate and ni - ki >= 2 and nj - kj >= 2:
        Ej[-2:] = Ei[-2:]  # discarded x discarded terms at E = 0
    sym = lambda k: (lambda a: (a + a.T) / 4)(rng.standard_normal((k, k)))  # noqa: E731
    p = dict(Ei=Ei, Ej=Ej, op1=rng.standard_normal((nj, ni)), op2=rng.standard_normal((nj, ni)), ri=sym(ki), rj=sym(kj),
             shape=shape, factor=float(rng.uniform(0.5, 2.0)))
    dev = {k: torch.tensor(v, device="cuda") for k, v in p.items() if isinstance(v, np.ndarray)}
    for k in ("op1", "op2"):
        wide = torch.full((nj, ni + 3), float("nan"), dtype=torch.float64, device="cuda")
        wide[:, 1:1 + ni] = dev[k]
        dev[k] = wide[:, 1:1 + ni]
    return p, dev


def rows_of(pairs, dm=False):
    from nrgljubljana_b200._lib import SPECPAIR_DTYPE
    out = []
    for p, d in pairs:
        ni, ki, nj, kj = p["shape"]
        out.append((d["Ei"].data_ptr(), d["Ej"].data_ptr(), d["op1"].data_ptr(), d["op1"].stride(0), d["op2"].data_ptr(),
                    d["op2"].stride(0), d["ri"].data_ptr(), max(ki, 1), d["rj"].data_ptr(), max(kj, 1),
                    ni, ki, nj, kj, ki, kj, p["factor"]))
    return np.array(out, dtype=SPECPAIR_DTYPE)


@pytest.mark.parametrize("algo", ["dmnrg", "gt", "ls"])
@pytest.mark.parametrize("bins,lo", [(3, -6.0), (500, -8.0)])
def test_bins(nb, oracle, algo, bins, lo):
    import torch
    from nrgljubljana_b200.api import spec_accumulate_array
    rng = np.random.default_rng(bins + len(algo))
    pairs = [pair(rng, s) for s in SHAPES]
    grid, cb = nb.BinGrid(lo, 1.0, bins), oracle.ChainBinning(lo, 1.0, bins)
    T, wnf = 0.3, 0.17
    for p, _ in pairs:
        ni, ki, nj, kj = p["shape"]
        if algo == "dmnrg":
            if ki and kj:
                cb.dmnrg_pair(p["Ei"][:ki], p["Ej"][:kj], p["op1"][:kj, :ki], p["op2"][:kj, :ki], p["ri"], p["rj"],
                              p["factor"], -1, 0.01, 1.5)
        else:
            cb.fdm_pair(algo, p["Ei"], ki, p["Ej"], kj, p["op1"], p["op2"], p["ri"] if algo == "gt" else p["rj"],
                        p["factor"], -1, T, wnf)
    pos = torch.zeros(grid.nbins, dtype=torch.float64, device="cuda")
    neg = torch.zeros_like(pos)
    spec_accumulate_array({"dmnrg": 0, "gt": 1, "ls": 2}[algo], rows_of(pairs), grid, pos, neg, sign=-1, T=T, wnf=wnf,
                          Emin=0.01, Emax=1.5)
    ref = np.concatenate([cb.pos_re, cb.neg_re])
    got = np.concatenate([pos.cpu().numpy(), neg.cpu().numpy()])
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("sign", [-1, 1])
@pytest.mark.parametrize("mats", [1, 3, 4, 5, 101])
def test_matsubara(nb, oracle, mats, sign):
    import torch
    from nrgljubljana_b200.api import spec_accumulate_mats_array
    from oracle.nrg_run_cpu import dmnrg_mats_pair, ft_mats_pair, mats_pair
    rng = np.random.default_rng(10 * mats + sign)
    T, wnf = 0.05, 0.21
    w = T * math.pi * (2 * np.arange(mats) + (0 if sign == 1 else 1))
    pairs = [pair(rng, s, degenerate=True) for s in SHAPES]
    for algo in ("fdm", "ft", "dmnrg"):
        ref = np.zeros(mats, dtype=complex)
        for p, _ in pairs:
            ni, ki, nj, kj = p["shape"]
            if algo == "fdm":
                ref += mats_pair(p["Ei"], ki, p["Ej"], kj, p["op1"], p["op2"], p["ri"], p["rj"], p["factor"], sign, T,
                                 wnf, w)
            elif algo == "ft":
                ref += ft_mats_pair(p["Ei"], p["Ej"], p["op1"], p["op2"], 1.0 / wnf, p["factor"], sign, T, w)
            elif ki and kj:
                ref += dmnrg_mats_pair(p["Ei"][:ki], p["Ej"][:kj], p["op1"][:kj, :ki], p["op2"][:kj, :ki], p["ri"],
                                       p["rj"], p["factor"], sign, T, w)
        re = torch.zeros(mats, dtype=torch.float64, device="cuda")
        im = torch.zeros_like(re)
        spec_accumulate_mats_array({"fdm": 3, "ft": 4, "dmnrg": 0}[algo], rows_of(pairs), mats, re, im, sign, T, wnf)
        got = re.cpu().numpy() + 1j * im.cpu().numpy()
        assert np.abs(got - ref).max() <= TOL * np.abs(ref).max(), algo


@pytest.mark.parametrize("E", [5e-155, 1e-155, 1e-120, 1e-9])
def test_matsubara_small_energy_at_zero_frequency(nb, E):
    """A discarded x kept term of energy E at the bosonic w_0 = 0 is -w / E, also where 1 / E^2 is out of range
    (E^2 is then a denormal number, whose spacing is the tolerance)."""
    import torch
    from nrgljubljana_b200.api import spec_accumulate_mats_array
    rng = np.random.default_rng(3)
    p, d = pair(rng, (1, 0, 1, 1))
    d["Ei"].zero_()
    d["Ej"].fill_(E)
    T, wnf = 0.05, 0.21
    re = torch.zeros(3, dtype=torch.float64, device="cuda")
    im = torch.zeros_like(re)
    spec_accumulate_mats_array(3, rows_of([(p, d)]), 3, re, im, 1, T, wnf)
    w = p["factor"] * p["op1"][0, 0] * p["op2"][0, 0] * (wnf - p["rj"][0, 0])
    assert abs(re[0].item() + w / E) <= abs(w / E) * (2.0 ** -48 + 2.0 ** -1074 / (E * E))
    assert im[0].item() == 0.0
    for n in (1, 2):
        wn = 2 * n * math.pi * T
        assert abs(re[n].item() + w * E / wn ** 2) <= 1e-14 * abs(w / wn) and abs(im[n].item() + w / wn) <= 1e-14 * abs(w / wn)
