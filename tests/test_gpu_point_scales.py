"""THC data have a free scale per interpolating point: X_P -> s_P X_P with V_PQ -> V_PQ / (s_P^2
s_Q^2) leaves Sigma and E_c as they are.  The mixed form's packed products (N_mu above 128) keep
their accuracy over spreads of s_P that FP16 words under one scale per matrix could not hold.

Tolerances: the 22-bit words and the truncating FP32 accumulation of a product (2e-5 of the largest
element for W and 1e-5 for a projection, as derived in the tests of the packed products) do not
depend on the scales, so Sigma and E_c of the scaled data are off by what they are for the unscaled
data (1.0e-5 and 1.8e-5 of the largest Sigma for these two systems), up to a factor of two for other
roundings of the same size."""
import numpy as np
import pytest

from coqui_b200 import capi
from coqui_b200.iaft import IAFT
from coqui_b200.symmetry import symmetric_system
from coqui_b200.synthetic import make_system

pytestmark = pytest.mark.gpu

FT = IAFT(100.0, 10.0, "low")


def context(s, mode):
    c = capi.Context(s.nk, s.nb, s.Np, FT.nt_f, FT.nw_b, s.kp_grid, mode=mode)
    c.set_ir(FT)
    c.set_kmesh(s.kpts, s.lattv, s.chi_bar)
    c.set_thc(s.X, s.V)
    return c


def scales(n, decades, seed):
    d = 10.0 ** np.random.default_rng(seed).uniform(-decades, 0, n)
    d[:2] = 1.0, 10.0 ** -decades
    return d


def dense_g(s):
    """G0 with MO coefficients that mix the orbitals (the synthetic system's are the identity)."""
    rng = np.random.default_rng(3)
    q, _ = np.linalg.qr(rng.standard_normal((s.nb, s.nb)) + 1j * rng.standard_normal((s.nb, s.nb)))
    return np.einsum("ia,tskab,jb->tskij", q, s.G0(FT), np.conj(q), optimize=True)


@pytest.mark.parametrize("Np", [129, 200, 290])
@pytest.mark.parametrize("decades", [2, 2.4, 3, 5, 8])  # 10^2.4: the largest that counts as ungraded
def test_w_of_graded_v_and_pi(Np, decades):
    """V = D V0 D with Pi = D^-1 Pi0 D^-1: D^-1 W D^-1 does not depend on D."""
    s = make_system((2, 1, 1), 3, 1, Np, seed=Np)
    rng = np.random.default_rng(Np)
    B = rng.standard_normal((FT.nw_half, s.nk, Np, Np)) + 1j * rng.standard_normal((FT.nw_half, s.nk, Np, Np))
    Pi = -(B @ np.conj(np.swapaxes(B, -1, -2))) * (0.5 / Np)
    d = 1.0 / scales(Np, decades, Np + int(decades))
    dd = d[:, None] * d[None, :]
    c = context(s, capi.FP64)
    ref = c.dyson_w(Pi)
    c.close()
    s.V = s.V * dd
    c = context(s, capi.MIXED)
    W = c.dyson_w(Pi / dd) / dd
    c.close()
    assert np.abs(W - ref).max() < 2e-5 * np.abs(ref).max()


@pytest.mark.parametrize("grid,nb,Np", [((2, 1, 1), 26, 160), ((1, 1, 1), 37, 300)])
@pytest.mark.parametrize("decades", [3, 5, 6])
def test_sigma_and_energy_do_not_depend_on_point_scales(grid, nb, Np, decades):
    s = make_system(grid, nb, nb // 2, Np, beta=100.0, seed=5)
    G = dense_g(s)
    res = {}
    for mode in (capi.FP64, capi.MIXED):
        c = context(s, mode)
        res[mode] = c.gw_iteration(G)[0], c.rpa_energy(G)
        c.close()
    (ref, e_ref), (S0, e0) = res[capi.FP64], res[capi.MIXED]
    assert np.abs(S0 - ref).max() < 4e-5 * np.abs(ref).max()
    f = scales(Np, decades, decades)
    s.X = s.X * f[:, None]
    s.V = s.V / (f[:, None] * f[None, :]) ** 2
    c = context(s, capi.MIXED)
    S, e = c.gw_iteration(G)[0], c.rpa_energy(G)
    c.close()
    assert np.abs(S - ref).max() < 2 * np.abs(S0 - ref).max()
    assert abs(e - e_ref) < 2 * abs(e0 - e_ref) + 1e-6 * abs(e_ref)


def test_batch_and_ibz_sigma_do_not_depend_on_point_scales():
    mols = [make_system(1, nb, nb // 2, Np, beta=100.0, seed=Np, gamma_only=True)
            for nb, Np in ((9, 60), (26, 150), (25, 300))]
    Gs = [dense_g(m)[:, 0, 0] for m in mols]
    out = []
    for decades in (0, 5):
        b = capi.Batch([m.nb for m in mols], [m.Np for m in mols], FT.nt_f, FT.nw_b)
        b.set_ir(FT)
        for i, m in enumerate(mols):
            # the second molecule stays as it is: graded and ordinary factors in one launch
            f = scales(m.Np, decades if i != 1 else 0, i)
            b.set_thc(i, m.X[0, 0] * f[:, None], m.V[0] / (f[:, None] * f[None, :]) ** 2)
        out.append(b.gw_iteration(Gs))
        b.close()
    for a, c in zip(*out):  # two results, each up to 4e-5 of the largest off
        assert np.abs(a - c).max() < 8e-5 * np.abs(a).max()

    d = symmetric_system("trev", (3, 1, 1), 25, 150, FT, seed=3)
    sym, res = d["sym"], []
    for decades in (0, 5):
        f = scales(150, decades, 1)
        c = capi.Context(sym["nk"], 25, 150, FT.nt_f, FT.nw_b, d["grid"], mode=capi.MIXED)
        c.set_ir(FT)
        c.set_kmesh(d["kpts_lex"], d["lattv"], d["chi_lex"])
        c.set_thc(d["X_lex"] * f[:, None], d["V_lex"] / (f[:, None] * f[None, :]) ** 2)
        c.set_symmetry(sym, d["D"])
        res.append(c.gw_iteration(d["G_ibz"])[0])
        c.close()
    assert np.abs(res[0] - res[1]).max() < 8e-5 * np.abs(res[0]).max()


@pytest.mark.parametrize("decades", [0, 4, 9])
def test_projection_of_graded_orbitals_and_tiny_values(decades):
    """X_Pa -> t_a X_Pa with G_ab -> G_ab / (t_a t_b) leaves G_PQ as it is; collocation values near
    2^-60 give G_PQ near 2^-120, which FP32 holds."""
    s = make_system((2, 1, 1), 27, 9, 131, beta=100.0, seed=8)
    G = dense_g(s)
    c = context(s, capi.FP64)
    ref = c.primary_to_aux(G)
    c.close()
    t = scales(27, decades, 2)
    s.X = s.X * t
    c = context(s, capi.MIXED)
    out = c.primary_to_aux(G / (t[:, None] * t[None, :]))
    c.close()
    assert np.abs(out - ref).max() < 1e-5 * np.abs(ref).max()
    if decades == 0:
        s.X = s.X * 2.0 ** -60
        s.V = s.V * 2.0 ** 60
        c = context(s, capi.MIXED)
        tiny = c.primary_to_aux(G)
        c.close()
        assert np.abs(tiny * 2.0 ** 120 - ref).max() < 1e-5 * np.abs(ref).max()
