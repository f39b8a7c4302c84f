"""The IBZ self-energy on grids where its rows are formed as convolutions (enough irreducible
k-points per operation; cubic and non-cubic grids, odd edges, one and two operations, whole and
partial groups of tau slices) against the k-space oracle, with an odd number of tau points too.
Tolerances as the other IBZ parity tests."""
import os

import numpy as np
import pytest

from coqui_b200 import capi
from coqui_b200.iaft import IAFT as ProductIAFT
from coqui_b200.symmetry import symmetric_system
from oracle import sym_oracle as SO
from oracle import thc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,grid,lam", [("trev", (2, 2, 2), 1e4), ("trev", (3, 3, 3), 1e5),
                                           ("trev", (5, 2, 3), 1e4), ("swap", (5, 5, 2), 1e4)])
@pytest.mark.parametrize("mode,tol", [(capi.FP64, 1e-10), (capi.MIXED, 1e-6)], ids=["fp64", "mixed"])
def test_convolution_rows_match_the_term_sums(kind, grid, lam, mode, tol):
    ft, pft = O.IAFT(1000.0, lam / 1000.0, "low"), ProductIAFT(1000.0, lam / 1000.0, "low")
    d = symmetric_system(kind, grid, 5, 19, ft, seed=3)
    sym = d["sym"]
    dW = SO.update_w_kspace(d["G_ibz"], d["X"], d["V"], ft, sym)
    ref = SO.eval_Sigma_all_kspace(d["G_ibz"], dW, d["X"], sym, d["D"])
    c = capi.Context(sym["nk"], 5, 19, ft.nt_f, ft.nw_b, d["grid"], mode=mode)
    c.set_ir(pft)
    c.set_kmesh(d["kpts_lex"], d["lattv"], d["chi_lex"])
    c.set_thc(d["X_lex"], d["V_lex"])
    c.set_symmetry(sym, d["D"])
    S, _ = c.gw_iteration(d["G_ibz"])
    assert np.abs(S - ref).max() < tol
    c.set_gcache_limit(0)  # every slice projected on its own
    S1, _ = c.gw_iteration(d["G_ibz"])
    assert np.abs(S1 - S).max() < 1e-12
    assert np.abs(ref).max() > 1e-3
    c.close()


@pytest.mark.parametrize("kind,grid,Np", [("trev", (2, 2, 2), 19), ("swap", (5, 5, 2), 20),
                                          ("trev", (3, 2, 1), 131)])
@pytest.mark.parametrize("mode,tol", [(capi.FP64, 1e-12), (capi.MIXED, 1e-6)], ids=["fp64", "mixed"])
def test_both_forms_of_the_rows_agree(kind, grid, Np, mode, tol):
    """COQUI_B200_IBZ_CONV picks the form: term sums launch once per tau slice, convolutions once
    per group of slices, and both give the same Sigma."""
    ft, pft = O.IAFT(1000.0, 10.0, "low"), ProductIAFT(1000.0, 10.0, "low")
    d = symmetric_system(kind, grid, 5, Np, ft, seed=4)
    sym, S, launches = d["sym"], [], []
    try:
        for form in "01":
            os.environ["COQUI_B200_IBZ_CONV"] = form
            c = capi.Context(sym["nk"], 5, Np, ft.nt_f, ft.nw_b, d["grid"], mode=mode)
            c.set_ir(pft)
            c.set_kmesh(d["kpts_lex"], d["lattv"], d["chi_lex"])
            c.set_thc(d["X_lex"], d["V_lex"])
            c.set_symmetry(sym, d["D"])
            c.gw_iteration(d["G_ibz"])
            n0 = c.kernel_launches()
            S.append(c.gw_iteration(d["G_ibz"])[0])
            launches.append(c.kernel_launches() - n0)
            c.close()
    finally:
        os.environ.pop("COQUI_B200_IBZ_CONV", None)
    assert launches[1] < launches[0]
    assert np.abs(S[0] - S[1]).max() < tol * max(1.0, np.abs(S[0]).max())


def test_sigma_fits_beside_other_allocations():
    """The rows of a group of tau slices are a buffer of up to 512 MB; with less memory left on the
    GPU the groups become smaller and the call succeeds."""
    import torch
    ft, pft = O.IAFT(1000.0, 10.0, "low"), ProductIAFT(1000.0, 10.0, "low")
    d = symmetric_system("trev", (2, 2, 2), 5, 640, ft, seed=3)
    sym = d["sym"]
    rows = sym["nk_ibz"] * 640 ** 2 * 8
    assert min(32, ft.nt_f // 2) * rows > 300 << 20
    c = capi.Context(sym["nk"], 5, 640, ft.nt_f, ft.nw_b, d["grid"], mode=capi.MIXED)
    c.set_ir(pft)
    c.set_kmesh(d["kpts_lex"], d["lattv"], d["chi_lex"])
    c.set_thc(d["X_lex"], d["V_lex"])
    c.set_symmetry(sym, d["D"])
    c.update_w(d["G_ibz"], want_w=False, want_head=False)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    ballast = torch.empty(free - (260 << 20), dtype=torch.uint8, device="cuda")
    try:
        S = c.eval_sigma(d["G_ibz"])
    finally:
        del ballast
        torch.cuda.empty_cache()
    c.close()
    c = capi.Context(sym["nk"], 5, 640, ft.nt_f, ft.nw_b, d["grid"], mode=capi.MIXED)
    c.set_ir(pft)
    c.set_kmesh(d["kpts_lex"], d["lattv"], d["chi_lex"])
    c.set_thc(d["X_lex"], d["V_lex"])
    c.set_symmetry(sym, d["D"])
    assert np.abs(c.gw_iteration(d["G_ibz"])[0] - S).max() < 1e-12
    c.close()
