"""The packed split-FP16 products at the edges of their range (N_mu above 128; projections also
nb of 24 and more): odd N_mu and nb (rows that are not 16-byte aligned, a ragged last block of 32
along K), nb above 256 (the two-stage form with a full left operand), the IBZ route's factors
gathered by q and X by row, and molecules of a batch.

Tolerances: 1e-5 of the largest element (22-bit words and a truncating FP32 accumulator, at most
2^-23 of the sum per 16 K); energies and the batch's Sigma the parity tests' 1e-6."""
import numpy as np
import pytest

from coqui_b200 import capi
from coqui_b200.iaft import IAFT
from coqui_b200.symmetry import symmetric_system
from coqui_b200.synthetic import make_system
from oracle import sym_oracle as SO
from oracle import thc_oracle as O

pytestmark = pytest.mark.gpu

FT, OFT = IAFT(100.0, 10.0, "low"), O.IAFT(100.0, 10.0, "low")


@pytest.mark.parametrize("grid,nb,Np", [((2, 1, 1), 24, 129), ((2, 1, 1), 25, 130), ((3, 1, 1), 37, 203),
                                        ((1, 1, 1), 31, 257), ((2, 1, 1), 261, 300)])
def test_projection_matches_the_fp64_form(grid, nb, Np):
    s = make_system(grid, nb, nb // 2, Np, beta=100.0, seed=nb)
    rng = np.random.default_rng(nb)
    G = rng.standard_normal((3, 1, s.nk, nb, nb)) + 1j * rng.standard_normal((3, 1, s.nk, nb, nb))
    out = {}
    for mode in (capi.FP64, capi.MIXED):
        c = capi.Context(s.nk, nb, Np, FT.nt_f, FT.nw_b, grid, mode=mode)
        c.set_ir(FT)
        c.set_kmesh(s.kpts, s.lattv, s.chi_bar)
        c.set_thc(s.X, s.V)
        out[mode] = c.primary_to_aux(G)
        c.close()
    ref = out[capi.FP64]
    assert np.abs(out[capi.MIXED] - ref).max() < 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("grid,nb,Np", [((3, 1, 1), 25, 131), ((2, 2, 1), 27, 160)])
def test_ibz_route_matches_the_oracle_and_the_whole_zone(grid, nb, Np):
    d = symmetric_system("trev", grid, nb, Np, OFT, seed=Np)
    sym, out = d["sym"], []
    ref = SO.eval_Sigma_all_kspace(d["G_ibz"], SO.update_w_kspace(d["G_ibz"], d["X"], d["V"], OFT, sym),
                                   d["X"], sym, d["D"])
    for with_sym in (True, False):
        c = capi.Context(sym["nk"], nb, Np, FT.nt_f, FT.nw_b, d["grid"], mode=capi.MIXED)
        c.set_ir(FT)
        c.set_kmesh(d["kpts_lex"], d["lattv"], d["chi_lex"])
        c.set_thc(d["X_lex"], d["V_lex"])
        if with_sym:
            c.set_symmetry(sym, d["D"])
        G = d["G_ibz"] if with_sym else d["G_lex"]
        out.append((c.gw_iteration(G)[0], c.rpa_energy(G)))
        c.close()
    assert np.abs(out[0][0] - ref).max() < 1e-5 * np.abs(ref).max()
    whole = out[1][0][:, :, d["lex"][:sym["nk_ibz"]]]
    assert np.abs(out[0][0] - whole).max() < 1e-5 * np.abs(ref).max()
    assert abs(out[0][1] - out[1][1]) < 1e-6


def test_batch_molecules_match_the_oracle():
    mols = [make_system(1, nb, nb // 2, Np, beta=100.0, seed=Np, gamma_only=True)
            for nb, Np in ((25, 131), (33, 203), (24, 256), (10, 60))]
    b = capi.Batch([m.nb for m in mols], [m.Np for m in mols], FT.nt_f, FT.nw_b)
    b.set_ir(FT)
    for i, m in enumerate(mols):
        b.set_thc(i, m.X[0, 0], m.V[0])
    Gs = [m.G0(OFT) for m in mols]
    out = b.gw_iteration([G[:, 0, 0] for G in Gs])
    for m, G, S in zip(mols, Gs, out):
        dW, _, _ = O.update_w(G, m.X, m.V, OFT, m.kpts, m.lattv, m.kp_grid)
        ref = O.eval_Sigma_all_Rspace(G, dW, m.X, m.kpts, m.lattv, m.kp_grid)
        assert np.abs(S - ref[:, 0, 0]).max() < 1e-6
    b.close()
