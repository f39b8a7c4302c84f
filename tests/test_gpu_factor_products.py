"""The Dyson step on packed factors (N_mu above 128: split-FP16 tensor-core products of L and L^H)
against the FP64 form of the same library: sizes around the 128-row tiles and the 32-wide K blocks,
odd sizes (unaligned rows), several q-points, scales of V and Pi far from one (powers of two
that FP16 cannot hold unscaled) and rows of very different size.

Tolerance: each of the K / 16 * 3 additions of a product into the tensor core's FP32 accumulator
rounds toward zero, at most 2^-23 of its value: 72 * 1.2e-7 = 8.6e-6 for K = 384, and W takes five
such products in a row, of which the last two weigh on it fully: 2e-5 of the largest element."""
import numpy as np
import pytest

from coqui_b200 import capi
from coqui_b200.iaft import IAFT
from coqui_b200.synthetic import make_system

pytestmark = pytest.mark.gpu

FT = IAFT(100.0, 10.0, "low")


def dyson(s, Pi, mode):
    c = capi.Context(s.nk, s.nb, s.Np, FT.nt_f, FT.nw_b, s.kp_grid, mode=mode)
    c.set_ir(FT)
    c.set_kmesh(s.kpts, s.lattv, s.chi_bar)
    c.set_thc(s.X, s.V)
    W = c.dyson_w(Pi)
    c.close()
    return W


@pytest.mark.parametrize("Np,scale,spread", [(129, 1.0, 0), (160, 1e-6, 0), (191, 1e7, 0), (256, 1.0, 6),
                                             (257, 1.0, 0), (301, 1e-3, 3), (384, 1.0, 0)])
def test_w_matches_the_fp64_form(Np, scale, spread):
    s = make_system((2, 1, 1), 3, 1, Np, seed=Np)
    rng = np.random.default_rng(Np)
    s.V *= scale
    # -Pi positive semidefinite, M = L^H Pi L of order one; rows spread over 10^(2 spread)
    B = rng.standard_normal((FT.nw_half, s.nk, Np, Np)) + 1j * rng.standard_normal((FT.nw_half, s.nk, Np, Np))
    B *= (10.0 ** rng.uniform(-spread, 0, Np))[:, None]
    Pi = -(B @ np.conj(np.swapaxes(B, -1, -2))) * (0.5 / (Np * scale))
    W = dyson(s, Pi, capi.MIXED)
    ref = dyson(s, Pi, capi.FP64)
    assert np.abs(W - ref).max() < 2e-5 * np.abs(ref).max()
    assert np.abs(W - np.conj(np.swapaxes(W, -1, -2))).max() <= 1e-6 * np.abs(ref).max()
