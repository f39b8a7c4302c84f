"""Consecutive calls with ordinary numpy arrays run directly, then capture, then replay the GW
iteration and the RPA energy of the resident G.  Every call of such a run gives what a fresh
context gives for its own inputs, also when the inputs, the THC data or the entry point change in
between, and non-finite inputs are refused on a replayed call too."""
import numpy as np
import pytest

from coqui_b200 import capi
from coqui_b200.iaft import IAFT
from coqui_b200.synthetic import make_system

pytestmark = pytest.mark.gpu

FT = IAFT(1000.0, 10.0, "low")


def context(s):
    c = capi.Context(s.nk, s.nb, s.Np, FT.nt_f, FT.nw_b, s.kp_grid, mode=capi.MIXED)
    c.set_ir(FT)
    c.set_kmesh(s.kpts, s.lattv, s.chi_bar)
    c.set_thc(s.X, s.V)
    return c


@pytest.mark.parametrize("grid,Np", [((1, 1, 1), 40), ((2, 2, 2), 130), ((3, 2, 1), 33)])
def test_replayed_calls_match_fresh_contexts(grid, Np):
    s, s2 = (make_system(grid, 7, 3, Np, seed=i) for i in (1, 2))
    Gs = [s.G0(FT), s2.G0(FT)]
    sigma, energy = {}, {}
    for t, sys in enumerate((s, s2)):
        for i, G in enumerate(Gs):
            c = context(sys)
            sigma[t, i] = c.gw_iteration(G)[0]
            c.close()
            c = context(sys)
            energy[t, i] = c.rpa_energy(G)
            c.close()
    c = context(s)
    for i in (0, 1, 0, 1, 1):
        assert np.array_equal(c.gw_iteration(Gs[i])[0], sigma[0, i])
    for i in (1, 0, 0, 1):
        assert c.rpa_energy(Gs[i]) == energy[0, i]
    c.set_thc(s2.X, s2.V)
    for i in (0, 1, 0):
        assert np.array_equal(c.gw_iteration(Gs[i])[0], sigma[1, i])
    bad = Gs[0].copy()
    bad[3, 0, 0, 1, 1] = np.nan
    with pytest.raises(capi.CoquiB200Error) as e:
        c.gw_iteration(bad)
    assert e.value.code == -1
    for i in (1, 0, 1):
        assert np.array_equal(c.gw_iteration(Gs[i])[0], sigma[1, i])
        assert c.rpa_energy(Gs[i]) == energy[1, i]
    c.close()


def test_replayed_calls_report_the_phases_of_the_direct_one():
    """To a caller that reads the breakdown; another one's graphs do not pay for the events."""
    s = make_system((2, 2, 2), 7, 3, 40, seed=1)
    G = s.G0(FT)
    c = context(s)
    for call in (lambda: c.gw_iteration(G), lambda: c.rpa_energy(G)):
        names, total = [], []
        for _ in range(4):  # direct, captured, replayed twice
            call()
            t = c.timings()
            names.append([n for n, _ in t])
            assert all(0 < ms < 1000 for _, ms in t), t
            total.append(sum(ms for _, ms in t))
        assert all(n == names[0] for n in names) and "EVALUATE_PI_R" in names[0]
        assert total[3] < 10 * total[2] and total[2] < 10 * total[3]
    c.close()
    c = context(s)  # nobody reads the breakdown of the first calls
    for call, one in ((lambda: c.gw_iteration(G), "GW_ITERATION_GRAPH"), (lambda: c.rpa_energy(G), None)):
        for _ in range(3):
            call()
        if one:
            assert one in [n for n, _ in c.timings()]
        for _ in range(2):
            call()
            assert "EVALUATE_PI_R" in [n for n, _ in c.timings()]
    c.close()
