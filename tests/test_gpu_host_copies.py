"""Large ordinary (pageable) host arrays, which cross the bus through the threaded staging copies,
give the same bytes as page-locked ones: a size that is no multiple of the staging piece, two
contexts driven from two threads at once, and a context created after the last one was closed."""
import ctypes
import threading

import numpy as np
import pytest

from coqui_b200 import capi
from coqui_b200.iaft import IAFT
from coqui_b200.synthetic import make_system

pytestmark = pytest.mark.gpu


def _context(s, ft):
    c = capi.Context(s.nk, s.nb, s.Np, ft.nt_f, ft.nw_b, s.kp_grid, mode=capi.MIXED)
    c.set_ir(ft)
    c.set_kmesh(s.kpts, s.lattv, s.chi_bar)
    c.set_thc(s.X, s.V)
    return c


@pytest.mark.parametrize("nb", [39, 53])  # 9.3 MB (just above the threaded form's limit), 17.3 MB
def test_pageable_arrays_match_page_locked_ones(nb):
    import torch
    ft = IAFT(1000.0, 10.0, "low")
    s = make_system(2, nb, nb // 2, 64, seed=nb)
    G = s.G0(ft)
    assert G.nbytes > 8 << 20 and G.nbytes % (1 << 20) != 0
    pin = torch.empty(G.shape, dtype=torch.complex128, pin_memory=True).numpy()
    out = torch.empty(G.shape, dtype=torch.complex128, pin_memory=True).numpy()
    pin[...] = G
    got, errors = {}, []

    def user(i):
        try:
            c = _context(s, ft)
            got[i] = [c.gw_iteration(G)[0] for _ in range(3)]
            c.close()
        except Exception as e:  # reported by the main thread
            errors.append(e)

    for _ in range(2):  # the second round starts after the last context was closed
        th = [threading.Thread(target=user, args=(i,)) for i in range(2)]
        [t.start() for t in th]
        [t.join() for t in th]
        assert not errors, errors
    c = _context(s, ft)
    c.gw_iteration(pin, sigma_out=out)
    for runs in got.values():
        for S in runs:
            assert np.array_equal(S, out)
    c.close()


@pytest.mark.parametrize("managed", [False, True])
def test_arrays_in_device_or_managed_memory_are_left_to_the_driver(managed):
    """The threaded copies read and write host memory themselves: they take ordinary host arrays
    only.  A pointer to device or managed memory goes to the driver's copy, which resolves it."""
    import torch
    ft = IAFT(1000.0, 10.0, "low")
    s = make_system(2, 53, 26, 64, seed=5)
    G = np.ascontiguousarray(s.G0(ft))
    assert G.nbytes > 16 << 20
    c = _context(s, ft)
    ref = c.gw_iteration(G)[0]
    if managed:
        rt = ctypes.CDLL("libcudart.so.12")
        addr = []
        for _ in range(2):
            p = ctypes.c_void_p()
            assert rt.cudaMallocManaged(ctypes.byref(p), ctypes.c_size_t(G.nbytes), 1) == 0
            addr.append(p.value)
        g, out = (np.ctypeslib.as_array((ctypes.c_double * (2 * G.size)).from_address(a))
                  for a in addr)
        g[...] = G.reshape(-1).view(np.float64)
        out[...] = 0
    else:
        g = torch.from_numpy(G).cuda()
        out = torch.zeros_like(g)
        addr = [g.data_ptr(), out.data_ptr()]
    torch.cuda.synchronize()
    for _ in range(3):
        rc = c.lib.coqui_b200_gw_iteration(c.h, addr[0], addr[1], None)
        assert rc == 0, c.lib.coqui_b200_last_error(c.h)
    got = out.view(np.complex128).reshape(G.shape) if managed else out.cpu().numpy()
    assert np.array_equal(got, ref)
    c.close()
    if managed:
        for a in addr:
            rt.cudaFree(ctypes.c_void_p(a))
