"""Performance cases: the calls a user of this package makes, over the sizes they are made at.

Every case goes through a public entry point of ``coqui_b200.capi`` with host arrays in and
host arrays out, as a host program with an ``MBState`` holds them.  ``kind`` names the call:

* ``gw``     one GW iteration (``Context.gw_iteration``: screened interaction + self-energy);
* ``rpa``    the RPA correlation energy (``Context.rpa_energy``);
* ``hf``     THC Hartree-Fock of a density matrix (``Context.hf_evaluate``, FP64);
* ``scgw``   two iterations of the self-consistent loop with Hartree-Fock and damping;
* ``ibz``    a GW iteration on the symmetry-reduced k-points (time reversal);
* ``batch``  a GW iteration of an uneven batch of Gamma-only molecules (``Batch``);
* ``mlp``    loss and gradient of the learned update's network (``Mlp.gradient``).

``mode`` is the context's precision (mixed or fp64), ``host`` whether the host arrays are
page-locked or ordinary numpy arrays.  Inputs are seeded and synthetic with the distributions
of ``coqui_b200.synthetic`` (X ~ CN(0, 1)/sqrt(Np), V = Z Z^H + 1e-3 I, orbital energies on
[-1, -0.1] and [0.1, 1]), the Green's function in a random unitary basis per k-point, so that
it is a full Hermitian matrix as in a self-consistent loop.
"""
import math
import random

import numpy as np
import torch

from coqui_b200 import capi
from coqui_b200.iaft import IAFT
from coqui_b200.symmetry import bz_symmetry


def _case(name, kind, grid=(1, 1, 1), nb=0, np_=0, beta=1000.0, lam=1e4, mode="mixed",
          host="pinned", div="ignore_g0", count=0):
    return {"name": name, "kind": kind, "n0": grid[0], "n1": grid[1], "n2": grid[2], "nb": nb,
            "np": np_, "beta": float(beta), "lam": float(lam), "mode": mode, "host": host,
            "div": div, "count": count}


def listed():
    return [
        # the smallest system of the benchmark: a quick RPA energy from plain numpy arrays,
        # where launches and host latency count
        _case("rpa_k222_nb16_np128", "rpa", (2, 2, 2), 16, 128, host="numpy"),
        # the same small system's GW iteration, also from plain numpy arrays
        _case("gw_k222_nb16_np128", "gw", (2, 2, 2), 16, 128, host="numpy"),
        # an ordinary G0W0 step with page-locked buffers
        _case("gw_k444_nb64_np512", "gw", (4, 4, 4), 64, 512),
        # RPA energy on a dense k-mesh of many small Dyson problems
        _case("rpa_k666_nb48_np384", "rpa", (6, 6, 6), 48, 384),
        # the largest matrices: 96 orbitals, 1024 interpolating points
        _case("gw_k333_nb96_np1024", "gw", (3, 3, 3), 96, 1024),
        # the FP64 form, chosen for tight convergence and quasiparticle continuation
        _case("gw_fp64_k333_nb48_np384", "gw", (3, 3, 3), 48, 384, mode="fp64"),
        # a non-cubic mesh with odd, ragged sizes and the gygi treatment with the dielectric
        # head, from plain numpy arrays
        _case("gw_gygi_k532_nb37_np203", "gw", (5, 3, 2), 37, 203, host="numpy", div="gygi"),
        # twelve molecules of uneven size in one call
        _case("batch12_nb30_150", "batch", nb=150, beta=500.0, count=12),
        # static Fock matrix of a density matrix
        _case("hf_k444_nb64_np512", "hf", (4, 4, 4), 64, 512, host="numpy", div="gygi"),
        # self-consistent loop with Hartree-Fock: two damped iterations from G0
        _case("scgw_k333_nb48_np384", "scgw", (3, 3, 3), 48, 384, host="numpy", div="gygi"),
        # time-reversal symmetric system on its irreducible k-points
        _case("ibz_k444_nb48_np384", "ibz", (4, 4, 4), 48, 384, host="numpy"),
        # training the learned update: loss and gradient of a large sample (forward, backward)
        _case("mlp_gradient_65536", "mlp", count=65536, host="numpy"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    top = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["gw", "gw", "gw", "rpa", "rpa", "hf", "scgw", "ibz", "batch", "mlp"])
        host = rng.choice(["pinned", "numpy"])
        if kind == "mlp":
            c = _case("", kind, count=_log_int(rng, 1000, 100000), host="numpy")
        elif kind == "batch":
            c = _case("", kind, nb=rng.randint(50, 180), beta=500.0, count=rng.randint(3, 14))
        else:
            grid = (rng.randint(1, 6), rng.randint(1, 6), rng.randint(1, 6))
            if kind == "ibz":
                grid = tuple(max(2, g) for g in grid)
            nb = _log_int(rng, 8, 96)
            np_ = min(1024, max(nb, int(nb * rng.uniform(4.0, 11.0))))
            mode = "fp64" if kind in ("gw", "rpa") and rng.random() < 0.3 else "mixed"
            div = rng.choice(["ignore_g0", "gygi"]) if kind in ("gw", "hf", "scgw") else "ignore_g0"
            if div == "gygi" and kind == "gw" and grid == (1, 1, 1):
                div = "ignore_g0"
            lam = rng.choice([1e3, 1e4])
            c = _case("", kind, grid, nb, np_, 100.0 if lam == 1e3 else 1000.0, lam, mode,
                      host if kind in ("gw", "rpa") else "numpy", div)
        if _cost(c) <= top:
            c.pop("name")
            return c


# ----------------------------------------------------------------------------------------
# sizes and work
# ----------------------------------------------------------------------------------------
def _grid(c):
    return (c["n0"], c["n1"], c["n2"])


def _nk(c):
    return c["n0"] * c["n1"] * c["n2"]


def _ft(c):
    return IAFT(c["beta"], c["lam"] / c["beta"], "low")


def _molecules(c):
    """Orbitals of each molecule: uneven, between 30 and c["nb"]; Np = 6 nb."""
    r = random.Random(1000 * c["count"] + c["nb"])
    return [r.randint(min(30, c["nb"]), c["nb"]) for _ in range(c["count"])]


def _pieces(c):
    """[(k-points, orbitals, points)] of the systems of a case."""
    if c["kind"] == "batch":
        return [(1, n, 6 * n) for n in _molecules(c)]
    return [(_nk(c), c["nb"], c["np"])]


def work(case):
    c = case
    if c["kind"] == "mlp":
        n, w = c["count"], 256
        per = 4 * w + w * w + 2 * w
        # forward, and backward through the weights (all layers) and the activations
        return {"bytes": 4.0 * (6 * n + 2 * (per + 2 * w + 2)),
                "flops": 2.0 * n * (2 * per + w * w + 2 * w)}
    ft = _ft(c) if c["kind"] != "hf" else None
    nbytes = flops = 0.0
    for nk, nb, Np in _pieces(c):
        nq = (nk + _self_conjugate(_grid(c))) // 2 if c["kind"] == "ibz" else nk
        x, v, g = nk * Np * nb, nk * Np * Np, nq * nb * nb
        p2a = nb * nb * Np + Np * Np * nb  # complex multiply-adds of X G X^H at one k
        if c["kind"] == "hf":
            nbytes += 16.0 * (x + v + 3 * g)
            flops += 8.0 * nk * 2 * p2a
            continue
        nt, nwh = ft.nt_f, ft.nw_half
        nbytes += 16.0 * (x + v + nt * g)
        macs = nt * nk * p2a  # projections of G
        macs += nwh * nq * Np ** 3 * (1 / 2 + 1 / 6)  # M = L^H Pi L and the factorisation
        if c["kind"] != "rpa":
            macs += nwh * nq * Np ** 3 * (1 / 6 + 2 / 3)  # inverse and W
            macs += nt * nk * p2a  # back-projection
            nbytes += 16.0 * nt * g
        if c["kind"] == "scgw":
            macs = 2 * (macs + 2 * nk * p2a + ft.nw_f * nk * nb ** 3)
        flops += 8.0 * macs
    return {"bytes": nbytes, "flops": flops}


def _self_conjugate(grid):
    return math.prod(2 if g % 2 == 0 else 1 for g in grid)


def _cost(c):
    return work(c)["flops"] * (3.5 if c["mode"] == "fp64" or c["kind"] == "hf" else 1.0)


def tolerance(case):
    """About four times the distance from ``exact`` that the largest sizes show: the mixed form's
    products carry 22 bits per operand and accumulate in FP32 in tensor memory, whose rounding
    towards zero adds up along K and in the products that follow (8.6e-5 of Sigma and 2.6e-5 of
    E_c at the largest listed sizes); the network's sums over the sample are FP32 (2.8e-6)."""
    if case["kind"] == "mlp":
        return {"rel": 1.2e-5}
    if case["mode"] == "fp64" or case["kind"] == "hf":
        return {"rel": 1e-12}  # FP64 throughout (1.3e-13 at the largest sizes)
    if case["kind"] == "rpa":
        return {"rel": 1e-4}
    return {"rel": 3.5e-4}


# ----------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------
def _cn(gen, shape, scale):
    return torch.randn(shape, dtype=torch.complex128, device="cuda", generator=gen) * scale


def _unitary(a):
    return torch.linalg.qr(a)[0]


def _green(eps, C, ft):
    """G(tau) (nt, nk, nb, nb) of orbital energies eps (nk, nb) with coefficients C."""
    tau = torch.from_numpy(ft.tau_mesh()).cuda()[:, None, None]
    x = eps[None]
    pos = x > 0
    xp, xn = torch.where(pos, x, 0.0), torch.where(pos, 0.0, x)
    g = torch.where(pos, -torch.exp(-xp * tau) / (1.0 + torch.exp(-xp * ft.beta)),
                    -torch.exp(xn * (ft.beta - tau)) / (1.0 + torch.exp(xn * ft.beta)))
    G = torch.empty((len(ft.tau_mesh()),) + C.shape, dtype=torch.complex128, device="cuda")
    for t in range(G.shape[0]):
        G[t] = (C * g[t][:, None, :]) @ C.mH
    return 0.5 * (G + G.mH)


def _system(gen, nk, nb, Np, ft):
    """Seeded inputs of one system without symmetry, on the device."""
    X = _cn(gen, (nk, Np, nb), 1.0 / math.sqrt(Np))
    Z = _cn(gen, (nk, Np, Np), 1.0 / math.sqrt(Np))
    V = Z @ Z.mH
    V = 0.5 * (V + V.mH) + 1e-3 * torch.eye(Np, dtype=V.dtype, device="cuda")
    del Z
    nocc = max(1, nb // 2)
    e = torch.rand((nk, nb), dtype=torch.float64, device="cuda", generator=gen) * 0.9 + 0.1
    e[:, :nocc] *= -1.0
    C = _unitary(_cn(gen, (nk, nb, nb), 1.0))
    chi = _cn(gen, (nk, Np), 1.0 / math.sqrt(Np))
    d = {"X": X, "V": V, "eps": e, "C": C, "chi": chi}
    if ft is not None:
        d["G"] = _green(e, C, ft)
    return d


def _kpts(grid):
    idx = np.stack(np.meshgrid(*[np.arange(g) / g for g in grid], indexing="ij"), -1)
    return 2.0 * np.pi * idx.reshape(-1, 3)


def _symmetric(gen, c, ft):
    """A time-reversal symmetric system: X(-k), H(-k), V(-q) are the complex conjugates."""
    sym = bz_symmetry(_grid(c), [np.eye(3, dtype=int)], True)
    nk, ni, lex = sym["nk"], sym["nk_ibz"], torch.from_numpy(sym["lex"])
    src = torch.from_numpy(sym["kp_to_ibz"].astype(np.int64)).cuda()
    trev = torch.from_numpy(np.asarray(sym["kp_trev"], bool)).cuda()
    kc = np.asarray(sym["kc"])[:ni]
    real = torch.from_numpy(np.all((2 * kc) % np.array(_grid(c)) == 0, axis=1)).cuda()
    nb, Np = c["nb"], c["np"]

    def own(a):  # real at k = -k
        m = real.reshape((-1,) + (1,) * (a.dim() - 1))
        return torch.where(m, a.real.to(a.dtype), a)

    X = own(_cn(gen, (ni, Np, nb), 1.0 / math.sqrt(Np)))
    Z = own(_cn(gen, (ni, Np, Np), 1.0 / math.sqrt(Np)))
    V = Z @ Z.mH
    V = 0.5 * (V + V.mH) + 0.05 * torch.eye(Np, dtype=V.dtype, device="cuda")
    del Z
    C = _unitary(own(_cn(gen, (ni, nb, nb), 1.0)))
    e = torch.rand((ni, nb), dtype=torch.float64, device="cuda", generator=gen) * 0.9 + 0.1
    e[:, :max(1, nb // 2)] *= -1.0
    G = _green(e, C, ft)  # on the irreducible k-points

    def unfold(a, axis):
        b = a.index_select(axis, src)
        shape = [1] * b.dim()
        shape[axis] = nk
        b = torch.where(trev.reshape(shape), b.conj(), b)
        out = torch.empty_like(b)
        out[(slice(None),) * axis + (lex.cuda(),)] = b
        return out

    return {"X": unfold(X, 0), "V": unfold(V, 0), "G": G, "G_full": unfold(G, 1), "sym": sym}


def _hf_dm(d):
    """Density matrix of the occupied orbitals of a system."""
    C = d["C"] * (d["eps"] < 0)[:, None, :]
    Dm = C @ d["C"].mH
    return 0.5 * (Dm + Dm.mH)


def _mlp_inputs(case, seed):
    r = np.random.default_rng(seed)
    n, w = case["count"], 256
    X = r.standard_normal((n, 4)).astype(np.float32)
    T = r.standard_normal((n, 2)).astype(np.float32)
    shapes = [(w, 4), (w,), (w, w), (w,), (2, w), (2,)]
    p = np.concatenate([(r.uniform(-1, 1, s) / math.sqrt(s[-1])).ravel() for s in shapes])
    return X, T, p.astype(np.float32), shapes


def _device_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    c, kind = case, case["kind"]
    if kind == "batch":
        ft = _ft(c)
        return ft, [_system(gen, nk, nb, Np, ft) for nk, nb, Np in _pieces(c)]
    if kind == "ibz":
        ft = _ft(c)
        return ft, _symmetric(gen, c, ft)
    ft = None if kind == "hf" else _ft(c)
    return ft, _system(gen, _nk(c), c["nb"], c["np"], ft)


def _host(a, host):
    """Host copy of a device tensor, page-locked or an ordinary numpy array."""
    out = torch.empty(a.shape, dtype=a.dtype, pin_memory=(host == "pinned"))
    out.copy_(a)
    return out.numpy()


MADELUNG = 0.5


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "mlp":
        X, T, p, _ = _mlp_inputs(c, seed)
        net = capi.Mlp(4, 256, 2, seed=1)
        net.set_params(p)
        return {"case": c, "net": net, "X": X, "T": T}
    ft, d = _device_inputs(c, seed)
    host = c["host"]
    s = {"case": c}
    if kind == "batch":
        b = capi.Batch([n for _, n, _ in _pieces(c)], [p for _, _, p in _pieces(c)], ft.nt_f,
                       ft.nw_b)
        b.set_ir(ft)
        for i, m in enumerate(d):
            b.set_thc(i, _host(m["X"][0], "numpy"), _host(m["V"][0], "numpy"))
        s["batch"] = b
        s["G"] = [_host(m["G"][:, 0], host) for m in d]
        s["Sigma"] = [_host(torch.zeros_like(m["G"][:, 0]), host) for m in d]
        del d
        torch.cuda.empty_cache()
        return s
    grid, nk = _grid(c), _nk(c)
    nt, nwb = (2, 1) if ft is None else (ft.nt_f, ft.nw_b)
    mode = capi.FP64 if c["mode"] == "fp64" else capi.MIXED
    ctx = capi.Context(nk, c["nb"], c["np"], nt, nwb, grid, mode=mode)
    if ft is not None:
        ctx.set_ir(ft)
    chi = None if "chi" not in d else _host(d["chi"], "numpy")
    ctx.set_kmesh(_kpts(grid), np.eye(3), chi)
    ctx.set_thc(_host(d["X"], "numpy")[None], _host(d["V"], "numpy"))
    s["ctx"] = ctx
    eye = np.ascontiguousarray(np.broadcast_to(np.eye(c["nb"], dtype=np.complex128),
                                               (1, nk, c["nb"], c["nb"])))
    if kind == "hf":
        s["Dm"], s["S"] = _host(_hf_dm(d), host)[None], eye
    elif kind == "scgw":
        ctx.set_ir_fermi(ft)
        H0 = (d["C"] * d["eps"][:, None, :]) @ d["C"].mH
        ctx.set_mean_field(_host(0.5 * (H0 + H0.mH), "numpy")[None], eye, np.zeros_like(eye), 0.0)
        ctx.set_iter_alg("damping", 0.7)
        ctx.set_hf(True, c["div"], MADELUNG)
        s["G"] = _host(d["G"], host)[:, None]
    else:
        if kind == "ibz":
            ctx.set_symmetry(d["sym"])
        if kind == "gw" and c["div"] != "ignore_g0":
            ctx.set_div_treatment(c["div"], MADELUNG, chi[0])
        s["G"] = _host(d["G"], host)[:, None]
        if kind == "gw" and host == "pinned":
            s["Sigma"] = _host(torch.zeros_like(d["G"]), host)[:, None]
    del d
    torch.cuda.empty_cache()
    return s


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "mlp":
        loss, g = state["net"].gradient(state["X"], state["T"])
        return {"loss": float(loss), "gradient": g}
    if kind == "batch":
        return state["batch"].gw_iteration(state["G"], state["Sigma"])
    ctx = state["ctx"]
    if kind == "rpa":
        return ctx.rpa_energy(state["G"])
    if kind == "hf":
        return ctx.hf_evaluate(state["Dm"], state["S"], True, True, c["div"], MADELUNG)
    if kind == "scgw":
        ctx.scgw_iteration(1, state["G"])
        e = ctx.scgw_iteration(2)
        G, S, Dm = ctx.get_scgw_state()
        return {"G": G, "Sigma": S, "Dm": Dm, "e_1e": e["e_1e"], "e_hf": e["e_hf"],
                "e_corr": e["e_corr"]}
    if c["div"] != "ignore_g0":
        S, head = ctx.gw_iteration(state["G"], sigma_out=state.get("Sigma"), want_head=True)
        return {"Sigma": S, "head": head}
    return ctx.gw_iteration(state["G"], sigma_out=state.get("Sigma"))[0]


# ----------------------------------------------------------------------------------------
# the same quantities in 64 bits
# ----------------------------------------------------------------------------------------
def _to_R(a, grid):
    """sum_k exp(-i k R) / nk over the leading k axis of (nk, ...)."""
    b = a.reshape(grid + a.shape[1:])
    return torch.fft.fftn(b, dim=(0, 1, 2), norm="forward").reshape(a.shape)


def _to_k(a, grid):
    b = a.reshape(grid + a.shape[1:])
    return torch.fft.ifftn(b, dim=(0, 1, 2), norm="forward").reshape(a.shape)


def _half(T, n_in_half, n_out_half, nt, nwb, to_w):
    """Particle-hole symmetric transform on the half grids."""
    T = torch.from_numpy(np.ascontiguousarray(T)).cuda()
    if to_w:
        rows = T[nwb // 2 + torch.arange(n_out_half)]
        out = rows[:, :n_in_half].clone()
        for it in range(n_in_half):
            if nt - 1 - it != it:
                out[:, it] += rows[:, nt - 1 - it]
        return out
    rows = T[:n_out_half]
    out = rows[:, nwb // 2 + torch.arange(n_in_half)].clone()
    for n in range(1, n_in_half):
        out[:, n] += rows[:, nwb // 2 - n]
    return out


def _p2a(X, O):
    return X @ O @ X.mH


def _pi_w(G, X, grid, ft):
    nt, nth = ft.nt_f, ft.nt_half
    nk, Np = X.shape[0], X.shape[1]
    Pi = torch.empty((nth, nk, Np, Np), dtype=torch.complex128, device="cuda")
    for t in range(nth):
        a, b = _to_R(_p2a(X, G[t]), grid), _to_R(_p2a(X, G[nt - 1 - t]), grid)
        Pi[t] = _to_k(-2.0 * a * b.conj(), grid)
    T = _half(ft.Twt_bb, nth, ft.nw_half, nt, ft.nw_b, True)
    out = torch.empty((ft.nw_half, nk, Np, Np), dtype=torch.complex128, device="cuda")
    for q in range(nk):
        out[:, q] = torch.tensordot(T, Pi[:, q], 1)
    return out


def _sigma(G, X, V, grid, ft):
    """(Sigma(tau), W(tau, q)) of one GW iteration."""
    nt, nth, nwh = ft.nt_f, ft.nt_half, ft.nw_half
    W = _pi_w(G, X, grid, ft)
    nk, Np = X.shape[0], X.shape[1]
    eye = torch.eye(Np, dtype=torch.complex128, device="cuda")
    T = _half(ft.Ttw_bb, nwh, nth, nt, ft.nw_b, False)
    Wt = torch.empty((nth, nk, Np, Np), dtype=torch.complex128, device="cuda")
    for q in range(nk):
        A = eye - V[q] @ W[:, q]
        # ([I - V Pi]^{-1} - I) V = [I - V Pi]^{-1} V Pi V
        Wt[:, q] = torch.tensordot(T, torch.linalg.solve(A, (V[q] @ W[:, q]) @ V[q]), 1)
    del W
    S = torch.zeros_like(G)
    for t in range(nth):
        WR = _to_R(Wt[t], grid)
        for u in ([t] if nt - 1 - t == t else [t, nt - 1 - t]):
            P = _to_k(-_to_R(_p2a(X, G[u]), grid) * WR, grid)
            S[u] = X.mH @ P @ X
    return S, Wt


def _hf(Dm, X, V, grid, div):
    D = _to_R(_p2a(X, Dm), grid)
    rho = 2.0 * torch.diagonal(D[0])
    K = _to_k(-D * _to_R(V, grid), grid)
    K = K + torch.diag(V[0] @ rho)
    F = X.mH @ K @ X
    return F - MADELUNG * Dm if div == "gygi" else F


def _herm(a):
    return 0.5 * (a + a.mH)


def _beta(ft, A):
    return torch.tensordot(torch.from_numpy(ft.T_beta_t_ff).cuda().to(A.dtype), A, 1)


def _corr_energy(G, S, ft):
    Twt, Ttw = torch.from_numpy(ft.Twt_ff).cuda(), torch.from_numpy(ft.Ttw_ff).cuda()
    Sw, Gw = torch.tensordot(Twt, S, 1), torch.tensordot(Twt, G, 1)
    e = torch.einsum("wkij,wkji->w", Sw, Gw) / G.shape[1]
    return float((-_beta(ft, Ttw @ e)).real)


def _scgw(c, ft, d):
    X, V, grid = d["X"], d["V"], _grid(c)
    H0 = _herm((d["C"] * d["eps"][:, None, :]) @ d["C"].mH)
    eye = torch.eye(c["nb"], dtype=torch.complex128, device="cuda")
    Twt, Ttw = torch.from_numpy(ft.Twt_ff).cuda(), torch.from_numpy(ft.Ttw_ff).cuda()
    wn = torch.from_numpy(np.asarray(ft.wn_mesh_f, np.float64)).cuda() * (math.pi / ft.beta)
    G = d["G"]
    Dm = _herm(-_beta(ft, G))
    F0 = S0 = None
    for it in (1, 2):
        F = _herm(_hf(Dm, X, V, grid, c["div"]))
        S = _herm(_sigma(G, X, V, grid, ft)[0])
        if it == 2:
            F, S = 0.7 * F + 0.3 * F0, 0.7 * S + 0.3 * S0
        A = (1j * wn)[:, None, None, None] * eye - H0 - F - torch.tensordot(Twt, S, 1)
        G = torch.tensordot(Ttw, torch.linalg.inv(A), 1)
        Dm, G = _herm(-_beta(ft, G)), _herm(G)
        F0, S0 = F, S
    nk = X.shape[0]
    e1 = 2.0 * float(torch.einsum("kij,kji->", Dm, H0).real) / nk
    eh = float(torch.einsum("kij,kji->", Dm, F).real) / nk
    return {"G": G[:, None].cpu().numpy(), "Sigma": S[:, None].cpu().numpy(),
            "Dm": Dm[None].cpu().numpy(), "e_1e": e1, "e_hf": eh, "e_corr": _corr_energy(G, S, ft)}


def _mlp_exact(case, seed):
    X, T, p, shapes = _mlp_inputs(case, seed)
    w, o = [], 0
    for s in shapes:
        n = int(np.prod(s))
        # the network runs with its parameters rounded to bfloat16
        w.append(torch.from_numpy(p[o:o + n].reshape(s)).bfloat16().double())
        o += n
    W1, b1, W2, b2, W3, b3 = w
    X, T = torch.from_numpy(X).double(), torch.from_numpy(T).double()
    h1 = torch.tanh(X @ W1.T + b1)
    h2 = torch.tanh(h1 @ W2.T + b2)
    Y = h2 @ W3.T + b3
    dY = 2.0 * (Y - T) / Y.numel()
    z2 = (dY @ W3) * (1.0 - h2 * h2)
    z1 = (z2 @ W2) * (1.0 - h1 * h1)
    g = [z1.T @ X, z1.sum(0), z2.T @ h1, z2.sum(0), dY.T @ h2, dY.sum(0)]
    return {"loss": float(((Y - T) ** 2).mean()),
            "gradient": torch.cat([a.reshape(-1) for a in g]).numpy()}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "mlp":
        return _mlp_exact(c, seed)
    ft, d = _device_inputs(c, seed)
    if kind == "batch":
        return [_sigma(m["G"], m["X"], m["V"], (1, 1, 1), ft)[0][:, 0].cpu().numpy() for m in d]
    grid, X, V = _grid(c), d["X"], d["V"]
    if kind == "hf":
        return _hf(_hf_dm(d), X, V, grid, c["div"])[None].cpu().numpy()
    if kind == "scgw":
        return _scgw(c, ft, d)
    if kind == "rpa":
        P = _pi_w(d["G"], X, grid, ft)
        eye = torch.eye(c["np"], dtype=torch.complex128, device="cuda")
        e = torch.zeros(ft.nw_b, dtype=torch.complex128, device="cuda")
        for n in range(ft.nw_half):
            A = P[n] @ V
            v = (torch.diagonal(A, dim1=1, dim2=2).sum() + torch.linalg.slogdet(eye - A)[1].sum())
            e[ft.nw_b // 2 + n] += v
            if n:
                e[ft.nw_b // 2 - n] += v
        et = torch.from_numpy(ft.Ttw_bb).cuda() @ e
        return float(_beta(ft, et).real) / (2.0 * X.shape[0])
    if kind == "ibz":
        S, _ = _sigma(d["G_full"], X, V, grid, ft)
        k = torch.from_numpy(d["sym"]["lex"][:d["sym"]["nk_ibz"]]).cuda()
        return S[:, k][:, None].cpu().numpy()
    S, W = _sigma(d["G"], X, V, grid, ft)
    if c["div"] == "ignore_g0":
        return S[:, None].cpu().numpy()
    # the dielectric head at the first smallest nonzero |q|, and its correction of Sigma
    q2 = (_kpts(grid) ** 2).sum(1)
    q = int(np.argmin(np.where(q2 > 0, q2, np.inf)))
    chi = d["chi"]
    head = torch.einsum("P,tPQ,Q->t", chi[q], W[:, q], chi[q].conj()) * float(q2[q] / (4.0 * np.pi))
    T = X.mH @ (chi[0].conj()[:, None] * X)
    for t in range(ft.nt_f):
        f = -MADELUNG * head[min(t, ft.nt_f - 1 - t)].real
        S[t] += f * (T @ d["G"][t] @ T.mH)
    return {"Sigma": S[:, None].cpu().numpy(), "head": head.cpu().numpy()}
