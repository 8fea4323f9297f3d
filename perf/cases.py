"""What the speed of this framework is measured on.

The listed cases are the calls that a self-consistency code makes every iteration, through the public
entry points (gb200.lib.Context, gb200.solvers, gb200.autograd and the batched call), from the smallest
system of the configurations to one that fills the GPU for about a second, in both contraction
precisions, with one and two spins, two-component input, odd sizes, forward and backward.  Inputs
follow the recipe of gb200.synth (Haar-random orbitals, Fermi-function Green's functions, complex
Gaussian integrals) and are made from the seed alone.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "green-mbpt_b200")
for _p in (os.path.join(os.getcwd(), "green-mbpt_b200"), _PKG):
    if os.path.isdir(_p) and _p not in sys.path:
        sys.path.insert(0, _p)
        break

from gb200 import autograd, grids, lib, solvers  # noqa: E402

C = torch.complex128


# --------------------------------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------------------------------
def _case(name, kind, mesh, nao, naux, nts, beta, ns=1, eps=2.0, slices=0, x2c=False, q0=False, madelung=0.0):
    """slices = 0: FP64 contractions, else split precision with that many slices."""
    return {"name": name, "kind": kind, "n1": mesh[0], "n2": mesh[1], "n3": mesh[2], "nao": nao, "naux": naux,
            "nts": nts, "beta": beta, "ns": ns, "eps": eps, "slices": slices, "x2c": x2c, "q0": q0,
            "madelung": madelung}


def listed():
    return [
        # the smallest configuration: one FP64 self-energy of a 2x2x2 mesh, bound by launches
        _case("gw_fp64_small", "gw", (2, 2, 2), 10, 40, 60, 100.0),
        # a small two-spin solid of odd sizes with the q -> 0 correction, at the default slice count
        _case("gw_split_odd", "gw", (3, 2, 1), 13, 57, 34, 50.0, ns=2, slices=4, q0=True),
        # the mid-size spin-polarised configuration's orbital, auxiliary and time shapes, FP64
        _case("gw_fp64_spin", "gw", (2, 2, 2), 26, 150, 100, 100.0, ns=2),
        # the headline workload's shapes in split precision, on a mesh of 8 and of 18 k-points
        _case("gw_split_mid", "gw", (2, 2, 2), 40, 250, 120, 200.0, eps=5.0, slices=5),
        _case("gw_split_large", "gw", (3, 3, 2), 40, 250, 120, 200.0, eps=5.0, slices=5),
        # relativistic (two-component) input, one slice more than usual
        _case("gw_split_x2c", "gw", (2, 2, 1), 18, 90, 80, 100.0, slices=6, x2c=True),
        # the Fock build at the headline workload's orbital and auxiliary sizes
        _case("hf_large", "hf", (3, 3, 3), 40, 250, 20, 100.0, madelung=0.4),
        # the Dyson step with the chemical-potential search at the headline workload's full size
        _case("dyson_large", "dyson", (5, 5, 5), 40, 1, 120, 200.0, eps=5.0),
        # gradient of a functional of the self-energy with respect to G and the integrals
        _case("grad_mid", "grad", (2, 2, 2), 20, 100, 80, 100.0),
        # many uneven systems in one call: "nao" and "naux" are the largest of them
        _case("batch_uneven", "batch", (3, 3, 3), 46, 220, 80, 100.0, slices=5),
        # one whole self-consistency iteration on device buffers, the headline workload's step
        _case("iteration_split", "iteration", (2, 2, 1), 40, 250, 120, 200.0, eps=5.0, slices=5),
        # one iteration of a small two-spin system through the host solvers (the drop-in interface)
        _case("scf_host_small", "scf_host", (2, 2, 1), 11, 45, 44, 50.0, ns=2, madelung=0.3),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


_MESHES = [(1, 1, 1), (2, 1, 1), (3, 1, 1), (2, 2, 1), (5, 1, 1), (3, 2, 1), (2, 2, 2), (3, 3, 1), (3, 2, 2), (3, 3, 2),
           (3, 3, 3)]


def draw(rng):
    limit = work(listed()[4])["flops"] * 0.5
    while True:
        kind = rng.choice(["gw", "gw", "gw", "gw", "hf", "dyson", "grad", "iteration", "scf_host"])
        mesh = rng.choice(_MESHES if kind in ("gw", "hf", "dyson") else _MESHES[:7])
        x2c = kind == "gw" and rng.random() < 0.2
        nao = _log_int(rng, 5, 30 if x2c else 46)
        naux = int(round(nao * rng.uniform(3.0, 6.0)))
        slices = rng.choice([0, 0, 4, 5, 5, 5, 6]) if kind in ("gw", "iteration") else 0
        beta, eps = rng.choice([20.0, 50.0, 100.0, 200.0]), rng.choice([2.0, 5.0])
        nts = 2 * max(_log_int(rng, 10, 60), math.ceil(1.9 * math.sqrt(beta * eps)))  # the time grid resolves exp(-eps tau)
        c = _case("", kind, mesh, nao, naux, min(nts, 120), beta, ns=1 if x2c else rng.choice([1, 1, 2]), eps=eps,
                  slices=slices, x2c=x2c, q0=kind == "gw" and mesh[0] == 3 and mesh[1] > 1 and rng.random() < 0.3,
                  madelung=rng.choice([0.0, 0.5]))
        del c["name"]
        if kind in ("dyson", "iteration", "scf_host") and (_nk(c) * nao < 60 or beta > 100.0):
            continue  # too few levels for a smooth electron count
        if kind == "dyson":
            c["naux"] = 1
        cost = work(c)["flops"] * (10.0 if slices == 0 and kind not in ("hf", "dyson") else 1.0)
        vbytes = 16.0 * _nk(c) ** 2 * c["naux"] * nao ** 2
        if cost <= limit and vbytes <= 6e9:
            return c


def _nk(c):
    return c["n1"] * c["n2"] * c["n3"]


def _batch_systems(c):
    """The systems of a batch: the largest orbital count on a small mesh and smaller ones beside it."""
    big = (2, 2, 2)
    n, q = c["nao"], c["naux"]
    shapes = [((2, 2, 2), max(8, n // 5), max(32, q // 5)), (big, n // 2, q // 2 + 1),
              ((c["n1"], c["n2"], c["n3"]), max(8, n // 4 + 1), max(32, q // 4 + 5)), (big, 3 * n // 4, 2 * q // 3),
              (big, n, q)]
    return [dict(c, kind="gw", n1=m[0], n2=m[1], n3=m[2], nao=a, naux=b) for m, a, b in shapes]


# --------------------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=16)
def _grid(beta, nts):
    # (a shorter candidate list than the default picks the same frequencies in a tenth of the time)
    return grids.ChebyshevGrid(beta, nts, nts, nts, candidates=max(512, (nts - 2) ** 2 // 8))


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _haar(gen, shape):
    z = torch.randn(shape, dtype=C, generator=gen)
    q, r = torch.linalg.qr(z)
    d = torch.diagonal(r, dim1=-2, dim2=-1)
    return q * (d / d.abs()).unsqueeze(-2)


def _fermi(eps, tau, beta):
    """exp(-eps tau) / (1 + exp(-beta eps)) without overflow: eps [...], tau [nts] -> [nts, ...]"""
    t = torch.as_tensor(tau).reshape((-1,) + (1,) * eps.dim())
    p, m = eps.clamp(min=0.0), eps.clamp(max=0.0)
    return torch.where(eps >= 0, torch.exp(-p * t) / (1 + torch.exp(-beta * p)),
                       torch.exp((beta - t) * m) / (1 + torch.exp(beta * m)))


def _herm(x):
    return 0.5 * (x + x.conj().transpose(-1, -2))


def _inputs(c, seed):
    """Everything a program has of one system, as torch tensors on the GPU (complex128)."""
    gen = torch.Generator().manual_seed(int(seed) * 7919 + 13)
    dev, nk, nao, NQ, ns = _device(), _nk(c), c["nao"], c["naux"], c["ns"]
    nso = 2 * nao if c["x2c"] else nao
    g = _grid(c["beta"], c["nts"])
    eps = (torch.rand((ns, nk, nso), dtype=torch.float64, generator=gen) * 2 - 1) * c["eps"]
    U = _haar(gen, (ns, nk, nso, nso)).to(dev)
    f = _fermi(eps, g.tau, c["beta"]).to(dev)
    eps = eps.to(dev)
    H = _herm((U * eps.unsqueeze(-2)) @ U.conj().transpose(-1, -2))
    G = -(U * f.unsqueeze(-2)) @ U.conj().transpose(-1, -2)
    S = torch.eye(nso, dtype=C).expand(ns, nk, nso, nso).clone()
    if not c["x2c"]:
        S = S + 0.05 * _herm(torch.randn((ns, nk, nso, nso), dtype=C, generator=gen)) / math.sqrt(nso)
    d = {"grid": g, "G": G.contiguous(), "H": H.contiguous(), "S": S.to(dev).contiguous(), "madelung": c["madelung"]}
    occ = 1.0 / (1.0 + torch.exp((c["beta"] * eps).clamp(-700, 700)))
    full = nso * ns * (2.0 if ns == 1 and not c["x2c"] else 1.0)
    d["nel"] = full * min(0.65, max(0.35, float(occ.mean())))
    if c["kind"] != "dyson":
        dgen = torch.Generator(device=dev).manual_seed(int(seed) * 104729 + 7)
        V = torch.empty((nk * (nk + 1) // 2, NQ, nao, nao), dtype=C, device=dev)
        for k1 in range(nk):
            lo = k1 * (k1 + 1) // 2
            V[lo:lo + k1 + 1] = torch.randn((k1 + 1, NQ, nao, nao), dtype=C, device=dev, generator=dgen) / math.sqrt(NQ)
            V[lo + k1] = _herm(V[lo + k1])
        d["V"] = V
    if c["q0"]:
        d["AqQ"] = torch.randn((nk, NQ), dtype=C, generator=gen).numpy() / math.sqrt(NQ)
        # |q| of the mesh points in units in which the fit's window (0, 1] holds a part of them
        i = np.arange(nk)
        fr = np.stack([i // (c["n2"] * c["n3"]) / c["n1"], i // c["n3"] % c["n2"] / c["n2"], i % c["n3"] / c["n3"]], 1)
        fr = fr - np.round(fr)
        d["q_abs"] = np.round(np.sqrt((fr ** 2 * np.array([1.0, 1.3, 1.7])).sum(1)) * 1.2, 12)
        d["madelung"] = 0.7
    if c["kind"] == "dyson":
        # a self-energy with the shape of a correlated one: negative, decaying from both ends
        e2 = (torch.rand((ns, nk, nso), dtype=torch.float64, generator=gen) * 2 - 1) * c["eps"]
        U2 = _haar(gen, (ns, nk, nso, nso)).to(dev)
        f2 = _fermi(e2, g.tau, c["beta"]).to(dev)
        d["Sigma"] = (-0.3 * (U2 * f2.unsqueeze(-2)) @ U2.conj().transpose(-1, -2)).contiguous()
        d["Sigma1"] = (0.5 * _herm(torch.randn((ns, nk, nso, nso), dtype=C, generator=gen)) / math.sqrt(nso)).to(dev)
    if c["kind"] == "grad":
        d["Sbar"] = torch.randn(G.shape, dtype=C, generator=gen).to(dev)
    return d


def _np(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _stream():
    h = torch.cuda.current_stream().cuda_stream
    return h if h else 1  # the legacy default stream's handle


def _context(c, d):
    g = d["grid"]
    ctx = lib.Context(_nk(c), c["nao"], c["ns"], c["naux"], g.nts, g.nw, g.nw_b, c["beta"],
                      nso=2 * c["nao"] if c["x2c"] else None)
    ctx.set_kq_maps(*solvers.kq_maps((c["n1"], c["n2"], c["n3"])))
    ctx.set_grid(g.Tnt_f, g.Ttn_f, g.Tnt_b, g.Ttn_b, g.wsample_f)
    if "V" in d:
        torch.cuda.synchronize()
        ctx.set_integrals_device(d["V"].data_ptr(), 0, d["V"].shape[0], stream=_stream())
    ctx.set_hamiltonian(_np(d["H"]), _np(d["S"]))
    if c["slices"]:
        ctx.set_precision(lib.PREC_SPLIT, c["slices"])
    if c["q0"]:
        ctx.set_q0_correction(d["AqQ"], d["q_abs"], d["madelung"])
    return ctx


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        parts = [prepare(b, seed * 31 + i) for i, b in enumerate(_batch_systems(case))]
        return {"kind": "batch", "parts": parts}
    d = _inputs(case, seed)
    st = {"kind": kind, "ctx": _context(case, d), "madelung": d["madelung"], "nel": d["nel"]}
    if kind == "gw":
        st["G"], st["Sigma"] = d["G"], torch.empty_like(d["G"])
    elif kind == "hf":
        st["dm"] = (-1.0 if case["ns"] == 2 else -2.0) * d["G"][-1]
        st["S"], st["F"] = d["S"], torch.empty_like(d["S"])
    elif kind == "dyson":
        st["S1_in"], st["St_in"] = d["Sigma1"], d["Sigma"]
        st["S1"], st["St"], st["G"] = d["Sigma1"].clone(), d["Sigma"].clone(), torch.empty_like(d["G"])
    elif kind == "grad":
        st["G"], st["V"], st["Sbar"] = d["G"].requires_grad_(True), d["V"].requires_grad_(True), d["Sbar"]
    elif kind == "iteration":
        st["G0"], st["G"] = d["G"], torch.empty_like(d["G"])
        st["S1"], st["Sigma"] = torch.empty_like(d["H"]), torch.empty_like(d["G"])
    elif kind == "scf_host":
        G = _np(d["G"])
        st["G0"], st["G"] = G, np.empty_like(G)
        st["S1"], st["Sigma"] = np.empty(G.shape[1:], dtype=np.complex128), np.empty_like(G)
        st["hf"] = solvers.hf_solver(st["ctx"], _np(d["S"]), d["madelung"], case["ns"])
        st["gw"] = solvers.gw_solver(st["ctx"])
    torch.cuda.synchronize()
    return st


# --------------------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "batch":
        p = state["parts"]
        lib.gw_sigma_batch_device([x["ctx"] for x in p], [x["G"].data_ptr() for x in p],
                                  [x["Sigma"].data_ptr() for x in p], _stream())
        return [x["Sigma"] for x in p]
    ctx = state["ctx"]
    if kind == "gw":
        ctx.gw_sigma_device(state["G"].data_ptr(), state["Sigma"].data_ptr(), _stream())
        return state["Sigma"]
    if kind == "hf":
        ctx.hf_fock_device(state["dm"].data_ptr(), state["S"].data_ptr(), state["madelung"], state["F"].data_ptr(),
                           _stream())
        return state["F"]
    if kind == "dyson":
        # the step hermitizes the self-energies in place, so a pass starts from the given ones
        state["S1"].copy_(state["S1_in"])
        state["St"].copy_(state["St_in"])
        mu = ctx.dyson_solve_device(state["S1"].data_ptr(), state["St"].data_ptr(), state["nel"], 1e-9, 0.0,
                                    state["G"].data_ptr(), _stream())
        return {"G": state["G"], "Sigma1": state["S1"], "Sigma": state["St"], "mu": mu}
    if kind == "grad":
        Sigma = autograd.gw_sigma(ctx, state["G"], state["V"])
        Gb, Vb = torch.autograd.grad(Sigma, (state["G"], state["V"]), state["Sbar"])
        return {"Sigma": Sigma.detach(), "G_bar": Gb, "V_bar": Vb}
    if kind == "iteration":
        state["G"].copy_(state["G0"])
        mu, e = ctx.iteration_device(state["G"].data_ptr(), state["S1"].data_ptr(), state["Sigma"].data_ptr(),
                                     state["madelung"], state["nel"], 1e-9, 0.0, _stream())
        return {"G": state["G"], "Sigma1": state["S1"], "Sigma": state["Sigma"], "mu": mu, "E": np.array(e)}
    np.copyto(state["G"], state["G0"])
    state["hf"].solve(state["G"], state["S1"], state["Sigma"])
    state["gw"].solve(state["G"], state["S1"], state["Sigma"])
    dy = solvers.dyson(ctx, state["nel"])
    dy.solve(state["G"], state["S1"], state["Sigma"])
    dy.diff(state["G"], state["S1"], state["Sigma"])
    return {"G": state["G"], "Sigma1": state["S1"], "Sigma": state["Sigma"], "mu": dy.mu, "E": np.array(dy.E)}


# --------------------------------------------------------------------------------------------------
# work and tolerance
# --------------------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "batch":
        w = [work(b) for b in _batch_systems(case)]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    nk, n, NQ, nts = _nk(case), float(case["nao"]), float(case["naux"]), float(case["nts"])
    nso = 2 * n if case["x2c"] else n
    sp = 4 if case["x2c"] else case["ns"]
    g = 16.0 * nts * case["ns"] * nk * nso ** 2
    m = g / nts
    v = 16.0 * nk * (nk + 1) / 2 * NQ * n * n
    # complex multiply-adds x 8; P0 over half the times, W V once per time pair and for all spins
    gw = 8.0 * nk * nk * (nts / 2) * (sp * (2 * n ** 3 * NQ + n * n * NQ * NQ) + n * n * NQ * NQ + 4 * sp * n ** 3 * NQ)
    gw += 8.0 * nk * (nts / 2) * NQ ** 2 * (3 * nts / 2 + 2 * NQ)
    hf = 8.0 * nk * nk * case["ns"] * 2 * n ** 3 * NQ
    dy = 8.0 * nk * case["ns"] * (2 * nts * nts * nso ** 2 + nts * nso ** 3 * 40)
    if kind == "gw":
        return {"bytes": v + 2 * g, "flops": gw}
    if kind == "hf":
        return {"bytes": v + 3 * m, "flops": hf}
    if kind == "dyson":
        return {"bytes": 3 * g + 4 * m, "flops": dy}
    if kind == "grad":
        return {"bytes": 2 * v + 4 * g, "flops": 4 * gw}
    return {"bytes": v + 4 * g + 3 * m, "flops": gw + hf + dy}


def tolerance(case):
    # four times the largest distance from the 64-bit results below that this path showed over several
    # seeds and shapes: sums in another order for FP64, the rounding of 7-bit slices otherwise
    s = case["slices"]
    if case["kind"] == "iteration" and s:
        # the chemical-potential search stops at 1e-9 of the electron count, so its last step may differ
        return {"rel": 1e-8, "max": 1e-7} if s >= 5 else {"rel": 1e-6, "max": 1e-5}
    if s:
        return {"rel": {4: 9e-8, 5: 9e-10, 6: 1.2e-11}[s], "max": {4: 8e-7, 5: 1.2e-8, 6: 2e-10}[s]}
    if case["kind"] in ("dyson", "iteration", "scf_host"):
        return {"rel": 2e-13, "max": 2e-12}  # through the inverse transforms
    return {"rel": 4e-14, "max": 4e-13}


# --------------------------------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# --------------------------------------------------------------------------------------------------
def _pair(V, k1, k2):
    if k1 >= k2:
        return V[k1 * (k1 + 1) // 2 + k2]
    return V[k2 * (k2 + 1) // 2 + k1].conj().transpose(-1, -2)


def _t(a, dev):
    return torch.as_tensor(np.asarray(a), dtype=C, device=dev)


def _exact_gw(c, d, G, V):
    dev, nk, n, NQ, nts = G.device, _nk(c), c["nao"], c["naux"], c["nts"]
    nth = nts // 2
    kp, km = solvers.kq_maps((c["n1"], c["n2"], c["n3"]))
    g = d["grid"]
    Tnt, Ttn = _t(g.Tnt_b, dev), _t(g.Ttn_b, dev)
    if c["x2c"]:
        b = [slice(0, n), slice(n, 2 * n)]
        Gs = [(G[:, 0, :, b[i], b[j]], G[:, 0, :, b[j], b[i]]) for i in (0, 1) for j in (0, 1)]
        pref = 1.0
    else:
        Gs = [(G[:, s], G[:, s]) for s in range(c["ns"])]
        pref = 1.0 if c["ns"] == 2 else 2.0
    Sig = [[0.0] * nk for _ in Gs]
    heads = np.zeros((g.nw_b, nk))
    for q in range(nk):
        P = 0.0
        for k in range(nk):
            v = _pair(V, k, int(kp[k, q]))
            vc = v.conj().reshape(NQ, n * n).T
            for Gf, Gbar in Gs:
                T1 = (v.reshape(NQ * n, n) @ Gf[:nth, int(kp[k, q])]).reshape(nth, NQ, n, n)
                Bt = Gbar[:, k].flip(0)[:nth].unsqueeze(1) @ T1
                P = P - pref * (Bt.reshape(nth, NQ, n * n) @ vc)
        P = _herm(P / nk)
        P = torch.cat([P, P.flip(0)])
        Pw = (Tnt @ P.reshape(nts, -1)).reshape(-1, NQ, NQ)
        A = torch.eye(NQ, dtype=C, device=dev) - Pw
        lo = torch.tril(A, -1)
        A = lo + lo.conj().transpose(-1, -2) + torch.diag_embed(torch.diagonal(A, dim1=-2, dim2=-1).real.to(C))
        Pt = _herm(torch.linalg.inv(A)) @ Pw
        if c["q0"]:
            a = _t(d["AqQ"][q], dev)
            heads[:, q] = (a.conj() @ (Pt @ a).T).real.cpu().numpy()
        W = (Ttn @ Pt.reshape(-1, NQ * NQ)).reshape(nts, NQ, NQ)
        for k in range(nk):
            v = _pair(V, k, int(km[k, q]))
            for s, (Gf, _) in enumerate(Gs):
                Y1 = (v.reshape(NQ * n, n) @ Gf[:, int(km[k, q])]).reshape(nts, NQ, n * n)
                Y2 = (W.transpose(-1, -2) @ Y1).reshape(nts, NQ, n, n)
                y = Y2.permute(0, 2, 1, 3).reshape(nts, n, NQ * n)
                Sig[s][k] = Sig[s][k] - y @ v.conj().permute(0, 2, 1).reshape(NQ * n, n)
    S = torch.stack([torch.stack(x, 1) for x in Sig], 1) / nk
    if c["x2c"]:
        top, bot = torch.cat([S[:, 0], S[:, 1]], -1), torch.cat([S[:, 2], S[:, 3]], -1)
        S = torch.cat([top, bot], -2).unsqueeze(1)
    if c["q0"]:
        # quadratic fit of the heads over the distinct |q| in (0, 1], taken to q = 0
        q_abs, first = np.unique(d["q_abs"], return_index=True)
        keep = (q_abs > 0) & (q_abs <= 1.0)
        A = np.vander(q_abs[keep], 3, increasing=True)
        e0 = np.linalg.lstsq(A, heads[:, first[keep]].T, rcond=None)[0][0]
        coef = (-d["madelung"] * (Ttn @ _t(e0, dev))).reshape(nts, 1, 1, 1, 1)
        ov = d["S"]
        if c["x2c"]:
            ov = torch.zeros_like(ov)
            ov[..., :n, :n] = ov[..., n:, n:] = d["S"][..., :n, :n]
        D = coef * (ov @ G @ ov)
        if c["x2c"]:
            D[..., n:, :n] = D[..., :n, n:].conj().transpose(-1, -2)
        S = S + D
    return S


def _exact_hf(c, d, dm):
    nk, n, NQ, ns, V = _nk(c), c["nao"], c["naux"], c["ns"], d["V"]
    pref = 1.0 if ns == 2 else 0.5
    F = torch.zeros_like(dm)
    u = sum(torch.einsum("qab,sba->q", _pair(V, k, k), dm[:, k]) for k in range(nk)) / nk
    for k in range(nk):
        F[:, k] += torch.einsum("q,qij->ij", u, _pair(V, k, k))
        for kp in range(nk):
            v = _pair(V, k, kp)
            vc = v.conj().permute(0, 2, 1).reshape(NQ * n, n)
            for s in range(ns):
                y = (v.reshape(NQ * n, n) @ dm[s, kp]).reshape(NQ, n, n).permute(1, 0, 2).reshape(n, NQ * n)
                F[s, k] -= (pref / nk) * (y @ vc)
    return F - pref * d["madelung"] * (d["S"] @ dm @ d["S"])


def _exact_dyson(c, d, S1, St):
    """mu, G, and the hermitized self-energies (the search reads them as given)."""
    dev, nk, ns = St.device, _nk(c), c["ns"]
    g = d["grid"]
    Tnt, Ttn = _t(g.Tnt_f, dev), _t(g.Ttn_f, dev)
    iw = 1j * _t(g.wsample_f, dev).reshape(-1, 1, 1, 1, 1)

    def matrix(S1, St):
        return d["H"] + S1 + (Tnt @ St.reshape(c["nts"], -1)).reshape((-1,) + S1.shape)

    X = matrix(S1, St)

    def electrons(mu):
        Gw = torch.linalg.inv((iw + mu) * d["S"] - X)
        tr = torch.einsum("wskij,skji->w", Gw, d["S"]) / nk
        return -(2.0 if ns == 1 else 1.0) * float((Ttn[-1] @ tr).real)

    nel0, tol, delta, mu = d["nel"], 1e-9, 0.5, 0.0
    nel = electrons(mu)
    if abs((nel - nel0) / nel0) > tol:
        lo = hi = mu
        if nel > nel0:
            while True:
                lo -= delta
                if electrons(lo) <= nel0:
                    break
            lo -= delta
        else:
            while True:
                hi += delta
                if electrons(hi) >= nel0:
                    break
            hi += delta
        while abs((nel - nel0) / nel0) > tol and abs(hi - lo) > 0.01 * tol:
            mu = (lo + hi) * 0.5
            nel = electrons(mu)
            if nel > nel0:
                hi = mu
            else:
                lo = mu
    S1, St = _herm(S1), _herm(St)
    Gw = torch.linalg.inv((iw + mu) * d["S"] - matrix(S1, St))
    G = (Ttn @ Gw.reshape(len(g.wsample_f), -1)).reshape(St.shape)
    return mu, G, S1, St


def _exact_energy(c, d, G, S1, St):
    dev, nk, ns = St.device, _nk(c), c["ns"]
    Tnt, Ttn = _t(d["grid"].Tnt_f, dev), _t(d["grid"].Ttn_f, dev)
    dm = (-1.0 if ns == 2 else -2.0) * G[-1]
    e1 = torch.einsum("skij,skji->", dm, d["H"]).real / nk
    ehf = 0.5 * torch.einsum("skij,skji->", dm, S1 + 2 * d["H"]).real / nk
    Gw, Sw = ((Tnt @ x.reshape(c["nts"], -1)).reshape((-1,) + S1.shape) for x in (G, St))
    tr = torch.einsum("wskij,wskji->w", Gw, Sw)
    ec = -float((Ttn[-1] @ tr).real) * (1.0 if ns == 1 else 0.5) / nk
    return np.array([float(e1), float(ehf), ec])


def _out(t):
    return t.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [exact(b, seed * 31 + i) for i, b in enumerate(_batch_systems(case))]
    d = _inputs(case, seed)
    if kind == "gw":
        return _out(_exact_gw(case, d, d["G"], d["V"]))
    if kind == "hf":
        return _out(_exact_hf(case, d, (-1.0 if case["ns"] == 2 else -2.0) * d["G"][-1]))
    if kind == "dyson":
        mu, G, S1, St = _exact_dyson(case, d, d["Sigma1"], d["Sigma"])
        return {"G": _out(G), "Sigma1": _out(S1), "Sigma": _out(St), "mu": mu}
    if kind == "grad":
        G, V = d["G"].requires_grad_(True), d["V"].requires_grad_(True)
        Sigma = _exact_gw(case, d, G, V)
        Gb, Vb = torch.autograd.grad(Sigma, (G, V), d["Sbar"])
        return {"Sigma": _out(Sigma.detach()), "G_bar": _out(Gb), "V_bar": _out(Vb)}
    S1 = _exact_hf(case, d, (-1.0 if case["ns"] == 2 else -2.0) * d["G"][-1])
    Sigma = _exact_gw(case, d, d["G"], d["V"])
    mu, G, S1, Sigma = _exact_dyson(case, d, S1, Sigma)
    return {"G": _out(G), "Sigma1": _out(S1), "Sigma": _out(Sigma), "mu": mu,
            "E": _exact_energy(case, d, G, S1, Sigma)}
