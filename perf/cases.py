"""Performance cases: the work a variational-MPS user has this library do.

Every case is one call (or the short sequence of calls) of a public entry
point, over the sizes the library is used at: bond dimensions from a handful
(the edges of a chain, small exact problems) to 1024 (the benchmark), spin 1/2
and spin 1, plain FP64 and precision form, square and ragged bonds.

``listed`` gives the fixed cases, ``draw`` more of the same ranges,
``prepare`` the inputs and handles that a program has in hand, ``run`` one
pass, ``work`` the bytes and operations a pass cannot do without, and
``exact`` the values in plain 64-bit torch or numpy where a result has one.
"""
from __future__ import annotations

import ctypes as ct
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (os.path.join(os.getcwd(), "nutcracker-1_b200"), os.path.join(_ROOT, "nutcracker-1_b200")):
    if os.path.isdir(_p) and _p not in sys.path:
        sys.path.append(_p)

C128 = torch.complex128


def listed():
    return [
        # H_eff product of an interior site at the benchmark's size (N=100
        # Heisenberg, chi=1024): the inner loop of an FP64 sweep.
        {"name": "heff_1024", "kind": "heff", "model": "heisenberg", "mixed": 0, "bl": 1024, "br": 1024},
        # The same product for spin 1 at odd, unequal bonds: a middling site of
        # a chain whose bond dimension was not chosen as a power of two.
        {"name": "heff_spin1_ragged", "kind": "heff", "model": "spin1", "mixed": 0, "bl": 301, "br": 243},
        # A small site of the transverse Ising chain: latency and launches.
        {"name": "heff_small", "kind": "heff", "model": "ising", "mixed": 0, "bl": 24, "br": 24},
        # The precision form's product at the benchmark's size.
        {"name": "heff_mixed_1024", "kind": "heff", "model": "heisenberg", "mixed": 1, "bl": 1024, "br": 1024},
        # Left environment update (the sweep's way right), FP64, a large bond.
        {"name": "env_left_640", "kind": "env", "model": "heisenberg", "mixed": 0, "side": 0, "bl": 640, "br": 640},
        # Right environment update (the way back) of a serving-size site with
        # unequal bonds, as next to a chain's end.
        {"name": "env_right_ragged", "kind": "env", "model": "ising", "mixed": 0, "side": 1, "bl": 150, "br": 97},
        # Precision-form right environment update of the spin-1 chain, chi=512.
        {"name": "env_mixed_spin1_512", "kind": "env", "model": "spin1", "mixed": 1, "side": 1, "bl": 512, "br": 512},
        # Gauge move at the benchmark's size, moving right.
        {"name": "gauge_right_1024", "kind": "gauge", "dir": 1, "d": 2, "bl": 1024, "bm": 1024, "br": 1024},
        # Gauge move at a serving size, moving left, odd bonds.
        {"name": "gauge_left_130", "kind": "gauge", "dir": -1, "d": 2, "bl": 130, "bm": 125, "br": 131},
        # The site eigen-solve on host buffers (the Fortran-ABI drop-in), with
        # one lower level projected out: an excited level's site step.
        {"name": "site_solve_48", "kind": "solve", "model": "heisenberg", "bl": 48, "br": 48, "nproj": 1},
        # A whole FP64 sweep of a 20-site chain from a given state: upload,
        # environments, 39 site solves and 38 moves, energy and centre site back.
        {"name": "sweep_heisenberg_20", "kind": "sweep", "model": "heisenberg", "sites": 20, "chi": 64},
        # A batch of small chains with random couplings in the lockstep engine.
        {"name": "batch_xxz", "kind": "batch", "chains": 12, "sites_min": 8, "sites_max": 10, "chi_max": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["heff", "heff", "heff", "env", "env", "gauge", "gauge", "solve", "sweep", "batch"])
    model = rng.choice(["heisenberg", "ising", "spin1"])
    d = _PHYS[model]
    top = 1024 if d == 2 else 640
    if kind in ("heff", "env"):
        mixed = int(rng.random() < 0.35)
        bl = _log(rng, 96 if mixed else 8, top)
        # neighbouring bonds are equal inside a chain, up to a factor d apart next to its ends
        br = bl if rng.random() < 0.4 else max(6, min(top, int(bl * rng.uniform(1.0 / d, 1.3))))
        c = {"kind": kind, "model": model, "mixed": mixed, "bl": bl, "br": br}
        if kind == "env":
            c["side"] = rng.randrange(2)
        return c
    if kind == "gauge":
        d = rng.choice([2, 2, 3])
        b = _log(rng, 12, 1024 if d == 2 else 640)
        return {"kind": kind, "dir": rng.choice([1, -1]), "d": d, "bl": b, "bm": max(4, b - rng.randrange(4)),
                "br": max(4, b - rng.randrange(6))}
    if kind == "solve":
        b = _log(rng, 10, 64 if d == 2 else 40)
        return {"kind": kind, "model": model, "bl": b, "br": max(8, b - rng.randrange(6)), "nproj": rng.randrange(3)}
    if kind == "sweep":
        return {"kind": kind, "model": rng.choice(["heisenberg", "ising"]), "sites": rng.randrange(8, 21),
                "chi": _log(rng, 8, 64)}
    lo = rng.randrange(6, 9)
    return {"kind": kind, "chains": rng.randrange(4, 13), "sites_min": lo, "sites_max": rng.randrange(lo, 11),
            "chi_max": rng.randrange(6, 17)}


# ---- the library -------------------------------------------------------------

_PHYS = {"heisenberg": 2, "ising": 2, "spin1": 3}
_STREAM = []


def _library():
    """The bindings, with the library's work on a stream of this program's."""
    import nutcracker_b200 as nb

    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    nb.lib.nc_set_stream(ct.c_void_p(_STREAM[0].cuda_stream))
    return nb


def _chain(model, n):
    from nutcracker_b200 import operators

    if model == "heisenberg":
        return operators.heisenberg(n)
    if model == "ising":
        return operators.ferromagnetic_transverse_ising(n, 1.2)
    return operators.heisenberg_spin1(n)


def _site(model):
    return _chain(model, 4)[1]


# ---- inputs ------------------------------------------------------------------
# Column-major tensors are held as contiguous torch tensors with the axes
# reversed: psi (br,bl,d) is a (d,bl,br) tensor.


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(*shape, dtype=C128, device="cuda", generator=g)


def _schmidt(n, least=1e-4):
    """A decaying Schmidt spectrum 1 .. least."""
    return torch.logspace(0, math.log10(least), n, dtype=torch.float64, device="cuda")


def _environment(g, b, c, identity, energy):
    """c Hermitian channels: the identity where the canonical gauge leaves it,
    a block energy with spread, and interaction terms of order one."""
    A = _randn(g, c, b, b) / math.sqrt(2.0 * b)
    E = A + A.conj().transpose(1, 2)
    eye = torch.eye(b, dtype=C128, device="cuda")
    E[energy] = 2.0 * E[energy] - 5.0 * eye
    E[identity] = eye
    return E.contiguous()


def _centre(g, d, bl, br):
    """A centre site of unit norm whose bonds carry decaying Schmidt values."""
    k = min(d * bl, br)
    left = _randn(g, d * bl, k) * _schmidt(k)
    x = left @ _randn(g, k, br)
    return (x / x.norm()).reshape(d, bl, br).contiguous()


def _mixed_columns(g, rows, cols):
    """rows x cols with full column rank: graded columns mixed by a unitary."""
    return torch.fft.fft(_randn(g, rows, cols) * _schmidt(cols), dim=1, norm="ortho")


def _pointers(*tensors):
    return [ct.c_void_p(t.data_ptr()) for t in tensors]


def _operator_on_device(op):
    return (torch.from_numpy(op.W.ravel(order="F").copy()).cuda(),
            torch.from_numpy(op.idx.ravel(order="F").astype(np.int32)).cuda())


def _site_inputs(case, seed):
    """L, R, psi of a heff or env case."""
    op, g = _site(case["model"]), _gen(seed)
    bl, br = case["bl"], case["br"]
    L = _environment(g, bl, op.cl, 0, op.cl - 1)
    R = _environment(g, br, op.cr, op.cr - 1, 0)
    return op, L, R, _centre(g, op.d, bl, br)


def _gauge_inputs(case, seed):
    g, d = _gen(seed), case["d"]
    bl, bm, br = case["bl"], case["bm"], case["br"]
    if case["dir"] > 0:                                  # A (bm,bl,d) gets normalised
        A = _mixed_columns(g, d * bl, bm).reshape(d, bl, bm)
        B = _randn(g, d, bm, br) / math.sqrt(d * br)
    else:                                                # B (br,bm,d) gets normalised
        A = _randn(g, d, bl, bm) / math.sqrt(d * bl)
        B = _mixed_columns(g, d * br, bm).reshape(d, br, bm).transpose(1, 2)
    return A.contiguous(), B.contiguous()


def _host_environment(rng, b, c, identity, energy):
    A = rng.standard_normal((b, b, c)) + 1j * rng.standard_normal((b, b, c))
    E = (A + A.conj().transpose(1, 0, 2)) / math.sqrt(8.0 * b)
    u = rng.standard_normal(b) + 1j * rng.standard_normal(b)
    u /= np.linalg.norm(u)
    E[:, :, energy] = 0.5 * E[:, :, energy] - 6.0 * np.outer(u, u.conj())   # a block ground state, gapped
    E[:, :, identity] = np.eye(b)
    return np.asfortranarray(E)


def _solve_inputs(case, seed):
    """Host buffers of a site solve: environments, guess, projector vectors."""
    rng, op = np.random.default_rng(seed), _site(case["model"])
    bl, br = case["bl"], case["br"]
    L = _host_environment(rng, bl, op.cl, 0, op.cl - 1)
    R = _host_environment(rng, br, op.cr, op.cr - 1, 0)
    n = bl * br * op.d
    guess = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    V = np.asfortranarray(rng.standard_normal((n, case["nproj"])) + 1j * rng.standard_normal((n, case["nproj"])))
    return op, L, R, guess, V


def _bonds(n, chi, d=2):
    edge = [1]
    while edge[-1] * d < chi and len(edge) < (n + 1) // 2:
        edge.append(edge[-1] * d)
    full = min(chi, d ** (n // 2))
    return edge + [full] * (n + 1 - 2 * len(edge)) + edge[::-1]


def _random_state(rng, bonds, d=2):
    """Random sites (br,bl,d): site 0 the centre, the rest right-normalised."""
    sites = []
    for i in range(len(bonds) - 1):
        bl, br = bonds[i], bonds[i + 1]
        x = rng.standard_normal((br * d, bl)) + 1j * rng.standard_normal((br * d, bl))
        if i == 0:
            q = x / np.linalg.norm(x)
        else:
            q = np.linalg.qr(x)[0]
        sites.append(np.asfortranarray(q.reshape(br, d, bl).transpose(0, 2, 1)))
    return sites


# ---- one state per case ----------------------------------------------------------


def prepare(case, seed):
    nb = _library()
    kind = case["kind"]
    if kind in ("heff", "env"):
        op, L, R, psi = _site_inputs(case, seed)
        W, idx = _operator_on_device(op)
        dims = [ct.c_uint32(v) for v in (case["bl"], case["br"], op.cl, op.cr, op.d, op.nnz)]
        if kind == "heff":
            out = torch.empty_like(psi)
            fn = nb.lib.nc_heff_apply_mixed_dev if case["mixed"] else nb.lib.nc_heff_apply_dev
            args, keep = dims + _pointers(idx, W, L, R, psi, out), (idx, W, L, R, psi)
        else:
            b, c, env = (case["br"], op.cr, L) if case["side"] == 0 else (case["bl"], op.cl, R)
            out = torch.empty((c, b, b), dtype=C128, device="cuda")
            fn = nb.lib.nc_env_update_dev
            args = [ct.c_int(case["side"]), ct.c_int(case["mixed"])] + dims + _pointers(idx, W, env, psi, out)
            keep = (idx, W, env, psi)
        return {"kind": kind, "nb": nb, "fn": fn, "args": args, "out": out, "keep": keep}
    if kind == "gauge":
        A, B = _gauge_inputs(case, seed)
        oA, oB = torch.empty_like(A), torch.empty_like(B)
        args = [ct.c_int(case["dir"])] + [ct.c_uint32(v) for v in (case["bl"], case["bm"], case["br"], case["d"],
                                                                    case["d"])] + _pointers(A, B, oA, oB)
        return {"kind": kind, "nb": nb, "fn": nb.lib.nc_gauge_move_dev, "args": args, "out": [oA, oB], "keep": (A, B)}
    if kind == "solve":
        op, L, R, guess, V = _solve_inputs(case, seed)
        n, m = len(guess), case["nproj"]
        if m:
            refl, rank, coeff, swaps = nb.Core.convert_vectors_to_reflectors(n, m, V)
            proj = (m, m, n - rank, refl, coeff, swaps)
            guess = nb.Core.filter_components_outside_orthog(n, *proj, guess)
        else:
            proj = (0, 0, n, None, None, None)
        guess = guess / np.linalg.norm(guess)
        args = (case["bl"], case["br"], op.cl, op.cr, op.d, L, op.nnz, op.idx, op.W, R, *proj, "SR", 1e-12, 1000,
                guess.reshape((case["br"], case["bl"], op.d), order="F"))
        return {"kind": kind, "nb": nb, "args": args}
    if kind == "sweep":
        from nutcracker_b200.chain import Chain

        bonds = _bonds(case["sites"], case["chi"])
        state = _random_state(np.random.default_rng(seed), bonds)
        chain = Chain(_chain(case["model"], case["sites"]), initial_bandwidth_dimension=max(bonds), seed=1)
        return {"kind": kind, "nb": nb, "chain": chain, "state": state}
    from nutcracker_b200 import operators
    from nutcracker_b200.batched import Batch

    rng = np.random.default_rng(seed)
    sites = [case["sites_min"] + k % (case["sites_max"] - case["sites_min"] + 1) for k in range(case["chains"])]
    chis = [min(2 ** (n // 2), case["chi_max"] - k % 3) for k, n in enumerate(sites)]
    batch = Batch([operators.xxz_random(n, rng) for n in sites], chis, seeds=[7 + k for k in range(len(sites))],
                  precision=0, maximum_sweeps=3)
    return {"kind": kind, "nb": nb, "batch": batch}


def run(state):
    kind, nb = state["kind"], state["nb"]
    if kind in ("heff", "env", "gauge"):
        if state["fn"](*state["args"]) != 0:
            nb._check()
        return state["out"]
    if kind == "solve":
        info, _, eigenvalue, result, normal = nb.Core.optimize(*state["args"])
        return {"info": info, "eigenvalue": np.array([eigenvalue]), "result": result, "normal": np.array([normal])}
    if kind == "sweep":
        chain = state["chain"]
        chain.set_state(state["state"])
        chain.perform_optimization_sweep()
        return {"energy": np.array([chain.get_energy()]), "centre": chain.get_site(0)}
    return np.array([r["energy"] for r in state["batch"].solve()])


# ---- what a pass cannot do without ---------------------------------------------------


def _heff_work(bl, br, op):
    d, cl, cr, nnz = op.d, op.cl, op.cr, op.nnz
    return (16 * (bl * bl * cl + br * br * cr + 2 * bl * br * d),
            8.0 * d * bl * br * (cl * bl + cr * br) + 8.0 * nnz * d * d * bl * br)


def _env_work(bl, br, op, side):
    d, cl, cr, nnz = op.d, op.cl, op.cr, op.nnz
    if side == 0:
        flops = 8.0 * d * bl * br * (cl * bl + cr * br)
    else:
        flops = 8.0 * d * bl * br * (cr * br + cl * bl)
    return 16 * (bl * bl * cl + br * br * cr + bl * br * d), flops + 8.0 * nnz * d * d * bl * br


def _gauge_work(b_free, bm, b_other, d):
    """Householder QR with explicit Q of a (d b_free) x bm matrix, and the absorption."""
    m = d * b_free
    return (16 * 2 * (m * bm + d * bm * b_other),
            4.0 * (4.0 * m * bm * bm - 4.0 / 3.0 * bm ** 3) + 8.0 * d * b_other * bm * bm)


def _chain_work(ops, bonds):
    """One sweep: per site step one H_eff product, one move, one environment update."""
    total_b, total_f = 0.0, 0.0
    for i, op in enumerate(ops):
        bl, br = bonds[i], bonds[i + 1]
        steps = 1 if i in (0, len(ops) - 1) else 2
        for b, f in (_heff_work(bl, br, op), _env_work(bl, br, op, 0), _gauge_work(bl, br, br, op.d)):
            total_b += steps * b
            total_f += steps * f
    return total_b, total_f


def work(case):
    kind = case["kind"]
    if kind == "heff":
        b, f = _heff_work(case["bl"], case["br"], _site(case["model"]))
    elif kind == "env":
        b, f = _env_work(case["bl"], case["br"], _site(case["model"]), case["side"])
    elif kind == "gauge":
        free, other = (case["bl"], case["br"]) if case["dir"] > 0 else (case["br"], case["bl"])
        b, f = _gauge_work(free, case["bm"], other, case["d"])
    elif kind == "solve":
        # a handful of products is the least a solve to 1e-12 takes from a cold guess
        op = _site(case["model"])
        b, f = _heff_work(case["bl"], case["br"], op)
        f *= 8
    elif kind == "sweep":
        b, f = _chain_work(_chain(case["model"], case["sites"]), _bonds(case["sites"], case["chi"]))
    else:
        from nutcracker_b200 import operators

        b = f = 0.0
        for k in range(case["chains"]):
            n = case["sites_min"] + k % (case["sites_max"] - case["sites_min"] + 1)
            cb, cf = _chain_work(operators.heisenberg(n), _bonds(n, case["chi_max"] - k % 3))
            b, f = b + 3 * cb, f + 3 * cf                # three sweeps
    return {"bytes": b, "flops": f}


# ---- the values in plain 64-bit arithmetic ---------------------------------------------


def _exact_site(case, seed):
    op, L, R, psi = _site_inputs(case, seed)
    W = torch.from_numpy(np.ascontiguousarray(op.W)).cuda()              # (o1, o2, n)
    links = [(int(op.idx[0, n]) - 1, int(op.idx[1, n]) - 1, W[:, :, n]) for n in range(op.nnz)]
    # psi as (a, l, r); L (k, j, i) for L(i=ket, j=bra, k); R (k, r=ket, r'=bra)
    if case["kind"] == "heff":
        T = torch.einsum("ali,kjl->kaji", psi, L)
        out = torch.zeros_like(psi)
        for k2 in range(op.cr):
            U = sum((torch.einsum("ab,ajr->bjr", w, T[f]) for f, t, w in links if t == k2), torch.zeros_like(T[0]))
            out += torch.einsum("bjr,rx->bjx", U, R[k2])
        return out
    if case["side"] == 0:
        T = torch.einsum("ali,kjl->kaji", psi, L)
        out = []
        for k2 in range(op.cr):
            U = sum((torch.einsum("ab,ajr->bjr", w, T[f]) for f, t, w in links if t == k2), torch.zeros_like(T[0]))
            out.append(torch.einsum("bjr,bjx->xr", U, psi.conj()))
        return torch.stack(out)
    Y = torch.einsum("bxq,krq->kbxr", psi.conj(), R)
    out = []
    for k1 in range(op.cl):
        Z = sum((torch.einsum("ab,bxr->axr", w, Y[t]) for f, t, w in links if f == k1), torch.zeros_like(Y[0]))
        out.append(torch.einsum("axr,ayr->yx", Z, psi))
    return torch.stack(out)


def _exact_gauge(case, seed):
    A, B = _gauge_inputs(case, seed)
    d, bl, bm, br = case["d"], case["bl"], case["bm"], case["br"]
    if case["dir"] > 0:
        X = A.reshape(d * bl, bm).conj().cpu().numpy()                   # A^H of the (bm, bl d) site
        q, r = np.linalg.qr(X)
        denorm = torch.einsum("smr,km->skr", B, torch.from_numpy(r).cuda().conj())
        return [torch.from_numpy(q.conj().reshape(d, bl, bm)).cuda(), denorm]
    X = B.transpose(1, 2).reshape(d * br, bm).conj().cpu().numpy()       # rows (s, r)
    # rows ordered with r fastest, as the library forms them
    q, r = np.linalg.qr(X)
    denorm = torch.einsum("slm,km->slk", A, torch.from_numpy(r).cuda().conj())
    norm = torch.from_numpy(q.conj().reshape(d, br, bm)).cuda().transpose(1, 2).contiguous()
    return [denorm, norm]


def _exact_solve(case, seed):
    op, L, R, guess, V = _solve_inputs(case, seed)
    n = len(guess)
    if n > 5000:
        return None
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (L, op.W, R)]
    H = torch.zeros((op.d, case["bl"], case["br"], op.d, case["bl"], case["br"]), dtype=C128, device="cuda")
    for q in range(op.nnz):
        f, to = int(op.idx[0, q]) - 1, int(op.idx[1, q]) - 1
        H += torch.einsum("ij,ab,xr->bjxair", t[0][:, :, f], t[1][:, :, q], t[2][:, :, to])
    H = H.reshape(n, n)
    if case["nproj"]:
        # the vectors are overlap vectors: the space removed is that of their conjugates
        Q = torch.from_numpy(np.linalg.qr(V.conj())[0]).cuda()
        P = torch.eye(n, dtype=C128, device="cuda") - Q @ Q.conj().T
        H = P @ H @ P + 1e3 * (Q @ Q.conj().T)
    w = torch.linalg.eigvalsh(0.5 * (H + H.conj().T))
    return {"info": None, "eigenvalue": w[:1].to(C128), "result": None, "normal": np.array([1.0])}


def exact(case, seed):
    if case["kind"] in ("heff", "env"):
        return _exact_site(case, seed)
    if case["kind"] == "gauge":
        return _exact_gauge(case, seed)
    if case["kind"] == "solve":
        return _exact_solve(case, seed)
    return None   # sweeps stop at their own thresholds: no value that a plain formula gives
