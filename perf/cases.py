"""The work that a user of the library has it do, as cases that can be timed and checked.

A case is one call of a public entry point on synthetic Fourier coefficients N(0,1)*exp(-alpha*n), with the
pad that every SFEMaNS caller uses (m_max_pad = 3*m_max/2).  The sizes come from the repository's
configurations and tests: meridian meshes of a thousand to a few hundred thousand Gauss points, 4 to 256
Fourier modes, odd point counts among them.

``listed`` gives the fixed cases, ``draw`` more of the same ranges, ``prepare`` what a program has in hand
before the call, ``run`` one pass, ``work`` the bytes and operations no implementation can avoid (each input
read once, each output written once, transforms as real FFTs of the dealiased length), and ``exact`` the
result from dense Fourier matrices in plain torch.
"""
import math

import numpy as np
import torch

import sfemans_b200 as sf
from sfemans_b200.profile_case import p2_rectangle

# linearised programs: base fields, slots of one tangent (cotangent), slots of one result
LINEAR = {"cross_jvp": (2, 12, 6), "cross_vjp": (2, 6, 12), "mhd_jvp": (3, 18, 12), "mhd_vjp": (3, 12, 18)}
GAUSS = ("gauss_ns", "gauss_lorentz", "gauss_advect")
GRID_ONLY = ("div", "svdiv", "tension")  # quotients: they depend on the grid of 2*m_max_pad-1 angles
LARGEST_BYTES = 4.0e9  # of a drawn case; the largest listed case moves more


def _pad(m):
    return max(3 * m // 2, 1)


def listed():
    return [
        # a regression-size mesh with a handful of modes: one step calls this many times, so latency counts
        {"name": "cross_small", "kind": "cross", "np": 1701, "m": 4, "alpha": 0.3},
        # the Navier-Stokes / induction product of an ordinary run: 4,000 P2 triangles, 16 modes
        {"name": "cross_ordinary", "kind": "cross", "np": 28000, "m": 16, "alpha": 0.3},
        # the same product at a mode count that is no power of two and an odd point count
        {"name": "cross_ragged", "kind": "cross", "np": 50001, "m": 40, "alpha": 0.2},
        # a strongly turbulent run: many modes
        {"name": "cross_many_modes", "kind": "cross", "np": 35000, "m": 128, "alpha": 0.05},
        # all nonlinear terms of an MHD step with temperature in one call
        {"name": "bundle", "kind": "bundle", "np": 280000, "m": 64, "alpha": 0.1},
        # the adjoint of the linearised product, one cotangent (backward)
        {"name": "adjoint", "kind": "cross_vjp", "np": 175000, "m": 32, "k": 1, "alpha": 0.2},
        # block-Krylov stability: several tangents of the linearised MHD products about one base state (forward)
        {"name": "krylov_block", "kind": "mhd_jvp", "np": 7000, "m": 256, "k": 16, "alpha": 0.05},
        # the split-precision form of the ordinary product
        {"name": "split_ordinary", "kind": "cross", "np": 28000, "m": 16, "alpha": 0.3, "split": 3},
        # momentum over density in variable-density flow (FFT_SCALAR_VECT_DCL, pb = 2): on the caller's grid
        {"name": "vector_over_scalar", "kind": "svdiv", "np": 28000, "m": 32, "alpha": 0.2},
        # the CFL number of every time step (FFT_MAX_VEL_DCL)
        {"name": "max_velocity", "kind": "max_vel", "np": 56000, "m": 32, "alpha": 0.2},
        # the Navier-Stokes term from the nodal velocity on a P2 mesh (curl and product at the Gauss points)
        {"name": "gauss_navier_stokes", "kind": "gauss_ns", "np": 100000, "m": 32, "alpha": 0.2},
        # the drop-in call of a host program: arrays in host memory, copied through the GPU
        {"name": "host_call", "kind": "host_cross", "np": 28000, "m": 16, "alpha": 0.3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cross", "cross", "dot", "prod", "svect", "tensor", "split", "bundle", "linear", "grid", "synth",
                       "gauss", "host_cross"])
    case = {"kind": kind, "alpha": round(rng.uniform(0.05, 0.4), 3)}
    if kind == "linear":
        case["kind"] = rng.choice(sorted(LINEAR))
        case["k"] = _log_int(rng, 1, 16)
        m, np_hi = _log_int(rng, 4, 256), 175000
    elif kind == "split":
        case["kind"] = rng.choice(["cross", "svect", "tensor", "bundle"])
        case["split"] = rng.choice([2, 3])
        m, np_hi = _log_int(rng, 4, 64), 60000
    elif kind == "grid":
        case["kind"] = rng.choice(GRID_ONLY)
        m, np_hi = _log_int(rng, 4, 64), 28000
    elif kind == "synth":
        case["kind"] = rng.choice(["max_vel", "real"])
        m, np_hi = _log_int(rng, 4, 64), 60000
    elif kind == "gauss":
        case["kind"] = rng.choice(GAUSS)
        m, np_hi = _log_int(rng, 4, 64), 200000
    elif kind == "host_cross":
        m, np_hi = _log_int(rng, 4, 64), 28000
    else:
        m, np_hi = _log_int(rng, 4, 64 if kind in ("bundle", "tensor") else 256), 200000
    case["m"] = m
    # the points of the case: its share of the largest drawn size, at most np_hi
    per_point = work(dict(case, np=7))["bytes"] / 7
    case["np"] = _log_int(rng, 1000, max(1001, min(np_hi, LARGEST_BYTES / per_point)))
    return case


def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _field(g, npts, nslot, m, alpha, k=None):
    """Coefficients (np, nslot, m[, k]) in Fortran order; the sine of mode 0 is zero."""
    lead = () if k is None else (k,)
    t = torch.randn(lead + (m, nslot, npts), generator=g, device="cuda", dtype=torch.float64)
    t *= torch.exp(-alpha * torch.arange(m, device="cuda", dtype=torch.float64))[:, None, None]
    t[..., 0, 1::2, :] = 0.0
    return t.permute(*range(t.dim() - 1, -1, -1))


_KIND_SLOTS = {"cross": (6, 6), "dot": (6, 6), "prod": (2, 2), "svect": (6, 2), "tensor": (6, 6), "div": (2, 2),
               "svdiv": (6, 2), "tension": (6, 6)}


def _mesh(npts):
    side = max(1, int(math.ceil(math.sqrt(npts / 14.0))))  # 7 Gauss points on each of 2*side*side triangles
    return p2_rectangle(side, side)


def prepare(case, seed):
    kind, npts, m, alpha = case["kind"], case["np"], case["m"], case["alpha"]
    g = _gen(seed)
    s = {"case": case, "pad": _pad(m)}
    if kind == "host_cross":
        rng = np.random.default_rng(int(seed))
        scale = np.exp(-alpha * np.arange(m))
        for name in ("a", "b"):
            v = np.asfortranarray(rng.standard_normal((m, 6, npts)).T * scale)
            v[:, 1::2, 0] = 0.0
            s[name] = v
        s["out"] = np.zeros((npts, 6, m), order="F")
    elif kind == "bundle":
        s["in"] = [_field(g, npts, 6, m, alpha) for _ in range(5)]
        s["out"] = tuple(sf.fortran_empty(npts, 6, m) for _ in range(3)) + (sf.fortran_empty(npts, 2, m),)
    elif kind in LINEAR:
        nbase, nin, nout = LINEAR[kind]
        s["in"] = [_field(g, npts, 6, m, alpha) for _ in range(nbase)]
        s["x"] = _field(g, npts, nin, m, alpha, case["k"])
        s["out"] = sf.fortran_empty(npts, nout, m, case["k"])
    elif kind in ("max_vel", "real"):
        s["a"] = _field(g, npts, 6, m, alpha)
        if kind == "real":
            s["out"] = sf.synthesis(s["a"])
    elif kind in GAUSS:
        mesh = _mesh(npts)
        s["mesh"] = {k: torch.from_numpy(np.ascontiguousarray(mesh[k].T)).cuda().permute(*range(mesh[k].ndim - 1, -1, -1))
                     for k in ("jj", "ww", "dw", "rr")}
        s["modes"] = torch.arange(m, dtype=torch.int32, device="cuda")
        s["v"] = _field(g, mesh["np"], 6, m, alpha)
        s["v2"] = _field(g, mesh["np"], 2 if kind == "gauss_advect" else 6, m, alpha)
        s["heat"] = 0.5 + 1.5 * torch.rand(mesh["me"], generator=g, device="cuda", dtype=torch.float64)
        s["out"] = sf.fortran_empty(7 * mesh["me"], 2 if kind == "gauss_advect" else 6, m)
    else:
        na, nb = _KIND_SLOTS[kind]
        s["op"] = sf.KINDS[kind][0]
        s["a"], s["b"] = _field(g, npts, na, m, alpha), _field(g, npts, nb, m, alpha)
        if kind in ("div", "svdiv"):
            # a density: positive on the whole circle
            s["b"] *= 0.05
            s["b"][:, 0, 0] = 3.0
        s["out"] = sf.out_empty(s["op"], npts, m)
    return s


def run(state):
    s, kind, pad = state, state["case"]["kind"], state["pad"]
    if kind == "host_cross":
        return sf.FFT_PAR_CROSS_PROD_DCL(None, s["a"], s["b"], s["out"], 1, s["a"].shape[0], pad)
    if kind == "bundle":
        return sf.bundle_mhd(*s["in"], m_max_pad=pad, outs=s["out"], split=s["case"].get("split"))
    if kind in LINEAR:
        return getattr(sf, kind)(*s["in"], s["x"], m_max_pad=pad, out=s["out"])
    if kind == "max_vel":
        return sf.max_vel(s["a"], pad)
    if kind == "real":
        return sf.synthesis(s["a"], out=s["out"])
    if kind == "gauss_ns":
        return sf.cross_gauss(s["v"], s["mesh"], s["modes"], m_max_pad=pad, out=s["out"])
    if kind == "gauss_lorentz":
        return sf.curlh_cross_b_gauss(s["v"], s["v2"], s["mesh"], s["modes"], m_max_pad=pad, out=s["out"])
    if kind == "gauss_advect":
        return sf.ugradc_gauss(s["v"], s["v2"], s["mesh"], s["modes"], heat=s["heat"], conservative=True, m_max_pad=pad,
                               out=s["out"])
    return sf.product(s["op"], s["a"], s["b"], out=s["out"], m_max_pad=pad, split=s["case"].get("split"))


def work(case):
    kind, npts, m, k = case["kind"], case["np"], case["m"], case.get("k", 1)
    N = 2 * _pad(m) - 1
    fft = 2.5 * N * math.log2(max(N, 2))  # of one real field of one point
    extra = 0.0
    if kind == "bundle":
        fin, fout, products = 15, 10, 21
    elif kind in LINEAR:
        nbase, nin, nout = LINEAR[kind]
        fin, fout, products = 3 * nbase + k * nin / 2, k * nout / 2, 4 * k * max(nin, nout) / 2
    elif kind in ("max_vel", "real"):
        fin, fout, products = 3, 0, 3
        extra = 8.0 * (3 * (2 * m - 1) * npts if kind == "real" else 1)
    elif kind in GAUSS:
        mesh_np = npts / 3.5  # P2 triangles: seven Gauss points and two nodes each
        nodal = 3 if kind == "gauss_ns" else 4 if kind == "gauss_advect" else 6
        fin, fout, products = nodal * mesh_np / npts, 1 if kind == "gauss_advect" else 3, 200
        extra = npts * 8.0 * (12 + 2)
    else:
        na, nb = _KIND_SLOTS.get(kind, (6, 6))
        fin, fout = (na + nb) / 2, {"dot": 1, "prod": 1, "div": 1, "tensor": 9, "tension": 9}.get(kind, 3)
        products = 3 * fout
    return {"bytes": npts * 16.0 * m * (fin + fout) + extra, "flops": npts * ((fin + fout) * fft + products * N)}


# ---------------------------------------------------------------------------
# the same results from dense Fourier matrices, in plain torch
# ---------------------------------------------------------------------------
def _matrices(m, N):
    r = torch.outer(torch.arange(m, device="cuda"), torch.arange(N, device="cuda")) % N
    th = r.to(torch.float64) * (2.0 * math.pi / N)
    syn = torch.stack([torch.cos(th), torch.sin(th)], 1)  # (m, 2, N)
    syn[0, 1] = 0.0
    weight = torch.full((m, 1, 1), 2.0 / N, device="cuda", dtype=torch.float64)
    weight[0] = 1.0 / N
    return syn, syn * weight


def _grid(v, syn):
    """Coefficients (np, nslot, m) to values (np, nslot/2, N)."""
    npts, nslot, m = v.shape
    x = v.reshape(npts, nslot // 2, 2, m)
    return torch.einsum("pcsm,msn->pcn", x, syn)


def _modes(f, ana):
    """Values (np, ncomp, N) to coefficients (np, 2*ncomp, m)."""
    y = torch.einsum("pcn,msn->pcsm", f, ana)
    return y.reshape(f.shape[0], -1, ana.shape[0])


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=1)


def _product(kind, a, b):
    if kind == "cross":
        return _cross(a, b)
    if kind == "dot":
        return (a * b).sum(1, keepdim=True)
    if kind in ("prod", "svect"):
        return a * b
    if kind in ("div", "svdiv"):
        return a / b
    if kind == "tensor":
        return a[:, :, None, :] * b[:, None, :, :]
    size = torch.sqrt((b * b).sum(1))[:, None, None, :]
    return a[:, :, None, :] * b[:, None, :, :] / (size + 1e-14) - size * torch.eye(3, device="cuda", dtype=torch.float64)[None, :, :, None]


def _operands(kind, s, pts):
    """The two or four operands of a Gauss-point caller at the points `pts`, (n, slots, m) each."""
    mesh, m = s["mesh"], s["case"]["m"]
    el, q = pts // 7, pts % 7
    jj = mesh["jj"].long() - 1
    node = jj[:, el].t()  # (n, 6)
    ww = mesh["ww"][:, q].t()
    d = mesh["dw"][:, :, q, el].permute(2, 0, 1)  # (n, 2, 6)
    ray = (mesh["rr"][0][node] * ww).sum(1)[:, None]
    mr = torch.arange(m, device="cuda", dtype=torch.float64)[None, :] / ray
    v = s["v"][node]  # (n, 6 nodes, slots, m)
    w, d1, d2 = (torch.einsum("pnsm,pn->psm", v, c) for c in (ww, d[:, 0], d[:, 1]))
    v2 = s["v2"][node]
    w2 = torch.einsum("pnsm,pn->psm", v2, ww)
    if kind == "gauss_advect":
        heat = s["heat"][el][:, None, None]
        c1, c2 = (torch.einsum("pnsm,pn->psm", v2, c) for c in (d[:, 0], d[:, 1]))
        grad = torch.stack([c1[:, 0], c1[:, 1], mr * w2[:, 1], -mr * w2[:, 0], c2[:, 0], c2[:, 1]], 1)
        div = torch.stack([d1[:, 0] + w[:, 0] / ray + mr * w[:, 3] + d2[:, 4],
                           d1[:, 1] + w[:, 1] / ray - mr * w[:, 2] + d2[:, 5]], 1)
        return heat * grad, w, div, heat * w2
    rot = torch.stack([mr * w[:, 5] - d2[:, 2], -mr * w[:, 4] - d2[:, 3], d2[:, 0] - d1[:, 4], d2[:, 1] - d1[:, 5],
                       w[:, 2] / ray + d1[:, 2] - mr * w[:, 1], w[:, 3] / ray + d1[:, 3] + mr * w[:, 0]], 1)
    return rot, (w if kind == "gauss_ns" else w2)


def _exact_chunk(case, s, lo, hi, syn, ana):
    """The outputs of points lo..hi-1, a list of (n, slots, m[, k]) tensors."""
    kind = case["kind"]
    if kind in GAUSS:
        f = [_grid(x, syn) for x in _operands(kind, s, torch.arange(lo, hi, device="cuda"))]
        y = _cross(f[0], f[1]) if len(f) == 2 else (f[0] * f[1]).sum(1, keepdim=True) + f[2] * f[3]
        return [_modes(y, ana)]
    if kind == "bundle":
        u, w, b, j, t = (_grid(x[lo:hi], syn) for x in s["in"])
        return [_modes(y, ana) for y in (_cross(u, w), _cross(u, b), _cross(j, b), (u * t).sum(1, keepdim=True))]
    if kind in LINEAR:
        base = [_grid(x[lo:hi], syn) for x in s["in"]]
        u, others = base[0], base[1:]
        ys = []
        for t in range(case["k"]):
            x = s["x"][lo:hi, :, :, t]
            if kind.endswith("jvp"):
                d = [_grid(x[:, 6 * i:6 * i + 6], syn) for i in range(len(base))]
                y = torch.cat([_cross(d[0], o) + _cross(u, do) for o, do in zip(others, d[1:])], 1)
                ys.append(_modes(y, ana))
            else:  # the transpose: cotangents synthesised with the analysis weights, no weights on the result
                c = [_grid(x[:, 6 * i:6 * i + 6], ana) for i in range(len(others))]
                y = torch.cat([sum(_cross(o, ci) for o, ci in zip(others, c))] + [_cross(ci, u) for ci in c], 1)
                ys.append(_modes(y, syn))
        return [torch.stack(ys, -1)]
    a, b = (torch.as_tensor(s[n][lo:hi], device="cuda") for n in ("a", "b"))
    a, b = _grid(a, syn), _grid(b, syn)
    y = _product("cross" if kind == "host_cross" else kind, a, b)
    if y.dim() == 4:  # tensors: V_out(k, p, 2l-1:2l, n) holds u_k v_l
        n = y.shape[0]
        z = _modes(y.reshape(n, 9, -1), ana).reshape(n, 3, 6, -1)
        return [z.permute(1, 0, 2, 3)]
    return [_modes(y, ana)]


def exact(case, seed):
    s = prepare(case, seed)
    kind, m = case["kind"], case["m"]
    if kind in ("max_vel", "real"):
        N = 2 * s["pad"] - 1 if kind == "max_vel" else 2 * m - 1
        syn, _ = _matrices(m, N)
        step, parts = max(1, int(2e7 / N)), []
        for lo in range(0, case["np"], step):
            f = _grid(s["a"][lo:lo + step], syn)
            parts.append(torch.sqrt((f * f).sum(1)).max() if kind == "max_vel" else f.permute(2, 1, 0))
        return float(torch.stack(parts).max()) if kind == "max_vel" else torch.cat(parts, 2)
    syn, ana = _matrices(m, 2 * s["pad"] - 1)
    out = s["out"] if isinstance(s["out"], tuple) else (s["out"],)
    tensor = kind in ("tensor", "tension")
    npts = out[0].shape[1 if tensor else 0]
    res = [torch.empty(tuple(o.shape), dtype=torch.float64, device="cuda") for o in out]
    step = max(1, int(4e7 / (m * 3 * 40)))
    for lo in range(0, npts, step):
        hi = min(npts, lo + step)
        for r, y in zip(res, _exact_chunk(case, s, lo, hi, syn, ana)):
            if tensor:
                r[:, lo:hi] = y
            else:
                r[lo:hi] = y
    return tuple(res) if isinstance(s["out"], tuple) else res[0]
