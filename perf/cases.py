"""Timed cases of the particle-coupling path, through the library's own entry points.

Every case is one call that a user's program makes again and again: an application of the coupling
operator (what the GMRES loop of a simulation, or a program's own Krylov solver, spends its time on),
a whole solve, the particle sum of the cross sections, the near field of a plane-wave expansion.
Sizes follow the seeded workloads of ``smuthi_gb300/workloads.py`` (100 and 2000 spheres on glass,
the 5000-sphere l_max = 4 shape, the sphere film), with fewer spheres where a pass would take long.

Inputs are synthetic: particles on a jittered lattice of the workload's density and minimum distance;
lookup tables with the radial behaviour of the real ones (spherical Hankel functions of the pair's
multipole orders, cut off below half the minimum distance, plus a smooth layer-mediated part);
vectors whose multipoles fall off with the order like scattered fields do.

Results of the FP32 operator, and of solves that use it, carry FP32-grade values in the library's
complex128 buffers; they are returned as complex64, the precision they have.
"""
import math

import numpy as np
import torch

from smuthi_gb300 import _lib

WAVELENGTH = 550.0
# density and minimum distance of the workloads: (lattice cell in nm, minimum distance in nm, refractive index)
GEOMETRY = {"glass": (268.3, 210.0, 1.0), "small": (282.8, 170.0, 1.0), "film": (300.0, 210.0, 1.8)}
PRECISION = {"fp64": _lib.SG_FP64, "df64": _lib.SG_DF64, "fp32": _lib.SG_FP32}


def listed():
    return [
        # the smallest simulation: the operator application inside a plain GMRES loop, latency counts
        dict(name="plain_100", do="apply", precision="fp64", n=100, l_max=3, rhs=1, kind="linear", res=5.0, geo="glass"),
        # the plain drop-in (default precision) on the 2000-sphere workload
        dict(name="plain_2000", do="apply", precision="fp64", n=2000, l_max=3, rhs=1, kind="cubic", res=5.0, geo="glass"),
        # the l_max = 4 workload's operator, plain, with an odd particle count
        dict(name="plain_l4_1201", do="apply", precision="fp64", n=1201, l_max=4, rhs=1, kind="cubic", res=2.0,
             geo="small"),
        # the refinement residual of the mixed form: 16 plane waves at once
        dict(name="residual_2000_16", do="apply", precision="df64", n=2000, l_max=3, rhs=16, kind="cubic", res=5.0,
             geo="glass"),
        # the inner operator of the mixed form, 16 plane waves at once
        dict(name="inner_2000_16", do="apply", precision="fp32", n=2000, l_max=3, rhs=16, kind="cubic", res=5.0,
             geo="glass"),
        # the same for the sphere film (linear lookup), odd count
        dict(name="inner_film_4001_16", do="apply", precision="fp32", n=4001, l_max=3, rhs=16, kind="linear", res=5.0,
             geo="film"),
        # 64 plane waves on the l_max = 4 shape
        dict(name="inner_l4_1500_64", do="apply", precision="fp32", n=1500, l_max=4, rhs=64, kind="cubic", res=2.0,
             geo="small"),
        # particles at different heights: the volume lookup
        dict(name="volume_250", do="volume", precision="fp64", n=250, l_max=3, rhs=1, kind="linear", res=10.0, geo="glass"),
        # a whole plain solve from host buffers, as Simulation.run does it; particles with two cut-offs
        dict(name="solve_plain_301", do="solve", precision="fp64", n=301, l_max=3, rhs=1, kind="linear", res=5.0,
             geo="glass", cutoffs="mixed", tol=1e-8),
        # a whole solve of 16 plane waves in the mixed form (FP32 operator, double-float residuals)
        dict(name="solve_mixed_1000_16", do="solve", precision="fp32", n=1000, l_max=3, rhs=16, kind="cubic", res=5.0,
             geo="glass", cutoffs="uniform", tol=1e-8),
        # total scattering cross section of one wave: half the default angular grid
        dict(name="cross_section_1000", do="farfield", n=1000, l_max=3, rhs=1, nk=181, na=721),
        # field on a 64 x 64 grid of points from an expansion on the default grids
        dict(name="near_field_4096", do="nearfield", n=4096, nk=279, na=721, field=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["plain", "plain", "residual", "inner", "inner", "volume", "solve", "farfield", "nearfield"])
    geo, res = rng.choice([("glass", 5.0), ("small", 2.0), ("film", 5.0)])
    kind = rng.choice(["linear", "cubic", "cubic", "cubic_hermite"])
    l_max = rng.choice([1, 2, 3, 3, 3, 4])
    if do == "plain":
        rhs = rng.choice([1, 1, 1, 2, 3, 4, 7])
        n = _log_int(rng, 40, (1500 if l_max < 4 else 1000) / math.sqrt(rhs))
        return dict(do="apply", precision="fp64", n=n, l_max=l_max, rhs=rhs, kind=kind, res=res, geo=geo,
                    cutoffs=rng.choice(["uniform", "uniform", "mixed"]))
    if do == "residual":
        rhs = rng.choice([1, 2, 5, 8, 16, 16, 32])
        n = _log_int(rng, 60, min(1800, (6000 if l_max < 4 else 3500) / math.sqrt(rhs)))
        return dict(do="apply", precision="df64", n=n, l_max=l_max, rhs=rhs, kind=kind, res=res, geo=geo)
    if do == "inner":
        rhs = rng.choice([1, 2, 3, 8, 12, 16, 16, 32, 64])
        n = _log_int(rng, 60, 3600 if l_max < 4 else 1400)
        return dict(do="apply", precision="fp32", n=n, l_max=l_max, rhs=rhs, kind=kind, res=max(res, 4.0 if n > 1500 else res),
                    geo=geo, cutoffs=rng.choice(["uniform", "uniform", "mixed"]))
    if do == "volume":
        return dict(do="volume", precision=rng.choice(["fp64", "fp32"]), n=_log_int(rng, 20, 400), l_max=rng.choice([2, 3]),
                    rhs=rng.choice([1, 1, 3, 8]), kind=rng.choice(["linear", "cubic"]), res=10.0, geo="glass")
    if do == "solve":
        if rng.random() < 0.5:
            return dict(do="solve", precision="fp64", n=_log_int(rng, 40, 500), l_max=rng.choice([2, 3]), rhs=rng.choice([1, 1, 2]),
                        kind=kind, res=5.0, geo="glass", cutoffs=rng.choice(["uniform", "mixed"]), tol=rng.choice([1e-6, 1e-8]))
        return dict(do="solve", precision="fp32", n=_log_int(rng, 40, 900), l_max=rng.choice([2, 3]),
                    rhs=rng.choice([1, 4, 16]), kind=kind, res=5.0, geo="glass", cutoffs="uniform", tol=1e-8)
    if do == "farfield":
        rhs = rng.choice([1, 1, 2, 5, 16])
        return dict(do="farfield", n=_log_int(rng, 50, 1400 / math.sqrt(rhs)), l_max=rng.choice([2, 3, 4]), rhs=rhs,
                    nk=rng.randint(40, 181), na=rng.choice([90, 181, 361, 721]))
    return dict(do="nearfield", n=_log_int(rng, 30, 4500), nk=rng.randint(60, 279), na=rng.choice([91, 180, 361, 721]),
                field=rng.choice([0, 1]))


# ---------------------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _normal(g, *shape):
    return torch.complex(torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64),
                         torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64))


def _multipoles(l_max):
    """(l, m) of every index of a block: both polarisations, l = 1 .. l_max, |m| <= l."""
    lm = [(l, m) for _ in range(2) for l in range(1, l_max + 1) for m in range(-l, l + 1)]
    return np.array([a for a, _ in lm], np.int32), np.array([b for _, b in lm], np.int32)


def _inputs(case, seed):
    """Everything the timed call is given: positions, the unknowns' layout, table, T-matrices, vectors."""
    g = _generator(seed)
    n, R = case["n"], case["rhs"]
    cell, d_min, index = GEOMETRY[case["geo"]]
    l_of_n, m_of_n = _multipoles(case["l_max"])
    B = len(l_of_n)
    side = math.ceil(math.sqrt(n))
    at = torch.randperm(side * side, generator=g, device="cuda")[:n]
    xy = torch.stack([at % side, at // side], 1).double() * cell
    xy = xy + (torch.rand(n, 2, generator=g, device="cuda", dtype=torch.float64) - 0.5) * (cell - d_min)
    xy = xy.cpu().numpy()
    own = np.ones((n, B), bool)
    if case.get("cutoffs") == "mixed":  # every third particle: one order less
        own[::3] = (l_of_n < max(2, case["l_max"]))[None]
    up, un = [a.astype(np.int32) for a in np.nonzero(own)]
    d = xy[:, None] - xy[None] if n < 700 else None
    r_max = float(np.sqrt((d ** 2).sum(-1)).max()) if d is not None else side * cell * math.sqrt(2.0)
    res = case["res"]
    rho = np.arange(-3 * res, r_max + 4 * res, res)
    fall = torch.tensor([0.3, 0.1, 0.02, 0.004], dtype=torch.float64, device="cuda")[torch.as_tensor(l_of_n - 1).long()]
    x = _normal(g, n, B, R) * fall[None, :, None]
    x = x.reshape(n * B, R)[torch.as_tensor(up.astype(np.int64) * B + un).cuda()].contiguous()
    t = torch.tensor([0.1, 0.02, 0.002, 0.0003], dtype=torch.float64, device="cuda")[torch.as_tensor(l_of_n - 1).long()]
    t = torch.stack([torch.polar(t, 6.28 * torch.rand(B, generator=g, device="cuda", dtype=torch.float64)) for _ in range(2)])
    t[1] *= torch.as_tensor(own[0]).cuda()  # the T-matrix of a lower cut-off has no entries above it
    return dict(g=g, n=n, B=B, R=R, l=l_of_n, m=m_of_n, xy=xy, up=up, un=un, rho=rho, x=x, t=t, k=2 * math.pi * index / WAVELENGTH,
                d_min=d_min, types=(np.arange(n) % 3 == 0).astype(np.int32))


def _hankel(order, z):
    """Spherical Hankel functions h_0 .. h_order of real z > 0, by upward recurrence."""
    e = torch.polar(torch.ones_like(z), z)
    h = [-1j * e / z, -e * (z + 1j) / z ** 2]
    for l in range(1, order):
        h.append((2 * l + 1) / z * h[l] - h[l - 1])
    return h


def _orders(inp):
    l = torch.as_tensor(inp["l"]).long().cuda()
    return l[:, None] + l[None, :]


def _radial_table(inp):
    """[len_rho, B, B]: direct part (cut off below half the minimum distance) plus layer-mediated part."""
    g, B = inp["g"], inp["B"]
    rho = torch.as_tensor(inp["rho"]).cuda()
    a, b = 0.5 * _normal(g, B, B), 0.15 * _normal(g, B, B)
    inside = (rho >= inp["d_min"] / 2).double()
    h = torch.stack(_hankel(2 * int(inp["l"].max()), inp["k"] * rho.clamp(min=inp["d_min"] / 2)), 1) * inside[:, None]
    z = inp["k"] * rho.abs()
    soft = torch.polar(1 / (1 + z), 1.2 * z)
    return a[None] * h[:, _orders(inp)] + b[None] * soft[:, None, None]


def _volume_tables(inp, res):
    """[len_rho, len_z, B, B] tables of z1 + z2 and z1 - z2, rounded to complex64 like the real ones."""
    g, B = inp["g"], inp["B"]
    z = torch.rand(inp["n"], generator=g, device="cuda", dtype=torch.float64) * 60.0 + 100.0
    rho = torch.as_tensor(inp["rho"]).cuda()
    nz = int(math.ceil(120.0 / res)) + 8
    sz, dz = 200.0 - 3 * res + res * torch.arange(nz).cuda().double(), -60.0 - 3 * res + res * torch.arange(nz).cuda().double()
    a, b = 0.5 * _normal(g, B, B), 0.15 * _normal(g, B, B)
    rp = inp["k"] * torch.sqrt(rho[:, None] ** 2 + sz[None] ** 2)
    plus = b[None, None] * torch.polar(1 / (1 + rp), rp)[:, :, None, None]
    rm = torch.sqrt(rho[:, None] ** 2 + dz[None] ** 2)
    direct = torch.stack(_hankel(2 * int(inp["l"].max()), inp["k"] * rm.clamp(min=inp["d_min"] / 2)), 2)
    direct = direct * (rho >= inp["d_min"] / 2).double()[:, None, None]
    minus = a[None, None] * direct[:, :, _orders(inp)]
    return z.cpu().numpy(), float(sz[0]), float(dz[0]), plus.to(torch.complex64), minus.to(torch.complex64)


def _farfield_inputs(case, seed):
    g = _generator(seed)
    n, R, nk, na = case["n"], case["rhs"], case["nk"], case["na"]
    l_of_n, m_of_n = _multipoles(case["l_max"])
    B = len(l_of_n)
    xy = torch.rand(n, 2, generator=g, device="cuda", dtype=torch.float64) * 268.3 * math.sqrt(n)
    fall = torch.tensor([0.3, 0.1, 0.02, 0.004], dtype=torch.float64, device="cuda")[torch.as_tensor(l_of_n - 1).long()]
    coef = _normal(g, n, B, R) * fall[None, :, None]
    kpar = 2 * math.pi / WAVELENGTH * torch.sin(torch.linspace(0, math.pi / 2, nk, dtype=torch.float64, device="cuda"))
    S = 0.4 * _normal(g, B, 2, nk)
    alpha = torch.linspace(0, 2 * math.pi, na, dtype=torch.float64, device="cuda")
    return xy, coef.contiguous(), m_of_n, kpar, S, alpha


def _nearfield_inputs(case, seed):
    g = _generator(seed)
    n, nk, na = case["n"], case["nk"], case["na"]
    k = 2 * math.pi / WAVELENGTH
    pts = (torch.rand(3, n, generator=g, device="cuda", dtype=torch.float64) - 0.5) * 6000.0
    pts[2] = pts[2].abs() / 10.0 + 250.0
    # Sommerfeld contour: real line with a dip into the lower half plane around the branch points
    s = torch.linspace(0, 1.4 * k, nk, dtype=torch.float64, device="cuda")
    dip = 0.05 * k * ((s > 0.8 * k) & (s < 1.2 * k)).double() * torch.sin((s / k - 0.8) / 0.4 * math.pi).clamp(min=0)
    kpar = torch.complex(s, -dip)
    kz = torch.sqrt(k ** 2 - kpar ** 2)
    kz = torch.where(kz.imag < 0, -kz, kz)
    alpha = torch.linspace(0, 2 * math.pi, na, dtype=torch.float64, device="cuda")
    return pts, kpar.contiguous(), kz.contiguous(), alpha, _normal(g, 2, nk, na), k


def prepare(case, seed):
    do = case["do"]
    ctx = _lib.Context(0)
    if do == "farfield":
        xy, coef, m_of_n, kpar, S, alpha = _farfield_inputs(case, seed)
        out = torch.empty(case["rhs"], 2, case["nk"], case["na"], dtype=torch.complex128, device="cuda")
        return dict(case=case, ctx=ctx, xy=xy, coef=coef, m=m_of_n, kpar=kpar, S=S, alpha=alpha, out=out)
    if do == "nearfield":
        pts, kpar, kz, alpha, amp, k = _nearfield_inputs(case, seed)
        out = torch.empty(3, case["n"], dtype=torch.complex128, device="cuda")
        return dict(case=case, ctx=ctx, pts=pts, kpar=kpar, kz=kz, alpha=alpha, amp=amp, k=k, out=out)
    inp = _inputs(case, seed)
    ctx.set_particles(inp["xy"], inp["up"], inp["un"], inp["B"], inp["m"])
    if do == "volume":
        z, sz0, dz0, plus, minus = _volume_tables(inp, case["res"])
        ctx.set_volume_lookup(case["kind"], z, plus.cpu().numpy(), minus.cpu().numpy(), inp["rho"][0], sz0, dz0, case["res"])
    else:
        ctx.set_lookup(case["kind"], _radial_table(inp).cpu().numpy(), inp["rho"][0], case["res"])
    ctx.set_tmatrix(torch.diag_embed(inp["t"]).cpu().numpy(), inp["types"], True)
    x = inp["x"]
    if do == "solve" and case["precision"] == "fp64":
        x = x.cpu().numpy()
        return dict(case=case, ctx=ctx, x=x if case["rhs"] > 1 else x[:, 0].copy())
    return dict(case=case, ctx=ctx, x=x, y=torch.zeros_like(x))


def run(state):
    case, ctx = state["case"], state["ctx"]
    do = case["do"]
    if do == "farfield":
        s = state
        ctx.farfield_sum_dev(case["n"], s["xy"].data_ptr(), len(s["m"]), case["rhs"], s["coef"].data_ptr(), int(s["m"].max()),
                             s["m"], case["nk"], s["kpar"].data_ptr(), s["S"].data_ptr(), case["na"], s["alpha"].data_ptr(),
                             s["out"].data_ptr())
        return s["out"]
    if do == "nearfield":
        s, p = state, state["pts"]
        ctx.pwe_field_dev(case["field"], case["n"], p[0].data_ptr(), p[1].data_ptr(), p[2].data_ptr(), case["nk"],
                          s["kpar"].data_ptr(), s["kz"].data_ptr(), case["na"], s["alpha"].data_ptr(), s["amp"].data_ptr(),
                          s["k"], 2 * math.pi / WAVELENGTH, s["out"].data_ptr())
        return s["out"]
    if do == "solve":
        if case["precision"] == "fp64":
            sol, _ = ctx.gmres(state["x"], state["x"], case["tol"], precision=_lib.SG_FP64)
            return sol
        state["y"].zero_()
        ctx.gmres_dev(state["x"].data_ptr(), state["y"].data_ptr(), case["rhs"], case["tol"],
                      precision=_lib.SG_FP32 | _lib.SG_DF64)
        return state["y"].to(torch.complex64)
    ctx.master_matvec_dev(state["x"].data_ptr(), state["y"].data_ptr(), case["rhs"], PRECISION[case["precision"]])
    return state["y"].to(torch.complex64) if case["precision"] == "fp32" else state["y"]


def work(case):
    do, n = case["do"], case["n"]
    if do == "nearfield":
        nodes = case["nk"] * case["na"]
        # one complex phase (counted as 30 operations) and three complex multiply-adds per point and node
        return {"bytes": 16.0 * (2 * nodes + 3 * n) + 24.0 * n, "flops": float(n) * nodes * (30 + 24)}
    B = len(_multipoles(case["l_max"])[0])
    R = case["rhs"]
    if do == "farfield":
        dirs, nm = case["nk"] * case["na"], 2 * case["l_max"] + 1
        return {"bytes": 16.0 * (n * B * R + 2 * B * case["nk"] + 2 * R * dirs), "flops": float(n) * dirs * (30 + 8.0 * 2 * R * nm)}
    word = 8.0 if case["precision"] == "fp32" else 16.0
    cell = GEOMETRY[case["geo"]][0]
    rows = cell * math.sqrt(2.0 * n) / case["res"] + 7
    taps = 4 if case["kind"] == "linear" else 12
    if do == "volume":
        rows, taps = 2 * rows * (120.0 / case["res"] + 8), 2 * (12 if case["kind"] == "linear" else 60)
    # operator applications: one; a solve needs about one per Krylov step and one per residual
    times = 1 if do != "solve" else (13 if case["precision"] == "fp64" else 16)
    return {"bytes": times * (rows * B * B * word + 2 * 16.0 * n * B * R),
            "flops": times * float(n) * n * B * B * (taps + 8.0 * R)}


# ---------------------------------------------------------------------------------------- 64-bit values
def _moments(y):
    """h^2 x second derivatives at the knots of the not-a-knot cubic spline through y[:, ...]."""
    L = y.shape[0]
    flat = torch.view_as_real(y.reshape(L, -1)).reshape(L, -1)
    A = torch.zeros(L, L, dtype=torch.float64, device=y.device)
    i = torch.arange(1, L - 1, device=y.device)
    A[i, i - 1], A[i, i], A[i, i + 1] = 1.0, 4.0, 1.0
    for row, s in ((0, 0), (L - 1, L - 3)):
        A[row, s], A[row, s + 1], A[row, s + 2] = 1.0, -2.0, 1.0
    rhs = torch.zeros_like(flat)
    rhs[1:-1] = 6 * (flat[2:] - 2 * flat[1:-1] + flat[:-2])
    return torch.view_as_complex(torch.linalg.solve(A, rhs).contiguous().reshape(L, -1, 2)).reshape(y.shape)


def _polynomials(kind, y):
    """Per interval k: coefficients of 1, t, t^2, t^3."""
    if kind == "linear":
        return [y[:-1], y[1:] - y[:-1]]
    if kind == "cubic":
        M = _moments(y)
        return [y[:-1], (y[1:] - y[:-1]) - (2 * M[:-1] + M[1:]) / 6, M[:-1] / 2, (M[1:] - M[:-1]) / 6]
    p = torch.cat([y[:1], y, y[-1:]])
    a, b, c, d = p[:-3], p[1:-2], p[2:-1], p[3:]
    return [b, (c - a) / 2, (2 * a - 5 * b + 4 * c - d) / 2, (-a + 3 * b - 3 * c + d) / 2]


def _geometry(inp, i0, i1, res):
    xy = torch.as_tensor(inp["xy"]).cuda()
    d = xy[i0:i1, None] - xy[None]
    rho = torch.sqrt((d ** 2).sum(-1))
    phi = torch.atan2(d[..., 1], d[..., 0])
    idx = (rho - inp["rho"][0]) / res
    return idx, phi


def _blocks(inp, case, polys, i0, i1):
    """W[i0:i1, :, B, B]: the interpolated blocks with their phases."""
    idx, phi = _geometry(inp, i0, i1, case["res"])
    k = idx.floor().long().clamp(0, polys[0].shape[0] - 1)
    t = (idx - k)[..., None, None]
    w = polys[-1][k]
    for p in polys[-2::-1]:
        w = w * t + p[k]
    m = torch.as_tensor(inp["m"]).cuda().double()
    return w * torch.polar(torch.ones((), dtype=torch.float64, device="cuda"), phi[..., None, None] * (m[None, :] - m[:, None]))


def _volume_blocks(inp, case, tables, i0, i1):
    z, sz0, dz0, plus, minus = tables
    z = torch.as_tensor(z).cuda()
    idx, phi = _geometry(inp, i0, i1, case["res"])
    w = 0
    for tab, pos in ((plus, z[i0:i1, None] + z[None] - sz0), (minus, z[i0:i1, None] - z[None] - dz0)):
        pos = pos / case["res"]
        k, q = idx.floor().long(), pos.floor().long()
        t, s = (idx - k)[..., None, None], (pos - q)[..., None, None]
        w = w + (1 - t) * ((1 - s) * tab[k, q] + s * tab[k, q + 1]) + t * ((1 - s) * tab[k + 1, q] + s * tab[k + 1, q + 1])
    m = torch.as_tensor(inp["m"]).cuda().double()
    return w * torch.polar(torch.ones((), dtype=torch.float64, device="cuda"), phi[..., None, None] * (m[None, :] - m[:, None]))


def _padded(inp, v):
    out = torch.zeros(inp["n"] * inp["B"], v.shape[1], dtype=torch.complex128, device="cuda")
    out[torch.as_tensor(inp["up"].astype(np.int64) * inp["B"] + inp["un"]).cuda()] = v
    return out


def _own(inp, v):
    return v[torch.as_tensor(inp["up"].astype(np.int64) * inp["B"] + inp["un"]).cuda()]


def _t_rows(inp):
    return inp["t"][torch.as_tensor(inp["types"]).long().cuda()].reshape(-1, 1)


def exact(case, seed):
    do = case["do"]
    if do == "farfield":
        xy, coef, m_of_n, kpar, S, alpha = _farfield_inputs(case, seed)
        R, na = case["rhs"], case["na"]
        ms = sorted(set(int(m) for m in m_of_n))
        em = torch.polar(torch.ones((), dtype=torch.float64, device="cuda"),
                         alpha[:, None] * torch.tensor(ms, dtype=torch.float64, device="cuda"))
        u = torch.cos(alpha)[:, None] * xy[None, :, 0] + torch.sin(alpha)[:, None] * xy[None, :, 1]
        out = torch.zeros(R, 2, case["nk"], na, dtype=torch.complex128, device="cuda")
        sel = [torch.as_tensor(np.nonzero(m_of_n == m)[0]).cuda() for m in ms]
        for k in range(case["nk"]):
            d = torch.stack([torch.einsum("inr,np->irp", coef[:, s], S[s, :, k]) for s in sel], 1)  # [i, m, r, p]
            f = torch.polar(torch.ones((), dtype=torch.float64, device="cuda"), -kpar[k] * u) @ d.reshape(case["n"], -1)
            out[:, :, k] = (f.reshape(na, len(ms), R, 2) * em[:, :, None, None]).sum(1).permute(1, 2, 0)
        return out
    if do == "nearfield":
        p, kpar, kz, alpha, amp, k = _nearfield_inputs(case, seed)
        ca, sa = torch.cos(alpha), torch.sin(alpha)
        u = ca[None] * p[0][:, None] + sa[None] * p[1][:, None]
        wa = torch.zeros_like(alpha)
        wa[1:] += 0.5 * (alpha[1:] - alpha[:-1])
        wa[:-1] += 0.5 * (alpha[1:] - alpha[:-1])
        wk = torch.zeros_like(kpar)
        wk[1:] += 0.5 * (kpar[1:] - kpar[:-1])
        wk[:-1] += 0.5 * (kpar[1:] - kpar[:-1])
        out = torch.zeros(3, case["n"], dtype=torch.complex128, device="cuda")
        for j in range(case["nk"]):
            te, tm = amp[0, j], amp[1, j]
            if case["field"] == 0:
                v = torch.stack([-sa * te + ca * kz[j] / k * tm, ca * te + sa * kz[j] / k * tm, -kpar[j] / k * tm], 1)
            else:
                v = torch.stack([-kz[j] * ca * te - k * sa * tm, -kz[j] * sa * te + k * ca * tm, kpar[j] * te], 1)
                v = v / (2 * math.pi / WAVELENGTH)
            f = torch.exp(1j * kpar[j] * u) @ (wa[:, None] * v)
            out += (wk[j] * kpar[j] * torch.exp(1j * kz[j] * p[2])[:, None] * f).T
        return out
    if do == "volume" and case["kind"] != "linear":
        return None
    inp = _inputs(case, seed)
    n, B, R = inp["n"], inp["B"], inp["R"]
    if do == "volume":
        tables = _volume_tables(inp, case["res"])
        tables = tables[:3] + tuple(t.to(torch.complex128) for t in tables[3:])

        def block(i0, i1):
            return _volume_blocks(inp, case, tables, i0, i1)
    else:
        polys = _polynomials(case["kind"], _radial_table(inp))

        def block(i0, i1):
            return _blocks(inp, case, polys, i0, i1)
    step = max(1, int(2e7 / (n * B * B)))

    def rows(i0):
        i1 = min(n, i0 + step)
        return block(i0, i1).permute(0, 2, 1, 3).reshape((i1 - i0) * B, n * B)
    x = _padded(inp, inp["x"])
    if do != "solve":
        y = torch.cat([rows(i0) @ x for i0 in range(0, n, step)])
        out = _own(inp, x - _t_rows(inp) * y)
        return out.to(torch.complex64) if case["precision"] == "fp32" else out
    # solve: dense T W, GMRES without restarts on every right-hand side, refined to 64-bit accuracy
    own = torch.zeros(n * B, 1, dtype=torch.float64, device="cuda")
    own[torch.as_tensor(inp["up"].astype(np.int64) * B + inp["un"]).cuda()] = 1.0
    TW = torch.cat([rows(i0) for i0 in range(0, n, step)])
    TW *= _t_rows(inp) * own

    def apply(v):
        return v - TW @ v
    sol = torch.zeros_like(x)
    for _ in range(3):
        r = x - apply(sol)
        beta = torch.linalg.vector_norm(r, dim=0)
        V, H = [r / beta], torch.zeros(R, 26, 25, dtype=torch.complex128, device="cuda")
        for j in range(25):
            w = apply(V[j])
            for _ in range(2):
                for q in range(j + 1):
                    h = (V[q].conj() * w).sum(0)
                    H[:, q, j] += h
                    w = w - h * V[q]
            h = torch.linalg.vector_norm(w, dim=0)
            H[:, j + 1, j] = h
            V.append(w / h)
        e = torch.zeros(R, 26, 1, dtype=torch.complex128, device="cuda")
        e[:, 0, 0] = beta
        y = torch.linalg.pinv(H) @ e
        for j in range(25):
            sol = sol + V[j] * y[:, j, 0]
    out = _own(inp, sol)
    if case["precision"] == "fp64":
        out = out.cpu().numpy()
        return out if R > 1 else out[:, 0]
    return out.to(torch.complex64)
