"""The work that a user of this package has it do, as cases to be timed: whole solutions of a body, wings with their
rigid wakes, load gradients, factorizations and sweeps of right hand sides, the free wake, and its point sums.

Every case goes through the package's public entry points with host arrays, as user programs call them. Sizes are
those of the tests, of the bench and of what lies between. Geometry, strengths and flow directions come from the seed
(a design variation of a few per cent about the named mesh). FP64 is the package's default precision; mixed precision
is what the large wings run in.

`run` leaves out what is rounding noise or a clock: the multipliers lambda and the residual (both vanish for the
compatible right hand sides of a closed body), and the statistics' times.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vortexpanel.jl_gb300"))
import vortexpanel_gpu as vp  # noqa: E402
from vortexpanel_gpu import adjoint, freewake, meshes  # noqa: E402

TIERS = ("self", "edge", "vertex", "contact", "near", "far")


def listed():
    return [
        # the smallest whole solution: an 80-triangle sphere (smoke checks, unit tests, the inside of a shape search),
        # where latency, launches and allocations count
        dict(name="sphere80_fp64", kind="body", shape="sphere", size=1, precision="fp64", test="hat"),
        # the test suite's sphere of 1,280 triangles, default options, the matrix read back as the reference's Matrix
        dict(name="sphere1280_fp64", kind="body", shape="sphere", size=3, precision="fp64", test="hat"),
        # the 3:1:1 ellipsoid of about 12k jittered triangles with slivers, default precision: a large closed body
        dict(name="ellipsoid12k_fp64", kind="body", shape="ellipsoid", size=32, stretch=3.0, precision="fp64", test="hat"),
        # the bench's wing (25,532 triangles) forward, mixed precision: assembly, factorization, solution, loads
        dict(name="wing25k_mixed", kind="wing", nchord=112, nspan=56, precision="mixed"),
        # load gradients of a small wing in the default precision: a gradient check or a small design loop
        dict(name="grad1700_fp64", kind="grad", nchord=28, nspan=14, precision="fp64"),
        # load gradients of a production wing in mixed precision (the mesh of the angle-of-attack sweep)
        dict(name="grad13k_mixed", kind="grad", nchord=80, nspan=40, precision="mixed"),
        # factor a 6.6k-unknown system in FP64 and solve it once
        dict(name="factor6600_fp64", kind="solve", nchord=80, nspan=40, precision="fp64", nrhs=1, kept=False),
        # an angle-of-attack sweep: 64 right hand sides with factors that the program keeps, mixed precision
        dict(name="sweep64_mixed", kind="solve", nchord=80, nspan=40, precision="mixed", nrhs=64, kept=True),
        # five steps of a free wake continued from a checkpoint
        dict(name="freewake_mixed", kind="freewake", nchord=28, nspan=28, precision="mixed", warm=30, steps=5),
        # the blob sum of a late free wake at its own particles and some more points
        dict(name="blobs100k_mixed", kind="blobs", nblob=100_000, npts=100_000, precision="mixed"),
        # the body's velocity at a cloud of field points (streamlines, a survey plane), default precision
        dict(name="field_fp64", kind="field", nchord=28, nspan=14, npts=20_000, precision="fp64"),
        # five wings of uneven sizes assembled in one call, mixed precision (a population of designs)
        dict(name="batch5_mixed", kind="batch", wings=5, nchord=18, nspan=12, growth=1.3, precision="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("body", "body", "wing", "wing", "grad", "grad", "solve", "solve", "freewake", "blobs", "field",
                       "batch"))
    precision = rng.choice(("fp64", "mixed"))
    if kind == "body":
        return dict(kind=kind, shape="ellipsoid", size=_log(rng, 3, 20), stretch=round(rng.uniform(1.0, 4.0), 2),
                    precision=precision, test=rng.choice(("hat", "hat", "onering", "dual")))
    if kind == "wing":
        nc = _log(rng, 5, 90 if precision == "mixed" else 48)
        return dict(kind=kind, nchord=nc, nspan=max(3, int(nc * rng.uniform(0.4, 0.8))), precision=precision)
    if kind == "grad":
        nc = _log(rng, 5, 56 if precision == "mixed" else 24)
        return dict(kind=kind, nchord=nc, nspan=max(3, int(nc * rng.uniform(0.4, 0.8))), precision=precision)
    if kind == "solve":
        nc = _log(rng, 5, 80)
        return dict(kind=kind, nchord=nc, nspan=max(3, int(nc * rng.uniform(0.4, 0.6))), precision=precision,
                    nrhs=_log(rng, 1, 64), kept=rng.random() < 0.5)
    if kind == "freewake":
        nc = _log(rng, 8, 28)
        return dict(kind=kind, nchord=nc, nspan=rng.randint(5, nc), precision=precision, warm=rng.randint(4, 16),
                    steps=rng.randint(1, 5))
    if kind == "blobs":
        hi = 150_000 if precision == "mixed" else 20_000
        return dict(kind=kind, nblob=_log(rng, 100, hi), npts=_log(rng, 100, hi), precision=precision)
    if kind == "field":
        nc = _log(rng, 5, 40)
        return dict(kind=kind, nchord=nc, nspan=max(3, nc // 2 + rng.randint(0, 3)), npts=_log(rng, 100, 15_000),
                    precision=precision)
    return dict(kind=kind, wings=rng.randint(2, 5), nchord=rng.randint(6, 18), nspan=rng.randint(4, 12),
                growth=round(rng.uniform(1.05, 1.3), 3), precision=precision)


# ---- inputs ------------------------------------------------------------------------------------------------------------


@functools.lru_cache(maxsize=4)
def _ellipsoid_mesh(n, stretch):
    return meshes.ellipsoid_case(n, axes=(stretch, 1.0, 1.0), seed=7)[0]


def _direction(rng):
    V = np.array([1.0, rng.uniform(-0.3, 0.3), rng.uniform(-0.3, 0.3)])
    return V / np.linalg.norm(V)


def _body(case, rng):
    if case["shape"] == "sphere":
        g = meshes.icosphere(case["size"])
    else:
        g = _ellipsoid_mesh(case["size"], case["stretch"])
    g = meshes.scale_nodes(g, 1.0 + rng.uniform(-0.03, 0.03, 3))
    return g, meshes.closed_body_dofmap(g)


def _wake_rows(nchord):
    """the rigid wake's rows to 20 chords downstream: the trailing edge panel's length, growing by 1.2"""
    rows = [0.0, (1 - math.cos(math.pi / nchord)) / 2]
    while rows[-1] < 20.0:
        rows.append(rows[-1] + (rows[-1] - rows[-2]) * 1.2)
    return rows


def _wing(nchord, nspan, rng):
    w = meshes.wing(nchord, nspan, aspect=8.0 * rng.uniform(0.9, 1.1), thickness=0.12 * rng.uniform(0.9, 1.1))
    wake = meshes.build_wake(w.g, w.dm, (1.0, 0.0, 0.0), rows=_wake_rows(nchord))
    return w, wake, meshes.wake_rows(w.dm, wake.te)


def _alpha(rng):
    return math.radians(rng.uniform(3.0, 7.0))


def _stream(alpha):
    return np.array([math.cos(alpha), 0.0, math.sin(alpha)])


def _unknowns(w, rng, k):
    """k smooth doublet distributions over the unknowns with the zero area mean of a closed body's solution"""
    dm, g = w.dm, w.g
    node = np.where(dm.free_slot < g.nnode, dm.free_slot, 0)
    lower = dm.free_slot >= g.nnode
    node[lower] = dm.wake_te.node[dm.free_slot[lower] - g.nnode]
    x, y, z = g.x[node].T
    y = 2 * y / w.span
    basis = np.stack([x, z, x * x, y * y, x * y * y, x * z, np.sqrt(np.clip(1 - y * y, 0, None)) * np.sign(z + 1e-9) * x,
                      np.cos(2 * x) * y], axis=1)
    q = basis @ rng.standard_normal((basis.shape[1], k)) + 1e-2 * rng.standard_normal((len(x), k))
    area = dm.C.T @ dm.slot_area
    return q - (area @ q) / area.sum()


def _cloud(case, rng):
    n, m = case["nblob"], case["npts"]
    lo, hi = np.array([0.0, -4.0, -1.0]), np.array([8.0, 4.0, 1.0])
    x = rng.uniform(lo, hi, (n, 3))
    blobs = np.hstack([x, 1e-3 * rng.standard_normal((n, 3)), rng.uniform(0.03, 0.07, (n, 1))])
    X = np.vstack([x[:min(n, m)], rng.uniform(lo, hi, (max(m - n, 0), 3))])
    return blobs, np.ascontiguousarray(X)


def _field(case, rng):
    w = meshes.wing(case["nchord"], case["nspan"], aspect=8.0 * rng.uniform(0.9, 1.1))
    sigma = 0.3 * rng.standard_normal(w.g.ntri)
    gamma = rng.standard_normal((w.g.ntri, 3))
    X = rng.uniform([-1.0, -6.0, -1.5], [4.0, 6.0, 1.5], (case["npts"], 3))
    return w, sigma, gamma, X


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = dict(case=case, kind=kind)
    if kind == "body":
        g, dm = _body(case, rng)
        s.update(g=g, dm=dm, V=_direction(rng), opts=vp.AssemblyOptions(precision=case["precision"], test=case["test"]))
    elif kind in ("wing", "grad"):
        w, wake, W = _wing(case["nchord"], case["nspan"], rng)
        s.update(w=w, wake=wake, W=W, alpha=_alpha(rng), opts=vp.AssemblyOptions(precision=case["precision"]))
    elif kind == "solve":
        w, wake, W = _wing(case["nchord"], case["nspan"], rng)
        V = _stream(_alpha(rng))
        els = vp.build_elements(w.g)
        A, _, _ = vp.assemble(w.g, w.dm, els, vp.source_strengths(els, V), V, wake=wake,
                              opts=vp.AssemblyOptions(precision="mixed"))
        # right hand sides whose solutions are known: b = A [C; W] q
        q = _unknowns(w, rng, case["nrhs"])
        b = A.download() @ np.vstack([w.dm.C @ q, W @ q])
        s.update(dm=w.dm, W=W, A=A, b=b[:, 0].copy() if case["nrhs"] == 1 else b)
        if case["kept"]:
            s["F"] = vp.factorize_galerkin(w.dm, A, W=W, precision=case["precision"])
    elif kind == "freewake":
        w = meshes.wing(case["nchord"], case["nspan"], aspect=8.0 * rng.uniform(0.9, 1.1))
        sim = freewake.FreeWakeSim(w.g, w.dm, _stream(math.radians(rng.uniform(6.0, 9.0))),
                                   freewake.FreeWakeOptions(dt=0.05, core=0.05),
                                   assembly=vp.AssemblyOptions(precision=case["precision"]), capacity=8192)
        sim.run(case["warm"])
        s.update(sim=sim, checkpoint=sim.checkpoint())
    elif kind == "blobs":
        s["blobs"], s["X"] = _cloud(case, rng)
    elif kind == "field":
        s["w"], s["sigma"], s["gamma"], s["X"] = _field(case, rng)
    else:
        cases = []
        for k in range(case["wings"]):
            f = case["growth"] ** k
            w, wake, _ = _wing(int(case["nchord"] * f), int(case["nspan"] * f), rng)
            V = _stream(_alpha(rng))
            cases.append((w.g, w.dm, vp.source_strengths(vp.build_elements(w.g), V), V, wake))
        s.update(cases=cases, opts=vp.AssemblyOptions(precision=case["precision"]))
    return s


# ---- one pass ------------------------------------------------------------------------------------------------------------


def _counts(stats):
    return {k: np.array([stats[k][t] for t in TIERS], dtype=np.int64) for k in ("pairs", "points")}


def run(s):
    return {"body": _run_body, "wing": _run_wing, "grad": _run_grad, "solve": _run_solve, "freewake": _run_freewake,
            "blobs": _run_blobs, "field": _run_field, "batch": _run_batch}[s["kind"]](s)


def _run_body(s):
    """the flow about a closed body: A (read back up to 2,000 triangles, as the reference returns it; larger ones stay
    on the device), b, the doublets, the surface velocities and pressures"""
    g, dm, V, opts = s["g"], s["dm"], s["V"], s["opts"]
    els = vp.build_elements(g)
    A, b, stats = vp.assemble(g, dm, els, vp.source_strengths(els, V), V, opts=opts)
    F = vp.factorize_galerkin(dm, A, precision=opts.precision)
    sol = vp.solve_galerkin(F, b)
    loads = vp.surface_loads(els, dm, sol["mu"], V)
    out = dict(b=b, q=sol["q"], mu=sol["mu"], cond=sol["cond"], u=loads["u"], cp=loads["cp"], **_counts(stats))
    if g.ntri <= 2000:
        out["A"] = np.asarray(A)
    return out


def _run_wing(s):
    """a wing at an angle of attack: the solution, the pressures, the pressure force, Kutta-Joukowski and Trefftz"""
    w, wake, opts = s["w"], s["wake"], s["opts"]
    V = _stream(s["alpha"])
    els = vp.build_elements(w.g)
    A, b, stats = vp.assemble(w.g, w.dm, els, vp.source_strengths(els, V), V, wake=wake, opts=opts)
    F = vp.factorize_galerkin(w.dm, A, W=s["W"], precision=opts.precision)
    sol = vp.solve_galerkin(F, b)
    loads = vp.surface_loads(els, w.dm, sol["mu"], V)
    Fkj, drag = vp.wake_loads(w.dm.wake_te, w.dm.K @ sol["q"], V)
    return dict(b=b, q=sol["q"], mu=sol["mu"], cond=sol["cond"], u=loads["u"], cp=loads["cp"], F=loads["F"],
                M=loads["M"], Fkj=Fkj, drag=np.array(drag), **_counts(stats))


def _run_grad(s):
    r = adjoint.wing_gradients(s["w"], s["wake"], s["W"], s["alpha"], precision=s["opts"].precision)
    return dict(loads=np.array([r["CL"], r["CDi"]]), q=r["q"], cond=r["cond"], dCL_dx=r["dCL_dx"],
                dCDi_dx=r["dCDi_dx"], dalpha=np.array([r["dCL_dalpha"], r["dCDi_dalpha"]]), **_counts(r["stats"]))


def _run_solve(s):
    F = s["F"] if s["case"]["kept"] else vp.factorize_galerkin(s["dm"], s["A"], W=s["W"], precision=s["case"]["precision"])
    r = vp.solve_galerkin(F, s["b"])
    return dict(q=r["q"], mu=r["mu"], cond=r["cond"])


def _run_freewake(s):
    sim = s["sim"]
    sim.restore(s["checkpoint"])
    out = {}
    for k in range(s["case"]["steps"]):
        r = sim.step()
        out[f"step{k}"] = dict(F_pressure=r["F_pressure"], F_kj=r["F_kj"], I=r["I"], mu_w=r["mu_w"],
                               particles=r["particles"], rows=r["rows"])
    st = sim.state
    out["state"] = dict(x=np.array(st.x), mu=np.array(st.mu), particles=st.particles, tag=st.tag)
    return out


def _run_blobs(s):
    return freewake.blob_velocities(s["blobs"], s["X"], precision=s["case"]["precision"])


def _run_field(s):
    return freewake.body_velocity(s["w"].g, s["sigma"], s["gamma"], s["X"], precision=s["case"]["precision"])


def _run_batch(s):
    return [dict(A=np.asarray(A), b=b, **_counts(stats)) for A, b, stats in vp.assemble_batch(s["cases"], opts=s["opts"])]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
# Flops of the pair integrals: every pair (test triangle x source triangle) has at least the three points of the far
# rule; a point is 60 flops of the multipole form and 18 of its contraction (forward), and 160 of the form's derivatives
# and 2 x 60 of the sums (gradients of two loads). Nearer pairs need more points, which only running tells. A dense LU
# of order n is 2/3 n^3, a solution 2 n^2 per right hand side.


def _wing_sizes(nchord, nspan):
    ntri = 4 * nchord * nspan + 2 * (2 * nchord - 2)
    nslot = (nspan + 1) * (2 * nchord + 1)
    rows = len(_wake_rows(nchord)) - 1
    return ntri, nslot, 2 * rows * nspan, (rows + 1) * (nspan + 1)


def work(case):
    kind = case["kind"]
    if kind == "body":
        ntri = 20 * 4 ** case["size"] if case["shape"] == "sphere" else 12 * case["size"] ** 2
        n = ntri // 2 + 2
        out = 8.0 * n * n if ntri <= 2000 else 0.0
        return dict(bytes=8.0 * n * n + 100.0 * ntri + out, flops=3.0 * 78 * ntri ** 2 + 2 / 3 * n ** 3 + 2.0 * n * n)
    if kind in ("wing", "grad"):
        ntri, n, wtri, wnode = _wing_sizes(case["nchord"], case["nspan"])
        pairs = 3.0 * ntri * (ntri + wtri)
        lu = 2 / 3 * n ** 3 + 2.0 * n * n * (3 if kind == "grad" else 1)
        return dict(bytes=8.0 * n * (n + wnode) + 8.0 * n * n + 200.0 * ntri,
                    flops=pairs * (78 + (280 if kind == "grad" else 0)) + lu)
    if kind == "solve":
        _, n, _, wnode = _wing_sizes(case["nchord"], case["nspan"])
        k = case["nrhs"]
        lu = 0.0 if case["kept"] else 2 / 3 * n ** 3
        return dict(bytes=(8.0 * n * n if case["kept"] else 8.0 * n * (n + wnode)) + 16.0 * n * k,
                    flops=lu + 2.0 * n * n * k)
    if kind == "freewake":
        ntri, n, _, _ = _wing_sizes(case["nchord"], case["nspan"])
        np_ = 2.0 * case["nspan"] * (case["warm"] + case["steps"])
        step = 3.0 * 28 * ntri * np_ + 78.0 * ntri * np_ + 28.0 * np_ * np_ + 2.0 * n * n
        return dict(bytes=case["steps"] * (8.0 * n * n + 100.0 * np_), flops=case["steps"] * step)
    if kind == "blobs":
        return dict(bytes=56.0 * case["nblob"] + 48.0 * case["npts"], flops=28.0 * case["nblob"] * case["npts"])
    if kind == "field":
        ntri = _wing_sizes(case["nchord"], case["nspan"])[0]
        return dict(bytes=104.0 * ntri + 48.0 * case["npts"], flops=78.0 * ntri * case["npts"])
    b = f = 0.0
    for k in range(case["wings"]):
        g = case["growth"] ** k
        ntri, n, wtri, wnode = _wing_sizes(int(case["nchord"] * g), int(case["nspan"] * g))
        b += 16.0 * n * (n + wnode) + 100.0 * ntri
        f += 3.0 * 78 * ntri * (ntri + wtri)
    return dict(bytes=b, flops=f)


# ---- the same in 64 bits, without the package's kernels ----------------------------------------------------------------


def exact(case, seed):
    """The solutions that the right hand sides of `solve` were made from, and the point sums as plain torch gives them
    in 64 bits (only the inputs are the package's meshes). The pair integrals have no plain counterpart here: they are
    defined by their adaptive rules, whose walk in plain numpy takes minutes on the listed meshes."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "solve":
        w, _, _ = _wing(case["nchord"], case["nspan"], rng)
        _alpha(rng)
        q = _unknowns(w, rng, case["nrhs"])
        q = q[:, 0] if case["nrhs"] == 1 else q
        return dict(q=q, mu=w.dm.C @ q, cond=None)
    if case["kind"] == "blobs":
        return _exact_blobs(*_cloud(case, rng))
    if case["kind"] == "field":
        w, sigma, gamma, X = _field(case, rng)
        return _exact_field(w.g.x[w.g.tris], sigma, gamma, X)
    return None


def _gpu(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda" if torch.cuda.is_available() else "cpu")


def _exact_blobs(blobs, X):
    """sum of alpha x r / (4 pi (|r|^2 + delta^2)^(3/2)), r = x - x_blob"""
    b, x = _gpu(blobs), _gpu(X)
    out = torch.empty_like(x)
    step = max(1, 50_000_000 // len(b))
    for i in range(0, len(x), step):
        r = [x[i:i + step, k, None] - b[None, :, k] for k in range(3)]
        d2 = r[0] ** 2 + r[1] ** 2 + r[2] ** 2 + b[None, :, 6] ** 2
        f = 1 / (4 * math.pi * d2 * d2.sqrt())
        a = [b[None, :, 3 + k] for k in range(3)]
        for k in range(3):
            p, q = (k + 1) % 3, (k + 2) % 3
            out[i:i + step, k] = ((a[p] * r[q] - a[q] * r[p]) * f).sum(1)
    return out.cpu().numpy()


def _exact_field(T, sigma, gamma, X, far=10.0):
    """sum of sigma w + gamma x w with w the unit source velocity of every triangle: the edge logs and the solid angle
    within `far` diameters, the multipole to third order beyond (source_triangle.jl:39-138)"""
    T, sigma, gamma, X = _gpu(T), _gpu(sigma), _gpu(gamma), _gpu(X)
    c = T.mean(1)
    nA = torch.linalg.cross(T[:, 1] - T[:, 0], T[:, 2] - T[:, 0])
    A2 = nA.norm(dim=1)
    n, area = nA / A2[:, None], A2 / 2
    edge = [T[:, (k + 1) % 3] - T[:, k] for k in range(3)]
    length = [e.norm(dim=1) for e in edge]
    nu = [torch.linalg.cross(e, n) / l[:, None] for e, l in zip(edge, length)]
    diam = torch.stack(length).amax(0)
    out = torch.empty_like(X)
    step = max(1, 3_000_000 // len(T))
    for i in range(0, len(X), step):
        x = X[i:i + step, None, :]
        r = x - c
        R2 = (r * r).sum(-1)
        w = r / R2[..., None] ** 1.5
        for k in range(3):
            d = T[:, k] - c
            dr, dd = (r * d).sum(-1)[..., None], (d * d).sum(-1)[:, None]
            R = R2[..., None].sqrt()
            w = w + (15 * dr ** 2 / R ** 7 * r - 6 * dr / R ** 5 * d - 3 * dd / R ** 5 * r) / 24
            w = w - (45 * dr ** 2 / R ** 7 * d - 105 * dr ** 3 / R ** 9 * r - 9 * dd / R ** 5 * d
                     + 45 * dd * dr / R ** 7 * r) / 180
        w = w * (area / (4 * math.pi))[:, None]
        rk = [x - T[:, k] for k in range(3)]
        lk = [v.norm(dim=-1) for v in rk]
        e = torch.zeros_like(r)
        for k in range(3):
            p, q = rk[k], rk[(k + 1) % 3]
            lp, lq = lk[k], lk[(k + 1) % 3]
            pq = (p * q).sum(-1)
            c2 = (torch.linalg.cross(p, q) ** 2).sum(-1)
            inv = torch.where(pq < 0, (lp * lq - pq) / (2 * c2), 1 / (2 * (lp * lq + pq)))
            e = e + ((lp + lq + length[k]) ** 2 * inv).log()[..., None] * nu[k]
        N = (rk[0] * torch.linalg.cross(rk[1], rk[2])).sum(-1)
        D = lk[0] * lk[1] * lk[2] + (rk[0] * rk[1]).sum(-1) * lk[2] + (rk[0] * rk[2]).sum(-1) * lk[1] + (rk[1] * rk[2]).sum(-1) * lk[0]
        e = (e + 2 * torch.atan2(N, D)[..., None] * n) / (4 * math.pi)
        w = torch.where((R2 > (far * diam) ** 2)[..., None], w, e)
        out[i:i + step] = (sigma[:, None] * w + torch.linalg.cross(gamma.expand_as(w), w)).sum(1)
    return out.cpu().numpy()
