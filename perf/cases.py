"""The work that programs have this library do, as measurable cases.

Every case is one call (or one output interval of a run) through the Python binding of the C ABI,
with the host arrays that lpm-v2 holds in Fortran: the sums are host-buffer calls, the solvers and
the ensemble keep their state on the GPU.  Meshes are the reference's uniform refinements at the
sizes of this repository's benchmark and tests, turned (sphere) or gently deformed (plane) by the
seed, so that another seed is another particle set; "n" below the mesh's own count drops particles
at random, as refinement and remeshing leave sets of any size.

LPM_MODE_FP32C evaluates its pairs in single precision, and the sweep shape that its tuner picks by
timing moves the last bits from one process to the next: its results are good to single precision
(1e-6 of the largest), and a program that asks for that mode keeps them in single-precision fields.
LPM_MODE_FP64 results are kept in double precision.
"""
import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "lpm-v2_gb300"))
import lpm_gpu as lg  # noqa: E402
import workloads as wl  # noqa: E402

EXACT_PAIRS = 4e10  # the most pairs that exact() evaluates (tens of seconds above it)


def listed():
    return [
        # one right-hand side of a coarse run: the call's latency is all there is
        {"name": "bve_small", "family": "bve", "mode": "fp32c", "nest": 3, "n": 1922, "block": False},
        # the headline problem: one velocity sum at icosahedral nest 8, 2.6e12 pairs
        {"name": "bve_large", "family": "bve", "mode": "fp32c", "nest": 8, "n": 1966082, "block": False},
        # one rank's block of targets of a set of odd size, as the MPI code calls it
        {"name": "bve_rank_block", "family": "bve", "mode": "fp32c", "nest": 6, "n": 100003, "block": True},
        # the reference's own single-vortex run, bit for bit, ten steps to the next output
        {"name": "bve_run_fp64", "family": "bve_run", "mode": "fp64", "nest": 4, "n": 7682, "steps": 10},
        # the same kind of run in the production mode, one refinement finer
        {"name": "bve_run", "family": "bve_run", "mode": "fp32c", "nest": 5, "n": 30722, "steps": 10},
        # the colliding dipoles' velocity, regularised
        {"name": "plane_quad7", "family": "plane", "mode": "fp32c", "nest": 7, "n": 131585, "delta": 0.02},
        # a remesh interval of the dipoles' run in the reference's arithmetic
        {"name": "plane_run_fp64", "family": "plane_run", "mode": "fp64", "nest": 5, "n": 8321, "delta": 0.02, "steps": 10},
        # the diffusion operator on the cubed sphere, K8 of the great-circle distance
        {"name": "pse_k8", "family": "pse", "mode": "fp32c", "nest": 7, "n": 196610, "op": "k8"},
        # the same in the reference's arithmetic, one refinement coarser
        {"name": "pse_k8_fp64", "family": "pse", "mode": "fp64", "nest": 6, "n": 49154, "op": "k8"},
        # a parameter study: 64 vortices on spheres of uneven refinement, one velocity evaluation
        {"name": "ensemble_64", "family": "ensemble", "mode": "fp32c", "count": 64, "lo": 3, "hi": 6, "mix": 0},
        # the stream functions a run writes at an output time, from the solver's own state
        {"name": "stream_output", "family": "stream", "mode": "fp32c", "nest": 6, "n": 122882},
        # the shallow-water right-hand side in the plane
        {"name": "swe_plane", "family": "swe_plane", "mode": "fp32c", "nest": 6, "n": 33025},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _nest_for(n, counts):
    return next(k for k, c in counts if c >= n)


_ICOS = [(k, 30 * 4 ** k + 2) for k in range(2, 9)]
_CUBED = [(k, 12 * 4 ** k + 2) for k in range(2, 8)]
_QUAD = [(k, 2 * 4 ** (k + 1) + 2 ** (k + 2) + 1) for k in range(2, 8)]


def draw(rng):
    family = rng.choice(["bve", "bve", "bve_run", "plane", "plane_run", "pse", "pse", "ensemble", "stream", "swe_plane"])
    mode = rng.choice(["fp32c", "fp32c", "fp64"])
    if family == "bve":
        n = _log_int(rng, 300, 400000 if mode == "fp32c" else 40000)
        return {"family": family, "mode": mode, "nest": _nest_for(n, _ICOS), "n": n, "block": rng.random() < 0.4}
    if family == "bve_run":
        n = _log_int(rng, 400, 40000 if mode == "fp32c" else 8000)
        return {"family": family, "mode": mode, "nest": _nest_for(n, _ICOS), "n": n, "steps": rng.randint(1, 12)}
    if family == "plane":
        n = _log_int(rng, 300, 131585 if mode == "fp32c" else 33025)
        return {"family": family, "mode": mode, "nest": _nest_for(n, _QUAD), "n": n, "delta": rng.choice([0.0, 0.02])}
    if family == "plane_run":
        n = _log_int(rng, 400, 30000 if mode == "fp32c" else 8321)
        return {"family": family, "mode": mode, "nest": _nest_for(n, _QUAD), "n": n, "delta": 0.02, "steps": rng.randint(1, 12)}
    if family == "pse":
        op = rng.choice(["k8", "k8", "gauss", "gradient", "divergence"])
        n = _log_int(rng, 1000, 196610 if mode == "fp32c" else 49154)
        return {"family": family, "mode": mode, "nest": _nest_for(n, _CUBED), "n": n, "op": op}
    if family == "ensemble":
        lo = rng.randint(3, 5)
        return {"family": family, "mode": "fp32c", "count": _log_int(rng, 4, 64), "lo": lo, "hi": rng.randint(lo, 6),
                "mix": rng.randrange(1, 1000)}
    if family == "stream":
        n = _log_int(rng, 400, 122882)
        return {"family": family, "mode": "fp32c", "nest": _nest_for(n, _ICOS), "n": n}
    n = _log_int(rng, 400, 60000)
    return {"family": family, "mode": "fp32c", "nest": _nest_for(n, _QUAD), "n": n}


# ------------------------------------------------------------------ particle sets
@functools.lru_cache(maxsize=None)
def _mesh(kind, nest):
    if kind == "quad":
        return lg.PolyMesh2d(lg.QUAD_RECT_SEED, nest, 4.0)
    return lg.PolyMesh2d(lg.ICOS_TRI_SPHERE_SEED if kind == "icos" else lg.CUBED_SPHERE_SEED, nest, 1.0)


class _Set:
    """A particle set: a mesh's particles, turned or deformed by the seed, n of them kept in their order."""

    def __init__(self, kind, nest, n, rng):
        m = _mesh(kind, nest)
        if m.spherical:
            r, _ = np.linalg.qr(rng.normal(size=(3, 3)))
            p = np.stack([m.x, m.y, m.z], 1) @ r.T
            p /= np.linalg.norm(p, axis=1, keepdims=True)
            x, y, z = p.T
        else:
            a, b, c, d = rng.uniform(0.0, 2.0 * math.pi, 4)
            x = m.x + 0.03 * np.sin(0.8 * m.y + a) * np.cos(0.6 * m.x + b)
            y = m.y + 0.03 * np.sin(0.8 * m.x + c) * np.cos(0.6 * m.y + d)
            z = m.z
        keep = np.sort(rng.permutation(m.n)[:n]) if n < m.n else slice(None)
        self.x, self.y, self.z, self.area = (np.ascontiguousarray(v[keep]) for v in (x, y, z, m.area))
        self.active = np.ascontiguousarray(m.active[keep])
        self.n = self.x.size
        self.eps_k8 = m.max_edge_length ** 0.75
        self.eps_gauss = 2.0 * m.avg_edge_length
        self.h = m.avg_edge_length


def _vorticity(s, rng):
    """Rossby-Haurwitz wave 4 plus a Gaussian vortex at a random place (the headline's field)."""
    return wl.rh54_vorticity(s) + wl.gaussian_vortex(s, 4.0 * math.pi, 36.0, wl.random_unit_vector(rng))


def _dipoles(s, rng):
    a, b = rng.uniform(-0.3, 0.3, 2)
    return wl.colliding_dipoles(s.x - a, s.y - b, amp=rng.uniform(30.0, 50.0))


def _inputs(case, seed):
    """The host arrays of a case."""
    rng = np.random.default_rng(seed)
    f = case["family"]
    if f == "ensemble":
        mix = np.random.default_rng(case["mix"])  # which refinements: the case's, not the seed's
        out = []
        for _ in range(case["count"]):
            nest = int(mix.integers(case["lo"], case["hi"] + 1))
            s = _Set("icos", nest, 30 * 4 ** nest + 2, rng)
            beta, amp = rng.uniform(2.0, 8.0), rng.uniform(2.0 * math.pi, 6.0 * math.pi)
            zeta = wl.gaussian_vortex(s, amp, beta * beta, wl.random_unit_vector(rng))
            out.append(dict(x=s.x, y=s.y, z=s.z, rel_vort=zeta, area=s.area, active=s.active, radius=1.0,
                            rotation_rate=2.0 * math.pi))
        return out
    kind = {"plane": "quad", "plane_run": "quad", "swe_plane": "quad", "pse": "cubed"}.get(f, "icos")
    s = _Set(kind, case["nest"], case["n"], rng)
    if f in ("plane", "plane_run"):
        s.q = _dipoles(s, rng)
    elif f == "swe_plane":
        s.q = _dipoles(s, rng) / 40.0
        a, b = rng.uniform(0.0, 2.0 * math.pi, 2)
        s.div = 0.3 * np.cos(0.7 * s.x + a) * np.sin(0.9 * s.y + b)
        s.surf = 1.0 + 0.1 * np.exp(-((s.x - 0.5) ** 2 + s.y ** 2)) + 1e-3 * rng.random(s.n)
        s.eps = 2.0 * s.h
    elif f == "pse":
        s.q = wl.y54(s.x, s.y, s.z) + 1e-3 * rng.random(s.n)
        s.eps = s.eps_gauss if case["op"] == "gauss" else s.eps_k8
        if case["op"] == "divergence":
            s.q, s.q2, s.q3 = wl.y54_surface_gradient(s.x, s.y, s.z)
    else:
        s.q = _vorticity(s, rng)
    s.ib, s.ie = (s.n // 3 + 1, s.n // 3 + s.n // 4) if case.get("block") else (1, s.n)
    return s


class _State:
    pass


def prepare(case, seed):
    st = _State()
    st.case, st.s = case, _inputs(case, seed)
    s, f, mode = st.s, case["family"], case["mode"]
    if f == "ensemble":
        st.handle = lg.Ensemble(s, mode=mode)
        return st
    if f in ("bve_run", "stream"):
        st.handle = lg.BVESolver(s.x, s.y, s.z, s.q, s.area, s.active, 1.0, 2.0 * math.pi, mode=mode)
        g = st.handle.get_state()
        st.start = [g[k] for k in ("x", "y", "z", "rel_vort", "u", "v", "w")]
    elif f == "plane_run":
        st.handle = lg.PlaneSolver(s.x, s.y, s.q, s.area, s.active, delta=case["delta"], mode=mode)
        g = st.handle.get_state()
        st.start = [g["u"], g["v"]]
    return st


def _fields(case, arrays):
    """The results as a program of this mode keeps them (see the top)."""
    return [a.astype(np.float32) for a in arrays] if case["mode"] == "fp32c" else list(arrays)


def run(st):
    case, s = st.case, st.s
    f, mode = case["family"], case["mode"]
    if f == "bve":
        out = lg.bve_sphere_velocity(s.x, s.y, s.z, s.q, s.area, s.active, 1.0, s.ib, s.ie, mode=mode)
    elif f == "bve_run":  # back to the run's start, on to its next output
        st.handle.set_state(*st.start)
        st.handle.timestep(0.01, case["steps"], renormalize=mode == "fp32c")
        out = st.handle.get_state().values()
    elif f == "plane":
        out = lg.planar_incompressible_velocity(s.x, s.y, s.q, s.area, s.active, case["delta"], mode=mode)
    elif f == "plane_run":  # a remeshed particle set, on to the next remesh
        st.handle.remesh(s.x, s.y, s.q, s.area, s.active, *st.start)
        st.handle.timestep(0.005, case["steps"])
        out = st.handle.get_state().values()
    elif f == "pse":
        a = (s.x, s.y, s.z, s.q)
        if case["op"] == "gradient":
            out = lg.pse_sphere_gradient_at_particles(*a, s.area, s.active, s.eps, mode=mode)
        elif case["op"] == "divergence":
            out = [lg.pse_sphere_divergence_at_particles(*a, s.q2, s.q3, s.area, s.active, s.eps, mode=mode)]
        else:
            kernel = lg.PSE_GAUSS_CHORD if case["op"] == "gauss" else lg.PSE_K8_GEODESIC
            out = [lg.pse_sphere_laplacian_at_particles(*a, s.area, s.active, s.eps, kernel=kernel, mode=mode)]
    elif f == "ensemble":
        st.handle.velocity()
        g = st.handle.get_state()
        out = [g[k] for k in ("u", "v", "w")]
    elif f == "stream":
        out = st.handle.stream_functions()
    else:
        out = lg.swe_plane_rhs_integrals(s.x, s.y, s.q, s.div, s.surf, s.area, s.active, s.eps, mode=mode)
    return _fields(case, out)


# ------------------------------------------------------------------ what a pass cannot do without
def _pairs(case):
    """Target-source pairs of one evaluation (the meshes' share of active particles: 2/3 icosahedral, 1/2 quadrilateral)."""
    if case["family"] == "ensemble":
        mix = np.random.default_rng(case["mix"])
        nests = [int(mix.integers(case["lo"], case["hi"] + 1)) for _ in range(case["count"])]
        return sum((30.0 * 4 ** k + 2) * 20.0 * 4 ** k for k in nests)
    share = 2.0 / 3.0 if case["family"] in ("bve", "bve_run", "stream") else 0.5
    return float(case["n"]) * (case["n"] // 4 if case.get("block") else case["n"]) * share


def work(case):
    """Flops of the reference's expressions per pair; the PSE sums' over the pairs inside r = 7, where the kernel is not yet zero."""
    f, n = case["family"], case.get("n", 0)
    pairs = _pairs(case)
    if f == "ensemble":
        particles = pairs ** 0.5 * 2.0
        return {"bytes": particles * 8 * 10, "flops": 24.0 * pairs}
    mesh = _mesh("icos" if f in ("bve", "bve_run", "stream") else "cubed" if f == "pse" else "quad", case["nest"])
    if f == "bve":
        return {"bytes": n * 44.0 + (n // 4 if case["block"] else n) * 24.0, "flops": 24.0 * pairs}
    if f == "bve_run":
        return {"bytes": n * 8.0 * 14, "flops": 24.0 * pairs * 4 * case["steps"]}
    if f == "plane":
        return {"bytes": n * (36.0 + 16.0), "flops": 13.0 * pairs}
    if f == "plane_run":
        return {"bytes": n * (52.0 + 32.0), "flops": 13.0 * pairs * 4 * case["steps"]}
    if f == "pse":
        eps = 2.0 * mesh.avg_edge_length if case["op"] == "gauss" else mesh.max_edge_length ** 0.75
        near = 0.5 * (1.0 - math.cos(min(math.pi, 7.0 * eps)))
        per = {"k8": 35.0, "gauss": 14.0, "gradient": 42.0, "divergence": 50.0}[case["op"]]
        outs = 3 if case["op"] == "gradient" else 1
        return {"bytes": n * (44.0 + (16.0 if case["op"] == "divergence" else 0.0) + 8.0 * outs), "flops": per * pairs * near}
    if f == "stream":
        return {"bytes": n * 8.0 * 7, "flops": 30.0 * pairs}
    near = min(1.0, math.pi * (14.0 * mesh.avg_edge_length) ** 2 / 64.0)
    return {"bytes": n * (52.0 + 32.0), "flops": 45.0 * pairs + 30.0 * pairs * near}


# ------------------------------------------------------------------ the same in 64 bits, by torch
def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def _rows(nt, ns):
    step = max(1, int(1.2e8 // max(1, ns)))
    return [(a, min(nt, a + step)) for a in range(0, nt, step)]


def _no_self(w, tgt, src):
    """Zero where a row's particle is its column's (both ascending)."""
    k = torch.searchsorted(src, tgt).clamp_(max=src.numel() - 1)
    hit = src[k] == tgt
    w[hit.nonzero()[:, 0], k[hit]] = 0.0


def _sq_dist(p, q):
    d = (p[:, :1] - q[:, 0]).square_()
    for c in range(1, p.shape[1]):
        d += (p[:, c:c + 1] - q[:, c]).square_()
    return d


def _bve_sum(p, zeta, area, src, lo, hi):
    """u_i = x_i x sum_j x_j w_ij, w_ij = -zeta_j A_j / (4 pi (1 - x_i.x_j)), with 1 - x_i.x_j = (|d|^2 - c_i - c_j) / 2."""
    q, c = p[src], p.square().sum(1) - 1.0
    s = -zeta[src] * area[src] / (2.0 * math.pi)
    out = torch.empty(hi - lo, 3, dtype=torch.float64, device="cuda")
    for a, b in _rows(hi - lo, src.numel()):
        t = torch.arange(lo + a, lo + b, device="cuda")
        w = _sq_dist(p[t], q).sub_(c[t, None]).sub_(c[src])
        w = s / w
        _no_self(w, t, src)
        out[a:b] = torch.linalg.cross(p[t], w @ q)
    return out


def _plane_sum(p, omega, area, src, delta):
    s = omega[src] * area[src] / (2.0 * math.pi)
    out = torch.empty(p.shape[0], 2, dtype=torch.float64, device="cuda")
    for a, b in _rows(p.shape[0], src.numel()):
        t = torch.arange(a, b, device="cuda")
        w = s / _sq_dist(p[t], p[src]).add_(delta * delta)
        _no_self(w, t, src)
        out[a:b, 0] = -(w * (p[t, 1:] - p[src, 1])).sum(1)
        out[a:b, 1] = (w * (p[t, :1] - p[src, 0])).sum(1)
    return out


def _rk4_bve(case, s):
    p, zeta, area = torch.stack([_dev(v) for v in (s.x, s.y, s.z)], 1), _dev(s.q), _dev(s.area)
    src = torch.from_numpy(np.flatnonzero(s.active)).cuda()
    dt, two_omega, n = 0.01, 4.0 * math.pi, s.n
    on = (lambda v: v / v.norm(dim=1, keepdim=True)) if case["mode"] == "fp32c" else (lambda v: v)
    u = _bve_sum(p, zeta, area, src, 0, n)
    for _ in range(case["steps"]):
        k, l = [dt * u], [-dt * two_omega * u[:, 2]]
        for h in (0.5, 0.5, 1.0):
            us = _bve_sum(on(p + h * k[-1]), zeta + h * l[-1], area, src, 0, n)
            k.append(dt * us)
            l.append(-dt * two_omega * us[:, 2])
        p = on(p + k[0] / 6 + k[1] / 3 + k[2] / 3 + k[3] / 6)
        zeta = zeta + l[0] / 6 + l[1] / 3 + l[2] / 3 + l[3] / 6
        u = _bve_sum(p, zeta, area, src, 0, n)
    return [*p.T, zeta, *u.T]


def _rk4_plane(case, s):
    p, omega, area = torch.stack([_dev(s.x), _dev(s.y)], 1), _dev(s.q), _dev(s.area)
    src = torch.from_numpy(np.flatnonzero(s.active)).cuda()
    dt, vel = 0.005, lambda v: _plane_sum(v, omega, area, src, case["delta"])
    u = vel(p)
    for _ in range(case["steps"]):
        k = [dt * u]
        for h in (0.5, 0.5, 1.0):
            k.append(dt * vel(p + h * k[-1]))
        p = p + k[0] / 6 + k[1] / 3 + k[2] / 3 + k[3] / 6
        u = vel(p)
    return [*p.T, *u.T]


def _k8(r2):
    return torch.exp(-r2) * (40.0 - 40.0 * r2 + 10.0 * r2 ** 2 - (2.0 / 3.0) * r2 ** 3) / math.pi


def _pse(case, s):
    p, q = torch.stack([_dev(v) for v in (s.x, s.y, s.z)], 1), _dev(s.q)
    src = torch.from_numpy(np.flatnonzero(s.active)).cuda()
    ps, area, eps, op = p[src], _dev(s.area)[src], s.eps, case["op"]
    out = torch.empty(s.n, 3 if op == "gradient" else 1, dtype=torch.float64, device="cuda")
    if op == "divergence":
        vec = torch.stack([q, _dev(s.q2), _dev(s.q3)], 1)
    for a, b in _rows(s.n, src.numel()):
        t = p[a:b]
        d2 = _sq_dist(t, ps)
        if op == "gauss":
            r2 = d2 / eps ** 2
            w = torch.exp(-r2) * (4.0 / math.pi)
        else:
            r2 = (2.0 * torch.asin((0.5 * d2.sqrt()).clamp_(max=1.0)) / eps).square_()
            w = _k8(r2) if op == "k8" else _k1(r2)
        w *= area
        if op in ("k8", "gauss"):
            out[a:b, 0] = ((q[src] - q[a:b, None]) * w).sum(1) / eps ** 4
            continue
        if op == "gradient":
            w *= q[src] + q[a:b, None]
            g = t * w.sum(1, keepdim=True) - w @ ps
            out[a:b] = (g - t * (g * t).sum(1, keepdim=True)) / eps ** 4
        else:  # sum_j w (P_i (x_i - x_j)) . (V_j + V_i)
            tot = torch.zeros(b - a, dtype=torch.float64, device="cuda")
            radial = d2 / 2.0  # (x_i - x_j).x_i on the unit sphere
            for c in range(3):
                tot += ((t[:, c:c + 1] - ps[:, c] - radial * t[:, c:c + 1]) * (vec[src, c] + vec[a:b, c:c + 1]) * w).sum(1)
            out[a:b, 0] = tot / eps ** 4
    return list(out.T)


def _k1(r2):
    """The first-derivative kernel of eighth order, without its factor r."""
    return -torch.exp(-r2) * (20.0 - 20.0 * r2 + 5.0 * r2 ** 2 - r2 ** 3 / 3.0) / math.pi


def _stream(s):
    p, area = torch.stack([_dev(v) for v in (s.x, s.y, s.z)], 1), _dev(s.area)
    rel = _dev(s.q)
    both = torch.stack([rel, rel + 4.0 * math.pi * p[:, 2]], 1) * area[:, None] / (-4.0 * math.pi)
    src = torch.from_numpy(np.flatnonzero(s.active)).cuda()
    c = p.square().sum(1) - 1.0
    out = torch.empty(s.n, 2, dtype=torch.float64, device="cuda")
    for a, b in _rows(s.n, src.numel()):
        t = torch.arange(a, b, device="cuda")
        g = _sq_dist(p[t], p[src]).sub_(c[t, None]).sub_(c[src]).mul_(0.5).log_()
        _no_self(g, t, src)
        out[a:b] = g @ both[src]
    return list(out.T)


def _swe_plane(s):
    p, area = torch.stack([_dev(s.x), _dev(s.y)], 1), _dev(s.area)
    src = torch.from_numpy(np.flatnonzero(s.active)).cuda()
    w, d, h = _dev(s.q)[src] * area[src] / (2.0 * math.pi), _dev(s.div)[src] * area[src] / (2.0 * math.pi), _dev(s.surf)
    out = torch.empty(s.n, 4, dtype=torch.float64, device="cuda")
    for a, b in _rows(s.n, 2 * src.numel()):
        t = torch.arange(a, b, device="cuda")
        dx, dy = p[t, :1] - p[src, 0], p[t, 1:] - p[src, 1]
        r2 = dx.square() + dy.square()
        inv = 1.0 / r2
        _no_self(inv, t, src)
        P, Q = (d * dx - w * dy) * inv, (w * dx + d * dy) * inv
        out[a:b, 0], out[a:b, 1] = P.sum(1), Q.sum(1)
        ux, uy = (d * inv - 2.0 * dx * P * inv).sum(1), (-w * inv - 2.0 * dy * P * inv).sum(1)
        vx, vy = (w * inv - 2.0 * dx * Q * inv).sum(1), (d * inv - 2.0 * dy * Q * inv).sum(1)
        out[a:b, 2] = ux * ux + 2.0 * uy * vx + vy * vy
        out[a:b, 3] = ((h[src] - h[t, None]) * area[src] * _k8(r2 / s.eps ** 2)).sum(1) / s.eps ** 4
    return list(out.T)


def exact(case, seed):
    f = case["family"]
    if _pairs(case) * (4 * case["steps"] if "steps" in case else 1) > EXACT_PAIRS:
        return None
    s = _inputs(case, seed)
    if f == "ensemble":
        parts = []
        for d in s:
            p = torch.stack([_dev(d[k]) for k in ("x", "y", "z")], 1)
            src = torch.from_numpy(np.flatnonzero(d["active"])).cuda()
            parts.append(_bve_sum(p, _dev(d["rel_vort"]), _dev(d["area"]), src, 0, p.shape[0]))
        return list(torch.cat(parts).T)
    if f == "bve":
        p = torch.stack([_dev(v) for v in (s.x, s.y, s.z)], 1)
        src = torch.from_numpy(np.flatnonzero(s.active)).cuda()
        out = torch.zeros(s.n, 3, dtype=torch.float64, device="cuda")
        out[s.ib - 1:s.ie] = _bve_sum(p, _dev(s.q), _dev(s.area), src, s.ib - 1, s.ie)
        return list(out.T)
    if f == "bve_run":
        return _rk4_bve(case, s)
    if f == "plane":
        p = torch.stack([_dev(s.x), _dev(s.y)], 1)
        src = torch.from_numpy(np.flatnonzero(s.active)).cuda()
        return list(_plane_sum(p, _dev(s.q), _dev(s.area), src, case["delta"]).T)
    if f == "plane_run":
        return _rk4_plane(case, s)
    if f == "pse":
        return _pse(case, s)
    if f == "stream":
        return _stream(s)
    return _swe_plane(s)
