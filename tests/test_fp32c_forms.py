"""CPU checks of the forms that the present sweeps evaluate: the curve on the cube's faces (csrc/hilbert.cuh,
compiled for the host), the polynomials (their coefficients read from the sources), the basis form of the sphere
velocity with its compact near form (csrc/bve_rel.cuh), the log1p form of the sphere stream functions
(csrc/stream_rel.cuh), the Laplacians' pair (csrc/pse_lap.cuh) and the four sums of the planar shallow-water
integrals (csrc/plane_rel.cuh).  float32 numpy rounds each addition and product as the GPU does; a fused multiply-add is
computed in float64 and rounded.  The GPU tests hold the kernels themselves to the oracle."""
import ctypes
import re
import subprocess

import numpy as np
import pytest

from conftest import PKG
from test_fp32c_arithmetic import _fma, _rcp, _split2, _two_sum

F, D, L = np.float32, np.float64, np.longdouble


# ------------------------------------------------------------------ the curve
@pytest.fixture(scope="module")
def curve(tmp_path_factory):
    d = tmp_path_factory.mktemp("curve")
    (d / "t.cpp").write_text('''
#define __host__
#define __device__
#include "hilbert.cuh"
extern "C" void keys(long n, const float* p, int bits, uint32_t* k) {
  for (long i = 0; i < n; ++i) k[i] = lpm::sphere_curve_index(p[3 * i], p[3 * i + 1], p[3 * i + 2], bits);
}
''')
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", str(PKG / "csrc"),
                    str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    fn = ctypes.CDLL(str(d / "t.so")).keys

    def keys(p, bits):
        p = np.ascontiguousarray(p, dtype=F)
        k = np.empty(len(p), np.uint32)
        fn(ctypes.c_long(len(p)), p.ctypes.data_as(ctypes.c_void_p), bits, k.ctypes.data_as(ctypes.c_void_p))
        return k

    return keys


def _face_cells(m):
    """The centres of m x m cells on each of the cube's faces, as directions."""
    w = (np.arange(m) + 0.5) * 2.0 / m - 1.0
    u = np.sign(w) * (1.273 - np.sqrt(1.273**2 - 4 * 0.273 * np.abs(w))) / (2 * 0.273)  # u (1.273 - 0.273 |u|) = w
    a, b = (v.ravel() for v in np.meshgrid(u, u))
    out = []
    for axis in range(3):
        for sign in (-1.0, 1.0):
            p = np.empty((m * m, 3))
            p[:, axis], p[:, axis - 2], p[:, axis - 1] = sign, a, b
            out.append(p)
    return np.concatenate(out)


def test_curve_visits_neighbouring_cells(curve):
    m = 16
    p = _face_cells(m)
    k = curve(p, 3 + 8)  # 16 x 16 cells a face
    assert np.array_equal(np.sort(k), np.arange(6 * m * m))
    p = p[np.argsort(k)] / np.linalg.norm(p[np.argsort(k)], axis=1, keepdims=True)
    step = np.linalg.norm(np.diff(p, axis=0), axis=1)
    assert step.max() <= 1.75 * (np.pi / 2) / m  # the next cell, also where one face's curve ends and the next starts
    faces = np.argsort(k) // (m * m)
    assert len(set(faces)) == 6 and np.count_nonzero(np.diff(faces)) == 5


def test_curve_widths_and_odd_directions(curve):
    p = np.random.default_rng(1).normal(size=(5000, 3))
    assert np.array_equal(curve(p, 27) >> 4, curve(p, 23))
    assert np.array_equal(curve(p * 2.0**20, 23), curve(p, 23))  # of a direction
    odd = np.array([[0, 0, 0], [np.nan, 0, 1], [np.nan] * 3, [np.inf, 1, 1], [1, -1, 1], [0, 0, -1]])
    assert np.all(curve(odd, 23) < (6 << 20))


# ------------------------------------------------------------------ the polynomials
def _coefficients(name, file):
    text = re.search(r"\b%s\[\d+\]\s*=\s*\{([^}]*)\}" % name, (PKG / "csrc" / file).read_text()).group(1)
    one = lambda t: float.fromhex(t) if "0x" in t else float(t.rstrip("f"))
    return [one(t.strip()) for t in text.split(",")]


@pytest.mark.parametrize("name, limit", [("c6", 0.1375), ("c9", 0.3125), ("c12", 0.46)])
def test_log1p_polynomials(name, limit):
    x = np.linspace(-limit, limit, 20001)
    q = np.polyval(np.array(_coefficients(name, "stream_rel.cuh"), F).astype(D)[::-1], x)
    assert np.abs(x + x * x * q - np.log1p(x)).max() <= 4.2e-9


@pytest.mark.parametrize("name, top, bound", [("kNear", 0.2, 4.5e-9), ("kFar", 1.3, 6.8e-9)])
def test_laplacian_angle_polynomials(name, top, bound):
    c = _coefficients(name, "sums.cu")
    v = np.linspace(1e-6, top, 20001)
    exact = 4 * np.arcsin(np.sqrt(v) / 2) ** 2
    assert np.abs(v * np.polyval(c[::-1], v) / exact - 1).max() <= bound
    w = np.linspace(top, 4.0, 2001)  # beyond, where the kernel is zero, only monotonic
    assert np.all(np.diff(w * np.polyval(c[::-1], w)) > 0)


@pytest.mark.parametrize("name, chord", [("kAngleNear", 0.45), ("kAngleFar", 1.14), ("kAngleWide", np.sqrt(2.0))])
def test_fp64_angle_polynomials(name, chord):
    c = [L(v) for v in _coefficients(name, "pse64.cuh")]
    v = np.linspace(L(1e-4), L(chord) ** 2, 4001)
    p = np.zeros_like(v)
    for k in c[::-1]:
        p = p * v + k
    exact = 4 * np.arcsin(np.sqrt(v) / 2) ** 2
    assert np.abs(v * p / exact - 1).max() <= 2.0**-56.5


# ------------------------------------------------------------------ sphere velocity
def _dot(h, l, e):
    """h . e + l . e as float32 pairs, the products' and sums' errors carried."""
    s, err = np.zeros(h.shape[:-1], F), np.zeros(h.shape[:-1], F)
    for k in range(3):
        p = h[..., k] * e[k]
        s, q = _two_sum(s, p)
        err = err + (q + _fma(h[..., k], e[k], -p) + l[..., k] * e[k])
    return s, err


def _group(P, S):
    """Origin, radius, basis and records of one group (unit-scaled positions, strengths)."""
    ph, pl = _split2(P)
    o = ph.mean(0, dtype=F)
    d = (ph - o) + pl
    R = F(np.sqrt((d * d).sum(1).max()) * F(1.000001))
    spc = F(((d[1:] - d[:-1]) ** 2).sum(1).min()) if len(P) > 1 else F(3e38)
    c = np.einsum("ij,ij->i", P, P) - 1.0
    g = dict(o=o, S=S.astype(F), nc=(-c).astype(F), compact=bool(R <= 0.5 and R <= 32 * np.sqrt(spc)))
    if g["compact"]:
        hi = (ph - o) + pl
        lo = ((ph - o) - hi) + pl
    else:
        off = P - o.astype(D)
        hi, lo = _split2(off)
    g["hi"], g["lo"] = hi, lo
    k = int(np.argmin(np.abs(o)))
    u = np.cross(o, np.eye(3, dtype=F)[k]).astype(F)
    e1 = (u / F(np.linalg.norm(u))).astype(F)
    w = np.cross(o, e1).astype(F)
    e2 = (w / F(np.linalg.norm(w))).astype(F)
    od, e1d, e2d = o.astype(D), e1.astype(D), e2.astype(D)
    k1, k2, g11, g12, g22 = (F(v) for v in (od @ e1d, od @ e2d, e1d @ e1d - 1, e1d @ e2d, e2d @ e2d - 1))
    g["k"] = F(-0.5 * (od @ od - 1.0))
    io2 = F(1) / F(od @ od)
    a0, b0, so = _dot(hi, lo, e1), _dot(hi, lo, e2), _dot(hi, lo, o)
    c0 = so[0] * io2
    af = a0[0] + (a0[1] - (a0[0] * g11 + b0[0] * g12 + c0 * k1))
    bf = b0[0] + (b0[1] - (a0[0] * g12 + b0[0] * g22 + c0 * k2))
    cf = (so[0] + (so[1] - (af * k1 + bf * k2))) * io2
    half = 0.5 * S
    g.update(e1=e1, e2=e2, k1=k1, k2=k2, a=af, b=bf, c=cf, W=(half * (1 + cf.astype(D))).astype(F),
             A=(-half * af.astype(D)).astype(F), B=(-half * bf.astype(D)).astype(F))
    r = (F(1.25 if R <= F(0.2) else 1.5) / F(3)) * R if g["compact"] else R
    g["near"] = F(3) * max(r, F(0.5) * np.sqrt(np.abs(g["k"])))
    return g


def _warp_velocity(T, groups, rng):
    """D = sum_j S_j d / q (up to a multiple of the target) for one warp's targets."""
    th, tl = _split2(T)
    nc = (1.0 - np.einsum("ij,ij->i", T, T)).astype(F) + F(2.0**-100)
    hi, lo = np.zeros((len(T), 3), F), np.zeros((len(T), 3), F)
    taken = dict(far=0, compact=0, near=0)
    for g in groups:
        t = (th - g["o"]) + tl
        n2 = _fma(t[:, 2], t[:, 2], _fma(t[:, 1], t[:, 1], t[:, 0] * t[:, 0]))
        if not np.any(n2 < g["near"] * g["near"]):
            taken["far"] += 1
            nq = n2 + nc
            cc, ga = _fma(nq, F(0.5), g["k"]), _fma(nq, F(-0.5), F(1) - g["k"])
            al, be = np.full(len(T), g["k1"]), np.full(len(T), g["k2"])
            for k in range(3):
                al, be = _fma(t[:, k], g["e1"][k], al), _fma(t[:, k], g["e2"][k], be)
            h = _fma(ga[:, None], -g["c"], cc[:, None])
            h = _fma(be[:, None], -g["b"], _fma(al[:, None], -g["a"], h))
            inv = _rcp(h, rng)
            W, A, B = (np.cumsum(inv * g[v], axis=1, dtype=F)[:, -1:] for v in ("W", "A", "B"))
            part = g["e1"] * A + (g["e2"] * B + t * W)
        else:
            taken["compact" if g["compact"] else "near"] += 1
            if g["compact"]:
                d = t[:, None, :] - g["hi"]
            else:
                uh, ul = _split2(T - g["o"].astype(D))
                d = (uh[:, None, :] - g["hi"]) + (ul[:, None, :] - g["lo"])
            q = _fma(d[..., 2], d[..., 2], _fma(d[..., 1], d[..., 1], d[..., 0] * d[..., 0])) + (nc[:, None] + g["nc"])
            w = g["S"] * _rcp(q, rng)
            part = np.cumsum(d * w[..., None], axis=1, dtype=F)[:, -1]
        hi, e = _two_sum(hi, part.astype(F))
        lo = lo + e
    return hi.astype(D) + lo.astype(D), taken


@pytest.mark.parametrize("nest, off", [(4, 0.0), (5, 0.0), (5, 1e-7)])
def test_basis_form_of_the_sphere_velocity(built_lib, oracle_mod, curve, nest, off):
    import workloads
    m = workloads.config_rh54_icos(nest)
    P = np.stack([m["x"], m["y"], m["z"]], 1)
    P = P * (1.0 + off * np.random.default_rng(5).standard_normal(len(P)))[:, None]
    src = np.flatnonzero(m["active"])
    src = src[np.argsort(curve(P[src], 23), kind="stable")]
    S = -m["zeta"] * m["area"] / (2 * np.pi)
    groups = [_group(P[src[i:i + 128]], S[src[i:i + 128]]) for i in range(0, len(src), 128)]
    rng, ref_max = np.random.default_rng(2), 0.0
    taken, err = dict(far=0, compact=0, near=0), 0.0
    for ib in range(0, len(P) - 192, len(P) // 7):
        T = P[ib:ib + 192]
        got, n = _warp_velocity(T, groups, rng)
        taken = {k: taken[k] + n[k] for k in taken}
        ref = np.stack(oracle_mod.bve_velocity(*(np.ascontiguousarray(v) for v in P.T), m["zeta"], m["area"], m["active"],
                                               ib=ib, ie=ib + 192), 1)
        err = max(err, np.abs(np.cross(got, T) - ref).max())
        ref_max = max(ref_max, np.abs(ref).max())
    assert taken["far"] > 0 and taken["compact"] > 0
    assert err <= 1e-6 * ref_max


# ------------------------------------------------------------------ sphere stream functions
def _log1p_degree(distance):
    """The degree that a group at this distance takes (None: a log per pair), with its sum held to the exact one."""
    rng = np.random.default_rng(int(1000 * distance))
    v = rng.uniform(-0.05, 0.05, (2, 64))
    p = np.stack([np.ones(64), *v], 1)
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    t = np.array([np.cos(distance), np.sin(distance) * 0.6, np.sin(distance) * 0.8])
    S = rng.uniform(0.5, 1.5, 64) / 64
    g = _group(p, S)
    o, e1, e2 = (g[k].astype(D) for k in ("o", "e1", "e2"))
    C = 1.0 - t @ o
    ga, al, be = (F(v / C) for v in (t @ o, t @ e1, t @ e2))
    x0 = F((C - D(F(C))) / C)
    x = _fma(be, -g["b"], _fma(al, -g["a"], _fma(ga, -g["c"], np.full(64, x0))))
    degree = next((n for n, limit in ((6, 0.1375), (9, 0.3125), (12, 0.46)) if np.abs(x).max() <= limit), None)
    if degree is not None:
        q = np.array(_coefficients("c%d" % degree, "stream_rel.cuh"), F)
        y = np.full(64, q[-1])
        for k in q[-2::-1]:
            y = _fma(y, x, np.full(64, k))
        y = _fma(x * x, y, x)
        got = np.log(2 * D(F(C))) * S.sum() + (g["S"] * y).sum(dtype=D)
        ref = (S * np.log(2 * (1.0 - p @ t))).sum()
        assert abs(got - ref) <= 3e-8 * S.sum()
    return degree


def test_log1p_form_of_far_groups():
    """sum S ln q over a group = ln(2 C) sum S + sum S log1p(x), by the lowest degree whose range holds every x."""
    degrees = [_log1p_degree(d) for d in np.geomspace(0.2, 3.0, 60)]
    assert set(degrees) == {None, 12, 9, 6}


# ------------------------------------------------------------------ Laplacians
@pytest.mark.parametrize("mean", [0.0, 1.0, 1e6])
def test_field_difference_of_the_laplacians_pair(mean):
    """F_j - F_i from float pairs of the field less the group's constant; a particle's own pair is zero."""
    rng = np.random.default_rng(3)
    f = mean + rng.normal(size=64)
    fh, fl = _split2(f)
    s, e = _two_sum(fh, np.full(64, -fh[0]))  # the records'
    fs, fe = _two_sum(s, e + fl)
    s, e = _two_sum(np.full(64, fh[0]), -fh)  # the targets'
    r = e - fl
    nf = s + r
    nl = r - (nf - s)
    m = (fs + nf[:, None]) + (fe + nl[:, None])
    assert np.all(np.diag(m) == 0.0)
    exact = f - f[:, None]
    assert np.abs(m - exact).max() <= 2.0**-23 * np.abs(exact).max() + 2.0**-47 * abs(mean)


def test_laplacian_kernel_in_the_exponents_unit():
    """40 - 40 r^2 + 10 r^4 - (2/3) r^6 at y = -r^2 log2 e, with the sweep's float constants."""
    text = (PKG / "csrc" / "pse_lap.cuh").read_text()
    body = text[text.index("lap_kernel(float2 y)"):]
    c = [D(F(float(v))) for v in re.findall(r"make_float2\(([\d.]+)f, [\d.]+f\)", body)[:4]]  # of y^3, y^2, y, 1
    r2 = np.linspace(0.0, 49.0, 5001)
    y = -r2 / np.log(2.0)
    got, ref = np.exp2(y) * np.polyval(c, y), np.exp(-r2) * (40 - 40 * r2 + 10 * r2**2 - 2 * r2**3 / 3)
    assert np.abs(got - ref).max() <= 1e-6 * 40


# ------------------------------------------------------------------ planar shallow water
def test_four_sums_of_the_planar_swe_integrals(oracle_mod):
    """u, v and the double dot product 2 (ux^2 + vx^2) from p = dx / r^2, q = -dy / r^2, in FP64."""
    rng = np.random.default_rng(4)
    n = 300
    x, y = rng.uniform(-2, 2, (2, n))
    vort, div, area, act = rng.normal(size=n), rng.normal(size=n), rng.uniform(0.5, 1.5, n) / n, (rng.random(n) < 0.6).astype(np.int32)
    ref = oracle_mod.swe_plane_rhs(x, y, vort, div, np.zeros(n), area, act, 0.3)
    src = np.flatnonzero(act)
    W, V = vort[src] * area[src] / (2 * np.pi), div[src] * area[src] / (2 * np.pi)
    dx, dy = x[:, None] - x[src], y[:, None] - y[src]
    r2 = dx * dx + dy * dy
    s = np.where(r2 > 0, 1.0 / np.where(r2 > 0, r2, 1.0), 0.0)
    p, q = s * dx, -s * dy
    a, t = s - 2 * q * q, -2 * p * q
    u, v = (V * p + W * q).sum(1), (W * p - V * q).sum(1)
    nux, nvx = (V * a - W * t).sum(1), (W * a + V * t).sum(1)
    for got, r in zip((u, v, 2 * (nux**2 + nvx**2)), ref):
        assert np.abs(got - r).max() <= 1e-12 * np.abs(r).max()
