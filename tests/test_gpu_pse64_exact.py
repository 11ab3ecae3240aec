"""The FP64 PSE sums' error against the same sums in extended precision (numpy's long double, 64 or more bits
of mantissa), beside that of the reference's own FP64 expressions (the oracle): particles on the sphere to their
rounding, off it by more and by different amounts, on the Earth's, and in the plane.  Bound: no larger than the
reference expressions', in the mean square over the targets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = np.longdouble
PI = L("3.14159265358979323846264338327950288")


@pytest.fixture(scope="module")
def lg(built_lib):
    return built_lib


def _k8(r2):
    return np.exp(-r2) * (40 - 40 * r2 + 10 * r2**2 - 2 * r2**3 / 3) / PI


def _k1(r2):
    return -np.exp(-r2) * (20 - 20 * r2 + 5 * r2**2 - r2**3 / 3) / PI


def _exact(p, fields, area, src, targets, eps, radius, op):
    """The sums of the targets; pairs beyond r = 8 (each below e^-64) left out."""
    q, eps, out = p[:, src], L(eps), []
    for i in targets:
        x = p[:, i]
        near = np.flatnonzero(((q - x[:, None]) ** 2).sum(0) <= (1.2 * 8 * float(eps)) ** 2)
        s, x, a, v = q[:, near].astype(L), x.astype(L), area[src[near]].astype(L), [f[src[near]].astype(L) for f in fields]
        d = x[:, None] - s
        if op == "plane":
            r2 = (d * d).sum(0) / eps**2
        else:
            c = np.stack([x[k - 2] * s[k - 1] - x[k - 1] * s[k - 2] for k in range(3)])
            r2 = (np.arctan2(np.sqrt((c * c).sum(0)), (x[:, None] * s).sum(0)) * L(radius) / eps) ** 2
        if op in ("k8", "plane"):
            out.append([((v[0] - fields[0][i]) * a * _k8(r2)).sum() / eps**4])
            continue
        w = a * _k1(r2)
        if op == "grad":
            g = (d * ((v[0] + fields[0][i]) * w)).sum(1)
            out.append(list((g - x * (x * g).sum()) / eps**4))
        else:
            t = d - x[:, None] * (x[:, None] * d).sum(0)
            out.append([sum(((v[k] + fields[k][i]) * t[k] * w).sum() for k in range(3)) / eps**4])
    return np.array(out).T


def _sphere_set(lg, kind):
    m = lg.PolyMesh2d(lg.CUBED_SPHERE_SEED, 5, 1.0)
    rng = np.random.default_rng(7)
    turn, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    p = turn @ np.stack([m.x, m.y, m.z])
    p /= np.linalg.norm(p, axis=0)
    radius = 6.37122e6 if kind == "earth" else 1.0
    if kind == "off":
        p = p * (1.0 + 1e-7 * rng.normal(size=m.n))
    p = np.ascontiguousarray(p * radius)
    x, y, z = p / radius
    fields = [x * y * z + x, y * z - 0.3 * x, x - y * y]
    eps = float(m.max_edge_length**0.75 * radius)
    return p, fields, m.area * radius**2, m.active, eps, radius


def _check(got, ref, exact):
    rms = [float(np.sqrt(np.mean(np.asarray((np.asarray(v) - exact), dtype=np.float64) ** 2))) for v in (got, ref)]
    assert rms[0] <= rms[1], rms


# (the derivatives' SphereProjection is the unit sphere's)
@pytest.mark.parametrize("kind, op", [("on", "k8"), ("on", "grad"), ("on", "div"), ("off", "k8"), ("off", "grad"),
                                      ("off", "div"), ("earth", "k8")])
def test_sphere(lg, oracle_mod, kind, op):
    p, fields, area, active, eps, radius = _sphere_set(lg, kind)
    n = p.shape[1]
    targets = np.sort(np.random.default_rng(1).permutation(n)[:250])
    args = (area, active, eps, radius)
    if op == "k8":
        ref = oracle_mod.pse_laplacian(*p, fields[0], *args, kernel=0)
        got = lg.pse_sphere_laplacian_at_particles(*p, fields[0], *args, mode="fp64")
    elif op == "grad":
        ref = oracle_mod.pse_sphere_gradient(*p, fields[0], *args)
        got = lg.pse_sphere_gradient_at_particles(*p, fields[0], *args, mode="fp64")
    else:
        ref = oracle_mod.pse_sphere_divergence(*p, *fields, *args)
        got = lg.pse_sphere_divergence_at_particles(*p, *fields, *args, mode="fp64")
    exact = _exact(p, fields, area, np.flatnonzero(active), targets, eps, radius, op)
    _check(np.atleast_2d(got)[:, targets], np.atleast_2d(ref)[:, targets], exact)


def test_plane(lg, oracle_mod):
    m = lg.PolyMesh2d(lg.QUAD_RECT_SEED, 5, 4.0)
    f, eps = m.x * m.y + 0.1 * m.x**3, 0.3
    targets = np.sort(np.random.default_rng(2).permutation(m.n)[:250])
    ref = oracle_mod.pse_laplacian(m.x, m.y, np.zeros(m.n), f, m.area, m.active, eps, kernel=2)
    got = lg.pse_plane_laplacian_at_particles(m.x, m.y, f, m.area, m.active, eps, mode="fp64")
    exact = _exact(np.stack([m.x, m.y, np.zeros(m.n)]), [f], m.area, np.flatnonzero(m.active), targets, eps, 1.0, "plane")
    _check(np.atleast_2d(got)[:, targets], np.atleast_2d(ref)[:, targets], exact)
