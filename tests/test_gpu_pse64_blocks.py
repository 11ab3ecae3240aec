"""The FP64 PSE sums of a block of targets, or of a batch of query points, are those of the whole set bit for
bit: a target's sum depends on the sources alone.  Sets on one sphere, on shells of several radii with particles at
the centre (whose pairs take the reference's expressions), and in the plane; the shells against the oracle too
(1e-12 of the largest value, the bound of the FP64 mode's PSE sums)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 30000  # blocks of every lane count of the whole set's rule
BLOCKS = [(1, 33), (200, 5000), (9000, 24000), (29990, 30000)]


@pytest.fixture(scope="module")
def lg(built_lib):
    return built_lib


def _set(kind):
    rng = np.random.default_rng(11)
    if kind == "plane":
        p = np.stack([*rng.uniform(-4.0, 4.0, (2, N)), np.zeros(N)])
    else:
        p = rng.normal(size=(3, N))
        p /= np.linalg.norm(p, axis=0)
        if kind == "shells":
            p *= rng.choice([0.5, 1.0, 1.0 + 1e-9, 1.1, 1.3, 4.0], N)
            p[:, [77, 15000, 29995]] = 0.0
    f = rng.normal(size=(4, N))
    return np.ascontiguousarray(p), f, rng.uniform(0.5, 1.5, N) / N, (rng.random(N) < 0.5).astype(np.int32)


def _operators(lg, kind, p, f, area, active):
    x, y, z = p
    if kind == "plane":
        a = (area, active, 0.12)
        return {
            "k8": lambda **k: lg.pse_plane_laplacian_at_particles(x, y, f[0], *a, mode="fp64", **k),
            "gauss": lambda **k: lg.pse_plane_laplacian_at_particles(x, y, f[0], *a, kernel=1, mode="fp64", **k),
            "gradient": lambda **k: lg.pse_plane_gradient_at_particles(x, y, f[0], *a, **k),
            "second": lambda **k: lg.pse_plane_second_partials_at_particles(x, y, f[0], f[1], *a, **k),
            "ddot": lambda **k: lg.pse_plane_double_dot_product_at_particles(x, y, f[0], f[1], *a, **k),
        }
    a = (area, active, 0.05)
    return {
        "k8": lambda **k: lg.pse_sphere_laplacian_at_particles(x, y, z, f[0], *a, mode="fp64", **k),
        "gauss": lambda **k: lg.pse_sphere_laplacian_at_particles(x, y, z, f[0], *a, kernel=1, mode="fp64", **k),
        "gradient": lambda **k: lg.pse_sphere_gradient_at_particles(x, y, z, f[0], *a, mode="fp64", **k),
        "divergence": lambda **k: lg.pse_sphere_divergence_at_particles(x, y, z, *f[:3], *a, mode="fp64", **k),
        "ddot": lambda **k: lg.pse_sphere_double_dot_product_at_particles(x, y, z, *f[:3], *a, **k),
    }


@pytest.mark.parametrize("kind", ["sphere", "shells", "plane"])
def test_blocks_of_targets(lg, kind):
    for name, op in _operators(lg, kind, *_set(kind)).items():
        whole = np.stack(np.atleast_2d(op()))
        for ib, ie in BLOCKS:
            part = np.stack(np.atleast_2d(op(i_begin=ib, i_end=ie)))
            assert np.array_equal(part[:, ib - 1:ie], whole[:, ib - 1:ie]), (name, ib, ie)


@pytest.mark.parametrize("kind", ["sphere", "plane"])
def test_batches_of_query_points(lg, kind):
    p, f, area, active = _set(kind)
    rng = np.random.default_rng(3)
    q = rng.normal(size=(3, 20000))
    if kind == "sphere":
        q /= np.linalg.norm(q, axis=0)
        kw = dict(geometry=lg.GEOMETRY_SPHERE)
    else:
        q[2] = 0.0
        kw = dict(geometry=lg.GEOMETRY_PLANE)
    call = lambda s: lg.pse_interpolate_scalar(*p, f[0], area, active, 0.06, *(np.ascontiguousarray(v[s]) for v in q), **kw)
    whole = np.asarray(call(slice(None)))
    for s in (slice(0, 1), slice(5, 700), slice(100, 16000)):
        assert np.array_equal(np.asarray(call(s)), whole[s])


def test_shells_against_the_oracle(lg, oracle_mod):
    p, f, area, active = _set("shells")
    for s in (slice(60, 360), slice(14990, 15010)):
        ib, ie = s.start, s.stop
        ref = oracle_mod.pse_laplacian(*p, f[0], area, active, 0.05, 1.0, kernel=0, ib=ib, ie=ie)
        got = lg.pse_sphere_laplacian_at_particles(*p, f[0], area, active, 0.05, 1.0, i_begin=ib + 1, i_end=ie, mode="fp64")
        assert np.abs(got[s] - ref).max() <= 1e-12 * np.abs(ref).max()


# 8, 4, 4 and 2 lanes per target on 152 SMs
@pytest.mark.parametrize("ns", [7295, 7296, 14591, 14592])
def test_every_lane_count(lg, oracle_mod, ns):
    rng = np.random.default_rng(ns)
    p = rng.normal(size=(3, 15000))
    p /= np.linalg.norm(p, axis=0)
    f, area = rng.normal(size=15000), rng.uniform(0.5, 1.5, 15000) / 15000
    active = (rng.permutation(15000) < ns).astype(np.int32)
    for kernel in (0, 1):
        ref = oracle_mod.pse_laplacian(*p, f, area, active, 0.05, 1.0, kernel=kernel, ib=700, ie=1200)
        got = lg.pse_sphere_laplacian_at_particles(*p, f, area, active, 0.05, 1.0, kernel=kernel, i_begin=701, i_end=1200,
                                                   mode="fp64")
        assert np.abs(got[700:1200] - ref).max() <= 1e-12 * np.abs(ref).max()
