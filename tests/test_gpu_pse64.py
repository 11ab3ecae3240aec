"""The FP64 PSE sums (csrc/pse64.cuh) against the oracle where their own path could go wrong: each
angle polynomial and the plain expressions beyond them, each lane count, target counts around a warp,
source counts around a tile, more in-reach tiles than a lane holds, sets far from the origin and of
small and large scale, particles without a direction, and rank blocks.  Tolerance: 1e-12 of the
largest value, the bound of the FP64 mode's PSE sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.fixture(scope="module")
def lg(built_lib):
    return built_lib


def _sphere(n, seed, radius=1.0):
    rng = np.random.default_rng(seed)
    p = rng.normal(size=(n, 3))
    p *= radius / np.linalg.norm(p, axis=1, keepdims=True)
    f, area = rng.normal(size=n), 4.0 * np.pi * radius ** 2 * rng.uniform(0.5, 1.5, n) / n
    return (*[np.ascontiguousarray(v) for v in p.T], f, area, (rng.random(n) < 0.6).astype(np.int32))


def _close(got, ref):
    got, ref = np.stack(np.atleast_2d(got)), np.stack(np.atleast_2d(ref))
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()


# reach / radius = 7 eps: the three polynomials, the last one past 90 degrees, the plain expressions
@pytest.mark.parametrize("eps", [0.02, 0.06, 0.0644, 0.15, 0.17, 0.3, 0.44, 0.6, 2.0])
@pytest.mark.parametrize("n", [31, 33, 1001])
def test_great_circle_laplacian_at_every_reach(lg, oracle_mod, eps, n):
    x, y, z, f, area, active = _sphere(n, n)
    ref = oracle_mod.pse_laplacian(x, y, z, f, area, active, eps, 1.0, kernel=0)
    _close(lg.pse_sphere_laplacian_at_particles(x, y, z, f, area, active, eps, 1.0, mode="fp64"), ref)


# 8, 8, 8, 4, 2 and 1 lanes per target on 152 SMs, blocks inside a larger set
@pytest.mark.parametrize("nt", [1, 7295, 7297, 14597, 29201, 58373])
def test_every_lane_count(lg, oracle_mod, nt):
    x, y, z, f, area, active = _sphere(60000, 5)
    active[::2] = 0
    for kernel, eps in ((0, 0.02), (1, 0.02)):
        got = lg.pse_sphere_laplacian_at_particles(x, y, z, f, area, active, eps, 1.0, kernel=kernel, i_begin=101,
                                                   i_end=100 + nt, mode="fp64")
        ref = oracle_mod.pse_laplacian(x, y, z, f, area, active, eps, 1.0, kernel=kernel, ib=100, ie=100 + nt)
        _close(got[100:100 + nt], ref)
        assert not got[:100].any() and not got[100 + nt:].any()


def test_more_tiles_in_reach_than_a_lane_holds(lg, oracle_mod):
    """Every target reaches a third of a sphere in random order: each of the ~94 tiles holds sources of
    every lane, so the held tiles are evaluated several times."""
    x, y, z, f, area, active = _sphere(10000, 9)
    ref = oracle_mod.pse_laplacian(x, y, z, f, area, active, 0.16, 1.0, kernel=0, ib=0, ie=500)
    got = lg.pse_sphere_laplacian_at_particles(x, y, z, f, area, active, 0.16, 1.0, i_begin=1, i_end=500, mode="fp64")
    _close(got[:500], ref)


@pytest.mark.parametrize("shift, scale", [((0.0, 0.0), 1.0), ((1000.0, -2000.0), 1.0), ((0.0, 0.0), 1e-25), ((3e12, 0.0), 1e12)])
@pytest.mark.parametrize("n", [63, 65, 2049])
def test_plane_far_from_the_origin_and_at_other_scales(lg, oracle_mod, shift, scale, n):
    rng = np.random.default_rng(n)
    x, y = (scale * rng.uniform(-4.0, 4.0, n) + s for s in shift)
    f, area, active = rng.normal(size=n), scale ** 2 * 64.0 * rng.uniform(0.5, 1.5, n) / n, (rng.random(n) < 0.7).astype(np.int32)
    for eps in (0.1 * scale, 0.6 * scale):
        got = lg.pse_plane_laplacian_at_particles(x, y, f, area, active, eps, mode="fp64")
        _close(got, oracle_mod.pse_laplacian(x, y, np.zeros(n), f, area, active, eps, kernel=2))


def test_particles_without_a_direction(lg, oracle_mod):
    """A passive and an active particle at the centre of the sphere: at distance 0 from everything."""
    x, y, z, f, area, active = _sphere(700, 3)
    for k, on in ((10, 1), (333, 0)):
        x[k] = y[k] = z[k] = 0.0
        active[k] = on
    ref = oracle_mod.pse_laplacian(x, y, z, f, area, active, 0.1, 1.0, kernel=0)
    _close(lg.pse_sphere_laplacian_at_particles(x, y, z, f, area, active, 0.1, 1.0, mode="fp64"), ref)


def test_earth_radius(lg, oracle_mod):
    a = 6.37122e6
    x, y, z, f, area, active = _sphere(3001, 4, a)
    for eps in (0.05 * a, 0.12 * a, 0.3 * a):
        ref = oracle_mod.pse_laplacian(x, y, z, f, area, active, eps, a, kernel=0)
        _close(lg.pse_sphere_laplacian_at_particles(x, y, z, f, area, active, eps, a, mode="fp64"), ref)
