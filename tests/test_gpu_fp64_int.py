"""The FP64 velocity sums, whose products and divisions run as integers (csrc/seq_i64.cuh), bit for
bit against the oracle where that could go wrong: zero coordinates and strengths, coordinates of few
bits (products that are ties), values outside the integer range (tiny, huge, subnormal, infinite),
coincident particles, radii outside it, and target counts of each lane count and ragged ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lg(built_lib):
    return built_lib


def _set(kind, n, seed):
    rng = np.random.default_rng(seed)
    p = rng.normal(size=(n, 3))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    q, area = rng.normal(size=n), rng.random(n) / n
    active = (rng.random(n) < 0.7).astype(np.int32)
    if kind == "zeros":
        p[rng.random((n, 3)) < 0.1] = 0.0
        p[rng.random(n) < 0.02] = -0.0
        q[rng.random(n) < 0.2] = 0.0
        q[rng.random(n) < 0.1] = -0.0
    elif kind == "few bits":
        p = np.round(p * 64.0) / 64.0
        p[::3] = np.round(p[::3] * 2.0 ** 26) / 2.0 ** 26
        area = np.round(area * n * 16.0 + 1.0) / 16.0
        q = np.round(q * 8.0)
    elif kind == "range":
        for v in (1e-40, 3e-310, 1e25, 1e-200):
            p[rng.integers(0, n, 2), rng.integers(0, 3, 2)] = v
        for v in (1e-300, 4e-320, 1e200, 1e-170, 1e290):
            q[rng.integers(0, n, 2)] = v
    elif kind == "inf":
        p[n // 2, 1] = np.inf
        q[n // 3] = np.inf
    elif kind == "same":
        p[n // 2:] = p[:n - n // 2]
    return [np.ascontiguousarray(v) for v in (*p.T, q, area)] + [active]


KINDS = ["plain", "zeros", "few bits", "range", "inf", "same"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [33, 1001, 5003])
@pytest.mark.parametrize("radius", [1.0, 6.37122e6, 1e-12])
def test_bve_fp64_is_the_oracle_bit_for_bit(lg, oracle_mod, kind, n, radius):
    x, y, z, q, area, active = _set(kind, n, n)
    a = (x * radius, y * radius, z * radius, q, area, active)
    for assoc, fn in ((oracle_mod.ASSOC_SOLVER, lg.bve_sphere_velocity), (oracle_mod.ASSOC_MESH, lg.set_velocity_from_vorticity)):
        with np.errstate(all="ignore"):
            ref = oracle_mod.bve_velocity(*a, radius, assoc)
        for g, r in zip(fn(*a, radius, mode="fp64"), ref):
            assert np.array_equal(g, r, equal_nan=True)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [33, 3001, 10007])
@pytest.mark.parametrize("delta", [0.0, 0.02, 1e-12])
def test_plane_fp64_is_the_oracle_bit_for_bit(lg, oracle_mod, kind, n, delta):
    x, y, _, q, area, active = _set(kind, n, n + 1)
    ref = oracle_mod.plane_velocity(x, y, q, area, active, delta)
    for g, r in zip(lg.planar_incompressible_velocity(x, y, q, area, active, delta, mode="fp64"), ref):
        assert np.array_equal(g, r, equal_nan=True)


def test_every_lane_count_at_a_ragged_block(lg, oracle_mod):
    """One target set per lane count of the sphere (8 and 4 lanes) and the plane (8, 4 and 2), as a
    rank's block inside a larger set."""
    n = 24001
    x, y, z, q, area, active = _set("zeros", n, 3)
    for nt in (1, 4861, 4867, 9733, 20011):
        ib, ie = 1001, 1000 + nt
        got = lg.bve_sphere_velocity(x, y, z, q, area, active, 1.0, ib, ie, mode="fp64")
        ref = oracle_mod.bve_velocity(x, y, z, q, area, active, 1.0, ib=ib - 1, ie=ie)
        for g, r in zip(got, ref):
            assert np.array_equal(g[ib - 1:ie], r, equal_nan=True)
        got = lg.planar_incompressible_velocity(x, y, q, area, active, 0.0, ib, ie, mode="fp64")
        ref = oracle_mod.plane_velocity(x, y, q, area, active, 0.0, ib=ib - 1, ie=ie)
        for g, r in zip(got, ref):
            assert np.array_equal(g[ib - 1:ie], r, equal_nan=True)
