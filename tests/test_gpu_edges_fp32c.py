"""FP32C sweeps where their forms and tiles meet: the Laplacians at every reach (angle polynomials, asin,
every pair of a small set), ragged sizes and groups spread over separate clusters, and the planar SWE
sums around a group and a tile.

Laplacians: the PSE sums' FP32C bound, 1e-4 of the largest value.  SWE sums, per target: a pair's 1/z and
1/z^2 carry at most 20 roundings of 2^-24, its running sum 32 and the sums above it 8 on average, so 2^-18 of
sum (|W| + |D|) / r for the velocity; the double dot product 2 (a^2 + b^2) of two such sums of
G = sum (|W| + |D|) / r^2 moves by at most 8 G (2^-18 G).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lg(built_lib):
    return built_lib


def _close(got, ref, tol=1e-4):
    assert np.abs(np.asarray(got) - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.parametrize("eps", [0.02, 0.1, 0.15, 0.17, 0.3, 1.0])
@pytest.mark.parametrize("n", [31, 65, 257, 1500])
@pytest.mark.parametrize("kernel", [0, 1])
def test_sphere_laplacian_at_every_reach(lg, oracle_mod, eps, n, kernel):
    rng = np.random.default_rng(n)
    p = rng.normal(size=(3, n))
    p /= np.linalg.norm(p, axis=0)
    f = 2.0 + p[0] * p[1] + rng.normal(size=n)
    area = 4 * np.pi / n * rng.uniform(0.5, 1.5, size=n)
    act = (rng.random(n) < 0.7).astype(np.int32)
    act[0] = 1
    ref = oracle_mod.pse_laplacian(p[0], p[1], p[2], f, area, act, eps, 1.0, kernel)
    _close(lg.pse_sphere_laplacian_at_particles(*p, f, area, act, eps, kernel=kernel, mode="fp32c"), ref)


@pytest.mark.parametrize("shift", [0.0, 100.0])
@pytest.mark.parametrize("n", [33, 300, 1025])
def test_plane_laplacian_of_separate_clusters(lg, oracle_mod, shift, n):
    rng = np.random.default_rng(n)
    x, y = rng.normal(scale=0.1, size=(2, n))
    x = x + 2.0 * rng.integers(0, 3, size=n) + shift
    f = 1.0 + np.sin(3 * x) + y
    area = np.full(n, 0.1 / n)
    act = np.ones(n, dtype=np.int32)
    ref = oracle_mod.pse_laplacian(x, y, np.zeros(n), f, area, act, 0.05, 1.0, 2)
    _close(lg.pse_plane_laplacian_at_particles(x, y, f, area, act, 0.05, mode="fp32c"), ref)


@pytest.mark.parametrize("n", [1, 2, 127, 129, 257, 1500])
@pytest.mark.parametrize("shift", [0.0, 50.0])
def test_plane_swe_group_and_tile_edges(lg, oracle_mod, n, shift):
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-1, 1, size=(2, n))
    x = x + shift
    w, d = rng.normal(size=(2, n))
    area = rng.uniform(0.5, 1.5, size=n) / n
    act = np.ones(n, dtype=np.int32)
    sh = 1.0 + 0.1 * x
    ref = oracle_mod.swe_plane_rhs(x, y, w, d, sh, area, act, 0.1)
    got = lg.swe_plane_rhs_integrals(x, y, w, d, sh, area, act, 0.1, mode="fp32c")
    r2 = (x[:, None] - x) ** 2 + (y[:, None] - y) ** 2
    inv = np.where(r2 > 0, 1.0 / np.where(r2 > 0, r2, 1.0), 0.0)
    s = (np.abs(w) + np.abs(d)) * area / (2 * np.pi)
    vel, g = np.sqrt(inv) @ s, inv @ s
    for c in (0, 1):
        assert np.all(np.abs(got[c] - ref[c]) <= 2.0**-18 * vel)
    assert np.all(np.abs(got[2] - ref[2]) <= 8 * 2.0**-18 * g**2)
