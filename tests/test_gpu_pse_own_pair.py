"""FP32C Laplacians of particles without a neighbour in reach: every target's sum is its own pair, whose f_j - f_i is
zero, times the kernel's peak.  All others have r >= 20, where the kernel is zero in any precision: the result is 0."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lg(built_lib):
    return built_lib


@pytest.mark.parametrize("n", [1, 2, 33, 700])
@pytest.mark.parametrize("mean", [0.0, 1.0, 1e5])
def test_own_pair_is_zero(lg, n, mean):
    rng = np.random.default_rng(n)
    k = np.arange(n) + 0.5
    z, ph = 1.0 - 2.0 * k / n, k * np.pi * (3.0 - np.sqrt(5.0))
    p = np.stack([np.sqrt(1 - z * z) * np.cos(ph), np.sqrt(1 - z * z) * np.sin(ph), z])
    grid = np.stack([k.astype(int) % 27, k.astype(int) // 27]) * 0.05 + 1e-3 * rng.random((2, n))
    f, area, active = mean + rng.normal(size=n), rng.uniform(0.5, 1.5, n) / n, np.ones(n, np.int32)
    for kernel in (0, 1):
        got = lg.pse_sphere_laplacian_at_particles(*p, f, area, active, 0.004, 1.0, kernel=kernel, mode="fp32c")
        assert not np.asarray(got).any()
    for kernel in (lg.PSE_K8_CHORD, lg.PSE_GAUSS_CHORD):
        got = lg.pse_plane_laplacian_at_particles(*grid, f, area, active, 0.002, kernel=kernel, mode="fp32c")
        assert not np.asarray(got).any()
