"""FP64 PSE sums of particles farther than 7 eps from each other.  Sets of up to 256 sources leave no pair out and hold
the FP64 mode's 1e-12 of the largest value; larger ones leave out the pairs beyond r = 7, each below 1e-14 of the
kernel's peak, so there the bound is 1e-14 of the sum of the pairs' sizes at the peak (40 / pi for K8)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lg(built_lib):
    return built_lib


@pytest.mark.parametrize("n", [255, 256, 257, 400])
def test_every_pair_beyond_the_cutoff(lg, oracle_mod, n):
    rng = np.random.default_rng(n)
    k = np.arange(n) + 0.5
    z, ph = 1.0 - 2.0 * k / n, k * np.pi * (3.0 - np.sqrt(5.0))  # even on the sphere
    p = np.stack([np.sqrt(1 - z * z) * np.cos(ph), np.sqrt(1 - z * z) * np.sin(ph), z])
    d = np.sqrt(((p[:, :, None] - p[:, None, :]) ** 2).sum(0)) + 10.0 * np.eye(n)
    eps = d.min() / 7.2
    f, area, active = rng.normal(size=n), np.full(n, 4.0 * np.pi / n), np.ones(n, np.int32)
    ref = oracle_mod.pse_laplacian(*p, f, area, active, eps, 1.0, kernel=0)
    got = lg.pse_sphere_laplacian_at_particles(*p, f, area, active, eps, 1.0, mode="fp64")
    if n <= 256:
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    else:
        size = (np.abs(f[:, None] - f[None, :]) * area).sum(1) * 40.0 / np.pi / eps**4
        assert np.all(np.abs(got - ref) <= 1e-14 * size)
