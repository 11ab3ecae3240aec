"""FP32C PSE sums with unused particles at the sphere's centre (passive, or active with no area): all outputs are finite,
and the others' are those of the oracle (the FP32C PSE sums' 1e-4 of the largest value), to which such a particle
adds nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lg(built_lib):
    return built_lib


@pytest.mark.parametrize("n", [40, 1500])
@pytest.mark.parametrize("active_too", [False, True])
def test_particles_at_the_centre(lg, oracle_mod, n, active_too):
    rng = np.random.default_rng(n)
    p = rng.normal(size=(3, n))
    p /= np.linalg.norm(p, axis=0)
    f, g, h = p[0] * p[1] + 0.2 * p[2], p[1] - p[2] ** 2, p[2] + p[0] * p[1]
    area, active = 4 * np.pi * rng.uniform(0.5, 1.5, n) / n, (rng.random(n) < 0.7).astype(np.int32)
    at = [0, n // 2, n - 1]
    p[:, at] = 0.0
    active[at], area[at] = (1, 0.0) if active_too else (0, 1.0)
    others = np.ones(n, bool)
    others[at] = False
    eps = 0.09

    def check(got, ref):
        got, ref = np.stack(np.atleast_2d(got)), np.stack(np.atleast_2d(ref))
        assert np.isfinite(got).all()
        assert np.abs(got - ref)[:, others].max() <= 1e-4 * np.abs(ref[:, others]).max()

    a = (area, active, eps, 1.0)
    for kernel in (0, 1):
        check(lg.pse_sphere_laplacian_at_particles(*p, f, *a, kernel=kernel, mode="fp32c"),
              oracle_mod.pse_laplacian(*p, f, *a, kernel=kernel))
    check(lg.pse_sphere_gradient_at_particles(*p, f, *a, mode="fp32c"), oracle_mod.pse_sphere_gradient(*p, f, *a))
    check(lg.pse_sphere_divergence_at_particles(*p, f, g, h, *a, mode="fp32c"), oracle_mod.pse_sphere_divergence(*p, f, g, h, *a))
