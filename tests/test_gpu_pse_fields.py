"""FP32C Laplacians of fields whose mean is large against their variation, where a pair's f_j - f_i lies in the
low parts of the two, and of sets whose last group of 32 holds a single source at a float position (a group of
radius 0).  Bound: the FP32C PSE sums' 1e-4 of the largest value; adding a constant to f changes no difference,
so the reference is the oracle's Laplacian of f without it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lg(built_lib):
    return built_lib


def _close(got, ref):
    assert np.abs(np.asarray(got) - ref).max() <= 1e-4 * np.abs(ref).max()


@pytest.mark.parametrize("mean", [1.0, 1e4, 1e6])
def test_field_with_a_large_mean(lg, oracle_mod, mean):
    m = lg.PolyMesh2d(lg.CUBED_SPHERE_SEED, 6, 1.0)
    f, eps = m.x * m.y + 0.3 * m.z, m.max_edge_length ** 0.75
    for kernel in (0, 1):
        ref = oracle_mod.pse_laplacian(m.x, m.y, m.z, f, m.area, m.active, eps, 1.0, kernel=kernel)
        got = lg.pse_sphere_laplacian_at_particles(m.x, m.y, m.z, f + mean, m.area, m.active, eps, 1.0, kernel=kernel,
                                                   mode="fp32c")
        _close(got, ref)
    rng = np.random.default_rng(3)
    x, y = rng.uniform(-2.0, 2.0, (2, 3000))
    f, area, act = np.sin(3 * x) * y, np.full(3000, 16.0 / 3000), np.ones(3000, np.int32)
    for kernel in (lg.PSE_K8_CHORD, lg.PSE_GAUSS_CHORD):
        ref = oracle_mod.pse_laplacian(x, y, np.zeros(3000), f, area, act, 0.08, kernel=kernel)
        _close(lg.pse_plane_laplacian_at_particles(x, y, f + mean, area, act, 0.08, kernel=kernel, mode="fp32c"), ref)


@pytest.mark.parametrize("n", [33, 65, 865])
@pytest.mark.parametrize("mean", [1.0, 1e4])
def test_a_last_group_of_one_source(lg, oracle_mod, n, mean):
    rng = np.random.default_rng(n)
    k = np.sort(rng.permutation(64 * 64)[:n])
    x, y = k % 64 / 32.0, k // 64 / 32.0
    f, area, act = 0.01 * np.sin(x + y), np.full(n, 4.0 / n), np.ones(n, np.int32)
    ref = oracle_mod.pse_laplacian(x, y, np.zeros(n), f, area, act, 0.1, kernel=2)
    _close(lg.pse_plane_laplacian_at_particles(x, y, f + mean, area, act, 0.1, mode="fp32c"), ref)
