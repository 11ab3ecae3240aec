"""FP32C sphere velocity around a group of a single source that lies off the sphere (the only source, or the last
one in curve order): its |p|^2 - 1 enters every pair, near ones too.  Bound: the velocity's 1e-6 of the target's
own sum of pair sizes, sum_j |zeta_j A_j| |x_i x x_j| / (4 pi |1 - x_i.x_j|)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lg(built_lib):
    return built_lib


@pytest.mark.parametrize("others", [0, 128])
@pytest.mark.parametrize("depth", [1e-5, 1e-3, 0.1])
def test_single_source_inside_the_sphere(lg, oracle_mod, others, depth):
    rng = np.random.default_rng(5)
    k = np.arange(others) + 0.5
    r, a = 0.3 * np.sqrt(k / max(others, 1)), k * np.pi * (3.0 - np.sqrt(5.0))
    patch = np.stack([-np.sqrt(1.0 - r * r), r * np.cos(a), r * np.sin(a)])  # the curve's first face; the single source is on its last
    th, ph = np.geomspace(1e-4, 1.5, 3000), rng.uniform(0, 2 * np.pi, 3000)
    targets = np.stack([np.cos(th), np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph)])
    p = np.ascontiguousarray(np.concatenate([patch, [[1.0 - depth], [0.0], [0.0]], targets], axis=1))
    n, m = p.shape[1], others + 1
    zeta, area = np.ones(n), np.full(n, 1.0 / m)
    act = (np.arange(n) < m).astype(np.int32)
    ref = np.stack(oracle_mod.bve_velocity(*p, zeta, area, act, 1.0))[:, m:]
    got = np.stack(lg.bve_sphere_velocity(*p, zeta, area, act, 1.0, mode="fp32c"))[:, m:]
    x, s = p[:, m:], p[:, :m]
    cross = np.linalg.norm(np.cross(x.T[:, None, :], s.T[None, :, :]), axis=2)
    size = (cross / np.abs(1.0 - x.T @ s)).sum(1) / m / (4.0 * np.pi)
    assert np.all(np.abs(got - ref) <= 1e-6 * size)
