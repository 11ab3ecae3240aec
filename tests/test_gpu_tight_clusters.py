"""FP32C sphere sums around clusters much tighter than the float spacing of their origin's place on the
sphere: targets at every distance from inside the cluster outward.

A cluster's own origin is off the sphere by up to 2^-24, which the far form must not see.  Bound: the
velocity's 1e-6 of the target's own sum of pair sizes, sum_j |S_j| / |d_ij| (every pair's relative error is a few
2^-24 to 2^-21); the stream functions' 2^-20 sum_j |S_j| (1 + |ln q_ij|) of the other sweep tests.
Smaller clusters have no reference: at 1e-6 the positions' own distance from the sphere (3e-16 in |x|^2)
exceeds the closest pairs' squared distance, and some of the reference's a^2 - x.x_j are negative.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lg(built_lib):
    return built_lib


def _cluster(size, m, seed):
    rng = np.random.default_rng(seed)
    k = np.arange(m) + 0.5
    r, a = size * np.sqrt(k / m), k * np.pi * (3.0 - np.sqrt(5.0))
    th = np.concatenate([np.geomspace(size / 10, 0.5, 1200), size * rng.uniform(1.5, 40.0, 800)])
    ph = rng.uniform(0, 2 * np.pi, th.size)
    p = np.stack([np.concatenate([r * np.cos(a), np.sin(th) * np.cos(ph)]),
                  np.concatenate([r * np.sin(a), np.sin(th) * np.sin(ph)]),
                  np.concatenate([np.sqrt(1 - r * r), np.cos(th)])])
    turn, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    p = turn @ p
    p /= np.linalg.norm(p, axis=0)
    n = p.shape[1]
    order = np.concatenate([np.arange(m), m + np.argsort(th)])
    return np.ascontiguousarray(p[:, order]), (np.arange(n) < m).astype(np.int32), rng


@pytest.mark.parametrize("size", [1e-5, 1e-4, 1e-2])
@pytest.mark.parametrize("m", [64, 128, 300])
def test_velocity_and_stream_around_a_tight_cluster(lg, oracle_mod, size, m):
    p, act, rng = _cluster(size, m, m)
    n = p.shape[1]
    zeta = 1.0 + 0.5 * rng.normal(size=n)
    area = np.full(n, 1.0 / m)
    src = act != 0
    d = p[:, :, None] - p[:, None, src]
    q = np.einsum("kij,kij->ij", d, d)
    s = np.abs(zeta * area)[src]
    ref = np.stack(oracle_mod.bve_velocity(*p, zeta, area, act, 1.0))
    got = np.stack(lg.bve_sphere_velocity(*p, zeta, area, act, 1.0, mode="fp32c"))
    size_u = np.where(q > 0, 1.0 / np.sqrt(np.where(q > 0, q, 1.0)), 0.0) @ s / (2 * np.pi)
    # the oracle's a^2 - x.x_j cancels: about 2^-52 / (q / 2) of a pair
    own = np.where(q > 0, 2.0**-51 / np.where(q > 0, q, 1.0) ** 1.5, 0.0) @ s / (2 * np.pi)
    assert np.all(np.abs(got - ref) <= 1e-6 * size_u + 4 * own)
    absv = zeta + 1.0
    ref = oracle_mod.bve_stream(*p, zeta, absv, area, act, 1.0)
    got = lg.set_stream_functions_on_mesh(*p, zeta, absv, area, act, 1.0, mode="fp32c")
    ln = 1.0 + np.abs(np.log(np.where(q > 0, q, 1.0)))
    rel = np.where(q > 0, 2.0**-50 / np.where(q > 0, q, 1.0), 0.0)
    for w, g, r in zip((zeta, absv), got, ref):
        a = np.abs(w * area)[src] / (4 * np.pi)
        assert np.all(np.abs(g - r) <= 2.0**-20 * ln @ a + 4 * rel @ a)
