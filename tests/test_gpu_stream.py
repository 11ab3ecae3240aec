"""The sphere stream functions' FP32C sweep where its forms meet: whole and ragged groups and tiles,
and targets at every distance of a patch, through the near limit and the log1p bounds.

Bound of a target: 2^-20 sum_j |S_j| (1 + |ln q_ij|).  A pair's log argument carries at most six
roundings of 2^-24 (offsets, expanded or squared distance), the log two units of its own size, and the
FP32 partials of at most 64 terms eight more on average: 16 x 2^-24 = 2^-20 in all.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lg(built_lib):
    return built_lib


def _check(lg, oracle_mod, p, qr, qa, area, act, radius=1.0):
    ref = oracle_mod.bve_stream(p[0], p[1], p[2], qr, qa, area, act, radius)
    got = lg.set_stream_functions_on_mesh(p[0], p[1], p[2], qr, qa, area, act, radius, mode="fp32c")
    src = act != 0
    d = p[:, :, None] - p[:, None, src]
    q = np.einsum("kij,kij->ij", d, d) / radius**2
    ln = 1.0 + np.abs(np.log(np.where(q > 0, q, 1.0)))
    for w, g, r in zip((qr, qa), got, ref):
        bound = 2.0**-20 * ln @ np.abs(w * area)[src] / (4 * np.pi)
        assert np.all(np.abs(g - r) <= bound + 1e-300)


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 255, 257, 769, 2500])
def test_sphere_stream_group_and_tile_edges(lg, oracle_mod, n):
    rng = np.random.default_rng(n)
    p = rng.normal(size=(3, n))
    p /= np.linalg.norm(p, axis=0)
    qr = 1.0 + rng.normal(size=n)
    qa = qr + 2.0 * p[2]
    area = rng.uniform(0.5, 1.5, size=n) * 4 * np.pi / n
    act = np.ones(n, dtype=np.int32)
    _check(lg, oracle_mod, p, qr, qa, area, act)


@pytest.mark.parametrize("patch,m", [(1e-3, 64), (0.02, 64), (0.02, 100), (0.1, 640)])
@pytest.mark.parametrize("radius", [1.0, 6.37122e6])
def test_sphere_stream_patch_at_every_distance(lg, oracle_mod, patch, m, radius):
    """m sources in an even patch around an axis, targets (no sources) from inside it to the far side."""
    rng = np.random.default_rng(m)
    k = np.arange(m) + 0.5
    r, a = patch * np.sqrt(k / m), k * np.pi * (3.0 - np.sqrt(5.0))
    src = np.stack([r * np.cos(a), r * np.sin(a), np.ones(m)])
    th = np.concatenate([np.geomspace(patch / 50, np.pi, 1500), patch * rng.uniform(1.0, 30.0, 500)])
    th = np.minimum(th, np.pi)
    ph = rng.uniform(0, 2 * np.pi, th.size)
    tgt = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)])
    p = np.concatenate([src / np.linalg.norm(src, axis=0), tgt], 1)
    turn, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    p = turn @ p
    p /= np.linalg.norm(p, axis=0)
    n = p.shape[1]
    act = (np.arange(n) < m).astype(np.int32)
    qr = 3.0 + rng.normal(size=n)
    qa = rng.normal(size=n)
    area = rng.uniform(0.5, 1.5, size=n) * radius**2 / m
    _check(lg, oracle_mod, p * radius, qr, qa, area, act, radius)
