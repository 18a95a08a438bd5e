"""The guide's training pass at batch sizes around its 16-sample tiles, its
12-warp blocks and the whole grid, against the float64 oracle with the same
BF16 roundings (oracle/mlp_ref.py)."""
import numpy as np
import pytest

from bulbit_b200 import lib
from oracle import mlp_ref

pytestmark = pytest.mark.gpu

AABB = np.array([-1, -1, -1, 1, 1, 1], np.float32)


def batch(n, seed):
    g = np.random.default_rng(seed)

    def unit():
        v = g.standard_normal((n, 3))
        return (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)

    raw = np.concatenate([g.uniform(-1, 1, (n, 3)), unit(), unit(), g.uniform(0.05, 1, (n, 1))], 1).astype(np.float32)
    return raw, unit(), g.exponential(1.0, n).astype(np.float32)


@pytest.mark.parametrize("n", [2, 15, 16, 17, 191, 193, 148 * 192 - 1, 148 * 192 + 17])
def test_gradient_at_tile_edges(n):
    g = np.random.default_rng(5)
    params = g.uniform(-0.25, 0.25, lib.GpuGuide.N_PARAMS).astype(np.float32)
    guide = lib.GpuGuide(AABB, seed=1)
    guide.set_params(params)
    raw, dirs, weights = batch(n, n)
    grad, loss = guide.gradient(raw, dirs, weights)
    # A sample's own arithmetic does not depend on its place in the batch, so a
    # batch is the sum of its parts up to 32-bit summation order (n terms of
    # 2^-24 each at worst, their square root in the mean).
    for cut in (1, n // 2, n - 1):
        a, la = guide.gradient(raw[:cut], dirs[:cut], weights[:cut])
        b, lb = guide.gradient(raw[cut:], dirs[cut:], weights[cut:])
        parts = a.astype(np.float64) + b
        assert np.linalg.norm(grad - parts) <= 1e-5 * np.linalg.norm(parts) + 1e-7
        assert abs(loss - (la + lb)) <= 1e-5 * (abs(la) + abs(lb)) + 1e-6
    if n > 100:
        # 3 % per layer, the bound of test_guide_gpu.py (a unit whose input
        # rounds to the other side of zero counts little in a large batch).
        ref, ref_loss = mlp_ref.gradient(params, raw, dirs, weights, AABB, bf=True)
        at = 0
        for shape in mlp_ref.SHAPES:
            m = int(np.prod(shape))
            assert np.linalg.norm(grad[at:at + m] - ref[at:at + m]) <= 3e-2 * np.linalg.norm(ref[at:at + m]), shape
            at += m
        assert abs(loss - ref_loss) <= 1e-3 * abs(ref_loss)
    guide.close()


def test_loss_is_summed_in_few_rounded_additions():
    """The blocks' losses reach the total by 148 additions in any order, each of
    a rounding error of about 0.4 * 2^-24 of a partial total of 0.58 of the sum
    (root mean squares): sqrt(148) times that, 1.7e-7 of the total. One addition
    per warp would be sqrt(12) times as much."""
    n, err = 32_768, []
    guide = lib.GpuGuide(AABB, seed=1)
    for seed in range(4):
        guide.set_params(np.random.default_rng(seed).uniform(-0.25, 0.25, lib.GpuGuide.N_PARAMS).astype(np.float32))
        raw, dirs, weights = batch(n, seed)
        parts = sum(float(guide.gradient(raw[i:i + 32], dirs[i:i + 32], weights[i:i + 32])[1]) for i in range(0, n, 32))
        err += [(guide.gradient(raw, dirs, weights)[1] - parts) / abs(parts) for _ in range(6)]
    assert np.sqrt(np.mean(np.square(err))) < 2.7e-7
    guide.close()
