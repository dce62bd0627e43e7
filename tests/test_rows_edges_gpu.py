"""Segment sums and SpMV at the edges of tiles (8192 elements) and of the SpMV's
product batches (4096), with bounds that crowd at one end; exact for int8,
within a bound on the FP32 roundings for the products."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TILE = 8192


def _bounds(kind, n, rng):
    if kind == "one":
        return np.array([0, n])
    if kind == "none_behind":  # every bound in the first tile, nothing behind
        return np.concatenate([[0], np.sort(rng.integers(0, min(n, 100) + 1, 2000))])
    if kind == "crowd_at_end":
        return np.concatenate([[0], np.sort(rng.integers(max(n - 50, 0), n + 1, 3000)), [n]])
    if kind == "dense":
        return np.concatenate([[0], np.sort(rng.integers(0, n + 1, n // 3 + 2)), [n]])
    return np.unique(np.concatenate([[0, n], np.arange(0, n + 1, TILE), np.minimum(np.arange(0, n + 1, TILE) + 1, n)]))


@pytest.mark.parametrize("kind", ["one", "none_behind", "crowd_at_end", "dense", "tile_edges"])
@pytest.mark.parametrize("n", [1, 4095, 4097, TILE - 1, TILE, TILE + 1, 40 * TILE, 40 * TILE + 5])
@pytest.mark.parametrize("wide", [False, True])
def test_bounds_and_products(kind, n, wide):
    import tcuscan_ops

    rng = np.random.default_rng(n)
    b = _bounds(kind, n, rng).astype(np.int64 if wide else np.int32)
    bd = torch.from_numpy(b).to(DEV)
    x8 = torch.from_numpy(rng.integers(-8, 9, n).astype(np.int8))
    cs = np.concatenate([[0], np.cumsum(x8.numpy().astype(np.int64))])
    got = tcuscan_ops.run_seg_sum_multi_core(x8.to(DEV), bd, 64).cpu().numpy()
    assert np.array_equal(got, cs[b[1:]] - cs[b[:-1]])
    cols = torch.from_numpy(rng.integers(0, 1000, n).astype(np.int32))
    for dt in (torch.float16, torch.float32):
        vals = torch.from_numpy(rng.standard_normal(n)).to(dt)
        xv = torch.from_numpy(rng.uniform(-1, 1, 1000)).to(dt)
        prod = vals.double().numpy() * xv.double().numpy()[cols.numpy()]
        ref = np.concatenate([[0.0], np.cumsum(prod)])
        mag = np.concatenate([[0.0], np.cumsum(np.abs(prod))])
        y = tcuscan_ops.run_spmv_v2(vals.to(DEV), bd, cols.to(DEV), xv.to(DEV), 64).cpu().double().numpy()
        err = np.abs(y - (ref[b[1:]] - ref[b[:-1]]))
        # A segment inside an aligned word of 32 elements is the difference of two of the word's FP32
        # prefixes: at most 2 * 31 roundings, each at most 2^-24 of the word's sum of magnitudes W.  A longer
        # one adds two such ends and FP32 sums of its words (half a unit, 2^-24, of the sum of magnitudes each,
        # 8 levels of words and threads in a tile; the tiles are joined in FP64).
        w = np.add.reduceat(np.abs(prod), np.arange(0, n, 32)).max()
        bound = 2 * 62 * 2.0 ** -24 * w + (31 + 2 * 8) * 2.0 ** -24 * (mag[b[1:]] - mag[b[:-1]])
        assert np.all(err <= bound + 1e-12)
