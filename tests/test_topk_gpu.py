"""Top-k at the edges of its three forms (one CTA, histograms, sampled) and on
inputs where a sample says little: bit-exact values and positions."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _input(kind, n):
    g = torch.Generator().manual_seed(n)
    if kind == "int16":
        return torch.randint(-32768, 32768, (n,), generator=g, dtype=torch.int32).to(torch.int16)
    x = torch.randn(n, generator=g).half()
    if kind == "sorted":
        return torch.sort(x).values
    if kind == "equal":
        return torch.full((n,), -2.5, dtype=torch.float16)
    if kind == "sparse":  # nearly all zeros of both signs, some NaN and infinities
        x = torch.where(torch.rand(n, generator=g) < 0.002, x, torch.zeros_like(x))
        x[::3] *= -1
        x[5::4097] = float("nan")
        x[9::8191] = float("inf")
        x[2::8191] = float("-inf")
    return x


# one CTA takes up to 32768 elements, the sampled form n >= 2^18 with k <= n / 32
@pytest.mark.parametrize("kind", ["normal", "int16", "sorted", "equal", "sparse"])
@pytest.mark.parametrize("n", [1, 511, 32767, 32768, 32769, (1 << 18) - 1, 1 << 18, 1_500_007])
def test_topk_forms(kind, n):
    import tcuscan_ops

    x = _input(kind, n)
    xd = x.to(DEV)
    fn = tcuscan_ops.run_topk_int16 if kind == "int16" else tcuscan_ops.run_topk_fp16
    for k in sorted({1, min(n, 3), n // 32, n // 32 + 1, n // 3, n - 1, n} - {0}):
        v, i = fn(xd, k, 0, 0, 64)
        rv, ri = oracle.topk(x.numpy(), k)
        assert np.array_equal(i.cpu().numpy(), ri), (k, "positions")
        assert np.array_equal(v.cpu().numpy().view(np.uint16), rv.view(np.uint16)), (k, "values")


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs in one process")
def test_every_device_of_a_process():
    """Kernels with more than 48 KB of shared memory on the second GPU after the first."""
    import tcuscan_ops

    x = _input("normal", 1_500_007)
    m = (x > 0).to(torch.int8)
    for dev in ("cuda:0", "cuda:1"):
        with torch.cuda.device(dev):
            for n in (30_000, x.numel()):
                v, i = tcuscan_ops.run_topk_fp16(x[:n].to(dev), 100, 0, 0, 64)
                rv, ri = oracle.topk(x[:n].numpy(), 100)
                assert np.array_equal(i.cpu().numpy(), ri) and np.array_equal(v.cpu().numpy(), rv)
            v, i = tcuscan_ops.run_compress_ind_no_arange(x.float().to(dev), m.to(dev), 64)
            assert np.array_equal(i.cpu().numpy(), np.nonzero(m.numpy())[0])
            s, _ = tcuscan_ops.run_radix_sort(x.to(dev), 128)
            assert torch.equal(s.cpu(), torch.sort(x).values)
            z = tcuscan_ops.run_scan_multi_core(m.to(dev).repeat(4), 64)
            assert torch.equal(z.cpu(), torch.cumsum(m.repeat(4).long(), 0).int())
