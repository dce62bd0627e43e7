"""Top-k at the edges of its three forms (one CTA, histograms, sampled), on
inputs where a sample says little or misleads, and through the C interface in
bfloat16 and on inputs that start on no 16 bytes: bit-exact values and
positions."""
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


def _key(bits, kind):
    """Selection key of 16-bit patterns: value order, -0 == +0, every NaN on top (fp16, bf16); int16 by value."""
    b = bits.astype(np.int64)
    if kind == "int16":
        return b ^ 0x8000
    mag = b & 0x7FFF
    k = np.where(b & 0x8000, 0x8000 - mag, 0x8000 + mag)
    return np.where(mag > (0x7C00 if kind == "float16" else 0x7F80), 0xFFFF, k)


def _expect(bits, kind, k):
    """Positions of the k largest by key: the oracle on the keys as int16 values."""
    return oracle.topk((_key(bits, kind) ^ 0x8000).astype(np.uint16).view(np.int16), k)[1]


def _run_c(bits, kind, k, off):
    """tcu_topk on 16-bit patterns that start `off` elements behind 16 bytes."""
    from tcuscan_ops import _lib as L

    buf = torch.zeros(bits.size + off, dtype=torch.int16, device=DEV)
    x = buf[off:]
    x.copy_(torch.from_numpy(bits.view(np.int16)))
    v = torch.empty(k, dtype=torch.int16, device=DEV)
    i = torch.empty(k, dtype=torch.int32, device=DEV)
    tb = L.lib.tcu_topk_tmp_bytes(bits.size)
    tmp = torch.empty(tb, dtype=torch.uint8, device=DEV)
    code = {"int16": L.TCU_INT16, "float16": L.TCU_FLOAT16, "bfloat16": L.TCU_BFLOAT16}[kind]
    assert L.lib.tcu_topk(x.data_ptr(), code, bits.size, k, v.data_ptr(), i.data_ptr(), tmp.data_ptr(), tb,
                          L.stream_ptr(torch.device(DEV))) == 0
    return v.cpu().numpy().view(np.uint16), i.cpu().numpy()


def _check_c(bits, kind, k, off=0):
    v, i = _run_c(bits, kind, k, off)
    ref = _expect(bits, kind, k)
    assert np.array_equal(i, ref), (kind, k, off, "positions")
    assert np.array_equal(v, bits[ref]), (kind, k, off, "values")


def _sample_positions(n):
    """The elements the sampled form looks at: one of each of 1024 equal parts, placed by its integer mix."""
    j = np.arange(1024, dtype=np.uint32)
    h = j ^ (j >> 16)
    h = h * np.uint32(0x7FEB352D)
    h ^= h >> 15
    h = h * np.uint32(0x846CA68B)
    h = (h ^ (h >> 16)).astype(np.uint64)
    a, b = np.uint64(n) * j // 1024, np.uint64(n) * (j.astype(np.uint64) + 1) // 1024
    return (a + (h * (b - a) >> np.uint64(32))).astype(np.int64)


def _rank(n, k):
    """The sample rank whose key bounds the candidates from below."""
    mu = 1024.0 * k / n
    return int(mu + 6.0 * np.sqrt(mu) + 8.0)


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("n", [1 << 18, 300_007])
def test_sampled_form_hands_over(n, off):
    """Inputs on which the collect pass cannot end the search: fewer than k candidates, and a k-th key in the last
    bin of the candidates' histogram (with its neighbours on either side)."""
    rng = np.random.default_rng(n)
    at = _sample_positions(n)
    # the samples hold the 1024 largest keys: the lower bound lies among them, above nearly all of the k largest
    for kind, big, small in (("int16", 20000, (-100, 100)), ("float16", 0x6000, (0x1000, 0x1100)),
                             ("bfloat16", 0x6000, (0x3000, 0x3100))):
        x = rng.integers(*small, n).astype(np.int16)
        x[at] = big + np.arange(1024)
        for k in (_rank(n, 2000) + 100, 2000, n // 32):
            assert k > _rank(n, k)  # only that many samples, and nothing else, reach the bound
            _check_c(x.view(np.uint16), kind, k, off)
    # 8191 keys above the bound and everything further share the last bin
    x = rng.integers(0, 3000, n).astype(np.int16)
    lo = np.sort(x[at])[::-1][_rank(n, 1) - 1]
    assert _rank(n, 1) == _rank(n, 3) == 8
    free = np.setdiff1d(np.arange(n), at)[[5, n // 2, n - 2000]]
    for d in (8189, 8190, 8191, 8192, 20000):
        for kk, other in ((1, 0), (2, 1), (3, -1)):
            y = x.copy()
            y[free] = [lo + d, lo + d + other, lo + d - other]
            _check_c(y.view(np.uint16), "int16", kk, off)


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("kind", ["float16", "bfloat16"])
def test_sampled_form_on_signs_and_specials(kind, off):
    """Candidates below zero (the bound and t negative), t among zeros of both signs, NaN and infinities among the
    candidates and as t."""
    n = (1 << 18) + 4099
    dt = {"float16": torch.float16, "bfloat16": torch.bfloat16}[kind]
    g = torch.Generator().manual_seed(7)
    neg = -torch.randn(n, generator=g).abs() - 1e-3
    neg = neg.to(dt).view(torch.int16).numpy().view(np.uint16).copy()
    for k in (1, 7, n // 100, n // 32):
        _check_c(neg, kind, k, off)
    x, r = neg.copy(), np.random.default_rng(5).permutation(n)
    inf = 0x7C00 if kind == "float16" else 0x7F80
    zeros, pos = r[: n // 100], r[n // 100: n // 100 + n // 200]
    x[zeros] = np.where(np.arange(zeros.size) % 3 == 0, 0x8000, 0)
    x[pos] ^= 0x8000
    s = r[n // 50: n // 50 + n // 1000]
    x[s] = np.resize(np.array([inf, inf | 0x8000, inf + 1, 0xFFFF], np.uint16), s.size)  # both infinities, both NaNs
    for k in (1, s.size // 2 - 3, s.size // 2 + 5, pos.size + 50, pos.size + n // 200, n // 64, n // 32):
        _check_c(x, kind, k, off)


@pytest.mark.parametrize("kind", ["int16", "float16", "bfloat16"])
@pytest.mark.parametrize("n", [1, 9, 4097, 32768, 32769, (1 << 18) - 1, 1_000_003])
def test_c_interface_types_and_alignment(kind, n):
    """All three forms on all bit patterns, from aligned inputs and from every other start."""
    bits = np.random.default_rng(n).integers(0, 1 << 16, n).astype(np.uint16)
    for off in (0, 1, 7):
        for k in sorted({1, min(n, 5), n // 40, n // 3, n} - {0}):
            _check_c(bits, kind, k, off)


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
