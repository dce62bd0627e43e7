"""The compaction at the edges of its tiles (2048 elements), groups (32 tiles)
and parts, for every element and index size: bit-exact, with outputs that do
not start on 16 bytes, capacities that cut a run, and both kinds of scratch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SIZES = [1, 511, 512, 513, 2047, 2048, 2049, 65535, 65536, 65537, 3 * 65536 + 2048 + 77]


def _ops():
    import tcuscan_ops
    from tcuscan_ops import _lib

    return tcuscan_ops, _lib


def _data(n, dtype, p, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randint(-100, 100, (n,), generator=g).to(dtype)
    # any nonzero byte selects
    m = torch.where(torch.rand(n, generator=g) < p, torch.randint(1, 256, (n,), generator=g), 0).to(torch.uint8)
    return x, m.view(torch.int8)


@pytest.mark.parametrize("dtype", [torch.int8, torch.int16, torch.float32, torch.int64])
@pytest.mark.parametrize("idx", [torch.int32, torch.int64])
@pytest.mark.parametrize("p", [0.0, 0.4, 1.0])
def test_compaction_edges(dtype, idx, p):
    ops, L = _ops()
    for n in SIZES:
        x, m = _data(n, dtype, p, n)
        xd, md = x.to(DEV), m.to(DEV)
        ix = torch.arange(n, dtype=idx) * 3 + 1
        sel = m.numpy() != 0
        assert np.array_equal(ops.run_compress(xd, md, 64).cpu().numpy(), x.numpy()[sel])
        v, i = ops.run_compress_ind(xd, ix.to(DEV), md, 64)
        assert np.array_equal(v.cpu().numpy(), x.numpy()[sel]) and np.array_equal(i.cpu().numpy(), ix.numpy()[sel])
        if idx == torch.int32:
            v, i = ops.run_compress_ind_no_arange(xd, md, 64)
            assert np.array_equal(v.cpu().numpy(), x.numpy()[sel]) and np.array_equal(i.cpu().numpy(), np.nonzero(sel)[0])
        v, i = ops.run_split_ind(xd, md, ix.to(DEV), 64)
        order = np.concatenate([np.nonzero(sel)[0], np.nonzero(~sel)[0]])
        assert np.array_equal(v.cpu().numpy(), x.numpy()[order]) and np.array_equal(i.cpu().numpy(), ix.numpy()[order])
        assert np.array_equal(ops.run_split(xd, md, 64).cpu().numpy(), x.numpy()[order])


@pytest.mark.parametrize("n", [2049, 70_001])
@pytest.mark.parametrize("dtype", [torch.int8, torch.float16, torch.float32, torch.float64])
def test_capacity_scratch_and_unaligned_indices(n, dtype):
    """The workspace entry points give what the scratch ones give; a capacity
    cuts the outputs; index outputs may start on any element."""
    ops, L = _ops()
    x, m = _data(n, dtype, 0.5, n + 1)
    xd, md = x.to(DEV), m.to(DEV)
    sel = np.nonzero(m.numpy())[0]
    ref = x.numpy()[sel]
    ws, wsb, sp = L.launch_context(torch.device(DEV), L.lib.tcu_workspace_bytes(n, 64))
    tb = L.lib.tcu_compact_tmp_bytes(n)
    tmp = torch.empty(tb, dtype=torch.uint8, device=DEV)
    eb = xd.element_size()
    for cap in (0, 1, 7, sel.size // 2 + 3, sel.size, sel.size + 100):
        for off in (0, 1, 3):
            for scratch in (False, True):
                z = torch.full((cap + 64,), 77, dtype=dtype, device=DEV)
                io = torch.full((cap + 64,), -5, dtype=torch.int32, device=DEV)
                cnt = torch.zeros(1, dtype=torch.int64, device=DEV)
                ip = io.data_ptr() + 4 * off
                if scratch:
                    L.check(L.lib.tcu_compact_count(md.data_ptr(), n, cnt.data_ptr(), tmp.data_ptr(), tb, sp), "count")
                    L.check(L.lib.tcu_compact_counted(xd.data_ptr(), eb, n, None, 4, 2, 0, z.data_ptr(), ip, cap,
                                                      tmp.data_ptr(), tb, sp), "counted")
                else:
                    L.check(L.lib.tcu_compress(xd.data_ptr(), eb, md.data_ptr(), n, None, 4, 2, z.data_ptr(), ip, cap,
                                               cnt.data_ptr(), ws, wsb, sp), "compress")
                k = min(cap, sel.size)
                assert int(cnt) == sel.size
                assert np.array_equal(z[:k].cpu().numpy(), ref[:k]) and bool((z[k:] == 77).all())
                assert np.array_equal(io[off:off + k].cpu().numpy(), sel[:k])
                assert bool((io[:off] == -5).all()) and bool((io[off + k:] == -5).all())


def test_compact_rejects():
    ops, L = _ops()
    x, m = _data(100, torch.int16, 0.5, 1)
    xd, md = x.to(DEV), m.to(DEV)
    tb = L.lib.tcu_compact_tmp_bytes(100)
    tmp = torch.empty(tb, dtype=torch.uint8, device=DEV)
    sp = L.stream_ptr(torch.device(DEV))
    assert L.lib.tcu_compact_count(md.data_ptr(), 100, None, tmp.data_ptr(), tb - 1, sp) == L.TCU_ERR_WORKSPACE
    assert L.lib.tcu_compact_count(md.data_ptr() + 1, 99, None, tmp.data_ptr(), tb, sp) == L.TCU_ERR_ALIGN
    assert L.lib.tcu_compact_counted(xd.data_ptr(), 3, 100, None, 0, 0, 0, tmp.data_ptr(), None, 0, tmp.data_ptr(), tb,
                                     sp) == L.TCU_ERR_DTYPE
    assert L.lib.tcu_compact_counted(xd.data_ptr(), 2, 100, None, 4, 2, 1, tmp.data_ptr(), tmp.data_ptr(), 100,
                                     tmp.data_ptr(), tb, sp) == L.TCU_ERR_ARG
