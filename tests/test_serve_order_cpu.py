"""Stream order of the serving loop, without a GPU.

The server runs on a model of CUDA streams: every operation it queues (through
the C interface or through torch) is written down with the set of operations
that are certain to come before it -- those of its own stream and those that a
recorded event or a stream wait brings along.  What the loop's correctness
needs is then a statement about these sets: the operations a caller queued
before must be in the set of every operation that reads or overwrites the same
memory.
"""
import contextlib
import ctypes
import types

import numpy as np
import pytest
import torch


class Stream:
    made = 0

    def __init__(self, model, name):
        self.model, self.name, self.before = model, name, frozenset()
        Stream.made += 1
        self.cuda_stream = 1000 + Stream.made
        model.streams[self.cuda_stream] = self

    def op(self, what):
        """Queue an operation; returns its id."""
        i = len(self.model.ops)
        self.model.ops.append((what, self, self.before))
        self.before = self.before | {i}
        return i

    def wait_stream(self, other):
        self.before = self.before | other.before

    def wait_event(self, ev):
        self.before = self.before | ev.point

    def synchronize(self):
        self.model.done |= self.before


class Event:
    def __init__(self, model):
        self.model, self.point = model, frozenset()

    def record(self, stream=None):
        self.point = (stream or self.model.current).before

    def query(self):
        if not self.model.busy:
            self.model.done |= self.point
        return not self.model.busy

    def synchronize(self):
        self.model.done |= self.point


class Model:
    """Streams, and a C interface whose calls only queue operations."""

    def __init__(self):
        self.ops, self.streams, self.done, self.fail, self.busy = [], {}, frozenset(), None, False
        self.error = (0, 0, 0)
        self.current = Stream(self, "caller")

    def __getattr__(self, name):  # lib.tcu_*
        if not name.startswith("tcu_"):
            raise AttributeError(name)

        def call(*args):
            if name.endswith("_bytes"):
                return 1 << 12
            if name == self.fail:
                return 3  # TCU_ERR_LAUNCH
            if name == "tcu_copy_async" and args[2] == 12:  # the slot's error words
                ctypes.memmove(args[0], (ctypes.c_uint32 * 3)(*self.error), 12)
            self.streams[args[-1].value].op(name)
            return 0

        return call

    def find(self, name):
        return [(i, s, before) for i, (what, s, before) in enumerate(self.ops) if what == name]


@pytest.fixture
def model(monkeypatch):
    from tcuscan_b200 import serve
    from tcuscan_ops import _lib

    m = Model()
    cuda = types.SimpleNamespace(
        current_device=lambda: 0, device=lambda d: contextlib.nullcontext(),
        Stream=lambda dev=None: Stream(m, "slot"), Event=lambda enable_timing=False: Event(m),
        current_stream=lambda dev=None: m.current, is_current_stream_capturing=lambda: False)

    class Torch:
        def __getattr__(self, name):
            return getattr(torch, name)

        @staticmethod
        def empty(*a, **k):
            k.pop("device", None)
            k.pop("pin_memory", None)
            return torch.zeros(*a, **k)

    shim = Torch()
    shim.cuda = cuda

    class Lib:
        def __getattr__(self, name):
            return getattr(_lib, name)

    lib = Lib()
    lib.lib = m
    lib._stream_key = lambda dev: (0, m.current.cuda_stream)
    monkeypatch.setattr(serve, "torch", shim)
    monkeypatch.setattr(serve, "_lib", lib)
    return m


def _server(m, **kw):
    from tcuscan_b200 import serve

    return serve.Server("cuda:0", budget_bytes=4 << 20, slots=2, keep_results=True, **kw)


def _submit(srv, op, n=5000, k=1, dt=0, nseg=40, iw=4):
    """k requests (int8 unless dt says otherwise) on memory of nobody's (the model reads nothing)."""
    n = np.broadcast_to(n, k)
    return srv.submit_many(np.full(k, op, np.int8), np.full(k, dt, np.int8), n, np.full(k, 4096, np.uint64),
                           np.full(k, 8192, np.uint64), np.broadcast_to(nseg if op == 1 else 0, k),
                           np.full(k, iw if op == 1 else 0, np.int8), np.full(k, srv.now()))


def test_construction_follows_the_callers_work(model):
    """The workspaces and the arena may be memory that the caller's queued work still uses (a temporary just
    freed): nothing of the server touches them before that work, and what the caller queues next on memory of a
    server that is gone comes after the server's own."""
    late = model.current.op("a temporary's last kernel")
    srv = _server(model)
    inits = model.find("tcu_workspace_init")
    assert len(inits) == 2
    for i, s, before in inits:
        assert late in before
        assert i in model.current.before  # the caller's next kernel may get this block again
    for sl in srv.slots:
        assert late in sl.stream.before and all(i in sl.stream.before for i, _, _ in inits)


def test_a_refused_server_leaves_nothing_queued(model):
    from tcuscan_b200 import serve

    with pytest.raises(ValueError):
        serve.Server("cuda:0", budget_bytes=1 << 16, slots=2)
    for i, s, before in model.find("tcu_workspace_init"):
        assert i in model.current.before


def test_batches_follow_the_work_that_fills_their_requests(model):
    """Whatever a caller queued on its stream before submit(), before run() or -- on another stream -- before
    submitting from there precedes every kernel of the batch."""
    from tcuscan_b200 import serve

    srv = _server(model)
    early = model.current.op("input of the first request")
    _submit(srv, serve.SCAN)
    main, side = model.current, Stream(model, "side")
    model.current = side
    aside = side.op("input of the second request")
    _submit(srv, serve.SEG_SUM)
    model.current = main
    late = main.op("queued between submit and run")
    n0 = len(model.ops)
    srv.run()
    queued = model.ops[n0:]
    assert {w for w, _, _ in queued} >= {"tcu_copy_async", "tcu_pack"}
    for what, s, before in queued:
        assert {early, aside, late} <= before, what


def test_release_keeps_the_readers_of_results_ahead(model):
    """After release() a block may be overwritten: the kernels that read the results queued before come first."""
    from tcuscan_b200 import serve

    srv = _server(model)
    r = _submit(srv, serve.SCAN)[0]
    srv.run()
    assert srv.result(r).numel() == 5000
    main, side = model.current, Stream(model, "side")
    model.current = side
    reader = side.op("reads the result")
    srv.release()
    model.current = main
    _submit(srv, serve.SCAN, k=3)
    n0 = len(model.ops)
    srv.run()
    assert len(model.ops) > n0 and all(reader in before for _, _, before in model.ops[n0:])


@pytest.mark.parametrize("op,fails", [(0, "tcu_seg_bounds"), (1, "tcu_pack"), (2, "tcu_compress_segments")])
def test_a_launch_that_fails_half_way_gives_everything_back(model, op, fails):
    """The copies and kernels queued before the failing call have ended before the error leaves the loop (the
    batch is not registered anywhere); the slot and the block are free again and serve the next batch."""
    from tcuscan_b200 import serve
    from tcuscan_ops import TcuError

    srv = _server(model)
    whole = list(srv.arena.free)
    _submit(srv, op)
    n0 = len(model.ops)
    model.fail = fails
    with pytest.raises(TcuError):
        srv.run()
    slot_ops = {i for i, (w, s, _) in enumerate(model.ops) if i >= n0 and s.name == "slot"}
    assert slot_ops and slot_ops <= model.done
    assert srv.used == 0 and srv.arena.free == whole
    assert sorted(srv.free_slots) == [0, 1] and not srv.inflight
    model.fail = None
    r = _submit(srv, op)[0]
    srv.run()
    srv.result(r)


def test_an_undersized_block_is_seen_before_anything_is_queued(model, monkeypatch):
    from tcuscan_b200 import serve

    srv = _server(model)
    whole = list(srv.arena.free)
    _submit(srv, serve.SCAN)
    monkeypatch.setattr(srv, "_take", lambda cls, room, take=srv._take: (take(cls, room)[0], 4096))
    n0 = len(model.ops)
    with pytest.raises(AssertionError):
        srv.run()
    assert {w for w, _, _ in model.ops[n0:]} <= {"tcu_workspace_init"}  # the slot's workspace, not the block
    assert srv.arena.free == whole and len(srv.free_slots) == 2


def test_a_server_that_goes_away_waits_for_its_streams(model):
    """PyTorch does not see the copies from the pinned tables: they have ended before the tables, the workspaces
    and the arena go back to their allocators -- also those of a batch that no list holds."""
    from tcuscan_b200 import serve

    srv = _server(model)
    _submit(srv, serve.COMPRESS)
    model.busy = True
    srv.step()
    srv.slots[1].stream.op("a copy that nothing registered")
    srv.__del__()
    assert {i for i, (w, s, _) in enumerate(model.ops) if s.name == "slot"} <= model.done
    serve.Server.__del__(object.__new__(serve.Server))  # a constructor that raised


@pytest.mark.parametrize("op", [0, 1, 2])
def test_a_device_error_is_raised_instead_of_results(model, op):
    """A bounded wait that ran out is recorded in the slot's workspace: the loop raises it, hands out nothing of
    the batch, and serves on with the slot's workspace reset."""
    from tcuscan_ops import TcuError

    srv = _server(model)
    whole = list(srv.arena.free)
    r = _submit(srv, op)[0]
    model.error = (4, 100, 7)
    with pytest.raises(TcuError, match="site 100, chunk 7"):
        srv.run()
    with pytest.raises(RuntimeError):
        srv.result(r)
    assert srv.arena.free == whole and srv.used == 0 and len(srv.free_slots) == 2 and not srv.inflight
    assert [s.name for _, s, _ in model.find("tcu_workspace_init")][2:] == ["slot"]
    model.error = (0, 0, 0)
    r = _submit(srv, op)[0]
    srv.run()
    srv.result(r)


@pytest.mark.parametrize("op,iw", [(0, 0), (1, 4), (1, 8), (2, 0)])
@pytest.mark.parametrize("dt", [0, 1, 2])
def test_blocks_hold_what_the_batches_lay_out(model, monkeypatch, op, iw, dt):
    """Admission sizes a block before the launch lays it out (and refuses one that is too small): every op, dtype
    and row-pointer width, requests of every length, packed and in place, with no more slack than the rounding of
    the block's buffers (at most six) to BLOCK_ALIGN takes."""
    from tcuscan_b200 import serve

    rng = np.random.default_rng(100 * op + 10 * iw + dt)
    monkeypatch.setattr(serve, "SOLO_MIN", 1 << 12)
    monkeypatch.setattr(serve, "BATCH_SLACK", 6 * serve.BLOCK_ALIGN)
    srv = serve.Server("cuda:0", budget_bytes=64 << 20, slots=2)
    for k in (1, 1, 2, 7, 40, 300):
        n = np.exp(rng.uniform(0, np.log(9000), size=k)).astype(np.int64)
        _submit(srv, op, n, k, dt, nseg=rng.integers(0, 400, size=k), iw=iw)
        srv.run()
    assert srv.used == 0 and np.isfinite(srv.done[: srv._n]).all()
