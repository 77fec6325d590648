"""Calls while device memory is short: the device's memory pool is replaced by one of a limited size, filled
up as far as a test wants, so that the library's stream-ordered allocations fail as they would with the
device's memory in other hands."""
import contextlib
import ctypes

import numpy as np
import pytest

from gazelle_plugin_gb300 import shuffle as S
from gazelle_plugin_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


class _Props(ctypes.Structure):  # CUmemPoolProps
    _fields_ = [("alloc_type", ctypes.c_int), ("handle_types", ctypes.c_int), ("location_type", ctypes.c_int),
                ("location_id", ctypes.c_int), ("security", ctypes.c_void_p), ("max_size", ctypes.c_size_t),
                ("usage", ctypes.c_ushort), ("reserved", ctypes.c_ubyte * 54)]


class Pool:
    """Device 0's current memory pool: at most `size` bytes."""

    def __init__(self, size):
        torch.zeros(1, device="cuda")  # the primary context is current
        self.cu = ctypes.CDLL("libcuda.so.1")
        self.dev = ctypes.c_int(0)
        props = _Props(alloc_type=1, location_type=1, max_size=size)  # PINNED on a DEVICE
        self.pool, self.before, self.held = ctypes.c_void_p(), ctypes.c_void_p(), []
        self._ok(self.cu.cuDeviceGetMemPool(ctypes.byref(self.before), self.dev))
        self._ok(self.cu.cuMemPoolCreate(ctypes.byref(self.pool), ctypes.byref(props)))
        self._ok(self.cu.cuDeviceSetMemPool(self.dev, self.pool))

    @staticmethod
    def _ok(r):
        assert r == 0, f"CUDA driver error {r}"

    def fill(self, leave=0):
        """Takes what is left of the pool, but for about `leave` bytes."""
        torch.cuda.synchronize()
        spare = ctypes.c_void_p()
        if leave:
            self._ok(self.cu.cuMemAllocFromPoolAsync(ctypes.byref(spare), ctypes.c_size_t(leave), self.pool, None))
        size = 1 << 30
        while size >= 4096:
            p = ctypes.c_void_p()
            r = self.cu.cuMemAllocFromPoolAsync(ctypes.byref(p), ctypes.c_size_t(size), self.pool, None)
            if r == 0:
                self.held.append(p)
            else:
                assert r == 2, r  # CUDA_ERROR_OUT_OF_MEMORY
                size //= 2
        if leave:
            self._ok(self.cu.cuMemFreeAsync(spare, None))
        torch.cuda.synchronize()

    def close(self):
        torch.cuda.synchronize()
        for p in self.held:
            self._ok(self.cu.cuMemFreeAsync(p, None))
        torch.cuda.synchronize()
        self._ok(self.cu.cuDeviceSetMemPool(self.dev, self.before))
        self._ok(self.cu.cuMemPoolDestroy(self.pool))


@contextlib.contextmanager
def pool(size):
    p = Pool(size)
    try:
        yield p
    finally:
        p.close()


def _resident_task(n, path, **kw):
    """A task whose outputs lie in device memory: the wide table in device buffers, split and waited for."""
    rng = np.random.default_rng(n)
    batches = [W.c2_batch(rng, 4096) for _ in range(n)]
    w = S.ShuffleSplitterJniWrapper()
    h = w.make(S.NativePartitioning("hash", 200, None, W.C2_KEYS, list(W.C2_SCHEMA)), dataFile=path,
               input_kind=S.GZ_INPUT_DEVICE_RETAINED, keep_output_on_device=1, **kw)
    keep = []
    for b in batches:
        t = [torch.from_numpy(x.view(np.uint8).copy()).cuda() if x.nbytes else None for x in b.buffers]
        keep.append(t)
        a = np.array([0 if x is None else x.data_ptr() for x in t], np.int64)
        torch.cuda.synchronize()
        w.split(h, b.num_rows, a, b.addrs_sizes()[1])
    w.sync(h)
    return w, h, batches, keep


def test_a_failed_stop_leaves_no_data_in_memory():
    """Without a data file Stop's bytes are read with gz_split_data: all of them after a Stop that worked, none
    after one that did not."""
    with pool(1 << 30) as p:
        w, h, batches, keep = _resident_task(40, "")
        p.fill()
        try:
            w.stop(h)
        except S.SplitterError:
            assert w.data(h) == b""
        else:
            assert w.data(h) == O.run_oracle(W.C2_SCHEMA, batches, 200, W.C2_KEYS).data
        w.close(h)
        del keep


@pytest.mark.parametrize("n", [40, 120])
@pytest.mark.parametrize("to_file", [False, True])
def test_stop_writes_without_device_memory_of_its_own(tmp_path, n, to_file):
    """Stop writes a task's outputs with no byte of device memory left (files of two windows and of several)."""
    path = str(tmp_path / "x.data") if to_file else ""
    with pool(1 << 30) as p:
        w, h, batches, keep = _resident_task(n, path)
        p.fill()
        w.stop(h)
        data = open(path, "rb").read() if to_file else w.data(h)
        w.close(h)
        del keep
    assert data == O.run_oracle(W.C2_SCHEMA, batches, 200, W.C2_KEYS).data


def test_stop_compresses_with_device_memory_for_the_bodies_only(tmp_path):
    """Under LZ4_FRAME Stop needs device memory for the compressed bodies: with less it says so, with that
    much and no more (the steps go past it) it writes the bytes of a Stop that has all it wants."""
    path = str(tmp_path / "x.data")
    want, states = None, []
    for leave in [256 << 20] + [x << 20 for x in range(16, 96, 4)]:
        with pool(1 << 30) as p:
            w, h, _, keep = _resident_task(60, path, codec="lz4")
            p.fill(leave)
            try:
                w.stop(h)
                data = open(path, "rb").read()
                want = want or data
                assert data == want
                states.append(True)
            except S.SplitterError as e:
                assert e.status == S.GZ_OOM and "partition" not in str(e) and "data file" not in str(e), e
                states.append(False)
            w.close(h)
            del keep
    assert states[1:] == sorted(states[1:]) and states[0] and states[-1] and not states[1]


def test_compressed_streams_are_read_with_memory_for_image_and_columns_only():
    """A compressed stream needs its image and its decoded buffers; the decoder that takes a block a CTA wants
    as much again, and without it the frames are decoded the slower way."""
    rng = np.random.default_rng(3)
    schema = [W.Field("k", "int64", False)]
    batches = [W.Batch(n, W._column(rng, schema[0], n, rng.integers(0, 50, size=n), 0.0)) for n in (2_000_000, 2_000_003)]
    res, data = S.split_batches(schema, batches, 1, [0], codec="lz4")
    stream = np.frombuffer(data, np.uint8)
    want = np.concatenate([b.buffers[1].view(np.int64) for b in batches])
    assert stream.nbytes < want.nbytes // 2
    read = []
    # the image, the decoded buffers and their tables, but not as much again; then all that is wanted
    for leave in (stream.nbytes + want.nbytes * 5 // 4 + (4 << 20), stream.nbytes + want.nbytes * 4):
        with pool(1 << 30) as p:
            r = S.PartitionReader(schema)
            p.fill(leave)
            r.addStream(stream)
            for q in p.held:
                p._ok(p.cu.cuMemFreeAsync(q, None))
            p.held = []
            torch.cuda.synchronize()
            r.finish()
            read.append(r.column_to_host(0))
            r.close()
    for c in read:
        assert np.array_equal(np.asarray(c[2]).view(np.int64), want)


def test_a_reader_without_device_memory_reads_streams_without_rows():
    """With no byte left a reader is made, takes streams without record batches, reports a malformed one as that
    and one with rows as out of memory; and reads it once there is memory."""
    schema = [W.Field("k", "int64", False)]
    rng = np.random.default_rng(4)
    batch = W.Batch(5000, W._column(rng, schema[0], 5000, rng.integers(0, 50, size=5000), 0.0))
    stream = S.split_batches(schema, [batch], 1, [0], writeSchema=True)[1]
    eos = stream[-8:]
    schema_only = stream[:8 + int.from_bytes(stream[4:8], "little")] + eos

    def status(r, s):
        try:
            r.addStream(np.frombuffer(s, np.uint8))
        except S.SplitterError as e:
            return e.status
        return S.GZ_OK

    with pool(64 << 20) as p:
        p.fill()
        r = S.PartitionReader(schema)
        assert [status(r, s) for s in (schema_only, eos, b"", stream[:-20], b"\1" * 64)] == [S.GZ_OK] * 3 + [S.GZ_INVALID] * 2
        assert status(r, stream) == S.GZ_OOM
        for q in p.held:
            p._ok(p.cu.cuMemFreeAsync(q, None))
        p.held = []
        torch.cuda.synchronize()
        assert status(r, stream) == S.GZ_OK
        assert r.finish()[0] == 5000
        assert np.array_equal(np.asarray(r.column_to_host(0)[2]).view(np.int64), batch.buffers[1].view(np.int64))
        r.close()
