"""Stop's data file put together by the device (k_emit, from four megabytes of input on): the bytes of the
oracle, and with a codec those of the path that gathers them on the host (taken when local-dir spill
files may hold passes), over host and device-resident inputs, one and many passes, data in a file
and in memory, record batches that span passes, files of one and of many windows."""
import os

import numpy as np
import pytest

from gazelle_plugin_gb300 import shuffle as S
from gazelle_plugin_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

F = W.Field
NESTED = [F("k", "int64", False), F("b", "bool"), F("d", "decimal128"), F("l", "list", True, "bool"),
          F("n", "list", True, None, (F("item", "struct", True, None, (F("a", "int32"), F("s", "utf8"))),)),
          F("z", "null"), F("u", "large_utf8")]


def _nested(rng, n):
    bufs = []
    for f in NESTED:
        if f.type == "null":
            bufs += [np.zeros(0, np.uint8)] * 2
        elif f.is_list:
            bufs += W.list_column(rng, f, n, 0.1, 0.1, 9)
        elif f.is_nested or f.is_binary or f.type in ("bool", "decimal128"):
            bufs += W.nested_column(rng, f, n, 0.1, 5)
        else:
            bufs += W._column(rng, f, n, rng.integers(0, 1 << 40, size=n), 0.0)
    return W.Batch(n, bufs)


def _batches(which, n):
    rng = np.random.default_rng(n)
    if which == "c1":
        return W.C1_SCHEMA, W.C1_KEYS, [W.c1_batch(rng, 3001) for _ in range(n)]
    if which == "c2":
        return W.C2_SCHEMA, W.C2_KEYS, [W.c2_batch(rng, 4096) for _ in range(n)]
    return NESTED, [0], [_nested(rng, 2500) for _ in range(n)]


def _run(schema, keys, P, batches, path, device=False, **kw):
    w = S.ShuffleSplitterJniWrapper()
    h = w.make(S.NativePartitioning("hash", P, None, keys, list(schema)), dataFile=path,
               input_kind=S.GZ_INPUT_DEVICE_RETAINED if device else S.GZ_INPUT_HOST, **kw)
    try:
        keep = []
        for b in batches:
            a, z = b.addrs_sizes()
            if device:
                t = [torch.from_numpy(x.view(np.uint8).copy()).cuda() if x.nbytes else None for x in b.buffers]
                keep.append(t)
                a = np.array([0 if x is None else x.data_ptr() for x in t], np.int64)
                torch.cuda.synchronize()
            w.split(h, b.num_rows, a, z)
        r = w.stop(h)
        data = open(path, "rb").read() if path else w.data(h)
    finally:
        w.close(h)
    assert len(data) == int(r.partitionLengths.sum())
    return data, r


# (input, batches, partitions): a little over that, two windows; several windows; many windows of
# tiny partitions; lists, nested columns and null-type columns; one partition with pieces of megabytes
CASES = [("c1", 44, 8), ("c2", 40, 200), ("c2", 40, 3000), ("nested", 30, 64), ("c2", 60, 1)]


@pytest.mark.parametrize("which,n,P", CASES)
@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("flush", [0, 1 << 20])
def test_emit_equals_oracle(tmp_path, which, n, P, device, flush):
    schema, keys, batches = _batches(which, n)
    assert sum(b.nbytes for b in batches) >= 4 << 20
    want = O.run_oracle(schema, batches, P, keys)
    opts = dict(flush_bytes=flush) if flush else {}
    for path in (str(tmp_path / "x.data"), ""):
        data, r = _run(schema, keys, P, batches, path, device, **opts)
        assert data == want.data
        assert np.array_equal(r.rawPartitionLengths, want.raw_partition_lengths)


@pytest.mark.parametrize("which,n,P", CASES)
def test_emit_lz4_equals_host_gather(tmp_path, which, n, P):
    schema, keys, batches = _batches(which, n)
    for device in (False, True):
        got, _ = _run(schema, keys, P, batches, str(tmp_path / "x.data"), device, codec="lz4", writeSchema=True, flush_bytes=3 << 20)
        want, _ = _run(schema, keys, P, batches, str(tmp_path / "y.data"), device, codec="lz4", writeSchema=True, flush_bytes=3 << 20,
                       host_budget=1 << 40, localDirs=str(tmp_path))
        assert got == want


@pytest.mark.parametrize("which,n,P", [("c1", 1, 8), ("c1", 10, 2500), ("c2", 5, 64), ("nested", 6, 900)])
def test_small_files_written_once_equal_oracle(tmp_path, which, n, P):
    """Below that the CPU gathers the partitions and writes them with one call."""
    schema, keys, batches = _batches(which, n)
    data, _ = _run(schema, keys, P, batches, str(tmp_path / "x.data"))
    assert data == O.run_oracle(schema, batches, P, keys).data


def test_emit_rewrites_a_longer_file_and_reports_a_bad_path(tmp_path):
    schema, keys, batches = _batches("c1", 44)
    path = str(tmp_path / "x.data")
    with open(path, "wb") as f:
        f.write(b"\xee" * (16 << 20))
    data, _ = _run(schema, keys, 8, batches, path)
    assert data == O.run_oracle(schema, batches, 8, keys).data
    with pytest.raises(S.SplitterError) as e:
        _run(schema, keys, 8, batches, str(tmp_path / "no" / "x.data"))
    assert e.value.status == S.GZ_IO
    _run_null = S.ShuffleSplitterJniWrapper()
    h = _run_null.make(S.NativePartitioning("hash", 8, None, keys, list(schema)), dataFile=os.devnull)
    for b in batches:
        a, z = b.addrs_sizes()
        _run_null.split(h, b.num_rows, a, z)
    assert int(_run_null.stop(h).partitionLengths.sum()) == len(data)
    _run_null.close(h)


@pytest.mark.parametrize("codec", ["uncompressed", "lz4"])
@pytest.mark.parametrize("device", [False, True])
def test_spill_after_stop(tmp_path, device, codec):
    """A memory manager may ask a task that has stopped to spill: the policy's bytes, as of a task whose file the
    host gathers, and nothing is moved any more."""
    schema, keys, batches = _batches("c2", 40)
    got = []
    for kw in ({}, dict(host_budget=1 << 40, localDirs=str(tmp_path))):
        w = S.ShuffleSplitterJniWrapper()
        h = w.make(S.NativePartitioning("hash", 200, None, keys, list(schema)), dataFile=str(tmp_path / "x.data"), codec=codec,
                   bufferSize=64, preferSpill=False, input_kind=S.GZ_INPUT_DEVICE_RETAINED if device else S.GZ_INPUT_HOST, **kw)
        keep = []
        for b in batches:
            a, z = b.addrs_sizes()
            if device:
                t = [torch.from_numpy(x.view(np.uint8).copy()).cuda() if x.nbytes else None for x in b.buffers]
                keep.append(t)
                a = np.array([0 if x is None else x.data_ptr() for x in t], np.int64)
                torch.cuda.synchronize()
            w.split(h, b.num_rows, a, z)
        w.stop(h)
        moved = w.stats(h)[3]
        got.append([w.nativeSpill(h, 1 << 40), w.nativeSpill(h, 1)])
        assert w.stats(h)[3] == moved or kw
        w.sync(h)
        w.close(h)
    assert got[0] == got[1] and got[0][0] > 0
