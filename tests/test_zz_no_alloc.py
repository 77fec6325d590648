"""gz_hash_partition_static, the entry point that allocates no device memory.

Some callers cannot call cudaMalloc: their device memory all belongs to another allocator (a
pool that reserved the free HBM up front, or an executor that charges every device byte to a
task's budget), or they must not let cudaMalloc / cudaFree stall the device.  For them the
library computes a batch's partition ids and per-partition row counts with its scratch in a
fixed 16 MiB device array of its own.

Checked through the C ABI, exactly, against the oracle's partition ids and against the
splitter's own (gz_split_last_pids) for the same batch, on calls in a row that share and reuse
that array (shared-memory and global-memory count paths, then the first case again, and a key
list with a null-type key, which leaves the hash unchanged).  Around every call after the first,
the device's free memory must not change: the call allocates nothing.  Collected last so that a
run stopping at the first failure has run every other test first; it also passes alone in a
fresh process.
"""
import ctypes

import numpy as np
import pytest

from gazelle_plugin_gb300 import shuffle as S
from gazelle_plugin_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

MAX_COUNTERS = 4 * 1024 * 1024  # per-tile counters the static array holds
TILE_ROWS = 1024


class GzKeyColumn(ctypes.Structure):
    _fields_ = [("type", ctypes.c_int32), ("reserved", ctypes.c_int32),
                ("validity", ctypes.c_void_p), ("values", ctypes.c_void_p)]


def _entry():
    f = S.lib().gz_hash_partition_static
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int32, ctypes.c_int32, ctypes.POINTER(GzKeyColumn), ctypes.c_int32,
                  ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    return f


def _last_error() -> str:
    buf = ctypes.create_string_buffer(1024)
    S.lib().gz_last_error(0, buf, len(buf))
    return buf.value.decode()


def _splitter_pids(schema, keys, P, batch):
    """Partition ids from the existing entry points: make, split (host buffers), last_pids."""
    w = S.ShuffleSplitterJniWrapper()
    h = w.make(S.NativePartitioning("hash", P, None, keys, list(schema)), writeSchema=False)
    try:
        addrs, sizes = batch.addrs_sizes()
        w.split(h, batch.num_rows, addrs, sizes)
        return w.lastPids(h, batch.num_rows)
    finally:
        w.close(h)


def _oracle_pids(schema, keys, P, batch):
    o = O.OracleSplitter(schema, P, keys)
    try:
        o.split(batch)
        return o.last_pids(batch.num_rows)
    finally:
        o.close()


def _device_keys(schema, keys, batch):
    """Key columns copied to the device; returns the ctypes array and the tensors that own it."""
    first = []
    b = 0
    for f in schema:
        first.append(b)
        b += 3 if f.is_binary else 2
    hold, cols = [], (GzKeyColumn * len(keys))()
    for j, k in enumerate(keys):
        cols[j].type = schema[k].code
        if schema[k].type == "null":  # no buffers are read
            cols[j].values = None
            cols[j].validity = None
            continue
        valid = batch.buffers[first[k]].view(np.uint8)
        vals = batch.buffers[first[k] + 1].view(np.uint8)
        dv = torch.from_numpy(vals.copy()).cuda()
        hold.append(dv)
        cols[j].values = dv.data_ptr()
        if valid.nbytes:
            dm = torch.from_numpy(valid.copy()).cuda()
            hold.append(dm)
            cols[j].validity = dm.data_ptr()
        else:
            cols[j].validity = None
    return cols, hold


def _static_call(schema, keys, P, batch):
    cols, hold = _device_keys(schema, keys, batch)
    n = batch.num_rows
    pids16 = torch.full((max(n, 1),), -1, dtype=torch.int16, device="cuda")  # 0xFFFF: unwritten
    counts = torch.full((P,), -1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    free_before = torch.cuda.mem_get_info()[0]
    st = _entry()(0, P, cols, len(keys), n, pids16.data_ptr(), counts.data_ptr(),
                  torch.cuda.current_stream().cuda_stream)
    assert st == 0, _last_error()
    torch.cuda.synchronize()
    free_after = torch.cuda.mem_get_info()[0]
    del hold
    got = pids16[:n].cpu().numpy().view(np.uint16)
    return got, counts.cpu().numpy(), free_before - free_after


def _with_null_key():
    """The c1 schema with a null-type field in front, listed first among the keys."""
    schema = [W.Field("n", "null")] + list(W.C1_SCHEMA)
    b = W.c1_batches(44, 1, 3000)[0]
    empty = np.zeros(0, np.uint8)
    batch = W.Batch(b.num_rows, [empty, empty] + list(b.buffers))
    return schema, [0] + [k + 1 for k in W.C1_KEYS], batch


CASES = [
    # P <= 12288: the tile histogram is counted in shared memory
    ("c2", W.C2_SCHEMA, W.C2_KEYS, 200, lambda: W.c2_batches(41, 1, 20000)[0]),
    # P > 12288: counted in the static array itself (cleared per tile), null keys
    ("c3", W.C3_SCHEMA, W.C3_KEYS, 20000, lambda: W.c3_batches(42, 1, 32768, 0.2, 0.05)[0]),
    # the first case again, after the second left its counts in the array
    ("c2-again", W.C2_SCHEMA, W.C2_KEYS, 200, lambda: W.c2_batches(41, 1, 20000)[0]),
    ("c1", W.C1_SCHEMA, W.C1_KEYS, 8, lambda: W.c1_batches(43, 1, 5000)[0]),
]


def test_static_scratch_matches_oracle_and_splitter_on_consecutive_calls():
    cases = [(tag, schema, keys, P, make()) for tag, schema, keys, P, make in CASES]
    nschema, nkeys, nbatch = _with_null_key()
    cases.append(("null-type key", nschema, nkeys, 8, nbatch))
    for i, (tag, schema, keys, P, batch) in enumerate(cases):
        want = _oracle_pids(schema, keys, P, batch)
        assert np.array_equal(_splitter_pids(schema, keys, P, batch), want), tag
        got, counts, grown = _static_call(schema, keys, P, batch)
        assert np.array_equal(got, want), tag
        assert np.array_equal(counts, np.bincount(want, minlength=P).astype(np.int64)), tag
        if i > 0:  # the first call on the device may load the module that holds the array
            assert grown == 0, f"{tag}: free device memory fell by {grown} bytes during the call"


def test_static_scratch_rejects_oversized_call():
    cols = (GzKeyColumn * 1)()
    dummy = torch.zeros(8, dtype=torch.int64, device="cuda")
    cols[0].type = W.TYPE_CODES["int64"]
    cols[0].values = dummy.data_ptr()
    P = 65536
    rows = (MAX_COUNTERS // P) * TILE_ROWS + 1  # one tile more than the array holds
    st = _entry()(0, P, cols, 1, rows, dummy.data_ptr(), dummy.data_ptr(), None)
    assert st == S.GZ_INVALID
    assert "static scratch" in _last_error()


@pytest.fixture(scope="module")
def many_keys():
    """One batch with a key of every width, nulls in all, and the Spark hash's ids by P."""
    n = 70001
    rng = np.random.default_rng(7)
    schema = [W.Field(f"k{i}", t) for i, t in enumerate(("int64", "int32", "int16", "int8", "bool", "float64"))]
    bufs = []
    for f in schema:
        v = rng.standard_normal(n) if f.type == "float64" else rng.integers(0, 2 if f.type == "bool" else 120, n)
        bufs += W._column(rng, f, n, v, 0.2)
    batch = W.Batch(n, bufs)
    ids = {}

    def pids(P):
        if P not in ids:
            ids[P] = _oracle_pids(schema, list(range(len(schema))), P, batch)
        return ids[P]

    return schema, batch, pids


# both sides of the lines of the dispatch by partitions (histograms of blocks of 512 and of 1024 threads, histograms
# counted in the scratch), over rows around the 1024 of the limit on a call and their multiples
@pytest.mark.parametrize("P", [1, 8, 2048, 2049, 12288, 12289, 24577, 57344, 57345])
@pytest.mark.parametrize("shift", [0, 1])
def test_static_ids_and_counts_over_sizes(many_keys, P, shift):
    schema, batch, pids = many_keys
    cols = (GzKeyColumn * len(schema))()
    hold = []
    for j, f in enumerate(schema):
        valid, vals = batch.buffers[2 * j].view(np.uint8), batch.buffers[2 * j + 1].view(np.uint8)
        w = W.BYTE_WIDTH.get(f.type, 1) * shift  # values one element off the allocation's alignment
        t = torch.from_numpy(np.concatenate([np.zeros(w, np.uint8), vals])).cuda()
        m = torch.from_numpy(np.concatenate([np.zeros(shift, np.uint8), valid])).cuda()
        hold += [t, m]
        cols[j].type, cols[j].values, cols[j].validity = f.code, t.data_ptr() + w, m.data_ptr() + shift
    for n in (1, 3, 1023, 1024, 1025, 8192, 8193, 32767, 32768, 32769, batch.num_rows):
        if -(-n // TILE_ROWS) * P > MAX_COUNTERS:
            continue
        out = torch.full((n + 1 + shift,), -1, dtype=torch.int16, device="cuda")
        counts = torch.full((P,), -1, dtype=torch.int64, device="cuda")
        st = _entry()(0, P, cols, len(schema), n, out.data_ptr() + 2 * shift, counts.data_ptr(),
                      torch.cuda.current_stream().cuda_stream)
        assert st == 0, _last_error()
        got = out.cpu().numpy().view(np.uint16)
        want = pids(P)[:n]
        assert np.array_equal(got[shift:shift + n], want), (n, P)
        assert got[shift + n] == 0xFFFF  # nothing past the last row
        assert np.array_equal(counts.cpu().numpy(), np.bincount(want, minlength=P)), (n, P)
    del hold


def test_static_calls_in_a_row_and_in_a_captured_graph(many_keys):
    """Calls whose kernels may come up while the previous call's still run: each call reads the keys that
    the kernel before it wrote and the scratch rows of its own counting kernel; the same in a graph."""
    schema, batch, pids = many_keys
    n, P = 20000, 2000
    v = torch.from_numpy(batch.buffers[1].view(np.int64)[:n].copy()).cuda()
    keys = [torch.empty_like(v) for _ in range(4)]
    outs = [(torch.empty(n, dtype=torch.int16, device="cuda"), torch.empty(P, dtype=torch.int64, device="cuda")) for _ in keys]
    cols = [(GzKeyColumn * 1)() for _ in keys]
    for c, k in zip(cols, keys):
        c[0].type, c[0].values, c[0].validity = W.TYPE_CODES["int64"], k.data_ptr(), None

    def calls(stream):
        for i, (k, (o, cnt)) in enumerate(zip(keys, outs)):
            k.copy_(v + i)
            assert _entry()(0, P, cols[i], 1, n, o.data_ptr(), cnt.data_ptr(), stream) == 0, _last_error()

    def check():
        for i, (o, cnt) in enumerate(outs):
            b = W.Batch(n, [np.zeros(0, np.uint8), (v.cpu().numpy() + i).view(np.uint8)])
            want = _oracle_pids([W.Field("k", "int64")], [0], P, b)
            assert np.array_equal(o.cpu().numpy().view(np.uint16), want)
            assert np.array_equal(cnt.cpu().numpy(), np.bincount(want, minlength=P))

    calls(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    check()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        calls(torch.cuda.current_stream().cuda_stream)
    for _ in range(3):
        for o, cnt in outs:
            o.zero_()
            cnt.zero_()
        g.replay()
        torch.cuda.synchronize()
        check()


# keys of one kind (their kernel, and the general one when a column or the ids lie off their boundaries)
@pytest.mark.parametrize("off", ["", "last key", "ids"])
@pytest.mark.parametrize("P", [1, 200, 3000, 57345])
@pytest.mark.parametrize("keys", [[1], [0], [0, 5]])
def test_static_ids_of_keys_of_one_kind(many_keys, keys, P, off):
    schema, batch, _ = many_keys
    want_all = _oracle_pids(schema, keys, P, batch)
    cols = (GzKeyColumn * len(keys))()
    hold = []
    for j, k in enumerate(keys):
        f = schema[k]
        w = W.BYTE_WIDTH[f.type] if off == "last key" and k == keys[-1] else 0
        t = torch.from_numpy(np.concatenate([np.zeros(w, np.uint8), batch.buffers[2 * k + 1].view(np.uint8)])).cuda()
        m = torch.from_numpy(batch.buffers[2 * k].view(np.uint8).copy()).cuda()
        hold += [t, m]
        cols[j].type, cols[j].values, cols[j].validity = f.code, t.data_ptr() + w, m.data_ptr()
    for n in (1, 4, 2047, 2048, 2051, 65533):
        if -(-n // TILE_ROWS) * P > MAX_COUNTERS:
            continue
        shift = int(off == "ids")
        out = torch.full((n + 2,), -1, dtype=torch.int16, device="cuda")
        counts = torch.full((P,), -1, dtype=torch.int64, device="cuda")
        st = _entry()(0, P, cols, len(keys), n, out.data_ptr() + 2 * shift, counts.data_ptr(),
                      torch.cuda.current_stream().cuda_stream)
        assert st == 0, _last_error()
        got = out.cpu().numpy().view(np.uint16)
        assert np.array_equal(got[shift:shift + n], want_all[:n])
        assert got[shift + n] == 0xFFFF
        assert np.array_equal(counts.cpu().numpy(), np.bincount(want_all[:n], minlength=P))
    del hold


# Both sides of what the launch is cut by: a sweep of a block's threads (2048 rows of 512 threads up to 2048
# partitions, 4096 of 1024 above), and the blocks that are resident at once (three an SM, or one: 933,888 and
# 622,592 rows on 152 SMs), from which on a block takes several sweeps, the next one's first key on its way.
@pytest.mark.parametrize("P,sizes", [(200, (2047, 2048, 2049, 933_888, 933_889, 1_000_003, 1_900_001)),
                                     (2049, (4095, 4096, 4097, 622_592, 622_593, 700_001, 1_300_003)),
                                     (5000, (4097, 800_003))])
@pytest.mark.parametrize("keys", [[0], [1], [0, 1], [0, 2, 3]])
def test_static_ids_of_blocks_with_several_sweeps(P, sizes, keys):
    n = max(sizes)
    rng = np.random.default_rng(P)
    schema = [W.Field(f"k{i}", t) for i, t in enumerate(("int64", "int32", "int16", "bool"))]
    bufs = []
    for f in schema:
        bufs += W._column(rng, f, n, rng.integers(0, 2 if f.type == "bool" else 30_000, n), 0.2)
    want = _oracle_pids(schema, keys, P, W.Batch(n, bufs))
    for shift in (0, 1):  # columns on their boundaries, and one element off them
        cols, hold = (GzKeyColumn * len(keys))(), []
        for j, k in enumerate(keys):
            w = W.BYTE_WIDTH.get(schema[k].type, 1) * shift
            t = torch.from_numpy(np.concatenate([np.zeros(w, np.uint8), bufs[2 * k + 1].view(np.uint8)])).cuda()
            m = torch.from_numpy(bufs[2 * k].view(np.uint8).copy()).cuda()
            hold += [t, m]
            cols[j].type, cols[j].values, cols[j].validity = schema[k].code, t.data_ptr() + w, m.data_ptr()
        for rows in sizes:
            assert -(-rows // TILE_ROWS) * P <= MAX_COUNTERS
            out = torch.full((rows + 2,), -1, dtype=torch.int16, device="cuda")
            counts = torch.full((P,), -1, dtype=torch.int64, device="cuda")
            st = _entry()(0, P, cols, len(keys), rows, out.data_ptr(), counts.data_ptr(), torch.cuda.current_stream().cuda_stream)
            assert st == 0, _last_error()
            got = out.cpu().numpy().view(np.uint16)
            assert np.array_equal(got[:rows], want[:rows]), (rows, shift)
            assert (got[rows:] == 0xFFFF).all()
            assert np.array_equal(counts.cpu().numpy(), np.bincount(want[:rows], minlength=P)), (rows, shift)
        del hold
