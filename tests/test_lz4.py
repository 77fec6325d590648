"""LZ4_FRAME shuffle compression: the framing on the host, the oracle decoder, and (GPU) the
CUDA compressor's output.

CPU: the oracle's LZ4 frame decoder (oracle/lz4_oracle.cc) against the LZ4 library pyarrow
ships; xxHash32 against its published empty-input value; the splitter's compressed record-batch
message (BodyCompression metadata, buffers as uncompressed length + LZ4 frame) read back by
pyarrow's IPC reader, with frames of stored blocks.
"""
import ctypes

import numpy as np
import pytest

from gazelle_plugin_gb300 import shuffle as S
from oracle import oracle as O


def test_xxh32_published_value():
    assert O.xxh32(b"") == 0x02CC5D05


@pytest.mark.parametrize("n", [1, 5, 100, 4096, 70000, 300000])
@pytest.mark.parametrize("kind", ["random", "repeat", "text"])
def test_oracle_lz4_decoder_matches_lz4_library(n, kind):
    pa = pytest.importorskip("pyarrow")
    rng = np.random.default_rng(n)
    if kind == "random":
        d = rng.integers(0, 256, n, dtype=np.uint8).tobytes()
    elif kind == "repeat":
        d = (b"abcabcabd" * (n // 9 + 1))[:n]
    else:
        d = rng.choice(np.frombuffer(b"abcdefghij  ", np.uint8), n).tobytes()
    frame = pa.compress(d, codec="lz4", asbytes=True)
    assert O.lz4f_decompress(frame, n) == d


def encode_lz4_stored(length, nodes, bufs):
    lib = S.lib()
    f = lib.gz_debug_encode_record_batch_lz4_stored
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int64, ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p,
                  ctypes.c_int32, ctypes.c_void_p, ctypes.c_int64, ctypes.POINTER(ctypes.c_int64)]
    n = np.array(nodes, np.int64).reshape(-1)
    ptrs = (ctypes.c_void_p * max(len(bufs), 1))(*[b.ctypes.data if b.nbytes else None for b in bufs])
    lens = np.array([b.nbytes for b in bufs], np.int64)
    out = np.zeros(4 << 20, np.uint8)
    olen = ctypes.c_int64(0)
    assert f(length, n.ctypes.data, len(nodes), ptrs, lens.ctypes.data, len(bufs), out.ctypes.data,
             out.nbytes, ctypes.byref(olen)) == 0
    return out[:olen.value].tobytes()


def test_compressed_record_batch_message_read_by_arrow():
    pa = pytest.importorskip("pyarrow")
    rng = np.random.default_rng(5)
    for trial in range(20):
        n = int(rng.integers(1, 100000 if trial % 5 == 0 else 500))
        mask = rng.random(n) < 0.1
        cols = [pa.array(rng.integers(-100, 100, n), pa.int64(), mask=mask),
                pa.array(["y" * int(k) for k in rng.integers(0, 12, n)], pa.string(),
                         mask=rng.random(n) < 0.05),
                pa.array(rng.integers(0, 2, n).astype(bool), pa.bool_()),
                pa.array(rng.integers(0, 9, n), pa.int32())]
        rb = pa.record_batch(cols, names=["a", "s", "b", "c"])
        nodes, bufs = [], []
        for col in rb.columns:
            nodes.append((len(col), col.null_count))
            bs = col.buffers()
            bufs.append(np.frombuffer(bs[0], np.uint8)[: (n + 7) // 8].copy() if (bs[0] is not None and col.null_count)
                        else np.zeros(0, np.uint8))
            if pa.types.is_string(col.type):
                off = np.frombuffer(bs[1], np.int32)[: n + 1]
                bufs.append(off.view(np.uint8).copy())
                bufs.append(np.frombuffer(bs[2], np.uint8)[: off[-1]].copy())
            elif pa.types.is_boolean(col.type):
                bufs.append(np.frombuffer(bs[1], np.uint8)[: (n + 7) // 8].copy())
            else:
                bufs.append(np.frombuffer(bs[1], np.uint8)[: n * (col.type.bit_width // 8)].copy())
        msg = pa.ipc.read_message(pa.py_buffer(encode_lz4_stored(n, nodes, bufs)))
        got = pa.ipc.read_record_batch(msg, rb.schema)
        assert got.equals(rb), trial


# ---------------------------------------------------------------------------------------- GPU
def _split(schema, batches, P, keys, **kw):
    return S.split_batches(schema, batches, P, keys, writeSchema=False, **kw)


def _partition_streams(res, data):
    starts = np.concatenate([[0], np.cumsum(np.asarray(res.partitionLengths))])
    return [data[starts[p]:starts[p + 1]] for p in range(len(starts) - 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["c1", "c2", "c3"])
def test_gpu_lz4_split_decodes_to_the_uncompressed_batches(which):
    """LZ4_FRAME output of the CUDA splitter: every record batch above batch_compress_threshold
    rows carries body compression, the others do not; decoded by the oracle's LZ4 frame decoder,
    every batch's buffers equal the uncompressed split's, which equal the oracle's."""
    from gazelle_plugin_gb300 import workloads as W
    from oracle import ipc_read as R
    if which == "c1":
        schema, keys, P, batches, kw = W.C1_SCHEMA, W.C1_KEYS, 8, W.c1_batches(21, 6, 4096), dict(bufferSize=1500)
    elif which == "c2":
        schema, keys, P, batches, kw = W.C2_SCHEMA, W.C2_KEYS, 200, W.c2_batches(22, 40, 4096), {}
    else:
        schema, keys, P, batches, kw = W.C3_SCHEMA, W.C3_KEYS, 16, W.c3_batches(23, 2, 32768, 0.2, 0.0), {}
    res_u, data_u = _split(schema, batches, P, keys, **kw)
    ref = O.run_oracle(schema, batches, P, keys, buffer_size=kw.get("bufferSize", 4096))
    assert data_u == ref.data
    res_z, data_z = _split(schema, batches, P, keys, codec="lz4", **kw)
    assert np.array_equal(res_z.rawPartitionLengths, res_u.rawPartitionLengths)
    # (random test data barely compresses: the frames may even add a few bytes)
    assert sum(res_z.partitionLengths) < 1.05 * sum(res_u.partitionLengths) + 4096
    for su, sz in zip(_partition_streams(res_u, data_u), _partition_streams(res_z, data_z)):
        bu, bz = R.parse_stream(su, schema), R.parse_stream(sz, schema)
        assert [r for r, _ in bu] == [r for r, _ in bz]
        assert R.batches_compressed(sz) == [r > 256 for r, _ in bz]
        for (_, cu), (_, cz) in zip(bu, bz):
            for fu, fz in zip(cu, cz):
                assert fu[0] == fz[0]  # null counts
                assert [bytes(b) for b in fu[1]] == [bytes(b) for b in fz[1]]


@pytest.mark.gpu
def test_gpu_reader_reads_lz4_streams():
    from gazelle_plugin_gb300 import workloads as W
    from oracle import ipc_read as R
    P = 200
    outs_u, outs_z = [], []
    for seed in (31, 32, 33):
        batches = W.c2_batches(seed, 6, 4096)
        outs_u.append(_partition_streams(*_split(W.C2_SCHEMA, batches, P, W.C2_KEYS)))
        outs_z.append(_partition_streams(*_split(W.C2_SCHEMA, batches, P, W.C2_KEYS, codec="lz4")))
    for p in range(0, P, 9):
        rows, cols = R.read_partition(W.C2_SCHEMA, [o[p] for o in outs_u])
        r = S.PartitionReader(list(W.C2_SCHEMA))
        for o in outs_z:
            r.addStream(o[p])
        assert r.finish()[0] == rows
        for fi, f in enumerate(W.C2_SCHEMA):
            valid, offs, vals = cols[fi]
            gv, go, gvals = r.column_to_host(fi)
            assert (gv is None) == (valid is None)
            if valid is not None:
                assert gv.tobytes() == R.pack_bits(valid)
            if f.is_binary:
                assert np.array_equal(go, offs)
            assert gvals.tobytes() == vals
        r.close()


@pytest.mark.gpu
def test_gpu_compressed_size_of_first_batch():
    """split(firstRecordBatch=True) with LZ4_FRAME: the batch's compressed IPC body length (the
    writer compares it between codecs, ColumnarShuffleWriter.scala:147-175), close to the body
    of the same batch split into one partition and compressed at Stop."""
    from gazelle_plugin_gb300 import workloads as W
    from oracle import ipc_read as R
    b = W.c2_batches(41, 1, 4096)[0]
    a, z = b.addrs_sizes()
    w = S.ShuffleSplitterJniWrapper()
    h = w.make(S.NativePartitioning("single", 1, None, [], list(W.C2_SCHEMA)), codec="lz4", writeSchema=False)
    plain = S.ShuffleSplitterJniWrapper()
    hp = plain.make(S.NativePartitioning("single", 1, None, [], list(W.C2_SCHEMA)), writeSchema=False)
    cs_lz4 = w.split(h, b.num_rows, a, z, True)
    cs_raw = plain.split(hp, b.num_rows, a, z, True)
    w.split(h, b.num_rows, a, z)
    w.stop(h)
    data = w.data(h)
    w.close(h)
    plain.close(hp)
    assert 0 < cs_lz4 < cs_raw
    # the body of the one record batch written: its message minus the metadata
    meta_len = int.from_bytes(data[4:8], "little")
    body = len(data) - 8 - 8 - meta_len  # continuation + length prefix, EOS at the end
    assert R.batches_compressed(data) == [True]
    assert abs(cs_lz4 - body) <= 0.01 * body + 64


def _lz4_block(rng, n, lits, mls, offs, history=b""):
    """A random LZ4 block of `n` decoded bytes and those bytes: sequences of literal lengths drawn from
    `lits`, match lengths from `mls` and offsets from `offs` (clipped to what precedes, `history`
    included), a literal tail."""
    out, blk = bytearray(history), bytearray()
    base = len(history)

    def ext(x):
        return b"" if x < 15 else b"\xff" * ((x - 15) // 255) + bytes([(x - 15) % 255])

    while True:
        lit, ml = int(rng.choice(lits)), int(rng.choice(mls))
        if len(out) == 0:
            lit = max(lit, 1)
        if len(out) - base + lit + ml + 5 > n:
            break
        data = rng.integers(0, 256, lit, dtype=np.uint8).tobytes()
        off = min(int(rng.choice(offs)), len(out) + lit)
        blk += bytes([(min(lit, 15) << 4) | min(ml - 4, 15)]) + ext(lit) + data + off.to_bytes(2, "little") + ext(ml - 4)
        out += data
        for _ in range(ml):
            out.append(out[-off])
    lit = n - (len(out) - base)
    data = rng.integers(0, 256, lit, dtype=np.uint8).tobytes()
    blk += bytes([min(lit, 15) << 4]) + ext(lit) + data
    return bytes(blk), bytes(out[base:]) + data


def _lz4_frame(blocks):
    """Frame of (payload, stored) blocks, as the splitter's frames are: independent blocks, no checksums."""
    f = b"\x04\x22\x4d\x18\x60\x40" + bytes([(O.xxh32(b"\x60\x40") >> 8) & 255])
    for b, stored in blocks:
        f += (len(b) | (0x80000000 if stored else 0)).to_bytes(4, "little") + b
    return f + bytes(4)


def _read_values_frame(frame, n):
    """The reader's value bytes of an int64 column of n bytes whose values buffer is `frame` (put over
    a longer frame of stored blocks; what follows a frame's end mark is not read)."""
    from gazelle_plugin_gb300 import workloads as W
    # the values' own bytes do not matter: they mark where the frame has to go
    plain = np.frombuffer(b"\xa5" * n, np.uint8)
    msg = bytearray(encode_lz4_stored(n // 8, [(n // 8, 0)], [np.zeros(0, np.uint8), plain]))
    at = msg.index(b"\x04\x22\x4d\x18")
    assert at + len(frame) <= len(msg)
    msg[at:at + len(frame)] = frame
    r = S.PartitionReader([W.Field("v", "int64", False)])
    try:
        r.addStream(bytes(msg))
        r.finish()
        return r.column_to_host(0)[2].tobytes()
    finally:
        r.close()


FRAME_SHAPES = {
    # sizes of the blocks, whether each is stored, and what their sequences look like
    "short sequences": ([8192, 8192, 3000], "ccc", range(0, 6), range(4, 12), range(1, 4000)),
    "overlapping matches": ([8192, 104], "cc", range(0, 3), range(4, 70), range(1, 40)),
    "long lengths": ([8192, 8184], "cc", [0, 14, 15, 16, 269, 270, 271, 600], [4, 18, 19, 20, 273, 274, 900], range(1, 9000)),
    "window edges": ([8192], "c", range(10, 18), range(14, 22), range(1, 300)),
    "pieces of a spanning batch": ([4, 8192, 1001, 8192, 3], "scscs", range(0, 9), range(4, 30), range(1, 2000)),
    "one short block": ([40], "c", range(0, 3), range(4, 6), range(1, 9)),
    "more blocks than slots": ([96] * 40, "c" * 40, range(0, 3), range(4, 9), range(1, 90)),
    "blocks over 8 KiB": ([20000, 65536], "cc", range(0, 9), range(4, 60), range(1, 65000)),
    "blocks that reach back": ([8192, 8192, 800], "lll", range(0, 6), range(4, 30), range(1, 20000)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("shape", list(FRAME_SHAPES))
def test_gpu_decoder_frame_shapes(shape):
    sizes, kinds, lits, mls, offs = FRAME_SHAPES[shape]
    for seed in range(4):
        rng = np.random.default_rng(seed)
        want, blocks = b"", []
        for n, kind in zip(sizes, kinds):
            if kind == "s":
                b = d = rng.integers(0, 256, n, dtype=np.uint8).tobytes()
            else:
                b, d = _lz4_block(rng, n, list(lits), list(mls), list(offs), want if kind == "l" else b"")
            blocks.append((b, kind == "s"))
            want += d
        pad = -len(want) % 8
        if pad:
            want += bytes(pad)
            blocks.append((bytes(pad), True))
        frame = _lz4_frame(blocks)
        assert O.lz4f_decompress(frame, len(want)) == want
        assert _read_values_frame(frame, len(want)) == want


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["offset 0", "offset before the frame", "cut block", "short", "long", "no end mark", "header"])
def test_gpu_decoder_malformed_frames(how):
    n = 8192 + 800
    rng = np.random.default_rng(3)
    b1, d1 = _lz4_block(rng, 8192, [3], [6], [100])
    b2, d2 = _lz4_block(rng, 800, [3], [6], [100])
    if how == "offset 0":
        b2 = b2[:4] + b"\x00\x00" + b2[6:]  # token, 3 literals, offset
    elif how == "offset before the frame":
        b1 = b1[:4] + b"\xff\xff" + b1[6:]
    elif how == "cut block":
        b2 = b2[:5]
    elif how == "short":
        b2 = _lz4_block(rng, 792, [3], [6], [100])[0]
    elif how == "long":
        b2 = _lz4_block(rng, 808, [3], [6], [100])[0]
    frame = _lz4_frame([(b1, False), (b2, False)])
    if how == "no end mark":
        frame = frame[:-4] + (0x7fffffff).to_bytes(4, "little")
    elif how == "header":
        frame = frame[:6] + bytes([frame[6] ^ 1]) + frame[7:]
    with pytest.raises(S.SplitterError) as e:
        _read_values_frame(frame, n)
    assert e.value.status == S.GZ_INVALID


DENSE_SHAPES = {
    # blocks, their size, FLG byte, and what their sequences look like
    "as many sequences as fit": (3, 8192, 0x60, [0], [4], range(1, 9)),
    "three-byte tokens, far sources": (2, 8192, 0x60, [0, 1], [4], range(1, 8190)),
    "one run": (2, 8192, 0x60, [1], [8180], [1]),
    "hardly a match": (2, 8192, 0x60, [3900], [80], [9]),
    "block checksums": (3, 4096, 0x70, range(0, 6), range(4, 12), range(1, 4000)),
    "content checksum": (3, 4096, 0x64, range(0, 6), range(4, 12), range(1, 4000)),
    "more blocks than run at once": (500, 8192, 0x60, range(0, 40), range(4, 30), range(1, 8000)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("shape", list(DENSE_SHAPES))
def test_gpu_decoder_blocks_at_their_limits(shape):
    """The most sequences a block can hold, one sequence over all segments, long chains of matches, frames
    with checksums, and more blocks than the device runs at once."""
    count, size, flg, lits, mls, offs = DENSE_SHAPES[shape]
    rng = np.random.default_rng(1)
    some = [_lz4_block(rng, size, list(lits), list(mls), list(offs)) for _ in range(min(count, 5))]
    desc = bytes([flg, 0x40])
    frame, want = b"\x04\x22\x4d\x18" + desc + bytes([(O.xxh32(desc) >> 8) & 255]), b""
    for i in range(count):
        b, d = some[i % len(some)]
        frame += len(b).to_bytes(4, "little") + b + (b"sums" if flg & 0x10 else b"")
        want += d
    frame += bytes(4) + (b"sum." if flg & 0x04 else b"")
    assert _read_values_frame(frame, len(want)) == want
