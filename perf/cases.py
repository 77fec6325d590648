"""Performance cases of the shuffle: the calls an executor makes, through the public entry points.

Four kinds of pass (``op``):

* ``pids``      gz_hash_partition_static on a batch that is already in device memory: partition id
                of every row and the row count of every partition;
* ``map``       map tasks as an executor runs them (shuffle.run_map_tasks: make, one split per
                record batch on pageable host buffers, stop writing the data file, close);
* ``resident``  one map task of a GPU-resident plan: batches in HBM, make, splitBatches, stop
                writing the data file, close;
* ``read``      one reduce task: a partition's IPC streams of many map outputs (page-cache bytes
                of memory-mapped data files) read into one set of device columns.

Inputs are the seeded workloads of ``gazelle_plugin_gb300.workloads`` at other sizes, generated on
the device.  Buffers start on 64-byte boundaries, as Arrow allocates them.
"""
import ctypes
import math
import os
import shutil
import tempfile

import numpy as np
import torch

from gazelle_plugin_gb300 import shuffle as S
from gazelle_plugin_gb300 import workloads as W

DEV = "cuda"
F = W.Field
NESTED_SCHEMA = [F("k", "int64", False), F("v", "float64"),
                 F("tags", "list", True, None, (F("item", "utf8"),)),
                 F("m", "list", True, "int32"),
                 F("st", "struct", True, None, (F("a", "int32"), F("b", "utf8")))]
SCHEMAS = {"small": (W.C1_SCHEMA, W.C1_KEYS), "wide": (W.C2_SCHEMA, W.C2_KEYS),
           "skew": (W.C3_SCHEMA, W.C3_KEYS), "mixed": (W.C4_SCHEMA_3, W.C4_KEYS_3),
           "nested": (NESTED_SCHEMA, [0])}
# input bytes per row, about: what sizes are chosen by
ROW_BYTES = {"small": 33, "wide": 180, "skew": 69, "mixed": 65, "nested": 64}
WORDS = (b"the of special pending ideas accounts carefully furiously express regular final "
         b"deposits requests packages slyly quickly bold theodolites ironic blithely even "
         b"instructions foxes unusual platelets dependencies silent pinto beans across asymptotes ")


def listed():
    return [
        # one small batch's ids, as a caller with its own allocator asks for them: latency
        dict(name="pids_call", op="pids", keys="int32", rows=4096, parts=8, nulls=0.05),
        # the key columns of a fact table chunk
        dict(name="pids_fact", op="pids", keys="int64,int64", rows=16_000_003, parts=200, nulls=0.02),
        # wide fan-out of a skewed, nullable key, a float and a bool beside it
        dict(name="pids_fanout", op="pids", keys="zipf,float64,bool", rows=500_009, parts=8000, nulls=0.2),
        # a short map task: one record batch of a dimension table (latency of the whole task)
        dict(name="map_first", op="map", schema="small", parts=8, tasks=1, batches=1, batch_rows=4096,
             nulls=0.05, codec="none", partitioner="hash"),
        # one map task over a slice of the wide fact table, ragged last batch
        dict(name="map_wide", op="map", schema="wide", parts=200, tasks=1, batches=64, batch_rows=4096,
             nulls=0.02, codec="none", partitioner="hash"),
        # an executor: 16 map tasks at once
        dict(name="map_executor", op="map", schema="wide", parts=200, tasks=16, batches=384, batch_rows=4096,
             nulls=0.02, codec="none", partitioner="hash"),
        # nested columns: list<utf8>, list<int32>, struct<int32, utf8>
        dict(name="map_nested", op="map", schema="nested", parts=64, tasks=1, batches=48, batch_rows=4096,
             nulls=0.1, codec="none", partitioner="hash"),
        # Spark's default shuffle codec over a slice of the wide table with worded comments
        dict(name="map_lz4", op="map", schema="wide", parts=200, tasks=1, batches=128, batch_rows=4096,
             nulls=0.02, codec="lz4", partitioner="hash"),
        # a GPU-resident plan's shuffle write of the wide table
        dict(name="resident_wide", op="resident", schema="wide", parts=200, batches=977, batch_rows=4096,
             nulls=0.02, codec="none", partitioner="hash"),
        # skewed key and wide fan-out, a fifth of the cells null, large batches
        dict(name="resident_skew", op="resident", schema="skew", parts=2000, batches=48, batch_rows=32768,
             nulls=0.2, codec="lz4", partitioner="hash"),
        # a reduce task: one partition of the wide table from 32 map outputs
        dict(name="read_wide", op="read", schema="wide", maps=32, map_rows=24_000, batch_rows=4085, nulls=0.02, codec="none"),
        # the same under LZ4_FRAME
        dict(name="read_lz4", op="read", schema="wide", maps=16, map_rows=12_000, batch_rows=4085, nulls=0.02, codec="lz4"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["pids", "pids", "map", "map", "resident", "read", "read"])
    if op == "pids":
        parts = _log(rng, 1, 16000)
        most = min(16_000_000, 1024 * (4_194_304 // parts))
        return dict(op=op, rows=_log(rng, 1000, most), parts=parts, nulls=rng.choice([0.0, 0.02, 0.3]),
                    keys=rng.choice(["int32", "int64", "int64,int64", "zipf", "int16,int64", "bool,float32,date32"]))
    schema = rng.choice(["small", "wide", "wide", "skew", "mixed", "nested"])
    nulls = rng.choice([0.0, 0.02, 0.2])
    codec = rng.choice(["none", "none", "lz4"])
    if op == "read":
        schema = "wide" if schema == "nested" else schema
        maps = _log(rng, 2, 16 if codec == "lz4" else 64)
        total = _log(rng, 200_000, 20_000_000 if codec == "lz4" else 130_000_000)
        return dict(op=op, schema=schema, maps=maps, map_rows=max(50, total // ROW_BYTES[schema] // maps),
                    batch_rows=rng.randint(1500, 4096), nulls=nulls, codec=codec)
    batch_rows = _log(rng, 500, 33_000)
    tasks = rng.choice([1, 1, 4, 16]) if op == "map" else 1
    total = _log(rng, 200_000, 300_000_000 if tasks > 1 or op == "resident" else 80_000_000)
    total //= 4 if codec == "lz4" else 8 if schema == "nested" else 1
    batches = max(tasks, min(2000, total // ROW_BYTES[schema] // batch_rows))
    d = dict(op=op, schema=schema, parts=_log(rng, 4, 3000), batches=batches, batch_rows=batch_rows, nulls=nulls,
             codec=codec, partitioner=rng.choice(["hash", "hash", "hash", "rr"]))
    if op == "map":
        d["tasks"] = tasks
    return d


# ---------------------------------------------------------------------------------------
# inputs
def _bits(v):
    """LSB-first bitmap of a bool tensor [batches, slots] (slots a multiple of 8)."""
    w = 2 ** torch.arange(8, device=v.device, dtype=torch.int32)
    return (v.view(v.shape[0], -1, 8).to(torch.int32) * w).sum(2).to(torch.uint8)


def _zipf(g, shape, s=1.1, ranks=10_000_000):
    u = torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)
    hs = (ranks ** (1 - s) - 1) / (1 - s)
    r = torch.floor((u * hs * (1 - s) + 1) ** (1 / (1 - s))).to(torch.int64).clamp(1, ranks)
    return r * (0x1E3779B97F4A7C15 | 1) + 2


class _Columns:
    """A task's batches of one flat schema: buffer j of every batch lies in one device tensor."""

    def __init__(self, rows, batch_rows, seed, nulls, worded):
        self.nb = -(-rows // batch_rows)
        self.br, self.slots = batch_rows, -(-batch_rows // 64) * 64
        self.rows = np.full(self.nb, batch_rows, np.int32)
        self.rows[-1] = rows - (self.nb - 1) * batch_rows
        self.nulls, self.worded = nulls, worded
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(seed)
        self.g0 = torch.Generator(device=DEV)  # null and length counts: the same for every seed
        self.g0.manual_seed(rows)
        self.shape = (self.nb, self.slots)
        self.tensors, self.starts, self.sizes = [], [], []
        self.live = torch.arange(self.slots, device=DEV)[None, :] < torch.from_numpy(self.rows).to(DEV)[:, None]

    def add(self, t, starts, sizes):
        self.tensors.append(t)
        self.starts.append(np.asarray(starts, np.int64))
        self.sizes.append(np.asarray(sizes, np.int64))

    def validity(self, nullable, lens=None):
        """A validity buffer, its nulls (and `lens` with them) in an order of the seed; the slots
        past a batch's last row stay where they are.  Returns the lengths, 0 at nulls."""
        if lens is None and not (nullable and self.nulls):
            self.add(None, np.zeros(self.nb), np.zeros(self.nb))
            return None
        v = torch.rand(self.shape, generator=self.g0, device=DEV) >= self.nulls
        at = self.live.view(-1).nonzero().view(-1)
        to = at[torch.randperm(at.numel(), generator=self.g, device=DEV)]
        if lens is not None:
            lens = (lens * v * self.live).view(-1)
            lens[to] = lens[at]
            lens = lens.view(self.shape)
        if not self.nulls:
            self.add(None, np.zeros(self.nb), np.zeros(self.nb))
            return lens
        v = v.view(-1)
        v[to] = v[at]
        t = _bits(v.view(self.shape))
        t = torch.nn.functional.pad(t, (0, -t.shape[1] % 64))
        self.add(t, np.arange(self.nb, dtype=np.int64) * t.shape[1], (self.rows.astype(np.int64) + 7) // 8)
        return lens

    def fixed(self, nullable, values):
        self.validity(nullable)
        w = values.element_size()
        self.add(values, np.arange(self.nb, dtype=np.int64) * self.slots * w, self.rows.astype(np.int64) * w)

    def randint(self, lo, hi, dtype):
        return torch.randint(lo, hi, self.shape, generator=self.g, device=DEV, dtype=dtype)

    def strings(self, lo, hi, alphabet):
        lens = self.validity(True, torch.randint(lo, hi + 1, self.shape, generator=self.g0, device=DEV,
                                                 dtype=torch.int32))
        ow = -(-(self.br + 1) // 16) * 16
        off = torch.zeros((self.nb, ow), dtype=torch.int32, device=DEV)
        off[:, 1:self.br + 1] = torch.cumsum(lens[:, :self.br], 1)
        totals = off[:, self.br].to(torch.int64)
        starts = torch.cumsum(-(-totals // 64) * 64, 0) - -(-totals // 64) * 64
        n = int(starts[-1] + totals[-1]) + 64
        if self.worded and hi > 4:  # rows cut out of a text of common words
            words = WORDS.split()
            pick = torch.randint(0, len(words), (16384,), generator=self.g, device=DEV).cpu().tolist()
            page = torch.tensor(list(b" ".join(words[i] for i in pick)), dtype=torch.uint8, device=DEV)
            jump = torch.randint(0, page.numel(), (n // 32 + 1,), generator=self.g, device=DEV)
            at = torch.arange(n, device=DEV)
            chars = page[(jump[at // 32] + at % 32) % page.numel()]
        else:
            a = torch.tensor(list(alphabet), dtype=torch.uint8, device=DEV)
            chars = a[torch.randint(0, len(alphabet), (n,), generator=self.g, device=DEV)]
        self.add(off, np.arange(self.nb, dtype=np.int64) * ow * 4, (self.rows.astype(np.int64) + 1) * 4)
        self.add(chars, starts.cpu().numpy(), totals.cpu().numpy())

    def on_device(self):
        a = np.stack([(0 if t is None else t.data_ptr()) + s for t, s in zip(self.tensors, self.starts)], 1)
        z = np.stack(self.sizes, 1)
        a[z == 0] = 0
        return a, z, self.tensors

    def on_host(self):
        """Pageable host copies, 64-byte aligned like Arrow's off-heap buffers."""
        keep, base = [], []
        for t in self.tensors:
            if t is None:
                keep.append(None)
                base.append(0)
                continue
            h = t.view(-1).view(torch.uint8).cpu().numpy()
            keep.append(h)
            base.append(h.ctypes.data)
        a = np.stack([b + s for b, s in zip(base, self.starts)], 1)
        z = np.stack(self.sizes, 1)
        a[z == 0] = 0
        return a, z, keep


def _flat(schema, rows, batch_rows, seed, nulls, worded=False):
    c = _Columns(rows, batch_rows, seed, nulls, worded)
    if schema == "small":
        c.fixed(False, c.randint(0, 2**31 - 1, torch.int32))
        c.fixed(True, c.randint(-2**62, 2**62, torch.int64))
        c.fixed(True, torch.randn(c.shape, generator=c.g, device=DEV, dtype=torch.float64))
        c.strings(0, 16, W.AZ)
    elif schema == "wide":
        for _ in range(4):
            c.fixed(False, c.randint(0, 600_000_000, torch.int64))
        for _ in range(4):
            c.fixed(True, torch.floor(torch.rand(c.shape, generator=c.g, device=DEV, dtype=torch.float64) * 1e7) / 100)
        for _ in range(2):
            c.fixed(True, c.randint(8000, 10600, torch.int32))
        for a in W.C2_FLAG_ALPHABETS:
            c.strings(1, 1, a)
        for _ in range(3):
            c.strings(10, 44, W.AZ_SPACE)
    elif schema == "skew":
        c.fixed(False, _zipf(c.g, c.shape))
        c.fixed(True, c.randint(-2**62, 2**62, torch.int64))
        c.fixed(True, c.randint(-2**62, 2**62, torch.int64))
        c.fixed(True, torch.randn(c.shape, generator=c.g, device=DEV, dtype=torch.float64))
        c.strings(0, 64, W.AZ)
    else:
        c.fixed(False, c.randint(-2**31, 2**31 - 1, torch.int32))
        for _ in range(5):
            c.fixed(True, c.randint(-2**31, 2**31 - 1, torch.int32))
        for _ in range(2):
            c.strings(0, 32, W.AZ)
    return c


def _nested(rows, batch_rows, seed, nulls):
    """Host batches of the nested schema: (rows, addresses, sizes, what keeps them alive)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    out, left = [], rows
    while left > 0:
        n = min(left, batch_rows)
        left -= n
        bufs = W._column(rng, NESTED_SCHEMA[0], n, rng.integers(0, 1 << 40, size=n), 0.0)
        bufs += W._column(rng, NESTED_SCHEMA[1], n, rng.standard_normal(n), nulls)
        bufs += W.nested_column(rng, NESTED_SCHEMA[2], n, nulls, 4)
        bufs += W.list_column(rng, NESTED_SCHEMA[3], n, nulls, nulls, 4)
        bufs += W.nested_column(rng, NESTED_SCHEMA[4], n, nulls, 4)
        out.append(W.Batch(n, bufs))
    pairs = [b.addrs_sizes() for b in out]
    return (np.array([b.num_rows for b in out], np.int32), np.stack([a for a, _ in pairs]),
            np.stack([z for _, z in pairs]), out)


def _scratch():
    base = "/dev/shm" if os.path.isdir("/dev/shm") and os.access("/dev/shm", os.W_OK) else None
    return tempfile.mkdtemp(prefix="gz-cases-", dir=base)


class _State:
    dir = None
    readers = ()

    def __del__(self):
        for r in self.readers:
            r.close()
        if self.dir:
            shutil.rmtree(self.dir, ignore_errors=True)


def _rows(case):
    # a ragged end: the last batch is about two thirds full
    return case["batches"] * case["batch_rows"] - case["batch_rows"] // 3


def _host_input(schema, rows, batch_rows, seed, nulls, worded):
    if schema == "nested":
        return _nested(rows, batch_rows, seed, nulls)
    c = _flat(schema, rows, batch_rows, seed, nulls, worded)
    a, z, keep = c.on_host()
    return c.rows, a, z, keep


class GzKeyColumn(ctypes.Structure):
    _fields_ = [("type", ctypes.c_int32), ("reserved", ctypes.c_int32), ("validity", ctypes.c_void_p),
                ("values", ctypes.c_void_p)]


def _prepare_pids(case, seed):
    st = _State()
    n = case["rows"]
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    kinds = case["keys"].split(",")
    st.keys = (GzKeyColumn * len(kinds))()
    st.keep = []
    for i, k in enumerate(kinds):
        if k == "zipf":
            k, v = "int64", _zipf(g, (n,))
        elif k == "int64":
            v = torch.randint(0, 600_000_000, (n,), generator=g, device=DEV, dtype=torch.int64)
        elif k in ("int32", "date32"):
            v = torch.randint(-2**31, 2**31 - 1, (n,), generator=g, device=DEV, dtype=torch.int32)
        elif k == "int16":
            v = torch.randint(-2**15, 2**15 - 1, (n,), generator=g, device=DEV, dtype=torch.int16)
        elif k == "bool":
            v = torch.randint(0, 256, ((n + 7) // 8,), generator=g, device=DEV, dtype=torch.uint8)
        else:
            v = torch.randn((n,), generator=g, device=DEV,
                            dtype=torch.float64 if k == "float64" else torch.float32)
        st.keep.append(v)
        st.keys[i].type = W.TYPE_CODES[k]
        st.keys[i].values = v.data_ptr()
        if case["nulls"]:
            v = _bits((torch.rand((1, -(-n // 8) * 8), generator=g, device=DEV) >= case["nulls"])).view(-1)
            st.keep.append(v)
            st.keys[i].validity = v.data_ptr()
    st.pids = torch.empty(n, dtype=torch.int16, device=DEV)  # uint16 ids: the same bits
    st.counts = torch.empty(case["parts"], dtype=torch.int64, device=DEV)
    st.args = (torch.cuda.current_device(), case["parts"], ctypes.addressof(st.keys), len(kinds), n,
               st.pids.data_ptr(), st.counts.data_ptr(), torch.cuda.current_stream().cuda_stream)
    f = S.lib().gz_hash_partition_static
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int32, ctypes.c_int32, ctypes.c_void_p, ctypes.c_int32, ctypes.c_int32,
                  ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    st.call = f
    return st


def _prepare_map(case, seed):
    st = _State()
    st.dir = _scratch()
    schema, keys = SCHEMAS[case["schema"]]
    st.part = S.NativePartitioning(case["partitioner"], case["parts"], None,
                                   keys if case["partitioner"] == "hash" else [], list(schema))
    st.rows, st.addrs, st.sizes, st.keep = _host_input(case["schema"], _rows(case), case["batch_rows"], seed,
                                                       case["nulls"], case["codec"] == "lz4")
    return st


def _prepare_resident(case, seed):
    st = _State()
    st.dir = _scratch()
    schema, keys = SCHEMAS[case["schema"]]
    st.part = S.NativePartitioning(case["partitioner"], case["parts"], None,
                                   keys if case["partitioner"] == "hash" else [], list(schema))
    if case["schema"] == "nested":
        st.rows, a, st.sizes, host = _nested(_rows(case), case["batch_rows"], seed, case["nulls"])
        flat = [b for x in host for b in x.buffers]  # one device block, buffers 64-byte aligned
        at = np.concatenate([[0], np.cumsum([-(-b.nbytes // 64) * 64 for b in flat])]).astype(np.int64)
        img = np.zeros(int(at[-1]) + 64, np.uint8)
        for b, o in zip(flat, at):
            img[o:o + b.nbytes] = b.view(np.uint8)
        st.keep = torch.from_numpy(img).to(DEV)
        st.addrs = np.where(st.sizes > 0, (at[:-1] + st.keep.data_ptr()).reshape(st.sizes.shape), 0)
    else:
        c = _flat(case["schema"], _rows(case), case["batch_rows"], seed, case["nulls"], case["codec"] == "lz4")
        st.rows = c.rows
        st.addrs, st.sizes, st.keep = c.on_device()
    st.wrapper = S.ShuffleSplitterJniWrapper()
    return st


def _prepare_read(case, seed):
    """The data files of `maps` map tasks, one partition each (its record batches hold batch_rows
    rows, as a hash split cuts them a little below the writer's buffer size)."""
    st = _State()
    st.dir = _scratch()
    schema, _ = SCHEMAS[case["schema"]]
    st.schema = list(schema)
    maps = case["maps"]
    br = min(case["batch_rows"], case["map_rows"])
    nb = -(-case["map_rows"] // br)
    rows, a, z, keep = _host_input(case["schema"], maps * nb * br - br // 3, br, seed, case["nulls"],
                                   case["codec"] == "lz4")
    S.run_map_tasks(S.NativePartitioning("single", 1, None, [], st.schema), rows, a, z, maps, st.dir,
                    codec=_codec(case))
    st.streams = [np.memmap(os.path.join(st.dir, f"task-{t:04d}.data"), dtype=np.uint8, mode="r")
                  for t in range(maps)]
    return st


def prepare(case, seed):
    return {"pids": _prepare_pids, "map": _prepare_map, "resident": _prepare_resident,
            "read": _prepare_read}[case["op"]](case, seed), case


# ---------------------------------------------------------------------------------------
class _DeviceBytes:
    """`n` device bytes at `p` for torch.as_tensor; `owner` keeps them alive."""

    def __init__(self, p, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (p, False), "version": 3}


def _device_bytes(p, n, owner):
    if not p or not n:
        return torch.empty(0, dtype=torch.uint8, device=DEV)
    return torch.as_tensor(_DeviceBytes(p, n, owner), device=DEV)


def _codec(case):
    return None if case["codec"] == "none" else case["codec"]


def _most_bytes(case, rows):
    """More than a task's data file of `rows` rows takes: the record batches' bodies, and their
    headers and padding (a partition's batches hold more than half a 4096-row buffer but for two)."""
    return int(1.1 * rows * ROW_BYTES[case["schema"]]) + 2500 * (2 * min(case["parts"], rows) + rows // 2048) + (1 << 20)


def _data_file(path, most):
    """The data file's bytes as a mapping of `most` bytes (its length differs with the inputs:
    past its end the mapping is a hole, zeros that take no memory)."""
    if os.path.getsize(path) > most:
        raise RuntimeError(f"{path} holds more than {most} bytes")
    os.truncate(path, most)
    return np.memmap(path, dtype=np.uint8, mode="r", shape=(most,))


def run(state):
    st, case = state
    op = case["op"]
    if op == "pids":
        if st.call(*st.args) != S.GZ_OK:
            raise RuntimeError("gz_hash_partition_static failed")
        return st.pids, st.counts
    if op == "map":
        r = S.run_map_tasks(st.part, st.rows, st.addrs, st.sizes, case["tasks"], st.dir, codec=_codec(case))
        most = _most_bytes(case, -(-case["batches"] // case["tasks"]) * case["batch_rows"])
        return [_data_file(os.path.join(st.dir, f"task-{t:04d}.data"), most)
                for t in range(case["tasks"])], r["partition_lengths"]
    if op == "resident":
        path = os.path.join(st.dir, "shuffle.data")
        w = st.wrapper
        h = w.make(st.part, dataFile=path, codec=_codec(case), input_kind=S.GZ_INPUT_DEVICE_RETAINED)
        w.splitBatches(h, st.rows, st.addrs, st.sizes)
        r = w.stop(h)
        w.close(h)
        return _data_file(path, _most_bytes(case, _rows(case))), r.partitionLengths, r.rawPartitionLengths
    for r in st.readers:  # the columns of the state's last pass are done with
        r.close()
    rd = S.PartitionReader(st.schema)
    st.readers = [rd]
    for s in st.streams:
        rd.addStream(s)
    n, _ = rd.finish()
    out = [n]
    for f in range(len(st.schema)):
        c = rd.column(f)
        ow = 8 if c.type in (21, 22, 24) else 4
        out += [_device_bytes(c.validity, (c.length + 7) // 8, rd),
                _device_bytes(c.offsets, (c.length + 1) * ow if c.offsets else 0, rd),
                _device_bytes(c.values, c.values_bytes, rd)]
    return out


def work(case):
    """Bytes every input is read and every output is written once (inputs that the host owns
    cross the host link, so do data files); no floating-point work."""
    n = case.get("rows") or (case["maps"] * case["map_rows"] if case["op"] == "read" else _rows(case))
    if case["op"] == "pids":
        w = sum({"bool": 0.125, "int16": 2, "int64": 8, "zipf": 8, "float64": 8}.get(k, 4)
                for k in case["keys"].split(","))
        w += len(case["keys"].split(",")) / 8 if case["nulls"] else 0
        return {"bytes": n * (w + 2) + 8 * case["parts"], "flops": 0}
    return {"bytes": 2 * n * ROW_BYTES[case["schema"]], "flops": 0}
