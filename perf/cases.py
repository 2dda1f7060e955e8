"""The work whose time is measured: counting, merging and reading k-mer databases
through the C ABI (include/kite_gpu.h), over the range of sizes, key widths and
options that `kite count`, `merge`, `dump`, `histo` and `query` are run with.

A case's `op` names the call:

  rows    kite_gpu_count_rows_noalloc: a small batch of reads already on the device
  device  FASTQ chunks already on the device, payloads left there
          (kite_gpu_count_submit_device + kite_gpu_count_finish without a callback)
  host    FASTQ chunks in pinned host memory, payloads handed out partition by
          partition: what `kite count` does between its reader and its writer
  batch   several samples counted as one (kite_gpu_count_submit_device_sample)
  merge   databases in pinned host memory merged into one, payloads handed out
  dump    a database written as TSV lines, handed out partition by partition
  histo   the histogram of a database's counts
  query   the counts of a list of keys

Reads have the shapes of kite_gb300/synth.py's workloads (lengths, error and N
rates, repeats, AT-rich stretches), made on the device from the seed, at about 30-fold
coverage, with quality values between "&" and "I" (which hold "+" and "@").  Chunks have
the planner's default size, partitions are its default 256 unless a case says so.
All outputs are whole numbers and bytes.
"""
import ctypes as C
import math

import numpy as np
import torch

from kite_gb300 import gpu, host
from kite_gb300.kitefile import KiteImage

CHUNK = 51_130_563  # the planner's chunk size for plain input at its default memory
HEADER = 12         # "@r" + 9 digits + newline


def listed():
    return [
        # a few hundred reads between other GPU work, in a process that cannot allocate
        {"name": "rows_800", "op": "rows", "reads": 800, "length": 150, "k": 31, "canonical": True, "parts": 256},
        # one small amplicon-sized batch: latency and launches
        {"name": "device_2k_k31", "op": "device", "reads": 2_000, "length": 150, "k": 31, "canonical": True,
         "parts": 256},
        # a bacterial sample: the 200,000-read configuration, from host chunks to host payloads
        {"name": "host_200k_k21", "op": "host", "reads": 200_000, "length": 150, "k": 21, "canonical": False,
         "parts": 16},
        # an ordinary sequencing sample counted where its reads already are
        {"name": "device_1m_k31", "op": "device", "reads": 1_000_000, "length": 150, "k": 31, "canonical": True,
         "parts": 256},
        # the 10M-read configuration, the largest
        {"name": "device_10m_k31", "op": "device", "reads": 10_000_000, "length": 150, "k": 31, "canonical": True,
         "parts": 256},
        # an ordinary sample end to end: copy in, count, copy out
        {"name": "host_2m_k31", "op": "host", "reads": 2_000_000, "length": 150, "k": 31, "canonical": True,
         "parts": 256},
        # long k-mers (u128 keys) of an AT-rich genome: the skewed configuration
        {"name": "device_1m_k63_skewed", "op": "device", "reads": 1_000_000, "length": 250, "k": 63,
         "canonical": True, "parts": 256, "skewed": True},
        # a run of metagenome samples of uneven sizes and read lengths
        {"name": "batch_16x50k_k31", "op": "batch", "samples": 16, "reads": 50_000, "length": 250, "k": 31,
         "canonical": True, "parts": 256},
        # eight databases of one species merged into one
        {"name": "merge_8x200k_k31", "op": "merge", "inputs": 8, "reads": 200_000, "length": 150, "k": 31,
         "canonical": True, "parts": 256, "least": 0},
        # a database of one segment as text, counts of 2 and more
        {"name": "dump_2m_k31", "op": "dump", "reads": 2_000_000, "length": 150, "k": 31, "canonical": True,
         "parts": 256, "segments": 1, "least": 2},
        # the count histogram (genome size, error rate) of a database flushed in four segments
        {"name": "histo_2m_k31", "op": "histo", "reads": 2_000_000, "length": 150, "k": 31, "canonical": True,
         "parts": 256, "segments": 4, "least": 0},
        # a panel of marker k-mers looked up, half of them present
        {"name": "query_100k_of_1m_k31", "op": "query", "reads": 1_000_000, "length": 150, "k": 31,
         "canonical": True, "parts": 256, "segments": 1, "least": 0, "keys": 100_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["rows", "device", "device", "device", "host", "host", "batch", "merge", "dump", "histo", "query"])
    k = rng.choice([rng.randint(11, 31), 21, 31, 31, rng.randint(32, 64), 51])
    c = {"op": op, "k": k, "canonical": rng.random() < 0.7, "parts": 256, "length": rng.randint(75, 300)}
    if op == "rows":
        c["reads"] = max(1, _log(rng, 8_000, 500_000) // (2 * c["length"] + 16))
        c["parts"] = rng.choice([16, 64, 256, 1024])
    elif op == "device":
        c["reads"] = _log(rng, 500, 4_000_000 if k <= 31 else 1_500_000)
        c["parts"] = rng.choice([16, 64, 256, 256, 256, 512, 2048])
        if c["reads"] < 100_000 and rng.random() < 0.3:
            c["parts"] = 4
        c["skewed"] = rng.random() < 0.3
    elif op == "host":
        c["reads"] = _log(rng, 2_000, 2_000_000 if k <= 31 else 800_000)
        c["parts"] = rng.choice([16, 64, 256, 256])
    elif op == "batch":
        c["samples"] = rng.randint(2, 24)
        c["reads"] = _log(rng, 300, 100_000 if k <= 31 else 40_000)
        c["length"] = rng.randint(150, 300)
    else:
        c["reads"] = _log(rng, 3_000, 2_000_000 if k <= 31 else 600_000)
        c["least"] = rng.choice([0, 2])
        if op == "merge":
            c["inputs"] = rng.randint(2, 12)
            c["reads"] = max(1_000, c["reads"] // c["inputs"])
        else:
            c["segments"] = rng.choice([1, 1, 2, 5])
        if op == "query":
            c["keys"] = _log(rng, 1, 1_000_000)
    return c


# ---- reads ---------------------------------------------------------------------

def _ints(gen, hi, *shape):
    return torch.randint(0, hi, shape, generator=gen, device="cuda")


def _genome(gen, n, skewed):
    """Base codes of a genome: a fifth of it copies of 2 kbp repeats, or (skewed) its first
    30% an AT-rich chain that keeps the previous base half the time."""
    g = _ints(gen, 4, n).to(torch.uint8)
    if skewed:
        m = int(n * 0.3)
        u = torch.rand(m, generator=gen, device="cuda")
        d = (u >= 0.4).to(torch.uint8) + (u >= 0.5).to(torch.uint8) + (u >= 0.6).to(torch.uint8)
        at = torch.arange(m, device="cuda")
        at[torch.rand(m, generator=gen, device="cuda") < 0.5] = 0
        g[:m] = d[torch.cummax(at, 0).values]
    elif n >= 20_000:
        slots, copies = n // 2000, n // 10_000
        elems = _ints(gen, 4, max(1, copies // 40), 2000).to(torch.uint8)
        c = elems[_ints(gen, elems.shape[0], copies)]
        c = (c + (torch.rand(c.shape, generator=gen, device="cuda") < 0.01) * _ints(gen, 4, *c.shape)) & 3
        g[:slots * 2000].view(slots, 2000)[torch.randperm(slots, generator=gen, device="cuda")[:copies]] = \
            c.to(torch.uint8)
    return g


def _records(gen, genome, n, length, first, errors, n_rate, both):
    """n FASTQ records of one read length as a (n, record) byte matrix."""
    start = _ints(gen, max(1, genome.numel() - length), n)
    codes = genome[start[:, None] + torch.arange(length, device="cuda")]
    if both:
        flip = torch.rand(n, 1, generator=gen, device="cuda") < 0.5
        codes = torch.where(flip, 3 - codes.flip(1), codes)
    u = torch.rand(n, length, generator=gen, device="cuda")
    codes = torch.where(u < errors, (codes + 1 + (u * (3 / errors)).to(torch.uint8)) & 3, codes)
    seq = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")[codes.long()]
    seq = torch.where(u > 1 - n_rate, 78, seq)
    out = torch.empty(n, HEADER + 2 * length + 4, dtype=torch.uint8, device="cuda")
    out[:, 0], out[:, 1], out[:, HEADER - 1] = 64, 114, 10
    idx = torch.arange(first, first + n, device="cuda")
    for d in range(9):
        out[:, 2 + d] = 48 + (idx // 10 ** (8 - d)) % 10
    o = HEADER + length
    out[:, HEADER:o] = seq
    out[:, o], out[:, o + 1], out[:, o + 2], out[:, -1] = 10, 43, 10, 10
    out[:, o + 3:-1] = torch.randint(38, 74, (n, length), generator=gen, device="cuda", dtype=torch.uint8)
    return out


def _fastq(gen, genome, reads, length, skewed):
    """Whole FASTQ chunks of at most CHUNK bytes in one device buffer, each on a 16-byte
    boundary with 16 readable bytes after it, and their (offset, length)."""
    record = HEADER + 2 * length + 4
    per = CHUNK // record
    room = (per * record + 31) & ~15
    n = -(-reads // per)
    buf = torch.zeros((n - 1) * room + (reads - (n - 1) * per) * record + 64, dtype=torch.uint8, device="cuda")
    chunks = []
    for i in range(n):
        m = min(per, reads - i * per)
        buf[i * room:i * room + m * record] = _records(gen, genome, m, length, i * per, 0.01,
                                                       0.0 if skewed else 0.001, not skewed).view(-1)
        chunks.append((i * room, m * record))
    return buf, chunks


def _bases(c):
    return c["reads"] * c["length"]


def _genome_of(gen, c, bases):
    return _genome(gen, max(5_000, c["length"] + 1, bases // 30), c.get("skewed", False))


# ---- databases -----------------------------------------------------------------

def _address(data):
    return C.cast(data, C.c_void_p).value


class _Out:
    """A caller's buffer: the payloads handed out so far, and each one's record."""

    def __init__(self, room, partitions):
        self.buf = torch.from_numpy(np.zeros(room, dtype=np.uint8))
        self.rec = np.zeros((partitions, 7), dtype=np.uint64)
        self.at = 0
        self.callback = gpu.EMIT(self._emit)

    def _emit(self, user, meta, data, n):
        m = meta.contents
        src = torch.from_numpy(np.ctypeslib.as_array(data, (n,)))
        self.buf[self.at:self.at + n].copy_(src)
        self.rec[m.partition_id] = (m.codec, m.row_count, n, m.key_min_lo[0], m.key_min_lo[1], m.key_max_lo[0],
                                    m.key_max_lo[1])
        self.at += n
        return 0

    def outputs(self):
        return {"payload": self.buf, "records": self.rec.view(np.int64)}


class _Database:
    """A .kite image in pinned host memory, as a program that opened the file has it."""

    def __init__(self, c, buf, chunks):
        width = 8 if c["k"] <= 31 else 16
        w = host.Writer(None, c["k"], c["canonical"], c["parts"], width, 2, 16 << 20, 2, c["least"] or None, None)
        segments = min(c.get("segments", 1), len(chunks))
        torch.cuda.synchronize()  # the reads are complete before the counter's own stream takes them up
        with gpu.Counter(c["k"], c["canonical"], c["parts"], splitter_mode=gpu.SPLIT_SAMPLED) as counter:
            for s in range(segments):
                for o, n in chunks[len(chunks) * s // segments:len(chunks) * (s + 1) // segments]:
                    counter.submit_device(buf.data_ptr() + o, n)
                for meta, payload in counter.finish():
                    w.append(meta, payload)
        w.finalize()
        data = w.image()
        w.close()
        self.image = KiteImage.parse(data)
        self.bytes = len(data)
        self.rows = sum(ch.row_count for ch in self.image.chunks)
        self.pinned = torch.frombuffer(bytearray(data), dtype=torch.uint8).pin_memory()
        self.image.data = b""
        self.input, self.keep = self.image.merge_input(self.pinned.data_ptr())
        self.input.base_len = self.bytes


def _split_for_segments(buf, chunks, segments, record):
    """The chunks cut finer, so that a small input still has `segments` flushes."""
    if len(chunks) >= segments:
        return buf, chunks
    (_, n), = chunks[:1]
    per = -(-(n // record) // segments) * record
    room = (per + 31) & ~15
    out = torch.zeros(segments * room + 64, dtype=torch.uint8, device="cuda")
    cut = []
    for i in range(segments):
        m = min(per, n - i * per)
        if m > 0:
            out[i * room:i * room + m] = buf[i * per:i * per + m]
            cut.append((i * room, m))
    return out, cut


def _some_keys(gen, genome, c):
    """Keys of a panel: half taken from the genome, half random, encoded as (low, high) words."""
    n, k = c["keys"], c["k"]
    g = genome.cpu().numpy()
    rng = np.random.default_rng(int(_ints(gen, 1 << 40, 1).item()))
    codes = rng.integers(0, 4, (n, k), dtype=np.uint8)
    at = rng.integers(0, len(g) - k + 1, n // 2)
    codes[:n // 2] = g[at[:, None] + np.arange(k)]
    words = np.zeros((2, n, 2), dtype=np.uint64)
    for s, strand in enumerate((codes, 3 - codes[:, ::-1])):
        for j in range(k):
            p = 2 * (k - 1 - j)
            words[s, :, p // 64] |= strand[:, j].astype(np.uint64) << np.uint64(p % 64)
    if not c["canonical"]:
        return np.ascontiguousarray(words[0])
    less = (words[1, :, 1] < words[0, :, 1]) | ((words[1, :, 1] == words[0, :, 1]) & (words[1, :, 0] < words[0, :, 0]))
    return np.ascontiguousarray(np.where(less[:, None], words[1], words[0]))


def _check(rc):
    if rc < 0:
        raise gpu.KiteGpuError(rc, "call failed")


class _DeviceBytes:
    def __init__(self, address, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (address, False), "version": 3,
                                         "strides": None}


class _Results:
    """A count whose payloads stay on the device (one partition after another), and the
    buffer of its caller that they are copied to, on the stream that the count runs on."""

    def __init__(self, c, room, samples=1):
        self.stream = torch.cuda.Stream()
        self.counter = gpu.Counter(c["k"], c["canonical"], c["parts"], stream=self.stream.cuda_stream,
                                   samples=samples)
        n = c["parts"] * samples
        self.meta = [gpu.ChunkMeta() for _ in range(n)]
        self.address = [C.c_void_p() for _ in range(n)]
        self.length = [C.c_size_t() for _ in range(n)]
        self.args = [(p, C.byref(m), C.byref(a), C.byref(n))
                     for p, (m, a, n) in enumerate(zip(self.meta, self.address, self.length))]
        self.payload = torch.zeros(room, dtype=torch.uint8, device="cuda")

    def outputs(self):
        get, handle = gpu.lib().kite_gpu_result_partition, self.counter._h
        for a in self.args:
            _check(get(handle, *a))
        lengths = np.array([n.value for n in self.length], dtype=np.int64)
        rows = np.array([m.row_count for m in self.meta], dtype=np.int64)
        total = int(lengths.sum())
        if total:
            first = self.address[int(np.argmax(lengths > 0))].value
            with torch.cuda.stream(self.stream):
                self.payload[:total].copy_(torch.as_tensor(_DeviceBytes(first, total), device="cuda"))
        return {"rows": rows, "lengths": lengths, "payload": self.payload}


# ---- the cases -----------------------------------------------------------------

def prepare(case, seed):
    c = dict(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 7919 + 17)
    op, record = c["op"], HEADER + 2 * c["length"] + 4
    s = {"op": op}
    if op == "rows":
        genome = _genome_of(gen, c, _bases(c))
        s["fastq"], ((_, n),) = _fastq(gen, genome, c["reads"], c["length"], False)
        width = 8 if c["k"] <= 31 else 16
        s["keys"] = torch.zeros(n * width, dtype=torch.uint8, device="cuda")
        s["counts"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        s["part_rows"] = torch.zeros(c["parts"], dtype=torch.int32, device="cuda")
        s["totals"] = (C.c_uint64 * 4)()
        call = gpu.lib().kite_gpu_count_rows_noalloc
        call.argtypes = [C.c_int, C.c_int, C.c_int, C.c_uint32, C.c_void_p, C.c_size_t, C.c_void_p, C.c_void_p,
                         C.c_uint64, C.c_void_p, C.POINTER(C.c_uint64), C.c_void_p, C.c_uint32]
        s["call"] = call
        s["args"] = (0, c["k"], 1 if c["canonical"] else 0, c["parts"], s["fastq"].data_ptr(), n,
                     s["keys"].data_ptr(), s["counts"].data_ptr(), n, s["part_rows"].data_ptr(), s["totals"], None, 0)
    elif op in ("device", "host"):
        genome = _genome_of(gen, c, _bases(c))
        buf, s["chunks"] = _fastq(gen, genome, c["reads"], c["length"], c.get("skewed", False))
        if op == "device":
            s["fastq"] = buf
            s["results"] = _Results(c, _payload_room(c))
            s["counter"] = s["results"].counter
        else:
            s["fastq"] = torch.empty(buf.numel(), dtype=torch.uint8).pin_memory()
            s["fastq"].copy_(buf)
            s["counter"] = gpu.Counter(c["k"], c["canonical"], c["parts"], arena_bytes=buf.numel() + (64 << 20))
            s["out"] = _Out(_payload_room(c), c["parts"])
    elif op == "batch":
        species = [_genome(gen, 300_000, False) for _ in range(8)]
        parts, s["chunks"], at = [], [], 0
        for i in range(c["samples"]):
            # uneven samples: half to one and a half times the mean, each of a few read lengths
            reads = max(1, int(c["reads"] * (0.5 + float(torch.rand(1, generator=gen, device="cuda")))))
            for j, length in enumerate((c["length"], c["length"] * 3 // 4, c["length"] // 2)):
                m = reads // 3 + (1 if j < reads % 3 else 0)
                if not m:
                    continue
                b, ch = _fastq(gen, species[(i + j) % 8], m, length, False)
                parts.append(torch.nn.functional.pad(b, (0, -b.numel() % 16)))
                s["chunks"] += [(at + o, n, i) for o, n in ch]
                at += parts[-1].numel()
        s["fastq"] = torch.cat(parts)
        room = c["samples"] * _payload_room(dict(c, reads=c["reads"] * 3 // 2 + 3))
        s["results"] = _Results(c, room, c["samples"])
        s["counter"] = s["results"].counter
        s["samples"] = c["samples"]
    else:
        many = c.get("inputs", 1)
        genome = _genome_of(gen, c, _bases(c) * many)
        s["db"] = []
        for i in range(many):
            buf, chunks = _fastq(gen, genome, c["reads"], c["length"], False)
            buf, chunks = _split_for_segments(buf, chunks, c.get("segments", 1), record)
            s["db"].append(_Database(c, buf, chunks))
            del buf
        s["inputs"] = (gpu.MergeInput * many)(*[d.input for d in s["db"]])
        s["counter"] = gpu.Counter(c["k"], c["canonical"], c["parts"])
        if op == "merge":
            s["out"] = _Out(_payload_room(dict(c, reads=c["reads"] * many)), c["parts"])
        elif op == "dump":
            s["out"] = _Out(_payload_room(c, c["k"] + 6), c["parts"])
        elif op == "histo":
            s["bins"] = []
            s["callback"] = gpu.HISTO(lambda user, count, keys: s["bins"].append((count, keys)) and 0 or 0)
        else:
            s["words"] = _some_keys(gen, genome, c)
            s["found"] = np.zeros(c["keys"], dtype=np.uint64)
    torch.cuda.synchronize()
    return s


def run(s):
    lib, op = gpu.lib(), s["op"]
    if op == "rows":
        _check(s["call"](*s["args"]))
        t = list(s["totals"])
        return {"totals": np.array(t, dtype=np.int64), "keys": s["keys"].view(torch.int64), "counts": s["counts"],
                "part_rows": s["part_rows"]}
    h = s["counter"]._h
    if op == "device":
        base = s["fastq"].data_ptr()
        for o, n in s["chunks"]:
            _check(lib.kite_gpu_count_submit_device(h, base + o, n))
        _check(lib.kite_gpu_count_finish(h, C.cast(None, gpu.EMIT), None))
        return s["results"].outputs()
    if op == "batch":
        base = s["fastq"].data_ptr()
        for o, n, sample in s["chunks"]:
            _check(lib.kite_gpu_count_submit_device_sample(h, sample, base + o, n))
        _check(lib.kite_gpu_count_finish(h, C.cast(None, gpu.EMIT), None))
        out = s["results"].outputs()
        out["totals"] = np.array([s["counter"].sample_totals(i) for i in range(s["samples"])], dtype=np.int64)
        return out
    if op == "host":
        base = s["fastq"].data_ptr()
        s["out"].at = 0
        for o, n in s["chunks"]:
            _check(lib.kite_gpu_count_submit(h, base + o, n))
        _check(lib.kite_gpu_count_finish(h, s["out"].callback, None))
        return s["out"].outputs()
    if op == "merge":
        s["out"].at = 0
        _check(lib.kite_gpu_merge(h, s["inputs"], len(s["db"]), s["out"].callback, None))
        return s["out"].outputs()
    if op == "dump":
        s["out"].at = 0
        _check(lib.kite_gpu_dump(h, s["inputs"], s["out"].callback, None))
        return s["out"].outputs()
    if op == "histo":
        s["bins"].clear()
        _check(lib.kite_gpu_histo(h, s["inputs"], s["callback"], None))
        out = np.zeros((16384, 2), dtype=np.int64)  # (count, keys) of every count that there is, then zeros
        out[:len(s["bins"])] = s["bins"]
        return {"histogram": out}
    u64p = C.POINTER(C.c_uint64)
    _check(lib.kite_gpu_query(h, s["inputs"], s["words"].ctypes.data_as(u64p), len(s["found"]),
                              s["found"].ctypes.data_as(u64p)))
    return {"counts": s["found"].view(np.int64)}


# ---- what a pass cannot do without ---------------------------------------------

def _kmers(c):
    return c["reads"] * max(0, c["length"] - c["k"] + 1)


def _rows(c, genome):
    """Rows of a database: the genome's k-mers that the reads cover, and those with an error."""
    n, k = _kmers(c), c["k"]
    clean = 0.99 ** k
    cells = 4.0 ** k / (2 if c["canonical"] else 1)
    distinct = -genome * math.expm1(-n * clean / genome) * (1 if c["canonical"] or c.get("skewed") else 2)
    seen = distinct + n * (1 - clean)
    return min(float(n), -cells * math.expm1(-seen / cells))


def _row_bytes(c, rows):
    """A key's distance to the one before it in its partition, 7 bits to a byte, and a count."""
    bits = 2 * c["k"] - math.log2(max(2.0, rows / c["parts"])) - (1 if c["canonical"] else 0)
    return max(1, math.ceil(max(1.0, bits) / 7)) + 1


def _payload_room(c, row=0):
    """A caller's estimate of the bytes that a database's rows take, with a good margin."""
    rows = _rows(c, max(5_000.0, _bases(c) / 30))
    return int(min(_kmers(c), 1.25 * rows + 5_000) * (row or _row_bytes(c, rows) + 1) * 1.1 + 65_536) & ~7


def work(case):
    c = dict(case)
    op, many = c["op"], c.get("inputs", 1)
    genome = max(5_000.0, _bases(c) * many / 30)
    fastq = float(c["reads"] * (HEADER + 2 * c["length"] + 4))
    if op == "batch":
        c["length"] = c["length"] * 3 // 4
        rows = _rows(c, max(5_000.0, _bases(c) / 30))
        return {"bytes": c["samples"] * (c["reads"] * (HEADER + 2 * c["length"] + 4) + rows * _row_bytes(c, rows)),
                "flops": 0}
    rows = _rows(c, genome)
    image = rows * _row_bytes(c, rows)
    if op == "rows":
        return {"bytes": fastq + rows * ((8 if c["k"] <= 31 else 16) + 4), "flops": 0}
    if op in ("device", "host"):
        return {"bytes": fastq + image, "flops": 0}
    kept = min(rows, genome) if c["least"] else rows
    if op == "merge":
        out = min(genome, many * rows) if c["least"] else _rows(dict(c, reads=c["reads"] * many), genome)
        return {"bytes": many * image + out * _row_bytes(c, out), "flops": 0}
    if op == "dump":
        return {"bytes": image + kept * (c["k"] + 4), "flops": 0}
    if op == "histo":
        return {"bytes": image + 16 * 256, "flops": 0}
    return {"bytes": image + c["keys"] * 24, "flops": 0}


def exact(case, seed):
    """None: every output is a whole number or a byte, and stays as it is."""
    return None
