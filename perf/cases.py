"""What the read-mapping library is timed on: the calls its users make, over the sizes they make them with.

A case is one call of a public entry point (hpgbwt.lib, the binding of the C ABI) on seeded synthetic
reads from one of three seeded synthetic genomes:

    iid       4 Mbp of uniform bases: an index that fits the L2 many times
    repeats   100 Mbp, GC 41 %, 5 % repeat copies: an index of about the L2's size
    large     600 Mbp, human-like repeats (45 %): an index several times the L2

`prepare` draws the reads on the GPU and keeps them where the call takes them from (device memory or
page-locked host memory).  The index of a genome is built once per process tree by the library's own
builder, kept in the temporary directory and opened once per process: an index is what a program opens
when it starts and searches for as long as it runs.  A server is started once, too.
"""
from __future__ import annotations

import ctypes
import hashlib
import os
import platform
import shutil
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT / "hpg-libs_gb300"))

from hpgbwt import lib, synth  # noqa: E402

GENOMES = {"iid": 4_000_000, "repeats": 100_000_000, "large": 600_000_000}
LOCATE_LIMIT = {"iid": 0, "repeats": 0, "large": 10_000}  # rows located per list, as a program sets it on a repeat-rich genome
SERVER_READS = 1 << 20  # reads per served batch at most
EDITS = ("none", "capped", "mix", "subst05", "subst1")


# ------------------------------------------------------------------ the cases --

def listed() -> list[dict]:
    return [
        # exact search of error-free reads on a small genome: the first pass of a mapper on a bacterial reference
        dict(name="exact_200k_iid", api="device", genome="iid", mode="exact", form="batched", reads=200_000, lo=100,
             hi=100, edits="none", max_results=1024),
        # the smallest served request size, as one call on host arrays: latency, launches
        dict(name="host_1k_repeats", api="host", genome="repeats", mode="search1", form="batched", reads=1000, lo=50,
             hi=300, edits="subst05", max_results=1024),
        # a pipeline stage's block of reads, host arrays in, host arrays out
        dict(name="host_64k_repeats", api="host", genome="repeats", mode="search1", form="batched", reads=65_536,
             lo=100, hi=100, edits="capped", max_results=1024),
        # the headline batch: 2M x 100 bp at most one edit, reads and results in device memory
        dict(name="device_2m_repeats", api="device", genome="repeats", mode="search1", form="batched",
             reads=2_000_000, lo=100, hi=100, edits="capped", max_results=1024),
        # reads of uneven length and error depth (trimmed reads): ragged work
        dict(name="device_4m_ragged", api="device", genome="repeats", mode="search1", form="batched",
             reads=4_000_000, lo=36, hi=250, edits="mix", max_results=1024),
        # a repeat-rich genome whose index is far larger than the caches, reads with more errors than are searched
        dict(name="device_2m_large", api="device", genome="large", mode="search1", form="batched", reads=2_000_000,
             lo=150, hi=150, edits="subst1", max_results=1024),
        # the same genome from host arrays, an odd count of reads of uneven length, the full result capacity
        dict(name="host_300k_large", api="host", genome="large", mode="search1", form="batched", reads=299_993, lo=50,
             hi=300, edits="subst05", max_results=65_536),
        # the plain form (one thread per read and strand)
        dict(name="plain_256k_repeats", api="device", genome="repeats", mode="search1", form="plain", reads=262_144,
             lo=100, hi=100, edits="capped", max_results=1024),
        # k-error block search with anchors, host arrays in and out
        dict(name="block_1m_repeats", api="block", genome="repeats", reads=1_000_000, lo=36, hi=150, edits="capped",
             max_results=1024),
        # requests of mixed sizes arriving together at a running server
        dict(name="serve_24_requests", api="serve", genome="repeats", requests=24, req_lo=1000, req_hi=131_072, lo=50,
             hi=300, edits="subst05"),
        # the reference's alignment-list call on a fastq batch
        dict(name="lists_64k_repeats", api="lists", genome="repeats", reads=65_536, lo=100, hi=100, edits="capped",
             max_results=200),
        # seeds and candidate alignment locations of the reads that did not map
        dict(name="cals_8k_repeats", api="cals", genome="repeats", reads=8192, lo=100, hi=100, edits="mix",
             max_results=300),
    ]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng) -> dict:
    """A case of the listed ones' ranges: call, genome, count of reads, lengths, error model and capacity."""
    api = rng.choice(["device", "device", "device", "host", "host", "block", "serve", "lists", "cals", "plain", "exact"])
    genome = rng.choice(["iid", "repeats", "repeats", "large"])
    lo = rng.randint(36, 150)
    hi = rng.choice([lo, rng.randint(lo, 250)])
    edits = rng.choice(EDITS)
    cap = rng.choice([64, 1024, 4096, 65_536])
    if api in ("device", "host"):
        n = _log_uniform(rng, 700, 1_100_000 if genome == "large" else 2_400_000 if api == "device" else 1_500_000)
        return dict(api=api, genome=genome, mode="search1", form="batched", reads=n, lo=lo, hi=hi, edits=edits,
                    max_results=cap)
    if api == "plain":
        return dict(api="device", genome=genome, mode="search1", form="plain", reads=_log_uniform(rng, 1000, 400_000),
                    lo=lo, hi=hi, edits=edits, max_results=cap)
    if api == "exact":
        return dict(api=rng.choice(["device", "host"]), genome=genome, mode="exact", form="batched",
                    reads=_log_uniform(rng, 1000, 2_000_000), lo=lo, hi=hi, edits=edits, max_results=cap)
    if api == "block":
        return dict(api="block", genome=genome, reads=_log_uniform(rng, 1000, 1_000_000), lo=lo, hi=hi, edits=edits,
                    max_results=cap)
    if api == "serve":
        return dict(api="serve", genome="repeats", requests=rng.randint(1, 24), req_lo=1000,
                    req_hi=rng.choice([4096, 32_768, 131_072]), lo=max(lo, 50), hi=max(hi, 50), edits=edits)
    if api == "lists":
        return dict(api="lists", genome=genome, reads=_log_uniform(rng, 500, 65_536), lo=lo, hi=hi, edits=edits,
                    max_results=200)
    return dict(api="cals", genome=genome, reads=_log_uniform(rng, 300, 8192), lo=lo, hi=hi, edits=edits,
                max_results=300)


# ------------------------------------------------------------------ genome, index, reads --

_held: dict = {}  # what this process keeps open: genomes on the GPU, indexes, the server


def _place(genome: str) -> Path:
    built = os.stat(lib.LIB_PATH).st_mtime_ns
    key = hashlib.sha1(f"{ROOT}|{built}".encode()).hexdigest()[:12]
    return Path(tempfile.gettempdir()) / f"hpgbwt_perf_{key}" / f"{genome}_{GENOMES[genome]}"


def _genome_and_index(genome: str):
    """The genome's codes on the GPU and the directory of its index."""
    if genome not in _held:
        at = _place(genome)
        if not (at / "genome.npy").exists():
            part = Path(f"{at}.{os.getpid()}")
            part.mkdir(parents=True)
            bp = GENOMES[genome]
            codes = synth.genome_large(bp, 1) if genome == "large" else synth.genome(genome, bp, 1)
            synth.write_fasta(str(part / "genome.fa"), codes)
            lib.build_index(str(part / "genome.fa"), str(part / "index"), 16, device=0)
            os.remove(part / "genome.fa")
            np.save(part / "genome.npy", codes)
            try:
                os.rename(part, at)
            except OSError:  # another process was first
                shutil.rmtree(part)
        _held[genome] = torch.from_numpy(np.load(at / "genome.npy")).cuda(), str(at / "index")
    return _held[genome]


def _index(genome: str, use: str = "calls") -> lib.GpuIndex:
    if (genome, use) not in _held:
        gi = lib.GpuIndex(_genome_and_index(genome)[1], device=0)
        gi.set_locate_limit(LOCATE_LIMIT[genome])
        _held[genome, use] = gi
    return _held[genome, use]


def _server(genome: str) -> lib.Server:
    if (genome, "server") not in _held:
        _held[genome, "server"] = lib.Server(_index(genome, "serving"), SERVER_READS, max_results=1024)
    return _held[genome, "server"]


def _reads(genome: str, n: int, lo: int, hi: int, edits: str, seed: int):
    """n reads of lo..hi bases (uniform) from uniform positions of either strand: ASCII bases and n+1 offsets on the GPU.
    capped: per base 0.5 % substitutions, 0.02 % insertions, 0.02 % deletions, at most one edit a read; mix: 30 % exact,
    50 % one substitution, 20 % one 1-bp indel; subst05 / subst1: 0.5 % / 1 % substitutions, as many as fall."""
    g = _genome_and_index(genome)[0]
    gen = torch.Generator(device="cuda").manual_seed(seed * 1_000_003 + n)
    ascii_of = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")

    def rand(*shape):
        return torch.rand(*shape, generator=gen, device="cuda")

    lens = torch.full((n,), lo, dtype=torch.int64, device="cuda") if lo == hi else \
        torch.randint(lo, hi + 1, (n,), generator=gen, device="cuda")
    offs = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=offs[1:])
    out = torch.empty(int(offs[-1]), dtype=torch.uint8, device="cuda")
    step = max(1, (1 << 25) // (hi + 1))
    for a in range(0, n, step):
        L = lens[a:a + step, None]
        m = L.shape[0]
        u, kind = rand(m), torch.zeros(m, dtype=torch.int64, device="cuda")  # 0 none, 1 substitution, 2 insertion, 3 deletion
        if edits == "mix":
            kind = (u >= 0.3).long() + (u >= 0.8).long() + (u >= 0.9).long()
        elif edits == "capped":
            some = u < 1 - (1 - 0.0054) ** L[:, 0].double()
            v = rand(m)
            kind = some.long() * (1 + (v >= 50 / 54).long() + (v >= 52 / 54).long())
        kind = kind[:, None]
        at = (rand(m, 1).double() * (L - 2)).long() + 1
        col = torch.arange(hi, device="cuda")[None, :]
        src = col + ((kind == 3) & (col >= at)).long() - ((kind == 2) & (col > at)).long()
        pos = (torch.rand(m, 1, generator=gen, device="cuda", dtype=torch.float64) * (g.numel() - L - 1)).long()
        base = g[(pos + src).clamp_(max=g.numel() - 1)]
        other = torch.randint(1, 4, (m, 1), generator=gen, device="cuda", dtype=torch.uint8)
        hit = (col == at) & ((kind == 1) | (kind == 2))
        base = torch.where(hit, (base + other) & 3, base)
        if edits.startswith("subst"):
            rate = 0.005 if edits == "subst05" else 0.01
            wrong = rand(m, hi) < rate
            base = torch.where(wrong, (base + torch.randint(1, 4, (m, hi), generator=gen, device="cuda",
                                                            dtype=torch.uint8)) & 3, base)
        rc = rand(m, 1) < 0.5
        base = torch.where(rc, 3 - base.gather(1, torch.where(rc, (L - 1 - col).clamp_(min=0), col)), base)
        out[int(offs[a]):int(offs[a + m])] = ascii_of[base[col < L].long()]
    return out, offs


def _host(t: torch.Tensor) -> torch.Tensor:
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


class _Kept:
    """Where a program keeps a call's records: arrays of a whole multiple of the batch's size, zero past the records."""

    def __init__(self, n: int, device: str):
        self.n, self.device, self.of = n, device, {}
        for key in ("hits", "locs"):
            self._grow(key, 4, n, torch.int64)

    def _grow(self, key: str, words: int, m: int, dtype) -> list:
        rows = self.n + (self.n >> 1)  # half as many again as reads, or eight times that, and so on
        while rows < m:
            rows *= 8
        buf = torch.empty(words * rows, dtype=dtype, device=self.device)
        self.of[key] = [buf.zero_(), 0]
        return self.of[key]

    def put(self, key: str, words: int, v: torch.Tensor, at: int = 0) -> None:
        """The records v (`words` values each) behind the `at` values kept already."""
        m = at + v.numel()
        slot = self.of.get(key)
        if slot is None or m > slot[0].numel():
            old, slot = slot, self._grow(key, words, -(-m // words), v.dtype)
            if at:
                slot[0][:at].copy_(old[0][:at])
        if v.numel():
            slot[0][at:m].copy_(v, non_blocking=True)

    def end(self, key: str, m: int) -> torch.Tensor:
        slot = self.of[key]
        if slot[1] > m:
            slot[0][m:slot[1]].zero_()
        slot[1] = m
        return slot[0]


class _OnDevice:
    """Device memory of the library seen as a torch tensor."""

    def __init__(self, ptr: int, n: int, typestr: str):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": typestr, "version": 3}


def _device_view(ptr, n: int, typestr: str, dtype) -> torch.Tensor:
    return torch.as_tensor(_OnDevice(ptr, n, typestr), device="cuda") if n else torch.empty(0, dtype=dtype, device="cuda")


def _host_view(ptr, n: int, dtype) -> np.ndarray:
    return np.frombuffer((ctypes.c_uint8 * (n * np.dtype(dtype).itemsize)).from_address(ptr), dtype=dtype) if n else \
        np.zeros(0, dtype)


def _host_results(rs: lib.ResultSetC) -> dict:
    """The records of a host result set, in place (32-byte records as four words each)."""
    return {"hits": torch.from_numpy(_host_view(rs.hits, 4 * rs.n_hits, np.int64)),
            "locs": torch.from_numpy(_host_view(rs.locs, 4 * rs.n_locs, np.int64)),
            "counts": torch.from_numpy(_host_view(rs.rs_count, 2 * rs.n_reads, np.int32)),
            "truncated": torch.from_numpy(_host_view(rs.rs_truncated, 2 * rs.n_reads, np.uint8))}


class _Results:
    """A host result set: the library's until it is given back, which a program does before its next batch."""

    def __init__(self):
        self.rs = lib.ResultSetC()
        self.free = lib.load().bwt_gpu_result_free

    def give_back(self) -> None:
        self.free(ctypes.byref(self.rs))
        self.rs = lib.ResultSetC()

    __del__ = give_back


def _peek(at: np.ndarray, size: int) -> np.ndarray:
    """`size` bytes at each of the addresses `at`, as rows."""
    if not len(at):
        return np.zeros((0, size), np.uint8)
    base = int(at.min())
    span = int(at.max()) - base + size
    mem = np.frombuffer((ctypes.c_uint8 * span).from_address(base), dtype=np.uint8)
    return mem[(at.astype(np.int64) - base)[:, None] + np.arange(size)[None, :]]


# array_list_t: size at 8, items behind the mutex (40 bytes on x86-64, 48 on Arm) and the condition (48)
LIST_ITEMS = 40 + (48 if platform.machine() == "aarch64" else 40) + 48


class FastqBatch(ctypes.Structure):  # fastq_batch_t of include/hpg_bwt_api.h
    _fields_ = [("num_reads", ctypes.c_ulong), ("data_indices_size", ctypes.c_ulong), ("data_size", ctypes.c_ulong),
                ("source_id", ctypes.c_int), ("header_indices", ctypes.c_void_p), ("header", ctypes.c_void_p),
                ("data_indices", ctypes.c_void_p), ("seq", ctypes.c_void_p), ("quality", ctypes.c_void_p)]


# ------------------------------------------------------------------ prepare and run --

def prepare(case: dict, seed: int) -> dict:
    s = dict(case=case, lib=lib.load())
    if case["api"] == "serve":
        r = np.random.default_rng(case["requests"] + case["req_hi"])  # the sizes are the case's, the reads the seed's
        sizes = np.exp(r.uniform(np.log(case["req_lo"]), np.log(case["req_hi"]), case["requests"])).astype(int)
        total = int(sizes.sum())
        seq, offs = (_host(t).numpy() for t in _reads(case["genome"], total, case["lo"], case["hi"], case["edits"], seed))
        cuts = np.concatenate([[0], np.cumsum(sizes)])
        s["requests"] = [(seq[offs[a]:offs[b]], (offs[a:b + 1] - offs[a]).astype(np.uint64))
                         for a, b in zip(cuts[:-1], cuts[1:])]
        s["server"] = _server(case["genome"])
        s["kept"] = _Kept(total, "cpu")
        return s
    s["index"] = _index(case["genome"])
    seq, offs = _reads(case["genome"], case["reads"], case["lo"], case["hi"], case["edits"], seed)
    n = case["reads"]
    if case["api"] == "device":
        s.update(seq=seq, offs=offs, bases=seq.numel(), kept=_Kept(n, "cuda"),
                 stream=torch.cuda.ExternalStream(s["index"].stream()))
    elif case["api"] in ("host", "block"):
        s.update(seq=_host(seq), offs=_host(offs), results=_Results(), kept=_Kept(n, "cpu"))
        if case["api"] == "block":
            s["anchors"] = torch.zeros(4 * n * lib.ANCHOR_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
            s["nth"] = torch.arange(2, dtype=torch.uint8)[None, :]
            s["n_anchors"] = torch.zeros(2 * n, dtype=torch.uint8, pin_memory=True)
    else:  # NUL-terminated reads of a fastq file
        s["kept"] = _Kept(n, "cpu")
        lens = offs[1:] - offs[:-1]
        z = torch.zeros(seq.numel() + n, dtype=torch.uint8, device="cuda")
        read_of = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
        z[torch.arange(seq.numel(), device="cuda") + read_of] = seq
        s["text"] = z.cpu().numpy()
        start = (offs + torch.arange(n + 1, device="cuda")).cpu().numpy()
        if case["api"] == "cals":
            s["reads"] = (ctypes.c_void_p * n)(*(start[:n] + s["text"].ctypes.data).tolist())
            s["bwt_opt"] = s["lib"].bwt_optarg_new(1, 1, 200, case["max_results"])
            s["cal_opt"] = s["lib"].cal_optarg_new(20, 0, 0, 0, 16, 0, 0, 500_000, 0)
        else:
            ids = np.frombuffer(b"".join(b"@r%09d\0" % i for i in range(n)), dtype=np.uint8)
            s["keep"] = [start.astype(np.int32), np.where(s["text"] == 0, 0, ord("I")).astype(np.uint8), ids,
                         (np.arange(n + 1) * 12).astype(np.int32)]
            room = n * (case["hi"] + 1) + 1
            s["left"] = [np.zeros(room, np.uint8), np.zeros(n + 1, np.int32), np.zeros(room, np.uint8),
                         np.zeros(len(ids) + 1, np.uint8), np.zeros(n + 1, np.int32)]
            s["bwt_opt"] = s["lib"].bwt_optarg_new(1, 1, case["max_results"], case["max_results"])
    return s


def _check(s: dict, rc: int) -> None:
    if rc != 0:
        raise RuntimeError(s["lib"].bwt_gpu_last_error().decode())


def _modes(case: dict) -> tuple[int, int]:
    return (lib.MODE_EXACT if case["mode"] == "exact" else lib.MODE_SEARCH1,
            lib.FORM_PLAIN if case["form"] == "plain" else lib.FORM_BATCHED)


def _run_device(s: dict):
    c = s["case"]
    mode, form = _modes(c)
    rs = s["index"].search_device(s["seq"].data_ptr(), s["offs"].data_ptr(), c["reads"], s["bases"], c["hi"], mode, form,
                                  c["max_results"])
    got = {"hits": (_device_view(rs.hits, 4 * rs.n_hits, "<i8", torch.int64), 4),
           "locs": (_device_view(rs.locs, 4 * rs.n_locs, "<i8", torch.int64), 4),
           "counts": (_device_view(rs.rs_count, 2 * rs.n_reads, "<i4", torch.int32), 2),
           "truncated": (_device_view(rs.rs_truncated, 2 * rs.n_reads, "|u1", torch.uint8), 2)}
    with torch.cuda.stream(s["stream"]):  # the index's own stream: ahead of the next call's work on these buffers
        for k, (v, words) in got.items():
            s["kept"].put(k, words, v)
        return {k: s["kept"].end(k, len(v)) for k, (v, _) in got.items()}


def _run_host(s: dict):
    c, r = s["case"], s["results"]
    mode, form = _modes(c)
    r.give_back()
    _check(s, s["lib"].bwt_gpu_search_batch(s["index"].handle, mode, form, s["seq"].data_ptr(), s["offs"].data_ptr(),
                                            c["reads"], c["max_results"], ctypes.byref(r.rs)))
    return _keep_host(s, r.rs)


def _keep_host(s: dict, rs: lib.ResultSetC) -> dict:
    """The result set's arrays into the program's own."""
    got = _host_results(rs)
    for k, v in got.items():
        s["kept"].put(k, 4 if k in ("hits", "locs") else 2, v)
    return {k: s["kept"].end(k, len(v)) for k, v in got.items()}


def _run_block(s: dict):
    c, r = s["case"], s["results"]
    r.give_back()
    _check(s, s["lib"].bwt_gpu_block_search(s["index"].handle, s["seq"].data_ptr(), s["offs"].data_ptr(), c["reads"],
                                            c["max_results"], ctypes.byref(r.rs), s["anchors"].data_ptr(),
                                            s["n_anchors"].data_ptr()))
    out = _keep_host(s, r.rs)
    # the anchors that a list has: slots past its count say nothing
    out["n_anchors"] = s["n_anchors"]
    out["anchors"] = s["anchors"].view(torch.int64).view(-1, 2, 3)
    out["anchors"].mul_((s["n_anchors"][:, None] > s["nth"])[:, :, None])
    return out


def _run_serve(s: dict):
    tickets = [s["server"].submit(seq, offs) for seq, offs in s["requests"]]
    n = {"hits": 0, "locs": 0, "counts": 0, "truncated": 0}
    for t in tickets:
        rs, _ = s["server"].wait(t, copy=False)
        for k, v in _host_results(rs).items():
            s["kept"].put(k, 4 if k in ("hits", "locs") else 2, v, n[k])
            n[k] += len(v)
        s["server"].release(t)
    return {k: s["kept"].end(k, m) for k, m in n.items()}


def _run_lists(s: dict):
    L, n = s["lib"], s["case"]["reads"]
    (didx, qual, ids, hidx), (useq, udidx, uqual, uids, uhidx) = s["keep"], s["left"]
    batch = FastqBatch(num_reads=n, header_indices=hidx.ctypes.data, header=ids.ctypes.data,
                       data_indices=didx.ctypes.data, seq=s["text"].ctypes.data, quality=qual.ctypes.data)
    left = FastqBatch(header_indices=uhidx.ctypes.data, header=uids.ctypes.data, data_indices=udidx.ctypes.data,
                      seq=useq.ctypes.data, quality=uqual.ctypes.data)
    lst = L.array_list_new(max(16, n), 1.25, 2)
    L.bwt_map_inexact_batch(ctypes.byref(batch), s["bwt_opt"], s["index"].handle, ctypes.byref(left), lst)
    m = int(L.array_list_size(lst))
    items = ctypes.c_void_p.from_address(lst + LIST_ITEMS).value
    rec = _peek(_host_view(items, m, np.int64), 50)  # alignment_t up to its flags
    s["kept"].put("numbers", 10, torch.from_numpy(np.ascontiguousarray(rec[:, :40]).view(np.int32).reshape(-1)))
    s["kept"].put("flags", 10, torch.from_numpy(np.ascontiguousarray(rec[:, 40:50]).reshape(-1)))
    out = {"numbers": s["kept"].end("numbers", 10 * m), "flags": s["kept"].end("flags", 10 * m),
           "unmapped": int(left.num_reads), "unmapped_bases": useq}
    L.array_list_free(lst, ctypes.cast(L.alignment_free, ctypes.c_void_p))
    return out


def _run_cals(s: dict):
    L, n = s["lib"], s["case"]["reads"]
    lists = (ctypes.c_void_p * n)(*[L.array_list_new(16, 1.25, 2) for _ in range(n)])
    L.bwt_generate_cals_batch(s["reads"], n, 16, s["bwt_opt"], s["cal_opt"], s["index"].handle, lists, 1)
    at = np.frombuffer(lists, dtype=np.int64)
    size = _peek(at + 8, 8).view(np.int64)[:, 0]
    items = _peek(at + LIST_ITEMS, 8).view(np.int64)[:, 0]
    first = np.repeat(items - 8 * np.concatenate([[0], np.cumsum(size)[:-1]]), size) + 8 * np.arange(int(size.sum()))
    rec = _peek(_peek(first, 8).view(np.int64)[:, 0], 44)  # cal_t: chromosome, strand, start, end, seeds, read area
    out = {"cals_per_read": size.copy()}
    places = np.delete(rec[:, :40], np.s_[8:16], 1)
    for key, size, v in (("places", 32, places), ("strand", 2, rec[:, 8:10]), ("area", 4, rec[:, 40:44])):
        v = torch.from_numpy(np.ascontiguousarray(v).reshape(-1))
        s["kept"].put(key, size, v)
        out[key] = s["kept"].end(key, v.numel())
    free = ctypes.cast(L.cal_free, ctypes.c_void_p)
    for p in lists:
        L.array_list_free(p, free)
    return out


def run(state: dict):
    return _RUN[state["case"]["api"]](state)


_RUN = {"device": _run_device, "host": _run_host, "block": _run_block, "serve": _run_serve, "lists": _run_lists,
        "cals": _run_cals}


# ------------------------------------------------------------------ what a pass cannot do without --

def work(case: dict) -> dict:
    """Bytes: the reads and their offsets once, the parts of the index that they can touch once (a 32-byte block per
    base and strand at most, the whole index at most), and the records of about one hit and one located row a read."""
    mean = (case["lo"] + case["hi"]) / 2
    n = case["reads"] if "reads" in case else \
        case["requests"] * (case["req_hi"] - case["req_lo"]) / np.log(case["req_hi"] / case["req_lo"])
    index = min(GENOMES[case["genome"]] * 2.0, n * mean * 2 * 32)
    return {"bytes": float(n * (mean + 8) + index + n * (2 * 32 + 10)), "flops": 0.0}


def exact(case: dict, seed: int):
    """Every output is whole numbers: intervals, places, counts, flags."""
    return None
