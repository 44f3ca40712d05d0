"""Cases that the caller's speed is measured on.

Each case is one call that a program of this package makes, through the C ABI
of include/gsnp_gb300.h (gsnp_gb300.api), on seeded synthetic alignments of one
of the shapes of gsnp_gb300.synth:

  op "call"       gsnp_call_chromosome_into: alignments in pinned host memory
                  to every site's 32-byte call in pinned host memory
  op "recall"     gsnp_recall_resident and gsnp_fetch_sites: the alignments of
                  the last call, still on the device, called again
  op "stream"     gsnp_call_streamed: the same as "call" with bounded device
                  memory, and the six -C files written on the way
  op "calibrate"  gsnp_calibrate: the first pass over the alignments
  op "text"       gsnp_format_cns: the cns text of the resident calls
  op "columns"    gsnp_write_columns: the six -C files of the resident calls

The inputs follow the shapes' distributions (depth, read lengths, quality
model, SNP and dbSNP rates, copy-number segments, hotspots, N runs), drawn on
the GPU from the seed alone.
"""
from __future__ import annotations

import ctypes
import functools
import math
import os
import shutil
import tempfile
import weakref

import numpy as np
import torch

from gsnp_gb300 import api, synth

CHR = "chr1"
COLUMN_FILES = ("1_2", "3_4_6", "5_7_8_9_14_16", "10", "11_12_13", "15_17")
# the -C files go to a RAM-backed directory where the host has one
RAM_DIR = "/dev/shm" if os.path.isdir("/dev/shm") and os.access("/dev/shm", os.W_OK) else None
# every field of a call that the cns row is made of; "flags" (which internal
# path decided the call) and "pad" are not part of the result.  The 16- and
# 32-bit counts are seen as signed numbers, which tensors have.
FIELDS = [f for f in api.SITE_DTYPE.names if f not in ("flags", "pad")]
SIGNED = {"<u2": "<i2", "<u4": "<i4"}
CALL_DTYPE = np.dtype([(n, SIGNED.get(api.SITE_DTYPE[n].str, api.SITE_DTYPE[n].str)) for n in api.SITE_DTYPE.names])
# room for a site's cns row, and for its share of one -C file
ROW_BYTES, COLUMN_BYTES = 96, 6

# mean depth of the copy-number shape: its segments' mean multiplier, and its
# hotspots (0.5% of sites at 300-1000 reads)
CN_MULT = (0.0, 0.5, 1.0, 2.0, 8.0)
CN_PROB = (0.05, 0.15, 0.6, 0.15, 0.05)


def listed():
    def case(name, op, shape, sites, form="fp32", packed=False):
        return {"name": name, "op": op, "shape": shape, "sites": sites, "form": form, "packed": packed}

    return [
        # a targeted region of 30 kb at 30x: the smallest calls, where launches and waits count
        case("region_30k", "call", "c1", 30_011),
        # the plain FP64 method at its own small configuration, 1 Mbp of 50 bp reads at 10x
        case("c0_fp64_1m", "call", "c0", 1_000_000, "fp64"),
        # the headline: 100 bp reads at 30x with known SNPs, packed reads, both forms
        case("c1_fp32_16m", "call", "c1", 16_000_000, "fp32", True),
        case("c1_fp64_6m", "call", "c1", 6_100_003, "fp64"),
        # very uneven depth: copy-number segments and hotspots of 300-1000 reads, mixed read lengths
        case("c2_fp32_10m", "call", "c2", 10_000_000, "fp32", True),
        case("c2_fp64_3m", "call", "c2", 3_000_000, "fp64"),
        # qualities up to 60
        case("c3_fp32_5m", "call", "c3", 5_000_000),
        # long reads, 150-250 bp
        case("c5_fp32_3m", "call", "c5", 2_999_999),
        # chromosome-scale: 40x streamed in chunks, calls and -C files written
        case("c4_stream_17m", "stream", "c4", 17_000_000, "fp32", True),
        # the resident alignments called again (another pass of the same chromosome)
        case("c1_recall_8m", "recall", "c1", 8_000_000, "fp32", True),
        # the two passes around the call: calibration before it, text after it
        case("c1_calibrate_8m", "calibrate", "c1", 8_000_000),
        case("c1_text_4m", "text", "c1", 4_000_000),
    ]


# the most sites a drawn case of each operation and shape has
MOST_SITES = {
    "call": {"c0": 16_000_000, "c1": 16_000_000, "c2": 10_000_000, "c3": 14_000_000, "c4": 11_000_000, "c5": 12_000_000},
    "recall": {"c0": 12_000_000, "c1": 10_000_000, "c2": 6_000_000, "c3": 10_000_000, "c4": 8_000_000, "c5": 8_000_000},
    "stream": {"c0": 16_000_000, "c1": 14_000_000, "c2": 8_000_000, "c3": 14_000_000, "c4": 14_000_000, "c5": 8_000_000},
    "calibrate": {"c0": 16_000_000, "c1": 12_000_000, "c2": 8_000_000, "c3": 12_000_000, "c4": 8_000_000, "c5": 8_000_000},
    "text": {"c0": 6_000_000, "c1": 6_000_000, "c2": 6_000_000, "c3": 6_000_000, "c4": 6_000_000, "c5": 6_000_000},
    "columns": {"c0": 8_000_000, "c1": 8_000_000, "c2": 6_000_000, "c3": 8_000_000, "c4": 8_000_000, "c5": 8_000_000},
}


def draw(rng):
    op = rng.choice(["call"] * 6 + ["recall", "stream", "calibrate", "text", "columns"])
    shape = rng.choice(["c0", "c1", "c1", "c2", "c2", "c3", "c4", "c5"])
    most = MOST_SITES[op][shape]
    form = rng.choice(["fp32", "fp32", "fp64"])
    if form == "fp64":
        most //= 3
    sites = int(round(math.exp(rng.uniform(math.log(25_000), math.log(most)))))
    return {"op": op, "shape": shape, "sites": sites, "form": form, "packed": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _mean_depth(cfg):
    d = cfg.depth
    if cfg.cn_segments:
        d *= sum(m * p for m, p in zip(CN_MULT, CN_PROB))
    if cfg.hotspots:
        d += 0.005 * 650.0 * float(np.mean(cfg.read_lens)) / 80.0
    return d


def _starts(cfg, G, isn_prefix, gen, dev):
    """Sorted read starts and their lengths: uniform over the genome, or by
    copy-number segment, plus the hotspots' reads; none over an N."""
    lens_of = torch.tensor(cfg.read_lens, device=dev)
    mean_len = float(np.mean(cfg.read_lens))

    def lengths(n):
        return lens_of[torch.randint(0, len(cfg.read_lens), (n,), generator=gen, device=dev)]

    def uniform(n):
        return torch.rand(n, generator=gen, device=dev, dtype=torch.float64)

    if cfg.cn_segments:
        m = max(4, int(G / 100_000 * 2) + 16)
        seg = (1 - torch.log(1 - uniform(m)) * 100_000).long()
        edge = torch.clamp(torch.cumsum(seg, 0), max=G)
        edge[-1] = G
        mult = torch.tensor(CN_MULT, device=dev, dtype=torch.float64)
        cdf = torch.cumsum(torch.tensor(CN_PROB, device=dev, dtype=torch.float64), 0)
        w = mult[torch.clamp(torch.searchsorted(cdf, uniform(m), right=True), max=4)]
        lo = torch.cat([torch.zeros(1, device=dev, dtype=torch.long), edge[:-1]])
        mass = torch.cumsum(w * (edge - lo).double(), 0)
        total = float(mass[-1])
        n = int(round(cfg.depth * total / mean_len))
        u = uniform(n) * total
        k = torch.clamp(torch.searchsorted(mass, u, right=True), max=m - 1)
        # the place within the segment, from the mass left of it
        start = (edge[k].double() - (mass[k] - u) / torch.clamp(w[k], min=1e-9)).long()
    else:
        n = int(round(cfg.depth * G / mean_len))
        start = (uniform(n) * G).long()
    length = lengths(n)
    if cfg.hotspots:
        n_hot = max(1, int(0.005 * G / 80))
        centre = 200 + (uniform(n_hot) * max(1, G - 400)).long()
        extra = 300 - int(cfg.depth) + (uniform(n_hot) * 701).long()
        at = torch.repeat_interleave(centre, extra)
        ln = lengths(at.numel())
        off = torch.randint(-10, 11, (at.numel(),), generator=gen, device=dev)
        start = torch.cat([start, at + off - torch.div(ln, 2, rounding_mode="floor")])
        length = torch.cat([length, ln])
    start = torch.clamp(start, min=0)
    ok = start + length < G
    ok &= isn_prefix[torch.clamp(start + length, max=G)] == isn_prefix[torch.clamp(start, max=G)]
    start, length = start[ok], length[ok]
    start, order = torch.sort(start, stable=True)
    return start, length[order]


def _host(t, pinned=True):
    """A device tensor's values in host memory, page-locked as a program keeps what it uploads."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=pinned)
    h.copy_(t)
    return h.numpy()


def _inputs(case, seed, with_counts=False):
    """The reference codes, dbSNP rows and alignments of a case (host arrays),
    and with with_counts the calibration counts of the alignments."""
    cfg = synth.CONFIGS[case["shape"]]
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(int(seed) * 7919 + 17)
    G = int(case["sites"])
    L = max(cfg.read_lens)

    def rand(n):
        return torch.rand(n, generator=gen, device=dev)

    # the reference (GC 41%), its N runs, and a diploid sample with SNPs
    code = torch.bucketize(rand(G), torch.tensor([0.295, 0.5, 0.795], device=dev), right=True).to(torch.uint8)
    isn = torch.zeros(G, dtype=torch.bool, device=dev)
    for run in cfg.n_runs:
        run = min(run, G // 8)
        lo = G // 3
        at = lo + int(torch.randint(0, max(1, G - run - G // 5 - lo), (1,), generator=gen, device=dev))
        isn[at:at + run] = True
    prefix = torch.cat([torch.zeros(1, dtype=torch.int32, device=dev), torch.cumsum(isn, 0, dtype=torch.int32)])
    hap = code.repeat(2, 1)
    snp = torch.nonzero((rand(G) < cfg.snp_rate) & ~isn).flatten()
    K = snp.numel()
    ref_s = code[snp]
    alt = torch.where(rand(K) < 2 / 3, ref_s ^ 3, torch.where(rand(K) < 0.5, ref_s ^ 1, ref_s ^ 2))
    het, first = rand(K) < 2 / 3, rand(K) < 0.5
    hap[0, snp] = torch.where(~het | first, alt, ref_s)
    hap[1, snp] = torch.where(~het | ~first, alt, ref_s)

    # known SNPs
    if cfg.dbsnp_frac > 0:
        db = torch.nonzero((rand(G) < cfg.dbsnp_frac) & ~isn).flatten()
        n_db = db.numel()
        second = code[db] ^ torch.where(rand(n_db) < 2 / 3, 3, torch.where(rand(n_db) < 0.5, 1, 2)).to(torch.uint8)
        true_alt = torch.full((G,), 255, dtype=torch.uint8, device=dev)
        true_alt[snp] = alt
        second = torch.where(true_alt[db] != 255, true_alt[db], second)
        f = torch.round(0.01 + 0.49 * rand(n_db).double(), decimals=4)
        freq = torch.zeros(n_db, 4, dtype=torch.float64, device=dev)
        freq.scatter_(1, code[db].long()[:, None], torch.round(1.0 - f, decimals=4)[:, None])
        freq.scatter_(1, second.long()[:, None], f[:, None])
        rows = np.zeros(n_db, dtype=api.SNP_DTYPE)
        rows["pos"] = db.cpu().numpy()
        rows["hapmap"] = (rand(n_db) < 0.5).cpu().numpy()
        rows["validated"] = (rand(n_db) < 0.8).cpu().numpy()
        rows["freq"] = freq.cpu().numpy()
    else:
        db, rows = None, None
    ascii_of = torch.tensor(list(b"ACTG"), dtype=torch.uint8, device=dev)
    site_code = torch.where(isn, torch.tensor(4 | ((ord("N") >> 1) & 3), dtype=torch.uint8, device=dev), code)
    if db is not None:
        site_code[db] |= 8

    # alignments: uniform starts, half of them reversed, 5% with several hits
    start, length = _starts(cfg, G, prefix, gen, dev)
    n = start.numel()
    minus = rand(n) < 0.5
    hit = torch.where(rand(n) < 0.05, 2 + torch.randint(0, 4, (n,), generator=gen, device=dev), 1)
    which = (rand(n) < 0.5).long()
    packed = bool(case["packed"])
    seq = np_empty((n, L))
    qual = None if packed else np_empty((n, L))
    n_q = cfg.q_hi + 1
    counts = torch.zeros((64, L, 4, 4), dtype=torch.int64, device=dev) if with_counts else None
    cyc = torch.arange(L, device=dev)
    for r0 in range(0, n, 1 << 20):
        r1 = min(n, r0 + (1 << 20))
        st, ln, mi = start[r0:r1, None], length[r0:r1, None], minus[r0:r1, None]
        # qualities and miscalls by cycle, then turned to reference order
        mu = cfg.q_mu0 + (cfg.q_mu1 - cfg.q_mu0) * (cyc[None, :] / torch.clamp(ln - 1, min=1))
        q = torch.round(mu + cfg.q_sd * torch.randn(r1 - r0, L, generator=gen, device=dev))
        q = torch.clamp(q, cfg.q_lo, cfg.q_hi)
        if cfg.lowq_clusters > 0:
            low = torch.rand(r1 - r0, L, generator=gen, device=dev) < cfg.lowq_clusters
            val = torch.randint(2, 9, (r1 - r0, L), generator=gen, device=dev).float()
            low[:, L - 5:] = False
            for d in range(5):
                q = torch.where(torch.roll(low, d, 1), torch.roll(val, d, 1), q)
        u = torch.rand(r1 - r0, L, generator=gen, device=dev)
        err = u < torch.pow(10.0, -q / 10.0)
        shift = torch.where(err, torch.randint(1, 4, (r1 - r0, L), generator=gen, device=dev), 0)
        valid = cyc[None, :] < ln
        cycle = torch.where(mi & valid, ln - 1 - cyc[None, :], cyc[None, :].expand(r1 - r0, L))
        q = torch.gather(q, 1, cycle).to(torch.uint8)
        site = torch.clamp(st + cyc[None, :], max=G - 1)
        truth = hap[which[r0:r1, None], site]
        obs = (truth + torch.gather(shift, 1, cycle).to(torch.uint8)) & 3
        if counts is not None:
            use = valid & (hit[r0:r1, None] == 1) & ((site_code[site] & 12) == 0)
            key = ((q.long() * L + cycle) * 4 + code[site].long()) * 4 + obs.long()
            counts += torch.bincount(key[use], minlength=64 * L * 16).reshape(64, L, 4, 4)
        if packed:
            s = torch.where(valid, (obs << 6) | q, torch.zeros_like(q))
            torch.from_numpy(seq[r0:r1]).copy_(s)
        else:
            zero = torch.zeros_like(q)
            torch.from_numpy(seq[r0:r1]).copy_(torch.where(valid, ascii_of[obs.long()], zero))
            torch.from_numpy(qual[r0:r1]).copy_(torch.where(valid, q + 64, zero))
    assert n_q <= 63
    return {
        "codes": site_code.cpu().numpy(), "snp": rows,
        "pos": _host(start.int()), "len": _host(length.int()), "hit": _host(hit.int()),
        "strand": _host(torch.where(minus, ord("-"), ord("+")).to(torch.uint8)),
        "seq": seq, "qual": qual, "counts": counts,
    }


def np_empty(shape):
    """A page-locked byte array."""
    return torch.empty(shape, dtype=torch.uint8, pin_memory=True).numpy()


def _flags(case):
    cfg = synth.CONFIGS[case["shape"]]
    return [f for f in cfg.flags if f != "-C"]


def _params(case):
    return api.params_from_flags(_flags(case), api.PRECISION_FP64 if case["form"] == "fp64" else api.PRECISION_FP32_FIXUP)


@functools.lru_cache(maxsize=1)
def _rank_table():
    """The rank-sum table, the same for every chromosome and parameter set; a program makes it once."""
    from gsnp_gb300 import native
    out = np.empty(64 * 64 * 2048, dtype=np.float64)
    if native().gsnp_rank_table(out.ctypes.data) != 0:
        raise RuntimeError("gsnp_rank_table failed")
    return out


class State:
    """What a program holds before the call: a context with the reference and
    the tables loaded, the alignments in pinned host memory, room for the result."""

    def __init__(self, case, seed):
        d = _inputs(case, seed)
        self.case = dict(case)
        self.caller = api.Caller(torch.cuda.current_device())
        self.dir = None
        self._closed = weakref.finalize(self, State._close, self.caller, self.__dict__)
        self.arrays = d
        packed = bool(case["packed"])
        self.reads = api.Caller.reads_struct(d["pos"], d["len"], d["hit"], d["strand"],
                                             None if packed else d["seq"], d["qual"],
                                             d["seq"] if packed else None, 64 if packed else 0)
        self.params = _params(case)
        self.caller.load_reference(d["codes"], d["snp"])
        op = case["op"]
        if op == "calibrate":
            return
        pm = self.caller.calibrate(self.params, self.reads)
        self.caller.load_tables(self.params, pm, self.caller.prior_table(self.params), _rank_table())
        if op in ("call", "recall", "stream"):
            self.raw = np_empty(int(case["sites"]) * api.SITE_DTYPE.itemsize)
            self.out = self.raw.view(CALL_DTYPE)
        if op in ("recall", "text", "columns"):
            self.caller.call(self.reads)
        if op in ("stream", "columns"):
            self.dir = tempfile.mkdtemp(prefix="gsnp_cases_", dir=RAM_DIR)
        if op == "text":
            self.text = np.zeros(ROW_BYTES * int(case["sites"]) + (1 << 16), dtype=np.uint8)

    @staticmethod
    def _close(caller, held):
        caller.close()
        if held.get("dir"):
            shutil.rmtree(held["dir"], ignore_errors=True)

    def calls(self):
        """every call's fields, where the caller wrote them"""
        return {f: self.out[f] for f in FIELDS}

    def files(self):
        """the six -C files, mapped: each with its length, the mapping going on
        in zeros to one length for every chromosome of this size (the files
        are lengthened without writing)"""
        got = {}
        room = COLUMN_BYTES * int(self.case["sites"]) + (1 << 20)
        for f in COLUMN_FILES:
            path = os.path.join(self.dir, "cns." + f)
            got["bytes " + f] = os.path.getsize(path)
            if got["bytes " + f] > room:
                raise RuntimeError("%s is longer than %d bytes" % (path, room))
            os.truncate(path, room)
            got["file " + f] = np.memmap(path, dtype=np.uint8, mode="r")
        return got


def prepare(case, seed):
    return State(case, seed)


def run(state):
    c, op = state.caller, state.case["op"]
    if op == "call":
        c.call_into(state.reads, state.raw.ctypes.data)
        return state.calls()
    if op == "recall":
        c.recall_resident()
        c._check(c.lib.gsnp_fetch_sites(c.ctx, 0, c.length, state.raw.ctypes.data), "gsnp_fetch_sites")
        return state.calls()
    if op == "stream":
        c.call_streamed(state.reads, CHR, state.raw.ctypes.data, None, os.path.join(state.dir, "cns"))
        return {**state.calls(), **state.files()}
    if op == "calibrate":
        return c.calibrate(state.params, state.reads)
    if op == "columns":
        c._check(c.lib.gsnp_write_columns(c.ctx, CHR.encode(), os.path.join(state.dir, "cns").encode()),
                 "gsnp_write_columns")
        return state.files()
    # the text: its size first, then the text into the program's buffer (zeros follow it)
    size = ctypes.c_int64(0)
    c._check(c.lib.gsnp_format_cns(c.ctx, CHR.encode(), None, ctypes.byref(size)), "gsnp_format_cns")
    if size.value > state.text.size:
        raise RuntimeError("the text is longer than %d bytes" % state.text.size)
    c._check(c.lib.gsnp_format_cns(c.ctx, CHR.encode(), state.text.ctypes.data, ctypes.byref(size)), "gsnp_format_cns")
    return {"text": state.text, "bytes": size.value}


def work(case):
    """Bytes: the alignments (base and quality, one byte when packed, and 13
    bytes of start, length, hits and strand per read), the 4-bit reference
    codes and the 32-byte calls, each once; a text row is about 66 bytes, a
    site of the -C files 6.  Operations: ten genotype terms per covering
    base and about 40 for the posterior of a site."""
    cfg = synth.CONFIGS[case["shape"]]
    G = float(case["sites"])
    bases = _mean_depth(cfg) * G
    reads = bases / float(np.mean(cfg.read_lens))
    alignments = bases * (1.0 if case["packed"] else 2.0) + 13.0 * reads
    calls, codes = 32.0 * G, 0.5 * G
    op = case["op"]
    if op == "calibrate":
        return {"bytes": alignments + codes + 8.0 * 256 * 256 * 16, "flops": bases}
    if op == "text":
        return {"bytes": calls + codes + 66.0 * G, "flops": 20.0 * G}
    if op == "columns":
        return {"bytes": calls + codes + 6.0 * G, "flops": 20.0 * G}
    files = 6.0 * G if op == "stream" else 0.0
    return {"bytes": alignments + codes + calls + files, "flops": 10.0 * bases + 40.0 * G}


def exact(case, seed):
    """The calibration matrix in 64 bits (the ratios of cpp/matrix.cc:129-205
    from the counts).  The calls' one floating field, the rank-sum value, takes
    the whole caller to reproduce (the genotype decides which reads it ranks),
    far over 20 seconds in numpy."""
    if case["op"] != "calibrate":
        return None
    p = _params(case)
    L = p.read_length
    nq = p.q_max - p.q_min + 1
    cnt = _inputs(case, seed, True)["counts"][:nq].cpu().numpy().astype(np.float64)   # [q][cycle][ref][obs]
    pm = np.ones((256, 256, 4, 4), dtype=np.float64)
    by_type = cnt.sum(axis=1)                                      # [q][ref][obs]
    total = by_type.sum(axis=(1, 2))
    mism = total - np.einsum("qii->q", by_type)
    same = np.eye(4, dtype=bool)[None, None]
    with np.errstate(divide="ignore", invalid="ignore"):
        v = np.where(cnt > 10, cnt / cnt.sum(axis=3, keepdims=True),
                     np.where((by_type > 10)[:, None], (by_type / by_type.sum(axis=2, keepdims=True))[:, None],
                              np.where(same, ((total - mism) / total)[:, None, None, None],
                                       (mism / total)[:, None, None, None])))
    v = np.where((total > 0)[:, None, None, None], v, 1.0)
    e = 10.0 ** (-np.arange(nq) / 10.0)[:, None, None, None]
    filled = np.where(same, np.maximum(1.0 - e, 0.25), np.minimum(e / 3.0, 0.25))
    pm[:nq, :L] = np.where((v == 0) | (v == 1), filled, v)
    return pm.reshape(-1)
