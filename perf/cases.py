"""What a user of this framework has it do, as cases that can be timed.

Two kinds of work: digests of files (stream mode and block mode, from host
buffers and from device memory) and comparisons of digests (all pairs of a
set, queries against a resident set, sets read from SDBF text).  Every case
goes through the public Context calls.

Content is the repository's seeded synthetic mixture (half uniform-random
regions, a quarter low-entropy runs, a quarter order-1 Markov text).  A case
fixes the sizes; the seed gives the bytes.  All outputs are whole numbers and
bytes: filters, counts and scores.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import sdhash_gb300 as sd
from sdhash_gb300 import synth

KIB, MIB = 1 << 10, 1 << 20
BLOCK = 16 * KIB            # the command line's -b 16
SEGMENT = 128 * MIB         # block mode digests large inputs in segments of this size
STREAM_FILTER = 12.3 * KIB  # mixture content per stream-mode filter, about

_context = None


def context():
    """One context per process, as a program that digests or compares keeps one."""
    global _context
    if _context is None:
        _context = sd.Context(0)
    return _context


# ------------------------------------------------------------------- cases
def listed():
    return [
        # one small file as it is read, one call each: where launches and waits count
        dict(name="stream_one_64k", path="stream_one", bytes=64 * KIB + 11),
        # 64 files of exactly 1 MiB in pinned host memory: a directory of ordinary files
        dict(name="stream_host_64x1m", path="stream_host", files=64, lo=MIB, hi=MIB),
        # very uneven files in pinned host memory, copy included
        dict(name="stream_host_bulk", path="stream_host", files=160, lo=4 * KIB, hi=64 * MIB),
        # very uneven files already on the device: the bulk digest
        dict(name="stream_device_bulk", path="stream_device", files=512, lo=4 * KIB, hi=64 * MIB),
        # one large file of several 32 MiB chunks and an odd tail
        dict(name="stream_device_large", path="stream_device", files=1, lo=200 * MIB + 4099, hi=200 * MIB + 4099),
        # a disk image in block mode, 128 MiB segments, on the device
        dict(name="block_device_image", path="block_device", files=8, lo=SEGMENT, hi=SEGMENT),
        # query fragments in block mode from host memory: short inputs with tail blocks
        dict(name="block_host_fragments", path="block_host", files=768, lo=4 * KIB, hi=MIB),
        # all pairs of 64 digests of 1 MiB files (sdhash -g): a small comparison
        dict(name="all_pairs_64x1m", path="all_pairs", digests=64, lo=85, hi=85, fast=False, where="host"),
        # all pairs of digests of very uneven filter counts, scores left on the device
        dict(name="all_pairs_uneven", path="all_pairs", digests=400, lo=1, hi=2000, fast=False, where="device"),
        # many query fragments against a resident image: the bulk query-target comparison
        dict(name="queries_image", path="queries", queries=2048, lo=4 * KIB, hi=MIB, segments=4, each_new=False),
        # one query against a resident image, uploaded as it arrives: a lookup
        dict(name="one_query_image", path="queries", queries=1, lo=600 * KIB, hi=600 * KIB, segments=4, each_new=True),
        # a set file read and compared with itself (sdhash -c): text in, scores out
        dict(name="text_all_pairs", path="text", files=200, lo=16 * KIB, hi=16 * MIB),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mean(lo, hi):
    """Mean of a log-uniform size."""
    return hi if hi <= lo + 1 else (hi - lo) / math.log(hi / lo)


def draw(rng):
    path = rng.choice(["stream_one", "stream_host", "stream_device", "stream_device", "block_device", "block_host",
                       "all_pairs", "all_pairs", "queries", "queries", "text"])
    if path == "stream_one":
        return dict(path=path, bytes=_log(rng, 4 * KIB, 8 * MIB))
    if path in ("stream_host", "stream_device"):
        hi = _log(rng, 64 * KIB, 64 * MIB)
        lo = _log(rng, 4 * KIB, hi)
        most = (600 * MIB if path == "stream_host" else 2400 * MIB) / _mean(lo, hi)
        return dict(path=path, files=max(1, min(2048, _log(rng, 1, max(2, most)))), lo=lo, hi=hi)
    if path == "block_device":
        size = _log(rng, 256 * KIB, SEGMENT)
        return dict(path=path, files=max(1, min(512, _log(rng, 1, max(2, 900 * MIB / size)))), lo=size, hi=size)
    if path == "block_host":
        hi = _log(rng, 32 * KIB, 4 * MIB)
        return dict(path=path, files=max(1, min(512, _log(rng, 4, max(5, 120 * MIB / hi)))), lo=min(hi, _log(rng, KIB, 64 * KIB)),
                    hi=hi)
    if path == "all_pairs":
        hi = _log(rng, 4, 2000)
        lo = _log(rng, 1, hi)
        most = 80000 / _mean(lo, hi)  # filters in all: fewer than the largest listed set has
        return dict(path=path, digests=max(2, min(1500, _log(rng, 16, max(17, most)))), lo=lo, hi=hi,
                    fast=rng.random() < 0.25, where=rng.choice(["host", "device"]))
    if path == "queries":
        if rng.random() < 0.4:
            size = _log(rng, 4 * KIB, 16 * MIB)
            return dict(path=path, queries=1, lo=size, hi=size, segments=rng.choice([1, 2, 4]), each_new=True)
        return dict(path=path, queries=_log(rng, 8, 1200), lo=_log(rng, 2 * KIB, 16 * KIB), hi=_log(rng, 64 * KIB, MIB),
                    segments=rng.choice([1, 2, 4]), each_new=rng.random() < 0.3)
    return dict(path=path, files=_log(rng, 8, 150), lo=_log(rng, 2 * KIB, 32 * KIB), hi=_log(rng, 64 * KIB, 16 * MIB))


# ------------------------------------------------------------------ inputs
def _sizes(count, lo, hi, which=7):
    """Log-uniform sizes fixed by the case (the seed gives the content)."""
    if lo == hi:
        return np.full(count, lo, dtype=np.uint64)
    return synth.log_uniform_sizes(which, count, lo, hi)


def _fill(seed, sizes, pinned=False):
    """Mixture content for inputs of these sizes, packed 16-byte aligned: (buffer, offsets, sizes)."""
    offs, total = synth.packed_layout(sizes)
    if pinned:
        data = torch.empty(max(16, total), dtype=torch.uint8, pin_memory=True).numpy()
    else:
        data = np.empty(max(16, total), dtype=np.uint8)
    # pieces of a few MiB, so that one large input is made by all host threads
    piece = 4 * MIB
    if total:
        cuts = [piece] * (total // piece) + ([total % piece] if total % piece else [])
        synth.fill_many(seed, "mixture", np.array(cuts, dtype=np.uint64), out=data)
    return data, offs, sizes


def _stream_digests(ctx, seed, sizes, tag):
    """Digests of a collection in which every second file shares a part of its content with the one before it."""
    data, offs, lens = _fill(seed, sizes)
    rng = np.random.default_rng(seed)
    for i in range(1, len(lens), 2):
        a, b, na = int(offs[i - 1]), int(offs[i]), int(lens[i - 1])
        share = int(min(na, int(lens[i])) * rng.uniform(0.2, 0.8))
        data[b:b + share] = data[a + na - share:a + na]
    return ctx.digest_packed(data, offs, lens, 0, names=[f"{tag}{i:05d}" for i in range(len(lens))])


def _segments(n):
    return np.full(n, SEGMENT, dtype=np.uint64)


def _fields(res, n):
    """The per-input results of a device digest call."""
    a = np.frombuffer(res, dtype=[("bf_count", "u4"), ("last_count", "u4"), ("status", "i4"), ("reserved", "u4"),
                                  ("filter_offset", "u8")], count=n)
    return {k: a[k].astype(np.int64) for k in ("bf_count", "last_count", "status", "filter_offset")}


def prepare(case, seed):
    ctx = context()
    path = case["path"]
    if path == "stream_one":
        data, offs, lens = _fill(seed, np.array([case["bytes"]], dtype=np.uint64))
        return dict(path=path, ctx=ctx, data=data, offs=offs, lens=lens,
                    filters=np.zeros(ctx.capacity(lens) * 256, dtype=np.uint8))
    if path in ("stream_host", "stream_device", "block_device", "block_host"):
        dd = BLOCK if path.startswith("block") else 0
        sizes = _sizes(case["files"], case["lo"], case["hi"])
        data, offs, lens = _fill(seed, sizes, pinned=path == "stream_host")
        cap = ctx.capacity(lens, dd)
        st = dict(path=path, ctx=ctx, offs=offs, lens=lens, dd=dd, cap=cap)
        if path.endswith("_device"):
            st["data"] = torch.from_numpy(data).cuda()
            st["filters"] = torch.zeros(max(1, cap) * 256, dtype=torch.uint8, device="cuda")
            st["counts"] = torch.zeros(max(1, cap), dtype=torch.int16, device="cuda") if dd else None
        else:
            st["data"] = data
            st["filters"] = torch.zeros(max(1, cap) * 256, dtype=torch.uint8, pin_memory=True).numpy()
        return st
    if path == "all_pairs":
        counts = _sizes(case["digests"], case["lo"], case["hi"])
        digs = _stream_digests(ctx, seed, (counts.astype(np.float64) * STREAM_FILTER).astype(np.uint64), "d")
        if case["fast"]:
            digs = [d.fast() for d in digs]
        st = dict(path=path, ctx=ctx, where=case["where"], set=ctx.upload(digs))
        if case["where"] == "device":
            n = len(digs)
            st["scores"] = torch.zeros(n * (n - 1) // 2, dtype=torch.int32, device="cuda")
        return st
    if path == "queries":
        # 60 % of the fragments are cut from the image (their first bytes changed), the others are fresh random bytes
        segs = _segments(case["segments"])
        image, offs, lens = _fill(seed, segs)
        target = ctx.digest_packed(image, offs, lens, BLOCK, names=[f"image{i:02d}" for i in range(len(lens))])
        sizes = _sizes(case["queries"], case["lo"], case["hi"])
        qoffs, qtot = synth.packed_layout(sizes)
        qdata, _, _ = synth.fill_many(seed + 1, "random", sizes)
        rng = np.random.default_rng(seed)
        for i in range(len(sizes)):
            n = int(sizes[i])
            if rng.random() < 0.6 or len(sizes) == 1:
                s, o, keep = int(rng.integers(0, image.size - n)), int(qoffs[i]), int(n * rng.uniform(0.0, 0.5))
                qdata[o + keep:o + n] = image[s + keep:s + n]
        queries = ctx.digest_packed(qdata, qoffs, sizes, BLOCK, names=[f"query{i:05d}" for i in range(len(sizes))])
        st = dict(path=path, ctx=ctx, target=ctx.upload(target), each_new=case["each_new"])
        if case["each_new"]:
            st["queries"] = queries
        else:
            st["queries"] = ctx.upload(queries)
            st["scores"] = torch.zeros(len(queries), len(target), dtype=torch.int32, device="cuda")
        return st
    assert path == "text"
    digs = _stream_digests(ctx, seed, _sizes(case["files"], case["lo"], case["hi"]), "f")
    return dict(path=path, ctx=ctx, text="".join(d.to_string() for d in digs).encode())


# --------------------------------------------------------------------- run
def run(st):
    ctx, path = st["ctx"], st["path"]
    if path == "stream_one":
        d = ctx.digest_packed(st["data"], st["offs"], st["lens"], 0, ["file"], st["filters"])[0]
        return [st["filters"], d.bf_count, d.last_count]
    if path.endswith("_device"):
        counts = st["counts"]
        res = ctx.digest_device(st["data"].data_ptr(), st["offs"], st["lens"], st["dd"], st["filters"].data_ptr(), st["cap"],
                                counts.data_ptr() if counts is not None else None)
        out = _fields(res, len(st["lens"]))
        out["filters"] = st["filters"]
        if counts is not None:
            out["counts"] = counts
        return out
    if path.endswith("_host"):
        digs = ctx.digest_packed(st["data"], st["offs"], st["lens"], st["dd"], out_filters=st["filters"])
        out = {"filters": st["filters"], "bf_count": np.array([d.bf_count if d else 0 for d in digs], dtype=np.int64)}
        if st["dd"]:
            out["counts"] = np.concatenate([d.elem_counts for d in digs if d]).astype(np.int64)
        else:
            out["last_count"] = np.array([d.last_count if d else 0 for d in digs], dtype=np.int64)
        return out
    if path == "all_pairs":
        if st["where"] == "host":
            return ctx.compare_all(st["set"])
        ctx.compare_all_device(st["set"], st["scores"].data_ptr())
        return st["scores"]
    if path == "queries":
        if st["each_new"]:
            return ctx.compare_to(ctx.upload(st["queries"]), st["target"])
        ctx.compare_to_device(st["queries"], st["target"], st["scores"].data_ptr())
        return st["scores"]
    return ctx.compare_all(ctx.load_text(st["text"]))


# -------------------------------------------------------------------- work
def _pair_work(filters_a, filters_b, pairs, scores):
    """Filters read once, scores written once; a filter pair is 2,048 ANDed and counted bits."""
    return {"bytes": 256 * (filters_a + filters_b) + 4 * scores, "flops": 2 * 2048 * pairs}


def work(case):
    path = case["path"]
    if path == "stream_one":
        return {"bytes": case["bytes"] * (1 + 256 / STREAM_FILTER), "flops": 0}
    if path.startswith("stream"):
        return {"bytes": float(_sizes(case["files"], case["lo"], case["hi"]).sum()) * (1 + 256 / STREAM_FILTER), "flops": 0}
    if path.startswith("block"):
        return {"bytes": float(_sizes(case["files"], case["lo"], case["hi"]).sum()) * (1 + 258 / BLOCK), "flops": 0}
    if path == "queries":
        q = float(np.ceil(_sizes(case["queries"], case["lo"], case["hi"]) / BLOCK).sum())
        t = case["segments"] * SEGMENT // BLOCK
        return _pair_work(q, t, q * t, case["queries"] * case["segments"])
    if path == "all_pairs":
        f = _sizes(case["digests"], case["lo"], case["hi"]).astype(np.float64)
    else:
        f = _sizes(case["files"], case["lo"], case["hi"]).astype(np.float64) / STREAM_FILTER
    n, pairs = len(f), (f.sum() ** 2 - (f * f).sum()) / 2
    w = _pair_work(f.sum(), 0, pairs, n * (n - 1) // 2)
    if path == "all_pairs" and case["fast"]:
        w["flops"] /= 4  # folded filters: 512 bits
    if path == "text":
        w["bytes"] += f.sum() * 256 * 4 / 3
    return w


def exact(case, seed):
    """Every output is a whole number or a byte, equal or wrong: no 64-bit value stands beside it."""
    return None
