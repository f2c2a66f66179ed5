"""What a Digest of a batch keeps alive: with a caller's output buffer a copy of
its own filters and a bounded number of its neighbours', never the buffer (the
library call is replaced, no GPU)."""
import ctypes as C

import numpy as np
import pytest


@pytest.mark.parametrize("dd", [0, 16384])
@pytest.mark.parametrize("count", [1, 3, 40, 3000])
def test_digest_keeps_a_bounded_array(native, monkeypatch, dd, count):
    import sdhash_gb300 as g

    rng = np.random.default_rng(count)
    lens = rng.integers(300, 400_000, count).astype(np.uint64)
    lens[0] = 40 << 20
    lens[count // 2] = 400 << 20  # more filters than are ever shared
    ok = lens >= 512
    per = np.where(ok, np.maximum(1, lens // 16384), 0).astype(np.int64)
    order = np.arange(count) if dd else np.argsort(-lens.astype(np.int64), kind="stable")
    offs = np.zeros(count, dtype=np.int64)
    offs[order] = np.cumsum(per[order]) - per[order]
    total = int(per.sum())
    want = rng.integers(0, 256, total * 256, dtype=np.uint8)
    want_counts = rng.integers(0, 193, total).astype(np.uint16)

    class Library:
        sdbfg_digest_capacity = native.sdbfg_digest_capacity

        @staticmethod
        def sdbfg_digest_batch(h, data, o, n_lens, n, block, out_filters, cap, out_counts, res):
            assert total <= cap
            C.memmove(out_filters, want.ctypes.data, want.nbytes)
            if block:
                C.memmove(out_counts, want_counts.ctypes.data, want_counts.nbytes)
            for i in range(n):
                res[i].status = 0 if ok[i] else -3
                res[i].bf_count, res[i].filter_offset, res[i].last_count = int(per[i]), int(offs[i]), 17
            return 0

    monkeypatch.setattr(g, "lib", lambda: Library)
    monkeypatch.setattr(g, "_SHARED_FILTERS", 1 << 14, raising=False)
    ctx = g.Context.__new__(g.Context)
    ctx.h = None
    buf = np.zeros(g.Context.capacity(lens, dd) * 256, dtype=np.uint8)
    data = np.zeros(16, dtype=np.uint8)
    digs = ctx.digest_packed(data, np.zeros(count, dtype=np.uint64), lens, dd, out_filters=buf)
    buf[:] = 0xEE  # the caller's again
    most = 4 << 20
    for i, d in enumerate(digs):
        assert (d is not None) == bool(ok[i])
        if d is None:
            continue
        a, b = int(offs[i]), int(offs[i] + per[i])
        assert np.array_equal(d.filters, want[a * 256:b * 256]) and d.bf_count == b - a
        held = d.filters if d.filters.base is None else d.filters.base
        assert held.nbytes <= max(2 * most, d.filters.nbytes)
        if dd:
            assert np.array_equal(d.elem_counts, want_counts[a:b])
            held = d.elem_counts if d.elem_counts.base is None else d.elem_counts.base
            assert held.nbytes * 128 <= max(2 * most, d.filters.nbytes)


def test_no_digest(native, monkeypatch):
    import sdhash_gb300 as g

    class Library:
        sdbfg_digest_capacity = native.sdbfg_digest_capacity

        @staticmethod
        def sdbfg_digest_batch(h, data, o, lens, n, block, out_filters, cap, out_counts, res):
            for i in range(n):
                res[i].status = -3
            return 0

    monkeypatch.setattr(g, "lib", lambda: Library)
    ctx = g.Context.__new__(g.Context)
    ctx.h = None
    for n in (0, 3):
        for out in (None, np.zeros(0, dtype=np.uint8), np.zeros(512, dtype=np.uint8)):
            assert ctx.digest_packed(np.zeros(16, np.uint8), [0] * n, [100] * n, 0, out_filters=out) == [None] * n
