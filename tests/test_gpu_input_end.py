"""Host inputs that end with their mapping: nothing behind them is read."""
import ctypes
import mmap

import numpy as np
import pytest

from sdhash_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dd", [0, 4096])
@pytest.mark.parametrize("n", [512, 1001, 70_001, 1 << 20])
def test_input_ends_with_its_mapping(ctx, oracle, n, dd):
    page = mmap.PAGESIZE
    size = (n + page - 1) // page * page
    area = mmap.mmap(-1, size + page)
    raw = synth.mixture_bytes(73, n, n)
    buf = np.frombuffer(area, dtype=np.uint8)[size - n:size]
    buf[:] = raw
    libc = ctypes.CDLL(None, use_errno=True)
    libc.mprotect.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int]
    behind = buf.ctypes.data + n
    assert behind % page == 0 and libc.mprotect(behind, page, 0) == 0
    try:
        got = ctx.digest_packed(buf, [0], [n], dd, ["f"])[0]
    finally:
        assert libc.mprotect(behind, page, 3) == 0
    assert got.to_string() == oracle.digest("f", raw.tobytes(), dd).to_string()
