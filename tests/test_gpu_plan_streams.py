"""A comparison plan made under one stream and run under another."""
import numpy as np
import pytest

from sdhash_gb300 import synth

pytestmark = pytest.mark.gpu


def test_plan_made_on_another_stream(ctx):
    import torch

    files = [synth.mixture_bytes(61, k, 20_000 + 9_000 * k) for k in range(12)]
    for k in range(1, 12, 2):
        files[k][:15_000] = files[k - 1][:15_000]
    digs = ctx.digest_buffers([f.tobytes() for f in files], [f"f{k}" for k in range(12)], 0)
    ds = ctx.upload(digs)
    ia, ib = np.triu_indices(12, 1)
    want = ctx.score_pairs(ds, ds, ia, ib)
    assert (want > 0).any()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    out = torch.zeros(len(want), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    try:
        with torch.cuda.stream(a):
            torch.cuda._sleep(20_000_000)  # the plan's tables wait behind this
        ctx.set_stream(a.cuda_stream)
        assert ctx.filter_pairs(ds) > 0
        ctx.set_stream(b.cuda_stream)
        ctx.compare_all_device(ds, out.data_ptr())
        b.synchronize()
        assert np.array_equal(out.cpu().numpy(), want)
    finally:
        ctx.set_stream(None)
        torch.cuda.synchronize()
