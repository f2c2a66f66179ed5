"""What a device digest call writes of its output buffer: nothing behind the
stated capacity, whatever the batch needs, and an error then."""
import numpy as np
import pytest

from sdhash_gb300 import synth

pytestmark = pytest.mark.gpu

SENTINEL = 0xA5


def device_batch(sizes):
    import torch

    offs, total = synth.packed_layout(np.array(sizes, dtype=np.uint64))
    data = np.zeros(total, dtype=np.uint8)
    for k, (o, n) in enumerate(zip(offs, sizes)):
        data[int(o):int(o) + n] = synth.mixture_bytes(71, k, n)
    return torch.from_numpy(data).cuda(), offs


# one file and several through the packing, a file long enough for the linked
# commit, and groups of both kinds
@pytest.mark.parametrize("sizes", [[200_000], [90_000, 300_000, 700, 40_000], [4 << 20], [4 << 20, 100_000]])
@pytest.mark.parametrize("room", ["none", "one", "all but one", "all"])
def test_capacity_is_kept(ctx, sizes, room):
    import torch

    import sdhash_gb300 as g

    data, offs = device_batch(sizes)
    bound = ctx.capacity(np.array(sizes, dtype=np.uint64), 0)

    def call(cap):
        dst = torch.full((bound * 256,), SENTINEL, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        try:
            res = ctx.digest_device(data.data_ptr(), offs, np.array(sizes, dtype=np.uint64), 0, dst.data_ptr(), cap)
        except g.EngineError as e:
            res = e
        return res, dst.cpu().numpy()

    full, want = call(bound)
    need = sum(r.bf_count for r in full)
    assert need < bound
    cap = {"none": 0, "one": 1, "all but one": need - 1, "all": need}[room]
    res, got = call(cap)
    if cap < need:
        assert res.code == -5  # SDBFG_ERR_CAPACITY
    else:
        assert [(r.bf_count, r.last_count, r.filter_offset) for r in res] == \
            [(r.bf_count, r.last_count, r.filter_offset) for r in full]
        assert np.array_equal(got[:need * 256], want[:need * 256])
    assert (got[cap * 256:] == SENTINEL).all()


# mixture files whose last filter has fewer than 20 elements and is dropped
@pytest.mark.parametrize("n", [60_000, 77_770, 97_317, 102_648, 106_202, 116_864, 129_303, 161_289])
def test_dropped_last_filter_is_not_written(ctx, oracle, n):
    import torch

    raw = synth.mixture_bytes(72, n, n)
    want = oracle.digest("f", raw.tobytes(), 0)
    assert want.st.last_count == 160
    data = torch.from_numpy(raw).cuda()
    bound = ctx.capacity([n], 0)
    dst = torch.full((bound * 256,), SENTINEL, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    r = ctx.digest_device(data.data_ptr(), [0], [n], 0, dst.data_ptr(), bound)[0]
    got = dst.cpu().numpy()
    assert (r.bf_count, r.last_count) == (want.st.bf_count, want.st.last_count)
    assert got[:r.bf_count * 256].tobytes() == bytes(want.filters())
    assert (got[r.bf_count * 256:] == SENTINEL).all()
