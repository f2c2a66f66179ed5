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
