"""Stream digests of small batches: sizes on both sides of every choice of
positions per ranking thread, one file (filters written in place) and several,
links that fail inside a group whose tiles are all resident.  Digests equal
the oracle's."""
import numpy as np
import pytest

from sdhash_gb300 import synth

pytestmark = pytest.mark.gpu

# ends of stretches (128 threads x 24, 40, 72 positions), of tiles, of the
# ranges in which a choice is taken on 148 to 152 SMs, and of a chunk
SIZES = [512, 513, 575, 3072, 3079, 5120, 5121, 8191, 8257, 9216, 65547, 1 << 20, (1 << 20) + 9, 1_400_003, 2_334_721,
         4_202_496, 8_871_937, 18_210_817, (32 << 20) + 8]


@pytest.mark.parametrize("n", SIZES)
def test_one_file(ctx, oracle, n):
    data = synth.mixture_bytes(31, n, n).tobytes()
    got = ctx.digest_buffers([data], ["f"], 0)[0]
    assert got.to_string() == oracle.digest("f", data, 0).to_string()


@pytest.mark.parametrize("lead", [0, 16])
@pytest.mark.parametrize("sizes", [[65_547], [1_000_003], [4096, 700, 300_001, 65_536, 1, 2_000_000]])
def test_failing_links(ctx, oracle, sizes, lead):
    files = [synth.mixture_bytes(32, k, n).tobytes() for k, n in enumerate(sizes)]
    names = [f"f{k}" for k in range(len(files))]
    before = ctx.relinked_tiles
    ctx.set_lead(lead)
    try:
        got = ctx.digest_buffers(files, names, 0)
    finally:
        ctx.set_lead(64)  # the default
    if lead == 0:
        assert ctx.relinked_tiles > before
    for k, f in enumerate(files):
        if len(f) >= 512:
            assert got[k].to_string() == oracle.digest(names[k], f, 0).to_string()


def test_one_file_in_place_and_packed(ctx):
    """A device output as large as the file's bound takes the filters in
    place, a smaller one takes them packed: the same bytes."""
    import torch

    n = 700_001
    data = torch.from_numpy(synth.mixture_bytes(33, 0, n)).cuda()
    bound = ctx.capacity([n], 0)
    out = []
    for cap in (bound, bound - 1):
        dst = torch.zeros(bound * 256, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        r = ctx.digest_device(data.data_ptr(), [0], [n], 0, dst.data_ptr(), cap)[0]
        out.append((r.bf_count, r.last_count, r.filter_offset, dst[:r.bf_count * 256].cpu().numpy()))
    assert out[0][:3] == out[1][:3] and out[0][0] > 1
    assert np.array_equal(out[0][3], out[1][3])
