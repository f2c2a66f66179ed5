"""Block batches on both sides of the number of blocks from which their ranks are
computed ahead (two per SM): the same inputs, few and many at a time, have the
oracle's digests."""
import numpy as np
import pytest

from sdhash_gb300 import synth

pytestmark = pytest.mark.gpu

SIZES = [512, 520, 1000, 1028, 4096, 8192, 8256, 8257, 8264, 8320, 12_345, 16_376, 16_384]


def content(seed, n):
    """Mixture content with stretches of zeros and of one short period."""
    d = synth.mixture_bytes(seed, 1, n)
    for k, o in enumerate(range(0, n, 30_000)):
        m = min(7_000, n - o)
        if k % 3 == 1:
            d[o:o + m] = 0
        elif k % 3 == 2:
            d[o:o + m] = np.resize(np.arange(97, 160, dtype=np.uint8), m)
    return d


@pytest.mark.parametrize("dd", SIZES)
def test_few_and_many_blocks(ctx, oracle, dd):
    import torch

    line = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    kinds = [content(91, n).tobytes() for n in (512, dd, dd + 511, dd + 512, 3 * dd - 1, 5 * dd + 701)]
    want = [oracle.digest("f", f, dd).to_string() for f in kinds]
    per = sum(len(f) // dd + (len(f) % dd >= 512) for f in kinds)
    for times in (1, line // per, line // per + 1, 2 * line // per):
        for extra in (0, 1):  # (a batch of exactly the line, and one block more, where the counts allow it)
            files = kinds * times + [kinds[1]] * (line + extra - per * times if 0 < line - per * times < per else 0)
            got = ctx.digest_buffers(files, ["f"] * len(files), dd)
            for k, d in enumerate(got):
                assert d.to_string() == (want[k % 6] if k < 6 * times else want[1]), (dd, times, extra, k)
