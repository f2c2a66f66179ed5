"""Block mode with ranks computed ahead: block sizes on both sides of one
walked tile (8,256 bytes) and of 8-byte alignment, tails of every kind, inputs
past one run of ranks (32 MiB) and past one slab (256 MiB)."""
import numpy as np
import pytest

from sdhash_gb300 import synth

pytestmark = pytest.mark.gpu

SIZES = [512, 520, 1000, 1028, 4096, 8192, 8256, 8257, 8264, 8320, 12_345, 16_376, 16_383, 16_384]


def mixed(seed, n):
    """Mixture content with runs of zeros, of one short period and of random bytes."""
    d = synth.mixture_bytes(seed, 0, n)
    for k, o in enumerate(range(0, n, 50_000)):
        m = min(9_000, n - o)
        if k % 4 == 1:
            d[o:o + m] = 0
        elif k % 4 == 2:
            d[o:o + m] = np.resize(np.arange(97, 160, dtype=np.uint8), m)
        elif k % 4 == 3:
            d[o:o + m] = synth.random_bytes(seed, k, m)
    return d


@pytest.mark.parametrize("dd", SIZES)
def test_block_sizes(ctx, oracle, dd):
    files = [mixed(41, n).tobytes() for n in (512, dd, dd + 511, dd + 512, 3 * dd - 1, 400_003, 5 * dd + 701)]
    names = [f"f{k}" for k in range(len(files))]
    got = ctx.digest_buffers(files, names, dd)
    for k, f in enumerate(files):
        assert got[k].to_string() == oracle.digest(names[k], f, dd).to_string(), (dd, len(f))


def crowded(n):
    """Content whose blocks select more than 192 positions, many of equal score."""
    d = synth.random_bytes(44, 0, n)
    for k, o in enumerate(range(0, n, 40_000)):
        m = min(30_000, n - o)
        d[o:o + m] = np.resize(synth.random_bytes(45, k, 65 + 37 * k), m)
    return d


CONTENT = {
    "random": lambda: synth.random_bytes(46, 0, 600_007),
    "random_low": lambda: synth.random_bytes(46, 1, 600_007) & 0x3F,
    "periods": lambda: crowded(1_000_003),
    "ramps": lambda: (np.arange(500_001) // 3 % 251).astype(np.uint8),
    "zeros": lambda: np.zeros(100_000, dtype=np.uint8),
}


@pytest.mark.parametrize("dd", [16_384, 16_379, 4096, 2048, 512])
@pytest.mark.parametrize("name", list(CONTENT))
def test_selection(ctx, oracle, name, dd):
    """The threshold, its allowance and the 192nd element of a block."""
    data = CONTENT[name]().tobytes()
    got = ctx.digest_buffers([data], [name], dd)[0]
    assert got.to_string() == oracle.digest(name, data, dd).to_string()


@pytest.mark.parametrize("lead", [0, 128])
@pytest.mark.parametrize("dd", [8264, 16_384])
def test_leads(ctx, oracle, dd, lead):
    data = mixed(42, 700_001).tobytes()
    ctx.set_lead(lead)
    try:
        got = ctx.digest_buffers([data], ["f"], dd)[0]
    finally:
        ctx.set_lead(64)  # the default
    assert got.to_string() == oracle.digest("f", data, dd).to_string()


@pytest.mark.parametrize("dd", [16_384, 5_000, 8_200])
def test_long_input_equals_its_pieces(ctx, dd):
    """Blocks are independent: a 300 MB input's filters are those of its pieces."""
    import torch

    n = 300_000_000 // dd * dd + 4_000
    piece = 37_000_000 // (2 * dd) * (2 * dd)
    data = torch.from_numpy(np.resize(mixed(43, 7_000_003), n)).cuda()

    def digest(o, m):
        cap = ctx.capacity([m], dd)
        out = torch.zeros(cap * 256, dtype=torch.uint8, device="cuda")
        cnt = torch.zeros(cap, dtype=torch.uint16, device="cuda")
        torch.cuda.synchronize()
        r = ctx.digest_device(data.data_ptr() + o, [0], [m], dd, out.data_ptr(), cap, cnt.data_ptr())[0]
        return out[:256 * r.bf_count].cpu().numpy(), cnt[:r.bf_count].cpu().numpy()

    whole, counts = digest(0, n)
    parts = [digest(o, min(piece, n - o)) for o in range(0, n, piece)]
    assert np.array_equal(whole, np.concatenate([p[0] for p in parts]))
    assert np.array_equal(counts, np.concatenate([p[1] for p in parts]))
    assert counts.max() > 16
