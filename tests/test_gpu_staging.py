"""Host inputs at every alignment and spacing, from pageable and from pinned
memory, in batches that the device gathers itself."""
import numpy as np
import pytest

from sdhash_gb300 import synth

pytestmark = pytest.mark.gpu

SIZES = [512, 513, 527, 528, 543, 544, 560, 1000, 4096, 4097, 31_744 + 61, 70_001, 130_000, 511, 16]


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("dd", [0, 2048])
@pytest.mark.parametrize("shift", [0, 1, 2, 3, 4, 6, 8, 11, 12, 15])
def test_gathered_inputs(ctx, oracle, shift, dd, pinned):
    import torch

    offs, at = [], 32 + shift
    for k, n in enumerate(SIZES):
        offs.append(at)
        at += n + (0 if k % 3 else 16 - n % 16)  # some follow at once, some keep the alignment
    buf = torch.empty(at + 32, dtype=torch.uint8, pin_memory=pinned).numpy()
    buf[:] = synth.mixture_bytes(51, shift, len(buf))
    names = [f"f{k}" for k in range(len(SIZES))]
    got = ctx.digest_packed(buf, np.array(offs), np.array(SIZES), dd, names)
    for k, (o, n) in enumerate(zip(offs, SIZES)):
        if n < 512:
            assert got[k] is None
            continue
        assert got[k].to_string() == oracle.digest(names[k], buf[o:o + n].tobytes(), dd).to_string(), (shift, n)


@pytest.mark.parametrize("shift,dd", [(0, 16_384), (5, 16_384), (0, 1028), (3, 1029)])
def test_block_slabs_from_host(ctx, shift, dd):
    """A host batch of several slabs has the filters of its inputs one by one."""
    rng = np.random.default_rng(52)
    lens = rng.integers(400, 3 << 20, 60).astype(np.uint64)
    lens[7] = 40 << 20
    offs = np.concatenate([[0], np.cumsum(lens[:-1] + 3)]).astype(np.uint64) + np.uint64(shift)
    buf = np.resize(synth.mixture_bytes(53, 0, 9_000_011), int(offs[-1] + lens[-1]))
    got = ctx.digest_packed(buf, offs, lens, dd)
    for k in range(len(lens)):
        one = ctx.digest_buffers([buf[int(offs[k]):int(offs[k] + lens[k])].tobytes()], [f"f{k}"], dd)[0]
        assert (got[k] is None) == (one is None)
        if one is not None:
            assert np.array_equal(got[k].filters, one.filters) and np.array_equal(got[k].elem_counts, one.elem_counts)


def test_file_backed_inputs(ctx, oracle, tmp_path):
    """Inputs in a mapped file, as a caller that maps its files passes them."""
    lens = [70_001, 513, 300_000]
    offs = [7, 80_000, 100_003]
    raw = synth.mixture_bytes(54, 0, 420_000)
    raw.tofile(tmp_path / "in.bin")
    buf = np.memmap(tmp_path / "in.bin", dtype=np.uint8, mode="r")
    for dd in (0, 4096):
        got = ctx.digest_packed(buf, np.array(offs), np.array(lens), dd, ["a", "b", "c"])
        for k in range(3):
            want = oracle.digest("abc"[k], raw[offs[k]:offs[k] + lens[k]].tobytes(), dd)
            assert got[k].to_string() == want.to_string()
