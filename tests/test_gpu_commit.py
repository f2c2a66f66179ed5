"""The ordered filter fill where its windows can go wrong: repeated content
at distances below, around and above a filter, a window and the big filter's
life, tiles without features between tiles with many, chunk ends inside a
window, inputs of a handful of features.  Digests equal the oracle's."""
import numpy as np
import pytest

from sdhash_gb300 import synth

pytestmark = pytest.mark.gpu


def periodic(period, n):
    return np.resize(synth.random_bytes(21, period, period), n)


def near_copies(n, block, back):
    """Random bytes in which every second block repeats the one `back` blocks earlier."""
    d = synth.random_bytes(22, block, n)
    for k in range(back | 1, n // block, 2):
        d[k * block:(k + 1) * block] = d[(k - back) * block:(k - back + 1) * block]
    return d


def gaps(n, step):
    """Mixture content with stretches of zeros (tiles without a feature)."""
    d = synth.mixture_bytes(23, step, n)
    for o in range(0, n, 2 * step):
        d[o:o + step] = 0
    return d


INPUTS = {
    "tiny": lambda: synth.mixture_bytes(24, 0, 512),
    "few_features": lambda: synth.random_bytes(24, 1, 3000),
    "one_window": lambda: synth.random_bytes(24, 2, 15100),
    "period_1500": lambda: periodic(1500, 1 << 20),
    "period_12600": lambda: periodic(12600, 1 << 20),
    "period_15200": lambda: periodic(15200, 3 << 20),
    "period_650k": lambda: periodic(650_000, 4 << 20),
    "period_720k": lambda: periodic(720_001, 4 << 20),
    "near_copies_700": lambda: near_copies(1 << 20, 700, 1),
    "near_copies_13k": lambda: near_copies(4 << 20, 13_000, 3),
    "gaps_40k": lambda: gaps(2 << 20, 40_000),
    "gaps_3m": lambda: gaps(24 << 20, 3 << 20),
    "zeros": lambda: np.zeros(300_000, dtype=np.uint8),
    "chunk_end": lambda: synth.mixture_bytes(25, 0, (32 << 20) + 70_001),
    "two_chunk_ends": lambda: periodic(5_000_011, (64 << 20) + 63),
}


@pytest.mark.parametrize("name", list(INPUTS))
def test_windows_against_oracle(ctx, oracle, name):
    data = INPUTS[name]().tobytes()
    got = ctx.digest_buffers([data], [name], 0)[0]
    assert got.to_string() == oracle.digest(name, data, 0).to_string()


def test_many_files_per_cta(ctx, oracle):
    """More files than resident CTAs: a CTA's shared state passes from file to file."""
    sizes = [600 + 37 * k for k in range(3000)]
    data = [synth.mixture_bytes(26, k, n).tobytes() for k, n in enumerate(sizes)]
    names = [f"m{k}" for k in range(len(sizes))]
    got = ctx.digest_buffers(data, names, 0)
    for k in range(0, len(sizes), 11):
        assert got[k].to_string() == oracle.digest(names[k], data[k], 0).to_string(), names[k]
