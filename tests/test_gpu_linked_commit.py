"""The commit of long files through links: the last holders of filter bits
across blocks of 1,024 features, filters that stay open for thousands of
features, the big filter's life, chunk ends, stretches of tiles without
features, batches that mix long files with short ones.  Digests equal the
oracle's."""
import numpy as np
import pytest

from sdhash_gb300 import synth

pytestmark = pytest.mark.gpu


def open_filter(n):
    """A filter left half full, then 3 MB that repeat what it already holds, then new content."""
    d = synth.random_bytes(61, 0, n)
    a = 9_000
    m = min(n, 3_000_000) - a
    d[a:a + m] = np.resize(d[:a], m)
    return d


def copies(n, block, back):
    """Every third block repeats the one `back` blocks earlier."""
    d = synth.mixture_bytes(62, block, n)
    for k in range(back, n // block, 3):
        d[k * block:(k + 1) * block] = d[(k - back) * block:(k - back + 1) * block]
    return d


def sparse(n):
    """Features in a few places only."""
    d = np.zeros(n, dtype=np.uint8)
    for o in (0, 70_000, 2_000_000, n - 50_000):
        d[o:o + 40_000] = synth.random_bytes(63, o, 40_000)
    return d


INPUTS = {
    "random": lambda: synth.random_bytes(64, 0, 5_000_003),
    "mixture": lambda: synth.mixture_bytes(64, 0, 3_100_000),
    "open_filter": lambda: open_filter(4_500_000),
    "period_77k": lambda: np.resize(synth.random_bytes(64, 1, 77_003), 4_000_000),
    "period_13k": lambda: np.resize(synth.random_bytes(64, 2, 13_001), 3_500_000),
    "period_300": lambda: np.resize(synth.random_bytes(64, 3, 300), 3_500_000),
    "copies_2k": lambda: copies(4_000_000, 2_000, 1),
    "copies_15k": lambda: copies(4_000_000, 15_000, 7),
    "copies_700k": lambda: copies(9_000_000, 700_000, 2),
    "sparse": lambda: sparse(8_000_000),
    "zeros": lambda: np.zeros(4_000_000, dtype=np.uint8),
    "chunks": lambda: synth.mixture_bytes(65, 0, (64 << 20) + 20),
    "copied_chunk": lambda: np.resize(synth.random_bytes(66, 0, (32 << 20) + 1_000), (64 << 20) + 300_000),
}


@pytest.mark.parametrize("name", list(INPUTS))
def test_one_file(ctx, oracle, name):
    data = INPUTS[name]().tobytes()
    got = ctx.digest_buffers([data], [name], 0)[0]
    assert got.to_string() == oracle.digest(name, data, 0).to_string()


@pytest.mark.parametrize("names", [["copied_chunk"], ["chunks", "sparse", "open_filter"], ["random", "sparse", "copies_15k"]])
def test_mixed_batch(ctx, oracle, names):
    files = [INPUTS[n]().tobytes() for n in names]
    short = [synth.mixture_bytes(67, k, 100 + 977 * k).tobytes() for k in range(60)]
    order = short[:20] + files[:1] + short[20:40] + files[1:] + short[40:]
    got = ctx.digest_buffers(order, [f"f{k}" for k in range(len(order))], 0)
    for k, f in enumerate(order):
        if len(f) >= 512:
            assert got[k].to_string() == oracle.digest(f"f{k}", f, 0).to_string(), k
        else:
            assert got[k] is None
