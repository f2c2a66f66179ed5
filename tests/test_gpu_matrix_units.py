"""The tensor-core comparison where its units and sums can go wrong: pairs cut
by target filters and by rows, groups against cut targets, tile edges, digests
of sparse filters, scores on exact halves (left to the ordered sum in double
precision) and more of them than the list of such pairs holds, folded
digests against unfolded ones.  Scores equal the one-CTA-per-pair path's,
which the other tests hold to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits_to_bytes(idx):
    b = np.zeros(2048, dtype=np.uint8)
    b[idx] = 1
    return np.packbits(b, bitorder="little")


def random_digest(g, rng, name, n, elems=None, pool=None, ham=660):
    """n filters of about `ham` bits, every fourth one taken from the pool with some bits changed."""
    f = np.zeros((n, 256), dtype=np.uint8)
    for i in range(n):
        if pool is not None and len(pool) and i % 4 == 1:
            f[i] = pool[int(rng.integers(len(pool)))] & rng.integers(64, 256, 256, dtype=np.uint8)
        else:
            f[i] = bits_to_bytes(rng.choice(2048, size=max(1, int(rng.normal(ham, 20))), replace=False))
    if elems is None:
        elems = np.where(rng.random(n) < 0.85, 192, rng.integers(0, 193, n))
    return g.Digest(name, 0, n, 0, 192, 16384, f.reshape(-1), np.asarray(elems, dtype=np.uint16))


def pairwise(ctx, q, t, nq, nt):
    ia, ib = np.meshgrid(np.arange(nq), np.arange(nt), indexing="ij")
    return ctx.score_pairs(q, t, ia.reshape(-1), ib.reshape(-1)).reshape(nq, nt)


@pytest.mark.parametrize("nq,nt", [([1], [3000]), ([38], [191, 192, 193, 2000]), ([5, 40, 83, 1], [2500, 384]),
                                   ([200], [1500]), ([129, 128, 127, 300], [128, 257, 1]), ([700], [650, 900])])
def test_cut_pairs_and_groups(ctx, nq, nt):
    import sdhash_gb300 as g
    rng = np.random.default_rng(sum(nq) + 7 * sum(nt))
    pool = np.stack([bits_to_bytes(rng.choice(2048, size=660, replace=False)) for _ in range(12)])
    qs = [random_digest(g, rng, f"q{i}", n, pool=pool) for i, n in enumerate(nq)]
    ts = [random_digest(g, rng, f"t{i}", n, pool=pool) for i, n in enumerate(nt)]
    q, t = ctx.upload(qs), ctx.upload(ts)
    want = pairwise(ctx, q, t, len(nq), len(nt))
    assert (want > 0).any()
    assert np.array_equal(ctx.compare_to(q, t), want)
    for work in (1, 1 << 16, 1 << 24):  # every pair cut into single tiles, ..., not at all
        ctx.set_compare_tuning(5, work, True)
        try:
            assert np.array_equal(ctx.compare_to(q, t), want), work
        finally:
            ctx.set_compare_tuning(5, 1 << 22, True)


def test_sparse_digests(ctx):
    """Digests without a filter of 16 elements, or whose last filter has none, on both sides."""
    import sdhash_gb300 as g
    rng = np.random.default_rng(3)
    ds = []
    for i, elems in enumerate([[3], [15], [16], [0, 0, 5], [160, 3], [3, 160], [15] * 20, [16] * 20, [160] * 30 + [2],
                               [2] + [160] * 30, [192] * 200, [7] * 150]):
        ds.append(random_digest(g, rng, f"s{i:02d}", len(elems), elems))
    dev, n = ctx.upload(ds), len(ds)
    iu = np.triu_indices(n, 1)
    assert np.array_equal(ctx.compare_all(dev), ctx.score_pairs(dev, dev, iu[0], iu[1]))


@pytest.mark.parametrize("n", [12, 100])
def test_exact_halves(ctx, oracle, n):
    """Single filters of 440 bits and 160 elements (cut 240): an overlap of 240 + k scores k / 2,
    a half for odd k; n = 100 has 9,900 such pairs."""
    import sdhash_gb300 as g
    rng = np.random.default_rng(n)
    perm = rng.permutation(2048)
    qs, ts = [], []
    for i in range(n):
        qs.append(g.Digest(f"q{i:03d}", 0, 1, 160, 160, 0, bits_to_bytes(perm[:440]), None))
        k = 2 * int(rng.integers(0, 99)) + 1
        own = perm[:240 + k]
        rest = rng.choice(perm[440:], size=200 - k, replace=False)
        ts.append(g.Digest(f"t{i:03d}", 0, 1, 160, 160, 0, bits_to_bytes(np.concatenate([own, rest])), None))
    q, t = ctx.upload(qs), ctx.upload(ts)
    got = ctx.compare_to(q, t)
    assert np.array_equal(got, pairwise(ctx, q, t, n, n))
    oq, ot = [oracle.parse(d.to_string()) for d in qs[:3]], [oracle.parse(d.to_string()) for d in ts]
    for i, a in enumerate(oq):
        assert [oracle.score(a, b) for b in ot] == list(got[i])


def test_folded_against_unfolded(ctx):
    """Folded queries, unfolded targets on either side of the swap rule: ratios
    above 1 and wrapped weights."""
    import sdhash_gb300 as g
    rng = np.random.default_rng(5)
    pool = np.stack([bits_to_bytes(rng.choice(2048, size=660, replace=False)) for _ in range(4)])
    qs = [random_digest(g, rng, f"q{i}", n, pool=pool, ham=300).fast() for i, n in enumerate([3, 20, 150, 260])]
    ts = [random_digest(g, rng, f"t{i}", n, pool=pool) for i, n in enumerate([1, 10, 64, 200, 400])]
    for d in ts:  # some target filters inside the folded ones' untouched bytes
        f = d.filters.reshape(-1, 256)
        for i in range(0, len(f), 3):
            f[i] = qs[i % 4].filters.reshape(-1, 256)[i % qs[i % 4].bf_count]
    q, t = ctx.upload(qs), ctx.upload(ts)
    assert np.array_equal(ctx.compare_to(q, t), pairwise(ctx, q, t, len(qs), len(ts)))


def test_repeated_runs_agree(ctx):
    """The roles of the tensor-core kernel hand each other a row's maximum while
    it changes: forty runs of targets of many tiles give the CUDA-core kernel's scores."""
    import sdhash_gb300 as g
    rng = np.random.default_rng(11)
    pool = np.stack([bits_to_bytes(rng.choice(2048, size=660, replace=False)) for _ in range(20)])
    counts = np.rint(np.exp(rng.uniform(0, np.log(900), 70))).astype(int)
    ds = [random_digest(g, rng, f"r{i:02d}", int(n), np.r_[np.full(int(n) - 1, 192), 40], pool) for i, n in enumerate(counts)]
    dev = ctx.upload(ds)
    ctx.set_compare_tuning(0, 1 << 22, False)
    try:
        want = ctx.compare_all(dev)
    finally:
        ctx.set_compare_tuning(5, 1 << 22, True)
    for k in range(40):
        assert np.array_equal(ctx.compare_all(dev), want), k


@pytest.mark.parametrize("counts", [list(range(1, 60)), [1] * 100 + [2] * 30 + [3] * 3 + [900], [5, 5, 6, 6, 6, 7, 127, 128, 129, 400],
                                    [60, 64, 64, 65, 2000], [1, 2, 3], [40] * 5 + [41] * 5 + [1500] * 2])
@pytest.mark.parametrize("folded", [False, True])
def test_bundles_of_small_digests(ctx, counts, folded):
    """All pairs of digests whose small ones share passes: every pair scored
    once, in the swap rule's order, classes of equal counts and folded digests among them."""
    import sdhash_gb300 as g
    rng = np.random.default_rng(len(counts) + sum(counts))
    pool = np.stack([bits_to_bytes(rng.choice(2048, size=660, replace=False)) for _ in range(12)])
    order = rng.permutation(len(counts))
    ds = [random_digest(g, rng, f"d{i:03d}", counts[k], pool=pool) for i, k in enumerate(order)]
    if folded:
        ds = [d.fast() if i % 3 == 1 else d for i, d in enumerate(ds)]
    s = ctx.upload(ds)
    i, j = np.triu_indices(len(ds), 1)
    want = ctx.score_pairs(s, s, i, j)
    assert (want > 0).any()
    assert np.array_equal(ctx.compare_all(s), want)
