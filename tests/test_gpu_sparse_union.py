"""The sparse grain-growth kernel (pf_sparse.cu) where its union and slot
tables can go wrong: unions below, at and above the 16 grains it keeps in
shared memory (above, the list-by-list path) within one block, lists longer
than the 4 items loaded at once, grains that only one neighbour has, empty
lists, axes of one and two cells, the appended order of fresh items.

Counts and indices in stored order exactly, values within 1e-12 relative, the
bounds of the model's other tests.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((40,), 30, 6, 4), ((1, 33), 12, 3, 4), ((2, 2), 16, 4, 3), ((9, 11), 30, 6, 3), ((13, 20), 17, 4, 3),
         ((5, 6, 7), 24, 3, 3), ((2, 1, 9), 30, 9, 2), ((70, 3), 16, 16, 3)]


@pytest.mark.parametrize("shape,grains,items,steps", CASES, ids=["%s-%d-%d" % ("x".join(map(str, s)), g, i) for s, g, i, _ in CASES])
def test_sparse_unions_against_oracle(gpu, oracle, shape, grains, items, steps):
    K = 32
    rng = np.random.default_rng(sum(shape) + grains)
    cells = int(np.prod(shape))
    cnt = rng.integers(0, items + 1, cells).astype(np.int32)
    idx = np.zeros((cells, K), np.int32)
    val = np.zeros((cells, K))
    for c in range(cells):
        idx[c, : cnt[c]] = rng.permutation(grains)[: cnt[c]] * 7 - 20
        val[c, : cnt[c]] = rng.random(cnt[c])
    cnt, idx, val = cnt.reshape(shape), idx.reshape(shape + (K,)), val.reshape(shape + (K,))
    d = gpu.make_desc(shape, K, np.float64, "sparse_gg")
    with gpu.Stepper(d) as s:
        s.sparse_upload(cnt, idx, val)
        s.step(steps)
        c1, i1, v1 = s.sparse_download()
    c2, i2, v2, _ = oracle.sparse_gg(cnt, idx, val, steps, 0.01, 1e-8)
    used = np.arange(K) < c2[..., None]
    assert np.array_equal(c1, c2)
    assert np.array_equal(i1[used], np.asarray(i2)[used])
    assert np.abs(v1 - v2)[used].max() <= 1e-12 * max(1.0, np.abs(v2[used]).max())


# grids whose warps take patches of four rows: row counts of one, two and three
# past a multiple of four, fewer rows than four, the smallest such grid
@pytest.mark.parametrize("shape", [(257, 257), (3, 22001), (66, 1001), (23, 7, 409), (40, 2, 821), (256, 256)],
                         ids=lambda s: "x".join(map(str, s)))
def test_sparse_bands_against_oracle(gpu, oracle, shape):
    K, grains, items, steps = 16, 9, 4, 3
    rng = np.random.default_rng(sum(shape))
    cells = int(np.prod(shape))
    cnt = rng.integers(0, items + 1, cells).astype(np.int32)
    used = np.arange(K) < cnt[:, None]
    idx = np.zeros((cells, K), np.int32)
    idx[:, :grains] = rng.random((cells, grains)).argsort(axis=1)
    idx[~used] = 0
    val = np.where(used, rng.random((cells, K)), 0.0)
    cnt, idx, val = cnt.reshape(shape), idx.reshape(shape + (K,)), val.reshape(shape + (K,))
    with gpu.Stepper(gpu.make_desc(shape, K, np.float64, "sparse_gg")) as s:
        s.sparse_upload(cnt, idx, val)
        s.step(steps)
        c1, i1, v1 = s.sparse_download()
    c2, i2, v2, _ = oracle.sparse_gg(cnt, idx, val, steps, 0.01, 1e-8)
    used = np.arange(K) < c2[..., None]
    assert np.array_equal(c1, c2)
    assert np.array_equal(i1[used], np.asarray(i2)[used])
    assert np.abs(v1 - v2)[used].max() <= 1e-12 * max(1.0, np.abs(v2[used]).max())
