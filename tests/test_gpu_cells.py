"""Counting and cell clustering at the sizes where they can go wrong: tiles of
0, 1 and 2 query slots, ragged last words, tiles tested lane = candidate and
lane = query, words settled by their boxes, more minpts of one epsilon than
one pass of the clustering takes, sparse and dense cells.  Labels and table
hashes must equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1


@pytest.fixture(scope="module")
def vdb():
    import variantdbscan_gb300 as v
    from variantdbscan_gb300 import build
    build.build()
    return v


@pytest.fixture(scope="module")
def ctx(vdb):
    c = vdb.Context()
    yield c
    c.close()


def _check(ctx, vdb, orc, x, y, eps, mp, mbb=70, **kw):
    want = orc.variants(x, y, eps, mp, mbb)
    out, st = ctx.run([vdb.BatchItem(x, y, eps, mp, mbb)], table_hash=True, **kw)
    np.testing.assert_array_equal(out[0], want)
    assert st["table_hash"] == sum(orc.table_hash(x, y, e, mbb) for e in np.unique(eps)) & M64
    assert st["clusters"] == int(want.max(axis=1).sum())
    out, _ = ctx.run([vdb.BatchItem(x, y, eps, mp, mbb)], table="border", **kw)
    np.testing.assert_array_equal(out[0], want)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [2, 15, 16, 17, 31, 33, 63, 65, 129, 1025, 4099])
def test_ragged_sizes(ctx, vdb, orc, n, precision):
    rng = np.random.default_rng(n)
    x, y = rng.uniform(0, 2, n), rng.uniform(0, 1, n)
    # one epsilon with 11 minpts (two passes of the clustering), one repeated
    eps = np.array([0.4] * 12 + [0.05, 0.05, 1.7])
    mp = np.array([1, 2, 3, 5, 8, 13, 21, 34, 55, 144, 500, 3, 2, 4, 30], np.uint32)
    _check(ctx, vdb, orc, x, y, eps, mp, precision=precision)


@pytest.mark.parametrize("lattice", [False, True])
@pytest.mark.parametrize("n", [32768, 40007])
def test_words_settled_by_their_boxes(ctx, vdb, orc, n, lattice):
    # hundreds of points per cell: most words lie inside or outside eps of a
    # whole tile; on the lattice many pairs are exactly eps apart
    rng = np.random.default_rng(n)
    x, y = rng.uniform(0, 3, n), rng.uniform(0, 2, n)
    x[: n // 8] = rng.normal(1.0, 0.05, n // 8)
    if lattice:
        x, y = np.rint(x * 50) / 50, np.rint(y * 50) / 50
    _check(ctx, vdb, orc, x, y, np.array([0.5, 0.2, 0.2]), np.array([50, 20, 400], np.uint32))


def test_sparse_cells_over_a_wide_box(ctx, vdb, orc):
    # a row directory instead of a dense cell array, cells of one point
    rng = np.random.default_rng(8)
    x, y = rng.uniform(0, 3000, 20000), rng.uniform(0, 3000, 20000)
    x[:6000] = rng.normal(700, 2, 6000)
    y[:6000] = rng.normal(700, 2, 6000)
    _check(ctx, vdb, orc, x, y, np.array([0.3, 0.3, 5.0]), np.array([4, 12, 3], np.uint32))


@pytest.mark.parametrize("entry_bytes", [2, 4])
@pytest.mark.parametrize("share", [1, 2, 3, 300])
def test_row_chunks_of_a_budget(ctx, vdb, orc, share, entry_bytes):
    # 2 chunks up to hundreds (more than one plan holds), and rows of a tile
    # that do not fit a chunk
    rng = np.random.default_rng(5)
    n = 40011
    x, y = rng.uniform(0, 40, n), rng.uniform(0, 40, n)
    eps, mp = np.array([0.4, 0.4]), np.array([9, 14], np.uint32)
    kw = dict(entry_bytes=entry_bytes, table_hash=True)
    item = vdb.BatchItem(x, y, eps, mp, 70)
    whole, sw = ctx.run([item], **kw)
    np.testing.assert_array_equal(whole[0], orc.variants(x, y, eps, mp, 70))
    out, st = ctx.run([item], budget=(sw["entry_bytes"] - 1) // share, **kw)
    np.testing.assert_array_equal(out[0], whole[0])
    assert st["table_hash"] == sw["table_hash"] == orc.table_hash(x, y, 0.4, 70) & M64
    assert st["table_chunks"] > share
    with pytest.raises(vdb.VDBError) as e:
        ctx.run([item], budget=2, **kw)
    assert e.value.code == -4  # no memory: the rows of one tile exceed the budget


@pytest.mark.parametrize("shift", [-9.0, -1.0, 0.0])
@pytest.mark.parametrize("n", [1, 33, 255, 257, 1025, 70001])
def test_boxes_of_signed_coordinates(ctx, vdb, orc, n, shift):
    # negative coordinates only, of both signs, and zeros of both signs; the
    # box's corners are the last points
    rng = np.random.default_rng(n)
    x, y = rng.uniform(0, 2, n) + shift, rng.uniform(0, 1, n) + shift
    x[: n // 4], y[n // 4 : n // 3] = 0.0, -0.0
    x[-1], y[-1] = 2.5 + shift, 1.5 + shift
    x[n // 2], y[n // 2] = shift - 0.5, shift - 0.5
    eps, mp = np.array([20.0 / np.sqrt(n) if n < 1000 else 0.01]), np.array([4], np.uint32)
    _check(ctx, vdb, orc, x, y, eps, mp)
    for bad in (np.nan, np.inf, -np.inf):
        x[-1] = bad
        with pytest.raises(vdb.VDBError):
            ctx.run([vdb.BatchItem(x, y, eps, mp, 70)])


@pytest.mark.parametrize("n", [262144, 262145, 786432, 786433])
def test_sort_tiles(ctx, vdb, orc, n):
    # the sizes at which the sorts change their tiles
    rng = np.random.default_rng(n)
    x, y = rng.uniform(0, 40, n), rng.uniform(0, 40, n)
    _check(ctx, vdb, orc, x, y, np.array([0.03, 0.02]), np.array([3, 2], np.uint32))


@pytest.mark.parametrize("entry_bytes", [2, 4])
@pytest.mark.parametrize("gap", [100, 1000, 7000, 100000])
def test_dense_regions_far_apart_in_the_same_rows(ctx, vdb, orc, gap, entry_bytes):
    # two dense lattice regions with nothing but empty cells between them (gap: in
    # cells of the middle epsilon), thousands of pairs at exactly eps: a run of
    # points that begins in the one region and ends in the other has a box whose
    # edges are far from its first point
    rng = np.random.default_rng(gap)
    n1, n2, step = 3500, 30000, 0.004
    x = np.concatenate([rng.uniform(1.0, 1.06, n1), rng.uniform(0.0, 0.06, n2) + 1.0 + gap * 0.01])
    x, y = np.rint(x / step) * step, np.rint(rng.uniform(40.0, 40.06, n1 + n2) / step) * step
    eps = np.array([0.01, 0.02, 0.05])
    mp = np.array([700, 9000, 20000], np.uint32)
    want = orc.variants(x, y, eps, mp, 70)
    item = vdb.BatchItem(x, y, eps, mp, 70)
    out, st = ctx.run([item], table_hash=True, entry_bytes=entry_bytes)
    np.testing.assert_array_equal(out[0], want)
    assert st["table_hash"] == sum(orc.table_hash(x, y, e, 70) for e in eps) & M64
    out, sb = ctx.run([item], table="border", entry_bytes=entry_bytes)
    np.testing.assert_array_equal(out[0], want)
    assert sb["pairs"] == st["pairs"]


@pytest.mark.parametrize("cpe", [4, 15, 16, 17, 24, 31, 32])
def test_many_cells_per_epsilon(ctx, vdb, orc, cpe):
    # up to 65 rows of up to 65 cells around each cell, most of them with points;
    # minpts near the degrees: cores and border points everywhere
    rng = np.random.default_rng(3)
    n = 9000
    x, y = rng.uniform(0, 6, n), rng.uniform(0, 4, n)
    x[:1500], y[:1500] = rng.normal(1.5, 0.4, 1500), rng.normal(3.0, 0.4, 1500)
    eps = np.array([1.0, 1.0, 1.0, 0.4, 0.4])
    mp = np.array([980, 1250, 2250, 160, 560], np.uint32)
    _check(ctx, vdb, orc, x, y, eps, mp, cells_per_eps=cpe)
    # two clusters that meet at one pair of cells, with up to 57 cells of noise
    # before it in the row: (0, 0) has its mass below, (0.95, 0.15) to the right
    px = np.concatenate([np.full(300, 0.2), np.zeros(5), np.full(5, 0.95), np.full(300, 1.9)])
    py = np.concatenate([np.full(300, -0.9), np.zeros(5), np.full(305, 0.15)])
    rx = np.arange(-0.9, 0.88, 1 / 32)
    x, y = np.concatenate([px, rx]), np.concatenate([py, np.full(len(rx), 0.15)])
    assert orc.variants(x, y, np.ones(1), np.array([200], np.uint32), 70).max() == 1
    _check(ctx, vdb, orc, x, y, np.ones(2), np.array([200, 3], np.uint32), cells_per_eps=cpe)


@pytest.mark.parametrize("cpe", [33, 50, 1000])
def test_more_cells_per_epsilon_than_the_rows_hold(ctx, vdb, orc, cpe):
    # the kernels hold 65 rows of cells: finer cells than 32 per epsilon are not made
    rng = np.random.default_rng(cpe)
    x, y = rng.uniform(0, 3, 2000), rng.uniform(0, 3, 2000)
    eps, mp = np.array([1.0, 0.3]), np.array([600, 60], np.uint32)
    _check(ctx, vdb, orc, x, y, eps, mp, cells_per_eps=cpe)


@pytest.mark.parametrize("entry_bytes", [2, 4])
def test_rows_built_twice_are_hashed_once(ctx, vdb, orc, entry_bytes):
    # row chunks that the labelling reads (cells that are no cliques) are built
    # for the unions and again for the border points
    rng = np.random.default_rng(6)
    n = 30011
    x, y = rng.uniform(0, 40, n), rng.uniform(0, 40, n)
    eps, mp = np.array([0.5, 0.5]), np.array([9, 14], np.uint32)
    kw = dict(entry_bytes=entry_bytes, table_hash=True, cells_per_eps=1)
    out, st = ctx.run([vdb.BatchItem(x, y, eps, mp, 70)], budget=200000, **kw)
    np.testing.assert_array_equal(out[0], orc.variants(x, y, eps, mp, 70))
    assert st["table_hash"] == orc.table_hash(x, y, 0.5, 70) & M64
    assert st["table_chunks"] > 2


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [33, 63, 64, 65, 97, 1500, 131100])
def test_tables_without_a_bitmap(ctx, vdb, orc, n, precision):
    # a far point makes one cell of all the others: every point a candidate of
    # all, few of them neighbours, so that the table fits a budget which the
    # bitmap of the tests exceeds (tiles of 32, of 64 from 2^17 points on)
    rng = np.random.default_rng(n)
    side = 1.0 if n < 1000 else 2.0
    x, y = rng.uniform(0, side, n), rng.uniform(0, side, n)
    x[0], y[0] = 1e5, 1e5
    eps, mp = np.array([0.004 if n > 1e5 else 0.02]), np.array([3], np.uint32)
    item = vdb.BatchItem(x, y, eps, mp, 70)
    want = orc.variants(x, y, eps, mp, 70)
    for entry_bytes in (2, 4):
        kw = dict(table_hash=True, precision=precision, entry_bytes=entry_bytes)
        _, sw = ctx.run([item], **kw)
        out, st = ctx.run([item], budget=sw["entry_bytes"], **kw)
        np.testing.assert_array_equal(out[0], want)
        assert st["table_chunks"] == 1
        assert st["table_hash"] == sw["table_hash"] == orc.table_hash(x, y, eps[0], 70) & M64
