"""Calls at the limits of device memory: what they hold, and when."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vdb():
    import variantdbscan_gb300 as v
    from variantdbscan_gb300 import build
    build.build()
    return v


def test_more_work_units_than_their_offsets_hold(vdb, orc):
    # every point a candidate of all the others: 2.2 thousand million units of
    # 1,024 candidates, refused before anything is sized by them
    rng = np.random.default_rng(1)
    n = 12_000_000
    x, y = rng.uniform(0, 1, n), rng.uniform(0, 1, n)
    c = vdb.Context()
    for table in ("border", "all"):
        with pytest.raises(vdb.VDBError) as e:
            c.run([vdb.BatchItem(x, y, [2.0], [5], 70)], table=table, unit_candidates=1024)
        assert e.value.code == -4
        out, _ = c.run([vdb.BatchItem(x[:3000], y[:3000], [0.02], [5], 70)], table=table)
        np.testing.assert_array_equal(out[0], orc.variants(x[:3000], y[:3000], [0.02], [5], 70))
    c.close()


@pytest.mark.parametrize("cpe", [0, 1])
def test_labelling_when_the_table_fills_the_memory(vdb, cpe):
    # a table that takes all the memory it is given, eight minpts to label after
    # it: the labelling's own memory has to be there (cells_per_eps 1 labels from
    # the table, over points)
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(12)
    n = 1_000_000
    x, y = rng.uniform(0, 100, n), rng.uniform(0, 100, n)
    eps = np.full(8, 1.2)
    mp = np.array([300, 350, 400, 430, 450, 470, 500, 550], np.uint32)
    item = vdb.BatchItem(x, y, eps, mp, 70)
    c = vdb.Context()
    want, sw = c.run([item], cells_per_eps=cpe)
    c.close()
    assert sw["table_chunks"] == 1
    c = vdb.Context()
    c.run([vdb.BatchItem(x[:5000], y[:5000], eps[:2], mp[:2], 70)], cells_per_eps=cpe)
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - (960 << 20), dtype=torch.uint8, device="cuda")
    try:
        out, st = c.run([item], cells_per_eps=cpe)
    finally:
        del hold
        torch.cuda.empty_cache()
        c.close()
    np.testing.assert_array_equal(out[0], want[0])
    assert st["table_chunks"] > 1


@pytest.mark.parametrize("kw", [dict(eps=[0.4], budget=100000), dict(eps=[-1.0], budget=0)])
def test_stats_of_a_call_that_no_graph_captures(vdb, kw):
    # row chunks and empty neighbourhoods are not captured: the first call with
    # graph=True records a run before it finds out
    rng = np.random.default_rng(9)
    x, y = rng.uniform(0, 30, 20000), rng.uniform(0, 30, 20000)
    lab = np.zeros((1, 20000), np.uint32)
    item = vdb.BatchItem(x, y, kw["eps"], [6], 70, lab)
    c = vdb.Context()
    want, sw = c.run([item], budget=kw["budget"], table_hash=True)
    for _ in range(2):
        out, st = c.run([item], budget=kw["budget"], table_hash=True, graph=True)
        assert st["graph"] == 4  # unsupported: ran directly
        for k in ("pairs", "candidates", "tables", "table_chunks", "clusters", "table_hash",
                  "entry_bytes", "worker_streams"):
            assert st[k] == sw[k], k
    c.close()


@pytest.mark.parametrize("graph", [False, True])
def test_work_units_when_memory_is_short(vdb, graph):
    # a far point makes one cell of all the others, but the cells look nearly
    # empty: units of 1,024 candidates, 1.1M of them, take 330 MB where 150 are
    # left; the largest ones take 80
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(13)
    n = 270_000
    x, y = rng.uniform(0, 1, n), rng.uniform(0, 1, n)
    x[0], y[0] = 1e6, 1e6
    item = vdb.BatchItem(x, y, [0.002], [3], 70, np.zeros((1, n), np.uint32))
    c = vdb.Context()
    want, _ = c.run([vdb.BatchItem(x, y, [0.002], [3], 70)])
    c.close()
    c = vdb.Context()
    c.run([vdb.BatchItem(x[1:5000], y[1:5000], [0.02], [3], 70)])
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - (300 << 20), dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2 if graph else 1):
            out, st = c.run([item], graph=graph)
            np.testing.assert_array_equal(out[0], want[0])
    finally:
        del hold
        torch.cuda.empty_cache()
        c.close()


@pytest.mark.parametrize("entry_bytes", [2, 4])
def test_memory_of_sparse_data(vdb, entry_bytes):
    # a few points per tile: counts per unit and query (256 bytes a unit) are kept
    # for the tiles that warps take only, so the index, the bitmap and the
    # labelling stay below 320 bytes a point beside the table
    rng = np.random.default_rng(14)
    n = 1_000_000
    x, y = rng.uniform(0, 100, n), rng.uniform(0, 100, n)
    c = vdb.Context()
    out, st = c.run([vdb.BatchItem(x, y, [0.3], [6], 70)], entry_bytes=entry_bytes)
    c.close()
    assert out[0].max() > 0
    assert st["device_bytes"] - st["table_bytes"] < 320 * n
