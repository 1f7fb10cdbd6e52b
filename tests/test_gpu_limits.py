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
