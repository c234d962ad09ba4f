"""The bucket cell build at the tile counts where its launch shape changes, with
empty, overfull and out-of-order cells, against a sort of the oracle's cells by
(key, z, particle id)."""
import numpy as np
import pytest

from particlebase_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(3, 3, 3), (3, 4, 16), (16, 37, 16), (16, 16, 37 + 1),
                                   (37, 48, 16), (37, 48, 17), (37, 64, 16), (37, 65, 16)])
def test_sorted_cells(cuda_lib, po, cells, monkeypatch):
    from particlebase_b200.md import from_system
    monkeypatch.setenv("PB_CELL_BUILD", "bucket")
    rng = np.random.default_rng(sum(cells))
    L = 2.6 * np.array(cells, np.float64)
    n = 20011
    r = rng.uniform(0, 1, (n, 3)) * L
    r[: n // 20] = rng.uniform(0, 2.0, (n // 20, 3))  # a cell past its bucket
    r[n // 20: n // 20 + 700] = L / 2 + rng.uniform(-1, 1, (700, 3))
    r[-50:, 2] = r[-100:-50, 2]  # equal z
    r = np.minimum(r.astype(np.float32), np.nextafter(L.astype(np.float32), np.float32(0)))
    box = np.array([0, L[0], 0, L[1], 0, L[2]], np.float32)
    s = W.LJSystem(box=box, r=r.astype(np.float64), v=np.zeros((n, 3)), mass=np.ones(n),
                   types=np.zeros(n, np.uint32), lj=W.single_type_lj(2.5), rc=2.5)
    p = from_system(s)
    assert p.cell_build_kernels() == 2
    for _ in range(2):  # the second build reuses the cleared counters
        p.calcBlockID()
        r4 = p.get("r")
        cid = p.get("cell_of")
        assert np.array_equal(cid, po.bin_cells(r4, box, 2.5))
        key = p.get("cell_key")[cid]
        order = np.lexsort((np.arange(n), r4[:, 2], key))
        assert np.array_equal(p.get("pid"), order)
        assert np.array_equal(p.get("r_sorted")[:, :3], r4[order, :3])
        start = np.concatenate([[0], np.cumsum(np.bincount(key, minlength=p.numBlocks()))])
        assert np.array_equal(p.get("cell_start"), start)
