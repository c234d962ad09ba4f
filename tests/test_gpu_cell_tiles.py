"""The bucket cell build at the tile counts where its launch shape changes, with
empty, overfull and out-of-order cells, against a sort of the oracle's cells by
(key, z, particle id)."""
import numpy as np
import pytest

from particlebase_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(3, 3, 3), (3, 4, 16), (16, 37, 16), (17, 35, 16),
                                   (37, 48, 16), (89, 20, 16), (37, 64, 16), (593, 8, 8)])
def test_sorted_cells(cuda_lib, po, cells, monkeypatch):
    monkeypatch.setenv("PB_CELL_BUILD", "bucket")
    rng = np.random.default_rng(sum(cells))
    check(cuda_lib, po, cells, 20011, 2, rng)


@pytest.mark.parametrize("cells,n,kernels", [
    ((3, 3, 3), 1, 1), ((3, 3, 3), 500, 1), ((3, 4, 16), 1023, 1), ((3, 4, 16), 1025, 1),
    ((8, 16, 16), 2047, 1), ((8, 16, 16), 2048, 1), ((8, 16, 16), 2049, 2), ((3, 3, 227), 1500, 1),
    ((3, 3, 228), 1500, 2)])
def test_sorted_cells_of_small_systems(cuda_lib, po, cells, n, kernels):
    """One block builds up to 2,048 atoms in up to 2,048 cells; on either side."""
    check(cuda_lib, po, cells, n, kernels, np.random.default_rng(n))


def check(cuda_lib, po, cells, n, kernels, rng):
    from particlebase_b200.md import from_system
    L = 2.5 * np.array(cells, np.float64) + 1.0
    r = rng.uniform(0, 1, (n, 3)) * L
    r[: n // 20] = rng.uniform(0, 2.0, (n // 20, 3))  # a cell past its bucket
    m = min(700, n // 4)
    r[n // 20: n // 20 + m] = L / 2 + rng.uniform(-1, 1, (m, 3))
    if n >= 100:
        r[-50:, 2] = r[-100:-50, 2]  # equal z
    r = np.minimum(r.astype(np.float32), np.nextafter(L.astype(np.float32), np.float32(0)))
    box = np.array([0, L[0], 0, L[1], 0, L[2]], np.float32)
    s = W.LJSystem(box=box, r=r.astype(np.float64), v=np.zeros((n, 3)), mass=np.ones(n),
                   types=np.zeros(n, np.uint32), lj=W.single_type_lj(2.5), rc=2.5)
    p = from_system(s)
    assert p.cell_build_kernels() == kernels
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
