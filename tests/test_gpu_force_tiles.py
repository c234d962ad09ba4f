"""The tiled force kernel at the edges of its tiles, blocks and tables, against
all pairs in FP64: partial and single-atom tiles, empty cells, columns of one
and of many runs, cells wider than the cutoff (more candidate blocks than the
warps' table holds), one to five atom types with their own cutoffs, 64-bit
sums, open boxes, atoms far outside their cells on every side, pairs that do
not interact, the soft core, and uneven density."""
import numpy as np
import pytest

from particlebase_b200 import workloads as W

pytestmark = pytest.mark.gpu

BAR = 1e-5  # relative RMS of the forces, the bar of the plain FP32 path


def system(L, n, ntypes, seed):
    """n atoms on a jittered grid of spacing 1.12 or more in a box of edges L."""
    rng = np.random.default_rng(seed)
    L = np.asarray(L, np.float32).astype(np.float64)
    k = np.floor(L / 1.12).astype(int)
    g = np.stack(np.meshgrid(*[np.arange(x) for x in k], indexing="ij"), -1).reshape(-1, 3)
    g = g[rng.permutation(len(g))[:n]]
    r = (g + 0.5 + rng.uniform(-0.12, 0.12, g.shape)) * (L / k)
    r = r.astype(np.float32).astype(np.float64)
    lj = np.zeros((ntypes, ntypes, 3))
    for a in range(ntypes):
        for b in range(ntypes):
            sig = 0.5 * (1.0 - 0.04 * a + 1.0 - 0.04 * b)
            lj[a, b] = sig, 1.0 + 0.1 * abs(a - b), 2.5 * sig
    lj = lj.astype(np.float32).astype(np.float64)
    box = np.array([0, L[0], 0, L[1], 0, L[2]], np.float32)
    types = rng.integers(0, ntypes, len(r)).astype(np.uint32)
    return W.LJSystem(box=box, r=r, v=np.zeros_like(r), mass=np.ones(len(r)), types=types, lj=lj,
                      rc=2.5)


def all_pairs(s, periodic=True):
    d = s.r[:, None] - s.r[None]
    if periodic:
        d -= s.L * np.round(d / s.L)
    r2 = (d ** 2).sum(-1)
    sig, eps, rc = np.moveaxis(s.lj[s.types[:, None], s.types[None]], -1, 0)
    near = (r2 < rc * rc) & (r2 > 0)
    r2 = np.where(near, r2, 1.0)
    s6 = (sig * sig / r2) ** 3
    f = np.where(near, 24 * eps * s6 * (2 * s6 - 1) / r2, 0.0)
    pe = np.where(near, 4 * eps * s6 * (s6 - 1), 0.0).sum() / 2
    return (f[..., None] * d).sum(1), pe


def check(s, periodic=True, rmax=2.5, **kw):
    from particlebase_b200.md import from_system
    p = from_system(s, cell_rmax=rmax, **kw)
    if not periodic:
        p.setupCutoffBlock(rmax, periodic=False)
    p.calcBlockID()
    F, pe = all_pairs(s, periodic)
    scale = max(np.sqrt((F ** 2).sum()), 1.0)
    for energy in (False, True):
        p.calcForce(energy=energy)
        got = p.get("F")[:, :3].astype(np.float64)
        assert np.sqrt(((got - F) ** 2).sum()) < BAR * scale
    assert abs(p.sums()["pe"] - pe) < BAR * max(abs(pe), 1.0)
    return p.status()


@pytest.mark.parametrize("L,n", [
    ((7.9, 7.9, 7.9), 1), ((7.9, 7.9, 7.9), 2), ((7.9, 8.2, 9.0), 15), ((7.9, 8.2, 9.0), 16),
    ((7.9, 8.2, 9.0), 17), ((7.9, 8.2, 9.0), 343), ((8.0, 13.0, 40.0), 33),
    ((8.0, 8.0, 60.0), 1500), ((20.0, 8.0, 8.0), 800), ((11.0, 10.4, 18.1), 1201)])
def test_one_type(cuda_lib, L, n):
    assert check(system(L, n, 1, n)) == 0


@pytest.mark.parametrize("ntypes", [2, 3, 4, 5, 8])
def test_types_with_their_own_cutoffs(cuda_lib, ntypes):
    assert check(system((9.0, 10.5, 16.0), 900, ntypes, ntypes)) == 0


@pytest.mark.parametrize("ntypes", [1, 2])
def test_64_bit_sums(cuda_lib, ntypes):
    assert check(system((9.0, 10.5, 16.0), 701, ntypes, 7), fp64_forces=True) == 0


@pytest.mark.parametrize("rmax,ntypes", [(4.9, 1), (4.9, 3), (3.7, 2)])
def test_cells_wider_than_the_cutoff(cuda_lib, rmax, ntypes):
    assert check(system((15.0, 15.0, 15.0), 2100, ntypes, 3), rmax=rmax) == 0


@pytest.mark.parametrize("far", [0.0, 30.0, 4000.0])
def test_open_box_and_atoms_far_outside(cuda_lib, far):
    """Past some hundred cell edges an atom leaves the range of the stage's fp16
    records, and the items whose home atom it is compute from global memory."""
    s = system((12.0, 11.0, 14.0), 700, 1, 5)
    if far:
        s.r[3] = (-far, 4.0, 5.0)
        s.r[90] = (3.0, -0.4, 2.0)
        s.r = s.r.astype(np.float32).astype(np.float64)
        d = s.r - s.r[90]
        keep = ((d ** 2).sum(1) > 0.9) | (np.arange(s.n) == 90)  # no overlap with the moved atom
        s.r, s.v, s.mass, s.types = s.r[keep], s.v[keep], s.mass[keep], s.types[keep]
    assert check(s, periodic=False) == 0


def test_non_finite_atoms_leave_the_others_alone(cuda_lib):
    """NaN and infinite coordinates: no force on or from those atoms."""
    from particlebase_b200.md import from_system
    s = system((9.0, 10.5, 16.0), 800, 1, 9)
    bad = {5: (np.nan, 1.0, 2.0), 77: (3.0, 3.0, np.nan), 200: (np.inf, 2.0, 2.0),
           333: (1.0, -np.inf, 9.0), 640: (4.0, 5.0, np.inf), 641: (np.nan,) * 3}
    p = from_system(s)
    r = p.get("r")
    for k, x in bad.items():
        r[k, :3] = x
    p.set("r", r)
    p.calcBlockID()
    p.calcForce()
    got = p.get("F")[:, :3].astype(np.float64)
    keep = np.setdiff1d(np.arange(s.n), list(bad))
    assert (got[list(bad)] == 0).all()
    s.r, s.types = s.r[keep], s.types[keep]
    F, _ = all_pairs(s)
    assert np.sqrt(((got[keep] - F) ** 2).sum()) < BAR * np.sqrt((F ** 2).sum())


def pair_sums(s):
    """Forces, and the sums over unordered pairs of the energy, the energy less its value
    at the cutoff, and F . r; the last is the number of ordered pairs inside the cutoff."""
    d = s.r[:, None] - s.r[None]
    d -= s.L * np.round(d / s.L)
    r2 = (d ** 2).sum(-1)
    sig, eps, rc = np.moveaxis(s.lj[s.types[:, None], s.types[None]], -1, 0)
    near = (r2 < rc * rc) & (r2 > 0)
    r2, rc2 = np.where(near, r2, 1.0), np.where(near, rc * rc, 1.0)
    s6, c6 = (sig * sig / r2) ** 3, (sig * sig / rc2) ** 3
    fr = np.where(near, 24 * eps * s6 * (2 * s6 - 1), 0.0)
    u = np.where(near, 4 * eps * s6 * (s6 - 1), 0.0)
    us = np.where(near, u - 4 * eps * c6 * (c6 - 1), 0.0)
    return ((fr / r2)[..., None] * d).sum(1), u.sum() / 2, us.sum() / 2, fr.sum() / 2, near.sum()


@pytest.mark.parametrize("acc64", [False, True])
@pytest.mark.parametrize("eps", [1.0, 0.0])
@pytest.mark.parametrize("ntypes", [2, 3, 5, 8])
def test_pairs_that_do_not_interact(cuda_lib, ntypes, eps, acc64):
    """A cutoff of zero switches a pair of types off, whatever its epsilon: no force, no
    energy, no virial and no pair counted, in dynamics and in the relaxation force (which
    caps no pair here: none is closer than half a sigma)."""
    from particlebase_b200.md import from_system
    s = system((9.0, 10.5, 16.0), 900, ntypes, 20 + ntypes)
    for a, b in ((0, 0), (0, ntypes - 1), (ntypes - 1, 0)):
        s.lj[a, b] = s.lj[a, b, 0], eps, 0.0
    F, *want = pair_sums(s)
    scale = np.sqrt((F ** 2).sum())
    p = from_system(s, fp64_forces=acc64)
    p.calcBlockID()
    for energy in (False, True):
        p.calcForce(energy=energy)
        got = p.get("F")[:, :3].astype(np.float64)
        assert np.sqrt(((got - F) ** 2).sum()) < BAR * scale
    e = p.sums()
    for k, w in zip(("pe", "pe_shift", "virial"), want):
        assert abs(e[k] - w) < BAR * max(abs(w), 1.0), k
    assert p.pair_stats()["nin"] == want[3]
    p.minimize(1)
    got = p.get("F")[:, :3].astype(np.float64)
    assert np.sqrt(((got - F) ** 2).sum()) < BAR * scale
    assert p.status() == 0


@pytest.mark.parametrize("up", [6.0, 60.0])
@pytest.mark.parametrize("Lz", [14.0, 45.0])
def test_open_box_atoms_above_the_top_face(cuda_lib, up, Lz):
    """Atoms more than a cell above the top of an open box are filed in cell 0, among
    atoms far below them: their column is not sorted by z.  One such atom or two above
    every column (of one run and of two), at several alignments of the columns' blocks
    and tiles."""
    full = system((12.0, 11.0, Lz), 10 ** 6, 1, 11)
    x, y = np.meshgrid(np.arange(1.25, 12, 2.5), np.arange(1.25, 12, 2.5), indexing="ij")
    odd = (np.round(x / 2.5 - 0.5) + np.round(y / 2.5 - 0.5)) % 2 == 1
    z = Lz + up + np.where(odd, 0.7, 0.0)
    high = np.stack([x, y, z], -1).reshape(-1, 3)
    high = np.concatenate([high, high[odd.reshape(-1)] + [0.0, 0.0, 1.1]])
    rng = np.random.default_rng(3)
    for k in range(16 if Lz < 20 else 6):
        # any atoms but a few of the lowest cells, so that every column's cell 0 shifts
        low = np.flatnonzero(full.r[:, 2] < 2.4)
        keep = np.setdiff1d(np.arange(full.n), rng.permutation(low)[:5 * k])
        r = np.concatenate([full.r[keep], high]).astype(np.float32).astype(np.float64)
        s = W.LJSystem(box=full.box, r=r, v=np.zeros_like(r), mass=np.ones(len(r)),
                       types=np.zeros(len(r), np.uint32), lj=full.lj, rc=2.5)
        assert check(s, periodic=False) == 0


@pytest.mark.parametrize("ntypes", [1, 3])
@pytest.mark.parametrize("far", [20.0, 150.0, 400.0, 430.0, 470.0, 640.0, 700.0, 5000.0])
def test_open_box_pairs_far_outside(cuda_lib, far, ntypes):
    """Bound pairs of atoms far from the box, beside which the box's own atoms keep their
    forces: within the range of the fp16 records (some 173 cell edges for a home atom, 256
    for a candidate's norm) and beyond it."""
    s = system((12.0, 11.0, 14.0), 650, ntypes, 6)
    y, z = np.arange(1.25, 11, 2.6), 1.25  # no two of them at the cutoff
    first = np.concatenate([[(-far, a, z) for a in y], [(12.0 + far, a + 0.1, z + 5) for a in y],
                            [(a, -far, z + 2.5) for a in y], [(a, 4.0, -far) for a in y]])
    pairs = np.concatenate([first, first + [0.4, 0.7, 0.8]])
    s.r = np.concatenate([s.r, pairs]).astype(np.float32).astype(np.float64)
    s.v, s.mass = np.zeros_like(s.r), np.ones(len(s.r))
    s.types = np.concatenate([s.types, np.arange(len(pairs)) % ntypes]).astype(np.uint32)
    assert check(s, periodic=False) == 0


@pytest.mark.parametrize("ntypes", [1, 2, 5])
@pytest.mark.parametrize("rc", [0.9, 2.0, 2.5, 3.1])
def test_soft_core(cuda_lib, ntypes, rc):
    """f0 cos(pi r / 2 rc) along r, within rc and the pair's own cutoff, against all pairs in
    FP64; also where the range ends beyond the cutoff, and in cells that go to global memory
    (a dense ball)."""
    from particlebase_b200.md import from_system
    a = system((9.0, 10.5, 16.0), 900, ntypes, 30 + ntypes)
    b = system((20.0, 20.0, 20.0), 600, ntypes, 5)
    ball = 10.0 + np.random.default_rng(1).uniform(-1.5, 1.5, (2500, 3))
    b.r = np.concatenate([b.r, ball]).astype(np.float32).astype(np.float64)
    b.v, b.mass = np.zeros_like(b.r), np.ones(len(b.r))
    b.types = (np.arange(len(b.r)) % ntypes).astype(np.uint32)
    for s, overflow in ((a, 0), (b, 1)):
        d = s.r[:, None] - s.r[None]
        d -= s.L * np.round(d / s.L)
        r2 = (d ** 2).sum(-1)
        pair = s.lj[s.types[:, None], s.types[None], 2]
        r = np.sqrt(r2)
        near = (r < np.minimum(rc, pair)) & (r2 > 0)
        f = np.where(near, 10.0 * np.cos(np.pi / 2 * r / rc) / np.where(near, r, 1.0), 0.0)
        F = (f[..., None] * d).sum(1)
        p = from_system(s)
        p.calcBlockID()
        p.calcForceSoftCore(rc, 10.0)
        got = p.get("F")[:, :3].astype(np.float64)
        assert np.sqrt(((got - F) ** 2).sum()) < BAR * np.sqrt((F ** 2).sum())
        assert p.status() == overflow


@pytest.mark.parametrize("ntypes,fill", [(1, 0.78), (1, 0.8), (2, 0.76), (2, 0.8)])
def test_density_contrast_that_fits_the_stage(cuda_lib, po, ntypes, fill):
    """A slab of liquid with empty space above it: the items inside it hold up to 1 / fill
    times the mean occupancy, which the stage has room for; an item that does not fit takes
    the slower global path and raises the status word."""
    from particlebase_b200.md import from_system
    L = np.array([20.0, 20.0, 150.0])
    k = np.round(L / (4 / 0.8442) ** (1 / 3)).astype(int)
    g = np.stack(np.meshgrid(*[np.arange(x) for x in k], indexing="ij"), -1).reshape(-1, 1, 3)
    r = (g + np.array([[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]]) + 0.25).reshape(-1, 3) / k * L
    r = r[r[:, 2] < fill * L[2]]
    r += np.random.default_rng(2).normal(0, 0.05, r.shape)
    r = r.astype(np.float32).astype(np.float64)
    lj = np.ones((ntypes, ntypes, 3)) * [1.0, 1.0, 2.5]
    s = W.LJSystem(box=np.array([0, L[0], 0, L[1], 0, L[2]], np.float32), r=r, v=np.zeros_like(r),
                   mass=np.ones(len(r)), types=(np.arange(len(r)) % ntypes).astype(np.uint32),
                   lj=lj, rc=2.5)
    p = from_system(s)
    p.calcBlockID()
    p.calcForce()
    assert p.status() == 0
    O = po.Oracle(s.box, s.lj, s.rc, s.r, types=s.types)
    O.forces()
    F = O.get("F")
    got = p.get("F")[:, :3].astype(np.float64)
    assert np.sqrt(((got - F) ** 2).sum()) < BAR * np.sqrt((F ** 2).sum())
