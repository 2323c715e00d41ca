"""Particles outside their tile's sort box (strays) in the tile sort: some in
a cell, many, and more than it takes (then the radix sort outside a graph)."""
import numpy as np
import pytest

from ctca_b200.emses import FX_ROW_SLOTS, Emses, EmsesError

from helpers import build, case, rel_l2

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "z", "vx", "vy", "vz")
STRAY_MAX = 16384


def key_of(cfg, tile, p):
    n = (cfg.nx, cfg.ny, cfg.nz)
    c = [np.floor(p[f]).astype(int) for f in "xyz"]
    nt = [-(-a // t) for a, t in zip(n, tile)]
    t = c[0] // tile[0] + nt[0] * (c[1] // tile[1] + nt[1] * (c[2] // tile[2]))
    return t * (tile[0] * tile[1] * tile[2]) + c[0] % tile[0] + tile[0] * (c[1] % tile[1] + tile[1] * (c[2] % tile[2]))


def strays(cfg, tile, before, after):
    ext = np.array([cfg.nx, cfg.ny, cfg.nz])
    c0, c1 = (np.stack([np.floor(p[f]) for f in "xyz"], 1).astype(int) for p in (before, after))
    off = c1 - (c0 // tile) * tile + 1
    off = np.where(off < 0, off + ext, np.where(off >= ext, off - ext, off))
    return int(np.any(off >= np.array(tile) + 2, axis=1).sum())


# (grid, ppc, thermal speed, more strays than the tile sort takes)
@pytest.mark.parametrize("n,ppc,vth,over", [
    ((24, 24, 24), (4, 3), 5.0, False),     # few
    ((24, 24, 24), (4, 3), 11.0, False),    # thousands, several in a cell
    ((20, 30, 26), (3, 2), 12.0, False),    # partial tiles
    ((32, 32, 32), (4, 1), 60.0, True),
])
def test_sort_with_strays(gpu, n, ppc, vth, over):
    tile = (8, 8, 8)
    c = case(n=n, ppc=ppc, vth_scale=vth, tile=tile)
    cfg, eb, p, tp = build(c, 1.2)
    runs = []
    for _ in range(2):
        g = Emses(cfg)
        g.upload_particles(p, tp)
        g.upload_field("eb", eb)
        g.fx_load()
        runs.append(g)
    a, b = runs
    a.fx_store()
    p0, _ = a.download_particles()
    for _ in range(4):
        a.fx_step(2, False)
    a.fx_store()
    p1, t1 = a.download_particles()
    ns = strays(cfg, tile, p0[:t1[0]], p1[:t1[0]])
    assert (ns > STRAY_MAX) if over else (0 < ns <= STRAY_MAX)
    a.fx_sort()
    a.fx_store()
    p2, t2 = a.download_particles()
    assert np.array_equal(t1, t2)
    base = np.concatenate([[0], np.cumsum(t1)])
    for s in range(cfg.nspec):
        u, v = p1[base[s]:base[s + 1]], p2[base[s]:base[s + 1]]
        assert np.all(np.diff(key_of(cfg, tile, v)) >= 0)
        ku, kv = (np.lexsort([q[f] for f in FIELDS]) for q in (u, v))
        for f in FIELDS:
            assert np.array_equal(u[f][ku], v[f][kv])
    # the same steps from a graph: the same bits where the tile sort takes the
    # strays; the order kept, and the sums equal to their FP32 rounding, where not
    a.fx_run(2, 8, 4, use_graph=False)
    for _ in range(4):
        b.fx_step(2, False)
    b.fx_sort()
    b.fx_run(2, 8, 4, use_graph=True)
    ra, ja = a.fx_download_accum()
    rb, jb = b.fx_download_accum()
    if over:
        # rounding of about 30 FP32 partial sums a node: 30 * 6e-8
        assert rel_l2(ra, rb) < 2e-6 and rel_l2(ja, jb) < 2e-6
    else:
        assert np.array_equal(ra, rb) and np.array_equal(ja, jb)
        a.fx_store()
        b.fx_store()
        pa, pb = a.download_particles()[0], b.download_particles()[0]
        assert np.array_equal(pa.view(np.uint8), pb.view(np.uint8))
    for g in runs:
        g.close()


def test_fallback_on_a_later_species_keeps_the_first(gpu):
    """Too many strays of the second species: the first, already through the
    tile sort, goes to the radix sort too, from its old layout.  Its tiles
    hold a few particles more than 9 rows at the load (13 ppc) and some of
    them fewer after the steps, so the new layout has fewer slots than the old
    one has in use."""
    tile = (8, 8, 8)
    c = case(n=(32, 32, 32), ppc=(13, 1), vth_scale=3.0, tile=tile)
    cfg, eb, p, tp = build(c, 1.2)
    p = p.copy()
    for f in ("vx", "vy", "vz"):
        p[f][tp[0]:] *= 600.0
    with Emses(cfg) as g:
        g.upload_particles(p, tp)
        g.upload_field("eb", eb)
        g.fx_load()
        g.fx_store()
        p0, _ = g.download_particles()
        for _ in range(4):
            g.fx_step(2, False)
        g.fx_store()
        p1, t1 = g.download_particles()
        n0 = int(t1[0])
        assert strays(cfg, tile, p0[:n0], p1[:n0]) <= STRAY_MAX < strays(cfg, tile, p0[n0:], p1[n0:])
        rows = [int(np.sum(-(-np.bincount(key_of(cfg, tile, q[:n0]) // 512) // FX_ROW_SLOTS))) for q in (p0, p1)]
        assert rows[1] < rows[0]
        g.fx_sort()
        assert np.array_equal(g.fx_counts(), t1)
        g.fx_store()
        p2, t2 = g.download_particles()
    assert np.array_equal(t1, t2)
    for u, v in ((p1[:n0], p2[:n0]), (p1[n0:], p2[n0:])):
        assert np.all(np.diff(key_of(cfg, tile, v)) >= 0)
        ku, kv = (np.lexsort([q[f] for f in FIELDS]) for q in (u, v))
        for f in FIELDS:
            assert np.array_equal(u[f][ku], v[f][kv])


# (grid, outer boundary, velocity): displacements of more than two axis lengths
# (ustep 2), where one wrap or reflection does not lead back into the grid
@pytest.mark.parametrize("n,npbnd,v", [
    ((2, 16, 16), 0, 2.2),
    ((20, 18, 13), 0, -40.0),       # partial tiles
    ((16, 16, 16), 1, 33.0),
    ((16, 16, 16), 0, 3e30),
])
@pytest.mark.parametrize("axis", range(3))
@pytest.mark.parametrize("sort", [False, True])
def test_displacement_past_the_grid_is_reported_and_dropped(gpu, n, npbnd, v, axis, sort):
    c = case(n=np.roll(n, axis), ppc=(6, 5), npbnd=(npbnd,) * 3, nfbnd=(npbnd,) * 3, e=False, b0=(0.0, 0.0, 0.0),
             tile=(8, 8, 8))
    cfg, eb, p, tp = build(c, 1.2)
    p = p.copy()
    m = int(tp[0]) // 2
    p["v" + "xyz"[axis]][m] = v
    with Emses(cfg) as g:
        g.upload_particles(p, tp)
        g.upload_field("eb", eb)
        g.fx_load()
        g.fx_step(2, sort)
        with pytest.raises(EmsesError, match="outside the field arrays"):
            g.synchronize()
        # the others go on without it
        g.fx_sort()
        g.fx_step(2, True)
        g.synchronize()
        assert np.array_equal(g.fx_counts(), tp[:cfg.nspec] - np.array([1, 0]))
