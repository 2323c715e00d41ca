"""The sort's move with many tiles (one buffer, several CTAs a
multiprocessor): a run that sorts after its first step against one that does
not.  Sorting only changes the order in which a node's FP32 partial sums are
formed; a particle lost, doubled or torn would change eight nodes by a
particle's charge, 7e-5 of the norm for these densities."""
import numpy as np
import pytest

from ctca_b200 import inputs
from ctca_b200.emses import Emses

from helpers import case, rel_l2

pytestmark = pytest.mark.gpu


def run(c, steps, sort):
    cfg = inputs.make_config(c)
    cfg.flags = 1
    with Emses(cfg) as g:
        g.upload_field("eb", inputs.make_fields(c))
        g.fx_load_plasma(inputs.plasma(c))
        for _ in range(steps):
            g.fx_step(2, sort)
        e1 = g.fx_energy()
        g.fx_step(2, False)
        rho, j = g.fx_download_accum()
        return g.fx_counts(), e1, rho, j


def same(a, b):
    (na, ea, ra, ja), (nb, eb, rb, jb) = a, b
    assert np.array_equal(na, nb)
    # the same FP64 terms in another order: about 1e7 of them, 1e-16 * sqrt(1e7)
    assert np.allclose(ea, eb, rtol=1e-12, atol=0)
    # FP32 partial sums of some ten terms: 6e-8 * sqrt(10) of a node's value,
    # and the out-of-place particles summed on their own
    assert rel_l2(ra, rb) < 2e-6
    assert rel_l2(ja, jb) < 2e-6


# (cells, tile, ppc): 512 tiles of 1 and 10 rows (small shape), 560 partial
# ones, 2197 tiles of 35 rows (mid shape)
@pytest.mark.parametrize("n,tile,ppc", [
    ((32, 32, 32), 4, (115, 2)),
    ((37, 30, 27), 4, (24, 60)),
    ((104, 104, 104), 8, (50, 1)),
])
def test_move_many_tiles(gpu, n, tile, ppc):
    c = case(n=n, ppc=ppc, vth_scale=2.0, tile=(tile, tile, tile))
    same(run(c, 1, True), run(c, 1, False))


def test_move_tiles_past_the_window(gpu):
    """The mid shape with many tiles, 35 rows a tile on the mean: a beam
    reflected at the upper x face doubles the density there (tiles of more
    rows than the 48 of a window, gathered unstaged) and leaves tiles empty
    at the lower one."""
    c = case(n=(104, 104, 104), ppc=(50, 1), e=False, b0=(0.0, 0.0, 0.0), npbnd=(1, 1, 1), nfbnd=(1, 1, 1), tile=(8, 8, 8))
    for s in c.species:
        s.drift = (1.8, 0.0, 0.0)  # 0.9 cells a step
    same(run(c, 9, True), run(c, 9, False))
