"""The FP64 projection's per-cell sums and sort at the edges of their warps: grids whose cell count is no
multiple of the ten cells of a warp, spacings that are a power of two and not, cells of no tracers, of more
than the 256 that a warp sorts in registers, and tracers on nodes and walls.  The oracle adds in the same
order, so the fields are compared bit for bit."""
import numpy as np
import pytest

from oracle.ptref import Oracle
from projectracer_gb300 import engine as eng
from tests.helpers import small_case, walls

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nx,nz", [("iso", 16, 16), ("chem", 24, 16), ("chem", 64, 32), ("chem", 40, 24)])
def test_projection_of_uneven_cells_is_bit_exact(kind, nx, nz):
    cfg, st = small_case(kind, nx=nx, nz=nz, tpc=16)
    st = walls(cfg, st)
    n = len(st["rtr"])
    dr = cfg.aspect / nx
    # 300 tracers in one cell (its neighbours lose theirs), some of them on its node
    st["rtr"][:300] = 5 * dr + np.linspace(-0.4, 0.4, 300) * dr
    st["str"][:300] = 7 / nz
    st["rtr"][::7][:40] = 5 * dr
    assert n > 600
    o = Oracle(cfg, iterate=1, nparts=0)
    o.load_restart(st["xg"], st["zg"], st["T"], st["Cnew"], st["SF"], st["rtr"], st["str"], st["Ctr"], st["Ttr"])
    e = eng.Engine(cfg)
    e.upload(st)
    assert np.array_equal(e.get(eng.F_NEMPTY), o.get(11)) and o.get(11).max() > 256
    g, r = e.get(eng.F_TRATIO), o.get(eng.F_TRATIO)
    assert np.array_equal(g[1:-1, 1:-1], r[1:-1, 1:-1])
    if cfg.comp:
        assert np.array_equal(e.get(eng.F_CNEW), o.get(4))
    e.close()


# tracers per cell on each side of the sort's widths (4 lanes up to a mean of 8 per cell, 8 up to 24, 32 above)
# and cells at and past what each width holds in registers (32, 64 and 256)
@pytest.mark.parametrize("tpc", [1, 7, 9, 25, 28])
def test_projection_is_bit_exact_at_every_width_of_the_sort(tpc):
    cfg, st = small_case("chem", nx=40, nz=24, tpc=tpc)
    n = len(st["rtr"])
    order = np.random.default_rng(2).permutation(n)
    for k in ("rtr", "str", "Ttr", "Ctr"):
        st[k] = np.ascontiguousarray(st[k][order])
    at, sizes = 0, (300, 70, 65, 64, 33, 32, 9, 8)
    for q, size in enumerate(sizes):  # cells (3 + 4 q, 5) get `size` tracers more
        st["rtr"][at:at + size] = (3 + 4 * q) * cfg.aspect / 40
        st["str"][at:at + size] = 5 / 24
        at += size
    o = Oracle(cfg, iterate=1, nparts=0)
    o.load_restart(st["xg"], st["zg"], st["T"], st["Cnew"], st["SF"], st["rtr"], st["str"], st["Ctr"], st["Ttr"])
    e = eng.Engine(cfg)
    e.upload(st)
    counts = o.get(11)
    assert np.array_equal(e.get(eng.F_NEMPTY), counts) and counts[5, 3:32:4].min() >= 8 and counts.max() >= 300
    g, r = e.get(eng.F_TRATIO), o.get(eng.F_TRATIO)
    assert np.array_equal(g[1:-1, 1:-1], r[1:-1, 1:-1])
    assert np.array_equal(e.get(eng.F_CNEW), o.get(4))
    e.close()
