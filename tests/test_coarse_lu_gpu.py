"""The coarse matrix's panel LU: coarsest grids whose order is a multiple of the panel's 16 columns or
not, below one panel and with bands wider than one, through the psi solve against the CPU oracle's
column-by-column LU."""
import pytest

from oracle.ptref import Oracle
from projectracer_gb300 import engine as eng
from tests.helpers import rel_err, small_case

pytestmark = pytest.mark.gpu


# coarsest grids of (nx+1)(nz+1) nodes and band kl = 3 (nz+1): 6x4 = 24, 8x6 = 48 (three panels of 16),
# 10x6 = 60, 8x8 = 64 (four), 14x8 = 112 (seven), 14x14 = 196, 18x14 = 252
@pytest.mark.parametrize("nx,nz", [(80, 48), (112, 80), (72, 40), (56, 56), (104, 56), (104, 104), (136, 104)])
@pytest.mark.parametrize("rounding", [0, 1])
def test_solves_on_coarse_grids_of_every_remainder_match_the_oracle(nx, nz, rounding):
    cfg, st = small_case("chem", nx=nx, nz=nz)
    cfg.reference_rounding = rounding
    o = Oracle(cfg, iterate=1, nparts=0)
    o.load_restart(st["xg"], st["zg"], st["T"], st["Cnew"], st["SF"], st["rtr"], st["str"], st["Ctr"], st["Ttr"])
    e = eng.Engine(cfg)
    e.upload(st)
    info = e.solve_psi()
    o.solve_psi()
    assert info["cycles"] == int(o.scalar("cycles"))
    # the bound of the solve's other comparisons with the oracle: sums that differ in the last bits
    assert rel_err(e.get(eng.F_SF), o.get(7)) < 1e-10
    e.close()


# two levels only, so that the inverse takes eight columns a CTA: 49 x 33 = 1617 nodes (a last panel of one
# column, a last CTA of one) and 41 x 33 = 1353 (nine columns, one)
@pytest.mark.parametrize("nx,nz", [(96, 64), (80, 64)])
def test_solves_with_two_levels_match_the_oracle(nx, nz):
    cfg, st = small_case("chem", nx=nx, nz=nz)
    cfg.grids = 2
    o = Oracle(cfg, iterate=1, nparts=0)
    o.load_restart(st["xg"], st["zg"], st["T"], st["Cnew"], st["SF"], st["rtr"], st["str"], st["Ctr"], st["Ttr"])
    e = eng.Engine(cfg)
    e.upload(st)
    info = e.solve_psi()
    o.solve_psi()
    assert info["cycles"] == int(o.scalar("cycles"))
    assert rel_err(e.get(eng.F_SF), o.get(7)) < 1e-10
    e.close()
