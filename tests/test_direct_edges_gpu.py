"""The direct solve's substitutions at the edges of their blocks: fewer unknowns than the band or two
blocks of 32 columns, orders that are no multiple of 32, a band narrower than a block, and one whose
window takes two elements per thread; psi bit-identical to the oracle's direct solve."""
import pytest

from tests.test_direct_gpu import test_direct_solve_matches_oracle_on_larger_grids as same_bits

pytestmark = pytest.mark.gpu


# band 3 (nz + 1): 27, 51, 39, 963 (two elements per thread)
@pytest.mark.parametrize("nx,nz", [(8, 8), (24, 16), (8, 12), (32, 320)])
def test_direct_solve_matches_oracle_at_block_edges(nx, nz):
    same_bits(nx, nz)


def test_bands_past_the_documented_bound_are_refused():
    """kl + ku = 6 (nz + 1) up to 6,950: nz = 1152 is accepted, 1168 refused (both with nz / 16 rows on the
    coarsest of four halvings)."""
    from projectracer_gb300 import engine as eng
    from projectracer_gb300.config import PT_PREC_FP64, workload

    cfg, _ = workload("C1", 1.0, PT_PREC_FP64)
    cfg.nx, cfg.direct, cfg.mingrid = 32, 1, 2
    for nz in (1168, 1152):
        cfg.nz, cfg.aspect, cfg.ntr = nz, 32 / nz, 32 * nz
        if nz == 1168:
            with pytest.raises(eng.PtError, match="band is too wide") as ex:
                eng.Engine(cfg)
            assert ex.value.code == -1
        else:
            eng.Engine(cfg).close()


def test_wide_bands_take_four_elements_per_thread():
    """kl = 3 (640 + 1) = 1923, past twice the row threads, with the shorter ring: psi has the oracle's bits."""
    import numpy as np

    from oracle.ptref import Oracle
    from projectracer_gb300 import engine as eng
    from projectracer_gb300.config import PT_PREC_FP64, workload
    from projectracer_gb300.inputs import make_state

    cfg, _ = workload("C1", 1.0, PT_PREC_FP64)
    cfg.nx, cfg.nz, cfg.aspect, cfg.mingrid = 8, 640, 8 / 640, 1  # (a coarsest grid that pt_init takes)
    cfg.direct, cfg.ntr = 1, 8 * 640 * 4
    st = make_state(cfg, 3)
    e = eng.Engine(cfg)
    e.upload(st)
    e.solve_psi()
    e.solve_psi()
    sf = e.get(eng.F_SF)
    e.close()
    o = Oracle(cfg, iterate=0, nparts=0)
    o.load_restart(st["xg"], st["zg"], st["T"], st["Cnew"], st["SF"], st["rtr"], st["str"], st["Ctr"], st["Ttr"])
    o.solve_psi()
    assert np.array_equal(sf.view(np.int64), o.get(7).view(np.int64))
