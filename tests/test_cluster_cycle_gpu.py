"""The levels of the mixed-precision cycle that run in one thread-block cluster, at the shapes where
their strips, columns and readers change: strips of one to several rows, partial last strips, idle
CTAs, one and several column segments, levels walked by every CTA alone, rigid walls, unequal
spacings, both schedules.

psi itself is fixed by the FP64 residual, so an error in the cycle shows in the number of cycles:
the FP64 path with the same schedule, smoother and correction scheme contracts the same error, and
FP32 rounding of a correction moves a residual by less than a cycle's contraction.  psi is compared
at the tolerance times the conditioning that the existing mixed tests use."""
import numpy as np
import pytest

from projectracer_gb300 import engine as eng
from projectracer_gb300.config import PT_CYCLE_REFERENCE, PT_CYCLE_V, PT_MG_CORRECTION, PT_PREC_FP64, PT_PREC_MIXED
from projectracer_gb300.inputs import make_state
from tests.helpers import rel_err, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nx,nz,grids,cycle,vbc", [
    ("iso", 32, 32, 3, PT_CYCLE_V, 0),      # level 2 of 16x16: 15 strips of one row, one CTA idle
    ("chem", 64, 64, 4, PT_CYCLE_V, 0),     # strips of two rows
    ("chem", 96, 48, 3, PT_CYCLE_V, 1),     # rigid walls, 23 rows over 16 CTAs
    ("chem", 128, 128, 6, PT_CYCLE_V, 0),   # strips of four rows, solo levels, solo coarsest solve
    ("chem", 128, 128, 5, PT_CYCLE_REFERENCE, 0),  # a level visited again and again, FP64 residuals
    ("depth", 256, 64, 4, PT_CYCLE_V, 0),   # four column segments, 31 rows
    ("depth", 48, 256, 4, PT_CYCLE_V, 1),   # tall: eight rows a strip, one segment
    ("chem", 112, 80, 4, PT_CYCLE_V, 0),    # strips of three rows, partial last strip, ragged segment
    ("c3", 256, 128, 4, PT_CYCLE_V, 0),     # coarsest solve over the whole cluster
])
def test_cluster_levels_contract_like_the_fp64_cycle(kind, nx, nz, grids, cycle, vbc):
    cfg, _ = small_case(kind, nx=nx, nz=nz, tpc=4)
    cfg.aspect = 1.1 * nx / nz if nx == 112 else nx / nz
    cfg.grids, cfg.mg_cycle, cfg.Vbc, cfg.mg_scheme = grids, cycle, vbc, PT_MG_CORRECTION
    cfg.nstageS = cfg.nstageC = 10
    cfg.dampingS, cfg.tolerance, cfg.max_cycles = 30.0, 1e-6, 200
    st = make_state(cfg, 8, noise=1e-3 if cfg.ivis else 0.0)
    out = {}
    for prec in (PT_PREC_FP64, PT_PREC_MIXED):
        c = cfg.copy()
        c.precision = prec
        e = eng.Engine(c)
        e.upload(st)
        info = e.solve_psi()
        assert info["resid_ratio"] <= c.tolerance
        out[prec] = (info["cycles"], e.get(eng.F_SF))
        e.close()
    assert abs(out[PT_PREC_MIXED][0] - out[PT_PREC_FP64][0]) <= 1 + out[PT_PREC_FP64][0] // 10
    assert rel_err(out[PT_PREC_MIXED][1], out[PT_PREC_FP64][1]) < 1e-4
    assert np.isfinite(out[PT_PREC_MIXED][1]).all()


@pytest.mark.parametrize("kind,nx,nz,grids,cycle,vbc,scheme", [
    ("iso", 32, 32, 3, PT_CYCLE_REFERENCE, 0, 0),    # level 2 of 16x16: strips of one row, one CTA idle
    ("chem", 96, 48, 3, PT_CYCLE_REFERENCE, 1, 0),   # rigid walls, two rows a strip, coarsest solve over the cluster
    ("chem", 128, 128, 6, PT_CYCLE_REFERENCE, 0, 0),  # stale corrections kept between visits
    ("depth", 256, 64, 4, PT_CYCLE_REFERENCE, 0, 1),  # four column segments
    ("depth", 48, 256, 4, PT_CYCLE_V, 1, 1),          # tall: eight rows a strip
    ("chem", 112, 80, 4, PT_CYCLE_REFERENCE, 0, 0),   # unequal spacings: ten derivative groups
])
def test_fp64_cluster_levels_match_the_reference_rounding(kind, nx, nz, grids, cycle, vbc, scheme):
    """The same solve with the reference's FP64 stencils, which runs a kernel per stage and the banded
    substitutions: the same outcome in the same number of cycles (the reference's stale corrections do
    not converge everywhere), and psi, or without convergence the first residuals, to the reference's
    rounding: 64 eps / h^4 of each stencil against the operator's smallest eigenvalue,
    (pi^2 (1 + 1 / aspect^2))^2."""
    cfg, _ = small_case(kind, nx=nx, nz=nz, tpc=4)
    cfg.aspect = 1.1 * nx / nz if nx == 112 else nx / nz
    cfg.grids, cfg.mg_cycle, cfg.Vbc, cfg.mg_scheme = grids, cycle, vbc, scheme
    cfg.tolerance, cfg.max_cycles = 1e-7, 100
    st = make_state(cfg, 9, noise=1e-3 if cfg.ivis else 0.0)
    out = []
    for rounding in (0, 1):
        c = cfg.copy()
        c.reference_rounding = rounding
        e = eng.Engine(c)
        e.upload(st)
        try:
            out.append((e.solve_psi()["cycles"], e.get(eng.F_SF)))
        except eng.PtError as ex:
            out.append((ex.code, np.array(e.residuals()[:8])))  # before rounding grows with a diverging cycle
        e.close()
    assert out[0][0] == out[1][0]
    bound = 64 * 1.1e-16 * max(nx / cfg.aspect, nz) ** 4 / (np.pi**2 * (1 + cfg.aspect**-2)) ** 2
    assert rel_err(out[0][1], out[1][1]) < bound
