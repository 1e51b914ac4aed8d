"""The stats row against the trapezoid rule in numpy on the engine's own fields, at row lengths and
row counts below, at and past the CTA sizes of the two summing kernels (256 columns, 512 rows)."""
import numpy as np
import pytest

from projectracer_gb300 import engine as eng
from projectracer_gb300.inputs import make_state
from tests.helpers import small_case

pytestmark = pytest.mark.gpu


def trapz2(f, dr, ds, k0=0):
    w = lambda n: np.where((np.arange(n) == 0) | (np.arange(n) == n - 1), 0.5, 1.0)  # noqa: E731
    g = f[k0:]
    return float(w(g.shape[0]) @ (g @ w(g.shape[1]))) * dr * ds


@pytest.mark.parametrize("nx,nz,dent", [(16, 16, 0.5), (256, 32, 0.0), (520, 40, 0.3), (40, 520, 0.99), (32, 32, 1.0)])
def test_stats_row_is_the_trapezoid_rule(nx, nz, dent):
    cfg, _ = small_case("chem", nx=nx, nz=nz, tpc=4)
    cfg.aspect, cfg.dent = nx / nz, dent
    st = make_state(cfg, 4, noise=1e-3)
    e = eng.Engine(cfg)
    e.upload(st)
    before = e.stats()  # velocities zero
    e.solve_psi()
    s = e.stats()
    dr, ds = cfg.aspect / nx, 1.0 / nz
    inner = lambda a, g: a[g:-g, g:-g]  # noqa: E731
    T, u, w, vis = (inner(e.get(f), 3) for f in (eng.F_T, eng.F_U, eng.F_W, eng.F_VIS))
    C, n = inner(e.get(eng.F_CNEW), 5), e.get(eng.F_NEMPTY)
    a = cfg.aspect
    # a sum of N values of one sign carries a relative error of at most N ulp in either order
    tol = 4 * (nx + nz) * 2.3e-16
    kent = int(np.max(np.nonzero(ds * np.arange(nz + 1) <= dent)[0]))
    mass = trapz2(C, dr, ds) / a
    assert before["vrms"] == 0.0
    assert s["Tavg"] == pytest.approx(trapz2(T, dr, ds) / a, rel=tol)
    assert s["Cavg"] == pytest.approx(mass, rel=tol)
    assert s["vrms"] == pytest.approx(np.sqrt(trapz2(u * u + w * w, dr, ds) / a), rel=tol)
    assert s["RaT_avg"] == pytest.approx(trapz2(cfg.RaT / vis, dr, ds) / a, rel=tol)
    ent = trapz2(C, dr, ds, kent) / a / mass if kent < nz else 0.0
    assert s["entrainment"] == pytest.approx(ent, rel=tol, abs=1e-300)
    assert (s["empty_cells"], s["tracer_min"], s["tracer_max"]) == (int((n == 0).sum()), int(n.min()), int(n.max()))
    e.close()


# rows and columns below, at and past the terms that a CTA adds at a time (255 columns, 511 rows or columns)
@pytest.mark.parametrize("kind,nx,nz,direct", [("iso", 64, 64, 0), ("iso", 64, 64, 1), ("iso", 100, 100, 1),
                                               ("chem", 256, 32, 0), ("chem", 520, 40, 0), ("chem", 40, 520, 0)])
def test_stats_row_has_the_oracles_bits_where_the_solve_rounds_like_it(kind, nx, nz, direct):
    """Every column of the isoviscous runs, whose psi has the oracle's bits; of the others the columns that
    psi does not enter."""
    from oracle.ptref import Oracle

    cfg, _ = small_case(kind, nx=nx, nz=nz, tpc=4)
    cfg.aspect, cfg.direct = nx / nz, direct
    cfg.reference_rounding = 1 - direct
    if kind == "chem":
        cfg.tolerance = 1e-2
    st = make_state(cfg, 4, noise=1e-3)
    o = Oracle(cfg, iterate=1 - direct, nparts=0)
    o.load_restart(st["xg"], st["zg"], st["T"], st["Cnew"], st["SF"], st["rtr"], st["str"], st["Ctr"], st["Ttr"])
    o.solve_psi()
    e = eng.Engine(cfg)
    e.upload(st)
    e.solve_psi()
    a, b = e.stats(), o.stats()
    e.close()
    names = list(b) if kind == "iso" else ["Tavg", "RaT_avg", "Nu", "Nu_bot", "q1", "q2", "q3", "q4", "empty_cells"]
    assert {k: a[k] for k in names} == {k: b[k] for k in names}
