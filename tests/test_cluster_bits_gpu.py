"""The mixed cycle's cluster levels give the per-stage kernels' bits: the same solves with the library as
built and with one whose pt_mixed.cu runs a kernel per stage on every level (PT_STAGE_KERNELS), each in a
process of its own; psi, cycles and the history of residuals are equal bit for bit."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# (kind, nx, nz, grids, V cycle, rigid, GCR directions); the shapes of test_cluster_cycle_gpu.py
CASES = [
    ("iso", 32, 32, 3, 1, 0, 0),      # strips of one row, one CTA idle
    ("chem", 64, 64, 4, 1, 0, 8),     # strips of two rows
    ("chem", 96, 48, 3, 1, 1, 0),     # rigid walls, 23 rows over 16 CTAs, level 1 in the cluster
    ("chem", 128, 128, 6, 1, 0, 8),   # strips of four rows, solo levels, solo coarsest solve
    ("chem", 128, 128, 5, 0, 0, 0),   # a level visited again and again, FP64 residuals
    ("depth", 256, 64, 4, 1, 0, 8),   # four column segments, 31 rows
    ("depth", 48, 256, 4, 1, 1, 0),   # tall: eight rows a strip, one segment
    ("chem", 112, 80, 4, 1, 0, 8),    # unequal spacings, partial last strip, ragged segment
    ("c3", 256, 128, 4, 1, 0, 0),     # coarsest solve over the whole cluster
]


def solve_all(lib, out):
    from projectracer_gb300 import engine as eng
    from projectracer_gb300.config import PT_CYCLE_REFERENCE, PT_CYCLE_V, PT_MG_CORRECTION, PT_PREC_MIXED
    from projectracer_gb300.inputs import make_state
    from tests.helpers import small_case

    eng.load_library(lib)
    res = {}
    for q, (kind, nx, nz, grids, v, vbc, krylov) in enumerate(CASES):
        cfg, _ = small_case(kind, nx=nx, nz=nz, tpc=4)
        cfg.aspect = 1.1 * nx / nz if nx == 112 else nx / nz
        cfg.precision, cfg.grids, cfg.Vbc, cfg.krylov = PT_PREC_MIXED, grids, vbc, krylov
        cfg.mg_cycle, cfg.mg_scheme = PT_CYCLE_V if v else PT_CYCLE_REFERENCE, PT_MG_CORRECTION
        cfg.nstageS = cfg.nstageC = 10
        cfg.dampingS, cfg.tolerance, cfg.max_cycles = 30.0, 1e-6, 200
        e = eng.Engine(cfg)
        e.upload(make_state(cfg, 8, noise=1e-3 if cfg.ivis else 0.0))
        n = e.launches()
        res[f"cycles{q}"] = e.solve_psi()["cycles"]
        res[f"launches{q}"] = e.launches() - n
        res[f"psi{q}"], res[f"residuals{q}"] = e.get(eng.F_SF).view(np.int64), np.array(e.residuals()).view(np.int64)
        e.close()
    np.savez(out, **res)


@pytest.fixture(scope="module")
def solves(tmp_path_factory):
    from projectracer_gb300 import build
    from projectracer_gb300.engine import LIB_PATH

    d = tmp_path_factory.mktemp("stage_kernels")
    obj, lib = str(d / "pt_mixed.o"), str(d / "libptgpu_stages.so")
    src = os.path.join(build.CSRC, "pt_mixed.cu")
    subprocess.run([build.nvcc()] + build.ARCH + build.COMMON + build.EXTRA.get("pt_mixed.cu", []) +
                   ["-DPT_STAGE_KERNELS", "-c", src, "-o", obj], check=True)
    objs = [obj if s == "pt_mixed.cu" else os.path.join(build.BUILD, s + ".o") for s in build.SOURCES]
    subprocess.run([build.nvcc()] + build.ARCH + ["-shared", "-o", lib] + objs + ["-Xcompiler", "-fopenmp", "-lgomp"],
                   check=True)
    out = []
    for name, path in (("cluster", LIB_PATH), ("stages", lib)):
        npz = str(d / (name + ".npz"))
        subprocess.run([sys.executable, "-m", "tests.test_cluster_bits_gpu", path, npz], check=True, cwd=ROOT, timeout=300)
        out.append(dict(np.load(npz)))
    return out


@pytest.mark.parametrize("q", range(len(CASES)), ids=lambda q: "-".join(map(str, CASES[q])))
def test_cluster_levels_have_the_stage_kernels_bits(solves, q):
    cluster, stages = solves
    assert cluster[f"launches{q}"] < stages[f"launches{q}"]  # the two do run different kernels
    assert cluster[f"cycles{q}"] == stages[f"cycles{q}"]
    assert np.array_equal(cluster[f"residuals{q}"], stages[f"residuals{q}"])
    assert np.array_equal(cluster[f"psi{q}"], stages[f"psi{q}"])


if __name__ == "__main__":
    solve_all(*sys.argv[1:3])
