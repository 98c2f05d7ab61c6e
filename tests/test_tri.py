"""Float-pair and -triple geodesic arithmetic (mahakala_gb300/csrc/mk_tri.cuh)
on the host, against long double."""

import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def test_tri_arithmetic(tmp_path):
    """The acceleration in pairs: 64 chained operations of 2^-45 each, 2e-12
    of the size of its terms.  The radius in triples: 1.4e-17 (2^-56), an
    eighth of binary64's rounding.  Triple sums and products: 1e-18."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = tmp_path / "tri_check"
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-Xcompiler",
                    "-ffp-contract=off", "-I", os.path.join(ROOT, "mahakala_gb300", "csrc"), "-I",
                    os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "tri_check.cu"), "-o", str(exe)],
                   check=True)
    n, accel, radius, add, mul, round_trip = subprocess.run([str(exe)], check=True, capture_output=True,
                                                            text=True).stdout.split()
    assert int(n) > 30000 and round_trip == "1"
    assert float(accel) < 2e-12, accel
    assert float(radius) < 1.4e-17, radius
    assert float(add) < 1e-18 and float(mul) < 1e-18, (add, mul)


def _table_by_loops(arrs):
    """The finest-level block table, one block at a time."""
    faces = np.stack([arrs.x1f[:, 0], arrs.x1f[:, -1], arrs.x2f[:, 0], arrs.x2f[:, -1], arrs.x3f[:, 0],
                      arrs.x3f[:, -1]], axis=1)
    left, w = faces[:, 0::2], faces[:, 1::2] - faces[:, 0::2]
    wf, lo = w.min(axis=0), left.min(axis=0)
    nb = [int(round((faces[:, 2 * a + 1].max() - lo[a]) / wf[a])) for a in range(3)]
    table = -np.ones(nb[::-1], np.int32)
    for m in range(len(faces)):
        i, j, k = np.rint((left[m] - lo) / wf).astype(int)
        si, sj, sk = np.rint(w[m] / wf).astype(int)
        table[k:k + sk, j:j + sj, i:i + si] = m
    return table


def _fine_ghosts_by_loops(arrs):
    """Blocks with a ghost region filled from finer neighbours."""
    have = {(int(lv),) + tuple(int(c) for c in u) for lv, u in zip(arrs.Levels, arrs.LogicalLocations)}
    out = []
    for lv, u in zip(arrs.Levels, arrs.LogicalLocations):
        fine = False
        for d in np.ndindex(3, 3, 3):
            t = [int(c) + e - 1 for c, e in zip(u, d)]
            if (d == (1, 1, 1) or (int(lv), *t) in have or (int(lv) - 1, *(c // 2 for c in t)) in have):
                continue
            fine |= (int(lv) + 1, *(2 * c for c in t)) in have
        out.append(fine)
    return np.array(out)


@pytest.mark.parametrize("nblocks,refine", [(1, ()), (3, ()), (2, ((0, 0, 0, 0),)),
                                            (4, ((0, 1, 1, 1), (0, 2, 2, 2), (1, 2, 2, 2))),
                                            (3, ((0, 1, 1, 1), (1, 2, 3, 2), (2, 5, 6, 5)))])
def test_mesh_tables_match_loops(nblocks, refine):
    from mahakala_gb300.grmhd.athenak import mesh_tables
    from mahakala_gb300.grmhd.synthetic import make_multilevel_snapshot
    arrs = make_multilevel_snapshot(nblocks=nblocks, cells_per_block=4, extent=10., refine=refine)
    t = mesh_tables(arrs)
    assert np.array_equal(t["table"], _table_by_loops(arrs))
    fine = _fine_ghosts_by_loops(arrs)
    assert np.array_equal(t["block64"] >= 0, fine) and t["n64"] == fine.sum()
    arrs.x1f[-1], arrs.x2f[-1], arrs.x3f[-1] = arrs.x1f[0], arrs.x2f[0], arrs.x3f[0]
    if len(arrs.Levels) > 1:
        with pytest.raises(ValueError):
            mesh_tables(arrs)
