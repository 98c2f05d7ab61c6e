"""Rules of the FP64 paths that need no GPU (mahakala_gb300/csrc/mk_sample_pair.cuh)
and of the host code, at their limits."""

import os
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_render_rules(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = tmp_path / "limits_check"
    subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I", os.path.join(ROOT, "mahakala_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "limits_check.cu"), "-o", str(exe)], check=True)
    out = dict(line.split() for line in subprocess.run([str(exe)], check=True, capture_output=True,
                                                       text=True).stdout.splitlines())
    assert out and set(out.values()) == {"1"}, out


@pytest.mark.parametrize("error_allowed,max_it", [(1e-3, 40), (1e-3, 10.5), (1e-3, 0.5), (1e-3, float("inf")), (0.0, 7),
                                                  (-1.0, 30), (1e-12, 40), (1e-3, 0), (float("nan"), 5)])
def test_bisections_of_any_count(monkeypatch, error_allowed, max_it):
    """Several bisections a pass take the midpoints and the decisions of one at
    a time, for every way to say when to stop."""
    import numpy as np
    from mahakala_gb300 import geodesics as g
    edge = np.array([1.3, 2.7182818, 5.0, 9.99])

    def far(inc, ca, sa, mid, *rest):   # in reality the radius each ray ends at
        n = len(mid) // len(edge)
        return np.where(np.asarray(mid).reshape(n, -1) < edge, 1.0, 1000.0).reshape(-1)

    monkeypatch.setattr(g, "_shadow_pass", far)
    monkeypatch.setattr(g, "SHADOW_RAYS", 600)
    got = g.find_shadow_bisection_angles(0.5, 60.0, np.arange(4.0), error_allowed=error_allowed, max_it=max_it)
    inner, outer, count = np.full(4, 0.5), np.full(4, 10.0), 0
    while np.max(outer - inner) > error_allowed and count < max_it:
        mid = (outer - inner) / 2 + inner
        inner, outer, count = np.where(mid < edge, mid, inner), np.where(mid < edge, outer, mid), count + 1
    assert np.array_equal(got, inner)


@pytest.mark.parametrize("nblocks,depth", [(4, 6), (2, 7), (8, 2)])
def test_mesh_tables_of_deep_meshes(nblocks, depth):
    """A corner refined again and again: the finest-level table, one block at a
    time, in little more memory than the table's own (a sixth of it for a
    plane's test, the tables of the blocks, and an indexing pass of 2^18 cells)."""
    import tracemalloc
    from types import SimpleNamespace

    import numpy as np
    from mahakala_gb300.grmhd.athenak import mesh_tables
    from test_tri import _table_by_loops
    blocks = {(0,) + t for t in np.ndindex(nblocks, nblocks, nblocks)}
    key = (0, 0, 0, 0)
    for _ in range(depth):
        blocks.remove(key)
        blocks |= {(key[0] + 1,) + tuple(2 * c + d for c, d in zip(key[1:], t)) for t in np.ndindex(2, 2, 2)}
        key = (key[0] + 1,) + tuple(2 * c + 1 for c in key[1:])
    order = np.array(sorted(blocks))
    width = 16.0 / nblocks / 2.0 ** order[:, 0]
    faces = [np.stack([-8 + width * order[:, 1 + a], -8 + width * (order[:, 1 + a] + 1)], axis=1) for a in range(3)]
    arrs = SimpleNamespace(Levels=order[:, 0], LogicalLocations=order[:, 1:], x1f=faces[0], x2f=faces[1], x3f=faces[2])
    tracemalloc.start()
    table = mesh_tables(arrs)["table"]
    peak = tracemalloc.get_traced_memory()[1]
    tracemalloc.stop()
    assert np.array_equal(table, _table_by_loops(arrs))
    assert peak <= 1.2 * table.nbytes + (16 << 20), (peak, table.nbytes)


def test_bench_line_is_short_and_last(capsys):
    """The contract's keys end up in one last JSON line, the long records before it."""
    import json
    import sys
    sys.path.insert(0, ROOT)
    import bench
    line = {k: 1 for k in bench.LINE_KEYS if k != "impl"}
    line.update(sweep512=[{"max_pixel_rel_err": 1.23456789e-4, "spin": 0.94}] * 400, serving={"latency": [1.0] * 500})
    bench.print_line(line)
    out = capsys.readouterr().out.splitlines()
    assert json.loads(out[-1]) == {k: 1 for k in bench.LINE_KEYS if k != "impl"}
    assert [x for x in out if x.startswith("{")] == out[-1:] and len(out) == 3
    key, value = out[0].split(" ", 2)[1:]
    assert key == "sweep512" and json.loads(value) == line["sweep512"]
