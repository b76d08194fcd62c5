"""Each precision's records are filled once per cross-section set, in the order
that the sweeps take them in: not again when a served request joins its batch or
its solo solver, nor when a batch chooses its form.  Counted from the trace
lines of a child process (TYCHO_TRACE=1)."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PRELUDE = """
import sys
import numpy as np
import tycho2_b200 as ty

def problem(n, sn, G):
    mesh = ty.TychoMesh.kuhn_cube(n, 0.05, 3, 1.0)
    return mesh, sn, G, np.ones(mesh.n_cells), np.full(mesh.n_cells, 0.4), np.ones((mesh.n_cells, 4, G))

def sweeper(n, sn, G, fp32=True):
    mesh, sn, G, st, ss, q = problem(n, sn, G)
    sw = ty.SweeperCuda(mesh, sn, G, fp32=fp32)
    sw.set_cross_sections(st, ss)
    sw.set_source(q, "isotropic")
    return sw

def serve(problems, **kw):
    srv = ty.SolveServer(method="mixed", budget_bytes=8e9, setup_threads=2, err_max=1e-8, **kw)
    for mesh, sn, G, st, ss, q in problems:
        srv.submit(mesh, sn, G, st, ss, None, q, arrival=0.0)
    srv.run()
    srv.close()

def batch(sweepers, method):
    b = ty.BatchSolver()
    for s in sweepers:
        b.add(s, method, err_max=1e-8)
    b.run()
    b.close()
"""

# name: (the program, fills of records)
CASES = {
    "served in the batch": ("serve([problem(4, 4, 2), problem(3, 4, 1)], large_items=1e9)", 4),
    "served alone": ("serve([problem(5, 4, 2)], large_items=1.0)", 2),
    "served alone, level launches": ("serve([problem(16, 4, 8)], large_items=1.0)", 2),
    "served in the large batch, level launches":
        ("serve([problem(24, 4, 8)], large_items=1.0, large_batched=True)", 2),
    "batch by chains": ("batch([sweeper(5, 4, 2), sweeper(4, 6, 1)], 'mixed')", 4),
    "batch by level launches": ("batch([sweeper(24, 4, 8)], 'mixed')", 2),
    "solved alone, then in a batch": ("s = sweeper(5, 4, 2); s.solve('mixed', iter_max=50, err_max=1e-8); "
                                      "batch([s], 'mixed')", 2),
    "applied and swept in turn": ("s = sweeper(15, 8, 2, False)\n"  # 166 MB: swept in chunks
                                  "from torch import zeros; x = zeros(s.phi_shape, dtype=float, device='cuda')\n"
                                  "psi = np.empty(s.psi_shape)\n"
                                  "for _ in range(3): s.apply(x, x.clone()); s.sweep(psi, psi * 0 + 1)", 1),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_records_are_filled_once(built, case):
    program, fills = CASES[case]
    env = dict(os.environ, TYCHO_TRACE="1")
    r = subprocess.run([sys.executable, "-c", PRELUDE + program], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stderr.count("[tycho] sweeper.records ") == fills
