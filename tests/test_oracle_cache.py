"""The oracle's cached colour gradient where ghost layers hold interface nodes: the stencil of a ghost node
reaches outside the arrays, so the cache is filled at fluid nodes alone.  The oracle is built with checked
vector indices and run in a child process, which a read outside ends."""
import os
import subprocess
import sys

import numpy as np

import mbcg
import oracle_lib as ol


def _check(lib):
    p = mbcg.rti_params(24, 22, q=27)
    p.bc[0], p.bc[2] = mbcg.BC_WALL, mbcg.BC_PERIODIC
    p.rti_position, p.rti_amplitude = 3.0, 4.0  # through both ends of the periodic axes
    a = ol.oracle_init(p, np.float64)
    assert (a[0, 0] * a[1, 0] > 1e-3).any()
    ol._oracle = None
    ol.build_oracle = lambda: lib
    out = [ol.oracle_step(p, a, 1, reference_cost=c)[:, 1:-1, 1:-1, 1:-1] for c in (False, True)]
    assert np.isfinite(out[0]).all()
    np.testing.assert_array_equal(out[0], out[1])


def test_cached_gradient_with_interface_nodes_in_ghost_layers(tmp_path):
    lib = str(tmp_path / "liboracle_checked.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-fopenmp", "-D_GLIBCXX_ASSERTIONS",
                    "-I", os.path.join(ol.ORACLE_DIR, "..", "include"), os.path.join(ol.ORACLE_DIR, "mbcg_oracle.cpp"),
                    "-o", lib], check=True)
    r = subprocess.run([sys.executable, "-c", f"import sys; sys.path[:] = {sys.path!r}; "
                        f"import test_oracle_cache as t; t._check({lib!r})"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
