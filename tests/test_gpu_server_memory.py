"""Fetching a served result when device memory is scarce: with room for two dense fields it succeeds, whatever
area a fetch would rather have.  cudaMalloc is made to refuse larger requests, in a child process."""
import os
import subprocess
import sys

import numpy as np
import pytest

import mbcg
from gpu_util import written_nodes

pytestmark = pytest.mark.gpu
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def _check():
    cases = [(mbcg.bubble_params(40, q=19), 3), (mbcg.jet_params(60, 50, 70, q=27, diameter=12.0), 4)]
    with mbcg.Server(arena_bytes=1 << 29, keep_results=1, calibrate=0) as srv:
        ids = [srv.submit(p, n) for p, n in cases]
        for rid in ids:
            assert srv.wait(rid).state == mbcg.REQ_DONE
        for rid, (p, n) in zip(ids, cases):
            field = 4 * p.nx * p.ny * p.nz
            os.environ["MBCG_TEST_MALLOC_LIMIT"] = str(2 * field - 1)
            try:
                srv.fetch(rid, p.shape)
            except mbcg.MbcgError:
                pass
            else:
                raise AssertionError("the preloaded cudaMalloc is not in use")
            os.environ["MBCG_TEST_MALLOC_LIMIT"] = str(2 * field)
            scarce = srv.fetch(rid, p.shape)
            del os.environ["MBCG_TEST_MALLOC_LIMIT"]
            np.testing.assert_array_equal(srv.fetch(rid, p.shape), scarce)
            with mbcg.Case(p) as c:
                c.init()
                c.step(n)
                np.testing.assert_array_equal(c.copy_out()[written_nodes(p)], scarce[written_nodes(p)])


def test_fetch_with_room_for_two_fields(tmp_path):
    shim = str(tmp_path / "fail_malloc.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", f"-I{CUDA}/include",
                    os.path.join(os.path.dirname(__file__), "cpp", "fail_malloc.cpp"), "-o", shim, f"-L{CUDA}/lib64",
                    "-Wl,--no-as-needed", "-lcudart", f"-Wl,-rpath,{CUDA}/lib64", "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", f"import sys; sys.path[:] = {sys.path!r}; "
                        "import test_gpu_server_memory as t; t._check()"], capture_output=True, text=True, timeout=600,
                       env={**os.environ, "LD_PRELOAD": shim})
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
