"""The server's planner on the CPU: the cut that building, sorting and scheduling every cut's tiles would give,
without building those that cannot be the best (the server plans with its lock held)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lightweight-mb-color-gradient-lbm_gb300", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "plan_check")
    subprocess.run([NVCC, "-O2", "-std=c++17", "-x", "cu", f"-I{CSRC}", f"-I{ROOT}/include",
                    os.path.join(ROOT, "tests", "cpp", "plan_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.fixture(scope="module")
def plans(exe):
    r = subprocess.run([exe, "7", "150"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-500:]
    return [[float(v) for v in line.split()] for line in r.stdout.split("\n") if line]


def test_same_cut_as_building_every_one(plans):
    assert len(plans) == 150
    # cuts within 0.1 % of each other count as equal
    assert all(c == b or ct <= bt / 0.999 for c, b, ct, bt, *_ in plans)
    assert sum(c == b for c, b, *_ in plans) >= 148


def test_tiles_built(plans):
    # 64 lattices of 192^3: no thin cut is built
    chosen, _, _, _, built, ntiles, all_ = plans[0]
    assert built <= 6 * ntiles and built <= 0.05 * all_
    # and never more than every cut's and the chosen one's again
    assert all(p[4] <= p[6] + p[5] for p in plans)


def test_long_lattices_are_covered(exe):
    """A tile's index along z has 16 bits: lattices of up to 524,280 fluid planes are accepted."""
    r = subprocess.run([exe, "cover"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
