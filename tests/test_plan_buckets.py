"""The clusterizer buckets of a plan, counted and filled strip by strip on the
planning threads, equal buckets filled node by node in index order (built for
the host by tests/cpp/plan_buckets_check.cpp)."""

import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.parametrize("threads", [1, 8])
def test_buckets_in_index_order(tmp_path, threads):
    out = str(tmp_path / "plan_buckets_check.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-pthread", "-o", out,
                    "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "cpp", "plan_buckets_check.cpp"),
                    os.path.join(ROOT, "hpgl_b200", "csrc", "plan.cpp"),
                    os.path.join(ROOT, "hpgl_b200", "csrc", "task_pool.cpp")], check=True, capture_output=True)
    assert C.CDLL(out).pbc_run(5 + threads, 120, threads) == 0
