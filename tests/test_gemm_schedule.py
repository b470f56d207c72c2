"""The GEMM kernels' tile scheduler (csrc/gemm_schedule.cuh, host/device code) on the host:
every element of C is produced exactly once for many shapes and both tile sizes
(tests/native/gemm_schedule_check.cc)."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_work_items_partition_the_output(tmp_path):
    exe = str(tmp_path / "sched")
    build = subprocess.run(["g++", "-std=c++17", "-O2", "-I",
                            os.path.join(ROOT, "bitscom_b200", "csrc"),
                            os.path.join(ROOT, "tests", "native", "gemm_schedule_check.cc"),
                            "-o", exe], capture_output=True, text=True, timeout=300)
    assert build.returncode == 0, build.stderr[-3000:]
    run = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stderr[-2000:]
    assert run.stdout.startswith("ok:")


def test_plan_of_every_shape_can_be_launched():
    """The rule that picks a kernel by shape: a share of K never exceeds the k-blocks, the
    workspace of shared-out products stays small, and a capped grid never takes them."""
    import random

    from bitscom_b200.ops import gemm as G

    for empty in ((0, 8, 64), (8, 0, 64), (8, 8, 0)):  # nothing to do, but not refused
        assert G._plan(*empty) >= 0
    rng = random.Random(5)
    for _ in range(2000):
        M, N, K = (rng.choice([1, 7, 64, 77, 128, 200, 577, 1000, 4096, 8192, 50432])
                   for _ in range(3))
        N = -(-N // 8) * 8
        for a_mn in (False, True):
            plan = G._plan(M, N, K, a_mn)
            assert -1 <= plan <= 8
            if plan >= 1:
                assert plan <= -(-K // 64)
                assert plan * -(-M // 128) * 128 * N * 4 <= 80 << 20 or plan == 1
            assert G._plan(M, N, K, a_mn, 1) == 0
            assert G._plan(M, N, K, a_mn, 64) in (-1, 0)
