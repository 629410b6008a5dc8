"""The way out of a tile kernel that gave up waits for the copies still in flight (csrc/kdnn_ring.cuh), on a host model."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_ring_drain_waits_for_the_last_copy(tmp_path):
    exe = str(tmp_path / "ring_drain_test")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-x", "c++", os.path.join(ROOT, "tests", "cpp", "ring_drain_test.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout


def test_kernels_drain_by_recorded_parity():
    """Both tcgen05 kernels use it, behind the barrier where all roles meet, and no copy is waited for by either parity."""
    for name in ("kdnn_tc.cuh", "kdnn_split.cuh"):
        src = open(os.path.join(ROOT, "dnn-for-kokkos_b200", "csrc", name)).read()
        assert src.count("ring_drain(") == 1 and src.count("ring.arm(") == 1
        assert "0u) || mbar_try_wait" not in src
        end = src[src.index("peer_out_finish(p.po, gridDim.x)"):]
        assert end.index("__syncthreads()") < end.index("ring_drain(") < end.index("tcgen05.dealloc")
