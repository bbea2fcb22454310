"""FP32 SRT: the velocity error of the library's update over a run is no larger
than that of the plain order of operations with fused multiply-adds (both on the
host, against FP64)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "nflow-red-poplar_b200", "csrc")


def test_velocity_error_of_a_run(tmp_path):
    exe = str(tmp_path / "srt")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2",
                    "--expt-relaxed-constexpr", "-Xcompiler", "-ffp-contract=off,-mfma", "-I", CSRC,
                    "-o", exe, os.path.join(HERE, "native", "srt_update.cu")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout
    rows = [tuple(map(float, line.split())) for line in out.splitlines()]
    assert len(rows) == 4
    for tau, library, plain in rows:
        assert library <= plain, (tau, library, plain)
