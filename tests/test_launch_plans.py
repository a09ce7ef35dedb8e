"""The planning functions of the library's boundary on the CPU (tests/cpp/launch_plans.cu)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launch_plans(tmp_path):
    exe = tmp_path / "launch_plans"
    # the launchers it never calls stay unresolved
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", "launch_plans.cu"), "-cudart", "static",
                    "-Xlinker", "--unresolved-symbols=ignore-all"], check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
