"""The fixed-point arithmetic of the FP64 hopping term (grid_gb300/csrc/gb_fx64.cuh), built for
the host with g++ (tests/cpp/test_fx64.cpp): conversions and limbs, the dot product at its
overflow bounds, and a site's error against long double, below the same site in double."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_fx64_arithmetic_on_the_host(tmp_path):
    exe = tmp_path / "test_fx64"
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-ffp-contract=off",
                    f"-I{ROOT / 'grid_gb300' / 'csrc'}", str(ROOT / "tests" / "cpp" / "test_fx64.cpp"), "-o",
                    str(exe)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "PASSED" in r.stdout
