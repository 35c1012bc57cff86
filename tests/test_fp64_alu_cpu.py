"""fp64_alu.cuh compiled for the host: products, squares, quotients and square
roots have to be the IEEE results bit for bit (estimates moved by -3 to +3
units, as the GPU's may be), the sine within half a unit of the result plus
2^-59 (its method's absolute error), and operands outside the functions' range
have to be refused."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_integer_unit_functions_against_ieee(tmp_path):
    exe = tmp_path / "fp64_alu"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-Wextra", "-Werror",
                        "-I", str(ROOT / "titan_gb300" / "csrc"), str(ROOT / "tests" / "cpp" / "fp64_alu.cpp"),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), "2000000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    lines = {k: (int(n), int(bad)) for k, n, bad in (x.split() for x in r.stdout.splitlines())}
    assert set(lines) == {"product", "square", "quotient", "root", "sine", "refused", "taken"}
    assert lines["sine"][0] > 1900000
    assert all(bad == 0 for _, bad in lines.values()), r.stdout
