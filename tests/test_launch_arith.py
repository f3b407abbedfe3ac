"""Launch arithmetic of the kernels at the largest sizes, compiled for the host (CPU only)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "sc2019_md_gb300" / "csrc"


def _run(tmp_path, body):
    if not shutil.which("g++"):
        pytest.skip("needs g++")
    src = tmp_path / "t.cpp"
    src.write_text("#include <cstdio>\n#include <cstdlib>\n#include \"mdrl_internal.h\"\nusing namespace mdrl;\n"
                   "#define CHECK(c) do { if (!(c)) { std::printf(\"%s\\n\", #c); std::exit(1); } } while (0)\n"
                   "int main() {\n" + body + "\nreturn 0; }\n")
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-o", str(exe), str(src)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout


@pytest.mark.parametrize("lanes", [16, 32])
def test_lanes_of_a_particle(tmp_path, lanes):
    """Every lane of the first and last CTA names its particle, past 2^31 threads too."""
    _run(tmp_path, f"""
    const unsigned L = {lanes}, T = 256, per = T / L;
    for (long long n : {{1LL, 1LL << 20, (1LL << 31) / L, (1LL << 31) / L + 1, 1LL << 28, (1LL << 31) - 1}})
        for (long long b : {{0LL, (n - 1) / per / 2, (n - 1) / per}})
            for (unsigned t = 0; t < T; ++t)
                CHECK((long long)lane_particle((unsigned)b, T, t, L) == b * per + t / L);
    """)


def test_blocks_of_a_launch(tmp_path):
    """Up to the largest int: mdrl_pair_eval copies 4 n elements for n up to 2^29 - 1."""
    _run(tmp_path, """
    for (long long n : {0LL, 1LL, 255LL, 256LL, 257LL, 4 * 536870848LL, 4 * 536870849LL, 4 * 536870911LL, (1LL << 31) - 1})
        for (int b : {8, 16, 256})
            CHECK(nblk((int)n, b) == (n + b - 1) / b);
    """)
