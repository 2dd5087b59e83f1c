"""Which join outputs of a wave are placed in a region: those that fit it one
after the other, and none of more rows than 32-bit offsets hold (nor what
follows it), however large the region is."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
HUGE = 1 << 50


@pytest.fixture(scope="module")
def place_check(built, tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ is missing")
    exe = str(tmp_path_factory.mktemp("place") / "place_check")
    lib = os.path.join(ROOT, "vedas_gb300")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(CUDA, "include"),
                    "-I" + os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "place_check.cpp"),
                    "-L" + lib, "-l:libvedas_gb300.so", "-Wl,-rpath," + lib, "-L" + os.path.join(CUDA, "lib64"),
                    "-lcudart_static", "-ldl", "-lrt", "-o", exe], check=True)

    def run(region_bytes, *totals):
        r = subprocess.run([exe, str(region_bytes)] + [str(t) for t in totals], capture_output=True, text=True,
                           check=True)
        placed, bump, blocks = r.stdout.split()
        return placed, int(bump), int(blocks)

    return run


@pytest.mark.parametrize("region,totals,placed", [
    (HUGE, (10, 0, 5), "101"),
    (512 + 2 * 512, (1, 64), "11"), (512 + 2 * 512, (1, 65), "10"), (512 + 2 * 512, (65, 1, 0, 1), "1000"),
    (HUGE, ((1 << 32) - 1, 7), "11"),
    (HUGE, (1 << 32, 7), "00"), (HUGE, (3, 1 << 32, 0, 7), "1000"), (HUGE, ((1 << 32) + 1, 1 << 33), "00"),
    (HUGE, ((1 << 62) + 1,), "0"),   # (its bytes wrap to a small number)
])
def test_placed_outputs(place_check, region, totals, placed):
    got, bump, blocks = place_check(region, *totals)
    assert got == placed
    rows = [t for t, p in zip(totals, placed) if p == "1"]
    assert bump == 512 + sum(2 * ((4 * t + 255) // 256 * 256) for t in rows)
    assert blocks == 2 * len(rows)
