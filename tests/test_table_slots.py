"""Sizes of the global hash tables of long contraction rows (host code, no GPU)."""
import os
import shutil
import subprocess

import pytest

from pennsylvaniagpugraphclustering_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(not (shutil.which("nvcc") or os.path.exists("/usr/local/cuda/bin/nvcc")), reason="no nvcc")
def test_slots_hold_the_keys_and_stay_below_2_30(tmp_path):
    exe = tmp_path / "table_slots"
    subprocess.run([build._nvcc(), *build.ARCH_FLAGS, "-std=c++17", "--expt-relaxed-constexpr", "-ccbin",
                    build._host_cxx(), "-I", build.CSRC, "-I", build.INCLUDE,
                    os.path.join(ROOT, "tests", "native", "table_slots.cu"), "-o", str(exe)], check=True)
    keys = [0, 1, 16, 17, 16384, 16385, (1 << 29) - 1, 1 << 29, (1 << 29) + 1, 1 << 30, (1 << 30) + 1, (1 << 31) - 2]
    out = subprocess.run([str(exe), *map(str, keys)], check=True, capture_output=True, text=True)
    slots = [int(x) for x in out.stdout.split()]
    for k, s in zip(keys, slots):
        assert s & (s - 1) == 0 and 32 <= s <= 1 << 30
        assert s == 1 << 30 or 2 * k <= s < max(4 * k, 33)
