"""Which graphs' lists are walked 32 to a row: those whose row positions and sums a 32-bit integer holds."""
import os
import subprocess

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rows_of_the_longest_lists_are_exact(tmp_path):
    src, exe = tmp_path / "rows.cpp", tmp_path / "rows"
    src.write_text('#include "pm_common.h"\nint main(int, char** v) { return pm::rows_of_lists(atoi(v[1])) ? 1 : 0; }\n')
    subprocess.run(["g++", "-std=c++17", "-include", "cstdlib", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "pumatch_b200", "csrc"), "-o", str(exe), str(src)], check=True)

    def rows(maxdeg):
        return subprocess.run([str(exe), str(maxdeg)]).returncode == 1

    assert rows(0) and rows(5214) and rows(10_000_000)
    longest = max(d for k in range(8, 31) for d in (2**k - 1, 2**k, 2**k + 1) if rows(d))
    ends = np.cumsum(np.full(32, longest, dtype=np.int32), dtype=np.int32)  # as the kernel's scan adds them
    assert np.array_equal(ends, np.arange(1, 33, dtype=np.int64) * longest)
    assert np.int64(2) * 3 * longest <= np.iinfo(np.int32).max
    assert not rows(2**26) and not rows(2**31 - 2)
