"""The counts of a launch's calls at the ends of their range.

A launch may be 2^31 - 1 iterations long; counts next to that are checked on
the host, through the functions that the kernels call.
"""
import ctypes as C
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TOP = 2 ** 31 - 1


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    d = tmp_path_factory.mktemp("counts")
    (d / "counts.c").write_text('''#include "xw_layout.h"
int32_t launch_calls(uint64_t iters) { return xw_launch_calls(iters); }
int32_t event_after(int32_t event, int32_t k) { return xw_event_after(event, k); }
int32_t calls_to(int32_t k, int32_t most, int32_t k_end) { return xw_calls_to(k, most, k_end); }
''')
    subprocess.run(["gcc", "-std=c11", "-O1", "-fwrapv", "-shared", "-fPIC",
                    "-I" + os.path.join(REPO, "xtax_b200", "csrc"), str(d / "counts.c"), "-o", str(d / "counts.so")],
                   check=True)
    L = C.CDLL(str(d / "counts.so"))
    L.launch_calls.argtypes = [C.c_uint64]
    return L


@pytest.mark.parametrize("iters", [0, 1, 4096, TOP - 2, TOP - 1, TOP])
def test_a_launch_makes_all_its_calls(counts, iters):
    assert counts.launch_calls(iters) == iters


@pytest.mark.parametrize("k", [0, 1, 62, 63, 64, TOP - 65, TOP - 64, TOP - 63, TOP - 2, TOP - 1, TOP])
def test_counts_stay_in_range(counts, k):
    for event in (-5, 0, 1, k - 1, k, min(k + 1, TOP), min(k + 2, TOP), TOP):
        assert counts.event_after(event, k) == min(max(event, k + 1), TOP)
    for most in (1, 64):
        for k_end in (k, min(k + 1, TOP), min(k + 63, TOP), min(k + 64, TOP), TOP):
            assert counts.calls_to(k, most, k_end) == min(k + most, k_end)
