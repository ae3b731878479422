"""Rules of the library's host side that decide which kernel a call may take (csrc/launch_rules.h), on
the CPU: a small C++ program built from the header evaluates them at sizes that no test machine
holds."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pasc_inference_gb300", "csrc")


def _run(tmp_path, body):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "rules.cpp", tmp_path / "rules"
    src.write_text('#include "launch_rules.h"\n#include <stdio.h>\nusing namespace pasc;\n' + body)
    subprocess.check_call([gxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)])
    return subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()


INT_MAX, UINT_MAX = 2**31 - 1, 2**32 - 1
FEM = [(10, 1, 1), (2_000_000, 200_000, 3), (INT_MAX - 256, 1, 1), (INT_MAX - 256, INT_MAX - 256, 1), (INT_MAX - 255, 1, 1),
       (INT_MAX, 10, 1), (2**31, 2**30, 1), (3 * 10**9, 3 * 10**8, 1), (6 * 10**8, 536_870_879, 8), (6 * 10**8, 536_870_880, 8),
       (6 * 10**8, 6 * 10**8, 8)]


def test_fem_sum_index_range(tmp_path):
    """Accepted exactly where no index of the kernels leaves its type: every fine timestep a thread
    forms (the last block's surplus threads included) fits an int, every coarse entry an unsigned int."""
    calls = "".join(f'printf("%d\\n", (int)fem_sum_indexable({a}L, {b}L, {k}));' for a, b, k in FEM)
    got = [int(v) for v in _run(tmp_path, "int main() {" + calls + "}")]

    def last_thread(n):  # largest index a launch over n items forms
        return (n + 255) // 256 * 256 - 1

    for (T1, T2, K), ok in zip(FEM, got):
        # in range: copy's and bounds' threads and the loop bounds T1, the residual's threads, the field's entries
        fits = max(last_thread(T1), last_thread(T2 + 1), T1) <= INT_MAX and last_thread(T2 * K) <= UINT_MAX
        assert not ok or fits, (T1, T2, K)
        if max(T1, T2 * K) <= 10**9:  # nothing ordinary is refused
            assert ok, (T1, T2, K)
    assert got == [1, 1, 1, 1, 0, 0, 0, 0, 1, 0, 0]


TAGS = r"""
int main()
{
    // adjoint solves (16384 tags each) and mixed launches of 1 to 4097: past 2^32 tags several times
    const unsigned int steps[] = {16384u, 4097u * 1021u, 1u << 31};
    for (unsigned int step : steps) {
        WordTags t;
        unsigned long long last = 0, cleared = 0, launches = 0;
        for (unsigned long long given = 0; given < 3ull << 32; launches++) {
            const unsigned int n = step > 65536 ? step : step - (unsigned int)(launches % 3);
            unsigned int first = 0;
            if (t.take(n, &first)) {
                cleared++;
                last = 0;
            }
            // above every tag since the buffer was cleared, never 0, no wrap inside the launch
            if (first <= last || (unsigned long long)first + n - 1 > UINT_MAX) return 1;
            last = (unsigned long long)first + n - 1;
            given += n;
        }
        printf("%llu\n", cleared);
    }
}
"""


def test_word_tags_never_repeat(tmp_path):
    assert [int(v) >= 2 for v in _run(tmp_path, TAGS)] == [True] * 3
