"""The pivot search of the register-window band LU (band_pivot.cuh), its 32 lanes run one beside the other
on the host from the header the kernel includes: whatever the column holds, NaN and infinities among
it, every lane ends with the same candidate, the first row of the largest magnitude that is not a NaN."""
import math
import random
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "strut_b200" / "csrc"

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include "pivot_candidate.cuh"
using namespace strut;
// stdin: columns of 64 entries; stdout: every lane's row and magnitude
int main() {
    double col[64];
    char word[64];
    for (;;) {
        for (int i = 0; i < 64; ++i) {
            if (scanf("%63s", word) != 1) return 0;
            col[i] = strtod(word, nullptr);
        }
        PivotCandidate c[32], o[32];
        for (int l = 0; l < 32; ++l) {
            pivot_offer(c[l], std::fabs(col[l]), l);
            pivot_offer(c[l], std::fabs(col[l + 32]), l + 32);
        }
        for (int m = 16; m > 0; m >>= 1) {
            for (int l = 0; l < 32; ++l) o[l] = c[l];
            for (int l = 0; l < 32; ++l) pivot_merge(c[l], o[l ^ m].v, o[l ^ m].row);
        }
        for (int l = 0; l < 32; ++l) printf("%d %.17g\n", c[l].row, c[l].v);
    }
}
"""


@pytest.fixture(scope="module")
def search(tmp_path_factory):
    d = tmp_path_factory.mktemp("pivot")
    (d / "search.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", str(CSRC), str(d / "search.cpp"), "-o", str(d / "search")])

    def run(columns):
        text = "\n".join(" ".join(repr(v) for v in c) for c in columns)
        out = subprocess.run([str(d / "search")], input=text, capture_output=True, text=True, check=True).stdout.split()
        vals = [(int(out[2 * k]), float(out[2 * k + 1])) for k in range(len(out) // 2)]
        return [vals[32 * k:32 * k + 32] for k in range(len(columns))]

    return run


def test_lanes_agree_on_the_first_largest(search):
    rng = random.Random(7)
    pool = [math.nan, math.inf, -math.inf, 0.0, -0.0, 1e-14, 1.0, -1.0, 2.0, 1e300]
    columns = [[rng.choice(pool) if rng.random() < share else rng.uniform(-2.0, 2.0) for _ in range(64)]
               for share in (0.0, 0.05, 0.3, 0.9) for _ in range(40)]
    columns += [[math.nan] * 64, [math.nan] + [0.5] * 63, [1.0] + [math.nan] * 63, [3.0] * 32 + [math.nan] * 31 + [4.0]]
    for col, lanes in zip(columns, search(columns)):
        finite = [abs(v) for v in col if not math.isnan(v)]
        want = (col.index(next(v for v in col if abs(v) == max(finite))), max(finite)) if finite else (0x7FFFFFFF, -1.0)
        assert lanes == [want] * 32
