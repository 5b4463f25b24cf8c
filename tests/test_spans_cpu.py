"""Address arithmetic of the kernels that copy whole words and vectors (csrc/spans.cuh), compiled for the host: no copy may
reach outside of its array, whatever the array's alignment, and every element has to be reachable."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include "spans.cuh"
#include <cstdio>
#include <initializer_list>
using namespace ftb200;
int main()
{
    long checked = 0;
    for (size_t off = 0; off < 16; off += 2) {
        const size_t t = 0x10000 + off;
        for (int stride : {1, 3, 7, 8, 9, 16, 23, 40, 1237, 2048}) {
            for (int cols : {1, 2, 7, stride - 1, stride}) {
                if (cols < 1 || cols > stride) continue;
                for (int rows : {1, 2, 5, 9, 20}) {
                    const size_t end = t + (size_t)rows * stride * 2;
                    for (int r = 0; r < rows; ++r) {
                        const size_t   row = t + (size_t)r * stride * 2;
                        const RowSpan  S   = row_span(row, cols);
                        const VecRange W   = whole_vectors(rows, stride, r, S.mis, S.nv);
                        if (S.base % 16 != 0 || S.base + 2 * (size_t)S.mis != row) return 1;
                        if (S.mis < 0 || S.mis > 7 || 8 * S.nv < S.mis + cols || 8 * (S.nv - 1) >= S.mis + cols) return 2;
                        if (W.first < 0 || W.first > 1 || W.last < W.first || W.last > S.nv) return 3;
                        if (W.last > W.first && (S.base + 16 * (size_t)W.first < t || S.base + 16 * (size_t)W.last > end)) return 4;
                        // at most the first and the last vector are left to single loads, and only where they reach outside
                        if (W.first == 1 && S.base >= t) return 5;
                        if (W.last < S.nv && W.last >= W.first && S.nv - W.last > 1) return 6;
                        if (W.last == S.nv - 1 && S.nv - 1 > W.first && S.base + 16 * (size_t)S.nv <= end) return 7;
                        ++checked;
                    }
                }
            }
        }
    }
    for (size_t a = 0x2000; a < 0x2004; ++a) {
        for (int n = 1; n < 20; ++n) {
            bool inside = true;
            for (int at = 0; at < n; ++at) {
                const size_t word = (a + at) & ~(size_t)3;
                inside            = inside && word >= a && word + 4 <= a + n;
                const WordSpan W  = word_span(a, n, at);
                if ((a + W.from) % 4 != 0 || W.from > at || W.from + 4 <= at) return 9;
                if (W.bytes == 0 ? W.from >= 0 : W.from < 0 || W.from + W.bytes > n || W.from + W.bytes <= at) return 10;
            }
            if (whole_words(n, a, 0, 0) != inside || whole_words(n, 0, a, 0) != inside || whole_words(n, 0, 0x3000, a) != inside) return 8;
            ++checked;
        }
    }
    std::printf("%ld\n", checked);
    return 0;
}
"""


def test_copies_stay_inside_their_arrays(tmp_path):
    src, exe = tmp_path / "spans.cc", tmp_path / "spans"
    src.write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "fastertransformer_b200", "csrc"), str(src), "-o", str(exe)])
    assert int(subprocess.check_output([str(exe)])) > 1500
