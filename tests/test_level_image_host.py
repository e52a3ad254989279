"""Host rules of a level's neighbourhood image, checked on the CPU: ImageShape,
image_run, row_part, src_index and outside_taps are taken verbatim from
libapr_b200/csrc/filter.cu and compiled with g++.  The image of a run, its halo
planes included, takes at most 1 GiB, or a tile's eight planes and their halo
where those are more; runs are whole tiles; in place, one run has all planes.
Parts of a row are whole steps that cover it.  The taps whose reflection leaves a
level are as many for each of its cells as the count says."""
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

MAIN = r"""
template <int R, typename T>
static long check(int xn, int yn, int zn) {
    const LD d{yn, xn, zn};
    long bad = image_run<R, T>(d, true) != zn;
    const int run = image_run<R, T>(d, false);
    bad += run < 1 || run > zn || (run < zn && run % kTZ != 0);
    const uint64_t bytes = ImageShape<R, T>(d, 0, run).elems() * sizeof(T);
    const uint64_t least = ImageShape<R, T>(d, 0, std::min(zn, kTZ)).elems() * sizeof(T);
    bad += bytes > std::max(uint64_t(1) << 30, least);
    // as many planes as the bound allows
    if (run < zn)
        bad += ImageShape<R, T>(d, 0, std::min(zn, run + kTZ)).elems() * sizeof(T) <= (uint64_t(1) << 30);
    if (bad) std::printf("R %d, %zu bytes: %d x %d x %d, run %d\n", R, sizeof(T), zn, xn, yn, run);
    return bad;
}

static long check_outside(int R, int zn, int xn, int yn) {
    const int S = 2 * R + 1;
    const LD d{yn, xn, zn};
    const uint64_t count = outside_taps(d, R);
    long bad = 0;
    for (int z = 0; z < zn; ++z)
        for (int x = 0; x < xn; ++x)
            for (int y = 0; y < yn; ++y) {
                uint64_t n = 0;
                for (int k = 0; k < S * S * S; ++k)
                    n += src_index(z + k / (S * S) - R, zn, 1) < 0 || src_index(x + k / S % S - R, xn, 1) < 0 ||
                         src_index(y + k % S - R, yn, 1) < 0;
                bad += n != count;
            }
    return bad;
}

static long check_part(uint64_t rows, int n, int step, uint64_t warps) {
    const int per = row_part(rows, n, step, warps);
    const uint64_t parts = (uint64_t)((n + per - 1) / per);
    return per % step != 0 || per < step || (rows >= warps && parts != 1) ||
           (rows * parts < warps && per != step) || parts > 65535;
}

int main() {
    long bad = 0;
    for (int zn = 1; zn < 6; ++zn)
        for (int xn = 1; xn < 6; ++xn)
            for (int yn = 1; yn < 6; ++yn) bad += check_outside(1, zn, xn, yn) + check_outside(2, zn, xn, yn);
    for (uint64_t rows : {1, 2, 7, 100, 1000, 4735, 4736, 5919, 5920, 100000})
        for (int n : {1, 2, 3, 31, 33, 255, 256, 257, 2047, 2048, 2049, 65535})
            bad += check_part(rows, n, 2, 148 * 8) + check_part(rows, n, 256, 148 * 40);
    for (int side : {1, 3, 100, 1000, 2048, 2900, 3400, 4096, 5800, 8192, 16384, 65535})
        for (int yn : {side, side / 2 + 1})
            for (int zn : {1, 7, 8, 9, 23, 24, 64, 67, 512, 2000, 65535}) {
                bad += check<1, float>(side, yn, zn) + check<2, float>(side, yn, zn);
                bad += check<1, double>(side, yn, zn) + check<2, double>(side, yn, zn);
            }
    std::printf("faults %ld\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_image_runs_keep_their_bound(tmp_path):
    with open(os.path.join(ROOT, "libapr_b200", "csrc", "filter.cu")) as f:
        src = f.read()

    def block(start, end="\n}\n"):
        a = src.index(start)
        return src[a:src.index(end, a) + len(end)]

    body = "".join([block("struct LD {", "};\n"), block("template <int R, typename T>\nstruct ImageShape {", "\n};\n"),
                    block("constexpr int kTX", "\n"), block("__host__ __device__ __forceinline__ int src_index("),
                    block("template <int R, typename T>\nint image_run("), block("int row_part("),
                    block("uint64_t outside_taps(")])
    text = ("#include <algorithm>\n#include <cstdint>\n#include <cstdio>\n#define __host__\n#define __device__\n"
            "#define __forceinline__ inline\n"
            + body + MAIN)
    path = tmp_path / "image_run.cpp"
    path.write_text(text)
    exe = str(tmp_path / "image_run")
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", exe, str(path)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "faults 0" in r.stdout, r.stdout[-2000:] + r.stderr
