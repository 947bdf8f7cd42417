"""CPU check of the fused coarse cycle's fit test (coarse_cycle_bytes, k2_coarse.cu): a level of any
size gets its true byte count or one beyond the shared-memory limit, also where the counts pass
2^31 and 2^32."""
import os
import subprocess

import pytest

from cedar_b200 import _lib, build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdlib>
#include "kernels2d.cuh"
using namespace cdrgpu;
template <typename T> static unsigned long long bytes(int nx, int ny, int nl, int relax, int ns)
{
	CoarseCycle<T> cc;
	cc.nl = nl;
	cc.relax = relax;
	for (int l = 0; l < nl; ++l) {
		cc.lv[l].nx = nx; cc.lv[l].ny = ny; cc.lv[l].ns = ns;
		cc.lv[l].pitch = (nx + 2 + 31) / 32 * 32; cc.lv[l].tpitch = (ny + 2 + 31) / 32 * 32;
		nx = (nx - 1) / 2 + 1; ny = (ny - 1) / 2 + 1;
	}
	return coarse_cycle_bytes<T>(cc);
}
int main(int n, char **a)
{
	const int nx = atoi(a[2]), ny = atoi(a[3]), nl = atoi(a[4]), relax = atoi(a[5]), ns = n > 6 ? atoi(a[6]) : 5;
	printf("%llu %llu\n", a[1][0] == 'd' ? bytes<double>(nx, ny, nl, relax, ns) : bytes<float>(nx, ny, nl, relax, ns),
	       (unsigned long long)kCoarseSmemMax);
	return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    build.build()
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(PROGRAM)
    exe = str(d / "plan")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "cedar_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(cuda, "include"), str(d / "plan.cpp"), "-o", exe, _lib.LIB_PATH,
                    "-Wl,-rpath," + os.path.dirname(_lib.LIB_PATH)], check=True)

    def run(prec, *numbers):
        out = subprocess.run([exe, prec] + [str(v) for v in numbers], capture_output=True, text=True,
                             check=True).stdout.split()
        return int(out[0]), int(out[1])
    return run


def wanted(prec, nx, ny, nl, relax):
    """Bytes of the levels' arrays with rows of nx + 2, and the coarsest solve's factor and vector."""
    size = 8 if prec == "d" else 4
    sor, sory = {0: (1, 0), 1: (2, 0), 2: (0, 2), 3: (2, 2)}[relax]
    n, lines = 0, 0
    for l in range(nl):
        last = l == nl - 1
        planes = 2 if l else 1  # x, b (the first level's b is staged, counted below)
        planes += 1 if l == 0 else 8
        if not last:
            planes += 1 + 5 + sor + sory
            if prec == "d" or max(nx, ny) > 64:
                lines = max(lines, (ny + 1) // 2 * nx, (nx + 1) // 2 * ny)
        n += planes * (nx + 2) * (ny + 2)
        cg = (nx * ny + (nx + 2) * nx * ny) * 8
        nx, ny = (nx - 1) // 2 + 1, (ny - 1) // 2 + 1
    return -(-(n + lines) * size // 8) * 8 + cg


@pytest.mark.parametrize("relax", [0, 1, 2, 3])
@pytest.mark.parametrize("prec", ["d", "f"])
def test_fit_test_of_any_size(program, prec, relax):
    sizes = [(31, 31, 4), (63, 50, 5), (64, 64, 7), (100, 7, 3), (128, 128, 6), (2047, 2047, 7), (70000, 9, 3)]
    # levels whose bytes end just past a multiple of 2^31 or 2^32
    for total in (2 ** 31, 2 ** 32, 2 ** 33):
        lo, hi = 64, 2 ** 28
        while lo < hi:
            mid = (lo + hi) // 2
            cut = (62, mid, 7, relax)
            lo, hi = (mid + 1, hi) if wanted(prec, *cut) < total else (lo, mid)
        sizes += [(62, lo, 7), (62, lo + 1, 7)]
    for nx, ny, nl in sizes:
        got, limit = program(prec, nx, ny, nl, relax)
        want = wanted(prec, nx, ny, nl, relax)
        assert got == want if want <= limit else got > limit, (nx, ny, nl, got, want)


def test_more_planes_than_the_table(program):
    """A hierarchy with more planes to stage than the launch's table holds does not fit, however small."""
    got, limit = program("f", 20, 20, 5, 3, 5)
    assert got <= limit
    got, limit = program("f", 20, 20, 5, 3, 30)  # 4 levels of 30 + 4 planes, 4 of 8, and b
    assert got > limit
