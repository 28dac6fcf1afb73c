"""The launch shapes of the persistent loops (loop_shape.h), on the CPU.

Over all block sizes and face counts the form chosen is the first that fits, two
of its blocks share an SM, and no block size gets the form with the normals in
global memory where the one without would fit.  The loops are taken where they
were measured faster than the kernels, by the sectors a warp's neighbour reads
touch; that count separates the kinds of mesh the rule names."""
import os
import shutil
import subprocess

import pytest

from graphite_b200 import meshgen

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "graphite_b200", "csrc")
SHAPES = r"""
#include "loop_shape.h"
#include <cstdio>
using namespace gb;
int main() {
    for (int faces = 4; faces <= 6; ++faces)
        for (int threads = 64; threads <= 576; threads += 32) {
            const LoopForm f = loop_form(faces, threads);
            std::printf("%d %d %d %d %d %d\n", faces, threads, (int)f, f == LoopForm::kNone ? 0 : loop_smem(f, faces, threads),
                        loop_smem(LoopForm::kWide, faces, threads), loop_smem(LoopForm::kNarrow, faces, threads));
        }
}
"""
RULES = r"""
#include "loop_shape.h"
#include <cstdio>
#include <cstdlib>
using namespace gb;
int main(int, char** a) {
    const int faces = std::atoi(a[1]), threads = std::atoi(a[2]);
    const float sectors = (float)std::atof(a[3]);
    const long long n = std::atoll(a[4]);
    const LoopForm f = loop_form(faces, threads);
    auto show = [](int64_t v) { std::printf("%lld ", v == kLoopNever ? -1LL : (long long)v); };
    show(loop_shortest(f, faces, threads, sectors, false, n));
    show(loop_shortest(f, faces, threads, sectors, true, n));
    show(nsi_loop_shortest(faces, threads, sectors, false, false, n));
    show(nsi_loop_shortest(faces, threads, sectors, true, false, n));
    show(nsi_loop_shortest(faces, threads, sectors, true, true, n));
}
"""
SECTORS = r"""
#include "gb_internal.h"
#include <cstdio>
namespace gb { void set_error(const std::string& s) { std::fprintf(stderr, "%s\n", s.c_str()); } void clear_error() {} }
using namespace gb;
int main(int n, char** path) {
    for (int k = 1; k < n; ++k) {
        ElementSet es;
        Topology t;
        Numbering num;
        if (!parse_su2(path[k], es) || !build_topology(es, t)) return 1;
        number_cells(t, true, num);
        std::printf("%f\n", neighbour_sectors(num));
    }
}
"""
NONE, WIDE, NARROW, LEAN = range(4)
SM_BYTES, RESERVED, STATIC = 228 * 1024, 1024, 3 * 1024      # per SM, per block by the system, per block at most

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


def build(tmp_path, source, *more):
    src, exe = tmp_path / "prog.cpp", tmp_path / "prog"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", os.path.join(ROOT, "include"), str(src), *more, "-o",
                    str(exe), "-lpthread"], check=True)
    return str(exe)


def test_every_shape_gets_the_first_form_that_fits(tmp_path):
    out = subprocess.check_output([build(tmp_path, SHAPES)], text=True)
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    fits = lambda dynamic: 2 * (dynamic + STATIC + RESERVED) <= SM_BYTES
    for faces, threads, form, smem, wide, narrow in rows:
        assert form == NONE or fits(smem), (faces, threads)
        want = (WIDE if threads <= 256 and fits(wide) else NARROW if threads <= 416 and fits(narrow) else
                LEAN if threads <= 512 else NONE)
        assert form == want, (faces, threads, form, want)
    form = {(r[0], r[1]): r[2] for r in rows}
    assert form[5, 224] == WIDE and form[5, 256] == NARROW and form[6, 192] == WIDE and form[6, 224] == NARROW
    assert form[4, 256] == WIDE and form[6, 384] == NARROW and form[6, 416] == LEAN


# (faces, threads, sectors, iterations of the run) -> launch from which Euler, batch, NSI, limited NSI (conditions by
# ghost kernels, inside the gradient pass) take the loop
@pytest.mark.parametrize("case,want", [
    ((4, 64, 103, 1000), [4, 4, 4, 4, 4]), ((4, 256, 110, 1000), [4, 4, 4, 4, 4]), ((4, 352, 110, 1000), [8, -1, 8, 8, -1]),
    ((4, 384, 110, 1000), [-1, -1, 8, 8, -1]), ((4, 512, 110, 1000), [-1, -1, 16, -1, -1]), ((4, 512, 110, 50), [-1, -1, 16, 16, 16]),
    ((5, 64, 50, 1000), [4, 4, 4, 4, 4]), ((5, 192, 50, 1000), [4, 4, 4, 4, 4]), ((5, 224, 50, 1000), [6, 6, 4, 4, 4]),
    ((5, 192, 91, 1000), [6, 6, 4, 4, 4]), ((5, 224, 91, 1000), [8, 8, 4, 4, 4]), ((5, 192, 112, 1000), [8, 8, 4, 4, 4]),
    ((5, 256, 50, 1000), [8, 8, 4, 4, 4]), ((6, 64, 98, 1000), [8, 4, 4, 4, 4]), ((6, 64, 112, 1000), [8, 6, 4, 4, 4]),
    ((5, 256, 91, 1000), [16, 16, 4, 4, 4]), ((5, 416, 50, 1000), [8, 8, 8, 8, 8]), ((5, 416, 91, 1000), [32, 32, 8, 8, -1]),
    ((5, 416, 112, 1000), [-1, -1, 8, -1, -1]), ((5, 480, 50, 1000), [32, -1, 16, 32, 32]), ((5, 480, 80, 1000), [-1, -1, -1, -1, -1]),
    ((6, 192, 66, 1000), [8, 8, 4, 4, 4]), ((6, 192, 98, 1000), [16, 8, 4, 4, 4]), ((6, 192, 112, 1000), [-1, 16, 4, 4, 4]),
    ((6, 256, 66, 1000), [16, 16, 4, 4, 4]), ((6, 352, 98, 1000), [-1, -1, 8, -1, -1]), ((6, 352, 98, 70), [32, -1, 8, -1, -1]),
    ((6, 352, 66, 1000), [16, 16, 8, 24, 24]), ((5, 224, 103, 1000), [16, 16, 4, 4, 4]), ((6, 512, 66, 1000), [32, -1, 16, 32, 32])])
def test_where_the_loops_are_taken(tmp_path, case, want):
    # (whether NSI's block fits its shared memory is asked before)
    out = subprocess.check_output([build(tmp_path, RULES), *map(str, case)], text=True)
    assert list(map(int, out.split())) == want


def test_sectors_separate_the_kinds_of_mesh(tmp_path):
    kinds = {"layer of prisms": (lambda: meshgen.airfoil_2d_prisms(66, 69), (40, 56)),
             "layer of hexes": (lambda: meshgen.cylinder_ogrid(96, 60), (56, 72)),
             "stacked prisms": (lambda: meshgen.channel_bump(40, 25, 8, cells="prism"), (72.01, 94)),
             "wing": (lambda: meshgen.swept_wing(40, 14, 10, 6), (72.01, 94)),
             "hexes": (lambda: meshgen.channel_bump(40, 25, 10, cells="hex"), (94.01, 105)),
             "tets": (lambda: meshgen.channel_bump(24, 15, 6, cells="tet"), (94.01, 128)),
             "pyramids": (lambda: meshgen.channel_bump(24, 15, 6, cells="pyramid"), (94.01, 130)),
             "mix": (lambda: meshgen.channel_bump(30, 15, 8, cells="mixed"), (105.01, 140)),
             "one cell": (lambda: meshgen.channel_bump(1, 1, 1, cells="hex"), (0, 0))}
    paths = []
    for k, (make, _) in enumerate(kinds.values()):
        paths.append(str(tmp_path / f"{k}.su2"))
        make().write_su2(paths[-1])
    exe = build(tmp_path, SECTORS, os.path.join(CSRC, "mesh_build.cpp"))
    got = list(map(float, subprocess.check_output([exe, *paths], text=True).split()))
    for (name, (_, (lo, hi))), s in zip(kinds.items(), got):
        assert lo <= s <= hi, (name, s)
