"""The index arithmetic of the row-pair kernels and the index-checked build's
answer to a bad index, on the CPU: a host program over hpcg_b200/csrc/pairs.cuh.

Good pairs: every row is taken once, and no access of a pair leaves its vector.
Bad ones (rows, storage rows and line offsets moved by every small amount): what
the checks let pass reads and writes inside the vector only, and a two-element
access only at an even element; a row that they redirect does too.
"""
import os
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "pairs.cuh"
#include <cstdio>
#include <cstdlib>
#include <vector>
using namespace hpcgx;

static void need(bool ok, const char *what) {
  if (!ok) { std::printf("%s\n", what); std::exit(1); }
}

// What the kernels access of a pair's own line: x[2i-1 .. 2i+2] as far as it
// exists, and both rows of r, x and y in one access where vec.
static bool own_ok(const LevelMat<double> &A, const PairId &id, bool vec) {
  const int64_t lo = id.row - (id.left ? 1 : 0);
  const int64_t hi = id.row + (id.right ? 2 : id.odd || vec ? 1 : 0);
  return lo >= 0 && hi < A.n && !(vec && (id.row & 1)) && id.ke >= 0 && id.ke < A.srows &&
         id.ko >= 0 && id.ko < A.srows;
}
// What load_line accesses of line l.
static bool line_ok(const LevelMat<double> &A, const PairId &id, bool vec, int l) {
  const int64_t at = id.row + A.off[3 * l + 1];
  auto in = [&](int64_t i) { return i >= A.lo && i < (int64_t)A.lo + A.span; };
  if (id.left && !in(at - 1)) return false;
  if (!in(at) || ((vec || id.odd) && !in(at + 1))) return false;
  if (id.right && !in(at + 2)) return false;
  return !(vec && (at & 1));
}

int main(int, char **argv) {
  const int nx = std::atoi(argv[1]), ny = std::atoi(argv[2]), nz = std::atoi(argv[3]);
  const int zlo = std::atoi(argv[4]), zhi = std::atoi(argv[5]);
  LevelMat<double> A = {};
  A.nx = nx; A.ny = ny; A.nz = nz;
  A.n = (int64_t)nx * ny * nz;
  A.zlo = zlo; A.zhi = zhi;
  A.lo = zlo ? -nx * ny : 0;
  A.span = (int)A.n - A.lo + (zhi ? nx * ny : 0);
  for (int s = 0; s < 27; ++s)
    A.off[s] = (s / 9 - 1) * nx * ny + ((s / 3) % 3 - 1) * nx + (s % 3 - 1);
  ClassInfo cls[4];
  for (int q = 0; q < 4; ++q) {
    ClassInfo &C = cls[q];
    C.q = q; C.py = q & 1; C.pz = q >> 1;
    C.nyq = (ny - C.py + 1) / 2;
    C.lines = C.nyq * ((nz - C.pz + 1) / 2);
    for (int px = 0; px < 2; ++px) {
      C.len[px] = (nx - px + 1) / 2;
      C.start[px] = A.srows;
      A.srows += ((int64_t)C.lines * C.len[px] + 31) / 32 * 32;
    }
    C.dlen = make_fastdiv((uint32_t)C.len[0]);
    C.dnyq = make_fastdiv((uint32_t)C.nyq);
  }
  const int vecs = nx % 2 == 0 ? 2 : 1;   // two-element accesses need even lines
  std::vector<int> taken(A.n);
  long passed = 0, refused = 0;
  for (const ClassInfo &C : cls)
    for (int t = 0; t < C.lines * C.len[0]; ++t) {
      const PairId id = pair_at(A, C, 0, t);
      need(pair_inside(A, id), "a good pair is refused");
      ++taken[id.row];
      if (id.odd) ++taken[id.row + 1];
      for (int vec = 0; vec < vecs; ++vec) {
        need(own_ok(A, id, vec), "a good pair leaves its vector");
        for (int l = 0; l < 9; ++l)
          if (has_line(id, l)) {
            need(line_inside(A, id, vec, l), "a good line is refused");
            need(line_ok(A, id, vec, l), "a good line leaves its vector");
          }
      }
      // bad rows and storage rows: an error of the index arithmetic moves a row
      // by whole pairs where lines are even
      for (int64_t d = -A.n - 4; d <= A.n + 4; ++d)
        for (int vec = 0; vec < vecs; ++vec) {
          PairId bad = id;
          bad.row += vec ? 2 * d : d;
          if (d % 3 == 0) bad.ke += d;
          if (d % 3 == 1) bad.ko += d;
          if (!pair_inside(A, bad)) { redirect(bad); ++refused; }
          need(own_ok(A, bad, vec), "a bad pair leaves its vector");
          for (int l = 0; l < 9; ++l) {
            LevelMat<double> B = A;
            B.off[3 * l + 1] += (int)d;
            if (!line_inside(B, bad, vec, l)) { ++refused; continue; }
            need(line_ok(B, bad, vec, l), "a bad line leaves its vector");
            ++passed;
          }
        }
    }
  for (int k : taken) need(k == 1, "a row is not taken once");
  need(passed > 0 && refused > 0, "nothing was checked");
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from hpcg_b200 import build
    d = tmp_path_factory.mktemp("pairs")
    src, exe = d / "pairs.cu", d / "pairs"
    src.write_text(PROGRAM)
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-I", os.path.join(ROOT, "hpcg_b200", "csrc"),
                    "-o", str(exe), str(src)], check=True)
    return str(exe)


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 1), (3, 1, 1), (1, 2, 3), (2, 2, 2), (4, 2, 2),
                                  (5, 3, 3), (6, 4, 5), (9, 7, 5), (8, 8, 8)])
@pytest.mark.parametrize("halo", [(0, 0), (1, 0), (1, 1)])
def test_pairs_stay_inside(program, dims, halo):
    r = subprocess.run([program, *map(str, dims + halo)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
