"""Index ranges of the cluster, slab and column kernels (csrc/sgh_fold.cuh,
csrc/sgh_volume.cuh) on the CPU, for every shape that the dispatch accepts up to
150 x 150 and for longer axes: each shared array that a pass reads or writes, in
this CTA and in the cluster's others, stays inside its own region; 16-byte
accesses are aligned; regions do not overlap and fit the shared memory; the
float quotients that pick an owner are exact; no bulk copy or fragment read
leaves the packed matrices."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "spectral_galerkin_heat_b200", "csrc")
NVCC = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "sgh_volume.cuh"
using namespace sgh;

static long checks = 0;
static int NX, NY, NN;
#define IN(i, lo, hi) do { const long i_ = (i); ++checks; if (i_ < (long)(lo) || i_ >= (long)(hi)) { \
  std::printf("line %d: %s = %ld outside [%ld, %ld) at %d x %d, %d CTAs\n", __LINE__, #i, i_, (long)(lo), (long)(hi), NX, NY, NN); std::exit(1); } } while (0)
#define OK(x) do { ++checks; if (!(x)) { std::printf("line %d: %s at %d x %d, %d CTAs\n", __LINE__, #x, NX, NY, NN); std::exit(1); } } while (0)

static int up8(int v) { return (v + 7) / 8 * 8; }

// Reads of one folded pass over nvec vectors of N elements at X[k sk + v sv]: vectors up to
// the next multiple of 8, slices clamped to the halves; fragments of the packed matrix.
static void pass(int N, int nvec, long sk, long sv, long lo, long hi) {
  if (nvec <= 0) return;
  const int h = fold::half_up(N), l = N - h, MT = fold::mtiles(N), KS = fold::ksteps(N);
  OK(h >= 1 && l >= (N > 1 ? 1 : 0));
  for (int v : {0, up8(nvec) - 1})
    for (int k : {0, h - 1, h, N - 1, h + (l > 0 ? l - 1 : -1), N - 1 - (h - 1)}) {
      if (k < 0 || k >= N) continue;
      IN(lo + k * sk + v * sv, lo, hi);
    }
  for (int ks = 0; ks < KS; ++ks)
    for (int t = 0; t < 4; ++t)
      for (int d : {0, 4}) {  // clamped slices of fold_mma (each half) and slab_pass
        const int s = 8 * ks + t + d;
        const int e = s < h - 1 ? s : h - 1;
        IN(e, 0, N); IN(N - 1 - e, 0, N);
        if (l > 0) { const int o = s < l - 1 ? s : l - 1; IN(o, 0, N); IN(N - 1 - o, 0, N); IN(h + o, 0, N); }
        else IN(h + (s < -1 ? s : -1), 0, N);
      }
  IN(((long)(MT - 1) * KS + KS - 1) * 256 + 2 * (31 + 96) + 1, 0, fold::pack_doubles(N));
}

// Owner of position p among shares of `share`, as the kernels compute it.
static void owners(int N, int share, int n) {
  const float r = 1.0f / (float)share;
  for (int p = 0; p < N; ++p) {
    const int d = (int)(((float)p + 0.5f) * r);
    OK(d == p / share);
    IN(d, 0, n);
  }
}

template <class W>
static void face(int nx, int ny, int n) {
  NX = nx; NY = ny; NN = n;
  const fold::FaceShape f = fold::face_shape<W>(nx, ny, n);
  if (f.bytes > fold::FACE_SMEM_MAX - 512) return;
  const int XC = (nx + 31) / 32, HC = (fold::half_up(nx) + 31) / 32;
  const long row = (long)f.R * f.ldr;
  const size_t md = 2 * (fold::pack_doubles(nx) + fold::pack_doubles(ny));
  // regions, in their order
  const long o_w = f.keep & fold::FACE_W ? f.o_w : f.bytes / 8;
  const long o_q = f.keep & fold::FACE_Q ? f.o_q : f.bytes / 8, o_m = f.keep & fold::FACE_M ? f.o_m : f.bytes / 8;
  const long e_row = std::min({o_w, o_q, o_m}), e_w = std::min(o_q, o_m), e_q = o_m, e_m = f.bytes / 8;
  OK(row <= f.o_xc && f.o_xc < f.o_xt && f.o_xt < f.o_sig && f.o_sig < f.o_part && f.o_part < f.o_row && f.o_row < e_row + 1);
  for (long o : {(long)f.o_xc, (long)f.o_xt, (long)f.o_sig, (long)f.o_part, (long)f.o_row, o_w, o_q, o_m}) OK(o % 2 == 0);
  OK(f.ldr % 4 == 0 && f.ldc % 4 == 0 && f.R % 8 == 0 && f.C % 8 == 0 && f.R * n >= ny && f.C * n >= nx);
  if (f.keep & fold::FACE_M) { OK((size_t)(e_m - o_m) >= md); OK((fold::pack_doubles(nx) * 8) % 16 == 0 && (f.o_m * 8) % 16 == 0); }
  owners(ny, f.R, n);
  owners(nx, f.C, n);
  const int NW = fold::threads_for(f) / 32;
  OK(NW <= fold::FACE_THREADS / 32 && n <= fold::FACE_MAX_CLUSTER && n <= 32);
  for (int rank = 0; rank < n; ++rank) {
    const int r0 = rank * f.R, c0 = rank * f.C;
    const int nr = std::max(0, std::min(f.R, ny - r0)), nc = std::max(0, std::min(f.C, nx - c0));
    const long xt = f.o_xt, xc = f.o_xc, ext = f.o_sig, exc = f.o_xt;
    if (nr > 0) {
      IN(xt + (long)(nr - 1) * f.ldr + nx - 1, xt, ext);                      // q_net
      IN(f.o_row + (long)(nr - 1) * XC + XC - 1, f.o_row, e_row);             // row sums
      if (f.keep & fold::FACE_Q) IN(f.o_q + (long)(nr - 1) * f.ldr + nx - 1, f.o_q, e_q);
      pass(nx, nr, 1, f.ldr, xt, ext);                                        // x-forward
      for (int p : {0, nx - 1})                                               // to_columns, remote xc
        for (int v : {0, nr - 1}) IN(xc + p % f.C + (long)(r0 + v) * f.ldc, xc, exc);
      pass(nx, nr, 1, f.ldr, 0, row);                                         // x-inverse
      IN(xt + (long)(up8(nr) - 1) * f.ldr + nx - 1, xt, ext);                 // keep_row
      IN((long)(r0 + nr - 1), 0, ny);
      OK(HC * 32 >= fold::half_up(nx));
    }
    if (nc > 0) {
      if (f.keep & fold::FACE_W) {
        const long per = (long)ny * f.ldc;
        IN(f.o_w * (8 / (long)sizeof(W)) + 3 * per + (long)(ny - 1) * f.ldc + nc - 1, 0, e_w * (8 / (long)sizeof(W)));
      }
      pass(ny, nc, f.ldc, 1, xc, exc);                                        // y-forward
      IN(xt + (long)(ny - 1) * f.ldc + up8(nc) - 1, xt, ext);                 // keep_col
      OK(up8(nc) <= f.ldc);
      IN(f.o_sig + (long)(ny - 1) * f.ldc + nc - 1, f.o_sig, f.o_part);
      pass(ny, nc, f.ldc, 1, xt, ext);                                        // y-inverse
      for (int y : {0, ny - 1}) {                                             // to_rows, remote xr
        IN((long)(y % f.R) * f.ldr + c0 + nc - 1, 0, row);
        OK(((long)(y % f.R) * f.ldr + c0) % 2 == 0);
      }
      const int PT = (ny + 7) / 8, VT = (nx + 7) / 8, vn = (nc + 7) / 8;
      IN(f.o_part + 2L * ((PT - 1) * VT + c0 / 8 + vn - 1) + 1, f.o_part, f.o_row);
      for (int t = 0; t < PT * vn; ++t) OK((int)(((float)t + 0.5f) / (float)vn) == t / vn);
      IN(fold::mode_at(c0 + nc - 1, nx), 0, nx);
    }
    IN(xc + ny + (long)rank * NW + NW - 1, xc, exc);                          // table of the commit, rank 0
  }
}

static void slab(int nx, int ny, int n) {
  NX = nx; NY = ny; NN = n;
  const vol::SlabShape f = vol::slab_shape(nx, ny, n);
  if (f.bytes > fold::FACE_SMEM_MAX - 1024) return;
  const long xin = 0, exin = f.o_xr, xr = f.o_xr, exr = f.o_xt, xt = f.o_xt, ext = f.o_m;
  OK((long)ny * f.ldc <= exin && (long)f.R * f.ldr <= exr - xr && (long)f.R * f.ldr <= ext - xt);
  OK(f.o_xr % 2 == 0 && f.o_xt % 2 == 0 && (f.o_m * 8) % 16 == 0 && f.ldr % 4 == 0 && f.ldc % 4 == 0);
  if (f.keep) OK((size_t)(f.bytes / 8 - f.o_m) >= 2 * (fold::pack_doubles(nx) + fold::pack_doubles(ny)));
  OK(f.R * n >= ny && f.C * n >= nx);
  owners(ny, f.R, n);
  owners(nx, f.C, n);
  for (int p = 0; p < nx; ++p) IN(vol::pos_of(p, nx), 0, nx);
  for (int rank = 0; rank < n; ++rank) {
    const int r0 = rank * f.R, c0 = rank * f.C;
    const int nr = std::max(0, std::min(f.R, ny - r0)), nc = std::max(0, std::min(f.C, nx - c0));
    if (nc > 0) {
      IN(xin + (long)(ny - 1) * f.ldc + nc - 1, xin, exin);
      pass(ny, nc, f.ldc, 1, xin, exin);                                      // y-forward and y-inverse
      for (int y : {0, ny - 1}) {                                             // remote xr
        IN(xr + (long)(y % f.R) * f.ldr + c0 + nc - 1, xr, exr);
        OK((xr + (long)(y % f.R) * f.ldr + c0) % 2 == 0);
      }
      IN((long)(ny - 1) * nx + c0 + nc - 1, 0, (long)nx * ny);                // global output
    }
    if (nr > 0) {
      pass(nx, nr, 1, f.ldr, xr, exr);                                        // x-forward
      pass(nx, nr, 1, f.ldr, xt, ext);                                        // x-inverse
      IN(xt + (long)(nr - 1) * f.ldr + nx - 1, xt, ext);
      for (int x : {0, nx - 1})                                               // remote xin
        IN(xin + x % f.C + (long)(r0 + nr - 1) * f.ldc, xin, exin);
      const int XB = (nx + 31) / 32;
      for (int t = 0; t < nr * XB; ++t) OK((int)(((float)t + 0.5f) / (float)XB) == t / XB);
    }
  }
}

static void column(int nx, int ny, int nz) {
  NX = nx; NY = ny; NN = nz;
  const vol::ColShape f = vol::col_shape(nx, ny, nz);
  if (f.bytes > vol::COL_SMEM_MAX) return;
  const int wn = vol::COL_THREADS / f.cc;
  const long b1 = 0, b2 = (long)nz * f.ld, end = f.bytes / 8;
  OK(f.cc % 8 == 0 && f.cc <= f.ld && f.ld % 4 == 0 && b2 % 2 == 0);
  IN(b1 + (long)(nz - 1) * f.ld + f.cc - 1, b1, b2);
  IN(b2 + (long)(wn - 1) * f.ld + f.cc - 1, b2, end);                         // surface partials
  IN(b2 + (long)(nz - 1) * f.ld + f.cc - 1, b2, end);
  const long S = (long)nx * ny;
  for (long blk : {0L, (S + f.cc - 1) / f.cc - 1}) {
    const int nc = (int)std::min<long>(f.cc, S - blk * f.cc);
    pass(nz, nc, f.ld, 1, b1, b2);
    pass(nz, nc, f.ld, 1, b2, end);
    IN((long)(nz - 1) * S + blk * f.cc + nc - 1, 0, S * nz);
  }
  for (int z = 0; z < nz; ++z) IN(vol::pos_of(z, nz), 0, nz);
}

int main() {
  std::vector<std::pair<int, int>> faces;
  for (int x = 2; x <= 150; ++x)
    for (int y = 2; y <= 150; ++y) faces.push_back({x, y});
  const int longer[] = {2, 3, 7, 8, 9, 16, 31, 64, 100, 120, 127, 128, 160, 192, 255, 256, 257, 300, 400, 511, 512, 513, 600, 1000, 1023, 2047, 4096};
  for (int x : longer)
    for (int y : longer) faces.push_back({x, y});
  for (const auto& q : faces)
    for (int n = 1; n <= 16; n *= 2) {
      face<double>(q.first, q.second, n);
      face<float>(q.first, q.second, n);
      slab(q.first, q.second, n);
    }
  for (const auto& q : faces)
    for (int nz : {1, 2, 3, 5, 8, 16, 17, 33, 64, 100, 255, 640})
      if ((q.first + q.second) % 7 == 0 || q.first > 150) column(q.first, q.second, nz);
  std::printf("ok %ld\n", checks);
  return 0;
}
"""


@pytest.mark.slow
@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
def test_every_shared_access_stays_in_its_region(tmp_path):
    src, exe = tmp_path / "ranges.cu", tmp_path / "ranges"
    src.write_text(PROGRAM)
    subprocess.run([NVCC, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-I", CSRC, "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout
