// sgh_fold.cuh -- FP64 cosine contractions halved by the transform's symmetry,
// and the whole face-space Picard step of one instance in one thread-block
// cluster built on them.
//
// The orthonormal DCT-II matrix has M[k][N-1-n] = (-1)^k M[k][n]. A forward
// pass therefore contracts X[n] + X[N-1-n] with the even rows and X[n] -
// X[N-1-n] with the odd rows over half the length; an inverse pass forms the
// even-mode and odd-mode halves e[n], o[n] of n < N/2 and gives out[n] = e + o,
// out[N-1-n] = e - o. Half the multiplications, the same sums up to FP64
// rounding (the products are those of the full contraction, added in another
// order).
//
// Contractions run on the FP64 tensor cores (mma.sync m16n8k8 .f64, the FP64
// MMA of sm_90 kept on sm_100a; tcgen05 has no FP64 kind) with the matrix as
// the 16 x 8 operand, read in fragment order from a packed copy (one
// coalesced 512-byte load per fragment half, no shared-memory staging, no
// bank conflicts), and the data as the 8 x 8 operand, read from shared
// memory, where both members of a mirrored pair are one load each. Vectors
// (rows or columns of the face) go 8 per MMA tile, so a cluster can share a
// small face out 8 rows at a time.
//
// In shared memory mode-space data is ordered even modes first: position p
// holds mode 2p for p < h, mode 2(p - h) + 1 above (h = ceil(N/2)).
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "sgh_axis.cuh"
#include "sgh_device.cuh"
#include "sgh_limits.h"
#include "sgh_umma.cuh"

namespace sgh {
namespace fold {

__host__ __device__ inline int half_up(int n) { return (n + 1) / 2; }
__host__ __device__ inline int mtiles(int n) { return (half_up(n) + 15) / 16; }
__host__ __device__ inline int ksteps(int n) { return (half_up(n) + 7) / 8; }
// doubles of one packed matrix (one direction): per 16-row tile and 8-slice
// step the even and the odd fragment, 4 doubles per lane each
__host__ __device__ inline size_t pack_doubles(int n) { return (size_t)mtiles(n) * ksteps(n) * 256; }
// mode at position p of an axis of n modes
__host__ __device__ inline int mode_at(int p, int n) {
  const int h = half_up(n);
  return p < h ? 2 * p : 2 * (p - h) + 1;
}

// Packs the N x N DCT-II matrix M[k][n] for both directions. Fragment (mt,
// ks), part q (0, 1: even rows, slices +0 / +4; 2, 3: odd rows), lane (g, t),
// element e: row 16 mt + g + 8 e, slice 8 ks + t + 4 (q & 1).
static __global__ void k_fold_pack(int N, const double* __restrict__ M, double* __restrict__ fwd,
                                   double* __restrict__ inv) {
  const int h = half_up(N), l = N - h, MT = mtiles(N), KS = ksteps(N);
  const long total = (long)MT * KS * 256;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int e = (int)(i & 1), lane = (int)(i >> 1) & 31, q = (int)(i >> 6) & 3;
    const int fr = (int)(i >> 8), ks = fr % KS, mt = fr / KS;
    const int row = 16 * mt + (lane >> 2) + 8 * e, k = 8 * ks + (lane & 3) + 4 * (q & 1);
    const bool odd = q >= 2, mid = (N & 1) && k == h - 1;
    double f = 0.0, v = 0.0;
    if (!odd) {
      // the middle sample of an odd length meets itself in the fold: half its weight
      if (row < h && k < h) f = M[(size_t)(2 * row) * N + k] * (mid ? 0.5 : 1.0);
      if (row < h && k < h) v = M[(size_t)(2 * k) * N + row];
    } else {
      if (row < l && k < l) f = M[(size_t)(2 * row + 1) * N + k];
      if (row < l && k < l) v = M[(size_t)(2 * k + 1) * N + row];  // row = middle: the odd half is 0
    }
    fwd[i] = f;
    inv[i] = v;
  }
}

// Accumulates one 16-row fragment row of a folded contraction over NV vector
// tiles: acc[v] += A x B(v), with A's fragments at ap (a 16 x 8 fragment every
// 128 double2, halves 32 apart) and B built from shared-memory vectors: lane
// (g, t) reads vector g of a tile. Forward (FOLD): slice k is X[k] + sgn
// X[N-1-k] (sgn = +-1: even, odd rows); inverse: slice k is X[k], X already at
// the even- or odd-mode half. kmax: last slice that may be read; slices beyond
// meet zero matrix entries. The MMA sustains its full rate on one dependent
// chain per scheduler (64 clocks each, measured), so a warp needs no second
// accumulator; the fragments of FU steps are loaded ahead of their MMAs, and
// the next FU steps' before those, to cover the L2 latency of matrices that
// did not fit in shared memory.

template <bool FOLD, int NV>
__device__ __forceinline__ void fold_mma(const double2* ap, int KS, const double* const (&x)[NV], int sk, int kmax,
                                         int nlast, double sgn, int t, double (&acc)[NV][4]) {
  constexpr int FU = NV == 1 ? 4 : 2;
  double2 an[FU][2];
#pragma unroll
  for (int u = 0; u < FU; ++u) {
    const int ks = u < KS ? u : KS - 1;
    an[u][0] = ap[ks * 128];
    an[u][1] = ap[ks * 128 + 32];
  }
#pragma unroll 1
  for (int k0 = 0; k0 < KS; k0 += FU) {
    double af[FU][4], bf[FU][NV][2];
#pragma unroll
    for (int u = 0; u < FU; ++u) {
      af[u][0] = an[u][0].x;
      af[u][1] = an[u][0].y;
      af[u][2] = an[u][1].x;
      af[u][3] = an[u][1].y;
    }
#pragma unroll
    for (int u = 0; u < FU; ++u) {
      const int ks = min(k0 + FU + u, KS - 1);
      an[u][0] = ap[ks * 128];
      an[u][1] = ap[ks * 128 + 32];
    }
#pragma unroll
    for (int u = 0; u < FU; ++u) {
      const int ka = min(8 * (k0 + u) + t, kmax), kb = min(8 * (k0 + u) + t + 4, kmax);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        bf[u][v][0] = x[v][ka * sk];
        bf[u][v][1] = x[v][kb * sk];
        if (FOLD) {
          bf[u][v][0] = fma(sgn, x[v][(nlast - ka) * sk], bf[u][v][0]);
          bf[u][v][1] = fma(sgn, x[v][(nlast - kb) * sk], bf[u][v][1]);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < FU; ++u)
      if (k0 + u < KS) {
#pragma unroll
        for (int v = 0; v < NV; ++v) mma_f64_m16n8k8(acc[v], af[u], bf[u][v]);
      }
  }
}

// One folded pass over nvec vectors, shared out over the block's warps. X:
// element k of vector v at X[k * sk + v * sv]; vectors up to the next multiple
// of 8 must be readable (their results are dropped).
//   KIND 0, forward: out(p, v, x0, x1) receives mode position p of vectors v, v + 1;
//   KIND 1, inverse halves: out(p, ...) receives e[p] for p < h (p natural) and
//     o[N-1-p] for p >= h: the caller forms e + o and e - o of a mirrored pair;
//   KIND 2, inverse: out(n, ...) receives natural index n.
// KIND 0 and 1 give the even and the odd half to different warps. The order of
// every sum depends on N only, so results do not depend on NV or on how
// vectors are dealt out.
template <int KIND, int NV, class Out>
__device__ __forceinline__ void fold_pass(const double* P, int N, const double* X, int sk, int sv, int nvec, int warp,
                                          int nwarps, const Out& out) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int h = half_up(N), l = N - h, MT = mtiles(N), KS = ksteps(N);
  const int nvt = (nvec + 7) / 8, ngrp = (nvt + NV - 1) / NV;
  const int rows = KIND == 2 ? MT : 2 * MT;  // fragment rows (x the two halves)
  int grp = 0, row = warp;
  while (row >= rows) {
    row -= rows;
    ++grp;
  }
  while (grp < ngrp) {
    const bool odd = KIND != 2 && row >= MT;
    const int mt = odd ? row - MT : row, vt0 = grp * NV;
    const double* xv[NV];
    double acc[NV][4];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      xv[v] = X + (size_t)(min(vt0 + v, nvt - 1) * 8 + g) * sv;
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[v][q] = 0.0;
    }
    const double2* ap = reinterpret_cast<const double2*>(P + (size_t)mt * KS * 256) + lane + (odd ? 64 : 0);
    if (KIND == 0) {
      fold_mma<true, NV>(ap, KS, xv, sk, odd ? l - 1 : h - 1, N - 1, odd ? -1.0 : 1.0, t, acc);
    } else {
      if (KIND == 1 && odd)
#pragma unroll
        for (int v = 0; v < NV; ++v) xv[v] += h * sk;
      fold_mma<false, NV>(ap, KS, xv, sk, odd ? l - 1 : h - 1, 0, 0.0, t, acc);
    }
    double ao[NV][4];
    if (KIND == 2) {
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        xv[v] += h * sk;
#pragma unroll
        for (int q = 0; q < 4; ++q) ao[v][q] = 0.0;
      }
      fold_mma<false, NV>(ap + 64, KS, xv, sk, l - 1, 0, 0.0, t, ao);
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      if (vt0 + v >= nvt) break;
      const int vec = (vt0 + v) * 8 + 2 * t;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = 16 * mt + g + 8 * e;
        if (KIND == 2) {
          if (r < h) {
            out(r, vec, acc[v][2 * e] + ao[v][2 * e], acc[v][2 * e + 1] + ao[v][2 * e + 1]);
            if (N - 1 - r != r) out(N - 1 - r, vec, acc[v][2 * e] - ao[v][2 * e], acc[v][2 * e + 1] - ao[v][2 * e + 1]);
          }
        } else if (r < (odd ? l : h)) {
          out(odd ? (KIND == 0 ? h + r : N - 1 - r) : r, vec, acc[v][2 * e], acc[v][2 * e + 1]);
        }
      }
    }
    row += nwarps;
    while (row >= rows) {
      row -= rows;
      ++grp;
    }
  }
}

// ---------------------------------------------------------------------------
// The face-space step of one instance in one cluster
// ---------------------------------------------------------------------------
// A face (ny x nx) is shared out over the n CTAs of a cluster twice: by rows
// for the x-passes (physical space and the x-side of the transposes), by mode
// columns for the y-passes (mode space). Each Picard iteration is
//   y-inverse (columns) -> x-inverse (rows), evaporation -> x-forward (rows)
//   -> y-forward (columns), relaxation
// with the two transposes written straight into the owners' shared memory and
// one cluster barrier behind each. The convergence test of an iteration rides
// on the next iteration's first barrier: that iteration's y-inverse is also
// what the commit's surface reconstruction needs, so nothing is wasted when
// the loop stops there.
// Every per-instance sum is taken over partials whose order depends on the face
// alone (per row, per 8 x 8 tile of modes), so a result does not depend on
// the cluster size or on the other instances of a launch.
constexpr int FACE_THREADS = 512;  // most threads of a face kernel
constexpr int FACE_MAX_CLUSTER = 16;
constexpr int FACE_SMEM_MAX = 227 * 1024;  // shapes leave 512 bytes of it to the kernels' static arrays

// Row stride of a shared array: at least n, 4 or 12 mod 16 doubles (fragment
// reads along and across rows then hit all banks).
__host__ __device__ inline int face_ld(int n) { return (n + 3) / 8 * 8 + 4; }

// What stays in shared memory beside the exchange buffers and sigma, in this
// order while it fits; the rest is read from global memory (L2) where needed.
enum { FACE_W = 1, FACE_Q = 2, FACE_M = 4 };

struct FaceShape {
  int nx, ny, n, R, C, ldr, ldc;   // rows / columns per CTA (multiples of 8), row strides
  int o_xc, o_xt, o_sig, o_w, o_q, o_m, o_part, o_row;  // offsets in doubles (xr at 0)
  int npart, bytes, keep;
};
template <class W>
__host__ inline FaceShape face_shape(int nx, int ny, int n) {
  FaceShape f;
  f.nx = nx; f.ny = ny; f.n = n;
  f.R = ((ny + 7) / 8 + n - 1) / n * 8;
  f.C = ((nx + 7) / 8 + n - 1) / n * 8;
  f.ldr = face_ld(nx);
  f.ldc = face_ld(f.C);
  f.npart = ((ny + 7) / 8) * ((nx + 7) / 8);
  const int row = f.R * f.ldr, col = ny * f.ldc;
  int o = row;
  f.o_xc = o; o += std::max(col, (ny + 1) / 2 * 2 + FACE_MAX_CLUSTER * FACE_THREADS / 32);
  f.o_xt = o; o += std::max(row, col);
  f.o_sig = o; o += col;
  f.o_part = o; o += 2 * f.npart;
  f.o_row = o; o += (f.R * ((nx + 31) / 32) + 1) / 2 * 2;
  f.keep = 0;
  f.o_w = f.o_q = f.o_m = 0;
  const int cap = FACE_SMEM_MAX / 8 - 64;
  const int wd = (int)((4 * (size_t)col * sizeof(W) + 7) / 8), qd = row;
  const size_t md = 2 * (pack_doubles(nx) + pack_doubles(ny));
  if (o + wd <= cap) { f.o_w = o; o += (wd + 1) / 2 * 2; f.keep |= FACE_W; }
  if (o + qd <= cap) { f.o_q = o; o += (qd + 1) / 2 * 2; f.keep |= FACE_Q; }
  if ((size_t)o + md <= (size_t)cap) { f.o_m = o; o += (int)md; f.keep |= FACE_M; }
  f.bytes = o * 8;
  return f;
}

// Cluster size for a face, 0 where the face does not fit a cluster. Small faces
// are bound by the latency of a pass and by the two cluster barriers of an
// iteration (0.5 us each), large ones by the FP64 tensor pipe of their CTAs.
// Measured on a B200, time of a Picard loop: up to 1024 elements one CTA is as
// fast as two or more (four slots of 24-64 columns: 1.85 ms at one or four CTAs
// by size, 2.01 ms at one CTA each); 64 x 32, 8 steps: 410 us at 4 CTAs, 508 at
// one; 18 FP64 slots with 128 x 64 faces on 4 CTAs 0.86 ms, on 8 (a second wave)
// 0.95; 192 x 96 and 256 x 128 gain 1.3x from 8 to 16 CTAs (256 x 128 x 64, 6
// steps: 564 against 748 us). The result does not depend on the choice.
template <class W>
__host__ inline int cluster_size(int nx, int ny) {
  const long S = (long)nx * ny;
  for (int n = S <= 1024 ? 1 : (S <= 8192 ? 4 : (S <= 16384 ? 8 : 16)); n <= FACE_MAX_CLUSTER; n *= 2)
    if (face_shape<W>(nx, ny, n).bytes <= FACE_SMEM_MAX - 512) return n;
  return 0;
}
// Cluster size of a face among so many that the chip is filled several times
// over: the fewest CTAs of at most FACE_SHARE_CROWDED elements each that hold it,
// since waves of clusters then count and the passes' latency does not.
constexpr long FACE_SHARE = 2048, FACE_SHARE_CROWDED = 4096;
template <class W>
__host__ inline int cluster_size_crowded(int nx, int ny) {
  for (int n = 1; n <= FACE_MAX_CLUSTER; n *= 2)
    if ((long)nx * ny <= FACE_SHARE_CROWDED * n && face_shape<W>(nx, ny, n).bytes <= FACE_SMEM_MAX - 512) return n;
  return cluster_size<W>(nx, ny);
}
// Estimated length of a Picard iteration's four passes on a cluster, in slice steps
// of its longest chain of tasks: 16 warps a CTA, a task is one 16-row fragment row
// of one half over the slices of one vector tile (see fold_pass). A long axis
// gives few CTAs many fragment rows, shares of several tiles give many tasks.
inline int face_chain(int nx, int ny, int n) {
  const int R = ((ny + 7) / 8 + n - 1) / n, C = ((nx + 7) / 8 + n - 1) / n;  // vector tiles a CTA
  const auto pass = [](int N, int tiles, int halves) {
    const bool two = tiles > 1 && mtiles(N) * ((tiles + 1) / 2) >= 16;
    const int tasks = halves * mtiles(N) * (two ? (tiles + 1) / 2 : tiles);
    return (tasks + 15) / 16 * ksteps(N) * (two ? 2 : 1);
  };
  return 2 * pass(nx, R, 2) + pass(ny, C, 2) + 2 * pass(ny, C, 1);
}
// Threads of a face kernel: eight warps cover the tasks of a small share
// (64 x 32 on 4 CTAs: 407 us with 256 or 512 threads, 437 with 128), larger
// ones want sixteen (256 x 128: 884 us with 256, 749 with 512, at 8 CTAs).
inline int threads_for(const FaceShape& f) { return (long)f.nx * f.ny / f.n <= 512 ? 256 : 512; }

template <class W>
struct FaceJob {
  // the fields laser_flux and evaporation read
  int cell_integrated;
  double dx, dy, r_x, r_y, order, T_liquidus, T_boil, evap_f1, evap_f2;
  double dct_scale, recon_scale, omega, tol, n_elements;
  int max_iter;
  double I0, lx, ly, shift_x, shift_y;
  const double *pxf, *pxi, *pyf, *pyi;  // packed matrices
  const W *Zt, *Yt, *Wtt, *Qtt;         // natural (ky, kx) order
  const double* part_n1;
  int n_n1;
  double *qlas, *qev, *sigma, *Tsurf;   // natural order; qev is q_evap_old on entry, q_evap on return
  double* hist;                         // (rms, rel) per iteration, or null
  int hist_cap;
};
struct FaceResult {
  int iter, status;
  double rel, tmax, qsum;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One element, global -> shared, asynchronously (4 or 8 bytes).
template <class W>
__device__ __forceinline__ void copy_async(W* dst, const W* src) {
  if (sizeof(W) == 8) {
    cp_async8(dst, src, 8);
  } else {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(src));
  }
}

// All threads of all CTAs of the cluster. The result is complete on rank 0,
// thread 0. bad: this CTA's operands are invalid (an expired wait): the cluster then
// writes no results (q_evap, sigma and the surface stay as they were) and the step
// ends non-finite. KEEPM: the packed matrices
// are in shared memory (FACE_M), addressed as such.
template <class W, bool KEEPM>
__device__ FaceResult face_step(const FaceShape& f, const FaceJob<W>& J, double* sm, bool bad) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ int sbad;
  const int n = f.n, rank = (int)cl.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int NW = blockDim.x >> 5;
  if (tid == 0) sbad = bad ? 1 : 0;
  auto sync_all = [&] {  // one CTA: a block barrier is a tenth of a cluster barrier
    if (n > 1) cl.sync();
    else __syncthreads();
  };
  const int nx = f.nx, ny = f.ny, ldr = f.ldr, ldc = f.ldc, R = f.R, C = f.C;
  const int r0 = rank * R, c0 = rank * C;
  const int nr = max(0, min(R, ny - r0)), nc = max(0, min(C, nx - c0));
  const float rR = 1.0f / (float)R, rC = 1.0f / (float)C;  // small exact quotients: (i + 0.5) / R
  double* xr = sm;
  double* xc = sm + f.o_xc;
  double* xt = sm + f.o_xt;
  double* sig = sm + f.o_sig;
  double* part = sm + f.o_part;
  double* rowsum = sm + f.o_row;
  const bool keepw = f.keep & FACE_W, keepq = f.keep & FACE_Q;
  W* sw = reinterpret_cast<W*>(sm + f.o_w);
  const int wstride = ny * ldc;
  double* sq = sm + f.o_q;
  const int nxp = (int)pack_doubles(nx), nyp = (int)pack_doubles(ny);
  const double* pxf = KEEPM ? sm + f.o_m : J.pxf;
  const double* pxi = KEEPM ? sm + f.o_m + nxp : J.pxi;
  const double* pyf = KEEPM ? sm + f.o_m + 2 * nxp : J.pyf;
  const double* pyi = KEEPM ? sm + f.o_m + 2 * nxp + nyp : J.pyi;

  if (keepw) {
    // this CTA's columns of the face sums and weights, in position order, copied
    // while the laser flux and the first passes run
    for (int p = warp; p < ny; p += NW) {
      const size_t g0 = (size_t)mode_at(p, ny) * nx;
      for (int c = lane; c < nc; c += 32) {
        const size_t gi = g0 + mode_at(c0 + c, nx);
        const int li = p * ldc + c;
        copy_async(&sw[li], J.Zt + gi);
        copy_async(&sw[wstride + li], J.Wtt + gi);
        copy_async(&sw[2 * wstride + li], J.Yt + gi);
        copy_async(&sw[3 * wstride + li], J.Qtt + gi);
      }
    }
    cp_async_commit();
  }
  // laser flux, warm-start shift (solvers/spectral.py:273-306); sums of q_las per 32 cells of a row
  const int XC = (nx + 31) / 32;
  for (int r = 0, xb = warp; r < nr; xb += NW) {
    while (xb >= XC && r < nr) {
      xb -= XC;
      ++r;
    }
    if (r >= nr) break;
    const int x = xb * 32 + lane, y = r0 + r;
    double q = 0.0;
    if (x < nx) {
      const ShiftTap ty = shift_tap(y, ny, J.shift_y), tx = shift_tap(x, nx, J.shift_x);
      double v = 0.0;
      if (ty.in && tx.in) {
        const double* f0 = J.qev + (size_t)ty.i0 * nx;
        const double* f1 = J.qev + (size_t)ty.i1 * nx;
        v = ty.w0 * (tx.w0 * f0[tx.i0] + tx.w1 * f0[tx.i1]) + ty.w1 * (tx.w0 * f1[tx.i0] + tx.w1 * f1[tx.i1]);
      }
      // cell centres rounded as the reference rounds them: fused into the
      // subtraction of the beam position they would differ between the kernels
      // this is compiled into
      q = laser_flux(J, J.I0, J.lx, J.ly, __dmul_rn((double)x + 0.5, J.dx), __dmul_rn((double)y + 0.5, J.dy));
      if (keepq) sq[r * ldr + x] = q;
      else J.qlas[(size_t)y * nx + x] = q;
      xt[r * ldr + x] = q - v;
    }
    q = warp_sum(q);
    if (lane == 0) rowsum[r * XC + xb] = q;
  }
  double n1 = 0.0;  // norm of the propagated modes, in a fixed order
  for (int k = lane; k < J.n_n1; k += 32) n1 += J.part_n1[k];
  n1 = warp_sum(n1);
  sync_all();  // also: every CTA of the cluster runs before any remote write

  FaceResult res;
  res.iter = -1;
  res.status = SGH_STEP_CAPPED;
  res.rel = nan("");
  // every warp reads every CTA's flag, so all leave here together or none does; the
  // second barrier keeps each CTA's shared memory until the others have read it
  if (__any_sync(0xffffffffu, lane < n && *cl.map_shared_rank(&sbad, lane < n ? lane : 0) != 0)) {
    cp_async_wait<0>();
    sync_all();
    res.iter = 0;
    res.status = SGH_STEP_NONFINITE;
    res.tmax = res.qsum = nan("");
    return res;
  }

  // transposes: row domain -> the column owners' xc, column domain -> the row owners' xr
  auto to_columns = [&](int p, int v, double x0, double x1) {
    const int dst = (int)(((float)p + 0.5f) * rC);
    double* o = cl.map_shared_rank(xc, dst) + (p - dst * C) + (r0 + v) * ldc;
    if (v < nr) o[0] = x0;
    if (v + 1 < nr) o[ldc] = x1;
  };
  auto to_rows = [&](int y, int v, double x0, double x1) {
    const int dst = (int)(((float)y + 0.5f) * rR);
    double* o = cl.map_shared_rank(xr, dst) + (y - dst * R) * ldr + c0 + v;
    if (v + 1 < nc) *reinterpret_cast<double2*>(o) = make_double2(x0, x1);
    else if (v < nc) *o = x0;
  };
  // results kept in this CTA's xt (vectors beyond the face land in its padding)
  auto keep_row = [&](int x, int v, double x0, double x1) {
    xt[v * ldr + x] = x0;
    xt[(v + 1) * ldr + x] = x1;
  };
  auto keep_col = [&](int p, int v, double x0, double x1) {
    *reinterpret_cast<double2*>(&xt[p * ldc + v]) = make_double2(x0, x1);
  };
  // two vector tiles per matrix fragment where there are two and that still leaves every
  // warp a task (with two for a share of one tile, half the products were
  // dropped: a 512 x 64 face, 12 iterations, 780 us a step, now 540)
  auto pass = [&](auto kind, const double* P, int N, const double* X, int sk, int sv, int nvec, const auto& out) {
    constexpr int KIND = decltype(kind)::value;
    if (nvec <= 0) return;
    if (nvec > 8 && mtiles(N) * ((nvec + 15) / 16) >= NW) fold_pass<KIND, 2>(P, N, X, sk, sv, nvec, warp, NW, out);
    else fold_pass<KIND, 1>(P, N, X, sk, sv, nvec, warp, NW, out);
  };
  auto weight = [&](int which, const W* src, int li, size_t gi) -> double {
    return keepw ? (double)sw[which * wstride + li] : (double)src[gi];
  };
  const int hx = half_up(nx), VT = (nx + 7) / 8, PT = (ny + 7) / 8, vt_n = (nc + 7) / 8;

  double mx = -INFINITY;
  for (;;) {
    // q_net -> its 2-D transform, first along rows, then along columns
    pass(std::integral_constant<int, 0>{}, pxf, nx, xt, 1, ldr, nr, to_columns);
    sync_all();
    pass(std::integral_constant<int, 0>{}, pyf, ny, xc, ldc, 1, nc, keep_col);
    if (res.iter < 0) cp_async_wait<0>();  // the weights of this thread's copies have landed
    __syncthreads();
    // 8 positions x 8 columns per warp, two elements per lane
    for (int task = warp; task < PT * vt_n; task += NW) {
      const int pt = (int)(((float)task + 0.5f) / (float)vt_n), vt = task - pt * vt_n;
      const int c = vt * 8 + (lane & 7);
      double r2 = 0.0, o2 = 0.0;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int p = pt * 8 + (lane >> 3) + 4 * j;
        if (p < ny && c < nc) {
          const int li = p * ldc + c;
          const size_t gi = keepw ? 0 : (size_t)mode_at(p, ny) * nx + mode_at(c0 + c, nx);
          const double S = J.dct_scale * xt[li], zt = weight(0, J.Zt, li, gi), wt = weight(1, J.Wtt, li, gi);
          double ns = S;  // initial guess: sigma = dct_scale DCT2(q_las - shift(q_evap_old))
          if (res.iter >= 0) {  // residual and iterate norms, relaxation (solvers/spectral.py:431-468)
            const double s = sig[li], q = weight(3, J.Qtt, li, gi), d = S - s;
            r2 += d * d * q;
            o2 += 2.0 * s * weight(2, J.Yt, li, gi) + s * s * q;
            ns = d * J.omega + s;
          }
          sig[li] = ns;
          xt[li] = zt + wt * ns;  // the iterate's top-surface input A = Zt + W_tt sigma
        }
      }
      if (res.iter >= 0) {  // this tile's partials into every CTA's table
        r2 = warp_sum(r2);
        o2 = warp_sum(o2);
        if (lane < n)
          *reinterpret_cast<double2*>(cl.map_shared_rank(part, lane) + 2 * (pt * VT + c0 / 8 + vt)) =
              make_double2(r2, o2);
      }
    }
    ++res.iter;
    __syncthreads();
    pass(std::integral_constant<int, 2>{}, pyi, ny, xt, ldc, 1, nc, to_rows);
    sync_all();
    bool stop = res.iter >= J.max_iter;
    if (res.iter > 0) {  // convergence test of the iteration just relaxed (solvers/spectral.py:464-499)
      double s0 = 0.0, s1 = 0.0;
      for (int k = lane; k < f.npart; k += 32) {
        const double2 q = *reinterpret_cast<const double2*>(part + 2 * k);
        s0 += q.x;
        s1 += q.y;
      }
      s0 = warp_sum(s0);
      s1 = warp_sum(s1) + n1;
      const double rms_d = sqrt(s0 / J.n_elements);
      res.rel = rms_d / fmax(sqrt(s1 / J.n_elements), 1e-9);
      if (J.hist && res.iter <= J.hist_cap && rank == 0 && tid == 0) {
        J.hist[2 * (res.iter - 1)] = rms_d;
        J.hist[2 * (res.iter - 1) + 1] = res.rel;
      }
      if (res.rel < J.tol) {
        res.status = SGH_STEP_CONVERGED;
        stop = true;
      } else if (!isfinite(res.rel)) {
        res.status = SGH_STEP_NONFINITE;
        stop = true;
      }
    }
    pass(std::integral_constant<int, 1>{}, pxi, nx, xr, 1, ldr, nr, keep_row);
    __syncthreads();
    // mirrored pairs of a row: T_s = recon_scale (e +- o), then evaporation and
    // q_net (solvers/spectral.py:388-404), or the commit (:502-512)
    for (int r = 0, xb = warp; r < nr; xb += NW) {
      const int HC = (hx + 31) / 32;
      while (xb >= HC && r < nr) {
        xb -= HC;
        ++r;
      }
      if (r >= nr) break;
      const int xa = xb * 32 + lane, xz = nx - 1 - xa;
      if (xa < hx) {
        double* row = xt + r * ldr;
        const double e = row[xa], o = xz != xa ? row[xz] : 0.0;
        const size_t g0 = (size_t)(r0 + r) * nx;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int x = j ? xz : xa;
          if (j && xz == xa) break;
          const double T = J.recon_scale * (j ? e - o : e + o);
          if (stop) {
            J.Tsurf[g0 + x] = T;
            mx = fmax(mx, T);
          } else {
            const double qe = evaporation(J, T);
            J.qev[g0 + x] = qe;
            row[x] = (keepq ? sq[r * ldr + x] : J.qlas[g0 + x]) - qe;
          }
        }
      }
    }
    if (stop) break;
    __syncthreads();
  }
  for (int p = warp; p < ny; p += NW) {
    const size_t g0 = (size_t)mode_at(p, ny) * nx;
    for (int c = lane; c < nc; c += 32) J.sigma[g0 + mode_at(c0 + c, nx)] = sig[p * ldc + c];
  }
  // P_laser and T_surface_max: per row sums and per CTA maxima into rank 0 (xc is free)
  double* tab = cl.map_shared_rank(xc, 0);
  for (int r = tid; r < nr; r += blockDim.x) {
    double s = 0.0;
    for (int k = 0; k < XC; ++k) s += rowsum[r * XC + k];
    tab[r0 + r] = s;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) tab[ny + rank * NW + warp] = mx;
  sync_all();
  res.tmax = -INFINITY;
  res.qsum = 0.0;
  if (rank == 0 && warp == 0) {
    double qs = 0.0, m = -INFINITY;
    for (int k = lane; k < ny; k += 32) qs += xc[k];
    for (int k = lane; k < n * NW; k += 32) m = fmax(m, xc[ny + k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    res.qsum = warp_sum(qs);
    res.tmax = m;
  }
  return res;
}

// Copies the packed matrices into shared memory (FACE_M) by bulk copies on one
// mbarrier, every thread waiting at most `lim` polls; false when the wait ran
// out (or, with `stall`, after a wait on a barrier that nothing completes): the
// error is recorded, and the copies in flight are waited for with the full
// bound. Called by all threads before face_step.
template <class W>
__device__ bool face_operands(const FaceShape& f, const FaceJob<W>& J, double* sm, uint64_t* bar, unsigned lim,
                              bool stall, int* err) {
  using namespace umma;
  if (threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    if (f.keep & FACE_M) {
      const uint32_t bx = (uint32_t)(pack_doubles(f.nx) * 8), by = (uint32_t)(pack_doubles(f.ny) * 8);
      mbar_expect_tx(&bar[0], 2 * (bx + by));
      char* o = reinterpret_cast<char*>(sm + f.o_m);
      bulk_g2s(o, J.pxf, bx, &bar[0]);
      bulk_g2s(o + bx, J.pxi, bx, &bar[0]);
      bulk_g2s(o + 2 * bx, J.pyf, by, &bar[0]);
      bulk_g2s(o + 2 * bx + by, J.pyi, by, &bar[0]);
    }
  }
  __syncthreads();
  bool ok = !stall || mbar_wait_bounded(&bar[1], 0u, lim);
  if (f.keep & FACE_M) {
    ok = ok && mbar_wait_bounded(&bar[0], 0u, lim);
    if (!ok) mbar_wait_bounded(&bar[0], 0u, WAIT_LIMIT);
  }
  ok = __syncthreads_and(ok ? 1 : 0) != 0;
  if (!ok && threadIdx.x == 0 && err) atomicExch(err, 1);
  return ok;
}

// Cluster launch of a face kernel; `pdl`: programmatic stream serialisation
// (the kernel executes griddepcontrol.wait before any global access).
template <class... KArgs, class... Args>
inline cudaError_t launch_cluster(void (*kernel)(KArgs...), int ctas, int n, int threads, int smem, bool pdl,
                                  cudaStream_t st,
                                  Args&&... args) {
  const cudaError_t e = kernel_limits(reinterpret_cast<const void*>(kernel), FACE_SMEM_MAX - 512, true);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute la[2];
  la[0].id = cudaLaunchAttributeClusterDimension;
  la[0].val.clusterDim.x = n;
  la[0].val.clusterDim.y = 1;
  la[0].val.clusterDim.z = 1;
  la[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  la[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = la;
  cfg.numAttrs = pdl ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace fold
}  // namespace sgh
