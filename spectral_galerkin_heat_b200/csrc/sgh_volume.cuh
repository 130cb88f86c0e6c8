// sgh_volume.cuh -- the Picard iteration of the grid-mode volume form as two
// kinds of fused kernels on the folded FP64 contractions of sgh_fold.cuh.
//
// An iteration is six 1-D transforms of the volume in each direction with
// pointwise work between them. As one pass per axis (14 launches of 4-5 us at
// 128 x 64 x 32) it is bound by the launches' fill, drain and L2 round trips.
// Here neighbouring passes share a kernel:
//   slab kernels (k_slab)   one cluster per z-mode: y and x transforms of one
//     slab, forward, then the modal update, then inverse, with the two
//     transposes through distributed shared memory;
//   column kernels (k_column) 16 or 32 (y, x) columns per CTA with all of z:
//     z-inverse, pointwise physics, z-forward.
// With latent heat and the property correction:
//   B = xy-inverse of the iterate (kept between iterations)
//   column LATENT : B -> T, latent source Q, top flux q_net -> G = z-DCT(Q)
//   slab TRIAL    : G + Ct q_net -> a_trial -> C = xy-inverse of a_trial
//   column TEMP   : C -> T, k'(T)
//   column STENCIL: f = div(k' grad T) - a'(T) dT/dt -> F = z-DCT(f)
//   slab RELAX    : F -> relaxation of the iterate, residual norms -> B
// and without the correction: column LATENT, slab TRIAL_RELAX. The top flux
// enters as (dct_scale / sqrt_dV) Ct[p] q_net added to every slab before its
// transform: Ct[p] S_top = Ct[p] dct_scale DCT2(q_net) by linearity.
#pragma once
#include "sgh_fold.cuh"

namespace sgh {
namespace vol {

using fold::half_up;
using fold::ksteps;
using fold::mode_at;
using fold::mtiles;

constexpr int SLAB_THREADS = 512;
constexpr int COL_THREADS = 256;
enum { SLAB_INIT, SLAB_TRIAL, SLAB_TRIAL_RELAX, SLAB_RELAX, SLAB_QM };
enum { COL_LATENT, COL_TEMP, COL_STENCIL, COL_COMMIT };

__host__ __device__ __forceinline__ int pos_of(int m, int n) { return (m & 1) ? half_up(n) + (m >> 1) : (m >> 1); }

// Where a pass puts its results: output p of vector v at row(p)[v * vs], for v <
// nv; pair: two neighbouring vectors (vs = 1) may be stored as one 16-byte word.
template <class Row>
struct Out {
  Row row;
  int vs, nv;
  bool pair;
  __device__ __forceinline__ void put(double* o, int v, double x0, double x1) const {
    if (pair && v + 1 < nv) {
      *reinterpret_cast<double2*>(o + v) = make_double2(x0, x1);
    } else {
      if (v < nv) o[v * vs] = x0;
      if (v + 1 < nv) o[(v + 1) * vs] = x1;
    }
  }
};
template <class Row>
__device__ __forceinline__ Out<Row> make_out(Row row, int vs, int nv, bool pair) {
  return Out<Row>{row, vs, nv, pair};
}

// One folded pass over nvec vectors, shared out over the block's warps. X:
// element k of vector v at X[k * sk + v * sv]; vectors up to the next multiple
// of 8 must be readable (their results are dropped). FWD: outputs are mode
// positions, else natural indices.
//
// A warp takes the even and the odd fragment row of 16 outputs together, for NV
// tiles of 8 vectors: the two halves of a forward pass share one read of each
// mirrored pair, and an inverse pass has e and o of a mirrored pair in the same
// lane. The FP64 MMA sustains its full rate on dependent chains (64 clocks each
// per scheduler, measured), so what binds is shared memory: a fragment is 1 KB
// and a mirrored pair of data fragments 1 KB, 128 bytes per clock and SM against
// 16 clocks per MMA and SM: 1.5 KB per MMA at NV = 1, 1 KB at NV = 2 (with the
// halves on different warps it was 2 KB, and a 128 x 64 slab's x-pass 5100
// clocks). PIPE: operands of the next step are loaded ahead of a step's MMAs
// (more registers; the column kernels' passes are short and share the SM with
// many warps).
// The order of every sum depends on N only, so results do not depend on NV or
// on how vectors are dealt out.
template <bool FWD, int NV, bool PIPE, class O>
__device__ __forceinline__ void slab_pass(const double* P, int N, const double* X, int sk, int sv, int nvec, int warp,
                                          int nwarps, const O& out) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int h = half_up(N), l = N - h, MT = mtiles(N), KS = ksteps(N);
  const int nvt = (nvec + 7) / 8, ngrp = (nvt + NV - 1) / NV;
  if (nvec <= 0) return;
  struct Frag {
    double2 a[4];
    double x[NV][4];
  };
  int grp = 0, mt = warp;
  while (mt >= MT) {
    mt -= MT;
    ++grp;
  }
  while (grp < ngrp) {
    const int vt0 = grp * NV;
    const double* xv[NV];
    double ae[NV][4], ao[NV][4];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      xv[v] = X + (min(vt0 + v, nvt - 1) * 8 + g) * sv;
#pragma unroll
      for (int q = 0; q < 4; ++q) ae[v][q] = ao[v][q] = 0.0;
    }
    const double2* ap = reinterpret_cast<const double2*>(P) + (size_t)mt * KS * 128 + lane;
    auto load = [&](Frag& f, int ks) {
#pragma unroll
      for (int q = 0; q < 4; ++q) f.a[q] = ap[ks * 128 + 32 * q];
      // slices beyond a half's length meet zero matrix entries; their reads stay inside the vector
      const int k0 = min(8 * ks + t, h - 1), k1 = min(8 * ks + t + 4, h - 1);
      const int m0 = FWD ? N - 1 - k0 : h + min(k0, l - 1), m1 = FWD ? N - 1 - k1 : h + min(k1, l - 1);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        f.x[v][0] = xv[v][k0 * sk];
        f.x[v][1] = xv[v][k1 * sk];
        f.x[v][2] = xv[v][m0 * sk];
        f.x[v][3] = xv[v][m1 * sk];
      }
    };
    auto step = [&](const Frag& f) {
      const double fe[4] = {f.a[0].x, f.a[0].y, f.a[1].x, f.a[1].y}, fo[4] = {f.a[2].x, f.a[2].y, f.a[3].x, f.a[3].y};
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const double be[2] = {FWD ? f.x[v][0] + f.x[v][2] : f.x[v][0], FWD ? f.x[v][1] + f.x[v][3] : f.x[v][1]};
        const double bo[2] = {FWD ? f.x[v][0] - f.x[v][2] : f.x[v][2], FWD ? f.x[v][1] - f.x[v][3] : f.x[v][3]};
        mma_f64_m16n8k8(ae[v], fe, be);
        mma_f64_m16n8k8(ao[v], fo, bo);
      }
    };
    Frag f0;
    if (!PIPE) {
#pragma unroll 1
      for (int ks = 0; ks < KS; ++ks) {
        load(f0, ks);
        step(f0);
      }
    }
    Frag f1;
    if (PIPE) load(f0, 0);
#pragma unroll 1
    for (int ks = 0; PIPE && ks < KS; ks += 2) {
      if (ks + 1 < KS) load(f1, ks + 1);
      step(f0);
      if (ks + 1 < KS) {
        if (ks + 2 < KS) load(f0, ks + 2);
        step(f1);
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = 16 * mt + g + 8 * e;
      if (r >= h) continue;
      const bool two = FWD ? r < l : N - 1 - r != r;  // the second output: odd mode, or the mirrored index
      double* o0 = out.row(r);
      double* o1 = two ? out.row(FWD ? h + r : N - 1 - r) : o0;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        if (vt0 + v >= nvt) break;
        const int vec = (vt0 + v) * 8 + 2 * t;
        const double e0 = ae[v][2 * e], e1 = ae[v][2 * e + 1], q0 = ao[v][2 * e], q1 = ao[v][2 * e + 1];
        out.put(o0, vec, FWD ? e0 : e0 + q0, FWD ? e1 : e1 + q1);
        if (two) out.put(o1, vec, FWD ? q0 : e0 - q0, FWD ? q1 : e1 - q1);
      }
    }
    mt += nwarps;
    while (mt >= MT) {
      mt -= MT;
      ++grp;
    }
  }
}

// Vector tiles per task: two where there are two and that still leaves eight tasks
// (512 x 128 x 32, an iteration: 744 us with two for shares of one tile, 576 now).
template <bool FWD, class O>
__device__ __forceinline__ void slab_run(const double* P, int N, const double* X, int sk, int sv, int nvec, int warp,
                                         int nwarps, const O& out) {
  if (nvec > 8 && mtiles(N) * ((nvec + 15) / 16) >= 8) slab_pass<FWD, 2, true>(P, N, X, sk, sv, nvec, warp, nwarps, out);
  else slab_pass<FWD, 1, true>(P, N, X, sk, sv, nvec, warp, nwarps, out);
}

// Division of a slab over the n CTAs of its cluster: R mode rows (positions),
// C natural columns; offsets in doubles.
struct SlabShape {
  int nx, ny, n, R, C, ldr, ldc, o_xr, o_xt, o_m, keep, bytes;
};
inline SlabShape slab_shape(int nx, int ny, int n) {
  SlabShape f;
  f.nx = nx; f.ny = ny; f.n = n;
  f.R = ((ny + 7) / 8 + n - 1) / n * 8;
  f.C = ((nx + 7) / 8 + n - 1) / n * 8;
  f.ldr = fold::face_ld(nx);
  f.ldc = fold::face_ld(f.C);
  int o = ny * f.ldc;
  f.o_xr = o; o += f.R * f.ldr;
  f.o_xt = o; o += f.R * f.ldr;
  const size_t md = 2 * (fold::pack_doubles(nx) + fold::pack_doubles(ny));
  f.o_m = o;
  f.keep = (size_t)o + md <= (size_t)(fold::FACE_SMEM_MAX / 8 - 128);
  if (f.keep) o += (int)md;
  f.bytes = o * 8;
  return f;
}
// CTAs per slab: a slab on n CTAs takes about its share of the folded
// multiplications (64 a clock and SM, half as much again for the operands) plus
// 9000 clocks of loads, pointwise work and three cluster barriers, and the slabs
// run in waves of the clusters a B200 holds at one CTA per SM (its GPCs leave
// some SMs out of large clusters). Measured: 128 x 64 x 32, 2 steps: 11.3 ms at
// n = 4 (32 slabs, 33 clusters), 14.5 at 2, 21.1 at 8; 75 x 45 x 37, 4 steps: 4.3
// ms at 2, 5.3 at 4 (two waves). 0 where a slab does not fit.
inline int slab_cluster(int nx, int ny, int nz) {
  const int active[5] = {148, 74, 33, 15, 7};
  int best = 0;
  double t = 0.0;
  for (int k = 0; k < 5; ++k) {
    const int n = 1 << k;
    if (slab_shape(nx, ny, n).bytes > fold::FACE_SMEM_MAX - 1024) continue;
    const double c = ((nz + active[k] - 1) / active[k]) * (1.5 / 64.0 * nx * ny * (nx + ny) / n + 9000.0);
    if (!best || c < t) {
      best = n;
      t = c;
    }
  }
  return best;
}

// Clocks of one folded pass over nvec vectors on a CTA's 16 warps (64 per MMA and
// scheduler, two halves a step; see slab_run for the tiles of a task).
inline long slab_pass_clocks(int N, int nvec) {
  const int tiles = (nvec + 7) / 8, pairs = (nvec + 15) / 16;
  const bool two = nvec > 8 && mtiles(N) * pairs >= 8;
  const int tasks = mtiles(N) * (two ? pairs : tiles);
  return 128L * ksteps(N) * (two ? 2 : 1) * ((tasks + 3) / 4);
}
// Multiplications of one axis pass, padded to the tiles it takes (axis_shape).
inline double axis_padded(int N, long ncol) {
  const int tiles[4][2] = {{64, 128}, {64, 64}, {32, 128}, {32, 64}};
  double w = 0.0;
  for (int q = 0; q < 4; ++q) {
    const long r = (N + tiles[q][0] - 1) / tiles[q][0], c = (ncol + tiles[q][1] - 1) / tiles[q][1];
    w = (double)r * tiles[q][0] * c * tiles[q][1] * N;
    if (r * c >= AXM_SMS) break;
  }
  return w;
}
// Whether an FP64 plan's Picard iteration is shorter fused than with one pass per
// axis. The slab kernels contract half as much, but in waves of the clusters that the
// GPU holds, and a share of one tile more than its warps divide costs a round. Both
// sides' us are fitted to 45 of 75 measured volumes (latent heat and property correction;
// plans with one of the two cross at the same places). The bound leaves room for
// the fit's error, so that no measured volume is slower fused:
//   volume          estimate  passes / fused us an iteration
//   128 x 64 x 32     0.73       76 /   58
//   256 x 128 x 64    0.67      485 /  337
//   512 x 128 x 32    0.85      641 /  576
//   200 x 200 x 100   0.91     1169 / 1011
//   384 x 192 x 64    0.92     1177 / 1238
//   320 x 160 x 32    1.22      517 /  540
//   288 x 144 x 64    1.08      750 /  817
// Up to 16384 modes, and slabs below 1000, 14 small launches take no longer than five
// larger ones: 16 x 16 x 8 37 / 41, 32 x 16 x 16 40 / 42, 64 x 32 x 8 44 / 44, 23 x 25
// x 31 45 / 49; 48 x 24 x 16 48 / 43, 31 x 33 x 17 57 / 48.
inline bool slab_wins(int nx, int ny, int nz, int n) {
  const int active[5] = {148, 74, 33, 15, 7};
  int k = 0;
  while ((1 << k) < n) ++k;
  const SlabShape f = slab_shape(nx, ny, n);
  const double M = 1e-6 * nx * ny * nz;
  if (M <= 0.016384 || nx * ny < 1000) return false;
  const double clocks = ((nz + active[k] - 1) / active[k]) *
                        (2.0 * (slab_pass_clocks(nx, f.R) + slab_pass_clocks(ny, f.C)) + 9000.0);
  const double fused = 1.6e-3 * clocks + 62.0 * M + 25.0;
  const double passes = 0.066e-6 * 4.0 * (axis_padded(nx, (long)ny * nz) + axis_padded(ny, (long)nx * nz)) +
                        119.0 * M + 46.0;
  return fused <= 0.915 * passes;
}

struct SlabArgs {
  PointPhys P;
  const double *pxf, *pxi, *pyf, *pyi;
  const double* in;       // G or F (z-mode slabs, physical y, x); null: only the top flux
  const double* qnet;     // TRIAL*: net top flux
  double flux_scale;      // dct_scale / sqrt_dV
  const double *aK, *KK, *Ct, *Cb, *S_bot;
  double* a_trial;        // written by TRIAL, read by RELAX
  double* a_it;           // iterate (INIT reads it, *RELAX update it)
  double* Qm;             // QM: latent modes
  double* out;            // xy-inverse of the result
  double* partials;
  Ctrl* ctrl;             // QM: skipped when no iteration ran; *RELAX: convergence test
  cudaGraphConditionalHandle h_picard;
  int in_graph;
  unsigned wait_limit;    // polls of the operand wait
  bool stall_test;        // it first waits on a barrier that nothing completes
};

// Waits for the packed matrices' copies on bar[0], at most lim polls a thread. A
// thread whose wait ran out (or, with `stall`, that first waited on bar[1], which
// nothing completes) records it in *err and waits for the copies with the full
// bound, so that none outlives the CTA.
__device__ __forceinline__ void slab_operands(uint64_t* bar, unsigned lim, bool stall, int* err) {
  bool ok = !stall || umma::mbar_wait_bounded(&bar[1], 0u, lim);
  ok = ok && umma::mbar_wait_bounded(&bar[0], 0u, lim);
  if (!ok) {
    atomicExch(err, 1);
    umma::mbar_wait_bounded(&bar[0], 0u, umma::WAIT_LIMIT);
  }
}

// KEEP: the packed matrices are in shared memory (f.keep), else read from L2.
// An expired wait is recorded in ctrl->umma_err: the convergence test then ends the
// Picard loop, and the step reports SGH_STEP_TC_TIMEOUT.
template <int MODE, bool KEEP>
__global__ void __launch_bounds__(SLAB_THREADS, 1) k_slab(SlabShape f, SlabArgs q) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(128) double sl_sh[];
  __shared__ uint64_t bar[2];
  __shared__ double red[2 * (SLAB_THREADS / 32)];
  constexpr int NW = SLAB_THREADS / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = f.n, rank = (int)cl.block_rank(), p = blockIdx.x / n;
  const int nx = f.nx, ny = f.ny, ldr = f.ldr, ldc = f.ldc, R = f.R, C = f.C, S = nx * ny;
  const int r0 = rank * R, c0 = rank * C;
  const int nr = max(0, min(R, ny - r0)), nc = max(0, min(C, nx - c0));
  const float rR = 1.0f / (float)R, rC = 1.0f / (float)C;
  double* xin = sl_sh;
  double* xr = sl_sh + f.o_xr;
  double* xt = sl_sh + f.o_xt;
  const int nxp = (int)fold::pack_doubles(nx), nyp = (int)fold::pack_doubles(ny);
  const double* pyf = KEEP ? sl_sh + f.o_m : q.pyf;
  const double* pxf = KEEP ? sl_sh + f.o_m + nyp : q.pxf;
  const double* pxi = KEEP ? sl_sh + f.o_m + nyp + nxp : q.pxi;
  const double* pyi = KEEP ? sl_sh + f.o_m + nyp + 2 * nxp : q.pyi;
  // The packed matrices never change: their copies start before the wait for
  // the previous kernel.
  if (KEEP && tid == 0) {
    double* o = sl_sh + f.o_m;
    umma::mbar_init(&bar[0], 1);
    umma::mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    umma::mbar_expect_tx(&bar[0], 16 * (nxp + nyp));
    umma::bulk_g2s(o, q.pyf, 8 * nyp, &bar[0]);
    umma::bulk_g2s(o + nyp, q.pxf, 8 * nxp, &bar[0]);
    umma::bulk_g2s(o + nyp + nxp, q.pxi, 8 * nxp, &bar[0]);
    umma::bulk_g2s(o + nyp + 2 * nxp, q.pyi, 8 * nyp, &bar[0]);
  }
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  if (MODE == SLAB_QM && q.ctrl->iter <= 0) {  // the same for every CTA
    if (KEEP) {
      __syncthreads();
      slab_operands(bar, q.wait_limit, q.stall_test, &q.ctrl->umma_err);  // no copy outlives the CTA
    }
    return;
  }
  const size_t g0 = (size_t)p * S;
  if (MODE == SLAB_INIT) {
    for (int r = warp; r < nr; r += NW) {
      const double* row = q.a_it + g0 + (size_t)mode_at(r0 + r, ny) * nx;
      for (int x = lane; x < nx; x += 32) xt[r * ldr + pos_of(x, nx)] = row[x];
    }
  } else {
    const double fl = (MODE == SLAB_TRIAL || MODE == SLAB_TRIAL_RELAX) ? q.flux_scale * q.Ct[p] : 0.0;
    constexpr int U = 4;  // rows whose loads are in flight together
    for (int y0 = warp; y0 < ny; y0 += U * NW)
      for (int c = lane; c < nc; c += 32) {
        double v[U], w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int y = y0 + u * NW;
          const size_t j = (size_t)(y < ny ? y : y0) * nx + c0 + c;
          v[u] = (MODE == SLAB_RELAX || MODE == SLAB_QM || q.in) ? q.in[g0 + j] : 0.0;
          w[u] = (MODE == SLAB_TRIAL || MODE == SLAB_TRIAL_RELAX) ? q.qnet[j] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int y = y0 + u * NW;
          if (y < ny)
            xin[y * ldc + c] = (MODE == SLAB_TRIAL || MODE == SLAB_TRIAL_RELAX) ? fma(fl, w[u], v[u]) : v[u];
        }
      }
  }
  if (KEEP) {
    __syncthreads();  // the barriers are initialised
    slab_operands(bar, q.wait_limit, q.stall_test, &q.ctrl->umma_err);
  }
  cl.sync();  // the slab is loaded; every CTA runs before any remote write
  double s0 = 0.0, s1 = 0.0;
  if (MODE != SLAB_INIT) {
    // y-forward of this CTA's columns, to the row owners; x-forward of the mode rows
    slab_run<true>(pyf, ny, xin, ldc, 1, nc, warp, NW,
                   make_out(
                       [&](int y) {
                         const int dst = (int)(((float)y + 0.5f) * rR);
                         return cl.map_shared_rank(xr, dst) + (y - dst * R) * ldr + c0;
                       },
                       1, nc, true));
    cl.sync();
    slab_run<true>(pxf, nx, xr, 1, ldr, nr, warp, NW, make_out([&](int x) { return xt + x; }, ldr, nr, false));
    __syncthreads();
    // modal update; natural columns, so that the global arrays are read along x
    const int XB = (nx + 31) / 32;
    constexpr int U = 4;
    for (int t0 = warp; t0 < nr * XB; t0 += U * NW) {
      double kk[U], b0[U], b1[U], ol[U];
      int li[U];
      size_t gi[U];
      bool in[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t0 + u * NW, r = (int)(((float)t + 0.5f) / (float)XB), x = (t - r * XB) * 32 + lane;
        in[u] = t < nr * XB && x < nx;
        li[u] = in[u] ? r * ldr + pos_of(x, nx) : 0;
        gi[u] = in[u] ? (size_t)mode_at(r0 + r, ny) * nx + x : 0;
        const size_t j = g0 + gi[u];
        if (MODE != SLAB_QM) kk[u] = q.KK[j];
        if (MODE == SLAB_TRIAL || MODE == SLAB_TRIAL_RELAX) b0[u] = q.aK[j];
        if (MODE == SLAB_RELAX) b0[u] = q.a_trial[j];
        if (MODE == SLAB_TRIAL || MODE == SLAB_TRIAL_RELAX) b1[u] = q.S_bot ? q.Cb[p] * q.S_bot[gi[u]] : 0.0;
        if (MODE == SLAB_RELAX || MODE == SLAB_TRIAL_RELAX) ol[u] = q.a_it[j];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!in[u]) continue;
        const size_t j = g0 + gi[u];
        const double v = q.P.sqrt_dV * xt[li[u]];
        if (MODE == SLAB_QM) {
          q.Qm[j] = v;
          continue;
        }
        double t = fma(kk[u], v, b0[u]);  // aK + KK (Ct S_top + Q_m), or a_trial + KK C
        if ((MODE == SLAB_TRIAL || MODE == SLAB_TRIAL_RELAX) && q.S_bot) t = fma(kk[u], b1[u], t);
        // a mixed plan's iterates stay in FP64 here; the commit rounds the modes
        if (MODE == SLAB_TRIAL) {
          q.a_trial[j] = t;
        } else {  // relaxation (solvers/spectral.py:456-468)
          const double res = t - ol[u];
          t = res * q.P.omega + ol[u];
          q.a_it[j] = t;
          s0 = fma(res, res, s0);
          s1 = fma(ol[u], ol[u], s1);
        }
        xt[li[u]] = t;
      }
    }
    if (MODE == SLAB_QM) return;  // no remote access is pending: the last one was before the second barrier
    __syncthreads();
  }
  // x-inverse of the mode rows, to the column owners; y-inverse into the output
  slab_run<false>(pxi, nx, xt, 1, ldr, nr, warp, NW,
                  make_out(
                      [&](int x) {
                        const int dst = (int)(((float)x + 0.5f) * rC);
                        return cl.map_shared_rank(xin, dst) + (x - dst * C) + r0 * ldc;
                      },
                      ldc, nr, false));
  cl.sync();
  double* dst0 = q.out + g0 + c0;
  slab_run<false>(pyi, ny, xin, ldc, 1, nc, warp, NW,
                  make_out([&](int y) { return dst0 + (size_t)y * nx; }, 1, nc, (nx & 1) == 0));
  if (MODE == SLAB_TRIAL_RELAX || MODE == SLAB_RELAX) {
    // partials of this CTA; the CTA that draws the last ticket adds them all in
    // a fixed order and runs the convergence test (solvers/spectral.py:464-499).
    // No CTA waits for another.
    __shared__ int last;
    block_sum2<SLAB_THREADS>(s0, s1, red);
    if (tid == 0) {
      q.partials[2 * blockIdx.x] = s0;
      q.partials[2 * blockIdx.x + 1] = s1;
      __threadfence();
      last = atomicAdd(&q.ctrl->tickets, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    s0 = s1 = 0.0;
    for (int b = tid; b < (int)gridDim.x; b += SLAB_THREADS) {
      s0 += __ldcg(q.partials + 2 * b);
      s1 += __ldcg(q.partials + 2 * b + 1);
    }
    block_sum2<SLAB_THREADS>(s0, s1, red);
    if (tid == 0) {
      q.ctrl->tickets = 0u;
      const int stop = converge_test(*q.P.full, q.ctrl, s0, s1);
      if (q.in_graph) cudaGraphSetConditional(q.h_picard, stop ? 0u : 1u);
    }
  }
}

constexpr int COL_SMEM_MAX = 200 * 1024;  // largest dynamic shared memory of a column kernel

struct ColShape {
  int nx, ny, nz, cc, ld, bytes;
};
inline ColShape col_shape(int nx, int ny, int nz) {
  ColShape f;
  f.nx = nx; f.ny = ny; f.nz = nz;
  // 16 columns per CTA (two vector tiles) up to 14,208 columns: the pointwise physics
  // wants every warp slot of the SMs; 32 where that many CTAs fill them anyway
  f.cc = (long)nx * ny <= 16 * 148 * 6 ? 16 : 32;
  f.ld = fold::face_ld(f.cc);
  f.bytes = (nz + std::max(nz, COL_THREADS / f.cc)) * f.ld * 8;
  return f;
}

struct ColArgs {
  PointPhys P;
  const double *pzf, *pzi;  // packed z matrices
  const double* in;         // B or C (z-mode slabs)
  const double* Ct;
  double inv_sqrt_dV;
  int latent, rescale;
  const double* Tprev;
  const double* q_las;
  double *q_evap, *q_net;
  double* out;              // G or F
  double *T, *kp;           // TEMP writes them, STENCIL reads them
  double *Tprev_out, *T_surf, *q_evap_old;
  double* partials;
};

// f at (z, y, x) = div(k' grad T) - a'(T) (T - T_prev)/dt, the numpy.gradient
// (edge_order = 1) stencil applied twice (spectral_cpu_kernels.py:165-252).
__device__ __forceinline__ double stencil_f(const DevParams& D, const PointPhys& P, const double* __restrict__ T,
                                            const double* __restrict__ kp, int i, int z, int y, int x, double tprev) {
  auto g_at = [&](int q, int n, int st, int b0, double inv) -> double {
    double d;
    if (q == 0) d = (__ldg(T + b0 + st) - __ldg(T + b0)) * inv;
    else if (q == n - 1) d = (__ldg(T + b0 + (n - 1) * st) - __ldg(T + b0 + (n - 2) * st)) * inv;
    else d = (__ldg(T + b0 + (q + 1) * st) - __ldg(T + b0 + (q - 1) * st)) * (0.5 * inv);
    return __ldg(kp + b0 + q * st) * d;
  };
  auto div_axis = [&](int q, int n, int st, int b0, double inv) -> double {
    if (q == 0) return (g_at(1, n, st, b0, inv) - g_at(0, n, st, b0, inv)) * inv;
    if (q == n - 1) return (g_at(n - 1, n, st, b0, inv) - g_at(n - 2, n, st, b0, inv)) * inv;
    return (g_at(q + 1, n, st, b0, inv) - g_at(q - 1, n, st, b0, inv)) * (0.5 * inv);
  };
  const double dgx = div_axis(x, D.nx, 1, i - x, D.inv_dx);
  const double dgy = div_axis(y, D.ny, D.nx, i - y * D.nx, D.inv_dy);
  const double dgz = div_axis(z, D.nz, D.S, i - z * D.S, D.inv_dz);
  const double t = __ldg(T + i);
  return dgx + dgy + dgz - a_prime(P, t) * ((t - tprev) * P.inv_dt);
}

template <int MODE>
__global__ void __launch_bounds__(COL_THREADS, 4) k_column(ColShape f, ColArgs q) {
  extern __shared__ __align__(128) double cs_sh[];
  __shared__ double red[2 * (COL_THREADS / 32)];
  constexpr int NW = COL_THREADS / 32;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int nz = f.nz, S = f.nx * f.ny, ld = f.ld, cc = f.cc;
  const int col0 = blockIdx.x * cc, nc = min(cc, S - col0);
  double* b1 = cs_sh;              // [nz][ld] input
  double* b2 = cs_sh + nz * ld;    // [nz][ld] T halves, then the forward input
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  const int c = tid % cc, w0 = tid / cc, wn = COL_THREADS / cc;  // column c, z rows w0, w0 + wn, ...
  const bool in = c < nc;
  double mx = -INFINITY;
  if (MODE == COL_STENCIL) {
    const int yx = col0 + c, y = yx / f.nx, x = yx - y * f.nx;
    for (int z = w0; z < nz; z += wn)
      if (in) {
        const int i = z * S + yx;
        b2[z * ld + c] = stencil_f(*q.P.full, q.P, q.T, q.kp, i, z, y, x, __ldg(q.Tprev + i));
      }
    __syncthreads();
  } else {
    constexpr int U = 8;
    for (int z0 = w0; z0 < nz; z0 += U * wn) {
      double v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int z = z0 + u * wn;
        v[u] = in && z < nz ? q.in[(size_t)z * S + col0 + c] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        // b1 in position order (even modes first)
        const int z = z0 + u * wn;
        if (z < nz) b1[pos_of(z, nz) * ld + c] = v[u];
      }
    }
    __syncthreads();
    if (MODE == COL_LATENT || MODE == COL_COMMIT) {  // surface row: Ts = recon_scale sum_p Ct[p] B[p]
      double s = 0.0;
      for (int p = w0; p < nz; p += wn) s = fma(__ldg(q.Ct + mode_at(p, nz)), b1[p * ld + c], s);
      b2[w0 * ld + c] = s;  // b2 has at least wn rows
      __syncthreads();
      if (w0 == 0 && in) {
        for (int k = 1; k < wn; ++k) s += b2[k * ld + c];
        const double Ts = q.P.recon_scale * s;
        const int i = col0 + c;
        if (MODE == COL_LATENT) {  // solvers/spectral.py:388-407
          const double qe = evaporation(q.P, Ts);
          q.q_evap[i] = qe;
          const double qc = q.P.has_top_conv ? q.P.h_top * (Ts - q.P.T0) : 0.0;
          double fl = __ldg(q.q_las + i) - qe - qc;
          if (q.rescale) fl = fl * (q.P.kbar / k_blended(q.P, Ts));
          q.q_net[i] = fl;
        } else {
          q.T_surf[i] = Ts;
          q.q_evap_old[i] = q.q_evap[i];
          mx = Ts;
        }
      }
      __syncthreads();
    }
    if (MODE == COL_LATENT && !q.latent) return;
    slab_pass<false, 1, false>(q.pzi, nz, b1, ld, 1, nc, warp, NW, make_out([&](int z) { return b2 + z * ld; }, 1, cc, true));
    __syncthreads();
    for (int z = w0; z < nz; z += wn) {
      if (!in) break;
      const double T = b2[z * ld + c] * q.inv_sqrt_dV;
      const size_t i = (size_t)z * S + col0 + c;
      if (MODE == COL_LATENT) {
        b2[z * ld + c] = latent_source(q.P, T, __ldg(q.Tprev + i));
      } else if (MODE == COL_TEMP) {
        q.T[i] = T;
        q.kp[i] = k_prime(q.P, T);
      } else {
        q.Tprev_out[i] = T;
      }
    }
    if (MODE == COL_LATENT) __syncthreads();
  }
  if (MODE == COL_LATENT || MODE == COL_STENCIL) {
    double* o = q.out + col0;
    slab_pass<true, 1, false>(q.pzf, nz, b2, ld, 1, nc, warp, NW,
                   make_out([&](int p) { return o + (size_t)mode_at(p, nz) * S; }, 1, nc, (S & 1) == 0));
  }
  if (MODE == COL_COMMIT) {
    double d = 0.0;
    block_max_sum<COL_THREADS>(mx, d, red);
    if (tid == 0) {
      q.partials[2 * blockIdx.x] = mx;
      q.partials[2 * blockIdx.x + 1] = 0.0;
    }
  }
}

}  // namespace vol
}  // namespace sgh
