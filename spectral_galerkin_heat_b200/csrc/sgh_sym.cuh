// sgh_sym.cuh -- one axis of a cosine transform as an FP64 tensor-core
// contraction halved by the symmetry of the cosine matrix, for transforms of
// whole arrays (the stand-alone DCT and the node-centred output field).
//
// View the array as [A][N][B] with N the transformed axis, c = (a, b) a column.
//   inverse form: Mat (Nout x N, row-major) has Mat[Nout-1-j][n] = (-1)^n Mat[j][n]
//     (transposed DCT-II matrices, node matrices). For j in the lower half the
//     sums e over even n and o over odd n give out[j] = e + o, out[Nout-1-j] =
//     e - o.
//   forward form: the DCT-II matrix has Mat[k][N-1-n] = (-1)^k Mat[k][n]. Even
//     outputs contract X[n] + X[N-1-n], odd ones X[n] - X[N-1-n], over n < N/2.
// Half the multiplications of the full contraction.
//
// One CTA: 32 output pairs x 64 columns, 8 warps as 2 x 4, each 16 pairs x 16
// columns with an even and an odd accumulator (mma.sync m16n8k8 .f64; tcgen05
// has no FP64 kind). A stage holds 16 slice pairs: 1024 matrix elements and 32
// slices of 64 columns, by cp.async, SYM_STAGES deep. Row strides keep fragment
// reads free of bank conflicts: 1 KB of shared-memory reads per MMA against 128
// bytes a clock and 16 clocks per MMA and SM, so the FP64 pipe binds, and two
// CTAs per SM cover each other's prologue and epilogue. Results leave through
// shared memory along the output's contiguous direction, whose strides the
// caller gives, so that an array can be written transposed.
// Measured on a B200: the 512 x 256 x 64 node field 390 us (18 TFLOP/s of halved
// work; 443 with the middle output as one more pair) against 667 with full
// contractions and a transposing copy; DCT-II and
// DCT-III of a 96 x 60 x 100 volume 66 us against 86.
#pragma once
#include <algorithm>

#include "sgh_axis.cuh"
#include "sgh_limits.h"

namespace sgh {
namespace sym {

constexpr int THREADS = 256;
constexpr int BJ = 32;        // output pairs per CTA
constexpr int BC = 64;        // columns per CTA
constexpr int KP = 16;        // slice pairs per stage
constexpr int SYM_STAGES = 3;

template <bool CONTIG, bool FWD>
struct Lay {
  // FWD: 64 matrix rows (2j, 2j + 1) x 16 slices; else 32 rows x 32 slices
  static constexpr int MR = FWD ? 2 * BJ : BJ, MS = FWD ? KP : 2 * KP, LDM = FWD ? 18 : 40;
  // CONTIG: [column][slice], FWD in two halves (direct, mirrored); else [slice][column]
  static constexpr int LDX = CONTIG ? (FWD ? 20 : 40) : (FWD ? BC + 4 : BC + 2);
  static constexpr int XH = FWD ? (CONTIG ? BC * LDX : KP * LDX) : 0;  // mirrored half
  static constexpr int XSIZE = CONTIG ? (FWD ? 2 * BC * LDX : BC * LDX) : 2 * KP * LDX;
  static constexpr int STAGE = MR * LDM + XSIZE;
  static constexpr int TILE = 2 * BJ * (BC + 1);  // epilogue
  static constexpr int BYTES = (SYM_STAGES * STAGE > TILE + THREADS ? SYM_STAGES * STAGE : TILE + THREADS) * 8;
};

struct Args {
  const double *X, *Mat;
  double* out;
  int Nout, N, A, B;
  long long sa, sk;  // output element (a, k, b) at a * sa + k * sk + b
  int kfast;         // the output is contiguous along k (else along columns)
};

template <bool CONTIG, bool FWD>
__global__ void __launch_bounds__(THREADS, 2) k_sym(Args q) {
  using L = Lay<CONTIG, FWD>;
  extern __shared__ __align__(16) double sy[];
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3, wm = warp >> 2, wn = warp & 3;
  const int N = q.N, Nout = q.Nout, B = q.B, ncol = q.A * B;
  // output pairs (the middle output of an odd inverse form is not one), slices a
  // forward pass keeps
  const int H = FWD ? (Nout + 1) / 2 : Nout / 2, h = (N + 1) / 2;
  // The middle output has zero weights on the odd slices. It is summed by the CUDA
  // cores of the last row of CTAs from the staged slices: as one more pair it would
  // cost a tile of 32 (N / 2 + 1 pairs of a node matrix: 3 tiles of 32 for 64). The
  // odd slices are added with their zeros, so that a NaN or an infinity among them
  // reaches this output as it reaches every other.
  const bool mid = !FWD && (Nout & 1) && blockIdx.y == gridDim.y - 1;
  double msum = 0.0;
  const int c0 = blockIdx.x * BC, j0 = blockIdx.y * BJ;
  const int nch = (h + KP - 1) / KP;
  const bool vm = (N % 2 == 0) && (reinterpret_cast<uintptr_t>(q.Mat) % 16 == 0) && !(FWD && (h & 1));
  const bool vx = (CONTIG ? (N % 2 == 0 && !(FWD && (h & 1))) : (B % 2 == 0)) &&
                  (reinterpret_cast<uintptr_t>(q.X) % 16 == 0);

  // Matrix element (row r, slice s) of the stage at slice pair p0, and whether it exists.
  auto mat_at = [&](int r, int s, int p0, bool& ok) -> const double* {
    const int k = FWD ? 2 * j0 + r : j0 + r, n = FWD ? p0 + s : 2 * p0 + s;
    ok = (FWD ? k < Nout && n < h : k < H && n < N);
    return q.Mat + (size_t)(ok ? k : 0) * N + (ok ? n : 0);
  };
  // Slice of X for stage slice s (FWD: s < KP direct, above mirrored).
  auto slice_at = [&](int s, int p0, bool& ok) -> int {
    if (!FWD) {
      const int n = 2 * p0 + s;
      ok = n < N;
      return ok ? n : 0;
    }
    const int i = p0 + (s < KP ? s : s - KP), n = s < KP ? i : N - 1 - i;
    // the middle sample of an odd length is its own mirror: kept once
    ok = i < h && (s < KP || n != i);
    return ok ? n : 0;
  };
  auto issue = [&](int st, int p0) {
    double* Ms = sy + st * L::STAGE;
    double* Xs = Ms + L::MR * L::LDM;
    if (vm) {
      for (int e = tid; e < L::MR * L::MS / 2; e += THREADS) {
        const int r = e / (L::MS / 2), s = 2 * (e % (L::MS / 2));
        bool ok;
        const double* p = mat_at(r, s, p0, ok);
        cp_async16(&Ms[r * L::LDM + s], p, ok ? 16 : 0);
      }
    } else {
      for (int e = tid; e < L::MR * L::MS; e += THREADS) {
        const int r = e / L::MS, s = e % L::MS;
        bool ok;
        const double* p = mat_at(r, s, p0, ok);
        cp_async8(&Ms[r * L::LDM + s], p, ok ? 8 : 0);
      }
    }
    if (CONTIG) {
      // element (column, slice); the mirrored half is stored in memory order,
      // index 15 - i for pair i
      if (vx) {
        for (int e = tid; e < BC * KP; e += THREADS) {
          const int cr = e / KP, s2 = e % KP;  // pair of slices 2 s2, 2 s2 + 1 of the 32
          const int c = c0 + cr;
          bool ok = c < ncol;
          if (!FWD) {
            const int n = 2 * p0 + 2 * s2;
            ok = ok && n < N;
            cp_async16(&Xs[cr * L::LDX + 2 * s2], q.X + (size_t)(ok ? c : 0) * N + (ok ? n : 0), ok ? 16 : 0);
          } else if (s2 < KP / 2) {
            const int n = p0 + 2 * s2;
            ok = ok && n < h;
            cp_async16(&Xs[cr * L::LDX + 2 * s2], q.X + (size_t)(ok ? c : 0) * N + (ok ? n : 0), ok ? 16 : 0);
          } else {
            const int m = 2 * s2 - KP, i = p0 + KP - 1 - m;  // memory index m holds pairs i and i - 1
            const int n = N - 1 - i;
            // pairs beyond the half (i >= h) meet zero matrix entries and direct halves
            ok = ok && i < h;
            cp_async16(&Xs[L::XH + cr * L::LDX + m], q.X + (size_t)(ok ? c : 0) * N + (ok ? n : 0), ok ? 16 : 0);
          }
        }
      } else {
        for (int e = tid; e < BC * 2 * KP; e += THREADS) {
          const int cr = e / (2 * KP), s = e % (2 * KP), c = c0 + cr;
          bool ok;
          const int n = slice_at(s, p0, ok);
          ok = ok && c < ncol;
          double* d = FWD ? (s < KP ? &Xs[cr * L::LDX + s] : &Xs[L::XH + cr * L::LDX + 2 * KP - 1 - s])
                          : &Xs[cr * L::LDX + s];
          cp_async8(d, q.X + (size_t)(ok ? c : 0) * N + (ok ? n : 0), ok ? 8 : 0);
        }
      }
    } else {
      if (vx) {
        for (int e = tid; e < KP * BC; e += THREADS) {
          const int s = e / (BC / 2), cr = 2 * (e % (BC / 2)), c = c0 + cr;
          bool ok;
          const int n = slice_at(s, p0, ok);
          ok = ok && c < ncol;
          const int cc = ok ? c : 0, a = cc / B, b = cc - a * B;
          cp_async16(&Xs[s * L::LDX + cr], q.X + ((size_t)a * N + n) * B + b, ok ? 16 : 0);
        }
      } else {
        for (int e = tid; e < 2 * KP * BC; e += THREADS) {
          const int s = e / BC, cr = e % BC, c = c0 + cr;
          bool ok;
          const int n = slice_at(s, p0, ok);
          ok = ok && c < ncol;
          const int cc = ok ? c : 0, a = cc / B, b = cc - a * B;
          cp_async8(&Xs[s * L::LDX + cr], q.X + ((size_t)a * N + n) * B + b, ok ? 8 : 0);
        }
      }
    }
    cp_async_commit();
  };

  double ae[2][4], ao[2][4];
#pragma unroll
  for (int v = 0; v < 2; ++v)
#pragma unroll
    for (int i = 0; i < 4; ++i) ae[v][i] = ao[v][i] = 0.0;
  for (int st = 0; st < SYM_STAGES - 1; ++st) {
    if (st < nch) issue(st, st * KP);
    else cp_async_commit();
  }
  for (int ch = 0; ch < nch; ++ch) {
    cp_async_wait<SYM_STAGES - 2>();
    __syncthreads();
    const int nxt = ch + SYM_STAGES - 1;
    if (nxt < nch) issue(nxt % SYM_STAGES, nxt * KP);
    else cp_async_commit();
    const double* Ms = sy + (ch % SYM_STAGES) * L::STAGE;
    const double* Xs = Ms + L::MR * L::LDM;
    if (mid) {
      const int col = tid % BC;
#pragma unroll
      for (int i = 0; i < KP * BC / THREADS; ++i) {
        const int s = 2 * (tid / BC + (THREADS / BC) * i), n = 2 * KP * ch + s;
        // the odd slice beyond the length is staged as zero
        const double x1 = CONTIG ? Xs[col * L::LDX + s + 1] : Xs[(s + 1) * L::LDX + col];
        if (n < N) msum = fma(__ldg(q.Mat + (size_t)(Nout / 2) * N + n), CONTIG ? Xs[col * L::LDX + s] : Xs[s * L::LDX + col], msum);
        msum = fma(0.0, x1, msum);
      }
    }
#pragma unroll
    for (int k8 = 0; k8 < KP; k8 += 8) {
      double fe[4], fo[4];
      const int jr = wm * 16 + g;
      if (FWD) {
        const double* m0 = Ms + 2 * jr * L::LDM + k8 + t;
        const double* m1 = m0 + 16 * L::LDM;
        fe[0] = m0[0]; fe[1] = m1[0]; fe[2] = m0[4]; fe[3] = m1[4];
        fo[0] = m0[L::LDM]; fo[1] = m1[L::LDM]; fo[2] = m0[L::LDM + 4]; fo[3] = m1[L::LDM + 4];
      } else {
        const double* m0 = Ms + jr * L::LDM + 2 * (k8 + t);
        const double* m1 = m0 + 8 * L::LDM;
        const double2 p0 = *reinterpret_cast<const double2*>(m0), p1 = *reinterpret_cast<const double2*>(m1);
        const double2 p2 = *reinterpret_cast<const double2*>(m0 + 8), p3 = *reinterpret_cast<const double2*>(m1 + 8);
        fe[0] = p0.x; fe[1] = p1.x; fe[2] = p2.x; fe[3] = p3.x;
        fo[0] = p0.y; fo[1] = p1.y; fo[2] = p2.y; fo[3] = p3.y;
      }
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const int col = wn * 16 + v * 8 + g;
        double be[2], bo[2];
        if (CONTIG && !FWD) {
          const double2 x0 = *reinterpret_cast<const double2*>(Xs + col * L::LDX + 2 * (k8 + t));
          const double2 x1 = *reinterpret_cast<const double2*>(Xs + col * L::LDX + 2 * (k8 + t) + 8);
          be[0] = x0.x; be[1] = x1.x;
          bo[0] = x0.y; bo[1] = x1.y;
        } else if (!FWD) {
          const double* x = Xs + 2 * (k8 + t) * L::LDX + col;
          be[0] = x[0]; be[1] = x[8 * L::LDX];
          bo[0] = x[L::LDX]; bo[1] = x[9 * L::LDX];
        } else {
          const double *x = CONTIG ? Xs + col * L::LDX + k8 + t : Xs + (k8 + t) * L::LDX + col;
          const double *y = CONTIG ? Xs + L::XH + col * L::LDX + KP - 1 - k8 - t : Xs + L::XH + (k8 + t) * L::LDX + col;
          const int s4 = CONTIG ? 4 : 4 * L::LDX, m4 = CONTIG ? -4 : 4 * L::LDX;
          const double u0 = x[0], u1 = x[s4], w0 = y[0], w1 = y[m4];
          be[0] = u0 + w0; be[1] = u1 + w1;
          bo[0] = u0 - w0; bo[1] = u1 - w1;
        }
        mma_f64_m16n8k8(ae[v], fe, be);
        mma_f64_m16n8k8(ao[v], fo, bo);
      }
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  // tile row r: FWD output 2 j0 + r; else output j0 + r for r < 32 and, ascending,
  // the mirrored outputs: Nout - 1 - (j0 + 63 - r)
  double* tile = sy;
  constexpr int LDT = BC + 1;
#pragma unroll
  for (int v = 0; v < 2; ++v)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int jr = wm * 16 + g + 8 * (i >> 1), col = wn * 16 + v * 8 + 2 * t + (i & 1);
      tile[(FWD ? 2 * jr : jr) * LDT + col] = FWD ? ae[v][i] : ae[v][i] + ao[v][i];
      tile[(FWD ? 2 * jr + 1 : 2 * BJ - 1 - jr) * LDT + col] = FWD ? ao[v][i] : ae[v][i] - ao[v][i];
    }
  if (mid) tile[L::TILE + tid] = msum;
  __syncthreads();
  if (mid && tid < BC && c0 + tid < ncol) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < THREADS / BC; ++i) s += tile[L::TILE + BC * i + tid];
    const int c = c0 + tid, a = CONTIG ? c : c / B, b = CONTIG ? 0 : c - a * B;
    q.out[a * q.sa + (Nout / 2) * q.sk + b] = s;
  }
  for (int e = tid; e < 2 * BJ * BC; e += THREADS) {
    const int r = q.kfast ? e % (2 * BJ) : e / BC, cr = q.kfast ? e / (2 * BJ) : e % BC;
    const int c = c0 + cr;
    int k;
    bool ok = c < ncol;
    if (FWD) {
      k = 2 * j0 + r;
      ok = ok && k < Nout;
    } else if (r < BJ) {
      k = j0 + r;
      ok = ok && k < H;
    } else {
      const int j = j0 + 2 * BJ - 1 - r;
      k = Nout - 1 - j;
      ok = ok && j < H;
    }
    if (ok) {
      const int a = CONTIG ? c : c / B, b = CONTIG ? 0 : c - a * B;
      q.out[a * q.sa + k * q.sk + b] = tile[r * LDT + cr];
    }
  }
}

// Whether a pass has enough CTAs for k_sym: past 128 its CTAs' chains of chunks are
// longer than those of launch_axis's smaller tiles, and under about 100 CTAs they
// leave SMs idle besides. A pair of transforms with every pass on the full
// contraction, with k_sym from 40 CTAs, with k_sym from 100: 512 x 512 (64 CTAs a
// pass) 96, 101, 82 us; 400 x 400 (49) 82, 87, 66; 20 x 600 x 20 (70) 89, 94, 77;
// 600 x 600 (100) 156, 119, 119; 30 x 600 x 20 (100) 115, 95, 95. Node field of 600 x
// 20 x 20 (70 CTAs in its x-pass) 48, 50, 44 us, of 1000 x 10 x 10 (32) 61, 81, 69.
constexpr int MIN_CTAS = 100;
inline bool fills(int Nout, int N, long long ncol) {
  const long long ctas = ((ncol + BC - 1) / BC) * ((std::max(1, (Nout + 1) / 2) + BJ - 1) / BJ);
  return N <= 128 || ctas >= MIN_CTAS;
}

// One pass; kind: 2 forward (DCT-II matrix), 3 inverse form. Output element (a, k, b)
// at a * sa + k * sk + b; kfast when that is contiguous along k.
template <bool CONTIG, bool FWD>
inline void launch_one(const Args& q, cudaStream_t st) {
  using L = Lay<CONTIG, FWD>;
  (void)kernel_limits(reinterpret_cast<const void*>(k_sym<CONTIG, FWD>), L::BYTES);
  const int H = FWD ? (q.Nout + 1) / 2 : std::max(1, q.Nout / 2);
  const dim3 grid((unsigned)(((long long)q.A * q.B + BC - 1) / BC), (unsigned)((H + BJ - 1) / BJ));
  launch_pdl(k_sym<CONTIG, FWD>, grid, THREADS, L::BYTES, st, q);
}
inline void launch(int kind, const double* X, const double* Mat, double* out, int Nout, int N, int A, int B,
                   long long sa, long long sk, bool kfast, cudaStream_t st) {
  const Args q = {X, Mat, out, Nout, N, A, B, sa, sk, kfast ? 1 : 0};
  if (B == 1) kind == 2 ? launch_one<true, true>(q, st) : launch_one<true, false>(q, st);
  else kind == 2 ? launch_one<false, true>(q, st) : launch_one<false, false>(q, st);
}

}  // namespace sym
}  // namespace sgh
