// Band-space complex products on the CUDA cores: the overlap (Gram) products
// of Wavefunction.dot and the projections <beta|psi>, the band rotations of
// Wavefunction.matmul and the back-projection beta (D proj), and the
// block-diagonal D apply.
//
// Replaces (qimpy/dft/electrons/_wavefunction_dot.py:18-107, 137-191;
// _wavefunction.py:106-123; qimpy/dft/electrons/_hamiltonian.py:22-24):
//   gram    out(i, j) = sum_g conj(A[i][g]) B[j][g]     (long g, small i/j)
//   rotate  out[j][g] (+)= sum_i W(i, j) X[i][g]         (short i, long g)
//   dapply  Dp[b][a pa + r] = sum_c D[a][r][c] proj[b][a pa + c]
// Arrays are batched over k-points with explicit strides.  GB300's FP64 rate
// (about 1 TFLOP/s) bounds the FP64 forms here, register-tiled multiply-add
// loops with shared-memory staging; larger FP64 products given a workspace go
// to the tensor cores instead (ozaki.cu).  The FP32 forms use the same tiling.
// Every product is deterministic: split-K partial tiles are summed by a
// second kernel in a fixed order (no atomics), so repeated calls, and calls
// from different host threads, give identical bits.
#include <algorithm>
#include <type_traits>

#include "bandgemm.cuh"

namespace qgb {
namespace bg {

constexpr int kSms = 152;  // GB300 streaming multiprocessors

template <typename T>
__device__ __forceinline__ void cmac_conj(cplx_t<T>& acc, const cplx_t<T>& a, const cplx_t<T>& b) {
  // acc += conj(a) * b
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(-a.y, b.x, acc.y);
}
template <typename T>
__device__ __forceinline__ void cmac(cplx_t<T>& acc, const cplx_t<T>& a, const cplx_t<T>& b) {
  // acc += a * b
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(-a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(a.y, b.x, acc.y);
}

// ---------------------------------------------------------------------------
// Gram / projection: out(i, j) = sum_g conj(A[i][g]) B[j][g]
// ---------------------------------------------------------------------------
//
// CTA: BI (i) x BJ (j) outputs of one k and one g range (split-K), 256
// threads as TI x TJ (TI TJ = 256), each 4 x 4 outputs: 64 x 64 in general,
// 128 x 32 or 32 x 128 when one side has at most 32 rows (the projections of
// a 32-band block), so that no thread multiplies padding.  g is staged 16 at a
// time: A and B tiles are loaded along g (coalesced rows) and stored
// transposed, [g][i] and [g][j], so each thread reads 4 consecutive i (or j)
// per g.
constexpr int GK = 16;   // g per stage
constexpr int GPAD = 1;  // row padding (elements) of the transposed tiles

struct GramArgs {
  const void* A;
  const void* B;
  long long a_batch, b_batch;  // element strides between k-points
  int lda, ldb;                // element stride between rows i (A) / j (B)
  int M, N, K;                 // i, j, g extents
  int splits, g_per_split;     // split-K (g_per_split a multiple of GK)
  void* partial;               // splits > 1: [split][k][M][N] of cplx_t<T>
  void* out;                   // splits == 1: OutT at out + k*out_batch + i*oi + j*oj
  long long out_batch;
  int oi, oj;
  const double* weight;        // optional per-g weight w_g (shared by all k): sum_g w_g conj(A) B
  int real_out;                // keep only the real part (imaginary part written as 0)
};

template <typename T, typename OutT, int TI>
__global__ void __launch_bounds__(256) k_gram(const GramArgs a) {
  using C2 = cplx_t<T>;
  using O2 = cplx_t<OutT>;
  constexpr int TJ = 256 / TI, BI = 4 * TI, BJ = 4 * TJ;
  __shared__ C2 As[GK][BI + GPAD];
  __shared__ C2 Bs[GK][BJ + GPAD];
  const int tid = threadIdx.x, tx = tid % TJ, ty = tid / TJ;
  const int i0 = blockIdx.x * BI, j0 = blockIdx.y * BJ;
  const int k = blockIdx.z / a.splits, split = blockIdx.z % a.splits;
  const int g_begin = split * a.g_per_split;
  const int g_end = min(a.K, g_begin + a.g_per_split);
  const C2* A = static_cast<const C2*>(a.A) + k * a.a_batch;
  const C2* B = static_cast<const C2*>(a.B) + k * a.b_batch;
  C2 acc[4][4];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[p][q] = mk<T>(T(0), T(0));
  for (int g0 = g_begin; g0 < g_end; g0 += GK) {
#pragma unroll
    for (int r = 0; r < BI * GK / 256; ++r) {
      const int e = tid + 256 * r, row = e >> 4, gg = e & 15, g = g0 + gg;
      As[gg][row] = (g < g_end && i0 + row < a.M) ? A[static_cast<long long>(i0 + row) * a.lda + g]
                                                  : mk<T>(T(0), T(0));
    }
#pragma unroll
    for (int r = 0; r < BJ * GK / 256; ++r) {
      const int e = tid + 256 * r, row = e >> 4, gg = e & 15, g = g0 + gg;
      const bool g_ok = g < g_end;
      C2 bv = (g_ok && j0 + row < a.N) ? B[static_cast<long long>(j0 + row) * a.ldb + g] : mk<T>(T(0), T(0));
      if (a.weight != nullptr && g_ok) {
        const T w = static_cast<T>(a.weight[g]);
        bv.x *= w;
        bv.y *= w;
      }
      Bs[gg][row] = bv;
    }
    __syncthreads();
#pragma unroll
    for (int gg = 0; gg < GK; ++gg) {
      C2 av[4], bv[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) av[p] = As[gg][ty * 4 + p];
#pragma unroll
      for (int q = 0; q < 4; ++q) bv[q] = Bs[gg][tx * 4 + q];
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) cmac_conj<T>(acc[p][q], av[p], bv[q]);
    }
    __syncthreads();
  }
  if (a.splits == 1) {
    O2* out = static_cast<O2*>(a.out) + k * a.out_batch;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int i = i0 + ty * 4 + p;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int j = j0 + tx * 4 + q;
        if (i < a.M && j < a.N)
          out[static_cast<long long>(i) * a.oi + static_cast<long long>(j) * a.oj] =
              mk<OutT>(static_cast<OutT>(acc[p][q].x), a.real_out ? OutT(0) : static_cast<OutT>(acc[p][q].y));
      }
    }
  } else {
    const int nk = gridDim.z / a.splits;
    C2* part = static_cast<C2*>(a.partial) + (static_cast<long long>(split) * nk + k) * a.M * a.N;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int i = i0 + ty * 4 + p;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int j = j0 + tx * 4 + q;
        if (i < a.M && j < a.N) part[static_cast<long long>(i) * a.N + j] = acc[p][q];
      }
    }
  }
}

// Sum of the split-K partials in split order (accumulated in OutT's precision
// or better), written with the caller's output strides.
template <typename T, typename OutT>
__global__ void k_gram_reduce(const cplx_t<T>* __restrict__ partial, int splits, int nk, int M, int N,
                              cplx_t<OutT>* __restrict__ out, long long out_batch, int oi, int oj, int real_out) {
  using Acc = typename std::conditional<sizeof(T) >= sizeof(OutT), T, OutT>::type;
  const long long per_k = static_cast<long long>(M) * N;
  const long long total = per_k * nk;
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int k = static_cast<int>(e / per_k);
    const long long r = e - k * per_k;
    const int i = static_cast<int>(r / N), j = static_cast<int>(r - static_cast<long long>(i) * N);
    Acc re = 0, im = 0;
    for (int s = 0; s < splits; ++s) {
      const cplx_t<T> v = partial[(static_cast<long long>(s) * nk + k) * per_k + r];
      re += static_cast<Acc>(v.x);
      im += static_cast<Acc>(v.y);
    }
    out[k * out_batch + static_cast<long long>(i) * oi + static_cast<long long>(j) * oj] =
        mk<OutT>(static_cast<OutT>(re), real_out ? OutT(0) : static_cast<OutT>(im));
  }
}

// Small overlaps: a CTA takes TI x TJ outputs, its threads run along g, and the
// sums are folded across the lanes (each step halves the values a lane keeps,
// so TI TJ complex sums cost about as many additions) and then the 8 warps.
// The 64 x 64 tiles above would multiply padding and leave most SMs idle (k = 8
// times 8 x 18 outputs over 1150 g: 517 us against 14 us here).  A few outputs
// over a long basis are split over g as well (launch_gram_small): 4 x 3 over
// 37073 is 4 tiles, 148 us on as many SMs, 11 us in 38 parts.
template <typename T, typename OutT, int TI, int TJ>
__global__ void __launch_bounds__(256) k_gram_small(const GramArgs a) {
  using C2 = cplx_t<T>;
  using Acc = typename std::conditional<sizeof(T) >= sizeof(OutT), T, OutT>::type;
  constexpr int V = 2 * TI * TJ;
  __shared__ Acc red[8][V];
  const int nj = (a.N + TJ - 1) / TJ;
  const int i0 = (blockIdx.x / nj) * TI, j0 = (blockIdx.x % nj) * TJ, k = blockIdx.y, split = blockIdx.z;
  const int g_end = min(a.K, (split + 1) * a.g_per_split);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const C2* A = static_cast<const C2*>(a.A) + k * a.a_batch;
  const C2* B = static_cast<const C2*>(a.B) + k * a.b_batch;
  C2 acc[TI][TJ];
#pragma unroll
  for (int p = 0; p < TI; ++p)
#pragma unroll
    for (int q = 0; q < TJ; ++q) acc[p][q] = mk<T>(T(0), T(0));
  for (int g = split * a.g_per_split + threadIdx.x; g < g_end; g += 256) {
    C2 av[TI], bv[TJ];
#pragma unroll
    for (int p = 0; p < TI; ++p) av[p] = A[static_cast<long long>(min(i0 + p, a.M - 1)) * a.lda + g];
#pragma unroll
    for (int q = 0; q < TJ; ++q) bv[q] = B[static_cast<long long>(min(j0 + q, a.N - 1)) * a.ldb + g];
    if (a.weight != nullptr) {
      const T w = static_cast<T>(a.weight[g]);
#pragma unroll
      for (int q = 0; q < TJ; ++q) {
        bv[q].x *= w;
        bv[q].y *= w;
      }
    }
#pragma unroll
    for (int p = 0; p < TI; ++p)
#pragma unroll
      for (int q = 0; q < TJ; ++q) cmac_conj<T>(acc[p][q], av[p], bv[q]);
  }
  Acc v[V];
#pragma unroll
  for (int p = 0; p < TI; ++p)
#pragma unroll
    for (int q = 0; q < TJ; ++q) {
      v[2 * (p * TJ + q)] = static_cast<Acc>(acc[p][q].x);
      v[2 * (p * TJ + q) + 1] = static_cast<Acc>(acc[p][q].y);
    }
  int n = V;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (n > 1) {
      n /= 2;
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < V / 2; ++i)
        if (i < n) {
          const Acc send = up ? v[i] : v[i + n];
          v[i] = (up ? v[i + n] : v[i]) + __shfl_xor_sync(0xffffffffu, send, o);
        }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  if (lane % (32 / V) == 0) red[warp][lane / (32 / V)] = v[0];
  __syncthreads();
  if (threadIdx.x < TI * TJ) {
    const int i = i0 + threadIdx.x / TJ, j = j0 + threadIdx.x % TJ;
    Acc re = red[0][2 * threadIdx.x], im = red[0][2 * threadIdx.x + 1];
#pragma unroll
    for (int w = 1; w < 8; ++w) {
      re += red[w][2 * threadIdx.x];
      im += red[w][2 * threadIdx.x + 1];
    }
    if (i >= a.M || j >= a.N) return;
    if (a.splits > 1)
      static_cast<cplx_t<Acc>*>(a.partial)[((static_cast<long long>(split) * gridDim.y + k) * a.M + i) * a.N + j] =
          mk<Acc>(re, im);
    else
      static_cast<cplx_t<OutT>*>(a.out)[k * a.out_batch + static_cast<long long>(i) * a.oi +
                                        static_cast<long long>(j) * a.oj] =
          mk<OutT>(static_cast<OutT>(re), a.real_out ? OutT(0) : static_cast<OutT>(im));
  }
}

// Sum of its partials: a warp an output, lane l those of splits l, l + 32, ...
template <typename T, typename OutT>
__global__ void __launch_bounds__(256) k_gram_small_reduce(const GramArgs a, int nk) {
  using Acc = typename std::conditional<sizeof(T) >= sizeof(OutT), T, OutT>::type;
  const long long per_k = static_cast<long long>(a.M) * a.N, e = blockIdx.x * 8ll + (threadIdx.x >> 5);
  if (e >= per_k * nk) return;
  const int lane = threadIdx.x & 31;
  Acc re = 0, im = 0;
  for (int s = lane; s < a.splits; s += 32) {
    const cplx_t<Acc> v = static_cast<const cplx_t<Acc>*>(a.partial)[s * per_k * nk + e];
    re += v.x;
    im += v.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    re += __shfl_xor_sync(0xffffffffu, re, o);
    im += __shfl_xor_sync(0xffffffffu, im, o);
  }
  const long long k = e / per_k, r = e - k * per_k, i = r / a.N, j = r - i * a.N;
  if (lane == 0)
    static_cast<cplx_t<OutT>*>(a.out)[k * a.out_batch + i * a.oi + j * a.oj] =
        mk<OutT>(static_cast<OutT>(re), a.real_out ? OutT(0) : static_cast<OutT>(im));
}

struct GramPlan {
  int shape;  // threads along i: 16 (64 x 64 tiles), 32 (128 x 32) or 8 (32 x 128)
  int ti, tj, splits, g_per_split;
  size_t partial_bytes;
};
static GramPlan gram_plan(int nk, int M, int N, int K, size_t elem) {
  GramPlan p;
  // Skinny tiles for skinny outputs; otherwise the tile shape that pads the
  // output least (M = 256 projectors x N = 160 bands: 128 x 32 tiles cover it
  // exactly, 64 x 64 tiles would compute 20% more), the square 64 x 64 tile
  // on ties, as its loads feed the most multiply-adds.
  auto padded = [M, N](int shape) {
    const long long bi = 4 * shape, bj = 4 * (256 / shape);
    return ((M + bi - 1) / bi) * bi * ((N + bj - 1) / bj) * bj;
  };
  p.shape = (N <= 32 && M > 32) ? 32 : ((M <= 32 && N > 32) ? 8 : 16);
  for (const int shape : {16, 32, 8})
    if (padded(shape) < padded(p.shape)) p.shape = shape;
  const int bi = 4 * p.shape, bj = 4 * (256 / p.shape);
  p.ti = (M + bi - 1) / bi;
  p.tj = (N + bj - 1) / bj;
  const int tiles = p.ti * p.tj * nk;
  const int kchunks = (K + GK - 1) / GK;
  // Enough CTAs for two waves over the SMs, with at least 8 stages of g each.
  int splits = std::max(1, std::min((2 * kSms + tiles - 1) / tiles, (kchunks + 7) / 8));
  const int chunks_per_split = (kchunks + splits - 1) / splits;
  p.g_per_split = chunks_per_split * GK;
  p.splits = (K + p.g_per_split - 1) / p.g_per_split;
  if (p.splits < 1) p.splits = 1;
  p.partial_bytes = p.splits > 1 ? static_cast<size_t>(p.splits) * nk * M * N * elem : 0;
  return p;
}

// ---------------------------------------------------------------------------
// Rotation / back-projection: out[j][g] (+)= sum_i W(i, j) X[i][g]
// ---------------------------------------------------------------------------
//
// CTA: TJ*8 (j) x 128 (g) outputs of one k, 256 threads as 32 (g) x 8 (j);
// each thread TJ j-values x 4 consecutive g.  i is staged 16 at a time: the
// X tile [16][128] along g (coalesced), the W tile [16][TJ*8].
constexpr int RG = 128;
constexpr int RK = 16;

struct RotArgs {
  const void* X;
  const void* W;
  void* out;
  long long x_batch, w_batch, out_batch;  // element strides between k-points
  int ldx, ldo;                           // element stride between rows i (X) / j (out)
  int wi, wj;                             // W(i, j) = W[i*wi + j*wj]
  int Kin, Nout, G;                       // i, j, g extents
  int accumulate;
};

template <typename T, int TJ>
__global__ void __launch_bounds__(256) k_rotate(const RotArgs a) {
  using C2 = cplx_t<T>;
  constexpr int BJ = TJ * 8;
  __shared__ C2 Xs[RK][RG];
  __shared__ C2 Ws[RK][BJ];
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  const int g0 = blockIdx.x * RG, j0 = blockIdx.y * BJ, k = blockIdx.z;
  const C2* X = static_cast<const C2*>(a.X) + k * a.x_batch;
  const C2* W = static_cast<const C2*>(a.W) + k * a.w_batch;
  C2 acc[TJ][4];
#pragma unroll
  for (int p = 0; p < TJ; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[p][q] = mk<T>(T(0), T(0));
  for (int i0 = 0; i0 < a.Kin; i0 += RK) {
#pragma unroll
    for (int r = 0; r < RK * RG / 256; ++r) {
      const int e = tid + 256 * r, ii = e / RG, gg = e % RG;
      const int i = i0 + ii, g = g0 + gg;
      Xs[ii][gg] = (i < a.Kin && g < a.G) ? X[static_cast<long long>(i) * a.ldx + g] : mk<T>(T(0), T(0));
    }
    for (int e = tid; e < RK * BJ; e += 256) {
      const int ii = e / BJ, jj = e % BJ, i = i0 + ii, j = j0 + jj;
      Ws[ii][jj] = (i < a.Kin && j < a.Nout) ? W[static_cast<long long>(i) * a.wi + static_cast<long long>(j) * a.wj]
                                             : mk<T>(T(0), T(0));
    }
    __syncthreads();
#pragma unroll 4
    for (int ii = 0; ii < RK; ++ii) {
      C2 xv[4], wv[TJ];
#pragma unroll
      for (int q = 0; q < 4; ++q) xv[q] = Xs[ii][tx * 4 + q];
#pragma unroll
      for (int p = 0; p < TJ; ++p) wv[p] = Ws[ii][ty * TJ + p];
#pragma unroll
      for (int p = 0; p < TJ; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) cmac<T>(acc[p][q], wv[p], xv[q]);
    }
    __syncthreads();
  }
  C2* out = static_cast<C2*>(a.out) + k * a.out_batch;
#pragma unroll
  for (int p = 0; p < TJ; ++p) {
    const int j = j0 + ty * TJ + p;
    if (j >= a.Nout) continue;
    C2* row = out + static_cast<long long>(j) * a.ldo;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int g = g0 + tx * 4 + q;
      if (g < a.G) {
        C2 v = acc[p][q];
        if (a.accumulate) {
          const C2 o = row[g];
          v.x += o.x;
          v.y += o.y;
        }
        row[g] = v;
      }
    }
  }
}

// Small rotations: one g and TJ j a thread, W broadcast.  (The 32 x 128 tiles
// above multiply padding and fill few SMs: 71 us for 8 x 18 over 1150 g and 8 k.)
// The FP64 pipe's 2 multiply-adds a clock and SM bound it, so the SM with the
// most threads times outputs does: the host picks TJ and the CTA size by that
// (pick_rotate_small; 10.9 -> 5.1 us for 12 x 6 over 300 g and 2 k, where CTAs of
// 64 x 4 would occupy 20 SMs).
// NL, the back-projection: W(i, j) = sum_c D[atom(i)][i % pa][c] proj[j][c], put in
// shared memory by each CTA for its TJ columns.  It repeats pa of every 64 (32)
// multiply-adds and saves k_dapply and its launch (3 to 4 us).
template <typename T, int TJ, bool NL>
__global__ void __launch_bounds__(64) k_rotate_small(const RotArgs a, const cplx_t<T>* __restrict__ D, int pa) {
  using C2 = cplx_t<T>;
  extern __shared__ __align__(16) unsigned char small_smem[];
  C2* Ws = reinterpret_cast<C2*>(small_smem);  // [TJ][Kin]
  const int g = blockIdx.x * blockDim.x + threadIdx.x, j0 = blockIdx.y * TJ, k = blockIdx.z;
  const C2* Wk = static_cast<const C2*>(a.W) + k * a.w_batch;
  if constexpr (NL) {
    for (int e = threadIdx.x; e < TJ * a.Kin; e += blockDim.x) {
      const int p = e / a.Kin, i = e - p * a.Kin, atom = i / pa;
      const C2* x = Wk + static_cast<long long>(min(j0 + p, a.Nout - 1)) * a.wj + atom * pa;
      const C2* d = D + static_cast<long long>(i) * pa;
      C2 acc = mk<T>(T(0), T(0));
      for (int c = 0; c < pa; ++c) cmac<T>(acc, d[c], x[c]);
      Ws[e] = acc;
    }
    __syncthreads();
  }
  if (g >= a.G) return;
  const C2* X = static_cast<const C2*>(a.X) + k * a.x_batch + g;
  const C2* W[TJ];
#pragma unroll
  for (int p = 0; p < TJ; ++p)
    W[p] = NL ? Ws + p * a.Kin : Wk + static_cast<long long>(min(j0 + p, a.Nout - 1)) * a.wj;
  const long long wi = NL ? 1 : a.wi;
  C2 acc[TJ];
#pragma unroll
  for (int p = 0; p < TJ; ++p) acc[p] = mk<T>(T(0), T(0));
#pragma unroll 4
  for (int i = 0; i < a.Kin; ++i) {
    const C2 x = X[static_cast<long long>(i) * a.ldx];
#pragma unroll
    for (int p = 0; p < TJ; ++p) cmac<T>(acc[p], W[p][i * wi], x);
  }
  C2* out = static_cast<C2*>(a.out) + k * a.out_batch + g;
#pragma unroll
  for (int p = 0; p < TJ; ++p) {
    if (j0 + p >= a.Nout) break;
    C2& o = out[static_cast<long long>(j0 + p) * a.ldo];
    if (a.accumulate) {
      acc[p].x += o.x;
      acc[p].y += o.y;
    }
    o = acc[p];
  }
}

// Dp[k][b][a*pa + r] = sum_c D[a][r][c] proj[k][b][a*pa + c]  (one thread per output)
template <typename T>
__global__ void k_dapply(const cplx_t<T>* __restrict__ proj, const cplx_t<T>* __restrict__ D, int n_atoms, int pa,
                         int nb, int nk, cplx_t<T>* __restrict__ Dp) {
  const int P = n_atoms * pa;
  const long long total = static_cast<long long>(nk) * nb * P;
  for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long kb = e / P;
    const int p = static_cast<int>(e - kb * P), atom = p / pa, r = p - atom * pa;
    const cplx_t<T>* x = proj + kb * P + atom * pa;
    const cplx_t<T>* d = D + (static_cast<long long>(atom) * pa + r) * pa;
    cplx_t<T> acc = mk<T>(T(0), T(0));
    for (int c = 0; c < pa; ++c) cmac<T>(acc, d[c], x[c]);
    Dp[e] = acc;
  }
}

}  // namespace bg

using namespace bg;

size_t gram_workspace_bytes(int dtype, int nk, int M, int N, int K, bool sliced) {
  if (nk < 1 || M < 1 || N < 1 || K < 1) return 0;
  const size_t partial = gram_plan(nk, M, N, K, elem_bytes(dtype)).partial_bytes;
  if (!sliced || dtype != QGB_F64 || !oz_gram_use(nk, M, N, K)) return partial;
  return std::max(partial, std::max(oz_gram_workspace_bytes(nk, M, N, K, false),
                                    oz_gram_workspace_bytes(nk, M, N, K, true)));
}

size_t rotate_workspace_bytes(int dtype, int nk, int Kin, int Nout, int G) {
  if (nk < 1 || Kin < 1 || Nout < 1 || G < 1 || dtype != QGB_F64 || !oz_rotate_use(nk, Kin, Nout, G)) return 0;
  return oz_rotate_workspace_bytes(nk, Kin, Nout, G);
}

template <typename T, typename OutT>
static void launch_gram(int shape, dim3 grid, const GramArgs& g, cudaStream_t st) {
  if (shape == 32)
    k_gram<T, OutT, 32><<<grid, 256, 0, st>>>(g);
  else if (shape == 8)
    k_gram<T, OutT, 8><<<grid, 256, 0, st>>>(g);
  else
    k_gram<T, OutT, 16><<<grid, 256, 0, st>>>(g);
}

// Products small enough that the FP64 pipe of all SMs takes about as long as
// the launches of the sliced form (ozaki.cu has both sides).
static bool small_product(int nk, int M, int N, int K, double limit = kSmallOverlap) {
  return static_cast<double>(nk) * M * N * K < limit && nk <= 65535;
}

// Work of the SM that gets the most of `ctas` equal CTAs.  `work` counts an
// output's multiply-add as 1 in FP64 (2 a clock and SM, nothing else is near);
// in FP32 the loads cost more than the multiply-adds, so larger tiles are kept
// longer.
static long long most_loaded(long long ctas, int work) { return (ctas + kSms - 1) / kSms * work; }

// The tile that loads the fullest SM least, the larger one on a tie: 8 x 18
// outputs of 8 k are 160 tiles of 2 x 4, two on 8 of the SMs, or 288 of 2 x 2,
// also two but half the size (1150 g, FP64: 23.7 -> 13.6 us).
// g is split where the tiles leave SMs idle, into as many parts as give no SM two
// of them, if that saves more than the second launch costs (9000 clocks): 256 g
// take a tile 512 clocks per output in FP64, 250 in all in FP32.  One part and
// split, us: 4 x 3 over 37073 FP64 148 and 11 (FP32 23 and 7), 16 x 16 over 10000 44
// and 27 (FP32, not split: 9.0 and 9.0), 18 x 18 over 8000 FP32, not split: 7.8 and 11.
struct GramSmall {
  int ti, tj, splits, g_per_split;
};
static GramSmall pick_gram_small(bool f64, int nk, int M, int N, int K, int max_splits) {
  GramSmall best{4, 4, 1, K};
  long long least = -1, ctas = 0;
  for (const GramSmall& c : {GramSmall{4, 4, 1, K}, GramSmall{2, 4, 1, K}, GramSmall{2, 2, 1, K}}) {
    const long long n = static_cast<long long>((M + c.ti - 1) / c.ti) * ((N + c.tj - 1) / c.tj) * nk;
    const long long cost = most_loaded(n, f64 ? c.ti * c.tj : c.ti * c.tj + 2 * (c.ti + c.tj));
    if (least < 0 || cost < least) {
      least = cost;
      best = c;
      ctas = n;
    }
  }
  const long long iterations = (K + 255) / 256;
  const long long s = std::min({static_cast<long long>(max_splits), iterations, kSms / ctas});
  if (s > 1 && (iterations - iterations / s) * (f64 ? 512 * best.ti * best.tj : 250) > 9000)
    best.g_per_split = static_cast<int>((iterations + s - 1) / s) * 256;
  best.splits = (K + best.g_per_split - 1) / best.g_per_split;
  return best;
}

template <typename T, typename OutT>
static int launch_gram_small(GramArgs g, int nk, int max_splits, cudaStream_t st) {
  const GramSmall p = pick_gram_small(sizeof(T) == 8, nk, g.M, g.N, g.K, max_splits);
  g.splits = p.splits;
  g.g_per_split = p.g_per_split;
  const dim3 grid(static_cast<unsigned>((g.M + p.ti - 1) / p.ti) * static_cast<unsigned>((g.N + p.tj - 1) / p.tj), nk,
                  p.splits);
  if (p.ti == 4)
    k_gram_small<T, OutT, 4, 4><<<grid, 256, 0, st>>>(g);
  else if (p.tj == 4)
    k_gram_small<T, OutT, 2, 4><<<grid, 256, 0, st>>>(g);
  else
    k_gram_small<T, OutT, 2, 2><<<grid, 256, 0, st>>>(g);
  QGB_LAUNCH_CHECK("k_gram_small");
  if (p.splits > 1) {
    const long long outputs = static_cast<long long>(nk) * g.M * g.N;
    k_gram_small_reduce<T, OutT><<<static_cast<unsigned>((outputs + 7) / 8), 256, 0, st>>>(g, nk);
    QGB_LAUNCH_CHECK("k_gram_small_reduce");
  }
  return QGB_OK;
}

// Columns a thread and threads a CTA of k_rotate_small, by the same rule: 4, 2 or
// 1 columns of 64 threads, or 1 of 32.
struct RotSmall {
  int tj, threads;
};
static RotSmall pick_rotate_small(int dtype, int nk, int Nout, int G) {
  RotSmall best{4, 64};
  long long least = -1;
  for (const RotSmall c : {RotSmall{4, 64}, RotSmall{2, 64}, RotSmall{1, 64}, RotSmall{1, 32}}) {
    const long long ctas = static_cast<long long>((G + c.threads - 1) / c.threads) * ((Nout + c.tj - 1) / c.tj) * nk;
    const long long cost = most_loaded(ctas, c.threads * (dtype == QGB_F64 ? c.tj : 2 * c.tj + 2));
    if ((Nout + c.tj - 1) / c.tj <= 65535 && (least < 0 || cost < least)) {
      least = cost;
      best = c;
    }
  }
  return best;
}

template <typename T, bool NL>
static void launch_rotate_small(const RotArgs& r, int nk, const void* D, int pa, RotSmall c, cudaStream_t st) {
  const dim3 grid((r.G + c.threads - 1) / c.threads, (r.Nout + c.tj - 1) / c.tj, nk);
  const size_t smem = NL ? static_cast<size_t>(c.tj) * r.Kin * sizeof(cplx_t<T>) : 0;
  const cplx_t<T>* d = static_cast<const cplx_t<T>*>(D);
  if (c.tj == 4)
    k_rotate_small<T, 4, NL><<<grid, c.threads, smem, st>>>(r, d, pa);
  else if (c.tj == 2)
    k_rotate_small<T, 2, NL><<<grid, c.threads, smem, st>>>(r, d, pa);
  else
    k_rotate_small<T, 1, NL><<<grid, c.threads, smem, st>>>(r, d, pa);
}

// out(i, j) of type out_dtype (complex) = sum_g conj(A(i, g)) B(j, g), per k.
int gram(int dtype, int out_dtype, const void* A, long long a_batch, int lda, const void* B, long long b_batch,
         int ldb, int nk, int M, int N, int K, void* out, long long out_batch, int oi, int oj, void* ws,
         size_t ws_bytes, cudaStream_t st, const double* weight, bool real_out) {
  if (nk < 0 || M < 0 || N < 0 || K < 0) return fail(QGB_ERR_INVALID, "negative gram extent");
  if (nk == 0 || M == 0 || N == 0) return QGB_OK;
  if (!A || !B || !out) return fail(QGB_ERR_INVALID, "NULL pointer in gram");
  if (dtype != QGB_F64 && dtype != QGB_F32) return fail(QGB_ERR_INVALID, "unknown dtype %d", dtype);
  if (out_dtype != QGB_F64 && out_dtype != QGB_F32) return fail(QGB_ERR_INVALID, "unknown out dtype %d", out_dtype);
  if (dtype == QGB_F64 && out_dtype == QGB_F32) return fail(QGB_ERR_UNSUPPORTED, "FP64 gram to FP32 output");
  if (K == 0) return fail(QGB_ERR_INVALID, "gram over an empty basis");
  const GramPlan p = gram_plan(nk, M, N, K, elem_bytes(dtype));
  if (p.splits > 1 && (!ws || ws_bytes < p.partial_bytes))
    return fail(QGB_ERR_WORKSPACE, "gram workspace %zu B < %zu B", ws_bytes, p.partial_bytes);
  if (dtype == QGB_F64 && ws && oz_gram_use(nk, M, N, K) &&
      ws_bytes >= oz_gram_workspace_bytes(nk, M, N, K, real_out))
    return oz_gram(A, a_batch, lda, B, b_batch, ldb, nk, M, N, K, out, out_batch, oi, oj, ws, st, weight, real_out);
  if (small_product(nk, M, N, K)) {
    const GramArgs g{A, B, a_batch, b_batch, lda, ldb, M, N, K, 1, K, ws, out, out_batch, oi, oj, weight,
                     real_out ? 1 : 0};
    // Its partial sums have the result's precision; the workspace holds p.splits of the operands'.
    const size_t acc = elem_bytes(out_dtype);
    const int room = reinterpret_cast<uintptr_t>(ws) % acc ? 1 : static_cast<int>(p.splits * elem_bytes(dtype) / acc);
    if (dtype == QGB_F64) return launch_gram_small<double, double>(g, nk, std::max(1, room), st);
    if (out_dtype == QGB_F64) return launch_gram_small<float, double>(g, nk, std::max(1, room), st);
    return launch_gram_small<float, float>(g, nk, std::max(1, room), st);
  }
  GramArgs g{A, B, a_batch, b_batch, lda, ldb, M, N, K, p.splits, p.g_per_split, ws, out, out_batch, oi, oj,
             weight, real_out ? 1 : 0};
  const dim3 grid(p.ti, p.tj, nk * p.splits);
  if (dtype == QGB_F64) {
    launch_gram<double, double>(p.shape, grid, g, st);
  } else if (out_dtype == QGB_F64) {
    launch_gram<float, double>(p.shape, grid, g, st);
  } else {
    launch_gram<float, float>(p.shape, grid, g, st);
  }
  QGB_LAUNCH_CHECK("k_gram");
  if (p.splits > 1) {
    const long long total = static_cast<long long>(nk) * M * N;
    const unsigned blocks = static_cast<unsigned>(std::min<long long>((total + 255) / 256, 8 * kSms));
    if (dtype == QGB_F64) {
      k_gram_reduce<double, double><<<blocks, 256, 0, st>>>(static_cast<const double2*>(ws), p.splits, nk, M, N,
                                                            static_cast<double2*>(out), out_batch, oi, oj, g.real_out);
    } else if (out_dtype == QGB_F64) {
      k_gram_reduce<float, double><<<blocks, 256, 0, st>>>(static_cast<const float2*>(ws), p.splits, nk, M, N,
                                                           static_cast<double2*>(out), out_batch, oi, oj, g.real_out);
    } else {
      k_gram_reduce<float, float><<<blocks, 256, 0, st>>>(static_cast<const float2*>(ws), p.splits, nk, M, N,
                                                          static_cast<float2*>(out), out_batch, oi, oj, g.real_out);
    }
    QGB_LAUNCH_CHECK("k_gram_reduce");
  }
  return QGB_OK;
}

// out[k][j][g] (+)= sum_i W(i, j) X[k][i][g] with W(i, j) = W[k*w_batch + i*wi + j*wj].
int rotate(int dtype, const void* X, long long x_batch, int ldx, const void* W, long long w_batch, int wi, int wj,
           int nk, int Kin, int Nout, int G, void* out, long long out_batch, int ldo, bool accumulate,
           cudaStream_t st, void* ws, size_t ws_bytes) {
  if (nk < 0 || Kin < 0 || Nout < 0 || G < 0) return fail(QGB_ERR_INVALID, "negative rotate extent");
  if (nk == 0 || Nout == 0 || G == 0) return QGB_OK;
  if (!out || (Kin > 0 && (!X || !W))) return fail(QGB_ERR_INVALID, "NULL pointer in rotate");
  if (dtype == QGB_F64 && Kin > 0 && ws && oz_rotate_use(nk, Kin, Nout, G) &&
      ws_bytes >= oz_rotate_workspace_bytes(nk, Kin, Nout, G))
    return oz_rotate(X, x_batch, ldx, W, w_batch, wi, wj, nk, Kin, Nout, G, out, out_batch, ldo, accumulate, ws, st);
  RotArgs r{X, W, out, x_batch, w_batch, out_batch, ldx, ldo, wi, wj, Kin, Nout, G, accumulate ? 1 : 0};
  if (small_product(nk, Kin, Nout, G, kSmallRotation) && (Nout + 3) / 4 <= 65535 && (dtype == QGB_F64 || dtype == QGB_F32)) {
    const RotSmall c = pick_rotate_small(dtype, nk, Nout, G);
    if (dtype == QGB_F64)
      launch_rotate_small<double, false>(r, nk, nullptr, 0, c, st);
    else
      launch_rotate_small<float, false>(r, nk, nullptr, 0, c, st);
    QGB_LAUNCH_CHECK("k_rotate_small");
    return QGB_OK;
  }
  if (dtype == QGB_F64) {
    constexpr int TJ = 4;
    const dim3 grid((G + RG - 1) / RG, (Nout + TJ * 8 - 1) / (TJ * 8), nk);
    k_rotate<double, TJ><<<grid, 256, 0, st>>>(r);
  } else if (dtype == QGB_F32) {
    constexpr int TJ = 8;
    const dim3 grid((G + RG - 1) / RG, (Nout + TJ * 8 - 1) / (TJ * 8), nk);
    k_rotate<float, TJ><<<grid, 256, 0, st>>>(r);
  } else {
    return fail(QGB_ERR_INVALID, "unknown dtype %d", dtype);
  }
  QGB_LAUNCH_CHECK("k_rotate");
  return QGB_OK;
}

bool backproject_small_use(int nk, int n_atoms, int pa, int nb, int n_tot) {
  const long long P = static_cast<long long>(n_atoms) * pa;
  return pa <= 8 && P <= 512 && small_product(nk, static_cast<int>(P), nb, n_tot) && (nb + 3) / 4 <= 65535;
}

int backproject_small(int dtype, const void* beta, const void* D, int n_atoms, int pa, const void* projT, void* out,
                      int nk, int nb, int n_tot, cudaStream_t st) {
  const int P = n_atoms * pa;
  const RotArgs r{beta, projT, out, static_cast<long long>(P) * n_tot, static_cast<long long>(nb) * P,
                  static_cast<long long>(nb) * n_tot, n_tot, n_tot, 1, P, P, nb, n_tot, 1};
  const RotSmall c = pick_rotate_small(dtype, nk, nb, n_tot);
  if (dtype == QGB_F64)
    launch_rotate_small<double, true>(r, nk, D, pa, c, st);
  else
    launch_rotate_small<float, true>(r, nk, D, pa, c, st);
  QGB_LAUNCH_CHECK("k_rotate_small");
  return QGB_OK;
}

int dapply(int dtype, const void* proj, const void* D, int n_atoms, int pa, int nb, int nk, void* Dp,
           cudaStream_t st) {
  const long long total = static_cast<long long>(nk) * nb * n_atoms * pa;
  if (total == 0) return QGB_OK;
  const unsigned blocks = static_cast<unsigned>(std::min<long long>((total + 255) / 256, 8 * kSms));
  if (dtype == QGB_F64)
    k_dapply<double><<<blocks, 256, 0, st>>>(static_cast<const double2*>(proj), static_cast<const double2*>(D),
                                             n_atoms, pa, nb, nk, static_cast<double2*>(Dp));
  else
    k_dapply<float><<<blocks, 256, 0, st>>>(static_cast<const float2*>(proj), static_cast<const float2*>(D), n_atoms,
                                            pa, nb, nk, static_cast<float2*>(Dp));
  QGB_LAUNCH_CHECK("k_dapply");
  return QGB_OK;
}

}  // namespace qgb
