// In-shared-memory batched 1D FFT passes built from the register codelets.
//
// A length-L transform with L = L1 * L2 is two passes of small DFTs (the
// "four-step" split without the reordering step):
//
//   inverse, natural in -> permuted out (SIGN +1)
//     pass 1: for each n1 < L1: DFT_L2 over x[n1 + L1 n2], times W[n1][k2],
//             stored back at n1 + L1 k2
//     pass 2: for each k2 < L2: DFT_L1 over the block [L1 k2, L1 k2 + L1)
//   forward, permuted in -> natural out (SIGN -1)
//     pass A: for each a < L2: DFT_L1 over the block [L1 a, L1 a + L1),
//             output c times conj(W[c][a])
//     pass B: for each c < L1: DFT_L2 over x[c + L1 a] -> natural index c + L1 d
//
// with W[i][j] = exp(+2 pi i i j / L).  Real-space index r = a + L2 b lives at
// position L1 a + b ("digit-permuted" order); every pass reads and writes the
// same addresses from one thread, so a pass needs no barrier inside it.
//
// All data and twiddles live in the kernel's dynamic shared memory and are
// addressed by element offsets from its base, so every access is a plain
// shared-memory load or store.
#pragma once

#include "block_fixed.cuh"
#include "codelets.cuh"
#include "qgb_common.cuh"

namespace qgb {

extern __shared__ __align__(16) unsigned char qgb_smem[];

// n / d by a multiplication, for n d < 2^32 and d >= 2 (a pass's items over its
// columns; the compiler's own division by a run-time d is some 20 instructions
// per item).
struct FastDiv {
  unsigned d, m;
  __device__ __forceinline__ explicit FastDiv(int divisor) : d(divisor), m(divisor > 1 ? 0xFFFFFFFFu / divisor + 1 : 0) {}
  __device__ __forceinline__ int quot(int n) const { return d > 1 ? static_cast<int>(__umulhi(n, m)) : n; }
};

template <typename T> __device__ __forceinline__ cplx_t<T>* smem_c() {
  return reinterpret_cast<cplx_t<T>*>(qgb_smem);
}

// One codelet applied in place to smem[off + j * stride], j < R, with an
// optional twiddle multiply by smem[tw + j * tw_stride] (tw < 0: none) on the
// outputs; the table holds exp(+i...) (pack_twiddle's form), conjugated when
// SIGN < 0.
template <typename T, int S, int R>
__device__ __forceinline__ void codelet_inplace(int off, int stride, int tw, int tw_stride, int lim,
                                                int tw_lim) {
  cplx_t<T>* sm = smem_c<T>();
  T re[R], im[R];
#pragma unroll
  for (int j = 0; j < R; ++j) {
    if (!QGB_OK_IDX(off + j * stride, lim, 10 + R)) return;
    const cplx_t<T> v = sm[off + j * stride];
    re[j] = v.x;
    im[j] = v.y;
  }
  Block<T, R> x;
  x.load(re, im);
  x.template run<S>();
  if (tw >= 0) {
#pragma unroll
    for (int j = 1; j < R; ++j) {
      if (!QGB_OK_IDX(tw + j * tw_stride, tw_lim, 40 + R)) return;
      x.template twiddle<S>(j, sm[tw + j * tw_stride]);
    }
  }
  x.store([&](int j, auto value) { sm[off + j * stride] = value(); });
}

// Geometry of one pass: item `it` in [0, nbatch * nsub) is (batch = it % nbatch,
// sub = it / nbatch); its codelet elements sit at shared offsets
//   base + boff(batch) + sub * sstride + j * estride,
// boff(batch) = (bmap ? bmap[batch] : batch) * bstride, bmap in global memory.
struct Pass {
  const int* bmap;
  int base, nbatch, bstride, nsub, sstride, estride;
  int tw, tw_sub, tw_el;  // tw < 0: no twiddles
  int lim, tw_lim;        // bounds of the data and twiddle regions (debug checks)
};

template <typename T, int S, int R>
__device__ __forceinline__ void run_pass_R(const Pass ps) {
  const int nitems = ps.nbatch * ps.nsub;
  const FastDiv div(ps.nbatch);
  for (int it = threadIdx.x; it < nitems; it += blockDim.x) {
    const int sub = div.quot(it);
    const int b = it - sub * ps.nbatch;
    const int boff = (ps.bmap != nullptr ? __ldg(ps.bmap + b) : b) * ps.bstride;
    codelet_inplace<T, S, R>(ps.base + boff + sub * ps.sstride, ps.estride,
                             ps.tw >= 0 ? ps.tw + sub * ps.tw_sub : -1, ps.tw_el, ps.lim, ps.tw_lim);
  }
}

template <typename T, int S>
__device__ __forceinline__ void run_pass(int R, const Pass ps) {
  switch (R) {
    case 2: run_pass_R<T, S, 2>(ps); break;
    case 3: run_pass_R<T, S, 3>(ps); break;
    case 4: run_pass_R<T, S, 4>(ps); break;
    case 5: run_pass_R<T, S, 5>(ps); break;
    case 6: run_pass_R<T, S, 6>(ps); break;
    case 7: run_pass_R<T, S, 7>(ps); break;
    case 8: run_pass_R<T, S, 8>(ps); break;
    case 9: run_pass_R<T, S, 9>(ps); break;
    case 10: run_pass_R<T, S, 10>(ps); break;
    case 12: run_pass_R<T, S, 12>(ps); break;
    case 14: run_pass_R<T, S, 14>(ps); break;
    case 15: run_pass_R<T, S, 15>(ps); break;
    case 16: run_pass_R<T, S, 16>(ps); break;
    default: break;  // R == 1: identity
  }
}

// One axis of nbatch pencils starting at shared offset `base`, element stride
// es: inverse (S > 0, natural -> permuted) or forward (S < 0, permuted ->
// natural); twiddles at shared offset W; `lim` bounds the data region.  Ends
// with __syncthreads().  The FP64 form runs both passes through one copy of the
// pass code (14 long codelets); in FP32 a copy each is 9% faster.
template <typename T, int S>
__device__ __forceinline__ void fft_axis(int base, const int* bmap, int nbatch, int bstride, int es, int L1, int L2,
                                         int W, int lim) {
  if constexpr (sizeof(T) == 8) {
    const bool single = L1 == 1 || L2 == 1;
#pragma unroll 1
    for (int i = single ? 1 : 0; i < 2; ++i) {
      const bool strided = !single && (i == 0) == (S > 0);  // DFT_L2 over x[n1 + L1 n2]; else DFT_L1 over blocks
      const bool tw = !single && i == 0;
      Pass ps{bmap, base, nbatch, bstride, strided ? L1 : L2, strided ? es : L1 * es, strided ? L1 * es : es,
              tw ? W : -1, S > 0 ? L2 : 1, S > 0 ? 1 : L2, lim, W + L1 * L2};
      if (single) {
        ps.nsub = 1;
        ps.estride = es;
      }
      run_pass<T, S>(single ? L1 * L2 : strided ? L2 : L1, ps);
      __syncthreads();
    }
  } else if constexpr (S > 0) {
    if (L2 > 1) {
      run_pass<T, +1>(L2, Pass{bmap, base, nbatch, bstride, L1, es, L1 * es, W, L2, 1, lim, W + L1 * L2});
      __syncthreads();
    }
    if (L1 > 1) {
      run_pass<T, +1>(L1, Pass{bmap, base, nbatch, bstride, L2, L1 * es, es, -1, 0, 0, lim, 0});
      __syncthreads();
    }
  } else {
    if (L1 > 1) {
      run_pass<T, -1>(L1, Pass{bmap, base, nbatch, bstride, L2, L1 * es, es, (L2 > 1) ? W : -1, 1, L2, lim,
                               W + L1 * L2});
      __syncthreads();
    }
    if (L2 > 1) {
      run_pass<T, -1>(L2, Pass{bmap, base, nbatch, bstride, L1, es, L1 * es, -1, 0, 0, lim, 0});
      __syncthreads();
    }
  }
}

}  // namespace qgb
