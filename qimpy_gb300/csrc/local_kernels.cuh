// Device code and launches of the local-potential kernels (local_potential.cu
// describes them).  Each precision and form is compiled in a translation unit
// of its own: local_f32.cu, local_f64.cu, batched_f32.cu, batched_f64.cu and the
// two density ones.
#pragma once

#include <algorithm>
#include <cmath>

#include "fft_steps.cuh"
#include "packed_f32.cuh"

namespace qgb {

static constexpr int kThreads = 256;

struct LocalParams {
  int nb_total;  // bands in C / out (stride of the band axis)
  int b0;        // first band of this chunk
  int nb;        // bands in this chunk
  unsigned flags;
};

template <typename T>
__device__ __forceinline__ void load_twiddles(int dst, const cplx_t<T>* src, int count) {
  cplx_t<T>* sm = smem_c<T>();
  for (int i = threadIdx.x; i < count; i += blockDim.x) sm[dst + i] = pack_twiddle(src[i]);
}

// Sphere points a thread of the scatter and the gather takes at a time: the
// gather's loads may alias its stores, so only loads written before the first
// store overlap.  1 -> 4, FP32 us: 72^3, 800 bands, scatter and its transforms 447
// -> 408, gather and its transforms 514 -> 485; 96^3, 160 bands 196 -> 181 and 211
// -> 204 (2 points: 188 and 207); 36^3, 57 points a slab, and FP64 within 1%.
constexpr int kPoints = 4;

// Plane workspace index of (k, band-in-chunk, slab).
__device__ __forceinline__ size_t plane_index(const qgb_sphere& s, int k, int b, int nb, int slab) {
  return (static_cast<size_t>(k) * nb + b) * s.max_slabs + slab;
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))),
               "l"(gsrc)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One complex element global -> shared without a register round trip (8 B
// for FP32, 16 B for FP64): many copies stay in flight per thread.
template <typename T>
__device__ __forceinline__ void cp_async_elem(cplx_t<T>* smem_dst, const cplx_t<T>* gsrc) {
  if constexpr (sizeof(cplx_t<T>) == 16) {
    cp_async16(smem_dst, gsrc);
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))),
                 "l"(gsrc)
                 : "memory");
  }
}


// ---------------------------------------------------------------------------
// y passes of the y/z kernels with the plane's boundaries folded in (used when
// both y factors exceed 1).  Rows y of the shared plane sit at offset y * ld,
// columns c < nz; `rowmask[y]` marks the rows the slab's sphere points touch.
// ---------------------------------------------------------------------------

// Inverse pass 1 (radix R = L2) over rows sub + j * L1 with the pass-1
// twiddles; untouched rows are read as zero (they are never zero-filled).
template <typename T, int R>
__device__ __forceinline__ void ypass_inv1_R(const int* rowmask, int nz, int L1, int ld, int W, int lim) {
  cplx_t<T>* sm = smem_c<T>();
  const int nitems = nz * L1;
  const FastDiv div(nz);
  for (int it = threadIdx.x; it < nitems; it += blockDim.x) {
    const int sub = div.quot(it);
    const int c = it - sub * nz;
    T re[R], im[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int y = sub + j * L1;
      const int off = y * ld + c;
      if (!QGB_OK_IDX(off, lim, 64)) return;
      cplx_t<T> v = mk<T>(T(0), T(0));
      if (rowmask[y]) v = sm[off];
      re[j] = v.x;
      im[j] = v.y;
    }
    Block<T, R> x;
    x.load(re, im);
    x.template run<+1>();
#pragma unroll
    for (int j = 1; j < R; ++j) x.template twiddle<+1>(j, sm[W + sub * R + j]);
    x.store([&](int j, auto value) { sm[(sub + j * L1) * ld + c] = value(); });
  }
}

// Inverse pass 2 (radix R = L1) over rows sub * L1 + j, stored straight to the
// plane in global memory (row stride N2), in the permuted order of the rows.
template <typename T, int R>
__device__ __forceinline__ void ypass_inv2_R(cplx_t<T>* __restrict__ out, int N2, int nz, int L2, int ld, int lim) {
  cplx_t<T>* sm = smem_c<T>();
  const int nitems = nz * L2;
  const FastDiv div(nz);
  for (int it = threadIdx.x; it < nitems; it += blockDim.x) {
    const int sub = div.quot(it);
    const int c = it - sub * nz;
    T re[R], im[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int off = (sub * R + j) * ld + c;
      if (!QGB_OK_IDX(off, lim, 65)) return;
      const cplx_t<T> v = sm[off];
      re[j] = v.x;
      im[j] = v.y;
    }
    Block<T, R> x;
    x.load(re, im);
    x.template run<+1>();
    x.store([&](int j, auto value) { out[static_cast<unsigned>((sub * R + j) * N2 + c)] = value(); });
  }
}

// Forward pass A (radix R = L1) over rows a * L1 + j, read straight from the
// plane in global memory, times the conjugated pass-A twiddles.
template <typename T, int R>
__device__ __forceinline__ void ypass_fwdA_R(const cplx_t<T>* __restrict__ in, int N2, int nz, int L2, int ld, int W,
                                             int lim) {
  cplx_t<T>* sm = smem_c<T>();
  const int nitems = nz * L2;
  const FastDiv div(nz);
  for (int it = threadIdx.x; it < nitems; it += blockDim.x) {
    const int a = div.quot(it);
    const int c = it - a * nz;
    T re[R], im[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const cplx_t<T> v = in[static_cast<unsigned>((a * R + j) * N2 + c)];
      re[j] = v.x;
      im[j] = v.y;
    }
    Block<T, R> x;
    x.load(re, im);
    x.template run<-1>();
#pragma unroll
    for (int j = 1; j < R; ++j) x.template twiddle<-1>(j, sm[W + a + j * L2]);
    x.store([&](int j, auto value) {
      const int off = (a * R + j) * ld + c;
      if (QGB_OK_IDX(off, lim, 66)) sm[off] = value();
    });
  }
}

// Forward pass B (radix R = L2) over rows sub + j * L1 (natural order out);
// only the rows the slab's sphere points touch are stored.
template <typename T, int R>
__device__ __forceinline__ void ypass_fwdB_R(const int* rowmask, int nz, int L1, int ld, int lim) {
  cplx_t<T>* sm = smem_c<T>();
  const int nitems = nz * L1;
  const FastDiv div(nz);
  for (int it = threadIdx.x; it < nitems; it += blockDim.x) {
    const int sub = div.quot(it);
    const int c = it - sub * nz;
    T re[R], im[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int off = (sub + j * L1) * ld + c;
      if (!QGB_OK_IDX(off, lim, 67)) return;
      const cplx_t<T> v = sm[off];
      re[j] = v.x;
      im[j] = v.y;
    }
    Block<T, R> x;
    x.load(re, im);
    x.template run<-1>();
    x.store([&](int j, auto value) {
      if (rowmask[sub + j * L1]) sm[(sub + j * L1) * ld + c] = value();
    });
  }
}

// kind 0: inverse pass 1; 1: inverse pass 2 (to global); 2: forward pass A
// (from global); 3: forward pass B.  R is the pass's radix.
template <typename T, int KIND>
__device__ __forceinline__ void ypass(int R, const int* rowmask, cplx_t<T>* g, int N2, int nz, int L1, int L2,
                                      int ld, int W, int lim) {
#define QGB_YP(RR)                                                                  \
  case RR:                                                                          \
    if constexpr (KIND == 0) ypass_inv1_R<T, RR>(rowmask, nz, L1, ld, W, lim);      \
    if constexpr (KIND == 1) ypass_inv2_R<T, RR>(g, N2, nz, L2, ld, lim);           \
    if constexpr (KIND == 2) ypass_fwdA_R<T, RR>(g, N2, nz, L2, ld, W, lim);        \
    if constexpr (KIND == 3) ypass_fwdB_R<T, RR>(rowmask, nz, L1, ld, lim);         \
    break;
  switch (R) {
    QGB_YP(2) QGB_YP(3) QGB_YP(4) QGB_YP(5) QGB_YP(6) QGB_YP(7) QGB_YP(8) QGB_YP(9) QGB_YP(10) QGB_YP(12)
    QGB_YP(14) QGB_YP(15) QGB_YP(16)
    default: break;
  }
#undef QGB_YP
}

template <typename T>
__device__ __forceinline__ void body_ifft_yz(const qgb_sphere& s, const LocalParams& lp,
                                             const cplx_t<T>* __restrict__ C, cplx_t<T>* __restrict__ planes,
                                             const int slab, const int b, const int k) {
  using C2 = cplx_t<T>;
  if (slab >= s.n_slabs[k]) return;
  const int N1 = s.N[1], N2 = s.N[2], ld = N2 + 1;
  const int L1y = s.L1[1], L2y = s.L2[1];
  const bool fold = L1y > 1 && L2y > 1;  // y passes with the plane's boundaries folded in
  // Shared layout: plane [N1][ld], W_y [N1], W_z [N2], row mask [N1] int.
  const int lim = N1 * ld, Wy = lim, Wz = Wy + N1;
  C2* sm = smem_c<T>();
  int* rowmask = reinterpret_cast<int*>(sm + Wz + N2);
  const C2* tw = static_cast<const C2*>(s.twiddle);
  load_twiddles<T>(Wy, tw + s.tw_off[1], N1);
  load_twiddles<T>(Wz, tw + s.tw_off[2], N2);
  const C2 zero = mk<T>(T(0), T(0));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int r0 = s.row_start[k * (s.max_slabs + 1) + slab];
  const int nrows = s.row_start[k * (s.max_slabs + 1) + slab + 1] - r0;
  const int* rows = s.rows + r0;
  if (fold) {
    // Only the touched rows are zero-filled: the first y pass reads the others as zero.
    for (int y = threadIdx.x; y < N1; y += blockDim.x) rowmask[y] = 0;
    for (int i = warp; i < nrows; i += nwarps) {
      const int y = rows[i];
      if (!QGB_OK_IDX(y, N1, 68)) continue;
      for (int c = lane; c < N2; c += 32) sm[y * ld + c] = zero;
    }
  } else {
    for (int r = warp; r < N1; r += nwarps)
      for (int c = lane; c < N2; c += 32) sm[r * ld + c] = zero;
  }
  __syncthreads();
  if (fold) {
    for (int i = threadIdx.x; i < nrows; i += blockDim.x) {
      const int y = rows[i];
      if (QGB_OK_IDX(y, N1, 68)) rowmask[y] = 1;
    }
  }

  // Scatter this slab's coefficients (contiguous in the basis) into the plane.
  const int g0 = s.slab_start[k * (s.max_slabs + 1) + slab];
  const int g1 = s.slab_start[k * (s.max_slabs + 1) + slab + 1];
  const C2* Cb = C + (static_cast<size_t>(k) * lp.nb_total + lp.b0 + b) * s.n_tot;
  const int* yz = s.yz + static_cast<size_t>(k) * s.n_tot;
  for (int gb = g0 + threadIdx.x; gb < g1; gb += kPoints * blockDim.x) {
    int v[kPoints];
#pragma unroll
    for (int u = 0; u < kPoints; ++u) {
      const int g = gb + u * blockDim.x;
      v[u] = g < g1 && QGB_OK_IDX(g, s.n[k], 1) ? yz[g] : 0;
    }
#pragma unroll
    for (int u = 0; u < kPoints; ++u) {
      const int g = gb + u * blockDim.x;
      if (g >= g1 || !QGB_OK_IDX(g, s.n[k], 1)) continue;
      const int pos = (v[u] >> 16) * ld + (v[u] & 0xFFFF);
      if (!QGB_OK_IDX(pos, lim, 2) || !QGB_OK_IDX(v[u] & 0xFFFF, N2, 3)) continue;
      cp_async_elem<T>(sm + pos, Cb + g);
    }
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();

  // Inverse z-FFT along the rows this slab touches (row stride ld, element
  // stride 1) and, where the y passes are not folded, the inverse y-FFT along
  // all N2 columns (column stride 1, element stride ld).
  if constexpr (sizeof(T) == 8) {  // one copy of the code
#pragma unroll 1
    for (int ax = 2; ax >= (fold ? 2 : 1); --ax)
      fft_axis<T, +1>(0, ax == 2 ? rows : nullptr, ax == 2 ? nrows : N2, ax == 2 ? ld : 1, ax == 2 ? 1 : ld, s.L1[ax],
                      s.L2[ax], ax == 2 ? Wz : Wy, lim);
  } else {
    fft_axis<T, +1>(0, rows, nrows, ld, 1, s.L1[2], s.L2[2], Wz, lim);
    if (!fold) fft_axis<T, +1>(0, nullptr, N2, 1, ld, L1y, L2y, Wy, lim);
  }
  if (!QGB_OK_IDX(plane_index(s, k, b, lp.nb, slab), (long long)s.nk * lp.nb * s.max_slabs, 4)) return;
  C2* out = planes + plane_index(s, k, b, lp.nb, slab) * (static_cast<size_t>(N1) * N2);
  if (fold) {
    // Inverse y-FFT along all N2 columns; its second pass stores the plane.
    ypass<T, 0>(L2y, rowmask, nullptr, N2, N2, L1y, L2y, ld, Wy, lim);
    __syncthreads();
    ypass<T, 1>(L1y, rowmask, out, N2, N2, L1y, L2y, ld, Wy, lim);
    return;
  }
  for (int r = warp; r < N1; r += nwarps)
    for (int c = lane; c < N2; c += 32) out[r * N2 + c] = sm[r * ld + c];
}

// The x-pass middle step on one item: inverse L1-point DFT, multiply by V,
// forward L1-point DFT, forward-pass twiddles; data at sm[p + j*ld], V at
// Vp[j * vstride] (global or shared), twiddles at sm[Wx + j*L2 + a].
template <typename T, int R, typename VPtr>
__device__ __forceinline__ void xmid_item(cplx_t<T>* sm, int p, int ld, VPtr Vp, unsigned vstride, int Wx, int L2,
                                          int a) {
  using C2 = cplx_t<T>;
  T re[R], im[R];
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const C2 v = sm[p + j * ld];
    re[j] = v.x;
    im[j] = v.y;
  }
  T v[R];
#pragma unroll
  for (int j = 0; j < R; ++j) v[j] = Vp[j * vstride];
  XBlock<T, R> x;
  x.load(re, im);
  x.template run<+1>();
  x.scale(v);
  x.template run<-1>();
  if (L2 > 1) {
#pragma unroll
    for (int j = 1; j < R; ++j) x.template twiddle<-1>(j, sm[Wx + j * L2 + a]);
  }
  x.store([&](int j, auto value) { sm[p + j * ld] = value(); });
}

template <typename T, typename VPtr>
__device__ __forceinline__ void xmid_dispatch(int L1, cplx_t<T>* sm, int p, int ld, VPtr Vp, unsigned vstride, int Wx,
                                              int L2, int a) {
  switch (L1) {
    case 1: xmid_item<T, 1>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 2: xmid_item<T, 2>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 3: xmid_item<T, 3>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 4: xmid_item<T, 4>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 5: xmid_item<T, 5>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 6: xmid_item<T, 6>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 7: xmid_item<T, 7>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 8: xmid_item<T, 8>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 9: xmid_item<T, 9>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 10: xmid_item<T, 10>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 12: xmid_item<T, 12>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 14: xmid_item<T, 14>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 15: xmid_item<T, 15>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    case 16: xmid_item<T, 16>(sm, p, ld, Vp, vstride, Wx, L2, a); break;
    default: break;
  }
}

// The x-pass's items (column c < nz, sub < nsub).  W32: tiles of 32 columns, a
// warp takes the 32 columns of a sub, so that twiddles, slab offsets and strides
// are uniform over the warp; its lanes c >= nz (the last tile) work on columns
// of their own that are never loaded or stored.  Otherwise columns and subs are
// flattened over the CTA's threads.
template <bool W32, typename F>
__device__ __forceinline__ void x_items(int nz, int nsub, F f) {
  if constexpr (W32) {
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    for (int sub = warp; sub < nsub; sub += blockDim.x >> 5) f(sub, static_cast<int>(threadIdx.x & 31));
  } else {
    const FastDiv div(nz);
    for (int it = threadIdx.x; it < nz * nsub; it += blockDim.x) {
      const int sub = div.quot(it);
      f(sub, it - sub * nz);
    }
  }
}

// x-pass first inverse pass straight from the slab planes: item (column c,
// sub) is the L2-point DFT over x = sub + j * L1 (natural order), read from the
// planes at offset xs[x] (zero where no slab), times the pass-1 twiddles, stored
// at the same shared rows.  Covers every row, so no zero fill is needed.
template <typename T, int R, bool W32>
__device__ __forceinline__ void xpass_first_R(const cplx_t<T>* __restrict__ base, const int* xs, int nz, int L1,
                                              int ld, int Wx, int lim) {
  cplx_t<T>* sm = smem_c<T>();
  x_items<W32>(nz, L1, [&](int sub, int c) {
    const bool in = !W32 || c < nz;
    T re[R], im[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int o = xs[sub + j * L1];
      cplx_t<T> v = mk<T>(T(0), T(0));
      if (o >= 0 && in) v = base[static_cast<unsigned>(o + c)];
      re[j] = v.x;
      im[j] = v.y;
    }
    XBlock<T, R> x;
    x.load(re, im);
    x.template run<+1>();
#pragma unroll
    for (int j = 1; j < R; ++j) x.template twiddle<+1>(j, sm[Wx + sub * R + j]);
    x.store([&](int j, auto value) {
      const int off = (sub + j * L1) * ld + c;
      if (QGB_OK_IDX(off, lim, 61)) sm[off] = value();
    });
  });
}

// x-pass last forward pass straight to the slab planes: the L2-point DFT over
// the shared rows sub + j * L1 gives natural x = sub + j * L1; only the rows of
// a slab (xs[x] >= 0) are stored.
template <typename T, int R, bool W32>
__device__ __forceinline__ void xpass_last_R(cplx_t<T>* __restrict__ base, const int* xs, int nz, int L1, int ld,
                                             int lim) {
  cplx_t<T>* sm = smem_c<T>();
  x_items<W32>(nz, L1, [&](int sub, int c) {
    const bool in = !W32 || c < nz;
    T re[R], im[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int off = (sub + j * L1) * ld + c;
      if (!QGB_OK_IDX(off, lim, 62)) return;
      const cplx_t<T> v = sm[off];
      re[j] = v.x;
      im[j] = v.y;
    }
    XBlock<T, R> x;
    x.load(re, im);
    x.template run<-1>();
    x.store([&](int j, auto value) {
      const int o = xs[sub + j * L1];
      if (o >= 0 && in) base[static_cast<unsigned>(o + c)] = value();
    });
  });
}

template <typename T, bool FIRST, bool W32>
__device__ __forceinline__ void xpass_outer(int R, cplx_t<T>* base, const int* xs, int nz, int L1, int ld, int Wx,
                                            int lim) {
#define QGB_XO(RR)                                                    \
  case RR:                                                            \
    if constexpr (FIRST)                                              \
      xpass_first_R<T, RR, W32>(base, xs, nz, L1, ld, Wx, lim);       \
    else                                                              \
      xpass_last_R<T, RR, W32>(base, xs, nz, L1, ld, lim);            \
    break;
  switch (R) {
    QGB_XO(2) QGB_XO(3) QGB_XO(4) QGB_XO(5) QGB_XO(6) QGB_XO(7) QGB_XO(8) QGB_XO(9) QGB_XO(10) QGB_XO(12)
    QGB_XO(14) QGB_XO(15) QGB_XO(16)
    default: break;
  }
#undef QGB_XO
}

// The x-pass's tables behind `lim` elements of data: W_x [N0] complex, x -> plane
// offset [N0] int (-1: no slab).  Ends with __syncthreads().
template <typename T>
__device__ __forceinline__ void x_tables(const qgb_sphere& s, const int k, const int lim) {
  const int N0 = s.N[0];
  int* xs = reinterpret_cast<int*>(smem_c<T>() + lim + N0);
  load_twiddles<T>(lim, static_cast<const cplx_t<T>*>(s.twiddle) + s.tw_off[0], N0);
  for (int x = threadIdx.x; x < N0; x += blockDim.x) xs[x] = -1;
  __syncthreads();
  const int* i0 = s.slab_i0 + k * s.max_slabs;
  for (int sl = threadIdx.x; sl < s.n_slabs[k]; sl += blockDim.x) {
    const int x = i0[sl];
    if (QGB_OK_IDX(x, N0, 63) && QGB_OK_IDX(sl, s.max_slabs, 6)) xs[x] = sl * s.N[1] * s.N[2];
  }
  __syncthreads();
}

// x-pass of the columns [c0, c0 + nz) of the N1 N2 (y, z) positions of a plane,
// with its outer passes on the slab planes: the first inverse pass reads the
// slab rows from global memory (L2) and the last forward pass stores the slab
// rows back, so shared memory sees each element in three passes only (no zero
// fill, staging or write-back).  The middle step reads V(r) from global memory
// (it stays in L2 across the bands).  An axis of a single codelet (L2 = 1) has
// the middle step alone and is staged.  Shared layout: pencils [N0][ld] complex
// (ld = 32 for W32, else nz; threads run along the columns, so rows need no
// padding), then x_tables.
template <typename T, bool W32>
__device__ __forceinline__ void body_xpass(const qgb_sphere& s, const LocalParams& lp, cplx_t<T>* __restrict__ planes,
                                           const int b, const int k, const int c0, const int nz) {
  using C2 = cplx_t<T>;
  const int N0 = s.N[0], N1 = s.N[1], N2 = s.N[2], ld = W32 ? 32 : nz;
  const int L1 = s.L1[0], L2 = s.L2[0];
  const int lim = N0 * ld, Wx = lim;
  C2* sm = smem_c<T>();
  int* xs = reinterpret_cast<int*>(sm + Wx + N0);
  const size_t plane = static_cast<size_t>(N1) * N2;
  if (!QGB_OK_IDX(plane_index(s, k, b, lp.nb, 0), (long long)s.nk * lp.nb * s.max_slabs, 5)) return;
  C2* base = planes + plane_index(s, k, b, lp.nb, 0) * plane + c0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  if (L2 > 1) {
    xpass_outer<T, true, W32>(L2, base, xs, nz, L1, ld, Wx, lim);
  } else {
    for (int x = warp; x < N0; x += nwarps) {
      const int o = xs[x];
      for (int c = lane; c < ld; c += 32) sm[x * ld + c] = o >= 0 && c < nz ? base[o + c] : mk<T>(T(0), T(0));
    }
  }
  __syncthreads();
  // V[p0][c0 + c] with p0 = a * L1 + j: j-stride N1 * N2.
  const T* V = static_cast<const T*>(s.V) + c0;
  x_items<W32>(nz, L2, [&](int a, int c) {
    if (!QGB_OK_IDX(c + (a * L1 + L1 - 1) * ld, lim, 7) || !QGB_OK_IDX((L1 - 1) * L2 + a, N0, 9) ||
        !QGB_OK_IDX(static_cast<long long>(a * L1 + L1 - 1) * plane + c0 + (W32 ? min(c, nz - 1) : c), N0 * plane, 8))
      return;
    xmid_dispatch<T>(L1, sm, c + a * L1 * ld, ld, V + static_cast<unsigned>(a * L1 * N1 * N2 + (W32 ? min(c, nz - 1) : c)),
                     N1 * N2, Wx, L2, a);
  });
  __syncthreads();
  if (L2 > 1) {
    xpass_outer<T, false, W32>(L2, base, xs, nz, L1, ld, Wx, lim);
  } else {
    for (int x = warp; x < N0; x += nwarps) {
      const int o = xs[x];
      if (o >= 0)
        for (int c = lane; c < nz; c += 32) base[o + c] = sm[x * ld + c];
    }
  }
}

// ---------------------------------------------------------------------------
// The FP32 x-pass on tiles of 64 columns: a lane takes columns c and c + 32 as a
// packed pair (packed_f32.cuh).  Otherwise as body_xpass<T, true>: the same
// passes, rows and items, with shared elements of 16 B and the twiddles doubled.
// One column a lane was bound by instruction issue (2.5 of 4 a clock): pairs
// issue 25.0 M instead of 35.8 M for 40 bands of 72^3.  What they need in return
// is that a thread's loads are all in flight before the first is used (loads and
// packing in one loop: 465 us instead of 360 at si64) and five CTAs' worth of
// warps at 96 registers (x_max_threads).  x-pass, us: 72^3, 800 bands 862 -> 751,
// 96^3, 160 bands 377 -> 367, 36^3, 144 bands 21.7 -> 20.3.
// ---------------------------------------------------------------------------

__device__ __forceinline__ cpair_t* smem_pairs() { return reinterpret_cast<cpair_t*>(qgb_smem); }

// The columns of a lane that the tile has (the last tile of a plane is ragged).
struct PairLane {
  int c;
  bool in0, in1;
};

__device__ __forceinline__ cpair_t pair_load(const float2* __restrict__ row, const PairLane l) {
  float2 a = make_float2(0.0f, 0.0f), b = a;
  if (l.in0) a = row[l.c];
  if (l.in1) b = row[l.c + 32];
  return make_ulonglong2(pair_of(a.x, b.x), pair_of(a.y, b.y));
}
__device__ __forceinline__ void pair_store(float2* __restrict__ row, const PairLane l, pair_t re, pair_t im) {
  const float2 x = pair_split(re), y = pair_split(im);
  if (l.in0) row[l.c] = make_float2(x.x, y.x);
  if (l.in1) row[l.c + 32] = make_float2(x.y, y.y);
}

template <int R>
__device__ __forceinline__ void xpair_first_R(const float2* __restrict__ base, const int* xs, const PairLane l, int L1,
                                              int Wx, int lim) {
  cpair_t* sm = smem_pairs();
  x_items<true>(0, L1, [&](int sub, int c) {
    PairBlock<R> x;
    float2 p[R], q[R];  // all loads in flight before the first is used
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int o = xs[sub + j * L1];
      p[j] = q[j] = make_float2(0.0f, 0.0f);
      if (o >= 0 && l.in0) p[j] = base[static_cast<unsigned>(o + c)];
      if (o >= 0 && l.in1) q[j] = base[static_cast<unsigned>(o + c + 32)];
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
      x.re[j] = F2::of(pair_of(p[j].x, q[j].x));
      x.im[j] = F2::of(pair_of(p[j].y, q[j].y));
    }
    x.template run<+1>();
#pragma unroll
    for (int j = 1; j < R; ++j) {
      const cpair_t w = sm[Wx + sub * R + j];
      x.template twiddle<+1>(j, w.x, w.y);
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int off = (sub + j * L1) * 32 + c;
      if (QGB_OK_IDX(off, lim, 61)) sm[off] = make_ulonglong2(x.re[j].value(), x.im[j].value());
    }
  });
}

template <int R>
__device__ __forceinline__ void xpair_last_R(float2* __restrict__ base, const int* xs, const PairLane l, int L1,
                                             int lim) {
  const cpair_t* sm = smem_pairs();
  x_items<true>(0, L1, [&](int sub, int c) {
    PairBlock<R> x;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int off = (sub + j * L1) * 32 + c;
      if (!QGB_OK_IDX(off, lim, 62)) return;
      const cpair_t v = sm[off];
      x.re[j] = F2::of(v.x);
      x.im[j] = F2::of(v.y);
    }
    x.template run<-1>();
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int o = xs[sub + j * L1];
      if (o >= 0) pair_store(base + static_cast<unsigned>(o), l, x.re[j].value(), x.im[j].value());
    }
  });
}

template <int R>
__device__ __forceinline__ void xpair_mid_R(const float* __restrict__ V, const PairLane l, unsigned plane, int v_lim,
                                            int L2, int Wx, int lim) {
  cpair_t* sm = smem_pairs();
  const int v0 = l.in0 ? l.c : 0, v1 = l.in1 ? l.c + 32 : v0;  // lanes beyond the tile read V of its first columns
  x_items<true>(0, L2, [&](int a, int c) {
    if (!QGB_OK_IDX(c + (a * R + R - 1) * 32, lim, 7) || !QGB_OK_IDX((a * R + R - 1) * plane + max(v0, v1), v_lim, 8))
      return;
    cpair_t* p = sm + a * R * 32 + c;
    const float* Va = V + static_cast<unsigned>(a * R) * plane;
    PairBlock<R> x;
    pair_t v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const cpair_t e = p[j * 32];
      x.re[j] = F2::of(e.x);
      x.im[j] = F2::of(e.y);
    }
    float f0[R], f1[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      f0[j] = Va[j * plane + v0];
      f1[j] = Va[j * plane + v1];
    }
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = pair_of(f0[j], f1[j]);
    x.template run<+1>();
#pragma unroll
    for (int j = 0; j < R; ++j) x.scale(j, v[j]);
    x.template run<-1>();
    if (L2 > 1) {
#pragma unroll
      for (int j = 1; j < R; ++j) {
        const cpair_t w = sm[Wx + j * L2 + a];
        x.template twiddle<-1>(j, w.x, w.y);
      }
    }
#pragma unroll
    for (int j = 0; j < R; ++j) p[j * 32] = make_ulonglong2(x.re[j].value(), x.im[j].value());
  });
}

// STEP 0: first inverse pass (radix L2), 1: middle step (L1), 2: last forward (L2).
template <int STEP>
__device__ __forceinline__ void xpair_step(int R, float2* base, const float* V, const int* xs, const PairLane l,
                                           unsigned plane, int v_lim, int L1, int L2, int Wx, int lim) {
#define QGB_XP(RR)                                             \
  case RR:                                                     \
    if constexpr (STEP == 0)                                   \
      xpair_first_R<RR>(base, xs, l, L1, Wx, lim);             \
    else if constexpr (STEP == 1)                              \
      xpair_mid_R<RR>(V, l, plane, v_lim, L2, Wx, lim);        \
    else                                                       \
      xpair_last_R<RR>(base, xs, l, L1, lim);                  \
    break;
  switch (R) {
    QGB_XP(2) QGB_XP(3) QGB_XP(4) QGB_XP(5) QGB_XP(6) QGB_XP(7) QGB_XP(8) QGB_XP(9) QGB_XP(10) QGB_XP(12)
    QGB_XP(14) QGB_XP(15) QGB_XP(16)
    default:  // radix 1: the middle step of an axis with L1 = 1
      if constexpr (STEP == 1) xpair_mid_R<1>(V, l, plane, v_lim, L2, Wx, lim);
      break;
  }
#undef QGB_XP
}

// As x_tables, behind 32 N0 pairs.
__device__ __forceinline__ void x_tables_pair(const qgb_sphere& s, const int k) {
  const int N0 = s.N[0];
  cpair_t* W = smem_pairs() + 32 * N0;
  int* xs = reinterpret_cast<int*>(W + N0);
  const float2* tw = static_cast<const float2*>(s.twiddle) + s.tw_off[0];
  for (int i = threadIdx.x; i < N0; i += blockDim.x) {
    const float2 w = tw[i];
    W[i] = make_ulonglong2(lane_const<pair_t>(w.x), lane_const<pair_t>(w.y));
    xs[i] = -1;
  }
  __syncthreads();
  const int* i0 = s.slab_i0 + k * s.max_slabs;
  for (int sl = threadIdx.x; sl < s.n_slabs[k]; sl += blockDim.x) {
    const int x = i0[sl];
    if (QGB_OK_IDX(x, N0, 63) && QGB_OK_IDX(sl, s.max_slabs, 6)) xs[x] = sl * s.N[1] * s.N[2];
  }
  __syncthreads();
}

__device__ __forceinline__ void body_xpass_pair(const qgb_sphere& s, const LocalParams& lp, float2* __restrict__ planes,
                                                const int b, const int k, const int c0, const int nz) {
  const int N0 = s.N[0], L1 = s.L1[0], L2 = s.L2[0];
  const int lim = 32 * N0;
  cpair_t* sm = smem_pairs();
  const int* xs = reinterpret_cast<const int*>(sm + lim + N0);
  const size_t plane = static_cast<size_t>(s.N[1]) * s.N[2];
  if (!QGB_OK_IDX(plane_index(s, k, b, lp.nb, 0), (long long)s.nk * lp.nb * s.max_slabs, 5)) return;
  float2* base = planes + plane_index(s, k, b, lp.nb, 0) * plane + c0;
  const float* V = static_cast<const float*>(s.V) + c0;
  const int v_lim = N0 * static_cast<int>(plane) - c0;  // V's elements from c0 on (range checks)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const PairLane l{lane, lane < nz, lane + 32 < nz};
  if (L2 > 1) {
    xpair_step<0>(L2, base, V, xs, l, plane, v_lim, L1, L2, lim, lim);
  } else {
    for (int x = warp; x < N0; x += nwarps) {
      const int o = xs[x];
      sm[x * 32 + lane] = o >= 0 ? pair_load(base + static_cast<unsigned>(o), l) : make_ulonglong2(0, 0);
    }
  }
  __syncthreads();
  xpair_step<1>(L1, base, V, xs, l, plane, v_lim, L1, L2, lim, lim);
  __syncthreads();
  if (L2 > 1) {
    xpair_step<2>(L2, base, V, xs, l, plane, v_lim, L1, L2, lim, lim);
  } else {
    for (int x = warp; x < N0; x += nwarps) {
      const int o = xs[x];
      const cpair_t v = sm[x * 32 + lane];
      if (o >= 0) pair_store(base + static_cast<unsigned>(o), l, v.x, v.y);
    }
  }
}

template <typename T>
__device__ __forceinline__ void body_fft_yz_gather(const qgb_sphere& s, const LocalParams& lp, const cplx_t<T>* C,
                                                   cplx_t<T>* out, const cplx_t<T>* __restrict__ planes,
                                                   const int slab, const int b, const int k) {
  using C2 = cplx_t<T>;
  const int nslabs = s.n_slabs[k];
  C2* Ob = out + (static_cast<size_t>(k) * lp.nb_total + lp.b0 + b) * s.n_tot;
  const bool accumulate = (lp.flags & QGB_ACCUMULATE) != 0;
  if (slab == 0 && !accumulate) {  // zero the padding entries of this band
    const int nk_in = s.n[k];
    for (int g = nk_in + threadIdx.x; g < s.n_tot; g += blockDim.x) Ob[g] = mk<T>(T(0), T(0));
  }
  if (slab >= nslabs) return;
  const int N0 = s.N[0], N1 = s.N[1], N2 = s.N[2], ld = N2 + 1;
  const int lim = N1 * ld, Wy = lim, Wz = Wy + N1;
  C2* sm = smem_c<T>();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  if (!QGB_OK_IDX(plane_index(s, k, b, lp.nb, slab), (long long)s.nk * lp.nb * s.max_slabs, 4)) return;
  const C2* in = planes + plane_index(s, k, b, lp.nb, slab) * (static_cast<size_t>(N1) * N2);
  const int L1y = s.L1[1], L2y = s.L2[1];
  const int r0 = s.row_start[k * (s.max_slabs + 1) + slab];
  const int nrows = s.row_start[k * (s.max_slabs + 1) + slab + 1] - r0;
  const C2* tw = static_cast<const C2*>(s.twiddle);
  const bool fold = L1y > 1 && L2y > 1;
  if (fold) {
    // The first forward y pass reads the plane from global memory; the second
    // stores only the rows the z-FFT and the gather use.
    int* rowmask = reinterpret_cast<int*>(sm + Wz + N2);
    for (int y = threadIdx.x; y < N1; y += blockDim.x) rowmask[y] = 0;
    load_twiddles<T>(Wy, tw + s.tw_off[1], N1);
    load_twiddles<T>(Wz, tw + s.tw_off[2], N2);
    __syncthreads();
    for (int i = threadIdx.x; i < nrows; i += blockDim.x) {
      const int y = s.rows[r0 + i];
      if (QGB_OK_IDX(y, N1, 68)) rowmask[y] = 1;
    }
    ypass<T, 2>(L1y, rowmask, const_cast<C2*>(in), N2, N2, L1y, L2y, ld, Wy, lim);
    __syncthreads();
    ypass<T, 3>(L2y, rowmask, nullptr, N2, N2, L1y, L2y, ld, Wy, lim);
    __syncthreads();
  } else {
    // Stage the plane asynchronously (padded rows are 8-byte aligned only, so one
    // element per copy), then the twiddles while the copies are in flight.
    for (int r = warp; r < N1; r += nwarps)
      for (int c = lane; c < N2; c += 32) cp_async_elem<T>(sm + r * ld + c, in + r * N2 + c);
    cp_async_commit();
    load_twiddles<T>(Wy, tw + s.tw_off[1], N1);
    load_twiddles<T>(Wz, tw + s.tw_off[2], N2);
    cp_async_wait<0>();
    __syncthreads();
  }
  // Forward y-FFT along all columns (unless folded above), then the forward
  // z-FFT along the touched rows.
  if constexpr (sizeof(T) == 8) {
#pragma unroll 1
    for (int ax = fold ? 2 : 1; ax <= 2; ++ax)
      fft_axis<T, -1>(0, ax == 2 ? s.rows + r0 : nullptr, ax == 2 ? nrows : N2, ax == 2 ? ld : 1, ax == 2 ? 1 : ld,
                      s.L1[ax], s.L2[ax], ax == 2 ? Wz : Wy, lim);
  } else {
    if (!fold) fft_axis<T, -1>(0, nullptr, N2, 1, ld, L1y, L2y, Wy, lim);
    fft_axis<T, -1>(0, s.rows + r0, nrows, ld, 1, s.L1[2], s.L2[2], Wz, lim);
  }

  const int g0 = s.slab_start[k * (s.max_slabs + 1) + slab];
  const int g1 = s.slab_start[k * (s.max_slabs + 1) + slab + 1];
  const C2* Cb = C + (static_cast<size_t>(k) * lp.nb_total + lp.b0 + b) * s.n_tot;
  const int* yz = s.yz + static_cast<size_t>(k) * s.n_tot;
  const T invN = T(1) / (T(N0) * T(N1) * T(N2));
  const bool add_ke = (lp.flags & QGB_ADD_KE) != 0;
  const T* ke = static_cast<const T*>(s.ke) + static_cast<size_t>(k) * s.n_tot;
  for (int gb = g0 + threadIdx.x; gb < g1; gb += kPoints * blockDim.x) {
    int v[kPoints];
    C2 c[kPoints], o[kPoints];
    T e[kPoints];
#pragma unroll
    for (int u = 0; u < kPoints; ++u) {
      const int g = gb + u * blockDim.x;
      const bool in = g < g1 && QGB_OK_IDX(g, s.n[k], 1);
      v[u] = in ? yz[g] : 0;
      c[u] = o[u] = mk<T>(T(0), T(0));
      e[u] = T(0);
      if (in && add_ke) {
        c[u] = Cb[g];
        e[u] = ke[g];
      }
      if (in && accumulate) o[u] = Ob[g];
    }
#pragma unroll
    for (int u = 0; u < kPoints; ++u) {
      const int g = gb + u * blockDim.x;
      if (g >= g1 || !QGB_OK_IDX(g, s.n[k], 1)) continue;
      const int pos = (v[u] >> 16) * ld + (v[u] & 0xFFFF);
      if (!QGB_OK_IDX(pos, lim, 2)) continue;
      const C2 f = sm[pos];
      T xr = f.x * invN, xi = f.y * invN;
      if (add_ke) {
        xr = fma(e[u], c[u].x, xr);  // (KE, the larger term at high G, unrounded)
        xi = fma(e[u], c[u].y, xi);
      }
      if (accumulate) {
        xr += o[u].x;
        xi += o[u].y;
      }
      Ob[g] = mk<T>(xr, xi);
    }
  }
}

// ---------------------------------------------------------------------------
// Kernels: one sphere (grid = work units of that sphere) ...
// ---------------------------------------------------------------------------

// The y/z kernels take 80 registers in FP32 (768 threads an SM), 128 in FP64 (block
// fixed point, 512 threads); the CTA sizes follow the grid, see launch_cost.
template <typename T> constexpr int kMaxThreadsYZ = sizeof(T) == 4 ? 384 : 512;

template <typename T>
__global__ void __launch_bounds__(kMaxThreadsYZ<T>, sizeof(T) == 4 ? 2 : 1) k_ifft_yz(const qgb_sphere s, LocalParams lp,
                                                              const cplx_t<T>* __restrict__ C,
                                                              cplx_t<T>* __restrict__ planes) {
  body_ifft_yz<T>(s, lp, C, planes, blockIdx.x, blockIdx.y, blockIdx.z);
}

// `tiles` tiles (x_cols<T> columns: 64 in FP32, 32 in FP64) per CTA, one after the
// other (one in FP64, whose body a loop costs 4%).
template <typename T> constexpr int x_cols = sizeof(T) == 4 ? 64 : 32;

template <typename T, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT > 160 ? 2 : 4) k_xpass(const qgb_sphere s, LocalParams lp,
                                                                   cplx_t<T>* __restrict__ planes, int tiles) {
  const int cols = s.N[1] * s.N[2];
  if constexpr (sizeof(T) == 4) {
    x_tables_pair(s, blockIdx.z);
    int c0 = blockIdx.x * tiles * 64;
    for (int t = 0; t < tiles && c0 < cols; ++t, c0 += 64) {
      if (t > 0) __syncthreads();  // the tile's shared memory is reused
      body_xpass_pair(s, lp, planes, blockIdx.y, blockIdx.z, c0, min(64, cols - c0));
    }
  } else {
    const int c0 = blockIdx.x * 32;
    x_tables<T>(s, blockIdx.z, 32 * s.N[0]);
    body_xpass<T, true>(s, lp, planes, blockIdx.y, blockIdx.z, c0, min(32, cols - c0));
  }
}

// C and out may alias (in-place apply): no __restrict__ on them.
template <typename T>
__global__ void __launch_bounds__(kMaxThreadsYZ<T>, sizeof(T) == 4 ? 2 : 1) k_fft_yz_gather(const qgb_sphere s, LocalParams lp,
                                                                    const cplx_t<T>* C, cplx_t<T>* out,
                                                                    const cplx_t<T>* __restrict__ planes) {
  body_fft_yz_gather<T>(s, lp, C, out, planes, blockIdx.x, blockIdx.y, blockIdx.z);
}

// ---------------------------------------------------------------------------
// Launches of one precision (instantiated in local_f32.cu and local_f64.cu)
// ---------------------------------------------------------------------------

inline size_t yz_smem_bytes(const qgb_sphere& s, size_t e) {
  return (static_cast<size_t>(s.N[1]) * (s.N[2] + 1) + s.N[1] + s.N[2]) * e + s.N[1] * sizeof(int);
}
inline size_t x_smem_bytes(const qgb_sphere& s, int nz, size_t e) {
  return (static_cast<size_t>(s.N[0]) * nz + s.N[0]) * e + s.N[0] * sizeof(int);
}

constexpr size_t kSmemPerSm = 227 * 1024;

// Relative cost of a launch: `ctas_total` CTAs of t threads and `smem` bytes,
// each doing `work` thread-rounds (a round counts its codelet's elements), where
// an SM's registers hold `resident` threads.  Wide CTAs wait longer at their
// barriers; a launch of few CTAs takes whole waves.
inline double launch_cost(int resident, double ctas_total, int t, size_t smem, double work) {
  const int ctas = std::max(1, static_cast<int>(std::min<size_t>(resident / t, (kSmemPerSm + 1024) / (smem + 1024))));
  double waves = std::max(1.0, ctas_total / (152.0 * ctas));
  if (waves < 8.0) waves = std::ceil(waves);
  const double on_sm = std::min<double>(ctas, std::ceil(ctas_total / 152.0)) * t;
  return waves * work * (1.0 + 0.0006 * t) * std::max(0.5, std::sqrt(on_sm / resident));
}

// CTA size of the y/z kernels: the one whose passes (y: N2 L1 items of radix L2
// and N2 L2 of L1; z: the touched rows, on average 0.8 of the most) fill their
// rounds.  Measured against 256 threads (FP32; 36^3 in FP64 against 224), us: 36^3,
// 144 bands, 43 -> 28 (FP64 144 -> 110); 72^3, 800 bands, inverse 513 -> 450.
template <typename T> int threads_yz(const qgb_sphere& s, int nb) {
  const size_t smem = yz_smem_bytes(s, sizeof(cplx_t<T>));
  const int zrows = std::max(1, s.max_rows * 4 / 5);
  double best = 1e30;
  int threads = 128;
  for (int t = 96; t <= kMaxThreadsYZ<T>; t += 32) {
    auto rounds = [t](int items) { return (items + t - 1) / t; };
    const double work = rounds(s.N[2] * s.L1[1]) * s.L2[1] + rounds(s.N[2] * s.L2[1]) * s.L1[1] +
                        rounds(zrows * s.L1[2]) * s.L2[2] + rounds(zrows * s.L2[2]) * s.L1[2] + 8.0;
    const double cost = launch_cost(sizeof(T) == 4 ? 768 : 512, static_cast<double>(s.max_slabs) * nb * s.nk, t, smem, work);
    if (cost < best * 0.999) {
      best = cost;
      threads = t;
    }
  }
  return threads;
}

// CTAs of the FP32 x-pass of up to 160 threads have 96 registers, four an SM, while
// shared memory lets three in (N0 <= 136); longer axes take up to 256 threads of
// 128 registers.  FP64 takes the latter always.  (96^3, 160 bands / 72^3, 800
// bands, us: 160 threads 367 / 774, 192 of 112 registers 354 / 842, 256 360 / 843.)
template <typename T> int x_max_threads(size_t smem) {
  return sizeof(T) == 4 && 3 * (smem + 1024) <= kSmemPerSm + 1024 ? 160 : kThreads;
}

// CTA size of the x-pass and the tiles a CTA takes.  A plane's N1 N2 columns are
// one contiguous range, so its tiles need not be y-rows: they are x_cols columns
// (512 B of a row), and the warps take the L1 subs of the outer passes
// (radix L2, twice) and the L2 of the middle step (radix L1, both directions) in
// as few rounds as launch_cost allows.  si64 (96^3): 3 + 2 full rounds of 4 warps.
// In FP32 up to 8 tiles share a CTA's tables while 4 waves of CTAs are left.
// Measured against whole y-rows flattened over 256 threads (x-pass, us): si64, 160
// bands 436 -> 367 (FP64, 32 bands 592 -> 568), 36^3, 144 bands 38 -> 20 (FP64 177 ->
// 136), 72^3, 800 bands 1046 -> 751.
template <typename T> void x_shape(const qgb_sphere& s, int nb, int* threads, int* tiles) {
  const int L1 = s.L1[0], L2 = s.L2[0];
  const size_t smem = x_smem_bytes(s, 32, 16);
  const int max_threads = x_max_threads<T>(smem), resident = max_threads == 160 ? 640 : 512;
  const double total = (static_cast<double>(s.N[1]) * s.N[2] + x_cols<T> - 1) / x_cols<T> * nb * s.nk;
  double best = 1e30;
  *threads = 128;
  for (int w = 1; w <= max_threads / 32; ++w) {
    const int outer = L2 > 1 ? (L1 + w - 1) / w : 0, mid = (L2 + w - 1) / w;
    const double work = 2.0 * (outer * L2 + mid * L1) + 8.0;
    const double cost = launch_cost(resident, total, 32 * w, smem, work);
    if (cost < best * 0.999) {
      best = cost;
      *threads = 32 * w;
    }
  }
  const int ctas = std::max(1, resident / *threads);
  *tiles = sizeof(T) == 8 ? 1 : std::max(1, std::min(8, static_cast<int>(total / (4.0 * 152.0 * ctas))));
}

template <typename T, int MAXT>
int launch_x(const qgb_sphere& s, const LocalParams& lp, void* planes, cudaStream_t st) {
  const size_t smem = x_smem_bytes(s, 32, 16);  // rows of 32 x 16 B: double complex, or two of float
  if (int rc = raise_smem_limit(k_xpass<T, MAXT>, smem)) return rc;
  int threads, tiles;
  x_shape<T>(s, lp.nb, &threads, &tiles);
  const int cta_cols = x_cols<T> * tiles;
  k_xpass<T, MAXT><<<dim3((s.N[1] * s.N[2] + cta_cols - 1) / cta_cols, lp.nb, s.nk), threads, smem, st>>>(
      s, lp, static_cast<cplx_t<T>*>(planes), tiles);
  QGB_LAUNCH_CHECK("k_xpass");
  return QGB_OK;
}

template <typename T>
int launch_ifft_yz(const qgb_sphere& s, const LocalParams& lp, const void* C, void* planes, cudaStream_t st) {
  const size_t smem = yz_smem_bytes(s, sizeof(cplx_t<T>));
  if (int rc = raise_smem_limit(k_ifft_yz<T>, smem)) return rc;
  k_ifft_yz<T><<<dim3(s.max_slabs, lp.nb, s.nk), threads_yz<T>(s, lp.nb), smem, st>>>(
      s, lp, static_cast<const cplx_t<T>*>(C), static_cast<cplx_t<T>*>(planes));
  QGB_LAUNCH_CHECK("k_ifft_yz");
  return QGB_OK;
}

template <typename T>
int launch_chunk(const qgb_sphere& s, const LocalParams& lp, const void* C, void* out, void* planes, cudaStream_t st,
                 cudaEvent_t gather_after) {
  using C2 = cplx_t<T>;
  int rc;
  if ((rc = launch_ifft_yz<T>(s, lp, C, planes, st))) return rc;
  if constexpr (sizeof(T) == 4) {
    rc = x_max_threads<T>(x_smem_bytes(s, 32, 16)) == 160 ? launch_x<T, 160>(s, lp, planes, st)
                                                          : launch_x<T, kThreads>(s, lp, planes, st);
  } else {
    rc = launch_x<T, kThreads>(s, lp, planes, st);
  }
  if (rc) return rc;
  if (gather_after) QGB_CUDA_CHECK(cudaStreamWaitEvent(st, gather_after, 0));
  const size_t smem = yz_smem_bytes(s, sizeof(C2));
  if ((rc = raise_smem_limit(k_fft_yz_gather<T>, smem))) return rc;
  k_fft_yz_gather<T><<<dim3(s.max_slabs, lp.nb, s.nk), threads_yz<T>(s, lp.nb), smem, st>>>(
      s, lp, static_cast<const C2*>(C), static_cast<C2*>(out), static_cast<const C2*>(planes));
  QGB_LAUNCH_CHECK("k_fft_yz_gather");
  return QGB_OK;
}

#ifdef QGB_DEBUG_CHECKS
// Debug builds: add this translation unit's first recorded range violation
// (site, index, limit, packed block index; site 0 = none) to out4 if that is
// still empty, and clear it.
static int unit_violation(unsigned long long* out4) {
  unsigned long long v[4];
  QGB_CUDA_CHECK(cudaMemcpyFromSymbol(v, g_qgb_violation, sizeof(v)));
  const unsigned long long zero[4] = {0, 0, 0, 0};
  QGB_CUDA_CHECK(cudaMemcpyToSymbol(g_qgb_violation, zero, sizeof(zero)));
  if (out4[0] == 0)
    for (int i = 0; i < 4; ++i) out4[i] = v[i];
  return QGB_OK;
}
#endif

}  // namespace qgb
