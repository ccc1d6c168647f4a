// Tensor-core (tcgen05) split-BF16x3 GEMM and the mixed-precision nonlocal term.
//
// D[m][n] = sum_k A[m][k] B[n][k] (both operands K-major, "TN") is computed as
//   A_hi B_hi^T + A_hi B_lo^T + A_lo B_hi^T,   x_hi = bf16(x), x_lo = bf16(x - x_hi),
// with FP32 accumulation in tensor memory: about 16 significant bits per
// product, the split-BF16x3 scheme.  How the three products meet (Order):
//   ORDER_SEGMENTS  one after the other over the whole K range, into one
//                   accumulator (the subspace overlaps, whose FP64 results keep
//                   their bits);
//   ORDER_BLOCKS    the three of a K block together, so a block takes 4 operand
//                   tiles from L2 and not 6;
//   ORDER_SPLIT     the same with the two small products in an accumulator of
//                   their own, added at the end: a third of the roundings at
//                   the size of the result, for long K ranges.
//
// Persistent CTAs, one per SM (192 threads); a unit is a 128 x BN output tile of
// one K range, N tiles fastest:
//   warps 0-3 - epilogue: tcgen05.ld of their 32 TMEM lanes, from one of two
//               accumulators (256 columns each) while the next unit's MMAs fill
//               the other;
//   warp 4    - TMA producer: 128B-swizzled boxes of A_hi, A_lo, B_hi and B_lo of
//               a K = 64 block into one stage of a shared-memory ring, so the
//               three products take 4 tiles from L2 and not 6 (the SM's ingest,
//               64 B a cycle, is the bound: 96 KB and 1536 MMA cycles per block
//               at BN = 256);
//   warp 5    - MMA issuer: tcgen05.mma.cta_group::1.kind::f16 with bf16 inputs
//               and an FP32 accumulator, twelve K = 16 steps per stage.
// BN is the smallest multiple of 32 that covers the band rows in equal tiles.
// Every mbarrier wait is bounded by a %globaltimer deadline; on timeout the
// kernel records an error code, drains its own TMA copies (bounded), frees its
// TMEM and returns.
//
// Complex products map onto this real GEMM by stacking real and imaginary
// parts as rows (see the nonlocal section below).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "tcgen05.cuh"

namespace qgb {
namespace tc {

constexpr int BM = 128;            // MMA M (rows of A per CTA)
constexpr int BK = 64;             // bf16 elements per stage along K (one 128 B swizzle atom)
constexpr int EPI_WARPS = 4;
constexpr int kThreads = (EPI_WARPS + 2) * 32;
constexpr int kSms = 152;
constexpr int ACC_COLS = 256;      // TMEM columns of one accumulator (two of them)
constexpr int MAX_STAGES = 4;

enum Epi { EPI_PARTIAL = 0, EPI_ADD_HC = 1 };
enum Order { ORDER_SEGMENTS = 0, ORDER_BLOCKS = 1, ORDER_SPLIT = 2 };

struct GemmArgs {
  int M, N, K;             // logical sizes (rows of A, rows of B, reduction)
  int BN, HB, stages;      // tile width (rows of B), bands per tile, ring depth
  int order;
  int units, m_tiles, n_tiles;
  int kb_per_split;        // 64-wide K blocks per split
  int splits;
  float* partial;          // EPI_PARTIAL: [batch][split][m_tiles*BM][n_tiles*BN]
  int part_ld;             // n_tiles * BN
  long long part_rows;     // m_tiles * BM
  float2* hc;              // EPI_ADD_HC: complex64 [batch][nb][hc_ld], += D
  long long hc_batch_stride;
  int hc_ld, nb;
  int hc_store;            // EPI_ADD_HC: 1 = store D instead of adding it
  int* err;                // device error word (0 = ok)
  unsigned long long timeout_ns;  // limit of each pipeline wait (kTimeoutNs)
  int skip_loads;          // test aid: the producer issues no copies, so the MMA wait runs out
};

constexpr int A_BYTES = BM * BK * 2;  // one of A_hi, A_lo: 16 KB
__host__ __device__ constexpr int stage_bytes(int bn, int order) {
  return (A_BYTES + bn * BK * 2) * (order == ORDER_SEGMENTS ? 1 : 2);
}
constexpr int BAR_BYTES = (2 * MAX_STAGES + 5) * 8 + 16;
__host__ __device__ constexpr int smem_bytes(int bn, int order, int stages) {
  return stages * stage_bytes(bn, order) + BAR_BYTES + 1024;  // + alignment slack
}

struct Unit {
  int n_tile, m_tile, split, batch;
};
__device__ __forceinline__ Unit unit_of(const GemmArgs& a, int u) {
  Unit t;
  t.n_tile = u % a.n_tiles;
  u /= a.n_tiles;
  t.m_tile = u % a.m_tiles;
  u /= a.m_tiles;
  t.split = u % a.splits;
  t.batch = u / a.splits;
  return t;
}

template <int EPI>
__global__ void __launch_bounds__(kThreads, 1)
    k_tc_gemm(const __grid_constant__ CUtensorMap mA_hi, const __grid_constant__ CUtensorMap mA_lo,
              const __grid_constant__ CUtensorMap mB_hi, const __grid_constant__ CUtensorMap mB_lo,
              const GemmArgs args) {
  extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
  // 1024-byte alignment for the 128B-swizzled tiles.
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int BN = args.BN, S = args.stages, STAGE = stage_bytes(BN, args.order), B_BYTES = BN * BK * 2;
  const int segments = args.order == ORDER_SEGMENTS ? 3 : 1;
  // Accumulators: two in turn, or (ORDER_SPLIT) the products' own two.
  const int bufs = args.order == ORDER_SPLIT ? 1 : 2;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * STAGE);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* acc_full = empty + MAX_STAGES;  // [2]
  uint64_t* acc_empty = acc_full + 2;       // [2]
  uint64_t* done = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nkb_total = (args.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], EPI_WARPS);
    }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == EPI_WARPS + 1) tmem_alloc(tmem_slot, 2 * ACC_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (threadIdx.x == EPI_WARPS * 32 && !args.skip_loads) {
    // ---------------- TMA producer ----------------
    int it = 0;  // stages filled so far, over all units
    bool live = true;
    for (int u = blockIdx.x; u < args.units && live; u += gridDim.x) {
      const Unit t = unit_of(args, u);
      const int kb0 = t.split * args.kb_per_split, nkb = min(nkb_total, kb0 + args.kb_per_split) - kb0;
      for (int i = 0; i < segments * nkb; ++i, ++it) {
        const int s = it % S, use = it / S;
        if (use > 0 && !mbar_wait(&empty[s], (use - 1) & 1, args.err, 1, args.timeout_ns)) {
          live = false;
          break;
        }
        const int seg = i / nkb, k = (kb0 + i - seg * nkb) * BK;
        unsigned char* dst = smem + s * STAGE;
        mbar_arrive_expect_tx(&full[s], STAGE);
        if (segments == 3) {
          tma_load_3d(dst, seg == 2 ? &mA_lo : &mA_hi, &full[s], k, t.m_tile * BM, t.batch);
          tma_load_3d(dst + A_BYTES, seg == 1 ? &mB_lo : &mB_hi, &full[s], k, t.n_tile * BN, t.batch);
        } else {
          tma_load_3d(dst, &mA_hi, &full[s], k, t.m_tile * BM, t.batch);
          tma_load_3d(dst + 2 * A_BYTES, &mB_hi, &full[s], k, t.n_tile * BN, t.batch);
          tma_load_3d(dst + 2 * A_BYTES + B_BYTES, &mB_lo, &full[s], k, t.n_tile * BN, t.batch);
          tma_load_3d(dst + A_BYTES, &mA_lo, &full[s], k, t.m_tile * BM, t.batch);
        }
      }
    }
    // Drain: every load issued lands before exit.  Loads before the last S were
    // waited for through the empty barriers (their MMAs consumed them); the
    // last min(S, issued) are waited for here, even after an error.
    for (int i = max(0, it - S); i < it; ++i) mbar_drain(&full[i % S], (i / S) & 1, args.err, 2);
  } else if (threadIdx.x == (EPI_WARPS + 1) * 32) {
    // ---------------- MMA issuer ----------------
    const uint32_t idesc = idesc_bf16_f32(BM, BN);
    const uint32_t b_step = static_cast<uint32_t>(B_BYTES / 16);
    int it = 0, n = 0;  // stages and units so far
    bool live = true;
    for (int u = blockIdx.x; u < args.units && live; u += gridDim.x, ++n) {
      const Unit t = unit_of(args, u);
      const int kb0 = t.split * args.kb_per_split, nkb = min(nkb_total, kb0 + args.kb_per_split) - kb0;
      const int buf = n % bufs;
      const uint32_t acc = tmem + buf * ACC_COLS, acc2 = bufs == 1 ? tmem + ACC_COLS : acc;
      if (n >= bufs && !mbar_wait(&acc_empty[buf], (n / bufs - 1) & 1, args.err, 5, args.timeout_ns)) break;
      tc_fence_after();
      for (int i = 0; i < segments * nkb; ++i, ++it) {
        const int s = it % S;
        if (!mbar_wait(&full[s], (it / S) & 1, args.err, 3, args.timeout_ns)) {
          live = false;
          break;
        }
        tc_fence_after();
        const uint32_t addr = smem_u32(smem + s * STAGE);
        const uint64_t a_hi = desc_kmajor_sw128(addr);
        const uint64_t b_hi = desc_kmajor_sw128(addr + (segments == 3 ? A_BYTES : 2 * A_BYTES));
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)  // K = 16 per MMA: advance 32 B = 2 descriptor units
          umma_bf16(acc, a_hi + 2 * k, b_hi + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
        if (segments == 1) {
          const uint64_t a_lo = a_hi + A_BYTES / 16, b_lo = b_hi + b_step;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_bf16(acc2, a_hi + 2 * k, b_lo + 2 * k, idesc, (bufs == 1 && i == 0 && k == 0) ? 0u : 1u);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) umma_bf16(acc2, a_lo + 2 * k, b_hi + 2 * k, idesc, 1u);
        }
        umma_commit(&empty[s]);
      }
      umma_commit(&acc_full[buf]);
    }
    umma_commit(done);  // fires once every MMA issued above has completed
  } else if (warp < EPI_WARPS) {
    // ---------------- Epilogue ----------------
    int n = 0;
    for (int u = blockIdx.x; u < args.units; u += gridDim.x, ++n) {
      const Unit t = unit_of(args, u);
      const int buf = n % bufs;
      bool ok = mbar_wait(&acc_full[buf], (n / bufs) & 1, args.err, 4, 2 * kTimeoutNs);
      // tcgen05.ld is warp-collective: decide per warp.
      ok = __all_sync(0xffffffffu, ok && *reinterpret_cast<volatile int*>(args.err) == 0);
      if (!ok) break;
      tc_fence_after();
      const bool any = t.split * args.kb_per_split < nkb_total;  // an empty K range adds nothing
      const int row = t.m_tile * BM + warp * 32 + lane;
      const uint32_t trow = tmem + buf * ACC_COLS + (static_cast<uint32_t>(warp * 32) << 16);
      if (EPI == EPI_PARTIAL) {
        float* out = args.partial + ((static_cast<long long>(t.batch) * args.splits + t.split) * args.part_rows + row) *
                                        args.part_ld + t.n_tile * BN;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 32) {
          float v[32];
          tmem_ld32(trow + c0, v);
          if (bufs == 1) {
            float w[32];
            tmem_ld32(trow + ACC_COLS + c0, w);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += w[i];
          }
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<float4*>(out + c0 + i) =
                any ? make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      } else {
        // Columns [0, HB) hold real parts and [HB, BN) imaginary parts of bands
        // n_tile * HB + j; rows are basis entries g.
        const int HB = args.HB;
        const bool row_ok = row < args.M;
        float2* hc = args.hc + t.batch * args.hc_batch_stride + row;
#pragma unroll 1
        for (int c0 = 0; c0 < HB; c0 += 16) {
          float vr[16], vi[16];
          // All loads of HC first, then the stores: interleaved read-modify-
          // writes through one pointer could alias, which would serialise the
          // memory round trips.
          float2 o[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int b = t.n_tile * HB + c0 + i;
            o[i] = (!args.hc_store && row_ok && b < args.nb) ? hc[static_cast<long long>(b) * args.hc_ld]
                                                             : make_float2(0.f, 0.f);
          }
          tmem_ld16(trow + c0, vr);
          tmem_ld16(trow + HB + c0, vi);
          if (bufs == 1) {
            float wr[16], wi[16];
            tmem_ld16(trow + ACC_COLS + c0, wr);
            tmem_ld16(trow + ACC_COLS + HB + c0, wi);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              vr[i] += wr[i];
              vi[i] += wi[i];
            }
          }
          if (row_ok) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int b = t.n_tile * HB + c0 + i;
              if (b < args.nb)
                hc[static_cast<long long>(b) * args.hc_ld] = make_float2(o[i].x + vr[i], o[i].y + vi[i]);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
    // Every MMA issued has completed before TMEM is freed, error or not.
    mbar_drain(done, 0, args.err, 6);
    tc_fence_before();
  }
  __syncwarp();
  __syncthreads();
  if (warp == EPI_WARPS + 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 2 * ACC_COLS);
  }
}

// ---------------------------------------------------------------------------
// Host: tensor maps and launches
// ---------------------------------------------------------------------------

// 3D bf16 tensor [batch][rows][ld] (K innermost, `k_extent` valid), box
// 64 x box_rows x 1 with 128-byte swizzle; out-of-range elements read as zero.
static int make_map(CUtensorMap* m, const void* base, long long k_extent, long long rows, long long batch,
                    long long ld, long long batch_stride, int box_rows) {
  auto enc = encode_fn();
  if (!enc) return fail(QGB_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable from the driver");
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (ld * 2) % 16 || (batch_stride * 2) % 16)
    return fail(QGB_ERR_INVALID, "tensor-map operand not 16-byte aligned (ld=%lld)", ld);
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(k_extent), static_cast<cuuint64_t>(rows),
                        static_cast<cuuint64_t>(batch)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld * 2), static_cast<cuuint64_t>(batch_stride * 2)};
  cuuint32_t box[3] = {static_cast<cuuint32_t>(BK), static_cast<cuuint32_t>(box_rows), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(QGB_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", static_cast<int>(r));
  return QGB_OK;
}

// Operand description for one side: hi/lo bf16 arrays [batch][rows][ld].
struct Operand {
  const void* hi;
  const void* lo;
  long long rows, ld, batch_stride;
};

// Tile of `nb` bands: rows of B per tile (real and imaginary rows of HB bands
// each, HB a multiple of 16), as few tiles as 256 rows allow and those equal.
static int band_tile(int nb) {
  const int tiles = (nb + 127) / 128, hb = (nb + tiles - 1) / tiles;
  return 2 * std::max(16, (hb + 15) / 16 * 16);
}
static int ring_depth(int bn, int order) {
  return std::min(MAX_STAGES, (227 * 1024 - BAR_BYTES - 1024) / stage_bytes(bn, order));
}

// K splits of a product of `tiles` output tiles of 128 x bn and nkb K blocks: the
// number that needs the least time, a block taking its copies' 64 B a cycle, a
// unit some 2000 cycles more, a split the write and read of its partial sums.
static int pick_splits(int tiles, int nkb, int bn) {
  int best = 1;
  double best_cost = 1e30;
  for (int s = 1; s <= std::min(nkb, 64); ++s) {
    const int per = (nkb + s - 1) / s;
    const double waves = std::ceil(static_cast<double>(tiles) * ((nkb + per - 1) / per) / kSms);
    const double cost = waves * (per * (stage_bytes(bn, ORDER_SPLIT) / 64.0) + 2000.0) +
                        static_cast<double>(tiles) * s * (BM * bn * 8.0) / 2500.0;
    if (cost < best_cost * 0.999) {
      best_cost = cost;
      best = s;
    }
  }
  return best;
}

template <int EPI>
static int launch(const Operand& A, const Operand& B, int K, int batch, const GemmArgs& args_in, cudaStream_t st) {
  GemmArgs args = args_in;
  if (args.timeout_ns == 0) args.timeout_ns = kTimeoutNs;
  CUtensorMap ma_hi, ma_lo, mb_hi, mb_lo;
  int rc;
  if ((rc = make_map(&ma_hi, A.hi, K, A.rows, batch, A.ld, A.batch_stride, BM))) return rc;
  if ((rc = make_map(&ma_lo, A.lo, K, A.rows, batch, A.ld, A.batch_stride, BM))) return rc;
  if ((rc = make_map(&mb_hi, B.hi, K, B.rows, batch, B.ld, B.batch_stride, args.BN))) return rc;
  if ((rc = make_map(&mb_lo, B.lo, K, B.rows, batch, B.ld, B.batch_stride, args.BN))) return rc;
  args.HB = args.BN / 2;
  args.stages = ring_depth(args.BN, args.order);
  const size_t smem = smem_bytes(args.BN, args.order, args.stages);
  if ((rc = raise_smem_limit(k_tc_gemm<EPI>, smem))) return rc;
  args.m_tiles = static_cast<int>((A.rows + BM - 1) / BM);
  args.n_tiles = static_cast<int>((B.rows + args.BN - 1) / args.BN);
  args.units = args.m_tiles * args.n_tiles * batch * args.splits;
  k_tc_gemm<EPI><<<std::min(args.units, kSms), kThreads, smem, st>>>(ma_hi, ma_lo, mb_hi, mb_lo, args);
  QGB_LAUNCH_CHECK("k_tc_gemm");
  return QGB_OK;
}

// ---------------------------------------------------------------------------
// Split kernels (FP32 -> bf16 hi/lo)
// ---------------------------------------------------------------------------

__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16& hi, __nv_bfloat16& lo) {
  hi = __float2bfloat16_rn(x);
  lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}

__device__ __forceinline__ unsigned pack_pair(__nv_bfloat16 a, __nv_bfloat16 b) {
  return static_cast<unsigned>(__bfloat16_as_ushort(a)) | (static_cast<unsigned>(__bfloat16_as_ushort(b)) << 16);
}
// 4 values -> their bf16 hi and lo parts, 8 B each.
__device__ __forceinline__ void split4(const float (&v)[4], uint2& hi, uint2& lo) {
  __nv_bfloat16 h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) split_bf16(v[i], h[i], l[i]);
  hi = make_uint2(pack_pair(h[0], h[1]), pack_pair(h[2], h[3]));
  lo = make_uint2(pack_pair(l[0], l[1]), pack_pair(l[2], l[3]));
}

// Bands as operand rows: complex64 C[k][nb][n_tot] -> rows r = t*2HB + part*HB + j
// (band t*HB + j, part 0 = real, 1 = imaginary) of [k][rows][ld] bf16 hi/lo;
// bands >= nb give zero rows.  With `weight` (real wavefunctions: 1 on the
// Gz = 0 plane, 2 elsewhere; powers of two, so the split stays exact) every
// coefficient is scaled by w_g.  A thread takes 4 basis entries of a band, both
// parts: bound by its 16 B moved per entry (one part and one entry a thread,
// reading everything twice: 107 us against 51 for 4 x 200 x 19926).
__global__ void __launch_bounds__(256) k_split_bands(const float2* __restrict__ C, int nb, int n_tot, int HB, int rows,
                                                     int ld, const double* __restrict__ weight,
                                                     __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo) {
  const int b = blockIdx.y, k = blockIdx.z;
  const int t = b / HB, r = t * 2 * HB + (b - t * HB);
  const float2* src = C + (static_cast<long long>(k) * nb + b) * n_tot;
  const long long o_re = (static_cast<long long>(k) * rows + r) * ld, o_im = o_re + static_cast<long long>(HB) * ld;
  for (int g = 4 * (blockIdx.x * blockDim.x + threadIdx.x); g < ld; g += 4 * gridDim.x * blockDim.x) {
    float re[4], im[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 c = make_float2(0.f, 0.f);
      if (b < nb && g + i < n_tot) {
        c = src[g + i];
        if (weight) {
          const float w = static_cast<float>(weight[g + i]);
          c.x *= w;
          c.y *= w;
        }
      }
      re[i] = c.x;
      im[i] = c.y;
    }
    uint2 h, l;
    split4(re, h, l);
    *reinterpret_cast<uint2*>(hi + o_re + g) = h;
    *reinterpret_cast<uint2*>(lo + o_re + g) = l;
    split4(im, h, l);
    *reinterpret_cast<uint2*>(hi + o_im + g) = h;
    *reinterpret_cast<uint2*>(lo + o_im + g) = l;
  }
}

static int launch_split_bands(const void* C, int nb, int nk, int n_tot, int HB, long long rows, long long ld,
                              const double* weight, __nv_bfloat16* hi, __nv_bfloat16* lo, cudaStream_t st) {
  const dim3 grid(static_cast<unsigned>(std::min<long long>(32, (ld + 1023) / 1024)), static_cast<unsigned>(rows / 2), nk);
  k_split_bands<<<grid, 256, 0, st>>>(static_cast<const float2*>(C), nb, n_tot, HB, static_cast<int>(rows),
                                      static_cast<int>(ld), weight, hi, lo);
  QGB_LAUNCH_CHECK("k_split_bands");
  return QGB_OK;
}

// Projector operands, once per basis: complex64 beta[k][P][n_tot] ->
//   A  [k][2P][ldA]  rows (Re beta_p; Im beta_p), K = basis  (for <beta|psi>)
//   AT [k][n_tot][ldT] row g = (Re beta_p(g), p < P; Im beta_p(g)), K = 2P
//                                                     (for beta (D proj))
__global__ void k_split_beta(const float2* __restrict__ beta, int P, int n_tot, int ldA, int ldT,
                             __nv_bfloat16* __restrict__ a_hi, __nv_bfloat16* __restrict__ a_lo,
                             __nv_bfloat16* __restrict__ t_hi, __nv_bfloat16* __restrict__ t_lo) {
  const int p = blockIdx.y, k = blockIdx.z;
  const float2* src = beta + (static_cast<long long>(k) * P + p) * n_tot;
  const long long oa_r = (static_cast<long long>(k) * 2 * P + p) * ldA;
  const long long oa_i = (static_cast<long long>(k) * 2 * P + P + p) * ldA;
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ldA; g += gridDim.x * blockDim.x) {
    const float2 c = (g < n_tot) ? src[g] : make_float2(0.f, 0.f);
    __nv_bfloat16 h, l;
    split_bf16(c.x, h, l);
    a_hi[oa_r + g] = h;
    a_lo[oa_r + g] = l;
    if (g < n_tot) {
      const long long ot = (static_cast<long long>(k) * n_tot + g) * ldT;
      t_hi[ot + p] = h;
      t_lo[ot + p] = l;
    }
    split_bf16(c.y, h, l);
    a_hi[oa_i + g] = h;
    a_lo[oa_i + g] = l;
    if (g < n_tot) {
      const long long ot = (static_cast<long long>(k) * n_tot + g) * ldT;
      t_hi[ot + P + p] = h;
      t_lo[ot + P + p] = l;
    }
  }
}

// Reduce split-K partials of <beta|psi> into projT[k][b][p] (complex64):
// D rows m < P are Re beta_m, rows P + m are Im beta_m; columns follow the
// band-row order of k_split_bands.
//   Re <b_p|psi_b> = D[p][re b] + D[P+p][im b],  Im = D[p][im b] - D[P+p][re b]
// Threads run along the band columns of a partial row (coalesced reads).
// Block (32, 8): threadIdx.x runs along bands, threadIdx.y strides the splits;
// the 8 partial sums of each band are combined in shared memory.
__global__ void k_reduce_proj(const float* __restrict__ partial, int splits, long long part_rows, int part_ld,
                              int P, int nb, int HB, int real_out, float2* __restrict__ projT) {
  __shared__ float2 acc[8][32];
  const int k = blockIdx.z, p = blockIdx.y;
  const int b = blockIdx.x * 32 + threadIdx.x;
  float re = 0.f, im = 0.f;
  if (b < nb) {
    const int t = b / HB, j = b - t * HB;
    const int c_re = t * 2 * HB + j, c_im = c_re + HB;
    for (int s = threadIdx.y; s < splits; s += 8) {
      const float* D = partial + (static_cast<long long>(k) * splits + s) * part_rows * part_ld;
      const float* r0 = D + static_cast<long long>(p) * part_ld;
      const float* r1 = D + static_cast<long long>(P + p) * part_ld;
      re += r0[c_re] + r1[c_im];
      im += r0[c_im] - r1[c_re];
    }
  }
  acc[threadIdx.y][threadIdx.x] = make_float2(re, im);
  __syncthreads();
  if (threadIdx.y == 0 && b < nb) {
    float2 sum = acc[0][threadIdx.x];
#pragma unroll
    for (int y = 1; y < 8; ++y) {
      sum.x += acc[y][threadIdx.x].x;
      sum.y += acc[y][threadIdx.x].y;
    }
    if (real_out) sum.y = 0.f;  // real wavefunctions: the implicit -G partners cancel it
    projT[(static_cast<long long>(k) * nb + b) * P + p] = sum;
  }
}

// Reduce split-K partials of a Gram product into out (complex128):
// out[k*out_batch + i*oi + j*oj] = <X_i|Y_j>, partial rows i < nx Re X_i,
// nx + i Im X_i; columns follow the band-row order of k_split_bands.  Splits
// are summed in FP64, in split order.
__global__ void k_reduce_gram(const float* __restrict__ partial, int splits, long long part_rows, int part_ld,
                              int nx, int ny, int HB, double2* __restrict__ out, long long out_batch, int oi,
                              int oj) {
  const int k = blockIdx.z, i = blockIdx.y;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < ny; j += gridDim.x * blockDim.x) {
    const int t = j / HB, jj = j - t * HB;
    const int c_re = t * 2 * HB + jj, c_im = c_re + HB;
    double re = 0.0, im = 0.0;
    for (int s = 0; s < splits; ++s) {
      const float* D = partial + (static_cast<long long>(k) * splits + s) * part_rows * part_ld;
      const float* r0 = D + static_cast<long long>(i) * part_ld;
      const float* r1 = D + static_cast<long long>(nx + i) * part_ld;
      re += static_cast<double>(r0[c_re]) + static_cast<double>(r1[c_im]);
      im += static_cast<double>(r0[c_im]) - static_cast<double>(r1[c_re]);
    }
    out[k * out_batch + static_cast<long long>(i) * oi + static_cast<long long>(j) * oj] = make_double2(re, im);
  }
}

// Dp[b][p] = sum_q D_atom[a][p'][q'] projT[b][a*pa + q'] (block-diagonal D),
// written as the back-projection B operand: rows r = t*2HB + part*HB + j for
// band t*HB + j, K = 2P: real-output row (Re Dp, -Im Dp), imaginary-output
// row (Im Dp, Re Dp).  One CTA per band computes both rows.
__global__ void k_dapply_split(const float2* __restrict__ projT, const float2* __restrict__ D, int n_atoms,
                               int pa, int nb, int HB, int rows, int ld, __nv_bfloat16* __restrict__ hi,
                               __nv_bfloat16* __restrict__ lo) {
  const int P = n_atoms * pa;
  const int b = blockIdx.y, k = blockIdx.z;
  const int t = b / HB, r = t * 2 * HB + (b - t * HB);
  const long long o_re = (static_cast<long long>(k) * rows + r) * ld, o_im = o_re + static_cast<long long>(HB) * ld;
  for (int p = threadIdx.x; p < ld; p += blockDim.x) {
    float re = 0.f, im = 0.f;
    if (b < nb && p < P) {
      const int a = p / pa, pp = p - a * pa;
      const float2* Drow = D + (static_cast<long long>(a) * pa + pp) * pa;
      const float2* x = projT + (static_cast<long long>(k) * nb + b) * P + a * pa;
      for (int q = 0; q < pa; ++q) {
        const float2 d = Drow[q], v = x[q];
        re += d.x * v.x - d.y * v.y;
        im += d.x * v.y + d.y * v.x;
      }
    }
    __nv_bfloat16 h, l;
    if (p < P) {
      split_bf16(re, h, l);
      hi[o_re + p] = hi[o_im + P + p] = h;
      lo[o_re + p] = lo[o_im + P + p] = l;
      split_bf16(im, h, l);
      hi[o_im + p] = h;
      lo[o_im + p] = l;
      hi[o_re + P + p] = __hneg(h);
      lo[o_re + P + p] = __hneg(l);
    } else if (p >= 2 * P) {
      const __nv_bfloat16 z = __float2bfloat16_rn(0.f);
      hi[o_re + p] = lo[o_re + p] = hi[o_im + p] = lo[o_im + p] = z;
    }
  }
}

// Band rotation operands.  C complex64 [k][n_in][n] -> A [k][n][ldA]: row g =
// (Re C_i(g), i < Kh; Im C_i(g)), K = 2 Kh with Kh = n_in rounded up to 4,
// through 64 (i) x 32 (g) tiles of shared memory: coalesced reads along g, 128 B
// written per row and array.
__global__ void __launch_bounds__(256) k_split_transpose(const float2* __restrict__ C, int n_in, int Kh, int n, int ldA,
                                                         __nv_bfloat16* __restrict__ hi,
                                                         __nv_bfloat16* __restrict__ lo) {
  __shared__ float2 tile[64][33];
  const int k = blockIdx.z;
  const int g0 = blockIdx.x * 32, i0 = blockIdx.y * 64;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int r = ty; r < 64; r += 8) {
    const int i = i0 + r, g = g0 + tx;
    tile[r][tx] = (i < n_in && g < n) ? C[(static_cast<long long>(k) * n_in + i) * n + g] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  const int seg = 4 * (threadIdx.x & 15);
  for (int r = threadIdx.x >> 4; r < 32; r += 16) {
    const int g = g0 + r, i = i0 + seg;
    if (g >= n || i >= Kh) continue;
    float re[4], im[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 v = tile[seg + j][r];
      re[j] = v.x;
      im[j] = v.y;
    }
    const long long o = (static_cast<long long>(k) * n + g) * ldA + i;
    uint2 h, l;
    split4(re, h, l);
    *reinterpret_cast<uint2*>(hi + o) = h;
    *reinterpret_cast<uint2*>(lo + o) = l;
    split4(im, h, l);
    *reinterpret_cast<uint2*>(hi + o + Kh) = h;
    *reinterpret_cast<uint2*>(lo + o + Kh) = l;
  }
}

// Rotation matrix rows for the B operand: M complex64 [k][n_in][n_out] ->
// rows r = t*BN + part*HB + jj (output band j = t*HB + jj) of [k][rows][ld],
// K = 2 Kh: real-output rows (Re M_ij, -Im M_ij), imaginary-output rows
// (Im M_ij, Re M_ij); bands >= n_out and the K padding are zero.
__global__ void k_split_matrix(const float2* __restrict__ M, int n_in, int Kh, int n_out, int HB, int rows, int ld,
                               __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo) {
  const int r = blockIdx.y, k = blockIdx.z;
  const int t = r / (2 * HB), rem = r - t * 2 * HB, part = rem / HB, j = t * HB + rem % HB;
  const long long o = (static_cast<long long>(k) * rows + r) * ld;
  for (int p = threadIdx.x; p < ld; p += blockDim.x) {
    float v = 0.f;
    const int i = p < Kh ? p : p - Kh;
    if (j < n_out && i < n_in) {
      const float2 m = M[(static_cast<long long>(k) * n_in + i) * n_out + j];
      v = p < Kh ? (part ? m.y : m.x) : (part ? m.x : -m.y);
    }
    __nv_bfloat16 h, l;
    split_bf16(v, h, l);
    hi[o + p] = h;
    lo[o + p] = l;
  }
}

}  // namespace tc

using namespace tc;

// Layout of the per-basis projector split (qgb_beta_split).
struct BetaSplitLayout {
  long long ldA, ldT, a_elems, t_elems;
};
static BetaSplitLayout beta_layout(int nk, int P, int n_tot) {
  BetaSplitLayout L;
  L.ldA = round_up(n_tot, 64);
  L.ldT = round_up(2LL * P, 64);
  L.a_elems = static_cast<long long>(nk) * 2 * P * L.ldA;
  L.t_elems = static_cast<long long>(nk) * n_tot * L.ldT;
  return L;
}
size_t beta_split_bytes(int nk, int P, int n_tot) {
  const BetaSplitLayout L = beta_layout(nk, P, n_tot);
  return static_cast<size_t>(2 * (L.a_elems + L.t_elems)) * 2 + 1024;
}

int beta_split(const void* beta, int nk, int P, int n_tot, void* out, size_t out_bytes, cudaStream_t st) {
  if (nk < 1 || P < 1 || n_tot < 1 || !beta || !out) return fail(QGB_ERR_INVALID, "bad beta_split arguments");
  if (out_bytes < beta_split_bytes(nk, P, n_tot)) return fail(QGB_ERR_WORKSPACE, "beta split buffer too small");
  const BetaSplitLayout L = beta_layout(nk, P, n_tot);
  auto* base = reinterpret_cast<__nv_bfloat16*>(round_up(reinterpret_cast<uintptr_t>(out), 256));
  __nv_bfloat16 *a_hi = base, *a_lo = a_hi + L.a_elems, *t_hi = a_lo + L.a_elems, *t_lo = t_hi + L.t_elems;
  QGB_CUDA_CHECK(cudaMemsetAsync(t_hi, 0, 2 * L.t_elems * 2, st));  // K padding of AT must read as zero
  dim3 grid(static_cast<unsigned>(std::min<long long>(64, (L.ldA + 255) / 256)), P, nk);
  k_split_beta<<<grid, 256, 0, st>>>(static_cast<const float2*>(beta), P, n_tot, static_cast<int>(L.ldA),
                                     static_cast<int>(L.ldT), a_hi, a_lo, t_hi, t_lo);
  QGB_LAUNCH_CHECK("k_split_beta");
  return QGB_OK;
}

struct NlWorkspace {
  long long ldB, rowsB, ldB2, partial_floats, psi_elems, b2_elems;
  int splits, kb_per_split, HB, BN;
};
static NlWorkspace nl_layout(int nk, int P, int nb, int n_tot) {
  NlWorkspace W;
  W.BN = band_tile(nb);
  W.HB = W.BN / 2;
  const long long n_tiles = (nb + W.HB - 1) / W.HB;
  W.rowsB = n_tiles * W.BN;
  W.ldB = round_up(n_tot, 64);
  W.ldB2 = round_up(2LL * P, 64);
  const int nkb = static_cast<int>((n_tot + BK - 1) / BK);
  const int m_tiles = static_cast<int>((2LL * P + BM - 1) / BM);
  const int tiles = m_tiles * static_cast<int>(n_tiles) * nk;
  const int splits = pick_splits(tiles, nkb, W.BN);
  W.kb_per_split = (nkb + splits - 1) / splits;
  W.splits = (nkb + W.kb_per_split - 1) / W.kb_per_split;
  W.partial_floats = static_cast<long long>(nk) * W.splits * m_tiles * BM * (n_tiles * W.BN);
  W.psi_elems = static_cast<long long>(nk) * W.rowsB * W.ldB;
  W.b2_elems = static_cast<long long>(nk) * W.rowsB * W.ldB2;
  return W;
}
size_t nonlocal_tc_workspace_bytes(int nk, int P, int nb, int n_tot) {
  const NlWorkspace W = nl_layout(nk, P, nb, n_tot);
  return static_cast<size_t>(W.partial_floats * 4 + 2 * W.psi_elems * 2 + 2 * W.b2_elems * 2) + 4 * 256 + 64;
}

// phases: 1 = steps 1-3 (everything that depends only on C), 2 = step 4 (the
// accumulation into HC), 3 = both; with 4 added, step 4 stores beta (D proj)
// into HC instead of adding it.  Phase 1 may run beside the local potential.
static int nonlocal_tc_impl(const void* split, const void* D, int n_atoms, int pa, const void* C, void* HC,
                            void* projT, int nk, int nb, int n_tot, const NlWorkspace& W, unsigned char* ws,
                            int* err, int phases, const double* weight, cudaStream_t st) {
  const int P = n_atoms * pa;
  const BetaSplitLayout BL = beta_layout(nk, P, n_tot);
  auto* sbase = reinterpret_cast<const __nv_bfloat16*>(round_up(reinterpret_cast<uintptr_t>(split), 256));
  const __nv_bfloat16 *a_hi = sbase, *a_lo = a_hi + BL.a_elems, *t_hi = a_lo + BL.a_elems,
                      *t_lo = t_hi + BL.t_elems;
  unsigned char* p = reinterpret_cast<unsigned char*>(round_up(reinterpret_cast<uintptr_t>(ws), 256));
  float* partial = reinterpret_cast<float*>(p);
  p += round_up(W.partial_floats * 4, 256);
  auto* b_hi = reinterpret_cast<__nv_bfloat16*>(p);
  auto* b_lo = b_hi + W.psi_elems;
  p += round_up(2 * W.psi_elems * 2, 256);
  auto* b2_hi = reinterpret_cast<__nv_bfloat16*>(p);
  auto* b2_lo = b2_hi + W.b2_elems;

  if (phases & 1) {
  // 1. Wavefunctions -> bf16 hi/lo band rows.
  int rc = launch_split_bands(C, nb, nk, n_tot, W.HB, W.rowsB, W.ldB, weight, b_hi, b_lo, st);
  if (rc) return rc;
  // 2. <beta|psi> partials: M = 2P, N = rowsB, K = basis, split-K.
  GemmArgs g1{};
  g1.M = 2 * P;
  g1.N = static_cast<int>(W.rowsB);
  g1.K = n_tot;
  g1.kb_per_split = W.kb_per_split;
  g1.splits = W.splits;
  g1.partial = partial;
  g1.part_ld = static_cast<int>(W.rowsB);
  g1.part_rows = (2LL * P + BM - 1) / BM * BM;
  g1.err = err;
  g1.BN = W.BN;
  g1.order = ORDER_SPLIT;
  rc = launch<EPI_PARTIAL>(
      Operand{a_hi, a_lo, 2LL * P, BL.ldA, 2LL * P * BL.ldA}, Operand{b_hi, b_lo, W.rowsB, W.ldB, W.rowsB * W.ldB},
      n_tot, nk, g1, st);
  if (rc) return rc;
  // 3. Reduce -> projT; apply D; build the back-projection operand.
  {
    dim3 grid((nb + 31) / 32, P, nk);
    k_reduce_proj<<<grid, dim3(32, 8), 0, st>>>(partial, W.splits, g1.part_rows, g1.part_ld, P, nb, W.HB,
                                                weight != nullptr, static_cast<float2*>(projT));
    QGB_LAUNCH_CHECK("k_reduce_proj");
    dim3 grid2(1, static_cast<unsigned>(W.rowsB / 2), nk);
    k_dapply_split<<<grid2, 256, 0, st>>>(static_cast<const float2*>(projT), static_cast<const float2*>(D),
                                          n_atoms, pa, nb, W.HB, static_cast<int>(W.rowsB),
                                          static_cast<int>(W.ldB2), b2_hi, b2_lo);
    QGB_LAUNCH_CHECK("k_dapply_split");
  }
  }
  if (!(phases & 2)) return QGB_OK;
  // 4. HC += beta (D proj): M = basis, N = rowsB, K = 2P.
  GemmArgs g2{};
  g2.M = n_tot;
  g2.N = static_cast<int>(W.rowsB);
  g2.K = 2 * P;
  g2.kb_per_split = static_cast<int>((2LL * P + BK - 1) / BK);
  g2.splits = 1;
  g2.hc = static_cast<float2*>(HC);
  g2.hc_batch_stride = static_cast<long long>(nb) * n_tot;
  g2.hc_ld = n_tot;
  g2.nb = nb;
  g2.hc_store = (phases & 4) ? 1 : 0;
  g2.err = err;
  g2.BN = W.BN;
  g2.order = ORDER_BLOCKS;
  return launch<EPI_ADD_HC>(
      Operand{t_hi, t_lo, n_tot, BL.ldT, static_cast<long long>(n_tot) * BL.ldT},
      Operand{b2_hi, b2_lo, W.rowsB, W.ldB2, W.rowsB * W.ldB2}, 2 * P, nk, g2, st);
}

int nonlocal_tc_phase(const void* split, const void* D, int n_atoms, int pa, const void* C, void* HC, void* projT,
                      int nk, int nb, int n_tot, void* ws, size_t ws_bytes, int* err, int phases, cudaStream_t st,
                      const double* weight) {
  const int P = n_atoms * pa;
  if (nk < 1 || nb < 0 || n_tot < 1 || P < 0) return fail(QGB_ERR_INVALID, "bad nonlocal_tc sizes");
  if (nb == 0 || P == 0) return QGB_OK;
  if (!split || !D || !C || !HC || !projT || !ws || !err) return fail(QGB_ERR_INVALID, "NULL pointer in nonlocal_tc");
  if (ws_bytes < nonlocal_tc_workspace_bytes(nk, P, nb, n_tot))
    return fail(QGB_ERR_WORKSPACE, "nonlocal_tc workspace too small");
  const NlWorkspace W = nl_layout(nk, P, nb, n_tot);
  unsigned char* w = static_cast<unsigned char*>(ws);
  return nonlocal_tc_impl(split, D, n_atoms, pa, C, HC, projT, nk, nb, n_tot, W, w, err, phases, weight, st);
}

// ---------------------------------------------------------------------------
// Subspace Gram on the tensor cores (mixed form)
// ---------------------------------------------------------------------------
//
// out[k][i][j] = sum_g conj(X[k][i][g]) Y[k][j][g] for complex64 X, Y: X split
// as the A operand (rows Re X_i, Im X_i, K = basis), Y as band rows (B), the
// split-K split-BF16x3 GEMM into FP32 partials, and the complex combination
// summed over the splits in FP64.
struct GramTcLayout {
  long long ldA, a_elems, partial_floats, psi_elems, ldB, rowsB;
  int splits, kb_per_split, HB, BN;
};
static GramTcLayout gram_tc_layout(int nk, int nx, int ny, int n) {
  GramTcLayout G;
  G.BN = band_tile(ny);
  G.HB = G.BN / 2;
  const long long n_tiles = (ny + G.HB - 1) / G.HB, m_tiles = (2LL * nx + BM - 1) / BM;
  G.ldA = G.ldB = round_up(n, 64);
  G.a_elems = static_cast<long long>(nk) * 2 * nx * G.ldA;
  G.rowsB = n_tiles * G.BN;
  G.psi_elems = static_cast<long long>(nk) * G.rowsB * G.ldB;
  // The ranges of K decide how an overlap is rounded (its FP64 value holds the
  // FP32 sums of the ranges), so they do not follow the tile width: about two
  // per SM, over tiles of 32, 64 or 128 bands.
  const int nkb = static_cast<int>((n + BK - 1) / BK);
  const int bands = ny <= 32 ? 32 : (ny <= 64 ? 64 : 128);
  const long long tiles = m_tiles * ((ny + bands - 1) / bands) * nk;
  const int splits = static_cast<int>(std::max(1LL, std::min<long long>(nkb, (2 * 152 + tiles - 1) / tiles)));
  G.kb_per_split = (nkb + splits - 1) / splits;
  G.splits = (nkb + G.kb_per_split - 1) / G.kb_per_split;
  G.partial_floats = static_cast<long long>(nk) * G.splits * m_tiles * BM * G.rowsB;
  return G;
}
size_t gram_tc_workspace_bytes(int nk, int nx, int ny, int n) {
  if (nk < 1 || nx < 1 || ny < 1 || n < 1) return 0;
  const GramTcLayout G = gram_tc_layout(nk, nx, ny, n);
  return static_cast<size_t>(round_up(G.partial_floats * 4, 256) + round_up(2 * G.a_elems * 2, 256) +
                             round_up(2 * G.psi_elems * 2, 256)) + 1024;
}

static int gram_tc_impl(const GramTcLayout& G, const void* X, int nx, const void* Y, int ny, int nk, int n,
                        double2* out, long long out_batch, int oi, int oj, unsigned char* ws, int* err,
                        cudaStream_t st) {
  unsigned char* p = reinterpret_cast<unsigned char*>(round_up(reinterpret_cast<uintptr_t>(ws), 256));
  float* partial = reinterpret_cast<float*>(p);
  p += round_up(G.partial_floats * 4, 256);
  auto* a_hi = reinterpret_cast<__nv_bfloat16*>(p);
  auto* a_lo = a_hi + G.a_elems;
  p += round_up(2 * G.a_elems * 2, 256);
  auto* b_hi = reinterpret_cast<__nv_bfloat16*>(p);
  auto* b_lo = b_hi + G.psi_elems;
  int rc = launch_split_bands(X, nx, nk, n, nx, 2LL * nx, G.ldA, nullptr, a_hi, a_lo, st);
  if (rc) return rc;
  if ((rc = launch_split_bands(Y, ny, nk, n, G.HB, G.rowsB, G.ldB, nullptr, b_hi, b_lo, st))) return rc;
  GemmArgs g{};
  g.M = 2 * nx;
  g.N = static_cast<int>(G.rowsB);
  g.K = n;
  g.kb_per_split = G.kb_per_split;
  g.splits = G.splits;
  g.partial = partial;
  g.part_ld = static_cast<int>(G.rowsB);
  g.part_rows = (2LL * nx + BM - 1) / BM * BM;
  g.err = err;
  g.BN = G.BN;
  g.order = ORDER_SEGMENTS;
  rc = launch<EPI_PARTIAL>(
      Operand{a_hi, a_lo, 2LL * nx, G.ldA, 2LL * nx * G.ldA}, Operand{b_hi, b_lo, G.rowsB, G.ldB, G.rowsB * G.ldB},
      n, nk, g, st);
  if (rc) return rc;
  dim3 grid3(static_cast<unsigned>((ny + 127) / 128), nx, nk);
  k_reduce_gram<<<grid3, 128, 0, st>>>(partial, G.splits, g.part_rows, g.part_ld, nx, ny, G.HB, out, out_batch, oi,
                                       oj);
  QGB_LAUNCH_CHECK("k_reduce_gram");
  return QGB_OK;
}

int gram_tc(const void* X, int nx, const void* Y, int ny, int nk, int n, double2* out, long long out_batch, int oi,
            int oj, void* ws, size_t ws_bytes, int* err, cudaStream_t st) {
  if (nk < 0 || nx < 0 || ny < 0 || n < 1) return fail(QGB_ERR_INVALID, "bad gram_tc sizes");
  if (nk == 0 || nx == 0 || ny == 0) return QGB_OK;
  if (nk > 65535 || nx > 65535) return fail(QGB_ERR_UNSUPPORTED, "gram_tc: nk or nx above 65535");
  if (!X || !Y || !out || !ws || !err) return fail(QGB_ERR_INVALID, "NULL pointer in gram_tc");
  if (ws_bytes < gram_tc_workspace_bytes(nk, nx, ny, n)) return fail(QGB_ERR_WORKSPACE, "gram_tc workspace too small");
  const GramTcLayout G = gram_tc_layout(nk, nx, ny, n);
  unsigned char* w = static_cast<unsigned char*>(ws);
  return gram_tc_impl(G, X, nx, Y, ny, nk, n, out, out_batch, oi, oj, w, err, st);
}

// ---------------------------------------------------------------------------
// Band rotation on the tensor cores (mixed form)
// ---------------------------------------------------------------------------
//
// out[k][j][g] (+)= sum_i M[k][i][j] C[k][i][g] for complex64 C, M, out: C
// transposed and split as the A operand (rows g, K = 2 n_in), M as rotation
// rows (B), one split-BF16x3 GEMM accumulating into out in its epilogue.
struct RotTcLayout {
  long long ldA, a_elems, ldB, rowsB, b_elems;
  int HB, BN, Kh;
};
static RotTcLayout rot_tc_layout(int nk, int n_in, int n_out, int n) {
  RotTcLayout R;
  R.BN = band_tile(n_out);
  R.HB = R.BN / 2;
  R.rowsB = (n_out + R.HB - 1) / R.HB * static_cast<long long>(R.BN);
  R.Kh = static_cast<int>(round_up(n_in, 4));
  R.ldA = round_up(2LL * R.Kh, 64);
  R.ldB = R.ldA;
  R.a_elems = static_cast<long long>(nk) * n * R.ldA;
  R.b_elems = static_cast<long long>(nk) * R.rowsB * R.ldB;
  return R;
}
size_t rotate_tc_workspace_bytes(int nk, int n_in, int n_out, int n) {
  if (nk < 1 || n_in < 1 || n_out < 1 || n < 1) return 0;
  const RotTcLayout R = rot_tc_layout(nk, n_in, n_out, n);
  return static_cast<size_t>(round_up(2 * R.a_elems * 2, 256) + round_up(2 * R.b_elems * 2, 256)) + 1024;
}

static int rotate_tc_impl(const RotTcLayout& R, const void* C, int n_in, int nk, int n, const void* M, int n_out,
                          void* out, bool accumulate, unsigned char* ws, int* err, cudaStream_t st) {
  unsigned char* p = reinterpret_cast<unsigned char*>(round_up(reinterpret_cast<uintptr_t>(ws), 256));
  auto* a_hi = reinterpret_cast<__nv_bfloat16*>(p);
  auto* a_lo = a_hi + R.a_elems;
  p += round_up(2 * R.a_elems * 2, 256);
  auto* b_hi = reinterpret_cast<__nv_bfloat16*>(p);
  auto* b_lo = b_hi + R.b_elems;
  // The K padding [2 Kh, ldA) of A is outside the tensor map's K extent and
  // reads as zero.
  {
    dim3 grid(static_cast<unsigned>((n + 31) / 32), static_cast<unsigned>((R.Kh + 63) / 64), nk);
    k_split_transpose<<<grid, 256, 0, st>>>(static_cast<const float2*>(C), n_in, R.Kh, n, static_cast<int>(R.ldA), a_hi,
                                            a_lo);
    QGB_LAUNCH_CHECK("k_split_transpose");
    dim3 grid2(1, static_cast<unsigned>(R.rowsB), nk);
    k_split_matrix<<<grid2, 256, 0, st>>>(static_cast<const float2*>(M), n_in, R.Kh, n_out, R.HB,
                                          static_cast<int>(R.rowsB), static_cast<int>(R.ldB), b_hi, b_lo);
    QGB_LAUNCH_CHECK("k_split_matrix");
  }
  GemmArgs g{};
  g.BN = R.BN;
  g.order = ORDER_BLOCKS;
  g.hc_store = accumulate ? 0 : 1;
  g.M = n;
  g.N = static_cast<int>(R.rowsB);
  g.K = 2 * R.Kh;
  g.kb_per_split = static_cast<int>((2LL * R.Kh + BK - 1) / BK);
  g.splits = 1;
  g.hc = static_cast<float2*>(out);
  g.hc_batch_stride = static_cast<long long>(n_out) * n;
  g.hc_ld = n;
  g.nb = n_out;
  g.err = err;
  return launch<EPI_ADD_HC>(Operand{a_hi, a_lo, n, R.ldA, static_cast<long long>(n) * R.ldA},
                            Operand{b_hi, b_lo, R.rowsB, R.ldB, R.rowsB * R.ldB}, 2 * R.Kh, nk, g, st);
}

int rotate_tc(const void* C, int n_in, int nk, int n, const void* M, int n_out, void* out, bool accumulate,
              void* ws, size_t ws_bytes, int* err, cudaStream_t st) {
  if (nk < 0 || n_in < 0 || n_out < 0 || n < 1) return fail(QGB_ERR_INVALID, "bad rotate_tc sizes");
  if (nk == 0 || n_out == 0) return QGB_OK;
  if (n_in == 0) {
    if (!accumulate) QGB_CUDA_CHECK(cudaMemsetAsync(out, 0, static_cast<size_t>(nk) * n_out * n * 8, st));
    return QGB_OK;
  }
  if (nk > 65535) return fail(QGB_ERR_UNSUPPORTED, "rotate_tc: nk above 65535");
  if (!C || !M || !out || !ws || !err) return fail(QGB_ERR_INVALID, "NULL pointer in rotate_tc");
  if (C == out) return fail(QGB_ERR_INVALID, "C and out must not alias");
  if (ws_bytes < rotate_tc_workspace_bytes(nk, n_in, n_out, n))
    return fail(QGB_ERR_WORKSPACE, "rotate_tc workspace too small");
  const RotTcLayout R = rot_tc_layout(nk, n_in, n_out, n);
  unsigned char* w = static_cast<unsigned char*>(ws);
  return rotate_tc_impl(R, C, n_in, nk, n, M, n_out, out, accumulate, w, err, st);
}

int nonlocal_tc(const void* split, const void* D, int n_atoms, int pa, const void* C, void* HC, void* projT,
                int nk, int nb, int n_tot, void* ws, size_t ws_bytes, int* err, cudaStream_t st) {
  return nonlocal_tc_phase(split, D, n_atoms, pa, C, HC, projT, nk, nb, n_tot, ws, ws_bytes, err, 3, st, nullptr);
}

// Test aid for the bounded waits: one CTA of the GEMM whose producer issues
// no copies, so the MMA issuer's first wait runs out after `timeout_ns` and
// records error 3; no copy or MMA is in flight when it returns.  Operands
// are valid (M = 128, N = 64, K = 64 bf16 rows of `ab`, 128 + 64 rows of 64
// elements), `ws` >= 128 * 64 floats.
int tc_wait_timeout_test(const void* ab, float* ws, int* err, unsigned long long timeout_ns, cudaStream_t st) {
  if (!ab || !ws || !err || timeout_ns == 0) return fail(QGB_ERR_INVALID, "tc_wait_timeout_test arguments");
  const auto* a = static_cast<const __nv_bfloat16*>(ab);
  const auto* b = a + 128 * 64;
  GemmArgs g{};
  g.M = 128;
  g.N = 64;
  g.K = 64;
  g.kb_per_split = 1;
  g.splits = 1;
  g.partial = ws;
  g.part_ld = 64;
  g.part_rows = 128;
  g.err = err;
  g.timeout_ns = timeout_ns;
  g.skip_loads = 1;
  g.BN = 64;
  return launch<EPI_PARTIAL>(Operand{a, a, 128, 64, 128 * 64}, Operand{b, b, 64, 64, 64 * 64}, 64, 1, g, st);
}

// Plain TN GEMM for tests: D (FP32 [M][N]) = A_hi B_hi^T + A_hi B_lo^T + A_lo B_hi^T.
int tc_gemm_test(const void* a_hi, const void* a_lo, const void* b_hi, const void* b_lo, int M, int N, int K,
                 int lda, int ldb, float* D, int* err, void* ws, size_t ws_bytes, cudaStream_t st) {
  if (M < 1 || N < 1 || K < 1 || N > 64 || lda % 8 || ldb % 8)
    return fail(QGB_ERR_INVALID, "tc_gemm_test: need N <= 64 and lda, ldb multiples of 8");
  const long long m_rows = (M + BM - 1) / BM * BM;
  if (ws_bytes < static_cast<size_t>(m_rows * 64 * 4)) return fail(QGB_ERR_WORKSPACE, "tc_gemm_test workspace");
  GemmArgs g{};
  g.M = M;
  g.N = N;
  g.K = K;
  g.kb_per_split = (K + BK - 1) / BK;
  g.splits = 1;
  g.partial = static_cast<float*>(ws);
  g.part_ld = 64;
  g.part_rows = m_rows;
  g.err = err;
  g.BN = 64;
  int rc = launch<EPI_PARTIAL>(Operand{a_hi, a_lo, M, lda, static_cast<long long>(M) * lda},
                               Operand{b_hi, b_lo, N, ldb, static_cast<long long>(N) * ldb}, K, 1, g, st);
  if (rc) return rc;
  QGB_CUDA_CHECK(cudaMemcpy2DAsync(D, N * sizeof(float), ws, 64 * sizeof(float), N * sizeof(float), M,
                                   cudaMemcpyDeviceToDevice, st));
  return QGB_OK;
}

}  // namespace qgb
