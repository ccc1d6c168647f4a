// FP64 band-space products on the tensor cores, with 55-bit operands (see Accuracy).
//
// GB300's FP64 pipe runs 2 multiply-adds a cycle on each SM (1.2 TFLOP/s per
// GPU), so the FP64 overlaps, projections and rotations were bound by it at
// any tiling.  Here they follow the error-free splitting of Ozaki, Ogita,
// Oishi and Rump (Numer. Algorithms 59, 2012), with integer slices:
//
//   a row x of an operand, scaled by its largest exponent, is the integer
//   X = round(x 2^54 / 2^floor(log2 max|x|)), |X| < 2^55, written with 7
//   signed base-256 digits, X = sum_p d_p 2^(8 (7 - p)), |d_p| <= 128, which
//   bf16 holds exactly;
//   a product of two such rows is sum_{p,q} 2^(-8 (p + q)) sum_k a_p[k] b_q[k],
//   and the tensor cores add the integers a_p b_q (|.| <= 2^14) of one
//   p + q = d into one FP32 accumulator without rounding while the sum stays
//   below 2^24: 128 terms of at most 7 pairs, 128 * 7 * 2^14 < 2^24;
//   after every 128 terms the 8 accumulators d = 2..9 are added into two
//   64-bit integers per output, again without rounding.
// The pairs with p + q > 9 are left out: together they are below 2^-59 max|x| max|y|
// a term.  The sums of a K range are rounded to FP64 once, and so is the result.
// The order is fixed: equal calls give equal bits.
//
// Accuracy.  A real product of rows a and b is off by at most
//   2^-54 (max|a| sum|b| + sum|a| max|b|) + 2^-59 K max|a| max|b|,
// where FP64 multiply-adds are off by at most (K + 1) 2^-53 sum|a||b|: at or below
// them relative to max|a| max|b| (measured 0.1 times their error on rows of even
// size), and above them relative to sum|a||b| as far as the entries that meet are
// below the largest.  max and sum are over
//   an overlap: g, within one K range, for rows a = X_i and b = Y_j.  Rows that
//     decay in opposite directions over the basis are fine (2^-58 sum|a||b|), rows that
//     do so within a range are not (decay 1e-13 and back every 128 g: 7e-7);
//   a rotation: the bands i, for a = X_i(g) / s_i and b = s_i W(i, j), s_i the power of
//     two of band i's largest entry (k_oz_band_exp): off by 2^-54 of the output
//     band's terms at their largest, whatever the norms of the bands.
// The multiply-add forms keep to sum|a||b| and are what a call without the larger
// workspace runs.  Falling back to them where sum|a||b| is small was not done: bands
// of a supercell that fold from different k have disjoint entries, and would all.
//
// Rows with a NaN or an infinity are marked by their scale and their outputs
// computed by plain FP64 multiply-adds.
//
// Measured (us, 352 x 176 over 37073, one k; FP64 multiply-adds before): overlap
// 25690 -> 812, rotation 16805 -> 787.  The GEMMs take 575 and 563 of these, a
// chunk of 128 K (34 pairs: 4.6 us at the tensor cores' peak) in 7.7 us: the copies
// of 14 digit tiles for 34 products bind (tensor pipe 45% active in captures of one
// panel); the slicing kernels run at 4.5 TB/s.
//
// Kernels (for each complex product as real ones: rows Re and Im stacked, or
// folded along K where only the real part is kept):
//   k_oz_slice_rows   A and B of an overlap: K-contiguous rows -> digits
//   k_oz_band_exp     a rotation's bands: their scales
//   k_oz_slice_cols   X of a rotation (contracted over its rows): transposed
//   k_oz_slice_mat    W of a rotation
//   k_oz_gemm         tcgen05 GEMM over digits, 128 x 64 outputs per CTA
//   k_oz_reduce       split sums of an overlap -> complex outputs
#include <cuda_bf16.h>

#include <algorithm>

#include "bandgemm.cuh"
#include "tcgen05.cuh"

namespace qgb {
namespace oz {

using namespace tc;

constexpr int kSms = 152;
constexpr int S = 7;              // digits per value
constexpr int ND = 8;             // digit-pair sums kept: p + q = 2 .. 9
constexpr int BM = 128;           // rows of A per CTA
constexpr int BN = 64;            // rows of B per CTA: ND * BN = 512 TMEM columns
constexpr int BK = 64;            // K per block of shared-memory tiles (128 B rows)
constexpr int CHUNK = 128;        // K per exact FP32 accumulation
constexpr int CHUNK_BLOCKS = CHUNK / BK;
constexpr int A_BYTES = BM * BK * 2;          // one digit of A: 16 KB
constexpr int B_BYTES = BN * BK * 2;          // one digit of B: 8 KB
constexpr int B_LO = 4;                       // digits 1..4 of B are double-buffered, 5..7 are not
constexpr int BLO_OFF = S * A_BYTES;
constexpr int BHI_OFF = BLO_OFF + 2 * B_LO * B_BYTES;
constexpr int BAR_OFF = BHI_OFF + (S - B_LO) * B_BYTES;
constexpr int EPI_WARPS = 16;      // (4 lane quarters) x (4 column quarters)
constexpr int WC = BN / (EPI_WARPS / 4);  // columns per epilogue warp
constexpr int SUMS_LD = 33;        // epilogue corner per warp: 2 columns x 32 rows (+ 1) of two int64
constexpr int SUMS_OFF = BAR_OFF + 512;
constexpr int SMEM_BYTES = SUMS_OFF + EPI_WARPS * 2 * SUMS_LD * 16 + 1024;
static_assert((2 * S + 6 + 2 * ND + 1) * 8 + 16 <= 512 && SMEM_BYTES <= 227 * 1024, "shared memory layout");
constexpr int kThreads = (EPI_WARPS + 2) * 32;
constexpr int kNonFinite = 0x7FF;  // exponent mark of an overlap's rows with a NaN or an infinity
constexpr int kBadRow = 1 << 16;   // the same mark of a rotation's rows, whose exponents go up to 2 * 2046
constexpr int kNoEntry = -4096;    // exponent of a rotation's row without a nonzero entry

enum Epi { EPI_PARTIAL = 0, EPI_ROTATE = 1 };

struct GemmArgs {
  int units, n_tiles, m_tiles;
  int chunks;              // K chunks of 128 per split
  int splits;
  const int* ea;           // exponent of A's complex rows: [batch][split][a_rows]
  const int* eb;           // exponent of B's complex rows: [batch][split][b_rows]
  int a_rows, b_rows;      // complex rows; real row r belongs to r % a_rows / b_rows (EPI_PARTIAL)
  int M, N;                // real rows of A and B
  int* err;
  // EPI_PARTIAL: FP64 [split][batch][M][N], this panel's from split0 on; add: to the earlier panels' sums
  double* partial;
  int split0, add, nbatch;
  // EPI_ROTATE: rows g0 + row < G; band j of column c (see k_oz_slice_mat)
  double2* out;
  long long out_batch;
  int ldo, g0, G, Nout, accumulate;
  const double2* X;        // operands, for rows marked non-finite
  const double2* W;
  long long x_batch, w_batch;
  int ldx, wi, wj, Kin;
};

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

// (hi 2^32 + lo) 2^e, rounded once to nearest-even.
__device__ __forceinline__ double to_double(long long hi, long long lo, int e) {
  long long h = hi + (lo >> 32);
  unsigned l = static_cast<unsigned>(lo);
  const bool neg = h < 0;
  if (neg) {
    h = ~h + (l == 0u ? 1 : 0);
    l = 0u - l;
  }
  unsigned long long top, uh = static_cast<unsigned long long>(h);
  unsigned sticky = 0;
  int msb;
  if (uh != 0) {
    const int z = __clzll(static_cast<long long>(uh));
    top = uh << z;
    if (z > 0) top |= (static_cast<unsigned long long>(l) << 32) >> (64 - z);
    sticky = z < 32 ? (l << z) : 0u;
    msb = 95 - z;
  } else {
    if (l == 0u) return 0.0;
    const int z = __clz(static_cast<int>(l));
    top = static_cast<unsigned long long>(l) << (32 + z);
    msb = 31 - z;
  }
  unsigned long long m = top >> 11;
  const unsigned rem = static_cast<unsigned>(top) & 0x7FFu;
  if (rem > 0x400u || (rem == 0x400u && (sticky != 0u || (m & 1ull)))) ++m;  // m in [2^52, 2^53]
  const int E = msb + e + 1023;
  double v;
  if (E >= 1 && E <= 2045)
    v = __longlong_as_double(static_cast<long long>((static_cast<unsigned long long>(E - 1) << 52) + m));
  else
    v = ldexp(static_cast<double>(m), msb - 52 + e);
  return neg ? -v : v;
}

__device__ __forceinline__ void mad_wide(long long& acc, int v, int w) {
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc) : "r"(v), "r"(w));
}

// One persistent CTA per SM; a unit is a 128 x 64 tile of one split of one
// batch entry, N tiles fastest (neighbouring CTAs read the same A digits from
// L2).  The epilogue holds a finished unit's sums in registers, so their
// conversion overlaps with the next unit's first chunk.
//
// The digit tiles of a K = 64 block fill shared memory, so there is no second
// block: each tile is refilled as soon as its last MMA of the block is done.
// Accumulator d = p + q sits at TMEM columns (d - 2) * BN; one MMA takes a
// digit of A against up to four digits of B (adjacent rows in shared memory,
// adjacent sums in TMEM).  Per block, in this order:
//   the 10 pairs of d <= 5:   p = 1: q = 1..4,  2: 1..3,  3: 1..2,  4: 1
//   the 24 pairs of d >= 6:   p = 1: q = 5..7,  2: 4..7,  3: 3..6,  4: 2..5,
//                             5: 1..4,  6: 1..3,  7: 1..2
// so that tiles are released evenly (A's from p = 1 to 7, B's digits 5..7 after
// p = 4; only digits 1..4 of B are needed from start to end and get a second
// buffer), and that sums are complete in the order d = 2..9, the first four
// early: the epilogue reads them while the MMAs go on with the others.
template <int EPI>
__global__ void __launch_bounds__(kThreads, 1)
    k_oz_gemm(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB, const GemmArgs args) {
  extern __shared__ __align__(1024) unsigned char oz_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(oz_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_a = reinterpret_cast<uint64_t*>(smem + BAR_OFF);  // [S], one per digit of A
  uint64_t* empty_a = full_a + S;
  uint64_t* full_lo = empty_a + S;       // [2]
  uint64_t* empty_lo = full_lo + 2;
  uint64_t* full_hi = empty_lo + 2;
  uint64_t* empty_hi = full_hi + 1;
  uint64_t* acc_full = empty_hi + 1;     // [ND] a digit-pair sum is complete in TMEM
  uint64_t* acc_empty = acc_full + ND;   // [ND] the epilogue has read it
  uint64_t* done = acc_empty + ND;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nblk = args.chunks * CHUNK_BLOCKS;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * S + 6; ++i) mbar_init(full_a + i, 1);
    for (int d = 0; d < ND; ++d) {
      mbar_init(&acc_full[d], 1);
      mbar_init(&acc_empty[d], EPI_WARPS);
    }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == EPI_WARPS + 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (threadIdx.x == EPI_WARPS * 32) {
    // ---------------- TMA producer ----------------
    int blk = 0;                    // blocks so far, over all units
    int na = 0, nlo = 0, nhi = 0;   // tiles issued
    bool live = true;
    for (int u = blockIdx.x; u < args.units && live; u += gridDim.x) {
      const Unit t = unit_of(args, u);
      for (int kb = 0; kb < nblk && live; ++kb, ++blk) {
        const int k = (t.split * nblk + kb) * BK;
        const uint32_t prev = (blk - 1) & 1;  // parity of the previous block's release
        const int sl = blk & 1;
        if (blk > 1 && !mbar_wait(&empty_lo[sl], ((blk >> 1) - 1) & 1, args.err, 1, kTimeoutNs)) {
          live = false;
          break;
        }
        mbar_arrive_expect_tx(&full_lo[sl], B_LO * B_BYTES);
        for (int q = 0; q < B_LO; ++q)
          tma_load_4d(smem + BLO_OFF + (sl * B_LO + q) * B_BYTES, &mB, &full_lo[sl], k, t.n_tile * BN, q, t.batch);
        ++nlo;
        for (int p = 0; p < S; ++p) {
          if (p == 4) {  // digits 5..7 of B, needed after the first four of A
            if (blk > 0 && !mbar_wait(empty_hi, prev, args.err, 1, kTimeoutNs)) {
              live = false;
              break;
            }
            mbar_arrive_expect_tx(full_hi, (S - B_LO) * B_BYTES);
            for (int q = B_LO; q < S; ++q)
              tma_load_4d(smem + BHI_OFF + (q - B_LO) * B_BYTES, &mB, full_hi, k, t.n_tile * BN, q, t.batch);
            ++nhi;
          }
          if (blk > 0 && !mbar_wait(&empty_a[p], prev, args.err, 1, kTimeoutNs)) {
            live = false;
            break;
          }
          mbar_arrive_expect_tx(&full_a[p], A_BYTES);
          tma_load_4d(smem + p * A_BYTES, &mA, &full_a[p], k, t.m_tile * BM, p, t.batch);
          ++na;
        }
      }
    }
    // Every copy issued lands before the CTA exits, also after an error: the
    // last one into each tile (the earlier ones were waited for through the
    // release of their tiles).
    for (int p = 0; p < S; ++p)
      if (na > p) mbar_drain(&full_a[p], ((na - 1 - p) / S) & 1, args.err, 2);
    for (int i = 0; i < 2; ++i)
      if (nlo > i) mbar_drain(&full_lo[i], ((nlo - 1 - i) / 2) & 1, args.err, 2);
    if (nhi > 0) mbar_drain(full_hi, (nhi - 1) & 1, args.err, 2);
  } else if (threadIdx.x == (EPI_WARPS + 1) * 32) {
    // ---------------- MMA issuer ----------------
    const uint32_t base = smem_u32(smem);
    const uint64_t da0 = desc_kmajor_sw128(base), dhi = desc_kmajor_sw128(base + BHI_OFF);
    // Digit p of A against digits q .. q + w - 1 of B (all below or above B_LO).
    auto mma = [&](int p, int q, int w, uint64_t dlo, bool fresh) {
      const uint64_t a = da0 + static_cast<uint64_t>((p - 1) * (A_BYTES / 16));
      const uint64_t b = q <= B_LO ? dlo + static_cast<uint64_t>((q - 1) * (B_BYTES / 16))
                                   : dhi + static_cast<uint64_t>((q - 1 - B_LO) * (B_BYTES / 16));
      const uint32_t idesc = idesc_bf16_f32(BM, BN) + (static_cast<uint32_t>((w - 1) * (BN >> 3)) << 17);
#pragma unroll
      for (int k = 0; k < BK / 16; ++k)
        umma_bf16(tmem + (p + q - 2) * BN, a + 2 * k, b + 2 * k, idesc, (fresh && k == 0) ? 0u : 1u);
    };
    bool live = true;
    auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
      if (live) live = mbar_wait(bar, parity, args.err, code, kTimeoutNs);
      return live;
    };
    int blk = 0, c = 0;  // blocks and chunks so far, over all units
    for (int u = blockIdx.x; u < args.units && live; u += gridDim.x) {
      for (int uc = 0; uc < args.chunks && live; ++uc, ++c) {
        for (int cb = 0; cb < CHUNK_BLOCKS && live; ++cb, ++blk) {
          const bool first = cb == 0, last = cb == CHUNK_BLOCKS - 1;
          const uint32_t ph = blk & 1, acc_ph = (c - 1) & 1;
          const uint64_t dlo = desc_kmajor_sw128(base + BLO_OFF + (blk & 1) * (B_LO * B_BYTES));
          wait(&full_lo[blk & 1], (blk >> 1) & 1, 3);
          if (first && c > 0)
            for (int d = 0; d < 4; ++d) wait(&acc_empty[d], acc_ph, 4);
          for (int p = 1; p <= 4; ++p) {
            if (!wait(&full_a[p - 1], ph, 3)) break;
            tc_fence_after();
            mma(p, 1, 5 - p, dlo, first && p == 1);
          }
          if (last)
            for (int d = 0; d < 4; ++d) umma_commit(&acc_full[d]);
          wait(full_hi, ph, 3);
          if (first && c > 0)
            for (int d = 4; d < ND; ++d) wait(&acc_empty[d], acc_ph, 4);
          if (!live) break;
          tc_fence_after();
          mma(1, 5, 3, dlo, first);
          umma_commit(&empty_a[0]);
          mma(2, 4, 1, dlo, false);
          if (first) {
            mma(2, 7, 1, dlo, true);  // the first of d = 9
            mma(2, 5, 2, dlo, false);
          } else {
            mma(2, 5, 3, dlo, false);
          }
          umma_commit(&empty_a[1]);
          mma(3, 3, 2, dlo, false);
          mma(3, 5, 2, dlo, false);
          umma_commit(&empty_a[2]);
          mma(4, 2, 3, dlo, false);
          mma(4, 5, 1, dlo, false);
          umma_commit(&empty_a[3]);
          umma_commit(empty_hi);
          for (int p = 5; p <= S; ++p) {
            if (!wait(&full_a[p - 1], ph, 3)) break;
            tc_fence_after();
            mma(p, 1, 9 - p, dlo, false);
            umma_commit(&empty_a[p - 1]);
            if (last) umma_commit(&acc_full[p - 1]);  // d = p + 1 is complete
          }
          if (last) umma_commit(&acc_full[ND - 1]);
          umma_commit(&empty_lo[blk & 1]);
        }
      }
    }
    umma_commit(done);
  } else if (warp < EPI_WARPS) {
    // ---------------- Epilogue: warps (lane quarter, column quarter) ----------------
    const int quarter = warp >> 2, row0 = (warp & 3) * 32 + lane;
    const uint32_t trow = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + quarter * WC;
    longlong2* sums = reinterpret_cast<longlong2*>(smem + SUMS_OFF) + warp * (2 * SUMS_LD);
    const double nan = __longlong_as_double(0x7FF8000000000000ll);
    bool ok = true;
    int c = 0;
#pragma unroll 1
    for (int u = blockIdx.x; u < args.units; u += gridDim.x) {
      const Unit t = unit_of(args, u);
      long long hi[WC], lo[WC];
#pragma unroll
      for (int i = 0; i < WC; ++i) hi[i] = lo[i] = 0;
#pragma unroll 1
      for (int uc = 0; uc < args.chunks && ok; ++uc, ++c) {
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          if (ok) ok = mbar_wait(&acc_full[d], c & 1, args.err, 5, kTimeoutNs);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          const int w = 1 << (8 * (3 - (d & 3)));
          float v[WC];
          tmem_ld16(trow + d * BN, v);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[d]);
#pragma unroll
          for (int i = 0; i < WC; ++i) mad_wide(d < 4 ? hi[i] : lo[i], __float2int_rn(v[i]), w);
        }
      }
      ok = __all_sync(0xffffffffu, ok && *reinterpret_cast<volatile int*>(args.err) == 0);
      // The sums go through this warp's corner of shared memory 2 columns at a
      // time, [column][row], so that the conversion is a short rolled loop:
      // unrolled over the registers it is some 30 KB of code, whose fetch alone
      // took longer than a chunk.
#pragma unroll 1
      for (int grp = 0; grp < WC / 2; ++grp) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < WC; ++i) {  // EPI_ROTATE: a band's real and imaginary column
          const int own = EPI == EPI_PARTIAL ? i / 2 : i & 7;
          const int slot = EPI == EPI_PARTIAL ? i % 2 : i / 8;
          if (own == grp) sums[slot * SUMS_LD + lane] = make_longlong2(hi[i], lo[i]);
        }
        __syncwarp();
        if (EPI == EPI_PARTIAL) {
          const int* ea = args.ea + (static_cast<long long>(t.batch) * args.splits + t.split) * args.a_rows;
          const int* eb = args.eb + (static_cast<long long>(t.batch) * args.splits + t.split) * args.b_rows;
          double* out = args.partial +
                        (static_cast<long long>(args.split0 + t.split) * args.nbatch + t.batch) * args.M * args.N;
          const int cc = lane & 1, col = t.n_tile * BN + quarter * WC + grp * 2 + cc;
          const int ec = col < args.N ? eb[col % args.b_rows] - 2 * 1021 - 72 : 0;
#pragma unroll
          for (int r = lane >> 1; r < 32; r += 16) {
            const int row = t.m_tile * BM + (warp & 3) * 32 + r;
            if (row < args.M && col < args.N) {
              const longlong2 v = sums[cc * SUMS_LD + r];
              double* o = out + static_cast<long long>(row) * args.N + col;
              const double d = ok ? to_double(v.x, v.y, ec + ea[row % args.a_rows]) : nan;
              *o = args.add ? *o + d : d;
            }
          }
        } else {
          const int row = t.m_tile * BM + row0, g = args.g0 + row;
          const int* ew = args.eb + static_cast<long long>(t.batch) * args.b_rows;
          const int j = t.n_tile * (BN / 2) + quarter * (WC / 2) + grp;
          if (row < args.M && g < args.G && j < args.Nout) {
            const int eg = args.ea[static_cast<long long>(t.batch) * args.a_rows + row];
            double2 v;
            if (!ok) {
              v = make_double2(nan, nan);
            } else if (eg == kBadRow || ew[j] == kBadRow) {
              const double2* x = args.X + t.batch * args.x_batch + g;
              const double2* wp = args.W + t.batch * args.w_batch + static_cast<long long>(j) * args.wj;
              v = make_double2(0.0, 0.0);
#pragma unroll 1
              for (int k = 0; k < args.Kin; ++k) {
                const double2 a = wp[static_cast<long long>(k) * args.wi];
                const double2 b = x[static_cast<long long>(k) * args.ldx];
                v.x = fma(a.x, b.x, v.x);
                v.x = fma(-a.y, b.y, v.x);
                v.y = fma(a.x, b.y, v.y);
                v.y = fma(a.y, b.x, v.y);
              }
            } else {
              const int e = eg + ew[j] - 2 * 1021 - 72;
              const longlong2 re = sums[lane], im = sums[SUMS_LD + lane];
              v = make_double2(to_double(re.x, re.y, e), to_double(im.x, im.y, e));
            }
            double2* o = args.out + t.batch * args.out_batch + static_cast<long long>(j) * args.ldo + g;
            if (args.accumulate) {
              v.x += o->x;
              v.y += o->y;
            }
            *o = v;
          }
        }
      }
    }
    // Every MMA has completed before TMEM is freed, also when one stopped early.
    mbar_drain(done, 0, args.err, 6);
    tc_fence_before();
  }
  __syncwarp();
  __syncthreads();
  if (warp == EPI_WARPS + 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------
// Slicing
// ---------------------------------------------------------------------------

__device__ __forceinline__ int exp_field(double x) { return (__double2hiint(x) >> 20) & 0x7FF; }

// Largest exponent field of a complex number, 1 if that is subnormal and 0 only
// for zero.  By integers: comparing doubles would take the FP64 pipe.
__device__ __forceinline__ int scale_field(double2 v) {
  const unsigned hi = max(static_cast<unsigned>(__double2hiint(v.x)) & 0x7FFFFFFFu,
                          static_cast<unsigned>(__double2hiint(v.y)) & 0x7FFFFFFFu);
  const unsigned any = hi | static_cast<unsigned>(__double2loint(v.x)) | static_cast<unsigned>(__double2loint(v.y));
  return static_cast<int>(max(hi >> 20, min(any, 1u)));
}

// round(x 2^(54 - (emax - 1023))) for |x| of exponent field at most emax: below
// 2^55 in magnitude, exact for the values within 2 bits of the largest.  Zero
// gives zero for any emax.
__device__ __forceinline__ long long fixed_point(double x, int emax) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(x));
  int E = static_cast<int>(b >> 52) & 0x7FF;
  unsigned long long m = b & 0x000FFFFFFFFFFFFFull;
  if (E > 0) m |= 0x0010000000000000ull; else E = 1;
  const int sh = emax - E - 2;
  const long long X = static_cast<long long>(sh <= 0 ? m << (-sh & 3) : (sh > 54 ? 0ull : (m + (1ull << (sh - 1))) >> sh));
  return static_cast<long long>(b) < 0 ? -X : X;
}

// The 7 base-256 digits of a fixed_point() value, biased by 128 below the top
// one: digit 7 in byte 0 .. digit 2 in byte 5, the signed digit 1 above.
__device__ __forceinline__ unsigned long long biased_digits(double x, int emax) {
  return static_cast<unsigned long long>(fixed_point(x, emax)) + 0x0000808080808080ull;
}

// Digit p (1 = most significant) of biased_digits() as a float.
template <int P> __device__ __forceinline__ float digit(unsigned long long X) {
  if (P == 1) return static_cast<float>(static_cast<int>(static_cast<long long>(X) >> 48));
  const unsigned word = P <= 3 ? static_cast<unsigned>(X >> 32) : static_cast<unsigned>(X);
  // bytes of X: digit 7 = byte 0 .. digit 4 = byte 3, digit 3 = byte 4, digit 2 = byte 5
  const unsigned sel = P <= 3 ? (3 - P) : (7 - P);
  return __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7650u | sel)) - 8388736.0f;  // 2^23 + 128
}

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {  // exact: |.| <= 128
  return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632u);
}

// Store the 7 digits of 4 consecutive K entries (8 B each) at dst + (p - 1) * step.
template <int P = 1>
__device__ __forceinline__ void store_digits4(__nv_bfloat16* dst, long long step, const unsigned long long (&X)[4]) {
  *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(digit<P>(X[0]), digit<P>(X[1])),
                                              pack_bf16(digit<P>(X[2]), digit<P>(X[3])));
  if constexpr (P < S) store_digits4<P + 1>(dst + step, step, X);
}

template <int THREADS> __device__ __forceinline__ int block_max(int v, int* red) {
  v = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  int m = red[0];
#pragma unroll
  for (int w = 1; w < THREADS / 32; ++w) m = max(m, red[w]);
  return m;
}

struct SliceArgs {
  const double2* src;      // [batch][rows][ld_src], K contiguous
  long long batch_stride;
  int ld_src, rows, K;
  int g0, Lg;              // this panel's first g, and g per split (a multiple of 64)
  int fold;                // 0: rows Re then Im stacked; 1: [Re | Im] of a split along K
  const double* weight;
  __nv_bfloat16* digits;   // [batch][7][real rows][ld]
  int ld;
  int* e;                  // [batch][split][rows]
};

// One CTA per (row, split, batch; A or B by blockIdx.z's parity): the row's
// range is read twice, the second time from L2, and written as digits.
// Bound by the 14 B per value it writes and the 16 B per complex it reads.
__global__ void __launch_bounds__(256) k_oz_slice_rows(const SliceArgs a0, const SliceArgs a1, int* err) {
  __shared__ int red[8];
  const SliceArgs& a = (blockIdx.z & 1) ? a1 : a0;
  const int row = blockIdx.x, split = blockIdx.y, batch = blockIdx.z >> 1;
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 0 && err) *err = 0;
  if (row >= a.rows) return;
  const double2* src = a.src + batch * a.batch_stride + static_cast<long long>(row) * a.ld_src;
  const int gb = a.g0 + split * a.Lg, n = max(0, min(a.Lg, a.K - gb));
  int em = 1;
  for (int i = threadIdx.x; i < n; i += 256) {
    double2 v = src[gb + i];
    if (a.weight) {
      const double w = a.weight[gb + i];
      v.x *= w;
      v.y *= w;
    }
    em = max(em, max(exp_field(v.x), exp_field(v.y)));
  }
  em = block_max<256>(em, red);
  if (threadIdx.x == 0) a.e[(static_cast<long long>(batch) * gridDim.y + split) * a.rows + row] = em;
  const int real_rows = a.fold ? a.rows : 2 * a.rows;
  const long long step = static_cast<long long>(real_rows) * a.ld;
  __nv_bfloat16* base = a.digits + batch * S * step;
  __nv_bfloat16* dre = base + static_cast<long long>(row) * a.ld + static_cast<long long>(split) * a.Lg * (a.fold ? 2 : 1);
  __nv_bfloat16* dim = a.fold ? dre + a.Lg : dre + static_cast<long long>(a.rows) * a.ld;
  for (int i = 4 * threadIdx.x; i < a.Lg; i += 1024) {
    unsigned long long re[4], im[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      double2 v = make_double2(0.0, 0.0);
      if (i + t < n && em != kNonFinite) {
        v = src[gb + i + t];
        if (a.weight) {
          const double w = a.weight[gb + i + t];
          v.x *= w;
          v.y *= w;
        }
      }
      re[t] = biased_digits(v.x, em);
      im[t] = biased_digits(v.y, em);
    }
    store_digits4(dre + i, step, re);
    store_digits4(dim + i, step, im);
  }
}

// The contracted index of a rotation is the band, and bands may differ by any
// factor (unnormalised ones, filtered ones, projectors of a back-projection): a
// common exponent would cut the small ones off.  So band i is scaled by its own
// power of two, s_i = 2^(e_i - 1023) with e_i the largest exponent field of its
// finite entries, and the product is of X_i / s_i and s_i W(i, j).  Both are
// shifts of the exponents the slices are taken at, exact, and cancel in the
// result.  A CTA takes kExpRange g of a band, all loads in flight: 39 us for
// 352 x 37073, of which the read takes 31 (ranges four times as long, in a loop: 44).
constexpr int kExpRange = 2048;
__global__ void __launch_bounds__(256) k_oz_band_exp(const double2* __restrict__ X, long long x_batch, int ldx, int Kin,
                                                     int G, int* __restrict__ e) {
  __shared__ int red[8];
  const int i = blockIdx.x, batch = blockIdx.z, g0 = blockIdx.y * kExpRange + threadIdx.x;
  const double2* x = X + batch * x_batch + static_cast<long long>(i) * ldx;
  double2 v[kExpRange / 256];
#pragma unroll
  for (int u = 0; u < kExpRange / 256; ++u) {
    const int g = g0 + 256 * u;
    v[u] = g < G ? x[g] : make_double2(0.0, 0.0);
  }
  int em = 0;
#pragma unroll
  for (int u = 0; u < kExpRange / 256; ++u) {
    // (an entry with a non-finite part counts by neither part: its row is marked)
    const int f = scale_field(v[u]);
    em = max(em, f == kNonFinite ? 0 : f);
  }
  em = block_max<256>(em, red);
  if (threadIdx.x == 0) atomicMax(e + static_cast<long long>(batch) * Kin + i, em);  // zero before the launch
}

// X [batch][Kin][ldx] of a rotation -> digits [batch][7][rows][ld], row = g,
// K = [Re X_i, i < Kh | Im X_i], one exponent per g, of the scaled bands.  One CTA
// per 32 g: pass 1 takes the exponents, pass 2 transposes 32 x 32 tiles through
// shared memory.
__global__ void __launch_bounds__(256) k_oz_slice_cols(const double2* __restrict__ X, long long x_batch, int ldx,
                                                       int Kin, int Kh, int g0, int G, int rows,
                                                       __nv_bfloat16* __restrict__ digits, int ld,
                                                       const int* __restrict__ eband, int* __restrict__ e, int* err) {
  __shared__ double2 tile[32][33];
  __shared__ int red[8][32], tile_e[32];
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && err) *err = 0;
  const int batch = blockIdx.y, r0 = blockIdx.x * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int g = g0 + r0 + tx;
  const bool gin = r0 + tx < rows && g < G;
  const double2* x = X + batch * x_batch + g;
  const int* eb = eband + static_cast<long long>(batch) * Kin;
  int em = kNoEntry;
  if (gin)
#pragma unroll 4
    for (int i = ty; i < Kin; i += 8) {
      const int f = scale_field(x[static_cast<long long>(i) * ldx]);
      em = max(em, f > 0 ? f - eb[i] : kNoEntry);  // above 0 only where f is kNonFinite
    }
  red[ty][tx] = em;
  __syncthreads();
  if (ty == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) em = max(em, red[w][tx]);
    if (em > 0) em = kBadRow;
    red[0][tx] = em;
    if (gin) e[static_cast<long long>(batch) * rows + r0 + tx] = em;
  }
  __syncthreads();
  const long long step = static_cast<long long>(rows) * ld;
  const int rr = threadIdx.x >> 3, seg = 4 * (threadIdx.x & 7);  // this thread's row and 4 of the 32 i
  const int er = red[0][rr];
  __nv_bfloat16* dst = digits + batch * S * step + static_cast<long long>(r0 + rr) * ld;
  for (int i0 = 0; i0 < Kh; i0 += 32) {
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const int i = i0 + ty + 8 * w;
      tile[ty + 8 * w][tx] = (gin && i < Kin) ? x[static_cast<long long>(i) * ldx] : make_double2(0.0, 0.0);
    }
    if (ty == 0) tile_e[tx] = i0 + tx < Kin ? eb[i0 + tx] : 0;
    __syncthreads();
    if (r0 + rr < rows && i0 + seg < Kh) {
      unsigned long long re[4], im[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        double2 v = tile[seg + t][rr];
        if (er == kBadRow) v = make_double2(0.0, 0.0);
        re[t] = biased_digits(v.x, er + tile_e[seg + t]);
        im[t] = biased_digits(v.y, er + tile_e[seg + t]);
      }
      store_digits4(dst + i0 + seg, step, re);
      store_digits4(dst + Kh + i0 + seg, step, im);
    }
    __syncthreads();
  }
}

// W(i, j) of a rotation -> digits of real rows [batch][7][2 * Npad][ld]: column
// tile t of 64 rows holds bands 32 t + 8 h + jj (h < 4, jj < 8) as rows
// 64 t + 16 h + jj (real output: Re W, -Im W) and + 8 (imaginary: Im W, Re W),
// so one epilogue warp has both parts of its bands.  One CTA per band.  Row i is
// scaled by the power of two of band i of X (a band of zeros adds nothing).
__global__ void __launch_bounds__(128) k_oz_slice_mat(const double2* __restrict__ W, long long w_batch, int wi, int wj,
                                                      int Kin, int Kh, int Nout, int Npad,
                                                      __nv_bfloat16* __restrict__ digits, int ld,
                                                      const int* __restrict__ eband, int* __restrict__ e) {
  __shared__ int red[4];
  const int j = blockIdx.x, batch = blockIdx.y;
  const double2* w = W + batch * w_batch + static_cast<long long>(j) * wj;
  const int* eb = eband + static_cast<long long>(batch) * Kin;
  int em = kNoEntry;
  if (j < Nout)
    for (int i = threadIdx.x; i < Kin; i += 128) {
      const double2 v = w[static_cast<long long>(i) * wi];
      const int f = scale_field(v);
      em = max(em, f == kNonFinite ? kBadRow : (f > 0 && eb[i] > 0 ? f + eb[i] : kNoEntry));
    }
  em = block_max<128>(em, red);
  if (threadIdx.x == 0) e[static_cast<long long>(batch) * Npad + j] = em;
  const long long step = 2ll * Npad * ld;
  const int r = (j / 32) * 64 + ((j >> 3) & 3) * 16 + (j & 7);
  __nv_bfloat16* dre = digits + batch * S * step + static_cast<long long>(r) * ld;
  __nv_bfloat16* dim = dre + 8ll * ld;
  for (int i = 4 * threadIdx.x; i < Kh; i += 512) {
    unsigned long long re[4], im[4], mi[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      double2 v = make_double2(0.0, 0.0);
      const int ei = i + t < Kin ? eb[i + t] : 0;
      if (j < Nout && ei > 0 && em != kBadRow) v = w[static_cast<long long>(i + t) * wi];
      re[t] = biased_digits(v.x, em - ei);
      im[t] = biased_digits(v.y, em - ei);
      mi[t] = biased_digits(-v.y, em - ei);
    }
    store_digits4(dre + i, step, re);
    store_digits4(dre + Kh + i, step, mi);
    store_digits4(dim + i, step, im);
    store_digits4(dim + Kh + i, step, re);
  }
}

// Split sums of an overlap: Re = P[i][j] + P[M + i][N + j], Im = P[i][N + j] -
// P[M + i][j] of the stacked real products (fold: the real part alone).  They
// are added as 64-bit integers in units of 2^-54 of the largest, which costs
// the FP64 pipe nothing and rounds once (two terms below 2^55 of each of at most
// kMaxSplits sets stay below 2^63).  Rows marked non-finite in any split of any
// panel (`exps` of them) are computed here by multiply-adds.
constexpr int kRed = 8;  // threads per output, over the splits
template <int FOLD>
__global__ void __launch_bounds__(256)
    k_oz_reduce(const double* __restrict__ partial, int sets, int panel_splits, int nbatch, int M, int N,
                double2* __restrict__ out, long long out_batch, int oi, int oj, const int* __restrict__ ea, const int* __restrict__ eb,
                int exps, const double2* __restrict__ A, const double2* __restrict__ B, long long a_batch,
                long long b_batch, int lda, int ldb, int K, const double* __restrict__ weight) {
  const long long per = static_cast<long long>(M) * N;
  const int R = FOLD ? 1 : 2;
  const long long per_split = per * R * R * nbatch;
  const int sub = threadIdx.x & (kRed - 1);
  const unsigned lanes = ((1u << kRed) - 1u) << (threadIdx.x & 31 & ~(kRed - 1));
  for (long long x = (blockIdx.x * 256ll + threadIdx.x) / kRed; x < per * nbatch; x += gridDim.x * (256ll / kRed)) {
    const int k = static_cast<int>(x / per);
    const int r = static_cast<int>(x - k * per), i = r / N, j = r - i * N;
    const double* P0 = partial + k * per * R * R + static_cast<long long>(i) * R * N + j;
    const double* P1 = P0 + static_cast<long long>(M) * R * N;  // the Im rows (not folded)
    int er = 1, ei = 1;
    bool bad = false;
    for (int s = sub; s < exps; s += kRed) {
      // The exponents are kept per panel, [batch][panel_splits][rows] each.
      const int pan = s / panel_splits, ps = s - pan * panel_splits;
      const long long es = (static_cast<long long>(pan) * nbatch + k) * panel_splits + ps;
      bad |= ea[es * M + i] == kNonFinite || eb[es * N + j] == kNonFinite;
    }
    for (int s = sub; s < sets; s += kRed) {
      er = max(er, exp_field(P0[s * per_split]));
      if (!FOLD) {
        er = max(er, exp_field(P1[s * per_split + N]));
        ei = max(ei, max(exp_field(P0[s * per_split + N]), exp_field(P1[s * per_split])));
      }
    }
    er = __reduce_max_sync(lanes, er);
    ei = __reduce_max_sync(lanes, ei);
    bad = __any_sync(lanes, bad);
    long long sr = 0, si = 0;
    if (!bad && max(er, ei) != kNonFinite) {
      for (int s = sub; s < sets; s += kRed) {
        sr += fixed_point(P0[s * per_split], er);
        if (!FOLD) {
          sr += fixed_point(P1[s * per_split + N], er);
          si += fixed_point(P0[s * per_split + N], ei) - fixed_point(P1[s * per_split], ei);
        }
      }
#pragma unroll
      for (int o = kRed / 2; o > 0; o >>= 1) {
        sr += __shfl_xor_sync(lanes, sr, o);
        if (!FOLD) si += __shfl_xor_sync(lanes, si, o);
      }
    }
    if (sub != 0) continue;
    double re = 0.0, im = 0.0;
    if (bad) {
      const double2* a = A + k * a_batch + static_cast<long long>(i) * lda;
      const double2* b = B + k * b_batch + static_cast<long long>(j) * ldb;
      for (int g = 0; g < K; ++g) {
        const double2 u = a[g];
        double2 v = b[g];
        if (weight) {
          v.x *= weight[g];
          v.y *= weight[g];
        }
        re = fma(u.x, v.x, re);
        re = fma(u.y, v.y, re);
        im = fma(u.x, v.y, im);
        im = fma(-u.y, v.x, im);
      }
    } else if (max(er, ei) == kNonFinite) {  // a product overflowed, or a pipeline wait ran out
      for (int s = 0; s < sets; ++s) {
        re += FOLD ? P0[s * per_split] : P0[s * per_split] + P1[s * per_split + N];
        if (!FOLD) im += P0[s * per_split + N] - P1[s * per_split];
      }
    } else {
      re = to_double(sr >> 32, sr & 0xFFFFFFFFll, er - 1077);
      if (!FOLD) im = to_double(si >> 32, si & 0xFFFFFFFFll, ei - 1077);
    }
    out[k * out_batch + static_cast<long long>(i) * oi + static_cast<long long>(j) * oj] =
        make_double2(re, FOLD ? 0.0 : im);
  }
}

// ---------------------------------------------------------------------------
// Host: plans and launches
// ---------------------------------------------------------------------------

// An operand is sliced in panels, of K for an overlap and of g for a rotation,
// whose digits stay below kPanelBytes (an overlap's panel takes at least
// kPanelChunks chunks of K: 28 B per value of 512 columns, below its operands from
// K = 900 on).  So a workspace is bounded, and most of a panel's digits are read
// back from L2.  (W of a rotation is sliced whole, 3.5 times its size.)  Every panel
// of an overlap has partial sums of its own while all of them stay below
// kPanelBytes too; otherwise the panels add into one set, of one wave of CTAs or of
// twice the output's size, which costs a panel some 5 us of reads (352 x 176 over
// 37073, 5 panels: 810 us in 45 sets, 837 us in 9).
constexpr long long kPanelBytes = 128ll << 20;
constexpr int kPanelChunks = 4;
constexpr int kMaxSplits = 127;  // partial sums of an overlap, see k_oz_reduce

// bf16 digits [batch][7][rows][ld], box 64 x box_rows of one digit with 128-byte
// swizzle; rows and columns past the end read as zero.
static int make_map(CUtensorMap* m, const void* base, long long rows, long long batch, long long ld, int box_rows) {
  auto enc = encode_fn();
  if (!enc) return fail(QGB_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable from the driver");
  cuuint64_t dims[4] = {static_cast<cuuint64_t>(ld), static_cast<cuuint64_t>(rows), S, static_cast<cuuint64_t>(batch)};
  cuuint64_t strides[3] = {static_cast<cuuint64_t>(ld * 2), static_cast<cuuint64_t>(rows * ld * 2),
                           static_cast<cuuint64_t>(S * rows * ld * 2)};
  cuuint32_t box[4] = {BK, static_cast<cuuint32_t>(box_rows), 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(QGB_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", static_cast<int>(r));
  return QGB_OK;
}

template <int EPI>
static int launch_gemm(const void* a, long long a_rows, const void* b, long long b_rows, long long batch, long long ld,
                       GemmArgs args, cudaStream_t st) {
  CUtensorMap ma, mb;
  int rc;
  if ((rc = make_map(&ma, a, a_rows, batch, ld, BM))) return rc;
  if ((rc = make_map(&mb, b, b_rows, batch, ld, BN))) return rc;
  if ((rc = raise_smem_limit(k_oz_gemm<EPI>, SMEM_BYTES))) return rc;
  args.n_tiles = static_cast<int>((b_rows + BN - 1) / BN);
  args.m_tiles = static_cast<int>((a_rows + BM - 1) / BM);
  args.units = static_cast<int>(batch * args.splits) * args.n_tiles * args.m_tiles;
  k_oz_gemm<EPI><<<std::min(args.units, kSms), kThreads, SMEM_BYTES, st>>>(ma, mb, args);
  QGB_LAUNCH_CHECK("k_oz_gemm");
  return QGB_OK;
}

struct OzGram {
  long long a_rows, b_rows;     // real rows
  int fold, Lg, chunks;         // g per split, K chunks per split
  int panel_splits, panels, sets;  // sets of partial sums: one a split of a panel, or of all panels
  long long ld, a_elems, b_elems;
  size_t digits_bytes, e_bytes, partial_bytes, total;
};

static OzGram gram_layout(int nk, int M, int N, int K, bool real_out) {
  OzGram L;
  L.fold = real_out ? 1 : 0;
  L.a_rows = real_out ? M : 2ll * M;
  L.b_rows = real_out ? N : 2ll * N;
  const long long mt = (L.a_rows + BM - 1) / BM, nt = (L.b_rows + BN - 1) / BN;
  const int gpc = L.fold ? CHUNK / 2 : CHUNK;  // g per K chunk
  const int nchunk = (K + gpc - 1) / gpc;
  const long long per_chunk = nk * (L.a_rows + L.b_rows) * CHUNK * S * 2;
  const int cap = static_cast<int>(std::min<long long>(nchunk, std::max<long long>(kPanelChunks, kPanelBytes / per_chunk)));
  L.panels = (nchunk + cap - 1) / cap;
  const int cpp = (nchunk + L.panels - 1) / L.panels;
  // One wave of CTAs over the SMs per panel (one CTA fills an SM).
  const int want = static_cast<int>(std::max(1ll, std::min({static_cast<long long>(cpp), kSms / (mt * nt * nk),
                                                            static_cast<long long>(kMaxSplits)})));
  L.chunks = (cpp + want - 1) / want;
  L.panel_splits = (cpp + L.chunks - 1) / L.chunks;
  L.Lg = L.chunks * gpc;
  L.panels = static_cast<int>((K + static_cast<long long>(L.Lg) * L.panel_splits - 1) /
                              (static_cast<long long>(L.Lg) * L.panel_splits));
  L.ld = static_cast<long long>(L.panel_splits) * L.chunks * CHUNK;
  L.a_elems = round_up(nk * S * L.a_rows * L.ld, 128);
  L.b_elems = round_up(nk * S * L.b_rows * L.ld, 128);
  L.digits_bytes = static_cast<size_t>(L.a_elems + L.b_elems) * 2;
  const long long splits = static_cast<long long>(L.panels) * L.panel_splits;
  L.e_bytes = static_cast<size_t>(round_up(splits * nk * (M + N) * 4, 256));
  const long long set_bytes = nk * L.a_rows * L.b_rows * 8;
  L.sets = static_cast<int>(splits <= kMaxSplits && splits * set_bytes <= kPanelBytes ? splits : L.panel_splits);
  L.partial_bytes = static_cast<size_t>(round_up(L.sets * set_bytes, 256));
  L.total = L.digits_bytes + L.e_bytes + L.partial_bytes + 256 + 256;
  return L;
}

struct OzRot {
  int Kh, chunks, Npad, nt, rows, panels;
  long long ld, a_elems, b_elems;
  size_t e_bytes, total;
};

static OzRot rot_layout(int nk, int Kin, int Nout, int G) {
  OzRot L;
  L.Kh = static_cast<int>(round_up(Kin, 4));
  L.chunks = (2 * L.Kh + CHUNK - 1) / CHUNK;
  L.ld = round_up(2ll * L.Kh, 8);
  L.nt = (Nout + BN / 2 - 1) / (BN / 2);
  L.Npad = L.nt * (BN / 2);
  const long long per_tile = static_cast<long long>(nk) * BM * L.ld * S * 2;
  const int mt = (G + BM - 1) / BM;
  const int cap = static_cast<int>(std::max<long long>(1, std::min<long long>(mt, kPanelBytes / per_tile)));
  L.panels = (mt + cap - 1) / cap;
  L.rows = (mt + L.panels - 1) / L.panels * BM;
  L.panels = (G + L.rows - 1) / L.rows;
  L.a_elems = round_up(nk * S * static_cast<long long>(L.rows) * L.ld, 128);
  L.b_elems = round_up(nk * S * 2ll * L.Npad * L.ld, 128);
  L.e_bytes = static_cast<size_t>(round_up(static_cast<long long>(nk) * (L.rows + L.Npad + Kin) * 4, 256));
  L.total = static_cast<size_t>(L.a_elems + L.b_elems) * 2 + L.e_bytes + 256 + 256;
  return L;
}

}  // namespace oz

using namespace oz;

// Where the sliced product is the faster form (kSmallOverlap, kSmallRotation).  Its
// launches and fills take 30-40 us whatever the size, the multiply-adds' time grows
// with the product:
//   overlap   18 x 18 x 8000 (2.6 M multiply-adds)  sliced 45 us, multiply-adds 35 us
//             8 k of 36 x 18 x 1150 (6 M)           43 us against 66 us
//   rotation  60 x 60 x 1000 (3.6 M)                33 us against 30 us
//             64 x 64 x 1000 (4.1 M)                33 us against 36 us
bool oz_gram_use(int nk, int M, int N, int K) {
  return static_cast<double>(nk) * M * N * K >= kSmallOverlap && nk <= 4096 && M <= 65535 && N <= 65535;
}
bool oz_rotate_use(int nk, int Kin, int Nout, int G) {
  return static_cast<double>(nk) * Kin * Nout * G >= kSmallRotation && nk <= 4096 && Nout <= 65535 &&
         G <= 65535 * kExpRange;
}

size_t oz_gram_workspace_bytes(int nk, int M, int N, int K, bool real_out) {
  return gram_layout(nk, M, N, K, real_out).total;
}
size_t oz_rotate_workspace_bytes(int nk, int Kin, int Nout, int G) { return rot_layout(nk, Kin, Nout, G).total; }

int oz_gram(const void* A, long long a_batch, int lda, const void* B, long long b_batch, int ldb, int nk, int M, int N,
            int K, void* out, long long out_batch, int oi, int oj, void* ws, cudaStream_t st, const double* weight,
            bool real_out) {
  const OzGram L = gram_layout(nk, M, N, K, real_out);
  unsigned char* p = reinterpret_cast<unsigned char*>(round_up(reinterpret_cast<uintptr_t>(ws), 256));
  int* err = reinterpret_cast<int*>(p);
  p += 256;
  auto* da = reinterpret_cast<__nv_bfloat16*>(p);
  auto* db = da + L.a_elems;
  p += L.digits_bytes;
  const long long splits = static_cast<long long>(L.panels) * L.panel_splits;
  int* ea = reinterpret_cast<int*>(p);
  int* eb = ea + splits * nk * M;
  p += L.e_bytes;
  double* partial = reinterpret_cast<double*>(p);
  for (int pan = 0; pan < L.panels; ++pan) {
    const int g0 = pan * L.panel_splits * L.Lg;
    int* eap = ea + static_cast<long long>(pan) * L.panel_splits * nk * M;
    int* ebp = eb + static_cast<long long>(pan) * L.panel_splits * nk * N;
    const SliceArgs sa{static_cast<const double2*>(A), a_batch, lda, M, K, g0, L.Lg, L.fold, nullptr, da,
                       static_cast<int>(L.ld), eap};
    const SliceArgs sb{static_cast<const double2*>(B), b_batch, ldb, N, K, g0, L.Lg, L.fold, weight, db,
                       static_cast<int>(L.ld), ebp};
    const dim3 grid(std::max(M, N), L.panel_splits, 2 * nk);
    k_oz_slice_rows<<<grid, 256, 0, st>>>(sa, sb, pan == 0 ? err : nullptr);
    QGB_LAUNCH_CHECK("k_oz_slice_rows");
    GemmArgs g{};
    g.chunks = L.chunks;
    g.splits = L.panel_splits;
    g.ea = eap;
    g.eb = ebp;
    g.a_rows = M;
    g.b_rows = N;
    g.M = static_cast<int>(L.a_rows);
    g.N = static_cast<int>(L.b_rows);
    g.err = err;
    g.partial = partial;
    const bool own = L.sets > L.panel_splits;  // (one panel: either)
    g.split0 = own ? pan * L.panel_splits : 0;
    g.add = !own && pan > 0 ? 1 : 0;
    g.nbatch = nk;
    if (int rc = launch_gemm<EPI_PARTIAL>(da, L.a_rows, db, L.b_rows, nk, L.ld, g, st)) return rc;
  }
  const long long total = static_cast<long long>(nk) * M * N;
  const unsigned blocks = static_cast<unsigned>(std::min<long long>((total * kRed + 255) / 256, 8 * kSms));
  auto* reduce = L.fold ? k_oz_reduce<1> : k_oz_reduce<0>;
  reduce<<<blocks, 256, 0, st>>>(partial, L.sets, L.panel_splits, nk, M, N, static_cast<double2*>(out), out_batch, oi,
                                 oj, ea, eb, static_cast<int>(splits), static_cast<const double2*>(A),
                                 static_cast<const double2*>(B), a_batch, b_batch, lda, ldb, K, weight);
  QGB_LAUNCH_CHECK("k_oz_reduce");
  return QGB_OK;
}

int oz_rotate(const void* X, long long x_batch, int ldx, const void* W, long long w_batch, int wi, int wj, int nk,
              int Kin, int Nout, int G, void* out, long long out_batch, int ldo, bool accumulate, void* ws,
              cudaStream_t st) {
  const OzRot L = rot_layout(nk, Kin, Nout, G);
  unsigned char* p = reinterpret_cast<unsigned char*>(round_up(reinterpret_cast<uintptr_t>(ws), 256));
  int* err = reinterpret_cast<int*>(p);
  p += 256;
  auto* da = reinterpret_cast<__nv_bfloat16*>(p);
  auto* db = da + L.a_elems;
  p += (L.a_elems + L.b_elems) * 2;
  int* eg = reinterpret_cast<int*>(p);
  int* ew = eg + static_cast<long long>(nk) * L.rows;
  int* eb = ew + static_cast<long long>(nk) * L.Npad;
  QGB_CUDA_CHECK(cudaMemsetAsync(eb, 0, static_cast<size_t>(nk) * Kin * sizeof(int), st));
  k_oz_band_exp<<<dim3(Kin, (G + kExpRange - 1) / kExpRange, nk), 256, 0, st>>>(static_cast<const double2*>(X), x_batch,
                                                                                ldx, Kin, G, eb);
  QGB_LAUNCH_CHECK("k_oz_band_exp");
  k_oz_slice_mat<<<dim3(L.Npad, nk), 128, 0, st>>>(static_cast<const double2*>(W), w_batch, wi, wj, Kin, L.Kh, Nout,
                                                   L.Npad, db, static_cast<int>(L.ld), eb, ew);
  QGB_LAUNCH_CHECK("k_oz_slice_mat");
  // The last panel first: its part of X is the one k_oz_band_exp left in L2.
  for (int pan = L.panels - 1; pan >= 0; --pan) {
    const int g0 = pan * L.rows;
    const int rows = std::min(L.rows, G - g0);
    k_oz_slice_cols<<<dim3((rows + 31) / 32, nk), 256, 0, st>>>(static_cast<const double2*>(X), x_batch, ldx, Kin, L.Kh,
                                                               g0, G, rows, da, static_cast<int>(L.ld), eb, eg,
                                                               pan == L.panels - 1 ? err : nullptr);
    QGB_LAUNCH_CHECK("k_oz_slice_cols");
    GemmArgs g{};
    g.chunks = L.chunks;
    g.splits = 1;
    g.ea = eg;
    g.eb = ew;
    g.a_rows = rows;
    g.b_rows = L.Npad;
    g.M = rows;
    g.N = 2 * L.Npad;
    g.err = err;
    g.out = static_cast<double2*>(out);
    g.out_batch = out_batch;
    g.ldo = ldo;
    g.g0 = g0;
    g.G = G;
    g.Nout = Nout;
    g.accumulate = accumulate ? 1 : 0;
    g.X = static_cast<const double2*>(X);
    g.W = static_cast<const double2*>(W);
    g.x_batch = x_batch;
    g.w_batch = w_batch;
    g.ldx = ldx;
    g.wi = wi;
    g.wj = wj;
    g.Kin = Kin;
    if (int rc = launch_gemm<EPI_ROTATE>(da, rows, db, 2ll * L.Npad, nk, L.ld, g, st)) return rc;
  }
  return QGB_OK;
}

}  // namespace qgb
