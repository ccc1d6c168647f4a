// Local-potential apply V*psi on the G-sphere: scatter -> 3D inverse FFT -> *V(r)
// -> 3D forward FFT -> gather (+ KE*psi), for a block of bands at every k.
//
// Replaces Basis.apply_potential (qimpy/dft/electrons/_basis_ops.py:39-113, with
// _KernelCommon.expand_ifft 152-163 and _ApplyPotentialKernel.__call__ 183-199)
// and fuses Basis.apply_ke (_basis_ops.py:29-36).  FFT conventions follow
// qimpy/grid/_fft.py: inverse unnormalised, forward scaled by 1/N.
//
// The 3D transform is split by the G-sphere's structure.  In-sphere points are
// sorted by linear grid index, so each "slab" (points sharing the first grid
// index i0) is a contiguous range of the basis, and only the n_slabs i0 values
// the sphere touches carry data:
//   k_ifft_yz      one CTA per (k, band, slab): scatter the slab's points into
//                  an N1 x N2 plane in shared memory, inverse z-FFT on the rows
//                  the sphere touches, inverse y-FFT on all columns, store the
//                  plane (real-space y, z in permuted order) to the workspace.
//   k_xpass        one CTA per (k, band, tiles of 64 (FP32) or 32 (FP64) of the
//                  plane's columns): gather the slabs' rows into pencils along
//                  x, inverse x-FFT, multiply by V(r), forward x-FFT, keep only
//                  the slab rows, store back.
//   k_fft_yz_gather one CTA per (k, band, slab): forward y-FFT on all columns,
//                  forward z-FFT on the touched rows, gather the slab's points,
//                  scale by 1/N and add KE*psi.
// Versus three full-grid passes each way this skips the empty x-planes in the
// y/z passes and the empty z-rows in the z passes.  Where both factors of an
// axis exceed 1, the passes next to global memory read or write it directly:
// the first inverse y pass reads untouched rows as zero (no zero fill), the
// last inverse y pass and the last forward x pass store straight to the
// planes, and the first inverse x pass and the first forward y pass read
// straight from them, so shared memory sees each element in the inner passes
// only.  With QGB_ACCUMULATE the gather adds to `out` (the mixed H.psi writes
// its nonlocal term there first, on another stream).  The FP64 codelets run in
// block fixed point on the integer pipes (block_fixed.cuh).
#include "batched_kernels.cuh"
#include "density_kernels.cuh"

namespace qgb {

extern template int launch_chunk<float>(const qgb_sphere&, const LocalParams&, const void*, void*, void*, cudaStream_t,
                                        cudaEvent_t);
extern template int launch_chunk<double>(const qgb_sphere&, const LocalParams&, const void*, void*, void*,
                                         cudaStream_t, cudaEvent_t);
extern template int launch_batched<float>(const qgb_batch_item*, const int*, const long long*, const int*,
                                          const long long*, long long, long long, size_t, size_t, cudaStream_t);
extern template int launch_batched<double>(const qgb_batch_item*, const int*, const long long*, const int*,
                                           const long long*, long long, long long, size_t, size_t, cudaStream_t);
extern template int launch_density_chunk<float>(const qgb_sphere&, const LocalParams&, const void*, void*,
                                                const double*, double*, cudaStream_t);
extern template int launch_density_chunk<double>(const qgb_sphere&, const LocalParams&, const void*, void*,
                                                 const double*, double*, cudaStream_t);

template <typename T>
__global__ void k_apply_ke(const qgb_sphere s, int nb, const cplx_t<T>* __restrict__ C,
                           cplx_t<T>* __restrict__ out) {
  const size_t total = static_cast<size_t>(s.nk) * nb * s.n_tot;
  const T* ke = static_cast<const T*>(s.ke);
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t g = i % s.n_tot;
    const size_t k = i / (static_cast<size_t>(nb) * s.n_tot);
    const T e = ke[k * s.n_tot + g];
    const cplx_t<T> c = C[i];
    out[i] = mk<T>(e * c.x, e * c.y);
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

#ifdef QGB_DEBUG_CHECKS
int violation_local_f32(unsigned long long*);
int violation_local_f64(unsigned long long*);
int violation_batched_f32(unsigned long long*);
int violation_batched_f64(unsigned long long*);
int violation_density_f32(unsigned long long*);
int violation_density_f64(unsigned long long*);
// Debug builds: copy out and clear the first recorded range violation
// (site, index, limit, packed block index); site 0 = none.
int debug_violation(unsigned long long* out4) {
  QGB_CUDA_CHECK(cudaDeviceSynchronize());
  for (int i = 0; i < 4; ++i) out4[i] = 0;
  for (auto* unit : {violation_local_f32, violation_local_f64, violation_batched_f32, violation_batched_f64,
                     violation_density_f32, violation_density_f64})
    if (int rc = unit(out4)) return rc;
  return QGB_OK;
}
#endif

static bool codelet_size(int R) {
  switch (R) {
    case 1: case 2: case 3: case 4: case 5: case 6: case 7: case 8: case 9: case 10:
    case 12: case 14: case 15: case 16:
      return true;
    default:
      return false;
  }
}

size_t plane_smem_bytes(const qgb_sphere& s, int dtype) {
  const size_t e = elem_bytes(dtype);
  const size_t yz = (static_cast<size_t>(s.N[1]) * (s.N[2] + 1) + s.N[1] + s.N[2]) * e + s.N[1] * sizeof(int);
  const size_t x = (static_cast<size_t>(s.N[0]) * (s.N[2] + 1) + s.N[0]) * e;
  return std::max(yz, x);
}

int validate_sphere(const qgb_sphere* s, int dtype, bool need_potential = true) {
  if (s == nullptr) return fail(QGB_ERR_INVALID, "sphere descriptor is NULL");
  if (dtype != QGB_F64 && dtype != QGB_F32) return fail(QGB_ERR_INVALID, "unknown dtype %d", dtype);
  if (s->nk < 1 || s->n_tot < 1 || s->max_slabs < 1)
    return fail(QGB_ERR_INVALID, "empty sphere (nk=%d n_tot=%d max_slabs=%d)", s->nk, s->n_tot,
                s->max_slabs);
  for (int a = 0; a < 3; ++a) {
    if (s->N[a] < 1 || s->N[a] > 65535)
      return fail(QGB_ERR_INVALID, "grid dimension %d = %d out of range", a, s->N[a]);
    if (!codelet_size(s->L1[a]) || !codelet_size(s->L2[a]) || s->L1[a] * s->L2[a] != s->N[a])
      return fail(QGB_ERR_INVALID, "axis %d: N=%d is not L1*L2 with L1=%d, L2=%d codelet sizes",
                  a, s->N[a], s->L1[a], s->L2[a]);
  }
  if (s->max_slabs > s->N[0]) return fail(QGB_ERR_INVALID, "max_slabs %d > N0", s->max_slabs);
  if (!s->n || !s->n_slabs || !s->slab_start || !s->slab_i0 || !s->yz || !s->row_start ||
      !s->rows || !s->twiddle || !s->ke)
    return fail(QGB_ERR_INVALID, "sphere descriptor has a NULL table");
  if (need_potential && !s->V) return fail(QGB_ERR_INVALID, "sphere descriptor has no potential V");
  if (plane_smem_bytes(*s, dtype) > 227 * 1024)
    return fail(QGB_ERR_UNSUPPORTED, "grid %dx%dx%d needs %zu B of shared memory per plane (max 227 KB)",
                s->N[0], s->N[1], s->N[2], plane_smem_bytes(*s, dtype));
  return QGB_OK;
}

size_t plane_bytes_per_band(const qgb_sphere& s, int dtype) {
  return static_cast<size_t>(s.nk) * s.max_slabs * s.N[1] * s.N[2] * elem_bytes(dtype);
}

// gather_after (optional): an event the gather kernels wait for, so that a
// term written into `out` on another stream (QGB_ACCUMULATE) can be produced
// while the inverse and x passes run.
int apply_potential(const qgb_sphere* s, int dtype, const void* C, void* out, int nb,
                    unsigned flags, void* ws, size_t ws_bytes, cudaStream_t st, cudaEvent_t gather_after = nullptr) {
  int rc = validate_sphere(s, dtype);
  if (rc) return rc;
  if (nb < 0) return fail(QGB_ERR_INVALID, "nb = %d < 0", nb);
  if (nb == 0) return QGB_OK;
  // C == out is allowed: every chunk reads its bands of C (k_ifft_yz, and the
  // KE term in k_fft_yz_gather before the same thread stores) before writing them.
  if (!C || !out) return fail(QGB_ERR_INVALID, "NULL wavefunction pointer");
  const size_t per_band = plane_bytes_per_band(*s, dtype);
  if (!ws || ws_bytes < per_band)
    return fail(QGB_ERR_WORKSPACE, "workspace %zu B < %zu B needed for one band", ws_bytes, per_band);
  const int chunk = static_cast<int>(std::min<size_t>(nb, std::min<size_t>(ws_bytes / per_band, 65535)));
  for (int b0 = 0; b0 < nb; b0 += chunk) {
    LocalParams lp{nb, b0, std::min(chunk, nb - b0), flags};
    rc = (dtype == QGB_F64) ? launch_chunk<double>(*s, lp, C, out, ws, st, gather_after)
                            : launch_chunk<float>(*s, lp, C, out, ws, st, gather_after);
    if (rc) return rc;
  }
  return QGB_OK;
}

// The x kernel of a batch takes whole y-rows.
size_t sphere_smem_bytes(const qgb_sphere& s, int dtype) {
  return std::max(plane_smem_bytes(s, dtype), x_smem_bytes(s, s.N[2], elem_bytes(dtype)));
}

int apply_potential_batched(const qgb_batch_item* items, int n_items, const int* slab_item,
                            const long long* slab_starts, const int* row_item, const long long* row_starts,
                            long long n_slab, long long n_row, int dtype, size_t smem_yz, size_t smem_x,
                            cudaStream_t st) {
  if (dtype != QGB_F64 && dtype != QGB_F32) return fail(QGB_ERR_INVALID, "unknown dtype %d", dtype);
  if (n_items < 0 || n_slab < 0 || n_row < 0) return fail(QGB_ERR_INVALID, "negative batch sizes");
  if (n_items == 0 || n_slab == 0) return QGB_OK;
  if (!items || !slab_starts || !row_starts || !slab_item || !row_item) return fail(QGB_ERR_INVALID, "NULL batch table");
  if (n_slab > 0x7FFFFFFFLL || n_row > 0x7FFFFFFFLL) return fail(QGB_ERR_UNSUPPORTED, "batch too large for one grid");
  if (smem_yz > 227 * 1024 || smem_x > 227 * 1024)
    return fail(QGB_ERR_UNSUPPORTED, "batched shared memory %zu / %zu B > 227 KB", smem_yz, smem_x);
  if (smem_x < smem_yz) return fail(QGB_ERR_INVALID, "smem_x %zu < smem_yz %zu", smem_x, smem_yz);
  return dtype == QGB_F64 ? launch_batched<double>(items, slab_item, slab_starts, row_item, row_starts, n_slab, n_row,
                                                   smem_yz, smem_x, st)
                          : launch_batched<float>(items, slab_item, slab_starts, row_item, row_starts, n_slab, n_row,
                                                  smem_yz, smem_x, st);
}

int apply_ke(const qgb_sphere* s, int dtype, const void* C, void* out, int nb, cudaStream_t st) {
  if (s == nullptr) return fail(QGB_ERR_INVALID, "sphere descriptor is NULL");
  if (nb < 0 || !C || !out || !s->ke) return fail(QGB_ERR_INVALID, "bad apply_ke arguments");
  if (nb == 0) return QGB_OK;
  const size_t total = static_cast<size_t>(s->nk) * nb * s->n_tot;
  const int blocks = static_cast<int>(std::min<size_t>((total + 255) / 256, 152 * 16));
  if (dtype == QGB_F64)
    k_apply_ke<double><<<blocks, 256, 0, st>>>(*s, nb, static_cast<const double2*>(C), static_cast<double2*>(out));
  else
    k_apply_ke<float><<<blocks, 256, 0, st>>>(*s, nb, static_cast<const float2*>(C), static_cast<float2*>(out));
  QGB_LAUNCH_CHECK("k_apply_ke");
  return QGB_OK;
}


int collect_density(const qgb_sphere* s, int dtype, const void* C, int nb, const double* prefac, double* rho,
                    unsigned flags, void* ws, size_t ws_bytes, cudaStream_t st) {
  int rc = validate_sphere(s, dtype, false);  // the density needs no potential
  if (rc) return rc;
  if (nb < 0) return fail(QGB_ERR_INVALID, "nb = %d < 0", nb);
  if (!rho) return fail(QGB_ERR_INVALID, "NULL density pointer");
  const size_t N = static_cast<size_t>(s->N[0]) * s->N[1] * s->N[2];
  if (!(flags & QGB_ACCUMULATE)) QGB_CUDA_CHECK(cudaMemsetAsync(rho, 0, N * sizeof(double), st));
  if (nb == 0) return QGB_OK;
  if (!C || !prefac) return fail(QGB_ERR_INVALID, "NULL wavefunction or prefactor pointer");
  const size_t per_band = plane_bytes_per_band(*s, dtype);
  if (!ws || ws_bytes < per_band)
    return fail(QGB_ERR_WORKSPACE, "workspace %zu B < %zu B needed for one band", ws_bytes, per_band);
  const int chunk = static_cast<int>(std::min<size_t>(nb, std::min<size_t>(ws_bytes / per_band, 65535)));
  for (int b0 = 0; b0 < nb; b0 += chunk) {
    LocalParams lp{nb, b0, std::min(chunk, nb - b0), 0u};
    rc = (dtype == QGB_F64) ? launch_density_chunk<double>(*s, lp, C, ws, prefac, rho, st)
                            : launch_density_chunk<float>(*s, lp, C, ws, prefac, rho, st);
    if (rc) return rc;
  }
  return QGB_OK;
}

}  // namespace qgb
