// Internal interface of the band-space products (bandgemm.cu) for the other
// translation units of the library.
#pragma once

#include "qgb_common.cuh"

namespace qgb {

// Workspace of a gram() call of these extents: the split-K partial sums of the
// multiply-add kernels, which it cannot do without (0: none), and with `sliced`
// also what the tensor-core form (ozaki.cu) takes where that is the faster one.
// A call with the smaller size runs the multiply-add kernels.
size_t gram_workspace_bytes(int dtype, int nk, int M, int N, int K, bool sliced = true);

// out(i, j) (complex of out_dtype, at out + k*out_batch + i*oi + j*oj) =
// sum_g [w_g] conj(A[k][i][g]) B[k][j][g]; real_out keeps the real part.
int gram(int dtype, int out_dtype, const void* A, long long a_batch, int lda, const void* B, long long b_batch,
         int ldb, int nk, int M, int N, int K, void* out, long long out_batch, int oi, int oj, void* ws,
         size_t ws_bytes, cudaStream_t st, const double* weight = nullptr, bool real_out = false);

// out[k][j][g] (+)= sum_i W(i, j) X[k][i][g], W(i, j) = W[k*w_batch + i*wi + j*wj].
// With rotate_workspace_bytes() of workspace (0: none) the FP64 product runs on
// the tensor cores where that is the faster form.
size_t rotate_workspace_bytes(int dtype, int nk, int Kin, int Nout, int G);
int rotate(int dtype, const void* X, long long x_batch, int ldx, const void* W, long long w_batch, int wi, int wj,
           int nk, int Kin, int Nout, int G, void* out, long long out_batch, int ldo, bool accumulate,
           cudaStream_t st, void* ws = nullptr, size_t ws_bytes = 0);

// FP64 products by integer slices on the tensor cores (ozaki.cu), from these many
// multiply-adds on; smaller ones take the small kernels.
constexpr double kSmallOverlap = 3e6, kSmallRotation = 4e6;
bool oz_gram_use(int nk, int M, int N, int K);
size_t oz_gram_workspace_bytes(int nk, int M, int N, int K, bool real_out);
int oz_gram(const void* A, long long a_batch, int lda, const void* B, long long b_batch, int ldb, int nk, int M, int N,
            int K, void* out, long long out_batch, int oi, int oj, void* ws, cudaStream_t st, const double* weight,
            bool real_out);
bool oz_rotate_use(int nk, int Kin, int Nout, int G);
size_t oz_rotate_workspace_bytes(int nk, int Kin, int Nout, int G);
int oz_rotate(const void* X, long long x_batch, int ldx, const void* W, long long w_batch, int wi, int wj, int nk,
              int Kin, int Nout, int G, void* out, long long out_batch, int ldo, bool accumulate, void* ws,
              cudaStream_t st);

// Dp[k][b][a pa + r] = sum_c D[a][r][c] proj[k][b][a pa + c].
int dapply(int dtype, const void* proj, const void* D, int n_atoms, int pa, int nb, int nk, void* Dp,
           cudaStream_t st);

// out[k][b][g] += sum_p beta[k][p][g] (D projT[k][b])[p] in one launch, D applied
// by every CTA: for products of `rotate`'s small kernel with blocks of at most 8
// (an eighth more multiply-adds, about what the launch saved costs at 3e6) and at
// most 512 projectors (32 KB of shared memory).
bool backproject_small_use(int nk, int n_atoms, int pa, int nb, int n_tot);
int backproject_small(int dtype, const void* beta, const void* D, int n_atoms, int pa, const void* projT, void* out,
                      int nk, int nb, int n_tot, cudaStream_t st);

}  // namespace qgb
