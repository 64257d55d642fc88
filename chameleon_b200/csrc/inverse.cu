// inverse.cu -- triangular inverse, triangular product and SPD inverse from
// the Cholesky factor (dtrtri, dlauum, dpotri), and the LAPACKE / Fortran
// LAPACK interfaces of the Cholesky path.
//
// Reference: compute/ztrtri.c, zlauum.c, zpotri.c (zpotri = pztrtri then
// pzlauum, compute/zpotri.c), lapack_api/src/lapack_z{posv,potrf,potrs,potri,
// trtri,lauum}.c.  All of them work on the lower triangle (an upper one is its
// transposed view) with FP64 tensor-core products, and skip the zero halves
// of triangular operands, so that each does its n^3 / 3 operations:
//   dtrtri: the inverted 64 x 64 diagonal blocks in one launch, then doubling:
//           at block size h = 64, 128, ... every pair of neighbouring h-blocks
//           gets X21 = -X22 (L21 X11), two launches for all pairs together; a
//           factor too ill-conditioned for that (INV_COND) by substitution,
//           whose residual does not grow with the condition (order 2500: 0.59
//           and 2.4 ms);
//   dlauum: A(i,j) = sum_{k >= i} L(k,i) L(k,j), one launch;
//   dpotri: dtrtri then dlauum, as LAPACK and the reference; the inverse of
//           the factor stays in the workspace between the two (order 2500:
//           4.26 ms as a dense solve and a dense product, 0.79 ms now).
// LAPACK's contract is kept: only the `uplo` triangle of A is read and
// written; dtrtri returns info = i when A(i,i) is exactly zero (A untouched),
// with diag = Unit the diagonal is neither read nor written.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "core.cuh"
#include "internal.h"
#include "rec.cuh"

struct cham_b200_handle_s;   // tile_abi.cu

namespace chb {

// Block edge of the products.  The k extents of the blocks differ by up to
// n / 64 times (triangular operands), so blocks are small and the longest come
// first: a 128-wide block of n = 2500 would run 0.65 ms alone, longer than the
// whole operation needs.
constexpr int HB = 64;
using CfgInv = Cfg64<double>;
constexpr int INV_CTAS_PER_SM = 3;
constexpr size_t LEAF_BYTES = 2 * IB * LEAF_LD * sizeof(double);

// What is known of a triangular matrix and its inverse: its first zero diagonal
// entry (1-based; INT_MAX: none) and the infinity norms of the two.
//
// Doubling keeps the residual X L - I of LAPACK's dtrtri, but L X - I grows with
// the condition: restated on the host (kernel, Wishart, Laplacian matrices,
// orders 512 and 1024), it is within 1.5 times a substitution's while the product
// of the norms is below 64, 4 times at 5e2, 1e2 times at 4e4, 1e4 times at 1e6.
// Beyond INV_COND (NaN included) the inverse is made by substitution instead.
constexpr double INV_COND = 64.0;
struct InvState {
    int first;
    double norm[2];
    __host__ __device__ bool ill() const { return !(norm[0] * norm[1] <= INV_COND); }
    __host__ __device__ bool usable() const { return first == INT_MAX && !ill(); }
};
constexpr int NORM_ROWS = 4;   // rows per CTA of the norms (a row is a chain of loads: 64 threads each)

// The inverted HB x HB diagonal blocks of the lower L (n x n), one CTA each, at
// X + q step (column-major, ld ldx); unit: with an implied unit diagonal.
__global__ void __launch_bounds__(NT_CTA, 1) diag_inv_kernel(View L, int n, int unit, double *X, int64_t ldx,
                                                             int64_t step) {
    extern __shared__ __align__(128) double smem[];
    const int j0 = blockIdx.x * HB, nb = min(HB, n - j0);
    rec::leaf64_load(L.sub(j0, j0), nb, smem);
    double *sX = smem + 64 * rec::LDS;
    rec::leaf64_core<double, false>(smem, sX, nb, unit != 0);
    double *D = X + blockIdx.x * step;
    for (int idx = threadIdx.x; idx < nb * nb; idx += NT_CTA)
        D[idx % nb + (int64_t)(idx / nb) * ldx] = sX[idx % nb + (idx / nb) * rec::LDS];
}

// X (column-major, ld ldx) <- L^-1 (trans: L^-T) for the lower L by substitution
// with its inverted diagonal blocks (HB x HB each, one after the other): strips
// of SUBST_W columns, one CTA each, the longest first; only the rows in which a
// strip of the result is not zero.  A strip is a chain of n / 64 products on one
// SM, so it is narrow, with two CTAs per SM and a deep pipeline.
constexpr int SUBST_W = 32;
using CfgSubst = GemmCfg<double, 64, SUBST_W, 4, 2, SPLIT_BF16X3, 4>;
__global__ void __launch_bounds__(NT_CTA, 2)
    inv_subst_kernel(View L, int n, const double *invd, double *X, int64_t ldx, int trans) {
    extern __shared__ __align__(128) double smem[];
    const int c0 = (trans ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * SUBST_W, w = min(SUBST_W, n - c0);
    const int b = c0 / HB, r0 = trans ? 0 : b * HB, m = trans ? min(n, (b + 1) * HB) : n - r0;
    const View S = View{X, 1, ldx}.sub(0, c0);
    for (int idx = threadIdx.x; idx < w * n; idx += NT_CTA) {
        const int i = idx % n, j = idx / n;
        *S.at(i, j) = i == c0 + j ? 1.0 : 0.0;
    }
    cta_sync_global();
    trsm_left<double, SPLIT_BF16X3, CfgSubst>(S.sub(r0, 0), w, L.sub(r0, r0), m, invd + (int64_t)(r0 / HB) * HB * HB,
                                              trans != 0, smem);
}

// One half of a doubling step on the pairs of h-blocks (rows [r, r + h2) below
// rows [r - h, r), r = h (2 q + 1), h2 = h or the matrix's end): output block
// (bi, bj) of pair q.  first: W21 = L21 X11, written into T (column-major, ld
// ldx); else X21 = -X22 W21, from T into X.
__global__ void __launch_bounds__(NT_CTA, INV_CTAS_PER_SM)
    trtri_pair_kernel(View L, int n, int h, double *X, double *T, int64_t ldx, int first) {
    extern __shared__ __align__(128) double smem[];
    const int r = h * (2 * (int)blockIdx.z + 1), c = r - h, h2 = min(h, n - r);
    // the longest products first: W needs k >= its column, X22 W k <= its row
    const int bi = first ? blockIdx.x : gridDim.x - 1 - blockIdx.x, bj = blockIdx.y;
    const int i0 = bi * HB, j0 = bj * HB;
    if (i0 >= h2) return;
    const int rows = min(HB, h2 - i0);
    Acc<CfgInv> acc;
    acc.zero();
    const View Xv{X, 1, ldx}, Tv{T, 1, ldx};
    if (first) {
        cta_gemm(acc, L.sub(r + i0, c + j0), Xv.sub(c + j0, c + j0).t(), rows, HB, h - j0, smem);
        acc.store_to(Tv.sub(r + i0, c + j0), rows, HB);
    } else {
        cta_gemm(acc, Xv.sub(r + i0, r), Tv.sub(r, c + j0).t(), rows, HB, i0 + rows, smem);
        acc.for_each([&](int i, int j, double v) {
            if (i < rows) *Xv.at(r + i0 + i, c + j0 + j) = -v;
        });
    }
}

// C (lower triangle, n x n view) = X^T X for the lower X (column-major, ld
// ldx): blocks of the lower triangle in row order, so that the longest sums
// (k from the block's first row to n) start first.  Nothing is written when
// st is given and its inverse is not to be used.
__global__ void __launch_bounds__(NT_CTA, INV_CTAS_PER_SM)
    lauum_kernel(View X, int n, View C, const InvState *st) {
    extern __shared__ __align__(128) double smem[];
    if (st && !st->usable()) return;
    int bi = (int)((sqrtf(8.f * (float)blockIdx.x + 1.f) - 1.f) * 0.5f);
    while ((bi + 1) * (bi + 2) / 2 <= (int)blockIdx.x) ++bi;
    while (bi * (bi + 1) / 2 > (int)blockIdx.x) --bi;
    const int bj = (int)blockIdx.x - bi * (bi + 1) / 2;
    const int i0 = bi * HB, j0 = bj * HB, rows = min(HB, n - i0), cols = min(HB, n - j0);
    Acc<CfgInv> acc;
    acc.zero();
    // k in this block row: X(k, i) is lower there, and is read in full
    cta_gemm(acc, X.sub(i0, i0).t(), X.sub(i0, j0).t(), rows, cols, n - i0, smem);
    acc.for_each([&](int i, int j, double v) {
        if (i < rows && j < cols && i0 + i >= j0 + j) *C.at(i0 + i, j0 + j) = v;
    });
}

// D <- the lower triangle of S (views of order n), zeros above it when
// zero_upper; the diagonal is left out when skip_diag; nothing when st is given
// and its inverse is not to be used.  Block (x, y): 64 rows of 4 columns per step, along the
// destination's contiguous direction.
__global__ void tri_copy_kernel(View S, View D, int n, int zero_upper, int skip_diag, const InvState *st) {
    if (st && !st->usable()) return;
    const bool cm = D.rs == 1;
    for (int y = blockIdx.y; y < n; y += gridDim.y)
        for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < n; x += gridDim.x * blockDim.x) {
            const int i = cm ? x : y, j = cm ? y : x;
            if (i < j ? !zero_upper : (i == j && skip_diag)) continue;
            *D.at(i, j) = i >= j ? *S.at(i, j) : 0.0;
        }
}

__global__ void inv_state_kernel(InvState *st) { *st = InvState{INT_MAX, {0.0, 0.0}}; }
// st->first = min over i of (i + 1) with A(i,i) == 0.
__global__ void zero_diag_kernel(View A, int N, InvState *st) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
        if (*A.at(i, i) == 0.0) atomicMin(&st->first, i + 1);
}
// st->norm = the infinity norms of L and of its inverse X.
__global__ void __launch_bounds__(NT_CTA, 4) inv_norm_kernel(View L, View X, int n, int unit, InvState *st) {
    const int r0 = (gridDim.x - 1 - blockIdx.x) * NORM_ROWS;   // the longest rows first
    rec::lower_norms<NORM_ROWS>(L, X, r0, min(NORM_ROWS, n - r0), unit != 0, st->norm);
}

namespace {
int grid_for(int64_t total) { return (int)std::min<int64_t>(std::max<int64_t>((total + 255) / 256, 1), 148 * 16); }

// A handle of the tile ABI on the library stream (kept).
cublasHandle_t lib_handle() {
    static cublasHandle_t h = nullptr;
    if (!h && CHAM_B200_Handle_Create(&h, ctx().stream) != 0) h = nullptr;
    return h;
}

double *g_w1 = nullptr, *g_w2 = nullptr, *g_w3 = nullptr, *g_w4 = nullptr, *g_w5 = nullptr;
size_t g_w1_bytes = 0, g_w2_bytes = 0, g_w3_bytes = 0, g_w4_bytes = 0, g_w5_bytes = 0;
InvState *g_state = nullptr;

double *work(double **buf, size_t *cap, size_t bytes) {
    if (bytes > *cap) {
        cudaStreamSynchronize(ctx().stream);
        dev_free(*buf);
        *cap = 0;
        if (!(*buf = (double *)dev_alloc(bytes))) return nullptr;
        *cap = bytes;
    }
    return *buf;
}
}  // namespace

// Lower view of the uplo triangle.
static View lower_view(cham_uplo_t uplo, double *A, int lda) {
    return uplo == ChamLower ? View{A, 1, lda} : View{A, lda, 1};
}

static int inv_attrs() {
    static bool done = false;
    if (done) return 0;
    CHB_CUDA(cudaFuncSetAttribute(trtri_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CfgInv::SMEM_BYTES));
    CHB_CUDA(cudaFuncSetAttribute(lauum_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CfgInv::SMEM_BYTES));
    CHB_CUDA(cudaFuncSetAttribute(inv_subst_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CfgSubst::SMEM_BYTES));
    CHB_CUDA(cudaFuncSetAttribute(diag_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)LEAF_BYTES));
    done = true;
    return 0;
}

static void tri_copy(View S, View D, int N, int zero_upper, int skip_diag, const InvState *st, cudaStream_t s) {
    const dim3 grid((N + 255) / 256, std::min(N, 2048));
    tri_copy_kernel<<<grid, 256, 0, s>>>(S, D, N, zero_upper, skip_diag, st);
    CHB_LAUNCHED(1);
}

// Workspace leading dimension: even (16-byte copies of the products' operands)
// and not a multiple of a power of two for the common orders.
static int64_t work_ld(int N) { return (N + 1) / 2 * 2 + 2; }

// The inverse of the lower L (view of order N) by doubling into the first
// workspace (column-major, ld work_ld(N), zeros above the diagonal of every
// HB-block), and g_state.  Returns the workspace, null when there is no memory
// for the two that doubling needs (g_state then has the first zero alone).
static int trtri_work(View L, cham_diag_t diag, int N, cudaStream_t s, double **Xp) {
    if (int rc = inv_attrs()) return rc;
    if (!g_state && !(g_state = (InvState *)dev_alloc(sizeof(InvState)))) return CHAMELEON_ERR_OUT_OF_RESOURCES;
    const int64_t ld = work_ld(N);
    const bool unit = diag == ChamUnit;
    inv_state_kernel<<<1, 1, 0, s>>>(g_state);
    CHB_LAUNCHED(1);
    if (!unit) {
        zero_diag_kernel<<<grid_for(N), 256, 0, s>>>(L, N, g_state);
        CHB_LAUNCHED(1);
    }
    double *X = work(&g_w1, &g_w1_bytes, (size_t)ld * N * sizeof(double));
    double *T = N > HB ? work(&g_w2, &g_w2_bytes, (size_t)ld * N * sizeof(double)) : X;
    *Xp = nullptr;
    if (!X || !T) return 0;
    diag_inv_kernel<<<(N + HB - 1) / HB, NT_CTA, LEAF_BYTES, s>>>(L, N, unit, X, ld, HB * (ld + 1));
    CHB_LAUNCHED(1);
    for (int64_t h = HB; h < N; h *= 2) {
        // pairs with any rows in their second block
        const int pairs = (int)((N - h + 2 * h - 1) / (2 * h)), nb = (int)(h / HB);
        for (int first = 1; first >= 0; --first)
            trtri_pair_kernel<<<dim3(nb, nb, pairs), NT_CTA, CfgInv::SMEM_BYTES, s>>>(L, N, (int)h, X, T, ld, first);
        CHB_LAUNCHED(2);
    }
    inv_norm_kernel<<<(N + NORM_ROWS - 1) / NORM_ROWS, NT_CTA, 0, s>>>(L, View{X, 1, ld}, N, unit, g_state);
    CHB_LAUNCHED(1);
    CHB_CUDA(cudaGetLastError());
    *Xp = X;
    return 0;
}

// The same inverse by substitution, as a lower view on the first workspace.
// For an upper matrix U = L^T it is U X = I that is solved, as for a lower one.
static int trtri_subst(cham_uplo_t uplo, View L, cham_diag_t diag, int N, cudaStream_t s, View *Xv) {
    if (int rc = inv_attrs()) return rc;
    const int64_t ld = work_ld(N);
    const int nb = (N + HB - 1) / HB, upper = uplo == ChamUpper;
    double *X = work(&g_w1, &g_w1_bytes, (size_t)ld * N * sizeof(double));
    double *invd = work(&g_w5, &g_w5_bytes, (size_t)nb * HB * HB * sizeof(double));
    if (!X || !invd) return CHAMELEON_ERR_OUT_OF_RESOURCES;
    diag_inv_kernel<<<nb, NT_CTA, LEAF_BYTES, s>>>(L, N, diag == ChamUnit, invd, HB, HB * HB);
    inv_subst_kernel<<<(N + SUBST_W - 1) / SUBST_W, NT_CTA, CfgSubst::SMEM_BYTES, s>>>(L, N, invd, X, ld, upper);
    CHB_LAUNCHED(2);
    CHB_CUDA(cudaGetLastError());
    *Xv = upper ? View{X, ld, 1} : View{X, 1, ld};
    return 0;
}

static int read_state(InvState *st, cudaStream_t s) {
    CHB_CUDA(cudaMemcpyAsync(st, g_state, sizeof(InvState), cudaMemcpyDeviceToHost, s));
    CHB_CUDA(cudaStreamSynchronize(s));
    return 0;
}

static void lauum_launch(View X, int N, View C, const InvState *st, cudaStream_t s) {
    const int nb = (N + HB - 1) / HB;
    lauum_kernel<<<nb * (nb + 1) / 2, NT_CTA, CfgInv::SMEM_BYTES, s>>>(X, N, C, st);
    CHB_LAUNCHED(1);
}

// The three operations on a device column-major A (ld lda), on the library
// stream; synchronous.  Return LAPACK's info (> 0) or a CHAMELEON_ERR_* code.
//
// dtrtri (potri: then dlauum): finish(X, st) writes the result from the lower
// inverse X, unless st says that it is not to be used.  The inverse by doubling
// is finished at once; what the host reads at the end decides whether that has
// happened, or A is singular (not modified), or the substitution has to run,
// which also serves when there is memory for one workspace only.
template <class Finish>
static int invert(cham_uplo_t uplo, cham_diag_t diag, int N, double *A, int lda, Finish finish) {
    cudaStream_t s = ctx().stream;
    double *X = nullptr;
    if (int rc = trtri_work(lower_view(uplo, A, lda), diag, N, s, &X)) return rc;
    if (X) finish(View{X, 1, work_ld(N)}, g_state);
    InvState st;
    if (int rc = read_state(&st, s)) return rc;
    if (st.first != INT_MAX) return st.first;
    if (X && !st.ill()) return 0;
    View Xv;
    if (int rc = trtri_subst(uplo, lower_view(uplo, A, lda), diag, N, s, &Xv)) return rc;
    finish(Xv, nullptr);
    CHB_CUDA(cudaGetLastError());
    CHB_CUDA(cudaStreamSynchronize(s));
    return 0;
}

int trtri_dev(cham_uplo_t uplo, cham_diag_t diag, int N, double *A, int lda) {
    cudaStream_t s = ctx().stream;
    return invert(uplo, diag, N, A, lda, [&](View X, const InvState *st) {
        tri_copy(X, lower_view(uplo, A, lda), N, 0, diag == ChamUnit, st, s);
    });
}

int lauum_dev(cham_uplo_t uplo, int N, double *A, int lda) {
    cudaStream_t s = ctx().stream;
    if (int rc = inv_attrs()) return rc;
    const View L = lower_view(uplo, A, lda);
    const int64_t ld = work_ld(N);
    double *T = work(&g_w1, &g_w1_bytes, (size_t)ld * N * sizeof(double));
    if (!T) return CHAMELEON_ERR_OUT_OF_RESOURCES;
    tri_copy(L, View{T, 1, ld}, N, 1, 0, nullptr, s);
    lauum_launch(View{T, 1, ld}, N, L, nullptr, s);
    CHB_CUDA(cudaGetLastError());
    CHB_CUDA(cudaStreamSynchronize(s));
    return 0;
}

int potri_dev(cham_uplo_t uplo, int N, double *A, int lda) {
    cudaStream_t s = ctx().stream;
    return invert(uplo, ChamNonUnit, N, A, lda, [&](View X, const InvState *st) {
        lauum_launch(X, N, lower_view(uplo, A, lda), st, s);
    });
}

// S (N x N, ld N) <- the symmetric matrix whose uplo triangle is in A.
__global__ void sym_full_kernel(const double *A, int64_t lda, double *S, int N, int upper) {
    const int64_t total = (int64_t)N * N;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(idx % N), j = (int)(idx / N);
        const bool in = upper ? i <= j : i >= j;
        S[i + (int64_t)j * N] = in ? A[i + (int64_t)j * lda] : A[j + (int64_t)i * lda];
    }
}

// compute/pzpotrimm.c: A <- A^-1 (uplo triangle; A is the SPD matrix on
// entry: potrf, trtri, lauum), then C = B A^-1 (the symm of its last loop
// nest, alpha = 1, beta = 0).  Device arrays.
int potrimm_dev(cham_uplo_t uplo, int N, double *A, int lda, const double *B, int ldb, double *C, int ldc) {
    int rc = CHAMELEON_dpotrf(uplo, N, A, lda);
    if (rc) return rc;
    if ((rc = potri_dev(uplo, N, A, lda))) return rc;
    cudaStream_t s = ctx().stream;
    cublasHandle_t h = lib_handle();
    if (!h) return CHAMELEON_ERR_UNEXPECTED;
    double *S = work(&g_w1, &g_w1_bytes, (size_t)N * N * sizeof(double));
    if (!S) return CHAMELEON_ERR_OUT_OF_RESOURCES;
    sym_full_kernel<<<grid_for((int64_t)N * N), 256, 0, s>>>(A, lda, S, N, uplo == ChamUpper);
    CHB_LAUNCHED(1);
    const double one = 1.0, zero = 0.0;
    if ((rc = CUDA_dgemm(ChamNoTrans, ChamNoTrans, N, N, N, &one, B, ldb, S, N, &zero, C, ldc, h))) return rc;
    CHB_CUDA(cudaGetLastError());
    CHB_CUDA(cudaStreamSynchronize(s));
    return 0;
}

// LAPACK layout: A on the host or the device.
enum InvOp { OP_TRTRI, OP_LAUUM, OP_POTRI };
int inverse_lapack(InvOp op, cham_uplo_t uplo, cham_diag_t diag, int N, double *A, int LDA) {
    cudaStream_t s = ctx().stream;
    cudaPointerAttributes at;
    bool dev = false;
    if (cudaPointerGetAttributes(&at, A) == cudaSuccess)
        dev = at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged;
    else
        cudaGetLastError();
    double *dA = A;
    int lda = LDA;
    if (!dev) {
        if (!(dA = stage_in(0, A, LDA, N, N, s))) return CHAMELEON_ERR_OUT_OF_RESOURCES;
        lda = N;
    }
    int rc = (op == OP_TRTRI) ? trtri_dev(uplo, diag, N, dA, lda)
                              : (op == OP_LAUUM) ? lauum_dev(uplo, N, dA, lda) : potri_dev(uplo, N, dA, lda);
    if (!dev && rc >= 0) {
        if (int r2 = stage_out(A, LDA, dA, N, N, s)) return r2;
        CHB_CUDA(cudaStreamSynchronize(s));
    }
    return rc;
}

// Tile layout: the descriptor's tiles <-> a dense device copy.
__global__ void tiles_dense_kernel(double *base, const int64_t *off, const int *ld, int mt, int mb, int nb, int N,
                                   double *D, int to_dense) {
    const int64_t total = (int64_t)N * N;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(idx % N), j = (int)(idx / N);
        const int m = i / mb, n = j / nb;
        double *t = base + off[m + (int64_t)mt * n] + (i - m * mb) + (int64_t)(j - n * nb) * ld[m];
        if (to_dense) D[i + (int64_t)j * N] = *t;
        else *t = D[i + (int64_t)j * N];
    }
}

int inverse_tile(InvOp op, cham_uplo_t uplo, cham_diag_t diag, CHAM_desc_t *A) {
    if (!A || A->dtyp != ChamRealDouble || A->m != A->n || A->mb != A->nb) return CHAMELEON_ERR_ILLEGAL_VALUE;
    const int N = A->n;
    if (N == 0) return 0;
    if (int rc = desc_upload(A)) return rc;
    cudaStream_t s = ctx().stream;
    double *D = staging(1, (size_t)N * N * sizeof(double));
    if (!D) return CHAMELEON_ERR_OUT_OF_RESOURCES;
    const DescDev &dv = priv(A)->dev;
    tiles_dense_kernel<<<grid_for((int64_t)N * N), 256, 0, s>>>((double *)A->mat, dv.off, dv.ld, A->mt, A->mb, A->nb,
                                                                N, D, 1);
    CHB_LAUNCHED(1);
    int rc = (op == OP_TRTRI) ? trtri_dev(uplo, diag, N, D, N)
                              : (op == OP_LAUUM) ? lauum_dev(uplo, N, D, N) : potri_dev(uplo, N, D, N);
    if (rc == 0) {
        tiles_dense_kernel<<<grid_for((int64_t)N * N), 256, 0, s>>>((double *)A->mat, dv.off, dv.ld, A->mt, A->mb,
                                                                    A->nb, N, D, 0);
        CHB_LAUNCHED(1);
        CHB_CUDA(cudaStreamSynchronize(s));
        if (int r2 = desc_sync_to_host(A)) return r2;
    }
    return rc;
}

}  // namespace chb

using namespace chb;

extern "C" {

// compute/ztrtri.c:ztrtri (LAPACK layout)
int CHAMELEON_dtrtri(cham_uplo_t uplo, cham_diag_t diag, int N, double *A, int LDA) {
    int rc = ensure_init();
    if (rc) return rc;
    if (uplo != ChamUpper && uplo != ChamLower) return -1;
    if (diag != ChamUnit && diag != ChamNonUnit) return -2;
    if (N < 0) return -3;
    if (LDA < std::max(1, N)) return -5;
    if (N == 0) return 0;
    return inverse_lapack(OP_TRTRI, uplo, diag, N, A, LDA);
}
int CHAMELEON_dlauum(cham_uplo_t uplo, int N, double *A, int LDA) {
    int rc = ensure_init();
    if (rc) return rc;
    if (uplo != ChamUpper && uplo != ChamLower) return -1;
    if (N < 0) return -2;
    if (LDA < std::max(1, N)) return -4;
    if (N == 0) return 0;
    return inverse_lapack(OP_LAUUM, uplo, ChamNonUnit, N, A, LDA);
}
int CHAMELEON_dpotri(cham_uplo_t uplo, int N, double *A, int LDA) {
    int rc = ensure_init();
    if (rc) return rc;
    if (uplo != ChamUpper && uplo != ChamLower) return -1;
    if (N < 0) return -2;
    if (LDA < std::max(1, N)) return -4;
    if (N == 0) return 0;
    return inverse_lapack(OP_POTRI, uplo, ChamNonUnit, N, A, LDA);
}
// compute/zpotrimm.c:72 (LAPACK layout): A, B, C host or device arrays.
int CHAMELEON_dpotrimm(cham_uplo_t uplo, int N, double *A, int LDA, double *B, int LDB, double *C, int LDC) {
    int rc = ensure_init();
    if (rc) return rc;
    if (uplo != ChamUpper && uplo != ChamLower) return -1;
    if (N < 0) return -2;
    if (LDA < std::max(1, N)) return -4;
    if (LDB < std::max(1, N)) return -6;
    if (LDC < std::max(1, N)) return -8;
    if (N == 0) return 0;
    cudaStream_t s = ctx().stream;
    auto on_dev = [](const void *p) {
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged;
    };
    const bool da = on_dev(A), db = on_dev(B), dc = on_dev(C);
    double *dA = A, *dB = B, *dC = C;
    int lda = LDA, ldb = LDB, ldc = LDC;
    if (!da) {
        if (!(dA = stage_in(0, A, LDA, N, N, s))) return CHAMELEON_ERR_OUT_OF_RESOURCES;
        lda = N;
    }
    if (!db) {
        if (!(dB = work(&g_w3, &g_w3_bytes, (size_t)N * N * sizeof(double)))) return CHAMELEON_ERR_OUT_OF_RESOURCES;
        CHB_CUDA(cudaMemcpy2DAsync(dB, (size_t)N * sizeof(double), B, (size_t)LDB * sizeof(double),
                                   (size_t)N * sizeof(double), N, cudaMemcpyHostToDevice, s));
        ldb = N;
    }
    if (!dc) {
        if (!(dC = work(&g_w4, &g_w4_bytes, (size_t)N * N * sizeof(double)))) return CHAMELEON_ERR_OUT_OF_RESOURCES;
        ldc = N;
    }
    rc = potrimm_dev(uplo, N, dA, lda, dB, ldb, dC, ldc);
    if (rc >= 0) {
        if (!da)
            if (int r2 = stage_out(A, LDA, dA, N, N, s)) return r2;
        if (!dc && rc == 0)
            CHB_CUDA(cudaMemcpy2DAsync(C, (size_t)LDC * sizeof(double), dC, (size_t)N * sizeof(double),
                                       (size_t)N * sizeof(double), N, cudaMemcpyDeviceToHost, s));
        CHB_CUDA(cudaStreamSynchronize(s));
    }
    return rc;
}

// compute/zpotrimm.c:202 (tile layout): square descriptors of one order.
int CHAMELEON_dpotrimm_Tile(cham_uplo_t uplo, CHAM_desc_t *A, CHAM_desc_t *B, CHAM_desc_t *C) {
    int rc = ensure_init();
    if (rc) return rc;
    if (uplo != ChamUpper && uplo != ChamLower) return CHAMELEON_ERR_ILLEGAL_VALUE;
    for (CHAM_desc_t *d : {A, B, C})
        if (!d || d->dtyp != ChamRealDouble || d->m != d->n || d->mb != d->nb) return CHAMELEON_ERR_ILLEGAL_VALUE;
    if (B->n != A->n || C->n != A->n) return CHAMELEON_ERR_ILLEGAL_VALUE;
    const int N = A->n;
    if (N == 0) return 0;
    cudaStream_t s = ctx().stream;
    double *DA = staging(1, (size_t)N * N * sizeof(double));
    double *DB = work(&g_w3, &g_w3_bytes, (size_t)N * N * sizeof(double));
    double *DC = work(&g_w4, &g_w4_bytes, (size_t)N * N * sizeof(double));
    if (!DA || !DB || !DC) return CHAMELEON_ERR_OUT_OF_RESOURCES;
    for (CHAM_desc_t *d : {A, B, C})
        if ((rc = desc_upload(d))) return rc;
    auto conv = [&](CHAM_desc_t *d, double *D, int to_dense) {
        const DescDev &dv = priv(d)->dev;
        tiles_dense_kernel<<<grid_for((int64_t)N * N), 256, 0, s>>>((double *)d->mat, dv.off, dv.ld, d->mt, d->mb,
                                                                    d->nb, N, D, to_dense);
        CHB_LAUNCHED(1);
    };
    conv(A, DA, 1);
    conv(B, DB, 1);
    rc = potrimm_dev(uplo, N, DA, N, DB, N, DC, N);
    if (rc == 0) {
        conv(A, DA, 0);
        conv(C, DC, 0);
        CHB_CUDA(cudaStreamSynchronize(s));
        if (int r2 = desc_sync_to_host(A)) return r2;
        if (int r2 = desc_sync_to_host(C)) return r2;
    }
    return rc;
}

int CHAMELEON_dtrtri_Tile(cham_uplo_t uplo, cham_diag_t diag, CHAM_desc_t *A) {
    int rc = ensure_init();
    if (rc) return rc;
    if ((uplo != ChamUpper && uplo != ChamLower) || (diag != ChamUnit && diag != ChamNonUnit))
        return CHAMELEON_ERR_ILLEGAL_VALUE;
    return inverse_tile(OP_TRTRI, uplo, diag, A);
}
int CHAMELEON_dlauum_Tile(cham_uplo_t uplo, CHAM_desc_t *A) {
    int rc = ensure_init();
    if (rc) return rc;
    if (uplo != ChamUpper && uplo != ChamLower) return CHAMELEON_ERR_ILLEGAL_VALUE;
    return inverse_tile(OP_LAUUM, uplo, ChamNonUnit, A);
}
int CHAMELEON_dpotri_Tile(cham_uplo_t uplo, CHAM_desc_t *A) {
    int rc = ensure_init();
    if (rc) return rc;
    if (uplo != ChamUpper && uplo != ChamLower) return CHAMELEON_ERR_ILLEGAL_VALUE;
    return inverse_tile(OP_POTRI, uplo, ChamNonUnit, A);
}

// ---- LAPACKE interface (lapack_api/src/lapack_z*.c after z->d) -------------
// The character arguments convert as lapack_api/src/lapack_api_common.c does:
// an illegal one prints the message and becomes CHAMELEON_ERR_ILLEGAL_VALUE,
// which the routine behind it then rejects with its own argument index.
static int lapacke_uplo(char c) {
    if (c == 'U' || c == 'u') return ChamUpper;
    if (c == 'L' || c == 'l') return ChamLower;
    fprintf(stderr, "CHAMELEON ERROR: %s(): %s\n", "chameleon_blastocblas_uplo",
            "illegal value of BLAS uplo parameter");
    return CHAMELEON_ERR_ILLEGAL_VALUE;
}
static int lapacke_diag(char c) {
    if (c == 'U' || c == 'u') return ChamUnit;
    if (c == 'N' || c == 'n') return ChamNonUnit;
    fprintf(stderr, "CHAMELEON ERROR: %s(): %s\n", "chameleon_blastocblas_diag",
            "illegal value of BLAS diag parameter");
    return CHAMELEON_ERR_ILLEGAL_VALUE;
}
#define CHB_LAPACKE_PROLOGUE(name)                                                                   \
    if (matrix_layout != CHAMELEON_LAPACK_COL_MAJOR) {                                               \
        fprintf(stderr, "CHAMELEON ERROR: %s(): %s\n", name, "illegal value of matrix_layout");      \
        return -1;                                                                                   \
    }                                                                                                \
    const int ul = lapacke_uplo(uplo);

int CHAMELEON_lapacke_dposv(int matrix_layout, char uplo, int N, int NRHS, double *A, int lda, double *B, int ldb) {
    CHB_LAPACKE_PROLOGUE("CHAMELEON_lapacke_dposv");
    return CHAMELEON_dposv((cham_uplo_t)ul, N, NRHS, A, lda, B, ldb);
}
int CHAMELEON_lapacke_dpotrf(int matrix_layout, char uplo, int N, double *A, int lda) {
    CHB_LAPACKE_PROLOGUE("CHAMELEON_lapacke_dpotrf");
    return CHAMELEON_dpotrf((cham_uplo_t)ul, N, A, lda);
}
int CHAMELEON_lapacke_dpotrs(int matrix_layout, char uplo, int N, int NRHS, const double *A, int lda, double *B,
                             int ldb) {
    CHB_LAPACKE_PROLOGUE("CHAMELEON_lapacke_dpotrs");
    return CHAMELEON_dpotrs((cham_uplo_t)ul, N, NRHS, const_cast<double *>(A), lda, B, ldb);
}
int CHAMELEON_lapacke_dpotri(int matrix_layout, char uplo, int N, double *A, int lda) {
    CHB_LAPACKE_PROLOGUE("CHAMELEON_lapacke_dpotri");
    return CHAMELEON_dpotri((cham_uplo_t)ul, N, A, lda);
}
int CHAMELEON_lapacke_dlauum(int matrix_layout, char uplo, int N, double *A, int lda) {
    CHB_LAPACKE_PROLOGUE("CHAMELEON_lapacke_dlauum");
    return CHAMELEON_dlauum((cham_uplo_t)ul, N, A, lda);
}
int CHAMELEON_lapacke_dtrtri(int matrix_layout, char uplo, char diag, int N, double *A, int lda) {
    CHB_LAPACKE_PROLOGUE("CHAMELEON_lapacke_dtrtri");
    const int dg = lapacke_diag(diag);
    return CHAMELEON_dtrtri((cham_uplo_t)ul, (cham_diag_t)dg, N, A, lda);
}

// ---- Fortran LAPACK interface (gfortran names: lower case, trailing _) ----
void chameleon_lapack_dposv_(const char *uplo, const int *n, const int *nrhs, double *a, const int *lda, double *b,
                             const int *ldb, int *info) {
    *info = CHAMELEON_lapacke_dposv(CHAMELEON_LAPACK_COL_MAJOR, *uplo, *n, *nrhs, a, *lda, b, *ldb);
}
void chameleon_lapack_dpotrf_(const char *uplo, const int *n, double *a, const int *lda, int *info) {
    *info = CHAMELEON_lapacke_dpotrf(CHAMELEON_LAPACK_COL_MAJOR, *uplo, *n, a, *lda);
}
void chameleon_lapack_dpotrs_(const char *uplo, const int *n, const int *nrhs, const double *a, const int *lda,
                              double *b, const int *ldb, int *info) {
    *info = CHAMELEON_lapacke_dpotrs(CHAMELEON_LAPACK_COL_MAJOR, *uplo, *n, *nrhs, a, *lda, b, *ldb);
}
void chameleon_lapack_dpotri_(const char *uplo, const int *n, double *a, const int *lda, int *info) {
    *info = CHAMELEON_lapacke_dpotri(CHAMELEON_LAPACK_COL_MAJOR, *uplo, *n, a, *lda);
}
void chameleon_lapack_dlauum_(const char *uplo, const int *n, double *a, const int *lda, int *info) {
    *info = CHAMELEON_lapacke_dlauum(CHAMELEON_LAPACK_COL_MAJOR, *uplo, *n, a, *lda);
}
void chameleon_lapack_dtrtri_(const char *uplo, const char *diag, const int *n, double *a, const int *lda, int *info) {
    *info = CHAMELEON_lapacke_dtrtri(CHAMELEON_LAPACK_COL_MAJOR, *uplo, *diag, *n, a, *lda);
}

}  // extern "C"
