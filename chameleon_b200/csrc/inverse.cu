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
//           gets X21 = -X22 (L21 X11), two launches for all pairs together;
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

// X (column-major, ld ldx) gets the inverted HB x HB diagonal blocks of the
// lower L (n x n), one CTA each; unit: with an implied unit diagonal.
__global__ void __launch_bounds__(NT_CTA, 1) diag_inv_kernel(View L, int n, int unit, double *X, int64_t ldx) {
    extern __shared__ __align__(128) double smem[];
    const int j0 = blockIdx.x * HB, nb = min(HB, n - j0);
    rec::leaf64_load(L.sub(j0, j0), nb, smem);
    double *sX = smem + 64 * rec::LDS;
    rec::leaf64_core<double, false>(smem, sX, nb, unit != 0);
    double *D = X + j0 + (int64_t)j0 * ldx;
    for (int idx = threadIdx.x; idx < nb * nb; idx += NT_CTA)
        D[idx % nb + (int64_t)(idx / nb) * ldx] = sX[idx % nb + (idx / nb) * rec::LDS];
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
// *skip is a valid index (a singular factor).
__global__ void __launch_bounds__(NT_CTA, INV_CTAS_PER_SM)
    lauum_kernel(View X, int n, View C, const int *skip) {
    extern __shared__ __align__(128) double smem[];
    if (skip && *skip != INT_MAX) return;
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
// zero_upper; the diagonal is left out when skip_diag; nothing when *skip is a
// valid index.  Block (x, y): 64 rows of 4 columns per step, along the
// destination's contiguous direction.
__global__ void tri_copy_kernel(View S, View D, int n, int zero_upper, int skip_diag, const int *skip) {
    if (skip && *skip != INT_MAX) return;
    const bool cm = D.rs == 1;
    for (int y = blockIdx.y; y < n; y += gridDim.y)
        for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < n; x += gridDim.x * blockDim.x) {
            const int i = cm ? x : y, j = cm ? y : x;
            if (i < j ? !zero_upper : (i == j && skip_diag)) continue;
            *D.at(i, j) = i >= j ? *S.at(i, j) : 0.0;
        }
}

// *first = min over i of (i + 1) with A(i,i) == 0 (INT_MAX: none).
__global__ void flag_kernel(int *first) {
    if (threadIdx.x == 0) *first = INT_MAX;
}
__global__ void zero_diag_kernel(View A, int N, int *first) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
        if (*A.at(i, i) == 0.0) atomicMin(first, i + 1);
}

namespace {
int grid_for(int64_t total) { return (int)std::min<int64_t>(std::max<int64_t>((total + 255) / 256, 1), 148 * 16); }

// A handle of the tile ABI on the library stream (kept).
cublasHandle_t lib_handle() {
    static cublasHandle_t h = nullptr;
    if (!h && CHAM_B200_Handle_Create(&h, ctx().stream) != 0) h = nullptr;
    return h;
}

double *g_w1 = nullptr, *g_w2 = nullptr, *g_w3 = nullptr, *g_w4 = nullptr;
size_t g_w1_bytes = 0, g_w2_bytes = 0, g_w3_bytes = 0, g_w4_bytes = 0;
int *g_flag = nullptr;

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
    CHB_CUDA(cudaFuncSetAttribute(diag_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(2 * IB * LEAF_LD * sizeof(double))));
    done = true;
    return 0;
}

static void tri_copy(View S, View D, int N, int zero_upper, int skip_diag, const int *skip, cudaStream_t s) {
    const dim3 grid((N + 255) / 256, std::min(N, 2048));
    tri_copy_kernel<<<grid, 256, 0, s>>>(S, D, N, zero_upper, skip_diag, skip);
    CHB_LAUNCHED(1);
}

// Workspace leading dimension: even (16-byte copies of the products' operands)
// and not a multiple of a power of two for the common orders.
static int64_t work_ld(int N) { return (N + 1) / 2 * 2 + 2; }

// The inverse of the lower L (view of order N) into the first workspace
// (column-major, ld work_ld(N), zeros above the diagonal of every HB-block);
// g_flag = the first zero diagonal entry (INT_MAX: none, or unit).  Stream
// operations only; returns the workspace.
static int trtri_work(View L, cham_diag_t diag, int N, cudaStream_t s, double **Xp) {
    if (int rc = inv_attrs()) return rc;
    if (!g_flag && !(g_flag = (int *)dev_alloc(sizeof(int)))) return CHAMELEON_ERR_OUT_OF_RESOURCES;
    const int64_t ld = work_ld(N);
    double *X = work(&g_w1, &g_w1_bytes, (size_t)ld * N * sizeof(double));
    double *T = N > HB ? work(&g_w2, &g_w2_bytes, (size_t)ld * N * sizeof(double)) : X;
    if (!X || !T) return CHAMELEON_ERR_OUT_OF_RESOURCES;
    flag_kernel<<<1, 32, 0, s>>>(g_flag);
    CHB_LAUNCHED(1);
    if (diag == ChamNonUnit) {
        zero_diag_kernel<<<grid_for(N), 256, 0, s>>>(L, N, g_flag);
        CHB_LAUNCHED(1);
    }
    diag_inv_kernel<<<(N + HB - 1) / HB, NT_CTA, 2 * IB * LEAF_LD * sizeof(double), s>>>(L, N, diag == ChamUnit, X, ld);
    CHB_LAUNCHED(1);
    for (int64_t h = HB; h < N; h *= 2) {
        // pairs with any rows in their second block
        const int pairs = (int)((N - h + 2 * h - 1) / (2 * h)), nb = (int)(h / HB);
        for (int first = 1; first >= 0; --first)
            trtri_pair_kernel<<<dim3(nb, nb, pairs), NT_CTA, CfgInv::SMEM_BYTES, s>>>(L, N, (int)h, X, T, ld, first);
        CHB_LAUNCHED(2);
    }
    CHB_CUDA(cudaGetLastError());
    *Xp = X;
    return 0;
}

static int read_flag(int *first, cudaStream_t s) {
    CHB_CUDA(cudaMemcpyAsync(first, g_flag, sizeof(int), cudaMemcpyDeviceToHost, s));
    CHB_CUDA(cudaStreamSynchronize(s));
    return 0;
}

// The three operations on a device column-major A (ld lda), on the library
// stream; synchronous.  Return LAPACK's info (> 0) or a CHAMELEON_ERR_* code.
int trtri_dev(cham_uplo_t uplo, cham_diag_t diag, int N, double *A, int lda) {
    cudaStream_t s = ctx().stream;
    const View L = lower_view(uplo, A, lda);
    double *X = nullptr;
    if (int rc = trtri_work(L, diag, N, s, &X)) return rc;
    tri_copy(View{X, 1, work_ld(N)}, L, N, 0, diag == ChamUnit, g_flag, s);
    int first = INT_MAX;
    if (int rc = read_flag(&first, s)) return rc;
    return first != INT_MAX ? first : 0;   // singular: A is not modified
}

int lauum_dev(cham_uplo_t uplo, int N, double *A, int lda) {
    cudaStream_t s = ctx().stream;
    if (int rc = inv_attrs()) return rc;
    const View L = lower_view(uplo, A, lda);
    const int64_t ld = work_ld(N);
    double *T = work(&g_w1, &g_w1_bytes, (size_t)ld * N * sizeof(double));
    if (!T) return CHAMELEON_ERR_OUT_OF_RESOURCES;
    tri_copy(L, View{T, 1, ld}, N, 1, 0, nullptr, s);
    const int nb = (N + HB - 1) / HB;
    lauum_kernel<<<nb * (nb + 1) / 2, NT_CTA, CfgInv::SMEM_BYTES, s>>>(View{T, 1, ld}, N, L, nullptr);
    CHB_LAUNCHED(1);
    CHB_CUDA(cudaGetLastError());
    CHB_CUDA(cudaStreamSynchronize(s));
    return 0;
}

int potri_dev(cham_uplo_t uplo, int N, double *A, int lda) {
    cudaStream_t s = ctx().stream;
    const View L = lower_view(uplo, A, lda);
    double *X = nullptr;
    if (int rc = trtri_work(L, ChamNonUnit, N, s, &X)) return rc;
    const int nb = (N + HB - 1) / HB;
    lauum_kernel<<<nb * (nb + 1) / 2, NT_CTA, CfgInv::SMEM_BYTES, s>>>(View{X, 1, work_ld(N)}, N, L, g_flag);
    CHB_LAUNCHED(1);
    CHB_CUDA(cudaGetLastError());
    int first = INT_MAX;
    if (int rc = read_flag(&first, s)) return rc;
    return first != INT_MAX ? first : 0;   // singular: A is not modified
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
