// potrf_smem.cuh -- Cholesky of an FP32 diagonal tile of order n <= 256 held
// entirely in shared memory, with the inverted 64 x 64 diagonal blocks.
//
// The diagonal-tile factorization is the critical path of the tile Cholesky
// DAG (compute/pzpotrf.c: potrf(k) -> trsm(m,k) -> update(k+1,k+1) ->
// potrf(k+1)).  The blocked tile kernels (rec.cuh) stream the tile through L2
// once per 64-column step; under the load of the trailing updates every such
// round trip costs microseconds, and their fully unrolled warp leaves are
// fetched from a busy L2 instruction by instruction.  Here the whole lower
// triangle (160 KB at n = 256) is loaded once, factored on chip by all 256
// threads with small loops, and written back once.
//
// Layout: the lower triangle by 64-wide block columns; block column b holds
// rows 64 b .. n-1, column-major with a padded leading dimension (blk_ld).  Right-looking over block columns:
//   leaf:     D_bb = L_bb L_bb^T and X_b = L_bb^-1 (the 64 x 64 leaf of
//             rec.cuh on a staged copy of the block)
//   panel:    L_ib = A_ib X_b^T                      (i > b)
//   trailing: A_ij -= L_ib L_jb^T                    (i >= j > b)
// (the panel and trailing products in FP32 FMA from shared memory)
// Same contract as CORE_spotrf on a lower view (coreblas/compute/core_zpotrf.c
// :75-81): lower triangle overwritten by L, upper untouched, LAPACK info; the
// inverted blocks go to invd (IB x IB, ld IB, zero outside the block), as the
// executor's panel solves expect.
#pragma once
#include "core.cuh"
#include "rec.cuh"

namespace chb {
namespace psm {

constexpr int MAXN = 256;   // largest tile order
constexpr int BW = 64;      // block-column width (= IB)
constexpr int LDI = rec::LDS;   // leading dimension of the staged block and its inverse

// Leading dimension of block column b: its rows rounded up to 32, plus 8 (a
// multiple of 4: the columns stay 16-byte aligned for the vector accesses).
__host__ __device__ constexpr int blk_ld(int n, int b) { return (((n - BW * b) + 31) & ~31) + 8; }
__host__ __device__ constexpr int blk_off(int n, int b) {
    int o = 0;
    for (int i = 0; i < b; ++i) o += BW * blk_ld(n, i);
    return o;
}
// Shared memory: the block columns, the staged diagonal block and its inverse
// (floats; 16-byte aligned base).
constexpr int SMEM_FLOATS = blk_off(MAXN, MAXN / BW) + 2 * BW * LDI + 8;
constexpr size_t SMEM_BYTES = (size_t)SMEM_FLOATS * sizeof(float);

// Cholesky of the nbk x nbk block (nbk <= 64) at D (column-major, ld ldd,
// lower triangle) in place, and its inverse into Xs (ld LDI, 64 x 64: zeros
// above the diagonal and outside nbk).  The block is staged, identity-padded,
// into sD (64 x LDI) for the 64 x 64 leaf of rec.cuh.  Returns LAPACK info.
// All 256 threads; ends with a barrier.
static __device__ __noinline__ int leaf(float *D, int ldd, int nbk, float *sD) {
    float *Xs = sD + BW * LDI;   // the leaf's inverse follows the staged block
    for (int idx = threadIdx.x; idx < 64 * 64; idx += NT_CTA) {
        const int r = idx & 63, c = idx >> 6;
        float v = (r == c) ? 1.f : 0.f;
        if (r < nbk && c < nbk) v = (r >= c) ? D[c * ldd + r] : 0.f;
        sD[c * LDI + r] = v;
    }
    __syncthreads();
    const int info = rec::leaf64_core<float, true>(sD, Xs, nbk);
    if (info) return info;
    for (int idx = threadIdx.x; idx < 64 * 64; idx += NT_CTA) {
        const int r = idx & 63, c = idx >> 6;
        if (r < nbk && c < nbk) {
            if (r >= c) D[c * ldd + r] = sD[c * LDI + r];
        } else {
            Xs[c * LDI + r] = 0.f;   // the identity padding's inverse
        }
    }
    __syncthreads();
    return 0;
}

// acc(i, c) = sum_{k < 64} Xm(i, k) Ym(c, k) for rows i < M (M <= 192) and
// columns c < 64, in FP32 FMA.  Xm: column-major (ld ldx), Ym(c, k) at
// Ym[k * ldy + c]; 16-byte aligned columns.  Thread (r = tid % 16, q = tid /
// 16) owns rows 4 r + 64 i .. + 3 (i < 3) and columns 4 q .. + 3, so that four
// 16-byte loads feed 48 FMAs.  The products are small and their operands are
// in shared memory, where the tensor-core form (three TF32 products per pair)
// spent its time on splitting operands and rounded more: order 256 137 us with
// it, 112 us with FMA.  Threads whose rows are all >= M, or columns >= N, sum
// those of row or column 0 instead (what follows may be written meanwhile);
// neither is stored.
struct Frag {
    float v[3][4][4];   // [row group][column][row]
};
static __device__ __forceinline__ void gemm64(Frag &acc, const float *Xm, int ldx, int M, const float *Ym, int ldy,
                                              int N) {
    const int r0 = 4 * (threadIdx.x & 15), c0 = 4 * (threadIdx.x >> 4);
    const float *x = Xm + r0, *y = Ym + (c0 < N ? c0 : 0);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc.v[i][j][e] = 0.f;
    const int ng = (M + 63) / 64;   // row groups (uniform across the CTA)
    const float *xl = Xm + (r0 + 64 * (ng - 1) < M ? r0 + 64 * (ng - 1) : 0);   // the last one
    auto sweep = [&](auto groups) {
        constexpr int G = decltype(groups)::value;
#pragma unroll 4
        for (int k = 0; k < BW; ++k) {
            const float4 b = *reinterpret_cast<const float4 *>(y + k * ldy);
#pragma unroll
            for (int i = 0; i < G; ++i) {
                const float4 a = *reinterpret_cast<const float4 *>((i == G - 1 ? xl : x + 64 * i) + k * ldx);
                const float bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc.v[i][j][0] = fmaf(a.x, bb[j], acc.v[i][j][0]);
                    acc.v[i][j][1] = fmaf(a.y, bb[j], acc.v[i][j][1]);
                    acc.v[i][j][2] = fmaf(a.z, bb[j], acc.v[i][j][2]);
                    acc.v[i][j][3] = fmaf(a.w, bb[j], acc.v[i][j][3]);
                }
            }
        }
    };
    if (ng == 1) sweep(std::integral_constant<int, 1>{});
    else if (ng == 2) sweep(std::integral_constant<int, 2>{});
    else sweep(std::integral_constant<int, 3>{});
}

// C(r, c) = acc (SUB: C -= acc) for r < M, c < N (and r >= c when lower), C
// column-major in shared memory (ld ldc, 16-byte aligned columns): four rows
// as one 16-byte access where all of them are stored.
template <bool SUB>
static __device__ __forceinline__ void frag_store(const Frag &acc, float *C, int ldc, int M, int N, bool lower) {
    const int r0 = 4 * (threadIdx.x & 15), c0 = 4 * (threadIdx.x >> 4);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = r0 + 64 * i, c = c0 + j;
            if (r >= M || c >= N) continue;
            const float(&v)[4] = acc.v[i][j];
            float *q = C + c * ldc + r;
            if (r + 3 < M && (!lower || r >= c)) {
                float4 o = make_float4(v[0], v[1], v[2], v[3]);
                if (SUB) {
                    const float4 w = *reinterpret_cast<const float4 *>(q);
                    o = make_float4(w.x - v[0], w.y - v[1], w.z - v[2], w.w - v[3]);
                }
                *reinterpret_cast<float4 *>(q) = o;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (r + e < M && (!lower || r + e >= c)) q[e] = SUB ? q[e] - v[e] : v[e];
            }
        }
}

// Factor the n x n lower view T (n <= MAXN) through shared memory `sm`
// (SMEM_BYTES, 16-byte aligned); inverted blocks to invd.  Returns info.
// All 256 threads.
static __device__ __noinline__ int potrf(const ViewF &T, int n, float *invd, float *sm, unsigned *ph = nullptr) {
    const int tid = threadIdx.x;
    const int nb = (n + BW - 1) / BW;
    float *sDl = sm + blk_off(n, nb);   // staged leaf block, then its inverse
    float *Xs = sDl + BW * LDI;
    // tracing (ph != null): thread 0 adds the clock cycles of the leaves, the
    // panel products and the trailing updates (with the load and the
    // write-back) to ph[0..2]
    long long c0 = (ph && tid == 0) ? clock64() : 0;
    auto lap = [&](int i) {
        if (ph && tid == 0) {
            const long long c1 = clock64();
            ph[i] += (unsigned)(c1 - c0);
            c0 = c1;
        }
    };
    // Load block column b (rows 64 b .. n-1, all 64 columns; the part above
    // the diagonal is never read).  A column-major tile with 16-byte aligned
    // columns is copied with 16-byte cp.async, every copy of the tile in
    // flight at once; otherwise element by element, coalesced along the
    // contiguous direction, eight loads in flight per thread.
    const bool colmajor = (T.rs == 1);
    const bool vec = colmajor && ((reinterpret_cast<uintptr_t>(T.p) & 15) == 0) && (T.cs % 4 == 0);
    if (vec) {
        for (int b = 0; b < nb; ++b) {
            const int rows = n - BW * b, ld = blk_ld(n, b), nq = ld / 4, wb = min(BW, n - BW * b);
            float *Sb = sm + blk_off(n, b);
            for (int idx = tid; idx < nq * wb; idx += NT_CTA) {
                const int q = idx % nq, c = idx / nq, r = 4 * q;
                const int nv = max(0, min(4, rows - r));
                const float *src = T.at(BW * b + r, BW * b + c);
                cp_async16(Sb + c * ld + r, nv ? src : T.p, nv * 4);
            }
        }
        cp_async_commit();
        cp_async_wait<0>();
    } else {
        for (int idx0 = tid; idx0 < n * n; idx0 += 8 * NT_CTA) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int idx = idx0 + u * NT_CTA;
                const int i = colmajor ? idx % n : idx / n, j = colmajor ? idx / n : idx % n;
                v[u] = (idx < n * n && i >= j) ? *T.at(i, j) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int idx = idx0 + u * NT_CTA;
                const int i = colmajor ? idx % n : idx / n, j = colmajor ? idx / n : idx % n;
                if (idx < n * n && i >= j) {
                    const int b = j / BW;
                    sm[blk_off(n, b) + (j - BW * b) * blk_ld(n, b) + (i - BW * b)] = v[u];
                }
            }
        }
    }
    __syncthreads();
    lap(2);
    int info = 0;
    for (int b = 0; b < nb; ++b) {
        float *Sb = sm + blk_off(n, b);
        const int ldb = blk_ld(n, b), nbk = min(BW, n - BW * b);
        const int linfo = leaf(Sb, ldb, nbk, sDl);
        lap(0);
        if (linfo) {
            info = BW * b + linfo;
            break;
        }
        float *inv = invd + (int64_t)b * IB * IB;
        for (int idx = tid; idx < IB * IB; idx += NT_CTA) inv[idx] = Xs[(idx / IB) * LDI + (idx % IB)];
        const int M = n - BW * (b + 1);   // rows below the diagonal block
        if (M <= 0) break;
        // panel: L_ib = A_ib X_b^T, computed in registers, then stored in place
        {
            Frag acc;
            gemm64(acc, Sb + BW, ldb, M, Xs, LDI, BW);   // X_b(c, k) at Xs[k * LDI + c]
            __syncthreads();
            frag_store<false>(acc, Sb + BW, ldb, M, nbk, false);
            __syncthreads();
        }
        lap(1);
        // trailing: block columns c > b
        for (int cb = b + 1; cb < nb; ++cb) {
            float *Sc = sm + blk_off(n, cb);
            const int ldc = blk_ld(n, cb), Mc = n - BW * cb, wc = min(BW, n - BW * cb);
            Frag acc;
            // rows i >= 64 cb of panel b, against its rows 64 cb .. 64 cb + 63
            gemm64(acc, Sb + BW * (cb - b), ldb, Mc, Sb + BW * (cb - b), ldb, wc);
            frag_store<true>(acc, Sc, ldc, Mc, wc, true);
        }
        __syncthreads();
        lap(2);
    }
    // write back the lower triangle, a line of the tile's contiguous direction
    // per warp and step, so that no index needs a division (the upper triangle
    // is never written)
    const int warp = tid >> 5, lane = tid & 31;
    for (int line = warp; line < n; line += NT_CTA / 32) {
        if (colmajor) {
            const int b = line / BW, ld = blk_ld(n, b);
            const float *q = sm + blk_off(n, b) + (line - BW * b) * ld - BW * b;
            float *g = T.at(0, line);
#pragma unroll 4
            for (int r = (line & ~31) + lane; r < n; r += 32)
                if (r >= line) g[r] = q[r];
        } else {
            float *g = T.at(line, 0);
            for (int c = lane; c <= line; c += 32) {
                const int b = c / BW;
                g[c] = sm[blk_off(n, b) + (c - BW * b) * blk_ld(n, b) + (line - BW * b)];
            }
        }
    }
    __syncthreads();
    lap(2);
    return info;
}

}  // namespace psm
}  // namespace chb
