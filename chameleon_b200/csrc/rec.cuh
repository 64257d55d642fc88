// rec.cuh -- recursive diagonal-tile Cholesky with the explicit tile inverse.
//
// The diagonal-tile POTRF is on the critical path of the tile Cholesky DAG
// (compute/pzpotrf.c: potrf(k) -> trsm(m,k) -> update(k+1,k+1) -> potrf(k+1)),
// so its latency, not its flops, bounds the factorization.  This variant
// factors an n x n tile (n <= 1024) by 2 x 2 recursion
//
//     [A11    ]   [L11    ]            L21 = A21 X11^T      (X11 = L11^-1)
//     [A21 A22] = [L21 L22] [..]^T,    A22 -= L21 L21^T,     L22 = chol(A22)
//
// and assembles the full inverse X = L^-1 on the way up
//
//     X21 = -X22 (L21 X11),
//
// so that every off-diagonal step is one GEMM-shaped pass (cta_gemm on the
// tensor cores).  The recursion ends in a 64 x 64 leaf (leaf64_core).
// With the full inverse, the panel solve A(m,k) <- A(m,k) L(k,k)^-T and the
// diagonal solves of the forward / backward substitutions are one GEMM each
// (apply_inv_right / apply_inv_left), done in place by ordering the output
// blocks so that no block is overwritten before it has been read.
//
// Using the explicit inverse of a whole tile trades the backward stability of
// a substitution for fewer dependent steps; the mixed-precision solver runs it
// in FP32 and its FP64 refinement restores the FP64 backward error.  The FP64
// substitutions, which nothing refines, use full inverses of well-conditioned
// tiles only (XINV_COND, executor.cuh).
#pragma once
#include "core.cuh"

namespace chb {
namespace rec {

// ---------------------------------------------------------------------------
// The 64 x 64 leaf: Cholesky factor and inverse of one diagonal block held in
// shared memory, by the whole CTA.
//
// It is the longest serial chain of every factorization here, so what bounds
// it is latency: 64 dependent pivots.  The block is factored by 8-wide panels,
// and the pivot chain is kept in registers.  Warp 0 owns the chain: every lane
// reads the panel's 8 x 8 diagonal block (36 broadcast loads) and factors it
// redundantly, so that consecutive pivots need no exchange between lanes (one
// reciprocal, one product and one FMA each), while it carries two rows of the panel along.
// After panel p the other warps bring block column p + 1 up to date, one 8 x 8
// tile each, and hand it to warp 0; while warp 0 factors panel p + 1 they
// update the remaining tiles (FP64 products on DMMA, FP32 ones on FMA).  The
// inverse trails the factorization by one panel and hides behind it: W(I, J) =
// sum_k L(I, k) X(k, J) is accumulated in the place of X(I, J), and block row
// p is finished as X(p, J) = -L(p,p)^-1 W(p, J) once panel p is factored.  The
// tiles stay in shared memory and are dealt out over the warps: with a row of
// tiles in each warp's registers the static register indices made every pass
// a chain of branches, and the warp with the longest row set the time (FP64
// 19.2 K cycles, FP32 18.8 K; now 14.6 K and 13.8 K; four 32 x 32 one-warp
// sweeps before: 42.2 K and 33.3 K).
// ---------------------------------------------------------------------------
constexpr int LDS = LEAF_LD;  // leaf leading dimension: 4 mod 16 doubles (and 4 mod 32
                              // floats), so that MMA fragments and 16-byte column reads
                              // are free of bank conflicts
constexpr int PW = 8;         // panel width

// The same pointer with its address space known: a function that is not inlined
// and takes a generic pointer would otherwise compile every access to a generic
// load or store, which takes about twice the latency of a shared one.
template <class T>
__device__ __forceinline__ T *in_shared(T *p) {
    return static_cast<T *>(__cvta_shared_to_generic(__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void bar_sync(int id) { asm volatile("bar.sync %0, 256;\n" ::"r"(id) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id) { asm volatile("bar.arrive %0, 256;\n" ::"r"(id) : "memory"); }

// Reciprocal (rc) and reciprocal square root (rs) of a pivot to working
// precision: the hardware estimates c and q (20 bits for FP64, 22 for FP32) and
// the residuals e = 1 - d c and h = 1 - d q^2, from which 1 / d = c / (1 - e) and
// d^(-1/2) = q (1 - h)^(-1/2) by the geometric and the binomial series
//   1 + e + e^2 + ..,   1 + h / 2 + 3 h^2 / 8 + ..,
// cut after the second power (FP64: the rest is below 2^-58) or the first (FP32:
// below 2^-40).  e comes from one FMA; h carries the rounding of d q, half of
// which reaches rs.  With the last rounding, and u = 2^-53 or 2^-24, the relative
// errors are within 1.01 u (rc) and 1.6 u (rs).  The next pivot waits for rc only.
// The estimates flush to zero or overflow near the ends of the exponent range:
// false outside (and for a pivot that is not positive, or NaN).
__device__ __forceinline__ bool pivot_recip(double d, double &rc, double &rs) {
    double c, q;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(c) : "d"(d));
    const double e = fma(-d, c, 1.0);
    rc = fma(c * e, 1.0 + e, c);
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(q) : "d"(d));
    const double h = fma(-d * q, q, 1.0);
    rs = fma(q * h, fma(0.375, h, 0.5), q);
    return d > 1e-280 && d < 1e280;
}
__device__ __forceinline__ bool pivot_recip(float d, float &rc, float &rs) {
    float c, q;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(c) : "f"(d));
    rc = fmaf(c, fmaf(-d, c, 1.f), c);
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(d));
    rs = fmaf(0.5f * q, fmaf(-d * q, q, 1.f), q);
    return d > 1e-30f && d < 1e30f;
}

// Panel p (columns 8 p .. 8 p + 7) of the block at S by one warp: L in place,
// the reciprocals of its diagonal to rd, and for p > 0 the inverse of its
// diagonal block to X (same place): lane k < 8 then carries the unit row e_k
// instead of the finished row k, which the column operations turn into column
// k of the inverse.  The pivots run on d and its reciprocal (an LDL^T
// recurrence on the unscaled columns); the square roots stay off the chain.
// SAFE: any pivot, subnormal and infinite ones too; the first one that is not
// positive (NaN included) is reported in info (1-based) and replaced by 1.  !SAFE: returns false, with
// nothing written, when a pivot is not positive or too extreme for the
// estimates.
template <class T, bool SAFE>
__device__ __forceinline__ bool leaf_panel(T *S, T *X, int p, T *rd, int &info) {
    const int lane = threadIdx.x & 31;
    T *P = S + PW * p * LDS;
    const T *D0 = P + PW * p;
    T d[PW][PW];
#pragma unroll
    for (int k = 0; k < PW; ++k)
#pragma unroll
        for (int i = k; i < PW; ++i) d[i][k] = D0[i + k * LDS];
    const bool unit = p > 0 && lane < PW;
    T a0[PW], a1[PW];
#pragma unroll
    for (int k = 0; k < PW; ++k) {
        a0[k] = P[lane + k * LDS];
        a1[k] = P[lane + 32 + k * LDS];
        if (unit) a0[k] = (k == lane) ? T(1) : T(0);
    }
    __syncwarp();   // every lane has read the diagonal block before it is overwritten
    T rs[PW], root[PW];   // root: SAFE only
    bool ok = true;
#pragma unroll
    for (int c = 0; c < PW; ++c) {
        T rc;
        if (SAFE) {
            T dc = d[c][c];
            if (!(dc > T(0))) {
                if (info == 0) info = PW * p + c + 1;
                dc = T(1);
            }
            root[c] = sqrt(dc);
            rs[c] = T(1) / root[c];
        } else {
            ok = pivot_recip(d[c][c], rc, rs[c]) && ok;
        }
        // (w first: a product of two unscaled entries could leave the exponent
        // range; and SAFE scales by the root, since the reciprocal of a small
        // subnormal pivot overflows)
#pragma unroll
        for (int k = c + 1; k < PW; ++k) {
            const T w = d[k][c] * (SAFE ? rs[c] : rc);
            const T f = SAFE ? rs[c] : T(1);
#pragma unroll
            for (int i = k; i < PW; ++i) d[i][k] -= SAFE ? d[i][c] * f * w : d[i][c] * w;
            a0[k] -= SAFE ? a0[c] * f * w : a0[c] * w;
            a1[k] -= SAFE ? a1[c] * f * w : a1[c] * w;
        }
    }
    if (!SAFE && !ok) return false;
    // one guarded store per entry through a per-lane pointer and stride
    // (separate branches for the two destinations cost twice the panel's time)
    T *q = unit ? X + PW * p * (LDS + 1) + lane * LDS : P + lane;
    const int st = unit ? 1 : LDS, last0 = unit ? PW : lane - PW * p, last1 = lane + 32 - PW * p;
#pragma unroll
    for (int c = 0; c < PW; ++c) {
        T v0 = a0[c] * rs[c], v1 = a1[c] * rs[c];
        if (SAFE) {   // the diagonal entry: an infinite pivot has an infinite root
            if (!unit && lane == PW * p + c) v0 = root[c];
            if (lane + 32 == PW * p + c) v1 = root[c];
        }
        if (c <= last0) q[c * st] = v0;
        if (c <= last1) P[lane + 32 + c * LDS] = v1;
    }
    T r = rs[0];
#pragma unroll
    for (int c = 1; c < PW; ++c)
        if (lane == c) r = rs[c];
    if (lane < PW) rd[PW * p + lane] = r;
    return true;
}
template <class T>
__device__ __noinline__ int leaf_panel_safe(T *S, T *X, int p, T *rd, int info) {
    leaf_panel<T, true>(in_shared(S), in_shared(X), p, in_shared(rd), info);
    return info;
}

// Inverse of the 8 x 8 lower block L(p, p) into X (full, zeros above the
// diagonal), by one warp: lane c < 8 solves for column c.
template <class T>
__device__ __forceinline__ void leaf_dinv(const T *S, T *X, int p, const T *rd) {
    const int lane = threadIdx.x & 31;
    const T *D0 = S + PW * p * (LDS + 1);
    T *X0 = X + PW * p * (LDS + 1);
    T s[PW];
#pragma unroll
    for (int i = 0; i < PW; ++i) s[i] = (i == lane) ? T(1) : T(0);
#pragma unroll
    for (int i = 0; i < PW; ++i) {
        s[i] *= rd[PW * p + i];
#pragma unroll
        for (int m = i + 1; m < PW; ++m) s[m] -= D0[m + i * LDS] * s[i];
    }
    if (lane < PW) {
#pragma unroll
        for (int i = 0; i < PW; ++i) X0[i + lane * LDS] = s[i];
    }
    __syncwarp();
}

// An 8 x 8 tile in the registers of one warp, with the DMMA accumulator's
// layout for both types: lane (g, t) = (lane / 4, lane % 4) holds the entries
// (g, 2 t) and (g, 2 t + 1).  LeafA is the left operand of a product, K = 8;
// the right operand is read from shared memory, B(k, n) at q[n + k LDS] (rows
// of L) or q[k + n LDS] (columns of X).
template <class T>
struct LeafA;
template <>
struct LeafA<double> {
    double a0, a1;
    __device__ __forceinline__ void load(const double *q, double sign) {
        const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
        a0 = sign * q[g + t * LDS];
        a1 = sign * q[g + (t + 4) * LDS];
    }
};
template <>
struct LeafA<float> {
    float a[PW];
    __device__ __forceinline__ void load(const float *q, float sign) {
        const int g = (threadIdx.x & 31) >> 2;
#pragma unroll
        for (int k = 0; k < PW; ++k) a[k] = sign * q[g + k * LDS];
    }
};
__device__ __forceinline__ void leaf_mm_l(double (&c)[2], const LeafA<double> &a, const double *q) {
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    dmma884(c, a.a0, q[g + t * LDS]);
    dmma884(c, a.a1, q[g + (t + 4) * LDS]);
}
__device__ __forceinline__ void leaf_mm_x(double (&c)[2], const LeafA<double> &a, const double *q) {
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    dmma884(c, a.a0, q[t + g * LDS]);
    dmma884(c, a.a1, q[t + 4 + g * LDS]);
}
__device__ __forceinline__ void leaf_mm_l(float (&c)[2], const LeafA<float> &a, const float *q) {
    const int t = threadIdx.x & 3;
#pragma unroll
    for (int k = 0; k < PW; ++k) {
        const float2 b = *reinterpret_cast<const float2 *>(q + 2 * t + k * LDS);
        c[0] = fmaf(a.a[k], b.x, c[0]);
        c[1] = fmaf(a.a[k], b.y, c[1]);
    }
}
__device__ __forceinline__ void leaf_mm_x(float (&c)[2], const LeafA<float> &a, const float *q) {
    const int t = threadIdx.x & 3;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const float4 x = *reinterpret_cast<const float4 *>(q + (2 * t + e) * LDS);
        const float4 y = *reinterpret_cast<const float4 *>(q + (2 * t + e) * LDS + 4);
        c[e] = fmaf(a.a[0], x.x, c[e]);
        c[e] = fmaf(a.a[1], x.y, c[e]);
        c[e] = fmaf(a.a[2], x.z, c[e]);
        c[e] = fmaf(a.a[3], x.w, c[e]);
        c[e] = fmaf(a.a[4], y.x, c[e]);
        c[e] = fmaf(a.a[5], y.y, c[e]);
        c[e] = fmaf(a.a[6], y.z, c[e]);
        c[e] = fmaf(a.a[7], y.w, c[e]);
    }
}
template <class T>
__device__ __forceinline__ void leaf_get(const T *q, T (&c)[2]) {   // q: the tile's (0, 0), ld LDS
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    c[0] = q[g + 2 * t * LDS];
    c[1] = q[g + (2 * t + 1) * LDS];
}
template <class T>
__device__ __forceinline__ void leaf_put(T *q, const T (&c)[2]) {
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    q[g + 2 * t * LDS] = c[0];
    q[g + (2 * t + 1) * LDS] = c[1];
}
// Tile (I, J) of S -= L(I, p) L(J, p)^T.  FP32 sums the 8 products first, so that
// an entry is rounded at its own size once per panel and not once per column
// (order 64, dominant diagonal: error of the factor 5.1e-8, 8.3e-8 the other way).
template <class T>
__device__ __forceinline__ void leaf_tile_c(T *S, int p, int I, int J) {
    const T *P = S + PW * p * LDS;
    LeafA<T> a;
    T c[2], o[2] = {T(0), T(0)};
    a.load(P + PW * I, T(-1));
    leaf_get(S + PW * I + PW * J * LDS, c);
    if constexpr (sizeof(T) == 4) {
        leaf_mm_l(o, a, P + PW * J);
        c[0] += o[0];
        c[1] += o[1];
    } else {
        leaf_mm_l(c, a, P + PW * J);
    }
    leaf_put(S + PW * I + PW * J * LDS, c);
}
// Tile (I, J) of W += L(I, k) X(k, J)
template <class T>
__device__ __forceinline__ void leaf_tile_w(const T *S, T *X, int k, int I, int J) {
    LeafA<T> a;
    T c[2];
    a.load(S + PW * k * LDS + PW * I, T(1));
    leaf_get(X + PW * I + PW * J * LDS, c);
    leaf_mm_x(c, a, X + PW * k + PW * J * LDS);
    leaf_put(X + PW * I + PW * J * LDS, c);
}
// Tile (p, J) of X = -X(p, p) W(p, J)
template <class T>
__device__ __forceinline__ void leaf_tile_x(T *X, int p, int J) {
    T *q = X + PW * p + PW * J * LDS;
    LeafA<T> a;
    T c[2] = {T(0), T(0)};
    a.load(X + PW * p * (LDS + 1), T(-1));
    leaf_mm_x(c, a, q);
    __syncwarp();   // every lane has read W
    leaf_put(q, c);
}
// q-th tile (row, column) of a lower triangle of tiles, row-major
__device__ __forceinline__ void leaf_tri(int q, int &i, int &j) {
    i = (q >= 1) + (q >= 3) + (q >= 6) + (q >= 10) + (q >= 15) + (q >= 21);
    j = q - i * (i + 1) / 2;
}

// 64 x 64 leaf on shared memory.  sD (ld LDS, 16-byte aligned) holds the
// block's lower triangle, identity-padded from n to the next multiple of 8.
// FACT: sD is factored in place (L), else it already holds L (unit: with an
// implied unit diagonal).  sX (ld LDS) receives the inverse of
// the leading 8 ceil(n / 8) rows and columns, lower triangle, with zeros
// above the diagonal and everywhere else.  Returns LAPACK info.  Called by all
// threads; ends with a barrier.
template <class T, bool FACT>
__device__ __noinline__ int leaf64_core(T *sD, T *sX, int n, bool unit = false) {
    sD = in_shared(sD);
    sX = in_shared(sX);
    __shared__ int s_info;
    __shared__ T s_rd[64];
    const int tid = threadIdx.x, warp = tid >> 5;
    const int nblk = (n + PW - 1) / PW;
    __syncthreads();   // the callers' last writes of the block
    if (!FACT && tid < PW * nblk) s_rd[tid] = unit ? T(1) : T(1) / sD[tid + tid * LDS];
#pragma unroll 4
    for (int idx = tid; idx < 64 * 64; idx += NT_CTA) sX[(idx & 63) + (idx >> 6) * LDS] = T(0);
    __syncthreads();
    if (FACT && warp == 0) {
        int info = 0;
        for (int p = 0; p < nblk; ++p) {
            if (p > 0) bar_sync(1);   // block column p is up to date in sD
            if (!leaf_panel<T, false>(sD, sX, p, s_rd, info)) info = leaf_panel_safe<T>(sD, sX, p, s_rd, info);
            if (p == nblk - 1 && tid == 0) s_info = info;
            bar_arrive(2);
        }
    } else {
        const int nw = FACT ? 7 : 8, w = FACT ? warp - 1 : warp;
        if (!FACT && w < nblk) leaf_dinv(sD, sX, w, s_rd);
        for (int p = 0; p < nblk; ++p) {
            if (FACT) bar_sync(2);   // panel p is factored; rows < p of the inverse are done
            else __syncthreads();
            if (FACT) {
                if (p + 1 + w < nblk) leaf_tile_c(sD, p, p + 1 + w, p + 1);   // gates the next panel
                if (p + 1 < nblk) bar_arrive(1);
            }
            if (w < p) {   // block row p of the inverse, one tile per warp
                leaf_tile_w(sD, sX, p - 1, p, w);
                __syncwarp();
                leaf_tile_x(sX, p, w);
            }
            const int m = FACT ? max(0, nblk - p - 2) : 0, nc = m * (m + 1) / 2;
            const int rows = nblk - 1 - p;
            // the first tiles go to the warps that had none above
            for (int q = nw - 1 - w; q < nc + rows * p; q += nw) {
                if (q < nc) {
                    int i, j;
                    leaf_tri(q, i, j);
                    leaf_tile_c(sD, p, p + 2 + i, p + 2 + j);
                } else {
                    const int q2 = q - nc;
                    leaf_tile_w(sD, sX, p - 1, p + 1 + q2 / p, q2 % p);
                }
            }
            // the diagonal block of the inverse comes with the panel, except panel 0's
            if (FACT && p == 0 && w == 6) leaf_dinv(sD, sX, 0, s_rd);
        }
    }
    __syncthreads();
    return FACT ? s_info : 0;
}

// Identity-padded load of the lower n x n block of A (n <= 64) into sD (its
// first 8 ceil(n / 8) columns).
template <class T>
__device__ __forceinline__ void leaf64_load(const ViewT<T> &A, int n, T *sD) {
    const int np = (n + PW - 1) / PW * PW;
    const bool cm = A.rs == 1;   // along the contiguous direction, all loads in flight together
    T v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int idx = threadIdx.x + u * NT_CTA;
        const int r = cm ? idx & 63 : idx >> 6, c = cm ? idx >> 6 : idx & 63;
        v[u] = (r < n && c < n) ? ((r >= c) ? *A.at(r, c) : T(0)) : (r == c ? T(1) : T(0));
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int idx = threadIdx.x + u * NT_CTA;
        const int r = cm ? idx & 63 : idx >> 6, c = cm ? idx >> 6 : idx & 63;
        if (c < np) sD[r + c * LDS] = v[u];
    }
    __syncthreads();
}

// 64 x 64 leaf on global views: FACT factors the lower n x n block of A in
// place; the full inverse goes to X (n x n, written in full).
template <class T, bool FACT>
__device__ __noinline__ int leaf64(const ViewT<T> &A, const ViewT<T> &X, int n, T *smem) {
    T *sD = smem;              // 64 x LDS
    T *sX = smem + 64 * LDS;   // 64 x LDS
    leaf64_load(A, n, sD);
    const int info = leaf64_core<T, FACT>(sD, sX, n);
    if (info) return info;
    for (int idx = threadIdx.x; idx < n * n; idx += NT_CTA) {
        const int r = idx % n, c = idx / n;
        if (FACT && r >= c) *A.at(r, c) = sD[r + c * LDS];
        *X.at(r, c) = sX[r + c * LDS];
    }
    cta_sync();
    return 0;
}

// Blocked left-looking diagonal-tile Cholesky (lower view Tv, n x n) with the
// 64-wide leaf: per inner block, one GEMM brings in the columns to its left,
// the leaf factors and inverts it in shared memory, and the rows below are
// updated and multiplied by the leaf's inverse.  Writes L into the lower
// triangle (upper untouched) and the inverted diagonal blocks (IB x IB, ld
// IB, zero outside the block) into invd.  Returns LAPACK info.  Same
// contract as CORE_dpotrf (coreblas/compute/core_zpotrf.c:75-81).
// ph (optional, tracing): thread 0 adds the clock cycles spent in the block-
// column updates, the leaves and the panels to ph[0..2].
// PR: rows of one panel step (128 or 64).  LEAN: the leaf's two 64 x 64
// blocks share the GEMM staging area instead of following it (the leaf runs
// between GEMMs), so that smem needs only lean_smem_elems() -- the footprint
// that lets several CTAs share an SM.
template <class T, int SP>
constexpr size_t lean_smem_elems() {
    return Cfg64<T, SP>::SMEM_ELEMS > 2 * IB * LDS ? Cfg64<T, SP>::SMEM_ELEMS : 2 * IB * LDS;
}
template <class T, int SP, int PR = 128, bool LEAN = false>
__device__ int tile_potrf_blk(const ViewT<T> &Tv, int n, T *invd, T *smem, unsigned *ph = nullptr) {
    static_assert(PR == 128 || PR == 64, "panel rows");
    using CP = typename std::conditional<PR == 128, Cfg12864<T, SP>, Cfg64<T, SP>>::type;
    using CD = Cfg64<T, SP>;
    T *sD = LEAN ? smem : smem + CP::SMEM_ELEMS;   // cta_gemm ends with a barrier
    T *sX = sD + IB * LDS;
    long long c0 = (ph && threadIdx.x == 0) ? clock64() : 0;
    auto lap = [&](int i) {
        if (ph && threadIdx.x == 0) {
            const long long c1 = clock64();
            ph[i] += (unsigned)(c1 - c0);
            c0 = c1;
        }
    };
    for (int jb = 0; jb < n; jb += IB) {
        const int nbk = min(IB, n - jb);
        Acc<CD> acc;
        acc.zero();
        if (jb > 0) cta_gemm(acc, Tv.sub(jb, 0), Tv.sub(jb, 0), nbk, nbk, jb, smem);
        leaf64_load(Tv.sub(jb, jb), nbk, sD);
        acc.for_each([&](int r, int c, T v) {
            if (r < nbk && c < nbk && r >= c) sD[r + c * LDS] -= v;
        });
        lap(0);
        const int info = leaf64_core<T, true>(sD, sX, nbk);
        lap(1);
        if (info) return jb + info;
        T *inv = invd + (int64_t)(jb / IB) * IB * IB;
        for (int idx = threadIdx.x; idx < IB * IB; idx += NT_CTA) {
            const int r = idx % IB, c = idx / IB;
            if (r < nbk && c < nbk && r >= c) *Tv.at(jb + r, jb + c) = sD[r + c * LDS];
            inv[idx] = (r < nbk && c < nbk) ? sX[r + c * LDS] : T(0);
        }
        cta_sync();
        // panel below the inner diagonal block
        for (int r0 = jb + nbk; r0 < n; r0 += PR) {
            const int mr = min(PR, n - r0);
            Acc<CP> pa;
            if (jb > 0) {
                pa.zero();
                cta_gemm(pa, Tv.sub(r0, 0), Tv.sub(jb, 0), mr, nbk, jb, smem);
                pa.sub_from(Tv.sub(r0, jb), mr, nbk, false);
                cta_sync();
            }
            pa.zero();
            const ViewT<T> Inv{inv, 1, IB};
            cta_gemm(pa, Tv.sub(r0, jb), Inv, mr, nbk, nbk, smem);
            pa.store_to(Tv.sub(r0, jb), mr, nbk);
            cta_sync();
        }
        lap(2);
    }
    return 0;
}

// acc (rows x 64) = P X^T for the 64 x 64 blocks P and X (lower) in shared
// memory (ld LDS), on DMMA: warp w owns rows 8 w .. 8 w + 7, all 64 columns.
struct RowAcc {
    double v[8][2];   // tile J: entries (8 w + g, 8 J + 2 t), (.., + 1)
    template <class F>
    __device__ __forceinline__ void for_each(F &&f) const {
        const int w = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
#pragma unroll
        for (int J = 0; J < 8; ++J)
#pragma unroll
            for (int e = 0; e < 2; ++e) f(8 * w + g, 8 * J + 2 * t + e, v[J][e]);
    }
};
static __device__ __forceinline__ void mul_xt64(RowAcc &acc, const double *P, const double *X) {
    const int w = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
#pragma unroll
    for (int J = 0; J < 8; ++J) acc.v[J][0] = acc.v[J][1] = 0.0;
#pragma unroll
    for (int kb = 0; kb < 8; ++kb) {   // X(c, k) is zero for k > c
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = 8 * kb + 4 * h + t;
            const double a = P[8 * w + g + k * LDS];
#pragma unroll
            for (int J = 0; J < 8; ++J)
                if (J >= kb) dmma884(acc.v[J], a, X[8 * J + g + k * LDS]);
        }
    }
}

// tile_potrf_blk for FP64 with the work between the leaves kept on chip: the
// leaf's inverse stays in shared memory beside the GEMM staging area (which
// the leaf block and the panel block alias in turn), so that a 64-row panel
// step is one product with the columns to its left, one subtraction into
// shared memory and one product with the inverse from there -- instead of two
// products with a write and two reads of global memory between them (order 128
// alone: 51 -> 38 us).  Same
// contract; smem: fused_smem_elems() doubles, two CTAs per SM.
constexpr int fused_smem_elems() { return Cfg64<double>::SMEM_ELEMS + IB * LDS; }
static_assert(2 * IB * LDS <= Cfg64<double>::SMEM_ELEMS, "leaf and panel block inside the staging area");
static __device__ int tile_potrf_fused(const View &Tv, int n, double *invd, double *smem, unsigned *ph = nullptr) {
    using C = Cfg64<double>;
    double *sD = smem, *sP = smem + IB * LDS, *sX = smem + C::SMEM_ELEMS;
    long long c0 = (ph && threadIdx.x == 0) ? clock64() : 0;
    auto lap = [&](int i) {
        if (ph && threadIdx.x == 0) {
            const long long c1 = clock64();
            ph[i] += (unsigned)(c1 - c0);
            c0 = c1;
        }
    };
    for (int jb = 0; jb < n; jb += IB) {
        const int nbk = min(IB, n - jb);
        Acc<C> acc;
        acc.zero();
        if (jb > 0) cta_gemm(acc, Tv.sub(jb, 0), Tv.sub(jb, 0), nbk, nbk, jb, smem);
        leaf64_load(Tv.sub(jb, jb), nbk, sD);
        if (jb > 0)
            acc.for_each([&](int r, int c, double v) {
                if (r < nbk && c < nbk && r >= c) sD[r + c * LDS] -= v;
            });
        lap(0);
        const int info = leaf64_core<double, true>(sD, sX, nbk);
        lap(1);
        if (info) return jb + info;
        double *inv = invd + (int64_t)(jb / IB) * IB * IB;
        const bool cm = Tv.rs == 1;
#pragma unroll 4
        for (int idx = threadIdx.x; idx < IB * IB; idx += NT_CTA) {
            const int r = idx % IB, c = idx / IB;
            inv[idx] = (r < nbk && c < nbk) ? sX[r + c * LDS] : 0.0;
            const int tr = cm ? r : c, tc = cm ? c : r;   // along the tile's contiguous direction
            if (tr < nbk && tc < nbk && tr >= tc) *Tv.at(jb + tr, jb + tc) = sD[tr + tc * LDS];
        }
        cta_sync();
        for (int r0 = jb + nbk; r0 < n; r0 += IB) {
            const int mr = min(IB, n - r0);
            acc.zero();
            if (jb > 0) cta_gemm(acc, Tv.sub(r0, 0), Tv.sub(jb, 0), mr, nbk, jb, smem);
            // (nbk == 64 here: rows below mean the block column is full)
            const View A = Tv.sub(r0, jb);
            Acc<C> old;
            acc.for_each_idx([&](int a, int b, int e, int r, int c, double) {
                old.v[a][b][e] = r < mr ? __ldcg(A.at(r, c)) : 0.0;
            });
            acc.for_each_idx([&](int a, int b, int e, int r, int c, double v) {
                sP[r + c * LDS] = old.v[a][b][e] - v;
            });
            __syncthreads();
            RowAcc x;
            mul_xt64(x, sP, sX);
            x.for_each([&](int r, int c, double v) {
                if (r < mr) *A.at(r, c) = v;
            });
            cta_sync();
        }
        lap(2);
    }
    return 0;
}

// One sweep (forward, or backward with the transpose) of the substitution on a
// strip of SW columns held in shared memory, X(r, c) at sX[r + c ld], rows n up
// to the next multiple of 64 zero, with the inverted diagonal blocks invd of
// the lower L.  The rows of L are used once per strip, so its MMA fragments
// come straight from L2 into registers, the next ones in flight during the
// products, and a 64-row step is two products and two barriers without a
// global round trip of X.  FP32 operands are multiplied in FP64.
// WITHIN: the blocks are those of a larger inverse with leading dimension ldi,
// whose entries outside the matrix are not read (a variant of its own: the
// guards on every call cost the batch 3%).  sR: SW x LEAF_LD doubles.  All
// threads; starts and ends with a barrier.
constexpr int SW = 8;
__host__ __device__ constexpr int strip_ld(int n) { return (n + IB - 1) / IB * IB + 4; }   // 4 mod 16: no conflicts
__host__ __device__ constexpr size_t strip_smem_elems(int n) { return (size_t)SW * (strip_ld(n) + LEAF_LD); }
template <class T, bool WITHIN = false>
__device__ __noinline__ void strip_sweep(const ViewT<T> &L, int n, const T *invd, double *sX, int ld, double *sR,
                                         bool trans, int ldi = IB) {
    sX = in_shared(sX);
    sR = in_shared(sR);
    const int warp = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    const int nblk = (n + IB - 1) / IB, row = 8 * warp + g;   // this lane's row of the 64-row step
    const int last = ld - 8;   // the strip's last group of four rows
    __syncthreads();
    for (int s = 0; s < nblk; ++s) {
        const int b = trans ? nblk - 1 - s : s, jb = b * IB;
        const bool live = jb + row < n;
        // fragments of the inverted diagonal block: independent of the sum below
        const T *inv = invd + (WITHIN ? (int64_t)jb * (ldi + 1) : (int64_t)b * IB * IB);
        T iv[IB / 4];
#pragma unroll
        for (int q = 0; q < IB / 4; ++q) {
            const int k = 4 * q + t, l = WITHIN ? ldi : IB;
            iv[q] = (!WITHIN || (live && jb + k < n)) ? (trans ? inv[k + row * l] : inv[row + k * l]) : T(0);
        }
        // rows jb .. of the sum over the columns solved so far
        const int k0 = trans ? jb + IB : 0, k1 = trans ? n : jb;
        const ViewT<T> Lr = trans ? L.sub(0, jb).t() : L.sub(jb, 0);   // (row, k)
        const T *lp = Lr.at(live ? row : 0, 0) + (int64_t)t * Lr.cs;
        const int64_t st = 4 * Lr.cs;
        double acc[4][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
        constexpr int U = 8;   // fragments of one round: 32 columns
        auto fetch = [&](T (&a)[U], int k) {
#pragma unroll
            for (int u = 0; u < U; ++u) a[u] = (live && k + 4 * u + t < k1) ? lp[(int64_t)(k / 4 + u) * st] : T(0);
        };
        T a0[U], a1[U];
        fetch(a0, k0);
        for (int k = k0; k < k1; k += 8 * U) {
            fetch(a1, k + 4 * U);
#pragma unroll
            for (int u = 0; u < U; ++u) dmma884(acc[u & 3], (double)a0[u], sX[min(k + 4 * u, last) + t + g * ld]);
            fetch(a0, k + 8 * U);
#pragma unroll
            for (int u = 0; u < U; ++u)
                dmma884(acc[u & 3], (double)a1[u], sX[min(k + 4 * (U + u), last) + t + g * ld]);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
            sR[row + (2 * t + e) * LEAF_LD] =
                sX[jb + row + (2 * t + e) * ld] - ((acc[0][e] + acc[1][e]) + (acc[2][e] + acc[3][e]));
        __syncthreads();
        double y[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
        for (int q = 0; q < IB / 4; ++q) dmma884(y[q & 1], (double)iv[q], sR[4 * q + t + g * LEAF_LD]);
#pragma unroll
        for (int e = 0; e < 2; ++e) sX[jb + row + (2 * t + e) * ld] = y[0][e] + y[1][e];
        __syncthreads();
    }
}

// The largest sum of absolute values of rows r0 .. r0 + n - 1 (n <= R) of the
// lower V (unit: with an implied unit diagonal), along the contiguous
// direction, as the bits of a double: maxima are taken on the bits, where NaN is
// above Inf.  The whole CTA; valid in every warp's lane 0 for what that warp
// has seen.
template <int R>
__device__ inline long long lower_row_norm(const View &V, int r0, int n, bool unit) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int Q = NT_CTA / R;
    __shared__ double s_part[Q][R];
    long long top = 0;
    const int skip = unit ? 1 : 0;
    if (V.rs == 1) {
        const int r = threadIdx.x % R, q = threadIdx.x / R;
        double s = (unit && q == 0) ? 1.0 : 0.0;
        if (r < n)
#pragma unroll 8
            for (int c = q; c <= r0 + r - skip; c += Q) s += fabs(*V.at(r0 + r, c));
        s_part[q][r] = s;
        __syncthreads();
        if (q == 0 && r < n) {
#pragma unroll
            for (int i = 1; i < Q; ++i) s += s_part[i][r];
            top = __double_as_longlong(fabs(s));
        }
        __syncthreads();
    } else {
        for (int r = warp; r < n; r += NT_CTA / 32) {
            double s = (unit && lane == 0) ? 1.0 : 0.0;
#pragma unroll 8
            for (int c = lane; c <= r0 + r - skip; c += 32) s += fabs(*V.at(r0 + r, c));
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            top = max(top, __double_as_longlong(fabs(s)));
        }
    }
    for (int o = 16; o; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    return top;
}
// norm[0], norm[1] = the infinity norms of the lower L and of its inverse X
// (zeroed before), R rows per CTA.
template <int R>
__device__ inline void lower_norms(const View &L, const View &X, int r0, int n, bool unit, double *norm) {
#pragma unroll 1
    for (int m = 0; m < 2; ++m) {
        const long long top = lower_row_norm<R>(m ? X : L, r0, n, unit && m == 0);
        if ((threadIdx.x & 31) == 0 && top) atomicMax(reinterpret_cast<long long *>(norm + m), top);
    }
}

// Inverted 64 x 64 diagonal blocks of an existing lower factor (n x n), for
// the solve-only executor mode.
template <class T>
__device__ void tile_inv_blk(const ViewT<T> &Tv, int n, T *invd, T *smem) {
    T *sD = smem;
    T *sX = sD + IB * LDS;
    for (int jb = 0; jb < n; jb += IB) {
        const int nbk = min(IB, n - jb);
        leaf64_load(Tv.sub(jb, jb), nbk, sD);
        leaf64_core<T, false>(sD, sX, nbk);
        T *inv = invd + (int64_t)(jb / IB) * IB * IB;
        for (int idx = threadIdx.x; idx < IB * IB; idx += NT_CTA) {
            const int r = idx % IB, c = idx / IB;
            inv[idx] = (r < nbk && c < nbk) ? sX[r + c * LDS] : T(0);
        }
        __syncthreads();
    }
}

// Output block sizes of the GEMM passes.
template <class T, int SP>
using CB = Cfg128<T, SP>;   // 128 x 128

// A (rows x n) <- A X^T in place, X lower n x n: column blocks from the last
// (each reads columns < its end, which later blocks do not overwrite).
template <class T, int SP>
__device__ __noinline__ void apply_inv_right(const ViewT<T> &A, int rows, const ViewT<T> &X, int n, T *smem) {
    using C = CB<T, SP>;
    const int ncb = (n + C::BN - 1) / C::BN;
    for (int r0 = 0; r0 < rows; r0 += C::BM) {
        const int mr = min(C::BM, rows - r0);
        for (int cb = ncb - 1; cb >= 0; --cb) {
            const int c0 = cb * C::BN, w = min(C::BN, n - c0);
            Acc<C> acc;
            acc.zero();
            cta_gemm(acc, A.sub(r0, 0), X.sub(c0, 0), mr, w, c0 + w, smem);
            acc.store_to(A.sub(r0, c0), mr, w);
            cta_sync();
        }
    }
}

// B (n x w) <- X B (TRANS: X^T B) in place, X lower n x n: row blocks from the
// last (forward) or the first (transposed), so that no row of B is
// overwritten before every block that reads it is done.
template <class T, int SP, bool TRANS>
__device__ __noinline__ void apply_inv_left(const ViewT<T> &B, int w, const ViewT<T> &X, int n, T *smem) {
    using C = Cfg12864<T, SP>;
    const int nrb = (n + C::BM - 1) / C::BM;
    for (int s = 0; s < nrb; ++s) {
        const int rb = TRANS ? s : nrb - 1 - s;
        const int r0 = rb * C::BM, mr = min(C::BM, n - r0);
        for (int c0 = 0; c0 < w; c0 += C::BN) {
            const int wc = min(C::BN, w - c0);
            Acc<C> acc;
            acc.zero();
            if (!TRANS) cta_gemm(acc, X.sub(r0, 0), B.sub(0, c0).t(), mr, wc, r0 + mr, smem);
            else cta_gemm(acc, X.sub(r0, r0).t(), B.sub(r0, c0).t(), mr, wc, n - r0, smem);
            acc.store_to(B.sub(r0, c0), mr, wc);
            cta_sync();
        }
    }
}

// Split point of an n-wide recursion level: a multiple of 64, at least half.
__device__ __forceinline__ int split_point(int n) { return ((n / 2 + 63) / 64) * 64; }

// Recursive factor (FACT) or inverse-only (!FACT) of an n x n lower tile,
// n <= 64 << LVL.  A: the tile (lower triangle read / written, upper never
// touched); X: its inverse, n x n, written in full.
template <class T, int SP, bool FACT, int LVL>
__device__ __noinline__ int rec_tile(const ViewT<T> &A, const ViewT<T> &X, int n, T *smem) {
    if constexpr (LVL == 0) {
        return leaf64<T, FACT>(A, X, n, smem);
    } else {
        if (n <= (64 << (LVL - 1))) return rec_tile<T, SP, FACT, LVL - 1>(A, X, n, smem);
        using C = CB<T, SP>;
        const int n1 = split_point(n), n2 = n - n1;
        const ViewT<T> A21 = A.sub(n1, 0), A22 = A.sub(n1, n1);
        const ViewT<T> X11 = X, X21 = X.sub(n1, 0), X22 = X.sub(n1, n1);
        int info = rec_tile<T, SP, FACT, LVL - 1>(A, X11, n1, smem);
        if (info) return info;
        if (FACT) {
            apply_inv_right<T, SP>(A21, n2, X11, n1, smem);   // L21 = A21 X11^T
            // A22 -= L21 L21^T, lower blocks only
            for (int r0 = 0; r0 < n2; r0 += C::BM) {
                const int mr = min(C::BM, n2 - r0);
                for (int c0 = 0; c0 <= r0; c0 += C::BN) {
                    const int w = min(C::BN, n2 - c0);
                    Acc<C> acc;
                    acc.zero();
                    cta_gemm(acc, A21.sub(r0, 0), A21.sub(c0, 0), mr, w, n1, smem);
                    acc.sub_from(A22.sub(r0, c0), mr, w, r0 == c0);
                }
            }
            cta_sync();
        }
        info = rec_tile<T, SP, FACT, LVL - 1>(A22, X22, n2, smem);
        if (info) return n1 + info;
        // W = L21 X11 into the X21 block (X11 lower: column block c0 needs k >= c0)
        for (int r0 = 0; r0 < n2; r0 += C::BM) {
            const int mr = min(C::BM, n2 - r0);
            for (int c0 = 0; c0 < n1; c0 += C::BN) {
                const int w = min(C::BN, n1 - c0);
                Acc<C> acc;
                acc.zero();
                cta_gemm(acc, A21.sub(r0, c0), X11.sub(c0, c0).t(), mr, w, n1 - c0, smem);
                acc.store_to(X21.sub(r0, c0), mr, w);
            }
        }
        cta_sync();
        // X21 = -X22 W in place, row blocks from the last
        const int nrb = (n2 + C::BM - 1) / C::BM;
        for (int rb = nrb - 1; rb >= 0; --rb) {
            const int r0 = rb * C::BM, mr = min(C::BM, n2 - r0);
            for (int c0 = 0; c0 < n1; c0 += C::BN) {
                const int w = min(C::BN, n1 - c0);
                Acc<C> acc;
                acc.zero();
                cta_gemm(acc, X22.sub(r0, 0), X21.sub(0, c0).t(), mr, w, r0 + mr, smem);
                acc.for_each([&](int r, int c, T v) {
                    if (r < mr && c < w) *X21.at(r0 + r, c0 + c) = -v;
                });
                cta_sync();
            }
        }
        // the upper-right block of the inverse is zero
        for (int idx = threadIdx.x; idx < n1 * n2; idx += NT_CTA) *X.at(idx % n1, n1 + idx / n1) = T(0);
        cta_sync();
        return 0;
    }
}

constexpr int MAX_LVL = 4;   // tiles up to 64 << 4 = 1024

template <class T, int SP>
__device__ __forceinline__ int tile_potrf_inv(const ViewT<T> &A, const ViewT<T> &X, int n, T *smem) {
    return rec_tile<T, SP, true, MAX_LVL>(A, X, n, smem);
}
template <class T, int SP>
__device__ __forceinline__ void tile_trtri(const ViewT<T> &A, const ViewT<T> &X, int n, T *smem) {
    rec_tile<T, SP, false, MAX_LVL>(A, X, n, smem);
}

// Shared memory of the leaf (the GEMM passes use the tile kernels' stages).
constexpr size_t leaf_smem_elems() { return 2 * 64 * LDS; }

}  // namespace rec
}  // namespace chb
