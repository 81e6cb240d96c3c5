// aca.cu -- batched ACA of all admissible blocks, FP64.
//
// The reference (linear_algebra.cu:3684-4012) advances all blocks in lock step:
// every rank step is ~10 kernel launches, Thrust reduce_by_key calls and a host
// synchronisation, over "batched" vectors that concatenate all blocks.  Here one CTA
// (small blocks: one warp) owns one block for its whole ACA: the residual row / column,
// the pivot searches and the norms are its reductions, and the only traffic is the
// block's own terms.
//
// Bound by the latency of the rank steps (a chain of r FP64 multiply-adds and a kernel
// entry, twice, with four barriers), not by bytes or FP64 rate: 30-50 % of issue slots
// used.  Measured at N = 2^17 (uniform 3D, Matern, eps 1e-8, mean rank 48, 108k blocks):
// 152 ms in the ACA kernels against 249 ms for a CTA of 256 threads (blocks to 512: a
// warp) that kept every term in device memory and ran the cross terms at every step;
// hmg_precompute_aca 190 ms against 575 (the rest: 16 GB of scratch in a pool that maps and
// unmaps it, now 4 GB).  Factors and ranks are the same to the last bit.
//
// Two modes:
//   * fixed (eps <= 0): the reference's semantics -- rank k_b = min(k,m1,m2)
//     (:769-787), row pivots taken in index order skipping residual rows of norm
//     < 1e-13 (:2009-2024, :2091, :1213-1230), column pivot = LAST index of the
//     largest |v| (tuple_absolute_maximum, :991-1018), v scaled by the pivot
//     (:963-986), residual updates with fused multiply-adds (:918-959, :1091-1147).
//     The reference's scaling kernel reads the pivot entry while other threads
//     overwrite it (:983); here the pivot is read once before any write.
//   * adaptive (eps > 0): standard partial pivoting -- next row = largest |u_r| over
//     unused rows, column = FIRST index of the largest |v| -- stopping when
//     |u_r| |v_r| <= eps ||S_r||_F with the Frobenius norm of the approximant
//     updated exactly (the criterion the reference keeps dormant at
//     :1595-1755, without its (1-eta) factor, which is negative for eta > 1).
//
// Factors are computed into FP64 scratch per batch of blocks and then compacted
// (converted to the storage precision, laid out as tile slices for U and as
// padded rows of V^T) into one allocation per batch.
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "hmg_matrix.cuh"
#include "stream.cuh"

namespace hmg {

static constexpr int ACA_KMAX = 512;

struct AcaBatch {
    const int* blocks;       // block indices of this batch
    const long long* uoff;   // FP64 scratch offsets
    const long long* voff;
    double* U;
    double* V;
    int* rank_out;           // per batch entry
    double* s2_out;          // per batch entry: |U V^T|_F^2 (adaptive mode), may be null
    const long long* soff;   // per batch entry: its first term among the batch's (mixed storage)
    double* tnorm;           // per term |u_l|^2, |v_l|^2, max |u_l| (mixed storage, else null)
};

struct BlockGeom {
    const int *r0, *m1, *c0, *m2;
    const double* param;  // per-block kernel parameter (grouped H-matrices), else null
};

// (value, index) argmax; last = true: ties go to the larger index, else the smaller.
__device__ __forceinline__ bool better(double a, int i, double b, int j, bool last)
{
    if (a != b) return a > b;
    return last ? i > j : i < j;
}

// The warp's entry of largest magnitude and its index (ties: the smaller index, or the
// larger with `last`; a NaN counts as 0), by integer reductions of the magnitude's words
// and the index: an FP64 compare-and-select butterfly takes five times the instructions.
__device__ __forceinline__ void warp_argmax(double& v, int& i, bool last)
{
    const unsigned long long key = v == v ? (unsigned long long)__double_as_longlong(fabs(v)) : 0ull;
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    const bool in = hi == mh && lo == ml;
    const int j = last ? __reduce_max_sync(0xffffffffu, in ? i : -1) : __reduce_min_sync(0xffffffffu, in ? i : 0x7fffffff);
    const unsigned at = __ballot_sync(0xffffffffu, in && i == j);
    v = __shfl_sync(0xffffffffu, v, at ? __ffs(at) - 1 : 0);
    i = j;
}

// c += A B of one 8 x 8 x 4 FP64 MMA: lane (g, t) has A[g][t], B[t][g], C[g][2t], C[g][2t+1]
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

// The share of warp w of nw in |sum_{l < r} u_l v_l^T|_F^2 = sum_{l, l'} (u_l . u_l')(v_l . v_l'):
// the 8 x 8 products of pairs of 8 terms, every nw-th pair (b0 <= b1).  The warp's lanes hold
// the parts of its sum.
template <class FU, class FV>
__device__ __forceinline__ double gram_share(int r, int m1, int m2, int w, int nw, FU term_u, FV term_v)
{
    const int lane = threadIdx.x & 31, nb = (r + 7) >> 3, g = lane >> 2, t = lane & 3;
    double acc = 0.0;
    int p = w;
    for (int b0 = 0; b0 < nb; b0++) {
        const int row = nb - b0;
        for (; p < row; p += nw) {
            const int b1 = b0 + p, l0 = 8 * b0 + g, l1 = 8 * b1 + g;
            double cu[2] = {0.0, 0.0}, cv[2] = {0.0, 0.0};
            const double *xu = l0 < r ? term_u(l0) : nullptr, *yu = l1 < r ? term_u(l1) : nullptr;
            const double *xv = l0 < r ? term_v(l0) : nullptr, *yv = l1 < r ? term_v(l1) : nullptr;
            for (int i0 = 0; i0 < m1; i0 += 4) {
                const bool in = i0 + t < m1;
                dmma(cu, xu && in ? xu[i0 + t] : 0.0, yu && in ? yu[i0 + t] : 0.0);
            }
            for (int i0 = 0; i0 < m2; i0 += 4) {
                const bool in = i0 + t < m2;
                dmma(cv, xv && in ? xv[i0 + t] : 0.0, yv && in ? yv[i0 + t] : 0.0);
            }
            acc += (b0 == b1 ? 1.0 : 2.0) * (cu[0] * cv[0] + cu[1] * cv[1]);
        }
        p -= row;
    }
    return acc;
}

// Kernel entries between one fixed point and the points of an array (SoA): the fixed
// point's coordinates are loaded once.
struct Entries {
    const double *cx, *cy, *cz;  // the points (cz: null in 2D)
    double fx, fy, fz;           // the fixed point
    int same;                    // the index whose entry is on the diagonal (gets the regularization)
    __device__ __forceinline__ Entries(const double* const* points, int p0, const double* const* fixed, int f, int dim, int d)
        : cx(points[0] + p0), cy(points[1] + p0), cz(dim > 2 ? points[2] + p0 : nullptr), fx(fixed[0][f]), fy(fixed[1][f]),
          fz(dim > 2 ? fixed[2][f] : 0.0), same(d)
    {
    }
    __device__ __forceinline__ double operator()(const KernelSpec& K, int j) const
    {
        const double x = fx - cx[j], y = fy - cy[j];
        double s = __fma_rn(x, x, 0.0);
        s = __fma_rn(y, y, s);
        if (cz) {
            const double z = fz - cz[j];
            s = __fma_rn(z, z, s);
        }
        const double v = kernel_from_sq(K, s);
        return j == same ? v + K.reg : v;
    }
};

// One block's ACA by one CTA of T threads.
//
// What a rank step reads is the block's earlier terms, twice: the residual of the pivot
// row needs every earlier v_l, that of the pivot column every earlier u_l.  The first
// `cap` terms (as many as the CTA's shared memory takes) are kept there, FP64 as in the
// scratch, and only later ones are read back from the scratch.  The residuals add the
// terms in order, one fused multiply-add each, wherever a term lies.
//
// The adaptive mode's third pass, the cross terms of |S_r|_F, is not run every step.
// |S_r|_F is at most the sum of the terms' norms; while a term is larger than eps times
// that bound the stopping test cannot hold.  When it no longer is, |S_r|_F^2 is computed
// once from the Gram matrices of the terms (FP64 tensor-core products of 8 x 8 terms), and
// updated exactly from there on (usually one to three steps).
template <int T> struct AcaShared {
    double v[T / 32], p[T / 32], q[T / 32], x[T / 32];
    int i[T / 32];
};

template <int T, int C>
struct AcaBlock {
    static constexpr int NW = T / 32;
    AcaShared<T>& sh;
    double* sp;           // the terms in shared memory: ms doubles each, u_l then v_l
    int ms, cap;
    double *U, *V;        // the terms in the scratch
    int m1, m2;
    int tid, lane, warp;

    __device__ __forceinline__ const double* term_u(int l) const { return l < cap ? sp + (size_t)l * ms : U + (size_t)l * m1; }
    __device__ __forceinline__ const double* term_v(int l) const { return l < cap ? sp + (size_t)l * ms + m1 : V + (size_t)l * m2; }
    // where entry j of v_r is kept until the pivot is known
    __device__ __forceinline__ double* slot_v(int r) const { return r < cap ? sp + (size_t)r * ms + m1 : V + (size_t)r * m2; }

    // val[q] = entry(idx[q]) - sum_l coef[l] term_l[idx[q]], l in order.  coef is 16-byte
    // aligned.  Where most terms lie in the scratch (two entries a thread: the largest
    // blocks), eight scratch loads an entry are in flight at any time, the first ones before
    // the entries are evaluated.
    template <int N, class F>
    __device__ __forceinline__ void residual(double (&val)[N], const int (&idx)[N], F entry, const double* s0,
                                             const double* g0, int ld, int r, const double* coef) const
    {
        constexpr bool AHEAD = C > 1;
        const int rs = r < cap ? r : cap;
        const double* g = g0 + (size_t)rs * ld;
        double t[8][N];
        if (AHEAD) {
#pragma unroll
            for (int u = 0; u < 8; u++)
#pragma unroll
                for (int q = 0; q < N; q++) t[u][q] = rs + u < r ? __ldcg(g + (size_t)u * ld + idx[q]) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < N; q++) val[q] = entry(idx[q]);
        const double* sq[N];
#pragma unroll
        for (int q = 0; q < N; q++) sq[q] = s0 + idx[q];
        int l = 0;
        for (; l + 4 <= rs; l += 4) {
            const double2 c0 = *reinterpret_cast<const double2*>(coef + l), c1 = *reinterpret_cast<const double2*>(coef + l + 2);
#pragma unroll
            for (int q = 0; q < N; q++) {
                val[q] = __fma_rn(-c0.x, sq[q][0], val[q]);
                val[q] = __fma_rn(-c0.y, sq[q][ms], val[q]);
                val[q] = __fma_rn(-c1.x, sq[q][2 * ms], val[q]);
                val[q] = __fma_rn(-c1.y, sq[q][3 * ms], val[q]);
                sq[q] += 4 * ms;
            }
        }
        for (; l < rs; l++)
#pragma unroll
            for (int q = 0; q < N; q++) {
                val[q] = __fma_rn(-coef[l], *sq[q], val[q]);
                sq[q] += ms;
            }
        // (l = cap, a multiple of 4, where there are terms in the scratch)
        if (AHEAD) {
            const double* p[N];  // the next term to load
#pragma unroll
            for (int q = 0; q < N; q++) p[q] = g + 8 * (size_t)ld + idx[q];
            for (; l + 16 <= r; l += 8) {
#pragma unroll
                for (int u = 0; u < 8; u += 2) {
                    const double2 c = *reinterpret_cast<const double2*>(coef + l + u);
#pragma unroll
                    for (int q = 0; q < N; q++) {
                        val[q] = __fma_rn(-c.x, t[u][q], val[q]);
                        t[u][q] = __ldcg(p[q]);
                        p[q] += ld;
                        val[q] = __fma_rn(-c.y, t[u + 1][q], val[q]);
                        t[u + 1][q] = __ldcg(p[q]);
                        p[q] += ld;
                    }
                }
            }
            const int have = min(8, r - l);  // loaded; then the rest, fewer than 8
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (u < have) {
                    const double c = coef[l + u];
#pragma unroll
                    for (int q = 0; q < N; q++) {
                        val[q] = __fma_rn(-c, t[u][q], val[q]);
                        if (l + u + 8 < r) t[u][q] = __ldcg(p[q] + (size_t)u * ld);
                    }
                }
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (l + u + 8 < r) {
                    const double c = coef[l + u + 8];
#pragma unroll
                    for (int q = 0; q < N; q++) val[q] = __fma_rn(-c, t[u][q], val[q]);
                }
        } else {
            for (; l + 8 <= r; l += 8, g += 8 * (size_t)ld) {
#pragma unroll
                for (int u = 0; u < 8; u++)
#pragma unroll
                    for (int q = 0; q < N; q++) t[u][q] = __ldcg(g + (size_t)u * ld + idx[q]);
#pragma unroll
                for (int u = 0; u < 8; u += 2) {
                    const double2 c = *reinterpret_cast<const double2*>(coef + l + u);
#pragma unroll
                    for (int q = 0; q < N; q++) {
                        val[q] = __fma_rn(-c.x, t[u][q], val[q]);
                        val[q] = __fma_rn(-c.y, t[u + 1][q], val[q]);
                    }
                }
            }
            for (; l < r; l++, g += ld)
#pragma unroll
                for (int q = 0; q < N; q++) val[q] = __fma_rn(-coef[l], __ldcg(g + idx[q]), val[q]);
        }
    }

    // Residuals of the n entries of a row or column, each handed to take(index, value), a
    // thread's own entry tid first: C at a time where the thread's warp has as many.
    template <class F, class G>
    __device__ __forceinline__ void residuals(int n, F entry, const double* s0, const double* g0, int ld, int r,
                                              const double* coef, G take) const
    {
        for (int j = tid; j < n; j += C * T) {
            if (C > 1 && (j & ~31) + T < n) {
                const int idx[2] = {j, min(j + T, n - 1)};
                double val[2];
                residual<2>(val, idx, entry, s0, g0, ld, r, coef);
                take(j, val[0]);
                if (j + T < n) take(j + T, val[1]);
            } else {
                const int idx[1] = {j};
                double val[1];
                residual<1>(val, idx, entry, s0, g0, ld, r, coef);
                take(j, val[0]);
            }
        }
    }

    // The CTA's entry of largest magnitude, and with SUMS the sums p, q and the maximum x;
    // every thread gets the results.  One barrier; the shared entries are free again at the
    // next.
    template <bool SUMS>
    __device__ __forceinline__ void reduce(double& v, int& i, double& p, double& q, double& x, bool last) const
    {
        warp_argmax(v, i, last);
        if (SUMS)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                p += __shfl_xor_sync(0xffffffffu, p, o);
                q += __shfl_xor_sync(0xffffffffu, q, o);
                x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
            }
        if (lane == 0) {
            sh.v[warp] = v;
            sh.i[warp] = i;
            if (SUMS) { sh.p[warp] = p; sh.q[warp] = q; sh.x[warp] = x; }
        }
        __syncthreads();
        const int w0 = lane & (NW - 1);
        v = sh.v[w0];
        i = sh.i[w0];
        warp_argmax(v, i, last);
        if (SUMS) {
            p = sh.p[w0]; q = sh.q[w0]; x = sh.x[w0];
#pragma unroll
            for (int o = NW / 2; o > 0; o >>= 1) {
                p += __shfl_xor_sync(0xffffffffu, p, o);
                q += __shfl_xor_sync(0xffffffffu, q, o);
                x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
            }
        }
    }

    // |sum_{l < r} u_l v_l^T|_F^2.  Barriers on both sides.
    __device__ __noinline__ double frobenius2(int r) const
    {
        return total(gram_share(r, m1, m2, warp, NW, [&](int l) { return term_u(l); }, [&](int l) { return term_v(l); }));
    }

    // cross terms of the last of r + 1 terms with the r before: sum_l (u_r . u_l)(v_r . v_l)
    __device__ __noinline__ double cross_terms(int r) const
    {
        const double *ur = term_u(r), *vr = term_v(r);
        double acc = 0.0;
        for (int l = warp; l < r; l += NW) {
            const double *ul = term_u(l), *vl = term_v(l);
            double x = 0.0, y = 0.0;
            for (int i = lane; i < m1; i += 32) x = __fma_rn(ur[i], ul[i], x);
            for (int j = lane; j < m2; j += 32) y = __fma_rn(vr[j], vl[j], y);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                x += __shfl_xor_sync(0xffffffffu, x, o);
                y += __shfl_xor_sync(0xffffffffu, y, o);
            }
            if (lane == 0) acc += x * y;
        }
        return total(acc);
    }

    __device__ double total(double s) const
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        __syncthreads();
        if (lane == 0) sh.p[warp] = s;
        __syncthreads();
        s = sh.p[lane & (NW - 1)];
#pragma unroll
        for (int o = NW / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        __syncthreads();
        return s;
    }
};

template <int T, int C, int CTAS>
__global__ void __launch_bounds__(T, CTAS)
k_aca(BlockGeom g, KernelSpec K0, PointsView P, AcaBatch B, int k, double eps, const int* elist, int panel, int kc)
{
    __shared__ AcaShared<T> sh;
    // panel doubles of terms, the pivot row's and column's coefficients (kc >= the largest
    // rank), then (adaptive mode) one bit per row
    extern __shared__ __align__(16) double aca_smem[];
    double *coef = aca_smem + panel, *coef2 = coef + kc;

    const int e = elist[blockIdx.x];
    const int b = B.blocks[e];
    KernelSpec K = K0;
    if (g.param) K.param = g.param[b];
    const int r0 = g.r0[b], m1 = g.m1[b], c0 = g.c0[b], m2 = g.m2[b];
    int kb = k < m1 ? k : m1;
    kb = kb < m2 ? kb : m2;
    const int tid = threadIdx.x;
    unsigned* used = reinterpret_cast<unsigned*>(coef2 + kc);
    const AcaBlock<T, C> A{sh, aca_smem, m1 + m2, panel / (m1 + m2) & ~3, B.U + B.uoff[e], B.V + B.voff[e], m1, m2,
                        tid, tid & 31, tid >> 5};
    const bool adaptive = eps > 0.0;
    int rank = 0;
    double S2 = 0.0;        // adaptive mode: squared Frobenius norm of the approximant
    double norms = 0.0;     // sum of the terms' norms, an upper bound of |S|_F
    bool have_s2 = false;

    if (adaptive) {
        for (int w = tid; w < ((m1 + 31) >> 5); w += T) used[w] = 0u;
        __syncthreads();
    }
    int ir = adaptive ? 0 : -1, nused = 0;
    for (int r = 0; r < kb; r++) {
        // ---- pivot row: the next usable row's residual, its largest entry
        double piv = 0.0, none = 0.0, nosum = 0.0;
        double mine = 0.0;  // the raw entry tid of v_r (the others wait in vr)
        int jr = -1;
        double* vr = A.slot_v(r);
        for (;;) {
            if (adaptive) {
                if (tid == 0) used[ir >> 5] |= 1u << (ir & 31);
                nused++;
            } else {
                if (ir >= m1 - 1) break;
                ir += 1;
            }
            for (int l = tid; l < r; l += T) coef[l] = A.term_u(l)[ir];
            __syncthreads();
            double bv = 0.0, ss = 0.0;
            int bj = adaptive ? 0x7fffffff : -1;
            const Entries row(P.c2, c0, P.c1, r0 + ir, K.dim, r0 + ir - c0);
            A.residuals(m2, [&](int q) { return row(K, q); }, A.sp + m1, A.V, m2, r, coef, [&](int j, double v) {
                if (j == tid) mine = v;
                else vr[j] = v;
                ss += v * v;
                if (better(fabs(v), j, fabs(bv), bj, !adaptive)) { bv = v; bj = j; }
            });
            if (adaptive) A.template reduce<false>(bv, bj, ss, nosum, none, false);
            else A.template reduce<true>(bv, bj, ss, nosum, none, true);
            if (adaptive ? fabs(bv) > 0.0 : sqrt(ss) >= 1.0e-13) {
                jr = bj;
                piv = bv;
                break;
            }
            __syncthreads();  // the reduction's entries and coef are used again
            if (adaptive) {
                // zero residual row: the next unused row in index order
                int cand = 0x7fffffff;
                for (int i = tid; i < m1; i += T)
                    if (!((used[i >> 5] >> (i & 31)) & 1u)) { cand = i; break; }
                double z = 0.0;
                A.template reduce<false>(z, cand, nosum, nosum, none, false);
                __syncthreads();
                if (cand == 0x7fffffff) break;
                ir = cand;
            }
        }
        if (jr < 0) break;
        // ---- the row scaled by the pivot
        for (int l = tid; l < r; l += T) coef2[l] = A.term_v(l)[jr];
        double pv = 0.0;
        for (int j = tid; j < m2; j += T) {
            const double v = (j == tid ? mine : vr[j]) / piv;
            if (r < A.cap) A.sp[(size_t)r * A.ms + m1 + j] = v;
            A.V[j + (size_t)r * m2] = v;
            pv += v * v;
        }
        __syncthreads();
        // ---- pivot column: residual, norm, and (adaptive) its largest unused row
        double pu = 0.0, bu = 0.0, mu = 0.0;
        int bi = 0x7fffffff;
        const Entries col(P.c1, r0, P.c2, c0 + jr, K.dim, c0 + jr - r0);
        A.residuals(m1, [&](int q) { return col(K, q); }, A.sp, A.U, m1, r, coef2, [&](int i, double v) {
            if (r < A.cap) A.sp[(size_t)r * A.ms + i] = v;
            A.U[i + (size_t)r * m1] = v;
            pu += v * v;
            mu = fmax(mu, fabs(v));
            if (adaptive && !((used[i >> 5] >> (i & 31)) & 1u) && better(fabs(v), i, fabs(bu), bi, false)) {
                bu = v;
                bi = i;
            }
        });
        rank = r + 1;
        if (!adaptive) {
            __syncthreads();
            continue;
        }
        A.template reduce<true>(bu, bi, pv, pu, mu, false);
        __syncthreads();  // u_r, v_r complete; the reduction's entries are used again
        if (B.tnorm && tid == 0) {
            double* tn = B.tnorm + 3 * (B.soff[e] + r);
            tn[0] = pu;
            tn[1] = pv;
            tn[2] = mu;
        }
        const double nn = sqrt(pu * pv);
        norms += nn;
        bool stop = false;
        if (have_s2) {
            const double cross = A.cross_terms(r);
            S2 = S2 + 2.0 * cross + pu * pv;
            stop = nn <= eps * sqrt(fabs(S2));
        } else if (!(nn > eps * norms * (1.0 + 1e-12))) {
            S2 = A.frobenius2(rank);
            have_s2 = true;
            stop = nn <= eps * sqrt(fabs(S2));
        }
        if (stop || nused >= m1 || bi == 0x7fffffff) break;
        ir = bi;
    }
    if (adaptive && B.s2_out && !have_s2 && rank > 0) {
        __syncthreads();
        S2 = A.frobenius2(rank);
    }
    if (tid == 0) {
        B.rank_out[e] = rank;
        if (B.s2_out) B.s2_out[e] = S2;
    }
}

// ---------------------------------------------------------------------------
// The adaptive ACA of a small block (m1, m2 <= ACA_WSMALL) by one warp: the steps of
// k_aca's adaptive mode with warp shuffles in place of CTA reductions and no CTA barriers.
// ---------------------------------------------------------------------------
static constexpr int ACA_WSMALL = 128;  // largest m1 and m2 of the warp variant
static constexpr int ACA_WPC = 8;       // warps (blocks) per CTA

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __noinline__ double warp_frobenius2(const double* U, const double* V, int m1, int m2, int r)
{
    return warp_sum(gram_share(r, m1, m2, 0, 1, [&](int l) { return U + (size_t)l * m1; },
                               [&](int l) { return V + (size_t)l * m2; }));
}

__global__ void __launch_bounds__(ACA_WPC * 32, 4)
k_aca_warp(BlockGeom g, KernelSpec K0, PointsView P, AcaBatch B, int k, double eps, const int* elist, int nlist)
{
    __shared__ double coefs[ACA_WPC][ACA_WSMALL];
    __shared__ unsigned usedw[ACA_WPC][ACA_WSMALL / 32];
    const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = blockIdx.x * ACA_WPC + wi;
    if (slot >= nlist) return;
    const int e = elist[slot];
    const int b = B.blocks[e];
    KernelSpec K = K0;
    if (g.param) K.param = g.param[b];
    const int r0 = g.r0[b], m1 = g.m1[b], c0 = g.c0[b], m2 = g.m2[b];
    int kb = k < m1 ? k : m1;
    kb = kb < m2 ? kb : m2;
    double* U = B.U + B.uoff[e];
    double* V = B.V + B.voff[e];
    double* coef = coefs[wi];
    unsigned* used = usedw[wi];
    for (int w = lane; w < ACA_WSMALL / 32; w += 32) used[w] = 0u;
    __syncwarp();
    int rank = 0, ir = 0, nused = 0;
    double S2 = 0.0, norms = 0.0;  // as in k_aca
    bool have_s2 = false;
    for (int r = 0; r < kb; r++) {
        int jr = -1;
        double piv = 0.0;
        bool have = false;
        for (;;) {
            if (lane == 0) used[ir >> 5] |= 1u << (ir & 31);
            nused++;
            for (int l = lane; l < r; l += 32) coef[l] = U[ir + (size_t)l * m1];
            __syncwarp();
            double best = 0.0;
            int bj = 0x7fffffff;
            const Entries row(P.c2, c0, P.c1, r0 + ir, K.dim, r0 + ir - c0);
            for (int j = lane; j < m2; j += 32) {
                double val = row(K, j);
                for (int l = 0; l < r; l++) val = __fma_rn(-coef[l], V[j + (size_t)l * m2], val);
                V[j + (size_t)r * m2] = val;
                if (better(fabs(val), j, fabs(best), bj, false)) { best = val; bj = j; }
            }
            warp_argmax(best, bj, false);
            if (fabs(best) > 0.0) {
                piv = best;
                jr = bj;
                have = true;
                break;
            }
            // zero residual row: the next unused row in index order
            int cand = 0x7fffffff;
            for (int i = lane; i < m1; i += 32)
                if (!((used[i >> 5] >> (i & 31)) & 1u)) { cand = i; break; }
            double dummy = 0.0;
            warp_argmax(dummy, cand, false);
            if (cand == 0x7fffffff) break;
            ir = cand;
            __syncwarp();
        }
        if (!have) break;
        __syncwarp();  // every lane's V[., r] written
        double pv = 0.0;
        for (int j = lane; j < m2; j += 32) {
            const double v = V[j + (size_t)r * m2] / piv;
            V[j + (size_t)r * m2] = v;
            pv += v * v;
        }
        __syncwarp();
        for (int l = lane; l < r; l += 32) coef[l] = V[jr + (size_t)l * m2];
        __syncwarp();
        double pu = 0.0, bu = 0.0, mu = 0.0;
        const Entries col(P.c1, r0, P.c2, c0 + jr, K.dim, c0 + jr - r0);
        int bi = 0x7fffffff;
        for (int i = lane; i < m1; i += 32) {
            double val = col(K, i);
            for (int l = 0; l < r; l++) val = __fma_rn(-coef[l], U[i + (size_t)l * m1], val);
            U[i + (size_t)r * m1] = val;
            pu += val * val;
            mu = fmax(mu, fabs(val));
            if (!((used[i >> 5] >> (i & 31)) & 1u) && better(fabs(val), i, fabs(bu), bi, false)) { bu = val; bi = i; }
        }
        const double nv2 = warp_sum(pv), nu2 = warp_sum(pu);
        warp_argmax(bu, bi, false);
        __syncwarp();  // every lane's U[., r] written
        if (B.tnorm) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mu = fmax(mu, __shfl_xor_sync(0xffffffffu, mu, o));
            if (lane == 0) {
                double* tn = B.tnorm + 3 * (B.soff[e] + r);
                tn[0] = nu2;
                tn[1] = nv2;
                tn[2] = mu;
            }
        }
        rank = r + 1;
        const double nn = sqrt(nu2 * nv2);
        norms += nn;
        if (have_s2) {
            // cross terms sum_l (u_r . U_l)(v_r . V_l), in l order
            double cross = 0.0;
            const double* ur = U + (size_t)r * m1;
            const double* vr = V + (size_t)r * m2;
            for (int l = 0; l < r; l++) {
                const double* ul = U + (size_t)l * m1;
                const double* vl = V + (size_t)l * m2;
                double a = 0.0, c = 0.0;
                for (int i = lane; i < m1; i += 32) a = __fma_rn(ur[i], ul[i], a);
                for (int j = lane; j < m2; j += 32) c = __fma_rn(vr[j], vl[j], c);
                cross += warp_sum(a) * warp_sum(c);
            }
            S2 = S2 + 2.0 * cross + nu2 * nv2;
            if (nn <= eps * sqrt(fabs(S2))) break;
        } else if (!(nn > eps * norms * (1.0 + 1e-12))) {
            S2 = warp_frobenius2(U, V, m1, m2, rank);
            have_s2 = true;
            if (nn <= eps * sqrt(fabs(S2))) break;
        }
        if (nused >= m1) break;
        if (bi == 0x7fffffff) break;
        ir = bi;
        __syncwarp();
    }
    if (B.s2_out && !have_s2 && rank > 0) S2 = warp_frobenius2(U, V, m1, m2, rank);
    if (lane == 0) {
        B.rank_out[e] = rank;
        if (B.s2_out) B.s2_out[e] = S2;
    }
}

// Classes of blocks by their longer side: a thread an entry, and as much shared memory for
// terms as leaves several CTAs an SM, whose rank steps (four barriers, an FP64 kernel entry
// and two chains of dependent FP64 multiply-adds each) overlap: 52 KB hold 40 terms of a
// 64 + 96 block, four CTAs to an SM.  Fewer threads than entries leave too few warps for the
// FP64 latencies (128 threads for blocks of 129 to 256: 62 ms against 38 ms at N = 2^17).
// Above 512 most terms lie in the scratch: two entries a thread keep sixteen loads in flight
// each, which takes the registers of a whole SM (with half of them: 111 ms against 79).
struct AcaClass {
    int side;      // longest m1 or m2
    int panel;     // bytes of terms in shared memory (the largest class: the row mask included)
};
static constexpr int ACA_NCLASS = 4;
static constexpr AcaClass ACA_CLASSES[ACA_NCLASS] = {{128, 52 << 10}, {256, 72 << 10}, {512, 104 << 10}, {0x7fffffff, 208 << 10}};

template <int T, int C, int CTAS>
static hmg_status launch_aca(BlockGeom g, const KernelSpec& K, const PointsView& P, const AcaBatch& B, int k, double eps,
                             const int* list, int n, int panel_bytes, int kc, int mask_bytes, cudaStream_t s)
{
    if (n == 0) return HMG_OK;
    const int dyn = panel_bytes + 16 * kc + mask_bytes;
    HMG_CUDA_TRY(cudaFuncSetAttribute(k_aca<T, C, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn));
    k_aca<T, C, CTAS><<<n, T, dyn, s>>>(g, K, P, B, k, eps, list, panel_bytes / 8, kc);
    HMG_LAUNCH_CHECK();
    return HMG_OK;
}

// The smallest class: a warp a block in the adaptive mode, whose ranks there are small
static hmg_status launch_small(BlockGeom g, const KernelSpec& K, const PointsView& P, const AcaBatch& B, int k, double eps,
                               const int* list, int n, int kc, int mask_bytes, cudaStream_t s)
{
    if (eps <= 0.0) return launch_aca<128, 1, 4>(g, K, P, B, k, eps, list, n, ACA_CLASSES[0].panel, kc, mask_bytes, s);
    if (n == 0) return HMG_OK;
    k_aca_warp<<<ceil_div(n, ACA_WPC), ACA_WPC * 32, 0, s>>>(g, K, P, B, k, eps, list, n);
    HMG_LAUNCH_CHECK();
    return HMG_OK;
}

// Write the FP64 scratch factors of one block into its final storage:
// U as tile slices (s_pad x r column-major, padding rows zero) and V^T as r rows
// of m2p entries (padding zero).
// A warp takes whole rows (of V^T) and whole columns of a tile slice (of U).
template <typename T>
__global__ void __launch_bounds__(256) k_aca_compact(BlockGeom g, AcaBatch B, const int* tile_r0, const int* tile_s,
                                                     const int* tile_pstart, const int* tfirst, const int* tlast,
                                                     T* const* ptrU, T* const* ptrV, unsigned* top)
{
    const int e = blockIdx.x;
    const int b = B.blocks[e];
    const int r0 = g.r0[b], m1 = g.m1[b], m2 = g.m2[b];
    const int r = B.rank_out[e];
    if (r == 0) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double* U = B.U + B.uoff[e];
    const double* V = B.V + B.voff[e];
    T* dU = ptrU[b];
    T* dV = ptrV[b];
    const int m2p = (m2 + 3) & ~3;
    unsigned top_u = 0u, top_v = 0u;
    for (int l = warp; l < r; l += 8)
        for (int j = lane; j < m2p; j += 32) {
            const T v = j < m2 ? (T)V[j + (size_t)l * m2] : (T)0;
            dV[(size_t)l * m2p + j] = v;
            if constexpr (sizeof(T) == 4) top_v = max(top_v, magnitude(v));
        }
    const int p0 = tile_pstart[tfirst[b]];
    for (int t = tfirst[b]; t <= tlast[b]; t++) {
        const int s = tile_s[t], sp = (s + 3) & ~3, tr = tile_r0[t] - r0;
        T* dst = dU + (size_t)(tile_pstart[t] - p0) * r;
        for (int l = warp; l < r; l += 8)
            for (int i = lane; i < sp; i += 32) {
                const T u = i < s ? (T)U[(size_t)l * m1 + tr + i] : (T)0;
                dst[(size_t)l * sp + i] = u;
                if constexpr (sizeof(T) == 4) top_u = max(top_u, magnitude(u));
            }
    }
    if constexpr (sizeof(T) == 4) {
        record_top(top_u, top + 1);
        record_top(top_v, top + 2);
    }
}

// ---------------------------------------------------------------------------
// Mixed-precision storage of the low-rank terms.
//
// The ACA terms u_l v_l^T of a block decay roughly geometrically.  A term whose
// rounding to a short format adds an error far below the ACA accuracy does not need
// FP32: with sigma_l = |u_l| |v_l| and S = |U V^T|_F, the terms l with
// sum_{l' >= l} sigma_l' <= TAU16 * S are stored in FP16 (unit roundoff 4.9e-4,
// error <~ 1e-3 TAU16 S) and those with a tail below TAU8 * S in FP8 e4m3 (error
// <~ 0.07 TAU8 S).  The FP8 count is rounded down to a multiple of 4 and the FP16
// count to a multiple of 2 (the remainder moves up a tier): short terms are stored
// interleaved in pairs (FP16) and quads (FP8), so that every 16-byte chunk of every
// tier holds four consecutive rows (U) or columns (V^T) of 1, 2 or 4 terms.  Each
// short term is scaled (u by su, v by sv: to [-1, 1] in FP16, to [-448, 448] in FP8)
// and su*sv is folded into t_l = v_l^T x.
// ---------------------------------------------------------------------------
static constexpr double TAU16 = 1e-4;
static constexpr double TAU8 = 1.5e-6;

struct TierOut {
    int* r32;          // per batch entry: terms kept in FP32
    int* r16;          // terms in FP16 (the rest, up to the rank, in FP8)
    const long long* soff;  // per batch entry: offset into the scale arrays
    float* su;         // per term: scale of u_l
    float* sv;         // per term: scale of v_l
};

// One warp per block: the tiers and scales from the terms' norms.
__global__ void __launch_bounds__(256) k_aca_tiers(AcaBatch B, TierOut T, int ne)
{
    const int e = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (e >= ne) return;
    const int r = B.rank_out[e];
    const double S = sqrt(fmax(B.s2_out[e], 0.0));
    const long long so = T.soff[e];
    const double* tn = B.tnorm + 3 * so;
    // the tails, added from the last term on (32 terms at a time, an in-order scan)
    int s16 = r, s8 = r;
    double tail = 0.0;
    for (int l1 = r; l1 > 0; l1 -= 32) {
        const int l = l1 - 1 - lane;
        const double sig = l >= 0 ? sqrt(tn[3 * l]) * sqrt(tn[3 * l + 1]) : 0.0;
        double mine = 0.0;
        for (int o = 0; o < 32; o++) {
            tail += __shfl_sync(0xffffffffu, sig, o);
            if (o == lane) mine = tail;
        }
        const bool ok16 = l >= 0 && mine <= TAU16 * S, ok8 = l >= 0 && mine <= TAU8 * S;
        const unsigned m16 = __ballot_sync(0xffffffffu, ok16), m8 = __ballot_sync(0xffffffffu, ok8);
        if (m16) s16 = l1 - 1 - (31 - __clz(m16));
        if (m8) s8 = l1 - 1 - (31 - __clz(m8));
    }
    if (s8 < s16) s8 = s16;
    s8 = r - ((r - s8) & ~3);          // FP8 terms: a multiple of 4
    s16 = s8 - ((s8 - s16) & ~1);      // FP16 terms: a multiple of 2
    if (lane == 0) {
        T.r32[e] = s16;
        T.r16[e] = s8 - s16;
    }
    // v_l's largest entry is its pivot, 1
    for (int l = lane; l < r; l += 32) {
        float a = 1.0f, c = 1.0f;
        if (l >= s8) {
            a = (float)(tn[3 * l + 2] / 448.0);
            c = (float)(1.0 / 448.0);
        } else if (l >= s16) {
            a = (float)tn[3 * l + 2];
        }
        if (!(a > 0.0f)) a = 1.0f;
        T.su[so + l] = a;
        T.sv[so + l] = c;
    }
}

// Mixed storage of one block (m2p = m2 rounded up to 4, s_pad = tile rows rounded up
// to 4).  V^T: r32 FP32 rows of m2p; r16/2 FP16 pair rows, element (j, t) of pair g
// at half index (g m2p + j) 2 + t; r8/4 FP8 quad rows, element (j, t) of quad g at
// byte (g m2p + j) 4 + t; then r FP32 factors su_l sv_l (1 for FP32 terms).  U tile
// slices: s_pad x r32 FP32 column-major, then the pairs [g][i][2] in FP16 and the
// quads [g][i][4] in FP8; a slice takes s_pad * (4 r32 + 2 r16 + r8) bytes.
__global__ void __launch_bounds__(256)
k_aca_compact_mixed(BlockGeom g, AcaBatch B, TierOut T, const int* tile_r0, const int* tile_s,
                    const int* tile_pstart, const int* tfirst, const int* tlast, void* const* ptrU,
                    void* const* ptrV, unsigned* top)
{
    const int e = blockIdx.x;
    const int b = B.blocks[e];
    const int r0 = g.r0[b], m1 = g.m1[b], m2 = g.m2[b];
    const int r = B.rank_out[e];
    if (r == 0) return;
    const int r32 = T.r32[e], r16 = T.r16[e], r8 = r - r32 - r16;
    const long long so = T.soff[e];
    const double* U = B.U + B.uoff[e];
    const double* V = B.V + B.voff[e];
    const int m2p = (m2 + 3) & ~3;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // dst[0 .. rows): the storage words of a word column -- FP32, FP16 pairs or FP8 quads --
    // from term l0 on, rows n.. zero (src + l ld: term l; sc: the terms' scales).  Four
    // entries a lane at a time, so that their loads overlap.
    auto convert = [&](uint32_t* dst, int rows, const double* src, size_t ld, int l0, int kind, int n, const float* sc,
                       unsigned& largest) {
        src += (size_t)l0 * ld;
        const int nt = 1 << kind;
        double q[4];
#pragma unroll
        for (int t = 0; t < 4; t++) q[t] = kind > 0 && t < nt ? (double)sc[l0 + t] : 1.0;
        for (int i0 = lane; i0 < rows; i0 += 128) {
            double x[4][4];
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int t = 0; t < 4; t++) x[u][t] = t < nt && i0 + 32 * u < n ? src[(size_t)t * ld + i0 + 32 * u] : 0.0;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (i0 + 32 * u >= rows) break;
                uint32_t w;
                if (kind == 0) {
                    w = __float_as_uint((float)x[u][0]);
                    largest = max(largest, w & 0x7fffffffu);
                } else if (kind == 1) {
                    const __half2 h = __halves2half2(__float2half_rn((float)(x[u][0] / q[0])), __float2half_rn((float)(x[u][1] / q[1])));
                    w = *reinterpret_cast<const uint32_t*>(&h);
                } else {
                    w = 0u;
#pragma unroll
                    for (int t = 0; t < 4; t++)
                        w |= (uint32_t)__nv_cvt_float_to_fp8((float)(x[u][t] / q[t]), __NV_SATFINITE, __NV_E4M3) << (8 * t);
                }
                dst[i0 + 32 * u] = w;
            }
        }
    };
    // word column c of a block: its tier and first term
    auto column = [&](int c, int& kind, int& l0) {
        kind = c < r32 ? 0 : (c < r32 + (r16 >> 1) ? 1 : 2);
        l0 = kind == 0 ? c : (kind == 1 ? r32 + 2 * (c - r32) : r32 + r16 + 4 * (c - r32 - (r16 >> 1)));
    };
    const int nc = r32 + (r16 >> 1) + (r8 >> 2);
    unsigned top_u = 0u, top_v = 0u;  // of the FP32 words
    uint32_t* vw = reinterpret_cast<uint32_t*>(ptrV[b]);
    for (int c = warp; c < nc; c += 8) {
        int kind, l0;
        column(c, kind, l0);
        convert(vw + (size_t)c * m2p, m2p, V, m2, l0, kind, m2, T.sv + so, top_v);
    }
    float* scal = reinterpret_cast<float*>(vw + (size_t)nc * m2p);
    for (int l = threadIdx.x; l < r; l += blockDim.x) scal[l] = T.su[so + l] * T.sv[so + l];
    // U tile slices
    const int bpr = 4 * nc;
    const int p0 = tile_pstart[tfirst[b]];
    char* ubase = static_cast<char*>(ptrU[b]);
    for (int t = tfirst[b]; t <= tlast[b]; t++) {
        const int s = tile_s[t], sp = (s + 3) & ~3, tr = tile_r0[t] - r0;
        uint32_t* slice = reinterpret_cast<uint32_t*>(ubase + (size_t)(tile_pstart[t] - p0) * bpr);
        for (int c = warp; c < nc; c += 8) {
            int kind, l0;
            column(c, kind, l0);
            convert(slice + (size_t)c * sp, sp, U + tr, m1, l0, kind, s, T.su + so, top_u);
        }
    }
    record_top(top_u, top + 1);
    record_top(top_v, top + 2);
}

void free_far(hmg_matrix* h)
{
    cudaStream_t s = h->stream;
    free_tc(h);
    for (void* p : h->far_chunks) cudaFree(p);
    h->far_chunks.clear();
    h->far_chunk_bytes.clear();
    dfree(h->rank, s);
    dfree(h->rank_off, s);
    dfree(h->ptrU, s);
    dfree(h->ptrV, s);
    dfree(h->tbuf, s);
    dfree(h->far_list, s);
    dfree(h->vt_tasks, s);
    h->vt_large = h->vt_small = 0;
    dfree(h->tier32, s);
    dfree(h->tier16, s);
    h->h_r32.clear();
    h->h_r16.clear();
    h->far_alg_u = h->far_alg_v = 0;
    h->nfar_list = 0;
    h->far_prec = -1;
    h->desc_near_mode = -1;
    h->rank_total = h->far_entries = h->far_rows = h->far_stored = 0;
    h->max_rank = 0;
    h->h_rank.clear();
}

// Scratch of the batches, grown to the largest batch and reused across batches; however
// run_aca returns, its kernels have ended and the scratch is given back.  The factors' part
// is up to 4 GB, which the stream-ordered pool maps and unmaps at 6.3 ms a GB each way; a
// cudaMalloc and its cudaFree take 0.7 ms and 0.8 more a GB (measured), so from 64 MB on it
// comes from there.  (cudaFree waits for the device.  Products of 1.53 ms on another stream,
// beside one construction of 131,072 points after another: p99 115 ms with 16 GB of pool
// scratch and the former kernels, 36 ms now.)
struct AcaScratch {
    static constexpr size_t POOLED = (64u << 20) / sizeof(double);
    hmg_matrix* h;
    double* uv = nullptr;  // the batch's u terms, then its v terms
    size_t cap_uv = 0;
    int *idx = nullptr, *rank = nullptr, *r32 = nullptr, *r16 = nullptr, *list = nullptr;
    long long *uo = nullptr, *vo = nullptr, *so = nullptr;
    double *s2 = nullptr, *tn = nullptr;
    float *su = nullptr, *sv = nullptr;

    explicit AcaScratch(hmg_matrix* m) : h(m) {}
    AcaScratch(const AcaScratch&) = delete;
    AcaScratch& operator=(const AcaScratch&) = delete;
    ~AcaScratch() { release(); }
    void release()
    {
        const cudaStream_t s = h->stream;
        for (cudaStream_t aux : h->k1_aux)
            if (aux) cudaStreamSynchronize(aux);
        cudaStreamSynchronize(s);
        drop();
        dfree(idx, s); dfree(rank, s); dfree(r32, s); dfree(r16, s); dfree(list, s);
        dfree(uo, s); dfree(vo, s); dfree(so, s);
        dfree(s2, s); dfree(tn, s); dfree(su, s); dfree(sv, s);
    }
    void drop()
    {
        if (cap_uv <= POOLED) dfree(uv, h->stream);
        else if (uv) cudaFree(uv);
        uv = nullptr;
        cap_uv = 0;
    }
    hmg_status grow(size_t n)
    {
        drop();
        cap_uv = n > 0 ? n : 1;
        if (cap_uv <= POOLED) return dalloc(&uv, cap_uv, h->stream);
        const cudaError_t e = cudaMalloc((void**)&uv, cap_uv * sizeof(double));
        if (e == cudaSuccess) return HMG_OK;
        cudaGetLastError();
        uv = nullptr;
        set_error("allocating %zu bytes of ACA scratch failed: %s", cap_uv * sizeof(double), cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? HMG_ERR_NOMEM : HMG_ERR_CUDA;
    }
};

hmg_status run_aca(hmg_matrix* h, int k, double eps, int precision)
{
    cudaStream_t s = h->stream;
    hmg_status st = HMG_OK;
    if (k < 1) { set_error("ACA rank bound k must be >= 1 (got %d)", k); return HMG_ERR_INVALID; }
    if (k > ACA_KMAX) {
        set_error("ACA rank bound k=%d exceeds the engine's limit %d", k, ACA_KMAX);
        return HMG_ERR_UNSUPPORTED;
    }
    const bool mixed = precision == HMG_PREC_MIXED;
    if (mixed && !(eps > 0.0)) {
        set_error("mixed-precision factors need the adaptive ACA (eps > 0)");
        return HMG_ERR_INVALID;
    }
    free_far(h);
    const int nb = h->nblocks;
    const size_t esz = precision == HMG_PREC_FP64 ? 8 : 4;
    std::vector<int> rank(nb, 0), r32v(nb, 0), r16v(nb, 0);
    std::vector<void*> pU(nb, nullptr), pV(nb, nullptr);
    long long alg_u = 0, alg_v = 0;
    if ((st = dalloc((int**)&h->rank, (size_t)nb, s)) ||
        (st = dalloc((long long**)&h->rank_off, (size_t)nb + 1, s)) ||
        (st = dalloc((void***)&h->ptrU, (size_t)nb, s)) ||
        (st = dalloc((void***)&h->ptrV, (size_t)nb, s)) ||
        (st = dalloc(&h->tier32, (size_t)nb, s)) || (st = dalloc(&h->tier16, (size_t)nb, s)))
        return st;
    HMG_CUDA_TRY(cudaMemsetAsync(h->stored_top + 1, 0, 2 * sizeof(unsigned), s));

    // batches of admissible blocks whose FP64 scratch fits the budget
    size_t free_b = 0, total_b = 0;
    HMG_CUDA_TRY(cudaMemGetInfo(&free_b, &total_b));
    size_t budget = free_b / 4;
    if (budget > ((size_t)4 << 30)) budget = (size_t)4 << 30;
    if (budget < ((size_t)64 << 20)) budget = (size_t)64 << 20;

    BlockGeom g{h->blk_r0, h->blk_m1, h->blk_c0, h->blk_m2, h->blk_param};
    PointsView P{};
    for (int d = 0; d < h->dim; d++) {
        P.c1[d] = h->zpts[0] + (size_t)d * h->n[0];
        P.c2[d] = h->zpts[1] + (size_t)d * h->n[1];
    }
    P.n1 = h->n[0];
    P.n2 = h->n[1];

    AcaScratch W(h);
    int *&d_idx = W.idx, *&d_rank = W.rank, *&d_r32 = W.r32, *&d_r16 = W.r16, *&d_list = W.list;
    long long *&d_uo = W.uo, *&d_vo = W.vo, *&d_so = W.so;
    double *&dU = W.uv, *&d_s2 = W.s2, *&d_tn = W.tn;
    float *&d_su = W.su, *&d_sv = W.sv;
    size_t cap_ne = 0, cap_sc = 0;
    int bstart = h->ndense;
    while (bstart < nb) {
        std::vector<int> idx;
        std::vector<long long> uo, vo;
        long long us = 0, vs = 0;
        int maxm1 = 1;
        int b = bstart;
        for (; b < nb; b++) {
            int m1 = h->h_m1[b], m2 = h->h_m2[b];
            int kb = std::min(k, std::min(m1, m2));
            long long need = ((long long)m1 + m2) * kb * 8;
            if (!idx.empty() && (us + vs) * 8 + need > (long long)budget) break;
            idx.push_back(b);
            uo.push_back(us);
            vo.push_back(vs);
            us += (long long)m1 * kb;
            vs += (long long)m2 * kb;
            maxm1 = std::max(maxm1, m1);
        }
        bstart = b;
        int ne = (int)idx.size();
        std::vector<long long> so(ne);
        long long nscale = 0;
        for (int e = 0; e < ne; e++) {
            so[e] = nscale;
            nscale += std::min(k, std::min(h->h_m1[idx[e]], h->h_m2[idx[e]]));
        }
        if ((size_t)ne > cap_ne) {
            dfree(d_idx, s); dfree(d_uo, s); dfree(d_vo, s); dfree(d_rank, s); dfree(d_s2, s);
            dfree(d_so, s); dfree(d_r32, s); dfree(d_r16, s); dfree(d_list, s);
            cap_ne = (size_t)ne;
            if ((st = dalloc(&d_idx, cap_ne, s)) || (st = dalloc(&d_uo, cap_ne, s)) || (st = dalloc(&d_vo, cap_ne, s)) ||
                (st = dalloc(&d_rank, cap_ne, s)) || (st = dalloc(&d_s2, cap_ne, s)) || (st = dalloc(&d_list, cap_ne, s)) ||
                (mixed && ((st = dalloc(&d_so, cap_ne, s)) || (st = dalloc(&d_r32, cap_ne, s)) ||
                           (st = dalloc(&d_r16, cap_ne, s)))))
                return st;
        }
        if ((size_t)(us + vs) > W.cap_uv && (st = W.grow((size_t)(us + vs)))) return st;
        if (mixed && (size_t)nscale > cap_sc) {
            dfree(d_su, s);
            dfree(d_sv, s);
            dfree(d_tn, s);
            cap_sc = (size_t)nscale;
            if ((st = dalloc(&d_su, cap_sc, s)) || (st = dalloc(&d_sv, cap_sc, s)) || (st = dalloc(&d_tn, 3 * cap_sc, s)))
                return st;
        }
        HMG_CUDA_TRY(cudaMemcpyAsync(d_idx, idx.data(), sizeof(int) * ne, cudaMemcpyHostToDevice, s));
        HMG_CUDA_TRY(cudaMemcpyAsync(d_uo, uo.data(), sizeof(long long) * ne, cudaMemcpyHostToDevice, s));
        HMG_CUDA_TRY(cudaMemcpyAsync(d_vo, vo.data(), sizeof(long long) * ne, cudaMemcpyHostToDevice, s));
        if (mixed) HMG_CUDA_TRY(cudaMemcpyAsync(d_so, so.data(), sizeof(long long) * ne, cudaMemcpyHostToDevice, s));
        AcaBatch B{d_idx, d_uo, d_vo, dU, dU + us, d_rank, d_s2, mixed ? d_so : nullptr, mixed ? d_tn : nullptr};
        TierOut T{d_r32, d_r16, d_so, d_su, d_sv};
        const size_t mask = eps > 0.0 ? ((size_t)((maxm1 + 31) / 32) * 4 + 7) & ~(size_t)7 : 0;
        if (mask > 200 * 1024) {
            set_error("block with %d rows exceeds the adaptive ACA's row-mask capacity", maxm1);
            return HMG_ERR_UNSUPPORTED;
        }
        // the blocks by class, in each the ones with most work first
        std::vector<int> list(ne);
        std::vector<int> cls(ne);
        int count[ACA_NCLASS] = {}, first[ACA_NCLASS], at[ACA_NCLASS];
        for (int e = 0; e < ne; e++) {
            const int side = std::max(h->h_m1[idx[e]], h->h_m2[idx[e]]);
            int c = 0;
            while (side > ACA_CLASSES[c].side) c++;
            cls[e] = c;
            count[c]++;
        }
        for (int c = ACA_NCLASS - 1, o = 0; c >= 0; o += count[c], c--) first[c] = at[c] = o;
        for (int e = 0; e < ne; e++) list[at[cls[e]]++] = e;
        std::stable_sort(list.begin(), list.begin() + count[ACA_NCLASS - 1], [&](int x, int y) {
            return (long long)h->h_m1[idx[x]] + h->h_m2[idx[x]] > (long long)h->h_m1[idx[y]] + h->h_m2[idx[y]];
        });
        HMG_CUDA_TRY(cudaMemcpyAsync(d_list, list.data(), sizeof(int) * ne, cudaMemcpyHostToDevice, s));
        // on three streams, so that one class's last blocks overlap the next class's first
        // ones; a small batch (the streams and events of a new handle take 0.25 ms to make and
        // destroy, 1700 points at rank 32 3.5 ms to build and multiply) stays on the handle's
        const bool fork = us + vs > (16ll << 20);
        cudaStream_t on[ACA_NCLASS] = {s, s, s, s};
        if (fork) {
            if ((st = ensure_side_streams(h))) return st;
            HMG_CUDA_TRY(cudaEventRecord(h->k1_ev[0], s));
            for (int i = 0; i < 2; i++) HMG_CUDA_TRY(cudaStreamWaitEvent(h->k1_aux[i], h->k1_ev[0], 0));
            on[0] = on[2] = h->k1_aux[0];
            on[1] = h->k1_aux[1];
        }
        auto kc = [&](int c) { return (std::min(k, ACA_CLASSES[c].side) + 1) & ~1; };
        auto bits = [&](int c) { return eps <= 0.0 ? 0 : (c < ACA_NCLASS - 1 ? ACA_CLASSES[c].side / 8 : (int)mask); };
        const int big = std::max(0, ACA_CLASSES[3].panel - bits(3)) & ~15;
        if ((st = launch_aca<512, 2, 1>(g, h->kspec, P, B, k, eps, d_list + first[3], count[3], big, kc(3), bits(3), s)) ||
            (st = launch_aca<512, 1, 2>(g, h->kspec, P, B, k, eps, d_list + first[2], count[2], ACA_CLASSES[2].panel, kc(2), bits(2), on[2])) ||
            (st = launch_aca<256, 1, 3>(g, h->kspec, P, B, k, eps, d_list + first[1], count[1], ACA_CLASSES[1].panel, kc(1), bits(1), on[1])) ||
            (st = launch_small(g, h->kspec, P, B, k, eps, d_list + first[0], count[0], kc(0), bits(0), on[0])))
            return st;
        for (int i = 0; i < 2 && fork; i++) {
            HMG_CUDA_TRY(cudaEventRecord(h->k1_ev[1 + i], h->k1_aux[i]));
            HMG_CUDA_TRY(cudaStreamWaitEvent(s, h->k1_ev[1 + i], 0));
        }
        if (mixed) {
            k_aca_tiers<<<ceil_div(ne, 8), 256, 0, s>>>(B, T, ne);
            HMG_LAUNCH_CHECK();
        }
        std::vector<int> br(ne), b32(ne, 0), b16(ne, 0);
        HMG_CUDA_TRY(cudaMemcpyAsync(br.data(), d_rank, sizeof(int) * ne, cudaMemcpyDeviceToHost, s));
        if (mixed) {
            HMG_CUDA_TRY(cudaMemcpyAsync(b32.data(), d_r32, sizeof(int) * ne, cudaMemcpyDeviceToHost, s));
            HMG_CUDA_TRY(cudaMemcpyAsync(b16.data(), d_r16, sizeof(int) * ne, cudaMemcpyDeviceToHost, s));
        }
        HMG_CUDA_TRY(cudaStreamSynchronize(s));
        // final storage of this batch
        long long bytes = 0;
        std::vector<long long> ofsU(ne), ofsV(ne);
        for (int e = 0; e < ne; e++) {
            int bb = idx[e], r = br[e];
            rank[bb] = r;
            const long long rows_p = h->h_tile_pstart[h->h_blk_tlast[bb] + 1] -
                                     h->h_tile_pstart[h->h_blk_tfirst[bb]];
            const long long m1 = h->h_m1[bb], m2 = h->h_m2[bb];
            ofsU[e] = bytes;
            if (mixed) {
                const int r32 = b32[e], r16 = b16[e], r8 = r - r32 - r16;
                r32v[bb] = r32;
                r16v[bb] = r16;
                const long long bpr = 4 * r32 + 2 * r16 + r8;
                bytes += rows_p * bpr;
                bytes = (bytes + 255) & ~255ll;
                ofsV[e] = bytes;
                bytes += ((m2 + 3) & ~3) * bpr + 4ll * r;
                alg_u += m1 * (4ll * r32 + 2ll * r16 + r8);
                alg_v += m2 * (4ll * r32 + 2ll * r16 + r8);
            } else {
                r32v[bb] = r;
                bytes += rows_p * r * (long long)esz;
                bytes = (bytes + 255) & ~255ll;
                ofsV[e] = bytes;
                bytes += (long long)r * ((m2 + 3) & ~3) * (long long)esz;
                alg_u += m1 * r * (long long)esz;
                alg_v += m2 * r * (long long)esz;
            }
            bytes = (bytes + 255) & ~255ll;
        }
        char* chunk = nullptr;
        if (bytes > 0) {
            cudaError_t ce = cudaMalloc((void**)&chunk, (size_t)bytes);
            if (ce != cudaSuccess) {
                cudaGetLastError();
                set_error("allocating %lld bytes of low-rank factors failed: %s", bytes,
                          cudaGetErrorString(ce));
                return ce == cudaErrorMemoryAllocation ? HMG_ERR_NOMEM : HMG_ERR_CUDA;
            }
            h->far_chunks.push_back(chunk);
            h->far_chunk_bytes.push_back((size_t)bytes);
            h->far_stored += bytes;
            for (int e = 0; e < ne; e++) {
                pU[idx[e]] = chunk + ofsU[e];
                pV[idx[e]] = chunk + ofsV[e];
            }
            // the batch is a contiguous block range
            HMG_CUDA_TRY(cudaMemcpyAsync(h->ptrU + idx[0], pU.data() + idx[0], sizeof(void*) * ne,
                                         cudaMemcpyHostToDevice, s));
            HMG_CUDA_TRY(cudaMemcpyAsync(h->ptrV + idx[0], pV.data() + idx[0], sizeof(void*) * ne,
                                         cudaMemcpyHostToDevice, s));
            if (mixed)
                k_aca_compact_mixed<<<ne, 256, 0, s>>>(g, B, T, h->tile_r0, h->tile_s, h->tile_pstart,
                                                       h->blk_tfirst, h->blk_tlast, h->ptrU, h->ptrV, h->stored_top);
            else if (precision == HMG_PREC_FP64)
                k_aca_compact<double><<<ne, 256, 0, s>>>(g, B, h->tile_r0, h->tile_s, h->tile_pstart,
                                                         h->blk_tfirst, h->blk_tlast,
                                                         (double* const*)h->ptrU, (double* const*)h->ptrV, nullptr);
            else
                k_aca_compact<float><<<ne, 256, 0, s>>>(g, B, h->tile_r0, h->tile_s, h->tile_pstart,
                                                        h->blk_tfirst, h->blk_tlast,
                                                        (float* const*)h->ptrU, (float* const*)h->ptrV, h->stored_top);
            HMG_LAUNCH_CHECK();
        }
        HMG_CUDA_TRY(cudaStreamSynchronize(s));
    }
    W.release();

    // ranks and their offsets
    std::vector<long long> roff(nb + 1, 0);
    h->far_entries = h->far_rows = 0;
    h->max_rank = 0;
    for (int b = 0; b < nb; b++) {
        roff[b + 1] = roff[b] + rank[b];
        if (h->h_type[b] == HMG_WT_ACA) {
            h->far_entries += (long long)(h->h_m1[b] + h->h_m2[b]) * rank[b];
            h->far_rows += h->h_m1[b] + h->h_m2[b];
            h->max_rank = std::max(h->max_rank, rank[b]);
        }
    }
    h->rank_total = roff[nb];
    HMG_CUDA_TRY(cudaMemcpyAsync(h->rank, rank.data(), sizeof(int) * nb, cudaMemcpyHostToDevice, s));
    HMG_CUDA_TRY(cudaMemcpyAsync(h->tier32, r32v.data(), sizeof(int) * nb, cudaMemcpyHostToDevice, s));
    HMG_CUDA_TRY(cudaMemcpyAsync(h->tier16, r16v.data(), sizeof(int) * nb, cudaMemcpyHostToDevice, s));
    h->h_r32 = r32v;
    h->h_r16 = r16v;
    h->far_alg_u = alg_u;
    h->far_alg_v = alg_v;
    HMG_CUDA_TRY(cudaMemcpyAsync(h->rank_off, roff.data(), sizeof(long long) * (nb + 1), cudaMemcpyHostToDevice, s));
    // padded and zeroed: the streaming product copies 16-byte-aligned supersets of t_b
    if ((st = dalloc((char**)&h->tbuf, (size_t)(h->rank_total + 32) * 8, s))) return st;
    HMG_CUDA_TRY(cudaMemsetAsync(h->tbuf, 0, (size_t)(h->rank_total + 32) * 8, s));
    HMG_CUDA_TRY(cudaStreamSynchronize(s));
    h->h_rank = rank;
    h->far_prec = precision;
    h->aca_k = k;
    h->aca_eps = eps;
    return HMG_OK;
}

}  // namespace hmg
