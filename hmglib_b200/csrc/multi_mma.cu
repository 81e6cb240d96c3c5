// multi_mma.cu -- Y = H X for 2 to 32 vectors over FP32 or mixed storage, on the
// tensor cores with FP32 accuracy.
//
// The reference multiplies one vector per call (apply_h_matrix_mvp, hmglib.cu:271-286).
// Here every stored value is read once for all vectors, straight into the fragments of
// mma.sync m16n8k16 (BF16 operands, FP32 accumulator): the product is bound by the bytes
// of the stored H-matrix, and a lane's own 16-byte loads already are its A fragments
// (4 rows of a chunk column, or 4 columns of a V row), so no operand passes through a
// shared tile or a descriptor.  The K order of an MMA is free as long as A and B agree:
// each storage tier orders its terms so that the loads fit.
//
// FP32 accuracy from BF16 operands.  A value is cut into BF16 parts of 8 bits each, exactly:
// three for FP32, two for FP16 and one for FP8.  All products of parts are formed but
// tail x tail, at most 2^-32 of the whole.  The accumulator truncates, and a chain of
// truncations is biased, so a chain is one step of 16 columns or terms: the heads' product
// e from zero; its remainder (the heads once more, from -e) and the other products in two
// chains, smallest first; these are added up, and added to the sum, on the CUDA cores
// (rounded to nearest).  A head product has 16 bits, so what e and the remainder miss lies below 2^-24
// of the step's largest product.  FP16 and FP8 terms, 1e-4 of a block and less, go without
// the remainder.  Against 64 bits, sums of 96 products: 5.5e-8 relative, without a mean
// shift, against 1.8e-7 for a chain of FP32 multiply-adds (values over a range of e^10, all
// of one sign: 5.7e-8, 3.5e-8 of it low, against 1.5e-7); a product with a unit vector
// returns the stored value.  Two TF32 parts and three products (6 MMAs for 16 columns, not
// 9) lost the last bit of a quarter of the values and 4e-8 of every sum: unit vectors
// were off by up to 1.6e-7, and CG on 8192 clustered points took 4785-4899 iterations instead
// of 4571-4778.
// Sums of a (tile, block) pair stay FP32 and pairs are added in FP64, as in the
// single-vector product.  Deterministic.
//
// Measured at N = 2^17 (uniform 3D, Matern, mixed storage, 8.0 GB: 1.23 ms at the copy
// peak) against the CUDA-core kernels (packed FP32 multiply-adds) this replaces: 8
// vectors 3.42 ms (7.18), 16 5.10 (9.45), 24 6.34 (14.1), 32 8.41 (14.1); with the two TF32
// parts 2.77, 3.95, 5.16 and 6.94.  Bound by instruction issue (8 vectors: 52-61 % active) and
// the latency of the MMA chains (32: tensor pipe 40-53 % busy), not by memory.
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "hmg_matrix.cuh"
#include "stream.cuh"

namespace hmg {

// 16-byte asynchronous copies global -> shared; an invalid source zeroes the destination.
// Stored data bypasses L1 and asks L2 for the whole 256-byte group; vectors stay in L1,
// where the warps of the neighbouring rows find them.
__device__ __forceinline__ void cp_stored16(uint32_t dst, const void* src, bool valid)
{
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
// the same where `on` (warp-uniform), without a branch
__device__ __forceinline__ void cp_stored16_if(uint32_t dst, const void* src, bool valid, bool on)
{
    const int n = valid ? 16 : 0;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t"
                 "@p cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;\n\t}" ::"r"(dst), "l"(src), "r"(n), "r"((int)on)
                 : "memory");
}
__device__ __forceinline__ void cp_vector16(uint32_t dst, const void* src, bool valid)
{
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// d = A B + c: A 16 x 16, B 16 x 8, d 16 x 8 (row g columns 2t, 2t + 1, then row g + 8).  A
// register of A or B holds two K slots; lane (g, t) has A rows g, g + 8 and B column g.  The
// kernels think of it as two K steps of 8: slot t or t + 4 (the register) of the first (its
// low half) and of the second step (its high half).
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2],
                                         const float (&c)[4])
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%10, %11, %12, %13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}

// The first PARTS runs of 8 bits of v0 and v1, as BF16 pairs (v0 in the low halves).  Cut,
// not rounded: each rest is exact and three parts hold an FP32 value.
template <int PARTS> __device__ __forceinline__ void split_pair(uint32_t v0, uint32_t v1, uint32_t (&p)[PARTS])
{
#pragma unroll
    for (int i = 0; i < PARTS; i++) {
        p[i] = __byte_perm(v0, v1, 0x7632);
        if (i + 1 < PARTS) {
            v0 = __float_as_uint(__uint_as_float(v0) - __uint_as_float(v0 & 0xffff0000u));
            v1 = __float_as_uint(__uint_as_float(v1) - __uint_as_float(v1 & 0xffff0000u));
        }
    }
}

// acc += d, two lanes of FP32 at a time
__device__ __forceinline__ void add4(float (&acc)[4], const float (&d)[4])
{
    asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%4, %5};\n\tadd.rn.f32x2 a, a, b;\n\t"
        "mov.b64 {%0, %1}, a;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%6, %7};\n\tadd.rn.f32x2 a, a, b;\n\t"
        "mov.b64 {%2, %3}, a;\n\t}"
        : "+f"(acc[0]), "+f"(acc[1]), "+f"(acc[2]), "+f"(acc[3])
        : "f"(d[0]), "f"(d[1]), "f"(d[2]), "f"(d[3]));
}

// The B fragments of a step for NT groups of 8 vectors, split: rows (lo0, hi0) and (lo1, hi1)
// are the K slots of its two registers.
template <int NT> struct FragB {
    uint32_t p[3][NT][2];
    __device__ __forceinline__ void get(const float* lo0, const float* lo1, const float* hi0, const float* hi1)
    {
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int q = 0; q < 2; q++) {
                uint32_t x[3];
                split_pair<3>(__float_as_uint((q ? lo1 : lo0)[8 * j]), __float_as_uint((q ? hi1 : hi0)[8 * j]), x);
                // kept in registers: loaded and split anew for every M tile otherwise
                asm volatile("" : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]));
#pragma unroll
                for (int i = 0; i < 3; i++) p[i][j][q] = x[i];
            }
    }
};

// What the MMAs multiply must split and must not overflow on the way: an infinity or a NaN
// does neither (inf - inf), nor does a part below BF16's range hold its bits.  The kernels
// that write vectors record their range: range[j] the largest magnitude of vector j of X (the
// bits of an FP32 value), range[RANGE_T] whether an entry of t is too large.  The kernels
// launched after them, which read these vectors, multiply with FP32 multiply-adds instead
// (step_fma) where a vector lies outside.  No kernel reads what it records itself: its warps
// would disagree.  The kernels that write the stored FP32 values record their largest
// (stored_top: near field, U, V), and a load looks for them (scan_stored_top).  Within the range, the sum of a pair, at most 512 products of a stored
// value below 2^40 and an entry of X or t below 2^78, is finite, and so is a sum over a block's
// columns, whose entries of V are below 2^9; the parts lose what lies below 2^-133, at most
// 2^-63 of a vector's and 2^-103 of the storage's largest value.
static constexpr unsigned RANGE_LARGE = (127u + 78) << 23, RANGE_SMALL = (127u - 70) << 23;
static constexpr unsigned STORED_LARGE = (127u + 40) << 23, STORED_SMALL = (127u - 30) << 23;
static constexpr unsigned V_LARGE = (127u + 9) << 23;
static constexpr int RANGE_T = 32;
static_assert(MULTI_RANGE_WORDS == RANGE_T + 1, "the record's words");
__device__ __forceinline__ bool too_large(float v) { return magnitude(v) >= RANGE_LARGE; }
// the same in every warp
__device__ __forceinline__ bool out_of_range(const unsigned* range, int R, const unsigned* stored)
{
    const int lane = threadIdx.x & 31;
    const unsigned a = max(stored[0], stored[1]);
    if (a >= STORED_LARGE || (a != 0u && a < STORED_SMALL) || stored[2] >= V_LARGE) return true;
    const unsigned top = lane < R ? range[lane] : 0u;
    return __any_sync(0xffffffffu, top >= RANGE_LARGE || (top != 0u && top < RANGE_SMALL));
}

// acc[j] += A B_j for one step: A cut into three parts (FP32: nine MMAs), two (FP16: six) or
// one (FP8: three)
template <int NT, int PARTS>
__device__ __forceinline__ void step_mma(float (&acc)[NT][4], const uint32_t (&a0)[4], const uint32_t (&a1)[4],
                                         const FragB<NT>& b)
{
    const float zero[4] = {0.f, 0.f, 0.f, 0.f};
    uint32_t a[PARTS][4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        uint32_t x[PARTS];
        split_pair<PARTS>(a0[q], a1[q], x);
#pragma unroll
        for (int i = 0; i < PARTS; i++) a[i][q] = x[i];
    }
#pragma unroll
    for (int j = 0; j < NT; j++) {
        float e[4], d[4], r[4];
        mma_bf16(e, a[0], b.p[0][j], zero);
        if constexpr (PARTS == 3) {
            mma_bf16(d, a[2], b.p[1][j], zero);
            mma_bf16(d, a[2], b.p[0][j], d);
            mma_bf16(d, a[1], b.p[1][j], d);
            mma_bf16(d, a[1], b.p[0][j], d);
            const float n[4] = {-e[0], -e[1], -e[2], -e[3]};
            mma_bf16(r, a[0], b.p[0][j], n);
            mma_bf16(r, a[1], b.p[2][j], r);
            mma_bf16(r, a[0], b.p[2][j], r);
            mma_bf16(r, a[0], b.p[1][j], r);
            add4(d, r);
        } else if constexpr (PARTS == 2) {
            mma_bf16(d, a[1], b.p[2][j], zero);
            mma_bf16(d, a[1], b.p[1][j], d);
            mma_bf16(d, a[0], b.p[2][j], d);
            mma_bf16(d, a[1], b.p[0][j], d);
            mma_bf16(d, a[0], b.p[1][j], d);
        } else {
            mma_bf16(d, a[0], b.p[2][j], zero);
            mma_bf16(d, a[0], b.p[1][j], d);
        }
        add4(d, e);
        add4(acc[j], d);
    }
}

// Half of the step (8 K slots) with FP32 multiply-adds: A from the warp's fragments, B row
// kk (slot order) at b(kk).
template <int NT, class F>
__device__ __forceinline__ void step_fma(float (&acc)[NT][4], const uint32_t (&a)[4], F b)
{
    const int lane = threadIdx.x & 31, lt = lane & 3;
#pragma unroll 1
    for (int kk = 0; kk < 8; kk++) {
        const int src = (lane & 28) | (kk & 3);
        const float x = __uint_as_float(__shfl_sync(0xffffffffu, kk < 4 ? a[0] : a[2], src));
        const float y = __uint_as_float(__shfl_sync(0xffffffffu, kk < 4 ? a[1] : a[3], src));
        const float* r = b(kk) + 2 * lt;
#pragma unroll
        for (int j = 0; j < NT; j++) {
            acc[j][0] = fmaf(x, r[8 * j], acc[j][0]);
            acc[j][1] = fmaf(x, r[8 * j + 1], acc[j][1]);
            acc[j][2] = fmaf(y, r[8 * j], acc[j][2]);
            acc[j][3] = fmaf(y, r[8 * j + 1], acc[j][3]);
        }
    }
}

__device__ __forceinline__ float2 half2_to_float2(uint32_t w)
{
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
__device__ __forceinline__ float2 e4m3x2_to_float2(uint32_t w)
{
    const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w & 0xffffu), __NV_E4M3);
    return __half22float2(*reinterpret_cast<const __half2*>(&h));
}

// X (caller order, column-major, FP64) as R FP32 values per point in Z order, and the
// vectors' largest magnitudes (256 threads a CTA)
__global__ void k_gather_mma(const double* X, int ldx, int nrhs, const int* perm2, int n, int R, float* xm, unsigned* range)
{
    __shared__ unsigned top[32];
    if (threadIdx.x < 32) top[threadIdx.x] = 0u;
    __syncthreads();
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx < (long long)n * R) {
        const int i = (int)(idx / R), j = (int)(idx - (long long)i * R);
        const float v = j < nrhs ? (float)X[perm2[i] + (size_t)j * ldx] : 0.0f;
        xm[idx] = v;
        atomicMax(&top[j], magnitude(v));
    }
    __syncthreads();
    // (read first: after a few CTAs hardly any has a larger one)
    if (threadIdx.x < R && top[threadIdx.x] > *static_cast<volatile unsigned*>(range + threadIdx.x))
        atomicMax(range + threadIdx.x, top[threadIdx.x]);
}

// ---------------------------------------------------------------------------
// V^T X
// ---------------------------------------------------------------------------
// Up to 64 terms of one block.  V_b^T is n32 FP32 rows, then n16 / 2 rows of FP16 pairs
// and n8 / 4 rows of FP8 quads, all with the same stride; its terms are cut into M tiles
// of 16 terms of one tier, and a task takes cnt of them from tile mt0.
struct VtTask {
    const char* v;
    const float* scal;   // scales of the block's terms (FP16 / FP8), else null
    long long tout;      // t row of the block's first term
    int c0, m2, chunks;  // columns; 16-byte chunks a row
    int n32, n16, n8;
    int mt0, cnt;
};

static constexpr int VT_MT = 4;         // most M tiles a task
static constexpr int VT_LD = 6;         // most 512-byte loads a step: two an FP32 tile, one an FP16 or FP8 tile
// Blocks with more columns than this are multiplied by all warps of a CTA, each over its
// share of the columns: one warp keeps about 4 KB in flight, so a 16384-column task
// (4 MB) would take it 200 us, as long as a whole product of 2^16 points.
static constexpr int VT_SPLIT_COLS = 1024;

template <int NT> struct VtShape {
    static constexpr int R = 8 * NT;
    // warps a CTA: what shared memory holds of rings and partial sums (206, 197, 159, 187 KB)
    static constexpr int WARPS = NT == 1 ? 16 : (NT == 2 ? 12 : 8);
    static constexpr int NS = 3;                                     // stages a warp
    static constexpr int BF = 16 * R + 32;                           // floats of a stage's 16 X rows
    static constexpr int STAGE = VT_LD * 512 + BF * 4;
    static constexpr int PART = VT_MT * 16 * R * 4;                  // one warp's partial sums
    static constexpr int SMEM = WARPS * (NS * STAGE + PART);
    static_assert(SMEM <= 227 * 1024, "the shared memory of a CTA");
};

// t_b = V_b^T X_b, scaled.  M = 16 terms, N = 8 vectors, K = 16 columns of each MMA, a step.
// A lane's 16 bytes are columns 4t .. 4t+3 of a row: columns 4t, 4t+1 are its K slots t, t+4
// of the first half of the step and 4t+2, 4t+3 of the second.  An FP16 row
// gives terms 2g, 2g+1 (M slots g, g+8); an FP8 row is read by two lane groups, each
// taking two of its four terms.  Copies run ahead across tasks in a ring per warp, each
// lane reading back what it copied (only X is shared by the warp).
template <int NT>
__global__ void __launch_bounds__(VtShape<NT>::WARPS * 32, 1)
k_vtx_mma(const VtTask* __restrict__ tasks, int nlarge, int nsmall, const float* __restrict__ xm,
           float* __restrict__ tm, unsigned* range, const unsigned* stored)
{
    typedef VtShape<NT> S;
    constexpr int R = S::R, NS = S::NS, WARPS = S::WARPS;
    extern __shared__ __align__(16) char vt_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lg = lane >> 2, lt = lane & 3;
    char* ring = vt_smem + (size_t)warp * NS * S::STAGE;
    float* part = reinterpret_cast<float*>(vt_smem + (size_t)WARPS * NS * S::STAGE);
    const uint32_t ring_s = static_cast<uint32_t>(__cvta_generic_to_shared(ring));
    const int nw = gridDim.x * WARPS, gw = blockIdx.x * WARPS + warp;

    // the warp's task sequence: the CTA's large tasks (its share of the columns), then
    // small tasks of its own
    auto first_task = [&]() { return (int)blockIdx.x < nlarge ? (int)blockIdx.x : nlarge + gw; };
    auto next_task = [&](int t) {
        if (t >= nlarge) return t + nw;
        return t + (int)gridDim.x < nlarge ? t + (int)gridDim.x : nlarge + gw;
    };
    auto steps_of = [&](int chunks, int ti, int& s0, int& s1) {
        const int ns = (chunks + 3) >> 2;
        s0 = 0;
        s1 = ns;
        if (ti < nlarge) {
            s0 = ns * warp / WARPS;  // ns > 64: no share is empty
            s1 = ns * (warp + 1) / WARPS;
        }
    };
    const int ntask = nlarge + nsmall;
    const bool plain = out_of_range(range, R, stored);
    bool large = false;

    // producer: the lane's rows of the task (offsets from the block's V, which may pass 4 GiB,
    // a bit per row that exists), its X rows, and the step
    int pt = first_task(), left = 0, cleft = 0, xleft = 0, nload = 0;
    const char* vp = nullptr;   // the lane's chunk of the next step, row 0
    const float* xp = nullptr;  // X row of the next step's first column
    size_t off[VT_LD];
    uint32_t rows = 0;
    uint32_t xdst[NT];
    int xsrc[NT], xcol[NT];
#pragma unroll
    for (int i = 0; i < NT; i++) {
        const int e = lane + 32 * i, c4 = e % (2 * NT);
        xcol[i] = e / (2 * NT);
        xsrc[i] = xcol[i] * R + c4 * 4;
        xdst[i] = VT_LD * 512 + (xcol[i] * R + (xcol[i] >> 2) * 8 + c4 * 4) * 4;
    }
    auto open_task = [&]() {
        if (pt >= ntask) return;
        const VtTask p = tasks[pt];
        int s0, s1;
        steps_of(p.chunks, pt, s0, s1);
        left = s1 - s0;
        cleft = p.chunks - 4 * s0 - lt;
        xleft = p.m2 - 16 * s0;
        vp = p.v + (size_t)(4 * s0 + lt) * 16;
        xp = xm + (size_t)(p.c0 + 16 * s0) * R;
        const int nm32 = (p.n32 + 15) >> 4, nm16 = (p.n16 + 15) >> 4;
        const int f = max(0, min(nm32 - p.mt0, p.cnt));  // FP32 tiles of the task
        nload = p.cnt + f;
        rows = 0;
#pragma unroll
        for (int i = 0; i < VT_LD; i++) {
            const int mt = p.mt0 + (i < 2 * f ? i >> 1 : i - f);
            int r, end;
            if (mt < nm32) {
                r = mt * 16 + lg + 8 * (i & 1);
                end = p.n32;
            } else if (mt < nm32 + nm16) {
                r = p.n32 + (mt - nm32) * 8 + lg;
                end = p.n32 + (p.n16 >> 1);
            } else {
                r = p.n32 + (p.n16 >> 1) + (mt - nm32 - nm16) * 4 + (lg >> 1);
                end = p.n32 + (p.n16 >> 1) + (p.n8 >> 2);
            }
            off[i] = (size_t)r * p.chunks * 16;
            if (r < end) rows |= 1u << i;
        }
    };
    open_task();
    uint32_t pslot = 0;  // byte offset of the producer's stage
    auto issue = [&]() {
        if (pt < ntask) {
            const uint32_t sa = ring_s + pslot + lane * 16;
            const uint32_t have = cleft > 0 ? rows : 0u;
#pragma unroll
            for (int i = 0; i < VT_LD; i++) {
                cp_stored16_if(sa + i * 512, vp + off[i], (have >> i) & 1u, i < nload);
            }
#pragma unroll
            for (int i = 0; i < NT; i++) cp_vector16(ring_s + pslot + xdst[i], xp + xsrc[i], xcol[i] < xleft);
            pslot = pslot + S::STAGE == NS * S::STAGE ? 0u : pslot + S::STAGE;
            vp += 64;
            xp += 16 * R;
            cleft -= 4;
            xleft -= 16;
            if (--left == 0) {
                pt = next_task(pt);
                open_task();
            }
        }
        cp_commit();
    };

    float acc[VT_MT][NT][4];
#pragma unroll
    for (int m = 0; m < VT_MT; m++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[m][j][q] = 0.0f;
    for (int i = 0; i < NS - 1; i++) issue();
    auto run = [&](auto plain_c) {
    constexpr bool PLAIN = decltype(plain_c)::value;
    uint32_t cslot = 0;
    for (int ct = first_task(); ct < ntask; ct = next_task(ct)) {
        const VtTask c = tasks[ct];
        const int nm32 = (c.n32 + 15) >> 4, nm16 = (c.n16 + 15) >> 4;
        const int c32 = max(0, nm32 - c.mt0), c16 = max(0, nm32 + nm16 - c.mt0);  // first tile of each short tier
        int s0, s1;
        steps_of(c.chunks, ct, s0, s1);
        for (int st = s0; st < s1; st++) {
            issue();
            cp_wait<NS - 1>();
            __syncwarp();
            const char* sa = ring + cslot + lane * 16;
            const float* sb = reinterpret_cast<const float*>(ring + cslot + VT_LD * 512);
            FragB<NT> b;
            const float* bp = sb + 4 * lt * R + lt * 8 + lg;
            b.get(bp, bp + R, bp + 2 * R, bp + 3 * R);
#pragma unroll
            for (int m = 0; m < VT_MT; m++) {
                if (m >= c.cnt) break;
                const char* sm = sa + (m + min(m, c32)) * 512;
                const uint4 w0 = *reinterpret_cast<const uint4*>(sm);
                uint32_t a[2][4];
                if (m < c32) {
                    const uint4 w1 = *reinterpret_cast<const uint4*>(sm + 512);
                    a[0][0] = w0.x; a[0][1] = w1.x; a[0][2] = w0.y; a[0][3] = w1.y;
                    a[1][0] = w0.z; a[1][1] = w1.z; a[1][2] = w0.w; a[1][3] = w1.w;
                    if constexpr (!PLAIN) step_mma<NT, 3>(acc[m], a[0], a[1], b);
                } else {
                    const uint32_t w[4] = {w0.x, w0.y, w0.z, w0.w};
                    const bool h16 = m < c16;
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float2 f = h16 ? half2_to_float2(w[q]) : e4m3x2_to_float2(w[q] >> (16 * (lg & 1)));
                        a[q >> 1][2 * (q & 1)] = __float_as_uint(f.x);
                        a[q >> 1][2 * (q & 1) + 1] = __float_as_uint(f.y);
                    }
                    if constexpr (!PLAIN) {
                        if (h16) step_mma<NT, 2>(acc[m], a[0], a[1], b);
                        else step_mma<NT, 1>(acc[m], a[0], a[1], b);
                    }
                }
                if constexpr (PLAIN)
                    for (int h = 0; h < 2; h++)
                        step_fma<NT>(acc[m], h ? a[1] : a[0], [&](int kk) {
                            const int col = 4 * (kk & 3) + 2 * h + (kk >> 2);
                            return sb + col * R + (col >> 2) * 8;
                        });
            }
            cslot = cslot + S::STAGE == NS * S::STAGE ? 0u : cslot + S::STAGE;
            __syncwarp();  // the slot is refilled next
        }
        // term of M slot (m, half): FP32 rows g, g + 8; pairs 2g, 2g + 1
        auto term_of = [&](int m, int half) {
            if (m < c32) {
                const int r = (c.mt0 + m) * 16 + lg + 8 * half;
                return r < c.n32 ? r : -1;
            }
            const bool h16 = m < c16;
            const int r = (c.mt0 + m - nm32 - (h16 ? 0 : nm16)) * 16 + 2 * lg + half;
            if (r >= (h16 ? c.n16 : c.n8)) return -1;
            return c.n32 + (h16 ? 0 : c.n16) + r;
        };
        if (ct < nlarge) {
            // the warps' shares of the columns, added in warp order
            float* mine = part + (size_t)warp * (VT_MT * 16 * R);
#pragma unroll
            for (int m = 0; m < VT_MT; m++)
#pragma unroll
                for (int j = 0; j < NT; j++)
#pragma unroll
                    for (int half = 0; half < 2; half++)
                        *reinterpret_cast<float2*>(mine + (m * 16 + lg + 8 * half) * R + 8 * j + 2 * lt) =
                            make_float2(acc[m][j][2 * half], acc[m][j][2 * half + 1]);
            __syncthreads();
#pragma unroll
            for (int m = 0; m < VT_MT; m++)
#pragma unroll
                for (int j = 0; j < NT; j++)
#pragma unroll
                    for (int half = 0; half < 2; half++) {
                        // warp w sums the w-th of the (m, j, half) pieces
                        if (((m * NT + j) * 2 + half) % WARPS != warp) continue;
                        float2 s = make_float2(0.f, 0.f);
#pragma unroll
                        for (int w = 0; w < WARPS; w++) {
                            const float2 v = *reinterpret_cast<const float2*>(
                                part + (size_t)w * (VT_MT * 16 * R) + (m * 16 + lg + 8 * half) * R + 8 * j + 2 * lt);
                            s.x += v.x;
                            s.y += v.y;
                        }
                        const int term = m < c.cnt ? term_of(m, half) : -1;
                        if (term >= 0) {
                            if (c.scal) {
                                s.x *= c.scal[term];
                                s.y *= c.scal[term];
                            }
                            large = large || too_large(s.x) || too_large(s.y);
                            *reinterpret_cast<float2*>(tm + (size_t)(c.tout + term) * R + 8 * j + 2 * lt) = s;
                        }
                    }
            __syncthreads();
        } else {
#pragma unroll
            for (int m = 0; m < VT_MT; m++)
#pragma unroll
                for (int half = 0; half < 2; half++) {
                    const int term = m < c.cnt ? term_of(m, half) : -1;
                    if (term < 0) continue;
                    const float sc = c.scal ? c.scal[term] : 1.0f;
#pragma unroll
                    for (int j = 0; j < NT; j++) {
                        const float2 s = make_float2(acc[m][j][2 * half] * sc, acc[m][j][2 * half + 1] * sc);
                        large = large || too_large(s.x) || too_large(s.y);
                        *reinterpret_cast<float2*>(tm + (size_t)(c.tout + term) * R + 8 * j + 2 * lt) = s;
                    }
                }
        }
#pragma unroll
        for (int m = 0; m < VT_MT; m++)
#pragma unroll
            for (int j = 0; j < NT; j++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[m][j][q] = 0.0f;
    }
    };
    if (plain) run(std::true_type{});
    else run(std::false_type{});
    cp_wait<0>();
    if (large) range[RANGE_T] = 1u;
}

struct VtItem {
    int b, mt0, cnt;
};

__global__ void k_build_vt(const VtItem* items, int n, const int* blk_c0, const int* blk_m2, const int* rank,
                           const int* tier32, const int* tier16, const long long* rank_off, void* const* ptrV,
                           int mixed, VtTask* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const VtItem it = items[i];
    const int b = it.b, r = rank[b];
    VtTask t;
    t.n32 = mixed ? tier32[b] : r;
    t.n16 = mixed ? tier16[b] : 0;
    t.n8 = r - t.n32 - t.n16;
    t.c0 = blk_c0[b];
    t.m2 = blk_m2[b];
    t.chunks = (t.m2 + 3) >> 2;
    t.v = static_cast<const char*>(ptrV[b]);
    t.scal = mixed ? reinterpret_cast<const float*>(t.v + (size_t)t.chunks * 16 * (t.n32 + (t.n16 >> 1) + (t.n8 >> 2)))
                   : nullptr;
    t.tout = rank_off[b];
    t.mt0 = it.mt0;
    t.cnt = it.cnt;
    out[i] = t;
}

// The V^T X tasks of the stored factors, the split (large) ones first.
static hmg_status ensure_vt(hmg_matrix* h)
{
    if (h->vt_tasks) return HMG_OK;
    cudaStream_t s = h->stream;
    hmg_status st;
    const bool mixed = h->far_prec == HMG_PREC_MIXED;
    std::vector<VtItem> large, small;
    for (int b = h->ndense; b < h->nblocks; b++) {
        const int r = h->h_rank.empty() ? 0 : h->h_rank[b];
        if (r == 0) continue;
        const int n32 = mixed ? h->h_r32[b] : r, n16 = mixed ? h->h_r16[b] : 0, n8 = r - n32 - n16;
        const int nm = ((n32 + 15) >> 4) + ((n16 + 15) >> 4) + ((n8 + 15) >> 4);
        const int nm32 = (n32 + 15) >> 4;
        std::vector<VtItem>& to = h->h_m2[b] > VT_SPLIT_COLS ? large : small;
        for (int m = 0; m < nm;) {
            int c = 0, ld = 0;
            while (c < VT_MT && m + c < nm && ld + (m + c < nm32 ? 2 : 1) <= VT_LD) ld += m + c < nm32 ? 2 : 1, c++;
            to.push_back({b, m, c});
            m += c;
        }
    }
    h->vt_large = (int)large.size();
    h->vt_small = (int)small.size();
    large.insert(large.end(), small.begin(), small.end());
    const int n = (int)large.size();
    VtTask* t = nullptr;
    VtItem* d = nullptr;
    if ((st = dalloc(&t, (size_t)n, s))) return st;
    if (n > 0) {
        if ((st = dalloc(&d, (size_t)n, s))) {
            dfree(t, s);
            return st;
        }
        cudaError_t e = cudaMemcpyAsync(d, large.data(), sizeof(VtItem) * n, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) {
            k_build_vt<<<ceil_div(n, 256), 256, 0, s>>>(d, n, h->blk_c0, h->blk_m2, h->rank, h->tier32, h->tier16,
                                                        h->rank_off, h->ptrV, mixed ? 1 : 0, t);
            e = cudaGetLastError();
        }
        dfree(d, s);
        const cudaError_t done = cudaStreamSynchronize(s);  // the host vector goes out of scope
        if (e == cudaSuccess) e = done;
        if (e != cudaSuccess) {
            dfree(t, s);
            set_error("building the V^T X tasks failed: %s", cudaGetErrorString(e));
            return HMG_ERR_CUDA;
        }
    }
    h->vt_tasks = t;
    return HMG_OK;
}

// ---------------------------------------------------------------------------
// the tile sums
// ---------------------------------------------------------------------------
template <int NT> struct TtShape {
    static constexpr int R = 8 * NT;
    // Warps a CTA: 8 leave the registers that the fragments of all parts take (at 2^17 points,
    // mixed: 8 vectors 3.42 ms against 4.30 with 12, 16 5.10 against 6.60, 32 8.41 against
    // 9.72); with 24 vectors 12, a multiple of a tile's 1 to 4 row groups, so that none is
    // without work (6.34 against 6.67; smaller tiles 3-4 % the other way).
    static constexpr int WARPS = NT == 3 ? 12 : 8;
    static constexpr int SB = NT % 2 ? R : R + 8;        // floats between vector rows: lanes (g, t) hit 32 banks
    static constexpr int NS = NT <= 2 ? 3 : 4;           // stages a warp
    static constexpr int CTAS = NT <= 2 ? 2 : 1;
    static constexpr int VOFF = 2048;                    // slices, vector rows, header
    static constexpr int STAGE = VOFF + 16 * SB * 4 + 16;
    static constexpr int RED = (WARPS - 1) * 256 * R;    // (G - 1) RG 32 rows x R sums in FP64, at most
    static constexpr int RING = WARPS * NS * STAGE;
    static constexpr int SMEM = RING > RED ? RING : RED;
};

// One CTA per row tile, a warp per 32 rows and group of the tile's pairs.  M = 16 rows,
// N = 8 vectors, K = 16 columns or terms of each MMA.  A lane's 16 bytes are 4 rows of a
// chunk column, the A rows g, g + 8 of two M tiles.  A stage is 16 terms of one tier (16
// FP32, 8 FP16 pair or 4 FP8 quad columns: one step) and the vector rows they multiply,
// put in slot order.  Copies run NS - 1 stages ahead, across pairs.
template <int NT>
__global__ void __launch_bounds__(TtShape<NT>::WARPS * 32, TtShape<NT>::CTAS)
k_tile_mma(const PairDesc* __restrict__ desc, const int* tile_pair_start, const int* tile_r0, const int* tile_s,
            const int* perm1, const float* __restrict__ xm, const float* __restrict__ tm, const char* tbase, int nrhs,
            double* Y, int ldy, int only_kind, const unsigned* range, const unsigned* stored)
{
    typedef TtShape<NT> S;
    constexpr int R = S::R, NS = S::NS, SB = S::SB;
    extern __shared__ __align__(16) char tt_smem[];
    const int t = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lg = lane >> 2, lt = lane & 3;
    const int s = tile_s[t], sp = (s + 3) & ~3, tr0 = tile_r0[t];
    const int RG = (sp + 31) >> 5, G = S::WARPS / RG;
    const int g = warp / RG, rw = warp % RG;
    const int row0 = rw * 32 + lg * 4;
    char* ring = tt_smem + (size_t)warp * NS * S::STAGE;
    const uint32_t ring_s = static_cast<uint32_t>(__cvta_generic_to_shared(ring));
    const int pend = g < G ? tile_pair_start[t + 1] : 0;
    const bool plain = out_of_range(range, R, stored) || range[RANGE_T] != 0u;

    // producer: pair; within it the tier (0 FP32, 1 FP16, 2 FP8), the lane's next slice and
    // vector addresses, chunk columns left in the tier
    int pp = (g < G ? tile_pair_start[t] : 0) + g;
    PairDesc nd{};
    if (pp < pend) nd = desc[pp];
    int n16 = 0, n8 = 0, kind = 0, left = 0;
    const char* ap = nullptr;   // the lane's 16 bytes of the stage's first load
    const float* wp = nullptr;  // vector row of the stage's first term
    // vector rows: source offset (terms in order) and slot-order destination per tier: FP16
    // term 8i + 2u + v goes to row 8i + u + 4v, FP8 term 4u + q to 8(q/2) + 4(q%2) + u
    uint32_t wdst[NT];
    auto wrow = [&](int i) { return (lane + 32 * i) / (2 * NT); };
    auto wc4 = [&](int i) { return (lane + 32 * i) % (2 * NT) * 4; };
    auto set_tier = [&](int k, int n) {
        kind = k;
        left = n;
#pragma unroll
        for (int i = 0; i < NT; i++) {
            const int rr = wrow(i);
            const int pos = k == 0 ? rr
                                   : (k == 1 ? (rr & 8) + ((rr >> 1) & 3) + 4 * (rr & 1)
                                             : 8 * ((rr >> 1) & 1) + 4 * (rr & 1) + (rr >> 2));
            wdst[i] = S::VOFF + (pos * SB + wc4(i)) * 4;
        }
    };
    auto open_pair = [&]() {  // the next pair with anything to multiply
        left = 0;
        while (pp < pend) {
            const PairDesc d = nd;
            if (pp + G < pend) nd = desc[pp + G];
            pp += G;
            const bool mixed = d.kind == PAIR_FAR_MIXED;
            n16 = mixed ? d.c0 >> 1 : 0;
            n8 = mixed ? d.pad >> 2 : 0;
            if (d.ncol + n16 + n8 > 0 && (only_kind < 0 || d.kind == only_kind)) {
                ap = static_cast<const char*>(d.data) + (size_t)(lt * sp + row0) * 4;
                wp = d.kind == PAIR_STORED ? xm + (size_t)d.c0 * R
                                           : tm + (size_t)((static_cast<const char*>(d.w) - tbase) / 4) * R;
                if (d.ncol > 0) set_tier(0, d.ncol);
                else if (n16 > 0) set_tier(1, n16);
                else set_tier(2, n8);
                return;
            }
        }
    };
    open_pair();
    int prod = 0;
    uint32_t pslot = 0;
    // the lane's columns of a stage, or none (beyond every pair's) where it has no rows
    const int lta = row0 < sp ? lt : 1 << 20;
    auto issue = [&]() {
        if (left > 0) {
            const uint32_t sa = ring_s + pslot + lane * 16;
            const int terms = left << kind, cols = 16 >> kind, used = min(left, cols);
            const char* src = ap;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const bool on = 4 * i < cols;
                cp_stored16_if(sa + i * 512, src, lta + 4 * i < left, on);
                src += (size_t)sp * 16;
            }
#pragma unroll
            for (int i = 0; i < NT; i++)
                cp_vector16(ring_s + pslot + wdst[i], wp + wrow(i) * R + wc4(i), wrow(i) < terms);
            // the next stage of the tier, of the pair's next tier, or of the next pair
            int hdr = kind;
            ap += (size_t)(used * sp) * 4;
            wp += (used << kind) * R;
            left -= used;
            if (left == 0) {
                if (kind == 0 && n16 > 0) set_tier(1, n16);
                else if (kind < 2 && n8 > 0) set_tier(2, n8);
                else {
                    hdr |= 4;  // the pair's last stage
                    open_pair();
                }
            }
            if (lane == 0) *reinterpret_cast<int*>(ring + pslot + S::STAGE - 16) = hdr;
            pslot = pslot + S::STAGE == NS * S::STAGE ? 0u : pslot + S::STAGE;
            prod++;
        }
        cp_commit();
    };

    constexpr int MT = 2;  // M tiles: rows row0 + 2m, row0 + 2m + 1
    double acc64[MT][NT][4];
    float acc[MT][NT][4];
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc64[m][j][q] = 0.0, acc[m][j][q] = 0.0f;

    for (int i = 0; i < NS - 1; i++) issue();
    auto run = [&](auto plain_c) {
    constexpr bool PLAIN = decltype(plain_c)::value;
    uint32_t cslot = 0;
    for (int cons = 0; cons != prod; cons++) {
        issue();
        cp_wait<NS - 1>();
        __syncwarp();
        const char* st = ring + cslot;
        const char* sa = st + lane * 16;
        const int hdr = *reinterpret_cast<const int*>(st + S::STAGE - 16);
        const int k = hdr & 3;
        const float* bp = reinterpret_cast<const float*>(st + S::VOFF);
        // the A fragments of half i of the step for the two M tiles
        auto frag = [&](int i, uint32_t (&a0)[4], uint32_t (&a1)[4]) {
            if (k == 0) {
                const uint4 w0 = *reinterpret_cast<const uint4*>(sa + (2 * i) * 512);
                const uint4 w1 = *reinterpret_cast<const uint4*>(sa + (2 * i + 1) * 512);
                a0[0] = w0.x; a0[1] = w0.y; a0[2] = w1.x; a0[3] = w1.y;
                a1[0] = w0.z; a1[1] = w0.w; a1[2] = w1.z; a1[3] = w1.w;
                return;
            }
            float2 f0, f1, f2, f3;
            if (k == 1) {
                const uint4 w = *reinterpret_cast<const uint4*>(sa + i * 512);
                f0 = half2_to_float2(w.x), f1 = half2_to_float2(w.y);
                f2 = half2_to_float2(w.z), f3 = half2_to_float2(w.w);
            } else {
                const uint4 w = *reinterpret_cast<const uint4*>(sa);
                f0 = e4m3x2_to_float2(w.x >> (16 * i)), f1 = e4m3x2_to_float2(w.y >> (16 * i));
                f2 = e4m3x2_to_float2(w.z >> (16 * i)), f3 = e4m3x2_to_float2(w.w >> (16 * i));
            }
            a0[0] = __float_as_uint(f0.x); a0[1] = __float_as_uint(f1.x);
            a0[2] = __float_as_uint(f0.y); a0[3] = __float_as_uint(f1.y);
            a1[0] = __float_as_uint(f2.x); a1[1] = __float_as_uint(f3.x);
            a1[2] = __float_as_uint(f2.y); a1[3] = __float_as_uint(f3.y);
        };
        if constexpr (!PLAIN) {
            FragB<NT> b;
            const float* br = bp + lt * SB + lg;
            b.get(br, br + 4 * SB, br + 8 * SB, br + 12 * SB);
            uint32_t a0[2][4], a1[2][4];
            frag(0, a0[0], a1[0]);
            frag(1, a0[1], a1[1]);
            if (k == 0) {
                step_mma<NT, 3>(acc[0], a0[0], a0[1], b);
                step_mma<NT, 3>(acc[1], a1[0], a1[1], b);
            } else if (k == 1) {
                step_mma<NT, 2>(acc[0], a0[0], a0[1], b);
                step_mma<NT, 2>(acc[1], a1[0], a1[1], b);
            } else {
                step_mma<NT, 1>(acc[0], a0[0], a0[1], b);
                step_mma<NT, 1>(acc[1], a1[0], a1[1], b);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                uint32_t a0[4], a1[4];
                frag(i, a0, a1);
                step_fma<NT>(acc[0], a0, [&](int kk) { return bp + (8 * i + kk) * SB; });
                step_fma<NT>(acc[1], a1, [&](int kk) { return bp + (8 * i + kk) * SB; });
            }
        }
        if (hdr & 4) {  // the pair's last stage
#pragma unroll
            for (int m = 0; m < MT; m++)
#pragma unroll
                for (int j = 0; j < NT; j++)
#pragma unroll
                    for (int q = 0; q < 4; q++) acc64[m][j][q] += acc[m][j][q], acc[m][j][q] = 0.0f;
        }
        cslot = cslot + S::STAGE == NS * S::STAGE ? 0u : cslot + S::STAGE;
        __syncwarp();  // the slot is refilled next
    }
    };
    if (plain) run(std::true_type{});
    else run(std::false_type{});
    cp_wait<0>();
    __syncthreads();
    // the groups' sums, added in group order
    double* red = reinterpret_cast<double*>(tt_smem);
    auto row_of = [&](int m, int half) { return row0 + 2 * m + half; };
    if (g > 0 && g < G) {
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int j = 0; j < NT; j++)
#pragma unroll
                for (int half = 0; half < 2; half++)
                    *reinterpret_cast<double2*>(red + ((size_t)(g - 1) * RG * 32 + row_of(m, half)) * R + 8 * j + 2 * lt) =
                        make_double2(acc64[m][j][2 * half], acc64[m][j][2 * half + 1]);
    }
    __syncthreads();
    if (g != 0) return;
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const int row = row_of(m, half);
            if (row >= s) continue;
            double* y = Y + perm1[tr0 + row];
#pragma unroll
            for (int j = 0; j < NT; j++) {
                double a = acc64[m][j][2 * half], b = acc64[m][j][2 * half + 1];
                for (int gg = 1; gg < G; gg++) {
                    const double2 v =
                        *reinterpret_cast<const double2*>(red + ((size_t)(gg - 1) * RG * 32 + row) * R + 8 * j + 2 * lt);
                    a += v.x;
                    b += v.y;
                }
                const int c = 8 * j + 2 * lt;
                if (c < nrhs) y[(size_t)c * ldy] = a;
                if (c + 1 < nrhs) y[(size_t)(c + 1) * ldy] = b;
            }
        }
}

// ---------------------------------------------------------------------------
// the range of loaded FP32 values
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned largest16(const uint4* p, long long n, long long i, long long step)
{
    unsigned top = 0u;
    for (; i < n; i += step) {
        const uint4 v = ld_stream(p + i);
        top = max(max(top, v.x & 0x7fffffffu), max(v.y & 0x7fffffffu, max(v.z & 0x7fffffffu, v.w & 0x7fffffffu)));
    }
    return top;
}

__global__ void k_near_top(const uint4* near, long long n16, unsigned* top)
{
    record_top(largest16(near, n16, blockIdx.x * (long long)blockDim.x + threadIdx.x, gridDim.x * (long long)blockDim.x), top);
}

// the FP32 terms of U and V, a CTA a block
__global__ void k_far_top(int b0, const int* tfirst, const int* tlast, const int* tile_s, const int* tile_pstart,
                          const int* blk_m2, const int* rank, const int* tier32, const int* tier16, int mixed,
                          void* const* ptrU, void* const* ptrV, unsigned* top)
{
    const int b = b0 + blockIdx.x, r = rank[b], r32 = mixed ? tier32[b] : r, r16 = mixed ? tier16[b] : 0;
    if (r == 0) return;
    const long long bpr = 4ll * r32 + 2ll * r16 + (r - r32 - r16);
    unsigned u = 0u;
    for (int t = tfirst[b]; t <= tlast[b]; t++) {
        const char* slice = static_cast<const char*>(ptrU[b]) + (tile_pstart[t] - tile_pstart[tfirst[b]]) * bpr;
        u = max(u, largest16(reinterpret_cast<const uint4*>(slice), (long long)((tile_s[t] + 3) >> 2) * r32, threadIdx.x, blockDim.x));
    }
    record_top(u, top + 1);
    record_top(largest16(static_cast<const uint4*>(ptrV[b]), (long long)((blk_m2[b] + 3) >> 2) * r32, threadIdx.x, blockDim.x),
               top + 2);
}

hmg_status scan_stored_top(hmg_matrix* h)
{
    cudaStream_t s = h->stream;
    HMG_CUDA_TRY(cudaMemsetAsync(h->stored_top, 0, 3 * sizeof(unsigned), s));
    if (h->ndense > 0 && h->near_prec == HMG_PREC_FP32) {
        const long long n16 = h->near_stored / 4;  // columns are padded to 16 bytes
        k_near_top<<<(int)std::min<long long>(h->nsm * 8, (n16 + 255) / 256 + 1), 256, 0, s>>>(
            static_cast<const uint4*>(h->near_data), n16, h->stored_top);
        HMG_LAUNCH_CHECK();
    }
    if (h->nblocks > h->ndense && (h->far_prec == HMG_PREC_FP32 || h->far_prec == HMG_PREC_MIXED)) {
        k_far_top<<<h->nblocks - h->ndense, 256, 0, s>>>(h->ndense, h->blk_tfirst, h->blk_tlast, h->tile_s, h->tile_pstart,
                                                         h->blk_m2, h->rank, h->tier32, h->tier16,
                                                         h->far_prec == HMG_PREC_MIXED ? 1 : 0, h->ptrU, h->ptrV, h->stored_top);
        HMG_LAUNCH_CHECK();
    }
    return HMG_OK;
}

template <int NT>
static hmg_status launch_tiles(hmg_matrix* h, const float* xm, const float* tm, int nrhs, double* Y, int ldy,
                               int only_kind, const unsigned* range)
{
    if (h->ntiles <= 0) return HMG_OK;
    HMG_CUDA_TRY(cudaFuncSetAttribute(k_tile_mma<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, TtShape<NT>::SMEM));
    k_tile_mma<NT><<<h->ntiles, TtShape<NT>::WARPS * 32, TtShape<NT>::SMEM, h->stream>>>(
        static_cast<const PairDesc*>(h->tile_desc), h->tile_desc_start, h->tile_r0, h->tile_s, h->perm[0], xm, tm,
        static_cast<const char*>(h->tbuf), nrhs, Y, ldy, only_kind, range, h->stored_top);
    HMG_LAUNCH_CHECK();
    return HMG_OK;
}

template <int NT>
static hmg_status launch_all(hmg_matrix* h, const float* xm, float* tm, int nrhs, double* Y, int ldy, unsigned* range)
{
    const int nl = h->vt_large, ns = h->vt_small;
    if (nl + ns > 0) {
        HMG_CUDA_TRY(cudaFuncSetAttribute(k_vtx_mma<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, VtShape<NT>::SMEM));
        const int grid = std::min(h->nsm, nl + ceil_div(ns, VtShape<NT>::WARPS));
        k_vtx_mma<NT><<<grid, VtShape<NT>::WARPS * 32, VtShape<NT>::SMEM, h->stream>>>(static_cast<const VtTask*>(h->vt_tasks), nl,
                                                                              ns, xm, tm, range, h->stored_top);
        HMG_LAUNCH_CHECK();
    }
    return launch_tiles<NT>(h, xm, tm, nrhs, Y, ldy, -1, range);
}

hmg_status matvec_multi_mma(hmg_matrix* h, int nrhs, const double* X, int ldx, double* Y, int ldy)
{
    cudaStream_t s = h->stream;
    hmg_status st;
    const int nt = (nrhs + 7) / 8, R = 8 * nt;
    if ((st = ensure_desc(h, 4)) || (st = ensure_vt(h))) return st;
    float* xm = nullptr;
    float* tm = nullptr;
    // the range record sits behind xm
    if ((st = dalloc(&xm, (size_t)h->n[1] * R + MULTI_RANGE_WORDS, s)) || (st = dalloc(&tm, (size_t)(h->rank_total + 1) * R, s))) {
        dfree(xm, s);
        return st;
    }
    unsigned* range = reinterpret_cast<unsigned*>(xm + (size_t)h->n[1] * R);
    cudaError_t e = cudaMemsetAsync(range, 0, MULTI_RANGE_WORDS * sizeof(unsigned), s);
    if (e == cudaSuccess) {
        k_gather_mma<<<ceil_div((long long)h->n[1] * R, 256), 256, 0, s>>>(X, ldx, nrhs, h->perm[1], h->n[1], R, xm, range);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        set_error("hmg_matvec_multi: gathering the vectors failed: %s", cudaGetErrorString(e));
        st = HMG_ERR_CUDA;
    } else {
        switch (nt) {
        case 1: st = launch_all<1>(h, xm, tm, nrhs, Y, ldy, range); break;
        case 2: st = launch_all<2>(h, xm, tm, nrhs, Y, ldy, range); break;
        case 3: st = launch_all<3>(h, xm, tm, nrhs, Y, ldy, range); break;
        default: st = launch_all<4>(h, xm, tm, nrhs, Y, ldy, range); break;
        }
    }
    dfree(xm, s);
    dfree(tm, s);
    return st;
}

// Y = the near-field part of H X for up to 32 vectors, FP32 stored near field (the BF16
// tensor-core path with its near field in FP32).  xm: n2 x 32 values and the range record.
hmg_status near_multi32(hmg_matrix* h, const double* X, int ldx, int nrhs, float* xm, double* Y, int ldy)
{
    // a product in another near-field mode or arithmetic may have left other descriptors, and
    // one that ran out of memory none
    hmg_status st = ensure_desc(h, 4);
    if (st) return st;
    unsigned* range = reinterpret_cast<unsigned*>(xm + (size_t)h->n[1] * 32);
    HMG_CUDA_TRY(cudaMemsetAsync(range, 0, MULTI_RANGE_WORDS * sizeof(unsigned), h->stream));
    k_gather_mma<<<ceil_div((long long)h->n[1] * 32, 256), 256, 0, h->stream>>>(X, ldx, nrhs, h->perm[1], h->n[1], 32,
                                                                                xm, range);
    HMG_LAUNCH_CHECK();
    return launch_tiles<4>(h, xm, nullptr, nrhs, Y, ldy, PAIR_STORED, range);
}

}  // namespace hmg
