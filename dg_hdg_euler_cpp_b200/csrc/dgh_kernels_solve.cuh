// Block solves with the slab-layout factors (dgh_slab.cuh): z = A^{-1} b per block
// (block_jacobi.hpp:24-39: permute, unit lower solve, upper solve) and its transpose.
//
// One warp owns one block, with no CTA-wide barriers, and streams its factors once per sweep.  What
// bounds it is that stream, and, where a warp has only one block to do, the chain of its latencies.  So
//  - the factors pass through a ring in shared memory, filled by 16-byte asynchronous copies that run on
//    across slabs, sweeps and blocks (4 KB a warp in flight, 20 to 24 warps an SM): nothing the warp waits for, a
//    triangle or a gather, stops them.  The stream's unit is a chunk, a slab's 32 columns (16 in FP64): it
//    is contiguous, and the diagonal square of a slab is one chunk (two), so that following it costs a few
//    instructions (with chunks cut by size and not by columns FP16 was bound by its instructions: 3.44 ms
//    in the last case below);
//  - the 32 x 32 diagonal triangles of the FP64 factors are stored inverted (k_slab_invert), so a triangle
//    is one more product instead of 32 dependent steps of a shuffle, an FMA and, going up, a division.  A
//    product's residual grows with the triangle's condition, substitution's does not, so a triangle above
//    INVERT_BOUND stays as it is, marked in a byte per square, and is solved by substitution.  On cell blocks
//    of degree 2 to 8 (condition at most 70) solutions are 3.4e-15 to 6.4e-14 from 64-bit solves with the
//    inverses, 3.1e-15 to 6.4e-14 without.  The FP32 and FP16 factors keep their triangles, since inverses
//    rounded to FP32 did lose accuracy, and solve them four columns to a shuffle, with the
//    reciprocals of the diagonal taken beforehand;
//  - a last slab of 4, 8 or 16 rows gives a row's column groups to 8, 4 or 2 lanes.
// Measured inside solves, before (four 16-byte loads in flight, triangles solved from global memory) and now:
// FP64, 4,096 blocks of 36: 36 and 16 us; 8,192 of 20: 40 and 15 us; 4,096 of 100, transposed: 126 and
// 75 us; FP32, 5,917 blocks of 144: 131 and 92 us (5.3 TB/s), 65,536 of 324: 4.78 and 4.77 ms (5.8 TB/s); FP16,
// 65,536 blocks of 324: 2.68 and 2.54 ms (5.7 TB/s), but 4,096, 1.15 rounds of warps, 200 and 207 us.
#pragma once
#include <type_traits>

#include "dgh_common.cuh"
#include "dgh_slab.cuh"

namespace dgh {

constexpr int SOLVE_WARPS = 4, SOLVE_THREADS = 32 * SOLVE_WARPS;

// Arithmetic type, elements per 16 bytes, columns per chunk, chunks in a warp's ring and row length of a
// block's slabs, by storage type.
// Aux: per block, the kept squares of FP64 factors (KEPT_L, KEPT_U) or the row scales of FP16 factors.
template <typename T> struct SolveType {
    using A = T;
    using Aux = typename std::conditional<sizeof(T) == 8, unsigned char, float>::type;
    static constexpr int W = SlabVec<T>::W, CW = sizeof(T) == 8 ? 16 : 32, STAGES = 2;
    __host__ __device__ static constexpr int row(int m) { return m; }
};
template <> struct SolveType<__half> {
    using A = float;
    using Aux = float;
    static constexpr int W = H_W, CW = 32, STAGES = 3;
    __host__ __device__ static constexpr int row(int m) { return pad8(m); }
};
// CTAs per SM that the registers are cut for: a warp more hides more of the solves' latencies than a chunk
// more in its ring (FP16, blocks of 324: 3 stages and 6 CTAs 633 us per 16,384 blocks, 4 and 5 641, 6 and 4
// 690, 8 and 3 791).
template <typename T> constexpr int SOLVE_CTAS = sizeof(T) == 2 ? 6 : 5;
template <typename T> constexpr int CHUNK_BYTES = 32 * SolveType<T>::CW * (int)sizeof(T);
template <typename T, bool TRANS> constexpr int RING_BYTES = CHUNK_BYTES<T> * (SolveType<T>::STAGES + TRANS);
// Blocks of at most this size are held whole instead of streamed: with a few chunks a sweep, a ring would wait
// for memory at each.
constexpr int WHOLE_BYTES = 16384;
template <typename T> __host__ __device__ constexpr size_t block_bytes(int m) { return sizeof(T) * (size_t)m * SolveType<T>::row(m); }
template <typename T> __host__ __device__ constexpr bool solve_whole(int m) { return block_bytes<T>(m) <= WHOLE_BYTES; }
// Shared memory per warp: the factors and the block's vector (the transposed solve adds a slab's results).
template <typename T, bool TRANS> __host__ __device__ constexpr size_t factor_bytes(int m) {
    return solve_whole<T>(m) ? (block_bytes<T>(m) + 15) / 16 * 16 : (size_t)RING_BYTES<T, TRANS>;
}
template <typename T, bool TRANS = false> __host__ __device__ constexpr size_t solve_warp_bytes(int m) {
    const size_t y = (sizeof(typename SolveType<T>::A) * (SolveType<T>::row(m) + (TRANS ? 32 : 0)) + 15) / 16 * 16;
    return factor_bytes<T, TRANS>(m) + y;
}

__device__ __forceinline__ unsigned long long pack2(unsigned lo, unsigned hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ void fma2(unsigned long long &d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 half_pair(unsigned w) { return __half22float2(*reinterpret_cast<const __half2 *>(&w)); }
__device__ __forceinline__ unsigned long long half_pack(unsigned w) {
    const float2 f = half_pair(w);
    return pack2(__float_as_uint(f.x), __float_as_uint(f.y));
}
// The accumulators of a row's products: a group's products are summed first and then added to one of four
// running sums (pairs of them in FP32), which keeps these short.
struct Acc64 {
    double a[4] = {0, 0, 0, 0};
    __device__ __forceinline__ double sum() const { return (a[0] + a[1]) + (a[2] + a[3]); }
};
struct Acc32 {
    unsigned long long a[4] = {0, 0, 0, 0};
    __device__ __forceinline__ float sum() const {
        const unsigned long long t = add2(add2(a[0], a[1]), add2(a[2], a[3]));
        return __uint_as_float((unsigned)t) + __uint_as_float((unsigned)(t >> 32));
    }
};
__device__ __forceinline__ void slab_fma(const uint4 &v, const double *y, double &acc, const double *) {
    const double2 a = *reinterpret_cast<const double2 *>(y);
    acc += fma(__hiloint2double((int)v.w, (int)v.z), a.y, __hiloint2double((int)v.y, (int)v.x) * a.x);
}
__device__ __forceinline__ void slab_fma(const uint4 &v, const float *y, unsigned long long &acc, const float *) {
    const uint4 a = *reinterpret_cast<const uint4 *>(y);
    unsigned long long d = mul2(pack2(v.x, v.y), pack2(a.x, a.y));
    fma2(d, pack2(v.z, v.w), pack2(a.z, a.w));
    acc = add2(acc, d);
}
__device__ __forceinline__ void slab_fma(const uint4 &v, const float *y, unsigned long long &acc, const __half *) {
    const uint4 a = *reinterpret_cast<const uint4 *>(y), b = *reinterpret_cast<const uint4 *>(y + 4);
    unsigned long long d = mul2(half_pack(v.x), pack2(a.x, a.y));
    fma2(d, half_pack(v.y), pack2(a.z, a.w));
    fma2(d, half_pack(v.z), pack2(b.x, b.y));
    fma2(d, half_pack(v.w), pack2(b.z, b.w));
    acc = add2(acc, d);
}

// FP32 blocks at least HALF_SQUARES wide fetch of a diagonal square only the triangle of the sweep, L going forward
// and U going back: fetched whole in both sweeps, the squares add a tenth to the bytes of 324-wide blocks.  65,536
// blocks of 324 (256, 144): 4.77 (2.71, 0.91) ms, with whole squares 5.06 (2.88, 0.98); 4,096 of 100: 55 against
// 53 us, where the bytes do not bound it.  (FP16, bound by instructions: 3 to 6 % slower at 100 to 196.)  Nor do
// they with few warps at work, whose chains the choice of a square's lanes lengthens: 324 (256, 196, 144) wide, 576 blocks
// 7 (10, 11, 17) % slower, 1,600 2 % faster (0, 0, 6 % slower), 2,500 4 (5, 6, 2) % faster.
constexpr int HALF_SQUARES = 128, HALF_BLOCKS = 2368;

__device__ __forceinline__ void ring_copy(unsigned dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// A warp's stream of chunks, copied ahead of their use: per sweep the slabs in order (sweep 0) or in reverse,
// a slab's chunks ascending (sweep 0) or descending, so that the diagonal's come last in a slab, or,
// transposed, first.  Chunk j of slab s lies at its offset in memory and in its ring slot alike (group by
// group, row by row), and unit i of its 16-byte units is copied by lane i % 32.
// HALF (D = 1): of a diagonal square only the triangle of the sweep.
template <typename T, bool TRANS, bool HALF = false> struct SlabStream {
    using S = SolveType<T>;
    static constexpr int D = 32 / S::CW, UNITS = S::CW / S::W;  // chunks in a diagonal square, groups in a chunk
    static constexpr int STAGES = S::STAGES + TRANS;
    const T *pool;
    size_t stride;
    int m, ml, slabs, chunks, ragged, count, warps;  // ragged: the chunk of fewer columns (-1: none)
    int blk, dir, s, j, left;                        // the next chunk, chunks left in its slab
    const uint4 *src;
    unsigned base;
    int fill_at, use_at;  // ring offsets in bytes
    __device__ __forceinline__ void slab() {
        const int d0 = D * s, d1 = min(D * s + D, chunks);
        if (dir == 0) {
            j = TRANS ? d0 : 0;
            left = (TRANS ? chunks : d1) - j;
        } else {
            j = (TRANS ? d1 : chunks) - 1;
            left = j + 1 - (TRANS ? 0 : d0);
        }
        const int nt = min(32, m - 32 * s);
        src = reinterpret_cast<const uint4 *>(pool + (size_t)blk * stride + (32 * s * ml + S::CW * j * nt)) + (threadIdx.x & 31);
    }
    __device__ __forceinline__ void fill() {
        if (blk < count) {
            const unsigned dst = base + fill_at + (threadIdx.x & 31) * 16;
            const bool rows = s < slabs - 1 || m % 32 == 0;
            if (HALF && rows && j == s) {  // the triangle that the sweep reads
                const int r = threadIdx.x & 31;
#pragma unroll
                for (int u = 0; u < UNITS; ++u)
                    if (dir == 0 ? r >= u * S::W : r < (u + 1) * S::W) ring_copy(dst + u * 512, src + u * 32);
            } else if (rows && j != ragged) {
#pragma unroll
                for (int u = 0; u < UNITS; ++u) ring_copy(dst + u * 512, src + u * 32);
            } else {
                const int units = min(32, m - 32 * s) * min(S::CW, ml - S::CW * j) / S::W;
                for (int u = 0; u < units; u += 32)
                    if (u + (int)(threadIdx.x & 31) < units) ring_copy(dst + u * 16, src + u);
            }
            if (--left) {
                const int step = UNITS * (rows ? 32 : m - 32 * s);
                j += dir == 0 ? 1 : -1;
                src += dir == 0 ? step : -step;
            } else {
                s += dir == 0 ? 1 : -1;
                if (s == slabs) dir = 1, s = slabs - 1;
                else if (s < 0) dir = 0, s = 0, blk += warps;
                slab();
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        fill_at = fill_at + CHUNK_BYTES<T> == RING_BYTES<T, TRANS> ? 0 : fill_at + CHUNK_BYTES<T>;
    }
    __device__ __forceinline__ SlabStream(const T *pool_, size_t stride_, int m_, int count_, int blk0, int warps_, void *ring)
        : pool(pool_), stride(stride_), m(m_), count(count_), warps(warps_), blk(blk0) {
        ml = S::row(m);
        slabs = (m + 31) / 32;
        chunks = (ml + S::CW - 1) / S::CW;
        ragged = ml % S::CW ? chunks - 1 : -1;
        dir = s = fill_at = use_at = 0;
        base = (unsigned)__cvta_generic_to_shared(ring);
        slab();
#pragma unroll
        for (int i = 0; i < STAGES - 1; ++i) fill();
    }
    __device__ __forceinline__ void block(int) {}  // (its chunks are on their way)
    // The next chunk's ring offset, once this lane's copies of it have landed.
    __device__ __forceinline__ int next() {
        fill();
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
        const int at = use_at;
        use_at = use_at + CHUNK_BYTES<T> == RING_BYTES<T, TRANS> ? 0 : use_at + CHUNK_BYTES<T>;
        return at;
    }
};

// The same interface for a block that is held whole: copied when its turn comes, the chunks read in place.
template <typename T, bool TRANS> struct SlabWhole {
    using S = SolveType<T>;
    static constexpr int D = 32 / S::CW;
    const T *pool;
    size_t stride;
    int m, ml, slabs, chunks;
    int dir, s, j, left;
    unsigned base;
    __device__ __forceinline__ SlabWhole(const T *pool_, size_t stride_, int m_, int, int, int, void *ring)
        : pool(pool_), stride(stride_), m(m_) {
        ml = S::row(m);
        slabs = (m + 31) / 32;
        chunks = (ml + S::CW - 1) / S::CW;
        base = (unsigned)__cvta_generic_to_shared(ring);
    }
    __device__ __forceinline__ void slab() {
        const int d0 = D * s, d1 = min(D * s + D, chunks);
        j = dir == 0 ? (TRANS ? d0 : 0) : (TRANS ? d1 : chunks) - 1;
        left = dir == 0 ? (TRANS ? chunks : d1) - j : j + 1 - (TRANS ? 0 : d0);
    }
    // Starts the block's copies (its predecessor has been read).
    __device__ __forceinline__ void block(int blk) {
        const uint4 *src = reinterpret_cast<const uint4 *>(pool + (size_t)blk * stride);
        const int units = m * ml / S::W;
        for (int u = threadIdx.x & 31; u < units; u += 32) ring_copy(base + u * 16, src + u);
        asm volatile("cp.async.commit_group;" ::: "memory");
        dir = s = 0;
        slab();
    }
    __device__ __forceinline__ int next() {
        if (dir == 0 && s == 0 && j == 0) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncwarp();
        }
        const int at = (int)sizeof(T) * (32 * s * ml + S::CW * j * min(32, m - 32 * s));
        if (--left) {
            j += dir == 0 ? 1 : -1;
        } else {
            s += dir == 0 ? 1 : -1;
            if (s == slabs) dir = 1, s = slabs - 1;
            if (s >= 0) slab();
        }
        return at;
    }
};

// A triangular system of nt <= 32 unknowns (a multiple of 4) in registers, ascending (lower) or descending
// (upper): lane i holds the right-hand side t and gets the unknown i.  own(c): the lane's coefficient of
// unknown c; four(r, c): row r's coefficients of c..c+3; d, rd: the diagonal and its reciprocal (UNIT: 1).
// EXACT corrects each product with the reciprocal to the quotient's rounding (FP32 factors; under the 2^-11 of
// FP16 factors the correction does not show: the solutions' rms distance from 64-bit ones over cells of degree 1
// to 8, 3.7e-4 to 9.3e-3, is the same to 2e-5 of itself with true quotients, and 100- to 196-wide solves are 4 to 7 %
// slower with it).  Four
// unknowns a step: they are shuffled at once and every lane finishes them itself, so a step's chain is
// one shuffle and a few FMAs, not four of each.
template <bool ASC, bool UNIT, bool EXACT, class Own, class Four>
__device__ __forceinline__ float triangle(float t, int lane, int nt, float d, const Own &own, const Four &four) {
    constexpr unsigned ALL = 0xffffffffu;
    const float rd = UNIT ? 1.f : 1.f / d;
    auto over = [&](float x, float r, float dd) {  // x / dd
        if (UNIT) return x;
        const float q = x * r;
        return EXACT ? fmaf(fmaf(-dd, q, x), r, q) : q;
    };
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int c = ASC ? 4 * k : 28 - 4 * k;
        if (c >= nt) continue;
        float y0 = __shfl_sync(ALL, t, c), y1 = __shfl_sync(ALL, t, c + 1);
        float y2 = __shfl_sync(ALL, t, c + 2), y3 = __shfl_sync(ALL, t, c + 3);
        float r0 = 1.f, r1 = 1.f, r2 = 1.f, r3 = 1.f;
        if (!UNIT) {
            r0 = __shfl_sync(ALL, rd, c);
            r1 = __shfl_sync(ALL, rd, c + 1);
            r2 = __shfl_sync(ALL, rd, c + 2);
            r3 = __shfl_sync(ALL, rd, c + 3);
        }
        float e0 = 1.f, e1 = 1.f, e2 = 1.f, e3 = 1.f;
        if (EXACT && !UNIT) {
            e0 = __shfl_sync(ALL, d, c);
            e1 = __shfl_sync(ALL, d, c + 1);
            e2 = __shfl_sync(ALL, d, c + 2);
            e3 = __shfl_sync(ALL, d, c + 3);
        }
        if (ASC) {
            const float4 l1 = four(c + 1, c), l2 = four(c + 2, c), l3 = four(c + 3, c);
            y0 = over(y0, r0, e0);
            y1 = fmaf(-l1.x, y0, y1);
            y1 = over(y1, r1, e1);
            y2 = fmaf(-l2.y, y1, fmaf(-l2.x, y0, y2));
            y2 = over(y2, r2, e2);
            y3 = fmaf(-l3.z, y2, fmaf(-l3.y, y1, fmaf(-l3.x, y0, y3)));
            y3 = over(y3, r3, e3);
        } else {
            const float4 u0 = four(c, c), u1 = four(c + 1, c), u2 = four(c + 2, c);
            y3 = over(y3, r3, e3);
            y2 = fmaf(-u2.w, y3, y2);
            y2 = over(y2, r2, e2);
            y1 = fmaf(-u1.z, y2, fmaf(-u1.w, y3, y1));
            y1 = over(y1, r1, e1);
            y0 = fmaf(-u0.y, y1, fmaf(-u0.z, y2, fmaf(-u0.w, y3, y0)));
            y0 = over(y0, r0, e0);
        }
        if (ASC ? lane > c + 3 : lane < c) {
            t = fmaf(-own(ASC ? c : c + 3), ASC ? y0 : y3, t);
            t = fmaf(-own(ASC ? c + 1 : c + 2), ASC ? y1 : y2, t);
            t = fmaf(-own(ASC ? c + 2 : c + 1), ASC ? y2 : y1, t);
            t = fmaf(-own(ASC ? c + 3 : c), ASC ? y3 : y0, t);
        } else if (lane >= c && lane < c + 4) {
            t = lane == c ? y0 : lane == c + 1 ? y1 : lane == c + 2 ? y2 : y3;
        }
    }
    return t;
}
// Entries of a diagonal square in its chunk: group q's row r at base[q nt + r].
__device__ __forceinline__ float square_at(const uint4 *base, int nt, int r, int c, const __half *) {
    return __half2float(reinterpret_cast<const __half *>(base + (c >> 3) * nt + r)[c & 7]);
}
__device__ __forceinline__ float square_at(const uint4 *base, int nt, int r, int c, const float *) {
    return reinterpret_cast<const float *>(base + (c >> 2) * nt + r)[c & 3];
}
__device__ __forceinline__ float4 square_four(const uint4 *base, int nt, int r, int c, const __half *) {
    const uint2 x = *reinterpret_cast<const uint2 *>(reinterpret_cast<const __half *>(base + (c >> 3) * nt + r) + (c & 7));
    const float2 lo = half_pair(x.x), hi = half_pair(x.y);
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ float4 square_four(const uint4 *base, int nt, int r, int c, const float *) {
    return *reinterpret_cast<const float4 *>(base + (c >> 2) * nt + r);
}
// A triangle with a subnormal diagonal entry, whose reciprocal may be out of range: true quotients, a column at a
// time, ascending or descending.  at(r, c): the triangle's entries.
template <bool ASC, class At> __device__ __forceinline__ float triangle_divided(float t, int lane, int nt, const At &at) {
#pragma unroll 1
    for (int k = 0; k < nt; ++k) {
        const int c = ASC ? k : nt - 1 - k;
        const float e = lane < nt && (ASC ? lane >= c : lane <= c) ? at(lane, c) : 1.f;
        if (lane == c) t = t / e;
        const float y = __shfl_sync(0xffffffffu, t, c);
        if (lane < nt && (ASC ? lane > c : lane < c)) t = fmaf(-e, y, t);
    }
    return t;
}
__device__ __forceinline__ bool any_subnormal(float d) { return __any_sync(0xffffffffu, fabsf(d) < 0x1p-126f); }
// The slab's triangle: L (dir 0) or U (dir 1), lane i holding row i's right-hand side.
template <typename T> __device__ __forceinline__ float slab_triangle(const uint4 *base, int lane, int nt, int dir, float t) {
    constexpr int W = SolveType<T>::W;
    const T *tag = nullptr;
    uint4 e[32 / W];
#pragma unroll
    for (int q = 0; q < 32 / W; ++q) e[q] = lane < nt && W * q < nt ? base[q * nt + lane] : make_uint4(0, 0, 0, 0);
    auto own = [&](int c) {  // c a constant
        const uint4 &x = e[c / W];
        const int w = sizeof(T) == 4 ? c & 3 : (c >> 1) & 3;
        const unsigned word = w == 0 ? x.x : w == 1 ? x.y : w == 2 ? x.z : x.w;
        if (sizeof(T) == 4) return __uint_as_float(word);
        const float2 p = half_pair(word);
        return c & 1 ? p.y : p.x;
    };
    auto four = [&](int r, int c) { return square_four(base, nt, r, c, tag); };
    if (dir == 0) return triangle<true, true, false>(t, lane, nt, 1.f, own, four);
    const float d = lane < nt ? square_at(base, nt, lane, lane, tag) : 1.f;
    if (sizeof(T) == 4 && any_subnormal(d))
        return triangle_divided<false>(t, lane, nt, [&](int r, int c) { return square_at(base, nt, r, c, tag); });
    return triangle<false, false, sizeof(T) == 4>(t, lane, nt, d, own, four);
}
// The same transposed: U^T (dir 0, lower) or L^T (dir 1, unit upper).
__device__ __forceinline__ float slab_triangle_t(const uint4 *base, int lane, int nt, int dir, float t) {
    const float *tag = nullptr;
    const int col = min(lane, nt - 1);
    auto own = [&](int c) { return square_at(base, nt, c, col, tag); };
    auto four = [&](int r, int c) {
        return make_float4(square_at(base, nt, c, r, tag), square_at(base, nt, c + 1, r, tag), square_at(base, nt, c + 2, r, tag),
                           square_at(base, nt, c + 3, r, tag));
    };
    if (dir == 1) return triangle<false, true, false>(t, lane, nt, 1.f, own, four);
    const float d = square_at(base, nt, col, col, tag);
    if (any_subnormal(d)) return triangle_divided<true>(t, lane, nt, [&](int r, int c) { return square_at(base, nt, c, r, tag); });
    return triangle<true, false, true>(t, lane, nt, d, own, four);
}

// Squares of FP64 factors whose triangle is kept (k_slab_invert): a byte per square, slab by slab.
constexpr unsigned char KEPT_L = 1, KEPT_U = 2;
// Lane s's byte of block blk, loaded beside the block's vector; ballots make it bits per slab.
template <typename T> __device__ __forceinline__ int kept_square(const typename SolveType<T>::Aux *aux, int blk, int slabs) {
    const int lane = threadIdx.x & 31;
    if constexpr (sizeof(T) == 8) return lane < slabs ? aux[(size_t)blk * slabs + lane] : 0;
    return 0;
}

// z = A^{-1} b.  T: the factors' storage; FP16 factors carry row scales (aux: the reciprocal of each U
// row's largest entry), FP64 factors their kept squares.  The body takes its block index bx and block count G explicitly (the batched
// solve of a lockstep batch runs it over each member's blocks).
template <typename T, class Stream>
__device__ __forceinline__ void lu_solve_blocks(int bx, int G, const T *__restrict__ pool, const typename SolveType<T>::Aux *__restrict__ aux,
                                              const int *__restrict__ perm, size_t stride, int m, int count,
                                              const double *__restrict__ rhs, double *__restrict__ z) {
    using S = SolveType<T>;
    using A = typename S::A;
    constexpr int W = S::W, CW = S::CW, UNITS = CW / W, D = 32 / CW;
    const T *tag = nullptr;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    unsigned char *ring = smraw + (size_t)wib * solve_warp_bytes<T>(m);
    A *y = reinterpret_cast<A *>(ring + factor_bytes<T, false>(m));
    const int warps = G * SOLVE_WARPS, blk0 = bx * SOLVE_WARPS + wib;
    if (blk0 >= count) return;
    Stream in(pool, stride, m, count, blk0, warps, ring);
    const int slabs = in.slabs, chunks = in.chunks, ml = in.ml;
    for (int blk = blk0; blk < count; blk += warps) {
        in.block(blk);
        const int *pm = perm + (size_t)blk * m;
        const double *b = rhs + (size_t)blk * m;
        const int kept = kept_square<T>(aux, blk, slabs);
        for (int i = lane; i < ml; i += 32) y[i] = i < m ? (A)b[pm[i]] : A(0);
        unsigned kept_l = 0, kept_u = 0;
        if constexpr (sizeof(T) == 8) {
            kept_l = __ballot_sync(0xffffffffu, kept & KEPT_L);
            kept_u = __ballot_sync(0xffffffffu, kept & KEPT_U);
        }
        __syncwarp();
        // sweep 0: forward, L y = P b (columns left of the slab); sweep 1: backward, U z = y (right of it)
        for (int dir = 0; dir < 2; ++dir)
            for (int si = 0; si < slabs; ++si) {
                const int s = dir == 0 ? si : slabs - 1 - si, r0 = 32 * s, nt = min(32, m - r0);
                const int d0 = D * s, d1 = min(D * s + D, chunks);
                typename std::conditional<sizeof(T) == 8, Acc64, Acc32>::type acc;
                A off;  // the off-diagonal products of row r0 + lane
                // lanes that share a row (in a short slab of 4, 8 or 16 rows), this lane's row and first group
                const bool share = nt < 32 && (nt & (nt - 1)) == 0;
                const int lg = share ? 31 - __clz(nt) : 5, sub = 32 >> lg, row = share ? lane & (nt - 1) : lane, k = lane >> lg;
                auto sum = [&](A x) {
                    if (share)
                        for (int o = nt; o < 32; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                    return x;
                };
                const int n_off = dir == 0 ? d0 : chunks - d1;
                const A *yj = y + (dir == 0 ? 0 : CW * (chunks - 1));
                if (nt == 32) {
                    for (int i = 0; i < n_off; ++i) {
                        const uint4 *v = reinterpret_cast<const uint4 *>(ring + in.next()) + lane;  // its own copies
                        const int groups = dir == 0 ? UNITS : min(UNITS, (ml - (int)(yj - y)) / W);
                        if (groups == UNITS) {
#pragma unroll
                            for (int u = 0; u < UNITS; ++u) slab_fma(v[u * 32], yj + u * W, acc.a[u & 3], tag);
                        } else {
                            for (int u = 0; u < groups; ++u) slab_fma(v[u * 32], yj + u * W, acc.a[0], tag);
                        }
                        yj += dir == 0 ? CW : -CW;
                    }
                } else {  // the last slab: all of its chunks left of the diagonal are whole
                    for (int i = 0; i < n_off; ++i) {
                        const uint4 *v = reinterpret_cast<const uint4 *>(ring + in.next());
                        __syncwarp();
                        if (row < nt)
                            for (int g = k; g < UNITS; g += sub) slab_fma(v[g * nt + row], yj + g * W, acc.a[0], tag);
                        yj += CW;
                        __syncwarp();
                    }
                }
                off = sum(acc.sum());
                if constexpr (sizeof(T) < 8) {
                    const uint4 *square = reinterpret_cast<const uint4 *>(ring + in.next());
                    __syncwarp();
                    float t = 0.f;
                    if (lane < nt)
                        t = sizeof(T) == 2 && dir == 1 ? fmaf(y[r0 + lane], aux[(size_t)blk * m + r0 + lane], -off)
                                                       : y[r0 + lane] - off;
                    t = slab_triangle<T>(square, lane, nt, dir, t);
                    if (lane < nt) y[r0 + lane] = t;
                    __syncwarp();
                } else if ((dir == 0 ? kept_l : kept_u) >> s & 1) {  // substitution, a column at a time
                    A t = lane < nt ? y[r0 + lane] - off : A(0);
                    for (int i = 0; i < d1 - d0; ++i) {
                        const T *e = reinterpret_cast<const T *>(ring + in.next()) + W * lane;
                        __syncwarp();
                        const int c0 = CW * (dir == 0 ? i : d1 - d0 - 1 - i), nc = min(CW, nt - c0);
                        for (int k = 0; k < nc; ++k) {
                            const int j = dir == 0 ? k : nc - 1 - k, c = c0 + j;
                            const T a = lane < nt && (dir == 0 ? lane > c : lane <= c) ? e[j / W * nt * W + j % W] : T(1);
                            if (dir == 1 && lane == c) t = t / a;
                            const A yc = __shfl_sync(0xffffffffu, t, c);
                            if (lane < nt && (dir == 0 ? lane > c : lane < c)) t = fma(-a, yc, t);
                        }
                        __syncwarp();
                    }
                    if (lane < nt) y[r0 + lane] = t;
                    __syncwarp();
                } else {  // the inverted triangle: the slab's right-hand side to y, then one more product
                    if (row < nt && k == 0) y[r0 + row] -= off;
                    __syncwarp();
                    acc = Acc64();
                    for (int i = 0; i < d1 - d0; ++i) {
                        const uint4 *v = reinterpret_cast<const uint4 *>(ring + in.next());
                        __syncwarp();
                        const int c0 = CW * (dir == 0 ? i : d1 - d0 - 1 - i), groups = min(UNITS, (nt - c0) / W);
                        if (row < nt)
#pragma unroll
                            for (int u = 0; u < UNITS; ++u) {
                                const int g = u * sub + k, c = c0 + g * W;
                                if (g < groups) {
                                    uint4 e = v[g * nt + row];  // the other triangle's columns dropped
                                    if (dir == 0 ? c >= row : c < row) e.x = e.y = 0;
                                    if (dir == 0 ? c + 1 >= row : c + 1 < row) e.z = e.w = 0;
                                    slab_fma(e, y + r0 + c, acc.a[u & 3], tag);
                                }
                            }
                        __syncwarp();
                    }
                    const A x = sum(acc.sum());
                    if (row < nt && k == 0) y[r0 + row] = dir == 0 ? y[r0 + row] + x : x;
                    __syncwarp();
                }
            }
        for (int i = lane; i < m; i += 32) z[(size_t)blk * m + i] = (double)y[i];
        __syncwarp();
    }
}
template <typename T>
__device__ __forceinline__ void lu_solve_body(int bx, int G, const T *__restrict__ pool, const typename SolveType<T>::Aux *__restrict__ aux,
                                              const int *__restrict__ perm, size_t stride, int m, int count,
                                              const double *__restrict__ rhs, double *__restrict__ z) {
    if (solve_whole<T>(m)) lu_solve_blocks<T, SlabWhole<T, false>>(bx, G, pool, aux, perm, stride, m, count, rhs, z);
    else if (sizeof(T) == 4 && m >= HALF_SQUARES && count >= HALF_BLOCKS)
        lu_solve_blocks<T, SlabStream<T, false, sizeof(T) == 4>>(bx, G, pool, aux, perm, stride, m, count, rhs, z);
    else lu_solve_blocks<T, SlabStream<T, false>>(bx, G, pool, aux, perm, stride, m, count, rhs, z);
}
template <typename T>
__global__ void __launch_bounds__(SOLVE_THREADS, SOLVE_CTAS<T>)
k_lu_solve(const T *__restrict__ pool, const typename SolveType<T>::Aux *__restrict__ aux, const int *__restrict__ perm, size_t stride, int m,
           int count, const double *__restrict__ rhs, double *__restrict__ z) {
    lu_solve_body<T>(blockIdx.x, gridDim.x, pool, aux, perm, stride, m, count, rhs, z);
}

// z = A^{-T} b with the same factors (A = P^T L U, so A^{-T} b = P^T L^{-T} U^{-T} b): a forward solve with
// U^T, a backward solve with L^T, then the scatter z[perm[i]] = x[i].  A slab's unknowns come first (its
// inverted triangle, transposed), then its rows are applied to the columns of the remaining unknowns.
// A lane owns a column of the chunk and walks its rows; the lanes start at different rows, so that a
// step's elements (and the unknowns they multiply) lie in different banks.
template <typename T, class Stream>
__device__ __forceinline__ void lu_solve_t_blocks(const T *__restrict__ pool, const typename SolveType<T>::Aux *__restrict__ aux,
                                                  const int *__restrict__ perm, size_t stride, int m, int count,
                                                  const double *__restrict__ rhs, double *__restrict__ z) {
    using S = SolveType<T>;
    constexpr int W = S::W, CW = S::CW, D = 32 / CW, PARTS = 32 / CW;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    unsigned char *ring = smraw + (size_t)wib * solve_warp_bytes<T, true>(m);
    T *x = reinterpret_cast<T *>(ring + factor_bytes<T, true>(m)), *y = x + 32;  // a slab's new unknowns; all of them
    const int warps = gridDim.x * SOLVE_WARPS, blk0 = blockIdx.x * SOLVE_WARPS + wib;
    if (blk0 >= count) return;
    Stream in(pool, stride, m, count, blk0, warps, ring);
    const int slabs = in.slabs, chunks = in.chunks;
    const int col = lane % CW, part = lane / CW, q = col / W;  // column and row part of this lane
    for (int blk = blk0; blk < count; blk += warps) {
        in.block(blk);
        const int *pm = perm + (size_t)blk * m;
        const double *b = rhs + (size_t)blk * m;
        for (int i = lane; i < m; i += 32) y[i] = (T)b[i];
        unsigned kept_l = 0, kept_u = 0;
        if constexpr (sizeof(T) == 8) {
            const int kept = kept_square<T>(aux, blk, slabs);
            kept_l = __ballot_sync(0xffffffffu, kept & KEPT_L);
            kept_u = __ballot_sync(0xffffffffu, kept & KEPT_U);
        }
        for (int dir = 0; dir < 2; ++dir)
            for (int si = 0; si < slabs; ++si) {
                const int s = dir == 0 ? si : slabs - 1 - si, r0 = 32 * s, nt = min(32, m - r0), span = nt / PARTS;
                const int d0 = D * s, d1 = min(D * s + D, chunks), n = dir == 0 ? chunks - d0 : d1;
                const T *yr = y + r0 + part * span;
                int jc = dir == 0 ? d0 : d1 - 1;
                for (int i = 0; i < n; ++i, jc += dir == 0 ? 1 : -1) {
                    __syncwarp();
                    const unsigned char *chunk = ring + in.next();
                    __syncwarp();
                    const int j = CW * jc + col;
                    const unsigned char *e = chunk + (q * nt + part * span) * 16 + (col % W) * sizeof(T);
                    T s0 = 0, s1 = 0;
                    if (i >= d1 - d0) {
                        if (nt == 32 && j < m) {
#pragma unroll
                            for (int k = 0; k < 32 / PARTS; ++k) {
                                const int r = (q + k) & (32 / PARTS - 1);
                                const T a = *reinterpret_cast<const T *>(e + r * 16);
                                if (k & 1) s1 = fma(a, yr[r], s1);
                                else s0 = fma(a, yr[r], s0);
                            }
                        } else if (j < m) {
                            int r = q % span;
                            for (int k = 0; k < span; ++k) {
                                s0 = fma(*reinterpret_cast<const T *>(e + r * 16), yr[r], s0);
                                r = r + 1 == span ? 0 : r + 1;
                            }
                        }
                        s0 += s1;
#pragma unroll
                        for (int o = CW; o < 32; o <<= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                        if (part == 0 && j < m) y[j] -= s0;
                    } else if (sizeof(T) == 4) {  // the triangle
                        const float t = slab_triangle_t(reinterpret_cast<const uint4 *>(chunk), lane, nt, dir,
                                                        lane < nt ? (float)y[r0 + lane] : 0.f);
                        if (lane < nt) y[r0 + lane] = t;
                    } else if ((dir == 0 ? kept_u : kept_l) >> s & 1) {
                        // the chunk's columns c0..c0 + nc - 1: the rows of known unknowns, halved between the
                        // lanes of a column, then the triangle, whose pivots are the chunk's own unknowns
                        const int c0 = CW * jc - r0, nc = min(CW, nt - c0);
                        const T *a = reinterpret_cast<const T *>(chunk) + q * nt * W + col % W;  // row r: a[r W]
                        const int lo = dir == 0 ? 0 : c0 + nc, hi = dir == 0 ? c0 : nt;
                        if (j < m)
                            for (int r = lo + part; r < hi; r += PARTS) s0 = fma(a[r * W], y[r0 + r], s0);
#pragma unroll
                        for (int o = CW; o < 32; o <<= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                        T t = j < m ? y[j] - s0 : T(0);
                        for (int k = 0; k < nc; ++k) {
                            const int r = dir == 0 ? k : nc - 1 - k;
                            const T e = j < m && (dir == 0 ? col >= r : col < r) ? a[(c0 + r) * W] : T(1);
                            if (dir == 0 && col == r) t = t / e;
                            const T xr = __shfl_sync(0xffffffffu, t, r);
                            if (j < m && (dir == 0 ? col > r : col < r)) t = fma(-e, xr, t);
                        }
                        __syncwarp();
                        if (part == 0 && j < m) y[j] = t;
                    } else {  // its inverse
                        const int cc = j - r0 - part * span;  // the diagonal's row, counted from yr
                        if (j < m) {
                            int r = q % span;
                            for (int k = 0; k < span; ++k) {
                                const T a = *reinterpret_cast<const T *>(e + r * 16);
                                if (dir == 0 ? r <= cc : r > cc) s0 = fma(a, yr[r], s0);
                                r = r + 1 == span ? 0 : r + 1;
                            }
                        }
#pragma unroll
                        for (int o = CW; o < 32; o <<= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                        if (part == 0 && j < m) x[j - r0] = s0;
                        if (i == d1 - d0 - 1) {
                            __syncwarp();
                            if (lane < nt) y[r0 + lane] = dir == 0 ? x[lane] : y[r0 + lane] + x[lane];
                        }
                    }
                }
            }
        __syncwarp();
        for (int i = lane; i < m; i += 32) z[(size_t)blk * m + pm[i]] = (double)y[i];
        __syncwarp();
    }
}

template <typename T>
__global__ void __launch_bounds__(SOLVE_THREADS, 4)
k_lu_solve_t(const T *__restrict__ pool, const typename SolveType<T>::Aux *__restrict__ aux, const int *__restrict__ perm,
             size_t stride, int m, int count, const double *__restrict__ rhs, double *__restrict__ z) {
    if (solve_whole<T>(m)) lu_solve_t_blocks<T, SlabWhole<T, true>>(pool, aux, perm, stride, m, count, rhs, z);
    else lu_solve_t_blocks<T, SlabStream<T, true>>(pool, aux, perm, stride, m, count, rhs, z);
}

// The diagonal squares of the slabs of `count` FP64 blocks, in place: the unit lower triangle's inverse below the
// diagonal, the upper triangle's on and above it.  One warp per square; lane j computes column j of both
// by substitution in FP64 registers, the triangles read from shared memory as broadcasts.  Bound by those
// reads and the FMAs: 296 us for 4,096 blocks of 324, whose factorisation takes 15.6 ms.
//
// A triangle T stays as it is (kept) where max|T| max|T^-1| is above INVERT_BOUND or not finite, or where either lies
// so far from 1 that products with the inverse could leave the normal range.  The residual of y = X b for a
// computed inverse X is of the order eps |T| |X| |b|, against eps |T| |y| by substitution: with triangles below 128
// the normwise backward error of random, graded and near-singular blocks of 32 to 100 rows stayed below 8 % of
// 8 m eps, at 256 to 1,024 it came to 46 %, above to any multiple of it.  The triangles of the solver's own cells
// and faces (degrees 0 to 8, CFL 1 to 50) lie at 2 to 12 in the median and at 70 (cells) and 153 (a face) at most.
constexpr int SQUARE_WARPS = 4, SQUARE_PITCH = 33;
constexpr double INVERT_BOUND = 128, INVERT_RANGE = 0x1p900;
// Largest entries by their high words, which order |v| and put infinities and NaN last.
__device__ __forceinline__ void most(unsigned &mx, double v) { mx = max(mx, (unsigned)__double2hiint(v) & 0x7fffffffu); }
__device__ __forceinline__ bool invertible(unsigned t_hi, unsigned x_hi) {  // the lanes' largest |T| and |T^-1|
    const double t = __hiloint2double((int)__reduce_max_sync(0xffffffffu, t_hi), -1);
    const double x = __hiloint2double((int)__reduce_max_sync(0xffffffffu, x_hi), -1);
    return t <= INVERT_RANGE && x <= INVERT_RANGE && t * x <= INVERT_BOUND;
}
__global__ void __launch_bounds__(32 * SQUARE_WARPS, 4)
k_slab_invert(double *__restrict__ pool, size_t stride, int m, int count, unsigned char *__restrict__ kept) {
    constexpr int W = 2;
    __shared__ double tile[SQUARE_WARPS][32 * SQUARE_PITCH + 32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, slabs = (m + 31) / 32;
    const long long job = (long long)blockIdx.x * SQUARE_WARPS + wib;
    if (job >= (long long)count * slabs) return;
    const int s = (int)(job % slabs), r0 = 32 * s, nt = min(32, m - r0);
    double *a = tile[wib], *rd = a + 32 * SQUARE_PITCH;
    double *S = pool + (size_t)(job / slabs) * stride + (size_t)r0 * m + (size_t)r0 * nt;  // group r0 / W, row 0
    // the largest entries of the lane's row (T) and column (T^-1) of L and U
    unsigned tl = 0x3ff00000u, tu = 0, xl = 0x3ff00000u, xu = 0;  // (L: its unit diagonal)
    for (int g = 0; g < 32 / W; ++g)
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const int c = g * W + w;
            const double v = lane < nt && c < nt ? S[((size_t)g * nt + lane) * W + w] : lane == c ? 1. : 0.;
            a[lane * SQUARE_PITCH + c] = v;
            if (lane < nt && c < nt) most(c < lane ? tl : tu, v);
        }
    rd[lane] = 1. / a[lane * SQUARE_PITCH + lane];
    __syncwarp();
    double x[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = i == lane ? 1. : 0.;
#pragma unroll
    for (int k = 0; k < 31; ++k)
#pragma unroll
        for (int i = k + 1; i < 32; ++i) x[i] = fma(-a[i * SQUARE_PITCH + k], x[k], x[i]);
#pragma unroll
    for (int i = 1; i < 32; ++i) most(xl, x[i]);
    const bool inv_l = invertible(tl, xl);
    __syncwarp();
#pragma unroll
    for (int i = 1; i < 32; ++i)
        if (i > lane && inv_l) a[i * SQUARE_PITCH + lane] = x[i];
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = i == lane ? 1. : 0.;
#pragma unroll
    for (int k = 31; k >= 0; --k) {
        x[k] *= rd[k];
#pragma unroll
        for (int i = 0; i < k; ++i) x[i] = fma(-a[i * SQUARE_PITCH + k], x[k], x[i]);
    }
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (lane < nt) most(xu, x[i]);
    const bool inv_u = invertible(tu, xu);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (i <= lane && inv_u) a[i * SQUARE_PITCH + lane] = x[i];
    __syncwarp();
    if (lane < nt && (inv_l || inv_u))
        for (int g = 0; g < nt / W; ++g)
#pragma unroll
            for (int w = 0; w < W; ++w) S[((size_t)g * nt + lane) * W + w] = a[lane * SQUARE_PITCH + g * W + w];
    if (lane == 0) kept[job] = (inv_l ? 0 : KEPT_L) | (inv_u ? 0 : KEPT_U);
}

}  // namespace dgh
