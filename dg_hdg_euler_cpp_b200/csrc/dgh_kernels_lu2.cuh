// Batched LU with row partial pivoting on the FP64 tensor pipe (DMMA), one CTA per matrix, for the
// batched DG cell blocks and the HDG condensation.
//
// Crout's order in panels of 32 columns.  Per panel: (1) the panel's columns, below the finished U
// rows, are brought up to date by one product with K = k0 (cr_col_tiles: A and L read from global
// memory through the row map, U staged once in shared memory) and left in shared memory; (2) they are
// factored there with one thread per row and one barrier per column (cr_panel); (3) the panel's block
// row of U is formed, again by one product with K = k0 and a 32-row triangular solve in registers
// (cr_row_tiles).  The left-looking form this replaces (column panels only) needs k0 / 32 dependent
// steps of a triangular solve and a rank-32 product per panel, each with two barriers; here a panel has
// about eight barriers besides its columns'.  Augmented columns [B | r] take part in step 3, so they
// come out as L^{-1} P [B | r] and only the back substitution (cr_back) remains.
//
// What bounds it: at m = 324 two matrices fit an SM (shared memory), and their chains of panel
// latencies (about 1100 cycles a column with both running) leave the FP64 tensor pipe 17 % busy (30 %
// with augmented columns); small widths run many CTAs per SM.  Measured on one B200, LU of 2368 blocks
// of 324 (4096 of 100, 36): 6.1 ms (0.73, 0.13) against 9.1 ms (2.41, 0.77) for the left-looking kernel; with 145 augmented
// columns, 1776 of 324: 9.7 against 11.1 ms.
//
// Storage: every row of L and U stays in the ORIGINAL row of the matrix (row interchanges only
// change the position -> row map piv[]), so no data moves on a pivot.  A final pass gathers the rows
// into position order.
//
// Pivoting: the first largest |a| in position order wins ties (LAPACK getrf, Eigen
// PartialPivLU), with LAPACK swap semantics, so the pivot sequence is the reference's.
#pragma once
#include "dgh_kernels_dg.cuh"
#include "dgh_slab.cuh"

#include <algorithm>
#include <type_traits>

namespace dgh {

// Fused DG mode of k_lu (FN = nodes per direction > 0): the kernel walks all cells in one persistent
// launch, assembling each cell's block (k_dg_assemble's entries, collocated volume rule) into its
// CTA's private FP64 slot, factoring it there and writing the factors out in the slab layout of the
// block solves (FP64 to out64, FP32 to out32, or FP16 with row scales to out16 / scale16).
struct LLFuse {
    const double *vol = nullptr, *fcache = nullptr, *speeds = nullptr;
    double *slots = nullptr;  // gridDim.x slots of m * m doubles
    double *out64 = nullptr;
    __half *out16 = nullptr;
    float *scale16 = nullptr;
    Basis1D b;
    Grid g;
    double inv_step = 0;
    int first = 0;  // cell of block 0 (outputs and perm_out are offset by the caller)
};

constexpr int CR_NB = 32;  // panel width
constexpr int CR_H = 16;   // columns held in registers at a time
constexpr int CR_AP = 33;  // shared pitch of the panel: odd, for column accesses and k-permuted fragments
constexpr int CR_IP = 36;  // shared pitch of the 32 x 32 triangles (= 4 mod 16: conflict-free DMMA fragments)
constexpr int CR_PR = CR_H + 2;

// Warps for width m, and panel rows a thread may hold: one thread per row where the registers of the
// CTAs that fit an SM allow it, else two rows in the widest panels.
__host__ __device__ constexpr int cr_warps(int m) {
    return m <= 32 ? 1 : m <= 64 ? 2 : m <= 128 ? 4 : m <= 160 ? 5 : m <= 224 ? 7 : m <= 384 ? 8 : 16;
}
__host__ __device__ constexpr int cr_rows(int warps) { return warps == 8 ? 2 : 1; }
// CTAs per SM that the registers are cut for (128 to 170 a thread): the most that leave the tiles without spills
// of any size and their loads in flight.  One step more (16, 8, 4, 3 CTAs of 1, 2, 5, 7 warps) spills up to 336 bytes a
// thread or cuts the loads: LU of 12,800 blocks of 64 1.38 against 1.22 ms, augmented 2.88 against 2.26; 5,913 of 144
// 3.14, 3.09 and 5.76, 5.53; 4,087 of 196 5.05, 4.53 and 8.66, 7.90.  One step less for 4 warps (3): 10,201 of 100
// 2.87, 2.82, but 4,096, which are 10 rounds in place of 7, 1.15 and 1.21; two less (2, of 5 warps too) 3.45 and, 144
// wide, 3.61.
template <int NW> constexpr int cr_min_ctas() {
    return NW == 1 ? 12 : NW == 2 ? 6 : NW == 4 ? 4 : NW == 5 ? 3 : NW <= 8 ? 2 : 1;
}
__host__ __device__ constexpr int cr_stage_pitch(int m) { return m + (18 - m % 16) % 16; }
__host__ __device__ constexpr int cr_area(int m) {  // doubles of the panel / staging area
    return m * CR_AP > 32 * cr_stage_pitch(m) ? (m * CR_AP + 1) / 2 * 2 : 32 * cr_stage_pitch(m);
}
inline size_t cr_smem_bytes(int m) {
    return sizeof(double) * ((size_t)cr_area(m) + CR_NB * 8 + CR_NB * CR_IP) + sizeof(int4) * 2 * 16 + sizeof(int) * ((size_t)(m + 15) / 16 * 16 + CR_NB + 1);
}

// The CTA's shared memory.
struct CrShared {
    double *acc;    // m x CR_AP: rows < k0 the U columns of the panel, rows >= k0 the panel (position order)
    double *inv;    // 4 x 8 x 8: the inverses of the triangle's diagonal blocks
    double *tri;    // CR_NB x CR_IP: the panel's diagonal triangle (shares its place with prow and u12)
    double *prow;   // per column parity and warp: the best row's half and its pivot's reciprocal (CR_PR)
    double *u12;    // CR_H x CR_H: U of the first half's pivot rows in the second half
    int4 *cand;     // per column parity and warp: key high, key low, position, row
    int *piv;       // position -> original row
    int *pslot;     // the panel's pivot rows (CR_NB)
    int *bad;       // set when a pivot is zero, subnormal or not finite
    __device__ explicit CrShared(int m) {
        extern __shared__ __align__(16) unsigned char smraw[];
        acc = reinterpret_cast<double *>(smraw);
        inv = acc + cr_area(m);
        tri = prow = inv + CR_NB * 8;
        u12 = prow + 2 * 16 * CR_PR;
        cand = reinterpret_cast<int4 *>(tri + CR_NB * CR_IP);
        piv = reinterpret_cast<int *>(cand + 2 * 16);  // 16-byte aligned, padded to 16 entries
        pslot = piv + (m + 15) / 16 * 16;
        bad = pslot + CR_NB;
    }
};
__device__ __forceinline__ double2 cr_ld2(const double *A, int off) { return *reinterpret_cast<const double2 *>(A + (unsigned)off); }
__device__ __forceinline__ int cr_get(const int4 &v, int u) { return u == 0 ? v.x : u == 1 ? v.y : u == 2 ? v.z : v.w; }

// High word of the pivot search's key of |a| (the low word is a's own): larger |a| first, a NaN below
// every number, 0 = no candidate.
__device__ __forceinline__ unsigned cr_key(double a, bool on) {
    const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
    return !on ? 0u : h > 0x7ff00000u ? 1u : h + 2u;
}
// The lanes (one) holding the largest key of the warp, the smallest position among ties; mh is the
// warp's largest high word.  Only a tie of high words, which is rare, needs the rest.
__device__ __forceinline__ unsigned cr_best(unsigned mh, unsigned hi, double a, int pos) {
    unsigned bal = __ballot_sync(0xffffffffu, hi == mh);
    if (bal & (bal - 1)) {
        const unsigned lo = hi > 1u ? (unsigned)__double2loint(a) : 0u;
        bool best = hi == mh;
        const unsigned ml = __reduce_max_sync(0xffffffffu, best ? lo : 0u);
        best = best && lo == ml;
        const unsigned mp = __reduce_min_sync(0xffffffffu, best ? (unsigned)pos : 0xffffffffu);
        bal = __ballot_sync(0xffffffffu, best && (unsigned)pos == mp);
    }
    return bal;
}
__device__ __forceinline__ void cr_bar(int threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }

// One half (16 columns from panel column c0) of the panel factorisation.  A thread holds R rows of
// the panel (slot[r] = slot[0] + r 32 NW), 16 entries each, in registers; pos[r]: the row's position
// (LAPACK swaps); on[r]: the row exists.
//
// A column is one chain of latencies (23 cycles a DFMA, 28 a warp reduction, 110 a store, barrier
// and load), so it has one barrier: every warp's best row writes itself, its key and its pivot's
// reciprocal to shared memory before the winner is known, and every thread then reads the winner's.
// The next column's search starts before the rest of the rank-1 update.
template <int NW, int R>
__device__ __forceinline__ void cr_half(const CrShared &s, double (&a)[R][CR_H], int k0, int c0, int nbh, int act_warps,
                                        const bool (&on)[R], const int (&slot)[R], int (&pos)[R]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned hi, mh;
    double v, rcp;  // the thread's best candidate
    int which;
    bool act[R];
    auto candidate = [&](int j) {
        which = 0;
        v = a[0][j];
        hi = cr_key(v, act[0]);
#pragma unroll
        for (int r = 1; r < R; ++r) {
            const unsigned h = cr_key(a[r][j], act[r]);
            bool better = h > hi;
            if (h == hi && h > 1u) {
                const unsigned l0 = __double2loint(v), l1 = __double2loint(a[r][j]);
                better = l1 != l0 ? l1 > l0 : pos[r] < pos[which];
            } else if (h == hi && h == 1u) {
                better = pos[r] < pos[which];
            }
            if (better) {
                which = r;
                hi = h;
                v = a[r][j];
            }
        }
        mh = __reduce_max_sync(0xffffffffu, hi);
        rcp = 1. / v;
    };
#pragma unroll
    for (int r = 0; r < R; ++r) act[r] = on[r] && pos[r] >= k0 + c0;
    candidate(0);
#pragma unroll
    for (int j = 0; j < CR_H; ++j) {
        if (j % 4 == 0 && j >= nbh) break;  // nbh is a multiple of 4
        const int tp = k0 + c0 + j, buf = (j & 1) * NW;
        const int cpos = R > 1 && which ? pos[R - 1] : pos[0];
        if ((cr_best(mh, hi, v, cpos) >> lane) & 1u) {
            s.cand[buf + warp] = make_int4((int)hi, __double2loint(v), cpos, R > 1 && which ? slot[R - 1] : slot[0]);
            double *out = s.prow + (size_t)(buf + warp) * CR_PR;
            out[CR_H] = v != 0. ? rcp : 1.;
            auto put = [&](const double (&w)[CR_H]) {
                if (j % 2 == 0 && j + 1 < CR_H) out[j + 1] = w[j + 1];
#pragma unroll
                for (int c = (j + 2) & ~1; c < CR_H; c += 2)
                    *reinterpret_cast<double2 *>(out + c) = make_double2(w[c], w[c + 1]);
            };
            if (R > 1 && which) put(a[R - 1]);
            else put(a[0]);
        }
        int w = 0;
        if (NW == 1) {
            __syncwarp();
        } else {
            cr_bar(32 * act_warps);
            const int4 k = lane < act_warps ? s.cand[buf + lane] : make_int4(0, 0, 0x7fffffff, 0);
            const unsigned gm = __reduce_max_sync(0xffffffffu, (unsigned)k.x);
            w = 31 - __clz(cr_best(gm, (unsigned)k.x, __hiloint2double(0, k.y), k.z));
        }
        const double *p = s.prow + (size_t)(buf + w) * CR_PR;
        const int4 win = s.cand[buf + w];
        double l[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (slot[r] == win.w) {
                s.pslot[c0 + j] = slot[r];
                pos[r] = tp;
            } else if (pos[r] == tp) {
                pos[r] = win.z;
            }
            act[r] = on[r] && pos[r] > tp;
            l[r] = a[r][j] * p[CR_H];
            if (act[r]) a[r][j] = l[r];
        }
        if (j + 1 < CR_H) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (act[r]) a[r][j + 1] -= l[r] * p[j + 1];
            candidate(j + 1);
#pragma unroll
            for (int c = (j + 2) & ~1; c < CR_H; c += 2) {
                const double2 q = *reinterpret_cast<const double2 *>(p + c);
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (act[r]) {
                        if (c > j + 1) a[r][c] -= l[r] * q.x;
                        a[r][c + 1] -= l[r] * q.y;
                    }
            }
        }
    }
}
// Factors the panel (columns 0..nb-1 of rows k0..m-1 of s.acc, the rows' positions at its start), R
// rows a thread, in two halves of 16 columns held in registers; writes the factors to the rows of
// A, leaves them in s.acc (pivot row i of the panel in row pslot[i]) and updates piv.
template <int NW, int R>
__device__ __noinline__ void cr_panel(double *A, int m, int ld, int k0, int nb) {
    const CrShared s(m);
    constexpr int T = 32 * NW;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int act_warps = min(NW, (m - k0 + 31) >> 5);
    int slot[R], pos[R], orig[R];
    bool on[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        slot[r] = pos[r] = k0 + tid + r * T;
        on[r] = slot[r] < m;
        orig[r] = on[r] ? s.piv[slot[r]] : 0;
    }
    if (warp < act_warps) {
        double *row[R];
        double a[R][CR_H];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            row[r] = s.acc + (size_t)(on[r] ? slot[r] : k0) * CR_AP;
#pragma unroll
            for (int c = 0; c < CR_H; ++c) a[r][c] = row[r][c];
        }
#pragma unroll 1
        for (int c0 = 0;; c0 += CR_H) {
            cr_half<NW, R>(s, a, k0, c0, min(nb - c0, CR_H), act_warps, on, slot, pos);
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (on[r])
#pragma unroll
                    for (int c = 0; c < CR_H; ++c) row[r][c0 + c] = a[r][c];
            if (c0 + CR_H >= nb) break;
            if (NW == 1) __syncwarp();
            else cr_bar(32 * act_warps);
            if (warp == 0 && lane < CR_H) {  // U12 = L11^{-1} A12, a column per lane
                double u[CR_H];
#pragma unroll
                for (int k = 0; k < CR_H; ++k) u[k] = s.acc[(size_t)s.pslot[k] * CR_AP + CR_H + lane];
#pragma unroll
                for (int k = 0; k < CR_H; ++k) {
                    s.acc[(size_t)s.pslot[k] * CR_AP + CR_H + lane] = s.u12[k * CR_H + lane] = u[k];
#pragma unroll
                    for (int i = k + 1; i < CR_H; ++i) u[i] -= s.acc[(size_t)s.pslot[i] * CR_AP + k] * u[k];
                }
            }
            if (NW == 1) __syncwarp();
            else cr_bar(32 * act_warps);
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int c = 0; c < CR_H; ++c) a[r][c] = row[r][CR_H + c];
#pragma unroll 2
            for (int j = 0; j < CR_H; ++j) {
                double l[R];
#pragma unroll
                for (int r = 0; r < R; ++r) l[r] = on[r] && pos[r] >= k0 + CR_H ? row[r][j] : 0.;
#pragma unroll
                for (int c = 0; c < CR_H; c += 2) {
                    const double2 u = *reinterpret_cast<const double2 *>(s.u12 + j * CR_H + c);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        a[r][c] -= l[r] * u.x;
                        a[r][c + 1] -= l[r] * u.y;
                    }
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (on[r] && pos[r] < k0 + nb) {  // a pivot row: its pivot
                const double d = row[r][pos[r] - k0];
                if (!isfinite(d) || !(fabs(d) > 2.2250738585072014e-308)) *s.bad = 1;
            }
            // the warp's rows to A (32 lanes = the panel's columns)
            const int first = k0 + r * T + 32 * warp, rows = min(32, m - first);
#pragma unroll 4
            for (int i = 0; i < rows; ++i) {
                const int o = __shfl_sync(0xffffffffu, orig[r], i);
                if (lane < nb) A[(size_t)o * ld + k0 + lane] = s.acc[(size_t)(first + i) * CR_AP + lane];
            }
        }
    }
    __syncthreads();  // every row and position map entry has been read
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (on[r]) s.piv[pos[r]] = orig[r];
    __syncthreads();
}

// s.inv gets the inverses of the four 8 x 8 diagonal blocks of the triangle in s.tri (unit lower, or
// upper with its diagonal): lane 8 b + i holds entry i of block b, a column of all four blocks per warp
// at a time.
template <int NW, bool UPPER> __device__ __forceinline__ void cr_diag_inverse(double *inv, const double *tri) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, base = lane & 24, i = lane & 7;
    const double *row = tri + lane * CR_IP + base;
    const double rd = UPPER ? 1. / row[i] : 1.;
    for (int c = warp; c < 8; c += NW) {
        double x = i == c ? 1. : 0.;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int q = UPPER ? 7 - k : k;
            if (UPPER && i == q) x *= rd;
            const double t = (UPPER ? i < q : i > q) ? row[q] : 0.;
            x -= t * __shfl_sync(0xffffffffu, x, base + q);
        }
        inv[lane * 8 + c] = x;
    }
}
// tri = the panel's diagonal triangle, identity outside nb x nb: element (i, c) from src(i, c).
template <int NW, bool UPPER, class F> __device__ __forceinline__ void cr_load_tri(double *tri, int nb, F src) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int C = (CR_NB + NW - 1) / NW;
#pragma unroll
    for (int e = 0; e < C; ++e) {
        const int i = warp + e * NW;
        if (i >= CR_NB) break;
        double v = i == lane ? 1. : 0.;
        if (i < nb && (UPPER ? lane < nb && lane >= i : lane < i)) v = src(i, lane);
        tri[i * CR_IP + lane] = v;
    }
}
// dst[i * pitch + k] = -A[piv[k0 + i]][c0 + k] for the panel's rows i (row nb - 1 repeated past the
// end) and k < K, zero up to Kp; eight loads in flight per lane.
template <int NW>
__device__ __forceinline__ void cr_stage_rows(double *dst, int pitch, const double *A, int ld, const int *piv, int k0, int nb,
                                              int c0, int K, int Kp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int chunks = (K + 31) / 32 * CR_NB;  // (32-column block, row)
    for (int q = warp; q < chunks; q += 8 * NW) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int c = q + u * NW, i = c & (CR_NB - 1), k = (c / CR_NB) * 32 + lane;
            v[u] = c < chunks && k < K ? A[(size_t)piv[k0 + min(i, nb - 1)] * ld + c0 + k] : 0.;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int c = q + u * NW, i = c & (CR_NB - 1), k = (c / CR_NB) * 32 + lane;
            if (c < chunks && k < Kp) dst[i * pitch + k] = -v[u];
        }
    }
}
// acc[i][c] = sign * A[piv[i]][j0 + c] for rows i < rows, c < ncols (zero up to 32).
template <int NW>
__device__ __forceinline__ void cr_stage_cols(double *acc, const double *A, int ld, const int *piv, int rows, int j0, int ncols,
                                              double sign) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int q = warp; q < rows; q += 8 * NW) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = q + u * NW;
            v[u] = i < rows && lane < ncols ? A[(size_t)piv[i] * ld + j0 + lane] : 0.;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = q + u * NW;
            if (i < rows) acc[i * CR_AP + lane] = sign * v[u];
        }
    }
}

// c = T^{-1} c for one warp's 32 x (8 NT) tile held in DMMA accumulators, T the panel's triangle (tri,
// with the inverses of its 8 x 8 diagonal blocks in inv): block substitution by 8 rows, each block's
// accumulators becoming B fragments by lane shuffles.
template <int NT, bool UPPER>
__device__ __forceinline__ void cr_tri(const double *inv, const double *tri, double (&c)[4][NT][2]) {
    const int lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
    auto frag = [&](const double (&t)[NT][2], int h, double (&b)[NT]) {  // rows 4 h .. 4 h + 3 of the block
        const int src = ((h * 4 + lc) << 2) | (lr >> 1);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const double v0 = __shfl_sync(0xffffffffu, t[nt][0], src), v1 = __shfl_sync(0xffffffffu, t[nt][1], src);
            b[nt] = (lr & 1) ? v1 : v0;
        }
    };
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int k = UPPER ? 3 - q : q;
        double x[NT][2];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) x[nt][0] = x[nt][1] = 0.;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            double b[NT];
            frag(c[k], h, b);
            const double a = inv[(k * 8 + lr) * 8 + 4 * h + lc];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) dmma8x8x4(x[nt], a, b[nt]);
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            c[k][nt][0] = x[nt][0];
            c[k][nt][1] = x[nt][1];
        }
        if (q == 3) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            double b[NT];
            frag(x, h, b);
#pragma unroll
            for (int mt = 0; mt < 4; ++mt) {
                if (UPPER ? mt >= k : mt <= k) continue;
                const double a = -tri[(mt * 8 + lr) * CR_IP + k * 8 + 4 * h + lc];
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) dmma8x8x4(c[mt][nt], a, b[nt]);
            }
        }
    }
}

// Row block of U: for the columns [c_begin, c_end) of the panel's nb rows (positions k0..),
// U = L_pp^{-1} (A - L[rows, 0:k0] U[0:k0, cols]).  The staged operand in s.acc holds -L (32 x k0,
// pitch k0 + 1).  A warp's tile is 32 x 16; tile column 8 nt + n is matrix column col0 + 2 n + nt, so
// that a lane reads its two columns of a row of U, and its four of A, as 16-byte vectors (c_begin, c_end
// and ld are even); MMA step u of a group of 16 k's takes k = 4 lc + u, so that a lane reads its
// four row numbers as one vector.
template <int NW>
__device__ __noinline__ void cr_row_tiles(double *A, int m, int ld, int k0, int nb, int c_begin, int c_end) {
    const CrShared s(m);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane >> 2, lc = lane & 3;
    const int pitch = k0 + 1;
    for (int col0 = c_begin + warp * 16; col0 < c_end; col0 += NW * 16) {
        const int bc = min(col0 + 2 * lr, c_end - 2);
        double2 b[2][4];  // the B operand: 16 k's in use, 16 on their way
        auto fetch = [&](double2 (&v)[4], int k) {
            const int4 rows = *reinterpret_cast<const int4 *>(s.piv + k + 4 * lc);
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = cr_ld2(A, cr_get(rows, u) * ld + bc);
        };
        if (k0 > 0) fetch(b[0], 0);
        double c[4][2][2];
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
            const int r = mt * 8 + lr, off = s.piv[k0 + min(r, nb - 1)] * ld + col0 + 4 * lc;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const double2 v = r < nb && col0 + 4 * lc + 2 * e < c_end ? cr_ld2(A, off + 2 * e) : make_double2(0., 0.);
                c[mt][0][e] = v.x;
                c[mt][1][e] = v.y;
            }
        }
        const double *as = s.acc + lr * pitch + 4 * lc;
#pragma unroll 1
        for (int kk = 0; kk < k0; kk += 32)  // k0 is a multiple of 32
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                if (g == 0 || kk + 32 < k0) fetch(b[g ^ 1], kk + 16 * (g + 1));
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int mt = 0; mt < 4; ++mt) {
                        const double a = as[mt * 8 * pitch + kk + 16 * g + u];
                        dmma8x8x4(c[mt][0], a, b[g][u].x);
                        dmma8x8x4(c[mt][1], a, b[g][u].y);
                    }
            }
        cr_tri<2, false>(s.inv, s.tri, c);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
            const int r = mt * 8 + lr, off = s.piv[k0 + min(r, nb - 1)] * ld + col0 + 4 * lc;
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (r < nb && col0 + 4 * lc + 2 * e < c_end)
                    *reinterpret_cast<double2 *>(A + (unsigned)(off + 2 * e)) = make_double2(c[mt][0][e], c[mt][1][e]);
        }
    }
}

// Panel columns k1.. of the rows at positions r >= k1: C = A - L[r, 0:k1] U[0:k1, cols], with -U
// staged in rows 0..k1-1 of s.acc; C goes to rows k1.. of s.acc.  8 MT rows x 8 NT columns a warp.  A lane
// reads 4 consecutive entries of its row of L (ld is even, rows are 16-byte aligned): MMA step i of a group
// of 16 k's takes k = 4 lc + i of both operands.
template <int NW, int MT, int NT>
__device__ __noinline__ void cr_col_tiles(const double *A, int m, int ld, int k1, int nb) {
    const CrShared s(m);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane >> 2, lc = lane & 3;
    constexpr int HALVES = 4 / NT;  // column halves of the panel
    for (int unit = warp;; unit += NW) {
        const int rb = k1 + unit / HALVES * 8 * MT, n0 = unit % HALVES * 8 * NT;
        if (rb >= m) break;
        double c[MT][NT][2];
        double2 a[2][MT][2];  // the A operand: 16 k's in use, 16 on their way
        int off[MT];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) off[mt] = s.piv[min(rb + mt * 8 + lr, m - 1)] * ld;
        auto fetch = [&](double2 (&v)[MT][2], int k) {
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int h = 0; h < 2; ++h) v[mt][h] = cr_ld2(A, off[mt] + k + 4 * lc + 2 * h);
        };
        fetch(a[0], 0);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int cc = n0 + nt * 8 + 2 * lc;
                const double2 v = cc < nb ? cr_ld2(A, off[mt] + k1 + cc) : make_double2(0., 0.);
                c[mt][nt][0] = v.x;
                c[mt][nt][1] = v.y;
            }
        const double *bs = s.acc + 4 * lc * CR_AP + n0 + lr;
#pragma unroll 1
        for (int kk = 0; kk < k1; kk += 32)  // k1 is a multiple of 32
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                if (g == 0 || kk + 32 < k1) fetch(a[g ^ 1], kk + 16 * (g + 1));
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    double b[NT];
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) b[nt] = bs[(kk + 16 * g + i) * CR_AP + nt * 8];
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt)
                            dmma8x8x4(c[mt][nt], i & 1 ? a[g][mt][i >> 1].y : a[g][mt][i >> 1].x, b[nt]);
                }
            }
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            const int r = rb + mt * 8 + lr;
            if (r >= m) continue;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) s.acc[(size_t)r * CR_AP + n0 + nt * 8 + 2 * lc + e] = c[mt][nt][e];
        }
    }
}

// cr_row_tiles for few columns (ncols <= 64): warps take 8 rows x 16 columns of the product each, so
// that its long dot products run side by side; the tiles meet in shared memory (behind the staged rows)
// for the triangle.
constexpr int CR_MEET = 66;  // pitch of the meeting place
template <int NW>
__device__ __noinline__ void cr_row_few(double *A, int m, int ld, int k0, int nb, int c_begin, int c_end) {
    const CrShared s(m);
    constexpr int P = CR_MEET;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane >> 2, lc = lane & 3;
    const int pitch = k0 + 1, tiles = (c_end - c_begin + 15) / 16;
    double *meet = s.acc + (32 * pitch + 1) / 2 * 2;
    for (int unit = warp; unit < 4 * tiles; unit += NW) {
        const int mt = unit & 3, off = (unit >> 2) * 16, bc = min(c_begin + off + 2 * lr, c_end - 2);
        double2 b[2][4];  // two groups of 16 k's in flight
        auto fetch = [&](double2 (&v)[4], int k) {
            const int4 rows = *reinterpret_cast<const int4 *>(s.piv + k + 4 * lc);
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = cr_ld2(A, cr_get(rows, u) * ld + bc);
        };
        fetch(b[0], 0);
        fetch(b[1], 16);  // k0 is a multiple of 32
        const int r = mt * 8 + lr, ro = s.piv[k0 + min(r, nb - 1)] * ld + c_begin + off + 4 * lc;
        double c[2][2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const double2 v = r < nb && c_begin + off + 4 * lc + 2 * e < c_end ? cr_ld2(A, ro + 2 * e) : make_double2(0., 0.);
            c[0][e] = v.x;
            c[1][e] = v.y;
        }
        const double *as = s.acc + r * pitch + 4 * lc;
#pragma unroll 1
        for (int kk = 0; kk < k0; kk += 32)
#pragma unroll
            for (int g = 0; g < 2; ++g) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const double a = as[kk + 16 * g + u];
                    dmma8x8x4(c[0], a, b[g][u].x);
                    dmma8x8x4(c[1], a, b[g][u].y);
                }
                if (kk + 32 < k0) fetch(b[g], kk + 32 + 16 * g);
            }
#pragma unroll
        for (int e = 0; e < 2; ++e)
            *reinterpret_cast<double2 *>(meet + r * P + off + 4 * lc + 2 * e) = make_double2(c[0][e], c[1][e]);
    }
    __syncthreads();
    for (int tile = warp; tile < tiles; tile += NW) {
        double c[4][2][2];
#pragma unroll
        for (int mt = 0; mt < 4; ++mt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const double2 v = *reinterpret_cast<const double2 *>(meet + (mt * 8 + lr) * P + tile * 16 + 2 * (2 * lc + e));
                c[mt][0][e] = v.x;
                c[mt][1][e] = v.y;
            }
        cr_tri<2, false>(s.inv, s.tri, c);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
            const int r = mt * 8 + lr;
            double *row = A + (size_t)s.piv[k0 + min(r, nb - 1)] * ld;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = c_begin + tile * 16 + 2 * (2 * lc + e);
                if (r < nb && col < c_end) *reinterpret_cast<double2 *>(row + col) = make_double2(c[mt][0][e], c[mt][1][e]);
            }
        }
    }
}

// LU of the m x m matrix A (row length ld >= m, m and ld multiples of 4, A 32-byte aligned; columns
// m..ld-1 receive L^{-1} P).  On exit every
// row of L and U is in its original row of A, piv[i] the row of position i.
template <int NW> __device__ __forceinline__ void cr_factor(double *A, int m, int ld) {
    constexpr int T = 32 * NW;
    const CrShared s(m);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < m; i += T) s.piv[i] = i;
    __syncthreads();
    cr_stage_cols<NW>(s.acc, A, ld, s.piv, m, 0, min(CR_NB, m), 1.);
    __syncthreads();
    for (int k0 = 0; k0 < m; k0 += CR_NB) {
        const int nb = min(CR_NB, m - k0), k1 = k0 + nb;
        if (cr_rows(NW) > 1 && m - k0 > T) cr_panel<NW, cr_rows(NW)>(A, m, ld, k0, nb);
        else cr_panel<NW, 1>(A, m, ld, k0, nb);
        if (k1 >= ld) break;
        cr_load_tri<NW, false>(s.tri, nb, [&](int i, int c) { return s.acc[(size_t)s.pslot[i] * CR_AP + c]; });
        __syncthreads();
        // -L of the panel's rows; it ends below row k0 of s.acc, where the panel starts
        cr_diag_inverse<NW, false>(s.inv, s.tri);
        if (k0 > 0) cr_stage_rows<NW>(s.acc, k0 + 1, A, ld, s.piv, k0, nb, 0, k0, k0);
        __syncthreads();
        if (k0 > 0 && ld - k1 <= 64 && 32 * (k0 + 1) + 2 + 32 * CR_MEET <= cr_area(m)) cr_row_few<NW>(A, m, ld, k0, nb, k1, ld);
        else cr_row_tiles<NW>(A, m, ld, k0, nb, k1, ld);
        __syncthreads();
        if (k1 >= m) break;
        const int nb1 = min(CR_NB, m - k1);
        cr_stage_cols<NW>(s.acc, A, ld, s.piv, k1, k1, nb1, -1.);
        __syncthreads();
        if (m - k1 > NW * 8) cr_col_tiles<NW, 2, 4>(A, m, ld, k1, nb1);
        else if (m - k1 > NW * 4) cr_col_tiles<NW, 1, 4>(A, m, ld, k1, nb1);
        else cr_col_tiles<NW, 1, 2>(A, m, ld, k1, nb1);
        __syncthreads();
    }
    __syncthreads();
}

// Back substitution of columns m..m+t of A: X | y = U^{-1} (those columns, position rows), row i =
// unknown i, to x (m x t; t even, 16-byte aligned) and y (m).  Column t is the last.  A warp's tile is
// 32 x 16 with cr_row_tiles' column order.
template <int NW>
__device__ __noinline__ void cr_back(const double *A, int m, int ld, int t, double *x, double *y) {
    const CrShared s(m);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane >> 2, lc = lane & 3;
    for (int p = (m + CR_NB - 1) / CR_NB - 1; p >= 0; --p) {
        const int k0 = p * CR_NB, nb = min(CR_NB, m - k0), k1 = k0 + nb, K = m - k1;
        const int Kp = (K + 15) / 16 * 16, pitch = Kp + 1;
        cr_load_tri<NW, true>(s.tri, nb, [&](int i, int c) { return A[(size_t)s.piv[k0 + i] * ld + k0 + c]; });
        cr_stage_rows<NW>(s.acc, pitch, A, ld, s.piv, k0, nb, k1, K, Kp);
        __syncthreads();
        cr_diag_inverse<NW, true>(s.inv, s.tri);
        __syncthreads();
        for (int col0 = warp * 16; col0 <= t; col0 += NW * 16) {
            const int bcol = col0 + 2 * lr;  // the lane's columns bcol, bcol + 1 (t even: y alone at bcol == t)
            auto fetch = [&](int k) {
                const int i = min(k1 + k, m - 1);  // past the end the staged operand is zero
                return bcol < t ? cr_ld2(x, i * t + bcol) : make_double2(bcol == t ? y[i] : 0., 0.);
            };
            double2 b[2][4];
            if (K > 0)
#pragma unroll
                for (int u = 0; u < 4; ++u) b[0][u] = fetch(4 * lc + u);
            double c[4][2][2];
#pragma unroll
            for (int mt = 0; mt < 4; ++mt) {
                const int r = mt * 8 + lr, off = s.piv[k0 + min(r, nb - 1)] * ld + m + col0 + 4 * lc;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const double2 v = r < nb && col0 + 4 * lc + 2 * e <= t ? cr_ld2(A, off + 2 * e) : make_double2(0., 0.);
                    c[mt][0][e] = v.x;
                    c[mt][1][e] = v.y;
                }
            }
            const double *as = s.acc + lr * pitch + 4 * lc;
#pragma unroll 1
            for (int kk = 0; kk < K; kk += 32)
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    if (kk + 16 * g >= K) break;
                    if (kk + 16 * (g + 1) < K)
#pragma unroll
                        for (int u = 0; u < 4; ++u) b[g ^ 1][u] = fetch(kk + 16 * (g + 1) + 4 * lc + u);
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int mt = 0; mt < 4; ++mt) {
                            const double a = as[mt * 8 * pitch + kk + 16 * g + u];
                            dmma8x8x4(c[mt][0], a, b[g][u].x);
                            dmma8x8x4(c[mt][1], a, b[g][u].y);
                        }
                }
            cr_tri<2, true>(s.inv, s.tri, c);
#pragma unroll
            for (int mt = 0; mt < 4; ++mt) {
                const int r = mt * 8 + lr;
                if (r >= nb) continue;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int col = col0 + 2 * (2 * lc + e);
                    if (col < t) *reinterpret_cast<double2 *>(x + (size_t)(k0 + r) * t + col) = make_double2(c[mt][0][e], c[mt][1][e]);
                    else if (col == t) y[k0 + r] = c[mt][0][e];
                }
            }
        }
        __syncthreads();
    }
}

// dst[0..m) = src[0..m) by one warp: 16-byte loads, up to four in flight per lane (m even and
// both rows 16-byte aligned: every row starts at a multiple of 8 m bytes, m = 4 n^2).
__device__ __forceinline__ void ll_stage_row(double *dst, const double *src, int m) {
    const int lane = threadIdx.x & 31, h = m / 2;
    const double2 *s2 = reinterpret_cast<const double2 *>(src);
    double2 *d2 = reinterpret_cast<double2 *>(dst);
    for (int c0 = lane; c0 < h; c0 += 4 * 32) {
        double2 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = c0 + 32 * u;
            if (c < h) v[u] = s2[c];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = c0 + 32 * u;
            if (c < h) d2[c] = v[u];
        }
    }
}

// Batched LU.  AUG = false: pool holds m x m blocks (ld = m); on exit row i of each block is position i
// of the factors (unit L below, U on and above the diagonal), perm_out[i] = its original row, and with
// slab_out the block is rewritten in the slab layout of k_lu_solve.  With out32 != nullptr the factors
// are instead written, rounded to FP32, in the FP32 slab layout to out32 (m x m per block) and pool is
// left in original-row order.  FN > 0: the fused DG mode (LLFuse).
// AUG = true: pool holds [A | B | r | pad] (t columns of B, ld >= m + t + 1, ld a multiple of 4); on exit
// X | y = A^{-1}[B r] (row i = unknown i) is in x_out (m x t row-major per matrix) and y_out (m per
// matrix), and the A part holds the factors in original-row order, perm_out[i] the row of position i.
template <int NW, bool AUG, int FN>
__global__ void __launch_bounds__(32 * NW, cr_min_ctas<NW>())
k_lu_crout(double *pool, size_t stride, int m, int ld, int t, int count, int *__restrict__ perm_out, int *status,
           int singular_bit, int slab_out, float *__restrict__ out32, double *x_out, double *y_out, LLFuse fu) {
    constexpr int T = 32 * NW;
    const CrShared s(m);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ Basis1D fsb;
    if constexpr (FN > 0) stage_basis<FN>(fu.b, fsb);
    for (int blk = blockIdx.x; blk < count; blk += gridDim.x) {
        double *A = pool + (size_t)blk * stride;
        if constexpr (FN > 0) {
            // assemble the cell's block into this CTA's slot (tables and rows in the panel area)
            constexpr int FP = FN * FN, FM = NVAR * FP, TABLES = 2 * FP * 16 + NFACES * FN * 16;
            constexpr int R = (cr_area(FM) - TABLES) / FM < FM ? (cr_area(FM) - TABLES) / FM : FM;
            A = fu.slots + (size_t)blockIdx.x * FM * FM;
            double *jx = s.acc, *jy = jx + FP * 16, *fj = jy + FP * 16, *buf = fj + NFACES * FN * 16;
            __syncthreads();
            cell_tables<FN, false>(fu.first + blk, fu.vol, fu.fcache, fu.speeds, fsb, fu.g, jx, jy, fj);
            for (int r0 = 0; r0 < FM; r0 += R) {
                const int rows = min(R, FM - r0);
                for (int i = tid; i < rows * FM / 2; i += T) reinterpret_cast<double2 *>(buf)[i] = make_double2(0., 0.);
                __syncthreads();
                cell_rows_fill<FN>(buf, FM, r0, rows, jx, jy, fj, fsb, fu.g, fu.inv_step, true, T);
                __syncthreads();
                rows_out(A + (size_t)r0 * FM, buf, rows * FM, T);
                __syncthreads();
            }
        }
        if (tid == 0) *s.bad = 0;
        __syncthreads();
        cr_factor<NW>(A, m, ld);
        if (perm_out)
            for (int i = tid; i < m; i += T) perm_out[(size_t)blk * m + i] = s.piv[i];
        if constexpr (AUG) {
            cr_back<NW>(A, m, ld, t, x_out + (size_t)blk * m * t, y_out + (size_t)blk * m);
        } else if (FN > 0 && fu.out16) {
            // ---- FP16 slabs with row scales (k_pack_half's layout) from the original-row storage:
            // stage 32 position rows, each row's largest |U| by a warp, then 8-column groups
            const int sp = cr_stage_pitch(m), mp8 = pad8(m);
            double *stage = s.acc;
            __shared__ float rsc[32];
            __half *out = fu.out16 + (size_t)blk * m * mp8;
            for (int r0 = 0; r0 < m; r0 += 32) {
                const int nt = min(32, m - r0);
                for (int rr = warp; rr < nt; rr += NW) {
                    double *row = stage + (size_t)rr * sp;
                    ll_stage_row(row, A + (size_t)s.piv[r0 + rr] * ld, m);
                    __syncwarp();
                    double big = 0;
                    for (int j = r0 + rr + lane; j < m; j += 32) big = fmax(big, fabs(row[j]));
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
                    if (lane == 0) {
                        rsc[rr] = big > 0 ? (float)(1. / big) : 1.f;
                        fu.scale16[(size_t)blk * m + r0 + rr] = rsc[rr];
                    }
                }
                __syncthreads();
                for (int gg = warp; gg < mp8 / H_W; gg += NW)
                    for (int rr = lane; rr < nt; rr += 32) {
                        __align__(16) __half v[H_W];
                        const double inv = (double)rsc[rr];
#pragma unroll
                        for (int w = 0; w < H_W; ++w) {
                            const int j = gg * H_W + w;
                            const double a = j < m ? stage[(size_t)rr * sp + j] : 0.;
                            v[w] = __double2half(j >= r0 + rr ? a * inv : a);
                        }
                        *reinterpret_cast<uint4 *>(out + (size_t)r0 * mp8 + (size_t)gg * nt * H_W + rr * H_W) =
                            *reinterpret_cast<const uint4 *>(v);
                    }
                __syncthreads();
            }
        } else if (out32 || (FN > 0 && fu.out64)) {
            // ---- FP32 or FP64 slabs straight from the original-row storage: stage 32 position rows
            // (16-byte loads, several in flight per thread), then a lane writes one row's slab group
            const int sp = cr_stage_pitch(m);
            double *stage = s.acc;
            for (int r0 = 0; r0 < m; r0 += 32) {
                const int nt = min(32, m - r0);
                for (int rr = warp; rr < nt; rr += NW) ll_stage_row(stage + (size_t)rr * sp, A + (size_t)s.piv[r0 + rr] * ld, m);
                __syncthreads();
                if (out32) {
                    constexpr int W = SlabVec<float>::W;
                    float4 *reg = reinterpret_cast<float4 *>(out32 + (size_t)blk * m * m + (size_t)r0 * m);
                    for (int g = warp; g < m / W; g += NW)
                        if (lane < nt) {
                            const double2 a = *reinterpret_cast<const double2 *>(stage + (size_t)lane * sp + g * W);
                            const double2 b = *reinterpret_cast<const double2 *>(stage + (size_t)lane * sp + g * W + 2);
                            reg[(size_t)g * nt + lane] = make_float4((float)a.x, (float)a.y, (float)b.x, (float)b.y);
                        }
                } else {
                    constexpr int W = SlabVec<double>::W;
                    double2 *reg = reinterpret_cast<double2 *>(fu.out64 + (size_t)blk * m * m + (size_t)r0 * m);
                    for (int g = warp; g < m / W; g += NW)
                        if (lane < nt)
                            reg[(size_t)g * nt + lane] = *reinterpret_cast<const double2 *>(stage + (size_t)lane * sp + g * W);
                }
                __syncthreads();
            }
        } else if constexpr (FN == 0) {
            // ---- gather the rows into position order, 32 columns at a time
            for (int c0 = 0; c0 < m; c0 += CR_NB) {
                const int w = min(CR_NB, m - c0);
                cr_stage_cols<NW>(s.acc, A, ld, s.piv, m, c0, w, 1.);
                __syncthreads();
                for (int i = warp; i < m; i += NW)
                    if (lane < w) A[(size_t)i * ld + c0 + lane] = s.acc[i * CR_AP + lane];
                __syncthreads();
            }
            if (slab_out) {  // in-place conversion to the slab layout read by k_lu_solve
                constexpr int W = SlabVec<double>::W;
                const int sp = cr_stage_pitch(m);
                double *stage = s.acc;
                for (int r0 = 0; r0 < m; r0 += 32) {
                    const int nt = min(32, m - r0);
                    double *reg = A + (size_t)r0 * m;
                    for (int rr = warp; rr < nt; rr += NW) ll_stage_row(stage + (size_t)rr * sp, reg + (size_t)rr * m, m);
                    __syncthreads();
                    double2 *reg2 = reinterpret_cast<double2 *>(reg);
                    for (int g = warp; g < m / W; g += NW)
                        if (lane < nt)
                            reg2[(size_t)g * nt + lane] = *reinterpret_cast<const double2 *>(stage + (size_t)lane * sp + g * W);
                    __syncthreads();
                }
            }
        }
        if (tid == 0 && *s.bad) atomicOr(status, singular_bit);
        __syncthreads();
    }
}

}  // namespace dgh
