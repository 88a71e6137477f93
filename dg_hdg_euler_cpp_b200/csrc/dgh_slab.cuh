// Factor storage shared by the LU kernels and the block solves, and the FP64 tensor instruction.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace dgh {

// Slab layout of a factored block (written by k_lu with slab_out, read by k_lu_solve): rows
// 32s..32s+nt-1 form slab s; inside a slab, columns come in groups of W = 16 bytes / sizeof(T)
// and each row's W values of a group are adjacent: element (32s + i, j) sits at
// 32 s m + (j / W) nt W + i W + j % W.  Lane i of a warp then loads its row's next W columns as
// one 16-byte vector, and the warp's load of a column group is nt*16 contiguous bytes.
// m = 4n^2 (cells) and 4n (faces) are multiples of W, so every group is complete.
// The 32 x 32 diagonal squares of FP64 slabs hold L^{-1} and U^{-1} in place of the triangles, but for
// those that are marked as kept (k_slab_invert); FP32 and FP16 slabs hold the triangles themselves.
__host__ __device__ constexpr int slab_count(int m) { return (m + 31) / 32; }
template <typename T> struct SlabVec;
template <> struct SlabVec<double> {
    using V = double2;
    static constexpr int W = 2;
};
template <> struct SlabVec<float> {
    using V = float4;
    static constexpr int W = 4;
};

// ---- 16-bit factor storage (the DG cell blocks, DGH_PRECISION_MIXED16) -------------------------
// FP16 slabs with 8 columns per 16-byte group and rows padded to mp = m rounded up to 8 (zeros
// past column m): element (32 s + i, j) at 32 s mp + (j / 8) nt 8 + 8 i + j % 8.  The strictly
// lower part holds L (|L| <= 1 under partial pivoting); each row's upper part U(i, i..m-1) is
// stored divided by that row's largest |U(i, j)|, whose reciprocal is kept as an FP32 row scale,
// so every stored U row peaks at 1 and stays in FP16's normal range.
constexpr int H_W = 8;
__host__ __device__ constexpr int pad8(int m) { return (m + 7) / 8 * 8; }

// FP64 DMMA m8n8k4: d = a b + d on one 8x8 tile, a the 8x4 and b the 4x8 operand fragment
// (lane l holds a[l/4][l%4], b[l%4][l/4] and d[l/4][2(l%4) .. 2(l%4)+1]).
__device__ __forceinline__ void dmma8x8x4(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

}  // namespace dgh
