// Host launchers of the batched pivoted LU (dgh_kernels_lu2.cuh), compiled in their own translation units
// (dgh_lu.cu, dgh_lu_fused.cu): the kernel is instantiated per CTA width, and per degree in its fused mode.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace dgh {
struct LLFuse;

// The widest block the kernel takes (a multiple of 4).
constexpr int LU_MAX_WIDTH = 512;
// Row length of an augmented matrix [A | B | r | pad]: rows start on 32 bytes.
__host__ __device__ constexpr int lu_aug_ld(int m, int t) { return (m + t + 1 + 3) / 4 * 4; }

// The dynamic shared-memory cap of a kernel is process-wide state that every context shares (and
// the contexts of a batch run on several host threads): it only ever rises, under a lock, so no
// launch sees a cap below the size it was launched with.  Throws std::runtime_error.
void allow_dynamic_smem(const void *fn, size_t bytes);

struct LuLaunch {
    cudaStream_t stream;
    int sms;
    int *status;
    int bit;  // status bit of a singular or non-finite factor
};
// Resident CTAs per SM of the pool / augmented form for width m, and of the fused DG form.
int lu_resident(int m, bool aug);
int lu_fused_resident(int n);
// pool: m x m blocks, factored in place (slab_out: slab layout), or rounded to FP32 slabs in out32.
void lu_pool(const LuLaunch &l, double *pool, int m, int count, int *perm, bool slab_out, float *out32);
// aug: [A | B | r | pad] with row length lu_aug_ld(m, t); X (m x t) and y (m) per matrix to x and y.
void lu_augmented(const LuLaunch &l, double *aug, int m, int t, int count, int *perm, double *x, double *y);
// The DG blocks of `count` cells assembled and factored by `grid` CTAs, each in its slot of fu.slots.
void lu_fused(const LuLaunch &l, int n, const LLFuse &fu, int grid, int count, int *perm, float *out32);
}  // namespace dgh
