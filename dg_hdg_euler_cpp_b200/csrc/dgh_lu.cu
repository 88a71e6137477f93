// The batched pivoted LU of caller-provided blocks and of augmented condensation matrices.
#include "dgh_lu.hpp"
#include "dgh_kernels_lu2.cuh"

#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <utility>

namespace dgh {
namespace {
void ck(cudaError_t e, const char *what) {
    if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}
// The kernel's CTA width for block width m.
template <class F> void with_warps(int m, F &&f) {
    if (m < 4 || m > LU_MAX_WIDTH || m % 4 != 0) throw std::runtime_error("LU block width unsupported");
    switch (cr_warps(m)) {
        case 1: f(std::integral_constant<int, 1>{}); break;
        case 2: f(std::integral_constant<int, 2>{}); break;
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 5: f(std::integral_constant<int, 5>{}); break;
        case 7: f(std::integral_constant<int, 7>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        default: f(std::integral_constant<int, 16>{}); break;
    }
}
template <int NW, bool AUG> int resident(int m) {
    const size_t smem = cr_smem_bytes(m);
    allow_dynamic_smem((const void *)k_lu_crout<NW, AUG, 0>, smem);
    int per_sm = 0;
    ck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lu_crout<NW, AUG, 0>, 32 * NW, smem), "occupancy");
    return std::max(1, per_sm);
}
}  // namespace

void allow_dynamic_smem(const void *fn, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, size_t> cap;
    int dev = 0;
    ck(cudaGetDevice(&dev), "cudaGetDevice");
    std::lock_guard<std::mutex> lock(mu);
    size_t &cur = cap[{fn, dev}];
    if (bytes <= cur) return;
    ck(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes), "shared memory attribute");
    cur = bytes;
}

int lu_resident(int m, bool aug) {
    int r = 0;
    with_warps(m, [&](auto nw) {
        constexpr int NW = decltype(nw)::value;
        r = aug ? resident<NW, true>(m) : resident<NW, false>(m);
    });
    return r;
}
void lu_pool(const LuLaunch &l, double *pool, int m, int count, int *perm, bool slab_out, float *out32) {
    with_warps(m, [&](auto nw) {
        constexpr int NW = decltype(nw)::value;
        const int grid = std::min(count, l.sms * resident<NW, false>(m));
        k_lu_crout<NW, false, 0><<<grid, 32 * NW, cr_smem_bytes(m), l.stream>>>(
            pool, (size_t)m * m, m, m, 0, count, perm, l.status, l.bit, slab_out ? 1 : 0, out32, nullptr, nullptr, LLFuse());
    });
    ck(cudaGetLastError(), "LU launch");
}
void lu_augmented(const LuLaunch &l, double *aug, int m, int t, int count, int *perm, double *x, double *y) {
    with_warps(m, [&](auto nw) {
        constexpr int NW = decltype(nw)::value;
        const int ld = lu_aug_ld(m, t), grid = std::min(count, l.sms * resident<NW, true>(m));
        k_lu_crout<NW, true, 0><<<grid, 32 * NW, cr_smem_bytes(m), l.stream>>>(
            aug, (size_t)m * ld, m, ld, t, count, perm, l.status, l.bit, 0, nullptr, x, y, LLFuse());
    });
    ck(cudaGetLastError(), "LU launch");
}
}  // namespace dgh
