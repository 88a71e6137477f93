// The fused DG form of the batched LU: cell-block assembly, factorisation and the slab write of all
// cells in one persistent launch, one instantiation per degree.
#include "dgh_lu.hpp"
#include "dgh_kernels_lu2.cuh"

#include <stdexcept>
#include <string>

namespace dgh {
namespace {
template <class F> void with_nodes(int n, F &&f) {
    switch (n) {
        case 1: f(std::integral_constant<int, 1>{}); break;
        case 2: f(std::integral_constant<int, 2>{}); break;
        case 3: f(std::integral_constant<int, 3>{}); break;
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 5: f(std::integral_constant<int, 5>{}); break;
        case 6: f(std::integral_constant<int, 6>{}); break;
        case 7: f(std::integral_constant<int, 7>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 9: f(std::integral_constant<int, 9>{}); break;
        default: throw std::runtime_error("Unsupported face degree");
    }
}
}  // namespace

int lu_fused_resident(int n) {
    int per_sm = 0;
    with_nodes(n, [&](auto nn) {
        constexpr int N = decltype(nn)::value, M = NVAR * N * N, NW = cr_warps(M);
        const size_t smem = cr_smem_bytes(M);
        allow_dynamic_smem((const void *)k_lu_crout<NW, false, N>, smem);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lu_crout<NW, false, N>, 32 * NW, smem) != cudaSuccess)
            throw std::runtime_error("occupancy");
    });
    return std::max(1, per_sm);
}
void lu_fused(const LuLaunch &l, int n, const LLFuse &fu, int grid, int count, int *perm, float *out32) {
    with_nodes(n, [&](auto nn) {
        constexpr int N = decltype(nn)::value, M = NVAR * N * N, NW = cr_warps(M);
        const size_t smem = cr_smem_bytes(M);
        allow_dynamic_smem((const void *)k_lu_crout<NW, false, N>, smem);
        k_lu_crout<NW, false, N><<<grid, 32 * NW, smem, l.stream>>>(fu.slots, 0, M, M, 0, count, perm, l.status, l.bit, 0, out32,
                                                                    nullptr, nullptr, fu);
    });
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw std::runtime_error(std::string("LU launch: ") + cudaGetErrorString(e));
}
}  // namespace dgh
