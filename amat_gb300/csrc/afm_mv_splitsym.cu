// Patch kernels, ArithSplitSym instances (split arithmetic on packed symmetric
// units), and the kernel that packs those units from a split arena. The whole
// units are what bounds a split patch product; packed they take 55% of the
// bytes (n = 10), and the ring twice the units: tet10 Poisson 52^3 x 6 157 -> 124
// us a product, 80^3 x 6 598 -> 452 (4 groups of 2 warps in both).
#define ARITH ArithSplitSym
#define CONFIG_FN configure_kernels_splitsym
#define PATCH_FN launch_patches_splitsym
#define PATCH_SMEM_FN patch_smem_splitsym
#include "afm_mv_launch.inl"

namespace afm {

namespace {

// Patch units (32 element slots, entry (r, c) of slot l at (r n + c) 32 + l in
// each plane) -> packed upper triangle, entry k = j (j + 1) / 2 + i at k 32 +
// l in each plane. A thread moves 4 slots of an entry; a block packs units of
// its own, so the triangle is walked once per unit and no index is divided.
__global__ void __launch_bounds__(256) k_pack_split(const float4* __restrict__ src, float4* __restrict__ dst,
                                                    uint32_t n, uint32_t units) {
    const uint32_t np = n * (n + 1) / 2, full = n * n;
    const uint32_t q = threadIdx.x & 7, plane = (threadIdx.x >> 3) & 1, k0 = threadIdx.x >> 4;
    for (uint32_t u = blockIdx.x; u < units; u += gridDim.x) {
        const float4* s = src + ((size_t)u * 2 + plane) * full * 8 + q;
        float4* d = dst + ((size_t)u * 2 + plane) * np * 8 + q;
        uint32_t j = 0;
        for (uint32_t k = k0; k < np; k += 16) {
            while ((j + 1) * (j + 2) / 2 <= k) j++;
            d[k * 8] = s[((k - j * (j + 1) / 2) * n + j) * 8];
        }
    }
}

}  // namespace

// packed: 2 x n (n + 1) / 2 x 32 floats per unit.
cudaError_t pack_split_units(const unsigned char* ke, uint32_t n, uint32_t units, unsigned char* packed, int sm_count,
                             cudaStream_t st) {
    if (units == 0) return cudaSuccess;
    const uint32_t most = (uint32_t)sm_count * 8;
    k_pack_split<<<units < most ? units : most, 256, 0, st>>>(reinterpret_cast<const float4*>(ke),
                                                              reinterpret_cast<float4*>(packed), n, units);
    return cudaGetLastError();
}

}  // namespace afm
