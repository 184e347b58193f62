// Warp-group kernels, ArithSplitBlk instances (split arithmetic on symmetric
// element units of 2 x 2 blocks), and the kernel that packs those units from a
// split arena.
#define ARITH ArithSplitBlk
#define LAUNCH_FN launch_segment_splitblk
#define SMEM_FN segment_smem_splitblk
#define CONFIG_FN configure_kernels_splitblk
#define FUSED_FN launch_fused_splitblk
#include "afm_mv_launch.inl"

namespace afm {

namespace {

constexpr uint32_t kPackThreads = 128;

// Element units (column-major, hi plane, lo plane `plane` entries on) -> the
// units of split_block_terms. A block packs units of its own in two passes over
// each, the largest difference K(c, r) - K(r, c) first; once per finalize, so
// the unit is simply read again (from L1 and L2).
__global__ void __launch_bounds__(kPackThreads) k_pack_blocks(const unsigned char* __restrict__ ke, uint64_t unit_bytes,
                                                              uint32_t plane, unsigned char* __restrict__ dst, uint32_t n,
                                                              uint32_t units) {
    __shared__ double smax[kPackThreads];
    const uint32_t nb = n / 2, cells = (nb / 2 + 1) * nb;
    for (uint32_t u = blockIdx.x; u < units; u += gridDim.x) {
        const float* s = reinterpret_cast<const float*>(ke + (size_t)u * unit_bytes);
        unsigned char* out = dst + (size_t)u * split_block_bytes(n);
        auto diff = [&](uint32_t r, uint32_t c) {
            const uint32_t x = c * n + r, y = r * n + c;
            return ((double)s[y] - (double)s[x]) + ((double)s[y + plane] - (double)s[x + plane]);
        };
        double most = 0.0;
        for (uint32_t t = threadIdx.x; t < cells; t += kPackThreads) {
            const uint32_t i = t % nb, j = (i + t / nb) % nb;
            for (uint32_t e = 0; e < 4; e++) most = fmax(most, fabs(diff(2 * i + (e >> 1), 2 * j + (e & 1))));
        }
        smax[threadIdx.x] = most;
        __syncthreads();
        for (uint32_t w = kPackThreads / 2; w; w /= 2) {
            if (threadIdx.x < w) smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + w]);
            __syncthreads();
        }
        most = smax[0];
        __syncthreads();
        // the smallest power of two that fits the differences into [-127, 127] (FP32, as the lo entries are)
        int ex = 0;
        frexp(most / 127.0, &ex);
        const double step = most > 0.0 ? ldexp(1.0, max(ex, -149)) : 0.0;
        for (uint32_t t = threadIdx.x; t < cells; t += kPackThreads) {
            const uint32_t i = t % nb, j = (i + t / nb) % nb;
            float h[4], l[4];
            uint32_t d = 0;
            for (uint32_t e = 0; e < 4; e++) {
                const uint32_t r = 2 * i + (e >> 1), c = 2 * j + (e & 1);
                h[e] = s[c * n + r];
                l[e] = s[c * n + r + plane];
                const int b = step > 0.0 ? (int)rint(diff(r, c) / step) : 0;
                d |= (uint32_t)(b + 128) << (8 * e);
            }
            reinterpret_cast<float4*>(out)[t] = make_float4(h[0], h[1], h[2], h[3]);
            reinterpret_cast<float4*>(out)[cells + t] = make_float4(l[0], l[1], l[2], l[3]);
            reinterpret_cast<uint32_t*>(out + (size_t)cells * 32)[t] = d;
        }
        if (threadIdx.x == 0)
            *reinterpret_cast<float4*>(out + (size_t)cells * 36) = make_float4((float)step, 0.0f, 0.0f, 0.0f);
    }
}

}  // namespace

cudaError_t pack_split_blocks(const unsigned char* ke, uint64_t unit_bytes, uint32_t plane, uint32_t n, uint32_t units,
                              unsigned char* dst, int sm_count, cudaStream_t st) {
    if (units == 0) return cudaSuccess;
    if (!split_block_bytes(n)) return cudaErrorInvalidValue;
    const uint32_t most = (uint32_t)sm_count * 16;
    k_pack_blocks<<<units < most ? units : most, kPackThreads, 0, st>>>(ke, unit_bytes, plane, dst, n, units);
    return cudaGetLastError();
}

}  // namespace afm
