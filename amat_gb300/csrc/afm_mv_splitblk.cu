// Warp-group kernels, ArithSplitBlk instances (split arithmetic on symmetric
// element units of 2 x 2 blocks), and the kernel that packs those units from a
// split arena.
#define ARITH ArithSplitBlk
#define LAUNCH_FN launch_segment_splitblk
#define CONFIG_FN configure_kernels_splitblk
#define FUSED_FN launch_fused_splitblk
#include "afm_mv_launch.inl"

namespace afm {

namespace {

constexpr uint32_t kPackThreads = 128;

// Element units (column-major, hi plane, lo plane `plane` entries on) -> the
// units of split_block_terms. Once per finalize.
__global__ void __launch_bounds__(kPackThreads) k_pack_blocks(const unsigned char* __restrict__ ke, uint64_t unit_bytes,
                                                              uint32_t plane, unsigned char* __restrict__ dst, uint32_t n,
                                                              uint32_t units) {
    const uint32_t nb = n / 2, nd = nb / 2 + 1, cells = nd * nb;
    for (uint32_t u = blockIdx.x; u < units; u += gridDim.x) {
        const float* s = reinterpret_cast<const float*>(ke + (size_t)u * unit_bytes);
        float4* out = reinterpret_cast<float4*>(dst + (size_t)u * split_block_bytes(n));
        for (uint32_t t = threadIdx.x; t < cells; t += kPackThreads) {
            const uint32_t i = t % nb, d = t / nb, j = (i + d) % nb;
            float h[4], l[4], x[4];
            for (uint32_t e = 0; e < 4; e++) {
                const uint32_t r = 2 * i + (e >> 1), c = 2 * j + (e & 1);
                h[e] = s[c * n + r];
                l[e] = s[c * n + r + plane];
                const float th = s[r * n + c], tl = s[r * n + c + plane];
                x[e] = split_transposed(h[e], th, tl);
                if (d != 0 && d + 1 != nd && !block_holds(h[e], th, tl)) h[e] = l[e] = x[e] = 0.0f;
            }
            out[t] = make_float4(h[0], h[1], h[2], h[3]);
            out[cells + t] = make_float4(l[0], l[1], l[2], l[3]);
            if (d != 0 && d + 1 != nd) out[2 * cells + t - nb] = make_float4(x[0], x[1], x[2], x[3]);
        }
    }
}

__global__ void __launch_bounds__(kPackThreads) k_add_pairs(double* v, const double* __restrict__ u,
                                                            const uint32_t* __restrict__ row,
                                                            const uint32_t* __restrict__ off,
                                                            const uint32_t* __restrict__ col,
                                                            const double* __restrict__ val, uint32_t rows, int bc_mode) {
    const uint32_t i = blockIdx.x * kPackThreads + threadIdx.x;
    if (i >= rows) return;
    double s = 0.0;
    for (uint32_t k = off[i]; k < off[i + 1]; k++)
        if (!(bc_mode && (col[k] & kBcFlag))) s = __fma_rn(val[k], u[col[k] & kDofMask], s);
    v[row[i]] += s;
}

}  // namespace

cudaError_t launch_add_pairs(double* v, const double* u, const uint32_t* row, const uint32_t* off, const uint32_t* col,
                             const double* val, uint32_t rows, int bc_mode, cudaStream_t st) {
    if (rows == 0) return cudaSuccess;
    k_add_pairs<<<(rows + kPackThreads - 1) / kPackThreads, kPackThreads, 0, st>>>(v, u, row, off, col, val, rows, bc_mode);
    return cudaGetLastError();
}

cudaError_t pack_split_blocks(const unsigned char* ke, uint64_t unit_bytes, uint32_t plane, uint32_t n, uint32_t units,
                              unsigned char* dst, int sm_count, cudaStream_t st) {
    if (units == 0) return cudaSuccess;
    if (!split_block_bytes(n)) return cudaErrorInvalidValue;
    const uint32_t most = (uint32_t)sm_count * 16;
    k_pack_blocks<<<units < most ? units : most, kPackThreads, 0, st>>>(ke, unit_bytes, plane, dst, n, units);
    return cudaGetLastError();
}

}  // namespace afm
