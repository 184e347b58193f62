// Vector kernels around the AFM matvec: boundary-condition wrapping of
// MatMult_mf and the Jacobi-preconditioned CG of the example drivers' solve
// (examples/include/solve.hpp:75-127). Vectors are T = double (the FP64 CG)
// or T = float (the inner CG of the mixed-precision solve); every dot product
// and step scalar is accumulated and held in FP64.
//
// Reductions are deterministic: a grid of nb = red_blocks(n) x kRedThreads
// threads sums fixed strided slices in index order, each block reduces in a
// fixed tree, and one block reduces the nb partials in a fixed tree. The
// result depends only on n, never on the device or on timing. (nb grows with
// n up to kRedBlocks, so a small solve occupies few SMs.)
#include <cuda_runtime.h>
#include <stdint.h>

#include "afm_solver.hpp"
#include "afm_internal.hpp"

namespace afm {

namespace {

// Sum over the block in a fixed tree: shuffles within each warp, then over
// the warps' sums (sh holds at least 33 doubles).
__device__ __forceinline__ double block_sum(double x, double* sh) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        double r = lane < kRedThreads / 32 ? sh[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
        if (lane == 0) sh[32] = r;
    }
    __syncthreads();
    const double r = sh[32];
    __syncthreads();
    return r;
}

__device__ __forceinline__ double final_sum(const double* part, double* sh, uint32_t nb) {
    double s = 0.0;
    for (uint32_t i = threadIdx.x; i < nb; i += kRedThreads) s += part[i];
    return block_sum(s, sh);
}

// The FP64 pipe takes 16 cycles per warp instruction, so in the small launches
// of a CG iteration the count of FP64 instructions per block is the time: a
// sum over the block goes through shared memory to one warp (12 FP64 adds
// instead of 43 with a shuffle tree in each warp), and one warp does what the
// whole block needs once (a division, a square root).

// Sum over the warp's lanes, in every lane.
__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// part[k * kRedBlocks + block] = the sums over the block of x[k], k < K. sh: K x kRedThreads.
template <int K>
__device__ __forceinline__ void block_partials(const double (&x)[K], double* sh, double* part) {
#pragma unroll
    for (int k = 0; k < K; k++) sh[k * kRedThreads + threadIdx.x] = x[k];
    __syncthreads();
    const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
    if (k >= K) return;
    double a[kRedThreads / 32];
#pragma unroll
    for (int i = 0; i < kRedThreads / 32; i++) a[i] = sh[k * kRedThreads + 32 * i + lane];
#pragma unroll
    for (int o = kRedThreads / 64; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; i++) a[i] += a[i + o];
    const double s = warp_sum(a[0]);
    if (lane == 0) part[k * kRedBlocks + blockIdx.x] = s;
}

// A warp's sum of nb partials, in every lane.
__device__ __forceinline__ double row_sum(const double* part, uint32_t nb) {
    double s = 0.0;
    for (uint32_t i = threadIdx.x & 31; i < nb; i += 32) s += part[i];
    return warp_sum(s);
}

#define kStride ((size_t)gridDim.x * kRedThreads)

// Dot-product accumulators of one thread. FP64 vectors: FP64 fused
// multiply-adds. FP32 vectors: compensated FP32 arithmetic (Ogita, Rump &
// Oishi, "Accurate sum and dot product", 2005, Dot2: TwoProduct by FMA and
// TwoSum, about twice FP32 precision per thread), which keeps the FP32
// recursion off GB300's FP64 pipe (1/64 of the FP32 rate). The _rn intrinsics
// keep the compiler from fusing the steps.
template <typename T>
struct DotAcc;
template <>
struct DotAcc<double> {
    double s = 0.0;
    __device__ __forceinline__ void add(double x, double y) { s = __fma_rn(x, y, s); }
    __device__ __forceinline__ double value() const { return s; }
};
template <>
struct DotAcc<float> {
    float hi = 0.0f, lo = 0.0f;
    __device__ __forceinline__ void add(float x, float y) {
        const float p = __fmul_rn(x, y);
        const float e = __fmaf_rn(x, y, -p);
        const float t = __fadd_rn(hi, p);
        const float bp = __fsub_rn(t, hi);
        const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(t, bp)), __fsub_rn(p, bp));
        hi = t;
        lo = __fadd_rn(lo, __fadd_rn(err, e));
    }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// Strided loops visit i = i0, i0 + stride, ... in index order; kUnroll of
// them load before any is used, so that each thread keeps several memory
// requests in flight (the order of every sum is unchanged).
constexpr int kUnroll = 4;



template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_set_constrained(T* v, const T* u, const uint32_t* idx, uint32_t n) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) v[idx[k]] = u[idx[k]];
}

// part[block]: partial sums of a.b
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_dot(const T* a, const T* b, size_t n, double* part) {
    __shared__ double sh[kRedThreads];
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    DotAcc<T> ab;
    size_t i = (size_t)blockIdx.x * kRedThreads + threadIdx.x;
    for (; i + (kUnroll - 1) * kStride < n; i += kUnroll * kStride) {
        T x[kUnroll], y[kUnroll];
#pragma unroll
        for (int q = 0; q < kUnroll; q++) {
            x[q] = a[i + q * kStride];
            y[q] = b[i + q * kStride];
        }
#pragma unroll
        for (int q = 0; q < kUnroll; q++) ab.add(x[q], y[q]);
    }
    for (; i < n; i += kStride) ab.add(a[i], b[i]);
    const double v[1] = {ab.value()};
    block_partials(v, sh, part);
}

// r = b - q (r may be q), with the partials of r.r: one pass where a copy, an update and a dot product were three. A
// mixed solve is bound by launches and host turns between its segments; with this, the update of the recursion in two
// launches and a segment's first batch enqueued with it, hex8 Poisson 24^3 (69 iterations, 11 segments) went from 2605
// to 2290 us.
__global__ void __launch_bounds__(kRedThreads) k_residual(double* r, const double* b, const double* q, size_t n,
                                                          double* part) {
    __shared__ double sh[kRedThreads];
    DotAcc<double> rr;
    for (size_t i = (size_t)blockIdx.x * kRedThreads + threadIdx.x; i < n; i += kUnroll * kStride) {
        double x[kUnroll], y[kUnroll];
#pragma unroll
        for (int k = 0; k < kUnroll; k++) {
            const size_t j = i + k * kStride;
            if (j < n) x[k] = b[j], y[k] = q[j];
        }
#pragma unroll
        for (int k = 0; k < kUnroll; k++) {
            const size_t j = i + k * kStride;
            if (j < n) {
                const double t = x[k] - y[k];
                r[j] = t;
                rr.add(t, t);
            }
        }
    }
    const double v[1] = {rr.value()};
    block_partials(v, sh, part);
}

// r = b - q, z = dinv r, p = z; partials of r.z, r.r, z.z, b.b, (dinv b).(dinv b)
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_cg_init(const T* __restrict__ b, const T* __restrict__ q,
                                                         const T* __restrict__ dinv, T* __restrict__ r,
                                                         T* __restrict__ z, T* __restrict__ p, size_t n, double* part) {
    __shared__ double sh[kRedThreads];
    double rz = 0, rr = 0, zz = 0, bb = 0, db = 0;
    for (size_t i = (size_t)blockIdx.x * kRedThreads + threadIdx.x; i < n; i += kStride) {
        const T bi = b[i], di = dinv[i];
        const T ri = bi - q[i];
        const T zi = di * ri;
        r[i] = ri;
        z[i] = zi;
        p[i] = zi;
        rz = __fma_rn((double)ri, (double)zi, rz);
        rr = __fma_rn((double)ri, (double)ri, rr);
        zz = __fma_rn((double)zi, (double)zi, zz);
        bb = __fma_rn((double)bi, (double)bi, bb);
        const double t = (double)di * (double)bi;
        db = __fma_rn(t, t, db);
    }
    double v[5] = {rz, rr, zz, bb, db};
    for (int j = 0; j < 5; j++) {
        const double s = block_sum(v[j], sh);
        if (threadIdx.x == 0) part[j * kRedBlocks + blockIdx.x] = s;
    }
}

__global__ void __launch_bounds__(kRedThreads) k_cg_init_final(double* sc, const double* part, uint32_t nb) {
    __shared__ double sh[kRedThreads];
    const double rz = final_sum(part, sh, nb);
    const double rr = final_sum(part + kRedBlocks, sh, nb);
    const double zz = final_sum(part + 2 * kRedBlocks, sh, nb);
    const double bb = final_sum(part + 3 * kRedBlocks, sh, nb);
    const double db = final_sum(part + 4 * kRedBlocks, sh, nb);
    if (threadIdx.x == 0) {
        sc[S_RZ] = rz;
        sc[S_RR] = rr;
        sc[S_ZZ] = zz;
        sc[S_BB] = bb;
        sc[S_DB] = db;
        const bool bad = rz < 0.0 || rz != rz;
        sc[S_FLAG] = bad ? 1.0 : 0.0;
        sc[S_DONE] = bad ? 1.0 : 0.0;
        sc[S_ITER] = 0.0;
    }
}

// Launches of one CG iteration follow one another with programmatic
// dependence: each waits for the one before it in full, but is on the SMs by
// then. What a launch before may write is read with plain loads (no
// __restrict__ const pointers, no ld.global.nc, whose lines may have been in
// L1 since before the write).
__device__ __forceinline__ void wait_launch() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release_next() { asm volatile("griddepcontrol.launch_dependents;"); }

// Reliable update of the FP32 recursion of the mixed-precision solve, pass 1:
// r = fl32(sigma r64) (the FP64 true residual in the new segment's scale),
// z = dinv r; partials of r.z, r.r, z.z and r.p (p = the last direction p_k,
// still in the previous segment's scale)
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_cg_reliable(const double* __restrict__ r64, T* __restrict__ r,
                                                             T* __restrict__ z, const T* __restrict__ p,
                                                             const T* __restrict__ dinv, size_t n, double* part,
                                                             double sigma) {
    __shared__ double sh[4 * kRedThreads];
    release_next();
    double rz = 0, rr = 0, zz = 0, rp = 0;
    for (size_t i = (size_t)blockIdx.x * kRedThreads + threadIdx.x; i < n; i += kStride) {
        const T ri = (T)(r64[i] * sigma);
        const T zi = dinv[i] * ri;
        r[i] = ri;
        z[i] = zi;
        rz = __fma_rn((double)ri, (double)zi, rz);
        rr = __fma_rn((double)ri, (double)ri, rr);
        zz = __fma_rn((double)zi, (double)zi, zz);
        rp = __fma_rn((double)ri, (double)p[i], rp);
    }
    const double v[4] = {rz, rr, zz, rp};
    block_partials(v, sh, part);
}

__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// pass 2: beta = r.z / (rho r_k.z_k), gamma = r.p / r.z (every block adds up
// the partials; the first writes the scalars and clears S_DONE, or sets it on
// breakdown, and S_ITER), p = z + beta (p - gamma z). rho = sigma_new /
// sigma_old, the change of the residual's scale: with r, z in the new scale and
// p, r_k.z_k in the old one this is the scaled form of the unscaled update.
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_cg_reliable_p(T* p, const T* z, size_t n, double* sc,
                                                               const double* part, uint32_t nb, double rho) {
    __shared__ double sums[4];
    __shared__ double coef[2];
    wait_launch();
    const uint32_t t = threadIdx.x;
    if (t < 128) {
        const double s = row_sum(part + (t >> 5) * kRedBlocks, nb);
        if ((t & 31) == 0) sums[t >> 5] = s;
    }
    __syncthreads();
    if (t == 0) {
        const double rz = sums[0], old = sc[S_RZOLD];
        const bool bad = rz < 0.0 || rz != rz;
        const double beta = (!bad && old > 0.0) ? rz / (old * rho) : 0.0;
        const double gamma = (!bad && rz > 0.0) ? sums[3] / rz : 0.0;
        coef[0] = beta;
        coef[1] = 1.0 - beta * gamma;
        if (blockIdx.x == 0) {
            sc[S_BETA] = beta;
            sc[S_GAMMA] = gamma;
            sc[S_RZ] = rz;
            sc[S_RR] = sums[1];
            sc[S_ZZ] = sums[2];
            sc[S_FLAG] = bad ? 1.0 : 0.0;
            sc[S_DONE] = bad ? 1.0 : 0.0;
            sc[S_ITER] = 0.0;
        }
    }
    __syncthreads();
    const T beta = (T)coef[0], c = (T)coef[1];
    for (size_t i = (size_t)blockIdx.x * kRedThreads + t; i < n; i += kStride) p[i] = fma_rn(beta, p[i], c * z[i]);
}

// sc[S_PQ] = sum of the partials (a plain reduction, no CG bookkeeping; one warp)
__global__ void k_sum(double* sc, const double* part, uint32_t nb) {
    const double s = row_sum(part, nb);
    if (threadIdx.x == 0) sc[S_PQ] = s;
}

// First half of an iteration: alpha = r.z / p.q (every block adds up the
// partials of p.q itself), x += alpha p, r -= alpha q; partials of r.z, r.r,
// z.z, z = dinv r. A solve that is done, or breaks down here (p.q <= 0 or NaN:
// out[S_BREAK]), changes nothing. A one-block launch for alpha (and one for
// beta) cost as much as the vector work up to 10^5 DoFs: the FP64 CG of hex8
// Poisson 32^3 took 4.10 ms with them, 2.49 ms without.
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_cg_xr(T* x, T* r, const T* p, const T* q, const T* dinv, size_t n,
                                                       const double* in, double* out, const double* part_pq,
                                                       uint32_t nb_pq, double* part) {
    __shared__ double sh[3 * kRedThreads];
    __shared__ double shared_alpha;
    __shared__ bool shared_bad;
    release_next();
    wait_launch();
    if (in[S_DONE] != 0.0) return;
    if (threadIdx.x < 32) {
        const double pq = row_sum(part_pq, nb_pq);
        const bool bad = !(pq > 0.0);
        const double a = in[S_RZ] / pq;
        if (threadIdx.x == 0) {
            shared_alpha = a;
            shared_bad = bad;
            if (blockIdx.x == 0) {
                out[S_PQ] = pq;
                out[S_ALPHA] = bad ? 0.0 : a;
                out[S_BREAK] = bad ? 1.0 : 0.0;
            }
        }
    }
    // the first entries load while the first warp finds alpha
    T xv[kUnroll], pv[kUnroll], qv[kUnroll], rv[kUnroll], dv[kUnroll];
    auto load = [&](size_t i0) {
#pragma unroll
        for (int k = 0; k < kUnroll; k++) {
            const size_t j = i0 + k * kStride;
            if (j < n) xv[k] = x[j], pv[k] = p[j], qv[k] = q[j], rv[k] = r[j], dv[k] = dinv[j];
        }
    };
    size_t i = (size_t)blockIdx.x * kRedThreads + threadIdx.x;
    load(i);
    __syncthreads();
    if (shared_bad) return;
    const T alpha = (T)shared_alpha;
    DotAcc<T> rz, rr, zz;
    for (; i < n; i += kUnroll * kStride, load(i)) {
#pragma unroll
        for (int k = 0; k < kUnroll; k++) {
            const size_t j = i + k * kStride;
            if (j < n) {
                x[j] = alpha * pv[k] + xv[k];
                const T ri = -alpha * qv[k] + rv[k];
                const T zi = dv[k] * ri;
                r[j] = ri;
                rz.add(ri, zi);
                rr.add(ri, ri);
                zz.add(zi, zi);
            }
        }
    }
    const double v[3] = {rz.value(), rr.value(), zz.value()};
    block_partials(v, sh, part);
}

// Second half: beta = r.z / (the previous r.z), the stopping test, p = dinv r +
// beta p. Block 0 writes the new scalars. A finished solve keeps its last
// direction (the mixed-precision solve continues from it after a reliable
// update).
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_cg_p(T* p, const T* r, const T* dinv, size_t n, const double* in,
                                                      double* out, const double* part, uint32_t nb) {
    __shared__ double sums[3];
    __shared__ double shared_beta;
    __shared__ int shared_done;  // 1: done, 2: broke down
    release_next();
    wait_launch();
    const uint32_t t = threadIdx.x;
    const bool lead = blockIdx.x == 0;
    if (in[S_DONE] != 0.0) {
        if (lead && t < kScalarSlots) out[t] = in[t];
        return;
    }
    if (out[S_BREAK] != 0.0) {  // (written by the first half)
        if (lead && t < kScalarSlots && t != S_PQ && t != S_BREAK)
            out[t] = t == S_FLAG || t == S_DONE ? 1.0 : t == S_ALPHA || t == S_BETA ? 0.0 : in[t];
        return;
    }
    const double it = in[S_ITER] + 1.0;
    if (t < 96) {
        const double s = row_sum(part + (t >> 5) * kRedBlocks, nb);
        if ((t & 31) == 0) sums[t >> 5] = s;
    }
    // the first entries load while the first warps find beta
    T pv[kUnroll], rv[kUnroll], dv[kUnroll];
    auto load = [&](size_t i0) {
#pragma unroll
        for (int k = 0; k < kUnroll; k++) {
            const size_t j = i0 + k * kStride;
            if (j < n) pv[k] = p[j], rv[k] = r[j], dv[k] = dinv[j];
        }
    };
    size_t i = (size_t)blockIdx.x * kRedThreads + t;
    load(i);
    __syncthreads();
    if (t < 32) {
        const double rz = sums[0], old = in[S_RZ];
        if (t == 0) shared_beta = old != 0.0 ? rz / old : 0.0;
    } else if (t < 64) {
        const double rz = sums[0], nrm = sqrt(in[S_NORM] != 0.0 ? sums[2] : sums[1]);
        const bool bad = rz < 0.0 || rz != rz || nrm != nrm;
        const bool done = nrm <= in[S_TOL] || (in[S_MAXIT] > 0.0 && it >= in[S_MAXIT]);
        if (t == 32) shared_done = bad ? 2 : done ? 1 : 0;
    }
    __syncthreads();
    const int done = shared_done;
    if (lead && t < kScalarSlots && t != S_PQ && t != S_ALPHA && t != S_BREAK) {
        double y = in[t];
        if (t == S_RZ) y = sums[0];
        if (t == S_RZOLD) y = in[S_RZ];
        if (t == S_RR) y = sums[1];
        if (t == S_ZZ) y = sums[2];
        if (t == S_BETA) y = shared_beta;
        if (t == S_ITER) y = it;
        if (t == S_FLAG && done == 2) y = 1.0;
        if (t == S_DONE && done) y = 1.0;
        out[t] = y;
    }
    if (done) return;
    const T beta = (T)shared_beta;
    for (; i < n; i += kUnroll * kStride, load(i)) {
#pragma unroll
        for (int k = 0; k < kUnroll; k++) {
            const size_t j = i + k * kStride;
            const T zi = dv[k] * rv[k];
            if (j < n) p[j] = beta * pv[k] + zi;
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_invert(T* __restrict__ dinv, const double* __restrict__ d,
                                                        size_t n) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) dinv[i] = (T)(1.0 / d[i]);
}

__global__ void __launch_bounds__(kRedThreads) k_axpby(double* __restrict__ y, const double* __restrict__ x,
                                                       double a, double b, size_t n) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        y[i] = __fma_rn(a, x[i], b * y[i]);
}

// out = (T)(scale in64) (scale a power of two: exact before the rounding)
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_to_f32(T* __restrict__ out, const double* __restrict__ in,
                                                        size_t n, double scale) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = (T)(in[i] * scale);
}

// x64 += inv d, d = 0 (inv a power of two)
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_add_f32(double* __restrict__ x, T* __restrict__ d, size_t n,
                                                         double inv) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        x[i] += (double)d[i] * inv;
        d[i] = (T)0;
    }
}

// |x| as the bits of a non-negative double: ordered like the values, with
// NaN above infinity, so that an integer max propagates both.
__device__ __forceinline__ unsigned long long abs_bits(double x) {
    return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}

__device__ __forceinline__ unsigned long long warp_max(unsigned long long m) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y = __shfl_down_sync(0xffffffffu, m, o);
        m = y > m ? y : m;
    }
    return m;
}

// w[0] = max |u[i]| over the DoFs not masked (mask[i] != 0: a constrained DoF
// that the product reads as zero), as double bits; vz[0 .. nv) = 0 on the way.
// The grid's blocks leave their maxima in w[2 + block]; the last block to
// finish (counted in the low word of w[1]) reduces them, writes w[0] and
// resets the counter, so one launch does it all and repeats cleanly inside a
// captured graph. The maximum is exact, hence independent of the order.
__global__ void __launch_bounds__(kRedThreads) k_umax(const double* u, const uint8_t* mask,
                                                      size_t n, double* vz, size_t nv,
                                                      unsigned long long* w) {
    __shared__ unsigned long long sh[kRedThreads / 32];
    __shared__ bool last;
    release_next();
    wait_launch();
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long m = 0;
    for (size_t i = i0; i < n; i += stride) {
        const unsigned long long b = abs_bits(u[i]);
        if ((!mask || !mask[i]) && b > m) m = b;
    }
    if (vz)
        for (size_t i = i0; i < nv; i += stride) vz[i] = 0.0;
    m = warp_max(m);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long bm = 0;
        for (int k = 0; k < kRedThreads / 32; k++) bm = sh[k] > bm ? sh[k] : bm;
        w[2 + blockIdx.x] = bm;
        __threadfence();
        const unsigned prev = atomicAdd(reinterpret_cast<unsigned*>(w + 1), 1u);
        last = (prev == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    unsigned long long r = 0;
    for (uint32_t k = threadIdx.x; k < gridDim.x; k += blockDim.x) {
        const unsigned long long b = __ldcg(w + 2 + k);
        r = b > r ? b : r;
    }
    r = warp_max(r);
    if (lane == 0) sh[wid] = r;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long bm = 0;
        for (int k = 0; k < kRedThreads / 32; k++) bm = sh[k] > bm ? sh[k] : bm;
        w[0] = bm;
        *reinterpret_cast<unsigned*>(w + 1) = 0u;
    }
}

// cm[j] = max over the unmasked rows i of |U[i ld + j]|, j < R (double bits;
// cm zeroed before the launch; R even, rows 16-byte aligned). A thread keeps
// the maxima of two columns over its rows, four rows in flight; per block they
// meet in shared memory, then one global atomic max per column. (An atomic per
// entry took 24 us for 46800 x 32, this 8.)
__global__ void __launch_bounds__(kRedThreads) k_umax_cols(const double* __restrict__ U, const uint8_t* __restrict__ mask,
                                                           size_t rows, uint32_t R, uint32_t ld,
                                                           unsigned long long* __restrict__ cm) {
    __shared__ unsigned long long sm[kMaxUmaxCols];
    for (uint32_t j = threadIdx.x; j < R; j += blockDim.x) sm[j] = 0;
    __syncthreads();
    const uint32_t cpr = R / 2, per = kRedThreads / cpr;  // threads of a row, rows of a pass
    const uint32_t k = threadIdx.x % cpr, r0 = threadIdx.x / cpr;
    unsigned long long m0 = 0, m1 = 0;
    if (r0 < per) {
        const size_t stride = (size_t)gridDim.x * per;
        for (size_t i = (size_t)blockIdx.x * per + r0; i < rows; i += kUnroll * stride) {
            double2 x[kUnroll];
#pragma unroll
            for (int q = 0; q < kUnroll; q++) {
                const size_t r = i + q * stride;
                x[q] = make_double2(0.0, 0.0);
                if (r < rows && !(mask && mask[r])) x[q] = *reinterpret_cast<const double2*>(U + r * ld + 2 * k);
            }
#pragma unroll
            for (int q = 0; q < kUnroll; q++) {
                const unsigned long long a = abs_bits(x[q].x), b = abs_bits(x[q].y);
                m0 = a > m0 ? a : m0;
                m1 = b > m1 ? b : m1;
            }
        }
        if (m0) atomicMax(sm + 2 * k, m0);
        if (m1) atomicMax(sm + 2 * k + 1, m1);
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < R; j += blockDim.x)
        if (sm[j]) atomicMax(cm + j, sm[j]);
}

// Combine pass of one-launch patches: v[dof[i]] = the entries of shared DoF
// i in the combine buffer, summed in patch order (the first entry, then each
// next one added), one thread per shared DoF. Waits for the patch launch
// (programmatic dependence) before reading.
template <typename VO>
__global__ void __launch_bounds__(kRedThreads) k_patch_combine(VO* v, const VO* pv,
                                                               const uint32_t* dof,
                                                               const uint32_t* off,
                                                               const uint32_t* idx, uint32_t nb,
                                                               const VO* u_rows) {
    wait_launch();
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += stride) {
        const uint32_t d = dof[i] & kDofMask;
        if (u_rows && (dof[i] & kBcFlag)) {
            v[d] = u_rows[d];
            continue;
        }
        const uint32_t k0 = off[i], k1 = off[i + 1];
        VO s = pv[idx[k0]];
        for (uint32_t k = k0 + 1; k < k1; k++) s += pv[idx[k]];
        v[d] = s;
    }
}

// The same over every DoF, with the partials of v.u: pos[d] = the DoF's place
// in the combine lists, or kNoElement (v[d] is there already).
template <typename VO>
__global__ void __launch_bounds__(kRedThreads) k_patch_combine_dot(VO* v, const VO* pv,
                                                                   const uint32_t* pos,
                                                                   const uint32_t* dof,
                                                                   const uint32_t* off,
                                                                   const uint32_t* idx, uint32_t n,
                                                                   const VO* u, double* part) {
    __shared__ double sh[kRedThreads];
    release_next();
    DotAcc<VO> acc;
    const uint32_t stride = gridDim.x * kRedThreads;
    bool waited = false;
    for (uint32_t d = blockIdx.x * kRedThreads + threadIdx.x; d < n; d += stride) {
        const uint32_t i = __ldg(pos + d);
        const bool sum = i != kNoElement;
        const bool fixed = sum && (__ldg(dof + i) & kBcFlag) != 0;
        const uint32_t k0 = sum ? __ldg(off + i) : 0u, k1 = sum ? __ldg(off + i + 1) : 0u;
        if (!waited) {
            wait_launch();
            waited = true;
        }
        const VO ud = u[d];
        VO s;
        if (!sum) {
            s = v[d];
        } else {
            s = fixed ? ud : pv[idx[k0]];
            if (!fixed)
                for (uint32_t k = k0 + 1; k < k1; k++) s += pv[idx[k]];
            v[d] = s;
        }
        acc.add(s, ud);
    }
    if (!waited) wait_launch();
    const double t[1] = {acc.value()};
    block_partials(t, sh, part);
}

// Gather pass of a plan whose elements run in one launch (launch_gather_sum):
// one thread per DoF; lists and mask are constant, so they load before the
// wait for the element launch. DOT: the partials of v.u too, kRedBlocks blocks
// at most.
template <typename VO, typename VT, uint32_t B, bool DOT>
__global__ void __launch_bounds__(kRedThreads) k_gather_sum(VT* v, const VO* ve,
                                                            const uint32_t* off,
                                                            const uint32_t* idx, uint32_t n,
                                                            const VT* u, const uint8_t* mask,
                                                            double* part) {
    constexpr int kAhead = 8;  // entries in flight per thread
    __shared__ double sh[DOT ? kRedThreads : 1];
    if constexpr (DOT) release_next();
    DotAcc<VT> acc;
    bool waited = false;
    for (uint32_t d = blockIdx.x * kRedThreads + threadIdx.x; d < n; d += gridDim.x * kRedThreads) {
        const uint32_t m = d / B, c = d - m * B;
        const uint32_t k0 = __ldg(off + m), k1 = __ldg(off + m + 1);
        const bool fixed = mask && mask[d];
        uint32_t at[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; q++) at[q] = k0 + q < k1 ? __ldg(idx + k0 + q) : 0u;
        if (!waited) {
            wait_launch();
            waited = true;
        }
        VT ud = VT(0);
        if (DOT || fixed) ud = u[d];
        VO s = VO(0);
        if (!fixed) {
            VO x[kAhead];
#pragma unroll
            for (int q = 0; q < kAhead; q++) x[q] = k0 + q < k1 ? __ldcg(ve + at[q] + c) : VO(0);
#pragma unroll
            for (int q = 0; q < kAhead; q++)
                if (k0 + q < k1) s += x[q];
            for (uint32_t k = k0 + kAhead; k < k1; k += kAhead) {
#pragma unroll
                for (int q = 0; q < kAhead; q++) at[q] = k + q < k1 ? __ldg(idx + k + q) : 0u;
#pragma unroll
                for (int q = 0; q < kAhead; q++) x[q] = k + q < k1 ? __ldcg(ve + at[q] + c) : VO(0);
#pragma unroll
                for (int q = 0; q < kAhead; q++)
                    if (k + q < k1) s += x[q];
            }
        }
        const VT out = fixed ? ud : (VT)s;
        v[d] = out;
        if constexpr (DOT) acc.add(out, ud);
    }
    if (!waited) wait_launch();
    if constexpr (DOT) {
        const double t[1] = {acc.value()};
        block_partials(t, sh, part);
    }
}

inline unsigned grid_for(size_t n) {
    size_t g = (n + kRedThreads - 1) / kRedThreads;
    if (g > 4096) g = 4096;
    if (g == 0) g = 1;
    return (unsigned)g;
}

}  // namespace

template <typename T>
cudaError_t launch_set_constrained(T* v, const T* u, const uint32_t* idx, uint32_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_set_constrained<T><<<(n + kRedThreads - 1) / kRedThreads, kRedThreads, 0, st>>>(v, u, idx, n);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_cg_init(const T* b, const T* q, const T* dinv, T* r, T* z, T* p, size_t n, double* sc,
                           double* part, cudaStream_t st) {
    const uint32_t nb = red_blocks(n);
    k_cg_init<T><<<nb, kRedThreads, 0, st>>>(b, q, dinv, r, z, p, n, part);
    k_cg_init_final<<<1, kRedThreads, 0, st>>>(sc, part, nb);
    return cudaGetLastError();
}

namespace {
// A launch of kRedThreads-thread blocks, with programmatic dependence on the
// launch before it if pdl.
template <typename... P, typename... A>
cudaError_t launch(void (*kernel)(P...), uint32_t blocks, bool pdl, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kRedThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Blocks of a CG iteration's launches: a DoF per thread while that fits
// kRedBlocks (a function of n only).
uint32_t cg_blocks(size_t n) {
    const size_t b = (n + kRedThreads - 1) / kRedThreads;
    return (uint32_t)(b < 1 ? 1 : b > (size_t)kRedBlocks ? (size_t)kRedBlocks : b);
}
}  // namespace

template <typename T>
cudaError_t launch_dot(const T* a, const T* b, size_t n, double* part, uint32_t* nb, cudaStream_t st) {
    *nb = red_blocks(n);
    return launch(k_dot<T>, *nb, false, st, a, b, n, part);
}

template <typename T>
cudaError_t launch_cg_iteration(T* x, T* r, T* p, const T* q, const T* dinv, size_t n, const double* in, double* out,
                                double* part, uint32_t nb_pq, cudaStream_t st) {
    const uint32_t nb = cg_blocks(n);
    const cudaError_t e = launch(k_cg_xr<T>, nb, true, st, x, r, p, q, dinv, n, in, out, part, nb_pq, part + kRedBlocks);
    if (e != cudaSuccess) return e;
    return launch(k_cg_p<T>, nb, true, st, p, r, dinv, n, in, out, part + kRedBlocks, nb);
}

template <typename T>
cudaError_t launch_invert(T* dinv, const double* d, size_t n, cudaStream_t st) {
    k_invert<T><<<grid_for(n), kRedThreads, 0, st>>>(dinv, d, n);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_norm2(const T* a, size_t n, double* sc, double* part, cudaStream_t st) {
    const uint32_t nb = red_blocks(n);
    k_dot<T><<<nb, kRedThreads, 0, st>>>(a, a, n, part);
    k_sum<<<1, 32, 0, st>>>(sc, part, nb);
    return cudaGetLastError();
}

cudaError_t launch_residual(double* r, const double* b, const double* q, size_t n, double* sc, double* part,
                            cudaStream_t st) {
    const uint32_t nb = cg_blocks(n);
    k_residual<<<nb, kRedThreads, 0, st>>>(r, b, q, n, part);
    k_sum<<<1, 32, 0, st>>>(sc, part, nb);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_cg_reliable(const double* r64, T* r, T* z, T* p, const T* dinv, size_t n, double* sc,
                               double* part, double sigma, double rho, cudaStream_t st) {
    const uint32_t nb = cg_blocks(n);
    k_cg_reliable<T><<<nb, kRedThreads, 0, st>>>(r64, r, z, p, dinv, n, part, sigma);
    return launch(k_cg_reliable_p<T>, nb, true, st, p, (const T*)z, n, sc, (const double*)part, nb, rho);
}
template cudaError_t launch_cg_reliable<float>(const double*, float*, float*, float*, const float*, size_t, double*,
                                               double*, double, double, cudaStream_t);
template cudaError_t launch_cg_reliable<double>(const double*, double*, double*, double*, const double*, size_t,
                                                double*, double*, double, double, cudaStream_t);

cudaError_t launch_axpby(double* y, const double* x, double a, double b, size_t n, cudaStream_t st) {
    k_axpby<<<grid_for(n), kRedThreads, 0, st>>>(y, x, a, b, n);
    return cudaGetLastError();
}

cudaError_t launch_to_f32(float* out, const double* in, size_t n, cudaStream_t st, double scale) {
    k_to_f32<float><<<grid_for(n), kRedThreads, 0, st>>>(out, in, n, scale);
    return cudaGetLastError();
}

cudaError_t launch_to_f32(double* out, const double* in, size_t n, cudaStream_t st, double scale) {
    k_to_f32<double><<<grid_for(n), kRedThreads, 0, st>>>(out, in, n, scale);
    return cudaGetLastError();
}

cudaError_t launch_add_f32(double* x, float* d, size_t n, cudaStream_t st, double inv) {
    k_add_f32<float><<<grid_for(n), kRedThreads, 0, st>>>(x, d, n, inv);
    return cudaGetLastError();
}

cudaError_t launch_add_f32(double* x, double* d, size_t n, cudaStream_t st, double inv) {
    k_add_f32<double><<<grid_for(n), kRedThreads, 0, st>>>(x, d, n, inv);
    return cudaGetLastError();
}

cudaError_t launch_patch_combine(int vo_bytes, void* v, const void* pv, const uint32_t* dof, const uint32_t* off,
                                 const uint32_t* idx, uint32_t nb, const void* u_rows, cudaStream_t st) {
    if (nb == 0) return cudaSuccess;
    if (vo_bytes == 8)
        return launch(k_patch_combine<double>, grid_for(nb), true, st, static_cast<double*>(v),
                      static_cast<const double*>(pv), dof, off, idx, nb, static_cast<const double*>(u_rows));
    return launch(k_patch_combine<float>, grid_for(nb), true, st, static_cast<float*>(v),
                  static_cast<const float*>(pv), dof, off, idx, nb, static_cast<const float*>(u_rows));
}

cudaError_t launch_patch_combine_dot(int vo_bytes, void* v, const void* pv, const uint32_t* pos, const uint32_t* dof,
                                     const uint32_t* off, const uint32_t* idx, uint32_t n, const void* u, double* part,
                                     uint32_t* nb, cudaStream_t st) {
    *nb = cg_blocks(n);
    if (vo_bytes == 8)
        return launch(k_patch_combine_dot<double>, *nb, true, st, static_cast<double*>(v),
                      static_cast<const double*>(pv), pos, dof, off, idx, n, static_cast<const double*>(u), part);
    return launch(k_patch_combine_dot<float>, *nb, true, st, static_cast<float*>(v), static_cast<const float*>(pv),
                  pos, dof, off, idx, n, static_cast<const float*>(u), part);
}

namespace {
template <typename VO, typename VT, uint32_t B>
cudaError_t gather_sum(void* v, const void* ve, const uint32_t* off, const uint32_t* idx, uint32_t n, const void* u,
                       const uint8_t* mask, double* part, uint32_t* nb, cudaStream_t st) {
    const uint32_t all = (n + kRedThreads - 1) / kRedThreads;
    VT* const vt = static_cast<VT*>(v);
    const VO* const vo = static_cast<const VO*>(ve);
    const VT* const ut = static_cast<const VT*>(u);
    if (!part) return launch(k_gather_sum<VO, VT, B, false>, all, true, st, vt, vo, off, idx, n, ut, mask, part);
    *nb = cg_blocks(n);
    return launch(k_gather_sum<VO, VT, B, true>, *nb, true, st, vt, vo, off, idx, n, ut, mask, part);
}
template <typename VO, typename VT>
cudaError_t gather_sum_b(uint32_t b, void* v, const void* ve, const uint32_t* off, const uint32_t* idx, uint32_t n,
                         const void* u, const uint8_t* mask, double* part, uint32_t* nb, cudaStream_t st) {
    return b == 3 ? gather_sum<VO, VT, 3>(v, ve, off, idx, n, u, mask, part, nb, st)
                  : gather_sum<VO, VT, 1>(v, ve, off, idx, n, u, mask, part, nb, st);
}
}  // namespace

cudaError_t launch_gather_sum(int ve_bytes, int vt_bytes, uint32_t b, void* v, const void* ve, const uint32_t* off,
                              const uint32_t* idx, uint32_t n, const void* u, const uint8_t* mask, double* part,
                              uint32_t* nb, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    if (ve_bytes == 8 && vt_bytes == 8)
        return gather_sum_b<double, double>(b, v, ve, off, idx, n, u, mask, part, nb, st);
    if (ve_bytes == 8) return gather_sum_b<double, float>(b, v, ve, off, idx, n, u, mask, part, nb, st);
    return gather_sum_b<float, float>(b, v, ve, off, idx, n, u, mask, part, nb, st);
}

cudaError_t launch_umax(const double* u, const uint8_t* mask, size_t n, double* vz, size_t nv,
                        unsigned long long* w, bool pdl, cudaStream_t st) {
    return launch(k_umax, red_blocks(n > nv ? n : nv), pdl, st, u, mask, n, vz, nv, w);
}

cudaError_t launch_umax_cols(const double* U, const uint8_t* mask, size_t rows, uint32_t R, uint32_t ld,
                             unsigned long long* cm, cudaStream_t st) {
    if (R == 0 || R % 2 || R > (uint32_t)kMaxUmaxCols) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(cm, 0, sizeof(unsigned long long) * R, st);
    if (e != cudaSuccess) return e;
    const size_t per = kRedThreads / (R / 2), passes = (rows + kUnroll * per - 1) / (kUnroll * per);
    k_umax_cols<<<(unsigned)(passes < kRedBlocks ? (passes ? passes : 1) : kRedBlocks), kRedThreads, 0, st>>>(U, mask, rows,
                                                                                                             R, ld, cm);
    return cudaGetLastError();
}

#define AFM_SOLVER_INSTANCES(T)                                                                                       \
    template cudaError_t launch_set_constrained<T>(T*, const T*, const uint32_t*, uint32_t, cudaStream_t);            \
    template cudaError_t launch_cg_init<T>(const T*, const T*, const T*, T*, T*, T*, size_t, double*, double*,        \
                                           cudaStream_t);                                                             \
    template cudaError_t launch_dot<T>(const T*, const T*, size_t, double*, uint32_t*, cudaStream_t);                 \
    template cudaError_t launch_cg_iteration<T>(T*, T*, T*, const T*, const T*, size_t, const double*, double*,       \
                                                double*, uint32_t, cudaStream_t);                                     \
    template cudaError_t launch_invert<T>(T*, const double*, size_t, cudaStream_t);                                   \
    template cudaError_t launch_norm2<T>(const T*, size_t, double*, double*, cudaStream_t);

AFM_SOLVER_INSTANCES(double)
AFM_SOLVER_INSTANCES(float)

}  // namespace afm
