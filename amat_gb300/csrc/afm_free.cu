// Matrix-free product (method 2, par::aMatFree with MATFREE_TYPE::FREE,
// include/aMatFree.hpp:2241-2745): no element matrix is stored; every product
// integrates each element's stiffness action from its node coordinates,
//   v_e = sum_q w_q |J_q| B_q^T D B_q u_e,
// which is Ke u_e of the reference's element kernels (the callback
// m_eleMatFunc computes Ke from xe, include/aMat.hpp:104-116, then multiplies)
// up to the order of the sums. It trades the Ke bytes for arithmetic: in FP32
// it needs ~0.5 KB per hex20 element instead of 7-29 KB of stored Ke.
//
// G = 8 or 32 lanes per element (32 / G elements per warp). A lane at
// quadrature point q forms J and the reference gradient R = du/dxi from the
// nodes, then, with C = adj(J) (J^-1 = C / |J|), the physical gradient times
// |J|, R C, the stress (or flux) of it times w / |J|, and its transform back
// to reference directions, P = S C^T: all per quadrature point, so that the
// nodes only see v_a = sum_q P_q dN_a(q). (Transforming dN_a to physical
// directions at every node and point, in both passes, cost 18 multiply-adds
// per node and point more: 36 against 27 in hex8 elasticity.)
//
// Coordinates are taken relative to the element's first node, which J does not
// depend on: their rounding no longer enters at the size of the domain over the
// size of the element (FP64 product of hex8 elasticity 32^3 against extended
// precision: 2.4e-15 -> 2.5e-16).
//
// What bounds it: FP64, the FP64 pipe (1/64 of the FP32 rate on GB300); FP32,
// instruction issue. So the count of multiply-adds decides, and lanes without
// work cost as much as busy ones (hence 8 lanes an element for tet10's 8 points
// and 10 nodes). Measured, with physical gradients at the nodes and a launch per
// colour -> this: FP64 hex8 elasticity 32^3 202 -> 103 us, hex20 elasticity
// 24^3 902 -> 511, tet10 Poisson 20^3 x 6 624 -> 144; FP32 hex20 elasticity
// 28x27x29 66 -> 30 us, hex8 elasticity 48^3 39 -> 18.
#include <cuda_runtime.h>
#include <stdint.h>

#include "afm_internal.hpp"

namespace afm {

namespace {

template <int KIND>
struct FreeKind;
// DoFs per node (and nodes, where a kernel takes them from tables; the tables follow afm_shape.hpp)
template <>
struct FreeKind<0> { static constexpr int DPN = 1; };
template <>
struct FreeKind<1> { static constexpr int DPN = 3; };
template <>
struct FreeKind<2> { static constexpr int NODES = 20, DPN = 3; };
template <>
struct FreeKind<3> { static constexpr int NODES = 10, DPN = 1; };
template <>
struct FreeKind<4> { static constexpr int NODES = 10, DPN = 3; };

constexpr int kFreeWarps = 4;
constexpr int kFreeMaxQ = 27;

// v[i] += x at L2, no load and no wait (round to nearest; the f32 form
// flushes subnormal values to zero). Elements of a launch share no DoF and
// launches are ordered, so each entry gets one add per colour, in colour order.
__device__ __forceinline__ void red_add(float* p, float x) {
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(x) : "memory");
}
__device__ __forceinline__ void red_add(double* p, double x) {
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(p), "d"(x) : "memory");
}

__device__ __forceinline__ float fm(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fm(double a, double b, double c) { return __fma_rn(a, b, c); }

// Smallest stride (in T) >= n that puts the slots of a warp's elements, read
// side by side in 16-byte pieces, on different shared-memory banks.
template <typename T>
constexpr int slot_stride(int n) {
    constexpr int W = (int)sizeof(T) / 4;
    int s = (n * W + 3) / 4 * 4;
    while (s % 32 != 8 && s % 32 != 24) s += 4;
    return s / W;
}

// The quadrature point's share: J[i][p] = dx_i / dxi_p and R[i][p] = du_i /
// dxi_p (i < DPN) to P[i][p] (in R); w: the point's weight.
template <int DPN, typename T>
__device__ __forceinline__ void point_flux(const T (&J)[3][3], T (&R)[DPN][3], T w, T lam, T mu) {
    T C[3][3];  // adj(J): C[p][i] = |J| d xi_p / d x_i
    C[0][0] = fm(J[1][1], J[2][2], -J[1][2] * J[2][1]);
    C[0][1] = fm(J[0][2], J[2][1], -J[0][1] * J[2][2]);
    C[0][2] = fm(J[0][1], J[1][2], -J[0][2] * J[1][1]);
    C[1][0] = fm(J[1][2], J[2][0], -J[1][0] * J[2][2]);
    C[1][1] = fm(J[0][0], J[2][2], -J[0][2] * J[2][0]);
    C[1][2] = fm(J[0][2], J[1][0], -J[0][0] * J[1][2]);
    C[2][0] = fm(J[1][0], J[2][1], -J[1][1] * J[2][0]);
    C[2][1] = fm(J[0][1], J[2][0], -J[0][0] * J[2][1]);
    C[2][2] = fm(J[0][0], J[1][1], -J[0][1] * J[1][0]);
    const T det = fm(J[0][0], C[0][0], fm(J[0][1], C[1][0], J[0][2] * C[2][0]));
    const T s = w / det;
    T H[DPN][3];  // |J| du_i / dx_j
#pragma unroll
    for (int i = 0; i < DPN; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) H[i][j] = fm(R[i][0], C[0][j], fm(R[i][1], C[1][j], R[i][2] * C[2][j]));
    if constexpr (DPN == 3) {
        const T ls = lam * s, ms = mu * s;
        const T tr = ls * (H[0][0] + H[1][1] + H[2][2]);
        const T xx = fm(ms, H[0][0] + H[0][0], tr), yy = fm(ms, H[1][1] + H[1][1], tr);
        const T zz = fm(ms, H[2][2] + H[2][2], tr);
        const T xy = ms * (H[0][1] + H[1][0]), yz = ms * (H[1][2] + H[2][1]), xz = ms * (H[0][2] + H[2][0]);
#pragma unroll
        for (int p = 0; p < 3; p++) {
            R[0][p] = fm(xx, C[p][0], fm(xy, C[p][1], xz * C[p][2]));
            R[1][p] = fm(xy, C[p][0], fm(yy, C[p][1], yz * C[p][2]));
            R[2][p] = fm(xz, C[p][0], fm(yz, C[p][1], zz * C[p][2]));
        }
    } else {
#pragma unroll
        for (int p = 0; p < 3; p++) R[0][p] = s * fm(H[0][0], C[p][0], fm(H[0][1], C[p][1], H[0][2] * C[p][2]));
    }
}

// ---- 8-node bricks -----------------------------------------------------------
// The trilinear fields x and u in monomials of (xi, eta, zeta): lane = node
// (lanes sl < 8) takes its node's values through three Hadamard stages (one
// shuffle and one add per value each) to the coefficient of one monomial,
// coefficient k (bit 0: xi, 1: eta, 2: zeta); a gradient is then 8
// multiply-adds per field component instead of 24, and so is its adjoint: the
// lane's P gives the seven coefficients of the test fields, a reduce-scatter
// over the lanes leaves each lane one coefficient's sum, and three Hadamard
// stages turn the coefficients into nodes. (Fields are held 8 times too large,
// which w / 512 undoes.)
template <int DPN, typename T, int G, bool VE>
__global__ void __launch_bounds__(kFreeWarps * 32, sizeof(T) == 4 ? 6 : 4) k_free_hex8(FreeArgs a) {
    constexpr int N = 8 * DPN, V = 3 + DPN;  // V: field components, x then u
    constexpr int EPW = 32 / G, SLOTS = kFreeWarps * EPW, CS = slot_stride<T>(8 * V);
    __shared__ __align__(16) T cf[SLOTS][CS];
    const int nq = (int)a.nq;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp * EPW + lane / G, sl = lane % G;
    const T* __restrict__ u = static_cast<const T*>(a.u);
    const T* __restrict__ xe = static_cast<const T*>(a.xe);
    const T lam = (T)a.lam, mu = (T)a.mu;
    // this lane's quadrature point (tables: dN, weights, points) and node signs (node order of hex8)
    const T* gw = static_cast<const T*>(a.ref) + nq * 24;
    const bool point = sl < nq, node = sl < 8;
    const T w = point ? gw[sl] * T(1.0 / 512.0) : T(0);
    const T X = point ? gw[nq + 3 * sl] : T(0), Y = point ? gw[nq + 3 * sl + 1] : T(0),
            Z = point ? gw[nq + 3 * sl + 2] : T(0);
    const bool b0 = ((sl ^ (sl >> 1)) & 1) != 0, b1 = (sl & 2) != 0, b2 = (sl & 4) != 0;
    const T s0 = b0 ? T(1) : T(-1), s1 = b1 ? T(1) : T(-1), s2 = b2 ? T(1) : T(-1);
    const int kc = (b0 ? 1 : 0) + (b1 ? 2 : 0) + (b2 ? 4 : 0);  // the lane's coefficient
    const uint32_t stride = gridDim.x * SLOTS;
    // every lane of the warp runs the same number of rounds; a slot past the end idles
    // Gather pipeline: the next round's values (and the map of the round after) load during this one.
    uint32_t mc[DPN], mn[DPN];
    T val[V], nxt[V];
    auto load_map = [&](uint32_t base_r, uint32_t* out) {
        const uint32_t el_r = base_r + lane / G;
#pragma unroll
        for (int i = 0; i < DPN; i++)
            out[i] = (node && el_r < a.count) ? __ldg(a.map + (size_t)(a.first + el_r) * N + DPN * sl + i) : 0u;
    };
    auto load_ux = [&](uint32_t base_r, const uint32_t* mp) {
        const uint32_t el_r = base_r + lane / G;
        const bool ok = node && el_r < a.count;
#pragma unroll
        for (int i = 0; i < 3; i++) nxt[i] = ok ? __ldg(xe + (size_t)(a.first + el_r) * 24 + 3 * sl + i) : T(0);
#pragma unroll
        for (int i = 0; i < DPN; i++) {
            T x = ok ? __ldg(u + (mp[i] & kDofMask)) : T(0);
            if (a.bc_mode && (mp[i] & kBcFlag)) x = T(0);
            nxt[3 + i] = x;
        }
    };
    uint32_t base = blockIdx.x * SLOTS + warp * EPW;
    load_map(base, mc);
    load_ux(base, mc);
    load_map(base + stride, mn);
    for (; base < a.count; base += stride) {
        const uint32_t el = base + lane / G;
        const bool live = el < a.count;
        uint32_t dof[DPN];
#pragma unroll
        for (int i = 0; i < V; i++) val[i] = nxt[i];
#pragma unroll
        for (int i = 0; i < DPN; i++) {
            dof[i] = mc[i];
            mc[i] = mn[i];
        }
        load_ux(base + stride, mc);
        load_map(base + 2 * stride, mn);
#pragma unroll
        for (int i = 0; i < V; i++) {
            T x = val[i];
            if (i < 3) x -= __shfl_sync(0xffffffffu, x, 0, G);  // from the element's first node
            x = fm(-s0, __shfl_xor_sync(0xffffffffu, x, 1), x);
            x = fm(-s1, __shfl_xor_sync(0xffffffffu, x, 3), x);
            x = fm(-s2, __shfl_xor_sync(0xffffffffu, x, 4), x);
            if (node) cf[slot][V * kc + i] = x;
        }
        __syncwarp();
        T R[DPN][3] = {};
        {
            T g[V][3];
            const T* c = cf[slot];
#pragma unroll
            for (int i = 0; i < V; i++) {
                const T c5 = c[5 * V + i], c6 = c[6 * V + i], c7 = c[7 * V + i];
                const T t = fm(c7, Z, c[3 * V + i]);
                g[i][0] = fm(Y, t, fm(c5, Z, c[V + i]));
                g[i][1] = fm(X, t, fm(c6, Z, c[2 * V + i]));
                g[i][2] = fm(Y, fm(c7, X, c6), fm(c5, X, c[4 * V + i]));
            }
            if (point && live) {
                T J[3][3];
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int p = 0; p < 3; p++) J[i][p] = g[i][p];
#pragma unroll
                for (int i = 0; i < DPN; i++)
#pragma unroll
                    for (int p = 0; p < 3; p++) R[i][p] = g[3 + i][p];
                point_flux<DPN, T>(J, R, w, lam, mu);
            }
        }
        __syncwarp();  // the coefficients are read before the next round's are written
        T out[DPN];
#pragma unroll
        for (int i = 0; i < DPN; i++) {
            T A[8];
            A[0] = T(0);
            A[1] = R[i][0];
            A[2] = R[i][1];
            A[4] = R[i][2];
            A[3] = fm(Y, R[i][0], X * R[i][1]);
            A[5] = fm(Z, R[i][0], X * R[i][2]);
            A[6] = fm(Z, R[i][1], Y * R[i][2]);
            A[7] = fm(Z, A[3], X * Y * R[i][2]);
            if constexpr (G == 32) {
#pragma unroll
                for (int k = 1; k < 8; k++) {
                    A[k] += __shfl_xor_sync(0xffffffffu, A[k], 16);
                    A[k] += __shfl_xor_sync(0xffffffffu, A[k], 8);
                }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const T keep = b2 ? A[k + 4] : A[k], send = b2 ? A[k] : A[k + 4];
                A[k] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
            }
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const T keep = b1 ? A[k + 2] : A[k], send = b1 ? A[k] : A[k + 2];
                A[k] = keep + __shfl_xor_sync(0xffffffffu, send, 3);
            }
            const T keep = b0 ? A[1] : A[0], send = b0 ? A[0] : A[1];
            T x = keep + __shfl_xor_sync(0xffffffffu, send, 1);
            x = fm(s0, __shfl_xor_sync(0xffffffffu, x, 1), x);
            x = fm(s1, __shfl_xor_sync(0xffffffffu, x, 3), x);
            out[i] = fm(s2, __shfl_xor_sync(0xffffffffu, x, 4), x);
        }
        if (live && node) {
#pragma unroll
            for (int i = 0; i < DPN; i++) {
                if constexpr (VE)
                    static_cast<T*>(a.ve)[(size_t)(a.first + el) * N + DPN * sl + i] = out[i];
                else
                    red_add(static_cast<T*>(a.v) + (dof[i] & kDofMask), out[i]);
            }
        }
    }
}

// ---- other elements: nodes and points from the tables of the reference element
template <int KIND, typename T, int G, bool VE>
__global__ void __launch_bounds__(kFreeWarps * 32, sizeof(T) == 4 ? 6 : 4) k_free(FreeArgs a) {
    constexpr int NN = FreeKind<KIND>::NODES, DPN = FreeKind<KIND>::DPN, N = NN * DPN, V = 3 + DPN;
    constexpr int EPW = 32 / G, SLOTS = kFreeWarps * EPW, QM = G < kFreeMaxQ ? G : kFreeMaxQ;
    constexpr int NS = slot_stride<T>(NN * V);             // nodes of one element: (x, u) per node
    constexpr int PS = (3 * DPN * (int)sizeof(T) + 15) / 16 * 16 / (int)sizeof(T);  // P of one point
    constexpr int QS = slot_stride<T>(QM * PS);
    constexpr int RS = NN * 3 + 1 - (NN * 3) % 2;  // odd: lanes at different points read different banks
    __shared__ T dNs[QM * RS];
    __shared__ __align__(16) T nd[SLOTS][NS];
    __shared__ __align__(16) T pq[SLOTS][QS];
    const int nq = (int)a.nq;
    const T* gref = static_cast<const T*>(a.ref);
    for (int i = threadIdx.x; i < nq * NN * 3; i += blockDim.x) dNs[i / (NN * 3) * RS + i % (NN * 3)] = gref[i];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp * EPW + lane / G, sl = lane % G;
    const T* __restrict__ u = static_cast<const T*>(a.u);
    const T* __restrict__ xe = static_cast<const T*>(a.xe);
    const T lam = (T)a.lam, mu = (T)a.mu;
    const T w = sl < nq ? gref[nq * NN * 3 + sl] : T(0);
    const uint32_t stride = gridDim.x * SLOTS;
    // every lane of the warp runs the same number of rounds (the __syncwarp calls); a slot past the end idles
    // Gather pipeline: the element of the next round has its u entries and coordinates loaded (and the one
    // after it its map) while the current element is integrated, so a round waits on no load of its own.
    constexpr int CN = (N + G - 1) / G, CX = (NN * 3 + G - 1) / G;
    uint32_t mc[CN], mn[CN];  // maps of the next round and of the one after
    T uc[CN], xc[CX];         // u entries and coordinates of the next round
    auto load_map = [&](uint32_t base_r, uint32_t* out) {
        const uint32_t el_r = base_r + lane / G;
#pragma unroll
        for (int k = 0; k < CN; k++) {
            const int i = sl + k * G;
            out[k] = (el_r < a.count && i < N) ? __ldg(a.map + (size_t)(a.first + el_r) * N + i) : 0u;
        }
    };
    auto load_ux = [&](uint32_t base_r, const uint32_t* mp) {
        const uint32_t el_r = base_r + lane / G;
        const bool ok = el_r < a.count;
#pragma unroll
        for (int k = 0; k < CN; k++) {
            const int i = sl + k * G;
            T x = (ok && i < N) ? __ldg(u + (mp[k] & kDofMask)) : T(0);
            if (a.bc_mode && (mp[k] & kBcFlag)) x = T(0);
            uc[k] = x;
        }
#pragma unroll
        for (int k = 0; k < CX; k++) {
            const int i = sl + k * G;
            xc[k] = (ok && i < NN * 3) ? __ldg(xe + (size_t)(a.first + el_r) * NN * 3 + i) : T(0);
        }
    };
    uint32_t base = blockIdx.x * SLOTS + warp * EPW;
    load_map(base, mc);
    load_ux(base, mc);
    load_map(base + stride, mn);
    for (; base < a.count; base += stride) {
        const uint32_t el = base + lane / G;
        const bool live = el < a.count;
        T x0[3];  // the element's first node
#pragma unroll
        for (int i = 0; i < 3; i++) x0[i] = __shfl_sync(0xffffffffu, xc[0], i, G);
        if (live) {
#pragma unroll
            for (int k = 0; k < CN; k++) {
                const int i = sl + k * G;
                if (i < N) nd[slot][i / DPN * V + 3 + i % DPN] = uc[k];
            }
#pragma unroll
            for (int k = 0; k < CX; k++) {
                const int i = sl + k * G;
                const T o = i % 3 == 0 ? x0[0] : i % 3 == 1 ? x0[1] : x0[2];
                if (i < NN * 3) nd[slot][i / 3 * V + i % 3] = xc[k] - o;
            }
        }
        __syncwarp();
        // next round: its u and coordinates from the map loaded a round ago; the map of the round after
#pragma unroll
        for (int k = 0; k < CN; k++) mc[k] = mn[k];
        load_ux(base + stride, mc);
        load_map(base + 2 * stride, mn);
        if (live && sl < nq) {
            const T* dN = dNs + sl * RS;
            T J[3][3] = {}, R[DPN][3] = {};  // J[i][p] = d x_i / d xi_p, R[i][p] = d u_i / d xi_p
#pragma unroll
            for (int b = 0; b < NN; b++) {
                const T* nb = nd[slot] + b * V;
                const T d0 = dN[3 * b], d1 = dN[3 * b + 1], d2 = dN[3 * b + 2];
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    const T x = nb[i];
                    J[i][0] = fm(x, d0, J[i][0]), J[i][1] = fm(x, d1, J[i][1]), J[i][2] = fm(x, d2, J[i][2]);
                }
#pragma unroll
                for (int i = 0; i < DPN; i++) {
                    const T x = nb[3 + i];
                    R[i][0] = fm(x, d0, R[i][0]), R[i][1] = fm(x, d1, R[i][1]), R[i][2] = fm(x, d2, R[i][2]);
                }
            }
            point_flux<DPN, T>(J, R, w, lam, mu);
            T* o = pq[slot] + sl * PS;
#pragma unroll
            for (int i = 0; i < DPN; i++)
#pragma unroll
                for (int p = 0; p < 3; p++) o[3 * i + p] = R[i][p];
        }
        __syncwarp();
        if (live)
            for (int b = sl; b < NN; b += G) {
                T acc[DPN] = {};
#pragma unroll 3
                for (int q = 0; q < nq; q++) {
                    const T* o = pq[slot] + q * PS;
                    const T* dN = dNs + q * RS + 3 * b;
                    const T d0 = dN[0], d1 = dN[1], d2 = dN[2];
#pragma unroll
                    for (int i = 0; i < DPN; i++)
                        acc[i] = fm(d0, o[3 * i], fm(d1, o[3 * i + 1], fm(d2, o[3 * i + 2], acc[i])));
                }
                const size_t row = (size_t)(a.first + el) * N + DPN * b;
#pragma unroll
                for (int i = 0; i < DPN; i++) {
                    if constexpr (VE)
                        static_cast<T*>(a.ve)[row + i] = acc[i];
                    else
                        red_add(static_cast<T*>(a.v) + (__ldg(a.map + row + i) & kDofMask), acc[i]);
                }
            }
        __syncwarp();
    }
}

template <int KIND, typename T, bool VE>
void* free_kernel_g(int g) {
    constexpr int DPN = FreeKind<KIND>::DPN;
    if constexpr (KIND < 2)
        return g == 8 ? (void*)k_free_hex8<DPN, T, 8, VE> : (void*)k_free_hex8<DPN, T, 32, VE>;
    else if constexpr (KIND > 2)
        return g == 8 ? (void*)k_free<KIND, T, 8, VE> : (void*)k_free<KIND, T, 32, VE>;
    else
        return (void*)k_free<KIND, T, 32, VE>;
}

template <typename T, bool VE>
void* free_kernel(int kind, int g) {
    switch (kind) {
        case 0: return free_kernel_g<0, T, VE>(g);
        case 1: return free_kernel_g<1, T, VE>(g);
        case 2: return free_kernel_g<2, T, VE>(g);
        case 3: return free_kernel_g<3, T, VE>(g);
        case 4: return free_kernel_g<4, T, VE>(g);
        default: return nullptr;
    }
}

}  // namespace

cudaError_t launch_free(int kind, bool f32, const FreeArgs& a, int sm_count, cudaStream_t st) {
    if (a.count == 0) return cudaSuccess;
    if (a.nq == 0 || a.nq > (uint32_t)kFreeMaxQ || kind < 0 || kind > 4) return cudaErrorInvalidValue;
    // lanes per element: the quadrature points (8 with two per direction, 27 with three); hex20's 20 nodes want 32
    const int g = a.nq <= 8 && kind != 2 ? 8 : 32;
    void* fn = a.ve ? (f32 ? free_kernel<float, true>(kind, g) : free_kernel<double, true>(kind, g))
                    : (f32 ? free_kernel<float, false>(kind, g) : free_kernel<double, false>(kind, g));
    const uint32_t slots = kFreeWarps * (32 / g);
    const uint32_t want = (a.count + slots - 1) / slots;
    const uint32_t most = (uint32_t)sm_count * (f32 ? 6 : 4);  // what the kernels' launch bounds keep resident
    FreeArgs args = a;
    void* params[] = {&args};
    return cudaLaunchKernel(fn, dim3(want < most ? want : most), dim3(kFreeWarps * 32), params, 0, st);
}

}  // namespace afm
