// Batched product V = K U over patches (elements of 24, 30 or 60 DoFs).
//
// The kernels that take a launch per colour read and write every V row once
// per element that lists it, through an L2 that the blocks do not fit: that
// traffic, not arithmetic, bounds them (hex8 elasticity 48^3 x 64 columns,
// FP32: 2.1 GB a product against 0.44 GB of element matrices and blocks). Here
// a warp takes a patch (up to 8 elements around a node, afm_batched_patch.hpp)
// and a block of CB columns, and sums the patch's rows of V in its own shared
// memory, element by element in a fixed order; rows of this patch alone go
// straight to V, the others to a combine buffer that a second pass adds up in
// patch order (bit-reproducible, no atomics, no colours). Warps share nothing,
// so there is no barrier but __syncwarp. Element matrices and U rows arrive by
// cp.async one element ahead, the next patch's header one patch ahead.
//
// Lane tile: RT rows x CT columns of V_e, RG row groups x CG column groups =
// 32 lanes, CB = CG CT columns. The products run on packed pairs of rows
// (fma.rn.f32x2: the same IEEE results, half the instructions; a column of Ke
// has its rows side by side, so only the entries of U_e are packed by hand): per
// column of Ke a lane reads RT entries of Ke, CT of U_e and issues RT CT / 2
// (FP32) or 6 RT CT (double-float) of them. What bounds it is latency: the
// shared memory of a warp (rows of V, two elements) sets the warps per SM, so a
// task is 32 columns (16 in double-float), not 64 (hex8 elasticity 48^3 x 64:
// 495 us with 64 columns and 5 warps per SM, 377 with 32 and 9); and next to it
// the shared-memory wavefronts of a lane tile (6 x 4: 10 per column of Ke; 12 x
// 2, whose rows load 16 bytes at a time: 14, 444 us). Measured, best tile of the
// launches per colour -> this: FP32 hex8 elasticity 48^3 x 64 639 -> 417 us, 20^3
// x 20 32 -> 17, hex20 20^3 x 64 417 -> 204, tet10 10^3 x 6 x 64 155 -> 44;
// split hex8 elasticity 24^3 x 32 525 -> 221 us.
#include <algorithm>

#include "afm_batched.cuh"
#include "afm_batched_patch.hpp"

namespace afm {

namespace {

constexpr int kBPatchWarps = 16;  // per CTA, at most

// cp.async of 16 bytes, or of 16 zero bytes
__device__ __forceinline__ void cp_async16z(void* dst, const void* src, bool zero) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(zero ? 0 : 16)
                 : "memory");
}

// Shared memory of one warp.
struct BPatchSmem {
    uint32_t vacc, u, u_bytes, k, k_bytes, total;
    __host__ __device__ BPatchSmem(const BPatchGeom& g, uint32_t cb, uint32_t vt, uint32_t ke_bytes) {
        vacc = 2 * g.hdr_bytes;
        u = vacc + g.max_rows * cb * vt;
        u_bytes = g.n * cb * vt;
        k = u + 2 * u_bytes;
        k_bytes = ((ke_bytes + 15u) & ~15u) + 32u;  // a lane tile past the last row reads on into the padding
        total = (k + 2 * k_bytes + 127u) & ~127u;
    }
};

template <int NT, int RT, int CT, bool SPLIT>
__global__ void __launch_bounds__(kBPatchWarps * 32, 1)
    k_bpatch(BPatchArgs a, BPatchGeom g, uint32_t ke_bytes, uint32_t ncb) {
    constexpr int RG = (NT + RT - 1) / RT, CG = 32 / RG, CB = CG * CT;
    static_assert(RG * CG == 32 && CT % 2 == 0 && RT % 2 == 0 && NT % 2 == 0 && CB <= 32, "lane tile");
    using VT = std::conditional_t<SPLIT, double, float>;
    constexpr int EPC = 16 / (int)sizeof(VT);  // entries of a 16-byte chunk
    constexpr int CPR = CB / EPC;              // chunks of a row
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
    const BPatchSmem L(g, CB, sizeof(VT), ke_bytes);
    unsigned char* const base = smem + (size_t)warp * L.total;
    VT* const vacc = reinterpret_cast<VT*>(base + L.vacc);
    const uint32_t rg = lane / CG, cg = lane % CG, r0 = rg * RT, col = cg * CT;
    const VT* __restrict__ U = static_cast<const VT*>(a.u);
    VT* __restrict__ V = static_cast<VT*>(a.v);
    VT* __restrict__ PV = static_cast<VT*>(a.pv);
    const uint32_t R = a.nrhs, tasks = g.patches * ncb, step = gridDim.x * W;

    auto header = [&](uint32_t b) { return reinterpret_cast<const uint32_t*>(base + b * g.hdr_bytes); };
    auto load_header = [&](uint32_t t, uint32_t b) {
        const unsigned char* src = a.hdr + (size_t)(t / ncb) * g.hdr_bytes;
        for (uint32_t q = lane * 16; q < g.hdr_bytes; q += 512) cp_async16(base + b * g.hdr_bytes + q, src + q);
    };
    // element e of the patch in header b: its matrix and its rows of U, columns [c0, c0 + CB)
    auto load_element = [&](uint32_t b, uint32_t e, uint32_t c0, uint32_t buf) {
        const uint32_t* h = header(b);
        const unsigned char* ks = a.ke + (size_t)h[8 + e] * a.unit_bytes;
        unsigned char* kd = base + L.k + buf * L.k_bytes;
        for (uint32_t q = lane * 16; q < ke_bytes; q += 512) cp_async16(kd + q, ks + q);
        const uint32_t* rows = h + bpatch_rows_off() / 4;
        const unsigned char* loc = reinterpret_cast<const unsigned char*>(h) + bpatch_loc_off(g.max_rows) + e * NT;
        unsigned char* ud = base + L.u + buf * L.u_bytes;
        const uint32_t k = lane % CPR, cc = c0 + k * EPC;
#pragma unroll 4
        for (uint32_t c = lane / CPR; c < NT; c += 32 / CPR) {
            const uint32_t d = rows[loc[c]];
            const bool zero = cc >= R || (a.bc_mode && (d & kBcFlag));
            const VT* src = zero ? U : U + (size_t)(d & kDofMask) * a.ld + cc;
            cp_async16z(ud + (c * CPR + k) * 16, src, zero);
        }
    };

    // CT values of a row of U_e, each twice; RT values of a column of Ke in pairs of rows
    auto load_u = [&](const float* p, f2* u2) {
#pragma unroll
        for (int y = 0; y < CT; y += 2) {
            const float2 w = *reinterpret_cast<const float2*>(p + y);
            u2[y] = pack2(w.x, w.x);
            u2[y + 1] = pack2(w.y, w.y);
        }
    };
    auto load_k = [&](const float* p, f2* k2) {
        if constexpr (RT % 4 == 0 && NT % 4 == 0) {
#pragma unroll
            for (int x = 0; x < RT; x += 4) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(p + x);
                k2[x / 2] = w.x, k2[x / 2 + 1] = w.y;
            }
        } else {
#pragma unroll
            for (int x = 0; x < RT; x += 2) k2[x / 2] = *reinterpret_cast<const f2*>(p + x);
        }
    };

    uint32_t t = blockIdx.x * W + warp;
    if (t >= tasks) return;
    uint32_t hb = 0, buf = 0;
    load_header(t, 0);
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();
    load_element(0, 0, (t % ncb) * CB, 0);
    cp_async_commit();
    for (; t < tasks; t += step, hb ^= 1) {
        const uint32_t tn = t + step, c0 = (t % ncb) * CB;
        const uint32_t* h = header(hb);
        const uint32_t ne = h[0], nr = h[1], own = h[2], pv0 = h[3];
        const unsigned char* loc = reinterpret_cast<const unsigned char*>(h) + bpatch_loc_off(g.max_rows);
        if (tn < tasks) load_header(tn, hb ^ 1);
        cp_async_commit();
        int usk = 0;  // of column c0 + lane
        if constexpr (SPLIT) usk = lane < CB && c0 + lane < R ? uscale_of(a.umax[c0 + lane]) : 0;
        for (uint32_t q = lane; q < nr * CPR; q += 32) reinterpret_cast<uint4*>(vacc)[q] = make_uint4(0, 0, 0, 0);
        for (uint32_t e = 0; e < ne; e++, buf ^= 1) {
            if (e + 1 < ne) {
                load_element(hb, e + 1, c0, buf ^ 1);
                cp_async_commit();
                cp_async_wait<1>();
                __syncwarp();
            } else {
                cp_async_wait<0>();  // this element and the next patch's header
                __syncwarp();
                if (tn < tasks) load_element(hb ^ 1, 0, (tn % ncb) * CB, buf ^ 1);
                cp_async_commit();
            }
            unsigned char* ub = base + L.u + buf * L.u_bytes;
            const float* kp = reinterpret_cast<const float*>(base + L.k + buf * L.k_bytes) + r0;
            const unsigned char* le = loc + e * NT;
            if constexpr (!SPLIT) {
                f2 acc[RT / 2][CT];
#pragma unroll
                for (int x = 0; x < RT / 2; x++)
#pragma unroll
                    for (int y = 0; y < CT; y++) acc[x][y] = 0ull;
                const float* up = reinterpret_cast<const float*>(ub) + col;
#pragma unroll 4
                for (int c = 0; c < NT; c++) {
                    f2 u2[CT], k2[RT / 2];
                    load_u(up + c * CB, u2);
                    load_k(kp + c * NT, k2);
#pragma unroll
                    for (int x = 0; x < RT / 2; x++)
#pragma unroll
                        for (int y = 0; y < CT; y++) acc[x][y] = fma2(k2[x], u2[y], acc[x][y]);
                }
#pragma unroll
                for (int x = 0; x < RT; x += 2)
                    if (r0 + x < NT) {  // (NT even: so is the second row of the pair)
                        float2 s[CT];
#pragma unroll
                        for (int y = 0; y < CT; y++) s[y] = unpack2(acc[x / 2][y]);
#pragma unroll
                        for (int h2 = 0; h2 < 2; h2++) {
                            float2* p = reinterpret_cast<float2*>(vacc + (uint32_t)le[r0 + x + h2] * CB + col);
#pragma unroll
                            for (int y = 0; y < CT; y += 2) {
                                float2 w = p[y / 2];
                                w.x += h2 ? s[y].y : s[y].x;
                                w.y += h2 ? s[y + 1].y : s[y + 1].x;
                                p[y / 2] = w;
                            }
                        }
                    }
            } else {
                // U_e as scaled float pairs, in place: a row's doubles become its leading parts, then the rest
                constexpr int RPP = 32 / CB;  // rows a pass of the warp converts
                const int my = __shfl_sync(0xffffffffu, usk, (int)(lane % CB));
#pragma unroll
                for (int c = 0; c < NT; c += 4 * RPP) {
                    double x[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int row = c + q * RPP + (int)lane / CB;
                        x[q] = row < NT ? reinterpret_cast<const double*>(ub)[row * CB + lane % CB] : 0.0;
                    }
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int row = c + q * RPP + (int)lane / CB;
                        if (row < NT) {
                            const float2 s = split_scaled(x[q], my);
                            float* w = reinterpret_cast<float*>(ub) + row * 2 * CB + lane % CB;
                            w[0] = s.x;
                            w[CB] = s.y;
                        }
                    }
                }
                __syncwarp();
                f2 hi[RT / 2][CT], lo[RT / 2][CT];
#pragma unroll
                for (int x = 0; x < RT / 2; x++)
#pragma unroll
                    for (int y = 0; y < CT; y++) hi[x][y] = lo[x][y] = 0ull;
                const float* up = reinterpret_cast<const float*>(ub) + col;
                const float* kl = kp + a.plane;
                const f2 m1 = pack2(-1.0f, -1.0f);
#pragma unroll 2
                for (int c = 0; c < NT; c++) {
                    // U pairs and their negatives: with -u the error terms of the products come out negated, so that
                    // every difference is a multiply-add by -1 (exact products: the roundings of ArithSplit::fma)
                    f2 uh[CT], nh[CT], nl[CT], kx[RT / 2], ky[RT / 2];
                    load_u(up + c * 2 * CB, uh);
                    load_u(up + c * 2 * CB + CB, nl);
#pragma unroll
                    for (int y = 0; y < CT; y++) nh[y] = mul2(uh[y], m1), nl[y] = mul2(nl[y], m1);
                    load_k(kp + c * NT, kx);
                    load_k(kl + c * NT, ky);
#pragma unroll
                    for (int x = 0; x < RT / 2; x++) {
#pragma unroll
                        for (int y = 0; y < CT; y++) {
                            const f2 p = mul2(kx[x], uh[y]);
                            const f2 nt = fma2(kx[x], nl[y], fma2(ky[x], nh[y], fma2(kx[x], nh[y], p)));
                            const f2 s = add2(hi[x][y], p);
                            const f2 bp = fma2(hi[x][y], m1, s);
                            const f2 err = add2(fma2(fma2(bp, m1, s), m1, hi[x][y]), fma2(bp, m1, p));
                            hi[x][y] = s;
                            lo[x][y] = add2(lo[x][y], fma2(nt, m1, err));
                        }
                    }
                }
#pragma unroll
                for (int x = 0; x < RT; x += 2)
                    if (r0 + x < NT) {
                        float2 s[CT], z[CT];
#pragma unroll
                        for (int y = 0; y < CT; y++) s[y] = unpack2(hi[x / 2][y]), z[y] = unpack2(lo[x / 2][y]);
#pragma unroll
                        for (int h2 = 0; h2 < 2; h2++) {
                            double2* p = reinterpret_cast<double2*>(vacc + (uint32_t)le[r0 + x + h2] * CB + col);
#pragma unroll
                            for (int y = 0; y < CT; y += 2) {
                                double2 w = p[y / 2];
                                w.x += (double)(h2 ? s[y].y : s[y].x) + (double)(h2 ? z[y].y : z[y].x);
                                w.y += (double)(h2 ? s[y + 1].y : s[y + 1].x) + (double)(h2 ? z[y + 1].y : z[y + 1].x);
                                p[y / 2] = w;
                            }
                        }
                    }
            }
            __syncwarp();
        }
        // the patch's rows: its own to V, the others to the combine buffer
        const uint32_t* rows = h + bpatch_rows_off() / 4;
        const uint32_t k = lane % CPR, cc = c0 + k * EPC;
        int k0 = 0, k1 = 0;
        if constexpr (SPLIT) {
            k0 = __shfl_sync(0xffffffffu, usk, (int)(2 * k));
            k1 = __shfl_sync(0xffffffffu, usk, (int)(2 * k + 1));
        }
        if (cc < R)
            for (uint32_t r = lane / CPR; r < nr; r += 32 / CPR) {
                uint4 w = reinterpret_cast<const uint4*>(vacc)[r * CPR + k];
                if constexpr (SPLIT) {
                    double2 d = *reinterpret_cast<double2*>(&w);
                    d.x = scale_pow2(d.x, -k0);
                    d.y = scale_pow2(d.y, -k1);
                    w = *reinterpret_cast<uint4*>(&d);
                }
                VT* dst;
                if (r < own) {
                    dst = V + (size_t)(rows[r] & kDofMask) * a.ld + cc;
                } else {
                    dst = PV + (size_t)(pv0 + r - own) * R + cc;
                }
                *reinterpret_cast<uint4*>(dst) = w;
            }
        __syncwarp();
    }
    allow_dependent_launch();
}

// V rows of DoFs of several patches: their rows of the combine buffer added in
// patch order; a thread owns 16 bytes of a row.
template <typename VT>
__global__ void __launch_bounds__(256) k_bpatch_combine(VT* __restrict__ V, const VT* PV,
                                                        const uint32_t* __restrict__ dof,
                                                        const uint32_t* __restrict__ off,
                                                        const uint32_t* __restrict__ idx, uint32_t n, uint32_t R,
                                                        uint32_t ld) {
    constexpr uint32_t EPC = 16 / sizeof(VT);
    const uint32_t cpr = R / EPC;
    const uint64_t q = (uint64_t)blockIdx.x * 256 + threadIdx.x;
    const uint32_t i = (uint32_t)(q / cpr), k = (uint32_t)(q % cpr) * EPC;
    const bool live = i < n;
    const uint32_t d = live ? __ldg(dof + i) : 0u;
    const uint32_t k0 = live ? __ldg(off + i) : 0u, k1 = live ? __ldg(off + i + 1) : 0u;
    constexpr uint32_t kAhead = 8;  // (the lists are constant: the first entries load before the wait)
    uint32_t at[kAhead];
#pragma unroll
    for (uint32_t j = 0; j < kAhead; j++) at[j] = k0 + j < k1 ? __ldg(idx + k0 + j) : 0u;
    wait_prior_grid();
    if (!live) return;
    VT s[EPC] = {};
    for (uint32_t e = k0; e < k1; e += kAhead) {
        if (e != k0) {
#pragma unroll
            for (uint32_t j = 0; j < kAhead; j++) at[j] = e + j < k1 ? __ldg(idx + e + j) : 0u;
        }
        uint4 x[kAhead];
#pragma unroll
        for (uint32_t j = 0; j < kAhead; j++)
            if (e + j < k1) x[j] = __ldcg(reinterpret_cast<const uint4*>(PV + (size_t)at[j] * R + k));
#pragma unroll
        for (uint32_t j = 0; j < kAhead; j++) {
            if (e + j >= k1) continue;
            VT y[EPC];
            memcpy(y, &x[j], 16);
#pragma unroll
            for (uint32_t q = 0; q < EPC; q++) s[q] = s[q] + y[q];
        }
    }
    uint4 w;
    memcpy(&w, s, 16);
    *reinterpret_cast<uint4*>(V + (size_t)d * ld + k) = w;
}

struct BTile {
    void* fn;
    uint32_t cb;  // columns of a task
};

// The lane tiles of an element size, widest first.
void tiles(uint32_t n, bool f32, BTile out[2], int* count) {
    *count = 0;
    auto put = [&](void* fn, uint32_t cb) { out[(*count)++] = {fn, cb}; };
    if (f32) {
        if (n == 24) {
            put((void*)k_bpatch<24, 6, 4, false>, 32);
            put((void*)k_bpatch<24, 6, 2, false>, 16);
        } else if (n == 30) {
            put((void*)k_bpatch<30, 8, 4, false>, 32);
            put((void*)k_bpatch<30, 8, 2, false>, 16);
        } else if (n == 60) {
            put((void*)k_bpatch<60, 16, 4, false>, 32);
            put((void*)k_bpatch<60, 16, 2, false>, 16);
        }
    } else if (n == 24) {
        put((void*)k_bpatch<24, 6, 2, true>, 16);
    } else if (n == 30) {
        put((void*)k_bpatch<30, 8, 2, true>, 16);
    }
}

}  // namespace

bool bpatch_supported(uint32_t n, bool f32) {
    BTile t[2];
    int count = 0;
    tiles(n, f32, t, &count);
    return count > 0;
}

cudaError_t configure_bpatch() {
    for (uint32_t n : {24u, 30u, 60u})
        for (int f = 0; f < 2; f++) {
            BTile t[2];
            int count = 0;
            tiles(n, f != 0, t, &count);
            for (int i = 0; i < count; i++) {
                const cudaError_t e = cudaFuncSetAttribute(t[i].fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                           (int)kSmemBudget);
                if (e != cudaSuccess) return e;
            }
        }
    return cudaSuccess;
}

cudaError_t launch_bpatch(const BPatchGeom& g, const BPatchArgs& a, bool f32, const uint32_t* shared_dof,
                          const uint32_t* shared_off, const uint32_t* shared_idx, int sm_count,
                          cudaStream_t st) {
    if (g.patches == 0) return cudaSuccess;
    BTile t[2];
    int count = 0;
    tiles(g.n, f32, t, &count);
    if (!count) return cudaErrorInvalidValue;
    const uint32_t vt = f32 ? 4 : 8;
    uint32_t ke_bytes = f32 ? g.n * g.n * 4 : 2 * a.plane * 4;
    // the narrowest tile that covers the columns, else the widest
    int pick = 0;
    while (pick + 1 < count && t[pick + 1].cb >= a.nrhs) pick++;
    const BPatchSmem L(g, t[pick].cb, vt, ke_bytes);
    uint32_t ncb = (a.nrhs + t[pick].cb - 1) / t[pick].cb;
    const uint64_t tasks = (uint64_t)g.patches * ncb;
    if (tasks > 0xffffffffull) return cudaErrorInvalidConfiguration;
    uint32_t W = std::min<uint32_t>((uint32_t)kBPatchWarps, kSmemBudget / L.total);
    if (W == 0) return cudaErrorInvalidConfiguration;
    W = std::min<uint32_t>(W, (uint32_t)((tasks + sm_count - 1) / sm_count));  // few tasks: over every SM first
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::min<uint64_t>((uint64_t)sm_count, (tasks + W - 1) / W));
    cfg.blockDim = dim3(W * 32);
    cfg.dynamicSmemBytes = W * L.total;
    cfg.stream = st;
    BPatchArgs args = a;
    BPatchGeom geom = g;
    void* params[] = {&args, &geom, &ke_bytes, &ncb};
    cudaError_t e = cudaLaunchKernelExC(&cfg, t[pick].fn, params);
    if (e != cudaSuccess || g.shared == 0) return e;
    const uint64_t threads = (uint64_t)g.shared * (a.nrhs * vt / 16);
    cfg.gridDim = dim3((unsigned)((threads + 255) / 256));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (f32)
        return cudaLaunchKernelEx(&cfg, k_bpatch_combine<float>, static_cast<float*>(a.v),
                                  static_cast<const float*>(a.pv), shared_dof, shared_off, shared_idx, g.shared, a.nrhs,
                                  a.ld);
    return cudaLaunchKernelEx(&cfg, k_bpatch_combine<double>, static_cast<double*>(a.v),
                              static_cast<const double*>(a.pv), shared_dof, shared_off, shared_idx, g.shared, a.nrhs,
                              a.ld);
}

}  // namespace afm
