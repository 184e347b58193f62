// Internal types shared by the host runtime (afm_capi.cpp) and the CUDA
// kernels (afm_kernels.cu, afm_solver.cu) of the GB300 AFM operator.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <string>
#include <vector>

#include "../../include/afm.h"

namespace afm {

// Kernel regimes, picked per element size n.
//   TPE (thread per element, n <= kTpeMaxN): 32 elements of one colour form a
//       unit; the unit's Ke is stored entry-major [k][32] so that lane l reads
//       entry k of element l; map [i][32].
//   WPE (warp per element, n > kTpeMaxN): one element per unit; its Ke is
//       stored column-major so lane r reads row r of column c; map [i].
enum Regime : int { REG_TPE = 0, REG_WPE = 1 };
constexpr uint32_t kTpeMaxN = 16;
constexpr uint32_t kTpeWidth = 32;
constexpr uint32_t kMaxN = 96;           // largest element supported (3 rows per lane)
constexpr uint32_t kBcFlag = 0x80000000u;  // map bit: DoF is constrained
constexpr uint32_t kDofMask = 0x7fffffffu;
// Patch index blocks also flag DoFs that more than one patch lists (their sums
// go through the combine pass), so their DoF ids keep 30 bits.
constexpr uint32_t kSharedFlag = 0x40000000u;
constexpr uint32_t kPatchDofMask = 0x3fffffffu;

// Device error flags (bit set in err[0]); err[1..6] record the first failed
// bounds check (kind, block, thread and three values); kErrWords ints in all.
constexpr int kErrTimeout = 1;
constexpr int kErrBounds = 2;
constexpr int kErrWords = 8;  // the last word is never written: the flag of afm_set_wait_probe

// One launch of the matvec: the elements of one colour that share n.
struct Segment {
    uint32_t color = 0;
    uint32_t n = 0;
    int regime = REG_WPE;
    uint64_t first_pos = 0;   // first element position (colour-sorted order)
    uint32_t count = 0;       // elements
    uint32_t units = 0;       // work units (TPE: ceil(count/32), WPE: count)
    uint64_t ke_offset = 0;   // byte offset of the first unit in the Ke arena
    uint64_t unit_bytes = 0;  // arena bytes per unit (16-byte multiple)
    uint64_t map_offset = 0;  // uint32 offset of the first unit in the map
    uint32_t plane = 0;       // FP64_SPLIT: entries per plane of a unit (the lo plane follows the hi plane)
    uint64_t sym_offset = 0;     // byte offset of the first unit in the symmetric inner arena
    uint64_t sym_unit_bytes = 0; // its bytes per unit (0: no symmetric form)
    uint64_t blk_offset = 0;     // byte offset of the first unit in the arena of block units
    uint32_t sym_plane = 0;      // entries of a unit's FP32 plane before its BF16 correction plane (0: none)
};

// Colours of one fused (cooperative) launch of the warp-group kernel, at most.
constexpr uint32_t kMaxFusedColours = 48;

// Arguments of one segment launch.
struct SegArgs {
    const unsigned char* ke;  // arena + segment offset
    const uint32_t* map;      // map + segment offset
    const void* u;            // double* or float*
    void* v;                  // double* or float*
    uint32_t units;
    uint32_t count;           // elements (TPE: last unit may be partial)
    uint64_t unit_bytes;      // stride between units in the arena
    uint32_t copy_bytes;      // bytes copied per unit (the hi plane only for FP32 on a split arena)
    uint32_t plane;           // entries per plane (split arena)
    int bc_mode;              // 1: constrained columns read as zero (MatMult_mf)
    int* err;
    const unsigned long long* umax;  // split arithmetic: max|u| (bits of a non-negative double)
    unsigned long long wait_ns;  // limit of each pipeline wait (afm_set_wait_limit)
    const int* probe;         // test hook: a flag nothing sets, or null (afm_set_wait_probe)
    void* ve = nullptr;       // warp-group kernel: element products go here (VO, n per element in arena order)
                              // for the gather pass (launch_gather_sum); null: added to v, one launch per colour
};

// Arguments of one batched (multi right-hand side) segment launch.
struct BatchArgs {
    const unsigned char* ke;
    const uint32_t* map;
    const void* u;  // n_dofs x ld, row-major
    void* v;
    uint32_t units, count;
    uint64_t unit_bytes;
    uint32_t copy_bytes, plane;
    uint32_t nrhs, ld;
    int bc_mode;
    int* err;
    uint32_t n_dofs;      // rows of U and V (bounds checks)
    uint32_t smem_total;  // dynamic shared memory of the launch (bounds checks)
    const unsigned long long* umax;  // split arithmetic: max|U(:, j)| per column j (double bits)
    unsigned long long wait_ns;  // limit of each pipeline wait
    const int* probe;         // test hook: a flag nothing sets, or null (afm_set_wait_probe)
};

// ---- patch path (small elements) -----------------------------------------
// Elements with at most kPatchMaxN DoFs (all of one size, no DoF listed twice
// in an element) run as patches: compact groups of up to kPatchElems elements,
// coloured so that patches of one colour share no DoF (see afm_patch.cuh).
constexpr uint32_t kPatchMaxN = 12;
constexpr uint32_t kPatchMaxDofs = 1024;  // local DoFs per patch (uint16 indices)

constexpr uint32_t kNoElement = 0xffffffffu;  // empty element slot

#ifdef __CUDACC__
#define AFM_HD __host__ __device__
#else
#define AFM_HD
#endif
// Byte offsets inside one patch index block (all 16-byte aligned): glob
// (uint32 x ndof), lmap (uint16 x units x n x 32), csr_off (uint16 x ndof+1),
// slot (uint16 x contributions).
AFM_HD inline uint32_t patch_r16(uint32_t x) { return (x + 15u) & ~15u; }
AFM_HD inline uint32_t patch_lmap_off(uint32_t ndof) { return patch_r16(ndof * 4u); }
AFM_HD inline uint32_t patch_csr_off(uint32_t ndof, uint32_t units, uint32_t n) {
    return patch_lmap_off(ndof) + units * n * 64u;
}
AFM_HD inline uint32_t patch_slot_off(uint32_t ndof, uint32_t units, uint32_t n) {
    return patch_csr_off(ndof, units, n) + patch_r16((ndof + 1u) * 2u);
}

// One patch: its Ke units and its index block (both 16-byte aligned).
struct PatchDesc {
    uint64_t ke_off;     // bytes into the Ke arena (unit0 x its unit size)
    uint64_t idx_off;    // bytes into the index arena
    uint32_t units;      // units of 32 element slots
    uint32_t ndof;       // local DoFs
    uint32_t idx_bytes;  // size of the index block (16-byte multiple)
    uint32_t elems;      // elements (the rest of the slots are empty)
    uint32_t unit0;      // first unit of the patch, in units of any arena
    uint32_t pv_off;     // first entry of the patch's local DoF sums in the combine buffer
};

// Arguments of one patch-colour launch.
struct PatchArgs {
    const PatchDesc* desc;    // the colour's first patch
    uint32_t count;           // patches of the colour
    const unsigned char* ke;  // Ke arena
    const unsigned char* idx; // index arena
    const void* u;
    void* v;
    uint64_t unit_bytes;      // stride between units
    uint32_t copy_bytes;      // bytes copied per unit (hi plane only for FP32 on a split arena)
    uint32_t plane;           // entries per plane (split arena)
    int bc_mode;
    int* err;
    void* pv;                 // one launch for every colour: sums of shared DoFs go here (VO), others to v;
                              // null: one launch per colour, every sum added to v
    int u_dep;                // u comes from the launch before: wait for it before reading
    int set_rows;             // one launch: v_c = u_c on constrained DoFs of one patch (u_rows has v's entry type)
    const void* u_rows;
    unsigned long long wait_ns;  // limit of each pipeline wait
    const int* probe;         // test hook: a flag nothing sets, or null (afm_set_wait_probe)
};

// Patch launch geometry shared by all colours of an operator.
struct PatchPlanGeom {
    uint32_t n = 0;           // DoFs per element
    uint32_t max_slots = 0;   // largest patch, in element slots (32 x units)
    uint32_t max_ndof = 0;    // largest local DoF count
    uint32_t max_idx = 0;     // largest index block, bytes
};

cudaError_t launch_patches(int prec, const PatchPlanGeom& pg, const PatchArgs& a, int sm_count, bool pdl,
                           cudaStream_t stream);
// The combine pass of one-launch patches: v[dof[i]] = sum over k in
// [off[i], off[i+1]) of pv[idx[k]], in order (vo_bytes 8: double, 4: float);
// where dof[i] carries kBcFlag and u_rows is not null, v = u_rows instead.
// Launched with programmatic dependence on the patch launch.
cudaError_t launch_patch_combine(int vo_bytes, void* v, const void* pv, const uint32_t* dof, const uint32_t* off,
                                 const uint32_t* idx, uint32_t nb, const void* u_rows, cudaStream_t st);
// The gather pass of a plan whose elements run in one launch: v[d] = sum over
// k in [off[m], off[m + 1]) of ve[idx[k] + d - b m], in order, m = d / b (b =
// 3: the map lists whole nodes of three consecutive DoFs; b = 1: one list per
// DoF); where mask is not null and mask[d] != 0, v[d] = u[d] instead. ve holds
// ve_bytes-wide entries, v and u vt_bytes-wide ones (8 and 8, 8 and 4, 4 and
// 4). part not null: also the partials of v.u, *nb of them. Launched with
// programmatic dependence on the element launch.
cudaError_t launch_gather_sum(int ve_bytes, int vt_bytes, uint32_t b, void* v, const void* ve, const uint32_t* off,
                              const uint32_t* idx, uint32_t n_dofs, const void* u, const uint8_t* mask, double* part,
                              uint32_t* nb, cudaStream_t st);
// The combine pass over every DoF (constrained rows as with u_rows = u), with
// the partials of v.u, *nb of them; pos[d]: the DoF's place in the combine
// lists, or kNoElement.
cudaError_t launch_patch_combine_dot(int vo_bytes, void* v, const void* pv, const uint32_t* pos, const uint32_t* dof,
                                     const uint32_t* off, const uint32_t* idx, uint32_t n, const void* u, double* part,
                                     uint32_t* nb, cudaStream_t st);
// Shared memory of a patch launch (0 if it does not fit).
size_t patch_smem_bytes(int prec, const PatchPlanGeom& pg, uint32_t copy_bytes);

// Arguments of one matrix-free (method 2) launch: the elements first ..
// first + count - 1 of the colour-sorted order (one colour).
struct FreeArgs {
    const void* xe;        // node coordinates, element-major (nodes x 3), double or float
    const uint32_t* map;   // n DoFs per element (kBcFlag on constrained DoFs)
    const void* ref;       // dN of every node at every quadrature point ([q][node][3]), the q weights, the q points
    const void* u;
    void* v;
    uint32_t first, count, nq;
    int bc_mode;
    double lam, mu;        // Lame parameters (elasticity)
    void* ve = nullptr;    // element products go here for the gather pass; null: added to v, one launch per colour
};
cudaError_t launch_free(int kind, bool f32, const FreeArgs& a, int sm_count, cudaStream_t st);

// Kernel arithmetic for FP32 products from the symmetric inner arena (an
// internal value beside the afm_precision codes).
constexpr int kPrecF32Sym = 16;
// ... and from the symmetric inner arena with its BF16 correction plane.
constexpr int kPrecF32SymX = 17;
// FP64 vectors, double-float products from that corrected arena (ArithSplitSymX).
constexpr int kPrecSplitSymX = 18;
// The corrected arena on FP32 u with FP32 row sums and FP64 v (ArithF32SymC).
constexpr int kPrecF32SymC = 19;

// FP64 vectors, the split arithmetic on packed symmetric patch units (ArithSplitSym).
constexpr int kPrecSplitSym = 20;
// ... and on symmetric element units of 2 x 2 blocks (ArithSplitBlk).
constexpr int kPrecSplitBlk = 21;
// Bytes of such a unit (0: no block kernel for this size): n/4 + 1 (rounded down) wrapped diagonals of n/2 blocks with
// 4 hi and 4 lo entries each, and for all but the first and the last the 4 lo entries of the transposed block.
constexpr uint32_t split_block_bytes(uint32_t n) {
    return n == 60 ? ((n / 4 + 1) * 32 + (n / 4 - 1) * 16) * (n / 2) : 0u;
}
// The lo part of K(c, r) in a block unit, beside the hi part of K(r, c) (h): what is left of the split pair (th, tl) of
// K(c, r), which is tl itself where the two hi parts agree.
AFM_HD inline float split_transposed(float h, float th, float tl) {
    return (float)(((double)th - (double)h) + (double)tl);
}
// Whether such a unit holds K(c, r) as the split pair does: to 2^-48 of itself, and as a leading part with a low part
// below its last place (2^-23 of it: the products round a low part to 24 bits and leave out its product with u's low
// part). Not where the rounding of the quadrature sums (2^-57 of the diagonal) is no small part of the entry: entries
// below 2^-34 of the diagonal, the zeros of regular meshes above all, and in jittered ones (15 x of the entries are below
// x of the diagonal) one in 1e9 or so. Such pairs are left out of the units and added by a pass of their own
// (launch_add_pairs).
AFM_HD inline bool block_holds(float h, float th, float tl) {
    if (h == th) return true;
    const double t = ((double)th - (double)h) + (double)tl;
    const float l = (float)t;
    return fabs(t - (double)l) <= 0x1p-49 * fabs((double)th) && fabs((double)l) <= 0x1p-23 * fabs((double)th);
}
// Whether a block unit stores entry (r, c) itself, its transpose beside it (1), as the transpose of (c, r) (-1), or both
// (0: the first and the last wrapped diagonal).
inline int block_side(uint32_t r, uint32_t c, uint32_t n) {
    const uint32_t nb = n / 2, d = (c / 2 + nb - r / 2) % nb;
    return d == 0 || d == nb / 2 ? 0 : d < nb / 2 ? 1 : -1;
}
// Pairs left out of block units, at most one in this many elements (a regular mesh has 84 an element: whole matrices).
constexpr uint32_t kElemsPerLoosePair = 8;
// v[row[i]] += the sum over k in [off[i], off[i + 1]) of val[k] u[col[k]], in order (bc_mode: constrained columns, kBcFlag
// in col, as zero).
cudaError_t launch_add_pairs(double* v, const double* u, const uint32_t* row, const uint32_t* off, const uint32_t* col,
                             const double* val, uint32_t rows, int bc_mode, cudaStream_t st);
// Elements per SM from which a plan takes block units (20 consumer warps hold 5 elements of an SM, so that below about ten
// each the ramps are most of the time): hex20 elasticity with 1000 elements 10.9 us on whole units, 10.9 on blocks; 1331
// 13.5 and 13.0; 1440 14.2 and 13.3; 1584 15.3 and 14.0; 2744 20.2 and 16.9.
constexpr uint32_t kBlockElemsPerSm = 10;
// Packs a segment's split units into block units (afm_mv_splitblk.cu).
cudaError_t pack_split_blocks(const unsigned char* ke, uint64_t unit_bytes, uint32_t plane, uint32_t n, uint32_t units,
                              unsigned char* dst, int sm_count, cudaStream_t st);

// Packs a patch plan's split units (afm_mv_splitsym.cu).
cudaError_t pack_split_units(const unsigned char* ke, uint32_t n, uint32_t units, unsigned char* packed, int sm_count,
                             cudaStream_t st);

// Fills segment s's part of the symmetric inner arena from its split-arena
// units (afm_mv_f32sym.cu).
cudaError_t build_sym_segment(const Segment& s, const unsigned char* ke, unsigned char* sym, int sm_count,
                              cudaStream_t st);

// Launches one segment on stream. prec: afm_precision (FP64, FP64_SPLIT, FP32)
// or kPrecF32Sym.
// pdl: allow the launch to begin while the previous kernel on the stream
// drains (programmatic dependent launch; v is touched only after it ends).
cudaError_t launch_segment(const Segment& s, int prec, const SegArgs& a, int sm_count, bool dup_in_element, bool pdl,
                           cudaStream_t stream);
// Dynamic shared memory the launch of segment s uses (for reporting).
size_t segment_smem_bytes(const Segment& s, int prec);

// ---- serving lane (afm_lane.cu) ---------------------------------------------
// One launch advances the FP32 CG recursion of many served solves at once:
// every request is one thread-block cluster of kLaneCtas CTAs that runs whole
// CG iterations (colour-ordered FP32 products on the hi plane of the split
// arena, dot products, vector updates) with cluster barriers between phases.
constexpr uint32_t kLaneCtas = 8;
constexpr uint32_t kLaneThreads = 512;

// One colour-size segment of a request, as the lane reads it.
struct LaneSeg {
    const float* ke;        // hi plane of the segment's first unit
    const uint32_t* map;    // the segment's map (kBcFlag on constrained DoFs)
    uint64_t unit_floats;   // floats from one unit to the next
    uint32_t n, regime, units, count;
    uint32_t sync_after;    // 1: the last segment of its colour (a cluster barrier follows)
    uint32_t pad;
};

// One request's FP32 recursion: the vectors of its solve (float, n_dofs) and
// its solver scalars on the device.
struct LaneJob {
    float *x, *r, *z, *p, *q;
    const float* dinv;
    const uint8_t* bcmask;  // 1 on constrained DoFs (q = p there), or null
    const LaneSeg* segs;
    double* sc;
    int* err;
    uint32_t n_dofs, n_segs;
};

// Runs at most iters CG iterations of each of the n_jobs requests (a request
// whose S_DONE is set does nothing), then writes every request's scalars to
// its sc.
cudaError_t launch_lane(const LaneJob* d_jobs, uint32_t n_jobs, uint32_t iters, cudaStream_t st);

// Replaces the operator's stream by one of the given priority (lower numbers
// run first, cudaDeviceGetStreamPriorityRange), after the old stream's work
// has finished. Call before any solve has captured work on the stream.
int set_stream_priority(afm_operator* op, int priority);

// Records the calling thread's last error message (returned by
// afm_last_error) and returns status.
int set_error(int status, const char* fmt, ...);


}  // namespace afm

// The operator handle.
struct afm_operator {
    int device = 0;
    int bc_method = AFM_BC_IMATRIX;
    int matfree_type = 1;
    int precision_req = AFM_PREC_AUTO;
    int precision = AFM_PREC_FP64;
    cudaStream_t stream = nullptr;
    int sm_count = 0;

    // maps (single rank: local == global)
    bool have_map = false;
    uint32_t n_elem = 0, n_dofs = 0, nmax = 0;
    std::vector<uint32_t> offsets;  // n_elem + 1
    std::vector<uint32_t> map;      // global DoF ids
    bool dup_in_element = false;    // some element lists a DoF twice
    uint32_t n_unlisted = 0;        // DoFs that no element lists (decided at finalize)
    int patch_mode = 1;             // small elements: patches, 1 one launch + combine pass when the patch colours
                                    // are small, else one launch per colour; 2 always per colour; 3 always one
                                    // launch; 0 colour segments
    bool patch_one_launch = false;  // the choice made at finalize

    // boundary conditions
    std::vector<uint64_t> constrained;
    std::vector<double> values;
    std::vector<uint32_t> bc_unique;  // sorted unique constrained ids

    // element matrices, host copy (row-major, reference layout)
    std::vector<uint64_t> kofs;     // n_elem + 1, entries
    std::vector<double> ke;
    bool ke_dirty = true;

    // finalize products
    bool finalized = false;
    std::vector<uint32_t> colors;
    uint32_t n_colors = 0;
    std::vector<uint32_t> perm;     // position -> element id
    std::vector<afm::Segment> segs;
    double trace = 0.0;
    std::vector<double> diag_host;  // Jacobi diagonal with BC rows

    // device state
    unsigned char* d_ke = nullptr;
    size_t ke_bytes = 0;
    uint32_t* d_map = nullptr;       // DoF map, constrained DoFs carry kBcFlag
    size_t map_bytes = 0;
    double* d_diag = nullptr;
    uint32_t* d_bc_idx = nullptr;    // constrained ids in reference order
    double* d_bc_val = nullptr;
    uint32_t n_bc = 0;
    int* d_err = nullptr;
    unsigned long long wait_ns = 4000000000ull;  // limit of each kernel pipeline wait (afm_set_wait_limit)
    bool wait_probe = false;         // afm_set_wait_probe
    int fail_skip = 0, fail_allocs = 0;  // afm_debug_fail_allocations
    unsigned long long* d_usc = nullptr;  // u-scale words of the split products (kUscWords, afm_solver.hpp), and as
                                          // many for products recorded in callers' graphs
    uint8_t* d_bcmask = nullptr;     // 1 per constrained DoF (null without constraints)
    // one cooperative launch for every colour of a split product (segment plans of one element size)
    bool fused_ok = false;           // the plan allows it (decided at finalize)
    bool fused = false;              // afm_set_fused_colours (off: measured slower than the colour launches)
    unsigned* d_gbar = nullptr;      // grid-barrier counters of the fused launch
    std::vector<int> trace_iters;    // the last mixed solve: inner iterations at each FP64 residual
    std::vector<double> trace_res;   // ... and that residual over ||b||
    double* d_work = nullptr;        // host-API staging and solver vectors
    size_t work_elems = 0;
    double* d_scalars = nullptr;     // solver scalars / reduction partials
    double* h_scalars = nullptr;     // pinned mirror
    float* d_work32 = nullptr;       // mixed-precision inner vectors
    size_t work32_elems = 0;
    double* d_work64i = nullptr;     // inner vectors of the FP64-vector mixed solve (symmetric inner format 3)
    size_t work64i_elems = 0;

    // captured CG iteration graphs (FP64 and FP32 inner), keyed by buffers
    struct CgGraph {
        cudaGraphExec_t exec = nullptr;
        const void* key[6] = {};
        int batch = 0;
        uint64_t gen = 0;
    };
    CgGraph cg64, cg32, cg64i, bcg64, bcg32;
    uint64_t generation = 0;  // bumped whenever device buffers are released

    // symmetric inner arena: FP32 element matrices with each symmetric pair of
    // entries stored once, built from the split arena on the first FP32 product
    bool ke_symmetric = false;      // every Ke symmetric to 1e-6 of its largest diagonal entry
    bool ke_sym_exact = false;      // every Ke equal to its transpose bit for bit
    uint64_t loose_pairs = 0;       // pairs of symmetric Ke of 60 DoFs that block units do not hold (block_holds)
    // ... and their entries, where the plan has block units: per row (DoF) its columns and values, row by row
    uint32_t n_loose_rows = 0;
    uint32_t* d_loose_row = nullptr;
    uint32_t* d_loose_off = nullptr;
    uint32_t* d_loose_col = nullptr;
    double* d_loose_val = nullptr;
    // the split units of a patch plan with exactly symmetric Ke, packed, or of a segment plan with Ke of 60 DoFs symmetric
    // up to rounding, as block units (FP64 products read them; null: they read d_ke)
    unsigned char* d_packed = nullptr;
    bool sym_ok = false;            // symmetric, split arena, and a layout the symmetric kernels cover
    int sym_mode = 1;               // afm_set_symmetric_inner: 0 off, 1 FP32, 2 FP32 + BF16 correction
    int sym_built = 0;              // format of d_sym (1 or 2; 0: not built)
    unsigned char* d_sym = nullptr;
    size_t sym_bytes = 0;
    double* d_vx = nullptr;         // format 2: FP64 product before its rounding to FP32 (n_dofs)

    // matrix-free operator (method 2, MATFREE_TYPE::FREE): element kind, material, quadrature and
    // node coordinates; on the device, coordinates and maps in colour order and the reference tables
    int elem_kind = -1;
    double elem_E = 1.0, elem_nu = 0.3;
    uint32_t elem_ngt = 2, elem_nodes = 0;
    std::vector<double> xe;         // n_elem x nodes x 3
    std::vector<uint32_t> free_color_first;  // colour offsets into the colour-sorted elements
    uint32_t free_nq = 0;
    double* d_free_xe64 = nullptr;
    float* d_free_xe32 = nullptr;
    double* d_free_ref64 = nullptr;
    float* d_free_ref32 = nullptr;

    // assembled operator (afm_assembled.cpp): CSR on the device
    uint64_t* d_csr_rp = nullptr;
    uint32_t* d_csr_cols = nullptr;
    double* d_csr_vals = nullptr;
    uint64_t csr_nnz = 0;
    int csr_width = 32;             // threads per row of the SpMV

    // patch path (small elements): patches in colour order
    bool use_patches = false;
    afm::PatchPlanGeom patch_geom;
    std::vector<uint32_t> patch_color_first;  // n_patch_colors + 1 offsets into the patch list
    uint32_t n_patches = 0;
    afm::PatchDesc* d_patch_desc = nullptr;
    unsigned char* d_patch_idx = nullptr;
    size_t patch_idx_bytes = 0;
    // one-launch patches: local sums of shared DoFs (pv_count entries of 8 bytes) and, per shared DoF,
    // the list of its entries in patch order
    size_t pv_count = 0;
    uint32_t n_shared = 0;
    std::vector<uint32_t> shared_dof, shared_off, shared_idx;  // host copies (finalize)
    double* d_pv = nullptr;
    uint32_t* d_shared_dof = nullptr;
    uint32_t* d_shared_off = nullptr;
    uint32_t* d_shared_idx = nullptr;
    uint32_t* d_shared_pos = nullptr;  // per DoF: its place in the shared lists, or kNoElement

    // one launch for every element (plans of one element size): the element products go to d_ve and a gather
    // pass sums each DoF's entries in arena (colour) order
    uint32_t gather_b = 0;          // DoFs per list of the gather pass (0: the plan has none)
    double* d_ve = nullptr;            // owns the lists too
    uint32_t* d_gather_idx = nullptr;
    uint32_t* d_gather_off = nullptr;
    // order of products on several streams (take_turn): 1 + the id of the stream of the last product (0: the operator's
    // own stream, or none yet), and the end of that product where the stream is a caller's
    unsigned long long turn_id = 0;
    cudaEvent_t turn_event = nullptr;
    bool own_capture = false;          // the operator's solver is capturing its iterations on `stream`

    // batched (multi right-hand side) state
    double* d_bwork = nullptr;
    size_t bwork_elems = 0;
    double* d_bsc = nullptr;        // per-column scalars and column partials
    size_t bsc_elems = 0;
    unsigned int* d_bremain = nullptr;
    unsigned int* h_bremain = nullptr;
    struct BatchTune {
        uint64_t key;
        int tr, ng;  // lane tile of the launches per colour: columns, rows
        float ms;
        bool patch = false;  // the patch plan beats every tile (ms is its time then)
    };
    // patch plan of the batched product (afm_batched_patch.hpp), built by the first batched call that can use it
    int bp_mode = 1;                // afm_set_batch_patches
    int bp_state = 0;               // 0 not looked at, 1 built, -1 none
    uint32_t bp_n = 0, bp_patches = 0, bp_max_rows = 0, bp_pv_rows = 0, bp_shared = 0;
    unsigned char* d_bp_hdr = nullptr;
    uint32_t* d_bp_dof = nullptr;
    uint32_t* d_bp_off = nullptr;
    uint32_t* d_bp_idx = nullptr;
    unsigned char* d_bp_pv = nullptr;  // combine buffer
    size_t bp_pv_bytes = 0;
    std::vector<BatchTune> batch_tune;  // autotuner choices
};
