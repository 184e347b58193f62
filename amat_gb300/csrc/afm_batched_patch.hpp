// Patch plan of the batched product (afm_batched_patch.cu): compact groups of
// elements of one size whose rows of V are summed in shared memory.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "afm_internal.hpp"

namespace afm {

constexpr uint32_t kBPatchElems = 8;  // elements per patch, at most
// rows (local DoFs) per patch, at most: 2 x 2 x 2 linear bricks have 81; one hex20 element has 60
constexpr uint32_t kBPatchRows = 128;
AFM_HD inline uint32_t bpatch_max_rows(uint32_t n) { return n <= 32 ? 96u : kBPatchRows; }

// One patch's block in the plan (hdr_bytes apart, 16-byte aligned):
//   uint32 {elements, rows, rows of this patch alone, first row of the others in the combine buffer}, 4 words free,
//   uint32 arena position of each element (kBPatchElems words),
//   uint32 global DoF of each row (kBcFlag on constrained ones), rows of this patch alone first,
//   uint8 local row of each element's DoFs (n per element).
struct BPatchGeom {
    uint32_t n = 0, patches = 0, max_rows = 0, hdr_bytes = 0;
    uint32_t pv_rows = 0;   // rows of the combine buffer
    uint32_t shared = 0;    // DoFs of several patches
};
AFM_HD inline uint32_t bpatch_rows_off() { return 32u + 4u * kBPatchElems; }
AFM_HD inline uint32_t bpatch_loc_off(uint32_t max_rows) { return bpatch_rows_off() + 4u * max_rows; }
AFM_HD inline uint32_t bpatch_hdr_bytes(uint32_t n, uint32_t max_rows) {
    return (bpatch_loc_off(max_rows) + kBPatchElems * n + 15u) & ~15u;
}

struct BPatchPlanHost {
    BPatchGeom geom;
    std::vector<unsigned char> hdr;
    std::vector<uint32_t> shared_dof, shared_off, shared_idx;  // combine lists: DoF, offsets, buffer rows
};

// The plan of n_elem elements of n DoFs each (perm[p]: the element at position p
// of the arena; color_first: its colours' first positions, and n_elem; is_bc:
// constrained DoFs).
void build_bpatch_plan(uint32_t n_elem, uint32_t n_dofs, uint32_t n, const uint32_t* map, const uint32_t* perm,
                       const std::vector<uint32_t>& color_first, const uint8_t* is_bc, BPatchPlanHost& out);

struct BPatchArgs {
    const unsigned char* hdr;
    const unsigned char* ke;
    uint64_t unit_bytes;      // stride between element matrices
    uint32_t plane;           // split arena: entries per plane
    const void* u;
    void* v;
    void* pv;                 // combine buffer, pv_rows x nrhs
    uint32_t nrhs, ld;
    int bc_mode;
    const unsigned long long* umax;  // split arithmetic: max|U(:, j)| per column (double bits)
};

// Whether the kernel takes elements of n DoFs in this arithmetic (f32: FP32
// products from an FP32 arena or the hi plane; else the split products).
bool bpatch_supported(uint32_t n, bool f32);
// V = K U: the patch launch and the combine pass (V rows of DoFs that no
// element lists are not written).
cudaError_t launch_bpatch(const BPatchGeom& g, const BPatchArgs& a, bool f32, const uint32_t* shared_dof,
                          const uint32_t* shared_off, const uint32_t* shared_idx, int sm_count,
                          cudaStream_t st);
cudaError_t configure_bpatch();

}  // namespace afm
