// Host side of the batched product's patch plan (afm_batched_patch.hpp).
#include <algorithm>
#include <cstring>
#include <utility>

#include "afm_batched_patch.hpp"

namespace afm {

void build_bpatch_plan(uint32_t n_elem, uint32_t n_dofs, uint32_t n, const uint32_t* map, const uint32_t* perm,
                       const std::vector<uint32_t>& color_first, const uint8_t* is_bc, BPatchPlanHost& out) {
    std::vector<uint32_t> pos(n_elem);
    for (uint32_t p = 0; p < n_elem; p++) pos[perm[p]] = p;
    // whole nodes of three consecutive DoFs where the map lists them, else single DoFs
    int nodes3 = n % 3 == 0 && n_dofs % 3 == 0;
#pragma omp parallel for schedule(static) reduction(&& : nodes3)
    for (int64_t k = 0; k < (int64_t)((uint64_t)n_elem * n / 3); k++) {
        if (!nodes3) continue;
        const uint32_t* m = map + 3 * k;
        nodes3 = m[0] % 3 == 0 && m[1] == m[0] + 1 && m[2] == m[0] + 2;
    }
    const uint32_t b = nodes3 ? 3 : 1, per = n / b, nodes = n_dofs / b;
    const uint32_t max_nodes = bpatch_max_rows(n) / b;
    // node -> elements, colour by colour: elements of one colour share no node
    std::vector<uint32_t> off((size_t)nodes + 1, 0), n2e((size_t)n_elem * per);
    for (int pass = 0; pass < 2; pass++) {
        std::vector<uint32_t> fill(off.begin(), off.end() - 1);
        for (size_t c = 0; c + 1 < color_first.size(); c++) {
#pragma omp parallel for schedule(static)
            for (int64_t p = color_first[c]; p < (int64_t)color_first[c + 1]; p++) {
                const uint32_t e = perm[p];
                for (uint32_t j = 0; j < per; j++) {
                    const uint32_t m = map[(uint64_t)e * n + j * b] / b;
                    if (pass == 0)
                        off[m + 1]++;
                    else
                        n2e[fill[m]++] = e;
                }
            }
        }
        if (pass == 0)
            for (uint32_t m = 0; m < nodes; m++) off[m + 1] += off[m];
    }
    // Patches: the lowest element left and the elements left around its highest node (on a structured mesh a
    // 2 x 2 x 2 block), then around the patch's other nodes, while the rows fit
    std::vector<uint8_t> taken(n_elem, 0);
    std::vector<uint32_t> stamp(nodes, UINT32_MAX);
    std::vector<uint32_t> first(1, 0), elems;  // patch -> its elements
    std::vector<uint32_t> nfirst(1, 0), pnodes, rank;  // patch -> its nodes, and each node's earlier patches
    std::vector<uint32_t> cnt(nodes, 0);               // patches of a node
    elems.reserve(n_elem);
    pnodes.reserve((size_t)n_elem * per / 2 + 16);
    rank.reserve((size_t)n_elem * per / 2 + 16);
    for (uint32_t s = 0; s < n_elem; s++) {
        if (taken[s]) continue;
        const uint32_t id = (uint32_t)first.size() - 1;
        const size_t n0 = pnodes.size();
        auto fresh = [&](uint32_t e) {  // nodes that e would add
            uint32_t f = 0;
            for (uint32_t j = 0; j < per; j++) f += stamp[map[(uint64_t)e * n + j * b] / b] != id;
            return f;
        };
        auto add = [&](uint32_t e) {
            taken[e] = 1;
            elems.push_back(e);
            for (uint32_t j = 0; j < per; j++) {
                const uint32_t m = map[(uint64_t)e * n + j * b] / b;
                if (stamp[m] != id) {
                    stamp[m] = id;
                    pnodes.push_back(m);
                    rank.push_back(cnt[m]++);
                }
            }
        };
        // the elements left around node m, the one that adds the fewest nodes first
        auto around = [&](uint32_t m) {
            while (elems.size() - first.back() < kBPatchElems) {
                uint32_t best = UINT32_MAX, at = 0;
                for (uint32_t k = off[m]; k < off[m + 1]; k++)
                    if (!taken[n2e[k]]) {
                        const uint32_t f = fresh(n2e[k]);
                        if (f < best) best = f, at = n2e[k];
                    }
                if (best == UINT32_MAX || pnodes.size() - n0 + best > max_nodes) return;
                add(at);
            }
        };
        add(s);
        uint32_t top = 0;
        for (uint32_t j = 0; j < per; j++) top = std::max(top, map[(uint64_t)s * n + j * b] / b);
        around(top);
        for (size_t q = n0; q < pnodes.size() && elems.size() - first.back() < kBPatchElems; q++) around(pnodes[q]);
        first.push_back((uint32_t)elems.size());
        nfirst.push_back((uint32_t)pnodes.size());
    }
    const uint32_t P = (uint32_t)first.size() - 1;
    uint32_t rows = 0;  // of the largest patch
    for (uint32_t p = 0; p < P; p++) rows = std::max(rows, (nfirst[p + 1] - nfirst[p]) * b);
    // combine buffer: the rows of each patch's shared nodes, in patch order
    std::vector<uint32_t> pv0(P + 1, 0);
    for (uint32_t p = 0; p < P; p++) {
        uint32_t c = 0;
        for (uint32_t q = nfirst[p]; q < nfirst[p + 1]; q++) c += cnt[pnodes[q]] > 1;
        pv0[p + 1] = pv0[p] + c * b;
    }
    std::vector<uint32_t> soff(nodes + 1, 0), srank(nodes + 1, 0);  // shared nodes: first list entry, place
    for (uint32_t m = 0; m < nodes; m++) {
        soff[m + 1] = soff[m] + (cnt[m] > 1 ? cnt[m] : 0);
        srank[m + 1] = srank[m] + (cnt[m] > 1 ? 1 : 0);
    }
    out.geom.n = n;
    out.geom.patches = P;
    out.geom.max_rows = (rows + 3u) & ~3u;
    out.geom.hdr_bytes = bpatch_hdr_bytes(n, out.geom.max_rows);
    out.geom.pv_rows = pv0[P];
    out.hdr.assign((size_t)P * out.geom.hdr_bytes, 0);
    // headers, and the combine lists' entries: entry r of a shared node is its row in its r-th patch
    out.shared_idx.assign((size_t)soff[nodes] * b, 0);
#pragma omp parallel for schedule(static)
    for (int64_t p = 0; p < (int64_t)P; p++) {
        unsigned char* h = out.hdr.data() + (size_t)p * out.geom.hdr_bytes;
        uint32_t* w = reinterpret_cast<uint32_t*>(h);
        const uint32_t ne = first[p + 1] - first[p], nn = nfirst[p + 1] - nfirst[p];
        uint32_t* ep = w + 8;
        uint32_t* rows = reinterpret_cast<uint32_t*>(h + bpatch_rows_off());
        unsigned char* loc = h + bpatch_loc_off(out.geom.max_rows);
        std::pair<uint32_t, uint32_t> place[kBPatchRows];  // the patch's nodes and their places, by node
        // the patch's own nodes first
        uint32_t own = 0, k = 0;
        for (int shared = 0; shared < 2; shared++) {
            for (uint32_t q = nfirst[p]; q < nfirst[p + 1]; q++) {
                const uint32_t m = pnodes[q];
                if ((cnt[m] > 1) != (shared == 1)) continue;
                place[k] = {m, k};
                for (uint32_t c = 0; c < b; c++) {
                    const uint32_t d = m * b + c;
                    rows[k * b + c] = d | (is_bc[d] ? kBcFlag : 0u);
                    if (shared)  // the node's DoFs have lists of equal length one after another
                        out.shared_idx[(size_t)soff[m] * b + c * cnt[m] + rank[q]] = pv0[p] + (k - own) * b + c;
                }
                k++;
            }
            if (!shared) own = k;
        }
        std::sort(place, place + nn);
        w[0] = ne;
        w[1] = nn * b;
        w[2] = own * b;
        w[3] = pv0[p];
        for (uint32_t q = 0; q < ne; q++) {
            const uint32_t e = elems[first[p] + q];
            ep[q] = pos[e];
            for (uint32_t j = 0; j < per; j++) {
                const std::pair<uint32_t, uint32_t> m(map[(uint64_t)e * n + j * b] / b, 0);
                const uint32_t at = std::lower_bound(place, place + nn, m)->second;
                for (uint32_t c = 0; c < b; c++) loc[q * n + j * b + c] = (unsigned char)(at * b + c);
            }
        }
    }
    // combine lists per DoF
    out.shared_dof.resize((size_t)srank[nodes] * b);
    out.shared_off.resize(out.shared_dof.size() + 1);
    out.shared_off[0] = 0;
#pragma omp parallel for schedule(static)
    for (int64_t m = 0; m < (int64_t)nodes; m++) {
        if (cnt[m] <= 1) continue;
        for (uint32_t c = 0; c < b; c++) {
            const size_t i = (size_t)srank[m] * b + c;
            out.shared_dof[i] = (uint32_t)m * b + c;
            out.shared_off[i + 1] = soff[m] * b + (c + 1) * cnt[m];
        }
    }
    out.geom.shared = (uint32_t)out.shared_dof.size();
}

}  // namespace afm
