// Host-side assembly plan: sparsity pattern of the free-DOF system and the
// element-to-nonzero scatter map (plain C++; built once per mesh + node book).
#pragma once

#include <stdint.h>

#include <memory>
#include <string>
#include <vector>

namespace rsg {

// One (row, adjacent tet) pair as the heat kernels read it: 16 bytes in slices of 32 rows -- pair t of row l of
// slice s at pair[(pair_ptr[s] + t) * 32 + l], padded with tet 0xffffffff.  Two forms:
//   wide   {tet, local index m of the row's node, offsets of the tet's four nodes in the row as 16 bits
//          each (0xffff: a fixed node)}; the node numbers come from the tet array;
//   near   for rows of at most 32 entries whose neighbour nodes are numbered within 32767 of the row's:
//          {tet, m | offsets as 6 bits each (63: a fixed node), node numbers less the row node's as
//          16 bits each}, which saves the tet array's scattered 16 bytes per pair and a dependent load.
struct alignas(16) AsmPair {
    uint32_t x, y, z, w;
};

struct AsmPlanHost {
    uint32_t n_nodes = 0, n_tets = 0, n_tris = 0, dofs = 1, n_free = 0;
    std::vector<uint32_t> row_node;   // node of each free row
    std::vector<uint8_t> row_comp;    // component of each free row
    std::vector<uint32_t> rp, ci;     // CSR pattern (sorted columns)
    // node -> tets adjacency in ascending tet order
    std::vector<uint32_t> adj_ptr, adj_elem;
    std::vector<uint8_t> adj_loc;     // local index of the node in the tet
    std::vector<uint16_t> adj_off;    // 4 per entry: offset of each tet node's column block in the row (0xffff: none)
    // with pack_pairs, instead of adj_off: the pairs
    std::vector<uint32_t> pair_ptr;   // slices + 1
    std::unique_ptr<AsmPair[]> pair;  // pair_ptr.back() * 32
    bool near = false;
    // node -> traction triangles adjacency (elasticity only)
    std::vector<uint32_t> tadj_ptr, tadj_tri;
    std::vector<uint8_t> node_mask;   // bit j set when component j of the node is free
};

// book has n_nodes * dofs entries (free position or 0xffffffff).  pack_pairs: for one component per node, the scatter
// map as AsmPair.  Returns false and sets err on bad input.
bool build_assembly_plan(uint32_t n_nodes, uint32_t n_tets, const uint32_t *tets, uint32_t n_tris,
                         const uint32_t *tris, const uint32_t *book, uint32_t dofs, uint32_t n_free, bool pack_pairs,
                         AsmPlanHost &plan, std::string &err);

}  // namespace rsg
