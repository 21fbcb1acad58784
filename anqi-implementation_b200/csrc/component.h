// The AKNN gather of rows in small components of the list graph (component.cu).
#pragma once

#include <vector>

#include "internal.h"

namespace anqi {

// Components of up to 2,048 rows take the component form: their distance
// matrix is at most 2,048 keys a row, 64 registers of a lane.
constexpr uint32_t kCompMaxWords = 64;
constexpr uint32_t kCompMaxRows = 32 * kCompMaxWords;

// One component: rows [start, start + size) of the locality numbering.
struct CompRange {
    uint32_t start, size;
};

struct CompDesc {
    uint32_t start, size, words, tile0;  // words = ceil(size / 32); tile0 = first Gram tile in the batch
    uint64_t goff, aoff;                 // first float of the distance matrix / word of the adjacency bitmaps
    uint32_t index, pad;                 // component number
};

// The gather's inputs in the locality numbering (GatherParams in build.cu).
struct CompGather {
    const float* x;
    const float* norms;
    uint64_t n;
    uint32_t stride, dim, cols;
    const uint32_t* g_ids;
    const float* g_vals;
    uint32_t K;
    const uint64_t* rev_off;
    const uint32_t* rev_ids;
    uint32_t ef, cap, out_k;
    const uint32_t* perm;
    uint32_t* out_ids;
    float* out_d;
    unsigned long long* pool_total;
};

// Gathers every row of the components `ranges` (ascending, disjoint, at most
// kCompMaxRows rows each).  row_comp (n entries) receives each row's component
// or kEmpty, bad (one flag per component) which of them hold a non-finite
// distance and were left out, any_bad whether there are any.
int run_component_gather(Ctx* c, const CompGather& g, const std::vector<CompRange>& ranges, DevBuf& row_comp,
                         DevBuf& bad, bool* any_bad);

// Select and commit of the G48 build when `ranges` cover every row (g.out_* and
// g.g_vals unused): final links (n x M) and degrees in the original numbering.
// With any_bad set the outputs are incomplete and the general path is to run.
int run_component_select_commit(Ctx* c, const CompGather& g, const std::vector<CompRange>& ranges, uint32_t M,
                                float alpha, uint32_t* links, uint32_t* deg, bool* any_bad);

}  // namespace anqi
