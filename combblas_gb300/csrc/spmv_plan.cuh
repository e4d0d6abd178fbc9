// The row-major form of a sparse matrix that the dense-vector SpMV runs on
// (spmv.cu), shared with the sparse-vector multiplies that fold rows in
// column order (spmspv_sr.cu).
#pragma once
#include "gbc_internal.cuh"

namespace gbc {

struct SpmvPlan {
    Context *ctx = nullptr;
    int64_t m = 0, n = 0, nnz = 0;
    int vt = 0;
    int64_t *rowptr = nullptr;  // [m+1]
    int32_t *col = nullptr;     // [nnz]
    void *val = nullptr;        // [nnz]
    bool tiles = true;          // laid out for the dense-vector SpMV (the members below)
    int64_t nrows = 0;             // rows with entries
    int32_t *rows = nullptr;       // [nrows] their ids, ascending
    uint32_t *starts = nullptr;    // [nnz / 32] bit p: entry p is the first of its row
    int32_t *group_row = nullptr;  // [nnz / kSpmvPer] row (index into rows) of each group's first entry
    int64_t ntiles = 0;            // blocks of k_spmv_tiles
    void *edge = nullptr;          // [2 ntiles] sums of the rows that cross tiles: before a tile's first start, behind its last
    int32_t *edge_row = nullptr;   // [ntiles] the row before a tile's first start; -1 none, -2 the tile has no start
};

// Build p (p->ctx and p->vt set) from A: rows ascending, each row's entries
// in ascending column order, by a stable device radix sort.
int spmv_plan_build(SpmvPlan *p, const gbc_matrix *A);
// Free p's device arrays (p itself stays).
void spmv_plan_release(SpmvPlan *p);

}  // namespace gbc
