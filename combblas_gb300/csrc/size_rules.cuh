// Rules by which the host sizes what kernels write, as plain functions of a
// matrix's counts (also compiled by the host compiler, where they are tested).
#pragma once

#include <stdint.h>

namespace gbc {

// Entries that k_ktl_fill writes at most for a matrix of nnz entries and ncol
// columns: a column touches at most as many row tiles as it has entries, and
// every column, empty ones included, has an end marker.
constexpr int64_t ktl_room(int64_t nnz, int64_t ncol) { return nnz + ncol; }

}  // namespace gbc
