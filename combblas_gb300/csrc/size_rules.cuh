// Rules by which the host sizes what kernels write, as plain functions of a
// matrix's counts (also compiled by the host compiler, where they are tested).
#pragma once

#include <stdint.h>

namespace gbc {

// Entries that k_ktl_fill writes at most for a matrix of nnz entries and ncol
// columns: a column touches at most as many row tiles as it has entries, and
// every column, empty ones included, has an end marker.
constexpr int64_t ktl_room(int64_t nnz, int64_t ncol) { return nnz + ncol; }

// Multi-source BFS with one bit per root holds positions among a graph's nnz
// entries in 32 bits and walks them in steps of up to kMbStep, one step past the
// last one included: nnz + kMbStep must not pass 2^32.
constexpr int64_t kMbStep = 128;
constexpr bool mb_positions_fit(int64_t nnz) { return nnz + kMbStep <= int64_t(1) << 32; }

}  // namespace gbc
