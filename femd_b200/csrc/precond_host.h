// precond_host.h -- the order in which ILU(0) and SSOR do a matrix's rows, computed on the host once per
// preconditioner (setup_host.cpp); precond.cu packs and uploads it.  Internal header (not installed).
#pragma once

#include <cstddef>
#include <vector>

namespace femd {

constexpr int PC_SLICE = 8;              // rows of a chunk that lie side by side
constexpr int PC_WARP = 32;              // rows that are filled up to the same number of entries
constexpr int PC_RECORD = 32, PC_HEAD = 16;   // bytes of a row's record and of a chunk's head
// Places within a chunk are 32-bit bytes: a level of more than this is cut into several chunks (its rows
// do not depend on one another, so it only takes a barrier more).
constexpr long long PC_CHUNK_MAX = 1ll << 30;

constexpr size_t pc_chunk_bytes(int m, int E)
{
    return PC_HEAD + PC_RECORD * (size_t)m + 12 * (size_t)E;   // E: a multiple of 4 PC_SLICE
}

// rows grouped by level: level(i) = 1 + max level over the rows that row i reads (its lower part
// for the forward sweep, its upper part for the backward one, taken from the last row down); dg: the
// positions of the diagonal
void level_schedule(int n, const std::vector<int> &ip, const std::vector<int> &ix, const std::vector<int> &dg, bool forward,
                    std::vector<int> &rows, std::vector<int> &ptr);

// The chunks of one sweep's levels, at most `limit` bytes each (or PC_SLICE rows): ptr becomes the chunks'
// first rows, the rows of a chunk are sorted by length; per row (in that order) its first entry, per chunk
// its entries and rows; the chunks' ends are appended to place (in 16 B, running).
void chunk_layout(const std::vector<int> &ip, const std::vector<int> &dg, bool forward, long long limit, std::vector<int> &rows,
                  std::vector<int> &ptr, std::vector<int> &eoff, std::vector<int> &etot, std::vector<int> &rtot,
                  std::vector<long long> &place);

}  // namespace femd
