// Where the one-ring and incidence records of a vertex lie (layout in vbd_kernels.cuh).
#pragma once
#include <cstddef>
#include <cstdint>
#include <limits>
#include <stdexcept>

#ifdef __CUDACC__
#define GAIA_HD __host__ __device__ __forceinline__
#else
#define GAIA_HD inline
#endif

namespace gaia {
namespace dev {

constexpr int kSegNbrs = 128;  // neighbours per segment at most (8-bit positions)
constexpr int kSlice = 8;      // vertices whose records are interleaved

// A row holds the k-th record of each vertex of a slice. Rows are counted in 32 bits, records
// (kSlice times as many) in 64: a scene has fewer rows of incidence records than incidences,
// the longest list of a slice being no longer than its lists together.
GAIA_HD size_t record_index(int32_t row, int32_t place) { return size_t(row) * kSlice + size_t(place); }

// vrec: (first row of NbrRec, first row of IncRec, neighbours | place in the slice << 8, incidences)
GAIA_HD int32_t pack_nbrs(int32_t n, int32_t place) { return n | place << 8; }
GAIA_HD int32_t nbrs_of(int32_t z) { return z & 255; }
GAIA_HD int32_t place_of(int32_t z) { return z >> 8; }

}  // namespace dev

// Incidences and rows are held in 32 bits.
inline int32_t checked_count(int64_t n) {
    if (n > std::numeric_limits<int32_t>::max()) throw std::runtime_error("too many incidences");
    return int32_t(n);
}

}  // namespace gaia
