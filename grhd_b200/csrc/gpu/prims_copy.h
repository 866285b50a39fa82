// prims_copy.h -- which parts of a ghosted primitive array an upload copies (host code only).
#pragma once

#include <cstddef>

namespace grhd {

constexpr size_t MAX_COPY_PITCH = 2147483647;  // cudaDevAttrMaxPitch: the pitch of a 2D copy, in bytes

// rows of `width` bytes, `pitch` bytes apart, from byte `offset` of the array on
struct CopyPiece {
  size_t offset, pitch, width, rows;
};

// The rows of the ghosted primitive array p(5, -ng:nx+ng, -ng:ny+ng, -ng:nz+ng) that k_prims_in
// reads: the interior rows (with their ghosts along i, which rows j = 1..ny of a plane hold
// contiguously) and, for two ghost cells, the rows at -ng along the active directions.  A 2D
// grid's ghost planes are most of its array: 27 MB against 3.4 MB of interior rows for
// 400x1x200, 8.7 against 1.4 MB for 257x131x1.  Calls copy(piece) for each; planes too large for
// the pitch of a 2D copy come one by one.  Stops at the first call that returns nonzero.
template <class Copy>
inline int prims_in_pieces(int nx, int ny, int nz, int ng, Copy &&copy) {
  const size_t row = (size_t)5 * sizeof(double) * ((size_t)nx + 2 * (size_t)ng + 1);
  const size_t plane = row * ((size_t)ny + 2 * (size_t)ng + 1);
  // rows j .. j + n - 1 of the planes k .. k + m - 1
  auto rows = [&](int j, int n, int k, int m) -> int {
    const size_t off = row * (size_t)(j + ng) + plane * (size_t)(k + ng), width = row * (size_t)n;
    if (m == 1 || plane <= MAX_COPY_PITCH) return copy(CopyPiece{off, plane, width, (size_t)m});
    for (int q = 0; q < m; ++q)
      if (int rc = copy(CopyPiece{off + plane * (size_t)q, plane, width, 1})) return rc;
    return 0;
  };
  if (int rc = rows(1, ny, 1, nz)) return rc;
  if (ng == 2 && ny > 1)
    if (int rc = rows(-ng, 1, 1, nz)) return rc;
  if (ng == 2 && nz > 1)
    if (int rc = rows(1, ny, -ng, 1)) return rc;
  return 0;
}

}  // namespace grhd
