/*
 * shl_cells.h -- the linked cells that a face's box covers, by their rank
 * (ShellSystem.C:1982-2001: the loops over the cells from lo to hi per axis).
 * Shared by the kernels, whose lanes share a face's cells, and the host tests.
 */
#ifndef SHL_CELLS_H_
#define SHL_CELLS_H_

#include "shl_distance.h"

/* How many cells lie in lo..hi; 0 if the range is empty on an axis.  (A face
 * whose three nodes are NaN on an axis has the empty box there, lo = INT_MAX
 * and hi = INT_MIN; the extent's difference would wrap around.) */
SHL_HD unsigned shl_cells_covered(const int* lo, const int* hi)
{
  if (lo[0] > hi[0] || lo[1] > hi[1] || lo[2] > hi[2]) return 0u;
  return (unsigned)(hi[0] - lo[0] + 1) * (unsigned)(hi[1] - lo[1] + 1) * (unsigned)(hi[2] - lo[2] + 1);
}

/* index, in a grid of ny x nz cells per layer, of the q-th of them */
SHL_HD unsigned shl_cells_at(unsigned q, const int* lo, const int* hi, unsigned ny, unsigned nz)
{
  const unsigned cy = (unsigned)(hi[1] - lo[1] + 1), cz = (unsigned)(hi[2] - lo[2] + 1);
  const unsigned z = q % cz, y = q / cz % cy, x = q / (cz * cy);
  return ((unsigned)lo[0] + x) * ny * nz + ((unsigned)lo[1] + y) * nz + (unsigned)lo[2] + z;
}

#endif /* SHL_CELLS_H_ */
