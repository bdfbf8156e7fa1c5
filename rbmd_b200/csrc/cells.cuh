// cells.cuh -- binning of one atom, shared by the standalone count kernel and the kick-drift kernel.
#pragma once

#include "kernels.h"

namespace rbmd {

// Puts atom i, at position pc, into its cell: the cell's count, the atom's place in the cell's bucket
// (in order of arrival; the build kernel orders the ids), and how far the atom lies outside the cell.
// Buckets hold cell_cap ids; the atoms beyond are chained per cell, kCellChains chains taken in turn.  A
// chain's length follows from the cell's count, so heads and links are never cleared.
__device__ __forceinline__ void bin_atom(const SysDev& s, int i, const double (&pc)[3]) {
  SysState* st = s.st;
  const int par = st->cell_epoch & 1;
  int ijk[3];
  double out = 0.0;  // how far the atom lies outside the cell it is binned into
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    long long c = (long long)((pc[k] - s.lo[k]) / s.d[k]);  // truncation, as vtkm::Id3(Vec3f)
    c = c < 0 ? 0 : c;
    c = c > s.dims[k] - 1 ? s.dims[k] - 1 : c;
    ijk[k] = (int)c;
    out = fmax(out, fmax(s.lo[k] + (double)c * s.d[k] - pc[k], pc[k] - (s.lo[k] + (double)(c + 1) * s.d[k])));
  }
  if (out > 0.0) atomicMax(&st->out_acc[par], __float_as_uint(__double2float_ru(out)));  // non-negative: bits order as values
  // internal numbering is z fastest so that the 2 nc + 1 cells of a traversal row (fixed x and y
  // offsets) are contiguous in cell order; get_cells reports the reference's x-fastest ids
  const int cell = ijk[2] + s.dims[2] * (ijk[1] + s.dims[1] * ijk[0]);
  s.cell_of_atom[i] = cell;
  const int slot = atomicAdd(&s.cell_count[(size_t)par * s.cell_stride + cell], 1);
  if (slot < s.cell_cap) s.cell_bucket[(size_t)cell * s.cell_cap + slot] = i;
  else s.cell_next[i] = atomicExch(&s.cell_head[(size_t)cell * kCellChains + ((slot - s.cell_cap) & (kCellChains - 1))], i);
}

}  // namespace rbmd
