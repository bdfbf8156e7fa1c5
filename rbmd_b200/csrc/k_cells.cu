// k_cells.cu -- cell-list binning by counting sort (replaces ContPointLocator::Build,
// framework/locator/ContPointLocator.cxx:70-92: BinPointsWorklet + SortByKey + Upper/LowerBounds).
//
// Two passes.  The first (bin_atom, in the kick-drift kernel of a step, in k_cells_count otherwise)
// counts each cell's atoms and drops their ids into a bucket per cell.  The second (k_cells_build)
// adds up the counts before its cells, orders each cell's ids (the stable order of the reference's
// sort of fresh 0..N-1 point ids) and writes the cell-ordered positions, charges and metadata that the
// pair kernels stream.  The counts live in two buffers taken in turn: building from one clears the
// other for the next list, so no launch is spent on clearing.
#include "cells.cuh"

namespace rbmd {

__global__ void k_cells_count(const SysDev* __restrict__ S, const int2* __restrict__ work) {
  const int2 w = work[blockIdx.x];
  const SysDev& s = S[w.x];
  const int i = w.y + threadIdx.x;
  if (i >= s.n) return;
  const double4 p = s.x[i];
  const double pc[3] = {p.x, p.y, p.z};
  bin_atom(s, i, pc);
}

// kBuildCells cells per block (one warp scans their counts), kBuildFew in systems of few cells, so that a
// box of a few hundred cells has a warp per cell and blocks for a third of the chip: with 32 cells per
// block the kernel took 9 us for 512 cells of 18 atoms and 58 us for 27 cells of 167.
constexpr int kBuildThreads = 256;
static_assert(kCellBlock % kBuildCells == 0 && kBuildCells % kBuildFew == 0 && kBuildCells == 32 && kBuildFew % 4 == 0 &&
                  kCellSuper % (4 * kBuildCells) == 0,
              "a work item is a whole number of build blocks, a block's counts start on 16 bytes");
static_assert((kCellChains & (kCellChains - 1)) == 0 && kCellChains <= 8, "a chain per lane of a cell");

// Atoms per group of kBuildCells cells, for systems of more than kCellBigGrid cells, and per kCellSuper
// cells in those of more than kCellHugeGrid (sums that the build clears).
__global__ void k_cells_group_sums(const SysDev* __restrict__ S, const int2* __restrict__ work) {
  const int2 w = work[blockIdx.x];
  const SysDev& s = S[w.x];
  const int c = w.y + threadIdx.x;
  const int par = s.st->cell_epoch & 1;
  const int cnt = c < s.ncell ? s.cell_count[(size_t)par * s.cell_stride + c] : 0;
  const int sum = __reduce_add_sync(0xffffffffu, cnt);
  if ((threadIdx.x & 31) == 0 && c < s.ncell) {
    s.cell_gsum[c / kBuildCells] = sum;
    if (s.ncell > kCellHugeGrid && sum > 0) atomicAdd(&s.cell_super[c / kCellSuper], sum);
  }
}

// Atom i at place k of the cell order.
__device__ __forceinline__ void place(const SysDev& s, int i, int k) {
  s.sorted[k] = i;
  s.rank[i] = k;
  const double4 p = s.x[i];
  s.sx[k] = p;
  s.sxf[k] = make_float4((float)p.x, (float)p.y, (float)p.z, (float)p.w);
  const int4 m = s.meta[i];
  s.smeta[k] = make_int4(i, m.x, m.y, m.z);
}

// How many of a bucket's n ids are below id (a bucket starts on 16 bytes).
__device__ __forceinline__ int rank_in(const int* ids, int n, int id) {
  int r = 0, j = 0;
  for (; j + 4 <= n; j += 4) {
    const int4 v = *reinterpret_cast<const int4*>(ids + j);
    r += (v.x < id ? 1 : 0) + (v.y < id ? 1 : 0) + (v.z < id ? 1 : 0) + (v.w < id ? 1 : 0);
  }
  for (; j < n; ++j) r += ids[j] < id ? 1 : 0;
  return r;
}

// A cell of more atoms than its bucket holds, by the cell's lanes (8, or a warp).  The rest hang on the
// cell's chains and are laid out one after the other first.  Not inlined: the build would spill.
__device__ __noinline__ void place_overfull(const SysDev& s, int c, int cnt, int start, int lanes, int lane) {
  const int cap = s.cell_cap, over = cnt - cap, gl = lane & (lanes - 1);
  const int* ids = s.cell_bucket + (size_t)c * cap;
  int* rest = s.cell_rest + start + cap;
  if (gl < kCellChains && gl < over) {
    int id = s.cell_head[(size_t)c * kCellChains + gl];
    for (int k = gl;;) {
      rest[k] = id;
      k += kCellChains;
      if (k >= over) break;
      id = s.cell_next[id];
    }
  }
  __syncwarp(lanes == 32 ? 0xffffffffu : 0xffu << (lane & 24));  // the cell's lanes
  for (int k = gl; k < cnt; k += lanes) {
    const int id = k < cap ? ids[k] : rest[k - cap];
    int r = rank_in(ids, cap, id);
    for (int j = 0; j < over; ++j) r += rest[j] < id ? 1 : 0;
    place(s, id, start + r);
  }
}

// One block per kBuildCells (or kBuildFew) cells.  Bound by latency: the loads of the preceding counts (at most
// kCellBigGrid / (4 x 256) 16-byte loads per thread; above that the sums of the kernel before, at most
// kCellHugeGrid / (32 x 4 x 256) such loads, or two and the sums of kCellSuper cells: with one level for
// any size a list of 17 M cells took 21.6 ms and of 64 M cells 331 ms, for now 2.9 and 12.6 ms),
// then one dependent gather per atom.  A cell's ids are taken by 8 lanes where buckets are small (cells
// of a few atoms) and by a warp otherwise; each lane ranks its ids against the whole cell, so cells
// of hundreds of atoms need no serial sort.  Atoms beyond the bucket are collected from their cell's
// chains first, so an atom is compared with those of its own cell only: in a slab that fills a tenth of
// its box (64,000 atoms, buckets of 8, 13 atoms per cell) a list takes 27 us, against 44 ms when each atom
// of an over-full cell went through the overflow of the whole system.  `items` is the number of work items
// where the table covers a single system's present cells only, 0 where it covers the ncell_cap of each.
__global__ void __launch_bounds__(kBuildThreads) k_cells_build(const SysDev* __restrict__ S,
                                                             const int2* __restrict__ work, int big, int items) {
  const int2 w = work[blockIdx.x];
  const SysDev& s = S[w.x];
  SysState* st = s.st;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int per = s.ncell_cap <= kFewCells ? kBuildFew : kBuildCells;
  if ((int)blockIdx.y * per >= kCellBlock) return;  // the grid is for the smaller blocks
  const int c0 = w.y + blockIdx.y * per;
  const int par = st->cell_epoch & 1;
  const int* count = s.cell_count + (size_t)par * s.cell_stride;
  int* other = s.cell_count + (size_t)(par ^ 1) * s.cell_stride;
  __shared__ int s_sum[kBuildThreads / 32], s_start[kBuildCells], s_cnt[kBuildCells];
  if (c0 < s.ncell) {  // block-uniform
    int sum = 0;
    if (big && per == kBuildCells) {
      const int super = s.ncell > kCellHugeGrid ? c0 / kCellSuper : 0, end = c0 / kBuildCells;
      const int* g = s.cell_gsum;  // 16 bytes per load from the first group of the super group on
      for (int k = super * (kCellSuper / kBuildCells) + 4 * tid; k < end; k += 4 * kBuildThreads) {
        const int4 v = *reinterpret_cast<const int4*>(g + k);
        sum += v.x + (k + 1 < end ? v.y : 0) + (k + 2 < end ? v.z : 0) + (k + 3 < end ? v.w : 0);
      }
      for (int k = tid; k < super; k += kBuildThreads) sum += s.cell_super[k];
    } else {
      const int4* c4 = reinterpret_cast<const int4*>(count);  // c0 is a multiple of 4
      for (int g = tid; g < c0 / 4; g += kBuildThreads) {
        const int4 v = c4[g];
        sum += (v.x + v.y) + (v.z + v.w);
      }
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) s_sum[wid] = sum;
    __syncthreads();
    if (wid == 0) {
      int base = lane < kBuildThreads / 32 ? s_sum[lane] : 0;
      base = __reduce_add_sync(0xffffffffu, base);
      const int c = c0 + lane;
      const bool mine = lane < per && c < s.ncell;
      const int cnt = mine ? count[c] : 0;
      const int incl = warp_incl_scan(cnt, lane);
      s_start[lane] = base + incl - cnt;
      s_cnt[lane] = cnt;
      if (mine) s.cell_start[c] = base + incl - cnt;
      if (mine && c == s.ncell - 1) s.cell_start[s.ncell] = base + incl;
    }
    __syncthreads();
    const int cap = s.cell_cap;
    const int lanes = cap <= 16 ? 8 : 32;  // lanes per cell
    const int gl = tid & (lanes - 1);
    for (int cc = tid / lanes; cc < per; cc += kBuildThreads / lanes) {
      const int cnt = s_cnt[cc];
      const int* ids = s.cell_bucket + (size_t)(c0 + cc) * cap;
      if (cnt <= cap) {
        for (int k = gl; k < cnt; k += lanes) place(s, ids[k], s_start[cc] + rank_in(ids, cnt, ids[k]));
      } else {
        place_overfull(s, c0 + cc, cnt, s_start[cc], lanes, lane);
      }
    }
    if (c0 == 0 && tid == 0) {  // a new cell list: nothing has moved since
      st->shake_disp_bits = 0u;
      st->mig_n = 0;
      st->out_bits = st->out_acc[par];
      st->out_acc[par ^ 1] = 0u;
    }
  }
  if (items == 0) items = (s.ncell_cap + kCellBlock - 1) / kCellBlock;
  if (tid < per && c0 + tid < s.ncell_cap) other[c0 + tid] = 0;
  if (c0 == 0)
    for (int c = items * kCellBlock + tid; c < s.ncell_cap; c += kBuildThreads) other[c] = 0;
  // every block has read this list's buffer index: the next list takes the other buffer
  if (arrive_last(&st->counter[7], (unsigned)(items * (kCellBlock / per)))) {
    if (tid == 0) st->cell_epoch ^= 1;
    if (big && s.ncell > kCellHugeGrid)
      for (int g = tid; g <= (s.ncell - 1) / kCellSuper; g += kBuildThreads) s.cell_super[g] = 0;
  }
}

void launch_cells_build(const Batch& b, cudaStream_t st) {
  if (b.big_cells) {
    k_cells_group_sums<<<b.cell.n, kCellBlock, 0, st>>>(b.sys, b.cell.d);
    note_launch();
  }
  const dim3 grid(b.cell.n, kCellBlock / (b.few_cells ? kBuildFew : kBuildCells));
  k_cells_build<<<grid, kBuildThreads, 0, st>>>(b.sys, b.cell.d, b.big_cells, b.cell_items);
  note_launch();
}

void launch_cells(const Batch& b, cudaStream_t st) {
  k_cells_count<<<b.atom.n, kAtomBlock, 0, st>>>(b.sys, b.atom.d);
  note_launch();
  launch_cells_build(b, st);
}

}  // namespace rbmd
