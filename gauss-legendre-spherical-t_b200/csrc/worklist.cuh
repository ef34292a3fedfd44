// Batched work-list kernels: one persistent launch per phase covers many
// independent systems.  Each system is described by a SysDesc (its grid,
// buffers, node tables and where its inputs and outputs live); each phase has
// a list of work items (system, block indices) -- the same block indices the
// system's own launch would use -- and a grid of resident CTAs that take the
// items in a fixed stride (CTA b: items b, b + gridDim.x, ...).  Every item
// runs exactly the code of the one-system kernels (the *_block functions of
// cells.cuh, shell_sums.cuh and kernels.cuh) on the same tables, so a system's
// results are bit for bit the ones it gets alone.  (The structure factors and
// the gather: far_field.cu.)
#pragma once

#include "cells.cuh"
#include "kernels.cuh"
#include "shell_sums.cuh"

namespace glst {
namespace dev {

// Cell counts to zero before binning: item a = block of 1024 cells.
__global__ void __launch_bounds__(1024) k_zero_counts_multi(const SysDesc *__restrict__ sys,
                                                            const WorkItem *__restrict__ items, uint32_t n) {
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const WorkItem w = items[it];
    const SysDesc &d = sys[w.sys];
    const uint32_t c = w.a * 1024u + threadIdx.x;
    if (c < d.g.ncell) d.cell_count[c] = 0u;
  }
}

__global__ void __launch_bounds__(256) k_bin_multi(const SysDesc *__restrict__ sys,
                                                   const WorkItem *__restrict__ items, uint32_t n) {
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const WorkItem w = items[it];
    const SysDesc &d = sys[w.sys];
    bin_block(d.rx, d.ry, d.rz, d.natom, d.g, d.atom_cell, d.atom_slot, d.cell_count, w.a);
  }
}

__global__ void __launch_bounds__(1024) k_scan_multi(const SysDesc *__restrict__ sys,
                                                     const WorkItem *__restrict__ items, uint32_t n) {
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const SysDesc &d = sys[items[it].sys];
    scan_body(d.cell_count, d.g.ncell, d.cell_point, d.pieces.cap, d.piece_list, d.n_pieces);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_scatter_multi(const SysDesc *__restrict__ sys,
                                                       const WorkItem *__restrict__ items, uint32_t n) {
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const WorkItem w = items[it];
    const SysDesc &d = sys[w.sys];
    scatter_block(d.atom_cell, d.atom_slot, d.cell_point, d.natom, d.perm, w.a);
  }
}

// item a = block of kSortCells cells; kSortCap u32 of dynamic shared memory
__global__ void __launch_bounds__(256) k_sort_pack_multi(const SysDesc *__restrict__ sys,
                                                         const WorkItem *__restrict__ items, uint32_t n) {
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const WorkItem w = items[it];
    const SysDesc &d = sys[w.sys];
    sort_pack_cells(d.perm, d.cell_count, d.cell_point, d.g, d.atom_cell, d.natom, d.rx, d.ry, d.rz, d.qc,
                    d.sorted_idx, d.pk, d.pd, w.a);
    __syncthreads();
  }
}

// item a = block of nb nodes; dynamic shared memory: the largest system's
// rows, twiddles and coordinate table
__global__ void __launch_bounds__(kSatThreads, 3) k_shell_sums_multi(const SysDesc *__restrict__ sys,
                                                                     const WorkItem *__restrict__ items,
                                                                     uint32_t n) {
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const WorkItem w = items[it];
    const SysDesc &d = sys[w.sys];
    shell_block<3>(d.g, d.sat, w.a);
    __syncthreads();
  }
}

// item (a, b) = (block of cells, row of neighbour cells)
__global__ void __launch_bounds__(kSrThreads) k_short_range_multi(const SysDesc *__restrict__ sys,
                                                                  const WorkItem *__restrict__ items,
                                                                  uint32_t n) {
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const WorkItem w = items[it];
    const SysDesc &d = sys[w.sys];
    const uint32_t width = sr_width(d.natom, d.sr_rows);
    sr_block<4>(d.pd, d.cell_count, d.cell_point, d.g, d.natom, d.sr, d.sr_rows,
             sr_warps_per_cell(d.natom, d.g.ncell, width), width, d.pieces, w.a, w.b);
    __syncthreads();
  }
}

// item a = block of kCombineAtoms atoms
__global__ void __launch_bounds__(kCombineThreads) k_combine_multi(const SysDesc *__restrict__ sys,
                                                                   const WorkItem *__restrict__ items,
                                                                   uint32_t n) {
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const WorkItem w = items[it];
    const SysDesc &d = sys[w.sys];
    combine_block(d.sr, d.sr_rows, d.part, d.part_rows, d.sorted_idx, d.natom, d.use_far, d.cfx, d.cfy, d.cfz, d.cen, d.ofx,
                  d.ofy, d.ofz, d.oen, d.block_energy, d.combine_blocks, d.ticket, d.energy, w.a);
    __syncthreads();
  }
}

// one item per system without atoms
__global__ void __launch_bounds__(256) k_energy_multi(const SysDesc *__restrict__ sys,
                                                      const WorkItem *__restrict__ items, uint32_t n) {
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const SysDesc &d = sys[items[it].sys];
    energy_body(d.block_energy, 0, d.energy);
    __syncthreads();
  }
}

}  // namespace dev
}  // namespace glst
