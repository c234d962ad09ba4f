// Host-side planning shared by the single-system and batched paths:
// the reference cell grid, Morton ranking of (x, y) columns and the force
// work items.
#pragma once

#include <cstdint>
#include <vector>

#include "md.cuh"

namespace pb {

// cudaCutoffBlock::setupCutoffBlock (cudaCutoffBlock.cu:97-113) in the same
// FP32 operations.  Periodic: blocknum = (uint32)(c / rmax),
// blocklen = c / (float)blocknum.  Open boundaries: blocklen = rmax and
// blocknum = (uint32)(c / rmax) + 1, one block past the top face.  Returns
// false if any axis has < 3 cells (the reference asserts blocknum > 2).
bool make_grid(const float cell6[6], float rmax, Grid &g, bool periodic = true);

// rank[d0 * ny + d1] = position of column (d0, d1) along a Z-order curve;
// xy[rank] = d0 * ny + d1.
void morton_columns(int nx, int ny, std::vector<uint32_t> &rank, std::vector<uint32_t> &xy);

// Reference 27-neighbour table (calc_BlockNeighbor, cudaCutoffBlock.cu:17-65)
// in reference cell numbering d2 + d1 nz + d0 nz ny; in an open box a
// neighbour outside the grid is kNoCell.
void neighbor_table(const Grid &g, std::vector<uint32_t> &out);

// z cells per force work item for a mean cell occupancy: about 124 * scale
// home atoms per item (8 tiles of 16), at most force_max_segment(), and short
// enough for the CTAs per SM of the launch shape (four with one atom type, three
// with more): at 14 atoms a cell and one type 7 cells, 98 atoms.
// `half`: the half-shell force kernel runs (about 200 * scale home atoms; its
// stage has to fit as well).
int choose_segment(double atoms_per_cell, int nz, double scale = 1.0, int nt = 1,
                   bool half = false);

// Shared-memory capacity (atoms) of a force CTA staging 9 columns x (seg + 2)
// cells at the given mean occupancy of a system of `nt` types, with headroom for
// fluctuations; `spare`: and whatever else the CTAs of an SM have room for.
int choose_capacity(double atoms_per_cell, int seg, int nt, bool spare);
// Member slots per cell bucket of the two-kernel cell build: at least 32 and
// about twice the mean occupancy (a fuller cell spills to the overflow list).
int choose_bucket_cap(double atoms_per_cell);
// Members a 64-cell tile block of the cell build stages in shared memory
// (9 B each): about 1.3 times the mean tile; fuller tiles take the slower path.
int choose_tile_atoms(double atoms_per_cell);
// The same for the half-shell force kernel, which stages 5 columns.
int choose_capacity_half(double atoms_per_cell, int seg);

// Force work items of one system whose packed cell keys start at cell0, with
// the column ranking `rank` (reference column -> rank) and its inverse `xy`.
void append_items(uint32_t sys, const Grid &g, int seg, uint32_t cell0,
                  const std::vector<uint32_t> &rank, const std::vector<uint32_t> &xy,
                  std::vector<ForceItem> &items);

int force_max_segment();
// Largest staged-atom capacity of a force CTA.
int force_max_capacity();
// The largest capacity with which the CTAs per SM that the default launch shape is built
// for stay resident.
int force_capacity_room(int nt);
// Shared memory of one default-shape force CTA with staged-atom capacity `cap` and
// `nt` types, with a margin.
int force_smem_per_cta(int cap, int nt);
// The shared memory a default-shape force CTA may use so that the CTAs per SM
// its launch shape is built for stay resident.
int force_smem_limit(int nt);
// The same two for the half-shell force kernel (force_half.cu).
int force_half_max_capacity(int nt);
int force_half_smem_per_cta(int cap, int nt);

}  // namespace pb
