// Persistent PCG kernels: whole solves (or steps of a solve) in one launch.
//
// k_team iterates systems whose matrix fits in the shared memory of the CTAs
// that share it (a "team"): the matrix is read once per launch, the vectors
// live in registers, and the CTAs of a team meet in two all-reduces per
// iteration over global memory.
#pragma once
#include "wsb_internal.h"

namespace wsb {

// A system's rows are cut into warp tiles (one row a lane, no block cut;
// kTeamWarpBrows block rows for BSR6), and those into parts of a fixed number
// of consecutive warp tiles (at most kTeamWarps). The cut depends on the matrix
// alone and sums are formed part by part, so a system's arithmetic does not
// depend on what else runs, nor on how many parts a CTA of its team holds: one,
// or two (a lane then owns a row of each). Two more warps reduce.
constexpr int kTeamWarps = 14;
constexpr int kTeamThreads = 32 * (kTeamWarps + 2);
constexpr int kTeamWarpBrows = 5;
constexpr int kTeamWarpRows = 6 * kTeamWarpBrows;
// Shared memory of a CTA: a fixed part; the CTA's rows of z and, for at most
// `ext` blocks whose columns lie outside the CTA, 6 more entries of z and a
// column; then per warp tile the LU factors and reciprocals of their diagonals
// (kTeamLuBytes), kTeamColBytes for each block of its longest block row
// (values, p at the block columns) and kTeamIdxBytes for each eight of them
// begun (places in z).
constexpr int kTeamLuBytes = (144 + 32) * kTeamWarpBrows;
constexpr int kTeamColBytes = 24 * kTeamWarpRows + 32 * kTeamWarpBrows;
constexpr int kTeamIdxBytes = 32 * (kTeamWarpBrows + 1);
constexpr int kTeamSmemMax = 227 * 1024;
__host__ __device__ constexpr int team_fixed_bytes(int parts) { return 512 + 2 * 8 * 32 * kTeamWarps * parts; }
__host__ __device__ constexpr uint32_t team_z_bytes(int parts, uint32_t ext) {
    return (4u * 32u * kTeamWarps * (uint32_t)parts + 28u * ext + 15u) & ~15u;
}
__host__ __device__ constexpr uint32_t team_tile_bytes(uint32_t cols) {
    return kTeamLuBytes + kTeamColBytes * cols + kTeamIdxBytes * ((cols + 7u) / 8u);
}
// CSR: 32 rows at most a warp tile, its blocks (1 to 6 rows) kTeamBlockLu bytes
// each, then 6 bytes a place of its longest row's length (a multiple of four)
// times 32; before the tiles z and p of the CTA's rows and of at most
// kTeamMaxExt columns outside, and those columns.
constexpr int kTeamBlockLu = 144 + 32;
constexpr uint32_t kTeamMaxExt = 4096;
__host__ __device__ constexpr uint32_t team_csr_tile_bytes(uint32_t cols, uint32_t blocks) {
    return (uint32_t)kTeamBlockLu * blocks + 192u * ((cols + 3u) & ~3u);
}
__host__ __device__ constexpr uint32_t team_csr_z_bytes(uint32_t ext) {
    return (8u * 32u * kTeamWarps + 12u * ext + 15u) & ~15u;
}
static_assert(kTeamBlockLu % 16 == 0, "16-byte operands");
static_assert(kTeamLuBytes % 16 == 0 && kTeamColBytes % 16 == 0 && kTeamIdxBytes % 16 == 0, "16-byte operands");

// Copies of the published partials of a team, each read by every copies-th
// CTA: with one copy, the polls of a hundred CTAs on the same few cache lines
// hold up the stores; fewer CTAs are faster with one store (B200, us an
// iteration with one, four and eight copies: 77 parts 5.4, 5.8, 5.7; 90 parts
// 7.0, 5.9, 5.8; 164 parts on 82 CTAs -, 8.2, 7.9; 148 CTAs in k_stream -, 13.5,
// 13.4).
__host__ __device__ constexpr uint32_t team_copies(uint32_t size) { return size <= 80u ? 1u : 8u; }
// (And one a CTA for the team to assemble.)
__host__ __device__ constexpr uint64_t team_red_entries(uint32_t size) {
    return ((uint64_t)kRedEntries * team_copies(size) + 1u) * size;
}

// The kernel whose CTAs hold up to `parts` (1 or 2) parts of a system, one item
// each or `lists` of them, launched cooperatively, one CTA per SM, with
// kTeamThreads threads and the arguments (const SysDesc *, StepParams *, const
// TeamItem *items, const uint32_t *item_off, uint32_t limit, uint32_t longest):
// CTA c works through items [item_off[c], item_off[c + 1]), `longest` at most,
// each for up to `limit` iterations. (More warps on an SM have too few registers:
// two CTAs of 512 threads spilled, and the spills did not fit in what L1 the
// shared memory leaves: 26 systems of 9^3 nodes 13.5 us an iteration against
// 10.7; so did one CTA of 24 warp tiles, 4^3 nodes 5.5 us against 2.9.)
const void *team_kernel(int parts, bool csr, bool single_reduction, bool lists);
// Fills D.tile_idx, D.ext_cols and D.ext_count (= count) of a CSR system whose
// tiles are set, `parts` parts of D.team_warps tiles. most[0] becomes the most
// columns outside a part, most[1] whether that is more than D.ext_cap (nothing
// is iterated from such a plan); both start as 0.
cudaError_t team_plan_csr(const SysDesc &D, uint32_t *count, uint32_t *most, uint32_t parts, cudaStream_t st);

}  // namespace wsb
