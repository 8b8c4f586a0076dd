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
// kTeamWarpBrows block rows for BSR6); a CTA of its team holds a fixed number
// of consecutive warp tiles. The cut depends on the matrix alone, so a
// system's arithmetic does not depend on what else runs. Two variants of the
// kernel hold at most kTeamWarps or kTeamWarpsWide warp tiles a CTA (128 or 96
// registers a thread); two more warps reduce.
constexpr int kTeamWarps = 14;
constexpr int kTeamWarpsWide = 18;
// Teams of more narrow CTAs than this are cut for the wide variant: polls among
// fewer CTAs then outweigh its longer product and its registers (B200, us an
// iteration, narrow against wide: 9^3 nodes, 11 CTAs, 4.7 and 5.1; 20^3, 115
// CTAs, 7.3 and 8.2; 21^3, 133 CTAs, 8.1 and 7.9), and it holds up to 23^3
// (8.7 against 12.9 in k_stream).
constexpr uint32_t kTeamNarrowCtas = 120;
constexpr int kTeamWarpBrows = 5;
constexpr int kTeamWarpRows = 6 * kTeamWarpBrows;
__host__ __device__ constexpr int team_threads(int warps) { return 32 * (warps + 2); }
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
__host__ __device__ constexpr int team_fixed_bytes(int warps) { return 512 + 2 * 8 * 32 * warps; }
__host__ __device__ constexpr uint32_t team_z_bytes(int warps, uint32_t ext) {
    return (4u * 32u * (uint32_t)warps + 28u * ext + 15u) & ~15u;
}
__host__ __device__ constexpr uint32_t team_tile_bytes(uint32_t cols) {
    return kTeamLuBytes + kTeamColBytes * cols + kTeamIdxBytes * ((cols + 7u) / 8u);
}
static_assert(kTeamLuBytes % 16 == 0 && kTeamColBytes % 16 == 0 && kTeamIdxBytes % 16 == 0, "16-byte operands");

// Copies of the published partials of a team, each read by every copies-th
// CTA: with one copy, the polls of a hundred CTAs on the same few cache lines
// hold up the stores (106 CTAs: 8.6 us an iteration against 7.5 with four);
// fewer CTAs are faster with one store (71 CTAs: 6.1 against 6.8 with three).
__host__ __device__ constexpr uint32_t team_copies(uint32_t size) { return size <= 96u ? 1u : 4u; }
__host__ __device__ constexpr uint64_t team_red_entries(uint32_t size) {
    return (uint64_t)kRedEntries * size * team_copies(size);
}

// The kernel whose CTAs hold up to `warps` (kTeamWarps or kTeamWarpsWide) warp
// tiles, launched cooperatively, one CTA per SM, with team_threads(warps)
// threads and the arguments (const SysDesc *, StepParams *, const TeamItem
// *items, const uint32_t *item_off, uint32_t limit): CTA c works through items
// [item_off[c], item_off[c + 1]), each for up to `limit` iterations. (More
// warps on an SM have too few registers: two CTAs of 512 threads spilled, and
// the spills did not fit in what L1 the shared memory leaves: 26 systems of 9^3
// nodes 13.5 us an iteration against 10.7; so did one CTA of 24 warp tiles, 4^3
// nodes 5.5 us against 2.9.)
const void *team_kernel(int warps);

}  // namespace wsb
