// k_stream: the persistent PCG loop for BSR6 systems that do not fit in the
// shared memory of the device. One CTA per SM; all of them share one system at
// a time and stream its matrix and factors in every iteration.
#pragma once
#include "wsb_internal.h"

namespace wsb {

constexpr int kStreamWarps = 16;
constexpr int kStreamThreads = 32 * kStreamWarps;
// Product tiles: 5 block rows (30 rows, one a lane), at most kStreamMaxBlocks
// blocks a tile and kStreamMaxCols a block row.
constexpr int kStreamBrows = 5;
constexpr int kStreamMaxBlocks = 36;
constexpr int kStreamMaxCols = 8;
constexpr int kStreamSpmvStage = 144 * kStreamMaxBlocks;
constexpr int kStreamColBytes = 4 * ((kStreamMaxBlocks + 3) / 4 * 4);     // a tile's block columns
constexpr int kStreamXgBytes = 32 * (kStreamBrows + 1) * kStreamMaxCols;  // p at a tile's block columns
// Update tiles: up to kStreamUpd(Sr)Brows block rows, one a lane: the factors,
// the slices of x and r (kSr: p and s too).
constexpr int kStreamUpdBrows = 32;
constexpr int kStreamUpdBrowsSr = 28;
constexpr int kStreamUpdStage = kStreamUpdBrowsSr * (144 + 4 * 24);
static_assert(kStreamUpdBrows * (144 + 2 * 24) <= kStreamUpdStage, "update stages");
static_assert(kStreamUpdBrows % 2 == 0 && kStreamUpdBrowsSr % 2 == 0, "16-byte slices");
// Each warp has two stages, used by both phases.
constexpr int kStreamWarpBytes = 2 * kStreamUpdStage;
static_assert(2 * kStreamSpmvStage + kStreamColBytes + kStreamXgBytes <= kStreamWarpBytes, "product stages");
static_assert(kStreamMaxBlocks <= 64, "two columns a lane");
static_assert(kStreamUpdStage % 16 == 0 && kStreamSpmvStage % 16 == 0 && kStreamColBytes % 16 == 0, "TMA alignment");
constexpr int kStreamFixedSmem = 2048;
constexpr int kStreamSmem = kStreamFixedSmem + kStreamWarps * kStreamWarpBytes;
static_assert(kStreamSmem <= 227 * 1024, "shared memory");

// The kernel for one recurrence, launched cooperatively with stream_grid CTAs
// of kStreamThreads threads and the arguments (const SysDesc *, StepParams *,
// uint32_t system, uint32_t limit): up to `limit` iterations of one system that
// the init kernels have started.
const void *stream_kernel(bool single_reduction);
// CTAs for a system of nbr block rows: one SM each, and work for every warp in
// both phases. A function of the system and the device: its FP64 sums are cut
// by it.
inline uint32_t stream_grid(uint32_t nbr, uint32_t sms) {
    const uint32_t want = (nbr + kStreamWarps * kStreamBrows - 1) / (kStreamWarps * kStreamBrows);
    return want < 1u ? 1u : want < sms ? want : sms;
}

}  // namespace wsb
