// k_team: see kernels_team.cuh.
//
// What bounds it: below about 25,000 block rows an iteration of the loop
// kernels (kernels_fused.cu) costs 22-28 us whatever the size: three
// dependent launches, each with its ramp, its chain of work-item loads and its
// last-CTA sum. Here an iteration is two exchanges between resident CTAs and
// the latency of one row sum and one block solve:
//   - a lane owns a row (or two): x, r, z and p stay in registers; the matrix, p at
//     every block's columns and the blocks' LU factors stay in shared memory,
//     so an iteration reads only other CTAs' z from the L2, each block of it
//     once a CTA (all row warps fetch, then all read it from shared memory);
//   - p.Ap and then r.r and r.z are all-reduced: every CTA stores its FP64
//     partial as one 16-byte {value, tag} and reads the whole team's in the
//     same fixed order, so all CTAs hold the same scalars and take the same
//     decisions after one hop (r.r by one warp, r.z by another);
//   - z travels as 8-byte {value, tag} packets: a reader waits for the packets
//     it needs and no fence or flag stands between the block solve and the
//     next product. Every CTA forms p = z + beta p for the block columns it
//     multiplies (same operation, same bits as the owner's), so p is never
//     exchanged.
// Measured (B200, us an iteration, loop kernels -> here): 4^3 nodes 24.4 -> 2.8,
// 9^3 23.5 -> 4.3, 12^3 24.8 -> 4.6, 17^3 25.7 -> 4.6, 21^3 27.5 -> 5.3; with
// two parts a CTA 9^3 6.0, 14^3 6.5 (one: 4.6), 20^3 6.8 (5.3), and 22^3 6.5,
// 24^3 6.6, 26^3 6.6 (in k_stream 10.5 to 11). CSR: 4^3 21.3 -> 3.3, 19^3 28.6
// -> 5.7. Single reduction: 4^3 24.6 -> 3.2, 16^3 25.8 -> 5.0, 26^3 28.6 -> 6.8.
// 48 systems of 4^3 to 24^3 nodes at once: 27.6 ms -> 13.2.
// What is left is latency (7 of 13 warps wait at a barrier at any time, issue
// slots 28 % used): per iteration two hops through the L2 (800 cycles for
// 8 CTAs, 1,400 for 31), the FP64 sums (nine cycles an add, 36 with the shuffle
// between lanes), two FP64 divisions and the block solve. So products are
// added through shared memory, 14 per lane as a tree, before the lanes, and two
// parts' side by side (one after the other: 0.6 us more at 22^3); a block
// is solved by one lane from shared memory (no shuffles between its steps); and
// all waits are warp-uniform loops: lanes that leave such a loop one by one
// stay apart and made the code after it up to ten times slower.
// Arithmetic is that of kernels_fused.cu operation by operation; only the
// grouping of the FP64 sums differs.
//
// CSR (kCsr): rows of different lengths have no blocks of columns to share, so z
// and p are kept once a CTA for every column it multiplies with, and each value
// has the 16-bit place of its column (k_team_plan_csr).
//
// Single reduction (kSr): the product multiplies u = M r (in z), p and s = A p
// are formed in the update; the exchanges are the same two.
//
// All CTAs of a launch are resident (cooperative launch); a CTA takes its
// items in list order, and the lists are cut from one global order of systems,
// so the first unfinished system always has all its CTAs. Every wait is
// bounded (StepParams::wait_cycles; that for a CTA which is still in another
// system, by the iterations of the launch): one that runs out sets kErrTeamWait,
// and every CTA leaves.
#include "kernels_team.cuh"
#include "team_device.cuh"

namespace wsb {
namespace {

// The fixed part of a CTA's shared memory.
struct TeamShared {
    double rz, beta;            // the last r.z and beta
    uint2 alpha;                // alpha; 0: the system stops here
    float beta_f;
    uint32_t go;                // 0: the system stops here
    uint32_t err;               // a wait ran out
    uint32_t ext;               // blocks outside the CTA's rows
    // Scalars of the recurrence, kept by one thread (the same in every CTA).
    double bb, rz_old, pap, alpha_d, rr, rel2, abs2;
    uint32_t iter, max_iter, status, breakdown;
    uint32_t bytes[2 * kTeamWarps];  // shared memory of each warp tile
    double rz_prev;             // kSr: the r.z before rz_old
    alignas(16) double v[1];     // the rows' products of a reduction, twice 32 a warp tile
};

struct WaitCtl {
    StepParams *sp;
    long long lim;
};

// Sums of one value per row of each of kT parts (v: 32 kTeamWarps a part), by
// one warp: lane l adds a pair per two warp tiles, as a tree, then the lanes;
// valid in lane 0. The parts' sums run side by side.
template <int kT>
__device__ __forceinline__ void part_sums(const double *v, uint32_t lane, double (&sum)[kT]) {
    constexpr int kPairs = kTeamWarps / 2;
    static_assert(kTeamWarps % 2 == 0, "pairs");
    const double2 *v2 = reinterpret_cast<const double2 *>(v) + lane;
    double s[kT][kPairs];
#pragma unroll
    for (int k = 0; k < kPairs; ++k)
#pragma unroll
        for (int t = 0; t < kT; ++t) {
            const double2 a = v2[16 * kTeamWarps * t + 32 * k];
            s[t][k] = a.x + a.y;
        }
#pragma unroll
    for (int n = kPairs; n > 1; n = (n + 1) / 2)
#pragma unroll
        for (int k = 0; k < n / 2; ++k)
#pragma unroll
            for (int t = 0; t < kT; ++t) s[t][k] += s[t][k + (n + 1) / 2];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int t = 0; t < kT; ++t) s[t][0] += __shfl_down_sync(kFull, s[t][0], o);
#pragma unroll
    for (int t = 0; t < kT; ++t) sum[t] = s[t][0];
}

// More SM cycles than an iteration of k_team takes (34 us at 1.9 GHz).
constexpr long long kTeamIterCycles = 65536;

// Where CTAs have lists of items, one that comes to a system may have to wait for
// one of its team that is still in others, for as long as those iterate
// (`others` cycles at most): the team assembles, and only then the limit of a
// wait counts. Apart from the system's own code, whose loop has no registers for
// it (inside, two parts a CTA ran 3 % slower).
__device__ __noinline__ void team_assemble(const SysDesc &D, uint32_t rank, uint32_t size, uint32_t parts, long long others,
                                           uint32_t *err, StepParams *sp) {
    if (parts >= size) return;
    if (threadIdx.x >> 5 == (uint32_t)kTeamWarps) {
        RedEntry *const red = D.red + (size_t)kRedEntries * team_copies(size) * size;
        const uint32_t tag = D.st->epoch + 1u;
        if ((threadIdx.x & 31u) == 0) st_entry(red + rank / parts, 0.0, tag);
        __syncwarp();
        team_gather(err, red, (size + parts - 1u) / parts, tag, sp, kTeamWaitCycles + others, 0);
    }
    __syncthreads();
}

// One system, this CTA's rows, up to `limit` iterations.
template <int kT, bool kCsr, bool kSr>
__device__ __forceinline__ void team_system(const SysDesc &D, const TeamItem it, uint32_t limit, TeamShared &S,
                                                 char *dyn, const WaitCtl &w) {
    static_assert(!kCsr || kT == 1, "CSR: one part a CTA");
    constexpr int kAhead = 8;  // block columns a lane handles at once
    constexpr uint32_t kRows = 32u * kTeamWarps;  // places for the rows of a part
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    SysState *st = D.st;
    if (!st->active) return;
    const uint32_t tw = D.team_warps;
    const bool lead = it.rank == 0, alone = it.parts >= it.size;
    // The CTA's block rows (BSR6) or rows (CSR).
    const uint32_t part_brows = tw * (uint32_t)kTeamWarpBrows, tile0 = it.rank * tw;
    const uint32_t br0 = kCsr ? D.tile_row[tile0] : min(it.rank * part_brows, D.n / 6u);
    const uint32_t br1 = kCsr ? D.tile_row[min(tile0 + tw, D.n_tiles)] : min(br0 + it.parts * part_brows, D.n / 6u);
    const bool fresh = st->fresh != 0;
    // The warps with rows; the last two warps have none: they reduce. The
    // first of them sums p.Ap and r.r and decides, the second sums r.z and
    // forms beta.
    const bool rows = warp < (uint32_t)kTeamWarps, red_a = warp == (uint32_t)kTeamWarps, red_b = warp == (uint32_t)kTeamWarps + 1u;
    // The lane's rows, one a part.
    const uint32_t bo = lane / 6u, a = lane % 6u;
    bool on[kT];
    uint32_t row[kT], k0[kT], nk[kT], cols[kT], most = 0;  // cols: most blocks of a block row of the warp tile
    float x[kT], r[kT], z[kT], p[kT], s[kT];  // (s: kSr)
    // CSR: the warp tile's first row and block, its rows and blocks.
    uint32_t row0 = 0, blk0 = 0, n_rows = 0, n_blk = 0;
    if (kCsr && warp < tw && tile0 + warp < D.n_tiles) {
        row0 = D.tile_row[tile0 + warp];
        blk0 = D.tile_blk[tile0 + warp];
        n_rows = D.tile_row[tile0 + warp + 1u] - row0;
        n_blk = D.tile_blk[tile0 + warp + 1u] - blk0;
    }
#pragma unroll
    for (int t = 0; t < kT; ++t) {
        const uint32_t br = br0 + (t * tw + warp) * (uint32_t)kTeamWarpBrows + bo;
        on[t] = kCsr ? lane < n_rows : lane < (uint32_t)kTeamWarpRows && warp < tw && (uint32_t)t < it.parts && br < br1;
        row[t] = !on[t] ? 0u : kCsr ? row0 + lane : 6u * br + a;
        k0[t] = nk[t] = 0;
        x[t] = r[t] = z[t] = p[t] = s[t] = 0.0f;
        if (on[t]) {
            const uint32_t *ptr = kCsr ? D.row_ptr + row[t] : D.brow_ptr + br;
            k0[t] = ptr[0];
            nk[t] = ptr[1] - k0[t];
            x[t] = D.x[row[t]];
            if (!fresh) {
                r[t] = D.r[row[t]];
                z[t] = D.z[row[t]];
                p[t] = D.p[row[t]];
                if (kSr) s[t] = D.s[row[t]];
            }
        }
        cols[t] = __reduce_max_sync(kFull, nk[t]);
        most = max(most, cols[t]);
        if (lane == 0 && rows) S.bytes[t * kTeamWarps + warp] = kCsr ? team_csr_tile_bytes(cols[t], n_blk) : team_tile_bytes(cols[t]);
    }
    double *const v0 = S.v, *const v1 = S.v + kT * kRows;
    if (rows)
#pragma unroll
        for (int t = 0; t < kT; ++t) v0[t * kRows + tid] = v1[t * kRows + tid] = 0.0;
    if (tid == 0) S.ext = 0;
    __syncthreads();
    // Dynamic shared memory: z of the CTA's rows (first r, then z, 32 a warp
    // tile) and of the blocks outside, and those blocks' first rows; then for
    // each warp tile its LU factors, 1 / diagonal and the range test of the
    // short division, and for block j of its block rows, lane by lane (no bank
    // conflicts), the row's first four values, its last two, p at the block's
    // columns, and where z of the block's columns is.
    // CSR: z and p of the CTA's rows and of the columns outside, and those
    // columns; then for each warp tile the factors (absent rows of a block are
    // rows of I), and four by four the rows' values and the places of their
    // columns in z and p.
    const uint32_t most_ext = D.team_ext[it.parts - 1u];
    float *const zx = reinterpret_cast<float *>(dyn);
    float *const px = zx + kRows + most_ext;  // (CSR)
    uint32_t *const ext = reinterpret_cast<uint32_t *>(kCsr ? px + kRows + most_ext : zx + kT * kRows + 6u * most_ext);
    char *const tiles = dyn + (kCsr ? team_csr_z_bytes(most_ext) : team_z_bytes(kT, most_ext));
    const float4 *val4 = nullptr;  // (CSR)
    const ushort4 *idx4 = nullptr;
    // (cols == 0: a warp tile without rows; it touches none of this.)
    float *lu[kT], *xg[kT];
    float4 *b4[kT];
    float2 *b2[kT];
    uint32_t *bc[kT];
    auto tile_at = [&](int t) {
        uint32_t before = 0;
        for (uint32_t q = 0; q < t * tw + min(warp, tw); ++q) before += S.bytes[q < tw ? q : kTeamWarps + q - tw];
        return tiles + before;
    };
    auto load_csr = [&]() {
        char *const mine = tile_at(0);
        lu[0] = reinterpret_cast<float *>(mine);
        const uint32_t colp = (cols[0] + 3u) & ~3u;
        float *const val = reinterpret_cast<float *>(mine + n_blk * (uint32_t)kTeamBlockLu);
        uint16_t *const idx = reinterpret_cast<uint16_t *>(val + 32u * colp);
        val4 = reinterpret_cast<const float4 *>(val) + lane;
        idx4 = reinterpret_cast<const ushort4 *>(idx) + lane;
        if (n_rows) {
            if (on[0]) px[32u * warp + lane] = fresh ? x[0] : kSr ? z[0] : p[0];
#pragma unroll 1
            for (uint32_t j = 0; j < nk[0]; ++j) cp_async4(val + 4u * (32u * (j >> 2) + lane) + (j & 3u), D.val + k0[0] + j);
            const char *from = reinterpret_cast<const char *>(D.tile_idx + D.tile_off[tile0 + warp]);
            for (uint32_t q = lane; q < 4u * colp; q += 32u) cp_async16(reinterpret_cast<char *>(idx) + 16u * q, from + 16u * q);
            if (lane < n_blk) {
                const uint32_t m = D.bstart[blk0 + lane + 1u] - D.bstart[blk0 + lane];
#pragma unroll
                for (uint32_t q = 0; q < 36u; ++q)
                    lu[0][36u * lane + q] =
                        q / 6u < m && q % 6u < m ? D.lu[36u * (size_t)(blk0 + lane) + q] : q % 7u == 0 ? 1.0f : 0.0f;
            }
        }
        // The columns outside, their first entries of p (kSr: u; x0 when fresh).
        const uint32_t n = D.ext_count[it.rank];
        if (tid == 0) S.ext = n;
        for (uint32_t i = tid; i < n; i += (uint32_t)kTeamThreads) {
            const uint32_t c = D.ext_cols[(size_t)it.rank * D.ext_cap + i];
            ext[i] = c;
            px[kRows + i] = (fresh ? D.x : kSr ? D.z : D.p)[c];
        }
    };
    auto load_bsr = [&](int t) {
        char *mine = tile_at(t);
        lu[t] = reinterpret_cast<float *>(mine);
        mine += kTeamLuBytes;
        const uint32_t colp = (cols[t] + 7u) & ~7u;
        b4[t] = reinterpret_cast<float4 *>(mine) + lane;
        b2[t] = reinterpret_cast<float2 *>(mine + (size_t)cols[t] * 16u * kTeamWarpRows) + lane;
        xg[t] = reinterpret_cast<float *>(mine + (size_t)cols[t] * 24u * kTeamWarpRows) + 8u * bo;
        bc[t] = reinterpret_cast<uint32_t *>(mine + (size_t)cols[t] * kTeamColBytes);
        for (uint32_t j = lane; j < colp * (uint32_t)(kTeamWarpBrows + 1); j += 32u) bc[t][j] = 0;  // past a row's end
        bc[t] += colp * bo;
        __syncwarp();
        if (on[t]) {
            // p (kSr: u; x0 for a fresh system) at the block columns, one component a lane.
            const float *src = (fresh ? D.x : kSr ? D.z : D.p) + a;
#pragma unroll 1
            for (uint32_t j = 0; j < nk[t]; ++j) {
                const float *v = D.bval + (size_t)(k0[t] + j) * 36u + 6u * a;
                float4 *d4 = b4[t] + j * kTeamWarpRows;
                cp_async8(d4, v);
                cp_async8(reinterpret_cast<float2 *>(d4) + 1, v + 2);
                cp_async8(b2[t] + j * kTeamWarpRows, v + 4);
                const uint32_t c = D.bcol[k0[t] + j];
                cp_async4(xg[t] + 8u * kTeamWarpBrows * j + a, src + 6u * (size_t)c);
                if (a == 0) {
                    if (c >= br0 && c < br1) {
                        const uint32_t q = (c - br0) / kTeamWarpBrows, part = q >= tw ? 1u : 0u;
                        bc[t][j] = part * kRows + 32u * (q - part * tw) + 6u * ((c - br0) % kTeamWarpBrows);
                    } else {
                        const uint32_t e = atomicAdd(&S.ext, 1u);  // (the order changes no value)
                        bc[t][j] = kT * kRows + 6u * e;
                        ext[e] = 6u * c;
                    }
                }
            }
            // The lane's row of the LU factors.
            const uint32_t br = row[t] / 6u;
#pragma unroll
            for (int q = 0; q < 3; ++q) cp_async8(lu[t] + 36u * bo + 6u * a + 2 * q, D.lu + (size_t)br * 36u + 6u * a + 2 * q);
        }
    };
    if (kCsr) load_csr();
    else
#pragma unroll
        for (int t = 0; t < kT; ++t) load_bsr(t);
    cp_async_wait_all();
    __syncwarp();
    // The block that this lane solves (BSR6: lanes 0..4 the first part's, 5..9
    // the second's), its rows, and the first of them in the warp tile.
    const uint32_t st_part = kCsr ? 0u : min(lane / (uint32_t)kTeamWarpBrows, (uint32_t)kT - 1u);
    const uint32_t sbo = kCsr ? min(lane, max(n_blk, 1u) - 1u)
                              : lane < (uint32_t)(kT * kTeamWarpBrows) ? lane % (uint32_t)kTeamWarpBrows : 0u;
    const bool solver = kCsr ? lane < n_blk
                             : lane < (uint32_t)(kT * kTeamWarpBrows) && warp < tw && st_part < it.parts &&
                                   br0 + (st_part * tw + warp) * (uint32_t)kTeamWarpBrows + sbo < br1;
    const uint32_t s_first = kCsr && solver ? D.bstart[blk0 + lane] - row0 : 6u * sbo;
    const uint32_t s_rows = kCsr && solver ? D.bstart[blk0 + lane + 1u] - D.bstart[blk0 + lane] : 6u;
    float *const slu0 = kT > 1 && st_part ? lu[kT - 1] : lu[0];
    const float *const slu = slu0 + 36u * sbo;
    float *const srd = slu0 + 36u * (kCsr ? n_blk : (uint32_t)kTeamWarpBrows) + 8u * sbo;
    if (solver) {
        float dlo = kDivLo;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const float u = slu[7 * i], au = fabsf(u);
            srd[i] = __frcp_rn(u);
            if (!(au >= kDivULo && au <= kDivUHi)) dlo = __int_as_float(0x7f800000);
        }
        srd[6] = dlo;
    }
    __syncthreads();
    const uint32_t n_ext = (kCsr ? 1u : 6u) * S.ext;

    // y = (row) . xg: products rounded, added in index order; the operands of
    // the next block are loaded before this block's products are added. Two
    // rows' sums run side by side.
    float ap[kT];
    auto row_sums_csr = [&]() {
        float acc = 0.0f;
        const float4 *V = val4;
        const ushort4 *I = idx4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f), q = v;
        ushort4 i = make_ushort4(0, 0, 0, 0);
        if (most) {
            v = V[0];
            i = I[0];
            q = make_float4(px[i.x], px[i.y], px[i.z], px[i.w]);
            if (most > 4u) i = I[32];
        }
#pragma unroll 2
        for (uint32_t j = 0; j < most; j += 4u) {
            const float2 p01 = mul2_rn(make_float2(v.x, v.y), make_float2(q.x, q.y));
            const float2 p23 = mul2_rn(make_float2(v.z, v.w), make_float2(q.z, q.w));
            V += 32, I += 32;
            if (j + 4u < most) {
                v = *V;
                q = make_float4(px[i.x], px[i.y], px[i.z], px[i.w]);
                if (j + 8u < most) i = I[32];
            }
            acc = j < nk[0] ? __fadd_rn(acc, p01.x) : acc;
            acc = j + 1u < nk[0] ? __fadd_rn(acc, p01.y) : acc;
            acc = j + 2u < nk[0] ? __fadd_rn(acc, p23.x) : acc;
            acc = j + 3u < nk[0] ? __fadd_rn(acc, p23.y) : acc;
        }
        ap[0] = acc;
    };
    auto row_sums_bsr = [&]() {
        const float4 *B4[kT], *X[kT];
        const float2 *B2[kT];
        float4 v[kT], xv[kT];
        float2 v2[kT], x2[kT];
#pragma unroll
        for (int t = 0; t < kT; ++t) {
            ap[t] = 0.0f;
            B4[t] = b4[t];
            B2[t] = b2[t];
            X[t] = reinterpret_cast<const float4 *>(xg[t]);
            if (nk[t]) v[t] = B4[t][0], v2[t] = B2[t][0], xv[t] = X[t][0], x2[t] = *reinterpret_cast<const float2 *>(X[t] + 1);
        }
#pragma unroll 2
        for (uint32_t j = 0; j < (kT == 1 ? nk[0] : most); ++j) {
            float2 q0[kT], q1[kT], q2[kT];
#pragma unroll
            for (int t = 0; t < kT; ++t) {
                q0[t] = mul2_rn(make_float2(v[t].x, v[t].y), make_float2(xv[t].x, xv[t].y));
                q1[t] = mul2_rn(make_float2(v[t].z, v[t].w), make_float2(xv[t].z, xv[t].w));
                q2[t] = mul2_rn(v2[t], x2[t]);
            }
#pragma unroll
            for (int t = 0; t < kT; ++t)
                if (j + 1 < nk[t]) {
                    B4[t] += kTeamWarpRows, B2[t] += kTeamWarpRows, X[t] += 2 * kTeamWarpBrows;
                    v[t] = *B4[t], v2[t] = *B2[t], xv[t] = X[t][0], x2[t] = *reinterpret_cast<const float2 *>(X[t] + 1);
                }
#pragma unroll
            for (int t = 0; t < kT; ++t) {
                float s = ap[t];
                s = __fadd_rn(s, q0[t].x);
                s = __fadd_rn(s, q0[t].y);
                s = __fadd_rn(s, q1[t].x);
                s = __fadd_rn(s, q1[t].y);
                s = __fadd_rn(s, q2[t].x);
                s = __fadd_rn(s, q2[t].y);
                ap[t] = kT == 1 || j < nk[t] ? s : ap[t];
            }
        }
    };
    // z = U^-1 L^-1 r of the warp tiles' blocks, one lane a block, in the order
    // of block_jacobi.wgsl:93-126; r comes and z goes through zx.
    float *const wz = zx + 32u * min(warp, (uint32_t)kTeamWarps - 1u);
    auto block_solve = [&]() {
#pragma unroll
        for (int t = 0; t < kT; ++t) wz[t * kRows + lane] = r[t];
        __syncwarp();
        if (solver) {
            float y[6], pr[6];
            bool ok = true;
            float *const rz = wz + st_part * kRows + s_first;
            float l[36];
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                const float4 v = reinterpret_cast<const float4 *>(slu)[q];
                l[4 * q] = v.x, l[4 * q + 1] = v.y, l[4 * q + 2] = v.z, l[4 * q + 3] = v.w;
            }
            if (kCsr) {
#pragma unroll
                for (int i = 0; i < 6; ++i) y[i] = (uint32_t)i < s_rows ? rz[i] : 0.0f;
            } else {
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const float2 v = reinterpret_cast<const float2 *>(rz)[i];
                    y[2 * i] = v.x, y[2 * i + 1] = v.y;
                }
            }
            const float4 d0 = reinterpret_cast<const float4 *>(srd)[0], d1 = reinterpret_cast<const float4 *>(srd)[1];
            const float rdiag[6] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y}, dlo = d1.z;
            // (CSR: what an absent row gives is 0 also beside infinities.)
#pragma unroll
            for (int i = 1; i < 6; ++i) {
#pragma unroll
                for (int q = 0; q < i; ++q) y[i] = __fsub_rn(y[i], __fmul_rn(l[6 * i + q], y[q]));
                if (kCsr && (uint32_t)i >= s_rows) y[i] = 0.0f;
            }
#pragma unroll
            for (int i = 5; i >= 0; --i) {
                float v = y[i];
#pragma unroll
                for (int q = i + 1; q < 6; ++q) v = __fsub_rn(v, __fmul_rn(l[6 * i + q], pr[q]));
                pr[i] = div_by(v, l[7 * i], rdiag[i], dlo, &ok);
            }
            if (kCsr) {
#pragma unroll
                for (int i = 0; i < 6; ++i)
                    if ((uint32_t)i < s_rows) rz[i] = ok ? pr[i] : y[i];
                if (!ok) back_general(slu, rz, rz, s_rows);
            } else if (ok) {
#pragma unroll
                for (int i = 0; i < 3; ++i) reinterpret_cast<float2 *>(rz)[i] = make_float2(pr[2 * i], pr[2 * i + 1]);
            } else {
#pragma unroll
                for (int i = 0; i < 6; ++i) rz[i] = y[i];
                back_general(slu, rz, rz, 6);
            }
        }
        __syncwarp();
#pragma unroll
        for (int t = 0; t < kT; ++t) z[t] = wz[t * kRows + lane];
    };

    uint32_t tag = st->epoch;
    // Published partials: one a part, or the sum of the CTA's two where the
    // system never has one part a CTA. This CTA's copy of them; lane l stores to
    // copy l % copies the CTA's partial l / copies.
    const bool pairs = kT > 1 && D.team_pairs;
    const uint32_t copies = team_copies(it.size), mine = lane / copies;
    const uint32_t entries = pairs ? (it.size + 1u) / 2u : it.size, first = pairs ? it.rank / 2u : it.rank;
    const bool publisher = mine < (pairs ? 1u : it.parts) && first + mine < entries;
    const RedEntry *const red = D.red + (size_t)(it.rank / it.parts % copies) * kRedEntries * it.size;
    RedEntry *const out = D.red + (size_t)(lane % copies) * kRedEntries * it.size + first + mine;
    unsigned long long *const zpk = D.zpk;
    // Sum over the system of one value a row, by one warp: the partials of all
    // CTAs in one fixed order (a CTA that holds all adds its two the same way).
    // Valid in lane 0.
    auto all_reduce = [&](const double *v, uint32_t slot, uint32_t tag) {
        double sums[kT];
        part_sums<kT>(v, lane, sums);
        double s = sums[0];
        if (kT > 1 && (alone || pairs)) s += sums[kT - 1];  // (an absent part's is 0)
        if (alone) return s;
        s = __shfl_sync(kFull, s, 0);
        if (kT > 1 && !pairs) {
            const double second = __shfl_sync(kFull, sums[kT - 1], 0);
            s = mine ? second : s;
        }
        if (publisher) st_entry(out + slot * it.size, s, tag);
        __syncwarp();
        return team_gather(&S.err, red + slot * it.size, entries, tag, w.sp, w.lim, quiet_cycles(entries));
    };
    if (red_a && lane == 0) {
        S.bb = st->bb;
        S.rr = S.pap = S.alpha_d = S.beta = 0.0;
        S.beta_f = 0.0f;
        S.rz = S.rz_old = st->rz_old;
        if (kSr && !fresh) {
            S.rz_prev = st->gamma_prev;
            S.alpha_d = st->alpha;
            S.beta = st->beta;
        }
        S.rel2 = st->rel2;
        S.abs2 = st->abs2;
        S.iter = st->iter;
        S.max_iter = st->max_iter;
        S.status = ST_RUNNING;
        S.breakdown = 0;
    }

    // The z packets of the blocks outside the CTA, by its warps with rows, into
    // shared memory, while the scalars are reduced.
    auto fetch_z = [&]() {
        constexpr uint32_t kBatch = 4;
        const uint32_t step = 32u * tw;
#pragma unroll 1
        for (uint32_t b = 0; b < n_ext; b += kBatch * step) {
            // (Only packets that have not come are asked for again: the polls of
            // all CTAs hold up the stores that they wait for.)
            unsigned long long zin[kBatch];
#pragma unroll
            for (uint32_t q = 0; q < kBatch; ++q) zin[q] = b + q * step + tid < n_ext ? 0ull : (unsigned long long)tag << 32;
            const long long t0 = clock64();
#pragma unroll 1
            for (uint32_t k = 1;; ++k) {
                uint32_t bad = 0;
#pragma unroll
                for (uint32_t q = 0; q < kBatch; ++q) {
                    const uint32_t i = b + q * step + tid, e = i / 6u;
                    const bool want = (uint32_t)(zin[q] >> 32) != tag;
                    zin[q] = ld_packet_if(zpk + (!want ? 0u : kCsr ? ext[i] : ext[e] + (i - 6u * e)), want, zin[q]);
                }
#pragma unroll
                for (uint32_t q = 0; q < kBatch; ++q) bad |= (uint32_t)(zin[q] >> 32) ^ tag;
                if (__all_sync(kFull, bad == 0)) break;
                if (__any_sync(kFull, clock64() - t0 > w.lim) ||
                    ((k & 255u) == 0 && __any_sync(kFull, ld_error(w.sp) != 0))) {
                    S.err = 1;
                    break;
                }
            }
#pragma unroll
            for (uint32_t q = 0; q < kBatch; ++q) {
                const uint32_t i = b + q * step + tid;
                if (i < n_ext) zx[kT * kRows + i] = __uint_as_float((uint32_t)zin[q]);
            }
        }
    };
    // p = z + beta p of the lane's rows and of their block columns (p = z when
    // first; kSr: u = z at the columns, p is the update's). All operands come
    // before the first store, which the compiler could not move a load across.
    auto advance_bsr = [&](bool first, float bf) {
#pragma unroll
        for (int t = 0; t < kT; ++t) {
            if (!kSr) p[t] = first ? z[t] : __fadd_rn(__fmul_rn(p[t], bf), z[t]);
#pragma unroll 1
            for (uint32_t j0 = 0; j0 < cols[t]; j0 += kAhead) {
                float *dst = xg[t] + 8u * kTeamWarpBrows * j0 + a;
                float pn[kAhead], zn[kAhead];
#pragma unroll
                for (int q = 0; q < kAhead / 4; ++q) {
                    const uint4 c = reinterpret_cast<const uint4 *>(bc[t] + j0)[q];
                    zn[4 * q] = zx[c.x + a], zn[4 * q + 1] = zx[c.y + a], zn[4 * q + 2] = zx[c.z + a], zn[4 * q + 3] = zx[c.w + a];
                }
#pragma unroll
                for (int j = 0; j < kAhead; ++j) pn[j] = !kSr && j0 + j < nk[t] ? dst[8u * kTeamWarpBrows * j] : 0.0f;
#pragma unroll
                for (int j = 0; j < kAhead; ++j)
                    if (j0 + j < nk[t])
                        dst[8u * kTeamWarpBrows * j] = kSr || first ? zn[j] : __fadd_rn(__fmul_rn(pn[j], bf), zn[j]);
            }
        }
        __syncwarp();
    };

    // CSR: p at every column, once a CTA.
    auto advance_csr = [&](bool first, float bf) {
        if (!kSr) p[0] = first ? z[0] : __fadd_rn(__fmul_rn(p[0], bf), z[0]);
        px[32u * warp + lane] = kSr ? z[0] : p[0];
        for (uint32_t i = kRows + tid; i < kRows + n_ext; i += kRows)
            px[i] = kSr || first ? zx[i] : __fadd_rn(__fmul_rn(px[i], bf), zx[i]);
    };

    // Results of a reduction are written between its two barriers and read by
    // all after the second; S.err may change at any time. The first pass of a
    // fresh system has xg = x0 and stands for k_init: r = b - A x0, z = M r,
    // b.b and r.z, p = z.
    bool init = fresh;
    uint32_t done = 0;
    for (;;) {
        ++tag;
        if (rows) {
            if (kCsr) row_sums_csr();
            else row_sums_bsr();
            __syncwarp();
        }
        if (init) {
            if (rows)
#pragma unroll
                for (int t = 0; t < kT; ++t) {
                    const float bi = on[t] ? __ldg(D.b + row[t]) : 0.0f;
                    r[t] = __fsub_rn(bi, ap[t]);
                    v0[t * kRows + tid] = (double)bi * (double)bi;
                }
        } else {
            if (rows)
#pragma unroll
                for (int t = 0; t < kT; ++t) v0[t * kRows + tid] = (double)(kSr ? z[t] : p[t]) * (double)ap[t];
            __syncthreads();
            if (red_a) {
                const double rz_old = S.rz, pap = all_reduce(v0, 0, tag);
                if (lane == 0) {
                    double den = pap;
                    if (kSr) {
                        // alpha, beta from gamma = (r, u) and delta = (A u, u).
                        double beta = 0.0;
                        if (S.iter != 0) {
                            beta = quotient(rz_old, S.rz_prev);
                            den = S.alpha_d != 0.0 ? pap - quotient(beta * rz_old, S.alpha_d) : 0.0;
                        }
                        S.beta = beta;
                        S.beta_f = (float)beta;
                    }
                    const double alpha = quotient(rz_old, den);
                    S.rz_old = rz_old;
                    S.pap = den;
                    S.alpha_d = alpha;
                    S.alpha = make_uint2(__float_as_uint((float)alpha), S.err ? 0u : 1u);
                }
            }
            __syncthreads();
            const uint2 al2 = S.alpha;
            if (!al2.y) break;
            const float al = __uint_as_float(al2.x), ma = -al;
            const float bf = kSr ? S.beta_f : 0.0f;
            const bool first = kSr && S.iter == 0;
            if (rows)
#pragma unroll
                for (int t = 0; t < kT; ++t) {
                    if (kSr) {
                        p[t] = first ? z[t] : __fadd_rn(__fmul_rn(p[t], bf), z[t]);
                        s[t] = first ? ap[t] : __fadd_rn(__fmul_rn(s[t], bf), ap[t]);
                    }
                    x[t] = __fadd_rn(x[t], __fmul_rn(al, p[t]));
                    r[t] = __fadd_rn(r[t], __fmul_rn(ma, kSr ? s[t] : ap[t]));
                    if (!on[t]) r[t] = 0.0f;
                }
        }
        if (rows) {
            block_solve();
#pragma unroll
            for (int t = 0; t < kT; ++t) {
                if (on[t] && !alone) st_packet(zpk + row[t], z[t], tag);
                if (!init) v0[t * kRows + tid] = (double)r[t] * (double)r[t];
                v1[t * kRows + tid] = (double)r[t] * (double)z[t];
            }
        }
        __syncthreads();
        if (red_a || red_b) {
            const double sum = all_reduce(red_a ? v0 : v1, red_a ? 1u : 2u, tag);
            if (lane == 0 && red_b) {
                if (kSr) {
                    S.rz_prev = S.rz_old;
                } else {
                    const double beta = quotient(sum, S.rz);
                    S.beta = beta;
                    S.beta_f = (float)beta;
                }
                S.rz = sum;
            } else if (lane == 0) {
                uint32_t status = ST_RUNNING;
                if (init) {
                    S.bb = sum;
                    if (sum == 0.0) status = ST_CONVERGED;
                    else if (S.max_iter == 0) status = ST_MAXITER;
                } else {
                    const uint32_t iter = S.iter;
                    S.rr = sum;
                    if (lead && D.history && iter < D.hist_cap) D.history[iter] = sum;
                    if (S.pap == 0.0) {
                        status = ST_BREAKDOWN;
                        S.breakdown = 1;
                    } else if (S.rz_old == 0.0) {
                        status = ST_BREAKDOWN;
                        S.breakdown = 2;
                    } else if (sum <= S.abs2 || sum <= S.rel2 * S.bb) {
                        status = ST_CONVERGED;
                    } else if (iter + 1 >= S.max_iter) {
                        status = ST_MAXITER;
                    }
                    S.iter = iter + 1;
                }
                S.status = status;
                S.go = status == ST_RUNNING && !S.err;
            }
        } else if (warp < tw) {
            fetch_z();
        }
        __syncthreads();
        if (!S.go) break;
        if (kCsr) {
            if (rows) advance_csr(init, S.beta_f);
            __syncthreads();  // p is shared by the CTA
        } else if (rows) {
            advance_bsr(init, S.beta_f);
        }
        if (!init && ++done >= limit) break;
        init = false;
    }
    __syncthreads();
    if (S.err) {
        if (tid == 0) atomicOr(&w.sp->error, kErrTeamWait);
        return;
    }
#pragma unroll
    for (int t = 0; t < kT; ++t)
        if (on[t]) {
            D.x[row[t]] = x[t];
            D.r[row[t]] = r[t];
            D.z[row[t]] = z[t];
            D.p[row[t]] = p[t];
            if (kSr) D.s[row[t]] = s[t];
        }
    if (lead && red_a && lane == 0) {
        const bool running = S.status == ST_RUNNING, none = S.iter == 0;  // none: stopped before the first iteration
        st->bb = S.bb;
        st->rz_old = running || none ? S.rz : S.rz_old;
        if (kSr) st->gamma_prev = S.rz_prev;
        st->pap = S.pap;
        st->rr = S.rr;
        st->rz_new = none ? 0.0 : S.rz;
        st->alpha = S.alpha_d;
        st->beta = none ? 0.0 : S.beta;
        st->alpha_f = (float)S.alpha_d;
        st->beta_f = none ? 0.0f : S.beta_f;
        st->iter = S.iter;
        st->status = S.status;
        st->breakdown = S.breakdown;
        st->epoch = tag;
        st->fresh = 0;
        st->active = running ? 1u : 0u;
    }
}

// kLists: CTAs may have several items. (With one part a CTA the call alone costs
// every iteration 0.02 to 0.05 us, so there is a variant without it.)
template <int kT, bool kCsr, bool kSr, bool kLists>
__global__ void __launch_bounds__(kTeamThreads, 1)
    k_team(const SysDesc *__restrict__ sys, StepParams *sp, const TeamItem *__restrict__ items,
           const uint32_t *__restrict__ item_off, uint32_t limit, uint32_t longest) {
    static_assert(offsetof(TeamShared, v) <= 512, "fixed shared memory");
    extern __shared__ __align__(128) char smem[];
    TeamShared &S = *reinterpret_cast<TeamShared *>(smem);
    const unsigned long long wl = sp->wait_cycles;
    const WaitCtl w{sp, wl == 0 || wl > (unsigned long long)kTeamWaitCycles ? kTeamWaitCycles : (long long)wl};
    if (threadIdx.x == 0) S.err = 0;
    __syncthreads();
    const uint32_t i1 = item_off[blockIdx.x + 1];
    for (uint32_t i = item_off[blockIdx.x]; i < i1; ++i) {
        const TeamItem it = items[i];
        if (kLists && longest > 1u) {
            team_assemble(sys[it.sys], it.rank, it.size, it.parts, kTeamIterCycles * longest * limit, &S.err, sp);
            if (S.err) {
                if (threadIdx.x == 0) atomicOr(&sp->error, kErrTeamWait);
                return;
            }
        }
        team_system<kT, kCsr, kSr>(sys[it.sys], it, limit, S, smem + team_fixed_bytes(kT), w);
        __syncthreads();
        if (S.err) {  // every CTA's later waits would run out as well
            // (Its teammates may have come to the end: the system has failed.)
            if (threadIdx.x == 0) sys[items[i].sys].st->failed = 1;
            return;
        }
    }
}

// The columns of one part (one CTA) that are not its own rows, each once, and
// for each nonzero the place of its column among the part's rows and those, in
// the order in which k_team keeps the values. The numbers come in any order:
// they choose places, not values. most[0]: the most such columns of a part;
// most[1]: more than D.ext_cap (nothing is iterated from such a plan).
constexpr uint32_t kPlanHash = 2 * kTeamMaxExt, kPlanThreads = 512;
static_assert((kPlanHash & (kPlanHash - 1)) == 0 && kTeamMaxExt + kPlanThreads < kPlanHash, "the table never fills");
__global__ void __launch_bounds__(kPlanThreads) k_team_plan_csr(SysDesc D, uint32_t *count, uint32_t *most) {
    extern __shared__ uint32_t table[];  // keys, then places
    __shared__ uint32_t found, first[kTeamWarps + 1];
    uint32_t *const place = table + kPlanHash;
    const uint32_t tid = threadIdx.x, tw = D.team_warps, tile0 = blockIdx.x * tw, tiles = min(tw, D.n_tiles - tile0);
    for (uint32_t i = tid; i < kPlanHash; i += kPlanThreads) table[i] = 0xffffffffu;
    if (tid <= tiles) first[tid] = D.tile_row[tile0 + tid];
    if (tid == 0) found = 0;
    __syncthreads();
    const uint32_t r0 = first[0], r1 = first[tiles], k0 = D.row_ptr[r0], k1 = D.row_ptr[r1];
    const volatile uint32_t *const now = &found;
    for (uint32_t k = k0 + tid; k < k1; k += kPlanThreads) {
        const uint32_t c = D.col[k];
        if (c >= r0 && c < r1) continue;
        uint32_t h = (c * 2654435761u) & (kPlanHash - 1u);
        while (*now <= D.ext_cap) {
            const uint32_t old = atomicCAS(&table[h], 0xffffffffu, c);
            if (old == c) break;
            if (old == 0xffffffffu) {
                const uint32_t e = atomicAdd(&found, 1u);
                place[h] = kTeamWarps * 32u + e;
                if (e < D.ext_cap) D.ext_cols[(size_t)blockIdx.x * D.ext_cap + e] = c;
                break;
            }
            h = (h + 1u) & (kPlanHash - 1u);
        }
    }
    __syncthreads();
    if (tid == 0) {
        count[blockIdx.x] = min(found, D.ext_cap);
        if (found > D.ext_cap) most[1] = 1u;
        atomicMax(most, found);
    }
    if (found > D.ext_cap) return;
    for (uint32_t t = 0; t < tiles; ++t) {
        uint16_t *const idx = D.tile_idx + D.tile_off[tile0 + t];
        const uint32_t lane = tid & 31u, nr = first[t + 1] - first[t];
        uint32_t s = 0, nk = 0;
        if (lane < nr) {
            s = D.row_ptr[first[t] + lane];
            nk = D.row_ptr[first[t] + lane + 1u] - s;
        }
        const uint32_t colp = (__reduce_max_sync(kFull, nk) + 3u) & ~3u;
        for (uint32_t j = tid >> 5; j < colp; j += kPlanThreads / 32u) {
            uint32_t at = 0;  // (past a row's end: not used)
            if (j < nk) {
                const uint32_t c = D.col[s + j];
                if (c >= r0 && c < r1) {
                    uint32_t q = 0;
                    while (c >= first[q + 1]) ++q;
                    at = 32u * q + (c - first[q]);
                } else {
                    uint32_t h = (c * 2654435761u) & (kPlanHash - 1u);
                    while (table[h] != c) h = (h + 1u) & (kPlanHash - 1u);
                    at = place[h];
                }
            }
            idx[4u * (32u * (j >> 2) + lane) + (j & 3u)] = (uint16_t)at;
        }
    }
}

}  // namespace

template <bool kSr>
static const void *team_kernel_of(int parts, bool csr, bool lists) {
    return parts == 2 ? (const void *)k_team<2, false, kSr, true>
           : csr      ? (lists ? (const void *)k_team<1, true, kSr, true> : (const void *)k_team<1, true, kSr, false>)
                      : (lists ? (const void *)k_team<1, false, kSr, true> : (const void *)k_team<1, false, kSr, false>);
}
const void *team_kernel(int parts, bool csr, bool single_reduction, bool lists) {
    return single_reduction ? team_kernel_of<true>(parts, csr, lists) : team_kernel_of<false>(parts, csr, lists);
}

cudaError_t team_plan_csr(const SysDesc &D, uint32_t *count, uint32_t *most, uint32_t parts, cudaStream_t st) {
    constexpr int bytes = 8 * (int)kPlanHash;
    cudaError_t e = cudaFuncSetAttribute(k_team_plan_csr, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    k_team_plan_csr<<<parts, kPlanThreads, bytes, st>>>(D, count, most);
    return cudaGetLastError();
}

}  // namespace wsb
