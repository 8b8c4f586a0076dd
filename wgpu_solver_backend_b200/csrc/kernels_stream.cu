// k_stream: see kernels_stream.cuh.
//
// What bounds it: the matrix and the LU factors, 171 bytes a row and iteration
// for a 7-point lattice, come from HBM (or, below about 100 MB, from the L2);
// the vectors stay in the L2. The loop kernels read the same bytes but paid
// three launches an iteration (ramp, drain and last-CTA sums, 23 us at any
// size) and computed each tile behind CTA-wide barriers. Here:
//   - every warp is its own pipeline: lane 0 keeps two bulk copies in flight
//     into the warp's two stages, the warp waits for its own stage only; no
//     CTA barrier inside a phase;
//   - an iteration is two phases with an all-reduce after each (one 16-byte
//     {value, tag} per CTA, polled by all, as in k_team). What the next phase
//     streams first (factors, x and r; matrix values) is requested before the
//     all-reduce ends, so HBM works through it;
//   - p = z + beta p is formed where p is gathered (both vectors in the L2) and
//     written once by its owner to the other of two buffers, so there is no
//     pass of its own for it.
// Product phase: a lane owns a row, its 6x6 blocks from the stage, products
// rounded and added in index order. Update phase: a lane owns a block (block
// solve in registers); x and r (kSr: p and s too) go back into the stage and out
// by bulk stores, z goes straight to memory.
// Arithmetic is that of kernels_fused.cu operation by operation; only the
// grouping of the FP64 sums differs (per lane over its tiles, warp, CTA, device).
//
// Measured (B200, us an iteration, loop kernels -> here): 32^3 nodes 31.8 ->
// 12.9, 40^3 41.5 -> 18.5 (single reduction 39.2 -> 18.5), 64^3 87.0 -> 61.3,
// 80^3 145.9 -> 114.5 (with the gathers behind the wait for the tile's values
// 15.2, 21, 65, 122). At 80^3 the product runs at the copy rate of HBM; up to
// 40^3 the two all-reduces (1.5 us each over 148 CTAs, as long alone) and the
// latencies around them are half of the time, and the product (200 cycles a
// tile and SM; its bytes need 70 from the L2) waits for shared-memory and
// gather wavefronts, 60 % of what the SM can issue.
//
// Single reduction (kSr): the update phase comes first with alpha and beta of
// the last iteration; the product multiplies u = M r (in z).
//
// All CTAs are resident (cooperative launch). Every wait is bounded: one that
// runs out sets kErrTeamWait, the CTA drains its copies in flight, and all
// leave at the next reduction.
#include "kernels_stream.cuh"
#include "kernels_team.cuh"
#include "team_device.cuh"

namespace wsb {
namespace {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P;\n\tmbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\tselp.u32 %0, 1, 0, P;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// By a whole warp, which leaves together.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, long long lim) {
    if (__all_sync(kFull, mbar_try(bar, parity))) return true;
    const long long t0 = clock64();
    while (!__all_sync(kFull, mbar_try(bar, parity)))
        if (__any_sync(kFull, clock64() - t0 > lim)) return false;
    return true;
}
// 1-D bulk copies (no multicast): addresses 16-byte aligned, bytes a multiple
// of 16 (none at 0). `pol`: an L2 eviction policy for data read once an iteration.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    if (bytes)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_u32(dst)),
                     "l"(src), "r"(bytes), "r"(smem_u32(bar))
                     : "memory");
}
__device__ __forceinline__ void bulk_load_hint(void *dst, const void *src, uint32_t bytes, uint64_t *bar, uint64_t pol) {
    if (bytes)
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::
                "r"(smem_u32(dst)),
            "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(pol)
            : "memory");
}
__device__ __forceinline__ void bulk_store(void *dst, const void *src, uint32_t bytes) {
    if (bytes)
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)),
                     "r"(bytes)
                     : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Orders this thread's accesses to shared memory before later bulk copies
// to or from it; the second also its global writes before later bulk loads.
__device__ __forceinline__ void fence_proxy_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

struct StreamShared {
    uint64_t bar[kStreamWarps][2];
    double w[2][kStreamWarps];  // warp partials of a reduction
    double rz, rz_prev, beta;
    double bb, rz_old, pap, alpha_d, rr, rel2, abs2;
    float alpha, beta_f;
    uint32_t iter, max_iter, status, breakdown;
    uint32_t go;   // 0: the system stops here
    uint32_t err;  // a wait ran out
};
static_assert(sizeof(StreamShared) <= kStreamFixedSmem, "fixed shared memory");

// Sum of the 16 warp partials of value `c`, by the calling warp, published.
__device__ __forceinline__ double publish(StreamShared &S, uint32_t c, RedEntry *out, uint32_t copies, uint32_t tag,
                                          bool release) {
    const uint32_t lane = threadIdx.x & 31u;
    double v = lane < (uint32_t)kStreamWarps ? S.w[c][lane] : 0.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
    v = __shfl_sync(kFull, v, 0);
    if (gridDim.x > 1) {
        if (release) __threadfence();  // the CTA's writes, ordered here by its barrier
        if (lane < copies) st_entry(out, v, tag);
    }
    __syncwarp();
    return v;
}

template <bool kSr>
__device__ __forceinline__ void stream_system(const SysDesc &D, uint32_t limit, StreamShared &S, char *dyn, StepParams *sp,
                                              long long lim) {
    // kVecs: vectors that an update tile stages.
    constexpr uint32_t kUpd = kSr ? kStreamUpdBrowsSr : kStreamUpdBrows, kVecs = kSr ? 4u : 2u;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    SysState *st = D.st;
    if (!st->active || st->fresh) return;  // (fresh: a wait of the init kernels ran out)
    // This CTA's block rows (an even first one: 16-byte aligned slices).
    const uint32_t nbr = D.n / 6u, half = (nbr + 1u) / 2u;
    const uint32_t b0 = min(nbr, 2u * (uint32_t)((uint64_t)blockIdx.x * half / gridDim.x));
    const uint32_t b1 = min(nbr, 2u * (uint32_t)((uint64_t)(blockIdx.x + 1) * half / gridDim.x));
    const uint32_t rows = b1 - b0;
    const uint32_t tiles_a = (rows + kStreamBrows - 1) / kStreamBrows;
    // Update tiles: as few passes over the warps as tiles of kUpd block rows
    // need, evenly filled.
    const uint32_t passes = (rows + kUpd * kStreamWarps - 1) / (kUpd * kStreamWarps);
    const uint32_t tu = passes ? min(kUpd, (((rows + passes * kStreamWarps - 1) / (passes * kStreamWarps)) + 1u) & ~1u) : kUpd;
    const uint32_t tiles_u = (rows + tu - 1) / tu;
    uint64_t *const bar = S.bar[warp];
    char *const stage = dyn + (size_t)warp * kStreamWarpBytes;
    uint32_t *const cols = reinterpret_cast<uint32_t *>(stage + 2 * kStreamSpmvStage);
    float *const xg = reinterpret_cast<float *>(stage + 2 * kStreamSpmvStage + kStreamColBytes);
    // The lane's row in a product tile: block row bo, row a of it. The third
    // block row's lanes are turned by two: with seven blocks a block row the
    // 16 lanes of a half-warp then read 16 different bank pairs.
    const uint32_t bo = lane / 6u, a = bo == 2u ? (lane - 10u) % 6u : lane % 6u, after = min(6u * (bo + 1u), 30u);
    const uint32_t trow = 6u * bo + a;  // the row in the tile
    // Data larger than the L2 streams past it.
    uint64_t pol;
    if (D.stream_past_l2) asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    else asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(pol));

    const uint32_t copies = team_copies(gridDim.x);
    const RedEntry *const red = D.red + (size_t)(blockIdx.x % copies) * kRedEntries * gridDim.x;
    RedEntry *const out = D.red + (size_t)(lane % copies) * kRedEntries * gridDim.x + blockIdx.x;
    uint32_t tag = st->epoch, phases = 0;  // phases: the parity each stage's barrier completes next
    if (tid == 0) {
        S.bb = st->bb;
        S.rz = S.rz_old = st->rz_old;
        S.rz_prev = st->gamma_prev;
        S.rr = st->rr;
        S.pap = st->pap;
        S.alpha_d = st->alpha;
        S.beta = st->beta;
        S.alpha = st->alpha_f;
        S.beta_f = st->beta_f;
        S.rel2 = st->rel2;
        S.abs2 = st->abs2;
        S.iter = st->iter;
        S.max_iter = st->max_iter;
        S.status = ST_RUNNING;
        S.breakdown = 0;
    }
    __syncthreads();

    // ---- product phase -----------------------------------------------------
    // Row pointers of tile t: a lane has that of its block row, lanes 30 and 31
    // the tile's end.
    auto row_ptrs = [&](uint32_t t) { return __ldg(D.brow_ptr + min(b0 + t * kStreamBrows + bo, b1)); };
    auto issue_a = [&](uint32_t rp, uint32_t s) {
        const uint32_t k0 = __shfl_sync(kFull, rp, 0), k1 = __shfl_sync(kFull, rp, 30);
        if (lane == 0) {
            mbar_expect(bar + s, 144u * (k1 - k0));
            bulk_load_hint(stage + s * kStreamSpmvStage, D.bval + (size_t)k0 * 36u, 144u * (k1 - k0), bar + s, pol);
        }
        __syncwarp();
    };
    // The block columns of a tile, two a lane.
    uint32_t col0 = 0, col1 = 0;
    auto load_cols = [&](uint32_t rp) {
        const uint32_t k = __shfl_sync(kFull, rp, 0) + lane, k1 = __shfl_sync(kFull, rp, 30);
        col0 = k < k1 ? __ldg(D.bcol + k) : 0u;
        col1 = k + 32u < k1 ? __ldg(D.bcol + k + 32u) : 0u;
    };
    auto stage_cols = [&]() {
        cols[lane] = col0;
        if (lane + 32u < kStreamColBytes / 4u) cols[lane + 32u] = col1;
        __syncwarp();
    };
    auto wait_stage = [&](uint32_t s) {
        if (!mbar_wait(bar + s, (phases >> s) & 1u, lim)) {
            S.err = 1;
            // The copies still land in this CTA's shared memory: wait for them.
            mbar_wait(bar + s, (phases >> s) & 1u, kTeamWaitCycles);
        }
        phases ^= 1u << s;
    };
    // Row pointers of the first three tiles, and of this tile and the next two.
    const uint32_t rpa = row_ptrs(warp), rpb = row_ptrs(warp + kStreamWarps), rpc = row_ptrs(warp + 2 * kStreamWarps);
    uint32_t rp0 = 0, rp1 = 0, rp2 = 0;
    auto start_a = [&]() {
        rp0 = rpa;
        rp1 = rpb;
        rp2 = rpc;
        if (warp < tiles_a) issue_a(rp0, 0);
        if (warp + kStreamWarps < tiles_a) issue_a(rp1, 1);
        load_cols(rp0);
    };
    float zq[kStreamMaxCols], pq[kStreamMaxCols], z_own = 0.0f, p_own = 0.0f;
    // Requests the gathered vectors of a tile whose columns are in `cols`. Plain
    // loads: the reduction's acquire has dropped the L1's older lines, and a
    // value is gathered by several rows of this SM.
    auto gather = [&](uint32_t t, uint32_t rp, const float *pv) {
        const uint32_t k0 = __shfl_sync(kFull, rp, 0), end = __shfl_sync(kFull, rp, after);
        const uint32_t nk = lane < 30u ? end - rp : 0u;
        const uint32_t *c = cols + (rp - k0);
#pragma unroll
        for (int j = 0; j < kStreamMaxCols; ++j) {
            zq[j] = pq[j] = 0.0f;
            if ((uint32_t)j < nk) {
                const uint32_t i = 6u * c[j] + a;
                zq[j] = D.z[i];
                if (!kSr) pq[j] = pv[i];
            }
        }
        z_own = p_own = 0.0f;
        if (nk) {
            const size_t i = 6u * (size_t)(b0 + t * kStreamBrows) + trow;
            z_own = D.z[i];
            if (!kSr) p_own = pv[i];
        }
    };
    // w = A v over the CTA's rows (v = z + beta p, or z: first, kSr); returns
    // the lane's FP64 sum of v . w.
    auto product = [&](bool first, float bf, const float *pv, float *pw) {
        double sum = 0.0;
        if (warp < tiles_a) {
            stage_cols();
            gather(warp, rp0, pv);
            load_cols(rp1);
        }
        uint32_t s = 0;
        for (uint32_t t = warp; t < tiles_a; t += kStreamWarps, s ^= 1u) {
            const uint32_t rp = rp0;
            const uint32_t next = __shfl_sync(kFull, rp, after), k0 = __shfl_sync(kFull, rp, 0);
            const uint32_t nk = lane < 30u ? next - rp : 0u;
            float *const xl = xg + 8u * bo;
#pragma unroll
            for (int j = 0; j < kStreamMaxCols; ++j)
                if ((uint32_t)j < nk)
                    xl[8u * (kStreamBrows + 1) * j + a] = kSr || first ? zq[j] : __fadd_rn(__fmul_rn(pq[j], bf), zq[j]);
            const float own = kSr || first ? z_own : __fadd_rn(__fmul_rn(p_own, bf), z_own);
            // The next tile's gathers, the columns of the one after it and the
            // row pointers of a third run behind this tile's sums; they do not
            // wait for the matrix values (that wait for each tile's bulk copy
            // took half of the product phase).
            stage_cols();
            if (t + kStreamWarps < tiles_a) gather(t + kStreamWarps, rp1, pv);
            if (t + 2 * kStreamWarps < tiles_a) load_cols(rp2);
            uint32_t rp3 = 0;
            if (t + 3 * kStreamWarps < tiles_a) rp3 = row_ptrs(t + 3 * kStreamWarps);
            wait_stage(s);
            float acc = 0.0f;
            const float2 *B = reinterpret_cast<const float2 *>(stage + s * kStreamSpmvStage) + (size_t)(rp - k0) * 18u + 3u * a;
            const float4 *X = reinterpret_cast<const float4 *>(xl);
#pragma unroll
            for (int j = 0; j < kStreamMaxCols; ++j) {
                if ((uint32_t)j < nk) {
                    const float4 x = X[2 * (kStreamBrows + 1) * j];
                    const float2 x2 = *reinterpret_cast<const float2 *>(X + 2 * (kStreamBrows + 1) * j + 1);
                    const float2 q0 = mul2_rn(B[18 * j], make_float2(x.x, x.y));
                    const float2 q1 = mul2_rn(B[18 * j + 1], make_float2(x.z, x.w));
                    const float2 q2 = mul2_rn(B[18 * j + 2], x2);
                    acc = __fadd_rn(acc, q0.x);
                    acc = __fadd_rn(acc, q0.y);
                    acc = __fadd_rn(acc, q1.x);
                    acc = __fadd_rn(acc, q1.y);
                    acc = __fadd_rn(acc, q2.x);
                    acc = __fadd_rn(acc, q2.y);
                }
            }
            __syncwarp();  // the stage and xg are read
            if (t + 2 * kStreamWarps < tiles_a) issue_a(rp2, s);
            rp0 = rp1;
            rp1 = rp2;
            rp2 = rp3;
            if (lane < 30u && b0 + t * kStreamBrows + bo < b1) {
                const size_t i = 6u * (size_t)(b0 + t * kStreamBrows) + trow;
                D.ap[i] = acc;
                if (!kSr) pw[i] = own;
                sum += (double)own * (double)acc;
            }
        }
        return sum;
    };

    // ---- update phase ------------------------------------------------------
    // Slices of a stage: x, r (kSr: p, s), which come and go by bulk copies. What
    // the product has just written (A p and p; kSr: w) and u = z are read and z is
    // written by plain accesses: a bulk load of them would need a proxy fence
    // behind the product, and a bulk store of z would have to be waited for before
    // the reduction. (z as {value, tag} packets, which need no fence, doubled the
    // gathers' bytes: 80^3 125 -> 139 us.)
    auto slice = [&](uint32_t s, uint32_t v) {
        return reinterpret_cast<float *>(stage + s * kStreamUpdStage + kUpd * 144u) + v * kUpd * 6u;
    };
    auto vec = [&](uint32_t v) -> float * { return v == 0 ? D.x : v == 1 ? D.r : v == 2 ? D.p : D.s; };
    // The factors and the slices, one bulk copy a lane.
    auto issue_u = [&](uint32_t u, uint32_t s) {
        const uint32_t r0 = b0 + u * tu, nb = min(tu, b1 - r0);
        const uint32_t vb = (24u * nb + 15u) & ~15u;
        if (lane == 0) mbar_expect(bar + s, 144u * nb + kVecs * vb);
        __syncwarp();
        if (lane == kVecs) bulk_load_hint(stage + s * kStreamUpdStage, D.lu + 36u * (size_t)r0, 144u * nb, bar + s, pol);
        else if (lane < kVecs) bulk_load(slice(s, lane), vec(lane) + 6u * (size_t)r0, vb, bar + s);
        __syncwarp();
    };
    auto start_u = [&]() {
        if (lane < kVecs) bulk_wait_all();  // the last update's stores: x and r are read again
        __syncwarp();
        if (warp < tiles_u) issue_u(warp, 0);
        if (warp + kStreamWarps < tiles_u) issue_u(warp + kStreamWarps, 1);
    };
    // The lane's rows of p (kSr: u) and A p, requested ahead. This SM wrote
    // them, so its L1 has no other value.
    float2 pv[3], wv[3];
    auto fetch_u = [&](uint32_t u, const float *pn) {
        const uint32_t r0 = b0 + u * tu, nb = min(tu, b1 - r0);
        if (lane < nb) {
            const size_t i = 6u * (size_t)(r0 + lane);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                pv[q] = *reinterpret_cast<const float2 *>((kSr ? D.z : pn) + i + 2 * q);
                wv[q] = *reinterpret_cast<const float2 *>(D.ap + i + 2 * q);
            }
        }
    };
    // Bulk stores of a tile's x and r (p and s), all but the last 8 bytes of an
    // odd number of block rows.
    auto store_u = [&](uint32_t u, uint32_t s) {
        const uint32_t r0 = b0 + u * tu, nb = min(tu, b1 - r0);
        if (lane < kVecs) {
            bulk_store(vec(lane) + 6u * (size_t)r0, slice(s, lane), (24u * nb) & ~15u);
            bulk_commit();
        }
    };
    // Those of the warp's last tile wait until the partials are published: the
    // fence before that would wait for them.
    uint32_t last_u = 0, last_s = 0;
    auto finish_u = [&]() {
        if (warp < tiles_u) store_u(last_u, last_s);
        if (lane < kVecs) bulk_wait_read();  // the stages are free
        fence_proxy_smem();
        __syncwarp();
    };
    auto update = [&](float al, float bf, bool first, const float *pn, double &rr, double &rz) {
        uint32_t s = 0;
        for (uint32_t u = warp; u < tiles_u; u += kStreamWarps, s ^= 1u) {
            const uint32_t r0 = b0 + u * tu, nb = min(tu, b1 - r0);
            wait_stage(s);
            if (lane < nb) {
                const float ma = -al;
                float2 *const x2 = reinterpret_cast<float2 *>(slice(s, 0)) + 3u * lane;
                float2 *const r2 = reinterpret_cast<float2 *>(slice(s, 1)) + 3u * lane;
                float2 *const p2 = reinterpret_cast<float2 *>(slice(s, 2)) + 3u * lane;
                float2 *const s2 = reinterpret_cast<float2 *>(slice(s, kSr ? 3 : 2)) + 3u * lane;
                const float4 *lu = reinterpret_cast<const float4 *>(stage + s * kStreamUpdStage) + 9u * lane;
                float L[36], r[6], y[6];
#pragma unroll
                for (int q = 0; q < 9; ++q) {
                    const float4 v = lu[q];
                    L[4 * q] = v.x, L[4 * q + 1] = v.y, L[4 * q + 2] = v.z, L[4 * q + 3] = v.w;
                }
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    float2 x = x2[q], p = pv[q], w = wv[q];
                    const float2 ro = r2[q];
                    if (kSr) {
                        const float2 uu = p, po = p2[q], so = s2[q];
                        p.x = first ? uu.x : __fadd_rn(__fmul_rn(po.x, bf), uu.x);
                        p.y = first ? uu.y : __fadd_rn(__fmul_rn(po.y, bf), uu.y);
                        w.x = first ? w.x : __fadd_rn(__fmul_rn(so.x, bf), w.x);
                        w.y = first ? w.y : __fadd_rn(__fmul_rn(so.y, bf), w.y);
                        p2[q] = p;
                        s2[q] = w;
                    }
                    x.x = __fadd_rn(x.x, __fmul_rn(al, p.x));
                    x.y = __fadd_rn(x.y, __fmul_rn(al, p.y));
                    r[2 * q] = __fadd_rn(ro.x, __fmul_rn(ma, w.x));
                    r[2 * q + 1] = __fadd_rn(ro.y, __fmul_rn(ma, w.y));
                    x2[q] = x;
                    r2[q] = make_float2(r[2 * q], r[2 * q + 1]);
                    rr += (double)r[2 * q] * (double)r[2 * q];
                    rr += (double)r[2 * q + 1] * (double)r[2 * q + 1];
                }
                if (u + kStreamWarps < tiles_u) fetch_u(u + kStreamWarps, pn);
#pragma unroll
                for (int i = 0; i < 6; ++i) {
                    float t = r[i];
#pragma unroll
                    for (int q = 0; q < i; ++q) t = __fsub_rn(t, __fmul_rn(L[6 * i + q], y[q]));
                    y[i] = t;
                }
#pragma unroll
                for (int i = 5; i >= 0; --i) {
                    float t = y[i];
#pragma unroll
                    for (int q = i + 1; q < 6; ++q) t = __fsub_rn(t, __fmul_rn(L[6 * i + q], y[q]));
                    y[i] = __fdiv_rn(t, L[7 * i]);
                }
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    reinterpret_cast<float2 *>(D.z + 6u * (size_t)(r0 + lane))[q] = make_float2(y[2 * q], y[2 * q + 1]);
#pragma unroll
                for (int i = 0; i < 6; ++i) rz += (double)r[i] * (double)y[i];
            }
            fence_proxy_smem();
            __syncwarp();
            const size_t i0 = 6u * (size_t)r0;
            const uint32_t bytes = (24u * nb) & ~15u;
            last_u = u;
            last_s = s;
            if (u + kStreamWarps < tiles_u) store_u(u, s);
            if (24u * nb > bytes && lane < 2u) {
                const uint32_t o = bytes / 4u + lane;
#pragma unroll
                for (uint32_t v = 0; v < kVecs; ++v) vec(v)[i0 + o] = slice(s, v)[o];
                fence_proxy_all();  // read by the next update's bulk loads
            }
            __syncwarp();
            if (u + 2 * kStreamWarps < tiles_u) {
                if (lane < kVecs) bulk_wait_read();
                fence_proxy_smem();
                __syncwarp();
                issue_u(u + 2 * kStreamWarps, s);
            }
        }
    };

    // ---- iterations --------------------------------------------------------
    start_a();
    bool asked = true;  // product stages are requested
    uint32_t done = 0;
    for (;;) {
        const uint32_t iter = S.iter;
        const bool first = iter == 0;
        // The two buffers of p: read from one, written to the other.
        float *const p_old = kSr ? D.p : (iter & 1u ? D.p2 : D.p), *const p_new = kSr ? D.p : (iter & 1u ? D.p : D.p2);
        const double pw = warp_sum(product(first, S.beta_f, p_old, p_new));
        ++tag;
        if (lane == 0) S.w[0][warp] = pw;
        fence_proxy_smem();
        __syncthreads();
        double pap = 0.0;
        if (warp == 0) pap = publish(S, 0, out, copies, tag, false);
        // The update's stages reuse the product's.
        start_u();
        if (warp < tiles_u) fetch_u(warp, p_new);
        if (warp == 0) {
            if (gridDim.x > 1) pap = team_gather(&S.err, red, gridDim.x, tag, sp, lim, 0);
            if (lane == 0) {
                double alpha;
                if (kSr) {
                    // alpha, beta from gamma = (r, u) and delta = (A u, u).
                    const double gamma = S.rz;
                    double beta = 0.0, den = pap;
                    if (!first) {
                        beta = quotient(gamma, S.rz_prev);
                        den = S.alpha_d != 0.0 ? pap - quotient(beta * gamma, S.alpha_d) : 0.0;
                    }
                    alpha = quotient(gamma, den);
                    S.pap = den;
                    S.beta = beta;
                    S.beta_f = (float)beta;
                } else {
                    alpha = quotient(S.rz, pap);
                    S.pap = pap;
                }
                S.rz_old = S.rz;
                S.alpha_d = alpha;
                S.alpha = (float)alpha;
                S.go = !S.err;
            }
        }
        __syncthreads();
        const bool go = S.go != 0;
        double rr = 0.0, rz = 0.0;
        update(S.alpha, S.beta_f, first, p_new, rr, rz);
        rr = warp_sum(rr);
        rz = warp_sum(rz);
        asked = go;
        if (!go) {
            finish_u();
            break;
        }
        if (lane == 0) {
            S.w[0][warp] = rr;
            S.w[1][warp] = rz;
        }
        __syncthreads();
        // The next product's stages are requested after the fence, which would
        // wait for them.
        const uint32_t slot = (warp + 1u) * gridDim.x;
        double sum = 0.0;
        if (warp < 2) sum = publish(S, warp, out + slot, copies, tag, true);
        finish_u();
        start_a();
        if (warp < 2 && gridDim.x > 1) {
            sum = team_gather(&S.err, red + slot, gridDim.x, tag, sp, lim, 0);
            __threadfence();  // what the publishers wrote is visible after this
        }
        if (warp == 1) {
            if (lane == 0) {
                if (!kSr) {
                    const double beta = quotient(sum, S.rz_old);
                    S.beta = beta;
                    S.beta_f = (float)beta;
                }
                S.rz_prev = S.rz_old;
                S.rz = sum;
            }
        } else if (warp == 0) {
            if (lane == 0) {
                uint32_t status = ST_RUNNING;
                S.rr = sum;
                if (blockIdx.x == 0 && D.history && iter < D.hist_cap) D.history[iter] = sum;
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
                S.status = status;
                S.go = status == ST_RUNNING && !S.err;
            }
        }
        __syncthreads();
        if (!S.go || ++done >= limit) break;
    }
    // The product stages requested for an iteration that does not come (an
    // error seen before the update left none).
    if (asked) {
        if (warp < tiles_a) wait_stage(0);
        if (warp + kStreamWarps < tiles_a) wait_stage(1);
    }
    __syncthreads();
    if (S.err) {
        if (tid == 0) {
            atomicOr(&sp->error, kErrTeamWait);
            st->failed = 1;
        }
        return;
    }
    if (blockIdx.x == 0 && tid == 0) {
        const bool running = S.status == ST_RUNNING;
        st->rz_old = running ? S.rz : S.rz_old;
        st->gamma_prev = S.rz_prev;
        st->pap = S.pap;
        st->rr = S.rr;
        st->rz_new = S.rz;
        st->alpha = S.alpha_d;
        st->beta = S.beta;
        st->alpha_f = S.alpha;
        st->beta_f = S.beta_f;
        st->iter = S.iter;
        st->status = S.status;
        st->breakdown = S.breakdown;
        st->epoch = tag;
        st->active = running ? 1u : 0u;
    }
}

template <bool kSr>
__global__ void __launch_bounds__(kStreamThreads, 1)
    k_stream(const SysDesc *__restrict__ sys, StepParams *sp, uint32_t system, uint32_t limit) {
    extern __shared__ __align__(128) char smem[];
    StreamShared &S = *reinterpret_cast<StreamShared *>(smem);
    const unsigned long long wl = sp->wait_cycles;
    const long long lim = wl == 0 || wl > (unsigned long long)kTeamWaitCycles ? kTeamWaitCycles : (long long)wl;
    if (threadIdx.x == 0) {
        S.err = 0;
        for (int w = 0; w < kStreamWarps; ++w)
            for (int s = 0; s < 2; ++s) mbar_init(&S.bar[w][s]);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    stream_system<kSr>(sys[system], limit, S, smem + kStreamFixedSmem, sp, lim);
}

}  // namespace

const void *stream_kernel(bool single_reduction) {
    return single_reduction ? (const void *)k_stream<true> : (const void *)k_stream<false>;
}

}  // namespace wsb
