// The reference's individual passes on the GPU with the reference's
// arithmetic (separately rounded FP32 multiply/add/divide, 256-wide shared
// memory tree for dot products). They back the executor entry points and the
// WSB_PREC_REFERENCE_F32 solve, whose iterates are bit-identical to the CPU
// restatement of compute.rs:189-495.
#include "kernels_ref.cuh"
#include "kernels_team.cuh"
#include "team_device.cuh"

namespace wsb {

// spmv.wgsl:43-64 - one row per thread, sequential sum in index order.
__global__ void k_ref_spmv(uint32_t n, const uint32_t *__restrict__ row_ptr, const uint32_t *__restrict__ col,
                           const float *__restrict__ val, const float *__restrict__ x, float *__restrict__ y) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float sum = 0.0f;
    for (uint32_t k = row_ptr[i]; k < row_ptr[i + 1]; ++k) sum = __fadd_rn(sum, __fmul_rn(val[k], __ldg(x + col[k])));
    y[i] = sum;
}

// 256-lane tree with offsets 128..1 (dot_partials.wgsl:57-69).
__device__ __forceinline__ float tree256(float *s) {
    const uint32_t t = threadIdx.x;
    for (uint32_t off = 128; off >= 1; off >>= 1) {
        if (t < off) s[t] = __fadd_rn(s[t], s[t + off]);
        __syncthreads();
    }
    return s[0];
}

// dot_partials.wgsl:37-75: partial[wg] = tree sum of a[i]*b[i] over 256 lanes.
__global__ void __launch_bounds__(256) k_ref_dot_partials(uint32_t n, const float *__restrict__ a,
                                                          const float *__restrict__ b, float *__restrict__ partial) {
    __shared__ float s[256];
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    s[threadIdx.x] = i < n ? __fmul_rn(a[i], b[i]) : 0.0f;
    __syncthreads();
    const float v = tree256(s);
    if (threadIdx.x == 0) partial[blockIdx.x] = v;
}

// dot_reduce.wgsl:36-74: output[wg] = tree sum of input[wg*256 .. +255].
__global__ void __launch_bounds__(256) k_ref_dot_reduce(uint32_t n, const float *__restrict__ in, float *__restrict__ out) {
    __shared__ float s[256];
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    s[threadIdx.x] = i < n ? in[i] : 0.0f;
    __syncthreads();
    const float v = tree256(s);
    if (threadIdx.x == 0) out[blockIdx.x] = v;
}

// copy_buffer_to_buffer of the final scalar (dot_scalar_exec.rs:239-246), or
// the n == 0 case that writes 0 (dot_scalar_exec.rs:165-174) when src is null.
__global__ void k_ref_store_scalar(const float *src, float *dst) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *dst = src ? *src : 0.0f;
}

// axpy.wgsl:32-42: y = y + alpha * x
__global__ void k_ref_axpy(uint32_t n, float alpha, const float *__restrict__ x, float *__restrict__ y) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __fadd_rn(y[i], __fmul_rn(alpha, x[i]));
}

// axpy_from_scalar_results.wgsl:28-42: y = y + s[k] * x
__global__ void k_ref_axpy_s(uint32_t n, const float *__restrict__ x, float *__restrict__ y,
                             const float *__restrict__ s, uint32_t k) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __fadd_rn(y[i], __fmul_rn(s[k], x[i]));
}

// scale_from_scalar_results.wgsl:26-38: x = x * s[k]
__global__ void k_ref_scale_s(uint32_t n, float *__restrict__ x, const float *__restrict__ s, uint32_t k) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = __fmul_rn(x[i], s[k]);
}

// block_jacobi.wgsl:63-127, one thread per block (the WGSL runs one
// single-invocation workgroup per block).
__global__ void k_ref_block_jacobi(uint32_t n, uint32_t nb, const float *__restrict__ lu,
                                   const uint32_t *__restrict__ bs, const float *__restrict__ r, float *__restrict__ z) {
    const uint32_t blk = blockIdx.x * blockDim.x + threadIdx.x;
    if (blk >= nb) return;
    const uint32_t offset = bs[blk], next = bs[blk + 1];
    if (offset >= n || next <= offset) return;
    const uint32_t m = min(6u, next - offset);
    const float *L = lu + (size_t)blk * 36u;
    float y[6] = {0, 0, 0, 0, 0, 0}, x[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        if ((uint32_t)i < m) {
            float sum = r[offset + i];
#pragma unroll
            for (int j = 0; j < i; ++j) sum = __fsub_rn(sum, __fmul_rn(L[i * 6 + j], y[j]));
            y[i] = sum;
        }
    }
#pragma unroll
    for (int i = 5; i >= 0; --i) {
        if ((uint32_t)i < m) {
            float sum = y[i];
#pragma unroll
            for (int j = i + 1; j < 6; ++j)
                if ((uint32_t)j < m) sum = __fsub_rn(sum, __fmul_rn(L[i * 6 + j], x[j]));
            x[i] = __fdiv_rn(sum, L[i * 6 + i]);
        }
    }
#pragma unroll
    for (int i = 0; i < 6; ++i)
        if ((uint32_t)i < m) z[offset + i] = x[i];
}

// pcg_update_scalars.wgsl:47-73 (one thread).
__global__ void k_ref_update_scalars(float *s, uint32_t p_ap, uint32_t rz_new, uint32_t rz_old, uint32_t alpha,
                                     uint32_t minus_alpha, uint32_t beta) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const float pap = s[p_ap], rzn = s[rz_new], rzo = s[rz_old];
    float a = 0.0f, b = 0.0f;
    if (pap != 0.0f) a = __fdiv_rn(rzo, pap);
    if (rzo != 0.0f) b = __fdiv_rn(rzn, rzo);
    s[alpha] = a;
    s[minus_alpha] = -a;
    s[beta] = b;
}

// After the ||b||^2 dot (compute.rs:228-257): store it, stop with Ok(0) when
// it is zero, otherwise open the iteration.
__global__ void k_ref_after_bnorm(RefState *st, const float *s) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    st->b_norm2 = s[0];
    st->rel2 = __fmul_rn(st->rel_tol, st->rel_tol);
    st->abs2 = __fmul_rn(st->abs_tol, st->abs_tol);
    st->iter = 0;
    st->breakdown = 0;
    if (st->b_norm2 == 0.0f) {
        st->status = ST_CONVERGED;
        st->active = 0;
    } else {
        st->status = ST_RUNNING;
        st->active = 1;
    }
}

// End of init (compute.rs:330): rz_old = scalar_results[3].
__global__ void k_ref_after_init(RefState *st, const float *s) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    st->rz_old = s[3];
    if (st->active && st->max_iter == 0) {
        st->status = ST_MAXITER;
        st->active = 0;
    }
}

// Step C (compute.rs:362-370): scalar_results[rz_old] = host rz_old.
__global__ void k_ref_write_rz_old(const RefState *st, float *s) {
    if (threadIdx.x == 0 && blockIdx.x == 0) s[3] = st->rz_old;
}

// The host side of one iteration (compute.rs:466-488) done on the device:
// breakdown checks, stop test in f32, rz_old = rz_new; clears the graph's
// while condition when the solve ends.
__global__ void k_ref_check(RefState *st, const float *s, double *history, uint64_t hist_cap,
                            cudaGraphConditionalHandle h) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const float p_ap = s[0], r_norm2 = s[1], rz_new = s[2];
    const uint32_t k = st->iter;
    if (history && k < hist_cap) history[k] = (double)r_norm2;
    st->iter = k + 1;
    st->last_rr = r_norm2;
    uint32_t status = ST_RUNNING;
    if (p_ap == 0.0f) {
        status = ST_BREAKDOWN;
        st->breakdown = 1;
    } else if (st->rz_old == 0.0f) {
        status = ST_BREAKDOWN;
        st->breakdown = 2;
    } else if (r_norm2 <= st->abs2 || r_norm2 <= __fmul_rn(st->rel2, st->b_norm2)) {
        status = ST_CONVERGED;
    } else if (k + 1 >= st->max_iter) {
        status = ST_MAXITER;
    } else {
        st->rz_old = rz_new;
    }
    if (status != ST_RUNNING) {
        st->status = status;
        st->active = 0;
    }
    if (h != 0 && (status != ST_RUNNING)) cudaGraphSetConditional(h, 0);
}

__global__ void k_ref_gate(const RefState *st, cudaGraphConditionalHandle h) {
    if (threadIdx.x == 0 && blockIdx.x == 0) cudaGraphSetConditional(h, st->active ? 1u : 0u);
}

}  // namespace wsb

namespace wsb {

size_t ref_dot_scratch_floats(uint64_t n) {
    const uint64_t l1 = (n + 255) / 256, l2 = (l1 + 255) / 256;
    return (size_t)(l1 + l2 + 2);
}

// The pass structure of encode_dot_scalar_into (dot_scalar_exec.rs:151-247):
// one dot_partials pass, then dot_reduce passes (ping-pong between the two
// halves of scratch) until one value is left, then a copy into s_out.
cudaError_t ref_dot(cudaStream_t st, uint32_t n, const float *a, const float *b, float *scratch, float *s_out) {
    if (n == 0) {
        k_ref_store_scalar<<<1, 32, 0, st>>>(nullptr, s_out);
        return cudaGetLastError();
    }
    const uint32_t l1 = (n + 255) / 256;
    float *in = scratch, *out = scratch + l1 + 1;
    k_ref_dot_partials<<<l1, 256, 0, st>>>(n, a, b, in);
    uint32_t len = l1;
    while (len > 1) {
        const uint32_t ol = (len + 255) / 256;
        k_ref_dot_reduce<<<ol, 256, 0, st>>>(len, in, out);
        len = ol;
        float *t = in;
        in = out;
        out = t;
    }
    k_ref_store_scalar<<<1, 32, 0, st>>>(in, s_out);
    return cudaGetLastError();
}


// ---------------------------------------------------------------------------
// k_ref_pcg: the passes above, one solve in one launch.
//
// What bounds the passes one by one is the number of launches, 19 an iteration
// of 27 us at any size below 20^3 nodes. Here a CTA of 256 rows (a workgroup of
// the dot products, so their trees stay the reference's) stays resident: its
// matrix rows are in shared memory, the factors of its blocks, x, r and p in
// registers. An iteration has two exchanges, as in k_team and k_stream:
// partials as {value, tag} packets that every CTA reads and adds by the
// reference's tree; z and p at other rows through global memory, ordered by the
// second exchange. The columns of a CTA's rows are listed once (a hash table in
// shared memory; a CTA with more than kRefCols of them reads z and p for each
// nonzero instead), so p = beta p + z is formed once for each.
// Blocks cross the CTAs' rows: a CTA also keeps r of up to five rows on either
// side and solves every block of its rows.
// Measured (B200, us an iteration, passes -> here): 4^3 nodes 27.4 -> 4.0, 9^3
// 31.1 -> 5.5, 12^3 30.8 -> 6.2, 16^3 33.6 -> 6.0; with two CTAs an SM 19^3 34.0
// -> 7.6, 23^3 40.1 -> 10.7. What is left is latency: two exchanges, the fence,
// the gather of p and z, one row sum, one block solve.
namespace {

struct RefShared {
    float v[2];     // results of an exchange
    uint32_t cols;  // columns listed
    uint32_t first_blk, n_blk;
    uint32_t err;
};

// Lane 0: tree sum (offsets 128..1) of the 256 values get(0..255), by one warp.
template <class F>
__device__ __forceinline__ float tree256_warp(F get) {
    const uint32_t t = threadIdx.x & 31u;
    float s[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) s[k] = get(t + 32u * k);
#pragma unroll
    for (int k = 0; k < 4; ++k) s[k] = __fadd_rn(s[k], s[k + 4]);
    s[0] = __fadd_rn(s[0], s[2]);
    s[1] = __fadd_rn(s[1], s[3]);
    float v = __fadd_rn(s[0], s[1]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_down_sync(kFull, v, o));
    return v;
}

// The dot product whose products of this workgroup are in `prod`, by one warp,
// valid in lane 0: the workgroups' trees, then trees over their results.
// `release`: the CTA's writes come before the partial.
__device__ __forceinline__ float ref_all_sum(const float *prod, unsigned long long *parts, uint32_t tag, bool release,
                                             RefShared &S, RefState *st, long long lim) {
    const uint32_t lane = threadIdx.x & 31u, wgs = gridDim.x, copies = team_copies(wgs);
    float v = tree256_warp([&](uint32_t i) { return prod[i]; });
    if (wgs == 1) return v;
    if (release) __threadfence();
    v = __shfl_sync(kFull, v, 0);
    if (lane < copies) st_packet(parts + (size_t)lane * 3u * wgs + blockIdx.x, v, tag);
    __syncwarp();
    parts += (size_t)(blockIdx.x % copies) * 3u * wgs;
    team_quiet(quiet_cycles(wgs));
    const long long t0 = clock64();
    uint32_t len = wgs;
    float mine = 0.0f;  // lane g: the tree over partials [256 g, 256 g + 256)
    for (uint32_t g = 0; 256u * g < wgs; ++g) {
        unsigned long long q[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) q[j] = 256u * g + lane + 32u * j < wgs ? 0ull : (unsigned long long)tag << 32;
#pragma unroll 1
        for (uint32_t k = 1;; ++k) {
            bool ok = true;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const bool want = (uint32_t)(q[j] >> 32) != tag;
                q[j] = ld_packet_if(parts + (want ? 256u * g + lane + 32u * j : 0u), want, q[j]);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) ok = ok && (uint32_t)(q[j] >> 32) == tag;
            if (__all_sync(kFull, ok)) break;
            if (__any_sync(kFull, clock64() - t0 > lim) || ((k & 255u) == 0 && __any_sync(kFull, ld_error(st) != 0))) {
                S.err = 1;
                atomicExch(&st->error, 1u);
                return 0.0f;
            }
        }
        float s[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] = __uint_as_float((uint32_t)q[j]);
#pragma unroll
        for (int k = 0; k < 4; ++k) s[k] = __fadd_rn(s[k], s[k + 4]);
        s[0] = __fadd_rn(s[0], s[2]);
        s[1] = __fadd_rn(s[1], s[3]);
        float w = __fadd_rn(s[0], s[1]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w = __fadd_rn(w, __shfl_down_sync(kFull, w, o));
        w = __shfl_sync(kFull, w, 0);
        if (lane == g) mine = w;
        len = g + 1u;
    }
    if (release) __threadfence();  // what the publishers wrote is visible after this
    if (len == 1) return mine;
    // (At most 32 values: the 256-wide tree adds zeros to them first.)
    v = __fadd_rn(__fadd_rn(__fadd_rn(mine, 0.0f), 0.0f), 0.0f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_down_sync(kFull, v, o));
    return v;
}

__global__ void __launch_bounds__(kRefThreads, 2) k_ref_pcg(const RefPcg D) {
    extern __shared__ __align__(16) char smem[];
    RefShared &S = *reinterpret_cast<RefShared *>(smem);
    float *const rw = reinterpret_cast<float *>(smem + 1024);  // r, then z, of the window's rows
    float *const zw = rw + kRefWin;
    float *const prod = zw + kRefWin;  // products of a dot, twice 256
    float *const px = prod + 512;      // p at the listed columns
    uint32_t *const list = reinterpret_cast<uint32_t *>(px + kRefCols);
    uint32_t *const table = list + kRefCols;
    uint16_t *const place = reinterpret_cast<uint16_t *>(table + kRefHash);
    const uint32_t width = (D.width + 1u) & ~1u;
    float *const val = reinterpret_cast<float *>(place + kRefHash);
    uint16_t *const idx = reinterpret_cast<uint16_t *>(val + (size_t)kRefThreads * width);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, row0 = 256u * blockIdx.x;
    const uint32_t row1 = min(row0 + 256u, D.n), win0 = row0 >= 5u ? row0 - 5u : 0u, win1 = min(row1 + 5u, D.n);
    // The thread's row: its own, or one beside the CTA's.
    uint32_t row = row0 + tid;
    bool own = tid < 256u && row < D.n, on = own;
    if (tid >= 256u) {
        const uint32_t k = tid - 256u;
        row = k < 5u ? row0 - 5u + k : row1 + k - 5u;
        on = k < 5u ? row0 >= 5u - k : k < 10u && row < win1;
    }
    const uint32_t k0 = on ? D.row_ptr[row] : 0u, nk = on ? D.row_ptr[row + 1u] - k0 : 0u;
    const uint32_t wr = on ? row - win0 : kRefWin - 1u;  // place in the window (the last: nobody's)
    if (tid == 0) {
        S.cols = S.err = 0;
        // Blocks with a solved row among the CTA's: those that start in
        // (row0 - 6, row1) and reach row0.
        auto at_least = [&](uint32_t r) {
            uint32_t lo = 0, hi = D.nb;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) / 2u;
                if (D.bs[mid] >= r) hi = mid;
                else lo = mid + 1u;
            }
            return lo;
        };
        S.first_blk = at_least(win0);
        S.n_blk = at_least(row1) - S.first_blk;
    }
    for (uint32_t i = tid; i < kRefHash; i += kRefThreads) table[i] = 0xffffffffu;
    for (uint32_t i = tid; i < kRefWin; i += kRefThreads) rw[i] = zw[i] = 0.0f;
    for (uint32_t i = tid; i < 512u; i += kRefThreads) prod[i] = 0.0f;
    __syncthreads();
    // The columns, each once; the numbers come in any order and choose places.
    const volatile uint32_t *const listed = &S.cols;
    for (uint32_t j = 0; j < nk; ++j) {
        const uint32_t c = D.col[k0 + j];
        uint32_t h = (c * 2654435761u) % kRefHash;
        while (*listed <= kRefCols) {
            const uint32_t old = atomicCAS(&table[h], 0xffffffffu, c);
            if (old == c) break;
            if (old == 0xffffffffu) {
                const uint32_t e = atomicAdd(&S.cols, 1u);
                place[h] = (uint16_t)e;
                if (e < kRefCols) list[e] = c;
                break;
            }
            h = (h + 1u) % kRefHash;
        }
    }
    __syncthreads();
    const uint32_t n_cols = S.cols;
    const bool direct = n_cols > kRefCols;
    for (uint32_t j = 0; j < nk; ++j) {
        val[kRefThreads * j + tid] = D.val[k0 + j];
        uint32_t h = 0;
        if (!direct) {
            const uint32_t c = D.col[k0 + j];
            h = (c * 2654435761u) % kRefHash;
            while (table[h] != c) h = (h + 1u) % kRefHash;
            h = place[h];
        }
        idx[kRefThreads * j + tid] = (uint16_t)h;
    }
    // A block a thread, spread over the warps; its factors in registers.
    const uint32_t bq = lane * (kRefThreads / 32u) + warp;
    const bool solver = bq < S.n_blk;
    uint32_t boff = 0, m = 0;
    float L[36];
    if (solver) {
        const uint32_t k = S.first_blk + bq, off = D.bs[k];
        boff = off - win0;
        m = min(6u, D.bs[k + 1u] - off);
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const float4 f = reinterpret_cast<const float4 *>(D.lu + 36u * (size_t)k)[q];
            L[4 * q] = f.x, L[4 * q + 1] = f.y, L[4 * q + 2] = f.z, L[4 * q + 3] = f.w;
        }
    }
    // block_jacobi.wgsl:63-127 on the window.
    auto block_solve = [&]() {
        if (solver) {
            float y[6], xs[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                y[i] = xs[i] = 0.0f;
                if ((uint32_t)i < m) {
                    float sum = rw[boff + i];
#pragma unroll
                    for (int j = 0; j < i; ++j) sum = __fsub_rn(sum, __fmul_rn(L[i * 6 + j], y[j]));
                    y[i] = sum;
                }
            }
#pragma unroll
            for (int i = 5; i >= 0; --i)
                if ((uint32_t)i < m) {
                    float sum = y[i];
#pragma unroll
                    for (int j = i + 1; j < 6; ++j)
                        if ((uint32_t)j < m) sum = __fsub_rn(sum, __fmul_rn(L[i * 6 + j], xs[j]));
                    xs[i] = __fdiv_rn(sum, L[i * 6 + i]);
                    zw[boff + i] = xs[i];
                }
        }
    };
    // spmv.wgsl:43-64 with p (x0 at first) at the listed columns.
    auto row_sum = [&](bool start, bool first, float beta, const float *p_old) {
        float sum = 0.0f;
        if (!direct) {
#pragma unroll 4
            for (uint32_t j = 0; j < nk; ++j)
                sum = __fadd_rn(sum, __fmul_rn(val[kRefThreads * j + tid], px[idx[kRefThreads * j + tid]]));
        } else {
#pragma unroll 4
            for (uint32_t j = 0; j < nk; ++j) {
                const uint32_t c = D.col[k0 + j];
                const float v = start ? D.x[c] : first ? D.z[c] : __fadd_rn(__fmul_rn(p_old[c], beta), D.z[c]);
                sum = __fadd_rn(sum, __fmul_rn(val[kRefThreads * j + tid], v));
            }
        }
        return sum;
    };
    const uint32_t wgs = gridDim.x;
    unsigned long long *const part0 = D.parts, *const part1 = part0 + wgs, *const part2 = part1 + wgs;
    const float rel2 = __fmul_rn(D.st->rel_tol, D.st->rel_tol), abs2 = __fmul_rn(D.st->abs_tol, D.st->abs_tol);
    const uint32_t max_iter = D.st->max_iter;
    uint32_t tag = 1, iter = 0, status = ST_RUNNING, breakdown = 0;
    // ||b||^2, r = b - A x0, z = M r, r.z (compute.rs:228-331).
    if (!direct)
        for (uint32_t i = tid; i < n_cols; i += kRefThreads) px[i] = D.x[list[i]];
    __syncthreads();
    float x = own ? D.x[row] : 0.0f, p = 0.0f, r = 0.0f, last_rr = 0.0f;
    {
        const float b = on ? D.b[row] : 0.0f;
        r = __fadd_rn(b, __fmul_rn(-1.0f, row_sum(true, false, 0.0f, nullptr)));
        if (on) rw[wr] = r;
        if (tid < 256u) prod[tid] = own ? __fmul_rn(b, b) : 0.0f;
    }
    __syncthreads();
    block_solve();
    __syncthreads();
    if (own) {
        D.z[row] = zw[wr];
        prod[256u + tid] = __fmul_rn(r, zw[wr]);
    }
    __syncthreads();
    if (warp < 2) {
        const float v = ref_all_sum(prod + 256u * warp, warp ? part2 : part1, tag, true, S, D.st, D.wait_cycles);
        if (lane == 0) S.v[warp] = v;
    }
    __syncthreads();
    const float bnorm2 = S.v[0];
    float rz_old = S.v[1], beta = 0.0f;
    if (bnorm2 == 0.0f) status = ST_CONVERGED;
    else if (max_iter == 0) status = ST_MAXITER;
    if (S.err) return;
    while (status == ST_RUNNING) {
        ++tag;
        const bool first = iter == 0;
        const float *const p_old = iter & 1u ? D.p1 : D.p0;
        float *const p_new = iter & 1u ? D.p0 : D.p1;
        // p = beta p + z (J of the iteration before), then A p and p.Ap.
        if (!direct)
            for (uint32_t i = tid; i < n_cols; i += kRefThreads) {
                const uint32_t c = list[i];
                px[i] = first ? D.z[c] : __fadd_rn(__fmul_rn(p_old[c], beta), D.z[c]);
            }
        if (own) {
            p = first ? zw[wr] : __fadd_rn(__fmul_rn(p, beta), zw[wr]);
            p_new[row] = p;
        }
        __syncthreads();
        const float ap = row_sum(false, first, beta, p_old);
        if (own) prod[tid] = __fmul_rn(p, ap);
        __syncthreads();
        if (warp == 0) {
            const float v = ref_all_sum(prod, part0, tag, false, S, D.st, D.wait_cycles);
            if (lane == 0) S.v[0] = v;
        }
        __syncthreads();
        if (S.err) return;
        const float pap = S.v[0], alpha = pap != 0.0f ? __fdiv_rn(rz_old, pap) : 0.0f, minus = -alpha;
        x = __fadd_rn(x, __fmul_rn(alpha, p));
        r = __fadd_rn(r, __fmul_rn(minus, ap));
        if (on) rw[wr] = r;
        __syncthreads();
        block_solve();
        __syncthreads();
        if (own) {
            const float z = zw[wr];
            D.z[row] = z;
            prod[tid] = __fmul_rn(r, r);
            prod[256u + tid] = __fmul_rn(r, z);
        }
        __syncthreads();
        if (warp < 2) {
            const float v = ref_all_sum(prod + 256u * warp, warp ? part2 : part1, tag, true, S, D.st, D.wait_cycles);
            if (lane == 0) S.v[warp] = v;
        }
        __syncthreads();
        if (S.err) return;
        const float rr = S.v[0], rz_new = S.v[1];
        // compute.rs:466-488
        if (D.history && blockIdx.x == 0 && tid == 0 && iter < D.hist_cap) D.history[iter] = (double)rr;
        last_rr = rr;
        if (pap == 0.0f) {
            status = ST_BREAKDOWN;
            breakdown = 1;
        } else if (rz_old == 0.0f) {
            status = ST_BREAKDOWN;
            breakdown = 2;
        } else if (rr <= abs2 || rr <= __fmul_rn(rel2, bnorm2)) {
            status = ST_CONVERGED;
        } else if (iter + 1u >= max_iter) {
            status = ST_MAXITER;
        }
        ++iter;
        beta = rz_old != 0.0f ? __fdiv_rn(rz_new, rz_old) : 0.0f;
        rz_old = rz_new;
    }
    if (own) D.x[row] = x;
    if (blockIdx.x == 0 && tid == 0) {
        D.st->b_norm2 = bnorm2;
        D.st->last_rr = last_rr;
        D.st->iter = iter;
        D.st->status = status;
        D.st->breakdown = breakdown;
        D.st->active = 0;
    }
}

}  // namespace

const void *ref_pcg_kernel() { return (const void *)k_ref_pcg; }

}  // namespace wsb
