// Device code shared by the persistent kernels (kernels_team.cu,
// kernels_stream.cu): published partials and packets, the all-reduce over a
// team's CTAs, and divisions shorter than the general ones.
#pragma once
#include "wsb_internal.h"

namespace wsb {
namespace {

constexpr uint32_t kFull = 0xffffffffu;

__device__ __forceinline__ void st_entry(RedEntry *e, double v, uint32_t tag) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(e),
                 "l"(__double_as_longlong(v)), "l"((long long)tag)
                 : "memory");
}
// Loads the entry where `miss`, which is cleared when it has arrived.
__device__ __forceinline__ void ld_entry_if(const RedEntry *e, bool &miss, uint32_t tag, double *v) {
    long long lo = __double_as_longlong(*v), hi = tag;
    asm volatile(
        "{\n\t.reg .pred q;\n\t.reg .b128 t;\n\tsetp.ne.u32 q, %3, 0;\n\tmov.b128 t, {%0, %1};\n\t"
        "@q ld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
        : "+l"(lo), "+l"(hi)
        : "l"(e), "r"((uint32_t)miss)
        : "memory");
    *v = __longlong_as_double(lo);
    miss = miss && (uint32_t)hi != tag;
}
__device__ __forceinline__ void st_packet(unsigned long long *p, float v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p),
                 "l"((unsigned long long)__float_as_uint(v) | ((unsigned long long)tag << 32))
                 : "memory");
}
// The packet, or `other` when !want.
__device__ __forceinline__ unsigned long long ld_packet_if(const unsigned long long *p, bool want,
                                                           unsigned long long other) {
    unsigned long long v = other;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.relaxed.gpu.global.u64 %0, [%1];\n\t}"
                 : "+l"(v)
                 : "l"(p), "r"((uint32_t)want)
                 : "memory");
    return v;
}
// The error word of a launch (StepParams, RefState).
template <class T>
__device__ __forceinline__ uint32_t ld_error(const T *sp) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&sp->error) : "memory");
    return v;
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Two FP32 products in one packed instruction, each rounded to nearest.
__device__ __forceinline__ float2 mul2_rn(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 ra, rb, rc;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "mul.rn.f32x2 rc, ra, rb;\n\tmov.b64 {%0, %1}, rc;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
    return v;
}

constexpr int kPollBatch = 5;
// A partial takes about 700 cycles to the L2 and on to a reader, so polls
// before that only hold up the stores. Where the CTAs of a team publish at
// nearly the same time (k_team, k_ref_pcg) and are many, the first poll waits
// (B200, us an iteration without, with 350, 650 and 1000 cycles: 63 parts 4.7,
// 4.8, 5.1, 5.5; 77 parts 5.3, 4.6, 4.9, 5.2; 124 parts 6.3, 5.9, 5.4, 5.5; 26^3
// nodes, 136 CTAs, 8.3, 7.7, 6.9, 6.9; in k_stream, 32^3, 13.0, 13.3, 13.5, 14.0).
__device__ __forceinline__ int quiet_cycles(uint32_t size) { return size <= 64u ? 0 : size <= 80u ? 350 : 700; }
__device__ __forceinline__ void team_quiet(int cycles) {
    if (cycles == 0) return;
    const long long t0 = clock64();
    while (clock64() - t0 < cycles) {}
    __syncwarp();
}
// Sum over the team of the partials in red[0 .. size), by one warp: lane l adds
// entries l, l + 32, ... in order, then the lanes; valid in lane 0. Each round
// keeps up to kPollBatch loads a lane in flight, for the entries that have not
// come (with all of them loaded again the polls hold up the stores they wait
// for: k_stream, 148 CTAs, 15.0 us an iteration on 32^3 nodes against 13.5;
// k_team, 124 CTAs, 6.7 against 6.2), the first after `quiet` cycles. *err is
// set when the wait runs out.
__device__ __noinline__ double team_gather(uint32_t *err, const RedEntry *red, uint32_t size, uint32_t tag, StepParams *sp,
                                           long long lim, int quiet) {
    const uint32_t lane = threadIdx.x & 31u;
    double sum = 0.0;
    const long long t0 = clock64();
    team_quiet(quiet);
#pragma unroll 1
    for (uint32_t b = 0; b < size; b += 32u * kPollBatch) {
        double v[kPollBatch] = {};
        bool miss[kPollBatch];
#pragma unroll
        for (int j = 0; j < kPollBatch; ++j) miss[j] = b + 32u * j + lane < size;
#pragma unroll 1
        for (uint32_t k = 1;; ++k) {
            bool any = false;
#pragma unroll
            for (int j = 0; j < kPollBatch; ++j) ld_entry_if(red + min(b + 32u * j + lane, size - 1u), miss[j], tag, &v[j]);
#pragma unroll
            for (int j = 0; j < kPollBatch; ++j) any = any || miss[j];
            if (!__any_sync(kFull, any)) break;
            if (__any_sync(kFull, clock64() - t0 > lim) || ((k & 255u) == 0 && __any_sync(kFull, ld_error(sp) != 0))) {
                *err = 1;
                return 0.0;
            }
        }
#pragma unroll
        for (int j = 0; j < kPollBatch; ++j)
            if (b + 32u * j + lane < size) sum += v[j];
    }
    return warp_sum(sum);
}

// a / b, or 0 when b is 0: an FP32 approximate reciprocal of b, two Newton steps, then
// the product corrected once by its residual (Markstein, IBM J. Res. Dev. 34,
// 1990); about 130 cycles against 420 for the division, which operands outside
// [2^-100, 2^100] take.
__device__ __noinline__ double quotient(double a, double b) {
    if (b == 0.0) return 0.0;
    const double aa = fabs(a), ab = fabs(b);
    if (!(aa >= 7.888609052210118e-31 && aa <= 1.2676506002282294e30 && ab >= 7.888609052210118e-31 &&
          ab <= 1.2676506002282294e30))
        return a / b;
    float seed;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(seed) : "f"((float)b));
    double y = (double)seed;
    y = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
    y = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

// v / u correctly rounded, y = RN(1 / u) formed beforehand: q = v y, then
// twice q += (v - u q) y in fused operations. By Markstein's theorem the last
// step rounds correctly when q is within one ulp and nothing under- or
// overflows, which lo <= |v| <= 2^60 ensures (lo = 2^-60 for |u| in
// [2^-40, 2^40], else infinity); a zero v keeps the product's sign. *ok is
// cleared for other operands, whose quotient is the division's.
constexpr float kDivLo = 8.673617e-19f, kDivHi = 1.1529215e18f;      // 2^-60, 2^60
constexpr float kDivULo = 9.094947e-13f, kDivUHi = 1.0995116e12f;  // 2^-40, 2^40
__device__ __forceinline__ float div_by(float v, float u, float y, float lo, bool *ok) {
    const float av = fabsf(v), q0 = __fmul_rn(v, y);
    float q = __fmaf_rn(__fmaf_rn(-u, q0, v), y, q0);
    q = __fmaf_rn(__fmaf_rn(-u, q, v), y, q);
    *ok = *ok && ((av >= lo && av <= kDivHi) || (av == 0.0f && lo <= kDivHi));
    return av == 0.0f ? q0 : q;
}
// Backward substitution of m rows with plain divisions.
__device__ __noinline__ void back_general(const float *lu, const float *y, float *x, int m) {
#pragma unroll 1
    for (int i = m - 1; i >= 0; --i) {
        float v = y[i];
#pragma unroll 1
        for (int q = i + 1; q < m; ++q) v = __fsub_rn(v, __fmul_rn(lu[6 * i + q], x[q]));
        x[i] = __fdiv_rn(v, lu[7 * i]);
    }
}

}  // namespace
}  // namespace wsb
