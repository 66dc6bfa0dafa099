// Device helpers shared by the kernels that walk a tile's list: asynchronous
// staging copies, the cull tests of a warp's 8x4 pixel block, packed pairs of
// entries and warp sums.
#pragma once
#include <cstdint>
#include <cmath>
#include "sf_math.cuh"

namespace sft {

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The cull's second test, for an entry whose power_max box reaches the warp's
// 8x4 block: whether the splat's quadratic form q(dx, dy) = hx dx^2 +
// cy dx dy + hz dy^2 stays above power_max at every pixel of the block. The
// pixel offsets (splat centre minus pixel centre) lie in [X0 - 7, X0] x
// [Y0 - 3, Y0], widened by 1e-3 for the rounding of X0 and Y0. The form is
// convex, so its minimum over that rectangle is 0 with the centre inside it,
// else the least of its minima along the four edges (each a 1-D quadratic,
// minimised at a clamped point; an approximate minimiser only raises q by
// the square of its error). The entry is skipped only when that minimum
// exceeds power_max by 1e-5 of the largest sum of |terms| over the block
// plus 1e-5: both this minimum and the per-pixel power are a few roundings
// of such terms (error below 1e-6 of their sum), so every pixel's computed
// power is then above power_max and the pixel would skip the pair itself.
// A form that is not positive definite has no box (ext infinite) and is
// never skipped.
__device__ __forceinline__ bool block_misses(const float4 g0, const float4 g1, const float2 e, float wxf,
                                             float wyf) {
    if (!(e.x < INFINITY)) return false;
    const float hx = g0.z, cy = g0.w, hz = g1.x, pmax = g1.z;
    const float x0 = g0.x - wxf, y0 = g0.y - wyf;
    const float xlo = x0 - 7.001f, xhi = x0 + 0.001f, ylo = y0 - 3.001f, yhi = y0 + 0.001f;
    if (xlo <= 0.0f && xhi >= 0.0f && ylo <= 0.0f && yhi >= 0.0f) return false;
    const float ky = __fdividef(-0.5f * cy, hz), kx = __fdividef(-0.5f * cy, hx);
    auto q = [&](float x, float y) { return fmaf(hx * x, x, fmaf(hz * y, y, (cy * x) * y)); };
    const float y1 = fminf(fmaxf(ky * xlo, ylo), yhi), y2 = fminf(fmaxf(ky * xhi, ylo), yhi);
    const float x1 = fminf(fmaxf(kx * ylo, xlo), xhi), x2 = fminf(fmaxf(kx * yhi, xlo), xhi);
    const float qmin = fminf(fminf(q(xlo, y1), q(xhi, y2)), fminf(q(x1, ylo), q(x2, yhi)));
    const float dx = fmaxf(fabsf(xlo), fabsf(xhi)), dy = fmaxf(fabsf(ylo), fabsf(yhi));
    const float smax = fmaf(hx * dx, dx, fmaf(hz * dy, dy, (fabsf(cy) * dx) * dy));
    return qmin > fmaf(1e-5f, smax, pmax + 1e-5f);
}

// Whether an entry (records g0 / g1, power_max box half extents e) may reach
// the 8x4 block whose first pixel centre is (wxf, wyf): the box test, then the
// exact one. A NaN anywhere (a splat of infinite extent) counts as a hit.
__device__ __forceinline__ bool block_hit(const float4 g0, const float4 g1, const float2 e, float wxf, float wyf) {
    const float lx = (g0.x - e.x) - wxf, hx = (g0.x + e.x) - wxf;
    const float ly = (g0.y - e.y) - wyf, hy = (g0.y + e.y) - wyf;
    if (lx > 7.0f || hx < 0.0f || ly > 3.0f || hy < 0.0f) return false;
    return !block_misses(g0, g1, e, wxf, wyf);
}

// Two consecutive list entries a and b of a warp's walk, each field of both
// side by side, so that one 16-byte load fills the operands of two packed f32
// operations: centres, negated form coefficients and power_max, opacity, the
// entries' places in the staged chunk and (RGB) colours. The stride (80 or 112
// bytes) starts the 16 records of a warp in eight different banks.
template <bool COLOR>
struct __align__(16) PairRec {
    float x[2], y[2], nhx[2], ncy[2], nhz[2], op[2], npm[2];
    uint32_t j[2];
    float r[COLOR ? 2 : 1], g[COLOR ? 2 : 1], b[COLOR ? 2 : 1];
    uint32_t pad[COLOR ? 6 : 1];
};
static_assert(sizeof(PairRec<true>) == 112 && sizeof(PairRec<false>) == 80, "record stride");

// Packed f32 pairs (sm_100a): each half rounds as the scalar operation does.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 both(float v) { return pack2(v, v); }

// exp_neg_ (sf_math.cuh) of two values, operation by operation.
__device__ __forceinline__ void exp_neg2(f32x2 x, float& ea, float& eb) {
    const f32x2 kr = add2(mul2(x, both(1.44269502f)), both(12582912.0f));
    const f32x2 kf = add2(kr, both(-12582912.0f));
    f32x2 r = fma2(kf, both(-0.693145751953125f), x);
    r = fma2(kf, both(-1.42860677e-06f), r);
    f32x2 p = both(1.98412701e-04f);
    p = fma2(p, r, both(1.38888892e-03f));
    p = fma2(p, r, both(8.33333377e-03f));
    p = fma2(p, r, both(4.16666679e-02f));
    p = fma2(p, r, both(1.66666672e-01f));
    p = fma2(p, r, both(0.5f));
    p = fma2(p, r, both(1.0f));
    p = fma2(p, r, both(1.0f));
    float pa, pb, ka, kb;
    unpack2(p, pa, pb);
    unpack2(kr, ka, kb);
    ea = sfm::u2f(sfm::f2u(pa) + (sfm::f2u(ka) << 23));
    eb = sfm::u2f(sfm::f2u(pb) + (sfm::f2u(kb) << 23));
}

// Sums N = 2^k values over the warp's lanes at once, halving the values held
// per lane at each of the first k steps (N - 1 + 5 - k shuffles instead of
// 5 N): on return v[0] of lane l is the warp's total of value l >> (5 - k).
template <uint32_t N>
__device__ __forceinline__ void warp_sum_scatter(float (&v)[N]) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t d = 16;
#pragma unroll
    for (uint32_t m = N / 2; m >= 1; m /= 2, d /= 2) {
        const bool up = lane & d;
#pragma unroll
        for (uint32_t i = 0; i < m; ++i) {
            const float send = up ? v[i] : v[i + m];
            const float keep = up ? v[i + m] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, d);
        }
    }
#pragma unroll
    for (uint32_t dd = 16 / N; dd >= 1; dd /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], dd);
}

}  // namespace sft
