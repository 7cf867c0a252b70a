// The update of one point and of four consecutive z, shared by the stencil
// kernels so that every path rounds alike.
#pragma once

#include "st_kernels.cuh"

namespace stg {
namespace {

__device__ __forceinline__ void f4_to(const float4& v, float a[4]) {
    a[0] = v.x;
    a[1] = v.y;
    a[2] = v.z;
    a[3] = v.w;
}

// The update of one point: out = 2u - upd + c * L u, upd = D * prev. Every operation is
// written out, so that no context or compiler setting contracts it otherwise than update2:
// points of one launch that two blocks form, and the launches of one step, two steps and
// all steps, agree bit for bit.
__device__ __forceinline__ float update_fast(float u, float upd, float xm, float xp, float ym, float yp, float zm,
                                             float zp, float c, float ax, float ay, float az) {
    const float lx = fmaf(-2.0f, u, __fadd_rn(xp, xm)), ly = fmaf(-2.0f, u, __fadd_rn(yp, ym)),
                lz = fmaf(-2.0f, u, __fadd_rn(zp, zm));
    const float lap = fmaf(lz, az, fmaf(lx, ax, __fmul_rn(ly, ay)));
    return fmaf(c, lap, fmaf(2.0f, u, -upd));
}

// The reference's guarded update (wave_equation.cpp:342-399), taken only when
// the fast result is non-finite or beyond the amplitude limit. A non-finite
// input always makes the fast result non-finite (c, 1/d^2 > 0), so the fast
// path is exact whenever it is taken. GINL: inlined at the call site (the
// two-step kernels measured faster so); otherwise one out-of-line copy
// shared by the call sites.
template <bool GINL = false>
__device__ __forceinline__ float update_guarded(float u, float upd, float xm, float xp, float ym, float yp, float zm,
                                                float zp, float c, float ax, float ay, float az, float amp,
                                                int* fired);
__device__ __forceinline__ float guarded_body(float u, float upd, float xm, float xp, float ym, float yp, float zm,
                                              float zp, float c, float ax, float ay, float az, float amp,
                                              int* fired) {
    if (!isfinite(u) || !isfinite(upd)) {
        *fired = 1;
        return 0.0f;
    }
    if (!isfinite(xm) || !isfinite(xp) || !isfinite(ym) || !isfinite(yp) || !isfinite(zm) || !isfinite(zp)) {
        *fired = 1;
        return u;
    }
    float nv = update_fast(u, upd, xm, xp, ym, yp, zm, zp, c, ax, ay, az);
    if (!isfinite(nv)) {
        nv = u;
        *fired = 1;
    }
    return fminf(fmaxf(nv, -amp), amp);
}
__device__ __noinline__ float guarded_call(float u, float upd, float xm, float xp, float ym, float yp, float zm,
                                           float zp, float c, float ax, float ay, float az, float amp, int* fired) {
    return guarded_body(u, upd, xm, xp, ym, yp, zm, zp, c, ax, ay, az, amp, fired);
}
template <bool GINL>
__device__ __forceinline__ float update_guarded(float u, float upd, float xm, float xp, float ym, float yp, float zm,
                                                float zp, float c, float ax, float ay, float az, float amp,
                                                int* fired) {
    if constexpr (GINL) return guarded_body(u, upd, xm, xp, ym, yp, zm, zp, c, ax, ay, az, amp, fired);
    else return guarded_call(u, upd, xm, xp, ym, yp, zm, zp, c, ax, ay, az, amp, fired);
}

__device__ __forceinline__ void ld4(const float* p, float v[4]) { f4_to(*reinterpret_cast<const float4*>(p), v); }
__device__ __forceinline__ void st4(float* p, const float v[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

// Two values per instruction, each rounded as the scalar form rounds it.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 pack(float x, float y) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void unpack(F2 a, float& x, float& y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// update_fast of two points; nD = -D.
__device__ __forceinline__ F2 update2(F2 u, F2 nD, F2 pv, F2 xs, F2 ys, F2 zs, F2 c, float ax, float ay, float az) {
    const F2 m2 = pack(-2.0f, -2.0f), p2 = pack(2.0f, 2.0f);
    const F2 lx = fma2(m2, u, xs), ly = fma2(m2, u, ys), lz = fma2(m2, u, zs);
    const F2 lap = fma2(lz, pack(az, az), fma2(lx, pack(ax, ax), mul2(ly, pack(ay, ay))));
    return fma2(c, lap, fma2(p2, u, mul2(nD, pv)));
}

// Four point updates in fd_step_kernel's order, first part: the update (the
// guarded form where the fast one is out of range), two points per instruction:
// the two-step kernels are bound by the latency of their instructions more than
// by memory (issue slots 50% busy, 39% of the DRAM rate at 192^3). With the sponge
// rule a compile-time choice: 150 x 203 x 171 RTM 6.60 -> 6.43 ms, 192^3 FWI 22.0 ->
// 21.7, 384 x 384 x 320 41.3 -> 40.4, 256^3 RTM 21.0 -> 20.9; the sponge rule alone gives
// about half. The caller then adds the adjoint receiver forcing, applies the
// stable damping (damp4) and, in the forward mode, samples the receivers and
// injects the source.
template <bool GINL>
__device__ __forceinline__ void update4(const StepArgs& a, const float u0[4], const float pv[4], const float um[4],
                                        const float up[4], const float ym[4], const float yp[4], float zm0, float zp3,
                                        const float cv[4], const float D[4], float res[4], int* fired) {
    bool bad = false;
    const float zs[4] = {u0[1] + zm0, u0[2] + u0[0], u0[3] + u0[1], zp3 + u0[2]};
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
        const F2 xs = add2(pack(up[j], up[j + 1]), pack(um[j], um[j + 1]));
        const F2 ys = add2(pack(yp[j], yp[j + 1]), pack(ym[j], ym[j + 1]));
        unpack(update2(pack(u0[j], u0[j + 1]), pack(-D[j], -D[j + 1]), pack(pv[j], pv[j + 1]), xs, ys,
                       pack(zs[j], zs[j + 1]), pack(cv[j], cv[j + 1]), a.ax, a.ay, a.az),
               res[j], res[j + 1]);
        bad = bad || !(fabsf(res[j]) <= a.amp) || !(fabsf(res[j + 1]) <= a.amp);
    }
    if (bad) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (fabsf(res[k]) <= a.amp) continue;
            const float zm = k == 0 ? zm0 : u0[k - 1];
            const float zp = k == 3 ? zp3 : u0[k + 1];
            res[k] = update_guarded<GINL>(u0[k], D[k] * pv[k], um[k], up[k], ym[k], yp[k], zm, zp, cv[k], a.ax, a.ay, a.az,
                                          a.amp, fired);
        }
    }
}

// The stable sponge mode damps the new values as well.
__device__ __forceinline__ void damp4(const float D[4], float res[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) res[k] *= D[k];
}

// Sponge factors of a 4-point group: D(min(dx, dyz)) for each point, formed
// as min(D(dx), D(dyz)) from the plane's x factor Dx and the y/z factors Dyz
// the thread looked up once (the table is non-decreasing in the distance and
// at most 1, so this is bit for bit the same).
__device__ __forceinline__ void sponge4f(float Dx, const float Dyz[4], float D[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) D[k] = fminf(Dx, Dyz[k]);
}

}  // namespace
}  // namespace stg
