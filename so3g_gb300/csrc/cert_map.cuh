// cert_map.cuh -- the certified chunked from_map's copy of the map and its
// certified float32 accumulation (cert_gather.cu).
#pragma once

#include "host.h"
#include "pair32.cuh"

namespace so3g {

namespace {

// float4 words per pixel of the map copy: the pairs (h, l), for a tiled map
// followed by the tile's presence in the last word's .w.
template <int NC, bool TILED>
struct CxMap {
    static constexpr int W = TILED ? (NC == 1 ? 1 : 2) : (NC + 1) / 2;
};

// The copy, over the parent map's pixels when tiled: h = +-0 for m = +-0,
// NaN where m is not finite or outside df_split's range (such a sample goes
// to the float64 path).
template <int P, int NC>
__global__ void k_cx_map(DGeom g, const double *map, long long npix, float4 *out, SkipIf gate) {
    if (gate.holds()) return;
    constexpr bool TILED = P == PX_FLAT_T_NN || P == PX_HP_T;
    constexpr int W = CxMap<NC, TILED>::W;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npix) return;
    long long off = i, plane = npix;
    bool present = true;
    if constexpr (TILED) {
        int pix[3];
        if (P == PX_HP_T) {
            hp_tile_split(g.nppt, i, pix[0], pix[1]);
            pix[2] = 0;
        } else {
            const int gy = (int)(i / g.nx), gx = (int)(i - (long long)gy * g.nx);
            flat_tile_tuple(g, gy, gx, pix);
        }
        present = locate<P>(g, pix, &off, &plane) < 0;
    }
    float hl[4 * W];
#pragma unroll
    for (int k = 0; k < 4 * W; k++) hl[k] = 0.f;
    if (present) {
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const double m = __ldg(map + off + c * plane);
            const unsigned mh = (unsigned)__double2hiint(m);
            float h = __int_as_float(0x7fc00000), l = 0.f;
            if (((mh & 0x7fffffffu) | (unsigned)__double2loint(m)) == 0u) {
                h = __uint_as_float(mh & 0x80000000u);
            } else {
                dfl d;
                if (df_split(m, d)) {
                    h = d.hi;
                    l = d.lo;
                }
            }
            hl[2 * c] = h;
            hl[2 * c + 1] = l;
        }
    }
    if (TILED) hl[4 * W - 1] = present ? 1.f : 0.f;
#pragma unroll
    for (int w = 0; w < W; w++)
        out[i * W + w] = make_float4(hl[4 * w], hl[4 * w + 1], hl[4 * w + 2], hl[4 * w + 3]);
}

// sig + m * pf rounded to float32 as the reference's `*sig += map * pf`, m =
// h + l from the map copy; false when that rounding is not certain.  S + L
// is the double-float sum (S = fl(sig + h pf)), within e of the reference's
// float64 sum (as fast_accum).
__device__ __forceinline__ bool cx_accum(float &sig, float h, float l, float pf) {
    const float p = h * pf;
    const float pe = fmaf(l, pf, fmaf(h, pf, -p));
    float S, x;
    two_sum(sig, p, S, x);
    const float L = x + pe, e = 5e-13f * (fabsf(p) + fabsf(sig));
    float r = S + (L + e);
    bool ok = (r == S + (L - e)) & (fabsf(r) > 1e-30f);
    if (!ok && (h == 0.f || (pf == 0.f && h == h))) {
        // An exact zero with the product's sign (as fast_accum).
        r = sig + __int_as_float((__float_as_int(h) ^ __float_as_int(pf)) & 0x80000000);
        ok = true;
    }
    if (ok) sig = r;
    return ok;
}

// The same for one component of two samples, without the exact zeros: c0 and
// c1 become false where a rounding is not certain (or the sum is zero).
__device__ __forceinline__ void cx_accum2(float &s0, float &s1, float h0, float h1, float l0,
                                          float l1, float f0, float f1, bool &c0, bool &c1) {
    const float p0 = h0 * f0, p1 = h1 * f1;
    const f32x2 s = f2_make(s0, s1), p = f2_make(p0, p1);
    const f32x2 pe = f2_make(fmaf(l0, f0, fmaf(h0, f0, -p0)), fmaf(l1, f1, fmaf(h1, f1, -p1)));
    f32x2 S, x;
    f2_two_sum(s, p, S, x);
    const f32x2 L = f2_add(x, pe);
    const f32x2 e = f2_mul(f2_both(5e-13f),
                           f2_make(fabsf(p0) + fabsf(s0), fabsf(p1) + fabsf(s1)));
    float q0, q1;
    f2_get(f2_add(S, f2_add(L, e)), s0, s1);
    f2_get(f2_add(S, f2_sub(L, e)), q0, q1);
    c0 = c0 & (s0 == q0) & (fabsf(s0) > 1e-30f);
    c1 = c1 & (s1 == q1) & (fabsf(s1) > 1e-30f);
}

// All NC components of one sample, one after the other (a sample that
// cx_accum2 did not take); out: the sum.
template <int NC, int W>
__device__ __noinline__ bool cx_accum_slow(float sig, float4 m0, float4 m1, float f0, float f1,
                                           float f2, float *out) {
    const float hl[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w}, pf[3] = {f0, f1, f2};
    bool ok = true;
#pragma unroll
    for (int c = 0; c < NC; c++) ok = ok & cx_accum(sig, hl[2 * c], hl[2 * c + 1], pf[c]);
    *out = sig;
    return ok;
}
template <int NC, int W>
__device__ __forceinline__ bool cx_accum_all(float sig, const float (&hl)[4 * W],
                                             const float (&pf)[3], float &out) {
    const float4 m0 = make_float4(hl[0], hl[1], hl[2], hl[3]);
    const float4 m1 = W > 1 ? make_float4(hl[4 * W - 4], hl[4 * W - 3], hl[4 * W - 2], hl[4 * W - 1])
                            : make_float4(0.f, 0.f, 0.f, 0.f);
    float r;
    const bool ok = cx_accum_slow<NC, W>(sig, m0, m1, pf[0], pf[1], pf[2], &r);
    out = r;
    return ok;
}

}  // namespace

}  // namespace so3g
