// gather_kernel.cuh -- from_map pieces shared by gather.cu and
// cert_gather.cu: the kernel arguments and the certified and exact
// per-sample paths.
#pragma once

#include "host.h"

namespace so3g {

struct GatherArgs {
    DGeom g;
    const double *bore;
    const double *dets;
    const float *resp;
    const double *map;
    float *signal;
    long long sig_stride;
    Segs segs;
    int piece;
    int *err;
    int fast;           // SO3G_POINTING_*: 0 exact, 1 certified, 2 mixed
    FastTables ft;
    FastConst fc;
    MixedConst mc;
    const float4 *bore32;   // float32 boresight (mixed pointing), or NULL
    const float4 *map32;    // float32 (T, Q, U, 0) per pixel (mixed pointing), or NULL
    SkipIf gate;            // the kernel's gate beside a chunked one, or none
};

// The chunked certified from_map (cert_gather.cu) of n_det whole detectors;
// 1 (nothing launched) where it does not apply, else the protocol of
// cert_to_map (scatter_kernel.cuh).
int cert_from_map(int coord, int kind, GatherArgs &args, int n_det, cudaStream_t st,
                  void **work);
// The chunked from_map with untiled bilinear TAN, ZEA and SIN maps in the mixed
// mode (bilinear_gather.cu; args.map32 must be set); as cert_from_map.
int chunked_bilinear_from_map(int coord, int kind, GatherArgs &args, int n_det, cudaStream_t st,
                              void **work);

namespace {

// Adds the sample's map terms to its signal (src/Projection.cxx:1763-1765).
template <int P, int NT>
__device__ __forceinline__ void gather_taps(const GatherArgs &a, float *sp, int n,
                                            const int (*pix)[3], const float *w,
                                            const float *pf) {
    float sig = *sp;
    const int nc = a.g.ncomp;
#pragma unroll
    for (int k = 0; k < NT; k++) {
        if (k >= n) break;
        long long off, plane;
        int bad = locate<P>(a.g, pix[k], &off, &plane);
        if (bad >= 0) {
            record_missing_tile(a.err, bad);
            continue;
        }
#pragma unroll
        for (int c = 0; c < 3; c++)
            if (c < nc) sig += __ldg(a.map + off + c * plane) * pf[c] * w[k];
    }
    *sp = sig;
}

template <int C, int P>
__device__ __noinline__ void exact_gather(const GatherArgs &a, int det, int t, const QuatD &ofs, float T,
                             float Pr) {
    constexpr int NT = PixTraits<P>::taps;
    double coords[4];
    float pf[3];
    int pix[NT][3];
    float w[NT];
    get_coords<C>(a.g.lut, load_quat(a.bore + 4LL * t), ofs, coords);
    spin_factors(a.g.ncomp, coords, T, Pr, pf);
    const int n = get_pixels<P>(a.g, coords, pix, w);
    gather_taps<P, NT>(a, a.signal + det * a.sig_stride + t, n, pix, w, pf);
}

// One sample of the certified float32 tier's fallback through the full
// certified double-float pointing and certified float32 roundings of the
// reference's float64 sums; false (signal untouched) when any of them is
// not certain.
template <int C, int P>
__device__ __forceinline__ bool df_gather_cert(const GatherArgs &a, int det, int t,
                                               const dfl (&qd)[4], float T, float Pr) {
    constexpr int NT = PixTraits<P>::taps;
    const double *bp = a.bore + 4LL * t;
    const double2 lo = __ldg(reinterpret_cast<const double2 *>(bp));
    const double2 hi = __ldg(reinterpret_cast<const double2 *>(bp) + 1);
    dfl qb[4];
    if (!(df_split(lo.x, qb[0]) & df_split(lo.y, qb[1]) & df_split(hi.x, qb[2]) &
          df_split(hi.y, qb[3])))
        return false;
    int pix[NT][3];
    float pf[3], w[NT];
    int n = 0;
    const int nc = a.g.ncomp;
    if (!fast_pointing<C, P>(a.g, a.ft, a.fc, qb, qd, nc, T, Pr, pix, w, n, pf)) return false;
    if (n == 0) return true;
    float *sp = a.signal + det * a.sig_stride + t;
    float s = *sp;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NT; k++) {
        if (k >= n || !ok) break;
        long long off, plane;
        const int bad = locate<P>(a.g, pix[k], &off, &plane);
        if (bad >= 0) {
            record_missing_tile(a.err, bad);
            continue;
        }
#pragma unroll
        for (int c = 0; c < 3; c++)
            if (ok && c < nc) ok = fast_accum(s, __ldg(a.map + off + c * plane), pf[c], w[k]);
    }
    if (ok) *sp = s;
    return ok;
}

// Index of a located sample's pixel in the float32 map copy: its element
// offset for an untiled map; for a tiled map its pixel in the parent map
// (flat: row-major over (ny, nx); HEALPix: the NEST index tile * nppt + sub).
template <int P>
__device__ __forceinline__ long long map32_index(const DGeom &g, const int *pix, long long off) {
    if (P == PX_FLAT_T_NN || P == PX_FLAT_T_BL) {
        const int t = pix[0], row = div_small(t, g.ntx, g.inv_ntx), col = t - row * g.ntx;
        return (long long)(row * g.ty + pix[1]) * g.nx + (long long)col * g.tx + pix[2];
    }
    if (P == PX_HP_T) return (long long)pix[0] * g.nppt + pix[1];
    return off;
}

// One sample of the mixed-pointing fallback through the double-float
// pointing; false (signal untouched) when its pixel is not certified.  Its
// spin factors and terms, like the float32 tier's, are float32 evaluations
// (the mixed-precision contract).
template <int C, int P>
__device__ __forceinline__ bool df_gather(const GatherArgs &a, int det, int t, const dfl (&qd)[4], float T,
                          float Pr) {
    constexpr int NT = PixTraits<P>::taps;
    const double *bp = a.bore + 4LL * t;
    const double2 lo = __ldg(reinterpret_cast<const double2 *>(bp));
    const double2 hi = __ldg(reinterpret_cast<const double2 *>(bp) + 1);
    dfl qb[4];
    if (!(df_split(lo.x, qb[0]) & df_split(lo.y, qb[1]) & df_split(hi.x, qb[2]) &
          df_split(hi.y, qb[3])))
        return false;
    int pix[NT][3];
    float pf[3], w[NT];
    int n = 0;
    const int nc = a.g.ncomp;
    if (!fast_pointing<C, P, false>(a.g, a.ft, a.fc, qb, qd, nc, T, Pr, pix, w, n, pf))
        return false;
    if (n == 0) return true;
    float *sp = a.signal + det * a.sig_stride + t;
    float s = *sp;
#pragma unroll
    for (int k = 0; k < NT; k++) {
        if (k >= n) break;
        long long off, plane;
        const int bad = locate<P>(a.g, pix[k], &off, &plane);
        if (bad >= 0) {
            record_missing_tile(a.err, bad);
            continue;
        }
        if (a.map32) {
            const float4 m = __ldg(a.map32 + map32_index<P>(a.g, pix[k], off));
            s = fmaf(m.x, pf[0] * w[k], s);
            if (nc > 1) s = fmaf(m.y, pf[1] * w[k], s);
            if (nc > 2) s = fmaf(m.z, pf[2] * w[k], s);
        } else {
#pragma unroll
            for (int c = 0; c < 3; c++)
                if (c < nc) s = fmaf(d2f_round(__ldg(a.map + off + c * plane)), pf[c] * w[k], s);
        }
    }
    *sp = s;
    return true;
}

}  // namespace

}  // namespace so3g
