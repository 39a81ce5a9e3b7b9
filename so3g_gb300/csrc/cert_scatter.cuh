// cert_scatter.cuh -- to_map / to_weight_map of the certified mode with the
// chunked pointing of cert_point.cuh (cert_scatter.cu: to_map, cert_weight.cu:
// to_weight_map).
//
// A warp sets up the models of up to 32 consecutive chunks of its detector
// (one lane each, in shared memory), then walks them in rounds of 128
// samples: two chunks (lanes 0-15 and 16-31), four consecutive samples per
// lane with one 16-byte signal load, the next round's signal loaded while
// the current one is evaluated.  A lane sums the runs of equal pixels among
// its four samples (TwoSum: to ~2^-46), one float64 atomic per run and
// component (CxRuns).  Samples the models
// do not certify go to a list and from there through the per-sample
// certified path and, if need be, the float64 one (k_scatter_cx_fix).
//
// Bound by instruction issue and the latency of dependent instructions (65 %
// of the issue slots at 20 warps per SM; ~195 warp-instructions per 32 samples,
// the per-sample path ~910), then by the L2 atomic units.  CAR TQU 3 x 2000 x
// 2000, 1000 det x 1M samples: to_map 26.1 -> 8.3 ms, with f32x2 instructions
// for the coordinates, the spin factors and the runs' sums 8.0 ms, with models
// for the longer side of the turn-arounds 7.9 ms, with the bounds on accelerating
// scans 8.0 ms (of which 0.78 ms the fallback), to_weight_map of 500 x 500k 7.4 ->
// 2.8 ms; HEALPix nside 1024, 400 det x 500k, to_map + from_map 14.8 -> 5.8 ms.
#pragma once

#include <algorithm>

#include "cert_point.cuh"
#include "scatter_kernel.cuh"

namespace so3g {

namespace {

// One sample the models left: the certified double-float pointing (false:
// not certain), the float64 pointing.
template <int C, int P, bool WEIGHT>
__device__ __noinline__ bool cx_df_sample(const ScatterArgs &a, int det, int t) {
    int mult[WEIGHT ? 6 : 3];
    const unsigned vmask = value_slots<WEIGHT>(a.g.ncomp, mult);
    const QuatD ofs = load_quat(a.dets + 4LL * det);
    const dfl qd[4] = {df_of(ofs.a), df_of(ofs.b), df_of(ofs.c), df_of(ofs.d)};
    const float T = __ldg(a.resp + 2 * det), Pr = __ldg(a.resp + 2 * det + 1);
    const float wt = a.det_weights ? __ldg(a.det_weights + det) : 1.f;
    return df_sample<C, P, WEIGHT, true>(a, det, t, qd, T, Pr, wt, mult, vmask);
}

template <int C, int P, bool WEIGHT>
__device__ __noinline__ void cx_exact_sample(const ScatterArgs &a, int det, int t) {
    constexpr int NV = WEIGHT ? 6 : 3;
    int mult[NV];
    const unsigned vmask = value_slots<WEIGHT>(a.g.ncomp, mult);
    const float T = __ldg(a.resp + 2 * det), Pr = __ldg(a.resp + 2 * det + 1);
    const float wt = a.det_weights ? __ldg(a.det_weights + det) : 1.f;
    if constexpr (P == PX_HP_NT || P == PX_HP_T) {
        int pix[3], n;
        float pf[3];
        if (cx_exact_spin<C, P>(a, det, t, pix, n, pf)) {
            if (n == 0) return;
            long long off, plane;
            const int bad = locate<P>(a.g, pix, &off, &plane);
            if (bad >= 0) {
                record_missing_tile(a.err, bad);
                return;
            }
            const float sig = WEIGHT ? 0.f : __ldg(a.signal + det * a.sig_stride + t);
            float v[NV];
            tap_values<WEIGHT, NV, true>(sig, pf, 1.f, wt, v);
#pragma unroll
            for (int k = 0; k < NV; k++)
                if ((vmask >> k) & 1u) atomicAdd(a.map + off + mult[k] * plane, f2d(v[k]));
            return;
        }
    }
    exact_sample<C, P, WEIGHT>(a, det, t, load_quat(a.dets + 4LL * det), T, Pr, wt, mult, vmask);
}

// Both in turn (a sample that does not fit the lists).
template <int C, int P, bool WEIGHT>
__device__ __noinline__ void cx_any_sample(const ScatterArgs &a, int det, int t) {
    if (!cx_df_sample<C, P, WEIGHT>(a, det, t)) cx_exact_sample<C, P, WEIGHT>(a, det, t);
}

// The lists of a call: TIER 0 the samples the models left, 1 those the
// double-float pointing left.
template <int C, int P, bool WEIGHT, int TIER>
__global__ void __launch_bounds__(kBlock) k_scatter_cx_fix(const __grid_constant__ ScatterArgs a,
                                                           CxList list, CxList next) {
    cx_for_each(list, next,
                [&](int det, int t) -> bool {
                    if (TIER == 0) return cx_df_sample<C, P, WEIGHT>(a, det, t);
                    cx_exact_sample<C, P, WEIGHT>(a, det, t);
                    return true;
                },
                [&](int det, int t) { cx_exact_sample<C, P, WEIGHT>(a, det, t); });
}

// Value k of a to_map (component k) or to_weight_map (upper-triangle pair
// in row order) of NC components: its pair and plane.
template <int NC>
__device__ constexpr int cx_pair_i(int k) {
    return NC == 3 ? (k < 3 ? 0 : (k < 5 ? 1 : 2)) : (NC == 2 ? (k < 2 ? 0 : 1) : 0);
}
template <int NC>
__device__ constexpr int cx_pair_j(int k) {
    return NC == 3 ? (k < 3 ? k : (k < 5 ? k - 2 : 2)) : (NC == 2 ? (k < 2 ? k : 1) : 0);
}
template <bool WEIGHT, int NC>
__device__ constexpr int cx_plane(int k) {
    return WEIGHT ? cx_pair_i<NC>(k) * NC + cx_pair_j<NC>(k) : k;
}

// Tiled maps: address and plane size of a key (flat: iy * nx + ix of the
// parent map; HEALPix: the pixel); NULL for an absent tile, which is
// recorded.  aux: log2 of the pixels per tile (tiled HEALPix), the bits of
// 1/nx as a float (tiled flat).
template <int P>
__device__ __forceinline__ double *cx_address(const ScatterArgs &a, int key, int aux, int &plane) {
    int tile, off;
    if constexpr (P == PX_HP_T) {
        tile = key >> aux;
        off = key & ((1 << aux) - 1);
    } else {
        // (flat_tile_tuple and locate in one: two divisions by the tile.)
        const int iy = div_small(key, a.g.nx, __int_as_float(aux)), ix = key - iy * a.g.nx;
        const int sy = div_small(iy, a.g.ty, a.g.inv_ty), sx = div_small(ix, a.g.tx, a.g.inv_tx);
        const int y0 = sy * a.g.ty, x0 = sx * a.g.tx;
        const int tnx = min(a.g.tx, a.g.nx - x0);
        tile = sy * a.g.ntx + sx;
        off = (iy - y0) * tnx + (ix - x0);
        plane = min(a.g.ty, a.g.ny - y0) * tnx;
    }
    const long long toff = __ldg(a.g.tile_offset + tile);
    if (toff < 0) {
        record_missing_tile(a.err, tile);
        return nullptr;
    }
    return a.map + toff + off;
}

// The term of value k of a sample (float32 products, left to right, as
// tap_values).
template <bool WEIGHT, int NC>
__device__ __forceinline__ float cx_value(int k, float sig, const float (&pf)[3], float det_wt) {
    if (WEIGHT) return pf[cx_pair_i<NC>(k)] * pf[cx_pair_j<NC>(k)] * det_wt;
    return sig * pf[k] * det_wt;
}

// Adds a run's totals (hi + lo) to the map (key < 0: nothing).  A lo that is
// NaN (an infinite hi) is left out.
template <int P, bool WEIGHT, int NC, int NV>
__device__ __forceinline__ void cx_flush(const ScatterArgs &a, int key, int aux, int plane,
                                         const float (&hi)[NV], const float (&lo)[NV]) {
    if (key < 0) return;
    double *p = nullptr;
    if constexpr (P == PX_FLAT_T_NN || P == PX_HP_T) {
        p = cx_address<P>(a, key, aux, plane);
        if (!p) return;
    }
#pragma unroll
    for (int c = 0; c < NV; c++) {
        double d = f2d(hi[c]);
        if (fabsf(lo[c]) > 0.f) d += f2d(lo[c]);
        const int pl = cx_plane<WEIGHT, NC>(c);
        // Untiled: the plane's base is the same in every lane.
        if constexpr (P == PX_FLAT_NT_NN || P == PX_HP_NT)
            atomicAdd((a.map + (long long)pl * plane) + key, d);
        else
            atomicAdd(p + pl * plane, d);
    }
}

// Runs a warp holds back until there are 32 to flush together: key, totals.
// A lane's first run is flushed at once (nearly every lane has one), its
// others (about half the lanes have one) go here: 1.6 full passes of atomics
// per 128 samples where flushing slot by slot took 2.2 part-filled ones, one
// copy of the flush code instead of four.
template <int NV>
struct CxRuns {
    // Most runs a round may add (else it is added term by term); six values
    // a run leave room for fewer (20 warps on an SM).
    static constexpr int more = NV > 3 ? 48 : 64;
    static constexpr int W = (1 + 2 * NV + 3) / 4;
    float4 rec[W][more + 32];
};

template <int NV>
__device__ __forceinline__ void cx_run_put(CxRuns<NV> &rb, int pos, int key, const float (&hi)[NV],
                                           const float (&lo)[NV]) {
    constexpr int W = CxRuns<NV>::W;
    float x[4 * W];
#pragma unroll
    for (int k = 0; k < 4 * W; k++)
        x[k] = k == 0 ? __int_as_float(key)
                      : (k <= NV ? hi[k <= NV ? k - 1 : 0]
                                 : (k <= 2 * NV ? lo[k <= 2 * NV && k > NV ? k - 1 - NV : 0] : 0.f));
#pragma unroll
    for (int w = 0; w < W; w++)
        rb.rec[w][pos] = make_float4(x[4 * w], x[4 * w + 1], x[4 * w + 2], x[4 * w + 3]);
}

// Flushes the last min(32, n) runs held back, one per lane.
template <int P, bool WEIGHT, int NC, int NV>
__device__ __forceinline__ void cx_run_flush(const ScatterArgs &a, CxRuns<NV> &rb, int n, int aux,
                                             int plane) {
    constexpr int W = CxRuns<NV>::W;
    const int i = n - 1 - (int)(threadIdx.x & 31);
    if (i < 0) return;
    float x[4 * W], hi[NV], lo[NV];
#pragma unroll
    for (int w = 0; w < W; w++) {
        const float4 v = rb.rec[w][i];
        x[4 * w] = v.x;
        x[4 * w + 1] = v.y;
        x[4 * w + 2] = v.z;
        x[4 * w + 3] = v.w;
    }
#pragma unroll
    for (int k = 0; k < NV; k++) {
        hi[k] = x[1 + k];
        lo[k] = x[1 + NV + k];
    }
    cx_flush<P, WEIGHT, NC, NV>(a, __float_as_int(x[0]), aux, plane, hi, lo);
}

// The total a of a run (a term) plus b's, the roundings in lo.
template <int NV>
__device__ __forceinline__ void cx_join(float (&a)[NV], float (&lo)[NV], const float (&b)[NV],
                                        const float (&blo)[NV]) {
    if constexpr (NV & 1) {
        float e;
        two_sum(a[0], b[0], a[0], e);
        lo[0] = blo[0] + e;
    }
#pragma unroll
    for (int c = NV & 1; c + 1 < NV; c += 2) {
        f32x2 s, e;
        f2_two_sum(f2_make(a[c], a[c + 1]), f2_make(b[c], b[c + 1]), s, e);
        f2_get(s, a[c], a[c + 1]);
        f2_get(f2_add(f2_make(blo[c], blo[c + 1]), e), lo[c], lo[c + 1]);
    }
}

// The runs of equal pixels among a lane's four samples: the first flushed,
// the others held back (nr: runs held back so far; flushed down to fewer
// than 32).  False (nothing done) when the round has too many further
// runs.  All lanes must call.
template <int P, bool WEIGHT, int NC, int NV>
__device__ __forceinline__ bool cx_runs4(const ScatterArgs &a, CxRuns<NV> &rb, int &nr, int aux,
                                         int plane, const int (&key)[4], const float (&sig)[4],
                                         const float (&pf)[4][3], float det_wt) {
    const bool h1 = key[1] != key[0], h2 = key[2] != key[1], h3 = key[3] != key[2];
    const bool p1 = h1 & (key[1] >= 0), p2 = h2 & (key[2] >= 0), p3 = h3 & (key[3] >= 0);
    const int n = (int)p1 + (int)p2 + (int)p3;
    const unsigned b0 = __ballot_sync(kFull, n & 1), b1 = __ballot_sync(kFull, n & 2);
    const int total = __popc(b0) + 2 * __popc(b1);
    if (total > CxRuns<NV>::more) return false;
    float v[4][NV], lo[4][NV];
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int c = 0; c < NV; c++) {
            v[j][c] = cx_value<WEIGHT, NC>(c, sig[j], pf[j], det_wt);
            lo[j][c] = 0.f;
        }
    // Right to left: v[i] + lo[i] becomes the total of the run from i on.
    if (!h3) cx_join<NV>(v[2], lo[2], v[3], lo[3]);
    if (!h2) cx_join<NV>(v[1], lo[1], v[2], lo[2]);
    if (!h1) cx_join<NV>(v[0], lo[0], v[1], lo[1]);
    if (total) {
        const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
        int pos = nr + __popc(b0 & lt) + 2 * __popc(b1 & lt);
        if (p1) cx_run_put<NV>(rb, pos, key[1], v[1], lo[1]);
        pos += p1;
        if (p2) cx_run_put<NV>(rb, pos, key[2], v[2], lo[2]);
        pos += p2;
        if (p3) cx_run_put<NV>(rb, pos, key[3], v[3], lo[3]);
        nr += total;
        __syncwarp();
    }
    cx_flush<P, WEIGHT, NC, NV>(a, key[0], aux, plane, v[0], lo[0]);
    while (nr >= 32) {
        cx_run_flush<P, WEIGHT, NC, NV>(a, rb, nr, aux, plane);
        nr -= 32;
        __syncwarp();
    }
    return true;
}

// Resident blocks per SM: 20 warps with 96 registers (to_map: 7.9 ms for 1000
// det x 1M samples; 24 warps with 80, more spills, 9.1 ms), 16 (to_weight_map,
// whose held-back runs take more shared memory; 20: 2 % slower).
template <bool WEIGHT>
struct CxScatterBlocks {
    static constexpr int value = WEIGHT ? 4 : 5;
};

template <int CL, int P, bool WEIGHT, int NC>
__global__ void __launch_bounds__(kCxBlock, CxScatterBlocks<WEIGHT>::value)
    k_scatter_cx(const __grid_constant__ ScatterArgs a, CxModel model, CxList left, int coord) {
    constexpr bool HP = P == PX_HP_NT || P == PX_HP_T;
    constexpr int NV = WEIGHT ? NC * (NC + 1) / 2 : NC;
    __shared__ float4 s_model[kCxWarps][kCxGroup][kCxWords];
    __shared__ CxWarp s_warp[kCxWarps];
    __shared__ CxRuns<NV> s_runs[kCxWarps];
    int det, t0, t1;
    if (a.gate.holds()) return;
    if (!seg_piece(a.segs, a.piece, det, t0, t1)) return;
    float det_wt = 1.f;
    if (a.det_weights) {
        det_wt = __ldg(a.det_weights + det);
        if (det_wt == 0.f) return;  // src/Projection.cxx:1784-1788
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    CxWarp &cw = s_warp[warp];
    dfl qd[4];
    {
        const QuatD ofs = load_quat(a.dets + 4LL * det);
        qd[0] = df_of(ofs.a);
        qd[1] = df_of(ofs.b);
        qd[2] = df_of(ofs.c);
        qd[3] = df_of(ofs.d);
        if (lane == 0) cw.n = 0;
        __syncwarp();
    }
    const float T = __ldg(a.resp + 2 * det), Pr = __ldg(a.resp + 2 * det + 1);
    const int n_time = a.segs.n_time;
    const int plane = P == PX_HP_NT ? (int)a.g.npix
                                    : (P == PX_HP_T ? (int)a.g.nppt : a.g.ny * a.g.nx);
    const int aux = P == PX_HP_T ? __ffsll(a.g.nppt) - 1
                    : (P == PX_FLAT_T_NN ? __float_as_int(1.f / (float)a.g.nx) : 0);
    // A run total that would leave float32's range (or an infinite or NaN
    // term) is added term by term: sums of |signal| (weights: 1) up to lim.
    const float lim = 1e36f / fmaxf(fmaxf(fabsf(T), fabsf(Pr)) *
                                        (WEIGHT ? fmaxf(fabsf(T), fabsf(Pr)) : 1.f) *
                                        fabsf(det_wt), 1e-30f);
    const float *sig = WEIGHT ? nullptr : a.signal + det * a.sig_stride;
    const bool vec = (reinterpret_cast<unsigned long long>(sig) & 15) == 0;
    auto load4 = [&](int tq) {
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (WEIGHT) return r;
        if (vec && tq >= t0 && tq + 3 < t1) {
            r = __ldg(reinterpret_cast<const float4 *>(sig + tq));
        } else {
            if (tq >= t0 && tq < t1) r.x = __ldg(sig + tq);
            if (tq + 1 >= t0 && tq + 1 < t1) r.y = __ldg(sig + tq + 1);
            if (tq + 2 >= t0 && tq + 2 < t1) r.z = __ldg(sig + tq + 2);
            if (tq + 3 >= t0 && tq + 3 < t1) r.w = __ldg(sig + tq + 3);
        }
        return r;
    };
    auto over = [&](int t) {
        if constexpr (CL == CX_CAR) {
            cx_any_sample<SO3G_COORD_CAR, P, WEIGHT>(a, det, t);
        } else {
            switch (coord) {
            case SO3G_COORD_TAN: cx_any_sample<SO3G_COORD_TAN, P, WEIGHT>(a, det, t); break;
            case SO3G_COORD_ZEA: cx_any_sample<SO3G_COORD_ZEA, P, WEIGHT>(a, det, t); break;
            default: cx_any_sample<SO3G_COORD_SIN, P, WEIGHT>(a, det, t); break;
            }
        }
    };
    int nr = 0;   // runs held back
    const int j0 = t0 / kCxLen, j1 = (t1 - 1) / kCxLen + 1;
    const int step = cx_step(j1 - j0);
    for (int g = j0 + warp * step; g < j1; g += kCxWarps * step) {
        const int nch = min(step, j1 - g);
        if (lane < nch)
            cx_setup<CL, HP, NC>(a, model.bore, coord, g + lane, n_time, qd, Pr, s_model[warp][lane]);
        __syncwarp();
        const int rounds = (nch + 1) / 2;
        const int half = lane >> 4;
        float4 sn = half < nch ? load4((g + half) * kCxLen + (lane & 15) * 4)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = 0; r < rounds; r++) {
            const float4 sc = sn;
            const int ck = 2 * r + half;
            if (r + 1 < rounds && ck + 2 < nch) sn = load4((g + ck + 2) * kCxLen + (lane & 15) * 4);
            const int tq = (g + ck) * kCxLen + (lane & 15) * 4;
            const bool lane_live = ck < nch;
            const float4 *w = s_model[warp][min(ck, nch - 1)];
            const float4 w3 = w[3];
            const float kq = (float)(tq - __float_as_int(w3.z));
            float res[4][3];
            if (w3.w != 0.f) cx_residuals(model.resid, tq, res);
            const float sg[4] = {sc.x, sc.y, sc.z, sc.w};
            int key[4];
            float pf[4][3];
            unsigned f4 = 0u;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                int kk = 0;
                bool on = false;
                const bool ok = cx_sample<P, NC>(w, f2_both(kq + (float)i), res[i], w3.w != 0.f,
                                                  a.g, T, kk, on, pf[i]);
                if (!ok) f4 |= 1u << i;
                key[i] = (ok & on) ? kk : -1;
            }
            // A round at the segment's ends, or the group's odd last chunk.
            const int tr = (g + 2 * r) * kCxLen;
            if (tr < t0 || tr + 2 * kCxLen > t1 || 2 * r + 2 > nch) {
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (!(lane_live && tq + i >= t0 && tq + i < t1)) {
                        f4 &= ~(1u << i);
                        key[i] = -1;
                    }
            }
            const float size = WEIGHT ? 1.f : fabsf(sg[0]) + fabsf(sg[1]) + fabsf(sg[2]) + fabsf(sg[3]);
            const bool by_run =
                a.accum == SO3G_ACCUM_WARP_RUNS && __all_sync(kFull, size < lim) &&
                cx_runs4<P, WEIGHT, NC, NV>(a, s_runs[warp], nr, aux, plane, key, sg, pf, det_wt);
            if (!by_run) {
#pragma unroll 1
                for (int i = 0; i < 4; i++) {
                    const int kk = i == 0 ? key[0] : (i == 1 ? key[1] : (i == 2 ? key[2] : key[3]));
                    const float s = i == 0 ? sg[0] : (i == 1 ? sg[1] : (i == 2 ? sg[2] : sg[3]));
                    float f[3], v[NV], z[NV];
#pragma unroll
                    for (int c = 0; c < 3; c++)
                        f[c] = i == 0 ? pf[0][c] : (i == 1 ? pf[1][c] : (i == 2 ? pf[2][c] : pf[3][c]));
#pragma unroll
                    for (int k = 0; k < NV; k++) {
                        v[k] = cx_value<WEIGHT, NC>(k, s, f, det_wt);
                        z[k] = 0.f;
                    }
                    cx_flush<P, WEIGHT, NC, NV>(a, kk, aux, plane, v, z);
                }
            }
            if (__any_sync(kFull, f4 != 0u) && cx_enqueue(cw, f4, tq) >= 32)
                cx_append(cw, left, det, over);
        }
        __syncwarp();
    }
    if (nr > 0) cx_run_flush<P, WEIGHT, NC, NV>(a, s_runs[warp], nr, aux, plane);
    cx_append(cw, left, det, over);
}

template <int C, int P, bool WEIGHT>
int cx_scatter_fix(const ScatterArgs &a, const CxWork &w, cudaStream_t st) {
    k_scatter_cx_fix<C, P, WEIGHT, 0><<<kCxFixBlocks, kBlock, 0, st>>>(a, w.left, w.exact);
    const int rc = after_launch("certified fallback");
    if (rc != SO3G_OK) return rc;
    k_scatter_cx_fix<C, P, WEIGHT, 1><<<kCxFixBlocks, kBlock, 0, st>>>(a, w.exact, w.exact);
    return after_launch("certified fallback (exact)");
}

template <int CL, int P, bool WEIGHT, int NC>
int cx_scatter_main(const ScatterArgs &a, const CxWork &w, int coord, dim3 grid, cudaStream_t st) {
    constexpr bool HP = P == PX_HP_NT || P == PX_HP_T;
    const int rc = cx_probe<CL, HP, NC, false>(a, w, coord, grid.x, a.det_weights, st);
    if (rc != SO3G_OK) return rc;
    k_scatter_cx<CL, P, WEIGHT, NC><<<grid, kCxBlock, 0, st>>>(a, w.model, w.left, coord);
    return after_launch(WEIGHT ? "to_weight_map (certified, chunked)"
                               : "to_map (certified, chunked)");
}

template <int CL, int P, bool WEIGHT>
int cx_scatter_launch(const ScatterArgs &a, const CxWork &w, int coord, dim3 grid,
                      cudaStream_t st) {
    int rc;
    switch (a.g.ncomp) {
    case 1: rc = cx_scatter_main<CL, P, WEIGHT, 1>(a, w, coord, grid, st); break;
    case 2: rc = cx_scatter_main<CL, P, WEIGHT, 2>(a, w, coord, grid, st); break;
    default: rc = cx_scatter_main<CL, P, WEIGHT, 3>(a, w, coord, grid, st); break;
    }
    if (rc != SO3G_OK) return rc;
    if constexpr (CL == CX_CAR) {
        return cx_scatter_fix<SO3G_COORD_CAR, P, WEIGHT>(a, w, st);
    } else {
        switch (coord) {
        case SO3G_COORD_TAN: return cx_scatter_fix<SO3G_COORD_TAN, P, WEIGHT>(a, w, st);
        case SO3G_COORD_ZEA: return cx_scatter_fix<SO3G_COORD_ZEA, P, WEIGHT>(a, w, st);
        default: return cx_scatter_fix<SO3G_COORD_SIN, P, WEIGHT>(a, w, st);
        }
    }
}

// Runs the chunked certified kernel on a call of n_seg segments of up to
// max_len samples; returns 1 (nothing launched) where it does not apply:
// another mode or pixelizor, planes whose offsets leave 32 bits, timelines
// shorter than a chunk, calls below cert_chunked_min_samples(), or no
// memory for the boresight models.
template <bool WEIGHT>
int cx_scatter(int coord, int kind, ScatterArgs &args, int n_det, long long n_seg,
               long long max_len, cudaStream_t st, void **work) {
    ScatterArgs a = args;
    const bool hp = kind == PX_HP_NT || kind == PX_HP_T;
    const bool flat = kind == PX_FLAT_NT_NN || kind == PX_FLAT_T_NN;
    const bool zen = coord == SO3G_COORD_TAN || coord == SO3G_COORD_ZEA ||
                     coord == SO3G_COORD_SIN;
    const long long nc = a.g.ncomp, npix = hp ? a.g.npix : (long long)a.g.ny * a.g.nx;
    // At most (sample ranges may overlap, but rarely do).
    const long long samples = std::min(n_seg * max_len, (long long)n_det * a.segs.n_time);
    if (a.fast != SO3G_POINTING_CERTIFIED || !(hp || flat) ||
        !(coord == SO3G_COORD_CAR || (flat && zen)) || a.segs.n_time <= kCxLen || npix <= 0 ||
        (WEIGHT ? nc * nc : nc) * npix >= (1LL << 31) || samples < cert_chunked_min_samples())
        return 1;
    CxWork w;
    if (!cx_work(w, a.bore, a.segs.n_time, samples, st)) return 1;
    a.piece = cx_piece(n_seg, max_len);
    a.gate = w.gate;
    const dim3 grid((unsigned)n_seg, (unsigned)((max_len + a.piece - 1) / a.piece));
    int rc;
    if (hp) {
        if (kind == PX_HP_NT) rc = cx_scatter_launch<CX_CAR, PX_HP_NT, WEIGHT>(a, w, coord, grid, st);
        else rc = cx_scatter_launch<CX_CAR, PX_HP_T, WEIGHT>(a, w, coord, grid, st);
    } else if (kind == PX_FLAT_NT_NN) {
        if (zen) rc = cx_scatter_launch<CX_ZEN, PX_FLAT_NT_NN, WEIGHT>(a, w, coord, grid, st);
        else rc = cx_scatter_launch<CX_CAR, PX_FLAT_NT_NN, WEIGHT>(a, w, coord, grid, st);
    } else {
        if (zen) rc = cx_scatter_launch<CX_ZEN, PX_FLAT_T_NN, WEIGHT>(a, w, coord, grid, st);
        else rc = cx_scatter_launch<CX_CAR, PX_FLAT_T_NN, WEIGHT>(a, w, coord, grid, st);
    }
    if (rc != SO3G_OK) {
        cudaFreeAsync(w.mem, st);
        return rc;
    }
    *work = w.mem;
    args.gate = w.gate;
    args.gate.skip = false;
    return SO3G_OK;
}

}  // namespace

}  // namespace so3g
