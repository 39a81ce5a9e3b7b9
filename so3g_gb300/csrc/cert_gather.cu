// cert_gather.cu -- from_map of the certified mode with the chunked pointing
// of cert_point.cuh, in the layout of cert_scatter.cuh: one 16-byte signal
// access per lane and four samples.
//
// The map is read from a copy made once per call (k_cx_map): per pixel, the
// components as double-float pairs side by side, so that a sample takes one
// or two 16-byte loads instead of a float64 load per plane and a split per
// value.  Each term's float32 rounding is certified as the spin factors'
// (cx_accum); a sample with an uncertain pixel, spin factor or term keeps
// its value in the main pass and goes through the per-sample paths.
//
// Bound by instruction issue and the latency of dependent instructions (67 %
// of the issue slots at 24 warps per SM).  CAR TQU 3 x 2000 x 2000, 1000 det x
// 1M samples: 30.9 -> 8.4 ms, and with the steps that two quantities or two
// samples share as f32x2 instructions 7.7 ms; with models for the longer side
// of the turn-arounds 7.3 ms (of which 0.93 ms the fallback).

#include "cert_point.cuh"
#include "cert_map.cuh"
#include "gather_kernel.cuh"

namespace so3g {

namespace {

// One sample the models left: the certified double-float pointing (false:
// not certain), the float64 pointing.
template <int C, int P>
__device__ __noinline__ bool cx_df_gather(const GatherArgs &a, int det, int t) {
    const QuatD ofs = load_quat(a.dets + 4LL * det);
    const dfl qd[4] = {df_of(ofs.a), df_of(ofs.b), df_of(ofs.c), df_of(ofs.d)};
    return df_gather_cert<C, P>(a, det, t, qd, __ldg(a.resp + 2 * det),
                                __ldg(a.resp + 2 * det + 1));
}

template <int C, int P>
__device__ __noinline__ void cx_exact_gather(const GatherArgs &a, int det, int t) {
    if constexpr (P == PX_HP_NT || P == PX_HP_T) {
        int pix[1][3], n;
        float pf[3];
        if (cx_exact_spin<C, P>(a, det, t, pix[0], n, pf)) {
            const float w[1] = {1.f};
            gather_taps<P, 1>(a, a.signal + det * a.sig_stride + t, n, pix, w, pf);
            return;
        }
    }
    exact_gather<C, P>(a, det, t, load_quat(a.dets + 4LL * det), __ldg(a.resp + 2 * det),
                       __ldg(a.resp + 2 * det + 1));
}

// Both in turn (a sample that does not fit the lists).
template <int C, int P>
__device__ __noinline__ void cx_any_gather(const GatherArgs &a, int det, int t) {
    if (!cx_df_gather<C, P>(a, det, t)) cx_exact_gather<C, P>(a, det, t);
}

// The lists of a call (as k_scatter_cx_fix).
template <int C, int P, int TIER>
__global__ void __launch_bounds__(kBlock) k_from_map_cx_fix(const __grid_constant__ GatherArgs a,
                                                            CxList list, CxList next) {
    cx_for_each(list, next,
                [&](int det, int t) -> bool {
                    if (TIER == 0) return cx_df_gather<C, P>(a, det, t);
                    cx_exact_gather<C, P>(a, det, t);
                    return true;
                },
                [&](int det, int t) { cx_exact_gather<C, P>(a, det, t); });
}

constexpr int kCxGatherBlocks = 6;   // resident blocks per SM (80 registers; 5 and 7 the same, 8: 3 % slower)

template <int CL, int P, int NC>
__global__ void __launch_bounds__(kCxBlock, kCxGatherBlocks)
    k_from_map_cx(const __grid_constant__ GatherArgs a, CxModel model, CxList left, int coord,
                  const float4 *cmap) {
    constexpr bool HP = P == PX_HP_NT || P == PX_HP_T;
    constexpr bool TILED = P == PX_FLAT_T_NN || P == PX_HP_T;
    constexpr int W = CxMap<NC, TILED>::W;
    __shared__ float4 s_model[kCxWarps][kCxGroup][kCxWords];
    __shared__ CxWarp s_warp[kCxWarps];
    int det, t0, t1;
    if (a.gate.holds()) return;
    if (!seg_piece(a.segs, a.piece, det, t0, t1)) return;
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
    const int tsh = P == PX_HP_T ? __ffsll(a.g.nppt) - 1 : 0;
    float *sig = a.signal + det * a.sig_stride;
    const bool vec = (reinterpret_cast<unsigned long long>(sig) & 15) == 0;
    auto over = [&](int t) {
        if constexpr (CL == CX_CAR) {
            cx_any_gather<SO3G_COORD_CAR, P>(a, det, t);
        } else {
            switch (coord) {
            case SO3G_COORD_TAN: cx_any_gather<SO3G_COORD_TAN, P>(a, det, t); break;
            case SO3G_COORD_ZEA: cx_any_gather<SO3G_COORD_ZEA, P>(a, det, t); break;
            default: cx_any_gather<SO3G_COORD_SIN, P>(a, det, t); break;
            }
        }
    };
    const int j0 = t0 / kCxLen, j1 = (t1 - 1) / kCxLen + 1;
    const int step = cx_step(j1 - j0);
    for (int g = j0 + warp * step; g < j1; g += kCxWarps * step) {
        const int nch = min(step, j1 - g);
        if (lane < nch)
            cx_setup<CL, HP, NC>(a, model.bore, coord, g + lane, n_time, qd, Pr, s_model[warp][lane]);
        __syncwarp();
        const int rounds = (nch + 1) / 2;
        for (int r = 0; r < rounds; r++) {
            const int ck = 2 * r + (lane >> 4);
            const int tq = (g + ck) * kCxLen + (lane & 15) * 4;
            const bool lane_live = ck < nch;
            const bool whole = vec && lane_live && tq + 3 < t1;
            // Loaded before the pointing, so that its latency overlaps it.
            float sv[4] = {0.f, 0.f, 0.f, 0.f};
            if (whole) {
                const float4 v = *reinterpret_cast<const float4 *>(sig + tq);
                sv[0] = v.x;
                sv[1] = v.y;
                sv[2] = v.z;
                sv[3] = v.w;
            } else if (lane_live) {
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (tq + i < t1) sv[i] = sig[tq + i];
            }
            const float4 *w = s_model[warp][min(ck, nch - 1)];
            const float4 w3 = w[3];
            const float kq = (float)(tq - __float_as_int(w3.z));
            float res[4][3];
            if (w3.w != 0.f) cx_residuals(model.resid, tq, res);
            unsigned f4 = 0u;
            // (In the whole warp: not a piece's end or an odd last chunk.)
            const bool full = (g + 2 * r + 2) * kCxLen <= t1 && 2 * r + 2 <= nch;
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
                bool act[2];
                float pf[2][3], hl[2][4 * W];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const bool live = full || (lane_live && tq + i + j < t1);
                    int key = 0;
                    bool on = false;
                    const bool ok = cx_sample<P, NC>(w, f2_both(kq + (float)(i + j)), res[i + j],
                                                     w3.w != 0.f, a.g, T, key, on, pf[j]);
                    if (live && !ok) f4 |= 1u << (i + j);
                    act[j] = live & ok & on;
#pragma unroll
                    for (int q = 0; q < W; q++) {
                        float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (act[j]) m = __ldg(cmap + (long long)key * W + q);
                        hl[j][4 * q] = m.x;
                        hl[j][4 * q + 1] = m.y;
                        hl[j][4 * q + 2] = m.z;
                        hl[j][4 * q + 3] = m.w;
                    }
                    if (TILED && act[j] && hl[j][4 * W - 1] == 0.f) {
                        act[j] = false;
                        if (P == PX_HP_T) {
                            record_missing_tile(a.err, key >> tsh);
                        } else {
                            int tp[3];
                            flat_tile_tuple(a.g, key / a.g.nx, key % a.g.nx, tp);
                            record_missing_tile(a.err, tp[0]);
                        }
                    }
                }
                float s0 = sv[i], s1 = sv[i + 1];
                bool c0 = true, c1 = true;
#pragma unroll
                for (int c = 0; c < NC; c++)
                    cx_accum2(s0, s1, hl[0][2 * c], hl[1][2 * c], hl[0][2 * c + 1], hl[1][2 * c + 1],
                              pf[0][c], pf[1][c], c0, c1);
                if (act[0] & !c0) c0 = cx_accum_all<NC, W>(sv[i], hl[0], pf[0], s0);
                if (act[1] & !c1) c1 = cx_accum_all<NC, W>(sv[i + 1], hl[1], pf[1], s1);
                if (act[0]) {
                    if (c0) sv[i] = s0;
                    else f4 |= 1u << i;
                }
                if (act[1]) {
                    if (c1) sv[i + 1] = s1;
                    else f4 |= 2u << i;
                }
            }
            if (whole) {
                *reinterpret_cast<float4 *>(sig + tq) = make_float4(sv[0], sv[1], sv[2], sv[3]);
            } else if (lane_live) {
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (tq + i < t1) sig[tq + i] = sv[i];
            }
            if (__any_sync(kFull, f4 != 0u) && cx_enqueue(cw, f4, tq) >= 32)
                cx_append(cw, left, det, over);
        }
        __syncwarp();
    }
    cx_append(cw, left, det, over);
}

template <int C, int P>
int cx_gather_fix(const GatherArgs &a, const CxWork &w, cudaStream_t st) {
    k_from_map_cx_fix<C, P, 0><<<kCxFixBlocks, kBlock, 0, st>>>(a, w.left, w.exact);
    const int rc = after_launch("certified fallback");
    if (rc != SO3G_OK) return rc;
    k_from_map_cx_fix<C, P, 1><<<kCxFixBlocks, kBlock, 0, st>>>(a, w.exact, w.exact);
    return after_launch("certified fallback (exact)");
}

template <int CL, int P, int NC>
int cx_gather_run(const GatherArgs &a, const CxWork &w, int coord, long long npix, dim3 grid,
                  cudaStream_t st) {
    constexpr int W = CxMap<NC, P == PX_FLAT_T_NN || P == PX_HP_T>::W;
    float4 *cmap = nullptr;
    if (cudaMallocAsync(reinterpret_cast<void **>(&cmap), sizeof(float4) * W * (size_t)npix, st) !=
        cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    int rc = cx_probe<CL, P == PX_HP_NT || P == PX_HP_T, NC, false>(a, w, coord, grid.x, nullptr, st);
    if (rc == SO3G_OK) {
        k_cx_map<P, NC><<<(unsigned)((npix + kBlock - 1) / kBlock), kBlock, 0, st>>>(
            a.g, a.map, npix, cmap, a.gate);
        rc = after_launch("from_map (map copy)");
    }
    if (rc == SO3G_OK) {
        k_from_map_cx<CL, P, NC><<<grid, kCxBlock, 0, st>>>(a, w.model, w.left, coord, cmap);
        rc = after_launch("from_map (certified, chunked)");
    }
    cudaFreeAsync(cmap, st);
    if (rc != SO3G_OK) return rc;
    if constexpr (CL == CX_CAR) {
        return cx_gather_fix<SO3G_COORD_CAR, P>(a, w, st);
    } else {
        switch (coord) {
        case SO3G_COORD_TAN: return cx_gather_fix<SO3G_COORD_TAN, P>(a, w, st);
        case SO3G_COORD_ZEA: return cx_gather_fix<SO3G_COORD_ZEA, P>(a, w, st);
        default: return cx_gather_fix<SO3G_COORD_SIN, P>(a, w, st);
        }
    }
}

template <int CL, int P>
int cx_gather_nc(const GatherArgs &a, const CxWork &w, int coord, long long npix, dim3 grid,
                 cudaStream_t st) {
    switch (a.g.ncomp) {
    case 1: return cx_gather_run<CL, P, 1>(a, w, coord, npix, grid, st);
    case 2: return cx_gather_run<CL, P, 2>(a, w, coord, npix, grid, st);
    default: return cx_gather_run<CL, P, 3>(a, w, coord, npix, grid, st);
    }
}

// Largest map (parent map when tiled) that gets the copy: 32 bytes a pixel.
constexpr long long kCxMapMaxPixels = 1LL << 28;

}  // namespace

int cert_from_map(int coord, int kind, GatherArgs &args, int n_det, cudaStream_t st,
                  void **work) {
    const bool hp = kind == PX_HP_NT || kind == PX_HP_T;
    const bool flat = kind == PX_FLAT_NT_NN || kind == PX_FLAT_T_NN;
    const bool zen = coord == SO3G_COORD_TAN || coord == SO3G_COORD_ZEA ||
                     coord == SO3G_COORD_SIN;
    GatherArgs a = args;
    const long long npix = hp ? a.g.npix : (long long)a.g.ny * a.g.nx;
    const long long n_time = a.segs.n_time, samples = n_time * n_det;
    const long long least = cert_chunked_min_samples();
    // The map copy (1e-5 us a pixel) must pay for itself, from the 2.4e-5 us
    // a sample that the chunked kernel saves (HEALPix nside 1024: 6.4M samples
    // 284 us against 268, 10M 329 against 392).
    if (a.fast != SO3G_POINTING_CERTIFIED || !(hp || flat) ||
        !(coord == SO3G_COORD_CAR || (flat && zen)) || n_time <= kCxLen || npix <= 0 ||
        npix > kCxMapMaxPixels || samples < least || (least > 0 && 2 * (samples - least) < npix))
        return 1;
    CxWork w;
    if (!cx_work(w, a.bore, (int)n_time, samples, st)) return 1;
    a.piece = cx_piece(n_det, n_time);
    a.gate = w.gate;
    const dim3 grid((unsigned)n_det, (unsigned)((n_time + a.piece - 1) / a.piece));
    int rc;
    if (hp) {
        if (kind == PX_HP_NT) rc = cx_gather_nc<CX_CAR, PX_HP_NT>(a, w, coord, npix, grid, st);
        else rc = cx_gather_nc<CX_CAR, PX_HP_T>(a, w, coord, npix, grid, st);
    } else if (kind == PX_FLAT_NT_NN) {
        if (zen) rc = cx_gather_nc<CX_ZEN, PX_FLAT_NT_NN>(a, w, coord, npix, grid, st);
        else rc = cx_gather_nc<CX_CAR, PX_FLAT_NT_NN>(a, w, coord, npix, grid, st);
    } else {
        if (zen) rc = cx_gather_nc<CX_ZEN, PX_FLAT_T_NN>(a, w, coord, npix, grid, st);
        else rc = cx_gather_nc<CX_CAR, PX_FLAT_T_NN>(a, w, coord, npix, grid, st);
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

}  // namespace so3g
