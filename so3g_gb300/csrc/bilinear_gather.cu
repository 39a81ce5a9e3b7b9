// bilinear_gather.cu -- from_map of untiled bilinear TAN, ZEA and SIN maps in
// the mixed mode with the chunked pointing of cert_point.cuh (its bilinear
// form).
//
// A bilinear weight needs the fraction of the pixel coordinate to float32
// accuracy, so the coordinates are held as the spin factors are, an exact
// float32 part plus a correction (within kCxBlPix of the reference's), and the
// weights formed from the fraction in double-float; the terms are float32 sums
// over the float32 map copy.  The certified mode keeps the per-sample kernels:
// its weights are the floats nearest the double-float coordinates' weights,
// which a float32 correction does not give in every last bit.  (CAR's
// coordinates come from interpolation tables, whose kinks the chunk models do
// not follow to that accuracy: it keeps the per-sample kernels; so does to_map,
// whose float64 sums keep the per-sample weights to the last bit.)
//
// Bound by instruction issue: the per-sample kernel ~850 warp-instructions
// per 32 samples (3000 x 3000 ZEA map of 0.5' pixels, 400 det x 300k: 2.9 -> 1.2
// ms; with f32x2 instructions the same, within 1 %).

#include "cert_point.cuh"
#include "gather_kernel.cuh"

namespace so3g {

namespace {

// One sample the models left: the double-float pointing (false: not
// certain), the float64 pointing.
template <int C>
__device__ __noinline__ bool bl_df_sample(const GatherArgs &a, int det, int t) {
    const QuatD ofs = load_quat(a.dets + 4LL * det);
    const dfl qd[4] = {df_of(ofs.a), df_of(ofs.b), df_of(ofs.c), df_of(ofs.d)};
    return df_gather<C, PX_FLAT_NT_BL>(a, det, t, qd, __ldg(a.resp + 2 * det),
                                       __ldg(a.resp + 2 * det + 1));
}

template <int C>
__device__ __noinline__ void bl_exact_sample(const GatherArgs &a, int det, int t) {
    exact_gather<C, PX_FLAT_NT_BL>(a, det, t, load_quat(a.dets + 4LL * det),
                                   __ldg(a.resp + 2 * det), __ldg(a.resp + 2 * det + 1));
}

template <int C>
__device__ __noinline__ void bl_any_sample(const GatherArgs &a, int det, int t) {
    if (!bl_df_sample<C>(a, det, t)) bl_exact_sample<C>(a, det, t);
}

template <int C, int TIER>
__global__ void __launch_bounds__(kBlock) k_from_map_bl_fix(const __grid_constant__ GatherArgs a,
                                                            CxList list, CxList next) {
    cx_for_each(list, next,
                [&](int det, int t) -> bool {
                    if (TIER == 0) return bl_df_sample<C>(a, det, t);
                    bl_exact_sample<C>(a, det, t);
                    return true;
                },
                [&](int det, int t) { bl_exact_sample<C>(a, det, t); });
}

// A pixel coordinate's floor and fraction from its exact part S and
// correction L (both less 1/2): false within e of an integer.
__device__ __forceinline__ bool bl_floor(float S, float L, float e, int base, int &i, dfl &frac) {
    const float r = (S + L) + kCxMagic, f = S - (r - kCxMagic);   // f exact
    i = base + __float_as_int(r);
    const dfl d = two_sum(f + 0.5f, L);
    frac = d;
    return (d.hi > e) & (d.hi < 1.f - e);
}

template <int NC>
__global__ void __launch_bounds__(kCxBlock, 5)
    k_from_map_bl(const __grid_constant__ GatherArgs a, CxModel model, CxList left, int coord) {
    __shared__ float4 s_model[kCxWarps][kCxGroup][kCxBlWords];
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
    float *sig = a.signal + det * a.sig_stride;
    const bool vec = (reinterpret_cast<unsigned long long>(sig) & 15) == 0;
    const int ny = a.g.ny, nx = a.g.nx;
    auto over = [&](int t) {
        switch (coord) {
        case SO3G_COORD_TAN: bl_any_sample<SO3G_COORD_TAN>(a, det, t); break;
        case SO3G_COORD_ZEA: bl_any_sample<SO3G_COORD_ZEA>(a, det, t); break;
        default: bl_any_sample<SO3G_COORD_SIN>(a, det, t); break;
        }
    };
    const int j0 = t0 / kCxLen, j1 = (t1 - 1) / kCxLen + 1;
    const int step = cx_step(j1 - j0);
    for (int g = j0 + warp * step; g < j1; g += kCxWarps * step) {
        const int nch = min(step, j1 - g);
        if (lane < nch)
            cx_setup<CX_ZEN, false, NC, true>(a, model.bore, coord, g + lane, a.segs.n_time, qd, Pr,
                                              s_model[warp][lane]);
        __syncwarp();
        const int rounds = (nch + 1) / 2;
        for (int r = 0; r < rounds; r++) {
            const int ck = 2 * r + (lane >> 4);
            const int tq = (g + ck) * kCxLen + (lane & 15) * 4;
            const bool lane_live = ck < nch;
            const bool whole = vec && lane_live && tq + 3 < t1;
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
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (!(lane_live && tq + i < t1)) continue;
                const float k = kq + (float)i;
                const f32x2 k2 = f2_both(k);
                const float4 W0 = w[0], W1 = w[1], W2 = w[2], W9 = w[9];
                f32x2 L = f2_fma(k2, f2_fma(k2, f2_fma(k2, f2_fma(k2, cx_lo(W9), cx_hi(W1)), cx_lo(W1)),
                                            cx_hi(W2)), cx_lo(W2));
                if (w3.w != 0.f) {
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const float4 J = w[10 + c];
                        L = f2_fma(f2_fma(k2, cx_hi(J), cx_lo(J)), f2_both(res[i][c]), L);
                    }
                }
                float Sx, Sy, Lx, Ly;
                f2_get(f2_fma(k2, cx_hi(W0), cx_lo(W0)), Sx, Sy);
                f2_get(L, Lx, Ly);
                int x1, y1;
                dfl wx0, wy0;
                bool ok = bl_floor(Sx, Lx, kCxBlPix, __float_as_int(w3.x), x1, wx0) &
                          bl_floor(Sy, Ly, kCxBlPix, __float_as_int(w3.y), y1, wy0) & (W9.z >= 0.f);
                const bool on = (x1 >= -1) & (x1 < nx) & (y1 >= -1) & (y1 < ny);
                float pf[3] = {T, 0.f, 0.f};
                if constexpr (NC > 1) {
                    f32x2 S, Lp;
                    float v1, v2;
                    cx_factors(w, k2, res[i], w3.w != 0.f, S, Lp);
                    f2_get(f2_add(S, Lp), v1, v2);
                    pf[NC - 2] = v1;
                    pf[NC - 1] = v2;
                }
                if (ok && on) {
                    // Taps as fast_pixels: the weight x - x1 goes with x1.
                    const dfl one{1.f, 0.f};
                    const dfl wx[2] = {wx0, df_sub(one, wx0)}, wy[2] = {wy0, df_sub(one, wy0)};
                    float s = sv[i];
#pragma unroll
                    for (int dy = 0; dy < 2; dy++) {
                        const int yy = y1 + dy;
                        if (yy < 0 || yy >= ny) continue;
#pragma unroll
                        for (int dx = 0; dx < 2; dx++) {
                            const int xx = x1 + dx;
                            if (xx < 0 || xx >= nx) continue;
                            const float wt = df_mul(wy[dy], wx[dx]).hi;
                            const long long off = (long long)yy * nx + xx;
                            const float4 m = __ldg(a.map32 + off);
                            s = fmaf(m.x, pf[0] * wt, s);
                            if constexpr (NC > 1) s = fmaf(m.y, pf[1] * wt, s);
                            if constexpr (NC > 2) s = fmaf(m.z, pf[2] * wt, s);
                        }
                    }
                    sv[i] = s;
                }
                if (!ok) f4 |= 1u << i;
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

template <int C>
int bl_fix(const GatherArgs &a, const CxWork &w, cudaStream_t st) {
    k_from_map_bl_fix<C, 0><<<kCxFixBlocks, kBlock, 0, st>>>(a, w.left, w.exact);
    const int rc = after_launch("bilinear fallback");
    if (rc != SO3G_OK) return rc;
    k_from_map_bl_fix<C, 1><<<kCxFixBlocks, kBlock, 0, st>>>(a, w.exact, w.exact);
    return after_launch("bilinear fallback (exact)");
}

template <int NC>
int bl_run(const GatherArgs &a, const CxWork &w, int coord, dim3 grid, cudaStream_t st) {
    int rc = cx_probe<CX_ZEN, false, NC, true>(a, w, coord, grid.x, nullptr, st);
    if (rc != SO3G_OK) return rc;
    k_from_map_bl<NC><<<grid, kCxBlock, 0, st>>>(a, w.model, w.left, coord);
    rc = after_launch("bilinear from_map (chunked)");
    if (rc != SO3G_OK) return rc;
    switch (coord) {
    case SO3G_COORD_TAN: return bl_fix<SO3G_COORD_TAN>(a, w, st);
    case SO3G_COORD_ZEA: return bl_fix<SO3G_COORD_ZEA>(a, w, st);
    default: return bl_fix<SO3G_COORD_SIN>(a, w, st);
    }
}

int bl_nc(const GatherArgs &a, const CxWork &w, int coord, dim3 grid, cudaStream_t st) {
    switch (a.g.ncomp) {
    case 1: return bl_run<1>(a, w, coord, grid, st);
    case 2: return bl_run<2>(a, w, coord, grid, st);
    default: return bl_run<3>(a, w, coord, grid, st);
    }
}

}  // namespace

int chunked_bilinear_from_map(int coord, int kind, GatherArgs &args, int n_det, cudaStream_t st,
                              void **work) {
    GatherArgs a = args;
    const bool zen = coord == SO3G_COORD_TAN || coord == SO3G_COORD_ZEA || coord == SO3G_COORD_SIN;
    const long long npix = (long long)a.g.ny * a.g.nx;
    const long long n_time = a.segs.n_time, samples = n_time * n_det;
    if (a.fast != SO3G_POINTING_MIXED || !a.map32 || kind != PX_FLAT_NT_BL || !zen ||
        n_time <= kCxLen || npix <= 0 || npix >= (1LL << 31) ||
        samples < cert_chunked_min_samples())
        return 1;
    CxWork w;
    if (!cx_work(w, a.bore, (int)n_time, samples, st)) return 1;
    a.piece = cx_piece(n_det, n_time);
    a.gate = w.gate;
    const dim3 grid((unsigned)n_det, (unsigned)((n_time + a.piece - 1) / a.piece));
    const int rc = bl_nc(a, w, coord, grid, st);
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
