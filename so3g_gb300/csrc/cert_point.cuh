// cert_point.cuh -- chunked pointing for the certified mode
// (SO3G_POINTING_CERTIFIED) with nearest-neighbour pixelizors: the pointing
// of 64 consecutive samples of a detector from one polynomial model whose
// results are the float64 path's, bit for bit.
//
// The certified double-float pointing (fastpoint.cuh) costs ~900
// instructions a sample, nearly all of them in the quaternion product and
// the spin factors, and the projection kernels are bound by instruction
// issue.  Along a scan the pointing is smooth, so here it is evaluated once
// per 64-sample chunk, at the chunk's middle, and expanded about it: per
// sample a float32 cubic for each pixel coordinate and, for each spin
// factor, an exactly representable float32 part plus a float32 correction.
// Both carry a bound on their distance from the reference's float64 value;
// a sample whose pixel or whose float32 rounding of a spin factor is not
// certain goes to the per-sample certified path (and from there, if need
// be, to the float64 path), so every result is that of the exact path.
//
// The boresight of a chunk is modelled by a polynomial Q(u) (u = (t - tm) /
// 64, tm its middle sample): the quartic through five of its samples where
// that fits every sample to 1.5e-13, else (time stamps and encoders jitter)
// the quadratic through its first, middle and last sample, with the
// residual of each sample kept as a small rotation rho, q(t) = Q (1 + rho),
// in 3 x 16 bits.  A chunk with a break (the turn-around of a triangle scan) gets
// the quadratic of the break's longer side; the samples of the other are
// marked and go to the per-sample path.  (rho is the vector part of conj(q)
// (q - Q); the scalar part, a change of norm, turns nothing: it goes into the
// bilinear form's bound, and through the samples' norm into the pixel's.)
//
// With A(u) = Q(u) q_det, alpha = a + i d and beta = c + i b are polynomials
// in u, alpha = alpha_0 (1 + z_1 u + z_2 u^2 + ...), and so are, to the order
// kept, their logarithms la(u) = log(alpha / alpha_0) and lb(u).  In these
// terms (Pointer<C>::GetCoords, src/Projection.cxx:337-507)
//   CAR   lon = arg(alpha) - arg(beta),   atanh(sin lat) = ln|alpha / beta|,
//         spin factors P exp(2 i (arg(alpha) + arg(beta)))
//   zenithal   Y - i X = 2 alpha conj(beta) g(|alpha|^2),   g(n) = 1 (SIN),
//         1 / (2n - 1) (TAN), 1 / sqrt(n) (ZEA),
//         spin factors P exp(4 i arg(alpha)).
// The spin factors are expanded to u^4, their u^1 coefficient in
// double-float, the pixel coordinates to u^3; the terms left out are
// bounded by the majorant series of the logarithms and the exponential
// (cx_tail_log, cx_tail_exp; ~1e-13 on the 1 deg/s scans of the workloads).
// The latitude and the modulus of CAR's spin factors also depend on the
// quaternions' norm, which the reference does not divide out: the bounds take
// it from the chunk's samples and the detector (eta, spread).  The residual
// turns the spin factors' phase phi by grad(phi) . rho, the gradient a linear
// function of u per chunk and detector, and moves the pixel by at most
// 2 |rho| / cos(lat), which goes into the pixel's bound.
#pragma once

#include "host.h"
#include "pair32.cuh"

namespace so3g {

namespace {

constexpr int kCxLen = 64;            // samples per chunk
constexpr int kCxMid = kCxLen / 2;
constexpr int kCxGroup = 32;          // chunks of a warp's group, one per lane
constexpr int kCxBlock = 128;         // threads per block (its warps are independent)
constexpr int kCxWarps = kCxBlock / 32;
// A chunk that its quadratic misses by more than this is searched for a break.
constexpr float kCxBreak = 6e-7f;
// (detector, chunk) models that k_cx_probe looks at.
constexpr int kCxProbes = 2048;
// A call whose models would leave more than one sample in this to the
// per-sample path takes the general kernel.  Up to there the list holds them
// (200 det x 500k, TQU, to_map / from_map against the general kernel: 7 % left
// on a CAR map 0.48 / 0.39 of its time, on a HEALPix map 0.57 / 0.47; 10 %
// 0.92 / 0.78; past the list's end the main kernel handles them in place, 25 %
// of a T map 1.2 / 1.0, all 2 to 3).
constexpr unsigned kCxShare = 12;

// The first residual word of a sample its chunk's model does not cover (the
// others' are within 32001).
constexpr int kCxUncovered = -32768;

// Classes of coordinate systems the models are compiled for.
enum { CX_CAR = 0, CX_ZEN = 1 };

// The boresight model of one chunk, Q = q + u a1 + u^2 a2 + u^3 a3 + u^4 a4.
struct __align__(16) CxBore {
    float4 q_hi, q_lo, a1_hi, a1_lo;   // double-float
    float4 a2, a3, a4;
    float e;               // max |q(t) - Q|
    float eta;             // max ||q(t)|^2 - 1|
    float spread;          // max ||q(t)|^2 - |Q(0)|^2|
    float lsb;             // residuals' unit; 0: none kept (e is negligible)
    float part;            // 1: some samples are not covered (residuals kCxUncovered)
    float rho0;            // max |Re(conj(q) (q - Q))|, the residuals' part that is no turn
    float q1, qr;          // sizes at the chunk's end: |a1| / 2; |a2| / 4 + |a3| / 8 + |a4| / 16
};

// The boresight models of a call: per chunk, and the residuals per sample.
struct CxModel {
    const CxBore *bore;
    const short4 *resid;
};

// Per (detector, chunk), nine 16-byte words (an odd number: neighbouring
// chunks' slots start on different shared-memory banks):
//   0: x0 y0 x1 y1   1: x2 y2 x3 y3   2: hx hy e e   3: xb yb mid flag
//   4: f0 h0 f1 h1   5: l0 m0 l1 m1   6: a2 b2 a3 b3   7: a4 b4 g1x g1y
//   8: g0x g0y g0z g1z
// (two quantities side by side: x and y, the two spin factors, so that one
// f32x2 instruction takes both).
// With k = t - mid: x = xb + 1/2 + x0 + k (x1 + k (x2 + k x3)) (xb less the
// bits of kCxMagic); a spin factor is
// (f0 + k f1), exact in float32, plus the correction l0 + k (l1 + k (a2 + k
// (a3 + k a4))), within e, plus (flag) the residual's turn.  hx, hy: 1/2 -
// bounds (pixels; -1: not modelled).  HEALPix: x is the longitude and y
// sin(lat), with xb = yb = 0 and hx, hy their error bounds (hx < 0: not
// modelled).  g0 + k g1: the gradient of phi, per residual unit.
constexpr int kCxWords = 9;
// The bilinear form (TAN, ZEA, SIN; thirteen words) holds the pixel
// coordinates as the spin factors are, exact part plus correction, and their
// gradients per residual unit:
//   0: fx0 fy0 fx1 fy1   1: x2 y2 x3 y3   2: lx0 ly0 lx1 ly1   3: xb yb mid flag
//   4 .. 8: as above   9: x4 y4 e e   10, 11, 12: jx0 jy0 jx1 jy1 for the
//   residual's components x, y, z (each g0 + k g1)
// with the unmodelled chunks' e = -1 (pixel bound kCxBlPix).
constexpr int kCxBlWords = 13;
// Bilinear weights need the fraction of a pixel to float32 accuracy: a chunk
// whose pixel coordinates are not within this of the reference's goes to the
// per-sample path (the bound is several times the error; a float32 weight is
// good to 3e-8).
constexpr float kCxBlPix = 2.5e-7f;
// 1.5 x 2^23: x + kCxMagic is x rounded to the nearest integer (|x| < 2^21),
// its low bits that integer -- one addition instead of a floor and a
// conversion on the slow conversion pipe.
constexpr float kCxMagic = 12582912.f;
constexpr int kCxMagicBits = 0x4b400000;

// Counters of a call: entries of the two lists, k_cx_probe's votes.
constexpr int kCxCounts = 4;

// Middle sample of chunk j (samples [64 j, 64 j + 64)); the last chunk's is
// moved back so that its model's samples mid - 32 .. mid + 32 exist.
__device__ __forceinline__ int cx_mid(int j, int n_time) {
    return min(j * kCxLen, n_time - 1 - kCxLen) + kCxMid;
}

// The chunks' boresight models and residuals, 16 threads per chunk (one per
// quaternion component and quarter of its samples), in double-float
// arithmetic (the float64 pipe would take ~0.1 ms per million samples).
__global__ void __launch_bounds__(128) k_cx_bore(const double *bore, int n_time, int n_chunks,
                                                 CxBore *out, short4 *resid,
                                                 unsigned long long *counts) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kCxCounts) counts[i] = 0;   // (of the kernels that follow)
    const int chunk = i >> 4, j = min(chunk, n_chunks - 1), comp = i & 3, part = (i >> 2) & 3;
    const int base = cx_mid(j, n_time) - kCxMid;
    const double *b = bore + 4LL * base + comp;
    bool bad = false;   // a value df_split does not take (or NaN, infinity)
    dfl q[5];
#pragma unroll
    for (int k = 0; k < 5; k++) bad |= !df_split(__ldg(b + kCxLen * k), q[k]);
    // Central differences about the middle, odd and even.
    const dfl o1 = df_sub(q[3], q[1]), o2 = df_sub(q[4], q[0]);
    const dfl two2 = df_mulf(q[2], 2.f);
    const dfl e1 = df_sub(df_add(q[1], q[3]), two2), e2 = df_sub(df_add(q[0], q[4]), two2);
    // Quartic, samples h = 1/4 apart: a1 = (8 o1 - o2) / (12 h), a2 = (16 e1 -
    // e2) / (24 h^2), a3 = (o2 - 2 o1) / (12 h^3), a4 = (e2 - 4 e1) / (24 h^4).
    const dfl third{0.33333334f, -9.934108e-09f};
    const dfl a1 = df_mul(df_sub(df_mulf(o1, 8.f), o2), third);
    const dfl a2 = df_mul(df_mulf(df_sub(df_mulf(e1, 16.f), e2), 2.f), third);
    const float a3 = df_sub(o2, df_mulf(o1, 2.f)).hi * (16.f / 3.f);
    const float a4 = df_sub(e2, df_mulf(e1, 4.f)).hi * (32.f / 3.f);
    // Quadratic through the first, middle and last sample.
    const dfl b1 = o2, b2 = df_mulf(e2, 2.f);
    const int k0 = j * kCxLen - base;                        // first own sample
    const int k1 = min(kCxLen - 1 + k0, n_time - 1 - base);  // last own sample
    // |q|^2 - 1 of one sample, from the four components' lanes.
    auto norm1 = [](const dfl &v) {
        dfl s = df_mul(v, v);
        s = df_add(s, dfl{__shfl_xor_sync(kFull, s.hi, 1), __shfl_xor_sync(kFull, s.lo, 1)});
        s = df_add(s, dfl{__shfl_xor_sync(kFull, s.hi, 2), __shfl_xor_sync(kFull, s.lo, 2)});
        return df_sub(s, dfl{1.f, 0.f}).hi;
    };
    float r4 = 0.f, r2 = 0.f;
    float top_n = norm1(q[2]), low_n = top_n;   // largest and smallest |q|^2 - 1
    for (int n = 0; n < kCxLen / 4; n++) {   // (the same count in every lane)
        const int k = min(k0 + part * (kCxLen / 4) + n, k1);
        dfl v;
        bad |= !df_split(__ldg(b + 4 * k), v);
        const float u = (float)(k - kCxMid) * (1.f / kCxLen);
        const dfl d = df_sub(v, q[2]);
        const dfl p4 =
            df_mulf(df_add(a1, df_mulf(df_add(a2, dfl{u * fmaf(u, a4, a3), 0.f}), u)), u);
        const dfl p2 = df_mulf(df_add(b1, df_mulf(b2, u)), u);
        r4 = fmaxf(r4, fabsf(df_sub(d, p4).hi));   // (fmaxf drops NaN: only a bad
        r2 = fmaxf(r2, fabsf(df_sub(d, p2).hi));   // value makes one)
        const float n1 = norm1(v);
        top_n = fmaxf(top_n, n1);
        low_n = fminf(low_n, n1);
    }
    bad = __any_sync(kFull, bad);   // (the warp's other chunk as well)
    auto max_parts = [](float x) {
        x = fmaxf(x, __shfl_xor_sync(kFull, x, 4));
        return fmaxf(x, __shfl_xor_sync(kFull, x, 8));
    };
    auto sum4 = [](float x) {
        x += __shfl_xor_sync(kFull, x, 1);
        return x + __shfl_xor_sync(kFull, x, 2);
    };
    r4 = max_parts(r4);
    r2 = max_parts(r2);
    top_n = max_parts(top_n);
    low_n = -max_parts(-low_n);
    float eta = fmaxf(fabsf(top_n), fabsf(low_n)), spread = top_n - low_n;
    // 1e-13: the double-float roundings.
    const float E4 = sqrtf(sum4(r4 * r4)) * 1.00001f + 1e-13f;
    float E2 = sqrtf(sum4(r2 * r2)) * 1.00001f + 1e-13f;
    const bool quad = !(E4 < 2.5e-13f);
    // A chunk that holds a break (a turn-around): its largest second
    // difference is there, and the longer side of it gets a quadratic of its
    // own (through its ends and middle, written about the chunk's middle): a
    // turn-around every 20 s had sent 1.6 % of a scan's samples to the
    // per-sample path, 0.78 ms of 1000 det x 1M samples; now 0.35 ms.
    dfl q0 = q[2], p1 = b1, p2 = b2;
    int c0 = k0, c1 = k1;   // samples covered
    const bool broken = quad && !bad && !(E2 < kCxBreak);
    if (__any_sync(kFull, broken)) {
        int top = 0;   // magnitude (float bits), its low bits the sample
        for (int n = 0; n < kCxLen / 4; n++) {
            const int k = min(max(k0 + part * (kCxLen / 4) + n, 1), min(k1, kCxLen - 1));
            const float d = (float)((__ldg(b + 4 * (k + 1)) - __ldg(b + 4 * k)) -
                                    (__ldg(b + 4 * k) - __ldg(b + 4 * (k - 1))));
            top = max(top, (__float_as_int(fabsf(d)) & ~127) | k);
        }
#pragma unroll
        for (int m = 1; m < 16; m <<= 1) top = max(top, __shfl_xor_sync(kFull, top, m));
        const int s = top & 127;
        int A = s + 1, B = k1;
        if (s - 1 - k0 > k1 - s - 1) {
            A = k0;
            B = s - 1;
        }
        if ((B - A) & 1) {   // (an even length, without the sample at the break)
            if (A == k0) B--;
            else A++;
        }
        const bool fit = broken && B - A >= 16;
        const int M = fit ? (A + B) >> 1 : kCxMid, H = fit ? (B - A) >> 1 : kCxMid;
        dfl x[3];
#pragma unroll
        for (int k = 0; k < 3; k++) df_split(__ldg(b + 4 * (M + (k - 1) * H)), x[k]);
        const float al = (float)kCxLen / (float)H, de = (float)(kCxMid - M) / (float)H;
        const dfl o = df_mulf(df_sub(x[2], x[0]), 0.5f);
        const dfl e = df_mulf(df_sub(df_add(x[0], x[2]), df_mulf(x[1], 2.f)), 0.5f);
        dfl w0 = df_add(x[1], df_mulf(df_add(o, df_mulf(e, de)), de));
        dfl w1 = df_mulf(df_add(o, df_mulf(e, 2.f * de)), al);
        dfl w2 = df_mulf(df_mulf(e, al), al);
        // To norm 1 (within off^2) at the chunk's middle, which may lie outside
        // the side.
        dfl nn = df_mul(w0, w0);
        nn = df_add(nn, dfl{__shfl_xor_sync(kFull, nn.hi, 1), __shfl_xor_sync(kFull, nn.lo, 1)});
        nn = df_add(nn, dfl{__shfl_xor_sync(kFull, nn.hi, 2), __shfl_xor_sync(kFull, nn.lo, 2)});
        const float off = df_sub(nn, dfl{1.f, 0.f}).hi, sc = -0.5f * off;
        w0 = df_add(w0, df_mulf(w0, sc));
        w1 = df_add(w1, df_mulf(w1, sc));
        w2 = df_add(w2, df_mulf(w2, sc));
        float r = 0.f;
        for (int n = 0; n < kCxLen / 4; n++) {
            const int k = fit ? min(max(k0 + part * (kCxLen / 4) + n, A), B) : kCxMid;
            dfl v;
            df_split(__ldg(b + 4 * k), v);
            const float u = (float)(k - kCxMid) * (1.f / kCxLen);
            r = fmaxf(r, fabsf(df_sub(df_sub(v, w0), df_mulf(df_add(w1, df_mulf(w2, u)), u)).hi));
        }
        r = max_parts(r);
        r = sqrtf(sum4(r * r)) * 1.00001f + 1e-13f;
        // (Noise without a break does not fit any side much better.)
        if (fit && fabsf(off) < 1e-5f && r < 0.1f * E2) {
            E2 = r;
            eta = fmaxf(eta, off * off + 1e-13f);
            spread = eta + off * off;
            q0 = w0;
            p1 = w1;
            p2 = w2;
            c0 = A;
            c1 = B;
        }
    }
    const float lsb = quad && !bad ? E2 * (1.f / 32000.f) : 0.f;
    const float b1_ = quad ? p1.hi : a1.hi, b2_ = quad ? p2.hi : a2.hi;
    const float n1 = sqrtf(sum4(b1_ * b1_)), n2 = sqrtf(sum4(b2_ * b2_)),
                n3 = sqrtf(sum4(a3 * a3)), n4 = sqrtf(sum4(a4 * a4));
    if (chunk < n_chunks && part == 0) {
        float *o = reinterpret_cast<float *>(out + j);
        o[comp] = q0.hi;
        o[4 + comp] = q0.lo;
        o[8 + comp] = b1_;
        o[12 + comp] = quad ? p1.lo : a1.lo;
        o[16 + comp] = b2_;
        o[20 + comp] = quad ? 0.f : a3;
        o[24 + comp] = quad ? 0.f : a4;
        if (comp == 0) {
            out[j].e = bad ? 1.f : (quad ? E2 : E4);
            out[j].eta = bad ? 1.f : eta * 1.00001f + 1e-14f;
            out[j].spread = bad ? 1.f : spread * 1.00001f + 1e-14f;
            out[j].lsb = lsb;
            if (!(lsb > 0.f)) out[j].rho0 = out[j].e;
            // (1.001: the detector quaternions' norm.)
            out[j].q1 = 1.001f * 0.5f * n1;
            out[j].qr = 1.001f * (0.25f * n2 + (quad ? 0.f : 0.125f * n3 + 0.0625f * n4));
            out[j].part = c0 > k0 || c1 < k1 ? 1.f : 0.f;
        }
    }
    // Residuals: rho = conj(Q) (q - Q), in units of lsb.
    if (!__any_sync(kFull, lsb > 0.f)) return;
    const float inv = lsb > 0.f ? 1.f / lsb : 0.f;
    const int lane0 = threadIdx.x & 28;
    float rho0 = 0.f;   // in units of lsb
    for (int n = 0; n < kCxLen / 4; n++) {
        const int k = k0 + part * (kCxLen / 4) + n, kc = min(k, k1);
        dfl v;
        df_split(__ldg(b + 4 * kc), v);
        const float u = (float)(kc - kCxMid) * (1.f / kCxLen);
        const dfl p = df_mulf(df_add(p1, df_mulf(p2, u)), u);
        const float r = df_sub(df_sub(v, q0), p).hi * inv, g = v.hi;
        float rr[4], qq[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            rr[c] = __shfl_sync(kFull, r, lane0 + c);
            qq[c] = __shfl_sync(kFull, g, lane0 + c);
        }
        if (kc >= c0 && kc <= c1)
            rho0 = fmaxf(rho0, fabsf(qq[0] * rr[0] + qq[1] * rr[1] + qq[2] * rr[2] +
                                     qq[3] * rr[3]));
        if (comp == (k & 3) && k <= k1 && chunk < n_chunks && inv > 0.f) {
            const float x = qq[0] * rr[1] - qq[1] * rr[0] - qq[2] * rr[3] + qq[3] * rr[2];
            const float y = qq[0] * rr[2] + qq[1] * rr[3] - qq[2] * rr[0] - qq[3] * rr[1];
            const float z = qq[0] * rr[3] - qq[1] * rr[2] + qq[2] * rr[1] - qq[3] * rr[0];
            resid[base + k] = k < c0 || k > c1
                                  ? make_short4((short)kCxUncovered, 0, 0, 0)
                                  : make_short4((short)__float2int_rn(x), (short)__float2int_rn(y),
                                                (short)__float2int_rn(z), 0);
        }
    }
    rho0 = max_parts(rho0);
    // (0.1 lsb: the sums' float32 roundings, 8u of 32000.)
    if (chunk < n_chunks && part == 0 && comp == 0 && lsb > 0.f)
        out[j].rho0 = (rho0 + 0.1f) * lsb;
}

// Complex float32.
struct cf {
    float r, i;
};
__device__ __forceinline__ cf operator+(cf a, cf b) { return cf{a.r + b.r, a.i + b.i}; }
__device__ __forceinline__ cf operator-(cf a, cf b) { return cf{a.r - b.r, a.i - b.i}; }
__device__ __forceinline__ cf operator*(float s, cf a) { return cf{s * a.r, s * a.i}; }
__device__ __forceinline__ cf operator*(cf a, cf b) {
    return cf{fmaf(a.r, b.r, -a.i * b.i), fmaf(a.r, b.i, a.i * b.r)};
}
__device__ __forceinline__ float cf_abs(cf a) {
    const float n = fmaf(a.r, a.r, a.i * a.i);
    return n > 1e-36f ? 1.000001f * n * rsqrtf(n) : 1e-18f;
}

__device__ __forceinline__ void cx_qmul(const float4 &p, const float (&q)[4], float (&r)[4]) {
    r[0] = p.x * q[0] - p.y * q[1] - p.z * q[2] - p.w * q[3];
    r[1] = p.x * q[1] + p.y * q[0] + p.z * q[3] - p.w * q[2];
    r[2] = p.x * q[2] - p.y * q[3] + p.z * q[0] + p.w * q[1];
    r[3] = p.x * q[3] + p.y * q[2] - p.z * q[1] + p.w * q[0];
}

// log(1 + z1 u + z2 u^2 + z3 u^3 + z4 u^4) to u^4.
struct CxLog {
    cf l1, l2, l3, l4;
};
__device__ __forceinline__ CxLog cx_log(cf z1, cf z2, cf z3, cf z4) {
    const cf s = z1 * z1;
    CxLog o;
    o.l1 = z1;
    o.l2 = z2 - 0.5f * s;
    o.l3 = z3 - z1 * z2 + (1.f / 3.f) * (s * z1);
    o.l4 = z4 - z1 * z3 - 0.5f * (z2 * z2) + s * z2 - 0.25f * (s * s);
    return o;
}

// For nonnegative c1..c4 (a polynomial's coefficients at the chunk's end),
// the terms of order >= 5 of X^2, X^3 and X^4, X = c1 t + ... + c4 t^4 at t =
// 1 (bounds: the differences' float32 cancellation is in the 1e-15).
struct CxTail {
    float t2, t3, t4, X;
};
__device__ __forceinline__ CxTail cx_tail(float c1, float c2, float c3, float c4) {
    CxTail o;
    const float X = c1 + c2 + c3 + c4, r = c2 + c3 + c4;
    o.X = X;
    o.t2 = 2.f * (c1 * c4 + c2 * (c3 + c4) + c3 * c4) + c3 * c3 + c4 * c4;
    // X^3 - c1^3 - 3 c1^2 c2 and X^4 - c1^4, with X = c1 + r.
    o.t3 = 3.f * c1 * c1 * (c3 + c4) + 3.f * c1 * r * r + r * r * r;
    o.t4 = r * (4.f * c1 * c1 * c1 + r * (6.f * c1 * c1 + r * (4.f * c1 + r)));
    return o;
}
// Terms of order >= 5 left out of the logarithm of 1 + X (n-th power / n).
__device__ __forceinline__ float cx_tail_log(const CxTail &t) {
    const float x2 = t.X * t.X;
    return 0.5f * t.t2 + (1.f / 3.f) * t.t3 + 0.25f * t.t4 + 0.25f * x2 * x2 * t.X;
}
// ... and of the exponential of X (n-th power / n!).
__device__ __forceinline__ float cx_tail_exp(const CxTail &t) {
    const float x2 = t.X * t.X;
    return 0.5f * t.t2 + (1.f / 6.f) * t.t3 + (1.f / 24.f) * t.t4 + (1.f / 100.f) * x2 * x2 * t.X;
}

// Size of the terms of order >= m of a zenithal projection's factor e(u)
// (cx_setup), m = 5 (BL) or 4, at the chunk's end, from the sizes a1 .. a4 of
// alpha's relative coefficients.  Nothing is taken to fall off from one order
// to the next: a scan may accelerate (a2 against a1^2), and the quartic of a
// short last chunk carries noise in every order.
// SIN: e = alpha / alpha_0.  ZEA: exp(i theta), m1 .. m4 theta's sizes.
// TAN: alpha / alpha_0 times G = 1 / (1 + x), x = f (|alpha / alpha_0|^2 - 1).
template <bool BL>
__device__ __forceinline__ float cx_rest_zea(float m1, float m2, float m3, float m4, float tail) {
    const float r5 = cx_tail_exp(cx_tail(m1, m2, m3, m4)) + 1.1f * tail;
    if (BL) return r5;
    return r5 + m4 + m1 * m3 + 0.5f * m2 * m2 + 0.5f * m1 * m1 * m2 +
           (1.f / 24.f) * m1 * m1 * m1 * m1;
}
template <bool BL>
__device__ __forceinline__ float cx_rest_tan(float f, float a1, float a2, float a3, float a4) {
    const float y1 = 2.f * f * a1, y2 = f * (2.f * a2 + a1 * a1), y3 = 2.f * f * (a3 + a1 * a2),
                y4 = f * (2.f * a4 + 2.f * a1 * a3 + a2 * a2);
    const float y5 = 2.f * f * (a4 * (a1 + a2 + a3) + a2 * a3) + f * (a3 * a3 + a4 * a4);
    const CxTail t = cx_tail(y1, y2, y3, y4);
    const float Y = t.X + y5, Y2 = Y * Y;
    const float g1 = y1, g2 = y2 + y1 * y1, g3 = y3 + 2.f * y1 * y2 + y1 * y1 * y1,
                g4 = y4 + 2.f * y1 * y3 + y2 * y2 + 3.f * y1 * y1 * y2 + y1 * y1 * y1 * y1;
    const float g5 = y5 * (1.f + 3.f * Y) + t.t2 + t.t3 + t.t4 + 1.3f * Y2 * Y2 * Y;
    const float r5 = g5 * (1.f + a1 + a2 + a3 + a4) + a4 * (g1 + g2 + g3 + g4) +
                     a3 * (g2 + g3 + g4) + a2 * (g3 + g4) + a1 * g4;
    if (BL) return r5;
    return r5 + a4 + a3 * g1 + a2 * g2 + a1 * g3 + g4;
}

// Gradient of phi with respect to a rotation rho of the boresight (q (1 +
// rho) q_det), at A = q q_det.  In the detector's frame (rho' = conj(q_det)
// rho q_det = (x, y, z)): d log(alpha) = i z - (y + i x) conj(beta) / alpha,
// d log(beta) = i z + (y + i x) conj(alpha) / beta, so dphi = 4 z + 2 Im((y
// + i x) kappa), kappa = (|alpha|^2 - |beta|^2) / (alpha beta) (CAR) or -2
// conj(beta) / alpha (zenithal).  Returns |kappa|.
template <int CL>
__device__ __forceinline__ float cx_gradient(const float (&A)[4], const float (&d)[4],
                                             float (&g)[3]) {
    const cf al{A[0], A[3]}, be{A[2], A[1]};
    cf k;
    if (CL == CX_CAR) {
        const cf v = al * be;
        const float z = (al.r * al.r + al.i * al.i) - (be.r * be.r + be.i * be.i);
        const float f = z * rcp_approx(v.r * v.r + v.i * v.i);
        k = cf{v.r * f, -v.i * f};
    } else {
        const cf v = al * be;
        const float f = -2.f * rcp_approx(al.r * al.r + al.i * al.i);
        k = cf{v.r * f, -v.i * f};
    }
    // To the boresight's frame: q_det g' conj(q_det).
    const float x = 2.f * k.r, y = 2.f * k.i, z = 4.f;
    const float tx = 2.f * (d[2] * z - d[3] * y), ty = 2.f * (d[3] * x - d[1] * z),
                tz = 2.f * (d[1] * y - d[2] * x);
    g[0] = x + d[0] * tx + d[2] * tz - d[3] * ty;
    g[1] = y + d[0] * ty + d[3] * tx - d[1] * tz;
    g[2] = z + d[0] * tz + d[1] * ty - d[2] * tx;
    return cf_abs(k);
}

// Gradient of the zenithal pixel coordinates (X, Y) with respect to rho, at A
// = q q_det, per unit of rotation: with W = alpha conj(beta) = (Y - i X) / G,
// G = g(n) 2, rho' = (x, y, z): dW = (y - i x) alpha^2 - (y + i x)
// conj(beta)^2, dn = -2 Re((y + i x) conj(alpha beta)).
__device__ __forceinline__ void cx_pixel_gradient(int coord, const float (&A)[4],
                                                  const float (&d)[4], float (&gx)[3],
                                                  float (&gy)[3]) {
    const cf al{A[0], A[3]}, be{A[2], A[1]}, bc{A[2], -A[1]};
    const cf a2 = al * al, b2 = bc * bc, v = al * be, W = al * bc;
    const float n = al.r * al.r + al.i * al.i;
    float G = 2.f, dG = 0.f;   // dG / dn
    if (coord == SO3G_COORD_TAN) {
        const float r = rcp_approx(2.f * n - 1.f);
        G = 2.f * r;
        dG = -4.f * r * r;
    } else if (coord == SO3G_COORD_ZEA) {
        const float r = rsqrtf(n);
        G = 2.f * r;
        dG = -r * r * r;
    }
    // y: dW = a2 - b2, dn = -2 Re v;  x: dW = -i (a2 + b2), dn = -2 Im v.
    const cf jy = G * (a2 - b2) + (-2.f * v.r * dG) * W;
    const cf sp = a2 + b2;
    const cf jx = G * cf{sp.i, -sp.r} + (-2.f * v.i * dG) * W;
    // (d(Y - i X): Y the real part, X minus the imaginary one); components
    // along x and y of the detector's frame, turned to the boresight's.
    const float in[2][2] = {{-jx.i, -jy.i}, {jx.r, jy.r}};
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const float x = in[c][0], y = in[c][1];
        const float tx = -2.f * d[3] * y, ty = 2.f * d[3] * x, tz = 2.f * (d[1] * y - d[2] * x);
        float(&g)[3] = c == 0 ? gx : gy;
        g[0] = x + d[0] * tx + d[2] * tz - d[3] * ty;
        g[1] = y + d[0] * ty + d[3] * tx - d[1] * tz;
        g[2] = d[0] * tz + d[1] * ty - d[2] * tx;
    }
}

// The model of chunk j for a detector (double-float qd), into w (kCxWords
// words; BL: the bilinear form, kCxBlWords).
template <int CL, bool HP, int NC, bool BL = false, class Args>
__device__ __forceinline__ void cx_setup(const Args &a, const CxBore *cxb, int coord, int j,
                                         int n_time, const dfl (&qd)[4], float Pr, float4 *w) {
    constexpr bool SPIN = NC > 1;
    constexpr float u = kU;
    const int mid = cx_mid(j, n_time);
    if (BL) w[9] = make_float4(0.f, 0.f, -1.f, -1.f);
    w[2] = make_float4(-1.f, -1.f, 0.f, 0.f);
    w[3] = make_float4(0.f, 0.f, __int_as_float(mid), 0.f);
    const CxBore &cb = cxb[j];
    const float E = __ldg(&cb.e), lsb = __ldg(&cb.lsb);
    // The norm of q(t) q_det: its distance from 1.
    auto norm_off = [&]() {
        const dfl qq = df_dot<4>(qd, qd);
        return __ldg(&cb.eta) + fabsf((qq.hi - 1.f) + qq.lo);
    };
    // (A side's norm may be off by E, which the bilinear form does not cover.)
    const bool covered = __ldg(&cb.part) == 0.f;
    if (!(E < 1e-6f) || (BL && !covered)) return;
    // The middle sample: its coordinates X0, Y0 (HEALPix: longitude and
    // sin(lat)) and spin quantities, certified double-float.
    dfl qa, qb, qc, qe, X0, Y0, Nc, Ns, D;
    {
        const float4 h = __ldg(&cb.q_hi), l = __ldg(&cb.q_lo);
        const dfl q[4] = {{h.x, l.x}, {h.y, l.y}, {h.z, l.z}, {h.w, l.w}};
        df_qmul(q, qd, qa, qb, qc, qe);
    }
    if constexpr (HP) {
        Y0 = df_dot<4>({qa, qb, qc, qe}, {qa, df_neg(qb), df_neg(qc), qe});
        if (!(fabsf(Y0.hi) < 0.99f) ||
            !fast_lon_spin(a.ft, a.fc, qa, qb, qc, qe, Y0, X0, Nc, Ns, D))
            return;
    } else if constexpr (CL == CX_CAR) {
        if (!fast_car(a.ft, a.fc, qa, qb, qc, qe, X0, Y0, Nc, Ns, D)) return;
    } else {
        dfl n, p, v;
        fast_zen_nuv(qa, qb, qc, qe, n, p, v);
        bool ok;
        if (coord == SO3G_COORD_TAN)
            ok = fast_zen_xy<SO3G_COORD_TAN>(a.ft, a.fc, qb, qc, n, p, v, X0, Y0);
        else if (coord == SO3G_COORD_ZEA)
            ok = fast_zen_xy<SO3G_COORD_ZEA>(a.ft, a.fc, qb, qc, n, p, v, X0, Y0);
        else
            ok = fast_zen_xy<SO3G_COORD_SIN>(a.ft, a.fc, qb, qc, n, p, v, X0, Y0);
        if (!ok) return;
        fast_zen_spin(qa, qe, n, Nc, Ns, D);
    }
    // The float32 polynomials of alpha and beta.
    const float d32[4] = {qd[0].hi, qd[1].hi, qd[2].hi, qd[3].hi};
    const float A[4] = {qa.hi, qb.hi, qc.hi, qe.hi};
    float A1[4], A2[4], A3[4], A4[4];
    dfl B1[4];   // BL: A1 in double-float
    if constexpr (BL) {
        const float4 h = __ldg(&cb.a1_hi), l = __ldg(&cb.a1_lo);
        const dfl q[4] = {{h.x, l.x}, {h.y, l.y}, {h.z, l.z}, {h.w, l.w}};
        df_qmul(q, qd, B1[0], B1[1], B1[2], B1[3]);
#pragma unroll
        for (int c = 0; c < 4; c++) A1[c] = B1[c].hi;
    } else {
        cx_qmul(__ldg(&cb.a1_hi), d32, A1);
    }
    cx_qmul(__ldg(&cb.a2), d32, A2);
    cx_qmul(__ldg(&cb.a3), d32, A3);
    cx_qmul(__ldg(&cb.a4), d32, A4);
    // Their sizes at the chunk's end: the coefficients' float32 errors go with
    // the quaternions', not with alpha's or beta's (6u each: the operands' roundings
    // and the product's).
    const float Q1 = __ldg(&cb.q1), Qr = __ldg(&cb.qr);
    const float al2 = A[0] * A[0] + A[3] * A[3], be2 = A[1] * A[1] + A[2] * A[2];
    const float nq2 = d32[0] * d32[0] + d32[1] * d32[1] + d32[2] * d32[2] + d32[3] * d32[3];
    if (!(fabsf(al2 + be2 - 1.f) < 1e-3f && fabsf(nq2 - 1.f) < 1e-3f && al2 > 0.004f)) return;
    const float ia = rcp_approx(al2);
    const cf inv_a{A[0] * ia, -A[3] * ia};
    const CxLog la = cx_log(cf{A1[0], A1[3]} * inv_a, cf{A2[0], A2[3]} * inv_a,
                            cf{A3[0], A3[3]} * inv_a, cf{A4[0], A4[3]} * inv_a);
    // |z_n| / 2^n: sizes at the chunk's end.
    const float ra = rsqrtf(al2) * 1.0001f;
    const CxTail ta = cx_tail(0.5f * ra * cf_abs(cf{A1[0], A1[3]}), 0.25f * ra * cf_abs(cf{A2[0], A2[3]}),
                              0.125f * ra * cf_abs(cf{A3[0], A3[3]}),
                              0.0625f * ra * cf_abs(cf{A4[0], A4[3]}));
    if (!(ta.X < 0.05f)) return;
    float tail = cx_tail_log(ta);    // logarithms' terms of order >= 5
    float phi1, phi2, phi3, phi4;    // phase of the spin factors
    float cx1, cx2, cx3, cy1, cy2, cy3;   // X, Y: cubic in u
    float tx, ty;                    // their terms of order >= 4
    float rx, ry;                    // X, Y per unit of residual
    float lutx = 0.f, luty = 0.f;    // the tables' errors at both ends
    float zz;                        // |z1|^2 of alpha and beta
    float gerr;                      // gradient of phi: error of its linear form
    float es;                        // spin factors (relative): change of the modulus over the
                                     // chunk, float32 errors of phi2 .. phi4
    float big;                       // size of the terms that X, Y's coefficients are sums of
    float curv = 0.f;                // BL: curvature of the pixel's gradient
    float sx2 = 0.f;                 // BL: terms of X, Y's coefficients of order >= 2
    cf x4{0.f, 0.f};                 // BL: the u^4 coefficient of Y - i X,
    float xs = 2.f;                  // and X, Y's change with the norm of q (relative)
    if constexpr (CL == CX_CAR) {
        if (!(be2 > 0.004f)) return;
        const float ib = rcp_approx(be2);
        const cf inv_b{A[2] * ib, -A[1] * ib};
        const CxLog lb = cx_log(cf{A1[2], A1[1]} * inv_b, cf{A2[2], A2[1]} * inv_b,
                                cf{A3[2], A3[1]} * inv_b, cf{A4[2], A4[1]} * inv_b);
        const float rb = rsqrtf(be2) * 1.0001f;
        const CxTail tb =
            cx_tail(0.5f * rb * cf_abs(cf{A1[2], A1[1]}), 0.25f * rb * cf_abs(cf{A2[2], A2[1]}),
                    0.125f * rb * cf_abs(cf{A3[2], A3[1]}), 0.0625f * rb * cf_abs(cf{A4[2], A4[1]}));
        if (!(tb.X < 0.05f)) return;
        tail += cx_tail_log(tb);
        phi1 = 2.f * (la.l1.i + lb.l1.i);
        phi2 = 2.f * (la.l2.i + lb.l2.i);
        phi3 = 2.f * (la.l3.i + lb.l3.i);
        phi4 = 2.f * (la.l4.i + lb.l4.i);
        zz = 4.f * (ta.X * ta.X + tb.X * tb.X);
        // 2 x 9u of each of la's and lb's (6u, and 3u of the division).
        es = 18.f * u * Qr * (ra + rb);
        big = 0.3f * (Q1 + Qr) * (ra + rb);   // (9u of Q1 + Qr)
        cx1 = la.l1.i - lb.l1.i;
        cx2 = la.l2.i - lb.l2.i;
        cx3 = la.l3.i - lb.l3.i;
        tx = 0.0625f * fabsf(la.l4.i - lb.l4.i) + tail;
        // Latitude from m = ln|alpha / beta| - its value at the middle: with
        // S, C = sin, cos of the latitude, dlat/dm = C, dS/dm = C^2.
        const float m1 = la.l1.r - lb.l1.r, m2 = la.l2.r - lb.l2.r, m3 = la.l3.r - lb.l3.r;
        const float S = al2 - be2, C2 = 4.f * al2 * be2, C = C2 * rsqrtf(C2);
        const float mu1 = 0.5f * fabsf(m1), mu2 = 0.25f * fabsf(m2), mu3 = 0.125f * fabsf(m3),
                    mu4 = 0.0625f * fabsf(la.l4.r - lb.l4.r) + tail;
        const float mu = mu1 + mu2 + mu3 + mu4;
        // kappa = S / v, |v| = C / 2: |kappa''| / 8 with |(1/v)'| <= |z1a| +
        // |z1b|, |(1/v)''| <= (...)^2 + 2 |l2a + l2b|, |S'| <= C^2 |m1|, |S''| <=
        // 2 C^2 (m1^2 + |m2|).
        const float zs1 = 2.f * (ta.X + tb.X);
        gerr = fabsf(S) * rsqrtf(C2) * (0.3f * zs1 * zs1 + 0.75f * cf_abs(la.l2 + lb.l2)) +
               C * fabsf(m1) * (0.6f * zs1 + 0.6f * fabsf(m1)) + 0.6f * C * fabsf(m2);
        // Order >= 4: m's own, those of m^2 / 2 and m^3 / 6 (derivatives at
        // most 2 and 4), and the fourth derivative's (at most 10).
        ty = mu4 + (2.f * mu1 * (mu3 + mu4) + (mu2 + mu3 + mu4) * (mu2 + mu3 + mu4)) +
             2.f * (mu * mu * mu - mu1 * mu1 * mu1) + 0.5f * mu * mu * mu * mu + 1e-12f;
        if constexpr (HP) {
            cy1 = C2 * m1;
            cy2 = C2 * (m2 - S * m1 * m1);
            cy3 = C2 * (m3 - 2.f * S * m1 * m2 - (C2 - 2.f * S * S) * (1.f / 3.f) * m1 * m1 * m1);
        } else {
            cy1 = C * m1;
            cy2 = C * (m2 - 0.5f * S * m1 * m1);
            cy3 = C * (m3 - S * m1 * m2 + (S * S - C2) * (1.f / 6.f) * m1 * m1 * m1);
        }
        rx = 1.05f * ra * rb;
        ry = 2.2f;
        // h^2/8 max|f''| of the tables: ATAN2 3.0e-10, ASIN 4.66e-10 S (1 -
        // S^2)^-3/2 (at an S beyond the chunk's); the middle's and the sample's.
        const float zs = fminf(fabsf(S) + 1.1f * C * mu, 0.9985f);
        const float rs = rsqrtf(1.f - zs * zs);
        lutx = 2.f * 3.1e-10f;
        luty = (HP ? 1.f : 2.f) * 4.7e-10f * zs * rs * rs * rs;
        // The norm N = |alpha|^2 + |beta|^2: the reference's sin(lat) is N
        // tanh(ln|alpha / beta|), so a sample's N off the middle's (by up to
        // spread) moves it by spread |tanh|, and the coefficients above, which
        // take C^2 for 1 - S^2 (it is N^2 - S^2) and N for 1, are off by up to 5
        // eta / (1 - S^2) of their terms (eta <= 1e-3 here, 1 - S^2 > 0.016).  (A
        // residual moves ln|alpha / beta| by 2 E / C.)
        const float eta = norm_off(), spread = 1.01f * __ldg(&cb.spread);
        const float ms = mu + 2.2f * E * rs;
        ty += (1.1f * spread * zs + 5.f * eta * ms) * (HP ? 1.f : rs);
        // The spin factors' modulus is (N^2 - S^2) / (1 - S^2), not 1.
        es += 1.1f * rs * rs * (2.2f * spread + 5.f * eta * zs * ms);
        // The longitude stays inside (-pi, pi) over the chunk (a HEALPix pixel
        // takes it modulo 2 pi).
        if (!HP && !(fabsf(X0.hi) + 1.05f * (ta.X + tb.X) + rx * E + 1e-6f < 3.1415f)) return;
    } else {
        phi1 = 4.f * la.l1.i;
        phi2 = 4.f * la.l2.i;
        phi3 = 4.f * la.l3.i;
        phi4 = 4.f * la.l4.i;
        zz = 4.f * ta.X * ta.X;
        if (!(al2 > 0.25f)) return;
        es = 36.f * u * Qr * ra;
        big = 4.f * (ta.X + Q1 + Qr);
        // kappa = -2 conj(beta) / alpha: |kappa''| / 8.
        gerr = 0.6f * ra * (cf_abs(cf{A2[2], A2[1]}) + 2.f * ta.X * cf_abs(cf{A1[2], A1[1]}) +
                            4.f * ta.X * ta.X + cf_abs(la.l2));
        // Y - i X = 2 g(n_0) alpha_0 e(u) conj(beta), e = (alpha / alpha_0)
        // g(n) / g(n_0): SIN alpha / alpha_0, ZEA exp(i Im la), TAN (alpha /
        // alpha_0) / (1 + x), x = 2 (n - n_0) / (2 n_0 - 1), n = n_0 exp(2 Re la).
        const cf z1 = la.l1;
        const cf z2 = cf{A2[0], A2[3]} * inv_a, z3 = cf{A3[0], A3[3]} * inv_a;
        cf e1, e2, e3;
        float g = 2.f, h = 1.1f * ta.X;   // h: size of e - 1 at the chunk's end
        float ft = 0.f;                   // TAN: f
        const float s1_ = 0.5f * cf_abs(z1), s2_ = 0.25f * cf_abs(z2), s3_ = 0.125f * cf_abs(z3),
                    s4_ = 0.0625f * cf_abs(cf{A4[0], A4[3]} * inv_a);
        float rest = BL ? 0.f : s4_;      // e's terms left out
        rx = 2.2f;
        if (coord == SO3G_COORD_TAN) {
            const float ct = 2.f * al2 - 1.f;
            if (!(ct > 0.1f)) return;
            const float ic = rcp_approx(ct), f = 2.f * al2 * ic;
            const float p1 = 2.f * la.l1.r, p2 = 2.f * la.l2.r, p3 = 2.f * la.l3.r;
            const float x1 = f * p1, x2 = f * (p2 + 0.5f * p1 * p1),
                        x3 = f * (p3 + p1 * p2 + (1.f / 6.f) * p1 * p1 * p1);
            const float g1 = -x1, g2 = x1 * x1 - x2, g3 = 2.f * x1 * x2 - x3 - x1 * x1 * x1;
            e1 = z1 + cf{g1, 0.f};
            e2 = z2 + g1 * z1 + cf{g2, 0.f};
            e3 = z3 + g1 * z2 + g2 * z1 + cf{g3, 0.f};
            g *= ic;
            xs = 2.f * ic;
            h += 2.4f * f * ta.X;
            ft = f;
            rest = cx_rest_tan<BL>(f, s1_, s2_, s3_, s4_);
            // (2 ic^2 for a turn, 2 ic^2 sin(theta) for a change of norm.)
            rx = 2.9f * ic * ic;
        } else if (coord == SO3G_COORD_ZEA) {
            const float t1 = la.l1.i, t2 = la.l2.i, t3 = la.l3.i;
            e1 = cf{0.f, t1};
            e2 = cf{-0.5f * t1 * t1, t2};
            e3 = cf{-t1 * t2, t3 - (1.f / 6.f) * t1 * t1 * t1};
            g *= rsqrtf(al2);
            rest = cx_rest_zea<BL>(0.5f * fabsf(t1), 0.25f * fabsf(t2), 0.125f * fabsf(t3),
                                   0.0625f * fabsf(la.l4.i), tail);
            xs = 1.f;
            rx = 2.4f * ia;
        } else {
            e1 = z1;
            e2 = z2;
            e3 = z3;
        }
        if (!(h < 0.1f)) return;
        ry = rx;
        const cf b0{A[2], -A[1]}, b1{A1[2], -A1[1]}, b2{A2[2], -A2[1]}, b3{A3[2], -A3[1]};
        const cf s = g * cf{A[0], A[3]};
        const cf p1 = s * (b1 + e1 * b0), p2 = s * (b2 + e1 * b1 + e2 * b0),
                 p3 = s * (b3 + e1 * b2 + e2 * b1 + e3 * b0);
        cy1 = p1.r;
        cy2 = p2.r;
        cy3 = p3.r;
        cx1 = -p1.i;
        cx2 = -p2.i;
        cx3 = -p3.i;
        // The terms left out of e times conj(beta) (order >= 4, BL: >= 5), with the
        // sizes kn = |b_n| / 2^n, dn = |e_n| / 2^n.
        const float d1 = 0.5f * cf_abs(e1), d2 = 0.25f * cf_abs(e2), d3 = 0.125f * cf_abs(e3);
        const float k0 = cf_abs(b0), k1 = 0.5f * cf_abs(b1), k2 = 0.25f * cf_abs(b2),
                    k3 = 0.125f * cf_abs(b3), k4 = 0.0625f * cf_abs(cf{A4[2], A4[1]});
        const float ks = k1 + k2 + k3 + k4;
        if constexpr (BL) {
            // (One order more.)
            const cf b4{A4[2], -A4[1]};
            cf e4;
            if (coord == SO3G_COORD_TAN) {
                const float ic = rcp_approx(2.f * al2 - 1.f), f = 2.f * al2 * ic;
                const float q1 = 2.f * la.l1.r, q2 = 2.f * la.l2.r, q3 = 2.f * la.l3.r,
                            q4 = 2.f * la.l4.r;
                const float x1 = f * q1, x2 = f * (q2 + 0.5f * q1 * q1),
                            x3 = f * (q3 + q1 * q2 + (1.f / 6.f) * q1 * q1 * q1),
                            x4_ = f * (q4 + q1 * q3 + 0.5f * q2 * q2 + 0.5f * q1 * q1 * q2 +
                                       (1.f / 24.f) * q1 * q1 * q1 * q1);
                const float g1 = -x1, g2 = x1 * x1 - x2, g3 = 2.f * x1 * x2 - x3 - x1 * x1 * x1,
                            g4 = 2.f * x1 * x3 - x4_ + x2 * x2 - 3.f * x1 * x1 * x2 +
                                 x1 * x1 * x1 * x1;
                e4 = cf{A4[0], A4[3]} * inv_a + g1 * z3 + g2 * z2 + g3 * z1 + cf{g4, 0.f};
            } else if (coord == SO3G_COORD_ZEA) {
                const float t1 = la.l1.i, t2 = la.l2.i, t3 = la.l3.i, t4 = la.l4.i;
                e4 = cf{-t1 * t3 - 0.5f * t2 * t2 + (1.f / 24.f) * t1 * t1 * t1 * t1,
                        t4 - 0.5f * t1 * t1 * t2};
            } else {
                e4 = cf{A4[0], A4[3]} * inv_a;
            }
            x4 = s * (b4 + e1 * b3 + e2 * b2 + e3 * b1 + e4 * b0);
            const float d4 = 0.0625f * cf_abs(e4);
            tx = ty = 1.2f * g * (rest * (k0 + ks) + d1 * k4 + d2 * (k3 + k4) +
                                  d3 * (k2 + k3 + k4) + d4 * ks) + 1e-13f;
            // (b_n and e_n: the quaternions' 6u, of A1 u, and 3u of a division; 24u
            // of the products' terms.)
            sx2 = g * (8.f * Qr * (1.f + 2.f * (1.f + ft) * (k0 + k1)) +
                       2.5f * (1.f + 2.f * ft) * Q1 * k1 +
                       24.f * (d1 * (ks + Q1) + (d2 + d3 + d4) * (k0 + ks)));
            const float zn = 2.f * s1_ * (1.f + 2.f * ft) + 2.f * k1;
            curv = 1.5f * (zn * zn + 4.f * s2_ * (1.f + ft) + 4.f * k2);
        } else {
            tx = ty = 1.2f * g * (rest * (k0 + ks) + k4 + d1 * (k3 + k4) + d2 * (ks - k1) +
                                  d3 * ks) + 1e-12f;
        }
    }
    // Pixel coordinates: the coefficients' float32 errors (24u of the terms'
    // sizes, of which cx1 .. carry products of at most a few factors), the
    // sample's polynomial (6u of its terms).
    const float icx = HP ? 1.f : a.mc.inv_cdx, icy = HP ? 1.f : a.mc.inv_cdy;
    const float aix = fabsf(icx), aiy = fabsf(icy);
    const float sx = 0.5f * fabsf(cx1) + 0.25f * fabsf(cx2) + 0.125f * fabsf(cx3);
    const float sy = 0.5f * fabsf(cy1) + 0.25f * fabsf(cy2) + 0.125f * fabsf(cy3);
    if (CL == CX_CAR) big = fmaxf(big, ta.X * 4.f + sx + sy + zz);
    else big *= 1.f + rx;
    float ex = (tx + lutx + rx * E + 32.f * u * (sx + big)) * aix;
    float ey = (ty + luty + ry * E + 32.f * u * (sy + big)) * aiy;
    int xb = 0, yb = 0;
    float xf, yf;
    if constexpr (HP) {
        xf = X0.hi + X0.lo;
        yf = Y0.hi + Y0.lo;
        ex = 1.5f * (ex + 3.f * u * (fabsf(xf) + sx) + 1e-11f);
        ey = 1.5f * (ey + 3.f * u * (fabsf(yf) + sy) + 1e-11f);
    } else {
        const dfl xa = df_add(df_mul(X0, a.fc.inv_cdx), a.fc.off_x);
        const dfl ya = df_add(df_mul(Y0, a.fc.inv_cdy), a.fc.off_y);
        if (!(fabsf(xa.hi) < 1e7f && fabsf(ya.hi) < 1e7f && sx * aix < 1e5f && sy * aiy < 1e5f))
            return;
        dfl fx, fy;
        xb = df_floor(xa, fx);
        yb = df_floor(ya, fy);
        xf = (fx.hi - 0.5f) + fx.lo;
        yf = (fy.hi - 0.5f) + fy.lo;
        xb -= kCxMagicBits;
        yb -= kCxMagicBits;
        // 2 kEpsPix: the reference's own rounding and the middle's error; u:
        // the final sum's rounding.
        ex = 1.5f * (ex + 2.f * kEpsPix + 2.f * u);
        ey = 1.5f * (ey + 2.f * kEpsPix + 2.f * u);
    }
    constexpr float s1 = 1.f / 64.f, s2 = s1 * s1, s3 = s2 * s1, s4 = s2 * s2;
    if constexpr (BL) {
        // X', Y' at the middle in double-float: Y' - i X' = s b1 + e1 (Y0 - i
        // X0), s = 2 g alpha_0, b1 = conj(beta_1), e1 = i Im z1 (ZEA), z1 (SIN)
        // or z1 - 4 n Re(z1) / (2n - 1) (TAN), z1 = alpha_1 / alpha_0.
        const dfl p = B1[0], r = B1[1], s = B1[2], t = B1[3];
        const dfl n = df_dot<2>({qa, qe}, {qa, qe}), rn = df_recip(n);
        const dfl ei = df_mul(df_dot<2>({t, p}, {qa, df_neg(qe)}), rn);
        dfl er = df_mul(df_dot<2>({p, t}, {qa, qe}), rn), G{2.f, 0.f};
        if (coord == SO3G_COORD_TAN) {
            const dfl rc = df_recip(df_sub(df_mulf(n, 2.f), dfl{1.f, 0.f}));
            G = df_mulf(rc, 2.f);
            er = df_sub(er, df_mul(df_mulf(df_mul(n, rc), 4.f), er));
        } else if (coord == SO3G_COORD_ZEA) {
            const float r0 = sqrtf(n.hi);
            const dfl sq = fast_two_sum(r0, (fmaf(-r0, r0, n.hi) + n.lo) / (2.f * r0));
            G = df_mulf(df_recip(sq), 2.f);
            er = dfl{0.f, 0.f};
        }
        const dfl yr = df_mul(G, df_dot<2>({qa, qe}, {s, r}));
        const dfl yi = df_mul(G, df_dot<2>({qe, qa}, {s, df_neg(r)}));
        const dfl Y1 = df_add(yr, df_dot<2>({er, ei}, {Y0, X0}));
        const dfl X1 = df_sub(df_dot<2>({er, ei}, {X0, df_neg(Y0)}), yi);
        const dfl xa = df_add(df_mul(X0, a.fc.inv_cdx), a.fc.off_x);
        const dfl ya = df_add(df_mul(Y0, a.fc.inv_cdy), a.fc.off_y);
        dfl fx, fy;
        df_floor(xa, fx);
        df_floor(ya, fy);
        fx = df_sub(fx, dfl{0.5f, 0.f});
        fy = df_sub(fy, dfl{0.5f, 0.f});
        // Exact parts in multiples of 2^-17 pixel (below 64 pixels in all).
        constexpr float cst = 96.f;
        const dfl vx = df_mulf(df_mul(X1, a.fc.inv_cdx), s1), vy = df_mulf(df_mul(Y1, a.fc.inv_cdy), s1);
        const float fx0 = (fx.hi + cst) - cst, fx1 = (vx.hi + cst) - cst;
        const float fy0 = (fy.hi + cst) - cst, fy1 = (vy.hi + cst) - cst;
        const float x2 = cx2 * icx * s2, x3 = cx3 * icx * s3, x4p = -x4.i * icx * s4;
        const float y2 = cy2 * icy * s2, y3 = cy3 * icy * s3, y4p = x4.r * icy * s4;
        // Errors: the terms left out, the corrections' float32 roundings and
        // those of the coefficients (sx2), the residual's
        // second order and quantisation, its gradient's linear form (which
        // takes the quaternions for unit ones), and the residual's part that is no turn: it scales q, and X and Y with it
        // (SIN 2, ZEA 1, TAN 2 / cos(theta) times their size).
        const float cor = 1024.f * (fabsf(cx2 * icx) + fabsf(cy2 * icy)) * s2 +
                          32768.f * (fabsf(cx3 * icx) + fabsf(cy3 * icy)) * s3 + 2e-4f;
        const float ai = fmaxf(aix, aiy);
        const float far = fmaxf(fabsf(X0.hi), fabsf(Y0.hi)) + fmaxf(sx, sy);
        const float eb = tx * ai + u * (4.f * cor + sx2 * ai) + 3e-12f * rx * ai +
                         1.2f * xs * far * __ldg(&cb.rho0) * ai +
                         (lsb > 0.f ? rx * ai * (E * (16.f * E + curv + 32.f * u + 4.f * norm_off()) +
                                                 2.f * lsb)
                                    : rx * ai * E);
        if (!(eb < kCxBlPix && (sx * aix + 1.f) < 60.f && (sy * aiy + 1.f) < 60.f)) return;
        w[0] = make_float4(fx0, fy0, fx1, fy1);
        w[1] = make_float4(x2, y2, x3, y3);
        w[2] = make_float4((fx.hi - fx0) + fx.lo, (fy.hi - fy0) + fy.lo, (vx.hi - fx1) + vx.lo,
                           (vy.hi - fy1) + vy.lo);
        w[9] = make_float4(x4p, y4p, -1.f, -1.f);
        if (lsb > 0.f) {
            float N0[4], N1[4], gx0[3], gx1[3], gy0[3], gy1[3];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                N0[c] = A[c] - 0.5f * A1[c] + 0.25f * A2[c];
                N1[c] = A[c] + 0.5f * A1[c] + 0.25f * A2[c];
            }
            cx_pixel_gradient(coord, N0, d32, gx0, gy0);
            cx_pixel_gradient(coord, N1, d32, gx1, gy1);
            const float hx = 0.5f * lsb * icx, hy = 0.5f * lsb * icy;
            const float dx = lsb * s1 * icx, dy = lsb * s1 * icy;
#pragma unroll
            for (int c = 0; c < 3; c++)
                w[10 + c] = make_float4((gx0[c] + gx1[c]) * hx, (gy0[c] + gy1[c]) * hy,
                                        (gx1[c] - gx0[c]) * dx, (gy1[c] - gy0[c]) * dy);
        }
    } else {
        w[0] = make_float4(xf, yf, cx1 * icx * s1, cy1 * icy * s1);
        w[1] = make_float4(cx2 * icx * s2, cy2 * icy * s2, cx3 * icx * s3, cy3 * icy * s3);
    }
    float e = 0.f;
    bool flag = (BL && lsb > 0.f) || !covered;
    if constexpr (SPIN) {
        // The spin factors at the middle, F1 + i F2 = P v^2 / D, and phi's
        // derivative there, 2 (Im(alpha_1 conj(alpha_0)) / |alpha_0|^2 + ...
        // beta) or 4 Im(alpha_1 conj(alpha_0)) / |alpha_0|^2, double-float.
        const dfl invD = df_recip(D);
        const dfl F1 = df_mulf(df_mul(df_dot<2>({Nc, Ns}, {Nc, df_neg(Ns)}), invD), Pr);
        const dfl F2 = df_mulf(df_mul(df_mulf(df_mul(Nc, Ns), 2.f), invD), Pr);
        dfl ph;
        {
            const float4 h = __ldg(&cb.a1_hi), l = __ldg(&cb.a1_lo);
            const dfl q[4] = {{h.x, l.x}, {h.y, l.y}, {h.z, l.z}, {h.w, l.w}};
            dfl p, r, s, t;
            df_qmul(q, qd, p, r, s, t);
            const dfl na = df_dot<2>({qa, qe}, {qa, qe});
            ph = df_mul(df_dot<2>({t, p}, {qa, df_neg(qe)}), df_recip(na));
            if (CL == CX_CAR) {
                const dfl nb = df_dot<2>({qb, qc}, {qb, qc});
                ph = df_add(ph, df_mul(df_dot<2>({r, s}, {qc, df_neg(qb)}), df_recip(nb)));
                ph = df_mulf(ph, 2.f);
            } else {
                ph = df_mulf(ph, 4.f);
            }
        }
        // exp(i (phi1 u + phi2 u^2 + ...)) - 1 = sum of (cr_k + i ci_k) u^k;
        // its first coefficient i phi1, the second -phi1^2 / 2 + i phi2.
        const dfl hp2 = df_mulf(df_mul(ph, ph), -0.5f);
        const float p1 = ph.hi, pp = p1 * p1;
        const cf c3{-p1 * phi2, phi3 - (1.f / 6.f) * pp * p1};
        const cf c4{-p1 * phi3 - 0.5f * phi2 * phi2 + (1.f / 24.f) * pp * pp,
                    phi4 - 0.5f * pp * phi2};
        // f0, f1 rounded to multiples of gr = 2^-22 of the power of two
        // >= |Pr|, so that f0 + k f1 (|k| <= 32, |sum| below twice that power)
        // is exact; the rest, l0 and l1, and the higher terms go into the
        // float32 correction.
        const float aP = fabsf(Pr);
        const int pe = ((__float_as_int(aP) - 1) >> 23) + 1;   // biased exponent
        const bool fine = pe > 24 && pe < 250 && fabsf(p1) < 0.5f;
        const float cst = fine ? 3.f * __int_as_float(pe << 23) : 0.f;
        const float gr = fine ? __int_as_float((pe - 22) << 23) : 0.f;
        float o[2][7];
#pragma unroll
        for (int f = 0; f < 2; f++) {
            // F1's terms: Re(c_k (F1 + i F2)); F2's: Im.
            const dfl F = f == 0 ? F1 : F2, G = f == 0 ? df_neg(F2) : F1;
            const dfl d1 = df_mul(ph, G);
            const dfl q1{d1.hi * s1, d1.lo * s1};
            const float f0 = (F.hi + cst) - cst, f1 = (q1.hi + cst) - cst;
            const float l0 = (F.hi - f0) + F.lo, l1 = (q1.hi - f1) + q1.lo;
            const float a2 = fmaf(phi2, G.hi, df_mul(hp2, F).hi);
            const float a3 = c3.r * F.hi + c3.i * G.hi, a4 = c4.r * F.hi + c4.i * G.hi;
            o[f][0] = f0;
            o[f][1] = f1;
            o[f][2] = l0;
            o[f][3] = l1;
            o[f][4] = a2 * s2;
            o[f][5] = a3 * s3;
            o[f][6] = a4 * s4;
        }
        w[4] = make_float4(o[0][0], o[1][0], o[0][1], o[1][1]);
        w[5] = make_float4(o[0][2], o[1][2], o[0][3], o[1][3]);
        w[6] = make_float4(o[0][4], o[1][4], o[0][5], o[1][5]);
        w[7] = make_float4(o[0][6], o[1][6], 0.f, 0.f);
        // e: the double-float error and the reference's roundings (kEpsPf;
        // phi1's is of the same size), the terms left out, the modulus'
        // change and the float32 errors of phi2, phi3 and phi4 (es, and 16u |z1|^2)
        // and of the products, the correction's roundings (3u of its
        // terms), and the boresight's distance from Q.
        const float h1 = 0.5f * fabsf(p1), h2 = 0.25f * fabsf(phi2) + u * zz,
                    h3 = 0.125f * fabsf(phi3) + 8.f * u * zz, h4 = 0.0625f * fabsf(phi4) + 8.f * u * zz;
        const CxTail tp = cx_tail(h1, h2, h3, h4);
        const float Df = D.hi;
        e = 1.2f * (cx_tail_exp(tp) + 4.f * tail) +
            kEpsPf * fmaxf(1.f, 0.25f / Df) * (1.f + h1) + es +
            u * (3.f * h1 * h1 + 8.f * h2 + 4.f * zz + 16.f * (h3 + h4 + h1 * (h2 + h1 * h1)));
        e = e * fmaxf(aP, 1e-3f) + 3.f * u * 18.f * gr;
        if (lsb > 0.f) {
            // The residual's turn: gradient at both ends, linear between;
            // second order in the residual; its quantisation; float32.
            flag = true;
            float N0[4], N1[4], g0[3], g1[3];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                N0[c] = A[c] - 0.5f * A1[c] + 0.25f * A2[c];
                N1[c] = A[c] + 0.5f * A1[c] + 0.25f * A2[c];
            }
            const float ka = cx_gradient<CL>(N0, d32, g0), kb = cx_gradient<CL>(N1, d32, g1);
            const float km = fmaxf(ka, kb) + 1.f;
            e += aP * (E * (2.1f * gerr + km * (64.f * u + 4.f * norm_off())) + 16.f * km * km * E * E +
                       2.f * (km + 4.f) * lsb);
            const float hm = 0.5f * lsb, hd = lsb * s1;
            w[7].z = (g1[0] - g0[0]) * hd;
            w[7].w = (g1[1] - g0[1]) * hd;
            w[8] = make_float4((g0[0] + g1[0]) * hm, (g0[1] + g1[1]) * hm, (g0[2] + g1[2]) * hm,
                               (g1[2] - g0[2]) * hd);
        } else {
            e += aP * (4.3f + 2.2f * rsqrtf(Df)) * E;
        }
        if (!fine) e = __int_as_float(0x7f800000);   // never certain
    }
    if constexpr (BL) w[9].z = w[9].w = e;
    else w[2] = make_float4(HP ? ex : 0.5f - ex, HP ? ey : 0.5f - ey, e, e);
    w[3] = make_float4(__int_as_float(xb), __int_as_float(yb), __int_as_float(mid),
                       flag ? 1.f : 0.f);
}

// The share of a modelled chunk's samples that the per-sample path will take
// (cx_sample finds the pixel or a spin factor's rounding not certain): the
// bounds against the pixel's size and the spacing of floats at the middle's
// factors.
template <bool HP, int NC, bool BL>
__device__ __forceinline__ float cx_share(const float4 *w, float nside, bool covered) {
    if constexpr (BL) return w[9].z >= 0.f ? 0.f : 1.f;
    const float hx = w[2].x, hy = w[2].y;
    if (HP ? !(hx >= 0.f) : !(hx > 0.f && hy > 0.f)) return 1.f;
    // (HEALPix: the two in-face indices, nside (4 lon / 2 pi +- 3/4 z) in the
    // equatorial belt, each within 1.5 times that; a third more for the caps.)
    float s = HP ? 8.f * nside * (0.64f * hx + 0.75f * hy) : 2.f - 2.f * (hx + hy);
    if constexpr (NC > 1) {
        const float e = w[2].z, v[2] = {w[4].x + w[5].x, w[4].y + w[5].y};
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const float ulp = __int_as_float(__float_as_int(v[c]) & 0x7f800000) * 1.1920929e-7f;
            s += ulp > 0.f ? 2.f * e / ulp : 1.f;
        }
    }
    if (!covered) s += 0.25f;   // (on average, of a chunk with a break)
    return s < 1.f ? s : 1.f;   // (1 for a NaN)
}

// Whether the models are worth it: kCxProbes of the call's chunks, spread over
// its segments and their time, give the share of samples that the models will
// leave (a rough boresight, quaternions off unit length, a scan over a pole, a
// detectors without polarisation response) as votes[0] of votes[1]; within a
// tenth of the share counted on flat maps, a third on HEALPix ones (200 det x
// 500k, pointing noise of 1e-9 to 1e-7, polar scans, interpolated boresights).
// One model per lane, 64 warps: a call pays the latency of one set-up.  Without
// it a boresight or detectors stored in 32 bits, or a scan over the pole, took
// 2 to 3 times the general kernel's time; now 1.02 to 1.05.
template <int CL, bool HP, int NC, bool BL, class Args>
__global__ void __launch_bounds__(32)
    k_cx_probe(const __grid_constant__ Args a, const CxBore *bore, int coord, int n_seg,
               const float *det_weights, unsigned long long *votes) {
    const int i = blockIdx.x * 32 + threadIdx.x;
    const int s = (int)((long long)i * n_seg / kCxProbes);
    int det = s, t0 = 0, t1 = a.segs.n_time;
    if (a.segs.seg) {
        det = __ldg(a.segs.seg + 3 * s);
        t0 = __ldg(a.segs.seg + 3 * s + 1);
        t1 = __ldg(a.segs.seg + 3 * s + 2);
    }
    unsigned long long left = 0, all = 0;
    if (t1 > t0 && !(det_weights && __ldg(det_weights + det) == 0.f)) {
        const int j0 = t0 / kCxLen, n = (t1 - 1) / kCxLen + 1 - j0;
        const int j = j0 + (int)__umulhi((unsigned)i * 2654435769u, (unsigned)n);
        const QuatD ofs = load_quat(a.dets + 4LL * det);
        const dfl qd[4] = {df_of(ofs.a), df_of(ofs.b), df_of(ofs.c), df_of(ofs.d)};
        float4 w[BL ? kCxBlWords : kCxWords];
        cx_setup<CL, HP, NC, BL>(a, bore, coord, j, a.segs.n_time, qd,
                                 __ldg(a.resp + 2 * det + 1), w);
        const float share =
            cx_share<HP, NC, BL>(w, (float)(int)a.g.nside, __ldg(&bore[j].part) == 0.f);
        all = 1024ULL * (unsigned)n;
        left = (unsigned long long)(share * 1024.f) * (unsigned)n;
    }
#pragma unroll
    for (int m = 16; m; m >>= 1) {
        left += __shfl_xor_sync(kFull, left, m);
        all += __shfl_xor_sync(kFull, all, m);
    }
    if (threadIdx.x == 0) {
        atomicAdd(votes, left);
        atomicAdd(votes + 1, all);
    }
}

__device__ __forceinline__ f32x2 cx_lo(const float4 &w) { return f2_make(w.x, w.y); }
__device__ __forceinline__ f32x2 cx_hi(const float4 &w) { return f2_make(w.z, w.w); }

// The exact parts S and corrections L of the spin factors at k = t - mid
// (k2: in both halves), with the residual's turn where `flag` is set.
__device__ __forceinline__ void cx_factors(const float4 *w, f32x2 k2, const float (&res)[3],
                                           bool flag, f32x2 &S, f32x2 &L) {
    const float4 W4 = w[4], W5 = w[5], W6 = w[6], W7 = w[7];
    L = f2_fma(k2, f2_fma(k2, f2_fma(k2, f2_fma(k2, cx_lo(W7), cx_hi(W6)), cx_lo(W6)), cx_hi(W5)),
               cx_lo(W5));
    S = f2_fma(k2, cx_hi(W4), cx_lo(W4));
    if (flag) {
        const float4 W8 = w[8];
        float k, k_, gx, gy, S1, S2, L1, L2;
        f2_get(k2, k, k_);
        f2_get(f2_fma(k2, cx_hi(W7), cx_lo(W8)), gx, gy);
        f2_get(S, S1, S2);
        f2_get(L, L1, L2);
        const float dphi = fmaf(gx, res[0], fmaf(gy, res[1], fmaf(k, W8.w, W8.z) * res[2]));
        L = f2_make(fmaf(-S2, dphi, L1), fmaf(S1, dphi, L2));
    }
}

// Their float32 values (within e2 of S + L); false when a rounding is not
// certain.
__device__ __forceinline__ bool cx_round(f32x2 S, f32x2 L, f32x2 e2, float &v1, float &v2) {
    float u1, u2;
    f2_get(f2_add(S, f2_add(L, e2)), v1, v2);
    f2_get(f2_add(S, f2_sub(L, e2)), u1, u2);
    return (v1 == u1) & (v2 == u2);
}

// The HEALPix pixel of longitude x (error ex; < 0: none) and sin(lat) y (ey),
// or -1 where it is not certain.  Not inlined: four copies of it in the main
// loop made the kernel wait for instructions (400 det x 500k, nside 1024, to_map
// and from_map: 7.5 -> 7.1 ms).
template <int P>
static __device__ __noinline__ int cx_hp_pixel(int nside, int nest, int npix, float x, float ex,
                                               float y, float ey) {
    if (!(ex >= 0.f)) return -1;
    DGeom g;
    g.nside = nside;
    g.nest = nest;
    g.npix = npix;
    int pix[1] = {0};
    return hp_pixel_f32<P, P == PX_HP_T, true>(g, x, ex, y, ey, 0.f, 0.f, pix) ? pix[0] : -1;
}

// One sample (k2: t - mid in both halves) of a modelled chunk: pixel key (flat: iy * nx +
// ix, of the parent map when tiled; HEALPix: the pixel), on the map or not,
// and the spin factors of an NC-component map; false when the pixel or
// (on the map) a spin factor is not certain.  res: the sample's residual
// (used where the chunk's flag is set).  P = PX_FLAT_T_NN: the tiled
// pixelizor's rule (int() truncation, src/Projection.cxx:1124-1138).
// A spin factor is within e of S + L (S exact), so the reference's value
// rounds to the same float32 when S + (L + e) and S + (L - e) do.
template <int P, int NC>
__device__ __forceinline__ bool cx_sample(const float4 *w, f32x2 k2, const float (&res)[3],
                                          bool flag, const DGeom &g, float T, int &key, bool &on,
                                          float (&pf)[3]) {
    const float4 P0 = w[0], P1 = w[1], P2 = w[2];
    const f32x2 xy =
        f2_fma(k2, f2_fma(k2, f2_fma(k2, cx_hi(P1), cx_lo(P1)), cx_hi(P0)), cx_lo(P0));
    bool ok;
    const bool left = flag && res[0] < (float)(kCxUncovered + 200);
    if constexpr (P == PX_HP_NT || P == PX_HP_T) {
        float x, y;
        f2_get(xy, x, y);
        key = cx_hp_pixel<P>((int)g.nside, g.nest, (int)g.npix, x, P2.x, y, P2.y);
        ok = (key >= 0) & !left;
        on = true;
    } else {
        const float4 P3 = w[3];
        // x, y less 1/2: the nearest integer is the floor, and the distance
        // from it the fraction less 1/2.
        const f32x2 magic = f2_both(kCxMagic), r2 = f2_add(xy, magic);
        float rx, ry, dx, dy;
        f2_get(r2, rx, ry);
        f2_get(f2_sub(xy, f2_sub(r2, magic)), dx, dy);
        ok = (fabsf(dx) < P2.x) & (fabsf(dy) < P2.y) & !left;
        int ix = __float_as_int(P3.x) + __float_as_int(rx),
            iy = __float_as_int(P3.y) + __float_as_int(ry);
        if constexpr (P == PX_FLAT_T_NN) {
            on = ((unsigned)(ix + 1) < (unsigned)(g.nx + 1)) &
                 ((unsigned)(iy + 1) < (unsigned)(g.ny + 1));
            ix = max(ix, 0);
            iy = max(iy, 0);
        } else {
            on = ((unsigned)ix < (unsigned)g.nx) & ((unsigned)iy < (unsigned)g.ny);
        }
        key = iy * g.nx + ix;
    }
    if constexpr (NC == 1) {
        pf[0] = T;
        pf[1] = pf[2] = 0.f;
    } else {
        f32x2 S, L;
        cx_factors(w, k2, res, flag, S, L);
        float v1, v2;
        const bool c = cx_round(S, L, cx_hi(P2), v1, v2);
        ok = ok & (c | !on);
        if constexpr (NC == 2) {
            pf[0] = v1;
            pf[1] = v2;
            pf[2] = 0.f;
        } else {
            pf[0] = T;
            pf[1] = v1;
            pf[2] = v2;
        }
    }
    return ok;
}

// The residuals of samples t .. t + 3 (t a multiple of 4, below kCxLen (n_chunks
// + 1): the lanes of a round without a chunk of their own read on past the last
// one, where the array is padded, and use nothing of it).
__device__ __forceinline__ void cx_residuals(const short4 *resid, int t, float (&r)[4][3]) {
    const int4 *p = reinterpret_cast<const int4 *>(resid + t);
    const int4 u = __ldg(p), v = __ldg(p + 1);
    const int lo[4] = {u.x, u.z, v.x, v.z}, hi[4] = {u.y, u.w, v.y, v.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        r[i][0] = (float)(short)(lo[i] & 0xffff);
        r[i][1] = (float)(lo[i] >> 16);
        r[i][2] = (float)(short)(hi[i] & 0xffff);
    }
}

// ---------------------------------------------------------------------------
// Samples the models leave.  Each warp collects them in shared memory and
// appends them, 32 or more at a time, to a list in global memory; a second
// kernel takes the list through the per-sample certified path and appends
// what that leaves to another list, for the float64 path: every path runs
// on full warps, and the main kernel's code stays small (with the per-sample
// paths called from it, instruction fetch stalls made it 2.2 times slower).
// Entries past a list's capacity are handled on the spot; a call that would
// fill the list takes the general kernel (k_cx_probe).

struct CxList {
    unsigned long long *count;
    int2 *entry;               // (det, t)
    unsigned long long cap;
};

// Samples a warp collects before it appends them: below 32 plus a round.
constexpr int kCxQueue = 160;

struct CxWarp {
    int n;                   // entries of queue
    int queue[kCxQueue];
};

// Appends samples tq + i for the bits i of f4; all lanes must call when any
// has a bit.  Returns the queue's length.
__device__ __forceinline__ int cx_enqueue(CxWarp &cw, unsigned f4, int tq) {
    if (f4) {
        int p = atomicAdd(&cw.n, __popc(f4));
        while (f4) {
            cw.queue[p++] = tq + __ffs(f4) - 1;
            f4 &= f4 - 1;
        }
    }
    __syncwarp();
    return cw.n;
}

// Moves the warp's queue to the list; over(t) handles a sample that does
// not fit.  All lanes must call.
template <class F>
__device__ __forceinline__ void cx_append(CxWarp &cw, const CxList &list, int det, F &&over) {
    const int lane = threadIdx.x & 31, n = cw.n;
    if (n == 0) return;
    unsigned long long p = 0;
    if (lane == 0) p = atomicAdd(list.count, (unsigned long long)n);
    p = __shfl_sync(kFull, p, 0);
    for (int i = lane; i < n; i += 32) {
        if (p + i < list.cap) list.entry[p + i] = make_int2(det, cw.queue[i]);
        else over(cw.queue[i]);
    }
    __syncwarp();
    if (lane == 0) cw.n = 0;
    __syncwarp();
}

// Calls f(det, t) for every entry of `list`, one lane each; where f returns
// false, the entry goes to `next` (over(det, t) when that is full).
template <class F, class G>
__device__ __forceinline__ void cx_for_each(const CxList &list, const CxList &next, F &&f,
                                            G &&over) {
    const unsigned long long n = min(*list.count, list.cap);
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
         (i & ~31ULL) < n; i += stride) {
        int2 e = make_int2(0, 0);
        bool left = false;
        if (i < n) {
            e = list.entry[i];
            left = !f(e.x, e.y);
        }
        const unsigned m = __ballot_sync(kFull, left);
        if (!m) continue;
        unsigned long long p = 0;
        if (lane == 0) p = atomicAdd(next.count, (unsigned long long)__popc(m));
        p = __shfl_sync(kFull, p, 0) + __popc(m & ((1u << lane) - 1u));
        if (left) {
            if (p < next.cap) next.entry[p] = e;
            else over(e.x, e.y);
        }
    }
}

// A HEALPix sample whose spin factors were not certain: its pixel (n taps, 0
// or 1) from the double-float pointing and only the spin factors in float64;
// false where the pixel is not certain.  (400 det x 500k, nside 1024, to_map and
// from_map: 6.9 -> 6.5 ms, the float64 pixel with its divisions left out.  A flat
// map's float64 pixel is two table lookups, and this made its calls 3 % slower:
// they take the whole float64 path.)
template <int C, int P, class Args>
__device__ __forceinline__ bool cx_exact_spin(const Args &a, int det, int t, int *pix, int &n,
                                              float (&pf)[3]) {
    const QuatD ofs = load_quat(a.dets + 4LL * det), b = load_quat(a.bore + 4LL * t);
    const dfl qd[4] = {df_of(ofs.a), df_of(ofs.b), df_of(ofs.c), df_of(ofs.d)};
    const float T = __ldg(a.resp + 2 * det), Pr = __ldg(a.resp + 2 * det + 1);
    dfl qb[4];
    if (!(df_split(b.a, qb[0]) & df_split(b.b, qb[1]) & df_split(b.c, qb[2]) &
          df_split(b.d, qb[3])))
        return false;
    int px[1][3];
    float w[1];
    n = 0;
    if (!fast_pointing<C, P, false>(a.g, a.ft, a.fc, qb, qd, a.g.ncomp, T, Pr, px, w, n, pf))
        return false;
    pix[0] = px[0][0];
    pix[1] = px[0][1];
    pix[2] = px[0][2];
    if (n == 0) return true;
    // (The coordinates themselves, and their tables, are not used.)
    double coords[4];
    get_coords<C>(a.g.lut, b, ofs, coords);
    spin_factors(a.g.ncomp, coords, T, Pr, pf);
    return true;
}

constexpr unsigned kCxFixBlocks = 152 * 8;   // of kBlock threads, striding over a list

// Chunks of a warp's group for a block that has n: even shares for its warps,
// in equal groups of at most kCxGroup, an even number (a round takes two).
__device__ __forceinline__ int cx_step(int n) {
    const int share = (n + kCxWarps - 1) / kCxWarps;
    const int groups = (share + kCxGroup - 1) / kCxGroup;
    return ((share + groups - 1) / groups + 1) & ~1;
}

// Samples per block of a call: each warp of a block takes up to kCxGroup
// chunks at once, fewer (even) when the call would not fill the GPU twice.
inline int cx_piece(long long n_seg, long long max_len) {
    constexpr long long kResident = 152 * 24;   // warps on the GPU at once
    const long long chunks = n_seg * ((max_len + kCxLen - 1) / kCxLen);
    long long per_warp = chunks / (2 * kResident);
    per_warp = per_warp < 2 ? 2 : (per_warp > kCxGroup ? kCxGroup : per_warp & ~1LL);
    long long p = per_warp * kCxWarps * kCxLen;
    while (per_warp == kCxGroup && p < 32768 && chunks * kCxLen > 16 * kResident / kCxWarps * p) p *= 2;
    while ((max_len + p - 1) / p > 65535) p *= 2;
    return (int)p;
}

// The workspace of a call, in stream-ordered memory: the chunks' boresight
// models, the residuals and the two lists (one entry for every 10 and 96
// samples: the workloads leave 1 in 50 and 1 in 1000).
struct CxWork {
    void *mem = nullptr;
    CxModel model;
    CxList left, exact;
    SkipIf gate;               // the chunked kernels skip when it holds (after cx_probe)
};

// Allocates the workspace and makes the boresight models; false (nothing
// left allocated) when that fails (the caller takes the per-sample path).
inline bool cx_work(CxWork &w, const double *bore, int n_time, long long samples,
                    cudaStream_t stream) {
    const long long n_chunks = (n_time + kCxLen - 1) / kCxLen;
    const long long cap1 = samples / 10 + 4096, cap2 = samples / 96 + 4096;
    const size_t o_res = 256 + sizeof(CxBore) * (size_t)n_chunks;
    // (One chunk of padding: cx_residuals.)
    const size_t o_l1 = o_res + sizeof(short4) * (size_t)((n_chunks + 1) * kCxLen);
    const size_t o_l2 = o_l1 + sizeof(int2) * (size_t)cap1;
    const size_t bytes = o_l2 + sizeof(int2) * (size_t)cap2;
    if (cudaMallocAsync(&w.mem, bytes, stream) != cudaSuccess) {
        cudaGetLastError();
        w.mem = nullptr;
        return false;
    }
    char *p = static_cast<char *>(w.mem);
    unsigned long long *counts = reinterpret_cast<unsigned long long *>(p);
    CxBore *models = reinterpret_cast<CxBore *>(p + 256);
    short4 *resid = reinterpret_cast<short4 *>(p + o_res);
    w.model = CxModel{models, resid};
    w.left = CxList{counts, reinterpret_cast<int2 *>(p + o_l1), (unsigned long long)cap1};
    w.exact = CxList{counts + 1, reinterpret_cast<int2 *>(p + o_l2), (unsigned long long)cap2};
    w.gate = SkipIf{counts + 2, kCxShare, true};
    const long long threads = 16 * n_chunks;
    k_cx_bore<<<(unsigned)((threads + 127) / 128), 128, 0, stream>>>(
        bore, n_time, (int)n_chunks, models, resid, counts);
    if (after_launch("boresight chunk models (certified)") != SO3G_OK) {
        cudaFreeAsync(w.mem, stream);
        w.mem = nullptr;
        clear_error();
        return false;
    }
    return true;
}

template <int CL, bool HP, int NC, bool BL, class Args>
int cx_probe(const Args &a, const CxWork &w, int coord, long long n_seg, const float *det_weights,
             cudaStream_t st) {
    k_cx_probe<CL, HP, NC, BL><<<kCxProbes / 32, 32, 0, st>>>(
        a, w.model.bore, coord, (int)n_seg, det_weights, w.left.count + 2);
    return after_launch("share of samples the chunk models leave");
}

}  // namespace

}  // namespace so3g
