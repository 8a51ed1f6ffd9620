// The D-step with the per-sequence dictionary state held as half-spectra.
//
// dict_update! (src/CDL/train.jl:46-89) transforms Y3, H = (G1 - g1) + (G3 - g3) and d to
// the frequency domain, solves per frequency, returns d to the time domain, updates the
// duals g1 += d - G1 and g3 += d - G3 (:70, :72) and averages d + g1, d + g3 and d over
// the sequences (:76, :83; and D_best, :91-98).  Every one of those steps after the
// solve is linear, and nothing outside the D-step reads d, g1 or g3.  So they are kept
// as half-spectra, with one more reduction:
//   * g1 and g3 start at zero and both receive the same d; their difference changes by
//     G3 - G1, the same for every sequence.  So g1 - g3 is one (M, F) spectrum Dg shared
//     by all sequences, and g3 = g1 - Dg: only d-hat and g1-hat are per sequence;
//   * H-hat = (G1-hat - g1-hat) + (G3-hat - g3-hat) with g3-hat = g1-hat - Dg, the duals
//     g1-hat += d-hat - G1-hat and Dg += G3-hat - G1-hat, and the averages of d + g1 and
//     d (that of d + g3 is the first minus Dg) are (M, F) spectra, returned to the time
//     domain once per D-step for the projections.  A D-step then transforms only Y3.
// The reference's statements applied to the transforms, with g3 recovered from the
// shared difference; results differ from the time-domain path by FP32 rounding.
#include "cdlgb_internal.h"

#include <cuda_pipeline_primitives.h>

#include <algorithm>

namespace {

__device__ __forceinline__ float2 cadd2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub2(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cfma2(float2 a, float2 b, float2 c) {   // a*b + c
    return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}
__device__ __forceinline__ float2 cjfma2(float2 a, float2 b, float2 c) {  // conj(a)*b + c
    return make_float2(fmaf(a.x, b.x, fmaf(a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(-a.y, b.x, c.y)));
}

struct SArgs {
    const float2* Yh;     // scratch (c1 - c0, M, La/2 + 1): Y3-hat's bins of sequences [c0, c1)
    const float2* G1h;    // (M, F)
    const float2* G3h;    // (M, F)
    const float2* Dg;     // (M, F): g1-hat - g3-hat, the same for every sequence
    float2* Dh;           // (N, M, F): rfft(d_old) in, the new d-hat out
    float2* g1h;          // (N, M, F)
    const float2* Zh;     // (N, F): rfft(G2 - g2)
    float2* Th;           // (N, F): scale * sum_m Y3h rfft(d_old)
    float2* part;         // (slots, 2, M, F): sums of d + g1 and of d over a sub-range
    double* rpart;        // (slots, nbb, 3): Parseval sums of |d-hat - G1-hat|^2,
                          // |d-hat - G3-hat|^2, |d-hat|^2 of a CTA (the residual record)
    int N, M, F, La, c0, c1, slot0;
    float kd, scale;
};

constexpr int kBins = 32, kWarps = 16;

// weight * q into the compensated sums rs, rc
template <bool RES>
__device__ __forceinline__ void add_residuals(const float (&q)[3], float weight, float (&rs)[3], float (&rc)[3]) {
#pragma unroll
    for (int k = 0; k < (RES ? 3 : 0); ++k) {
        const float y = __fsub_rn(__fmul_rn(weight, q[k]), rc[k]);
        const float t = __fadd_rn(rs[k], y);
        rc[k] = __fsub_rn(__fsub_rn(t, rs[k]), y);
        rs[k] = t;
    }
}
// the CTA's residual partials, in float64, added in warp order
__device__ __forceinline__ void store_residuals(const SArgs& A, const float (&rs)[3], const float (&rc)[3]) {
    __shared__ double rsh[3][kWarps];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double v = (double)rs[k] - (double)rc[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) rsh[k][w] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double t = 0.0;
        for (int v = 0; v < kWarps; ++v) t += rsh[threadIdx.x][v];
        A.rpart[((size_t)(A.slot0 + blockIdx.y) * gridDim.x + blockIdx.x) * 3 + threadIdx.x] = t;
    }
}

// grid (ceil(F / 32), nsub): a CTA takes 32 bins and sub-range s of the sequences
// [c0, c1), in order, and writes that sub-range's sums to slot slot0 + s; warp w owns
// filters w, w + 16, ... (MW of them at most, M <= 16 MW; k_dspec_wide takes more).
//
// A sequence is a chain -- its three spectra's loads, the sums over the filters (over the
// warps), the solve, the stores -- of little arithmetic, so what counts is what is in flight:
//   * each thread's spectra of the next NST - 2 sequences are on their way to shared memory
//     (asynchronous copies into the thread's own slots, NST buffers);
//   * sequence n's sums are formed while sequence n - 1 is solved from its own, one barrier
//     per sequence;
//   * what a thread uses at every sequence (G1-hat, G1-hat + G3-hat + Dg of its filters) is in
//     registers, addresses are stepped, and for M <= 32 two CTAs share an SM.
// With every filter slot loaded, two barriers, one sequence ahead and whole Y3 spectra, a
// D-step after the first took 6.66 ms at 20000 sequences, 64 filters and 465 bins, 4.29 at
// (5000, 32, 1065), 1.04 at (5000, 10, 417) and 0.207 at (1000, 16, 249); now 5.89, 2.11, 0.417
// and 0.137.
// The copies and the stores through L1, a few bytes per thread, hold it at two thirds of the
// HBM rate.
//
// RES: also the residual partials (compiled out when false).  INIT: the first D-step of a
// training, whose d-hat is G1-hat for every sequence and whose g1-hat is zero: neither is
// read, nor was it written.
template <int MW, int NST, bool RES, bool INIT>
__global__ void __launch_bounds__(kBins * kWarps, MW <= 2 ? 2 : 1) k_dspec(SArgs A) {
    extern __shared__ float4 sm4[];
    constexpr int kArr = INIT ? 1 : 3;                     // staged spectra: Y3-hat, g1-hat, d-hat
    constexpr int NT = kBins * kWarps;
    const int M = A.M, F = A.F;
    const int j = blockIdx.y, cn = A.c1 - A.c0;
    const int n0 = A.c0 + (int)((int64_t)cn * j / gridDim.y);
    const int n1 = A.c0 + (int)((int64_t)cn * (j + 1) / gridDim.y);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int f = blockIdx.x * kBins + lane;
    const bool on = f < F;
    const bool edge = f == 0 || f == F - 1;
    const int fl = on ? f : 0;                             // lanes past F take bin 0, store nothing
    // Y3 is zero off every fourth row: its transform repeats with period La = Lg / 4 and is
    // stored as the La/2 + 1 bins of the real rows kept
    const int FY = A.La / 2 + 1, fy = fl % A.La;
    const float ysign = 2 * fy > A.La ? -1.f : 1.f;
    const int yl = 2 * fy > A.La ? A.La - fy : fy;
    // the warps' partial sums of B, Q.x, Q.y, T.x, T.y per bin, [2][5][kWarps][32], and
    // their totals, [2][5][32]: each total is summed once, by one thread, in warp order
    float* pp = reinterpret_cast<float*>(sm4);
    float* tot = pp + 2 * 5 * kWarps * kBins;
    float2* stg = reinterpret_cast<float2*>(tot + 2 * 5 * kBins) + threadIdx.x;   // [NST][kArr][MW][NT]
    float2 G1r[MW], Kr[MW], s1[MW], sd[MW];
#pragma unroll
    for (int k = 0; k < MW; ++k) {
        const size_t i = (size_t)min(w + kWarps * k, M - 1) * F + fl;
        G1r[k] = A.G1h[i];
        // H = (G1 - g1) + (G3 - g3) with g3 = g1 - Dg (train.jl:52-54) is Kr - 2 g1
        Kr[k] = cadd2(cadd2(G1r[k], A.G3h[i]), A.Dg[i]);
        s1[k] = sd[k] = make_float2(0.f, 0.f);
    }
    // compensated (Kahan) float32 sums over this thread's sequences of the g1 and g3
    // increments' and d's squared magnitudes (Parseval weights: 1 at the edge bins, 2
    // elsewhere), combined in float64 at the end
    float rs[3] = {0.f, 0.f, 0.f}, rc[3] = {0.f, 0.f, 0.f};
    const int ystep = kWarps * FY, step = kWarps * F;      // from a filter of a thread to its next
    const float2* yp = A.Yh + ((size_t)(n0 - A.c0) * M + w) * FY + yl;   // the sequence to stage next
    size_t sp = ((size_t)n0 * M + w) * F + fl;             // ... in g1-hat and d-hat
    auto stage = [&](int buf) {
        float2* d0 = stg + buf * (kArr * MW * NT);
#pragma unroll
        for (int k = 0; k < MW; ++k) {
            if (w + kWarps * k >= M) break;
            __pipeline_memcpy_async(d0 + k * NT, yp + k * ystep, sizeof(float2));
            if (INIT) continue;
            __pipeline_memcpy_async(d0 + (MW + k) * NT, A.g1h + sp + k * step, sizeof(float2));
            __pipeline_memcpy_async(d0 + (2 * MW + k) * NT, A.Dh + sp + k * step, sizeof(float2));
        }
        yp += (size_t)M * FY;
        sp += (size_t)M * F;
    };
    size_t op = ((size_t)n0 * M + w) * F + fl;             // the sequence to solve next
    for (int s = 0; s < NST - 2; ++s) {
        if (n0 + s < n1) stage(s);
        __pipeline_commit();
    }
    // rfft(G2 - g2) of the bin, loaded a sequence ahead
    float2 z = make_float2(0.f, 0.f);
    int cur = 0, prev = NST - 1, ahead = NST - 2;          // buffers of sequences n, n - 1, n + NST - 2
    int par = 0;
    for (int n = n0; n <= n1; ++n) {
        float2 zn = z;
        if (n < n1) {
            zn = A.Zh[(size_t)n * F + fl];
            // a group per sequence, empty past the last; its buffer held sequence n - 2
            if (n + NST - 2 < n1) stage(ahead);
            __pipeline_commit();
            __pipeline_wait_prior(NST - 2);
            const float2* s0 = stg + cur * (kArr * MW * NT);
            float B = 0.f;
            float2 Q = make_float2(0.f, 0.f), T = make_float2(0.f, 0.f);
#pragma unroll
            for (int k = 0; k < MW; ++k) {
                if (w + kWarps * k >= M) break;
                float2 y = s0[k * NT];
                y.y *= ysign;
                float2 h = Kr[k], d = G1r[k];
                if (INIT) {
                    if (edge) d.y = 0.f;
                } else {
                    const float2 g = s0[(MW + k) * NT];
                    h = csub2(h, cadd2(g, g));
                    d = s0[(2 * MW + k) * NT];
                }
                B = fmaf(y.x, y.x, fmaf(y.y, y.y, B));
                Q = cfma2(y, h, Q);
                T = cfma2(y, d, T);
            }
            float* p = pp + (par * 5 * kWarps + w) * kBins + lane;
            p[0] = B;
            p[kWarps * kBins] = Q.x;
            p[2 * kWarps * kBins] = Q.y;
            p[3 * kWarps * kBins] = T.x;
            p[4 * kWarps * kBins] = T.y;
        }
        __syncthreads();     // sequence n's partial sums and n - 1's totals are written
        if (w < 5 && n < n1) {
            const float* src = pp + (par * 5 + w) * kWarps * kBins + lane;
            float acc = 0.f;
#pragma unroll
            for (int v = 0; v < kWarps; ++v) acc += src[v * kBins];
            tot[(par * 5 + w) * kBins + lane] = acc;
        }
        par ^= 1;
        if (n > n0 && on) {
            const float* t = tot + par * 5 * kBins + lane;
            const float B = t[0];
            const float inv = 1.f / (B + A.kd);
            const float2 beta = make_float2(fmaf(z.x, B, t[kBins]) * inv, fmaf(z.y, B, t[2 * kBins]) * inv);
            const float2 W = csub2(z, beta);
            const float2* s0 = stg + prev * (kArr * MW * NT);
            float q[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < MW; ++k) {
                if (w + kWarps * k >= M) break;
                float2 y = s0[k * NT], g = make_float2(0.f, 0.f), h = Kr[k];
                y.y *= ysign;
                if (!INIT) {
                    g = s0[(MW + k) * NT];
                    h = csub2(h, cadd2(g, g));
                }
                // REF_QUIRK_Q1: the combine has no 1/2, unlike the X-step's (cdl_kernels.jl:30)
                float2 dh = cjfma2(y, W, h);
                if (edge) dh.y = 0.f;                      // the transform of a real d
                // g1 += d - G1 with G1 before the update (train.jl:70)
                const float2 e1 = csub2(dh, G1r[k]);
                const float2 g1n = cadd2(g, e1);
                A.Dh[op + k * step] = dh;
                A.g1h[op + k * step] = g1n;
                s1[k] = cadd2(s1[k], cadd2(dh, g1n));
                sd[k] = cadd2(sd[k], dh);
                if (!RES) continue;
                const float2 G3 = __ldg(A.G3h + (w + kWarps * k) * (size_t)F + f);
                const float2 e3 = csub2(dh, G3);           // g3 += d - G3 (:72)
                q[0] = fmaf(e1.x, e1.x, fmaf(e1.y, e1.y, q[0]));
                q[1] = fmaf(e3.x, e3.x, fmaf(e3.y, e3.y, q[1]));
                q[2] = fmaf(dh.x, dh.x, fmaf(dh.y, dh.y, q[2]));
            }
            add_residuals<RES>(q, edge ? 1.f : 2.f, rs, rc);
            if (w == 0) A.Th[(size_t)(n - 1) * F + f] = make_float2(t[3 * kBins] * A.scale, t[4 * kBins] * A.scale);
            op += (size_t)M * F;
        }
        z = zn;
        prev = cur;
        cur = cur + 1 == NST ? 0 : cur + 1;
        ahead = ahead + 1 == NST ? 0 : ahead + 1;
    }
    if (RES) store_residuals(A, rs, rc);
    if (!on) return;
    float2* out = A.part + (size_t)(A.slot0 + j) * 2 * M * F + (size_t)w * F + f;
#pragma unroll
    for (int k = 0; k < MW; ++k) {
        if (w + kWarps * k >= M) break;
        out[k * step] = s1[k];
        out[(size_t)M * F + k * step] = sd[k];
    }
}

// The same for M up to 16 MW = 128 filters, whose spectra fit neither the registers nor the
// staging: loaded as they are needed, kept in registers between the sums and the solve.
template <bool RES, bool INIT>
__global__ void __launch_bounds__(kBins * kWarps, 1) k_dspec_wide(SArgs A) {
    constexpr int MW = 8;
    extern __shared__ float4 sm4[];
    const int M = A.M, F = A.F;
    const int j = blockIdx.y, cn = A.c1 - A.c0;
    const int n0 = A.c0 + (int)((int64_t)cn * j / gridDim.y);
    const int n1 = A.c0 + (int)((int64_t)cn * (j + 1) / gridDim.y);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int f = blockIdx.x * kBins + lane;
    const bool on = f < F;
    const bool edge = f == 0 || f == F - 1;
    float2* G1s = reinterpret_cast<float2*>(sm4);          // [M][32]
    // Ks = G1-hat + G3-hat + Dg: H = (G1 - g1) + (G3 - g3) with g3 = g1 - Dg is
    // Ks - 2 g1, one shared spectrum instead of three (G3s is kept for the residuals)
    float2* Ks = G1s + (size_t)M * kBins;                  // [M][32]
    float2* G3s = Ks + (size_t)M * kBins;                  // [M][32]
    // the warps' partial sums of B, Q.x, Q.y, T.x, T.y per bin, [5][kWarps][32], and
    // their totals, [5][32]: each total is summed once, by one thread, in warp order
    float* pp = reinterpret_cast<float*>(G3s + (size_t)M * kBins);
    float* tot = pp + 5 * kWarps * kBins;
    for (int i = threadIdx.x; i < M * kBins; i += blockDim.x) {
        const int m = i / kBins, ff = blockIdx.x * kBins + i % kBins;
        const bool in = ff < F;
        const float2 g1 = in ? A.G1h[(size_t)m * F + ff] : make_float2(0.f, 0.f);
        const float2 g3 = in ? A.G3h[(size_t)m * F + ff] : make_float2(0.f, 0.f);
        const float2 dg = in ? A.Dg[(size_t)m * F + ff] : make_float2(0.f, 0.f);
        G1s[i] = g1;
        G3s[i] = g3;
        Ks[i] = cadd2(cadd2(g1, g3), dg);
    }
    float2 s1[MW], sd[MW];
#pragma unroll
    for (int k = 0; k < MW; ++k) s1[k] = sd[k] = make_float2(0.f, 0.f);
    // compensated (Kahan) float32 sums over this thread's sequences of the g1 and g3
    // increments' and d's squared magnitudes (Parseval weights: 1 at the edge bins, 2
    // elsewhere), combined in float64 at the end
    float rs[3] = {0.f, 0.f, 0.f}, rc[3] = {0.f, 0.f, 0.f};
    __syncthreads();
    const int fl = on ? f : 0;                             // lanes past F load bin 0
    // Y3 is zero off every fourth row: its transform repeats with period La = Lg / 4 and is
    // stored as the La/2 + 1 bins of the real rows kept
    const int FY = A.La / 2 + 1, fy = fl % A.La;
    const bool mirror = 2 * fy > A.La;
    const int yl = mirror ? A.La - fy : fy;
    // rfft(G2 - g2) of the bin, loaded one sequence ahead (it is needed after the
    // cross-warp sums, where a load issued then would stall every warp)
    float2 zn = (on && n0 < n1) ? A.Zh[(size_t)n0 * F + f] : make_float2(0.f, 0.f);
    for (int n = n0; n < n1; ++n) {
        const float2 z = zn;
        if (on && n + 1 < n1) zn = A.Zh[(size_t)(n + 1) * F + f];
        // every load of this sequence first (independent), then the arithmetic
        float2 yv[MW], g1v[MW], dv[MW];
        const size_t base = (size_t)n * M * F + fl;
        const size_t ybase = (size_t)(n - A.c0) * M * FY + yl;
#pragma unroll
        for (int k = 0; k < MW; ++k) {
            const int m = min(w + kWarps * k, M - 1);  // in bounds; unused when m >= M
            yv[k] = A.Yh[ybase + (size_t)m * FY];
            if (INIT) continue;
            g1v[k] = A.g1h[base + (size_t)m * F];
            dv[k] = A.Dh[base + (size_t)m * F];
        }
        if (INIT) {
#pragma unroll
            for (int k = 0; k < MW; ++k) {
                g1v[k] = make_float2(0.f, 0.f);
                dv[k] = G1s[min(w + kWarps * k, M - 1) * kBins + lane];
            }
        }
        if (mirror) {
#pragma unroll
            for (int k = 0; k < MW; ++k) yv[k].y = -yv[k].y;
        }
        float2 hv[MW];
        float B = 0.f;
        float2 Q = make_float2(0.f, 0.f), T = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < MW; ++k) {
            const int m = w + kWarps * k;
            const bool use = on && m < M;
            const int ms = use ? m : 0;
            const float2 y = use ? yv[k] : make_float2(0.f, 0.f);
            float2 d = use ? dv[k] : make_float2(0.f, 0.f);
            if (edge) d.y = 0.f;
            // H = (G1 - g1) + (G3 - g3) with g3 = g1 - Dg  (train.jl:52-54), = Ks - 2 g1
            const float2 h = use ? csub2(Ks[ms * kBins + lane], cadd2(g1v[k], g1v[k]))
                                 : make_float2(0.f, 0.f);
            hv[k] = h;
            B = fmaf(y.x, y.x, fmaf(y.y, y.y, B));
            Q = cfma2(y, h, Q);
            T = cfma2(y, d, T);
        }
        pp[(0 * kWarps + w) * kBins + lane] = B;
        pp[(1 * kWarps + w) * kBins + lane] = Q.x;
        pp[(2 * kWarps + w) * kBins + lane] = Q.y;
        pp[(3 * kWarps + w) * kBins + lane] = T.x;
        pp[(4 * kWarps + w) * kBins + lane] = T.y;
        __syncthreads();
        if (w < 5) {
            // warp w sums component w over the warps for its lane's bin, warp 0 first
            // (the order every thread summed all of them in before: the same bits)
            const float* src = pp + w * kWarps * kBins + lane;
            float acc = 0.f;
#pragma unroll
            for (int v = 0; v < kWarps; ++v) acc += src[v * kBins];
            tot[w * kBins + lane] = acc;
        }
        __syncthreads();                                   // totals written; partials read
        B = tot[lane];
        Q = make_float2(tot[kBins + lane], tot[2 * kBins + lane]);
        T = make_float2(tot[3 * kBins + lane], tot[4 * kBins + lane]);
        if (on) {
            const float inv = 1.f / (B + A.kd);
            const float2 beta = make_float2(fmaf(z.x, B, Q.x) * inv, fmaf(z.y, B, Q.y) * inv);
            const float2 W = csub2(z, beta);
            float q[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < MW; ++k) {
                const int m = w + kWarps * k;
                if (m >= M) continue;
                // REF_QUIRK_Q1: the combine has no 1/2, unlike the X-step's (cdl_kernels.jl:30)
                float2 dh = cjfma2(yv[k], W, hv[k]);
                if (edge) dh.y = 0.f;                      // the transform of a real d
                const size_t i = (size_t)n * M * F + (size_t)m * F + f;
                // g1 += d - G1 with G1 before the update (train.jl:70)
                const float2 e1 = csub2(dh, G1s[m * kBins + lane]);
                const float2 g1n = cadd2(g1v[k], e1);
                A.Dh[i] = dh;
                A.g1h[i] = g1n;
                s1[k] = cadd2(s1[k], cadd2(dh, g1n));
                sd[k] = cadd2(sd[k], dh);
                if (!RES) continue;
                const float2 e3 = csub2(dh, G3s[m * kBins + lane]);   // g3 += d - G3 (:72)
                q[0] = fmaf(e1.x, e1.x, fmaf(e1.y, e1.y, q[0]));
                q[1] = fmaf(e3.x, e3.x, fmaf(e3.y, e3.y, q[1]));
                q[2] = fmaf(dh.x, dh.x, fmaf(dh.y, dh.y, q[2]));
            }
            add_residuals<RES>(q, edge ? 1.f : 2.f, rs, rc);
            if (w == 0) A.Th[(size_t)n * F + f] = make_float2(T.x * A.scale, T.y * A.scale);
        }
    }
    if (RES) store_residuals(A, rs, rc);
    if (!on) return;
#pragma unroll
    for (int k = 0; k < MW; ++k) {
        const int m = w + kWarps * k;
        if (m >= M) continue;
        const size_t pi = (size_t)m * F + f;
        const size_t q = (size_t)(A.slot0 + j) * 2 * M * F;
        A.part[q + pi] = s1[k];
        A.part[q + (size_t)M * F + pi] = sd[k];
    }
}

// The three sums' spectra, scaled by 1/Lg so that the unnormalised inverse transform
// gives the time-domain sums: out[0] = sum (d + g1), out[2] = sum d (over the slots, in
// double), out[1] = sum (d + g3) = out[0] - N Dg after this D-step's Dg += G3-hat - G1-hat
// (the change of g1 - g3, train.jl:70, 72; the solves have used the old one).  Four
// threads per output take the slots j = t mod 4 in order; the four partials are added in
// a fixed order.
__global__ void k_dspec_sum(const float2* __restrict__ part, float2* __restrict__ Dg,
                            const float2* __restrict__ G1h, const float2* __restrict__ G3h, float2* __restrict__ out, size_t mf, int slots, int N, double inv_lg) {
    const size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t i = g >> 2;                                // 0 .. 2 mf - 1
    const int t = (int)(g & 3);
    double re = 0.0, im = 0.0;
    if (i < 2 * mf)
        for (int j = t; j < slots; j += 4) {
            const float2 v = part[(size_t)j * 2 * mf + i];
            re += v.x;
            im += v.y;
        }
    re += __shfl_down_sync(0xffffffffu, re, 1);
    im += __shfl_down_sync(0xffffffffu, im, 1);
    re += __shfl_down_sync(0xffffffffu, re, 2);
    im += __shfl_down_sync(0xffffffffu, im, 2);
    if (t != 0 || i >= 2 * mf) return;
    if (i < mf) {
        out[i] = make_float2((float)(re * inv_lg), (float)(im * inv_lg));
        const float2 dg = cadd2(Dg[i], csub2(G3h[i], G1h[i]));
        Dg[i] = dg;
        out[mf + i] = make_float2((float)((re - (double)N * dg.x) * inv_lg),
                                  (float)((im - (double)N * dg.y) * inv_lg));
    } else {
        out[mf + i] = make_float2((float)(re * inv_lg), (float)(im * inv_lg));
    }
}

// dst = a - plane, the plane broadcast over n (g3-hat = g1-hat - Dg)
__global__ void k_sub_bcast(float2* __restrict__ dst, const float2* __restrict__ a,
                            const float2* __restrict__ plane, size_t mf, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        dst[i] = csub2(a[i], plane[i % mf]);
}

__global__ void k_scale(float* __restrict__ x, size_t n, float s) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        x[i] *= s;
}

}  // namespace

int dspec_max_m() { return kWarps * 8; }

size_t dspec_part_bytes(int M, int F, int slots) { return (size_t)slots * 2 * M * F * sizeof(float2); }

// CTAs per SM (k_dspec's launch bounds; its shared memory fits)
static int dspec_ctas(int M) { return M <= 2 * kWarps ? 2 : 1; }

// Sub-ranges of one launch over cn sequences.  One or two CTAs fit per SM, so a launch runs
// ceil(nbb nsub / CTAs) waves of CTAs that each take ceil(cn / nsub) sequences after a
// start-up (the block's G1-hat, G3-hat, Dg and the first staged sequence) worth about
// two sequences; the count minimising that estimate is taken (the smallest on ties).
// It depends only on (cn, M, F, nsm), so the slot layout and the order of the sums are
// fixed for a given device and size.
int dspec_nsub(int cn, int M, int F, int nsm) {
    const int nbb = (F + kBins - 1) / kBins;
    nsm = std::max(nsm, 1) * dspec_ctas(M);
    int best = 1;
    long long bt = -1;
    for (int s = 1; s <= std::min(cn, 2048); ++s) {
        const long long waves = ((long long)nbb * s + nsm - 1) / nsm;
        const long long t = waves * ((cn + s - 1) / s + 2);
        if (bt < 0 || t < bt) { bt = t; best = s; }
    }
    return best;
}

int dspec_slots(int N, int chunk, int M, int F, int nsm) {
    int slots = 0;
    for (int n0 = 0; n0 < N; n0 += chunk) slots += dspec_nsub(std::min(chunk, N - n0), M, F, nsm);
    return slots;
}

template <int MW, int NST, bool INIT>
static int launch_form(cdlgb_ctx* c, const SArgs& a, dim3 g) {
    auto k = c->res_on ? k_dspec<MW, NST, true, INIT> : k_dspec<MW, NST, false, INIT>;
    constexpr size_t sm = (size_t)2 * 5 * (kWarps + 1) * kBins * sizeof(float) +
                          (size_t)(INIT ? 1 : 3) * NST * MW * kBins * kWarps * sizeof(float2);
    CU_TRY(c, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k<<<g, kBins * kWarps, sm, c->stream>>>(a);
    LAUNCH_CHECK(c, "k_dspec");
    return CDLGB_OK;
}
// NST buffers; the first D-step stages one spectrum of three, so twice as many sequences ahead
template <int MW, int NST>
static int launch(cdlgb_ctx* c, const SArgs& a, dim3 g) {
    return c->spec_init ? launch_form<MW, 2 * NST, true>(c, a, g) : launch_form<MW, NST, false>(c, a, g);
}

int dspec_launch(cdlgb_ctx* c, const float2* Yh, const float2* G3h, int c0, int c1, int slot0) {
    SArgs a;
    a.Yh = Yh; a.G1h = c->G1h; a.G3h = G3h; a.Dg = c->Dg; a.Dh = c->Dhs; a.g1h = c->g1h;
    a.Zh = c->sUh; a.Th = c->sVh; a.part = c->spart; a.rpart = c->rpart;
    a.N = c->N; a.M = c->M; a.F = c->F; a.La = c->Lg / 4; a.c0 = c0; a.c1 = c1; a.slot0 = slot0;
    a.kd = c->p.sherman_const_cdl; a.scale = 1.f / (float)c->Lg;
    const dim3 g((unsigned)((c->F + kBins - 1) / kBins), (unsigned)dspec_nsub(c1 - c0, c->M, c->F, c->nsm));
    if (c->M <= kWarps) return launch<1, 4>(c, a, g);
    if (c->M <= 2 * kWarps) return launch<2, 3>(c, a, g);
    // (three buffers, not the four that fit: with 218 KB of shared memory the L1 that the
    // copies pass through is left 28 KB, and 64 filters took 5.65 ms instead of 4.65)
    if (c->M <= 4 * kWarps) return launch<4, 3>(c, a, g);
    const size_t sm = (size_t)3 * c->M * kBins * sizeof(float2) + (size_t)kWarps * kBins * 5 * sizeof(float) +
                      (size_t)5 * kBins * sizeof(float);
    auto k = c->res_on ? (c->spec_init ? k_dspec_wide<true, true> : k_dspec_wide<true, false>)
                       : (c->spec_init ? k_dspec_wide<false, true> : k_dspec_wide<false, false>);
    // process-wide per kernel: the same cap for every context (M = 128 takes 107 KB)
    CU_TRY(c, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024));
    k<<<g, kBins * kWarps, sm, c->stream>>>(a);
    LAUNCH_CHECK(c, "k_dspec_wide");
    return CDLGB_OK;
}

// the Dg update (after every chunk has used the old Dg) and the three sums: out (3, M, F)
int dspec_sums(cdlgb_ctx* c, const float2* G3h, float2* out) {
    const size_t mf = (size_t)c->M * c->F;
    k_dspec_sum<<<(unsigned)((4 * 2 * mf + 255) / 256), 256, 0, c->stream>>>(
        c->spart, c->Dg, c->G1h, G3h, out, mf, c->dslots, c->N, 1.0 / (double)c->Lg);
    LAUNCH_CHECK(c, "k_dspec_sum");
    return CDLGB_OK;
}

// g3-hat of rows (sequence x filter) [0, rows) of g1h into dst
int dspec_g3(cdlgb_ctx* c, float2* dst, const float2* g1h, size_t rows) {
    const size_t mf = (size_t)c->M * c->F;
    k_sub_bcast<<<grid_for(rows * c->F, 256), 256, 0, c->stream>>>(dst, g1h, c->Dg, mf, rows * c->F);
    LAUNCH_CHECK(c, "k_sub_bcast");
    return CDLGB_OK;
}

int dspec_scale(cdlgb_ctx* c, float* x, size_t n, float s) {
    k_scale<<<grid_for(n, 256), 256, 0, c->stream>>>(x, n, s);
    LAUNCH_CHECK(c, "k_scale");
    return CDLGB_OK;
}
