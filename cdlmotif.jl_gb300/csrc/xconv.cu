// X-steps by short convolutions (code_update!, src/CDL/train.jl:1-44), for any Lg.
//
// G1 is zero outside its first T = 4W rows (prox_simplex_zeros!, cdl_kernels.jl:53-66, and
// the constructor's mask), so the X-step needs no transform of the M code rows: with
//   P = sum_m g_m (*) v_m      (circular, T taps)
//   W = irfft( rfft(k U - P) / (k + A) ),   DX = U - W,   A = sum_m |G1-hat[m]|^2
//   X_m[l] = (v_m[l] + sum_j g_m[j] W[l + j]) / k
// this is the Sherman-Morrison solve of train.jl:18-27 (csc_kernels.jl:8-49) in the time
// domain, and only W, one row per sequence, goes through a transform.
//
// An X-step has two parts:
//   codes   a CTA takes B pairs of filters of one sequence: X from the previous step's V
//           and W, then shrink!, projectionX! and the dual updates (csc_kernels.jl:53-82,
//           train.jl:12-14) give this step's V, which goes through shared memory and is
//           convolved with the taps into the CTA's part of P;
//   solve   a CTA takes one sequence: P, the transforms, W, DX, Y1 (update_Y1!,
//           csc_kernels.jl:86-95), y1 and U.
// Between the steps a code is kept as t = X + y2 and u = X + y3, from which V and both duals
// follow by the operations that define them (xsplit2: the same bits): two arrays read and
// written per X-step instead of V, y2 and y3 (a code update of 15 X-steps 3.60 -> 3.43 ms at
// 5000 sequences, L = 200, 10 filters of 4 bases, 8.18 -> 7.81 at 500, 1000, 32, 16).
// Each is a launch over all sequences (k_xc_codes, k_xc_solve), started early with
// griddepcontrol; where one CTA holds all filters of a sequence and all sequences are
// resident at once, one launch runs all X-steps instead (k_xc_all).
#include "cdlgb_internal.h"
#include "regfft.cuh"

#include <math.h>
#include <stdlib.h>
#include <algorithm>

namespace {

constexpr int kMaxStages = 10;
constexpr int kR = 16;                  // rows per thread
constexpr int kMaxTaps = 128;
constexpr int kMaxLg = 16384;
constexpr int kMaxThreads = 320;        // at most, two CTAs per SM: 96 registers a thread
constexpr size_t kSmemSm = 228 * 1024;  // per SM; a CTA also has 1 KB reserved
constexpr size_t kSmemCta = 226 * 1024;

// Two packed floats as one 64-bit register, as loaded from shared memory: the operands of
// the packed FMAs stay in aligned register pairs without moves.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 ffma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float2 unpack(f32x2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}

struct Args {
    const float* Xin;       // X
    float* V;               // t = X + y2 between the steps, X after the last
    float* y2;              // read by the first, written after the last
    float* y3;              // u = X + y3 between the steps
    float* Y1;
    float* y1;
    float* DX;
    const float* S;
    const float* G1;
    float* P;               // [cn][G][Lg] parts of sum_m g_m (*) v_m, of PB pairs each
    float* W;               // [cn][Lg]
    float* U;               // [cn][Lg]
    double* absx_part;      // [N][CTAs per sequence] sum |X|
    const float2* tw;       // per stage [radix - 1][s] exp(-2 pi i o q / m), s = m / radix
    const float2* wk;       // [n/2 + 1] exp(-pi i k / n)
    const ushort2* pos;     // [n/2 + 1] places of bins k and n - k after the forward stages
    const float2* Hsd;      // [n/2 + 1] (H[k] + H[n-k])/2n, (H[k] - H[n-k])/2n
    int n0, M, Lg, L4, gamma, iters, T, G;
    int first, last;        // k_xc_solve: the code update's first, last X-step
    int zero;               // y2, y3 are zero and not written yet (the initial state)
    float lam, rho, kc;
    int NB;                 // blocks of 16 taps (the last one filled up with zeros)
    int B, CG, nchunk;      // pairs per CTA, row blocks per warp, row blocks
    int PB, PCG;            // pairs per part of P, row blocks per warp that forms one
    int pitch;              // places of V per pair in shared memory
    int n, nst;
    int radix[kMaxStages], twoff[kMaxStages];
};

// places in the transform buffer: one complex of padding per 16, so that the stages with
// short strides spread over the banks
__device__ __forceinline__ int fp(int i) { return i + (i >> 4); }

template <int SIGN>
__device__ __forceinline__ void dft4(float2& a, float2& b, float2& c, float2& d) {
    const float2 s0 = cadd(a, c), s1 = csub(a, c), s2 = cadd(b, d), s3 = mul_i<SIGN>(csub(b, d));
    a = cadd(s0, s2);
    c = csub(s0, s2);
    b = cadd(s1, s3);
    d = csub(s1, s3);
}

// DFT of R values in natural order, in registers
template <int R, int SIGN>
__device__ __forceinline__ void dft_small(float2 (&x)[R]) {
    if (R == 2) {
        const float2 t = x[0];
        x[0] = cadd(t, x[1]);
        x[1] = csub(t, x[1]);
    } else if (R == 3) {
        constexpr float s = 0.866025403784438647f;
        const float2 t = cadd(x[1], x[2]);
        const float2 u = csub(x[1], x[2]);
        const float2 a = rfma(t, -0.5f, x[0]);
        const float2 b = mul_i<SIGN>(f2(u.x * s, u.y * s));
        x[0] = cadd(x[0], t);
        x[1] = cadd(a, b);
        x[2] = csub(a, b);
    } else if (R == 4) {
        dft4<SIGN>(x[0], x[1], x[2], x[3]);
    } else if (R == 5) {
        constexpr float c1 = 0.309016994374947424f, c2 = -0.809016994374947424f;
        constexpr float s1 = 0.951056516295153572f, s2 = 0.587785252292473129f;
        const float2 t1 = cadd(x[1], x[4]), t2 = cadd(x[2], x[3]);
        const float2 u1 = csub(x[1], x[4]), u2 = csub(x[2], x[3]);
        const float2 a1 = rfma(t1, c1, rfma(t2, c2, x[0])), a2 = rfma(t1, c2, rfma(t2, c1, x[0]));
        const float2 b1 = mul_i<SIGN>(rfma(u1, s1, f2(u2.x * s2, u2.y * s2)));
        const float2 b2 = mul_i<SIGN>(rfma(u1, s2, f2(u2.x * -s1, u2.y * -s1)));
        x[0] = cadd(x[0], cadd(t1, t2));
        x[1] = cadd(a1, b1);
        x[4] = csub(a1, b1);
        x[2] = cadd(a2, b2);
        x[3] = csub(a2, b2);
    } else if (R == 8) {
        constexpr float h = 0.707106781186547524f;
        float2 e0 = x[0], e1 = x[2], e2 = x[4], e3 = x[6];
        float2 o0 = x[1], o1 = x[3], o2 = x[5], o3 = x[7];
        dft4<SIGN>(e0, e1, e2, e3);
        dft4<SIGN>(o0, o1, o2, o3);
        const float2 r1 = mul_i<SIGN>(o1), r3 = mul_i<SIGN>(o3);
        const float2 q1 = cadd(o1, r1), q3 = csub(r3, o3);          // sqrt(2) times w8 o1, w8^3 o3
        o2 = mul_i<SIGN>(o2);
        x[0] = cadd(e0, o0);
        x[4] = csub(e0, o0);
        x[1] = rfma(q1, h, e1);
        x[5] = rfma(q1, -h, e1);
        x[2] = cadd(e2, o2);
        x[6] = csub(e2, o2);
        x[3] = rfma(q3, h, e3);
        x[7] = rfma(q3, -h, e3);
    }
}

// One stage over sub-transforms of length m, in place.  Forward (decimation in frequency):
// the DFT, then the twiddles; inverse (decimation in time): the conjugate twiddles, then
// the inverse DFT.  m / R is a power of two except at the first stage, where m = n.  The
// twiddles of a stage lie one after another (a common table's strided entries cost a
// cache line per lane).
template <int R, bool INV>
__device__ __forceinline__ void stage(float2* __restrict__ buf, const float2* __restrict__ tw, int n,
                                      int m, int nt) {
    const int s = m / R;
    const int sh = m == n ? 31 : 31 - __clz(s);
    __syncthreads();
#pragma unroll 1
    for (int t = threadIdx.x; t < n / R; t += nt) {
        const int b = t >> sh;                    // 0 at the first stage
        const int o = t - (b << sh) * (m != n);
        const int base = b * m + o;
        float2 x[R], w[R];
#pragma unroll
        for (int q = 1; q < R; ++q) w[q] = __ldg(tw + (q - 1) * s + o);
#pragma unroll
        for (int q = 0; q < R; ++q) x[q] = buf[fp(base + q * s)];
        if (INV) {
#pragma unroll
            for (int q = 1; q < R; ++q) x[q] = cmulc(x[q], w[q]);
        }
        dft_small<R, INV ? 1 : -1>(x);
        if (!INV) {
#pragma unroll
            for (int q = 1; q < R; ++q) x[q] = cmul(x[q], w[q]);
        }
#pragma unroll
        for (int q = 0; q < R; ++q) buf[fp(base + q * s)] = x[q];
    }
}

template <bool INV>
__device__ __forceinline__ void run_stage(float2* buf, const Args& A, int st, int m, int nt) {
    const int r = A.radix[st];
    const float2* tw = A.tw + A.twoff[st];
    if (r == 8) stage<8, INV>(buf, tw, A.n, m, nt);
    else if (r == 4) stage<4, INV>(buf, tw, A.n, m, nt);
    else if (r == 2) stage<2, INV>(buf, tw, A.n, m, nt);
    else if (r == 3) stage<3, INV>(buf, tw, A.n, m, nt);
    else stage<5, INV>(buf, tw, A.n, m, nt);
}

// One sequence's solve.  W = irfft(rfft(k U - P) / (k + A)) multiplies by a real, even
// spectrum, so it is a circular convolution with a symmetric kernel; that is evaluated as
// a linear one on the padded length 2n >= 2 Lg with n = 2^a 3^b 5^c, folded back, which
// leaves Lg free.  The 2n real values go as n complex ones (even, odd) through buf.
__device__ __forceinline__ void solve(const Args& A, float2* buf, size_t c, size_t n, bool first, bool last) {
    const int NT = blockDim.x, Lg = A.Lg, half = Lg / 2, n_ = A.n;
    const float2* Pg = reinterpret_cast<const float2*>(A.P + c * A.G * Lg);
    float2* Ug = reinterpret_cast<float2*>(A.U + c * Lg);
    float2* Y1g = reinterpret_cast<float2*>(A.Y1 + n * Lg);
    float2* y1g = reinterpret_cast<float2*>(A.y1 + n * Lg);
    float2* DXg = reinterpret_cast<float2*>(A.DX + n * Lg);
    // Z = k U - P (the parts in order), zero-padded.  The code update's first step forms
    // U = Y1 - y1', y1' = y1 + DX - Y1 (train.jl:12; REF_QUIRK_Q6: the previous iteration's Y1)
    for (int i = threadIdx.x; i < n_; i += NT) {
        float2 z = f2(0.f, 0.f);
        if (i < half) {
            float2 P_ = Pg[i];
            for (int g = 1; g < A.G; ++g) P_ = cadd(P_, Pg[(size_t)g * half + i]);
            float2 U;
            if (first) {
                const float2 Yv = Y1g[i], yv = y1g[i], dv = DXg[i];
                const float2 yn = f2((yv.x + dv.x) - Yv.x, (yv.y + dv.y) - Yv.y);
                U = f2(Yv.x - yn.x, Yv.y - yn.y);
                y1g[i] = yn;
                Ug[i] = U;
            } else {
                U = Ug[i];
            }
            z = f2(fmaf(A.kc, U.x, -P_.x), fmaf(A.kc, U.y, -P_.y));
        }
        buf[fp(i)] = z;
    }
    int m = n_;
#pragma unroll 1
    for (int st = 0; st < A.nst; ++st) {
        run_stage<false>(buf, A, st, m, NT);
        m /= A.radix[st];
    }
    __syncthreads();
    // the real spectrum of the 2n values from the n complex ones, times H, and back
    for (int k = threadIdx.x; k <= n_ / 2; k += NT) {
        const ushort2 pp = __ldg(A.pos + k);
        const float2 hh = __ldg(A.Hsd + k), w = __ldg(A.wk + k);
        const float2 c1 = buf[fp(pp.x)], c2 = buf[fp(pp.y)];
        const float2 E = f2(0.5f * (c1.x + c2.x), 0.5f * (c1.y - c2.y));
        const float2 O = f2(0.5f * (c1.y + c2.y), 0.5f * (c2.x - c1.x));
        const float2 wO = cmul(O, w), wE = cmulc(E, w);
        const float2 E2 = f2(fmaf(hh.x, E.x, hh.y * wO.x), fmaf(hh.x, E.y, hh.y * wO.y));
        const float2 O2 = f2(fmaf(hh.x, O.x, hh.y * wE.x), fmaf(hh.x, O.y, hh.y * wE.y));
        buf[fp(pp.x)] = f2(E2.x - O2.y, E2.y + O2.x);
        if (pp.x != pp.y) buf[fp(pp.y)] = f2(E2.x + O2.y, O2.x - E2.y);
    }
#pragma unroll 1
    for (int st = A.nst - 1; st >= 0; --st) {
        m *= A.radix[st];
        run_stage<true>(buf, A, st, m, NT);
    }
    __syncthreads();
    // W folded, DX = U - W, Y1 = (W'S + rho (DX + y1')) / (W'W + rho), then the next
    // iteration's y1' and U
    float2* Wg = reinterpret_cast<float2*>(A.W + c * Lg);
    for (int i = threadIdx.x; i < half; i += NT) {
        const float2 a = buf[fp(i)];
        const float2 b = buf[fp(2 * i >= half ? i - half + n_ : i + half)];
        const float2 W = cadd(a, b);
        const float2 dx = csub(Ug[i], W), yp = y1g[i];
        const int l = 2 * i;
        Wg[i] = W;
        const bool in = l >= A.gamma && l < A.gamma + A.L4;
        const float2 wts = in ? *reinterpret_cast<const float2*>(A.S + n * A.L4 + (l - A.gamma)) : f2(0.f, 0.f);
        const float dg = in ? 1.f : 0.f;
        const float2 Yn = f2(__fadd_rn(wts.x, __fmul_rn(A.rho, dx.x + yp.x)) / (dg + A.rho),
                             __fadd_rn(wts.y, __fmul_rn(A.rho, dx.y + yp.y)) / (dg + A.rho));
        if (!last) {
            const float2 yn = f2((yp.x + dx.x) - Yn.x, (yp.y + dx.y) - Yn.y);
            y1g[i] = yn;
            Ug[i] = f2(Yn.x - yn.x, Yn.y - yn.y);
        } else {
            DXg[i] = dx;
            Y1g[i] = Yn;
        }
    }
}

// FIRST: t, u and V from X and the duals; MID: X from the previous V and W, then t, u and V;
// LAST: X and the duals.
// A thread owns 16 consecutive rows of a pair of filters, two packed floats per row: it
// keeps 16 sums in registers and slides over the taps, one shared-memory load per 16
// packed FMAs.  gs: [8 NB][B] two taps of a pair; ws: [9 (nchunk + NB)] two values of W,
// twice each, 16 values and a gap; Vs: [B][pitch], a row l of V at place l % 16 of row block
// l / 16 + NB, 17 places of 8 bytes per block (the pitch has a residue modulo 16 for which
// a warp's lanes, pair fastest, then block, spread over the banks); the NB blocks before
// the first hold the last 16 NB rows again (the circular wrap).  LAST returns sum |X|: four
// rows of a filter in float32, as k_abssum adds them, and these in float64.
enum { FIRST, MID, LAST };
template <int MODE>
__device__ __forceinline__ double codes(const Args& A, const float4* gs, const float4* ws, float2* Vs, size_t n, int m0,
                                       int Mr) {
    constexpr int R = kR;
    const int NB = A.NB, TP = 16 * NB, Lg = A.Lg, B = A.B, M = A.M;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int p = lane % B, cl = lane / B;
    const bool lane_on = cl < A.CG && 2 * p < Mr;
    const ulonglong2* gp = reinterpret_cast<const ulonglong2*>(gs) + p;
    const float lam = A.lam, ik = 1.f / A.kc;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    double absacc = 0.0;
    for (int q0 = warp * A.CG; q0 < A.nchunk; q0 += nwarps * A.CG) {
        // ---------------- sum_j g[j] W[l + j], left in V's place
        const int q = q0 + cl;
        if (MODE != FIRST && lane_on && q < A.nchunk) {
            f32x2 acc[R];
            const ulonglong2* wq = reinterpret_cast<const ulonglong2*>(ws) + 9 * q;
            f32x2 w[R];
#pragma unroll
            for (int i = 0; i < R; i += 2) {
                const ulonglong2 u = wq[i >> 1];
                w[i] = u.x;
                w[i + 1] = u.y;
                acc[i] = acc[i + 1] = 0;
            }
            const ulonglong2* gb = gp;
            // 16 taps at a time: after them every row is back at its place in w
#pragma unroll 1
            for (int b = 0; b < NB; ++b, gb += 8 * B) {
                wq += 9;
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    const ulonglong2 gg = gb[(j >> 1) * B];
                    const ulonglong2 u = wq[j >> 1];          // the two values of W after these 16
#pragma unroll
                    for (int i = 0; i < R; ++i) acc[i] = ffma2(gg.x, w[(i + j) & 15], acc[i]);
                    w[j] = u.x;
#pragma unroll
                    for (int i = 0; i < R; ++i) acc[i] = ffma2(gg.y, w[(i + j + 1) & 15], acc[i]);
                    w[j + 1] = u.y;
                }
            }
            f32x2* vq = reinterpret_cast<f32x2*>(Vs + p * A.pitch + 17 * (q + NB));
#pragma unroll
            for (int i = 0; i < R; ++i) vq[i] = acc[i];
        }
        __syncwarp();
        // ---------------- X, the duals and V of the warp's own row blocks: four rows of a
        // pair per lane, neighbouring lanes along the rows (whole lines of the arrays)
        const int per = min(4 * A.CG, Lg / 4 - 4 * q0), groups = (Mr + 1) / 2 * per;
        int pp = 0, k4 = lane;
        for (int e = lane; e < groups; e += 64) {
            // two groups of four rows in flight
            float4 xa[2], xb[2], aa[2], ab[2], ba[2], bb[2];       // X (t), y2, y3 (u) of both filters
            int pu[2], ku[2];
            size_t ra[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                while (k4 >= per) { k4 -= per; ++pp; }
                pu[u] = pp;
                ku[u] = k4;
                ra[u] = (n * M + m0 + 2 * pp) * Lg + R * q0 + 4 * k4;
                const bool on = e + 32 * u < groups;
                const bool two = on && 2 * pp + 1 < Mr;              // the pair's second filter exists
                const float* src = (MODE == FIRST ? A.Xin : A.V) + ra[u];
                xa[u] = on ? *reinterpret_cast<const float4*>(src) : z4;
                xb[u] = two ? *reinterpret_cast<const float4*>(src + Lg) : z4;
                if (MODE == FIRST && A.zero) {
                    aa[u] = ab[u] = ba[u] = bb[u] = z4;
                } else {
                    ba[u] = on ? *reinterpret_cast<const float4*>(A.y3 + ra[u]) : z4;
                    bb[u] = two ? *reinterpret_cast<const float4*>(A.y3 + ra[u] + Lg) : z4;
                    if (MODE == FIRST) {
                        aa[u] = on ? *reinterpret_cast<const float4*>(A.y2 + ra[u]) : z4;
                        ab[u] = two ? *reinterpret_cast<const float4*>(A.y2 + ra[u] + Lg) : z4;
                    }
                }
                k4 += 32;
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (e + 32 * u >= groups) break;
                const bool two = 2 * pu[u] + 1 < Mr;
                const int l = R * q0 + 4 * ku[u];
                float2 x[4] = {f2(xa[u].x, xb[u].x), f2(xa[u].y, xb[u].y), f2(xa[u].z, xb[u].z), f2(xa[u].w, xb[u].w)};
                float2 a3[4] = {f2(ba[u].x, bb[u].x), f2(ba[u].y, bb[u].y), f2(ba[u].z, bb[u].z), f2(ba[u].w, bb[u].w)};
                float2 a2[4];
                if (MODE == FIRST) {
                    a2[0] = f2(aa[u].x, ab[u].x);
                    a2[1] = f2(aa[u].y, ab[u].y);
                    a2[2] = f2(aa[u].z, ab[u].z);
                    a2[3] = f2(aa[u].w, ab[u].w);
                }
                float2* vq = Vs + pu[u] * A.pitch + 17 * (q0 + (ku[u] >> 2) + NB) + 4 * (ku[u] & 3);
                if (MODE != FIRST) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float2 v = xsplit2(x[k], a3[k], a2[k], a3[k], lam, k == 0);
                        x[k] = cadd(v, vq[k]);
                        x[k] = f2(x[k].x * ik, x[k].y * ik);
                    }
                }
                float* dst = A.V + ra[u];
                if (MODE == LAST) {
                    *reinterpret_cast<float4*>(dst) = make_float4(x[0].x, x[1].x, x[2].x, x[3].x);
                    *reinterpret_cast<float4*>(A.y2 + ra[u]) = make_float4(a2[0].x, a2[1].x, a2[2].x, a2[3].x);
                    *reinterpret_cast<float4*>(A.y3 + ra[u]) = make_float4(0.f, a3[1].x, a3[2].x, a3[3].x);
                    if (two) {
                        *reinterpret_cast<float4*>(dst + Lg) = make_float4(x[0].y, x[1].y, x[2].y, x[3].y);
                        *reinterpret_cast<float4*>(A.y2 + ra[u] + Lg) = make_float4(a2[0].y, a2[1].y, a2[2].y, a2[3].y);
                        *reinterpret_cast<float4*>(A.y3 + ra[u] + Lg) = make_float4(0.f, a3[1].y, a3[2].y, a3[3].y);
                    }
                    absacc += (double)((fabsf(x[0].x) + fabsf(x[1].x)) + (fabsf(x[2].x) + fabsf(x[3].x)));
                    if (two) absacc += (double)((fabsf(x[0].y) + fabsf(x[1].y)) + (fabsf(x[2].y) + fabsf(x[3].y)));
                    continue;
                }
                float2 v[4], w[4];                                   // V; u (x becomes t)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    w[k] = cadd(x[k], a3[k]);
                    x[k] = cadd(x[k], a2[k]);
                    v[k] = xsplit2(x[k], w[k], a2[k], a3[k], lam, k == 0);
                    vq[k] = v[k];
                }
                if (l + 3 >= Lg - TP) {                              // again before the first row
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int at = l + k - Lg + TP;
                        if (at >= 0) Vs[pu[u] * A.pitch + fp(at)] = v[k];
                    }
                }
                *reinterpret_cast<float4*>(dst) = make_float4(x[0].x, x[1].x, x[2].x, x[3].x);
                *reinterpret_cast<float4*>(A.y3 + ra[u]) = make_float4(w[0].x, w[1].x, w[2].x, w[3].x);
                if (two) {
                    *reinterpret_cast<float4*>(dst + Lg) = make_float4(x[0].y, x[1].y, x[2].y, x[3].y);
                    *reinterpret_cast<float4*>(A.y3 + ra[u] + Lg) = make_float4(w[0].y, w[1].y, w[2].y, w[3].y);
                }
            }
        }
    }
    return absacc;
}

// This CTA's parts of P = sum_m g_m (*) v_m, as in codes(): one (k_xc_codes, which holds a
// part's pairs), or with ALL the A.G of its sequence, part g from pair g A.PB on, so that
// either way a part is the same sum in the same order and solve() adds the same parts.  A
// part's pairs of a row block sit in neighbouring lanes: the sum over them is a few shuffles.
template <bool ALL>
__device__ __forceinline__ void convolve(const Args& A, const float4* gs, const float2* Vs, float* P, int Mr) {
    constexpr int R = kR;
    const int NB = A.NB, Lg = A.Lg, B = A.PB, CG = A.PCG, GB = ALL ? A.B : B;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int p = lane % B, cl = lane / B;
    const int pg2 = B >= 16 ? 16 : B >= 8 ? 8 : B >= 4 ? 4 : B >= 2 ? 2 : 1;
    const int passes = (A.nchunk + CG - 1) / CG;                      // over a part's row blocks
    for (int it = warp; it < (ALL ? A.G : 1) * passes; it += nwarps) {
        const int part = ALL ? it / passes : 0, pr = part * B + p;
        const int q = (it - part * passes) * CG + cl;
        const bool lane_on = cl < CG && 2 * pr < Mr;
        f32x2 acc[R];
#pragma unroll
        for (int i = 0; i < R; ++i) acc[i] = 0;
        if (lane_on && q < A.nchunk) {
            const f32x2* v = reinterpret_cast<const f32x2*>(Vs + pr * A.pitch + 17 * (q + NB));
            f32x2 w[R];
#pragma unroll
            for (int i = 0; i < R; ++i) w[i] = v[i];
            const ulonglong2* gb = reinterpret_cast<const ulonglong2*>(gs) + pr;
#pragma unroll 1
            for (int b = 0; b < NB; ++b, gb += 8 * GB) {
                v -= 17;
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    const ulonglong2 gg = gb[(j >> 1) * GB];
#pragma unroll
                    for (int i = 0; i < R; ++i) acc[i] = ffma2(gg.x, w[(i - j) & 15], acc[i]);
                    w[(-j - 1) & 15] = v[15 - j];
#pragma unroll
                    for (int i = 0; i < R; ++i) acc[i] = ffma2(gg.y, w[(i - j - 1) & 15], acc[i]);
                    w[(-j - 2) & 15] = v[14 - j];
                }
            }
        }
        // over the pairs: lanes p >= pg2 first, then halves of the 16 rows in turn
        float s[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const float2 a = unpack(acc[i]);
            s[i] = a.x + a.y;
        }
        if (B > pg2) {
            const bool take = p + pg2 < B;
            const int from = take ? lane + pg2 : lane;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const float o = __shfl_sync(0xffffffffu, s[i], from & 31);
                if (take) s[i] += o;
            }
        }
        int off = 0, cnt = R;
#pragma unroll
        for (int h = 8; h >= 1; h >>= 1) {
            const int x = pg2 * h / 16;                     // rows 2h -> h: lanes p and p ^ x
            if (x >= 1) {
                const bool hi = (p & x) != 0;
                const int from = (lane - p + (p ^ x)) & 31;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (k >= h) break;
                    const float send = hi ? s[k] : s[k + h];
                    const float keep = hi ? s[k + h] : s[k];
                    s[k] = keep + __shfl_sync(0xffffffffu, send, from);
                }
                off += hi ? h : 0;
                cnt = h;
            }
        }
        if (cl < CG && p < pg2 && q < A.nchunk) {
            float* Pt = P + (size_t)part * Lg;
            const int l = R * q + off;
#pragma unroll
            for (int k = 0; k < R; ++k)
                if (k < cnt && l + k < Lg) Pt[l + k] = s[k];
        }
    }
}

// the taps of a CTA's filters and W of a sequence in codes()'s layouts
__device__ __forceinline__ void load_taps(const Args& A, float4* gs, int m0, int Mr) {
    for (int t = threadIdx.x; t < 8 * A.NB * A.B; t += blockDim.x) {
        const int j = 2 * (t / A.B), p = t % A.B;
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int tap = j + (e >> 1), m = 2 * p + (e & 1);
            v[e] = tap < A.T && m < Mr ? A.G1[(size_t)(m0 + m) * A.Lg + tap] : 0.f;
        }
        gs[t] = make_float4(v[0], v[1], v[2], v[3]);
    }
}
__device__ __forceinline__ void load_w(const Args& A, float4* ws, size_t c) {
    const float4* Wg = reinterpret_cast<const float4*>(A.W + c * A.Lg);
    for (int i = threadIdx.x; i < A.Lg / 4; i += blockDim.x) {
        const float4 w = Wg[i];
        const float4 lo = make_float4(w.x, w.x, w.y, w.y), hi = make_float4(w.z, w.z, w.w, w.w);
        float4* d = ws + 2 * i + (i >> 2);
        d[0] = lo;
        d[1] = hi;
        if (i < 4 * A.NB) {
            const int k = i + A.Lg / 4;
            d = ws + 2 * k + (k >> 2);
            d[0] = lo;
            d[1] = hi;
        }
    }
}

// the CTA's sum of v, by thread 0
__device__ __forceinline__ void block_sum(double v, double* out) {
    __shared__ double red[kMaxThreads / 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        *out = t;
    }
}

// waits for the launches this one depends on (it is launched while the last one's CTAs
// finish), and lets the next launch do the same
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <int MODE>
__global__ void __launch_bounds__(kMaxThreads, 2) k_xc_codes(const __grid_constant__ Args A) {
    extern __shared__ float4 smem4[];
    float4* gs = smem4;
    float4* ws = gs + 8 * A.NB * A.B;
    float2* Vs = reinterpret_cast<float2*>(ws + 9 * (A.nchunk + A.NB));
    const size_t c = blockIdx.x / A.G, n = A.n0 + c;
    const int g = blockIdx.x % A.G, m0 = g * 2 * A.B, Mr = min(2 * A.B, A.M - m0);
    load_taps(A, gs, m0, Mr);           // G1 is older than the launch before this one
    after_previous();
    // this CTA's rows towards L2 while it convolves (hints; a row is a multiple of 16 bytes)
    if (MODE != FIRST && threadIdx.x >= blockDim.x - 32) {
        const size_t r0 = (n * A.M + m0) * A.Lg;
        for (int k = threadIdx.x & 31; k < 2 * Mr; k += 32) {
            const float* a = (k < Mr ? A.V : A.y3) + r0 + (size_t)(k % Mr) * A.Lg;
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(a), "r"(4 * A.Lg) : "memory");
        }
    }
    if (MODE != FIRST) load_w(A, ws, c);
    __syncthreads();
    const double s = codes<MODE>(A, gs, ws, Vs, n, m0, Mr);
    __syncthreads();
    if (MODE == LAST) block_sum(s, A.absx_part + n * A.G + g);
    else convolve<false>(A, gs, Vs, A.P + (c * A.G + g) * A.Lg, Mr);
}

__global__ void __launch_bounds__(256) k_xc_solve(const __grid_constant__ Args A) {
    extern __shared__ float4 smem4[];
    const size_t c = blockIdx.x, n = A.n0 + c;
    after_previous();
    if (threadIdx.x < 2) {
        // what the end reads, towards L2 (hints; rows are multiples of 16 bytes)
        const float* a = threadIdx.x == 0 ? A.y1 + n * A.Lg : A.S + n * A.L4;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;"
                     :: "l"(a), "r"(threadIdx.x == 0 ? 4 * A.Lg : 4 * A.L4) : "memory");
    }
    solve(A, reinterpret_cast<float2*>(smem4), c, n, A.first, A.last);
}

// all X-steps of one sequence by one CTA that holds all its filters: no launch between the
// parts, and what they leave in global memory is found in the caches
__global__ void __launch_bounds__(kMaxThreads, 2) k_xc_all(const __grid_constant__ Args A) {
    extern __shared__ float4 smem4[];
    float4* gs = smem4;
    float4* ws = gs + 8 * A.NB * A.B;
    float2* Vs = reinterpret_cast<float2*>(ws + 9 * (A.nchunk + A.NB));
    const size_t n = blockIdx.x;
    load_taps(A, gs, 0, A.M);
    __syncthreads();
    for (int it = 0; it < A.iters; ++it) {
        if (it == 0) {
            codes<FIRST>(A, gs, ws, Vs, n, 0, A.M);
        } else {
            load_w(A, ws, n);
            __syncthreads();
            codes<MID>(A, gs, ws, Vs, n, 0, A.M);
        }
        __syncthreads();
        convolve<true>(A, gs, Vs, A.P + n * A.G * A.Lg, A.M);
        __syncthreads();
        solve(A, Vs, n, n, it == 0, it == A.iters - 1);      // the transform in V's place
        __syncthreads();
    }
    load_w(A, ws, n);
    __syncthreads();
    block_sum(codes<LAST>(A, gs, ws, Vs, n, 0, A.M), A.absx_part + n);
}

// The smallest n >= Lg of the form {1, 3, 5, 9, 15, 25} 2^a and its stages: the odd
// radices first (at most two, so that every later sub-length is a power of two), then 8,
// with one 4 or 2 or two 4s to finish.
int transform_length(int Lg, int* radix, int* nst) {
    int best = 0, odd = 1;
    for (int c : {1, 3, 5, 9, 15, 25}) {
        int v = 16 * c;
        while (v < Lg) v *= 2;
        if (!best || v < best) { best = v; odd = c; }
    }
    int k = 0, p2 = 0;
    for (int c = odd; c > 1;) {
        const int r = c % 5 == 0 ? 5 : 3;
        radix[k++] = r;
        c /= r;
    }
    for (int v = best / odd; v > 1; v /= 2) ++p2;
    while (p2 > 0) {
        const int b = p2 == 4 || p2 == 2 ? 2 : p2 >= 3 ? 3 : 1;
        radix[k++] = 1 << b;
        p2 -= b;
    }
    *nst = k;
    return best;
}

// The tables of a transform length and Lg, in double then rounded.
struct Tables {
    float2* tw;
    float2* wk;
    ushort2* pos;
    double* cosL;           // cos(2 pi t / Lg), t < Lg
    double* cosN;           // cos(pi t / n), t < 2n
    int n, nst, Lg;
    int radix[kMaxStages], twoff[kMaxStages];
};
__global__ void k_tables(const __grid_constant__ Tables T) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, n = T.n;       // 2n threads
    double s, c;
    if (t < 2 * n) T.cosN[t] = cospi((double)t / n);
    for (int u = t; u < T.Lg; u += gridDim.x * blockDim.x) T.cosL[u] = cospi(2.0 * u / T.Lg);
    if (t <= n / 2) {
        sincospi((double)t / n, &s, &c);
        T.wk[t] = make_float2((float)c, (float)-s);
        // bin k leaves the stages at sum_i q_i m_i for k = q_0 + r_0 (q_1 + r_1 (...))
        int at[2], k[2] = {t, (n - t) % n};
        for (int b = 0; b < 2; ++b) {
            int m = n;
            at[b] = 0;
            for (int st = 0; st < T.nst; ++st) {
                m /= T.radix[st];
                at[b] += (k[b] % T.radix[st]) * m;
                k[b] /= T.radix[st];
            }
        }
        T.pos[t] = make_ushort2((unsigned short)at[0], (unsigned short)at[1]);
    }
    int m = n;
    for (int st = 0; st < T.nst; ++st) {
        const int sl = m / T.radix[st], e = t - T.twoff[st];
        if (e >= 0 && e < (T.radix[st] - 1) * sl) {
            const int q = e / sl + 1, o = e % sl;
            sincospi(2.0 * ((double)o * q) / m, &s, &c);
            T.tw[t] = make_float2((float)c, (float)-s);
        }
        m = sl;
    }
}

// h[d] = (1/Lg) sum_f r[f] cos(2 pi f d / Lg) over all Lg bins, r = 1 / (k + A); a block per d
__global__ void k_solve_kernel(const float* __restrict__ Ah, const double* __restrict__ cosL,
                               double* __restrict__ h, int Lg, double kc) {
    __shared__ double sh[4];
    const int d = blockIdx.x, half = Lg / 2;
    double a = 0.0;
    for (int f = threadIdx.x; f <= half; f += blockDim.x) {
        const double r = 1.0 / (kc + (double)Ah[f]);
        const unsigned k = (unsigned)f * (unsigned)d % (unsigned)Lg;
        a += (f == 0 || f == half ? r : 2.0 * r) * cosL[k];
    }
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) h[d] = ((sh[0] + sh[1]) + (sh[2] + sh[3])) / Lg;
}

// The kernel's spectrum at bins k and n - k of the length 2n, as half sum and half
// difference over n (h reaches Lg/2 on both sides, that last value split between them)
__global__ void k_solve_spectrum(const double* __restrict__ h, const double* __restrict__ cosN,
                                 float2* __restrict__ Hsd, int Lg, int n) {
    __shared__ double sh[4][2];
    const int k = blockIdx.x, half = Lg / 2;
    double a = 0.0, b = 0.0;
    for (int d = threadIdx.x; d <= half; d += blockDim.x) {
        const double v = d == 0 || d == half ? h[d] : 2.0 * h[d];
        a += v * cosN[(unsigned)k * (unsigned)d % (2u * n)];
        b += v * cosN[(unsigned)(n - k) * (unsigned)d % (2u * n)];
    }
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) { sh[threadIdx.x >> 5][0] = a; sh[threadIdx.x >> 5][1] = b; }
    __syncthreads();
    if (threadIdx.x == 0) {
        a = (sh[0][0] + sh[1][0]) + (sh[2][0] + sh[3][0]);
        b = (sh[0][1] + sh[1][1]) + (sh[2][1] + sh[3][1]);
        Hsd[k] = make_float2((float)(0.5 * (a + b) / n), (float)(0.5 * (a - b) / n));
    }
}


struct Shape {
    int NB, G, B, CG, nchunk, pitch, threads;
    size_t smem, smem_all;
};

struct XconvPlan {
    Shape s;
    int G, PB, PCG;         // the parts of P: k_xc_codes's CTAs, in either form
    int n, nst, radix[kMaxStages], twoff[kMaxStages];
    int chunk, solve_threads;
    size_t solve_smem;
    bool all;               // k_xc_all
    float2* tw;
    float2* wk;
    ushort2* pos;
    float2* Hsd;
    double* cosL;           // cos(2 pi t / Lg), t < Lg
    double* cosN;           // cos(pi t / n), t < 2n
    double* h;              // [Lg/2 + 1] the solve's circular kernel
    double* absx_part;      // [N][s.G]
    int absx_n;
};

// the layout with at most B pairs per CTA
Shape shape_for(int Lg, int M, int T, int B, int n) {
    Shape s;
    const int pairs = (M + 1) / 2;
    s.NB = (T + 15) / 16;
    s.G = (pairs + B - 1) / B;
    s.B = (pairs + s.G - 1) / s.G;                  // as even as it goes
    s.CG = 32 / s.B;
    s.nchunk = (Lg + 15) / 16;
    const int warps = (s.nchunk + s.CG - 1) / s.CG, most = kMaxThreads / 32;
    const int loops = (warps + most - 1) / most;
    s.threads = 32 * ((warps + loops - 1) / loops);
    const size_t blocks = (size_t)s.nchunk + s.NB;
    static const int residue[17] = {0, 1, 8, 6, 4, 3, 3, 2, 2, 1, 1, 1, 1, 1, 1, 1, 1};
    s.pitch = (int)(17 * blocks);
    while (s.pitch % 16 != residue[s.B]) ++s.pitch;
    const size_t fixed = (size_t)8 * s.NB * s.B * 16 + 9 * blocks * 16, places = (size_t)s.B * s.pitch;
    s.smem = fixed + places * 8;
    s.smem_all = fixed + std::max(places, (size_t)n + n / 16 + 1) * 8;
    return s;
}

// k_xc_codes takes up to 5 pairs per CTA, fewer while two CTAs do not fit an SM's shared
// memory.  Measured (ms for 15 X-steps): N=1500, L=137, M=25, W=9: 2.76 at 4 pairs per
// CTA, 2.98 at 7, 3.04 at 13; N=5000, L=500, M=32, W=16: 35.6 at 4, 40.9 at 2, 54 at 8 (one
// CTA per SM); N=500, L=1000: 8.5 at 2, 10.3 at 1, 10.8 at 4 (one per SM).
bool choose_shape(int Lg, int M, int T, int n, Shape* s) {
    for (int B = 5; B >= 1; --B) {
        *s = shape_for(Lg, M, T, B, n);
        if (2 * (s->smem + 1024) <= kSmemSm) return true;
    }
    return s->smem <= kSmemCta;
}

void free_arrays(cdlgb_ctx* c, XconvPlan* P) {
    dev_free(c, P->tw);
    dev_free(c, P->wk);
    dev_free(c, P->pos);
    dev_free(c, P->Hsd);
    dev_free(c, P->cosL);
    dev_free(c, P->cosN);
    dev_free(c, P->h);
    dev_free(c, P->absx_part);
}

}  // namespace

// Whether the automatic choice (fft_mode 0; 1 and 2 ask for the transforms) may take this
// X-step for a context.  CDLGB_XCONV=0 and the switches that pick an FFT form leave it out.
static bool xconv_allowed(const cdlgb_ctx* c) {
    const int T = 4 * c->p.filter_size, TP = (T + 15) / 16 * 16;
    if (c->p.fft_mode != 0 || T > kMaxTaps || c->Lg % 4 || c->Lg > kMaxLg || c->Lg < TP) return false;
    if (getenv("CDLGB_GENERIC_FFT")) return false;
    for (const char* v : {"CDLGB_XCONV", "CDLGB_XITER"}) {
        const char* e = getenv(v);
        if (e && atoi(e) == 0) return false;
    }
    return true;
}

// Whether an allowed context takes it.  Up to 64 taps and Lg = 4128: every length without a
// multi-iteration register-FFT kernel (slots: its filter slots for all of M, 16 per CTA; else
// 0), and where those slots are empty enough, 5.5 + 0.03 T ps per filter against 4.8 per slot.
// It is the more exact form there (32 trainings of 16 sizes, after one outer iteration against
// float64: DX 2 to 20 times nearer than by the transforms, codes 2 to 6) and mostly the faster
// one; where it is not (0.76 to 0.95 of the transforms' speed: M = 8, 10 with W = 16 at L = 200;
// odd M at Lg = 496 and 928; M = 9 at Lg = 4096) the more exact one is kept.  Past those sizes
// the cheaper one is taken, by estimates in ps per X-step and code value from 2300 measured
// sizes (Lg = 40-12288, M = 1-256, T = 4-128, 2 to 6e7 code values; 15 X-steps each way).  The
// number of sequences has no say: a sequence's route, and with it its bits, must not depend
// on how many others there are.
//   * these kernels, 8 % rms: the taps, filled up to 16s, in lanes of which 1 / pad have work
//     (short rows are not bound by that); the element-wise pass; the solve, a transform per
//     sequence; 2.5 where two CTAs per SM leave each one pair of filters, 6 where one CTA
//     fits.  M = 32, T = 64: 6.6 measured at Lg = 512, 7.3 at 2048, 8.7 at 4224, 10.1 at 5120,
//     12.6 at 8192; M = 9: 9.5, 9.9, 11.2, 10.9, 14.3;
//   * the multi-iteration register-FFT kernel, per slot: 4.5-5.0, 4.8-5.6 with three CTAs or
//     more, 4.2-4.8 up to 8 filters in one, 3.6-4.0 with 32 lanes per transform.  A tenth less
//     is granted, which these kernels lose with a few hundred sequences;
//   * the other transforms, from below: the one-X-step register FFTs (M = 33: 7.5, 17: 7.9, 9:
//     8.4, 5: 9.7); the in-kernel mixed radix (10.0 at Lg = 1024, 11-19 elsewhere, 15 and more
//     at M = 5); cuFFT by the largest prime factor of Lg (M = 32: 9.5 at 2048 and 4096; 12.2-19
//     up to 19; 14.7-24 up to 47; 21-65 past it).
static bool xconv_wanted(const cdlgb_ctx* c, const Shape& s, int n, int slots) {
    const int T = 4 * c->p.filter_size, Lg = c->Lg;
    const double M = c->M;
    const bool empty = (c->M + 1) / 2 * 2 * (5.5 + 0.03 * T) < 4.8 * slots;
    if (T <= 64 && Lg <= 4128) return slots == 0 || empty;
    double pad = 64.0 * s.G * ((s.nchunk + s.CG - 1) / s.CG) / (s.nchunk * M);
    if (Lg < 320) pad = std::min(pad, 1.5);
    const bool two = 2 * (s.smem + 1024) <= kSmemSm;
    const double room = !two ? 6.0 : s.B == 1 && c->M > 2 ? 2.5 : 0.0;
    const double conv = 1.3 + pad * (1.63 + 0.0594 * 16 * s.NB) + 16.0 * n / (Lg * M) + room;
    if (slots) {
        const double per_slot = c->M > 8 ? (slots <= 32 ? 4.0 : 4.4) : Lg < 520 ? 4.0 : 3.4;
        return empty && conv < per_slot * slots / M;
    }
    int odd = Lg, most = 1;
    while (odd % 2 == 0) odd /= 2;
    for (int p = 3; odd > 1; p += 2)
        for (; odd % p == 0; odd /= p) most = p;
    double fft;
    if (fused_one_step_regs(c)) fft = 7.2 + 10 / M + 9 / (M * M);
    else if (c->fused) fft = (Lg == 1024 ? 10.0 : 11.5) + (c->M < 9 ? 15 / M + 15 / (M * M) : 0.0);
    else if (most == 1) fft = 8.5 + 8.5 / M;
    else fft = (most <= 19 ? 11.0 : most <= 47 ? 14.0 : 20.0) + 11 / M;
    return conv < fft;
}

void* xconv_plan_create(cdlgb_ctx* c, int slots, int* status) {
    *status = CDLGB_OK;
    if (!xconv_allowed(c)) return nullptr;
    const int Lg = c->Lg;
    XconvPlan* P = new XconvPlan();
    P->n = transform_length(Lg, P->radix, &P->nst);
    const int n = P->n;
    P->solve_smem = (size_t)(n + n / 16 + 1) * sizeof(float2);
    P->solve_threads = n <= 512 ? 64 : n <= 1536 ? 128 : 256;
    const int T = 4 * c->p.filter_size;
    if (P->solve_smem > kSmemCta || !choose_shape(Lg, c->M, T, n, &P->s) || !xconv_wanted(c, P->s, n, slots)) {
        delete P;
        return nullptr;
    }
    P->G = P->s.G;
    P->PB = P->s.B;
    P->PCG = P->s.CG;
    // the parts of P lie in the cuFFT passes' scratch
    P->chunk = (int)std::min<size_t>((size_t)c->chunk * c->M / P->G, c->N);
    // One CTA per sequence (M <= 32) where that keeps every sequence resident and a
    // sequence's work, one CTA's chain, is short.  15 X-steps of 30 sequences, so and with a
    // launch per part: 0.17 and 0.27 ms at Lg = 436, M = 16, T = 16 (0.4 million in the rule's
    // units), 0.47 / 0.44 at 1060, 16, 64 (1.9), 0.59 / 0.45 at 1456, 32, 16 (3.0), 1.18 / 0.72
    // at 4096, 9, 64 (4.1); of 200 sequences: 0.51 / 0.61 at 1456, 16, 16 (1.5).
    P->all = false;
    if (c->M <= 32 && P->chunk == c->N && (long long)c->M * Lg * (48 + T) <= 2000000) {
        Shape a = shape_for(Lg, c->M, T, 16, n);
        // as few warps as finish both passes (codes, parts of P) in the fewest rounds
        const int codes_n = (a.nchunk + a.CG - 1) / a.CG, parts_n = P->G * ((a.nchunk + P->PCG - 1) / P->PCG);
        const auto rounds = [&](int w) { return (codes_n + w - 1) / w + (parts_n + w - 1) / w; };
        int warps = kMaxThreads / 32;
        for (int w = warps; w >= 1; --w)
            if (rounds(w) <= rounds(warps)) warps = w;
        a.threads = 32 * warps;
        int per_sm = 0;
        if (a.smem_all <= kSmemCta &&
            (cudaFuncSetAttribute(k_xc_all, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCta) != cudaSuccess ||
             cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_xc_all, a.threads, a.smem_all) != cudaSuccess)) {
            cudaGetLastError();
            per_sm = 0;
        }
        P->all = c->N <= per_sm * c->nsm;
        if (P->all) P->s = a;
    }
    P->absx_n = c->N * P->s.G;
    Tables t = {};
    t.n = n;
    t.nst = P->nst;
    t.Lg = Lg;
    for (int st = 0, m = n, off = 0; st < P->nst; ++st) {
        P->twoff[st] = off;
        m /= P->radix[st];
        off += (P->radix[st] - 1) * m;
        t.radix[st] = P->radix[st];
        t.twoff[st] = P->twoff[st];
    }
    cudaError_t e = dev_malloc(c, (void**)&P->tw, (size_t)n * sizeof(float2));
    if (e == cudaSuccess) e = dev_malloc(c, (void**)&P->wk, (size_t)(n / 2 + 1) * sizeof(float2));
    if (e == cudaSuccess) e = dev_malloc(c, (void**)&P->pos, (size_t)(n / 2 + 1) * sizeof(ushort2));
    if (e == cudaSuccess) e = dev_malloc(c, (void**)&P->cosL, (size_t)Lg * sizeof(double));
    if (e == cudaSuccess) e = dev_malloc(c, (void**)&P->cosN, (size_t)2 * n * sizeof(double));
    if (e == cudaSuccess) e = dev_malloc(c, (void**)&P->h, (size_t)(Lg / 2 + 1) * sizeof(double));
    if (e == cudaSuccess) e = dev_malloc(c, (void**)&P->Hsd, (size_t)(n / 2 + 1) * sizeof(float2));
    if (e == cudaSuccess) e = dev_malloc(c, (void**)&P->absx_part, (size_t)P->absx_n * sizeof(double));
    // process-wide per kernel: the same cap for every context
    for (auto k : {k_xc_codes<FIRST>, k_xc_codes<MID>, k_xc_codes<LAST>, k_xc_solve})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCta);
    if (e == cudaSuccess) {
        t.tw = P->tw; t.wk = P->wk; t.pos = P->pos; t.cosL = P->cosL; t.cosN = P->cosN;
        k_tables<<<(2 * n + 127) / 128, 128, 0, c->stream>>>(t);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        *status = cdlgb_seterr(c, CDLGB_ECUDA, "convolution X-step setup failed: %s", cudaGetErrorString(e));
        free_arrays(c, P);
        delete P;
        return nullptr;
    }
    return P;
}

void xconv_plan_free(cdlgb_ctx* c, void* p) {
    XconvPlan* P = (XconvPlan*)p;
    if (!P) return;
    free_arrays(c, P);
    delete P;
}

int xconv_plan_parts(void* p) { return ((XconvPlan*)p)->s.G; }
int xconv_plan_filters(void* p) { return 2 * ((XconvPlan*)p)->s.B; }

// a launch that may start while the previous one finishes (griddepcontrol.wait in the kernel)
static cudaError_t launch_after(cdlgb_ctx* c, void (*k)(Args), unsigned grid, int threads, size_t smem,
                                const Args& a) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, a);
}

// `iters` X-steps over the first Nlim sequences
int xconv_xsteps(cdlgb_ctx* c, void* p, const float* Xin, float* Xout, int iters, int Nlim) {
    XconvPlan* P = (XconvPlan*)p;
    const Shape& s = P->s;
    k_solve_kernel<<<c->Lg / 2 + 1, 128, 0, c->stream>>>(c->Ah, P->cosL, P->h, c->Lg,
                                                         (double)c->p.sherman_const_csc);
    LAUNCH_CHECK(c, "k_solve_kernel");
    k_solve_spectrum<<<P->n / 2 + 1, 128, 0, c->stream>>>(P->h, P->cosN, P->Hsd, c->Lg, P->n);
    LAUNCH_CHECK(c, "k_solve_spectrum");
    Args a = {};
    a.Xin = Xin; a.V = Xout; a.y2 = c->y2; a.y3 = c->y3;
    a.Y1 = c->Y1; a.y1 = c->y1; a.DX = c->DX; a.S = c->S; a.G1 = c->G1;
    a.P = c->sA; a.W = reinterpret_cast<float*>(c->sVh); a.U = c->sU;
    a.absx_part = P->absx_part;
    a.tw = P->tw; a.wk = P->wk; a.pos = P->pos; a.Hsd = P->Hsd;
    a.M = c->M; a.Lg = c->Lg; a.L4 = c->L4; a.gamma = c->gamma; a.iters = iters;
    a.T = 4 * c->p.filter_size; a.G = P->G; a.PB = P->PB; a.PCG = P->PCG;
    a.lam = c->p.lambda; a.rho = c->p.rho; a.kc = c->p.sherman_const_csc;
    a.NB = s.NB; a.B = s.B; a.CG = s.CG; a.nchunk = s.nchunk; a.pitch = s.pitch;
    a.n = P->n; a.nst = P->nst; a.zero = c->zero_duals;
    for (int i = 0; i < P->nst; ++i) { a.radix[i] = P->radix[i]; a.twoff[i] = P->twoff[i]; }
    // the fused kernel's timer, in X-steps, where a fused form exists for the size
    if (c->fused) cdlgb_phase_begin(c, PH_XFUSED);
    if (P->all) {
        k_xc_all<<<(unsigned)Nlim, s.threads, s.smem_all, c->stream>>>(a);
        LAUNCH_CHECK(c, "k_xc_all");
    }
    for (int n0 = P->all ? Nlim : 0; n0 < Nlim; n0 += P->chunk) {
        const int cn = std::min(P->chunk, Nlim - n0);
        a.n0 = n0;
        for (int it = 0; it <= iters; ++it) {
            CU_TRY(c, launch_after(c, it == 0 ? k_xc_codes<FIRST> : it < iters ? k_xc_codes<MID> : k_xc_codes<LAST>,
                                   (unsigned)cn * s.G, s.threads, s.smem, a));
            LAUNCH_CHECK(c, "k_xc_codes");
            if (it == iters) break;
            a.first = it == 0;
            a.last = it == iters - 1;
            CU_TRY(c, launch_after(c, k_xc_solve, (unsigned)cn, P->solve_threads, P->solve_smem, a));
            LAUNCH_CHECK(c, "k_xc_solve");
        }
    }
    if (c->fused) cdlgb_phase_end_n(c, PH_XFUSED, iters);
    return CDLGB_OK;
}

int xconv_absx(void* p, const double** part, int* n) {
    XconvPlan* P = (XconvPlan*)p;
    *part = P->absx_part;
    *n = P->absx_n;
    return 1;
}
