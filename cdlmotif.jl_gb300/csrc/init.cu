// The initial state of a training (CDL_setup, src/CDL/CDL_setup.jl:180-230): the drawn
// dictionary, and in one pass the drawn codes, their reconstruction DX = sum_m d_m (*) x_m
// and sum |X|.
//
// X is zero off the rows l % 4 == 0 and a filter off its first T = 4W rows, so with x the
// kept rows (La = Lg / 4 of them) and four taps g[b][0..3] per base
//   DX[4a + r] = sum_m sum_{b < W} g_m[b][r] x_m[a - b]         (circular in a)
// is a short convolution: a CTA draws a range of a sequence's codes filter by filter,
// writes them and convolves them from shared memory.  The transforms of all codes that
// gave DX before (their spectra written and read, N M Lg / 2 complex values, and X read
// back) are not formed.
#include "cdlgb_internal.h"
#include "regfft.cuh"

#include <math.h>
#include <algorithm>

namespace {

constexpr int kNT = 256, kWarps = kNT / 32;
constexpr int kRows = 8;                // consecutive a per thread
constexpr int kTaps = 256;              // taps (bases) per pass over a range, at most
constexpr int kPart = 152 * 8;          // partial sums of |X|, at most

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// standard normal of a counter: Box-Muller on two 53-bit uniforms
__device__ double normal(uint64_t seed, uint64_t i) {
    const uint64_t h = splitmix64(seed * 0x2545F4914F6CDD1Dull ^ (i + 0x9E37ull));
    const double u1 = ((double)(h >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    const uint64_t h2 = splitmix64(h);
    const double u2 = ((double)(h2 >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    return sqrt(-2.0 * log(u1)) * cos(2.0 * M_PI * u2);
}

// D0: filter m's first T rows standard normal, scaled to norm 1, zero elsewhere
// (CDL_setup.jl:182-183), into the four arrays that start as D0.  A block per filter; row l
// draws from counter m T + l.  On the host the M T draws were a serial stretch before the
// first dependent launch, and the LM rows a copy.
__global__ void k_init_d(uint64_t seed, int Lg, int T, float* __restrict__ a, float* __restrict__ b,
                         float* __restrict__ c, float* __restrict__ d) {
    __shared__ double sh[kWarps];
    const uint64_t at = (uint64_t)blockIdx.x * T;
    const size_t row = (size_t)blockIdx.x * Lg;
    double mine = 0.0, sq = 0.0;
    for (int l = threadIdx.x; l < T; l += kNT) {
        const double v = normal(seed, at + l);
        if (l < kNT) mine = v;
        sq += v * v;
    }
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = sq;
    __syncthreads();
    double norm = 0.0;
    for (int w = 0; w < kWarps; ++w) norm += sh[w];
    norm = sqrt(norm);
    for (int l = threadIdx.x; l < Lg; l += kNT) {
        const float v = l >= T ? 0.f : (float)((l < kNT ? mine : normal(seed, at + l)) / norm);
        a[row + l] = b[row + l] = c[row + l] = d[row + l] = v;
    }
}

struct XArgs {
    float4* X;              // (N, M, La)
    const float4* G1;       // (M, La): taps b < W, zero after them
    float4* DX;             // (N, La)
    float4* G2;
    double* out;            // per CTA sum |X|
    uint64_t seed;
    int N, M, La, W;
    int nr, RA;             // ranges of a sequence, a per range (a multiple of kRows)
    int nq, ms;             // threads along a range, along the filters
    int MG, pitch;          // filters per pass, places per filter in shared memory
};

__device__ __forceinline__ int place(int i) { return (i >> 3) * 12 + (i & 7); }
__device__ __forceinline__ unsigned long long twice(float x) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ unsigned long long pair(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ unsigned long long ffma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float2 unpack(unsigned long long a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}

// X (CDL_setup.jl:191-192): standard normal on the rows l % 4 == 0, float4 j of (N, M, La)
// from counter 4 j of the seed's splitmix64 stream (Box-Muller on two 24-bit uniforms); a
// given X is masked to those rows instead (!DRAW).  DX and G2 = DX (CDL_setup.jl:197-203).
//
// A CTA takes ranges of RA values of a of one sequence, MG filters at a time: each warp
// fills whole rows (with the values before the range that the taps reach, drawn again),
// then a thread convolves kRows values of a, all four r, with every ms-th filter's taps,
// eight packed FMAs per row of taps and value.  The ms partial results meet in shared
// memory.  The row blocks of 8 values sit 12 places apart: 16-byte loads of neighbouring
// threads' blocks spread over the banks.
template <bool DRAW>
__global__ void __launch_bounds__(kNT, 3) k_init_x(XArgs A) {
    extern __shared__ float4 sm4[];
    __shared__ double sh[kWarps];
    float* xs = reinterpret_cast<float*>(sm4);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = threadIdx.x % A.nq, mi = threadIdx.x / A.nq;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const size_t items = (size_t)A.N * A.nr;
    float s = 0.f, sc = 0.f;
    double total = 0.0, rest = 0.0;
    for (size_t item = blockIdx.x; item < items; item += gridDim.x) {
        const size_t n = item / A.nr;
        const int a0 = (int)(item - n * A.nr) * A.RA, an = min(A.RA, A.La - a0);
        unsigned long long acc[kRows][2];
#pragma unroll
        for (int i = 0; i < kRows; ++i) acc[i][0] = acc[i][1] = 0;
        for (int m0 = 0; m0 < A.M; m0 += A.MG) {
            const int mg = min(A.MG, A.M - m0);
            for (int t0 = 0; t0 < A.W; t0 += kTaps) {
                const int taps = min(kTaps, A.W - t0), Hp = (taps + 7) & ~7;
                __syncthreads();                           // the previous pass has read xs
                for (int mm = warp; mm < mg; mm += kWarps) {
                    const size_t row = (n * A.M + m0 + mm) * A.La;
                    for (int i = lane; i < A.nq * kRows + Hp; i += 32) {
                        float v = 0.f;
                        if (i - Hp < an) {
                            int a = a0 + i - Hp - t0;
                            while (a < 0) a += A.La;
                            const size_t j = row + a;
                            if (DRAW) {
                                const uint64_t h = splitmix64(A.seed * 0x2545F4914F6CDD1Dull ^ (uint64_t)(4 * j));
                                const float u1 = ((float)(uint32_t)(h >> 40) + 0.5f) * (1.0f / 16777216.0f);
                                const float u2 = ((float)((uint32_t)h & 0xFFFFFFu) + 0.5f) * (1.0f / 16777216.0f);
                                v = sqrtf(-2.f * logf(u1)) * cospif(2.f * u2);
                            } else {
                                v = A.X[j].x;
                            }
                            if (i >= Hp && t0 == 0) {      // the range's own
                                A.X[j] = make_float4(v, 0.f, 0.f, 0.f);
                                // sum |X| (two-sum): drawn codes as a float32 pair per
                                // range, which for them has the bits of a float64 sum;
                                // given ones, of any size, as a float64 pair
                                if (DRAW) {
                                    const float x = fabsf(v), t = __fadd_rn(s, x), b = __fsub_rn(t, s);
                                    sc = __fadd_rn(sc, __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(x, b)));
                                    s = t;
                                } else {
                                    const double x = (double)fabsf(v), t = total + x, b = t - total;
                                    rest += (total - (t - b)) + (x - b);
                                    total = t;
                                }
                            }
                        }
                        xs[mm * A.pitch + place(i)] = v;
                    }
                }
                __syncthreads();
                if (mi < A.ms) {
                    for (int mm = mi; mm < mg; mm += A.ms) {
                        const float4* g = A.G1 + (size_t)(m0 + mm) * A.La + t0;
                        const float* xr = xs + mm * A.pitch;
                        const int base = Hp + kRows * q;
                        // w[4 + i - t]: x[a - b] of the thread's value i, b = k + t
                        unsigned long long w[kRows + 4];
#pragma unroll
                        for (int i = 0; i < kRows; i += 4) {
                            const float4 x = *reinterpret_cast<const float4*>(xr + place(base + i));
                            w[4 + i] = twice(x.x);
                            w[5 + i] = twice(x.y);
                            w[6 + i] = twice(x.z);
                            w[7 + i] = twice(x.w);
                        }
#pragma unroll 1
                        for (int k = 0; k < taps; k += 4) {
                            float4 gg[4];
#pragma unroll
                            for (int t = 0; t < 4; ++t) gg[t] = k + t < taps ? __ldg(g + k + t) : z;
                            const float4 x = *reinterpret_cast<const float4*>(xr + place(base - k - 4));
                            w[0] = twice(x.x);
                            w[1] = twice(x.y);
                            w[2] = twice(x.z);
                            w[3] = twice(x.w);
#pragma unroll
                            for (int t = 0; t < 4; ++t) {
                                const unsigned long long lo = pair(gg[t].x, gg[t].y), hi = pair(gg[t].z, gg[t].w);
#pragma unroll
                                for (int i = 0; i < kRows; ++i) {
                                    acc[i][0] = ffma2(lo, w[4 + i - t], acc[i][0]);
                                    acc[i][1] = ffma2(hi, w[4 + i - t], acc[i][1]);
                                }
                            }
#pragma unroll
                            for (int i = kRows + 3; i >= 4; --i) w[i] = w[i - 4];
                        }
                    }
                }
            }
        }
        // the filters' parts; 9 places per thread's 8 rows, so that the stores spread
        __syncthreads();
        float4* red = sm4;
        if (mi < A.ms) {
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const float2 lo = unpack(acc[i][0]), hi = unpack(acc[i][1]);
                red[(mi * A.nq + q) * 9 + i] = make_float4(lo.x, lo.y, hi.x, hi.y);
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < an; i += kNT) {
            const float4* r = red + (i >> 3) * 9 + (i & 7);
            float4 v = r[0];
            for (int k = 1; k < A.ms; ++k) {
                const float4 u = r[(size_t)k * A.nq * 9];
                v = make_float4(v.x + u.x, v.y + u.y, v.z + u.z, v.w + u.w);
            }
            const size_t j = n * A.La + a0 + i;
            A.DX[j] = v;
            A.G2[j] = v;
        }
        if (DRAW) total += (double)s + (double)sc;
        s = sc = 0.f;
    }
    total += rest;
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    __syncthreads();
    if (lane == 0) sh[warp] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kWarps; ++w) t += sh[w];
        A.out[blockIdx.x] = t;
    }
}

}  // namespace

int init_d(cdlgb_ctx* c, uint64_t seed) {
    k_init_d<<<(unsigned)c->M, kNT, 0, c->stream>>>(seed, c->Lg, 4 * c->p.filter_size, c->G1, c->G3, c->Dbest,
                                                    c->dsum);
    LAUNCH_CHECK(c, "k_init_d");
    return CDLGB_OK;
}

// X (drawn, or masked where it stands), DX, G2 from G1; *np partial sums of |X| in out
int init_x(cdlgb_ctx* c, float* X, bool draw, uint64_t seed, double* out, int* np) {
    XArgs a;
    a.X = (float4*)X; a.G1 = (const float4*)c->G1;
    a.DX = (float4*)c->DX; a.G2 = (float4*)c->G2; a.out = out; a.seed = seed;
    a.N = c->N; a.M = c->M; a.La = c->Lg / 4; a.W = c->p.filter_size;
    // A range per CTA: a thread per 8 values, times as many filters at a time as fill the
    // threads; a whole sequence at best.  Cut where a sequence is longer than the CTA or where
    // more than a sixth of the threads would have no work; not below 16 threads along the
    // range, where the values that are drawn twice (up to W + 7 per range) begin to count.
    // The number of sequences has no say: the cut sets ms, and with it the order of the sums
    // over the filters, and a sequence's bits must not depend on how many others there are.
    const int chunks = (a.La + kRows - 1) / kRows;
    auto used = [&](int nq) { return std::min(kNT / nq, a.M) * nq; };
    for (a.nr = (chunks + kNT - 1) / kNT;; ++a.nr) {
        const int nq = (chunks + a.nr - 1) / a.nr, next = (chunks + a.nr) / (a.nr + 1);
        if (next < 16 || used(nq) * 6 >= kNT * 5) break;
    }
    a.nq = (chunks + a.nr - 1) / a.nr;
    a.RA = a.nq * kRows;
    a.nr = (a.La + a.RA - 1) / a.RA;
    a.ms = std::max(1, std::min(kNT / a.nq, a.M));
    const int Hp = (std::min(kTaps, a.W) + 7) & ~7;
    a.pitch = (a.RA + Hp) / 8 * 12;
    // two rows of filters per part and per warp, in about a third of an SM's shared memory
    const int unit = std::max(a.ms, kWarps);
    constexpr size_t room = 72 * 1024;
    a.MG = (int)std::min<size_t>((size_t)2 * unit, std::max<size_t>(1, room / ((size_t)a.pitch * 4)));
    a.MG = std::min(a.MG, a.M);
    const size_t smem = std::max((size_t)a.MG * a.pitch * 4, (size_t)a.ms * a.nq * 9 * 16);
    auto k = draw ? k_init_x<true> : k_init_x<false>;
    int per_sm = 0;
    // process-wide per kernel: the same cap for every context (smem is at most room)
    CU_TRY(c, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room));
    CU_TRY(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kNT, smem));
    const size_t items = (size_t)a.N * a.nr;
    const int grid = (int)std::min<size_t>({items, (size_t)std::max(1, per_sm) * std::max(1, c->nsm), (size_t)kPart});
    k<<<grid, kNT, smem, c->stream>>>(a);
    LAUNCH_CHECK(c, "k_init_x");
    *np = grid;
    return CDLGB_OK;
}
