// PWM scan and count kernels (src/SEARCH/scan.jl, src/SEARCH/helpers.jl).
//
// Scores are summed in float32 with one rounded multiply and one rounded add per
// term (__fmul_rn / __fadd_rn: no FMA contraction), in the order of the reference
// path being replaced, so positions and scores are bit-identical to it (REF_QUIRK_Q7):
//   greedy_search! (scan.jl:223-239): position-major, ind outer, nucleotide inner;
//   scan_n (scan.jl:10-21):           nucleotide-major, j outer, k inner.
#include "cdlgb_internal.h"

#include <math.h>
#include <algorithm>
#include <vector>

namespace {

constexpr int kScanThreads = 256;

// order-preserving reduction of (value, index): larger value wins, ties -> lower index
struct VI { float v; int i; };
__device__ __forceinline__ VI vi_best(VI a, VI b) {
    bool take_b = (b.v > a.v) || (b.v == a.v && b.i < a.i);
    return take_b ? b : a;
}
__device__ VI block_argmax(VI x, VI* sh) {
    for (int o = 16; o > 0; o >>= 1) {
        VI y;
        y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
        y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
        x = vi_best(x, y);
    }
    int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        x = lane < (int)(blockDim.x >> 5) ? sh[lane] : VI{-INFINITY, 0x7fffffff};
        for (int o = 16; o > 0; o >>= 1) {
            VI y;
            y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
            y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
            x = vi_best(x, y);
        }
        if (lane == 0) sh[0] = x;
    }
    __syncthreads();
    VI r = sh[0];
    __syncthreads();
    return r;
}

// one block per sequence n; loops over motifs k; threads over positions.
// pwms: (K, 4, maxlen) col-major; out pos: (K, N) col-major.
__global__ void k_scan_fwd(const float* __restrict__ data, const float* __restrict__ pwms,
                           const int32_t* __restrict__ lens, const float* __restrict__ thresh,
                           int K, int maxlen, int L, int32_t* __restrict__ pos) {
    extern __shared__ float xs[];      // one-hot column, 4L floats
    __shared__ VI red[32];
    const int n = blockIdx.x;
    const float* col = data + (size_t)n * 4 * L;
    for (int i = threadIdx.x; i < 4 * L; i += blockDim.x) xs[i] = col[i];
    __syncthreads();
    for (int k = 0; k < K; ++k) {
        const int w = lens[k];
        const float th = thresh[k];
        VI best{-INFINITY, 0x7fffffff};
        for (int l = threadIdx.x; l < L; l += blockDim.x) {
            float v = 0.f;
            if (l <= L - w) {
                float s = 0.f;
                for (int ind = 0; ind < w; ++ind)
#pragma unroll
                    for (int a = 0; a < 4; ++a)
                        s = __fadd_rn(s, __fmul_rn(pwms[k + K * (a + 4 * ind)], xs[(l + ind) * 4 + a]));
                v = s > th ? s : 0.f;
            }
            best = vi_best(best, VI{v, l});
        }
        VI r = block_argmax(best, red);
        // REF_QUIRK_Q3: a best hit at the first position reads as no hit (scan.jl:197)
        if (threadIdx.x == 0) pos[k + (size_t)K * n] = (r.i == 0) ? 0 : r.i + 1;
    }
}

// scan_n on both strands; complement pwm_c[j, kk] = pwm[3-j, w-1-kk] (reverse of the
// matrix).  Strict '>' from -Inf: NaN and -Inf never become the maximum.
__global__ void k_scan_both(const float* __restrict__ data, const float* __restrict__ pwms,
                            const int32_t* __restrict__ lens, const float* __restrict__ thresh,
                            int K, int maxlen, int L, int32_t* __restrict__ pos,
                            float* __restrict__ score, uint8_t* __restrict__ comp) {
    extern __shared__ float xs[];
    __shared__ VI red[32];
    const int n = blockIdx.x;
    const float* col = data + (size_t)n * 4 * L;
    for (int i = threadIdx.x; i < 4 * L; i += blockDim.x) xs[i] = col[i];
    __syncthreads();
    for (int k = 0; k < K; ++k) {
        const int w = lens[k];
        VI bf{-INFINITY, 0x7fffffff}, bc{-INFINITY, 0x7fffffff};
        for (int l = threadIdx.x; l <= L - w; l += blockDim.x) {
            float sf = 0.f, sc = 0.f;
            for (int j = 0; j < 4; ++j)
                for (int kk = 0; kk < w; ++kk) {
                    float x = xs[(l + kk) * 4 + j];
                    sf = __fadd_rn(sf, __fmul_rn(pwms[k + K * (j + 4 * kk)], x));
                    sc = __fadd_rn(sc, __fmul_rn(pwms[k + K * ((3 - j) + 4 * (w - 1 - kk))], x));
                }
            if (sf > -INFINITY) bf = vi_best(bf, VI{sf, l});
            if (sc > -INFINITY) bc = vi_best(bc, VI{sc, l});
        }
        VI rf = block_argmax(bf, red);
        VI rc = block_argmax(bc, red);
        if (threadIdx.x == 0) {
            // no candidate -> (-1, -Inf) as scan_n returns
            float sF = rf.i == 0x7fffffff ? -INFINITY : rf.v;
            float sC = rc.i == 0x7fffffff ? -INFINITY : rc.v;
            int iF = rf.i == 0x7fffffff ? -1 : rf.i + 1;
            int iC = rc.i == 0x7fffffff ? -1 : rc.i + 1;
            bool fwd = sF >= sC;
            float s = fwd ? sF : sC;
            bool keep = s > thresh[k];
            size_t o = k + (size_t)K * n;
            if (pos) pos[o] = keep ? (fwd ? iF : iC) : 0;
            if (score) score[o] = keep ? s : 0.f;
            if (comp) comp[o] = (keep && !fwd) ? 1 : 0;
        }
    }
}

// k_scan_both with the block's inputs staged once: the sequence base-major (xt[j][p],
// so consecutive positions are consecutive words), every PWM and its reverse complement
// as (fwd, comp) pairs in the order the sums consume them (pw[k][j][kk]), one position
// per thread, and the argmax of each motif reduced within each warp by shuffles (no
// barrier) and across the warps once, after the last motif.  The products and sums are
// k_scan_both's, in its order, and the (value, index) reduction is the same total order,
// so positions, scores and strands are bit-identical to it.
__global__ void k_scan_both_staged(const float* __restrict__ data, const float* __restrict__ pwms,
                                   const int32_t* __restrict__ lens, const float* __restrict__ thresh,
                                   int K, int maxlen, int L, int32_t* __restrict__ pos,
                                   float* __restrict__ score, uint8_t* __restrict__ comp) {
    extern __shared__ float4 sm4s[];
    const int nw = blockDim.x >> 5, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float2* pw = reinterpret_cast<float2*>(sm4s);                  // [K][4][maxlen]
    VI* wb = reinterpret_cast<VI*>(pw + (size_t)K * 4 * maxlen);     // [K][nw][2]
    float* xt = reinterpret_cast<float*>(wb + (size_t)K * nw * 2);  // [4][L]
    const int n = blockIdx.x;
    const float* col = data + (size_t)n * 4 * L;
    for (int i = threadIdx.x; i < 4 * L; i += blockDim.x) xt[(i & 3) * L + (i >> 2)] = col[i];
    const int per = 4 * maxlen;
    for (int i = threadIdx.x; i < K * per; i += blockDim.x) {
        const int k = i / per, r = i - k * per, j = r / maxlen, kk = r - j * maxlen;
        const int w = lens[k];
        float f = 0.f, cc = 0.f;
        if (kk < w) {
            f = pwms[k + K * (j + 4 * kk)];
            cc = pwms[k + K * ((3 - j) + 4 * (w - 1 - kk))];
        }
        pw[i] = make_float2(f, cc);
    }
    __syncthreads();
    const int l = threadIdx.x;
    for (int k = 0; k < K; ++k) {
        const int w = lens[k];
        VI bf{-INFINITY, 0x7fffffff}, bc{-INFINITY, 0x7fffffff};
        if (l <= L - w) {
            const float2* p = pw + (size_t)k * per;
            float sf = 0.f, sc = 0.f;
            for (int j = 0; j < 4; ++j) {
                const float* xr = xt + j * L + l;
                const float2* pj = p + j * maxlen;
#pragma unroll 4
                for (int kk = 0; kk < w; ++kk) {
                    const float x = xr[kk];
                    const float2 q = pj[kk];
                    sf = __fadd_rn(sf, __fmul_rn(q.x, x));
                    sc = __fadd_rn(sc, __fmul_rn(q.y, x));
                }
            }
            if (sf > -INFINITY) bf = VI{sf, l};
            if (sc > -INFINITY) bc = VI{sc, l};
        }
        for (int o = 16; o > 0; o >>= 1) {
            VI y;
            y.v = __shfl_xor_sync(0xffffffffu, bf.v, o);
            y.i = __shfl_xor_sync(0xffffffffu, bf.i, o);
            bf = vi_best(bf, y);
            y.v = __shfl_xor_sync(0xffffffffu, bc.v, o);
            y.i = __shfl_xor_sync(0xffffffffu, bc.i, o);
            bc = vi_best(bc, y);
        }
        if (lane == 0) {
            wb[((size_t)k * nw + wid) * 2] = bf;
            wb[((size_t)k * nw + wid) * 2 + 1] = bc;
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        VI rf{-INFINITY, 0x7fffffff}, rc{-INFINITY, 0x7fffffff};
        for (int v = 0; v < nw; ++v) {
            rf = vi_best(rf, wb[((size_t)k * nw + v) * 2]);
            rc = vi_best(rc, wb[((size_t)k * nw + v) * 2 + 1]);
        }
        const float sF = rf.i == 0x7fffffff ? -INFINITY : rf.v;
        const float sC = rc.i == 0x7fffffff ? -INFINITY : rc.v;
        const int iF = rf.i == 0x7fffffff ? -1 : rf.i + 1;
        const int iC = rc.i == 0x7fffffff ? -1 : rc.i + 1;
        const bool fwd = sF >= sC;
        const float sv = fwd ? sF : sC;
        const bool keep = sv > thresh[k];
        const size_t o = k + (size_t)K * n;
        if (pos) pos[o] = keep ? (fwd ? iF : iC) : 0;
        if (score) score[o] = keep ? sv : 0.f;
        if (comp) comp[o] = (keep && !fwd) ? 1 : 0;
    }
}

// ---------------------------------------------------------------- sparse scans
// On 0/1 data every term whose one-hot entry is 0 is pwm * 0 = +-0 for a finite pwm,
// and adding +-0 to a partial sum that starts at +0 leaves it unchanged (s + -0 = s for
// s != 0, +0 + -0 = +0, and the sum is never -0); a term whose entry is 1 is pwm * 1 =
// pwm.  So the sum of the nonzero terms alone, added in the reference's order, has the
// same bits: about w terms per window instead of 4 w products and sums.  Taken only
// when the data is exact 0/1 and every PWM entry finite (an infinite entry times 0 is
// NaN, which the dense kernels keep).

// the base bits of position p of the staged sequence: bit j set when entry j is 1
__device__ __forceinline__ uint32_t base_bits(const float* col, int p) {
    const float4 v = reinterpret_cast<const float4*>(col)[p];
    return (v.x != 0.f ? 1u : 0u) | (v.y != 0.f ? 2u : 0u) | (v.z != 0.f ? 4u : 0u) | (v.w != 0.f ? 8u : 0u);
}

// greedy_search! (scan.jl:223-239: position-major, nucleotide inner) on 0/1 data, one
// position per thread: for ind = 0 .. w-1 the entries of base(l + ind) in nucleotide
// order.  Same candidates and (value, index) order as k_scan_fwd.
__global__ void k_scan_fwd_sparse(const float* __restrict__ data, const float* __restrict__ pwms,
                                  const int32_t* __restrict__ lens, const float* __restrict__ thresh,
                                  int K, int maxlen, int L, int32_t* __restrict__ pos) {
    extern __shared__ float4 sm4f[];
    const int nw = blockDim.x >> 5, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float* pw = reinterpret_cast<float*>(sm4f);                    // [K][maxlen][4]
    VI* wb = reinterpret_cast<VI*>(pw + (size_t)K * 4 * maxlen);     // [K][nw]
    uint8_t* bb = reinterpret_cast<uint8_t*>(wb + (size_t)K * nw);  // [L] base bits
    const int n = blockIdx.x;
    const float* col = data + (size_t)n * 4 * L;
    for (int i = threadIdx.x; i < L; i += blockDim.x) bb[i] = (uint8_t)base_bits(col, i);
    for (int i = threadIdx.x; i < K * 4 * maxlen; i += blockDim.x) {
        const int k = i / (4 * maxlen), r = i - k * 4 * maxlen, ind = r >> 2, a = r & 3;
        pw[i] = pwms[k + K * (a + 4 * ind)];
    }
    __syncthreads();
    const int l = threadIdx.x;
    for (int k = 0; k < K; ++k) {
        const int w = lens[k];
        VI best{-INFINITY, 0x7fffffff};
        if (l < L) {
            float v = 0.f;
            if (l <= L - w) {
                const float* p = pw + (size_t)k * 4 * maxlen;
                float s = 0.f;
                for (int ind = 0; ind < w; ++ind) {
                    uint32_t b = bb[l + ind];
                    while (b) {
                        const int a = __ffs(b) - 1;
                        b &= b - 1;
                        s = __fadd_rn(s, p[4 * ind + a]);
                    }
                }
                v = s > thresh[k] ? s : 0.f;
            }
            best = VI{v, l};
        }
        for (int o = 16; o > 0; o >>= 1) {
            VI y;
            y.v = __shfl_xor_sync(0xffffffffu, best.v, o);
            y.i = __shfl_xor_sync(0xffffffffu, best.i, o);
            best = vi_best(best, y);
        }
        if (lane == 0) wb[(size_t)k * nw + wid] = best;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        VI r{-INFINITY, 0x7fffffff};
        for (int v = 0; v < nw; ++v) r = vi_best(r, wb[(size_t)k * nw + v]);
        // REF_QUIRK_Q3: a best hit at the first position reads as no hit (scan.jl:197)
        pos[k + (size_t)K * n] = (r.i == 0) ? 0 : r.i + 1;
    }
}

// scan_n on both strands (scan.jl:10-21: nucleotide-major) on 0/1 data, one position
// per thread, w <= 64 (what k_scan_lut leaves: 33 columns and more): the window's positions
// of base j are the set bits of a mask cut from the sequence's bit plane of j (built
// with one ballot per base and warp of positions), so the nonzero terms are visited j by
// j, ind ascending -- the dense order -- in one loop of exactly that many steps.  The
// (forward, complement) coefficient pairs, the per-warp argmax and the final reduction
// are k_scan_both_staged's.
__global__ void k_scan_both_sparse(const float* __restrict__ data, const float* __restrict__ pwms,
                                   const int32_t* __restrict__ lens, const float* __restrict__ thresh,
                                   int K, int maxlen, int L, int32_t* __restrict__ pos,
                                   float* __restrict__ score, uint8_t* __restrict__ comp) {
    extern __shared__ float4 sm4p[];
    const int nw = blockDim.x >> 5, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nwords = (L + 31) / 32 + 2;                           // two zero words of padding
    float2* pw = reinterpret_cast<float2*>(sm4p);                   // [K][4][maxlen]
    VI* wb = reinterpret_cast<VI*>(pw + (size_t)K * 4 * maxlen);     // [K][nw][2]
    uint32_t* planes = reinterpret_cast<uint32_t*>(wb + (size_t)K * nw * 2);   // [4][nwords]
    const int n = blockIdx.x;
    const float* col = data + (size_t)n * 4 * L;
    {
        // blockDim.x = 32 ceil(L / 32): warp w's ballots are word w of the planes
        const uint32_t bits = threadIdx.x < L ? base_bits(col, threadIdx.x) : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t b = __ballot_sync(0xffffffffu, (bits >> j) & 1u);
            if (lane == 0) planes[j * nwords + wid] = b;
        }
        if (threadIdx.x < 8) planes[(threadIdx.x >> 1) * nwords + nw + (threadIdx.x & 1)] = 0u;
    }
    const int per = 4 * maxlen;
    for (int i = threadIdx.x; i < K * per; i += blockDim.x) {
        const int k = i / per, r = i - k * per, j = r / maxlen, kk = r - j * maxlen;
        const int w = lens[k];
        float f = 0.f, cc = 0.f;
        if (kk < w) {
            f = pwms[k + K * (j + 4 * kk)];
            cc = pwms[k + K * ((3 - j) + 4 * (w - 1 - kk))];
        }
        pw[i] = make_float2(f, cc);
    }
    __syncthreads();
    const int l = threadIdx.x;
    const int wi = l >> 5, sh = l & 31;
    typedef uint64_t MT;
    constexpr int MB = 8 * (int)sizeof(MT);
    for (int k = 0; k < K; ++k) {
        const int w = lens[k];
        VI bf{-INFINITY, 0x7fffffff}, bc{-INFINITY, 0x7fffffff};
        if (l <= L - w) {
            const MT keep = w >= MB ? ~(MT)0 : (((MT)1 << w) - 1);
            MT mj[4];
            int cnt = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t* pl = planes + j * nwords + wi;
                MT m;
                if (MB == 32) {
                    m = (MT)__funnelshift_r(pl[0], pl[1], sh);
                } else {
                    const uint64_t lo = ((uint64_t)pl[1] << 32) | pl[0];
                    uint64_t m64 = lo >> sh;
                    if (sh) m64 |= (uint64_t)pl[2] << (64 - sh);
                    m = (MT)m64;
                }
                mj[j] = m & keep;
                cnt += MB == 32 ? __popc((uint32_t)mj[j]) : __popcll((unsigned long long)mj[j]);
            }
            const float2* p = pw + (size_t)k * per;
            float sf = 0.f, sc = 0.f;
            int j = 0;
            MT m = mj[0];
            for (int t = 0; t < cnt; ++t) {
                while (m == 0) {
                    ++j;
                    m = j == 1 ? mj[1] : (j == 2 ? mj[2] : mj[3]);
                }
                const int kk = (MB == 32 ? __ffs((int)(uint32_t)m) : __ffsll((long long)m)) - 1;
                m &= m - 1;
                const float2 q = p[j * maxlen + kk];
                sf = __fadd_rn(sf, q.x);
                sc = __fadd_rn(sc, q.y);
            }
            bf = VI{sf, l};
            bc = VI{sc, l};
        }
        for (int o = 16; o > 0; o >>= 1) {
            VI y;
            y.v = __shfl_xor_sync(0xffffffffu, bf.v, o);
            y.i = __shfl_xor_sync(0xffffffffu, bf.i, o);
            bf = vi_best(bf, y);
            y.v = __shfl_xor_sync(0xffffffffu, bc.v, o);
            y.i = __shfl_xor_sync(0xffffffffu, bc.i, o);
            bc = vi_best(bc, y);
        }
        if (lane == 0) {
            wb[((size_t)k * nw + wid) * 2] = bf;
            wb[((size_t)k * nw + wid) * 2 + 1] = bc;
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        VI rf{-INFINITY, 0x7fffffff}, rc{-INFINITY, 0x7fffffff};
        for (int v = 0; v < nw; ++v) {
            rf = vi_best(rf, wb[((size_t)k * nw + v) * 2]);
            rc = vi_best(rc, wb[((size_t)k * nw + v) * 2 + 1]);
        }
        const float sF = rf.i == 0x7fffffff ? -INFINITY : rf.v;
        const float sC = rc.i == 0x7fffffff ? -INFINITY : rc.v;
        const int iF = rf.i == 0x7fffffff ? -1 : rf.i + 1;
        const int iC = rc.i == 0x7fffffff ? -1 : rc.i + 1;
        const bool fwd = sF >= sC;
        const float sv = fwd ? sF : sC;
        const bool keepk = sv > thresh[k];
        const size_t o = k + (size_t)K * n;
        if (pos) pos[o] = keepk ? (fwd ? iF : iC) : 0;
        if (score) score[o] = keepk ? sv : 0.f;
        if (comp) comp[o] = (keepk && !fwd) ? 1 : 0;
    }
}

// ---------------------------------------------------------------- filtered scans
// The best window of a motif needs the exact, ordered sum at few windows only.  Every
// window gets an approximate score first, in steps of 1 / scale with scale * sum_i max_j
// |pwm[j, i]| = 32000: tables of the sum over four bases, rounded to a step, both strands
// in the halves of one integer (256 entries per four columns; the first four's entries
// hold 32768, so a sum's halves are its strands' scores + 32768 and never carry).  Sums of
// rounded entries add exactly, so an approximation is within half a step per segment of
// the real sum, and the float32 sum in any order within 0.06 steps of that: eps =
// segments / 2 + 1 steps holds.  A motif whose best approximation stays eps below its
// threshold has no hit (nine in ten at the usual p-value); else the windows within 2 eps
// of the best approximation are summed exactly, in the reference's order, and the first
// maximum among them is the first maximum of all.  Sequences with a column that is not
// one base take the exact sums for all windows.
// Instructions bound it.  N = 20000, L = 200, K = 32: 1.24 ms for both strands with the
// sparse sums of every window, 0.33 ms so (0.41 with half-precision tables, whose eps of
// 0.4 % sends a third of the motifs to the exact sums); forward, N = 10000, K = 24: 0.44, 0.15.
constexpr int kLutWarps = 16, kLutBlocks = 8;             // 32-position blocks in registers at a time
constexpr int kLutSegs = 104;                             // KB of tables per CTA (two CTAs per SM)

struct LutArgs {
    const float* data;
    const float* pwms;      // (K, 4, columns) col-major
    const int32_t* lens;
    const float* thresh;
    const int32_t* limit;   // [K] best approximations (+ 32768) from here on may hit
    const float* scale;
    int32_t* pos;
    float* score;
    uint8_t* comp;
    int K, KG, widest, L, N, words;                       // widest: columns; words: 32-position words of a sequence
};

// the larger of each 16-bit half
__device__ __forceinline__ unsigned max_halves(unsigned a, unsigned b) {
    unsigned r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// the window's exact sums (order of k_scan_both / k_scan_fwd), m: the masks of its bases,
// p: the motif, [column][base]
template <bool BOTH>
__device__ __forceinline__ float2 exact_sums(const float* __restrict__ p, int w, const unsigned (&m)[4]) {
    float2 s = make_float2(0.f, 0.f);
    if (BOTH) {
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
            unsigned b = j == 0 ? m[0] : j == 1 ? m[1] : j == 2 ? m[2] : m[3];
            for (; b; b &= b - 1) {
                const int i = __ffs((int)b) - 1;
                s.x = __fadd_rn(s.x, p[4 * i + j]);
                s.y = __fadd_rn(s.y, p[4 * (w - 1 - i) + 3 - j]);
            }
        }
    } else {
#pragma unroll 1
        for (int i = 0; i < w; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (m[j] >> i & 1) s.x = __fadd_rn(s.x, p[4 * i + j]);
    }
    return s;
}

template <bool BOTH>
__global__ void __launch_bounds__(32 * kLutWarps, 2) k_scan_lut(const __grid_constant__ LutArgs A) {
    extern __shared__ unsigned lut[];
    const int L = A.L, K = A.K, words = A.words;
    const int k0 = blockIdx.y * A.KG, k1 = min(K, k0 + A.KG);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned full = 0xffffffffu;
    // the motifs, [motif][column][base], behind the tables and the warps' planes
    const int kl = 4 * A.widest;
    int segs = 0;
    for (int k = k0; k < k1; ++k) segs += (A.lens[k] + 3) / 4;
    unsigned* planes = reinterpret_cast<unsigned*>(lut + 256 * segs) + warp * 4 * (words + 1);   // [4][words + 1]
    float* pw = reinterpret_cast<float*>(reinterpret_cast<unsigned*>(lut + 256 * segs) + kLutWarps * 4 * (words + 1));
    for (int e = threadIdx.x; e < (k1 - k0) * kl; e += blockDim.x) {
        const int k = e % (k1 - k0), r = e / (k1 - k0);               // pwms: motif fastest
        pw[k * kl + r] = A.pwms[k0 + k + (size_t)K * r];
    }
    __syncthreads();
    for (int k = k0, at = 0; k < k1; ++k) {
        const int w = A.lens[k], ns = (w + 3) / 4;
        const float* p = pw + (k - k0) * kl;
        const float sc = A.scale[k];
        for (int e = threadIdx.x; e < 256 * ns; e += blockDim.x) {
            const int i0 = e >> 8 << 2;
            float f = 0.f, c = 0.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                // base = bit q of the low nibble + 2 (bit q of the high nibble)
                const int i = i0 + q, b = (e >> q & 1) | (e >> (4 + q) & 1) << 1;
                if (i < w) {
                    f += p[4 * i + b];
                    if (BOTH) c += p[4 * (w - 1 - i) + 3 - b];
                }
            }
            const int fi = __float2int_rn(f * sc) + (i0 == 0 ? 32768 : 0), ci = __float2int_rn(c * sc) + (i0 == 0 ? 32768 : 0);
            lut[256 * at + e] = ((unsigned)ci << 16) + (unsigned)fi;
        }
        at += ns;
    }
    __syncthreads();
    for (int n = blockIdx.x * kLutWarps + warp; n < A.N; n += gridDim.x * kLutWarps) {
        const float* col = A.data + (size_t)n * 4 * L;
        bool odd = false;
        __syncwarp();
        for (int v0 = 0; v0 <= words; v0 += 4) {
            unsigned b[4];                                            // four words' loads in flight
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int l = 32 * (v0 + u) + lane;
                b[u] = l < L ? base_bits(col, l) : 0u;
                odd |= l < L && (b[u] == 0 || (b[u] & (b[u] - 1)) != 0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (v0 + u > words) break;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const unsigned m = __ballot_sync(full, b[u] >> j & 1);
                    if (lane == j) planes[j * (words + 1) + v0 + u] = m;
                }
            }
        }
        odd = __any_sync(full, odd);
        __syncwarp();
        // the masks of the 32 bases from this lane's position in word v on
        const auto masks = [&](int v, unsigned (&m)[4]) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const unsigned* pl = planes + j * (words + 1) + v;
                m[j] = __funnelshift_r(pl[0], pl[1], lane);
            }
        };
        // table indices of the windows' eight segments, a byte each
        uint2 win[kLutBlocks];
        const auto windows = [&](int v0) {
#pragma unroll
            for (int u = 0; u < kLutBlocks; ++u) {
                win[u] = make_uint2(0u, 0u);
                if (v0 + u < words) {
                    unsigned m[4];
                    masks(v0 + u, m);
                    const unsigned lo = m[1] | m[3], hi = m[2] | m[3];
                    const auto nibbles = [](unsigned x) {             // 16 bits -> a nibble per byte
                        x = (x | x << 8) & 0x00ff00ffu;
                        return (x | x << 4) & 0x0f0f0f0fu;
                    };
                    win[u].x = nibbles(lo & 0xffffu) | nibbles(hi & 0xffffu) << 4;
                    win[u].y = nibbles(lo >> 16) | nibbles(hi >> 16) << 4;
                }
            }
        };
        const int groups = (words + kLutBlocks - 1) / kLutBlocks;
        if (groups == 1) windows(0);
        int rp = 0;
        float rs = 0.f;
        unsigned rc = 0;
        const unsigned* tab = lut;
        for (int k = k0; k < k1; ++k) {
            const int w = A.lens[k], ns = (w + 3) / 4, eps = ns / 2 + 1, limit = A.limit[k];
            const float thr = A.thresh[k];
            unsigned acc[kLutBlocks];
            const auto approximate = [&](int v0) {
#pragma unroll
                for (int u = 0; u < kLutBlocks; ++u) acc[u] = 0u;
#pragma unroll
                for (int sg = 0; sg < 8; ++sg) {
                    if (sg >= ns) break;
                    const unsigned* t = tab + 256 * sg;
#pragma unroll
                    for (int u = 0; u < kLutBlocks; ++u)
                        if (v0 + u < words)
                            acc[u] += t[__byte_perm(sg < 4 ? win[u].x : win[u].y, 0u, 0x4440u + (sg & 3))];
                }
                // windows that leave the sequence are below every other (whose halves are >= 768)
#pragma unroll
                for (int u = 0; u < kLutBlocks; ++u)
                    if (32 * (v0 + u) + lane > L - w) acc[u] = 0u;
            };
            unsigned best = 0u;
            for (int g = 0; g < groups; ++g) {
                if (groups > 1) windows(kLutBlocks * g);
                approximate(kLutBlocks * g);
#pragma unroll
                for (int u = 0; u < kLutBlocks; ++u) best = max_halves(best, acc[u]);
            }
            tab += 256 * ns;
            int mf = (int)(best & 0xffffu), mc = BOTH ? (int)(best >> 16) : 0;
            VI bf{-INFINITY, 0x7fffffff}, bc{-INFINITY, 0x7fffffff};
            if (odd || __any_sync(full, max(mf, mc) >= limit)) {
                mf = __reduce_max_sync(full, mf);
                mc = __reduce_max_sync(full, mc);
                // a strand that is 2 eps behind cannot win
                const int cf = mf >= mc - 2 * eps ? mf - 2 * eps : 0x10000;
                const int cc = BOTH && mc >= mf - 2 * eps ? mc - 2 * eps : 0x10000;
                for (int g = 0; g < groups; ++g) {
                    if (groups > 1) {
                        tab -= 256 * ns;
                        windows(kLutBlocks * g);
                        approximate(kLutBlocks * g);
                        tab += 256 * ns;
                    }
#pragma unroll
                    for (int u = 0; u < kLutBlocks; ++u) {
                        const int v = kLutBlocks * g + u, l = 32 * v + lane;
                        const bool cand = v < words && l <= L - w &&
                                          (odd || (int)(acc[u] & 0xffffu) >= cf || (BOTH && (int)(acc[u] >> 16) >= cc));
                        if (!cand) continue;
                        unsigned m[4];
                        masks(v, m);
#pragma unroll
                        for (int j = 0; j < 4; ++j) m[j] &= w == 32 ? full : (1u << w) - 1u;
                        const float2 s = exact_sums<BOTH>(pw + (k - k0) * kl, w, m);
                        if (s.x > bf.v) bf = VI{s.x, l};
                        if (BOTH && s.y > bc.v) bc = VI{s.y, l};
                    }
                }
                for (int o = 16; o > 0; o >>= 1) {
                    VI y;
                    y.v = __shfl_xor_sync(full, bf.v, o);
                    y.i = __shfl_xor_sync(full, bf.i, o);
                    bf = vi_best(bf, y);
                    if (BOTH) {
                        y.v = __shfl_xor_sync(full, bc.v, o);
                        y.i = __shfl_xor_sync(full, bc.i, o);
                        bc = vi_best(bc, y);
                    }
                }
            }
            const bool fwd = bf.v >= bc.v;                // forward kept on ties
            const VI b = fwd ? bf : bc;
            const bool hit = b.v > thr;
            const int at = (k - k0) & 31;
            if (lane == at) {
                // REF_QUIRK_Q3: the forward scan's best hit at the first position reads as none
                rp = hit && (BOTH || b.i != 0) ? b.i + 1 : 0;
                rs = hit ? b.v : 0.f;
                rc = hit && !fwd;
            }
            if ((at == 31 || k == k1 - 1) && lane <= at) {
                const size_t o = (k - at + lane) + (size_t)K * n;
                if (A.pos) A.pos[o] = rp;
                if (BOTH && A.score) A.score[o] = rs;
                if (BOTH && A.comp) A.comp[o] = (uint8_t)rc;
            }
        }
    }
}

// the sparse scans apply: exact 0/1 data, finite PWM entries (within each motif's
// length), not turned off by CDLGB_SCAN_DENSE
bool sparse_ok(const cdlgb_ctx* c, const float* pwms, const int32_t* lens, int K, int maxlen) {
    if (!c->onehot_exact) return false;
    if (const char* e = getenv("CDLGB_SCAN_DENSE"))
        if (atoi(e) != 0) return false;
    for (int k = 0; k < K; ++k)
        for (int kk = 0; kk < lens[k]; ++kk)
            for (int a = 0; a < 4; ++a)
                if (!isfinite(pwms[k + (size_t)K * (a + 4 * kk)])) return false;
    return true;
}

// integer count matrices: grid (K, chunks); counts (4, maxlen, K) col-major
__global__ void k_count(const float* __restrict__ data, const int32_t* __restrict__ pos,
                        const uint8_t* __restrict__ comp, const int32_t* __restrict__ lens, int K,
                        int maxlen, int L, int N, int32_t* __restrict__ counts,
                        int32_t* __restrict__ nseq) {
    extern __shared__ int cnt[];       // 4*maxlen + 1
    const int k = blockIdx.x;
    const int w = lens[k];
    for (int i = threadIdx.x; i < 4 * maxlen + 1; i += blockDim.x) cnt[i] = 0;
    __syncthreads();
    int per = (N + gridDim.y - 1) / gridDim.y;
    int n0 = blockIdx.y * per, n1 = min(N, n0 + per);
    for (int n = n0 + threadIdx.x; n < n1; n += blockDim.x) {
        int p = pos[k + (size_t)K * n];
        if (p <= 0) continue;
        bool rc = comp && comp[k + (size_t)K * n];
        const float* x = data + (size_t)n * 4 * L + (size_t)(p - 1) * 4;
        for (int i = 0; i < w; ++i)
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                int v = (int)(rc ? x[(w - 1 - i) * 4 + (3 - a)] : x[i * 4 + a]);
                if (v) atomicAdd(&cnt[a + 4 * i], v);
            }
        atomicAdd(&cnt[4 * maxlen], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * maxlen; i += blockDim.x)
        if (cnt[i]) atomicAdd(&counts[i + (size_t)4 * maxlen * k], cnt[i]);
    if (threadIdx.x == 0 && cnt[4 * maxlen]) atomicAdd(&nseq[k], cnt[4 * maxlen]);
}

int check_pwm_args(cdlgb_ctx* c, const float* pwms, const int32_t* lens, const float* thresh,
                   int K, int maxlen) {
    if (!c->loaded) return cdlgb_seterr(c, CDLGB_ESTATE, "no data loaded");
    if (K <= 0 || maxlen <= 0 || !pwms || !lens || !thresh)
        return cdlgb_seterr(c, CDLGB_EINVAL, "scan: bad K=%d / maxlen=%d / null input", K, maxlen);
    for (int k = 0; k < K; ++k)
        if (lens[k] < 1 || lens[k] > maxlen)
            return cdlgb_seterr(c, CDLGB_EINVAL, "scan: lens[%d]=%d outside 1..maxlen=%d", k,
                                lens[k], maxlen);
    return CDLGB_OK;
}

// The filtered scans take motifs of at most 32 columns and sequences of at most 4096 bases;
// the forward scan's threshold is not negative (below zero its first maximum can be a
// window that is no hit).  Fills the motifs' thresholds, scales and limits (as floats' bits), the
// motifs per CTA and the widest motif's columns: the array may be wider than any of them
// (zero padding up to maxlen), and the tables go by the motifs alone.
bool lut_ok(const cdlgb_ctx* c, const float* pwms, const int32_t* lens, const float* thresh, int K, int maxlen,
            bool both, std::vector<float>& meta, int* KG, int* widest) {
    if (maxlen > 32 || c->L4 / 4 > 4096 || !sparse_ok(c, pwms, lens, K, maxlen)) return false;
    meta.resize(3 * (size_t)K);
    int segs = 0, most = 1;
    *widest = 1;
    for (int k = 0; k < K; ++k) {
        if (!both && !(thresh[k] >= 0.f)) return false;
        double S = 0.0;
        for (int i = 0; i < lens[k]; ++i) {
            float a = 0.f;
            for (int j = 0; j < 4; ++j) a = fmaxf(a, fabsf(pwms[k + (size_t)K * (j + 4 * i)]));
            S += a;
        }
        // sums in float32 have to stay far from its range's ends
        if (!(S < 1e30) || (S > 0.0 && S < 1e-25)) return false;
        const int ns = (lens[k] + 3) / 4;
        const float scale = S > 0.0 ? (float)(32000.0 / S) : 0.f;
        meta[k] = thresh[k];
        meta[K + k] = scale;
        const double at = floor((double)scale * (double)thresh[k]) + 32768.0 - (ns / 2 + 1);
        // a NaN threshold has no hit; a motif of zeros is left to the exact sums
        const int32_t limit = thresh[k] != thresh[k] ? 65536 : scale == 0.f ? 1
                            : at > 65536.0 ? 65536 : at < 1.0 ? 1 : (int32_t)at;
        memcpy(&meta[2 * (size_t)K + k], &limit, 4);
        segs += ns;
        most = std::max(most, ns);
        *widest = std::max(*widest, (int)lens[k]);
    }
    const int parts = (segs + kLutSegs - 1) / kLutSegs;
    *KG = std::min((K + parts - 1) / parts, kLutSegs / most);
    return true;
}

// device scratch layout: [pwms K*4*maxlen f32][per motif, 3 K f32: the threshold, and for the
// filtered scans what lut_ok fills][scores K*N f32] and [lens K i32][pos K*N i32]
int upload_pwms(cdlgb_ctx* c, const float* pwms, const int32_t* lens, const float* thresh,
                const std::vector<float>& meta, int K, int maxlen, size_t extra_i) {
    const size_t np = (size_t)K * 4 * maxlen;
    ST_TRY(ensure_scratch(c, &c->scan_f, &c->scan_f_cap, np + 3 * (size_t)K + (size_t)K * c->N));
    ST_TRY(ensure_scratch(c, &c->scan_i, &c->scan_i_cap, (size_t)K + extra_i));
    CU_TRY(c, cudaMemcpyAsync(c->scan_f, pwms, np * 4, cudaMemcpyHostToDevice, c->stream));
    if (meta.empty())
        CU_TRY(c, cudaMemcpyAsync(c->scan_f + np, thresh, (size_t)K * 4, cudaMemcpyHostToDevice, c->stream));
    else
        CU_TRY(c, cudaMemcpyAsync(c->scan_f + np, meta.data(), meta.size() * 4, cudaMemcpyHostToDevice, c->stream));
    CU_TRY(c, cudaMemcpyAsync(c->scan_i, lens, (size_t)K * 4, cudaMemcpyHostToDevice, c->stream));
    return CDLGB_OK;
}

// The filtered scan of one or both strands.  Shared memory: KG ceil(widest / 4) <= kLutSegs KB
// of tables, at most 33 KB of planes (4096 bases) and KG 16 widest <= 6.5 KB of motifs.  A warp
// takes a sequence, so few sequences leave SMs idle and a warp's motifs in a row are the
// time: there the motifs are cut further, as long as the CTAs are no more than two per SM
// (500 sequences of 4000, 24 motifs: 1.21 -> 0.37 ms for the forward call; 20 of 1000, 8 motifs:
// 0.139 -> 0.073).
template <bool BOTH>
int launch_lut(cdlgb_ctx* c, int KG, int widest, int K, int maxlen, int32_t* dpos, float* dscore, uint8_t* dcomp) {
    LutArgs a;
    a.data = scan_data(c); a.pwms = c->scan_f; a.lens = c->scan_i; a.thresh = c->scan_f + (size_t)K * 4 * maxlen;
    a.scale = a.thresh + K; a.limit = reinterpret_cast<const int32_t*>(a.thresh + 2 * (size_t)K);
    a.pos = dpos; a.score = dscore; a.comp = dcomp;
    const int blocks = (c->N + kLutWarps - 1) / kLutWarps, cut = std::min(K, 2 * 152 / blocks);
    if (cut > 1) KG = std::min(KG, (K + cut - 1) / cut);
    a.K = K; a.KG = KG; a.widest = widest; a.L = c->L4 / 4; a.N = c->N; a.words = (a.L + 31) / 32;
    const size_t shm = (size_t)KG * ((widest + 3) / 4) * 1024 + (size_t)kLutWarps * 16 * (a.words + 1) +
                       (size_t)KG * 16 * widest;
    CU_TRY(c, cudaFuncSetAttribute(k_scan_lut<BOTH>, cudaFuncAttributeMaxDynamicSharedMemorySize, 150 * 1024));
    const int parts = (K + KG - 1) / KG;
    const int gx = std::max(1, std::min(blocks, 2 * 152 / parts));
    k_scan_lut<BOTH><<<dim3(gx, parts), 32 * kLutWarps, shm, c->stream>>>(a);
    LAUNCH_CHECK(c, "k_scan_lut");
    return CDLGB_OK;
}

}  // namespace

int scan_fwd(cdlgb_ctx* c, const float* pwms, const int32_t* lens, const float* thresh, int K,
             int maxlen, int32_t* pos_out) {
    ST_TRY(check_pwm_args(c, pwms, lens, thresh, K, maxlen));
    const int N = c->N, L = c->L4 / 4;
    cdlgb_phase_begin(c, PH_SCAN);
    std::vector<float> meta;
    int KG = 0, widest = 0;
    const bool lut = lut_ok(c, pwms, lens, thresh, K, maxlen, false, meta, &KG, &widest);
    if (!lut) meta.clear();
    ST_TRY(upload_pwms(c, pwms, lens, thresh, meta, K, maxlen, (size_t)K * N));
    int32_t* dpos = c->scan_i + K;
    size_t shm = (size_t)4 * L * sizeof(float);
    if (shm > 200 * 1024) return cdlgb_seterr(c, CDLGB_ENOTSUP, "scan: L=%d too long", L);
    // one position per thread with the inputs staged, on exact one-hot data with finite
    // PWMs: the sparse sums (at most 1024 positions and 64 KB of staged inputs)
    const int nts = ((L + 31) / 32) * 32;
    const size_t shs = (size_t)K * 4 * maxlen * sizeof(float) + (size_t)K * (nts / 32) * sizeof(VI) +
                       (size_t)L;
    if (lut) {
        ST_TRY(launch_lut<false>(c, KG, widest, K, maxlen, dpos, nullptr, nullptr));
    } else if (nts <= 1024 && shs <= 64 * 1024 && sparse_ok(c, pwms, lens, K, maxlen)) {
        if (shs > 48 * 1024)
            CU_TRY(c, cudaFuncSetAttribute(k_scan_fwd_sparse, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           64 * 1024));
        k_scan_fwd_sparse<<<N, nts, shs, c->stream>>>(scan_data(c), c->scan_f, c->scan_i,
                                                       c->scan_f + (size_t)K * 4 * maxlen, K, maxlen,
                                                       L, dpos);
        LAUNCH_CHECK(c, "k_scan_fwd_sparse");
    } else {
        if (shm > 48 * 1024)
            CU_TRY(c, cudaFuncSetAttribute(k_scan_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        k_scan_fwd<<<N, kScanThreads, shm, c->stream>>>(scan_data(c), c->scan_f, c->scan_i,
                                                         c->scan_f + (size_t)K * 4 * maxlen, K, maxlen,
                                                         L, dpos);
        LAUNCH_CHECK(c, "k_scan_fwd");
    }
    CU_TRY(c, cudaMemcpyAsync(pos_out, dpos, (size_t)K * N * 4, cudaMemcpyDeviceToHost, c->stream));
    cdlgb_phase_end(c, PH_SCAN);
    CU_TRY(c, cudaStreamSynchronize(c->stream));
    return CDLGB_OK;
}

int scan_both(cdlgb_ctx* c, const float* pwms, const int32_t* lens, const float* thresh, int K,
              int maxlen, int32_t* pos_out, float* score_out, uint8_t* comp_out) {
    ST_TRY(check_pwm_args(c, pwms, lens, thresh, K, maxlen));
    const int N = c->N, L = c->L4 / 4;
    cdlgb_phase_begin(c, PH_SCAN);
    std::vector<float> meta;
    int KG = 0, widest = 0;
    const bool lut = lut_ok(c, pwms, lens, thresh, K, maxlen, true, meta, &KG, &widest);
    if (!lut) meta.clear();
    ST_TRY(upload_pwms(c, pwms, lens, thresh, meta, K, maxlen, (size_t)K * N));
    ST_TRY(ensure_scratch(c, &c->scan_u, &c->scan_u_cap, (size_t)K * N));
    int32_t* dpos = c->scan_i + K;
    float* dscore = c->scan_f + (size_t)K * 4 * maxlen + 3 * (size_t)K;
    size_t shm = (size_t)4 * L * sizeof(float);
    if (shm > 200 * 1024) return cdlgb_seterr(c, CDLGB_ENOTSUP, "scan: L=%d too long", L);
    // one position per thread and the staged PWMs when they fit: at most 1024 positions
    // and 64 KB of staged inputs (several blocks per SM)
    const int nts = ((L + 31) / 32) * 32;
    const size_t shs = (size_t)K * 4 * maxlen * sizeof(float2) + (size_t)K * (nts / 32) * 2 * sizeof(VI) +
                       (size_t)4 * L * sizeof(float);
    const size_t shp = (size_t)K * 4 * maxlen * sizeof(float2) + (size_t)K * (nts / 32) * 2 * sizeof(VI) +
                       (size_t)4 * ((L + 31) / 32 + 2) * sizeof(uint32_t);
    if (lut) {
        ST_TRY(launch_lut<true>(c, KG, widest, K, maxlen, dpos, dscore, c->scan_u));
    } else if (nts <= 1024 && maxlen <= 64 && shp <= 64 * 1024 && sparse_ok(c, pwms, lens, K, maxlen)) {
        if (shp > 48 * 1024)
            CU_TRY(c, cudaFuncSetAttribute(k_scan_both_sparse, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
        k_scan_both_sparse<<<N, nts, shp, c->stream>>>(scan_data(c), c->scan_f, c->scan_i,
                                                        c->scan_f + (size_t)K * 4 * maxlen, K, maxlen, L,
                                                        dpos, dscore, c->scan_u);
        LAUNCH_CHECK(c, "k_scan_both_sparse");
    } else if (nts <= 1024 && shs <= 64 * 1024) {
        if (shs > 48 * 1024)
            CU_TRY(c, cudaFuncSetAttribute(k_scan_both_staged, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           64 * 1024));
        k_scan_both_staged<<<N, nts, shs, c->stream>>>(scan_data(c), c->scan_f, c->scan_i,
                                                        c->scan_f + (size_t)K * 4 * maxlen, K, maxlen, L,
                                                        dpos, dscore, c->scan_u);
        LAUNCH_CHECK(c, "k_scan_both_staged");
    } else {
        if (shm > 48 * 1024)
            CU_TRY(c, cudaFuncSetAttribute(k_scan_both, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        k_scan_both<<<N, kScanThreads, shm, c->stream>>>(scan_data(c), c->scan_f, c->scan_i,
                                                          c->scan_f + (size_t)K * 4 * maxlen, K,
                                                          maxlen, L, dpos, dscore, c->scan_u);
        LAUNCH_CHECK(c, "k_scan_both");
    }
    if (pos_out)
        CU_TRY(c, cudaMemcpyAsync(pos_out, dpos, (size_t)K * N * 4, cudaMemcpyDeviceToHost, c->stream));
    if (score_out)
        CU_TRY(c, cudaMemcpyAsync(score_out, dscore, (size_t)K * N * 4, cudaMemcpyDeviceToHost, c->stream));
    if (comp_out)
        CU_TRY(c, cudaMemcpyAsync(comp_out, c->scan_u, (size_t)K * N, cudaMemcpyDeviceToHost, c->stream));
    cdlgb_phase_end(c, PH_SCAN);
    CU_TRY(c, cudaStreamSynchronize(c->stream));
    return CDLGB_OK;
}

int count_pfms(cdlgb_ctx* c, const int32_t* pos, const uint8_t* use_comp, const int32_t* lens,
               int K, int maxlen, int32_t* counts_out, int32_t* nseq_out) {
    if (!c->loaded) return cdlgb_seterr(c, CDLGB_ESTATE, "no data loaded");
    if (!c->onehot_exact)
        return cdlgb_seterr(c, CDLGB_ENOTSUP, "count_pfms needs 0/1 one-hot data");
    if (K <= 0 || maxlen <= 0 || !pos || !lens || !counts_out)
        return cdlgb_seterr(c, CDLGB_EINVAL, "count_pfms: bad arguments");
    const int N = c->N, L = c->L4 / 4;
    for (int k = 0; k < K; ++k)
        if (lens[k] < 1 || lens[k] > maxlen)
            return cdlgb_seterr(c, CDLGB_EINVAL, "count_pfms: lens[%d]=%d", k, lens[k]);
    if (const long long i = first_bad_position(pos, lens, K, (size_t)N, L); i >= 0) {
        const int k = (int)(i % K), n = (int)(i / K);
        return cdlgb_seterr(c, CDLGB_EINVAL,
                            "count_pfms: window at pos[%d,%d]=%d (len %d) leaves the sequence (L=%d)",
                            k, n, pos[i], lens[k], L);
    }
    size_t ncnt = (size_t)4 * maxlen * K;
    ST_TRY(ensure_scratch(c, &c->scan_i, &c->scan_i_cap, (size_t)K + (size_t)K * N + ncnt + K));
    ST_TRY(ensure_scratch(c, &c->scan_u, &c->scan_u_cap, (size_t)K * N));
    int32_t* dlens = c->scan_i;
    int32_t* dpos = c->scan_i + K;
    int32_t* dcnt = dpos + (size_t)K * N;
    int32_t* dnseq = dcnt + ncnt;
    CU_TRY(c, cudaMemcpyAsync(dlens, lens, (size_t)K * 4, cudaMemcpyHostToDevice, c->stream));
    CU_TRY(c, cudaMemcpyAsync(dpos, pos, (size_t)K * N * 4, cudaMemcpyHostToDevice, c->stream));
    if (use_comp)
        CU_TRY(c, cudaMemcpyAsync(c->scan_u, use_comp, (size_t)K * N, cudaMemcpyHostToDevice, c->stream));
    CU_TRY(c, cudaMemsetAsync(dcnt, 0, (ncnt + K) * 4, c->stream));
    int chunks = (N + 1023) / 1024;
    if (chunks > 64) chunks = 64;
    size_t shm = (size_t)(4 * maxlen + 1) * 4;
    k_count<<<dim3(K, chunks), 256, shm, c->stream>>>(scan_data(c), dpos, use_comp ? c->scan_u : nullptr,
                                                      dlens, K, maxlen, L, N, dcnt, dnseq);
    LAUNCH_CHECK(c, "k_count");
    CU_TRY(c, cudaMemcpyAsync(counts_out, dcnt, ncnt * 4, cudaMemcpyDeviceToHost, c->stream));
    if (nseq_out)
        CU_TRY(c, cudaMemcpyAsync(nseq_out, dnseq, (size_t)K * 4, cudaMemcpyDeviceToHost, c->stream));
    CU_TRY(c, cudaStreamSynchronize(c->stream));
    return CDLGB_OK;
}

namespace {
// non_overlap_scan! (scan.jl:123-174): one thread per sequence n over its K entries
// (k fastest).  sc is a scratch copy of the scores (taken entries are zeroed, as the
// reference zeroes scores_n), keep a scratch of flags; the intersection test walks the
// kept entries in the order they were taken.
__global__ void k_nonoverlap(int32_t* __restrict__ pos, float* __restrict__ score,
                             uint8_t* __restrict__ comp, const int32_t* __restrict__ lens,
                             int K, int N, float* __restrict__ sc, int32_t* __restrict__ order) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    int32_t* P = pos + (size_t)n * K;
    float* Sc = sc + (size_t)n * K;
    int32_t* ord = order + (size_t)n * K;         // kept entries in the order taken
    for (int k = 0; k < K; ++k) Sc[k] = P[k] != 0 ? score[(size_t)n * K + k] : 0.f;
    int nkept = 0;
    for (int iter = 0; iter < K; ++iter) {
        int best = 0;
        float bv = Sc[0];
        for (int k = 1; k < K; ++k)
            if (Sc[k] > bv) { bv = Sc[k]; best = k; }  // first maximum
        if (bv == 0.f) break;
        const int pm = P[best], pme = pm + lens[best] - 1;
        bool hit = false;
        for (int j = 0; j < nkept; ++j) {
            const int q = ord[j], p = P[q], pe = p + lens[q] - 1;
            if ((p <= pm && pm <= pe) || (p <= pme && pme <= pe) || (pm <= p && p <= pme) ||
                (pm <= pe && pe <= pme))
                hit = true;
        }
        if (!hit) ord[nkept++] = best;
        Sc[best] = 0.f;
    }
    // delete what was not kept: mark kept entries in sc (1), the rest (0)
    for (int k = 0; k < K; ++k) Sc[k] = 0.f;
    for (int j = 0; j < nkept; ++j) Sc[ord[j]] = 1.f;
    for (int k = 0; k < K; ++k)
        if (Sc[k] == 0.f && P[k] != 0) {
            P[k] = 0;
            score[(size_t)n * K + k] = 0.f;
            if (comp) comp[(size_t)n * K + k] = 0;
        }
}
}  // namespace

int nonoverlap_select(cdlgb_ctx* c, int32_t* pos, float* score, uint8_t* use_comp,
                      const int32_t* lens, int K) {
    if (!c->loaded) return cdlgb_seterr(c, CDLGB_ESTATE, "no data loaded");
    if (K <= 0 || !pos || !score || !lens)
        return cdlgb_seterr(c, CDLGB_EINVAL, "select_nonoverlapping: bad arguments");
    for (int k = 0; k < K; ++k)
        if (lens[k] < 1) return cdlgb_seterr(c, CDLGB_EINVAL, "select_nonoverlapping: lens[%d]=%d", k, lens[k]);
    const int N = c->N;
    const size_t KN = (size_t)K * N;
    ST_TRY(ensure_scratch(c, &c->scan_i, &c->scan_i_cap, (size_t)K + 2 * KN));
    ST_TRY(ensure_scratch(c, &c->scan_f, &c->scan_f_cap, 2 * KN));
    ST_TRY(ensure_scratch(c, &c->scan_u, &c->scan_u_cap, KN));
    int32_t* dlens = c->scan_i;
    int32_t* dpos = c->scan_i + K;
    int32_t* dord = dpos + KN;
    float* dscore = c->scan_f;
    float* dsc = c->scan_f + KN;
    CU_TRY(c, cudaMemcpyAsync(dlens, lens, (size_t)K * 4, cudaMemcpyHostToDevice, c->stream));
    CU_TRY(c, cudaMemcpyAsync(dpos, pos, KN * 4, cudaMemcpyHostToDevice, c->stream));
    CU_TRY(c, cudaMemcpyAsync(dscore, score, KN * 4, cudaMemcpyHostToDevice, c->stream));
    if (use_comp) CU_TRY(c, cudaMemcpyAsync(c->scan_u, use_comp, KN, cudaMemcpyHostToDevice, c->stream));
    cdlgb_phase_begin(c, PH_SCAN);
    k_nonoverlap<<<(N + 127) / 128, 128, 0, c->stream>>>(dpos, dscore, use_comp ? c->scan_u : nullptr,
                                                         dlens, K, N, dsc, dord);
    LAUNCH_CHECK(c, "k_nonoverlap");
    cdlgb_phase_end(c, PH_SCAN);
    CU_TRY(c, cudaMemcpyAsync(pos, dpos, KN * 4, cudaMemcpyDeviceToHost, c->stream));
    CU_TRY(c, cudaMemcpyAsync(score, dscore, KN * 4, cudaMemcpyDeviceToHost, c->stream));
    if (use_comp) CU_TRY(c, cudaMemcpyAsync(use_comp, c->scan_u, KN, cudaMemcpyDeviceToHost, c->stream));
    CU_TRY(c, cudaStreamSynchronize(c->stream));
    return CDLGB_OK;
}

namespace {
// pvalue2score (src/SEARCH/PWM_Touzet.jl:199-217) with the reference's granularity
// eps = 0.1 (a Float64) and flat background: the rounded entries floor(x / eps) eps are
// exact multiples k eps, every score reached is K eps for an integer K, and every
// probability is count / 4^m, so the reference's Double64 distribution Q[m]
// (score_distribution, :79-102) is the integer count table below, exactly.  One CTA per
// PWM: dense DP over K in shared memory, then find_largest_alpha (:130-142) over the
// reached keys in ascending order.
constexpr int kTouzetMaxR = 6144;     // score range per PWM (two uint64 tables in smem)

// The table's last pass (tail sums) runs in parallel: one thread over up to 6144 entries
// twice was 55 of the kernel's 74 us at widths of 20 columns.
constexpr int kTouzetThreads = 256;
__global__ void __launch_bounds__(kTouzetThreads) k_touzet(
    const int32_t* __restrict__ kq, const int32_t* __restrict__ lens, const int32_t* __restrict__ kmin,
    const int32_t* __restrict__ range, int maxlen, const unsigned long long* __restrict__ thr_count,
    int32_t* __restrict__ alpha_k, int32_t* __restrict__ status) {
    extern __shared__ unsigned long long tab[];
    __shared__ unsigned long long part[kTouzetThreads];
    __shared__ int first[kTouzetThreads / 32], last[kTouzetThreads / 32];
    const int p = blockIdx.x;
    const int m = lens[p], R = range[p];
    unsigned long long* Q0 = tab;
    unsigned long long* Q1 = tab + kTouzetMaxR;
    const int32_t* kp = kq + (size_t)p * 4 * maxlen;       // k[j][i] at j * maxlen + i
    if (threadIdx.x == 0) Q0[0] = 1ull;
    __syncthreads();
    int lo = 0;      // sum of the column minima so far
    int width = 1;   // reached keys lie in [lo, lo + width)
    for (int i = 0; i < m; ++i) {
        int k[4];
        for (int j = 0; j < 4; ++j) k[j] = kp[j * maxlen + i];
        const int cmin = min(min(k[0], k[1]), min(k[2], k[3])), cmax = max(max(k[0], k[1]), max(k[2], k[3]));
        const int nw = width + (cmax - cmin);
        for (int s = threadIdx.x; s < nw; s += kTouzetThreads) {
            unsigned long long acc = 0ull;
            for (int j = 0; j < 4; ++j) {
                const int src = s - (k[j] - cmin);
                if (src >= 0 && src < width) acc += Q0[src];
            }
            Q1[s] = acc;
        }
        __syncthreads();
        unsigned long long* t = Q0;
        Q0 = Q1;
        Q1 = t;
        lo += cmin;
        width = nw;
    }
    if (lo != kmin[p] || width != R) {
        if (threadIdx.x == 0) status[p] = 1;
        return;
    }
    // find_largest_alpha: q_sum starts at the total (4^m counts), keys ascending;
    // q_sum >= pval  <=>  tail >= ceil(pval 4^m)  (integers, exact).  The answer is the first
    // reached key whose tail is below, or the last reached key.  Thread t takes keys
    // [t per, (t + 1) per); tails of whole threads' keys by a suffix sum over the threads.
    const int per = (width + kTouzetThreads - 1) / kTouzetThreads;
    const int s0 = threadIdx.x * per, s1 = min(width, s0 + per);
    unsigned long long sum = 0ull;
    int end = -1;
    for (int s = s0; s < s1; ++s) {
        sum += Q0[s];
        if (Q0[s]) end = s;
    }
    part[threadIdx.x] = sum;
    for (int o = 1; o < kTouzetThreads; o <<= 1) {
        __syncthreads();
        const unsigned long long v = threadIdx.x + o < kTouzetThreads ? part[threadIdx.x + o] : 0ull;
        __syncthreads();
        part[threadIdx.x] += v;
    }
    unsigned long long tail = part[threadIdx.x];             // keys from s0 on
    int at = 0x7fffffff;
    for (int s = s0; s < s1 && at == 0x7fffffff; ++s) {
        const unsigned long long v = Q0[s];
        if (v == 0ull) continue;                             // keys never reached are absent
        if (tail < thr_count[p]) at = s;
        tail -= v;
    }
    at = __reduce_min_sync(0xffffffffu, at);
    end = __reduce_max_sync(0xffffffffu, end);
    if ((threadIdx.x & 31) == 0) {
        first[threadIdx.x >> 5] = at;
        last[threadIdx.x >> 5] = end;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kTouzetThreads / 32; ++w) {
            at = min(at, first[w]);
            end = max(end, last[w]);
        }
        alpha_k[p] = lo + (at != 0x7fffffff ? at : end);
        status[p] = 0;
    }
}
}  // namespace

int touzet_thresholds(cdlgb_ctx* c, const float* pwms, const int32_t* lens, int K, int maxlen,
                      double pval, float* thresh_out) {
    if (K <= 0 || maxlen <= 0 || !pwms || !lens || !thresh_out)
        return cdlgb_seterr(c, CDLGB_EINVAL, "pvalue_thresholds: bad arguments");
    if (!(pval >= 0.0 && pval <= 1.0)) return cdlgb_seterr(c, CDLGB_EINVAL, "pvalue must be in [0,1]");
    const double eps = 1e-1;                                 // _granularity_
    const size_t nk = (size_t)K * 4 * maxlen;
    std::vector<int32_t> host((size_t)nk + 5 * (size_t)K, 0);
    int32_t* kq = host.data() + 2 * (size_t)K;
    int32_t* kmin = kq + nk;
    int32_t* range = kmin + K;
    int32_t* hl = range + K;
    std::vector<unsigned long long> thr(K);
    for (int p = 0; p < K; ++p) {
        const int m = lens[p];
        if (m < 1 || m > maxlen || m > 31)
            return cdlgb_seterr(c, CDLGB_EINVAL, "pvalue_thresholds: lens[%d]=%d (1..31, <= maxlen)", p, m);
        hl[p] = m;
        long lo = 0, hi = 0;
        for (int i = 0; i < m; ++i) {
            int cmin = 0, cmax = 0;
            for (int j = 0; j < 4; ++j) {
                // pwms (K, 4, maxlen) col-major: element (p, j, i) at p + K (j + 4 i)
                const double x = (double)pwms[p + (size_t)K * (j + 4 * (size_t)i)];
                if (!(fabs(x) < 1e6))
                    return cdlgb_seterr(c, CDLGB_EINVAL, "pvalue_thresholds: PWM entry %g", x);
                // exact floor(x / eps): the double quotient corrected by exact fma residuals
                double q = floor(x / eps);
                if (fma(q, eps, -x) > 0.0) q -= 1.0;
                else if (fma(q + 1.0, eps, -x) <= 0.0) q += 1.0;
                const int k = (int)q;
                kq[(size_t)p * 4 * maxlen + j * maxlen + i] = k;
                if (j == 0 || k < cmin) cmin = k;
                if (j == 0 || k > cmax) cmax = k;
            }
            lo += cmin;
            hi += cmax;
        }
        if (hi - lo + 1 > kTouzetMaxR)
            return cdlgb_seterr(c, CDLGB_ENOTSUP, "pvalue_thresholds: score range %ld of PWM %d exceeds %d",
                                hi - lo + 1, p, kTouzetMaxR);
        kmin[p] = (int32_t)lo;
        range[p] = (int32_t)(hi - lo + 1);
        thr[p] = (unsigned long long)ceil(ldexp(pval, 2 * m));   // pval 4^m is exact; <= 2^62
    }
    // thr, kq, kmin, range and lens in one copy (thr first: 8-byte aligned), then alpha, status
    const size_t up = 2 * (size_t)K + nk + 3 * (size_t)K;
    memcpy(host.data(), thr.data(), (size_t)K * 8);
    ST_TRY(ensure_scratch(c, &c->scan_i, &c->scan_i_cap, up + 2 * (size_t)K));
    int32_t* d_kq = c->scan_i + 2 * (size_t)K;
    int32_t* d_alpha = c->scan_i + up;
    int32_t* d_status = d_alpha + K;
    CU_TRY(c, cudaMemcpyAsync(c->scan_i, host.data(), up * 4, cudaMemcpyHostToDevice, c->stream));
    constexpr int shm = 2 * kTouzetMaxR * (int)sizeof(unsigned long long);
    CU_TRY(c, cudaFuncSetAttribute(k_touzet, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
    k_touzet<<<K, kTouzetThreads, shm, c->stream>>>(d_kq, d_kq + nk + 2 * (size_t)K, d_kq + nk, d_kq + nk + K, maxlen,
                                                    reinterpret_cast<const unsigned long long*>(c->scan_i), d_alpha,
                                                    d_status);
    LAUNCH_CHECK(c, "k_touzet");
    std::vector<int32_t> out(2 * (size_t)K);
    CU_TRY(c, cudaMemcpyAsync(out.data(), d_alpha, 2 * (size_t)K * 4, cudaMemcpyDeviceToHost, c->stream));
    CU_TRY(c, cudaStreamSynchronize(c->stream));
    for (int p = 0; p < K; ++p) {
        if (out[K + p] != 0) return cdlgb_seterr(c, CDLGB_ECUDA, "pvalue_thresholds: table mismatch for PWM %d", p);
        // the Double64 key K eps is exact; its high part rounded to float32 (get_thresh's
        // type_real conversion)
        thresh_out[p] = (float)((double)out[p] * eps);
    }
    return CDLGB_OK;
}

void scan_free(cdlgb_ctx* c) {
    dev_free(c, c->scan_i);
    dev_free(c, c->scan_f);
    dev_free(c, c->scan_u);
    c->scan_i = nullptr; c->scan_f = nullptr; c->scan_u = nullptr;
    c->scan_i_cap = c->scan_f_cap = c->scan_u_cap = 0;
}
