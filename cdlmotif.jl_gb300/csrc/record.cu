// Code -> activations -> filter-pair topology -> pair count matrices
// (src/SEARCH/store.jl:1-144, src/SEARCH/extractions.jl:18-190), device resident.
//
// The activation record keeps, for each training t, the codes
//   codes[t][n][m][c] = X_best[gamma + 4c, m, n]   (store.jl:15, c = 0..L-1)
// and its threshold; a filter k of the record is (t, m) for every m of training t with
// at least one activation (the reference's uinds, store.jl:22).  Activations are
// codes > thresh[t] (store.jl:17), evaluated on the fly.
//
// topology_at_nth_pt! (store.jl:64-107) launches a thread per (r, c, n) over
// (C*K)^2 * N; here the record keeps every filter's activations in a sequence as a bit
// mask, a CTA takes some ordered filter pairs (fr, fc) over some sequences and counts
// their distances in shared memory from the set bits alone, with the reference's
// conditions (integer counts: exact and order-independent).
#include "cdlgb_internal.h"

#include <algorithm>
#include <new>
#include <string>
#include <vector>

struct cdlgb_ar {
    int dev = 0;
    cudaStream_t stream = nullptr;
    char err[512];
    int N = 0, C = 0, M = 0, T = 0;
    std::vector<int> uinds, training_num, filter_lengths;   // per registered filter (1-based)
    std::vector<int> recorded;                               // training recorded?
    float* codes = nullptr;                                  // (T, N, M, C)
    int* anym = nullptr;                                     // (M) scratch
    int* kmap = nullptr;                                     // (Kcap) t*M + m
    int* klen = nullptr;                                     // (Kcap) filter length (bases)
    unsigned* mask = nullptr;                                // (T, N, M, ceil(C/32)): codes > thresh[t]; behind codes
    int* dcount = nullptr;                                   // topology outputs (device)
    size_t dcount_cap = 0;
    float* msa = nullptr;                                    // pair MSA partials
    size_t msa_cap = 0;
};

namespace {

int ar_err(cdlgb_ar* a, int code, const char* fmt, ...) {
    if (a) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(a->err, sizeof(a->err), fmt, ap);
        va_end(ap);
    }
    return code;
}

#define AR_CU(a, call)                                                                   \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess)                                                           \
            return ar_err((a), CDLGB_ECUDA, "%s failed: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

// codes[t] <- X_best rows gamma, gamma+4, ...; the bits code > thresh; anym[m] |= any.
// A warp takes 256 positions of a row (n, m), their loads in flight together; long rows of
// few sequences so spread over the warps too (two records of 50 x 8 rows of 20000, with the
// allocations: 844 us with a warp per row and a word at a time, 399 so).
// X_best is read whole (its sectors hold 8 rows each).
constexpr int kRecWords = 8;
__global__ void __launch_bounds__(256) k_record(const float* __restrict__ Xb, float* __restrict__ codes,
                                                unsigned* __restrict__ mask, size_t rows, int M, int C, int Lg,
                                                int gamma, float thresh, int* __restrict__ anym) {
    const int lane = threadIdx.x & 31, words = (C + 31) / 32, segs = (words + kRecWords - 1) / kRecWords;
    const size_t stride = (size_t)gridDim.x * (blockDim.x / 32);
    for (size_t i = blockIdx.x * (size_t)(blockDim.x / 32) + (threadIdx.x >> 5); i < rows * segs; i += stride) {
        const size_t r = segs == 1 ? i : i / segs;
        const int w0 = kRecWords * (int)(i - r * segs);
        const float* x = Xb + r * Lg + gamma;
        float v[kRecWords];
#pragma unroll
        for (int u = 0; u < kRecWords; ++u) {
            const int c = 32 * (w0 + u) + lane;
            v[u] = c < C ? x[4 * c] : 0.f;
        }
        unsigned mine = 0;
        bool any = false;
#pragma unroll
        for (int u = 0; u < kRecWords; ++u) {
            const int c = 32 * (w0 + u) + lane;
            if (c < C) codes[r * C + c] = v[u];
            const unsigned b = __ballot_sync(0xffffffffu, c < C && v[u] > thresh);
            if (lane == u) mine = b;
            any |= b != 0;
        }
        if (lane < kRecWords && w0 + lane < words) mask[r * words + w0 + lane] = mine;
        const int m = (int)(r % M);
        if (any && lane == 0 && !anym[m]) atomicOr(&anym[m], 1);
    }
}

// Ordered filter pairs of different trainings: fr in a tile of up to FG filters, fc in one
// of up to FC, each tile of one training and one length, over one chunk of the sequences.
// The distance counts of the tile stay in shared memory, [FG][FC][dn] (of the D = maxlen
// overlaps, CmFm1 gaps and "next to", dn from blockIdx.z dn on), and are added to the
// outputs at the end.  A warp takes a sequence: it lists the tile's fc activations, then
// for each activation of an fr its lanes go over the list, so that every lane counts.
// Instructions and shared-memory atomics bound it.  N = 5000, L = 200, K = 64, 3.5 % of the
// codes active (250 M pairs): 3.7 ms with global atomics over 3.3 MB and a pair loop of
// 64-bit divisions, 3.5 ms with a lane per fc over its own mask bits (lanes wait for the
// fullest mask), 1.2 ms with the lists.
// over (K, K, maxlen), non_over (K, K, CmFm1), next_to (K, K), all col-major int32.
struct TopoTile { int fr0, nr, fc0, nc; };
constexpr int kTopoThreads = 1024, kTopoList = 512;           // list entries per warp; 8 mask words add up to 256
__global__ void __launch_bounds__(kTopoThreads) k_topology(
    const unsigned* __restrict__ mask, const int* __restrict__ kmap, const int* __restrict__ klen,
    const TopoTile* __restrict__ tiles, int FG, int FC, int dn, int N, int M, int C, int K, int maxlen, int CmFm1,
    int* __restrict__ over, int* __restrict__ non_over, int* __restrict__ next_to) {
    extern __shared__ int hist[];
    const int words = (C + 31) / 32, D = maxlen + CmFm1 + 1, dlo = blockIdx.z * dn;
    const TopoTile tile = tiles[blockIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    unsigned* list = reinterpret_cast<unsigned*>(hist + (size_t)FG * FC * dn) + warp * kTopoList;
    for (int i = threadIdx.x; i < FG * FC * dn; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const int lr = klen[tile.fr0], same = klen[tile.fc0] == lr;  // equal lengths at one place: excluded
    const int n0 = (int)((long long)N * blockIdx.y / gridDim.y), n1 = (int)((long long)N * (blockIdx.y + 1) / gridDim.y);
    const int nrw = tile.nr * words, ncw = tile.nc * words;
    const auto word = [&](int k0, int n, int i) {               // word i of the rows of filters k0, k0 + 1, ...
        const int tm = kmap[k0 + i / words], t = tm / M, m = tm - t * M;
        return mask[(((size_t)t * N + n) * M + m) * words + i % words];
    };
    for (int n = n0 + warp; n < n1; n += nwarps) {
        for (int c0 = 0; c0 < ncw;) {
            // (filter << 16 | position) of the next words' bits, of as many of 32 words as fit
            // (8 at least; 8 at a time took 1.20 instead of 0.72 ms, with the copies, for 2 x 32
            // filters, 500 sequences of 1000 and 0.3 % of the codes active)
            int cnt = 0;
            while (c0 < ncw && cnt + 256 <= kTopoList) {
                const int i = c0 + lane;
                unsigned b = i < ncw ? word(tile.fc0, n, i) : 0u;
                int at = __popc(b);
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, at, o);
                    if (lane >= o) at += v;
                }
                const int taken = __popc(__ballot_sync(0xffffffffu, cnt + at <= kTopoList));
                const int sum = __shfl_sync(0xffffffffu, at, taken - 1);
                at += cnt - __popc(b);
                const unsigned base = (unsigned)(i / words) << 16 | (unsigned)(i % words) << 5;
                if (lane < taken)
                    for (; b; b &= b - 1) list[at++] = base + __ffs(b) - 1;
                c0 += taken;
                cnt += sum;
            }
            __syncwarp();
            for (int r0 = 0; r0 < nrw; r0 += 32) {
                const unsigned a = r0 + lane < nrw ? word(tile.fr0, n, r0 + lane) : 0u;
                for (unsigned any = __ballot_sync(0xffffffffu, a != 0); any; any &= any - 1) {
                    const int src = __ffs(any) - 1, i = r0 + src;
                    int* h = hist + (size_t)(i / words) * FC * dn - dlo;
                    for (unsigned b = __shfl_sync(0xffffffffu, a, src); b; b &= b - 1) {
                        const int pr = 32 * (i % words) + __ffs(b) - 1;
                        for (int e = lane; e < cnt; e += 32) {
                            const unsigned v = list[e];
                            const int off = (int)(v & 0xffffu) - pr, dist = off - lr;
                            if (off < same) continue;
                            const int d = dist < 0 ? -dist - 1 : dist > 0 && dist <= CmFm1 ? maxlen + dist - 1 : D - 1;
                            if ((unsigned)(d - dlo) < (unsigned)dn) atomicAdd(h + (v >> 16) * dn + d, 1);
                        }
                    }
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < tile.nr * FC * dn; i += blockDim.x) {
        const int v = hist[i];
        if (!v) continue;
        const int d = dlo + i % dn, f = i / dn % FC, r = i / dn / FC;
        const size_t at = (tile.fr0 + r) + (size_t)K * (tile.fc0 + f);
        if (d < maxlen) atomicAdd(&over[at + (size_t)K * K * d], v);
        else if (d < D - 1) atomicAdd(&non_over[at + (size_t)K * K * (d - maxlen)], v);
        else atomicAdd(&next_to[at], v);
    }
}

// Pair MSAs (get_f_pair_starts + msa_fill, extractions.jl:116-181): grid (P, chunks); a
// warp finds the pair's starts in a sequence from the two masks (fr's bits and fc's
// shifted by the pair's distance) and adds the code-weighted one-hot windows to its row
// of shared memory, its lanes along the window; the warps' rows are added in order into
// one partial per chunk (summed in order afterwards).
constexpr int kMsaWarps = 8;
constexpr int kMaxSpan = 1536;                                // k_pair_finish holds it in 48 KB of float64
__global__ void __launch_bounds__(32 * kMsaWarps) k_pair_msa(
    const float* __restrict__ codes, const unsigned* __restrict__ mask, const float* __restrict__ S,
    const int* __restrict__ pairs, const int* __restrict__ kmap, const int* __restrict__ klen, int N, int M, int C,
    int max_span, float* __restrict__ part) {
    extern __shared__ float acc[];                            // [kMsaWarps][4 * max_span]
    const int p = blockIdx.x, ch = blockIdx.y, nch = gridDim.y;
    const int fr = pairs[3 * p] - 1, fc = pairs[3 * p + 1] - 1, o_len = pairs[3 * p + 2];
    const int fl1 = klen[fr], fl2 = klen[fc];
    const int span = o_len >= fl2 ? o_len : fl1 - o_len + fl2;   // get_span_len
    const int t1 = kmap[fr] / M, f1 = kmap[fr] % M;
    const int t2 = kmap[fc] / M, f2 = kmap[fc] % M;
    const int words = (C + 31) / 32, ml = 4 * max_span;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* my = acc + warp * ml;
    for (int i = lane; i < ml; i += 32) my[i] = 0.f;
    __syncwarp();
    const int n0 = (int)((long long)N * ch / nch), n1 = (int)((long long)N * (ch + 1) / nch);
    const int nl = 4 * span, sh = fl1 - o_len, sw = sh >> 5, sb = sh & 31;
    // fr starts at 0-based s, fc at s + sh; the window [s, s + span) inside the sequence
    const int last = C - span;
    for (int n = n0 + warp; n < n1; n += kMsaWarps) {
        const size_t r1 = ((size_t)t1 * N + n) * M + f1, r2 = ((size_t)t2 * N + n) * M + f2;
        const unsigned* m1 = mask + r1 * words;
        const unsigned* m2 = mask + r2 * words;
        const float* x = S + (size_t)n * 4 * C;
        for (int w0 = 0; w0 < words; w0 += 32) {
            const int w = w0 + lane;
            unsigned hit = 0;
            if (w < words) {
                const unsigned lo = w + sw < words ? m2[w + sw] : 0u, hi = w + sw + 1 < words ? m2[w + sw + 1] : 0u;
                hit = m1[w] & __funnelshift_r(lo, hi, sb);
                if (32 * w + 31 > last) hit &= last < 32 * w ? 0u : ~0u >> (31 - (last - 32 * w));
            }
            for (unsigned any = __ballot_sync(0xffffffffu, hit != 0); any; any &= any - 1) {
                const int src = __ffs(any) - 1;
                for (unsigned b = __shfl_sync(0xffffffffu, hit, src); b; b &= b - 1) {
                    const int s = 32 * (w0 + src) + __ffs(b) - 1;
                    const float avg = (codes[r1 * C + s] + codes[r2 * C + s + sh]) / 2;
                    for (int l = lane; l < nl; l += 32) my[l] += avg * x[4 * s + l];
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ml; i += blockDim.x) {
        float v = 0.f;
        for (int w = 0; w < kMsaWarps; ++w) v += acc[w * ml + i];
        part[((size_t)p * nch + ch) * ml + i] = v;
    }
}

// sum the chunk partials in order, + 0.1 inside the span (msa_pseudocount), normalise
// by the first column's total; pfms (P, 4, max_span) col-major
__global__ void k_pair_finish(const float* __restrict__ part, const int* __restrict__ pairs,
                              const int* __restrict__ klen, int P, int nch, int max_span,
                              float* __restrict__ pfm, int* __restrict__ spans) {
    extern __shared__ double col[];                           // 4 * max_span
    const int p = blockIdx.x;
    const int fr = pairs[3 * p] - 1, fc = pairs[3 * p + 1] - 1, o_len = pairs[3 * p + 2];
    const int fl1 = klen[fr], fl2 = klen[fc];
    const int span = o_len >= fl2 ? o_len : fl1 - o_len + fl2;
    for (int i = threadIdx.x; i < 4 * max_span; i += blockDim.x) {
        double s = 0.0;
        for (int ch = 0; ch < nch; ++ch) s += part[((size_t)p * nch + ch) * 4 * max_span + i];
        float v = (float)s;
        if (i < 4 * span) v += 0.1f;
        col[i] = v;
    }
    __syncthreads();
    const double tot = col[0] + col[1] + col[2] + col[3];
    for (int i = threadIdx.x; i < 4 * max_span; i += blockDim.x) {
        const int a = i % 4, j = i / 4;
        pfm[p + (size_t)P * (a + 4 * (size_t)j)] = (float)(col[i] / tot);
    }
    if (threadIdx.x == 0) spans[p] = span;
}

}  // namespace

extern "C" {

int cdlgb_ar_create(int32_t N, int32_t L, int32_t M, int32_t T, int32_t device, cdlgb_ar** out) {
    if (!out || N <= 0 || L <= 0 || M <= 0 || T <= 0 || L > 65535)
        return noctx_seterr(CDLGB_EINVAL, "cdlgb_ar_create: N=%d, L=%d, M=%d, T=%d (L <= 65535)",
                            N, L, M, T);
    *out = nullptr;
    cdlgb_ar* a = new (std::nothrow) cdlgb_ar();
    if (!a) return noctx_seterr(CDLGB_EINVAL, "cdlgb_ar_create: out of host memory");
    a->err[0] = 0;
    a->dev = device;
    a->N = N; a->C = L; a->M = M; a->T = T;
    a->recorded.assign(T, 0);
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&a->stream, cudaStreamNonBlocking);
    size_t kcap = (size_t)T * M;
    // the codes and, in the same block (an allocation less: 20 us), their masks
    const size_t rows = (size_t)T * N * M;
    if (e == cudaSuccess) e = cudaMalloc((void**)&a->codes, rows * L * sizeof(float) + rows * ((L + 31) / 32) * sizeof(unsigned));
    if (e == cudaSuccess) a->mask = reinterpret_cast<unsigned*>(a->codes + rows * L);
    if (e == cudaSuccess) e = cudaMalloc((void**)&a->anym, M * sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc((void**)&a->kmap, kcap * sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc((void**)&a->klen, kcap * sizeof(int));
    if (e != cudaSuccess) {
        noctx_seterr(CDLGB_ECUDA, "cdlgb_ar_create: %s", cudaGetErrorString(e));
        cdlgb_ar_destroy(a);
        return CDLGB_ECUDA;
    }
    *out = a;
    return CDLGB_OK;
}

int cdlgb_ar_destroy(cdlgb_ar* a) {
    if (!a) return CDLGB_OK;
    cudaSetDevice(a->dev);
    if (a->stream) cudaStreamSynchronize(a->stream);
    void* ptrs[] = {a->codes, a->anym, a->kmap, a->klen, a->dcount, a->msa};
    for (void* p : ptrs) if (p) cudaFree(p);
    if (a->stream) cudaStreamDestroy(a->stream);
    delete a;
    return CDLGB_OK;
}

const char* cdlgb_ar_last_error(const cdlgb_ar* a) {
    if (a) return a->err;
    const char* m = noctx_err();
    return m ? m : "null record";
}

int cdlgb_ar_record(cdlgb_ar* a, cdlgb_ctx* c, double thresh, int32_t train_num,
                    int32_t filter_size, int32_t* added) {
    if (!a || !c) return CDLGB_EINVAL;
    // store.jl:8
    if (!(thresh > 0)) return ar_err(a, CDLGB_EINVAL, "threshold must be greater than 0");
    if (train_num < 1 || train_num > a->T || a->recorded[train_num - 1])
        return ar_err(a, CDLGB_EINVAL, "train_num %d outside 1..%d or already recorded", train_num, a->T);
    if (!c->initialized || c->N != a->N || c->L4 != 4 * a->C || c->M != a->M)
        return ar_err(a, CDLGB_EINVAL, "context does not hold an initialised N=%d, L=%d, M=%d problem",
                      a->N, a->C, a->M);
    if (filter_size < 1 || filter_size > a->C) return ar_err(a, CDLGB_EINVAL, "bad filter_size");
    AR_CU(a, cudaSetDevice(a->dev));
    AR_CU(a, cudaStreamSynchronize(c->stream));     // X_best is final
    const int t = train_num - 1;
    const float th = (float)thresh;                 // activations compare Float32 codes
    const float* Xb = c->best_is_cur ? c->Xb[c->xcur] : c->Xb[1 - c->xcur];
    AR_CU(a, cudaMemsetAsync(a->anym, 0, a->M * sizeof(int), a->stream));
    const size_t rows = (size_t)a->N * a->M, words = (a->C + 31) / 32;
    k_record<<<grid_for(rows * ((words + kRecWords - 1) / kRecWords), 8), 256, 0, a->stream>>>(Xb, a->codes + t * rows * a->C, a->mask + t * rows * words,
                                                       rows, a->M, a->C, c->Lg, c->gamma, th, a->anym);
    AR_CU(a, cudaGetLastError());
    std::vector<int> any(a->M);
    AR_CU(a, cudaMemcpyAsync(any.data(), a->anym, a->M * sizeof(int), cudaMemcpyDeviceToHost, a->stream));
    AR_CU(a, cudaStreamSynchronize(a->stream));
    int cnt = 0;
    for (int m = 0; m < a->M; ++m)
        if (any[m]) {
            a->uinds.push_back(m + 1);
            a->training_num.push_back(train_num);
            a->filter_lengths.push_back(filter_size);
            ++cnt;
        }
    a->recorded[t] = 1;
    const int K = (int)a->uinds.size();
    std::vector<int> km(K), kl(K);
    for (int k = 0; k < K; ++k) {
        km[k] = (a->training_num[k] - 1) * a->M + (a->uinds[k] - 1);
        kl[k] = a->filter_lengths[k];
    }
    // on the record's stream, ahead of the kernels that read them (a blocking copy from
    // pageable memory may return before it lands, and that stream does not wait on the
    // legacy stream); each call returns once its host bytes are staged
    AR_CU(a, cudaMemcpyAsync(a->kmap, km.data(), K * sizeof(int), cudaMemcpyHostToDevice, a->stream));
    AR_CU(a, cudaMemcpyAsync(a->klen, kl.data(), K * sizeof(int), cudaMemcpyHostToDevice, a->stream));
    if (added) *added = cnt;
    return CDLGB_OK;
}

int cdlgb_ar_info(const cdlgb_ar* a, int32_t* K, int32_t* uinds, int32_t* training_num,
                  int32_t* filter_lengths, int32_t cap) {
    if (!a || !K) return CDLGB_EINVAL;
    const int k = (int)a->uinds.size();
    *K = k;
    if (cap < k && (uinds || training_num || filter_lengths)) return CDLGB_EINVAL;
    for (int i = 0; i < k; ++i) {
        if (uinds) uinds[i] = a->uinds[i];
        if (training_num) training_num[i] = a->training_num[i];
        if (filter_lengths) filter_lengths[i] = a->filter_lengths[i];
    }
    return CDLGB_OK;
}

int cdlgb_ar_topology(cdlgb_ar* a, int32_t* over, int32_t* non_over, int32_t* next_to) {
    if (!a || !over || !non_over || !next_to) return CDLGB_EINVAL;
    const int K = (int)a->uinds.size();
    if (K == 0) return ar_err(a, CDLGB_ESTATE, "no filters recorded");
    AR_CU(a, cudaSetDevice(a->dev));
    int maxlen = *std::max_element(a->filter_lengths.begin(), a->filter_lengths.end());
    int minlen = *std::min_element(a->filter_lengths.begin(), a->filter_lengths.end());
    const int CmFm1 = a->C - minlen - 1;       // maximum_apart_length (helpers.jl:11)
    if (CmFm1 < 0) return ar_err(a, CDLGB_EINVAL, "filters longer than the sequences");
    const size_t n_over = (size_t)K * K * maxlen, n_non = (size_t)K * K * CmFm1, n_next = (size_t)K * K;
    // tiles of filter pairs whose distance counts fit a CTA's shared memory beside the warps'
    // lists, as many fc as a list has use for
    const int D = maxlen + CmFm1 + 1;
    const size_t lists = (size_t)(kTopoThreads / 32) * kTopoList * 4, cap = 220 * 1024 - lists;
    int dn = D, FC = std::min(K, 32), FG = std::min(K, 32);
    while (FC > 1 && (size_t)FC * dn * 4 > cap) FC = (FC + 1) / 2;
    while (FG > 1 && (size_t)FG * FC * dn * 4 > cap) --FG;
    while ((size_t)FG * FC * dn * 4 > cap) dn = (dn + 1) / 2;   // one pair, its distances in parts
    // runs of recorded filters of one training and length, cut into tiles
    std::vector<TopoTile> tiles;
    const auto run = [&](int k0, int most) {
        int k = k0;
        while (k < K && a->training_num[k] == a->training_num[k0] && a->filter_lengths[k] == a->filter_lengths[k0]) ++k;
        const int parts = (k - k0 + most - 1) / most;
        return (k - k0 + parts - 1) / parts;
    };
    for (int r = 0, nr; r < K; r += nr) {
        nr = run(r, FG);
        for (int f = 0, nc; f < K; f += nc) {
            nc = run(f, FC);
            if (a->training_num[r] != a->training_num[f]) tiles.push_back({r, nr, f, nc});
        }
    }
    const size_t n_counts = (n_over + n_non + n_next + 3) & ~(size_t)3;
    const size_t need = n_counts + 4 * tiles.size();
    if (a->dcount_cap < need) {
        if (a->dcount) cudaFree(a->dcount);
        a->dcount = nullptr;
        AR_CU(a, cudaMalloc((void**)&a->dcount, need * sizeof(int)));
        a->dcount_cap = need;
    }
    AR_CU(a, cudaMemsetAsync(a->dcount, 0, n_counts * sizeof(int), a->stream));
    if (!tiles.empty()) {
        TopoTile* dt = (TopoTile*)(a->dcount + n_counts);
        AR_CU(a, cudaMemcpyAsync(dt, tiles.data(), tiles.size() * sizeof(TopoTile), cudaMemcpyHostToDevice, a->stream));
        AR_CU(a, cudaFuncSetAttribute(k_topology, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
        // one CTA per SM, 32 warps: at least one sequence per warp; the chunks of the sequences
        // that leave the least of the SMs idle (a chunk's counts cleared and added up are put
        // at a twentieth of a pass over all sequences)
        const int most = std::max(1, std::min((a->N + 31) / 32, std::max(8, 152 / (int)tiles.size())));
        const auto cost = [&](int n) { return (double)((tiles.size() * n + 151) / 152) * (1.0 / n + 0.05); };
        int nch = 1;
        for (int n = 2; n <= most; ++n)
            if (cost(n) < cost(nch)) nch = n;
        k_topology<<<dim3((unsigned)tiles.size(), nch, (D + dn - 1) / dn), kTopoThreads,
                     lists + (size_t)FG * FC * dn * 4, a->stream>>>(
            a->mask, a->kmap, a->klen, dt, FG, FC, dn, a->N, a->M, a->C, K, maxlen, CmFm1, a->dcount,
            a->dcount + n_over, a->dcount + n_over + n_non);
    }
    AR_CU(a, cudaGetLastError());
    AR_CU(a, cudaMemcpyAsync(over, a->dcount, n_over * sizeof(int), cudaMemcpyDeviceToHost, a->stream));
    AR_CU(a, cudaMemcpyAsync(non_over, a->dcount + n_over, n_non * sizeof(int), cudaMemcpyDeviceToHost, a->stream));
    AR_CU(a, cudaMemcpyAsync(next_to, a->dcount + n_over + n_non, n_next * sizeof(int), cudaMemcpyDeviceToHost, a->stream));
    AR_CU(a, cudaStreamSynchronize(a->stream));
    return CDLGB_OK;
}

int cdlgb_ar_pair_pfms(cdlgb_ar* a, cdlgb_ctx* c, const int32_t* pairs, int32_t P,
                       int32_t filter_size, float* pfms, int32_t* span_lens) {
    if (!a || !c || !pairs || !pfms || !span_lens || P <= 0 || filter_size < 1) return CDLGB_EINVAL;
    if (!c->loaded || c->N != a->N || c->L4 != 4 * a->C)
        return ar_err(a, CDLGB_EINVAL, "context does not hold the record's data");
    const int K = (int)a->uinds.size();
    if (filter_size > (kMaxSpan + 1) / 2)
        return ar_err(a, CDLGB_EINVAL, "filter size %d: pairs span at most %d bases", filter_size, kMaxSpan);
    const int max_span = 2 * filter_size - 1;   // extractions.jl:22
    for (int p = 0; p < P; ++p) {
        const int fr = pairs[3 * p], fc = pairs[3 * p + 1], o = pairs[3 * p + 2];
        if (fr < 1 || fr > K || fc < 1 || fc > K || o < 1 || o > a->filter_lengths[fr - 1])
            return ar_err(a, CDLGB_EINVAL, "pair %d = (%d, %d, %d) out of range (K=%d)", p, fr, fc, o, K);
        const int fl1 = a->filter_lengths[fr - 1], fl2 = a->filter_lengths[fc - 1];
        const int span = o >= fl2 ? o : fl1 - o + fl2;
        if (span > max_span || span > a->C)
            return ar_err(a, CDLGB_EINVAL, "pair %d spans %d bases (> %d)", p, span, max_span);
    }
    AR_CU(a, cudaSetDevice(a->dev));
    AR_CU(a, cudaStreamSynchronize(c->stream));
    const int nch = std::max(1, std::min(64, a->N / 64));
    const size_t npart = (size_t)P * nch * 4 * max_span;
    const size_t need = npart + (size_t)P * 4 * max_span + 3 * (size_t)P + P;
    if (a->msa_cap < need) {
        if (a->msa) cudaFree(a->msa);
        a->msa = nullptr;
        AR_CU(a, cudaMalloc((void**)&a->msa, need * sizeof(float)));
        a->msa_cap = need;
    }
    float* part = a->msa;
    float* dpfm = part + npart;
    int* dpairs = (int*)(dpfm + (size_t)P * 4 * max_span);
    int* dspan = dpairs + 3 * P;
    AR_CU(a, cudaMemcpyAsync(dpairs, pairs, 3 * (size_t)P * sizeof(int), cudaMemcpyHostToDevice, a->stream));
    // (a process-wide cap, the same for every context)
    constexpr int cap = kMsaWarps * 4 * kMaxSpan * (int)sizeof(float);
    const size_t sm = (size_t)kMsaWarps * 4 * max_span * sizeof(float);
    if (sm > 48 * 1024) AR_CU(a, cudaFuncSetAttribute(k_pair_msa, cudaFuncAttributeMaxDynamicSharedMemorySize, cap));
    k_pair_msa<<<dim3(P, nch), 32 * kMsaWarps, sm, a->stream>>>(a->codes, a->mask, c->S, dpairs, a->kmap, a->klen,
                                                               a->N, a->M, a->C, max_span, part);
    AR_CU(a, cudaGetLastError());
    k_pair_finish<<<P, 128, 4 * max_span * sizeof(double), a->stream>>>(part, dpairs, a->klen, P, nch,
                                                                       max_span, dpfm, dspan);
    AR_CU(a, cudaGetLastError());
    AR_CU(a, cudaMemcpyAsync(pfms, dpfm, (size_t)P * 4 * max_span * sizeof(float), cudaMemcpyDeviceToHost, a->stream));
    AR_CU(a, cudaMemcpyAsync(span_lens, dspan, P * sizeof(int), cudaMemcpyDeviceToHost, a->stream));
    AR_CU(a, cudaStreamSynchronize(a->stream));
    return CDLGB_OK;
}

}  // extern "C"
