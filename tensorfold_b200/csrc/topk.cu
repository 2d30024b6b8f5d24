// Exact top-k over vocabulary rows and the keyed Gumbel-max draw.
//
// top-k: a bf16 logit is a 16-bit sortable key. A row is cut into contiguous slices, one CTA each. A CTA reads its
// slice once, 64 keys a thread into registers, and needs no histogram: K keys reach the smallest, over the warps, of a
// warp's ceil(K / warps)-th largest THREAD maximum, so that is a lower bound T0 of the slice's K-th largest key.
// The keys that reach T0 are few, they are ranked against each other by (key descending, id ascending), and the first
// K are the slice's candidates, in order. Only a slice whose keys tie or crowd at T0 (more than kCand reach it) takes the
// exact route: bisect the key range on the count of all keys, then the smallest ids among the ties. A second kernel does the
// same over the slices' ordered candidates. The row's k largest are among its slices' k largest, so the result is
// exact and a function of the row alone.
//
// draw: token = argmax over the kept candidates of logit/T + Gumbel(hash(seed, position, id)), the
// candidates being the top_k cut to the smallest prefix whose tempered probability reaches top_p.
// The hash (splitmix64) and the arithmetic (fp64) follow the host rule, so a row gets the same
// token whether it is drawn alone or inside a window. A warp draws a row: a lane does two candidates' exponentials
// and logarithms, and the sums run over the candidates in order.
//
// Bound: the row bytes from HBM (128 rows x 248320: 63.6 MB, 9.7 us at 6.55 TB/s). The former histogram kernel
// (keys staged in shared memory, two atomic histograms with a match per key) took 111 us there, its merge 12 us and a
// draw of one thread a row 19.5 us.

#include <algorithm>

#include "common.cuh"

namespace tf {
namespace {

constexpr int kMaxK = 64;
constexpr int kSliceThreads = 256, kChunks = 8;                       // a thread holds kChunks x 8 keys
constexpr int kSliceMax = kSliceThreads * kChunks * 8 - 8;            // a slice off a 16-byte boundary takes one chunk more
constexpr int kSliceMin = 4096;
constexpr int kCand = 1024, kMaxSlices = 64, kMergeThreads = 128, kSms = 148;

// Slices are cut so that a few rows still give every SM a CTA (down to kSliceMin entries a slice, at most kMaxSlices),
// many rows the longest slices: the result does not depend on the cut.
// A vocabulary too long for kMaxSlices slices of kSliceMax, up to kMaxSlices of all the keys that a CTA's threads hold (1048576
// entries), still has kMaxSlices: where such a slice is off a 16-byte boundary it takes the exact route.
inline int least_slices(int V) {
    const int slices = (V + kSliceMax - 1) / kSliceMax;
    return slices > kMaxSlices && V <= kMaxSlices * kSliceThreads * kChunks * 8 ? kMaxSlices : slices;
}
inline int most_slices(int V) { return std::min(V / kSliceMin, kMaxSlices); }
inline int slice_len(int V, int rows) {
    const int slices = std::max(least_slices(V), std::min(most_slices(V), (kSms + rows - 1) / rows));
    return (((V + slices - 1) / slices) + 7) & ~7;          // a multiple of 8 entries: slices of an aligned row are aligned
}
inline int slice_count(int V, int rows) { const int L = slice_len(V, rows); return (V + L - 1) / L; }

__device__ __forceinline__ uint32_t unsort_key(uint32_t k) { return (k & 0x8000u) ? (k & 0x7FFFu) : (~k & 0xFFFFu); }
// two bf16 values -> two sortable keys: a negative value's bits are inverted, a positive one's sign bit is set
__device__ __forceinline__ uint32_t sort_keys2(uint32_t w) {
    const uint32_t neg = (w >> 15) & 0x00010001u;
    return w ^ (0x80008000u | (neg * 0x7FFFu));
}

// the largest T such that `count(T) >= K`, bisected over 16-bit keys (count(0) >= K must hold); `count` is block-wide
template <class Count>
__device__ __forceinline__ uint32_t bisect_key(int K, Count count) {
    uint32_t T = 0;
#pragma unroll 1
    for (int bit = 15; bit >= 0; --bit) {
        const uint32_t t = T | (1u << bit);
        if (count(t) >= K) T = t;
    }
    return T;
}

// Order of candidates: key descending, then id ascending, as one 64-bit number.
__device__ __forceinline__ unsigned long long rank_code(uint32_t key, uint32_t id) { return ((unsigned long long)key << 32) | (0xFFFFFFFFu - id); }

// The exact route, for a slice whose keys crowd: its kk largest (ties to the smallest ids) into c_s, unordered. Reads the
// slice from memory again: a thread's registers then hold no more than the ordinary route needs.
__device__ __noinline__ void exact_slice(const uint16_t* xr, int n, int v0, int kk, unsigned long long* c_s, int* n_s, int* scan_s) {
    const int tid = threadIdx.x, passes = (n + kSliceThreads - 1) / kSliceThreads;
    auto key_at = [&](int e) { return sort_keys2(xr[e]) & 0xFFFFu; };
    const uint32_t T = bisect_key(kk, [&](uint32_t t) {
        int mine = 0;
        for (int e = tid; e < n; e += kSliceThreads) mine += key_at(e) >= t;
        mine = __reduce_add_sync(0xffffffffu, mine);
        if ((tid & 31) == 0) scan_s[tid >> 5] = mine;
        __syncthreads();
        int all = 0;
        for (int w = 0; w < kSliceThreads / 32; ++w) all += scan_s[w];
        __syncthreads();
        return all;
    });
    if (tid == 0) *n_s = 0;
    __syncthreads();
    for (int e = tid; e < n; e += kSliceThreads)
        if (key_at(e) > T) c_s[atomicAdd(n_s, 1)] = rank_code(key_at(e), (uint32_t)(v0 + e));      // at most kk - 1
    __syncthreads();
    int taken = *n_s;
    for (int i = 0; i < passes && taken < kk; ++i) {
        const int e = i * kSliceThreads + tid;
        const bool tie = e < n && key_at(e) == T;
        const unsigned m = __ballot_sync(0xffffffffu, tie);
        if ((tid & 31) == 0) scan_s[tid >> 5] = __popc(m);
        __syncthreads();
        int at = taken + __popc(m & ((1u << (tid & 31)) - 1u));
        for (int w = 0; w < kSliceThreads / 32; ++w) {
            if (w < (tid >> 5)) at += scan_s[w];
            taken += scan_s[w];
        }
        if (tie && at < kk) c_s[at] = rank_code(T, (uint32_t)(v0 + e));
        __syncthreads();
    }
}

// DEALT: a row of at most 8 entries a thread (always one slice; the slices of a cut row are longer) is dealt out entry by entry, round
// the warps, so that every warp and thread has its share whatever its length. 1 row of 300 / 600 / 1024 / 1500 entries, k = 28: 4.1 / 4.7 /
// 4.3 / 4.4 us; 10.7 / 19.6 / 37.8 / 12.6 by chunks, which leave warps empty, so that T0 is 0 and every entry a candidate.
template <bool DEALT>
__global__ void __launch_bounds__(kSliceThreads, 4) topk_slice_kernel(const __nv_bfloat16* x, size_t row_stride, int V, int K, int L,
                                                                   unsigned long long* cand) {
    __shared__ unsigned long long c_s[kCand];
    __shared__ int n_s, scan_s[kSliceThreads / 32 + 1];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, row = blockIdx.y;
    const int v0 = blockIdx.x * L, n = min(L, V - v0);
    const uint16_t* xr = reinterpret_cast<const uint16_t*>(x) + (size_t)row * row_stride + v0;
    unsigned long long* out = cand + ((size_t)row * gridDim.x + blockIdx.x) * K;
    const int kk = min(K, n);                                   // a short slice yields all it has
    // chunks of 16 aligned bytes that hold the slice: chunk c has entries 8c - off .. 8c - off + 7
    const int off = (int)((reinterpret_cast<uintptr_t>(xr) & 15) >> 1), chunks = (n + off + 7) >> 3;
    constexpr int kWarps = kSliceThreads / 32, kHeld = DEALT ? 1 : kChunks;
    const int warp = tid >> 5;
    constexpr int kStep = DEALT ? kSliceThreads : 1;            // entries from one key of a thread's eight to the next
    uint4 key[kHeld];
    if constexpr (!DEALT) {
#pragma unroll
        for (int i = 0; i < kHeld; ++i) {
            const int c = i * kSliceThreads + tid, e0 = 8 * c - off;
            if (c < chunks && e0 >= 0 && e0 + 8 <= n) key[i] = __ldcs(reinterpret_cast<const uint4*>(xr + e0));
        }
    }
    if (tid == 0) n_s = 0;
    uint32_t top2 = 0;
#pragma unroll
    for (int i = 0; i < kHeld; ++i) {
        const int c = i * kSliceThreads + tid, e0 = DEALT ? (tid & 31) * kWarps + warp : 8 * c - off;
        if (!DEALT && c < chunks && e0 >= 0 && e0 + 8 <= n) {
            key[i] = make_uint4(sort_keys2(key[i].x), sort_keys2(key[i].y), sort_keys2(key[i].z), sort_keys2(key[i].w));
        } else {                                                // dealt entries, an end chunk, or none: entries outside the slice are key 0
            uint32_t w[4] = {0u, 0u, 0u, 0u};
            if (DEALT || c < chunks)
                for (int j = 0; j < 8; ++j)
                    if (e0 + j * kStep >= 0 && e0 + j * kStep < n) w[j >> 1] |= (sort_keys2(xr[e0 + j * kStep]) & 0xFFFFu) << (16 * (j & 1));
            key[i] = make_uint4(w[0], w[1], w[2], w[3]);
        }
        top2 = __vmaxu2(top2, __vmaxu2(__vmaxu2(key[i].x, key[i].y), __vmaxu2(key[i].z, key[i].w)));
    }
    const uint32_t top = max(top2 & 0xFFFFu, top2 >> 16);
    // T0: each warp's ceil(kk / warps)-th largest thread maximum, the smallest of them over the warps: kk keys reach it. A warp with
    // fewer threads that hold entries (dealt rows of less than 256) gives its smallest one: an entry is then a thread's only one.
    {
        const int most = DEALT ? min(kk, kWarps * ((n - warp + kWarps - 1) / kWarps)) : kk;
        uint32_t left = top + 1, reached = DEALT ? 0x10000u : 0u;      // 0: taken; a warp without entries bounds nothing
        for (int r = 0; r < most; r += kWarps) {
            reached = __reduce_max_sync(0xffffffffu, left);
            if ((tid & 31) == __ffs(__ballot_sync(0xffffffffu, left == reached)) - 1) left = 0;
        }
        if ((tid & 31) == 0) scan_s[warp] = (int)(reached - 1);
    }
    __syncthreads();
    uint32_t T = 0xFFFFu;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) T = min(T, (uint32_t)scan_s[w]);
    if (top >= T) {
#pragma unroll
        for (int i = 0; i < kHeld; ++i) {
            const uint32_t m = __vmaxu2(__vmaxu2(key[i].x, key[i].y), __vmaxu2(key[i].z, key[i].w));
            if (max(m & 0xFFFFu, m >> 16) < T) continue;
            const uint32_t w[4] = {key[i].x, key[i].y, key[i].z, key[i].w};
            const int e0 = DEALT ? (tid & 31) * kWarps + warp : 8 * (i * kSliceThreads + tid) - off;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t k = (w[j >> 1] >> (16 * (j & 1))) & 0xFFFFu;
                if (k >= T && (unsigned)(e0 + j * kStep) < (unsigned)n) {
                    const int at = atomicAdd(&n_s, 1);
                    if (at < kCand) c_s[at] = rank_code(k, (uint32_t)(v0 + e0 + j * kStep));
                }
            }
        }
    }
    __syncthreads();
    int have = n_s;
    if (have > kCand || (!DEALT && chunks > kChunks * kSliceThreads)) {
        __syncthreads();
        exact_slice(xr, n, v0, kk, c_s, &n_s, scan_s);
        have = kk;
    }
    for (int i = tid; i < have; i += kSliceThreads) {
        const unsigned long long me = c_s[i];
        int rank = 0;
        for (int j = 0; j < have; ++j) rank += c_s[j] > me;
        if (rank < kk) out[rank] = me;
    }
    for (int j = tid + kk; j < K; j += kSliceThreads) out[j] = 0ull;       // ranks behind every real entry
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
    x ^= x >> 30; x *= 0xBF58476D1CE4E5B9ull;
    x ^= x >> 27; x *= 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

struct Draw {
    const long long* positions;
    unsigned long long seed;
    double temperature, top_p;
    int top_k;
    int* tokens;
};

// One warp draws a row from its candidates, ordered by (value desc, id asc). Lane l holds candidates l and l + 32; the
// sums add the candidates one by one in order (the host rule's order), fetched from their lanes.
__device__ __forceinline__ int draw_row(const int (&id)[2], const float (&val)[2], int width, long long position, const Draw& d) {
    const int lane = threadIdx.x & 31;
    const int k = max(1, min(d.top_k > 0 ? d.top_k : width, width));
    const double t = fmax(d.temperature, 1e-6);
    const double s0 = (double)val[0] / t, s1 = (double)val[1] / t;
    const double top = __shfl_sync(0xffffffffu, s0, 0);
    int keep = k;
    if (d.top_p > 0.0 && d.top_p < 1.0) {
        const double e0 = lane < k ? exp(s0 - top) : 0.0, e1 = lane + 32 < k ? exp(s1 - top) : 0.0;
        double denom = 0.0;
        for (int j = 0; j < k; ++j) denom += __shfl_sync(0xffffffffu, j < 32 ? e0 : e1, j & 31);
        const double p0 = e0 / denom, p1 = e1 / denom;
        double cum = 0.0;
        int below = 0;
        for (int j = 0; j < k; ++j) {
            cum += __shfl_sync(0xffffffffu, j < 32 ? p0 : p1, j & 31);
            below += cum < d.top_p;
        }
        keep = min(k, below + 1);
    }
    const unsigned long long h0 = mix64(d.seed + 0x9E3779B97F4A7C15ull);
    const unsigned long long h1 = mix64(h0 ^ ((unsigned long long)position * 0xD1B54A32D192ED03ull));
    double best = -INFINITY;
    int at = 0x7FFFFFFF, pick = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (lane + 32 * h < keep) {
            const unsigned long long hash = mix64(h1 ^ (unsigned long long)(long long)id[h]);
            const double u = (double)(hash >> 11) * 0x1.0p-53 + 0x1.0p-54;
            const double score = (h ? s1 : s0) - log(-log(u));
            if (score > best) { best = score; at = lane + 32 * h; pick = id[h]; }
        }
    }
    // the first candidate of the largest score, as a scan in order would keep it
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o), op = __shfl_xor_sync(0xffffffffu, pick, o);
        if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; pick = op; }
    }
    const int first = __shfl_sync(0xffffffffu, id[0], 0);
    return at == 0x7FFFFFFF ? first : pick;                    // no score above -inf: the first candidate
}

// One CTA per row: the slices' candidates that reach a lower bound of the K-th largest, ranked; with `d.tokens` the row's
// token is drawn from them in the same launch (idx_out and val_out may then be null).
__global__ void __launch_bounds__(kMergeThreads) topk_merge_kernel(const unsigned long long* cand, int n, int K, int* idx_out, float* val_out,
                                                                   const Draw d) {
    __shared__ unsigned long long c_s[kMaxSlices * kMaxK];
    __shared__ unsigned long long best_s[kMaxK];
    __shared__ int n_s;
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, slices = n / K;
    const unsigned long long* c = cand + (size_t)row * n;
    if (tid == 0) n_s = 0;
    // every slice's list is in order: with the first ceil(K / slices) of each, K candidates reach the smallest of those
    // lists' last entries (0, below every real entry, where a slice has fewer)
    const int at = (K + slices - 1) / slices - 1;
    unsigned long long T = ~0ull;
    for (int s = lane; s < slices; s += 32) T = min(T, c[s * K + at]);
#pragma unroll
    for (int o = 16; o; o >>= 1) T = min(T, __shfl_xor_sync(0xffffffffu, T, o));
    __syncthreads();
    constexpr int U = 4;                                       // loads in flight
    for (int i0 = tid; i0 < n; i0 += U * kMergeThreads) {
        unsigned long long mine[U];
#pragma unroll
        for (int u = 0; u < U; ++u) mine[u] = i0 + u * kMergeThreads < n ? c[i0 + u * kMergeThreads] : 0ull;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (mine[u] != 0ull && mine[u] >= T) c_s[atomicAdd(&n_s, 1)] = mine[u];
    }
    __syncthreads();
    const int have = n_s;
    for (int i = tid; i < have; i += kMergeThreads) {
        const unsigned long long me = c_s[i];
        int rank = 0;
        for (int j = 0; j < have; ++j) rank += c_s[j] > me;
        if (rank < K) {
            best_s[rank] = me;
            if (idx_out != nullptr) {
                idx_out[(size_t)row * K + rank] = (int)(0xFFFFFFFFu - (uint32_t)me);
                val_out[(size_t)row * K + rank] = __uint_as_float(unsort_key((uint32_t)(me >> 32)) << 16);
            }
        }
    }
    if (d.tokens == nullptr) return;
    __syncthreads();
    if (tid >= 32) return;
    int id[2];
    float val[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const unsigned long long c = tid + 32 * h < K ? best_s[tid + 32 * h] : best_s[0];
        id[h] = (int)(0xFFFFFFFFu - (uint32_t)c);
        val[h] = __uint_as_float(unsort_key((uint32_t)(c >> 32)) << 16);
    }
    const int token = draw_row(id, val, K, d.positions[row], d);
    if (tid == 0) d.tokens[row] = token;
}

// The draw alone, from candidates already ordered: a warp per row.
__global__ void sample_kernel(const int* idx, const float* val, int width, const Draw d, int rows) {
    pdl_launch_dependents();
    pdl_wait();
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= rows) return;
    int id[2];
    float v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int j = lane + 32 * h < width ? lane + 32 * h : 0;
        id[h] = idx[(size_t)row * width + j];
        v[h] = val[(size_t)row * width + j];
    }
    const int token = draw_row(id, v, width, d.positions[row], d);
    if (lane == 0) d.tokens[row] = token;
}

}  // namespace
}  // namespace tf

extern "C" {

// Fewer rows are cut into more slices, so a call's own lists, rows x slice_count, may be more than those of a call with more
// rows (vocabulary 248320: 154 for 7 rows, 152 for 8). The size is a bound of them that grows with the rows, the
// vocabulary and k, so that a workspace made for the largest call serves every smaller one.
size_t tf_topk_scratch_bytes(int rows, int vocab, int k) {
    if (rows < 1 || vocab < 1 || k < 1 || k > tf::kMaxK) return 0;
    const size_t least = (size_t)rows * tf::least_slices(vocab), most = (size_t)rows * tf::most_slices(vocab), wanted = (size_t)rows + tf::kSms - 1;
    const size_t lists = std::max(least, std::min(most, wanted));
    return lists * k * sizeof(unsigned long long);
}

static int topk(const void* x, size_t row_stride, int rows, int vocab, int k, int* idx, float* val, tf::Draw draw, void* scratch,
                size_t scratch_bytes, void* stream) {
    if (rows < 1 || rows > 65535 || vocab < 1 || k < 1 || k > tf::kMaxK || k > vocab || row_stride < (size_t)vocab) return TF_EINVAL;
    if (!x || (!idx != !val) || (!idx && !draw.tokens)) return TF_EINVAL;
    if (reinterpret_cast<uintptr_t>(x) & 1) return TF_EALIGN;
    const int slices = tf::slice_count(vocab, rows);
    if (slices > tf::kMaxSlices) return TF_EINVAL;
    if (!scratch || scratch_bytes < (size_t)rows * slices * k * sizeof(unsigned long long)) return TF_ESCRATCH;
    if (reinterpret_cast<uintptr_t>(scratch) & 7) return TF_EALIGN;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int len = tf::slice_len(vocab, rows), n = slices * k;
    void* a1[] = {&x, &row_stride, &vocab, &k, &len, &scratch};
    const void* slice = len <= tf::kSliceThreads * 8 ? (const void*)tf::topk_slice_kernel<true> : (const void*)tf::topk_slice_kernel<false>;
    if (tf::launch_pdl(slice, dim3(slices, rows), dim3(tf::kSliceThreads), 0, st, a1) != cudaSuccess) {
        cudaGetLastError();
        return TF_ECUDA;
    }
    void* a2[] = {&scratch, &n, &k, &idx, &val, &draw};
    if (tf::launch_pdl((const void*)tf::topk_merge_kernel, dim3(rows), dim3(tf::kMergeThreads), 0, st, a2) != cudaSuccess) {
        cudaGetLastError();
        return TF_ECUDA;
    }
    return TF_OK;
}

int tf_topk_rows(const void* x, size_t row_stride, int rows, int vocab, int k, int* idx, float* val, void* scratch,
                 size_t scratch_bytes, void* stream) {
    if (!idx) return TF_EINVAL;
    return topk(x, row_stride, rows, vocab, k, idx, val, tf::Draw{}, scratch, scratch_bytes, stream);
}

int tf_topk_sample_rows(const void* x, size_t row_stride, int rows, int vocab, int k, const long long* positions, unsigned long long seed,
                        double temperature, int top_k, double top_p, int* tokens, void* scratch, size_t scratch_bytes, void* stream) {
    if (!positions || !tokens) return TF_EINVAL;
    return topk(x, row_stride, rows, vocab, k, nullptr, nullptr, tf::Draw{positions, seed, temperature, top_p, top_k, tokens}, scratch,
                scratch_bytes, stream);
}

int tf_sample_rows(const int* idx, const float* val, int width, const long long* positions, unsigned long long seed,
                   double temperature, int top_k, double top_p, int* tokens, int rows, void* stream) {
    if (rows < 1 || width < 1 || width > tf::kMaxK || !idx || !val || !positions || !tokens) return TF_EINVAL;
    tf::Draw draw{positions, seed, temperature, top_p, top_k, tokens};
    void* args[] = {&idx, &val, &width, &draw, &rows};
    if (tf::launch_pdl((const void*)tf::sample_kernel, dim3((rows + 3) / 4), dim3(128), 0, static_cast<cudaStream_t>(stream), args) !=
        cudaSuccess) { cudaGetLastError(); return TF_ECUDA; }
    return TF_OK;
}

}  // extern "C"
