// 4-bit group-affine lane matmul for sm_100a: weights stream once from HBM through a bulk-copy
// (TMA) pipeline into shared memory, are expanded to bf16 in registers and multiplied on the
// tensor cores; the scale/bias epilogue and the K-segment sums run in fp32.
//
// Arithmetic, per output element (row m, column n):
//   for each weight group g of the segment, in order:
//       P   = tensor-core chain over the group's 16-wide k-steps of  x[m,k] * (q[n,k] + 128),
//             started from  -128 * xs[m,g]            (so P = x . q up to fp32 rounding)
//       acc = fma(b[n,g], xs[m,g], fma(s[n,g], P, acc))
//   segments of K (fixed by N, K and the worker count only) are added in k order,
//   then one rounding to bf16.
// The chain never looks at the row count, so row m of an M-row call has the bits of a 1-row call.
//
// Weight tile layout (built by tf_qmm_tile): records indexed [column block of 256][k tile of 64]
// [column tile of 16 inside the block]; a pipeline stage (all 16 column tiles of a block, a few k
// tiles) is therefore ONE contiguous range and arrives with a single bulk copy. Each record is
// 512 bytes of nibbles + 64*(64/group) bytes of (scale, bias) pairs.
//   nibbles: lane (g = lane/4, t = lane%4) owns 16 bytes = 4 words; word s (k-step s) holds, at
//            nibble j, column 16c + g + 8*(j&1) and input tile_k(t, s, nibble_quad(j)) of the k tile,
//            so that (w >> 4i) & 0x000F000F is register i of the mma A fragment. K-steps 0,1 cover
//            inputs 0..31 of the tile and k-steps 2,3 inputs 32..63: a group of 32 is two whole k-steps.
//   pairs  : for each half-tile h (one per group inside the k tile) and g in 0..7:
//            bf16 s[16c+g], b[16c+g], s[16c+g+8], b[16c+g+8]   (8 bytes, one load per lane)
//
// Activations arrive "packed" (tf_pack_rows, or written directly by the glue kernels): per k tile,
// Mp rows (M rounded up to its bucket 8/16/32/64/128, extra rows zero) of 128 bytes (the tile's 64
// bf16 inputs, with the two 64-byte halves swapped on odd rows so that shared-memory reads spread
// over all banks), then the tile's group sums as [groups in tile][Mp] fp32. A stage's activations
// are again one contiguous range.
//
// Warp roles in a CTA: consumer warps (each one or two 16-column tiles of the block) and one producer
// thread (bulk copies).
//
// What bounds the loop once the bytes arrive is the integer pipe (16 lanes a cycle per sub-partition):
// a 16 x 64 record costs 12 shifts + 16 and-or operations there, so each of the 16 is one lop3.

#include <type_traits>

#include "common.cuh"

namespace tf {
namespace {

constexpr int kWorkers = 148;
// k tiles per schedule item: a function of the weight's shape only, the same for every row bucket, so that
// the K segments (hence the bits) do not depend on the row count. One tile keeps the workers' shares within
// a tile of each other; a narrow weight (fewer than 18 column blocks) would then be cut into dozens of
// segments a block, so its blocks are cut into eight items instead.
constexpr int kMaxCutsNarrow = 8;
__host__ __device__ inline int item_tiles_for(int CB, int KT) {
    return CB * kMaxCutsNarrow < kWorkers ? (KT + kMaxCutsNarrow - 1) / kMaxCutsNarrow : 1;
}
constexpr int kWarps = 16;      // column tiles per column block (baked into the layout)
constexpr int kCols = kWarps * 16;

__host__ __device__ constexpr int rec_bytes(int group) { return 512 + (64 / group) * 64; }

// position inside the 4-element k quad that nibble j of a word carries
__host__ __device__ constexpr int nibble_quad(int j) { return ((j >> 1) & 1) * 2 + ((j >> 2) & 1); }
// input (0..63) of a k tile that lane t feeds to k-step s at quad position `quad`
__host__ __device__ constexpr int tile_k(int t, int s, int quad) { return 32 * (s >> 1) + 8 * t + 4 * (s & 1) + quad; }

// One instantiation per row bucket: MB blocks of 8 rows, KTS k tiles a pipeline stage, T column tiles per
// consumer warp (they share the activation loads), HALVES passes over the weights, each for its own MB * 8 rows of a
// bucket of HALVES times as many.
template <int G_, int MB_, int KTS_, int T_, int HALVES_ = 1>
struct Cfg {
    static constexpr int G = G_, MB = MB_, KTS = KTS_, T = T_, HALVES = HALVES_;
    static constexpr int REC = rec_bytes(G);
    static constexpr int GPT = 64 / G;                 // groups per k tile
    static constexpr int ROWS = MB * 8;                // rows of a pass; ROWS * HALVES = tf_padded_rows(M) for every M of the bucket
    static constexpr int XTILE = ROWS * (128 + 4 * GPT);   // packed activation bytes per k tile and pass
    static constexpr int W_BYTES = kWarps * KTS * REC;
    static constexpr int X_BYTES = KTS * XTILE;
    static constexpr int STAGE_BYTES = ((W_BYTES + X_BYTES + 127) / 128) * 128;
    static constexpr int CW = kWarps / T;               // consumer warps
    // With 64 rows the eight consumer warps want more than the 168 registers a thread that nine warps get (the allocation
    // is by four warps): the producer's warp group hands its own over (256 x 216 + 128 x 72 = the 384 x 168 of the launch).
    static constexpr bool REGS = MB >= 8;
    static constexpr int THREADS = REGS ? 384 : (CW + 1) * 32;       // consumers + producer warp
    static_assert(!REGS || CW == 8, "two consumer warp groups");
    // the ring takes the SM's shared memory (1 KB belongs to the system)
    static constexpr int BUDGET = 226 * 1024 - 512;
    static constexpr int STAGES = BUDGET / (STAGE_BYTES + 16) > 12 ? 12 : BUDGET / (STAGE_BYTES + 16);
    static constexpr int SMEM = STAGES * STAGE_BYTES + 2 * STAGES * 8 + 128;
    static_assert(STAGES >= 2, "the ring needs at least two stages");
};

// Optional per-CTA timeline for profiling: when set (tf_qmm_set_trace), each launch writes eight
// globaltimer stamps per CTA: 0 kernel entry, 1 first weight copy issued, 2 predecessor's memory visible
// (griddepcontrol.wait passed), 3 consumers past their first full barrier, 4 main loop done, 5 a cut block's
// segment parked, 6 its ordered sum done, 7 producer's last copy issued, 9 end.
__device__ unsigned long long* g_trace = nullptr;
__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
constexpr int kTraceLaunches = 512, kTraceSlots = 16;
// layout: [148] per-CTA launch counters, then [launch % 512][cta][16] stamps
__device__ __forceinline__ void stamp(unsigned long long* tr, int slot) {
    if (tr != nullptr) tr[blockIdx.x * kTraceSlots + slot] = now_ns();
}

struct Args {
    const uint8_t* xp;
    const uint8_t* w;
    void* y;
    uint32_t* epochs;
    uint32_t* flags;
    float* slots;
    float* packets;
    int* status;
    int M, N, K;
    int f32_out;
    // grouped form (MoE experts): `max_probs` problems of 8 rows each, problem p multiplying its own
    // packed rows (xp + p * xp_stride) with the weight of expert prob_expert[p] (w + e * w_stride)
    // into y + p * y_stride elements; the live count is read on the device. nullptr: one problem.
    // With prob_sel, the launch covers the problems prob_sel[0 .. count) only (an expert-parallel rank's
    // own experts); addresses are still formed from the selected problem's index.
    // the matmul that runs next on this stream (may be null): once this kernel's own copies are all
    // issued, each worker asks L2 for the first bytes the SAME worker of that launch will stream
    const uint8_t* next_w;
    int next_N, next_K, next_group, prefetch_bytes;
    // tensor-parallel partial (may be null): instead of y, the fp32 sums go as 16-byte packets
    // {row 2i, n, row 2i+1, n} (n = exchange number = *peer_seq + 1) into block peer_rank of slot n & 1 of
    // EVERY rank's exchange buffer (plain peer stores); the consuming norm kernel waits for the number
    uint8_t* const* peer_bufs;
    const uint32_t* peer_seq;
    size_t peer_slot_bytes;
    int peer_rank, peer_world;
    // SwiGLU epilogue (may be null): the weight is a [gate; up] stack interleaved by column tile (tile 2a = gate
    // columns 16a..16a+15, tile 2a+1 = up columns 16a..16a+15), a consumer warp owns both tiles of an activation tile,
    // and instead of y the block's owner writes bf16(silu(bf16 gate) * bf16 up) with its group sums as the packed
    // input of the down projection (N / 2 inputs) - the bits the separate SwiGLU kernel would write
    uint8_t* act_packed;
    const int* prob_expert;
    const int* prob_count;
    const int* prob_sel;
    int max_probs;
    long long w_stride, xp_stride, y_stride;
};

// Work items (column block, group of item_tiles_for k tiles) are split evenly over kWorkers CTAs.
// cta * total stays below 2^31: the entry points refuse shapes with more than 2^30 / kWorkers items
__host__ __device__ inline int range_begin(int cta, int total) { return (int)((unsigned)cta * (unsigned)total / (unsigned)kWorkers); }

// the worker that holds item i: the last one whose range begins at or before it
__device__ __forceinline__ int holder(int i, int total) { return (int)(((unsigned)(i + 1) * (unsigned)kWorkers + (unsigned)total - 1u) / (unsigned)total) - 1; }

constexpr size_t kSlotFloats = (size_t)TF_QMM_MAX_ROWS * kCols;
// scratch: [ticket words of the wide-row kernel][parked segments, two slots of 128 x 256 floats a worker]
//          [launch numbers, one a worker][ready flags][packets]
constexpr size_t kEpochOffset = TF_QMM_COUNTER_BYTES + 2 * kWorkers * kSlotFloats * sizeof(float);
// ready flags of the parked segments (two a worker), behind the launch numbers; each in a 128-byte line of its own worker
constexpr size_t kFlagOffset = kEpochOffset + 1024;
constexpr size_t kFlagStride = 32;      // words
// the self-tagged packets of launches of up to 8 rows have a place that nothing else writes: a stale word there is an older tag
constexpr size_t kPacketOffset = kFlagOffset + kWorkers * kFlagStride * sizeof(uint32_t);
constexpr size_t kPacketFloats = (size_t)2 * 8 * kCols;               // a worker's segment of 8 rows, half values, half tags
constexpr size_t kScratchBytes = kPacketOffset + kWorkers * kPacketFloats * sizeof(float);

// 16-byte load that is performed every time it is executed (a polled location)
__device__ __forceinline__ float4 ld_volatile16(const float4* p) {
    float4 v;
    asm volatile("ld.volatile.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release(uint32_t* p, uint32_t v) { asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// How a column block cut along K is put together. The work items of a block are consecutive, so its
// segments belong to consecutive workers: the first segment (the block's first k items) ends one
// worker's range, every later segment starts the next worker's range. A worker therefore "parks" at
// most one segment, the first of its range, early in the kernel: each consumer thread stores its
// accumulators as 16-byte packets {value, value, launch number, launch number} (thread-major, so the
// stores coalesce; a packet is stored whole, so whoever reads this launch's number in it has the values).
// The worker that holds the block's FIRST segment is the one that finishes the block: at the end of its
// range it keeps that segment in registers, fetches the later segments' packets (again, bounded, while
// one still carries an older number), which were parked long before unless their worker started late,
// adds them in worker order, which is k order, and writes the output. No tickets, flags or fences, one
// round trip on the critical path, and nothing to reset. The launch number is the worker's own counter in scratch, advanced once
// per launch before dependents may start, so every worker of a launch holds the same number.
//
// Above 8 rows a segment is 16 to 128 KB, and one worker that fetches up to nine of them in turn was half of the
// launch (5120 x 4096 at 128 rows: 74 us). There every worker of a cut block parks its segment (plain values, then a
// fence and a ready flag that carries the launch number), and the block's workers share the sum: each adds all the
// segments of every nseg-th accumulator unit, in k order from the first segment on, and writes those outputs. All parking comes
// before any waiting, and a launch's workers are all resident, so the waits end. Only the workers that hold a segment are visited
// (fewer items than workers leave idle ones between), eight segments at a time where a worker has one unit: 64 x 5120 at 16 / 32 rows
// 9.3 / 11.1 us, 256 x 1024 6.3 / 6.9 (30 / 35 and 28 / 31 over every worker from the first to the last, two at a time).
template <class C, bool MULTI>
__global__ void __launch_bounds__(C::THREADS, 1) qmm_kernel(const Args a) {
    constexpr int MB = C::MB, KTS = C::KTS, STAGES = C::STAGES, CW = C::CW, T = C::T, NC = CW * 32;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint32_t epoch_s;
    // every thread derives the same per-launch trace base: the CTA's launch counter is bumped by thread 0
    // only after all threads have read it (the barrier below)
    unsigned long long* tr = g_trace;
    if (tr != nullptr) tr += kWorkers + (tr[blockIdx.x] % kTraceLaunches) * (kWorkers * kTraceSlots);
    if (threadIdx.x == 0) stamp(tr, 0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int KT = a.K >> 6;                              // k tiles
    const int CB = (a.N + kCols - 1) / kCols;             // column blocks
    constexpr bool multi = MULTI;      // the grouped form is its own instantiation: the plain one pays nothing for it
    // Grouped launches never cut a column block along K: where the cut falls would depend on how many
    // problems the launch holds, that is on the other rows' routing. One item = a whole (problem, block).
    const int item_tiles = multi ? ((KT + KTS - 1) / KTS) * KTS : item_tiles_for(CB, KT);
    const int SPB = (KT + item_tiles - 1) / item_tiles;   // schedule items per column block
    if (multi) pdl_wait();                                // the problem list is the previous kernel's output
    const int probs = multi ? min(*a.prob_count, a.max_probs) : 1;
    const int total = probs * CB * SPB;                   // "column block" below: (problem, column block) pairs
    const int begin = range_begin(blockIdx.x, total), end = range_begin(blockIdx.x + 1, total);

    uint8_t* stage0 = smem;
    const uint32_t bars = smem_u32(smem + STAGES * C::STAGE_BYTES);
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), CW);
        }
        mbar_fence_init();
        epoch_s = atomicAdd(a.epochs + blockIdx.x, 1u) + 1u;   // this launch's number: the same on every worker
        if (g_trace != nullptr) g_trace[blockIdx.x] += 1;
    }
    __syncthreads();
    pdl_launch_dependents();     // the next kernel may be scheduled; it still waits for this one's memory

    if (warp >= CW) {
        if constexpr (C::REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        // ------------------------------- producer: one thread ----------------------------------
        // Weights never change during a forward, so the first ring of weight copies is issued before
        // waiting for the previous kernel; the activations (its output) follow after the wait.
        if (warp == CW && lane == 0 && begin < end) {
            auto picked = [&](int q) { return (MULTI && a.prob_sel) ? a.prob_sel[q] : q; };
            // walks the range's pipeline stages: passes over the rows, items, k tiles of an item's segment
            struct Walk {
                int half, it, kt0, kt_end, gb, begin, end, SPB, KT, item_tiles;
                __device__ void open() {                             // the segment that starts at item `it`
                    gb = it / SPB;
                    const int cb_begin = gb * SPB, seg_end = min(cb_begin + SPB, end);
                    kt0 = (it - cb_begin) * item_tiles;
                    kt_end = min(KT, (seg_end - cb_begin) * item_tiles);
                }
                __device__ bool valid() const { return half < C::HALVES; }
                __device__ int nkt() const { return min(KTS, kt_end - kt0); }
                __device__ void next() {
                    kt0 += KTS;
                    if (kt0 < kt_end) return;
                    it = min((gb + 1) * SPB, end);
                    if (it == end) { ++half; it = begin; }
                    open();
                }
            };
            bool prefetched = MULTI;
            auto prefetch_next = [&] {
                prefetched = true;
                if (a.next_w == nullptr) return;
                // where this worker's range of the next matmul starts (its items are cut like this one's)
                const int nKT = a.next_K >> 6, nCB = (a.next_N + kCols - 1) / kCols, nIT = item_tiles_for(nCB, nKT), nSPB = (nKT + nIT - 1) / nIT;
                const int ntotal = nCB * nSPB;
                const int nb = range_begin(blockIdx.x, ntotal), ne = range_begin(blockIdx.x + 1, ntotal);
                const size_t tile_bytes = (size_t)kWarps * rec_bytes(a.next_group);      // one k tile of a column block
                const size_t at = ((size_t)(nb / nSPB) * nKT + (size_t)(nb % nSPB) * nIT) * tile_bytes;
                const size_t whole = (size_t)nCB * nKT * tile_bytes;
                size_t len = (size_t)(ne - nb) * nIT * tile_bytes;
                if (len > (size_t)a.prefetch_bytes) len = (size_t)a.prefetch_bytes;
                if (at + len > whole) len = whole > at ? whole - at : 0;
                for (size_t off = 0; off < len; off += 32768) {
                    const uint32_t piece = (uint32_t)(len - off < 32768 ? len - off : 32768);
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.next_w + at + off), "r"(piece) : "memory");
                }
            };
            Walk w{0, begin, 0, 0, 0, begin, end, SPB, KT, item_tiles};
            w.open();
            Walk x = w;
            int ws = 0, xs = 0, ahead = 0;                            // stages whose weights are under way and activations are not
            uint32_t phase = 1;
            auto issue_w = [&] {
                const int pq = MULTI ? w.gb / CB : 0, cb = w.gb - pq * CB, nkt = w.nkt();
                const uint8_t* wbase = a.w + (multi ? (size_t)a.prob_expert[picked(pq)] * a.w_stride : 0) + (size_t)cb * KT * (kWarps * C::REC);
                mbar_wait(empty_bar(ws), phase, a.status);
                const uint32_t wbytes = (uint32_t)(nkt * kWarps * C::REC);
                mbar_arrive_expect_tx(full_bar(ws), wbytes + (uint32_t)(nkt * C::XTILE));
                bulk_g2s(smem_u32(stage0 + ws * C::STAGE_BYTES), wbase + (size_t)w.kt0 * (kWarps * C::REC), wbytes, full_bar(ws));
                if (++ws == STAGES) { ws = 0; phase ^= 1; }
                w.next();
                ++ahead;
            };
            auto issue_x = [&] {
                const uint8_t* xbase = a.xp + (multi ? (size_t)picked(x.gb / CB) * a.xp_stride : 0);
                const uint32_t dst = smem_u32(stage0 + xs * C::STAGE_BYTES + C::W_BYTES);
                const int nkt = x.nkt();
                if constexpr (C::HALVES == 1) {
                    bulk_g2s(dst, xbase + (size_t)x.kt0 * C::XTILE, (uint32_t)(nkt * C::XTILE), full_bar(xs));
                } else {                                              // this pass's rows and sums of every k tile
                    for (int kt = 0; kt < nkt; ++kt) {
                        const uint8_t* tile = xbase + (size_t)(x.kt0 + kt) * (C::HALVES * C::XTILE);
                        bulk_g2s(dst + kt * C::XTILE, tile + x.half * (C::ROWS * 128), C::ROWS * 128, full_bar(xs));
                        for (int h = 0; h < C::GPT; ++h)
                            bulk_g2s(dst + kt * C::XTILE + C::ROWS * (128 + 4 * h),
                                     tile + C::HALVES * C::ROWS * (128 + 4 * h) + x.half * (C::ROWS * 4), C::ROWS * 4, full_bar(xs));
                    }
                }
                if (++xs == STAGES) xs = 0;
                x.next();
                --ahead;
            };
            if (!multi) {
                while (ahead < STAGES && w.valid()) {
                    issue_w();
                    if (ahead == 1) stamp(tr, 1);
                }
                if (!w.valid()) prefetch_next();
                pdl_wait();
            }
            while (x.valid()) {
                if (ahead == 0) issue_w();
                issue_x();
                if (!w.valid() && !prefetched) prefetch_next();
            }
            stamp(tr, 7);
        }
        return;
    }
    if constexpr (C::REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    pdl_wait();                  // everything below reads or writes what other kernels produce or read
    if (threadIdx.x == 0) stamp(tr, 2);
    if (begin >= end) return;

    // ----------------------------------- consumer warps ---------------------------------------
    const int g = lane >> 2, t = lane & 3;
    const int xlane = g * 128 + ((t * 16) ^ ((g & 1) << 6));   // this lane's B-operand bytes inside a row block
    // opaque to the compiler on purpose: as registers they let (w >> s) & mask | magic be one lop3
    uint32_t nib_mask = 0x000F000Fu, magic = 0x43004300u;
    asm volatile("" : "+r"(nib_mask), "+r"(magic));
    const uint32_t epoch = epoch_s;
    // one accumulator unit (16 columns x 8 rows, a lane's 4 values) of column block `cb` to its destination
    auto store_unit = [&](int cb, int prob, int half, int ti, int rb_pass, const float (&v)[4]) {
        const int col0 = cb * kCols + (warp * T + ti) * 16 + g, rb = half * MB + rb_pass;
        if (!MULTI && a.peer_bufs != nullptr) {
            // a tensor-parallel rank's partial: straight into every rank's exchange buffer, self-signalling
            const uint32_t want = *reinterpret_cast<const volatile uint32_t*>(a.peer_seq) + 1u;
            const size_t base = (want & 1u) * a.peer_slot_bytes + (size_t)a.peer_rank * ((a.M + 1) / 2) * a.N * 16;
#pragma unroll
            for (int hsel = 0; hsel < 2; ++hsel) {
                const int row = rb * 8 + 2 * t, col = col0 + hsel * 8;
                if (row < a.M && col < a.N) {
                    const size_t at = base + ((size_t)(row >> 1) * a.N + col) * 16;
                    for (int peer = 0; peer < a.peer_world; ++peer)
                        asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(a.peer_bufs[peer] + at),
                                     "r"(__float_as_uint(v[2 * hsel])), "r"(want), "r"(__float_as_uint(v[2 * hsel + 1])), "r"(want) : "memory");
                }
            }
            return;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = rb * 8 + 2 * t + (i & 1), col = col0 + (i >> 1) * 8;
            if (row < a.M && col < a.N) {
                const size_t at = (size_t)prob * a.y_stride + (size_t)row * a.N + col;
                if (a.f32_out) reinterpret_cast<float*>(a.y)[at] = v[i];
                else reinterpret_cast<__nv_bfloat16*>(a.y)[at] = f2bf(v[i]);
            }
        }
    };
    constexpr bool SHARED_SUM = MB > 1;
    int parked = 0;                      // bit 2 * half: this range's first segment is parked, bit 2 * half + 1: its last
    float acc[T][MB][4];
    int s = 0;
    uint32_t phase = 0;
#pragma unroll 1
    for (int half = 0; half < C::HALVES; ++half)
    for (int it = begin; it < end;) {
        const int gb = it / SPB, pq = MULTI ? gb / CB : 0, cb = gb - pq * CB;
        const int prob = (MULTI && a.prob_sel) ? a.prob_sel[pq] : pq;
        const int cb_begin = gb * SPB, cb_end = cb_begin + SPB;
        const int seg_begin = it, seg_end = cb_end < end ? cb_end : end;
#pragma unroll
        for (int ti = 0; ti < T; ++ti)
#pragma unroll
            for (int rb = 0; rb < MB; ++rb) acc[ti][rb][0] = acc[ti][rb][1] = acc[ti][rb][2] = acc[ti][rb][3] = 0.f;

        const int kt_end = min(KT, (seg_end - cb_begin) * item_tiles);
        for (int kt0 = (it - cb_begin) * item_tiles; kt0 < kt_end; kt0 += KTS) {
            const int nkt = min(KTS, kt_end - kt0);
            mbar_wait(full_bar(s), phase, a.status);
            if (tr != nullptr && threadIdx.x == 0 && it == begin && kt0 == (it - cb_begin) * item_tiles) stamp(tr, 3);
            const uint8_t* sb = stage0 + s * C::STAGE_BYTES;
            const uint8_t* wrec = sb + warp * T * C::REC;
            const uint8_t* xst = sb + C::W_BYTES;
#pragma unroll
            for (int kt = 0; kt < KTS; ++kt) {
                if (kt < nkt) {
                    const uint8_t* xt = xst + kt * C::XTILE;
                    const float* xsums = reinterpret_cast<const float*>(xt + C::ROWS * 128) + 2 * t;
                    uint32_t af[T][4][4];
                    float sc[T][C::GPT][2], bi[T][C::GPT][2];
#pragma unroll
                    for (int ti = 0; ti < T; ++ti) {
                        const uint8_t* rec = wrec + kt * (kWarps * C::REC) + ti * C::REC;
                        const uint4 wq = *reinterpret_cast<const uint4*>(rec + lane * 16);
                        const uint32_t wv[4] = {wq.x, wq.y, wq.z, wq.w};
#pragma unroll
                        for (int s4 = 0; s4 < 4; ++s4)
#pragma unroll
                            for (int i = 0; i < 4; ++i) af[ti][s4][i] = and_or(i ? wv[s4] >> (4 * i) : wv[s4], nib_mask, magic);
#pragma unroll
                        for (int h = 0; h < C::GPT; ++h) {
                            const uint2 p = *reinterpret_cast<const uint2*>(rec + 512 + h * 64 + g * 8);
                            sc[ti][h][0] = bf16_lo(p.x); bi[ti][h][0] = bf16_hi(p.x);
                            sc[ti][h][1] = bf16_lo(p.y); bi[ti][h][1] = bf16_hi(p.y);
                        }
                    }
                    // RP row blocks at a time: their chains of dependent products (25 cycles a step) run interleaved
                    constexpr int RP = MB == 4 ? 4 : MB > 1 ? 2 : 1;
#pragma unroll
                    for (int rb0 = 0; rb0 < MB; rb0 += RP) {
                        uint32_t xb[RP][8];
#pragma unroll
                        for (int r = 0; r < RP; ++r) {
                            const uint4 x0 = *reinterpret_cast<const uint4*>(xt + (rb0 + r) * 1024 + xlane);
                            const uint4 x1 = *reinterpret_cast<const uint4*>(xt + (rb0 + r) * 1024 + (xlane ^ 64));
                            xb[r][0] = x0.x; xb[r][1] = x0.y; xb[r][2] = x0.z; xb[r][3] = x0.w;
                            xb[r][4] = x1.x; xb[r][5] = x1.y; xb[r][6] = x1.z; xb[r][7] = x1.w;
                        }
                        constexpr int SPG = 4 / C::GPT;   // k-steps per group
#pragma unroll
                        for (int h = 0; h < C::GPT; ++h) {
                            float2 xs[RP];
                            float p[RP][T][4];
#pragma unroll
                            for (int r = 0; r < RP; ++r) xs[r] = *reinterpret_cast<const float2*>(xsums + h * C::ROWS + (rb0 + r) * 8);
#pragma unroll
                            for (int s4 = h * SPG; s4 < (h + 1) * SPG; ++s4)
#pragma unroll
                                for (int r = 0; r < RP; ++r) {
                                    const float i0 = -128.f * xs[r].x, i1 = -128.f * xs[r].y;
                                    const float start[4] = {i0, i1, i0, i1};
#pragma unroll
                                    for (int ti = 0; ti < T; ++ti) {
                                        if (s4 == h * SPG) mma_bf16_16816(p[r][ti], af[ti][s4], xb[r][2 * s4], xb[r][2 * s4 + 1], start);
                                        else mma_bf16_16816(p[r][ti], af[ti][s4], xb[r][2 * s4], xb[r][2 * s4 + 1], p[r][ti]);
                                    }
                                }
#pragma unroll
                            for (int r = 0; r < RP; ++r)
#pragma unroll
                                for (int ti = 0; ti < T; ++ti) {
                                    float* ac = acc[ti][rb0 + r];
                                    ac[0] = __fmaf_rn(bi[ti][h][0], xs[r].x, __fmaf_rn(sc[ti][h][0], p[r][ti][0], ac[0]));
                                    ac[1] = __fmaf_rn(bi[ti][h][0], xs[r].y, __fmaf_rn(sc[ti][h][0], p[r][ti][1], ac[1]));
                                    ac[2] = __fmaf_rn(bi[ti][h][1], xs[r].x, __fmaf_rn(sc[ti][h][1], p[r][ti][2], ac[2]));
                                    ac[3] = __fmaf_rn(bi[ti][h][1], xs[r].y, __fmaf_rn(sc[ti][h][1], p[r][ti][3], ac[3]));
                                }
                        }
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty_bar(s));
            if (++s == STAGES) { s = 0; phase ^= 1; }
        }
        it = seg_end;

        // ---- segment done ----
        if (tr != nullptr && threadIdx.x == 0 && seg_end == end) stamp(tr, 4);
        if constexpr (SHARED_SUM) {
            if (seg_begin > cb_begin || seg_end < cb_end) {
                const int which = seg_begin > cb_begin ? 0 : 1;        // a worker's first and last segments may both be parts
                float4* slot = reinterpret_cast<float4*>(a.slots + (size_t)(2 * blockIdx.x + which) * kSlotFloats) + half * (T * MB * NC);
#pragma unroll
                for (int ti = 0; ti < T; ++ti)
#pragma unroll
                    for (int rb = 0; rb < MB; ++rb)
                        __stcg(slot + (ti * MB + rb) * NC + threadIdx.x, make_float4(acc[ti][rb][0], acc[ti][rb][1], acc[ti][rb][2], acc[ti][rb][3]));
                __threadfence();
                named_bar_sync(4, NC);
                if (threadIdx.x == 0) st_release(a.flags + blockIdx.x * kFlagStride + 2 * half + which, epoch);
                parked |= 1 << (2 * half + which);
                if (threadIdx.x == 0) stamp(tr, 5);
                continue;
            }
        } else if (seg_begin > cb_begin) {
            // a later segment of a block some earlier worker finishes: park it (always the first of this range)
            // as 16-byte packets {value, value, launch number, launch number}: a packet is stored whole, so a
            // reader that sees this launch's number in it has the values too. No fence, no flag.
            float4* slot = reinterpret_cast<float4*>(a.packets + (size_t)blockIdx.x * kPacketFloats);
            const float tagf = __uint_as_float(epoch);
#pragma unroll
            for (int ti = 0; ti < T; ++ti)
#pragma unroll
                for (int rb = 0; rb < MB; ++rb) {
                    __stcg(slot + ((ti * MB + rb) * 2 + 0) * NC + threadIdx.x, make_float4(acc[ti][rb][0], acc[ti][rb][1], tagf, tagf));
                    __stcg(slot + ((ti * MB + rb) * 2 + 1) * NC + threadIdx.x, make_float4(acc[ti][rb][2], acc[ti][rb][3], tagf, tagf));
                }
            if (tr != nullptr && threadIdx.x == 0) stamp(tr, 5);
            continue;
        }
        if (!SHARED_SUM && seg_end < cb_end) {
            // the block's first segment: add the later ones, parked by the next workers, in worker order.
            // Up to four segments are waited for and fetched together (their latencies overlap) and then
            // added one by one, so the sum is the plain sequential one.
            int o = blockIdx.x + 1;
            bool more = true;
            while (more) {
                constexpr int SB = 4;                            // segments fetched together
                constexpr int UN = T * MB, UB = UN >= 4 ? 4 : UN;  // accumulator units (4 values each), units per fetch
                int who[SB], cnt = 0;
                for (; o < kWorkers && cnt < SB; ++o) {
                    const int ob = range_begin(o, total);
                    if (ob >= cb_end) { more = false; break; }
                    if (range_begin(o + 1, total) == ob) continue;       // a worker without work
                    who[cnt++] = o;
                }
                if (o >= kWorkers) more = false;
                if (cnt == 0) break;
#pragma unroll
                for (int u0 = 0; u0 < UN; u0 += UB) {
                    // fetch the packets of these units from every segment of the batch; a packet that does not
                    // carry this launch's number yet is fetched again (bounded)
                    float4 v[SB][UB][2];
                    bool ready = false;
                    for (int spin = 0; spin < (1 << 20) && !ready; ++spin) {
                        ready = true;
#pragma unroll
                        for (int j = 0; j < SB; ++j)
                            if (j < cnt) {
                                const float4* slot = reinterpret_cast<const float4*>(a.packets + (size_t)who[j] * kPacketFloats);
#pragma unroll
                                for (int u = 0; u < UB; ++u)
#pragma unroll
                                    for (int h = 0; h < 2; ++h) {
                                        const float4 pk = ld_volatile16(slot + ((u0 + u) * 2 + h) * NC + threadIdx.x);
                                        v[j][u][h] = pk;
                                        ready = ready && __float_as_uint(pk.z) == epoch && __float_as_uint(pk.w) == epoch;
                                    }
                            }
                    }
                    if (!ready) report(a.status, TF_ESTALL);
#pragma unroll
                    for (int j = 0; j < SB; ++j)
                        if (j < cnt) {
#pragma unroll
                            for (int u = 0; u < UB; ++u) {
                                float* ac = acc[(u0 + u) / MB][(u0 + u) % MB];
                                ac[0] += v[j][u][0].x; ac[1] += v[j][u][0].y;
                                ac[2] += v[j][u][1].x; ac[3] += v[j][u][1].y;
                            }
                        }
                }
            }
            if (tr != nullptr && threadIdx.x == 0) stamp(tr, 6);
        }
        // a whole block, or a finished one: write the output
        if constexpr (!MULTI && MB == 1 && T == 2) {
            if (a.act_packed != nullptr) {
                __shared__ float act_part[kWarps / 2][C::ROWS];
                const int at = cb * (kWarps / 2) + warp;            // activation tile: 16 inputs of the down projection
                const int q4 = at & 3;                              // its place in the down projection's k tile
                uint8_t* tile = a.act_packed + (size_t)(at >> 2) * (C::ROWS * (128 + 4 * C::GPT));
                const bool in_range = at * 16 < (a.N >> 1);
#pragma unroll
                for (int rb = 0; rb < MB; ++rb)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int row = rb * 8 + 2 * t + j;
                        float pair = 0.f;
#pragma unroll
                        for (int hsel = 0; hsel < 2; ++hsel) {
                            const float gv = round_bf16(acc[0][rb][2 * hsel + j]), uv = round_bf16(acc[1][rb][2 * hsel + j]);
                            const float ov = round_bf16(gv * sigmoidf_(gv) * uv);
                            if (in_range)
                                *reinterpret_cast<__nv_bfloat16*>(tile + row * 128 + (((2 * q4 + hsel) * 16) ^ ((row & 1) << 6)) + g * 2) = f2bf(ov);
                            // the chunk's eight values added in column order (as the separate kernel's lane does), then the pair of chunks
                            float cs = 0.f;
#pragma unroll
                            for (int i = 0; i < 8; ++i) cs += __shfl_sync(0xffffffffu, ov, i * 4 + t);
                            pair = hsel == 0 ? cs : pair + cs;
                        }
                        if (g == 0) act_part[warp][row] = pair;
                    }
                named_bar_sync(4, NC);
                constexpr int WPG = 4 / C::GPT;                     // warps (activation tiles) per group
                if ((warp % WPG) == 0 && lane < C::ROWS && in_range) {
                    float sum = act_part[warp][lane] + act_part[warp + 1][lane];
                    if (WPG == 4) sum = sum + (act_part[warp + 2][lane] + act_part[warp + 3][lane]);
                    reinterpret_cast<float*>(tile + C::ROWS * 128)[(C::GPT == 1 ? 0 : (q4 >> 1)) * C::ROWS + lane] = sum;
                }
                named_bar_sync(4, NC);
                continue;
            }
        }
#pragma unroll
        for (int ti = 0; ti < T; ++ti)
#pragma unroll
            for (int rb = 0; rb < MB; ++rb) store_unit(cb, prob, half, ti, rb, acc[ti][rb]);
    }
    if constexpr (SHARED_SUM) {
#pragma unroll 1
        for (int part = 0; part < 2 * C::HALVES; ++part) {
            if (!(parked >> part & 1)) continue;
            const int half = part >> 1, which = part & 1;
            // the cut block at this end of the range, and the workers that hold its segments, in k order
            const int gb = (which == 0 ? begin : end - 1) / SPB, cb_begin = gb * SPB, cb_end = cb_begin + SPB;
            // Fewer items than workers: every item has a worker of its own, with idle workers between. Otherwise every worker has items.
            const bool sparse = total < kWorkers;
            const int first = holder(cb_begin, total), nseg = sparse ? SPB : holder(cb_end - 1, total) - first + 1;
            const int mine = sparse ? begin - cb_begin : (int)blockIdx.x - first;
            auto worker = [&](int j) { return sparse ? holder(cb_begin + j, total) : first + j; };
            bool ready = false;
            for (int spin = 0; spin < (1 << 20) && !ready; ++spin) {
                ready = true;
                // the first segment is its worker's last part, every later one its worker's first part
                for (int j = lane; j < nseg; j += 32)
                    ready = ready && ld_acquire(a.flags + worker(j) * kFlagStride + 2 * half + (j == 0 ? 1 : 0)) == epoch;
                ready = __all_sync(0xffffffffu, ready);
            }
            if (!ready) report(a.status, TF_ESTALL);
            const float4* parts = reinterpret_cast<const float4*>(a.slots) + half * (T * MB * NC) + threadIdx.x;
            auto part_of = [&](int j) { return parts + (size_t)(2 * worker(j) + (j == 0 ? 1 : 0)) * (kSlotFloats / 4); };
            // A fetch is an L2 round trip, whatever its size: UB units of SB segments are under way together. A block of many
            // segments leaves a worker one unit, which takes more segments at a time.
            auto sum_units = [&](auto ub, auto sb) {
                constexpr int UB = decltype(ub)::value, SB = decltype(sb)::value, UN = T * MB;
#pragma unroll 1
                for (int u0 = mine; u0 < UN; u0 += UB * nseg) {
                    float4 sum[UB];
                    const float4* p0 = part_of(0);
#pragma unroll
                    for (int i = 0; i < UB; ++i)
                        if (u0 + i * nseg < UN) sum[i] = __ldcg(p0 + (u0 + i * nseg) * NC);
#pragma unroll 1
                    for (int j0 = 1; j0 < nseg; j0 += SB) {
                        float4 v[SB][UB];
#pragma unroll
                        for (int j = 0; j < SB; ++j) {
                            if (j0 + j >= nseg) continue;
                            const float4* pj = part_of(j0 + j);
#pragma unroll
                            for (int i = 0; i < UB; ++i)
                                if (u0 + i * nseg < UN) v[j][i] = __ldcg(pj + (u0 + i * nseg) * NC);
                        }
#pragma unroll
                        for (int j = 0; j < SB; ++j) {
                            if (j0 + j >= nseg) continue;
#pragma unroll
                            for (int i = 0; i < UB; ++i) { sum[i].x += v[j][i].x; sum[i].y += v[j][i].y; sum[i].z += v[j][i].z; sum[i].w += v[j][i].w; }
                        }
                    }
#pragma unroll
                    for (int i = 0; i < UB; ++i)
                        if (u0 + i * nseg < UN) {
                            const float r[4] = {sum[i].x, sum[i].y, sum[i].z, sum[i].w};
                            store_unit(gb, 0, half, (u0 + i * nseg) / MB, (u0 + i * nseg) % MB, r);
                        }
                }
            };
            if (nseg >= T * MB) sum_units(std::integral_constant<int, 1>(), std::integral_constant<int, 8>());
            else sum_units(std::integral_constant<int, MB == 2 ? 2 : 4>(), std::integral_constant<int, MB == 2 ? 4 : 2>());
            if (threadIdx.x == 0) stamp(tr, 6);
        }
    }
    if (threadIdx.x == 0) stamp(tr, 9);
}

template <class C, bool MULTI = false>
int launch(const Args& a, cudaStream_t stream) {
    static_assert(C::SMEM <= 227 * 1024, "stage ring does not fit shared memory");
    auto kern = qmm_kernel<C, MULTI>;
    // the opt-in is per device: keep one flag per device ordinal
    static bool configured[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return TF_ECUDA; }
    if (!configured[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess)
            return TF_ECUDA;
        configured[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kWorkers);
    cfg.blockDim = dim3(C::THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled(1) ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, kern, a) != cudaSuccess) { cudaGetLastError(); return TF_ECUDA; }
    return TF_OK;
}

// bytes of the next matmul's weight each worker asks L2 for (TF_QMM_PREFETCH_KB, default the ring's size)
// the peer destination of the launch being set up (tf_qmm_peer hands it to tf_qmm_next on the same thread)
struct PeerOut {
    uint8_t* const* bufs = nullptr;
    const uint32_t* seq = nullptr;
    size_t slot_bytes = 0;
    int rank = 0, world = 0;
};
thread_local PeerOut g_peer;
// the SwiGLU destination of the launch being set up (tf_qmm_act hands it to tf_qmm_next on the same thread)
thread_local uint8_t* g_act = nullptr;

inline int prefetch_bytes() {
    static const int v = [] { const char* e = std::getenv("TF_QMM_PREFETCH_KB"); return (e ? atoi(e) : 224) * 1024; }();
    return v;
}

template <int G>
int dispatch(const Args& a, cudaStream_t stream) {
    // Eight consumer warps of two column tiles in every bucket. What bounds the loop above 8 rows is the sum of the warps'
    // tensor, fma and integer instructions, not one of them: per SM, k tile and 8 rows 134 cycles of mma.sync (8.4 a
    // sub-partition and m16n8k16, 545 TFLOP/s measured) and about 64 of fma, per k tile 270 of weight expansion. 16 warps
    // of one tile, 16 warps of two tiles and half of the rows, and shorter stages measured the same or slower
    // (17408 x 5120, 32 / 64 rows: 27.4 / 51.8 us; 34.1 / 53.2 with 16 warps of one tile; 31.7 / 59.8).
    // 128 rows take the 64-row pass twice (92 us, the weights' second pass comes out of L2): 128 accumulators a thread spill
    // (104 us, and 143 us as 16 warps of one tile with one owner adding up the K segments).
    if (a.M <= 8) return launch<Cfg<G, 1, 4, 2>>(a, stream);
    if (a.M <= 16) return launch<Cfg<G, 2, 4, 2>>(a, stream);
    if (a.M <= 32) return launch<Cfg<G, 4, 4, 2>>(a, stream);
    if (a.M <= 64) return launch<Cfg<G, 8, 2, 2>>(a, stream);
    return launch<Cfg<G, 8, 2, 2, 2>>(a, stream);
}

// ---- relayout kernels: one thread per output word / pair -----------------------------------------
__device__ __forceinline__ size_t record_offset(int col_tile, int kt, int KT, int REC) {
    return (((size_t)(col_tile / kWarps) * KT + kt) * kWarps + (col_tile % kWarps)) * REC;
}

__global__ void tile_kernel(const uint32_t* words, const uint16_t* scales, const uint16_t* biases, uint8_t* out,
                            int N, int K, int G) {
    const int KT = K >> 6, CB = (N + kCols - 1) / kCols, REC = rec_bytes(G), GPT = 64 / G;
    const long long recs = (long long)CB * kWarps * KT;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int per = 128 + 16 * GPT;                 // threads per record: 128 words + 16*GPT (s,b) pairs
    if (id >= recs * per) return;
    const long long rec = id / per;
    const int e = (int)(id % per);
    const int c = (int)(rec / KT), kt = (int)(rec % KT);
    uint8_t* r = out + record_offset(c, kt, KT, REC);
    if (e < 128) {
        const int lane = e >> 2, s = e & 3, g = lane >> 2, t = lane & 3;
        uint32_t w = 0;
        for (int j = 0; j < 8; ++j) {
            const int col = 16 * c + g + 8 * (j & 1);
            const int k = 64 * kt + tile_k(t, s, nibble_quad(j));
            uint32_t q = 0;
            if (col < N) q = (words[(size_t)col * (K >> 3) + (k >> 3)] >> (4 * (k & 7))) & 0xFu;
            w |= q << (4 * j);
        }
        reinterpret_cast<uint32_t*>(r)[e] = w;
    } else {
        const int p = e - 128, h = p >> 4, q = p & 15, g = q >> 1, hi = q & 1;
        const int col = 16 * c + g + 8 * hi, grp = kt * GPT + h;
        uint16_t s = 0, b = 0;
        if (col < N) { s = scales[(size_t)col * (K / G) + grp]; b = biases[(size_t)col * (K / G) + grp]; }
        uint16_t* dst = reinterpret_cast<uint16_t*>(r + 512 + h * 64 + g * 8 + hi * 4);
        dst[0] = s; dst[1] = b;
    }
}

__global__ void untile_kernel(const uint8_t* in, uint32_t* words, uint16_t* scales, uint16_t* biases, int N, int K,
                              int G) {
    const int KT = K >> 6, REC = rec_bytes(G), GPT = 64 / G;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long nwords = (long long)N * (K >> 3), npairs = (long long)N * (K / G);
    if (id < nwords) {
        const int col = (int)(id / (K >> 3)), wi = (int)(id % (K >> 3));
        uint32_t w = 0;
        for (int i = 0; i < 8; ++i) {
            const int k = wi * 8 + i, kt = k >> 6, kin = k & 63, t = (kin >> 3) & 3, s = 2 * (kin >> 5) + ((kin >> 2) & 1),
                      quad = kin & 3;
            const int c = col >> 4, cin = col & 15, g = cin & 7, hi = cin >> 3;
            // inverse of nibble_quad: quad {0,1,2,3} sits at (j>>1) = {0,2,1,3}
            const int j = hi + 2 * (((quad & 1) << 1) | (quad >> 1));
            const uint32_t v = reinterpret_cast<const uint32_t*>(in + record_offset(c, kt, KT, REC))[(g * 4 + t) * 4 + s];
            w |= ((v >> (4 * j)) & 0xFu) << (4 * i);
        }
        words[id] = w;
    } else if (id < nwords + npairs) {
        const long long p = id - nwords;
        const int col = (int)(p / (K / G)), grp = (int)(p % (K / G));
        const int kt = grp / GPT, h = grp % GPT, c = col >> 4, cin = col & 15, g = cin & 7, hi = cin >> 3;
        const uint16_t* src =
            reinterpret_cast<const uint16_t*>(in + record_offset(c, kt, KT, REC) + 512 + h * 64 + g * 8 + hi * 4);
        scales[p] = src[0];
        biases[p] = src[1];
    }
}

// Row-major bf16 rows -> packed activations (+ group sums). One lane per 8 contiguous inputs:
// sequential sum of 8, then a pairwise tree across the G/8 lanes of a group.
template <int G>
__global__ void pack_rows_kernel(const __nv_bfloat16* x, uint8_t* xp, float* xs_out, int M, int K) {
    // The wait comes before the trigger: the matmul behind copies its first ring of weights without waiting, and a weight may
    // have been written by the kernel in front of this one. Back to back, 1 row x 1024 x 5120 takes 11.7 us, 8 rows x 17408 x 5120
    // 18.9 (11.2 and 17.4 with the trigger first, where nothing orders those copies behind the writer).
    pdl_wait();
    pdl_launch_dependents();
    const int Mp = tf_padded_rows(M);
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long chunks = (long long)Mp * (K >> 3);
    const int row = (int)(id / (K >> 3)), c = (int)(id % (K >> 3));       // chunk c = inputs 8c..8c+7
    uint4 v = make_uint4(0, 0, 0, 0);
    if (id < chunks && row < M) v = reinterpret_cast<const uint4*>(x)[(size_t)row * (K >> 3) + c];
    const float s = group_sum8<G>(v);
    if (id >= chunks) return;
    packed_store<G>(xp, Mp, row, c, v, s);
    if ((c & (G / 8 - 1)) == 0 && xs_out != nullptr && row < M) xs_out[(size_t)row * (K / G) + c / (G / 8)] = s;
}

}  // namespace
}  // namespace tf

extern "C" {

int tf_version(void) { return 1001; }

int tf_qmm_set_trace(void* stamps) {
    unsigned long long* p = static_cast<unsigned long long*>(stamps);
    return cudaMemcpyToSymbol(tf::g_trace, &p, sizeof(p)) == cudaSuccess ? TF_OK : TF_ECUDA;
}
int tf_qmm_workers(void) { return tf::kWorkers; }

size_t tf_qmm_tiled_bytes(int N, int K, int group) {
    if (N <= 0 || K <= 0 || K % 64 || (group != 64 && group != 32)) return 0;
    return (size_t)((N + tf::kCols - 1) / tf::kCols) * tf::kWarps * (K / 64) * tf::rec_bytes(group);
}

size_t tf_packed_bytes(int M, int K, int group) {
    if (M <= 0 || K <= 0 || K % 64 || (group != 64 && group != 32)) return 0;
    return (size_t)(K / 64) * tf::tf_padded_rows(M) * (128 + 4 * (64 / group));
}

size_t tf_qmm_scratch_bytes(void) {
    return tf::kScratchBytes;
}

int tf_qmm(const void* x_packed, const void* w_tiled, void* y, void* scratch, size_t scratch_bytes, int M, int N, int K,
           int group, int flags, int* status, void* stream) {
    return tf_qmm_next(x_packed, w_tiled, y, scratch, scratch_bytes, M, N, K, group, flags, nullptr, 0, 0, 0, status, stream);
}

int tf_qmm_next(const void* x_packed, const void* w_tiled, void* y, void* scratch, size_t scratch_bytes, int M, int N, int K,
                int group, int flags, const void* next_w_tiled, int next_N, int next_K, int next_group, int* status, void* stream) {
    if (next_w_tiled && (next_N < 1 || next_K < 64 || next_K % 64 || (next_group != 64 && next_group != 32) || ((uintptr_t)next_w_tiled & 15)))
        return TF_EINVAL;
    if (M < 1 || M > TF_QMM_MAX_ROWS || N < 1 || K < 64 || K % 64) return TF_EINVAL;
    if (group != 64 && group != 32) return TF_EINVAL;
    if (flags & ~TF_QMM_F32_OUT) return TF_EINVAL;
    if (!x_packed || !w_tiled || (!y && tf::g_peer.bufs == nullptr && tf::g_act == nullptr)) return TF_EINVAL;
    const long long CB = (N + tf::kCols - 1) / tf::kCols, IT = tf::item_tiles_for((int)CB, K / 64), SPB = (K / 64 + IT - 1) / IT;
    if (CB * SPB > (1 << 30) / tf::kWorkers) return TF_EINVAL;
    if (((uintptr_t)x_packed | (uintptr_t)w_tiled) & 15) return TF_EALIGN;
    if ((uintptr_t)y & 3) return TF_EALIGN;
    if (!scratch || ((uintptr_t)scratch & 255)) return TF_ESCRATCH;
    if (scratch_bytes < tf_qmm_scratch_bytes()) return TF_ESCRATCH;
    tf::Args a;
    a.xp = static_cast<const uint8_t*>(x_packed);
    a.w = static_cast<const uint8_t*>(w_tiled);
    a.y = y;
    a.epochs = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(scratch) + tf::kEpochOffset);
    a.flags = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(scratch) + tf::kFlagOffset);
    a.slots = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + TF_QMM_COUNTER_BYTES);
    a.packets = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + tf::kPacketOffset);
    a.status = status;
    a.M = M; a.N = N; a.K = K;
    a.f32_out = (flags & TF_QMM_F32_OUT) ? 1 : 0;
    a.prob_expert = nullptr; a.prob_count = nullptr; a.prob_sel = nullptr; a.max_probs = 1;
    a.w_stride = a.xp_stride = a.y_stride = 0;
    a.next_w = static_cast<const uint8_t*>(next_w_tiled); a.next_N = next_N; a.next_K = next_K; a.next_group = next_group;
    a.prefetch_bytes = tf::prefetch_bytes();
    a.peer_bufs = tf::g_peer.bufs; a.peer_seq = tf::g_peer.seq; a.peer_slot_bytes = tf::g_peer.slot_bytes;
    a.peer_rank = tf::g_peer.rank; a.peer_world = tf::g_peer.world;
    tf::g_peer = tf::PeerOut();
    if (a.peer_bufs != nullptr) a.y = nullptr;
    a.act_packed = tf::g_act;
    tf::g_act = nullptr;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return group == 64 ? tf::dispatch<64>(a, st) : tf::dispatch<32>(a, st);
}

int tf_qmm_act(const void* x_packed, const void* w_tiled, void* act_packed, void* scratch, size_t scratch_bytes, int M, int N, int K,
               int group, const void* next_w_tiled, int next_N, int next_K, int next_group, int* status, void* stream) {
    // the row bucket whose consumer warps own a gate tile and its up tile; whole activation tiles
    if (M < 1 || M > 8 || N < 32 || N % 32 || !act_packed || ((uintptr_t)act_packed & 15)) return TF_EINVAL;
    tf::g_act = static_cast<uint8_t*>(act_packed);
    const int rc = tf_qmm_next(x_packed, w_tiled, nullptr, scratch, scratch_bytes, M, N, K, group, 0, next_w_tiled, next_N, next_K,
                               next_group, status, stream);
    tf::g_act = nullptr;
    return rc;
}

int tf_qmm_peer(const void* x_packed, const void* w_tiled, void* scratch, size_t scratch_bytes, int M, int N, int K, int group,
                void* const* peer_bufs, size_t slot_bytes, const void* seq, int rank, int world, const void* next_w_tiled,
                int next_N, int next_K, int next_group, int* status, void* stream) {
    if (!peer_bufs || !seq || world < 2 || world > 64 || rank < 0 || rank >= world) return TF_EINVAL;
    if (slot_bytes < tf_peer_slot_bytes(M, N, world) || (slot_bytes & 15)) return TF_EINVAL;
    tf::g_peer.bufs = reinterpret_cast<uint8_t* const*>(peer_bufs);
    tf::g_peer.seq = static_cast<const uint32_t*>(seq);
    tf::g_peer.slot_bytes = slot_bytes; tf::g_peer.rank = rank; tf::g_peer.world = world;
    const int rc = tf_qmm_next(x_packed, w_tiled, nullptr, scratch, scratch_bytes, M, N, K, group, TF_QMM_F32_OUT, next_w_tiled, next_N,
                               next_K, next_group, status, stream);
    tf::g_peer = tf::PeerOut();
    return rc;
}

int tf_qmm_grouped(const void* x_packed, const void* w_tiled, const int* prob_expert, const int* prob_count,
                   const int* prob_sel, int max_probs, void* y, void* scratch, size_t scratch_bytes, int N, int K, int group, int flags, int* status,
                   void* stream) {
    if (max_probs < 1 || N < 1 || K < 64 || K % 64) return TF_EINVAL;
    if (group != 64 && group != 32) return TF_EINVAL;
    if (flags & ~TF_QMM_F32_OUT) return TF_EINVAL;
    if (!x_packed || !w_tiled || !y || !prob_expert || !prob_count) return TF_EINVAL;
    const long long CB = (N + tf::kCols - 1) / tf::kCols;     // one schedule item per (problem, column block)
    if (CB * max_probs > (1 << 30) / tf::kWorkers) return TF_EINVAL;
    if (((uintptr_t)x_packed | (uintptr_t)w_tiled) & 15) return TF_EALIGN;
    if ((uintptr_t)y & 3) return TF_EALIGN;
    if (!scratch || ((uintptr_t)scratch & 255)) return TF_ESCRATCH;
    if (scratch_bytes < tf_qmm_scratch_bytes()) return TF_ESCRATCH;
    tf::Args a;
    a.xp = static_cast<const uint8_t*>(x_packed);
    a.w = static_cast<const uint8_t*>(w_tiled);
    a.y = y;
    a.epochs = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(scratch) + tf::kEpochOffset);
    a.flags = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(scratch) + tf::kFlagOffset);
    a.slots = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + TF_QMM_COUNTER_BYTES);
    a.packets = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + tf::kPacketOffset);
    a.status = status;
    a.M = 8; a.N = N; a.K = K;
    a.f32_out = (flags & TF_QMM_F32_OUT) ? 1 : 0;
    a.prob_expert = prob_expert; a.prob_count = prob_count; a.prob_sel = prob_sel; a.max_probs = max_probs;
    a.next_w = nullptr; a.next_N = a.next_K = a.next_group = a.prefetch_bytes = 0;
    a.peer_bufs = nullptr; a.peer_seq = nullptr; a.peer_slot_bytes = 0; a.peer_rank = a.peer_world = 0;
    a.act_packed = nullptr;
    a.w_stride = (long long)tf_qmm_tiled_bytes(N, K, group);
    a.xp_stride = (long long)tf_packed_bytes(8, K, group);
    a.y_stride = 8ll * N;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return group == 64 ? tf::launch<tf::Cfg<64, 1, 4, 2>, true>(a, st) : tf::launch<tf::Cfg<32, 1, 4, 2>, true>(a, st);
}

int tf_qmm_tile(const void* words, const void* scales, const void* biases, void* w_tiled, int N, int K, int group,
                void* stream) {
    if (N < 1 || K < 64 || K % 64 || (group != 64 && group != 32)) return TF_EINVAL;
    if (!words || !scales || !biases || !w_tiled) return TF_EINVAL;
    const long long recs = (long long)((N + tf::kCols - 1) / tf::kCols) * tf::kWarps * (K / 64);
    const long long threads = recs * (128 + 16 * (64 / group));
    tf::tile_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint32_t*>(words), static_cast<const uint16_t*>(scales), static_cast<const uint16_t*>(biases),
        static_cast<uint8_t*>(w_tiled), N, K, group);
    return cudaGetLastError() == cudaSuccess ? TF_OK : TF_ECUDA;
}

int tf_qmm_untile(const void* w_tiled, void* words, void* scales, void* biases, int N, int K, int group,
                  void* stream) {
    if (N < 1 || K < 64 || K % 64 || (group != 64 && group != 32)) return TF_EINVAL;
    if (!words || !scales || !biases || !w_tiled) return TF_EINVAL;
    const long long threads = (long long)N * (K / 8) + (long long)N * (K / group);
    tf::untile_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint8_t*>(w_tiled), static_cast<uint32_t*>(words), static_cast<uint16_t*>(scales),
        static_cast<uint16_t*>(biases), N, K, group);
    return cudaGetLastError() == cudaSuccess ? TF_OK : TF_ECUDA;
}

int tf_pack_rows(const void* x, void* x_packed, void* xs, int M, int K, int group, void* stream) {
    if (M < 1 || K < 64 || K % 64 || (group != 64 && group != 32)) return TF_EINVAL;
    if (!x || !x_packed) return TF_EINVAL;
    if (((uintptr_t)x | (uintptr_t)x_packed) & 15) return TF_EALIGN;
    const long long chunks = (long long)tf::tf_padded_rows(M) * (K / 8);
    const unsigned blocks = (unsigned)((chunks + 255) / 256);
    void* args[] = {&x, &x_packed, &xs, &M, &K};
    const void* fn = group == 64 ? (const void*)tf::pack_rows_kernel<64> : (const void*)tf::pack_rows_kernel<32>;
    return tf::launch_pdl(fn, dim3(blocks), dim3(256), 0, static_cast<cudaStream_t>(stream), args, 3) == cudaSuccess
               ? TF_OK : (cudaGetLastError(), TF_ECUDA);
}

}  // extern "C"
