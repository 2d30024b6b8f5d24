// Gated-DeltaNet recurrence over the rows of each sequence's verify window, and the commit replay.
//
// Per (sequence, value head, value row) the fp32 state row S[0..127] (key dimension) stays in
// registers across the window's rows, split over 4 lanes of 32 values each (one or two value rows a thread):
//     S    <- S * g
//     mem   = S . k                      (fp32: per lane four 8-term fma chains combined pairwise, then a 4-lane xor tree)
//     delta = (v - mem) * beta
//     S    <- S + k * delta              (fma)
//     y     = S . q
// rows in chain order. The committed state is only read; `tf_gdn_replay` later advances it over the
// accepted rows with the same statements in the same order, so a replayed state has the bits a
// serial one-row step would have produced, and row t of a window equals the t-th serial step.
//
// q and k of the rows being processed are staged as fp32 in shared memory, 8 rows at a time, and
// shared by the 32 or 64 value rows a CTA owns.

#include "common.cuh"

namespace tf {
namespace {

constexpr int kDk = 128;            // key head dim (state row length)
constexpr int kRowUnit = 32;        // value rows come in multiples of this
constexpr int kGdnThreads = 128;    // threads per CTA of gdn_kernel: 4 lanes a value row, VR rows a thread -> 32 VR value rows
constexpr int kTile = 8;            // window rows staged per pass

// ---- two fp32 lanes in one instruction: each half rounds as its scalar counterpart does ----
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// The 32 state values a lane holds of one value row: key elements 16*i + 4*j + e as pairs (e = 0,1) and (2,3).
struct StateRow { ulonglong2 v[8]; };
__device__ __forceinline__ void load_row(StateRow& s, const float* row, int j) {
#pragma unroll
    for (int i = 0; i < 8; ++i) s.v[i] = reinterpret_cast<const ulonglong2*>(row)[i * 4 + j];
}

// One window row applied to the VR value rows a lane holds, the same statements in the chain, replay and fused
// kernels: four partial dot products per value row and lane (one per element of the float4s, eight terms each,
// so the fma chains are short), combined pairwise, then the 4-lane xor tree.
//
// A head's 128 x 128 state takes 65536 fp32 operations a window row, 512 cycles of an SM; one block alone spends about
// 1050 (measured with clock64), the rest being the two dot products' reductions, which the next statement needs, and the loads of k
// and q, which every lane of a value row's four repeats. Two value rows a thread share each load, k stays in registers
// from the first dot product to the update, and the arithmetic runs on pairs (f32x2: the same rounding, half the
// instructions): 128 warp loads of 16 bytes a head and row instead of 384.
template <int VR, bool OUT>
__device__ __forceinline__ void gdn_row_step(StateRow (&s)[VR], const float* krow, const float* qrow, int j, float decay, const float (&vval)[VR],
                                             float beta, float (&out)[VR]) {
    ulonglong2 kv[8];
    f32x2 m01[VR], m23[VR];
    const f32x2 decay2 = pack2(decay, decay);
#pragma unroll
    for (int r = 0; r < VR; ++r) m01[r] = m23[r] = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        kv[i] = *reinterpret_cast<const ulonglong2*>(krow + i * 16 + j * 4);
#pragma unroll
        for (int r = 0; r < VR; ++r) {
            s[r].v[i].x = mul2(s[r].v[i].x, decay2);
            s[r].v[i].y = mul2(s[r].v[i].y, decay2);
            m01[r] = fma2(s[r].v[i].x, kv[i].x, m01[r]);
            m23[r] = fma2(s[r].v[i].y, kv[i].y, m23[r]);
        }
    }
    float mem[VR];
#pragma unroll
    for (int r = 0; r < VR; ++r) {
        const float2 a = unpack2(m01[r]), b = unpack2(m23[r]);
        mem[r] = (a.x + a.y) + (b.x + b.y);
    }
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1)
#pragma unroll
        for (int r = 0; r < VR; ++r) mem[r] += __shfl_xor_sync(0xffffffffu, mem[r], o);
    f32x2 delta[VR], o01[VR], o23[VR];
#pragma unroll
    for (int r = 0; r < VR; ++r) {
        const float d = (vval[r] - mem[r]) * beta;
        delta[r] = pack2(d, d);
        o01[r] = o23[r] = 0;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        ulonglong2 qv = make_ulonglong2(0, 0);
        if (OUT) qv = *reinterpret_cast<const ulonglong2*>(qrow + i * 16 + j * 4);
#pragma unroll
        for (int r = 0; r < VR; ++r) {
            s[r].v[i].x = fma2(kv[i].x, delta[r], s[r].v[i].x);
            s[r].v[i].y = fma2(kv[i].y, delta[r], s[r].v[i].y);
            if (OUT) {
                o01[r] = fma2(s[r].v[i].x, qv.x, o01[r]);
                o23[r] = fma2(s[r].v[i].y, qv.y, o23[r]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < VR; ++r) {
        out[r] = 0.f;
        if (OUT) {
            const float2 a = unpack2(o01[r]), b = unpack2(o23[r]);
            out[r] = (a.x + a.y) + (b.x + b.y);
        }
    }
    if (OUT) {
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1)
#pragma unroll
            for (int r = 0; r < VR; ++r) out[r] += __shfl_xor_sync(0xffffffffu, out[r], o);
    }
}

struct GdnArgs {
    const __nv_bfloat16* q;         // [R, KH, 128]   (unused by replay)
    const __nv_bfloat16* k;         // [R, KH, 128]
    const __nv_bfloat16* v;         // [R, VH, DV]
    const float* g;                 // [R, VH]
    const float* beta;              // [R, VH]
    const float* state_in;          // [S, VH, DV, 128]
    float* state_out;               // same shape, or null
    __nv_bfloat16* y;               // [R, VH, DV], or null
    const int* seq_start;           // [S + 1] first packed row of each sequence
    const int* keep;                // [S] rows to apply (null: all rows of the window)
    int KH, VH, DV;
    // several layers in one launch (commit): element strides between layers, 0 for one layer
    long long rec_q, rec_v, rec_g, rec_state;
    int S;
};

template <bool OUT, int VR, int CTAS>
__global__ void __launch_bounds__(kGdnThreads, CTAS) gdn_kernel(const GdnArgs a) {
    constexpr int THREADS = kGdnThreads, kRowsPerCta = kRowUnit * VR;
    __shared__ __align__(16) float ks[kTile][kDk];
    __shared__ __align__(16) float qs[OUT ? kTile : 1][kDk];
    __shared__ float vs[kTile][kRowsPerCta];
    __shared__ float gs[kTile], bs[kTile];
    pdl_launch_dependents();
    pdl_wait();
    const int layer = blockIdx.z / a.S, seq = blockIdx.z % a.S, head = blockIdx.y;
    const int tid = threadIdx.x, j = tid & 3, lr = tid >> 2;       // this thread's value rows: lr (and lr + 32) of the CTA's
    const int dv0 = blockIdx.x * kRowsPerCta;
    const int kh = head / (a.VH / a.KH);
    const int r0 = a.seq_start[seq];
    int n = a.seq_start[seq + 1] - r0;
    if (a.keep != nullptr) n = min(n, a.keep[seq]);
    const __nv_bfloat16* qp = a.q + layer * a.rec_q;
    const __nv_bfloat16* kp = a.k + layer * a.rec_q;
    const __nv_bfloat16* vp = a.v + layer * a.rec_v;
    const float* gp = a.g + layer * a.rec_g;
    const float* bp = a.beta + layer * a.rec_g;

    // lane j of a value row holds key elements 16*i + 4*j + e (i = 0..7, e = 0..3): 16-byte loads that coalesce
    StateRow s[VR];
    size_t srow[VR];
    bool live[VR];
#pragma unroll
    for (int x = 0; x < VR; ++x) {
        const int dvrow = dv0 + lr + x * kRowUnit;
        live[x] = dvrow < a.DV;
        srow[x] = (size_t)layer * a.rec_state + (((size_t)seq * a.VH + head) * a.DV + dvrow) * kDk;
        if (live[x]) load_row(s[x], a.state_in + srow[x], j);
        else {
#pragma unroll
            for (int i = 0; i < 8; ++i) s[x].v[i] = make_ulonglong2(0, 0);
        }
    }

    for (int t0 = 0; t0 < n; t0 += kTile) {
        const int rows = min(kTile, n - t0);
        __syncthreads();
        // 16-byte loads: 8 bf16 values of a key/query row, or of a row's 64 values, per thread
        for (int e = tid; e < rows * (kDk / 8); e += THREADS) {
            const int r = e / (kDk / 8), d = (e % (kDk / 8)) * 8;
            const size_t at = ((size_t)(r0 + t0 + r) * a.KH + kh) * kDk + d;
            float f[8];
            unpack8(*reinterpret_cast<const uint4*>(kp + at), f);
#pragma unroll
            for (int i = 0; i < 8; ++i) ks[r][d + i] = f[i];
            if (OUT) {
                unpack8(*reinterpret_cast<const uint4*>(qp + at), f);
#pragma unroll
                for (int i = 0; i < 8; ++i) qs[r][d + i] = f[i];
            }
        }
        for (int e = tid; e < rows * (kRowsPerCta / 8); e += THREADS) {
            const int r = e / (kRowsPerCta / 8), c = (e % (kRowsPerCta / 8)) * 8;
            float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (dv0 + c < a.DV) unpack8(*reinterpret_cast<const uint4*>(vp + ((size_t)(r0 + t0 + r) * a.VH + head) * a.DV + dv0 + c), f);
#pragma unroll
            for (int i = 0; i < 8; ++i) vs[r][c + i] = f[i];
        }
        if (tid < rows) {
            gs[tid] = gp[(size_t)(r0 + t0 + tid) * a.VH + head];
            bs[tid] = bp[(size_t)(r0 + t0 + tid) * a.VH + head];
        }
        __syncthreads();
        for (int r = 0; r < rows; ++r) {
            float v[VR], out[VR];
#pragma unroll
            for (int x = 0; x < VR; ++x) v[x] = vs[r][lr + x * kRowUnit];
            gdn_row_step<VR, OUT>(s, ks[r], qs[OUT ? r : 0], j, gs[r], v, bs[r], out);
            if (OUT && j < VR && (j == 0 ? live[0] : live[VR - 1]))
                a.y[((size_t)(r0 + t0 + r) * a.VH + head) * a.DV + dv0 + lr + j * kRowUnit] = f2bf(j == 0 ? out[0] : out[VR - 1]);
        }
    }
    if (a.state_out != nullptr) {
#pragma unroll
        for (int x = 0; x < VR; ++x)
            if (live[x]) {
#pragma unroll
                for (int i = 0; i < 8; ++i) reinterpret_cast<ulonglong2*>(a.state_out + srow[x])[i * 4 + j] = s[x].v[i];
            }
    }
}

// ---- the whole GDN mixer between its two projections, one launch ----------------------------------------
// One CTA of 256 threads per (value head, sequence) does, for the sequence's window rows in passes of 8:
//   1. the causal 4-tap conv + SiLU on the head's q, k and v channels, the RMS scale of q and k, the decay
//      g and the write strength beta (one warp per row, a lane's 4 channels of q, k and v: the statements of
//      gdn_pre_kernel), into shared memory, with SiLU(z) beside them; k, v, g, beta also go to the record the commit replays;
//   2. the delta-rule recurrence over the pass's rows with the fp32 state row in registers (4 lanes x 32
//      values per value row: the statements of gdn_kernel), y rounded to bf16 into shared memory;
//   3. the gated RMSNorm of y with SiLU(z) (16 lanes per row: the statements of gated_norm_kernel) written
//      as the output projection's packed input with its group sums.
// q, k, v, g, beta, y never travel through HBM between the steps and the three launches become one; every
// statement is the unfused kernel's, so the results carry the same bits.
struct GdnFusedArgs {
    const __nv_bfloat16* qkv; size_t qkv_stride;      // [R, 2*KH*128 + VH*128] conv input rows
    const __nv_bfloat16* z; size_t z_stride;          // [R, VH*128]
    const __nv_bfloat16* a_in; const __nv_bfloat16* b_in; size_t ab_stride;   // [R, VH]
    const __nv_bfloat16* conv_state;                  // [S, 3, C]
    const __nv_bfloat16* conv_w;                      // [C, 4]
    const float* a_log; const float* dt_bias;         // [VH]
    const __nv_bfloat16* norm_w;                      // [128]
    const float* state_in;                            // [S, VH, 128, 128]
    __nv_bfloat16* k_out; __nv_bfloat16* v_out; float* g_out; float* beta_out;   // the record
    uint8_t* out_packed; __nv_bfloat16* out_rows;     // [R, VH*128] packed (and optionally plain rows)
    const int* seq_start;
    int KH, VH, S, R, group;
    float eps;
};

constexpr int kFusedThreads = 256;

// CTAS: thread blocks an SM the registers are cut for. One block's time is a chain of phases (8 rows: conv 1.6 us,
// recurrence 4.4, norm 1) whose latencies only another block fills; a grid of at most one block an SM is faster with all the
// registers (32 heads x 8 rows: 9.5 against 11.7 us), a larger one with two blocks an SM (512 blocks: 33 against 36 us).
// Before the pairs, the staged conv inputs and the gates up front: 10.2 us, 38.2 for 512 blocks, 135 (now 121) for a window of 128 rows.
template <int G, int CTAS>
__global__ void __launch_bounds__(kFusedThreads, CTAS) gdn_fused_kernel(const GdnFusedArgs a) {
    __shared__ __align__(16) float ks[kTile][kDk], qs[kTile][kDk], vs[kTile][kDk], ys[kTile][kDk], zs[kTile][kDk];
    __shared__ float gs[TF_QMM_MAX_ROWS], bs[TF_QMM_MAX_ROWS];
    // conv inputs of a pass: its rows and the three before them, the head's q, k and v channels. The next pass's
    // arrive (cp.async) while this pass's recurrence runs, so that a long window pays their trip once.
    __shared__ __align__(16) __nv_bfloat16 raw[2][kTile + 3][3][kDk];
    pdl_launch_dependents();
    pdl_wait();
    const int head = blockIdx.x, seq = blockIdx.y;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int j = tid & 3, lr = tid >> 2;                          // recurrence roles: value rows lr and lr + 64, quarter of the key axis
    const int kh = head / (a.VH / a.KH);
    const int C = (2 * a.KH + a.VH) * 128;
    const int r0 = a.seq_start[seq], n = a.seq_start[seq + 1] - r0;
    const int Mp = tf_padded_rows(a.R), total = a.VH * 16;         // chunks of 8 in an output row
    // the last sequence's CTAs also zero the packed buffer's padding rows for their head
    if (seq == a.S - 1 && a.out_packed != nullptr) {
        for (int e = tid; e < (Mp - a.R) * 16; e += kFusedThreads)
            packed_store<G>(a.out_packed, Mp, a.R + e / 16, head * 16 + (e & 15), make_uint4(0, 0, 0, 0), 0.f);
    }
    if (n <= 0) return;
    // rows t0 .. t0 + rows + 2 of [conv_state (3 rows); window rows], 8 bytes a copy (the strides are multiples of four values)
    auto stage = [&](int t0, int rows, int buf) {
        for (int e = tid; e < (rows + 3) * 96; e += kFusedThreads) {
            const int i = e / 96, part = (e % 96) >> 5, src = t0 + i;
            const int ch0 = (part == 0 ? kh : part == 1 ? a.KH + kh : 2 * a.KH + head) * 128 + (e & 31) * 4;
            const __nv_bfloat16* p = src < 3 ? a.conv_state + ((size_t)seq * 3 + src) * C + ch0 : a.qkv + (size_t)(r0 + src - 3) * a.qkv_stride + ch0;
            cp_async8(smem_u32(&raw[buf][i][part][(e & 31) * 4]), p);
        }
        cp_async_commit();
    };
    stage(0, min(kTile, n), 0);
    StateRow s[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) load_row(s[x], a.state_in + (((size_t)seq * a.VH + head) * kDk + lr + x * 64) * kDk, j);
    // the window's gates, a thread a row
    for (int t = tid; t < n; t += kFusedThreads) {
        const size_t row = (size_t)(r0 + t);
        const float av = bf2f(a.a_in[row * a.ab_stride + head]), bv = bf2f(a.b_in[row * a.ab_stride + head]);
        const float ag = av + a.dt_bias[head];
        const float sp = ag > 20.0f ? ag : logf(1.0f + expf(ag));
        const float gv = expf(-expf(a.a_log[head]) * sp);
        const float bvv = sigmoidf_(bv);
        gs[t] = gv; bs[t] = bvv;
        a.g_out[row * a.VH + head] = gv;
        a.beta_out[row * a.VH + head] = bvv;
    }

    for (int t0 = 0; t0 < n; t0 += kTile) {
        const int rows = min(kTile, n - t0), buf = (t0 / kTile) & 1;
        // ---- 1. conv: warp r takes q, k and v of row r and its output gate z, side by side (each is one long dependent chain) ----
        uint4 wq[3][2];
#pragma unroll
        for (int part = 0; part < 3; ++part) {
            const int ch0 = (part == 0 ? kh : part == 1 ? a.KH + kh : 2 * a.KH + head) * 128 + lane * 4;
            const uint4* wp = reinterpret_cast<const uint4*>(a.conv_w + (size_t)ch0 * 4);
            wq[part][0] = wp[0]; wq[part][1] = wp[1];
        }
        uint2 zv = make_uint2(0, 0);                               // 8 bytes: the row stride is a multiple of four values (narrow shards)
        if (warp < rows) zv = *reinterpret_cast<const uint2*>(a.z + (size_t)(r0 + t0 + warp) * a.z_stride + head * 128 + lane * 4);
        cp_async_wait<0>();
        __syncthreads();                                           // also: the last pass's readers of the shared rows are done
        if (warp < rows) {
            const int r = warp, row = r0 + t0 + r;
            float c[4][4] = {{}, {}, {}, {bf16_lo(zv.x), bf16_hi(zv.x), bf16_lo(zv.y), bf16_hi(zv.y)}};
#pragma unroll
            for (int part = 0; part < 3; ++part) {
                float wt[16];
                {
                    float lo[8], hi[8];
                    unpack8(wq[part][0], lo);
                    unpack8(wq[part][1], hi);
#pragma unroll
                    for (int i = 0; i < 8; ++i) { wt[i] = lo[i]; wt[8 + i] = hi[i]; }
                }
#pragma unroll
                for (int tap = 0; tap < 4; ++tap) {
                    const uint2 xv = *reinterpret_cast<const uint2*>(&raw[buf][r + tap][part][lane * 4]);
                    const float xf[4] = {bf16_lo(xv.x), bf16_hi(xv.x), bf16_lo(xv.y), bf16_hi(xv.y)};
#pragma unroll
                    for (int i = 0; i < 4; ++i) c[part][i] = __fmaf_rn(xf[i], wt[i * 4 + tap], c[part][i]);
                }
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {                         // SiLU of q, k, v (rounded) and of z
                const float y = c[i >> 2][i & 3] * sigmoidf_(c[i >> 2][i & 3]);
                c[i >> 2][i & 3] = i < 12 ? round_bf16(y) : y;
            }
            *reinterpret_cast<float4*>(zs[r] + lane * 4) = make_float4(c[3][0], c[3][1], c[3][2], c[3][3]);
            float ss[2] = {0.f, 0.f};
#pragma unroll
            for (int part = 0; part < 2; ++part)
#pragma unroll
                for (int i = 0; i < 4; ++i) ss[part] += c[part][i] * c[part][i];
#pragma unroll
            for (int o = 16; o; o >>= 1)
#pragma unroll
                for (int part = 0; part < 2; ++part) ss[part] += __shfl_xor_sync(0xffffffffu, ss[part], o);
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                const float inv = 1.0f / sqrtf(ss[part] / 128.0f + 1e-6f);
                const float scale = part == 0 ? 1.0f / 128.0f : 0.08838834764831845f;   // 1/dk, dk^-1/2
                const uint2 packed = make_uint2(pack_bf16(c[part][0] * inv * scale, c[part][1] * inv * scale),
                                                pack_bf16(c[part][2] * inv * scale, c[part][3] * inv * scale));
                *reinterpret_cast<float4*>((part == 0 ? qs[r] : ks[r]) + lane * 4) =
                    make_float4(bf16_lo(packed.x), bf16_hi(packed.x), bf16_lo(packed.y), bf16_hi(packed.y));
                // one of the value heads that share this key head keeps k for the commit
                if (part == 1 && head % (a.VH / a.KH) == 0)
                    *reinterpret_cast<uint2*>(a.k_out + ((size_t)row * a.KH + kh) * 128 + lane * 4) = packed;
            }
            *reinterpret_cast<float4*>(vs[r] + lane * 4) = make_float4(c[2][0], c[2][1], c[2][2], c[2][3]);
            *reinterpret_cast<uint2*>(a.v_out + ((size_t)row * a.VH + head) * 128 + lane * 4) = make_uint2(pack_bf16(c[2][0], c[2][1]), pack_bf16(c[2][2], c[2][3]));
        }
        // the next pass's conv inputs and the norm's weight: their trips hide behind the recurrence
        if (t0 + kTile < n) stage(t0 + kTile, min(kTile, n - t0 - kTile), buf ^ 1);
        const uint4 w_pre = reinterpret_cast<const uint4*>(a.norm_w)[lane & 15];
        __syncthreads();
        // ---- 2. recurrence over the pass's rows ----
        for (int r = 0; r < rows; ++r) {
            const float v[2] = {vs[r][lr], vs[r][lr + 64]};
            float out[2];
            gdn_row_step<2, true>(s, ks[r], qs[r], j, gs[t0 + r], v, bs[t0 + r], out);
            if (j < 2) ys[r][lr + j * 64] = round_bf16(j == 0 ? out[0] : out[1]);
        }
        __syncthreads();
        // ---- 3. gated norm + packing: 16 lanes per row, 8 values a lane ----
        if (warp * 2 < rows) {
            const int r = warp * 2 + (lane >> 4), l16 = lane & 15;
            const bool live = r < rows;
            const int row = r0 + t0 + (live ? r : 0);
            __align__(16) float yv[8], zv[8];
            float wv[8], o[8];
            float ss = 0.f;
            uint4 ov = make_uint4(0, 0, 0, 0);
            if (live) {
#pragma unroll
                for (int i = 0; i < 8; i += 4) {
                    *reinterpret_cast<float4*>(yv + i) = *reinterpret_cast<const float4*>(ys[r] + l16 * 8 + i);
                    *reinterpret_cast<float4*>(zv + i) = *reinterpret_cast<const float4*>(zs[r] + l16 * 8 + i);
                }
                unpack8(w_pre, wv);
#pragma unroll
                for (int i = 0; i < 8; ++i) ss += yv[i] * yv[i];
            }
#pragma unroll
            for (int o2 = 1; o2 < 16; o2 <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o2);
            if (live) {
                const float inv = 1.0f / sqrtf(ss / 128.0f + a.eps);
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = zv[i] * (yv[i] * inv * wv[i]);
                ov = pack8(o);
            }
            const float gsum = group_sum8<G>(ov);
            if (live) {
                const int c = head * 16 + l16;
                if (a.out_rows != nullptr) reinterpret_cast<uint4*>(a.out_rows)[(size_t)row * total + c] = ov;
                if (a.out_packed != nullptr) packed_store<G>(a.out_packed, Mp, row, c, ov, gsum);
            }
        }
    }
}

// Conv tail after a commit: the last 3 rows of [old tail (3 rows); the sequence's kept window rows].
__global__ void conv_commit_kernel(const __nv_bfloat16* qkv, size_t qkv_stride, long long rec_qkv, __nv_bfloat16* conv_state,
                                   long long rec_state, const int* seq_start, const int* keep, int C, int S) {
    pdl_launch_dependents();
    pdl_wait();
    const int layer = blockIdx.z / S, seq = blockIdx.z % S;
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (c >= C) return;
    const int r0 = seq_start[seq];
    const int n = min(keep[seq], seq_start[seq + 1] - r0);
    __nv_bfloat16* st = conv_state + layer * rec_state + (size_t)seq * 3 * C + c;
    const __nv_bfloat16* rows = qkv + layer * rec_qkv + c;
    uint4 out[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int src = n + i;                    // index into [old tail; kept rows]
        out[i] = src < 3 ? *reinterpret_cast<const uint4*>(st + (size_t)src * C)
                         : *reinterpret_cast<const uint4*>(rows + (size_t)(r0 + src - 3) * qkv_stride);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(st + (size_t)i * C) = out[i];
}

// A value row a thread where its 32-row blocks find an SM each: a window row is then a chain of half the arithmetic (replay, 32 heads x 1 row:
// 3.4 -> 2.9 us, 4 heads x 8 rows 4.4 -> 3.7; chain, 4 heads x 8 rows 5.1 -> 4.3; the chain's 64-row blocks hide theirs from about 100 small
// blocks on: 32 heads x 8 rows 5.4 against 5.8). Larger grids take two rows a thread, for the shared loads of k and q; a replay of many
// waves with the registers of four blocks an SM (12 layers x 16 x 8 rows: 185 against 204 us), one of few with those of three
// (6 layers x 1 x 8 rows: 7.7 against 9.5).
template <bool OUT>
cudaError_t launch_gdn(GdnArgs a, int windows, void* stream) {
    const long long blocks = (long long)(a.DV / kRowUnit) * a.VH * windows;
    const bool one = blocks <= (OUT ? 100 : 148);
    const void* fn = one ? (const void*)gdn_kernel<OUT, 1, 4> : blocks > 888 ? (const void*)gdn_kernel<OUT, 2, 4> : (const void*)gdn_kernel<OUT, 2, OUT ? 4 : 3>;
    void* args[] = {&a};
    const int per = kRowUnit * (one ? 1 : 2);
    return launch_pdl(fn, dim3((a.DV + per - 1) / per, a.VH, windows), dim3(kGdnThreads), 0, static_cast<cudaStream_t>(stream), args);
}

int check(int S, int layers, int KH, int VH, int DK, int DV) {
    if (S < 1 || layers < 1 || KH < 1 || VH < 1 || VH % KH || DK != kDk || DV < 1 || DV % kRowUnit) return TF_EINVAL;
    if ((long long)S * layers > 65535) return TF_EINVAL;
    return TF_OK;
}

}  // namespace
}  // namespace tf

extern "C" {

int tf_gdn_chain(const void* q, const void* k, const void* v, const float* g, const float* beta, const float* state,
                 float* state_out, void* y, const int* seq_start, int n_seqs, int k_heads, int v_heads, int dk, int dv,
                 void* stream) {
    if (tf::check(n_seqs, 1, k_heads, v_heads, dk, dv) != TF_OK) return TF_EINVAL;
    if (!q || !k || !v || !g || !beta || !state || !y || !seq_start) return TF_EINVAL;
    if (((uintptr_t)state | (uintptr_t)state_out | (uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15) return TF_EALIGN;
    tf::GdnArgs a = {};
    a.q = static_cast<const __nv_bfloat16*>(q); a.k = static_cast<const __nv_bfloat16*>(k);
    a.v = static_cast<const __nv_bfloat16*>(v); a.g = g; a.beta = beta;
    a.state_in = state; a.state_out = state_out; a.y = static_cast<__nv_bfloat16*>(y);
    a.seq_start = seq_start; a.keep = nullptr;
    a.KH = k_heads; a.VH = v_heads; a.DV = dv; a.S = n_seqs;
    const cudaError_t e = tf::launch_gdn<true>(a, n_seqs, stream);
    if (e != cudaSuccess) { cudaGetLastError(); return TF_ECUDA; }
    return TF_OK;
}

int tf_gdn_fused(const void* qkv, size_t qkv_stride, const void* z, size_t z_stride, const void* a, const void* b, size_t ab_stride,
                 const void* conv_state, const void* conv_w, const float* a_log, const float* dt_bias, const void* norm_w,
                 const float* state, void* k_out, void* v_out, float* g_out, float* beta_out, void* out_packed, void* out_rows,
                 const int* seq_start, int rows, int n_seqs, int k_heads, int v_heads, int dk, int dv, int taps, int group, float eps,
                 void* stream) {
    if (rows < 1 || rows > TF_QMM_MAX_ROWS || n_seqs < 1 || n_seqs > 65535 || k_heads < 1 || v_heads < 1 || v_heads % k_heads) return TF_EINVAL;
    if (dk != 128 || dv != 128 || taps != 4 || (group != 64 && group != 32)) return TF_EINVAL;
    if (!qkv || !z || !a || !b || !conv_state || !conv_w || !a_log || !dt_bias || !norm_w || !state || !seq_start) return TF_EINVAL;
    if (!k_out || !v_out || !g_out || !beta_out || (!out_packed && !out_rows) || qkv_stride % 4 || z_stride % 4) return TF_EINVAL;
    if (((uintptr_t)qkv | (uintptr_t)conv_state | (uintptr_t)k_out | (uintptr_t)v_out) & 7) return TF_EALIGN;
    if (((uintptr_t)z) & 7) return TF_EALIGN;
    if (((uintptr_t)conv_w | (uintptr_t)norm_w | (uintptr_t)state | (uintptr_t)out_packed | (uintptr_t)out_rows) & 15) return TF_EALIGN;
    tf::GdnFusedArgs g = {};
    g.qkv = static_cast<const __nv_bfloat16*>(qkv); g.qkv_stride = qkv_stride;
    g.z = static_cast<const __nv_bfloat16*>(z); g.z_stride = z_stride;
    g.a_in = static_cast<const __nv_bfloat16*>(a); g.b_in = static_cast<const __nv_bfloat16*>(b); g.ab_stride = ab_stride;
    g.conv_state = static_cast<const __nv_bfloat16*>(conv_state); g.conv_w = static_cast<const __nv_bfloat16*>(conv_w);
    g.a_log = a_log; g.dt_bias = dt_bias; g.norm_w = static_cast<const __nv_bfloat16*>(norm_w); g.state_in = state;
    g.k_out = static_cast<__nv_bfloat16*>(k_out); g.v_out = static_cast<__nv_bfloat16*>(v_out); g.g_out = g_out; g.beta_out = beta_out;
    g.out_packed = static_cast<uint8_t*>(out_packed); g.out_rows = static_cast<__nv_bfloat16*>(out_rows);
    g.seq_start = seq_start; g.KH = k_heads; g.VH = v_heads; g.S = n_seqs; g.R = rows; g.group = group; g.eps = eps;
    void* args[] = {&g};
    const bool one = (long long)v_heads * n_seqs <= 148;         // a thread block an SM at most
    const void* fn = group == 64 ? (one ? (const void*)tf::gdn_fused_kernel<64, 1> : (const void*)tf::gdn_fused_kernel<64, 2>)
                                 : (one ? (const void*)tf::gdn_fused_kernel<32, 1> : (const void*)tf::gdn_fused_kernel<32, 2>);
    cudaError_t e = tf::launch_pdl(fn, dim3(v_heads, n_seqs), dim3(tf::kFusedThreads), 0, static_cast<cudaStream_t>(stream), args);
    if (e != cudaSuccess) { cudaGetLastError(); return TF_ECUDA; }
    return TF_OK;
}

int tf_gdn_replay(const void* k, const void* v, const float* g, const float* beta, float* state, const int* seq_start,
                  const int* keep, int n_seqs, int layers, long long rec_k_stride, long long rec_v_stride,
                  long long rec_g_stride, long long state_stride, int k_heads, int v_heads, int dk, int dv, void* stream) {
    if (tf::check(n_seqs, layers, k_heads, v_heads, dk, dv) != TF_OK) return TF_EINVAL;
    if (!k || !v || !g || !beta || !state || !seq_start || !keep) return TF_EINVAL;
    if ((uintptr_t)state & 15 || state_stride % 4 || (((uintptr_t)k | (uintptr_t)v) & 15) || rec_k_stride % 8 || rec_v_stride % 8) return TF_EALIGN;
    tf::GdnArgs a = {};
    a.q = nullptr; a.k = static_cast<const __nv_bfloat16*>(k);
    a.v = static_cast<const __nv_bfloat16*>(v); a.g = g; a.beta = beta;
    a.state_in = state; a.state_out = state; a.y = nullptr;          // each thread rewrites only what it read
    a.seq_start = seq_start; a.keep = keep;
    a.KH = k_heads; a.VH = v_heads; a.DV = dv; a.S = n_seqs;
    a.rec_q = rec_k_stride; a.rec_v = rec_v_stride; a.rec_g = rec_g_stride; a.rec_state = state_stride;
    const cudaError_t e = tf::launch_gdn<false>(a, n_seqs * layers, stream);
    if (e != cudaSuccess) { cudaGetLastError(); return TF_ECUDA; }
    return TF_OK;
}

int tf_conv_commit(const void* qkv, size_t qkv_stride, long long rec_qkv_stride, void* conv_state, long long state_stride,
                   const int* seq_start, const int* keep, int n_seqs, int layers, int channels, void* stream) {
    if (n_seqs < 1 || layers < 1 || channels < 8 || channels % 8 || qkv_stride % 8) return TF_EINVAL;
    if (!qkv || !conv_state || !seq_start || !keep || (long long)n_seqs * layers > 65535) return TF_EINVAL;
    if (((uintptr_t)qkv | (uintptr_t)conv_state) & 15 || rec_qkv_stride % 8 || state_stride % 8) return TF_EALIGN;
    void* args[] = {&qkv, &qkv_stride, &rec_qkv_stride, &conv_state, &state_stride, &seq_start, &keep, &channels, &n_seqs};
    dim3 grid((channels / 8 + 127) / 128, 1, n_seqs * layers);
    cudaError_t e = tf::launch_pdl((const void*)tf::conv_commit_kernel, grid, dim3(128), 0, static_cast<cudaStream_t>(stream), args);
    if (e != cudaSuccess) { cudaGetLastError(); return TF_ECUDA; }
    return TF_OK;
}

}  // extern "C"
