// Causal grouped-query attention over the paged cache, for every head size and group.
//
//   tb_attn_prefill  queries of a ragged step; keys before the step come from the cache, keys of
//                    the step itself from the step's own K | V rows (so a ring cache can be
//                    written after attention)
//   tb_attn_decode   one query per sequence over its cached keys, cut into splits by the sequence's
//                    own length (tb_split_keys), each giving (max, sum, unnormalised output)
//   tb_attn_merge    log-sum-exp merge of the chunks in chunk order (a block per sequence and head, or, with
//                    AttnArgs.pair_lambda, per sequence and pair of heads, whose difference it finishes)
//
// The general kernels have one warp per (query, head): a lane scores one key per round with the whole query in shared
// memory, the warp folds 32 scores into the running softmax, then every lane accumulates its
// output dims over the 32 values.  Scores, softmax and PV are float32 with precise expf.
// Plain float32 prompts go in tiles of queries and keys (runs of a few tokens by the row, in the same order of sums), decode steps with rows of up to 32
// 16-byte units with lanes across a row.
// A chunk's borders depend on the sequence's own length only, never on the batch.
//
// berniehans/titan: flash_attention_2_kernel (engine/engine-cuda/kernels/flash_attention_2.cu:22-106),
// paged_attention_decode_kernel, flash_decoding_split_kernel and flash_decoding_reduce_kernel
// (kernels/paged_attention.cu:6-103, 200-309, 314-369): score = q.k / sqrt(hd), keys t <= position,
// query head h reads kv head h / (nh/nkv), partials merged with exp(m_s - m_max).
#include <float.h>

#include <atomic>

#include "attention_args.h"
#include "common.cuh"

#define ATT_MAXE 8        // head_dim <= 256 (the wide instantiation: 32 values a lane, rows up to 1,024)
#define ATT_MAXE_WIDE 32
#define ATT_WARPS 4


template <typename T> __device__ __forceinline__ void load8(const T* p, float* o);
template <> __device__ __forceinline__ void load8<float>(const float* p, float* o) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
}
template <> __device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float* o) {
    const uint4 r = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        o[2 * i] = __uint_as_float(w[i] << 16);
        o[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

// The elements of a 16-byte unit.
template <typename T> __device__ __forceinline__ void unpack16(const uint4& r, float* o);
template <> __device__ __forceinline__ void unpack16<float>(const uint4& r, float* o) {
    o[0] = __uint_as_float(r.x); o[1] = __uint_as_float(r.y); o[2] = __uint_as_float(r.z); o[3] = __uint_as_float(r.w);
}
template <> __device__ __forceinline__ void unpack16<__nv_bfloat16>(const uint4& r, float* o) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { o[2 * i] = __uint_as_float(w[i] << 16); o[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
}

// kv_row_offset with the page's size as a shift where it is a power of two (``shift`` >= 0): two divisions less a key.
__device__ __forceinline__ int page_shift(const TbKvView& c) { return (c.page_size & (c.page_size - 1)) == 0 ? 31 - __clz(c.page_size) : -1; }
__device__ __forceinline__ size_t row_offset(const TbKvView& c, int slot, int pos, int head, int shift) {
    if (shift < 0) return kv_row_offset(c, slot, pos, head);
    const int row = c.ring_rows ? pos % c.ring_rows : pos;
    const int page = c.table[(size_t)slot * c.table_width + (row >> shift)];
    return (((size_t)page * c.kv_heads + head << shift) + (row & (c.page_size - 1))) * c.head_dim;
}

// Running softmax state of one warp: every lane holds the same m and l, and acc for dims lane + 32 j.
template <int MAXE>
struct Running {
    float m, l;
    float acc[MAXE];
};

// Width of a value row (and of an output row): the key's width unless the launch says otherwise.
__device__ __host__ __forceinline__ int value_width(const AttnArgs& a) { return a.hd_v > 0 ? a.hd_v : a.hd; }

// Folds keys [lo, hi) of one sequence into ``st``.  Keys at positions >= first_new are read from the
// step's own rows (row index first_new_row + pos - first_new), earlier ones from the cache.
template <typename T, int MAXE>
__device__ __forceinline__ void attend_range(Running<MAXE>& st, const float* qs, const AttnArgs& a, int lo, int hi,
                                             int first_new, int first_new_row, int slot, int kh, int lane) {
    const int hd = a.hd, hdv = value_width(a);
    const T* knew = (const T*)a.kv_new;
    const T* cache = (const T*)a.cache.storage;
    const size_t vhalf = (cache && !a.v_alias) ? kv_half_elems(a.cache) : 0;
    const int vnew = a.v_alias ? 0 : a.nkv * hd;
    for (int base = lo; base < hi; base += 32) {
        const int kpos = base + lane;
        const bool valid = kpos < hi;
        const T* kp = nullptr;
        const T* vp = nullptr;
        if (valid) {
            if (kpos >= first_new) {
                kp = knew + (size_t)(first_new_row + kpos - first_new) * a.kv_stride + kh * hd;
                vp = kp + vnew;
            } else {
                kp = cache + kv_row_offset(a.cache, slot, kpos, kh);
                vp = kp + vhalf;
            }
        }
        float s = -FLT_MAX;
        if (valid) {
            float dot = 0.f;
            for (int e = 0; e < hd; e += 8) {
                float kv[8];
                load8<T>(kp + e, kv);
#pragma unroll
                for (int i = 0; i < 8; ++i) dot = fmaf(qs[e + i], kv[i], dot);
            }
            s = dot * a.scale;
        }
        const float m_new = fmaxf(st.m, warp_max(s));
        const float alpha = expf(st.m - m_new);           // st.m = -FLT_MAX at the start: exp(-huge) = 0
        const float p = valid ? expf(s - m_new) : 0.f;
        st.l = st.l * alpha + warp_sum(p);
        st.m = m_new;
#pragma unroll
        for (int j = 0; j < MAXE; ++j) st.acc[j] *= alpha;
        const int n_valid = min(32, hi - base);
        for (int kk = 0; kk < n_valid; ++kk) {
            const float pk = __shfl_sync(0xffffffffu, p, kk);
            const T* v = (const T*)__shfl_sync(0xffffffffu, (unsigned long long)vp, kk);
#pragma unroll
            for (int j = 0; j < MAXE; ++j) {
                const int d = lane + 32 * j;
                if (d < hdv) st.acc[j] = fmaf(pk, ldf(v + d), st.acc[j]);
            }
        }
    }
}

template <typename T>
__device__ __forceinline__ void load_query(float* qs, const T* q, int hd, int lane) {
    for (int e = lane; e < hd; e += 32) qs[e] = ldf(q + e);
    __syncwarp();
}

// ------------------------------------------------------------------ prefill
// grid (T, ceil(nh / ATT_WARPS)); warp = one head of one query token.
template <typename T, int MAXE>
__global__ void __launch_bounds__(ATT_WARPS * 32) attn_prefill_kernel(AttnArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float q_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.x, h = blockIdx.y * ATT_WARPS + warp;
    if (h >= a.nh) return;                             // (the two heads of a pair leave or stay together)
    const int hd = a.hd;
    float* qs = q_smem + warp * hd;
    load_query<T>(qs, (const T*)a.q + (size_t)t * a.q_stride + h * hd, hd, lane);
    const int seq = a.batch.seq_of[t], pos = a.batch.pos_of[t];
    const int slot = a.batch.slot_of_seq[seq];
    const int first_new = a.kv_new ? a.batch.start_pos[seq] : 0x7fffffff;
    const int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    Running<MAXE> st;
    st.m = -FLT_MAX; st.l = 0.f;
#pragma unroll
    for (int j = 0; j < MAXE; ++j) st.acc[j] = 0.f;
    if (a.keep_first > 0 && lo > 0)                    // the kept first tokens that the window has left behind
        attend_range<T, MAXE>(st, qs, a, 0, min(a.keep_first, lo), first_new, a.batch.q_start[seq], slot, h / (a.nh / a.nkv), lane);
    attend_range<T, MAXE>(st, qs, a, lo, pos + 1, first_new, a.batch.q_start[seq], slot, h / (a.nh / a.nkv), lane);
    if (a.sink) {                                     // one more term of the denominator, against the larger of the two maxima
        const float sk = a.sink[h], m_new = fmaxf(st.m, sk), alpha = expf(st.m - m_new);
        st.l = st.l * alpha + expf(sk - m_new);
#pragma unroll
        for (int j = 0; j < MAXE; ++j) st.acc[j] *= alpha;
    }
    const float inv = 1.0f / st.l;
    const int hdv = value_width(a);
    if (a.pair_lambda) {
        // heads 2p and 2p + 1 sit in neighbouring warps: the second leaves its output where its query lay, and the first
        // takes it off its own, divides by the root mean square and writes the pair's row
        if (h & 1) {
            __syncwarp();
#pragma unroll
            for (int j = 0; j < MAXE; ++j) {
                const int d = lane + 32 * j;
                if (d < hdv) qs[d] = st.acc[j] * inv;
            }
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp >> 1)) : "memory");      // the pair's two warps
        if (h & 1) return;
        const float lam = *a.pair_lambda;
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < MAXE; ++j) {
            const int d = lane + 32 * j;
            st.acc[j] = d < a.pair_width ? fmaf(-lam, qs[hd + d], st.acc[j] * inv) : 0.f;
            ss = fmaf(st.acc[j], st.acc[j], ss);
        }
        const float r = a.pair_scale / sqrtf(warp_sum(ss) / (float)a.pair_width + a.pair_eps);
        T* o = (T*)a.out + (size_t)t * a.out_stride + (h >> 1) * a.pair_width;
#pragma unroll
        for (int j = 0; j < MAXE; ++j) {
            const int d = lane + 32 * j;
            if (d < a.pair_width) stf(o + d, st.acc[j] * r);
        }
        return;
    }
    T* o = (T*)a.out + (size_t)t * a.out_stride + h * hdv;
#pragma unroll
    for (int j = 0; j < MAXE; ++j) {
        const int d = lane + 32 * j;
        if (d < hdv) stf(o + d, st.acc[j] * inv);
    }
}

// ------------------------------------------------------------------ prefill in float32, tiles of queries
// Runs of TILE_FROM tokens and more: grid (query tiles, nh), 256 threads: 64 queries of one head against tiles of 64 keys.  The kernel
// above reads every key and value once a query and head (L1 and L2 bound: 637 us for 1,125 tokens of three sequences,
// 16 heads of 64); here a tile of keys serves 64 queries.  Scores and outputs are sums in registers, 4 x 4 and
// 4 x HD / 16 a thread, two at a time (fma.rn.f32x2: float32, rounded as fmaf rounds), the weights pass through shared memory.
// Bound by the FMA pipes and shared memory: 119 us for the tokens above.  HD: the head size rounded up to 64 or 128, the rest is zero.
// Shorter runs (running sequences beside a prompt's piece, drafts): attend_row, a warp a query and head, which walks the same
// 64 keys at a time and adds in the same order, so that a query is the same bits however its prompt is cut.  By the row / in tiles, 16 heads
// of 64: 2 tokens at 4,000 273 / 535 us, 32 prompts of 20 19 / 25, 64 sequences of 100 with 1 or 2 tokens each 17 / 91; from 32 tokens on
// a tile is the faster form (a prompt of 64: 20 / 11).  Where a step has both kinds, one launch holds them: beside 63 single tokens at 4,000 the
// tiles of 64 more cost nothing.
constexpr int TILE_FROM = 32;

// One head of one query of a short run by one warp, VW neighbouring elements of the head a lane.  A lane scores two neighbouring keys of 64;
// weights and value rows' addresses pass through the warp's piece of shared memory, sixteen value rows are requested at once.
// Bound by the latency of a key's row (a lane walks it alone: a sum over a row has one order).
constexpr int TILE_Q = 64, TILE_K = 64, TILE_P = 68;       // rows of 64 in shared memory lie 68 apart: 16-byte aligned, spread over the banks
template <int VW> struct __align__(16) RowShared {
    float q[32 * VW];
    const float* v[TILE_K];
    float p[TILE_K];
};

template <int VW>
__device__ __forceinline__ void attend_row(const AttnArgs& a, RowShared<VW>& sh, int item) {
    const int lane = threadIdx.x & 31, hd = a.hd, h = item % a.nh, kh = h / (a.nh / a.nkv);
    int place = item / a.nh;
    const int seq = tb_find_run(a.batch.q_start, a.batch.B, place, [](int n) { return n < TILE_FROM ? n : 0; });
    if (seq < 0) return;
    const int t0 = a.batch.q_start[seq], first = a.batch.start_pos[seq], slot = a.batch.slot_of_seq[seq], pos = first + place;
    const int first_new = a.kv_new ? first : 0x7fffffff;
    const float* knew = (const float*)a.kv_new;
    const float* cache = (const float*)a.cache.storage;
    const size_t vhalf = cache ? kv_half_elems(a.cache) : 0;
    const int shift = page_shift(a.cache), at = lane * VW;
    {
        const float* q = (const float*)a.q + (size_t)(t0 + place) * a.q_stride + (size_t)h * hd;
        for (int d = lane; d < hd; d += 32) sh.q[d] = q[d];
        __syncwarp();
    }
    float m = -FLT_MAX, l = 0.f, o[VW];
#pragma unroll
    for (int e = 0; e < VW; ++e) o[e] = 0.f;
    const int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    for (int k0 = lo & ~(TILE_K - 1); k0 <= pos; k0 += TILE_K) {
        const float* row[2] = {nullptr, nullptr};
        bool ok[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int key = k0 + 2 * lane + j;
            ok[j] = key <= pos && key >= lo;
            if (!ok[j]) continue;
            if (key >= first_new) {
                row[j] = knew + (size_t)(t0 + key - first_new) * a.kv_stride + (size_t)kh * hd;
                sh.v[2 * lane + j] = row[j] + (size_t)a.nkv * hd;
            } else {
                row[j] = cache + row_offset(a.cache, slot, key, kh, shift);
                sh.v[2 * lane + j] = row[j] + vhalf;
            }
        }
        __syncwarp();
        const int begin = max(0, lo - k0), end = min(TILE_K, pos + 1 - k0);
        constexpr int AHEAD = 16;
        float v[AHEAD][VW];
        auto load_values = [&](int k) {
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const float* r = sh.v[min(k + u, end - 1)] + min(at, hd - VW);
                if constexpr (VW == 4) { const float4 f = *reinterpret_cast<const float4*>(r); v[u][0] = f.x; v[u][1] = f.y; v[u][2] = f.z; v[u][3] = f.w; }
                else if constexpr (VW == 2) { const float2 f = *reinterpret_cast<const float2*>(r); v[u][0] = f.x; v[u][1] = f.y; }
                else v[u][0] = *r;
            }
        };
        float s[2] = {0.f, 0.f};
        if (ok[0] || ok[1]) {
            const float* r0 = ok[0] ? row[0] : row[1];
            const float* r1 = ok[1] ? row[1] : row[0];
#pragma unroll 8
            for (int d = 0; d < hd; d += 4) {
                const float4 q4 = *reinterpret_cast<const float4*>(sh.q + d), x = *reinterpret_cast<const float4*>(r0 + d), y = *reinterpret_cast<const float4*>(r1 + d);
                s[0] = fmaf(q4.x, x.x, s[0]); s[1] = fmaf(q4.x, y.x, s[1]);
                s[0] = fmaf(q4.y, x.y, s[0]); s[1] = fmaf(q4.y, y.y, s[1]);
                s[0] = fmaf(q4.z, x.z, s[0]); s[1] = fmaf(q4.z, y.z, s[1]);
                s[0] = fmaf(q4.w, x.w, s[0]); s[1] = fmaf(q4.w, y.w, s[1]);
            }
        }
        __syncwarp();
        load_values(begin);                                // on their way while the weights are made
        float top = -FLT_MAX, p[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            s[j] = __fmul_rn(s[j], a.scale);
            if (ok[j]) top = fmaxf(top, s[j]);
        }
        const float m_new = fmaxf(m, warp_max(top)), alpha = expf(m - m_new);
#pragma unroll
        for (int j = 0; j < 2; ++j) { p[j] = ok[j] ? expf(__fsub_rn(s[j], m_new)) : 0.f; sh.p[2 * lane + j] = p[j]; }
        // the order of the tiles: four neighbouring keys one after the other, then the sixteen fours in pairs (on the odd lanes)
        const float before = __shfl_up_sync(0xffffffffu, p[0] + p[1], 1);
        float sum = (lane & 1 ? before : 0.f) + p[0] + p[1];
#pragma unroll
        for (int x = 2; x < 32; x *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, x);
        l = __fmaf_rn(l, alpha, __shfl_sync(0xffffffffu, sum, 31));
        m = m_new;
#pragma unroll
        for (int e = 0; e < VW; ++e) o[e] = __fmul_rn(o[e], alpha);
        __syncwarp();
        for (int k = begin; k < end; k += AHEAD) {
            if (k > begin) load_values(k);
#pragma unroll
            for (int u = 0; u < AHEAD; ++u)
                if (k + u < end) {
                    const float w = sh.p[k + u];
#pragma unroll
                    for (int e = 0; e < VW; ++e) o[e] = fmaf(w, v[u][e], o[e]);
                }
        }
        __syncwarp();                                      // (weights and addresses have been read)
    }
    float scale = 1.f;
    if (a.sink) {                                          // one more term of the denominator, against the larger of the two maxima
        const float sk = a.sink[h], m_new = fmaxf(m, sk);
        scale = expf(m - m_new);
        l = __fmaf_rn(l, scale, expf(sk - m_new));
    }
    const float inv = scale / l;
    float* out = (float*)a.out + (size_t)(t0 + place) * a.out_stride + (size_t)h * hd;
#pragma unroll
    for (int e = 0; e < VW; ++e) if (at < hd) out[at + e] = o[e] * inv;
}

// A step of short runs only: grid (items / 4), an item is a (token, head).
template <int VW>
__global__ void __launch_bounds__(ATT_WARPS * 32) attn_prefill_row_kernel(AttnArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ RowShared<VW> sh[ATT_WARPS];
    const int warp = threadIdx.x >> 5;
    const long long item = (long long)blockIdx.x * ATT_WARPS + warp;
    if (item < (long long)a.batch.T * a.nh) attend_row<VW>(a, sh[warp], (int)item);
}

__device__ __forceinline__ void att_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long att_twice(float v) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float att_low(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float att_high(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }

template <int HD> constexpr size_t tile_smem() { return (size_t)(2 * HD * TILE_P + TILE_K * HD + TILE_K * TILE_P) * sizeof(float); }

template <int HD>
__global__ void __launch_bounds__(256) attn_prefill_tile_kernel(AttnArgs a, int tiles_x) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float sm_tile[];
    float* qt = sm_tile;                                   // [HD][TILE_P]: queries, transposed, scaled
    float* kt = qt + HD * TILE_P;                          // [HD][TILE_P]: keys, transposed
    float* vs = kt + HD * TILE_P;                          // [TILE_K][HD]
    float* pt = vs + TILE_K * HD;                          // [TILE_K][TILE_P]: weights, transposed
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int h = blockIdx.y, kh = h / (a.nh / a.nkv), hd = a.hd;
    if ((int)blockIdx.x >= tiles_x) {                      // short runs beside the long ones, eight (token, head) a block
        const long long item = ((long long)(blockIdx.x - tiles_x) * gridDim.y + h) * 8 + (tid >> 5);
        if (item < (long long)a.batch.T * a.nh) attend_row<HD / 32>(a, reinterpret_cast<RowShared<HD / 32>*>(sm_tile)[tid >> 5], (int)item);
        return;
    }
    // which sequence, which tile of it; a sequence's last tiles, which see the most keys, start first
    int tile = blockIdx.x;
    const int seq = tb_find_run(a.batch.q_start, a.batch.B, tile, [](int n) { return n >= TILE_FROM ? (n + TILE_Q - 1) / TILE_Q : 0; });
    if (seq < 0) return;
    const int t0 = a.batch.q_start[seq], n_new = a.batch.q_start[seq + 1] - t0;
    tile = (n_new + TILE_Q - 1) / TILE_Q - 1 - tile;
    const int first = a.batch.start_pos[seq], slot = a.batch.slot_of_seq[seq];
    const int q0 = tile * TILE_Q, nq = min(TILE_Q, n_new - q0), pos0 = first + q0;
    const int first_new = a.kv_new ? first : 0x7fffffff;
    const float* knew = (const float*)a.kv_new;
    const float* cache = (const float*)a.cache.storage;
    const size_t vhalf = cache ? kv_half_elems(a.cache) : 0;
    const int shift = page_shift(a.cache);
    const int row = tid >> 2, quarter = tid & 3;           // loads: four threads a row, a row's 16-byte units in turn
    {
        const float* q = (const float*)a.q + (size_t)(t0 + q0 + min(row, nq - 1)) * a.q_stride + (size_t)h * hd;
#pragma unroll
        for (int u = 0; u < HD / 16; ++u) {
            const int d = (u * 4 + quarter) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row < nq && d < hd) v = *reinterpret_cast<const float4*>(q + d);
            qt[d * TILE_P + row] = v.x; qt[(d + 1) * TILE_P + row] = v.y; qt[(d + 2) * TILE_P + row] = v.z; qt[(d + 3) * TILE_P + row] = v.w;
        }
    }
    float m[4], l[4];
    unsigned long long o[4][HD / 32];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -FLT_MAX; l[i] = 0.f;
#pragma unroll
        for (int j = 0; j < HD / 32; ++j) o[i][j] = 0ull;
    }
    const int hi = pos0 + nq, lo = a.window > 0 ? max(0, pos0 - a.window + 1) & ~(TILE_K - 1) : 0;      // tiles of keys begin at multiples of 64: a query's sums are the same in any step
    for (int k0 = lo; k0 < hi; k0 += TILE_K) {
        const int kpos = k0 + row;
        const float* kp = nullptr;
        const float* vp = nullptr;
        if (kpos < hi) {
            if (kpos >= first_new) {
                kp = knew + (size_t)(t0 + kpos - first_new) * a.kv_stride + (size_t)kh * hd;
                vp = kp + (size_t)a.nkv * hd;
            } else {
                kp = cache + row_offset(a.cache, slot, kpos, kh, shift);
                vp = kp + vhalf;
            }
        }
        __syncthreads();                                   // the tile before has been read
        int odd = 0;                                       // a value that is not finite: it must not reach queries that do not see it
#pragma unroll
        for (int u = 0; u < HD / 16; ++u) {
            const int d = (u * 4 + quarter) * 4;
            float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), vv = kv;
            if (kp && d < hd) { kv = *reinterpret_cast<const float4*>(kp + d); vv = *reinterpret_cast<const float4*>(vp + d); }
            kt[d * TILE_P + row] = kv.x; kt[(d + 1) * TILE_P + row] = kv.y; kt[(d + 2) * TILE_P + row] = kv.z; kt[(d + 3) * TILE_P + row] = kv.w;
            *reinterpret_cast<float4*>(vs + row * HD + d) = vv;
            odd |= !(fmaxf(fmaxf(fabsf(vv.x), fabsf(vv.y)), fmaxf(fabsf(vv.z), fabsf(vv.w))) <= FLT_MAX) | (vv.x != vv.x) | (vv.y != vv.y) | (vv.z != vv.z) | (vv.w != vv.w);
        }
        odd = __syncthreads_or(odd);
        unsigned long long sc[4][2] = {};
#pragma unroll 8
        for (int d = 0; d < HD; ++d) {
            const float4 q4 = *reinterpret_cast<const float4*>(qt + d * TILE_P + ty * 4);
            const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(kt + d * TILE_P + tx * 4);
            const float qv[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const unsigned long long qq = att_twice(qv[i]);
                att_fma2(sc[i][0], qq, k2.x);
                att_fma2(sc[i][1], qq, k2.y);
            }
        }
        float p[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pos = pos0 + ty * 4 + i;
            float s[4] = {att_low(sc[i][0]), att_high(sc[i][0]), att_low(sc[i][1]), att_high(sc[i][1])};
            bool ok[4];
            float top = -FLT_MAX;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = k0 + tx * 4 + j;
                ok[j] = key <= pos && (a.window <= 0 || key > pos - a.window);
                s[j] = __fmul_rn(s[j], a.scale);           // (roundings spelled out: those of attend_row)
                if (ok[j]) top = fmaxf(top, s[j]);
            }
#pragma unroll
            for (int x = 1; x < 16; x *= 2) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
            const float m_new = fmaxf(m[i], top), alpha = expf(m[i] - m_new);      // m = -FLT_MAX at the start: the sums it scales are zero
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) { p[i][j] = ok[j] ? expf(__fsub_rn(s[j], m_new)) : 0.f; sum += p[i][j]; }
#pragma unroll
            for (int x = 1; x < 16; x *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, x);
            l[i] = __fmaf_rn(l[i], alpha, sum);
            m[i] = m_new;
            const unsigned long long aa = att_twice(alpha);
#pragma unroll
            for (int j = 0; j < HD / 32; ++j) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(o[i][j]) : "l"(aa));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(pt + (tx * 4 + j) * TILE_P + ty * 4) = make_float4(p[0][j], p[1][j], p[2][j], p[3][j]);
        __syncwarp();                                      // a warp reads the weights of its own eight rows only
        const int n_keys = min(TILE_K, hi - k0);
#pragma unroll 4
        for (int k = 0; k < n_keys; ++k) {
            const float4 p4 = *reinterpret_cast<const float4*>(pt + k * TILE_P + ty * 4);
            const float pv[4] = {p4.x, p4.y, p4.z, p4.w};
            unsigned long long v2[HD / 32];
#pragma unroll
            for (int j = 0; j < HD / 64; ++j) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(vs + k * HD + j * 64 + tx * 4);
                v2[2 * j] = v.x; v2[2 * j + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (odd && (k0 + k > pos0 + ty * 4 + i || (a.window > 0 && k0 + k <= pos0 + ty * 4 + i - a.window))) continue;
                const unsigned long long pp = att_twice(pv[i]);
#pragma unroll
                for (int j = 0; j < HD / 32; ++j) att_fma2(o[i][j], pp, v2[j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i;
        if (r >= nq) continue;
        float scale = 1.f;
        if (a.sink) {                                      // one more term of the denominator, against the larger of the two maxima
            const float sk = a.sink[h], m_new = fmaxf(m[i], sk);
            scale = expf(m[i] - m_new);
            l[i] = __fmaf_rn(l[i], scale, expf(sk - m_new));
        }
        const float inv = scale / l[i];
        float* out = (float*)a.out + (size_t)(t0 + q0 + r) * a.out_stride + (size_t)h * hd;
#pragma unroll
        for (int j = 0; j < HD / 64; ++j) {
            const int d = j * 64 + tx * 4;
            if (d < hd)
                *reinterpret_cast<float4*>(out + d) = make_float4(att_low(o[i][2 * j]) * inv, att_high(o[i][2 * j]) * inv,
                                                                  att_low(o[i][2 * j + 1]) * inv, att_high(o[i][2 * j + 1]) * inv);
        }
    }
}

template <int HD>
static int launch_tile(const AttnArgs& a, cudaStream_t stream) {
    static std::atomic<bool> configured[64];              // a device each
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 64 || !configured[dev].load()) {
        const cudaError_t e = cudaFuncSetAttribute(attn_prefill_tile_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_smem<HD>());
        TB_REQUIRE(e == cudaSuccess, "attn_prefill: cannot reserve %zu bytes of shared memory: %s", tile_smem<HD>(), cudaGetErrorString(e));
        if (dev < 64) configured[dev].store(true);
    }
    // At least the tiles of all long runs, and blocks for the tokens of the short ones (none where all runs are as long as the longest).
    const int B = a.batch.B, T = a.batch.T, most = a.batch.max_new;
    const int tiles_x = T / TILE_Q + min(B, T / TILE_FROM), others = most > 0 ? (int)min((long long)T - most, (long long)(B - 1) * (TILE_FROM - 1)) : T;
    const dim3 grid(tiles_x + (most > 0 && (long long)B * most == T ? 0 : (others + 7) / 8), a.nh);
    tb_launch(attn_prefill_tile_kernel<HD>, grid, 256, tile_smem<HD>(), stream, a, tiles_x);
    return 0;
}

static void launch_rows(const AttnArgs& a, cudaStream_t stream) {
    const unsigned blocks = (unsigned)(((long long)a.batch.T * a.nh + ATT_WARPS - 1) / ATT_WARPS);
    if (a.hd <= 32) tb_launch(attn_prefill_row_kernel<1>, dim3(blocks), ATT_WARPS * 32, 0, stream, a);
    else if (a.hd <= 64) tb_launch(attn_prefill_row_kernel<2>, dim3(blocks), ATT_WARPS * 32, 0, stream, a);
    else tb_launch(attn_prefill_row_kernel<4>, dim3(blocks), ATT_WARPS * 32, 0, stream, a);
}

// ------------------------------------------------------------------ decode, split over the keys
// grid (B, nkv, n_splits); the warps of a block take the query heads of one kv head in turn.
// Partial of (sequence b, head h, split s) at scratch[((b * nh + h) * n_splits + s) * (hd + 2)]:
// hd unnormalised outputs, then m, then l (l = 0: the split saw no key).
template <typename T, int MAXE>
__global__ void __launch_bounds__(ATT_WARPS * 32) attn_decode_kernel(AttnArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float q_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int blocks_y = a.head_blocks > 0 ? a.head_blocks : a.nkv;
    const int b = blockIdx.x, kh = (int)blockIdx.y * a.nkv / blocks_y, split = blockIdx.z;
    const int hd = a.hd, hdv = value_width(a), group = a.nh / blocks_y;
    const int len = a.batch.kv_len[b];
    const int keys = tb_split_keys(len, a.chunk, a.n_splits);
    if ((long long)split * keys >= len) return;     // the merge reads ceil(len / keys) splits only
    const int pos = len - 1;
    const int slot = a.batch.slot_of_seq[b];
    const int wlo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    const int lo = max(wlo, split * keys), hi = min(len, (split + 1) * keys);
    // the kept first tokens that lie in this split and before the window
    const int klo = split * keys, khi = a.window > 0 ? min(min(a.keep_first, wlo), hi) : 0;
    float* qs = q_smem + warp * hd;
    for (int g = warp; g < group; g += ATT_WARPS) {
        const int h = (int)blockIdx.y * group + g;
        float* part = a.scratch + ((size_t)(b * a.nh + h) * a.n_splits + split) * (hdv + 2);
        Running<MAXE> st;
        st.m = -FLT_MAX; st.l = 0.f;
#pragma unroll
        for (int j = 0; j < MAXE; ++j) st.acc[j] = 0.f;
        if (lo < hi || klo < khi) {
            __syncwarp();
            load_query<T>(qs, (const T*)a.q + (size_t)b * a.q_stride + h * hd, hd, lane);
            if (klo < khi) attend_range<T, MAXE>(st, qs, a, klo, khi, 0x7fffffff, 0, slot, kh, lane);
            if (lo < hi) attend_range<T, MAXE>(st, qs, a, lo, hi, 0x7fffffff, 0, slot, kh, lane);
        }
#pragma unroll
        for (int j = 0; j < MAXE; ++j) {
            const int d = lane + 32 * j;
            if (d < hdv) part[d] = st.acc[j];
        }
        if (lane == 0) { part[hdv] = st.m; part[hdv + 1] = st.l; }
    }
}

// The same for rows of up to 32 16-byte units (float32: 128 elements, bfloat16: 256).  LPK lanes share a key, a 16-byte unit of its row
// each, so that a load covers whole rows of 32 / LPK keys (in the kernel above every lane walks a row of its own, and a warp a
// whole split).  Each group of LPK lanes is a stream of its own: keys st, st + streams, ... of the split, eight keys and
// values requested at once, an own running softmax.  A warp merges its streams by shuffles; ``share`` warps, a power of two, take
// a head together and meet in shared memory.  They are as many as leave a stream a whole round of eight keys of the launch's ``chunk``
// (more only add parts to merge: 32 keys a split, 64 sequences of 2,000, 8 heads of 8: 2,700 us with sixteen warps a head).
// Bound by the latency of the loads at a few hundred keys a split: three
// sequences of 500 tokens, 16 heads of 64 on 8, float32: 210 -> 12.3 us a layer.
constexpr int VEC_WARPS = 16, VEC_KEYS = 8;

template <typename T, int LPK>
__global__ void __launch_bounds__(VEC_WARPS * 32) attn_decode_vec_kernel(AttnArgs a, int share) {
    constexpr int PER = 16 / (int)sizeof(T), STREAMS = 32 / LPK;
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float parts[];                   // [warps][hdv + 2]: what a warp made of its keys (share > 1)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, unit = lane % LPK;
    const int blocks_y = a.head_blocks > 0 ? a.head_blocks : a.nkv;
    const int b = blockIdx.x, kh = (int)blockIdx.y * a.nkv / blocks_y, split = blockIdx.z;
    const int hd = a.hd, hdv = value_width(a), group = a.nh / blocks_y;
    const int len = a.batch.kv_len[b];
    const int keys = tb_split_keys(len, a.chunk, a.n_splits);
    if ((long long)split * keys >= len) return;     // the merge reads ceil(len / keys) splits only
    const int pos = len - 1;
    const int slot = a.batch.slot_of_seq[b];
    const int wlo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    const int lo = max(wlo, split * keys), hi = min(len, (split + 1) * keys);
    // the kept first tokens that lie in this split and before the window
    const int klo = split * keys, khi = a.window > 0 ? min(min(a.keep_first, wlo), hi) : 0;
    if (lo >= hi && a.keep_first <= 0) return;         // a split before the window: the merge begins behind it
    const T* cache = (const T*)a.cache.storage;
    const size_t vhalf = a.v_alias ? 0 : kv_half_elems(a.cache);
    const int shift = page_shift(a.cache);
    const int streams = share * STREAMS, st = (warp % share) * STREAMS + lane / LPK;
    const int at = unit * PER, at_once = (int)(blockDim.x >> 5) / share;
    const bool key_part = at < hd, value_part = at < hdv;
    for (int g0 = 0; g0 < group; g0 += at_once) {
        const int g = g0 + warp / share;
        const int h = (int)blockIdx.y * group + min(g, group - 1);
        float q[PER], acc[PER], m = -FLT_MAX, l = 0.f;
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            q[e] = at + e < hd ? ldf((const T*)a.q + (size_t)b * a.q_stride + h * hd + at + e) : 0.f;
            acc[e] = 0.f;
        }
        auto attend = [&](int first, int last) {
            for (int base = first; base < last; base += VEC_KEYS * streams) {      // (the bounds are the warp's: its lanes stay together)
                uint4 kr[VEC_KEYS], vr[VEC_KEYS];
#pragma unroll
                for (int u = 0; u < VEC_KEYS; ++u) {
                    const T* row = cache + row_offset(a.cache, slot, min(base + u * streams + st, last - 1), kh, shift) + at;
                    kr[u] = vr[u] = make_uint4(0, 0, 0, 0);
                    if (key_part) kr[u] = *reinterpret_cast<const uint4*>(row);
                    if (value_part) vr[u] = *reinterpret_cast<const uint4*>(row + vhalf);
                }
                float s[VEC_KEYS], top = m;
#pragma unroll
                for (int u = 0; u < VEC_KEYS; ++u) {
                    float k[PER], dot = 0.f;
                    unpack16<T>(kr[u], k);
#pragma unroll
                    for (int e = 0; e < PER; ++e) dot = fmaf(q[e], k[e], dot);
#pragma unroll
                    for (int o = LPK / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
                    s[u] = dot * a.scale;
                    if (base + u * streams + st < last) top = fmaxf(top, s[u]);
                }
                const float alpha = expf(m - top);     // m = -FLT_MAX at the start: the sums it scales are zero
                m = top;
                l *= alpha;
#pragma unroll
                for (int e = 0; e < PER; ++e) acc[e] *= alpha;
#pragma unroll
                for (int u = 0; u < VEC_KEYS; ++u) {
                    if (base + u * streams + st >= last) continue;
                    const float p = expf(s[u] - m);
                    float v[PER];
                    unpack16<T>(vr[u], v);
                    l += p;
#pragma unroll
                    for (int e = 0; e < PER; ++e) acc[e] = fmaf(p, v[e], acc[e]);
                }
            }
        };
        if (g < group) {
            if (klo < khi) attend(klo, khi);
            if (lo < hi) attend(lo, hi);
        }
        // the warp's streams as one
        float top = m;
#pragma unroll
        for (int o = LPK; o < 32; o *= 2) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        const float mine = expf(m - top);              // (a stream that saw no key: its sums are zero)
        l *= mine;
#pragma unroll
        for (int e = 0; e < PER; ++e) acc[e] *= mine;
#pragma unroll
        for (int o = LPK; o < 32; o *= 2) {
            l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
            for (int e = 0; e < PER; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
        }
        float* part = a.scratch + ((size_t)(b * a.nh + h) * a.n_splits + split) * (hdv + 2);
        float* to = share == 1 ? part : parts + warp * (hdv + 2);
        if (g0 > 0 && share > 1) __syncthreads();      // the heads before have been read
        if (lane < LPK && (share > 1 || g < group)) {
#pragma unroll
            for (int e = 0; e < PER; ++e) if (at + e < hdv) to[at + e] = acc[e];
            if (unit == 0) { to[hdv] = top; to[hdv + 1] = l; }
        }
        if (share == 1) continue;
        __syncthreads();
        if (g >= group) continue;                      // (every warp takes every turn of the loop)
        const float* of = parts + warp / share * share * (hdv + 2);      // the head's warps lie side by side
        float all = -FLT_MAX, sum = 0.f;
        for (int w = 0; w < share; ++w) all = fmaxf(all, of[w * (hdv + 2) + hdv]);
        for (int d = (warp % share) * 32 + lane; d < hdv + 1; d += share * 32) {      // (place hdv: the weights' sum)
            sum = 0.f;
            for (int w = 0; w < share; ++w) {
                const float* p = of + w * (hdv + 2);
                sum = fmaf(expf(p[hdv] - all), p[d < hdv ? d : hdv + 1], sum);
            }
            part[d < hdv ? d : hdv + 1] = sum;
        }
        if (warp % share == 0 && lane == 0) part[hdv] = all;
    }
}

// The splits of NH neighbouring heads (h0 ..) merged for output dims ``d0 + threadIdx.x + blockDim.x * j``: acc[k][j] =
// sum_s exp(m_s - m) acc_s and l[k] = sum_s exp(m_s - m) l_s (the sink's term included), both in the order of the splits.  The
// block first turns the splits' (m, l) pairs into weights, a thread a split, MERGE_TILE splits at a time; the loads of the
// sums then wait for nothing but the weights in shared memory.  Splits that saw no key (l = 0) get the weight zero.
#define MERGE_TILE 128
template <int NH, int PER>
__device__ __forceinline__ void merge_splits(const AttnArgs& a, int b, int h0, int hd, int d0, int used, int first, float (&acc)[NH][PER], float (&l)[NH]) {
    __shared__ float sm[NH][MERGE_TILE], sl[NH][MERGE_TILE], red[NH][32];
    const int stride = hd + 2, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const float* part = a.scratch + (size_t)(b * a.nh + h0) * a.n_splits * stride;
    const size_t head = (size_t)a.n_splits * stride;
    float m[NH];
#pragma unroll
    for (int k = 0; k < NH; ++k) {
        m[k] = -FLT_MAX; l[k] = 0.f;
#pragma unroll
        for (int j = 0; j < PER; ++j) acc[k][j] = 0.f;
    }
    // the first tile's pairs stay in shared memory; the maximum runs over all of them
    for (int s = threadIdx.x; s < used - first; s += blockDim.x)
#pragma unroll
        for (int k = 0; k < NH; ++k) {
            const float* p = part + k * head + (size_t)(first + s) * stride + hd;
            const float ms = p[0], ls = p[1];
            if (ls > 0.f) m[k] = fmaxf(m[k], ms);
            if (s < MERGE_TILE) { sm[k][s] = ms; sl[k][s] = ls; }
        }
#pragma unroll
    for (int k = 0; k < NH; ++k) {
        m[k] = warp_max(m[k]);
        if (lane == 0) red[k][warp] = m[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NH; ++k) {
        for (int w = 0; w < nwarp; ++w) m[k] = fmaxf(m[k], red[k][w]);
        if (a.sink) m[k] = fmaxf(m[k], a.sink[h0 + k]);
    }
    for (int s0 = 0; s0 < used - first; s0 += MERGE_TILE) {
        const int n = min(MERGE_TILE, used - first - s0);
        if (s0 > 0) __syncthreads();
        for (int s = threadIdx.x; s < n; s += blockDim.x)
#pragma unroll
            for (int k = 0; k < NH; ++k) {
                const float* p = part + k * head + (size_t)(first + s0 + s) * stride + hd;
                const float ms = s0 > 0 ? p[0] : sm[k][s], ls = s0 > 0 ? p[1] : sl[k][s];      // (a thread reads back what it wrote itself)
                const float w = ls > 0.f ? expf(ms - m[k]) : 0.f;
                sm[k][s] = w; sl[k][s] = w * ls;
            }
        __syncthreads();
        const float* p = part + (size_t)(first + s0) * stride + d0 + threadIdx.x;
#pragma unroll 8
        for (int s = 0; s < n; ++s)
#pragma unroll
            for (int k = 0; k < NH; ++k) {
                const float w = sm[k][s];
                l[k] += sl[k][s];
#pragma unroll
                for (int j = 0; j < PER; ++j)
                    if (d0 + (int)threadIdx.x + (int)blockDim.x * j < hd) acc[k][j] = fmaf(w, p[k * head + (size_t)s * stride + blockDim.x * j], acc[k][j]);
            }
    }
    if (a.sink)                                        // the sink counts once, here, not once a split
#pragma unroll
        for (int k = 0; k < NH; ++k) l[k] += expf(a.sink[h0 + k] - m[k]);
}

// grid (B, nh, ceil(value width / 128)), 128 threads: out = sum_s exp(m_s - m) acc_s / sum_s exp(m_s - m) l_s.
template <typename T>
__global__ void __launch_bounds__(128) attn_merge_kernel(AttnArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    const int b = blockIdx.x, h = blockIdx.y, hd = value_width(a), d = blockIdx.z * 128 + threadIdx.x;
    const int len = a.batch.kv_len[b], keys = tb_split_keys(len, a.chunk, a.n_splits);
    const int used = min(a.n_splits, (len + keys - 1) / keys);
    const int first = (a.window > 0 && a.keep_first <= 0) ? max(0, len - a.window) / keys : 0;      // splits before the window's first key hold nothing
    float acc[1][1], l[1];
    merge_splits<1, 1>(a, b, h, hd, blockIdx.z * 128, used, first, acc, l);
    float inv = 1.0f / l[0];
    if (a.head_gate) inv *= 1.0f / (1.0f + expf(-a.head_gate[(size_t)b * a.head_gate_stride + h]));      // the head's gate
    if (d < hd) stf((T*)a.out + (size_t)b * a.out_stride + h * hd + d, acc[0][0] * inv);
}

// grid (B, nh / 2), 128 threads: both maps of a pair merged, the second times lambda taken off the first, the difference
// divided by its root mean square (AttnArgs.pair_lambda).
template <typename T, int PER>
__global__ void __launch_bounds__(128) attn_merge_pair_kernel(AttnArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[33];
    const int b = blockIdx.x, p = blockIdx.y, hd = value_width(a);
    const int len = a.batch.kv_len[b], keys = tb_split_keys(len, a.chunk, a.n_splits);
    const int used = min(a.n_splits, (len + keys - 1) / keys);
    const int first = (a.window > 0 && a.keep_first <= 0) ? max(0, len - a.window) / keys : 0;
    float acc[2][PER], l[2];
    merge_splits<2, PER>(a, b, 2 * p, hd, 0, used, first, acc, l);
    const float lam = *a.pair_lambda, inv1 = 1.0f / l[0], inv2 = 1.0f / l[1];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int d = threadIdx.x + 128 * j;
        acc[0][j] = d < a.pair_width ? fmaf(-lam, acc[1][j] * inv2, acc[0][j] * inv1) : 0.f;
        ss = fmaf(acc[0][j], acc[0][j], ss);
    }
    const float r = a.pair_scale / sqrtf(block_sum(ss, red) / (float)a.pair_width + a.pair_eps);
    T* o = (T*)a.out + (size_t)b * a.out_stride + p * a.pair_width;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int d = threadIdx.x + 128 * j;
        if (d < a.pair_width) stf(o + d, acc[0][j] * r);
    }
}

static int check_common(const AttnArgs& a, const char* who) {
    TB_REQUIRE(a.nh > 0 && a.nkv > 0 && a.nh % a.nkv == 0, "%s: %d query heads are not a multiple of %d kv heads", who, a.nh, a.nkv);
    TB_REQUIRE(a.hd >= 8 && a.hd % 8 == 0 && a.hd <= 32 * ATT_MAXE_WIDE, "%s: head_dim %d must be a multiple of 8 up to %d", who, a.hd, 32 * ATT_MAXE_WIDE);
    TB_REQUIRE(a.hd_v >= 0 && a.hd_v <= 32 * ATT_MAXE_WIDE, "%s: a value row of %d elements (at most %d)", who, a.hd_v, 32 * ATT_MAXE_WIDE);
    TB_REQUIRE(!a.v_alias || value_width(a) <= a.hd, "%s: a value that is the head of its key row cannot be wider (%d) than the key (%d)", who, value_width(a), a.hd);
    TB_REQUIRE(a.q_stride % 8 == 0 && a.kv_stride % 8 == 0, "%s: row strides must be multiples of 8 elements", who);
    TB_REQUIRE(a.window >= 0 && a.keep_first >= 0, "%s: negative window or kept tokens", who);
    TB_REQUIRE(!(a.softcap > 0.f) && !a.rel_bias && !a.head_mix, "%s: capped, biased or mixed scores run on the mixed-heads kernels", who);
    TB_REQUIRE(!a.out_f32, "%s: float32 output rows are the tensor-core prompt kernels'", who);
    TB_REQUIRE(!a.pair_lambda || (a.nh % 2 == 0 && a.pair_width > 0 && a.pair_width <= value_width(a) && a.pair_eps > 0.f && !a.head_gate && !a.sink),
               "%s: pairs of heads need an even number of them (%d), a width (%d) within the value's and no gate or sink a head", who, a.nh, a.pair_width);
    TB_REQUIRE(!a.pair_lambda || value_width(a) <= a.hd, "%s: a pair's value row (%d) may not be wider than its key row (%d)", who, value_width(a), a.hd);
    TB_REQUIRE(!a.cache.storage || (a.cache.head_dim == a.hd && a.cache.kv_heads == a.nkv), "%s: the cache view does not match the heads", who);
    return 0;
}

// Rows of up to 256 elements take 8 values a lane, wider ones 32.
static bool wide_rows(const AttnArgs& a) { return a.hd > 32 * ATT_MAXE || value_width(a) > 32 * ATT_MAXE; }

#define ATT_DISPATCH(kernel, grid, threads, smem)                                                              \
    do {                                                                                                       \
        if (dtype == TB_F32) {                                                                                 \
            if (wide) tb_launch(kernel<float, ATT_MAXE_WIDE>, grid, threads, smem, stream, a);                 \
            else tb_launch(kernel<float, ATT_MAXE>, grid, threads, smem, stream, a);                           \
        } else {                                                                                               \
            if (wide) tb_launch(kernel<__nv_bfloat16, ATT_MAXE_WIDE>, grid, threads, smem, stream, a);         \
            else tb_launch(kernel<__nv_bfloat16, ATT_MAXE>, grid, threads, smem, stream, a);                   \
        }                                                                                                      \
    } while (0)

extern "C" int tb_attn_prefill(const AttnArgs* args, int dtype, cudaStream_t stream) {
    AttnArgs a = *args;
    if (check_common(a, "attn_prefill")) return 1;
    TB_REQUIRE(dtype == TB_F32 || dtype == TB_BF16, "attn_prefill: unknown dtype %d", dtype);
    TB_REQUIRE(a.batch.T > 0, "attn_prefill: no tokens");
    TB_REQUIRE(a.kv_new || a.cache.storage, "attn_prefill: neither new keys nor a cache");
    TB_REQUIRE(!a.head_gate, "attn_prefill: a gate on the heads is applied by the merge of decode splits or by the mixed-heads kernels");
    // The tiles take plain float32 heads: keys and values of one width of up to 128 that lie in separate planes, no kept first tokens
    // and no pairs of heads, rows that 16-byte loads and stores can take.
    if (dtype == TB_F32 && a.hd <= 128 && value_width(a) == a.hd && !a.v_alias && a.keep_first <= 0 && !a.pair_lambda && a.out_stride % 4 == 0 &&
        (uintptr_t)a.q % 16 == 0 && (uintptr_t)a.kv_new % 16 == 0 && (uintptr_t)a.out % 16 == 0 && (uintptr_t)a.cache.storage % 16 == 0 && a.nh <= 65535) {
        if (a.batch.max_new > 0 && a.batch.max_new < TILE_FROM) launch_rows(a, stream);
        else if (a.hd <= 64 ? launch_tile<64>(a, stream) : launch_tile<128>(a, stream)) return 1;
        TB_CHECK_LAUNCH("attn_prefill");
        return 0;
    }
    dim3 grid(a.batch.T, (a.nh + ATT_WARPS - 1) / ATT_WARPS);
    const size_t smem = (size_t)ATT_WARPS * a.hd * sizeof(float);
    const bool wide = wide_rows(a);
    ATT_DISPATCH(attn_prefill_kernel, grid, ATT_WARPS * 32, smem);
    TB_CHECK_LAUNCH("attn_prefill");
    return 0;
}

extern "C" int tb_attn_merge(const AttnArgs* args, int dtype, cudaStream_t stream) {
    AttnArgs a = *args;
    TB_REQUIRE(dtype == TB_F32 || dtype == TB_BF16, "attn_merge: unknown dtype %d", dtype);
    const int width = value_width(a);
    if (a.pair_lambda) {
        TB_REQUIRE(a.nh % 2 == 0 && a.pair_width > 0 && a.pair_width <= width && !a.head_gate && !a.sink, "attn_merge: pairs of heads do not fit");
        const dim3 grid(a.batch.B, a.nh / 2);
        if (dtype == TB_F32) {
            if (width <= 128) tb_launch(attn_merge_pair_kernel<float, 1>, grid, 128, 0, stream, a);
            else if (width <= 256) tb_launch(attn_merge_pair_kernel<float, 2>, grid, 128, 0, stream, a);
            else tb_launch(attn_merge_pair_kernel<float, 8>, grid, 128, 0, stream, a);
        } else {
            if (width <= 128) tb_launch(attn_merge_pair_kernel<__nv_bfloat16, 1>, grid, 128, 0, stream, a);
            else if (width <= 256) tb_launch(attn_merge_pair_kernel<__nv_bfloat16, 2>, grid, 128, 0, stream, a);
            else tb_launch(attn_merge_pair_kernel<__nv_bfloat16, 8>, grid, 128, 0, stream, a);
        }
    } else {
        const dim3 grid(a.batch.B, a.nh, (width + 127) / 128);
        if (dtype == TB_F32) tb_launch(attn_merge_kernel<float>, grid, 128, 0, stream, a);
        else tb_launch(attn_merge_kernel<__nv_bfloat16>, grid, 128, 0, stream, a);
    }
    TB_CHECK_LAUNCH("attn_merge");
    return 0;
}

extern "C" int tb_attn_decode(const AttnArgs* args, int dtype, cudaStream_t stream) {
    AttnArgs a = *args;
    if (check_common(a, "attn_decode")) return 1;
    TB_REQUIRE(dtype == TB_F32 || dtype == TB_BF16, "attn_decode: unknown dtype %d", dtype);
    TB_REQUIRE(a.batch.B > 0 && a.cache.storage && a.scratch, "attn_decode: needs sequences, a cache and scratch");
    TB_REQUIRE(a.chunk > 0 && a.n_splits > 0 && a.n_splits <= 65535, "attn_decode: bad split (chunk=%d splits=%d)", a.chunk, a.n_splits);
    TB_REQUIRE(a.nkv <= 65535 && a.head_blocks <= 65535, "attn_decode: too many kv heads");
    TB_REQUIRE(a.head_blocks == 0 || (a.head_blocks > 0 && a.nh % a.head_blocks == 0 && a.head_blocks % a.nkv == 0),
               "attn_decode: %d blocks for %d query heads on %d kv heads", a.head_blocks, a.nh, a.nkv);
    dim3 grid(a.batch.B, a.head_blocks > 0 ? a.head_blocks : a.nkv, a.n_splits);
    const int width = a.hd > value_width(a) ? a.hd : value_width(a), units = (width * (dtype == TB_F32 ? 4 : 2) + 15) / 16;
    if (units <= 32 && a.hd % 8 == 0 && value_width(a) % (dtype == TB_F32 ? 4 : 8) == 0 && (uintptr_t)a.cache.storage % 16 == 0) {
        // lanes a key: as few as hold its row; warps a head: see the kernel (a rule of the launch's numbers, not of the lengths)
        const int lanes = units <= 4 ? 4 : (units <= 8 ? 8 : (units <= 16 ? 16 : 32)), group = a.nh / (int)grid.y;
        const int turns = (group + VEC_WARPS - 1) / VEC_WARPS, heads = (group + turns - 1) / turns;      // equal turns
        int share = 1;
        while (share * 2 * heads <= VEC_WARPS && share * 2 * (32 / lanes) * VEC_KEYS <= a.chunk) share *= 2;
        const int warps = share * heads;
#define ATT_VEC(TT, L) tb_launch(attn_decode_vec_kernel<TT, L>, grid, warps * 32, (size_t)warps * (value_width(a) + 2) * sizeof(float), stream, a, share)
#define ATT_VEC_ANY(TT) do { if (lanes == 4) ATT_VEC(TT, 4); else if (lanes == 8) ATT_VEC(TT, 8); else if (lanes == 16) ATT_VEC(TT, 16); else ATT_VEC(TT, 32); } while (0)
        if (dtype == TB_F32) ATT_VEC_ANY(float); else ATT_VEC_ANY(__nv_bfloat16);
#undef ATT_VEC_ANY
#undef ATT_VEC
    } else {
        const size_t smem = (size_t)ATT_WARPS * a.hd * sizeof(float);
        const bool wide = wide_rows(a);
        ATT_DISPATCH(attn_decode_kernel, grid, ATT_WARPS * 32, smem);
    }
    TB_CHECK_LAUNCH("attn_decode");
    return tb_attn_merge(args, dtype, stream);
}
