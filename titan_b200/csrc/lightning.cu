// Linear attention with a per-head decay ("lightning" mixer): the recurrence and the gated norm after it.
//
//   S_t = decay_h S_{t-1} + k_t v_t^T        S: [dk][dv] float32 per (sequence, head), kept in the cache's state group
//   o_t = S_t^T q_t
// with q = silu(.), k = silu(.), v = silu(.) of the projection's columns (the projection may be in the compute
// dtype; the activation, the state and the sums are float32).  A sequence's tokens are taken in order, so a prompt
// run whole, in pieces or token by token leaves the same state up to the order of float32 sums: runs of few tokens are added one
// after the other, longer ones in chunks of 64 that begin where the step's run begins, so that a cut changes the last bits (what a
// sequence gives does not depend on the other sequences of the step).
//
// tb_lightning_scan   grid (sequences, heads, ceil(dv / 32)): a block owns 32 value columns of one head's state;
//                     four neighbouring lanes share a column (each keeps a quarter of its rows in registers) and
//                     add their parts of o with two shuffles.  Tokens are staged in shared memory sixteen at a time,
//                     the next sixteen requested while these are worked through.  Runs of CHUNKED_FROM tokens and
//                     more go in chunks as small matrix products instead (lightning_parts_kernel and the two behind it).
// tb_gated_rmsnorm    y = o / sqrt(mean(o^2) + eps) * w * sigmoid(g) over the concatenated heads, one block a token.
// tb_rotary_rows      rotates heads that lie side by side in float32 rows, in place, and scales some of them: what the
//                     retention mixer does to q and k between its projection and this recurrence (LightningArgs.plain).
#include <atomic>

#include "common.cuh"
#include "qk_args.h"

struct LightningArgs {
    const void* proj; int stride;           // [T][stride]: q (H*dk) | k (H*dk) | v (H*dv) | g (H*dv), compute dtype
    float* out; int out_stride;             // [T][out_stride] float32: head h at h * dv
    float* state;                           // [slots][H][dk][dv] float32
    const float* decay;                     // [H]
    const int* q_start; const int* slot_of_seq;
    int B; int H; int dk; int dv;
    int max_new;                            // most tokens a sequence brings in this step (1: a step of single tokens)
    int plain;                              // 1: q, k and v enter the recurrence as they stand in the rows (no silu): the retention mixer, whose rows are float32
    float* work; int work_chunks;           // room for the chunked form; work_chunks >= the chunks of all its runs (tb_lightning_work); null: token by token
    int work_room;                          // chunks that ``work`` holds at a time: more go one segment after the other
    int below;                              // > 0: only runs of fewer tokens (set by the launcher)
    int segment;                            // first chunk of the segment at work (set by the launcher)
};

namespace {

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }

// CH tokens of a sequence are staged in shared memory at a time (q and k of the head with the activation applied, and the
// block's 32 value columns), requested into registers while the chunk before is worked through, so that the latency of
// the loads is paid once a chunk and not once a token.  Within a chunk the tokens are taken one after the other from
// shared memory: a thread keeps rows [s * R, (s + 1) * R) of its column of the state in registers (s = lane & 3), reads
// the matching q and k as 16-byte loads (rows of the four s are 16 bytes apart in the banks), and the four partial sums
// of o meet by two shuffles.
template <typename T, int R, int CH>
__global__ void __launch_bounds__(128) lightning_scan_kernel(LightningArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    constexpr int DKP = 4 * (R + 4);                    // a q or k row in shared memory: four runs of R, each padded by 4
    constexpr int ROW = 2 * DKP + 32;                   // q | k | 32 values
    constexpr int PER = (CH * ROW + 127) / 128;         // staged elements a thread
    const int b = blockIdx.x, h = blockIdx.y;
    const int tid = threadIdx.x, s = tid & 3, col = tid >> 2, j = blockIdx.z * 32 + col;
    const int dk = a.dk, dv = a.dv;
    const int t0 = a.q_start[b], t1 = a.q_start[b + 1];
    if (a.below > 0 && t1 - t0 >= a.below) return;
    const bool live = j < dv;
    float* S_g = a.state + (((size_t)a.slot_of_seq[b] * a.H + h) * dk) * dv + j;
    float S[R];
#pragma unroll
    for (int ii = 0; ii < R; ++ii) {
        const int i = s * R + ii;
        S[ii] = (live && i < dk) ? S_g[(size_t)i * dv] : 0.f;
    }
    const float decay = a.decay[h];
    const T* base = (const T*)a.proj;
    const int kq = h * dk, kk = a.H * dk + h * dk, kvv = 2 * a.H * dk + h * dv + blockIdx.z * 32;
    float stage[PER];
    // Element e of a chunk's staging area: token e / ROW, and within the row q (padded), k (padded) or a value.  Gives
    // the address to read (always a valid one: indices are clamped, so that the load needs no condition and nothing
    // waits for it before the chunk is due) and whether the element is real or padding.
    auto source = [&](int u, int first, bool* real) -> const T* {
        const int e = tid + 128 * u, ec = min(e, CH * ROW - 1), tok = ec / ROW, x = ec % ROW;
        bool ok = e < CH * ROW && first + tok < t1;
        const T* row = base + (size_t)min(first + tok, t1 - 1) * a.stride;
        if (x < 2 * DKP) {
            const int y = x < DKP ? x : x - DKP, run = y / (R + 4), within = y % (R + 4), i = run * R + within;
            ok = ok && within < R && i < dk;
            *real = ok;
            return row + (x < DKP ? kq : kk) + (ok ? i : 0);
        }
        const int c = x - 2 * DKP;
        ok = ok && blockIdx.z * 32 + c < dv;
        *real = ok;
        return row + kvv + (ok ? c : 0);
    };
    auto request = [&](int first) {
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            bool real;
            stage[u] = ldf(source(u, first, &real));
        }
    };
    if (t0 < t1) request(t0);
    for (int c0 = t0; c0 < t1; c0 += CH) {
        __syncthreads();                                // the chunk before has been read from shared memory
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int e = tid + 128 * u;
            bool real;
            source(u, c0, &real);
            if (e < CH * ROW) sm[e] = real ? (a.plain ? stage[u] : silu_f(stage[u])) : 0.f;
        }
        __syncthreads();
        if (c0 + CH < t1) request(c0 + CH);
        const int n = min(CH, t1 - c0);
        for (int tt = 0; tt < n; ++tt) {
            const float* qs = sm + tt * ROW + s * (R + 4);
            const float* ks = qs + DKP;
            const float vj = sm[tt * ROW + 2 * DKP + col];
            float acc = 0.f;
#pragma unroll
            for (int ii = 0; ii < R; ii += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(ks + ii), q4 = *reinterpret_cast<const float4*>(qs + ii);
                S[ii] = fmaf(decay, S[ii], k4.x * vj);         acc = fmaf(S[ii], q4.x, acc);
                S[ii + 1] = fmaf(decay, S[ii + 1], k4.y * vj); acc = fmaf(S[ii + 1], q4.y, acc);
                S[ii + 2] = fmaf(decay, S[ii + 2], k4.z * vj); acc = fmaf(S[ii + 2], q4.z, acc);
                S[ii + 3] = fmaf(decay, S[ii + 3], k4.w * vj); acc = fmaf(S[ii + 3], q4.w, acc);
            }
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            if (s == 0 && live) a.out[(size_t)(c0 + tt) * a.out_stride + h * dv + j] = acc;
        }
    }
    if (live) {
#pragma unroll
        for (int ii = 0; ii < R; ++ii) {
            const int i = s * R + ii;
            if (i < dk) S_g[(size_t)i * dv] = S[ii];
        }
    }
}

// Eight consecutive elements of a row, as they come from one (bfloat16) or two (float32) 16-byte loads.
template <typename T> struct Pack8;
template <> struct Pack8<__nv_bfloat16> {
    uint4 a;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { a = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ void get(float* o) const {
        const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { o[2 * i] = __uint_as_float(w[i] << 16); o[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
    }
};
template <> struct Pack8<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float* p) { a = *reinterpret_cast<const float4*>(p); b = *reinterpret_cast<const float4*>(p + 4); }
    __device__ __forceinline__ void get(float* o) const { o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w; }
};

// The same recurrence for sizes in multiples of 8 (dk, dv, the projection's row stride): a block owns 16 value columns,
// eight neighbouring lanes share a column (R rows of it each, dk <= 8 R), and a chunk of tokens is staged by 16-byte
// loads of eight elements, a few a thread.  Twice the blocks of the kernel above, half the arithmetic a thread and
// token, and an eighth of the load instructions.
template <typename T, int R, int CH>
__global__ void __launch_bounds__(128) lightning_scan_vec_kernel(LightningArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    constexpr int DKP = 8 * (R + 4);                    // a q or k row in shared memory: eight runs of R, each padded by 4
    constexpr int ROW = 2 * DKP + 16;                   // q | k | 16 values
    const int b = blockIdx.x, h = blockIdx.y;
    const int tid = threadIdx.x, s = tid & 7, col = tid >> 3, j = blockIdx.z * 16 + col;
    const int dk = a.dk, dv = a.dv;
    const int t0 = a.q_start[b], t1 = a.q_start[b + 1];
    if (a.below > 0 && t1 - t0 >= a.below) return;
    const bool live = j < dv;
    float* S_g = a.state + (((size_t)a.slot_of_seq[b] * a.H + h) * dk) * dv + j;
    float S[R];
#pragma unroll
    for (int ii = 0; ii < R; ++ii) {
        const int i = s * R + ii;
        S[ii] = (live && i < dk) ? S_g[(size_t)i * dv] : 0.f;
    }
    const float decay = a.decay[h];
    const T* base = (const T*)a.proj;
    const int kq = h * dk, kk = a.H * dk + h * dk, kvv = 2 * a.H * dk + h * dv + blockIdx.z * 16;
    const int qk_units = dk >> 3, units = 2 * qk_units + 2, total = CH * units;       // units of eight elements a token, a chunk
    constexpr int PERU = (CH * (2 * R + 2) + 127) / 128;                              // at most 8 R / 8 = R units of q and of k a token
    Pack8<T> stage[PERU];
    // unit n of a chunk: token n / units; then q (qk_units of them), k, and two units of values.  Gives a valid address
    // (clamped, so the load carries no condition), where the eight floats go in shared memory, and whether they are real.
    auto source = [&](int u, int first, bool* real, int* to) -> const T* {
        const int n = tid + 128 * u, nc = min(n, total - 1), tok = nc / units, x = nc % units;
        bool ok = n < total && first + tok < t1;
        const T* row = base + (size_t)min(first + tok, t1 - 1) * a.stride;
        if (x < 2 * qk_units) {
            const int g = x < qk_units ? x : x - qk_units, i = g * 8;
            *to = tok * ROW + (x < qk_units ? 0 : DKP) + (i / R) * (R + 4) + (i % R);
            *real = ok;
            return row + (x < qk_units ? kq : kk) + i;
        }
        const int c = (x - 2 * qk_units) * 8;
        ok = ok && blockIdx.z * 16 + c < dv;
        *to = tok * ROW + 2 * DKP + c;
        *real = ok;
        return row + kvv + (ok ? c : 0);
    };
    auto request = [&](int first) {
#pragma unroll
        for (int u = 0; u < PERU; ++u) {
            bool real; int to;
            stage[u].load(source(u, first, &real, &to));
        }
    };
    // rows of the padded q and k areas beyond dk are never written by a unit: zero them once (they are read as factors)
    for (int e = tid; e < CH * ROW; e += 128) sm[e] = 0.f;
    if (t0 < t1) request(t0);
    for (int c0 = t0; c0 < t1; c0 += CH) {
        __syncthreads();                                // the chunk before has been read from shared memory (or the zeros are in place)
#pragma unroll
        for (int u = 0; u < PERU; ++u) {
            bool real; int to;
            source(u, c0, &real, &to);
            if (tid + 128 * u < total) {
                float v[8];
                stage[u].get(v);
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = real ? (a.plain ? v[i] : silu_f(v[i])) : 0.f;
                *reinterpret_cast<float4*>(sm + to) = make_float4(v[0], v[1], v[2], v[3]);
                *reinterpret_cast<float4*>(sm + to + 4) = make_float4(v[4], v[5], v[6], v[7]);
            }
        }
        __syncthreads();
        if (c0 + CH < t1) request(c0 + CH);
        const int n = min(CH, t1 - c0);
        for (int tt = 0; tt < n; ++tt) {
            const float* qs = sm + tt * ROW + s * (R + 4);
            const float* ks = qs + DKP;
            const float vj = sm[tt * ROW + 2 * DKP + col];
            float acc = 0.f;
#pragma unroll
            for (int ii = 0; ii < R; ii += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(ks + ii), q4 = *reinterpret_cast<const float4*>(qs + ii);
                S[ii] = fmaf(decay, S[ii], k4.x * vj);         acc = fmaf(S[ii], q4.x, acc);
                S[ii + 1] = fmaf(decay, S[ii + 1], k4.y * vj); acc = fmaf(S[ii + 1], q4.y, acc);
                S[ii + 2] = fmaf(decay, S[ii + 2], k4.z * vj); acc = fmaf(S[ii + 2], q4.z, acc);
                S[ii + 3] = fmaf(decay, S[ii + 3], k4.w * vj); acc = fmaf(S[ii + 3], q4.w, acc);
            }
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            acc += __shfl_xor_sync(0xffffffffu, acc, 4);
            if (s == 0 && live) a.out[(size_t)(c0 + tt) * a.out_stride + h * dv + j] = acc;
        }
    }
    if (live) {
#pragma unroll
        for (int ii = 0; ii < R; ++ii) {
            const int i = s * R + ii;
            if (i < dk) S_g[(size_t)i * dv] = S[ii];
        }
    }
}

// ---------------------------------------------------------------- prompts: chunks of 64 tokens
// Token by token the recurrence is a chain of 2,000 dependent steps of half a microsecond each and more (measured: 965 us for 2,000 bfloat16 tokens, 1,531 within a
// step, 16 heads of 128 x 128).  With S the state before a chunk, r a token's place in it and n its length,
//     o_r = decay^(r+1) q_r . S + sum over j <= r of decay^(r-j) (q_r . k_j) v_j,     S' = decay^n S + sum_j decay^(n-1-j) k_j v_j^T
// so that all that waits for the chunk before is one multiply-add an element of the state.  Three kernels:
//   lightning_parts_kernel    all chunks at once: M = sum_j decay^(n-1-j) k_j v_j^T, a block for 64 value columns, and, by one block more,
//                             A = [decay^(r-j) (q_r . k_j), zero above r]; both go to the room.
//   lightning_states_kernel   a thread four elements of a head's state, chunk after chunk: takes M, leaves the state before the chunk in its place.
//   lightning_outputs_kernel  all chunks at once: [A | decay^(r+1) q] . [v; S], a block for 64 value columns.
// Everything stays float32, fused multiply-adds only (two at a time, fma.rn.f32x2, each rounded as fmaf rounds); powers of the
// decay are formed in 64 bits.  Bound by the FMA pipes (3.4 GFLOP for 2,000 tokens of 16 heads of 128 x 128: 47 us) and by what a block waits for
// its operands; a chain of chunks that made outputs and states in turn, a block for 16 value columns, took 174 us there.
// Chunks are numbered through all long runs of the step; a segment of them is worked off before the next, so that their rows need
// a bounded room however long the prompt is: the state passes from segment to segment through the cache, the bits are the same.
constexpr int CHUNK = 64, VCOLS = 64;
// Tokens of a run from which it goes in chunks: where one sequence is the faster so (token by token / in chunks, us: 16 heads of 128 x 128, 32
// tokens 18 / 30, 40 23 / 30, 64 33 / 29, 100 53 / 31; 32 heads of 64 x 128, 40 tokens 17 / 20, 64 24 / 22, 100 38 / 29; with the chain of chunks).  Many short
// runs together are no reason for another border: what a run gives may not depend on the runs beside it.
constexpr int CHUNKED_FROM = 64;

__device__ __forceinline__ void lf_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long lf_twice(float v) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float lf_low(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float lf_high(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }

// Room of a (chunk, head): A [64][64], then M, later the state before the chunk, [dk][dv] as in the cache.
__host__ __device__ __forceinline__ size_t room_floats(int dk, int dv) { return (size_t)CHUNK * CHUNK + (((size_t)dk * dv + 3) & ~(size_t)3); }

// The chunk that the ``at``-th of the segment is: its first token and number of tokens; false behind the last.
__device__ __forceinline__ bool chunk_of(const LightningArgs& a, int at, int& t0, int& n) {
    int chunk = a.segment + at;
    const int b = tb_find_run(a.q_start, a.B, chunk, [](int m) { return m >= CHUNKED_FROM ? (m + CHUNK - 1) / CHUNK : 0; });
    if (b < 0) return false;
    t0 = a.q_start[b] + chunk * CHUNK;
    n = min(CHUNK, a.q_start[b + 1] - t0);
    return true;
}

// Columns [col, col + WIDTH) of CHUNK rows of the projection into shared memory (row stride LD), activated unless ``plain``, row r times power[first + step * r]
// (null: as they are); rows from n on and columns from ``cols`` on are zero.  256 threads.  Returns whether this thread met a value that is not finite.
template <typename T, int WIDTH, int LD>
__device__ __forceinline__ bool load_rows(float* to, const LightningArgs& a, int t0, int n, int col, int cols, const float* power, int first, int step) {
    const T* base = (const T*)a.proj + (size_t)t0 * a.stride + col;
    bool odd = false;
    auto value = [&](float z, int r, bool real) {
        const float y = real ? (a.plain ? z : silu_f(z)) : 0.f;
        odd = odd || !(fabsf(y) <= 3.402823466e38f);
        return power && real ? y * power[first + step * r] : y;
    };
    if (cols >= 8 && cols % 8 == 0 && a.stride % 8 == 0 && col % 8 == 0 && (uintptr_t)a.proj % 16 == 0) {
        constexpr int UNITS = CHUNK * WIDTH / 8 / 256;      // units of eight elements a thread, all requested at once
        Pack8<T> u8[UNITS];
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int e = (threadIdx.x + 256 * u) * 8;
            u8[u].load(base + (size_t)min(e / WIDTH, n - 1) * a.stride + min(e % WIDTH, cols - 8));
        }
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int e = (threadIdx.x + 256 * u) * 8, r = e / WIDTH, d = e % WIDTH;
            float f[8];
            u8[u].get(f);
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = value(f[i], r, r < n && d < cols);
            float4* out = reinterpret_cast<float4*>(to + r * LD + d);
            out[0] = make_float4(f[0], f[1], f[2], f[3]); out[1] = make_float4(f[4], f[5], f[6], f[7]);
        }
    } else {
        for (int e = threadIdx.x; e < CHUNK * WIDTH; e += 256) {
            const int r = e / WIDTH, d = e % WIDTH;
            const bool real = r < n && d < cols;
            to[r * LD + d] = value(real ? ldf(base + (size_t)r * a.stride + d) : 0.f, r, real);
        }
    }
    return odd;
}

__device__ __forceinline__ void put_four(float* to, const float* v, int left, bool wide) {      // up to ``left`` of four neighbours
    if (wide) { if (left > 0) *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]); return; }
#pragma unroll
    for (int i = 0; i < 4; ++i) if (i < left) to[i] = v[i];
}

template <int DK> constexpr size_t parts_smem() { return (size_t)(2 * CHUNK * (DK + 4) + CHUNK + 1) * sizeof(float); }
template <int DK> constexpr size_t outputs_smem() { return (size_t)(CHUNK * (CHUNK + DK + 4) + (CHUNK + DK) * (VCOLS + 4) + CHUNK + 1) * sizeof(float); }

// grid (chunks of a segment, H, blocks of value columns + 1), 256 threads
template <typename T, int DK>
__global__ void __launch_bounds__(256) lightning_parts_kernel(LightningArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    constexpr int LD = DK + 4;
    float* ks = sm;                                     // [64][LD]
    float* other = ks + CHUNK * LD;                     // [64][LD]: the queries, or [64][VCOLS + 4]: the values
    float* power = other + CHUNK * LD;                  // decay^0 .. decay^64
    const int tid = threadIdx.x, h = blockIdx.y, dk = a.dk, dv = a.dv, tx = tid & 15, ty = tid >> 4;
    int t0, n;
    if (!chunk_of(a, blockIdx.x, t0, n)) return;
    if (tid <= CHUNK) power[tid] = (float)pow((double)a.decay[h], (double)tid);
    __syncthreads();
    float* room = a.work + ((size_t)blockIdx.x * a.H + h) * room_floats(dk, dv);
    if ((int)blockIdx.z * VCOLS >= dv) {                // A
        load_rows<T, DK, LD>(other, a, t0, n, h * dk, dk, nullptr, 0, 0);
        load_rows<T, DK, LD>(ks, a, t0, n, (a.H + h) * dk, dk, nullptr, 0, 0);
        __syncthreads();
        unsigned long long acc[4][4] = {};              // rows ty + 16 i, keys tx + 16 j; sums over even and over odd dimensions
#pragma unroll 4
        for (int d = 0; d < DK; d += 4) {
            ulonglong2 q[4], k[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                q[i] = *reinterpret_cast<const ulonglong2*>(other + (ty + 16 * i) * LD + d);
                k[i] = *reinterpret_cast<const ulonglong2*>(ks + (tx + 16 * i) * LD + d);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j) { lf_fma2(acc[i][j], q[i].x, k[j].x); lf_fma2(acc[i][j], q[i].y, k[j].y); }      // (j > i: keys after every query)
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int r = ty + 16 * i, c = tx + 16 * j;
                room[r * CHUNK + c] = c <= r && r < n ? (lf_low(acc[i][j]) + lf_high(acc[i][j])) * power[r - c] : 0.f;
            }
        return;
    }
    constexpr int RD = DK / 16, LV = VCOLS + 4;         // M: dimensions RD ty .., columns 4 tx ..
    const int j0 = blockIdx.z * VCOLS;
    load_rows<T, DK, LD>(ks, a, t0, n, (a.H + h) * dk, dk, power, n - 1, -1);
    load_rows<T, VCOLS, LV>(other, a, t0, n, 2 * a.H * dk + h * dv + j0, min(VCOLS, dv - j0), nullptr, 0, 0);
    __syncthreads();
    unsigned long long acc[RD][2] = {};
#pragma unroll 4
    for (int t = 0; t < CHUNK; ++t) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(other + t * LV + 4 * tx);
        float k[RD];
#pragma unroll
        for (int i = 0; i < RD; i += 4) {
            const float4 f = *reinterpret_cast<const float4*>(ks + t * LD + RD * ty + i);
            k[i] = f.x; k[i + 1] = f.y; k[i + 2] = f.z; k[i + 3] = f.w;
        }
#pragma unroll
        for (int i = 0; i < RD; ++i) {
            const unsigned long long kk = lf_twice(k[i]);
            lf_fma2(acc[i][0], kk, v.x); lf_fma2(acc[i][1], kk, v.y);
        }
    }
    float* M = room + CHUNK * CHUNK;
#pragma unroll
    for (int i = 0; i < RD; ++i) {
        const float v[4] = {lf_low(acc[i][0]), lf_high(acc[i][0]), lf_low(acc[i][1]), lf_high(acc[i][1])};
        if (RD * ty + i < dk) put_four(M + (size_t)(RD * ty + i) * dv + j0 + 4 * tx, v, dv - j0 - 4 * tx, dv % 4 == 0);
    }
}

// grid (long runs at most, H, ceil(dk dv / 1024)), 256 threads
__global__ void __launch_bounds__(256) lightning_states_kernel(LightningArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    const int h = blockIdx.y, lane = threadIdx.x & 31, size = a.dk * a.dv, e0 = ((int)blockIdx.z * 256 + (int)threadIdx.x) * 4;
    int which = blockIdx.x;
    const int b = tb_find_run(a.q_start, a.B, which, [](int m) { return m >= CHUNKED_FROM ? 1 : 0; });
    if (b < 0) return;
    int chunk0 = 0;                                     // the run's first chunk
    for (int i = lane; i < b; i += 32) {
        const int m = a.q_start[i + 1] - a.q_start[i];
        if (m >= CHUNKED_FROM) chunk0 += (m + CHUNK - 1) / CHUNK;
    }
    chunk0 = __reduce_add_sync(0xffffffffu, chunk0);
    const int tokens = a.q_start[b + 1] - a.q_start[b];
    // the run's chunks in this segment
    const int begin = max(0, a.segment - chunk0), end = min((tokens + CHUNK - 1) / CHUNK, a.segment + a.work_room - chunk0);
    if (begin >= end || e0 >= size) return;
    const double decay = (double)a.decay[h];
    const float whole = (float)pow(decay, (double)CHUNK), last = (float)pow(decay, (double)min(CHUNK, tokens - (end - 1) * CHUNK));
    const bool wide = size % 4 == 0;                    // states and rooms then start on 16-byte borders
    float* S_g = a.state + ((size_t)a.slot_of_seq[b] * a.H + h) * size + e0;
    const size_t step = (size_t)a.H * room_floats(a.dk, a.dv);
    float* M = a.work + (size_t)(chunk0 + begin - a.segment) * step + (size_t)h * room_floats(a.dk, a.dv) + CHUNK * CHUNK + e0;
    auto get = [&](const float* p, float* v) {
        if (wide) {
            const float4 f = *reinterpret_cast<const float4*>(p);
            v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = e0 + i < size ? p[i] : 0.f;
        }
    };
    float S[4];
    get(S_g, S);
    constexpr int AHEAD = 8;                            // chunks requested at once
    for (int c0 = begin; c0 < end; c0 += AHEAD) {
        float m[AHEAD][4];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) if (c0 + u < end) get(M + (size_t)u * step, m[u]);
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            if (c0 + u >= end) continue;
            put_four(M + (size_t)u * step, S, size - e0, wide);
            const float f = c0 + u == end - 1 ? last : whole;
#pragma unroll
            for (int i = 0; i < 4; ++i) S[i] = fmaf(f, S[i], m[u][i]);
        }
        M += AHEAD * step;
    }
    put_four(S_g, S, size - e0, wide);
}

// grid (chunks of a segment, H, blocks of value columns), 256 threads
template <typename T, int DK>
__global__ void __launch_bounds__(256) lightning_outputs_kernel(LightningArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    constexpr int ROW = CHUNK + DK, LX = ROW + 4, LY = VCOLS + 4;
    float* X = sm;                                      // [64][LX]: A | decay^(r+1) q
    float* Y = X + CHUNK * LX;                          // [ROW][LY]: v, then S
    float* power = Y + ROW * LY;
    const int tid = threadIdx.x, h = blockIdx.y, dk = a.dk, dv = a.dv, j0 = blockIdx.z * VCOLS, tx = tid & 15, ty = tid >> 4;
    int t0, n;
    if (!chunk_of(a, blockIdx.x, t0, n)) return;
    const float* room = a.work + ((size_t)blockIdx.x * a.H + h) * room_floats(dk, dv);
    for (int e = tid; e < CHUNK * CHUNK / 4; e += 256)
        *reinterpret_cast<float4*>(X + e / 16 * LX + e % 16 * 4) = reinterpret_cast<const float4*>(room)[e];
    const float* S = room + CHUNK * CHUNK + j0;
    if (dv % 4 == 0) {
        for (int e = tid; e < DK * VCOLS / 4; e += 256) {
            const int d = e / (VCOLS / 4), c = e % (VCOLS / 4) * 4;
            *reinterpret_cast<float4*>(Y + (CHUNK + d) * LY + c) = d < dk && j0 + c < dv ? *reinterpret_cast<const float4*>(S + (size_t)d * dv + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    } else {
        for (int e = tid; e < DK * VCOLS; e += 256) {
            const int d = e / VCOLS, c = e % VCOLS;
            Y[(CHUNK + d) * LY + c] = d < dk && j0 + c < dv ? S[(size_t)d * dv + c] : 0.f;
        }
    }
    if (tid <= CHUNK) power[tid] = (float)pow((double)a.decay[h], (double)tid);
    __syncthreads();
    load_rows<T, DK, LX>(X + CHUNK, a, t0, n, h * dk, dk, power, 1, 1);
    // a value that is not finite: its product with a zero weight is no zero
    const bool odd = __syncthreads_or(load_rows<T, VCOLS, LY>(Y, a, t0, n, 2 * a.H * dk + h * dv + j0, min(VCOLS, dv - j0), nullptr, 0, 0));
    unsigned long long acc[4][2] = {};                  // rows ty + 16 i, columns 4 tx ..
    if (odd) {
        for (int j = 0; j < CHUNK; ++j) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(Y + j * LY + 4 * tx);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (j > ty + 16 * i) continue;
                const unsigned long long x = lf_twice(X[(ty + 16 * i) * LX + j]);
                lf_fma2(acc[i][0], x, v.x); lf_fma2(acc[i][1], x, v.y);
            }
        }
    }
#pragma unroll 2
    for (int k = odd ? CHUNK : 0; k < ROW; k += 4) {
        float x[4][4];
        ulonglong2 y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 f = *reinterpret_cast<const float4*>(X + (ty + 16 * i) * LX + k);
            x[i][0] = f.x; x[i][1] = f.y; x[i][2] = f.z; x[i][3] = f.w;
            y[i] = *reinterpret_cast<const ulonglong2*>(Y + (k + i) * LY + 4 * tx);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const unsigned long long xx = lf_twice(x[i][e]);
                lf_fma2(acc[i][0], xx, y[e].x); lf_fma2(acc[i][1], xx, y[e].y);
            }
    }
    const bool wide = dv % 4 == 0 && a.out_stride % 4 == 0 && (uintptr_t)a.out % 16 == 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty + 16 * i;
        const float v[4] = {lf_low(acc[i][0]), lf_high(acc[i][0]), lf_low(acc[i][1]), lf_high(acc[i][1])};
        if (r < n) put_four(a.out + (size_t)(t0 + r) * a.out_stride + h * dv + j0 + 4 * tx, v, dv - j0 - 4 * tx, wide);
    }
}

template <typename T>
int launch_scan(const LightningArgs& a, bool single, cudaStream_t stream);

template <typename T, int DK>
int launch_chunks(const LightningArgs& a, cudaStream_t stream) {
    static std::atomic<bool> configured[64];            // a device each
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 64 || !configured[dev].load()) {
        cudaError_t e = cudaFuncSetAttribute(lightning_parts_kernel<T, DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)parts_smem<DK>());
        if (e == cudaSuccess) e = cudaFuncSetAttribute(lightning_outputs_kernel<T, DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)outputs_smem<DK>());
        TB_REQUIRE(e == cudaSuccess, "lightning_scan: cannot reserve %zu bytes of shared memory: %s", outputs_smem<DK>(), cudaGetErrorString(e));
        if (dev < 64) configured[dev].store(true);
    }
    LightningArgs part = a;
    const int runs = min(a.B, a.work_chunks);           // (a long run has a chunk at least)
    for (part.segment = 0; part.segment < a.work_chunks; part.segment += a.work_room) {
        const int chunks = min(a.work_room, a.work_chunks - part.segment), columns = (a.dv + VCOLS - 1) / VCOLS;
        tb_launch(lightning_parts_kernel<T, DK>, dim3(chunks, a.H, columns + 1), 256, parts_smem<DK>(), stream, part);
        tb_launch(lightning_states_kernel, dim3(runs, a.H, (a.dk * a.dv + 1023) / 1024), 256, 0, stream, part);
        tb_launch(lightning_outputs_kernel<T, DK>, dim3(chunks, a.H, columns), 256, outputs_smem<DK>(), stream, part);
    }
    if (a.B > 1) {                                      // shorter runs beside them go token by token, as they would alone
        LightningArgs rest = a;
        rest.work = nullptr; rest.below = CHUNKED_FROM;
        return launch_scan<T>(rest, false, stream);
    }
    return 0;
}

template <typename T>
__global__ void gated_rmsnorm_kernel(const float* __restrict__ o, int ldo, const float* __restrict__ w, const T* __restrict__ gate,
                                     int ldg, T* __restrict__ y, int ldy, int N, float eps) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[33];
    const size_t t = blockIdx.x;
    const float* row = o + t * ldo;
    float ss = 0.f;
    for (int i = threadIdx.x; i < N; i += blockDim.x) ss += row[i] * row[i];
    ss = block_sum(ss, red);
    const float scale = 1.0f / sqrtf(ss / (float)N + eps);
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        const float g = ldf(gate + t * ldg + i);
        stf(y + t * ldy + i, row[i] * scale * w[i] * (1.0f / (1.0f + expf(-g))));
    }
}

// The same for rows of whole 16-byte units: a thread keeps up to UNITS runs of eight columns in registers, row and gate requested together
// (the weight before the wait: nothing makes it), so that a row costs one round trip to memory instead of one a column and thread, twice.  Bound by
// its bytes at 2,000 rows of 2,048 (18.6 us above), by latency at eight (8.1 us above).
template <typename T, int UNITS>
__global__ void __launch_bounds__(512) gated_rmsnorm_vec_kernel(const float* o, int ldo, const float* __restrict__ w, const T* gate, int ldg, T* y, int ldy,
                                                                int N, float eps) {
    pdl_launch_dependents();
    __shared__ float red[33];
    const size_t t = blockIdx.x;
    const int n8 = N >> 3;
    float4 ww[UNITS][2], v[UNITS][2];
    Pack8<T> g[UNITS];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < UNITS; ++j) {
        const int i = threadIdx.x + j * blockDim.x;
        const float4* from = reinterpret_cast<const float4*>(w) + 2 * i;
        ww[j][0] = i < n8 ? from[0] : zero; ww[j][1] = i < n8 ? from[1] : zero;
    }
    pdl_wait();
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < UNITS; ++j) {
        const int i = threadIdx.x + j * blockDim.x;
        const float4* from = reinterpret_cast<const float4*>(o + t * ldo) + 2 * i;
        v[j][0] = i < n8 ? from[0] : zero; v[j][1] = i < n8 ? from[1] : zero;
        if (i < n8) g[j].load(gate + t * ldg + 8 * i);
    }
#pragma unroll
    for (int j = 0; j < UNITS; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) ss += v[j][e].x * v[j][e].x + v[j][e].y * v[j][e].y + v[j][e].z * v[j][e].z + v[j][e].w * v[j][e].w;
    ss = block_sum(ss, red);
    const float scale = 1.0f / sqrtf(ss / (float)N + eps);
#pragma unroll
    for (int j = 0; j < UNITS; ++j) {
        const int i = threadIdx.x + j * blockDim.x;
        if (i >= n8) continue;
        const float x[8] = {v[j][0].x, v[j][0].y, v[j][0].z, v[j][0].w, v[j][1].x, v[j][1].y, v[j][1].z, v[j][1].w};
        const float m[8] = {ww[j][0].x, ww[j][0].y, ww[j][0].z, ww[j][0].w, ww[j][1].x, ww[j][1].y, ww[j][1].z, ww[j][1].w};
        float f[8];
        g[j].get(f);
        alignas(16) T r[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) stf(r + e, x[e] * scale * m[e] * (1.0f / (1.0f + expf(-f[e]))));
        uint4* to = reinterpret_cast<uint4*>(y + t * ldy + 8 * i);
#pragma unroll
        for (int e = 0; e < (int)sizeof(T) / 2; ++e) to[e] = reinterpret_cast<const uint4*>(r)[e];
    }
}

// One block a token; a thread takes pairs of one head's rotated dimensions (both members, so the rotation is in place),
// then the elements that pass unrotated.  Heads from ``scale_from`` on are multiplied by ``scale`` after the rotation.
__global__ void __launch_bounds__(128) rotary_rows_kernel(float* x, int stride, const int* __restrict__ pos_of, int heads, int hd,
                                                          TbRotary rope, int scale_from, float scale) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float cs[];           // [half] cosines, [half] sines
    const int t = blockIdx.x, half = rope.rot >> 1;
    float* sn = cs + half;
    const float p = (float)pos_of[t] + rope.offset;
    for (int k = threadIdx.x; k < half; k += blockDim.x) {
        float sv, cv;
        sincosf(p * rope.inv_freq[k], &sv, &cv);
        sn[k] = sv * rope.magnitude; cs[k] = cv * rope.magnitude;
    }
    __syncthreads();
    float* row = x + (size_t)t * stride;
    const int per = half + (hd - rope.rot);          // work items a head: pairs, then single elements
    for (int i = threadIdx.x; i < heads * per; i += blockDim.x) {
        const int h = i / per, w = i % per;
        float* head = row + (size_t)h * hd;
        const float f = h >= scale_from ? scale : 1.f;
        if (w < half) {
            const int ia = rope.adjacent ? 2 * w : w, ib = rope.adjacent ? 2 * w + 1 : w + half;
            const float u = head[ia], v = head[ib];
            head[ia] = (u * cs[w] - v * sn[w]) * f;
            head[ib] = (v * cs[w] + u * sn[w]) * f;
        } else {
            head[rope.rot + (w - half)] *= f;
        }
    }
}

template <typename T, int R, int CH>
int launch_one(const LightningArgs& a, dim3 grid, cudaStream_t stream) {
    constexpr size_t smem = (size_t)CH * (2 * 4 * (R + 4) + 32) * sizeof(float);
    static bool configured = false;
    if (!configured && smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(lightning_scan_kernel<T, R, CH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        TB_REQUIRE(e == cudaSuccess, "lightning_scan: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
        configured = true;
    }
    tb_launch(lightning_scan_kernel<T, R, CH>, grid, 128, smem, stream, a);
    return 0;
}

// Rows of the state a thread keeps (a quarter of dk, rounded up to 8, 16, 32 or 64) and tokens staged at a time: sixteen for
// prompts, one for steps of single tokens (nothing to amortise, and less to request).
template <typename T, int R, int CH>
int launch_vec(const LightningArgs& a, cudaStream_t stream) {
    constexpr size_t smem = (size_t)CH * (2 * 8 * (R + 4) + 16) * sizeof(float);
    static_assert(smem <= 48 * 1024, "the staging area fits the default shared memory");
    dim3 grid(a.B, a.H, (a.dv + 15) / 16);
    tb_launch(lightning_scan_vec_kernel<T, R, CH>, grid, 128, smem, stream, a);
    return 0;
}

template <typename T>
int launch_scan(const LightningArgs& a, bool single, cudaStream_t stream) {
    if (a.work) return a.dk <= 64 ? launch_chunks<T, 64>(a, stream) : launch_chunks<T, 128>(a, stream);
    // sizes in multiples of 8 and rows that 16-byte loads can take: the kernel of eight lanes a column
    if (a.dk % 8 == 0 && a.dv % 8 == 0 && a.stride % 8 == 0 && ((uintptr_t)a.proj % 16 == 0) && a.dk >= 64 && (a.dv + 15) / 16 <= 65535) {
        const int rows = a.dk / 8;
        if (single) {
            if (rows <= 8) return launch_vec<T, 8, 1>(a, stream);
            if (rows <= 16) return launch_vec<T, 16, 1>(a, stream);
            return launch_vec<T, 32, 1>(a, stream);
        }
        if (rows <= 8) return launch_vec<T, 8, 16>(a, stream);
        if (rows <= 16) return launch_vec<T, 16, 16>(a, stream);
        return launch_vec<T, 32, 8>(a, stream);
    }
    dim3 grid(a.B, a.H, (a.dv + 31) / 32);
    const int rows = (a.dk + 3) / 4;
    if (single) {
        if (rows <= 8) return launch_one<T, 8, 1>(a, grid, stream);
        if (rows <= 16) return launch_one<T, 16, 1>(a, grid, stream);
        if (rows <= 32) return launch_one<T, 32, 1>(a, grid, stream);
        return launch_one<T, 64, 1>(a, grid, stream);
    }
    if (rows <= 8) return launch_one<T, 8, 16>(a, grid, stream);
    if (rows <= 16) return launch_one<T, 16, 16>(a, grid, stream);
    if (rows <= 32) return launch_one<T, 32, 16>(a, grid, stream);
    return launch_one<T, 64, 8>(a, grid, stream);
}

}  // namespace

// Floats a chunk takes in ``work``, and in ``chunks`` how many chunks a step of T tokens in B runs, the longest of max_new, has at most; 0: no run is
// long enough for the chunked form (or a head has more than 128 key dimensions).  The caller gives room for as many as it likes, one at least.
extern "C" long long tb_lightning_work(int T, int B, int H, int dk, int dv, int max_new, int* chunks) {
    *chunks = 0;
    if (max_new < CHUNKED_FROM || dk > 128 || ((long long)dk * dv + 1023) / 1024 > 65535) return 0;
    *chunks = T / CHUNK + min(B, T / CHUNKED_FROM);
    return (long long)H * (long long)room_floats(dk, dv);
}

extern "C" int tb_lightning_scan(const LightningArgs* args, int dtype, cudaStream_t stream) {
    LightningArgs a = *args;
    a.below = a.segment = 0;
    TB_REQUIRE(a.B > 0 && a.H > 0 && a.dk > 0 && a.dv > 0, "lightning_scan: sizes must be positive");
    TB_REQUIRE(a.dk <= 256, "lightning_scan: %d key dimensions a head (at most 256)", a.dk);
    TB_REQUIRE(a.H <= 65535 && (a.dv + 31) / 32 <= 65535, "lightning_scan: too many heads or value columns");
    TB_REQUIRE(a.proj && a.out && a.state && a.decay && a.q_start && a.slot_of_seq, "lightning_scan: missing buffers");
    TB_REQUIRE(a.stride >= 2 * a.H * a.dk + a.H * a.dv, "lightning_scan: the projection row is too short");
    TB_REQUIRE(dtype == TB_F32 || dtype == TB_BF16, "lightning_scan: unknown dtype %d", dtype);
    const bool single = a.max_new <= 1;
    TB_REQUIRE(!a.work || (a.dk <= 128 && a.work_chunks > 0 && a.work_room > 0 && ((long long)a.dk * a.dv + 1023) / 1024 <= 65535 && (uintptr_t)a.work % 16 == 0),
               "lightning_scan: the chunked form takes heads of up to 128 key dimensions (%d)", a.dk);
    if (dtype == TB_F32 ? launch_scan<float>(a, single, stream) : launch_scan<__nv_bfloat16>(a, single, stream)) return 1;
    TB_CHECK_LAUNCH("lightning_scan");
    return 0;
}

template <typename T>
static void launch_gated_rmsnorm(const float* o, int ldo, const float* w, const T* gate, int ldg, T* y, int ldy, int n_rows, int N, float eps, cudaStream_t stream) {
    // 16-byte units of every row, up to four a thread of 512; other widths, strides and addresses column by column
    if (N % 8 == 0 && N <= 16384 && ldo % 4 == 0 && ldg % 8 == 0 && ldy % 8 == 0 && (((uintptr_t)o | (uintptr_t)w | (uintptr_t)gate | (uintptr_t)y) & 15) == 0) {
        const int threads = N >= 4096 ? 512 : (N / 8 + 31) / 32 * 32;
        if (N <= 8 * threads) tb_launch(gated_rmsnorm_vec_kernel<T, 1>, n_rows, threads, 0, stream, o, ldo, w, gate, ldg, y, ldy, N, eps);
        else tb_launch(gated_rmsnorm_vec_kernel<T, 4>, n_rows, threads, 0, stream, o, ldo, w, gate, ldg, y, ldy, N, eps);
        return;
    }
    tb_launch(gated_rmsnorm_kernel<T>, n_rows, N >= 2048 ? 256 : (N >= 512 ? 128 : 64), 0, stream, o, ldo, w, gate, ldg, y, ldy, N, eps);
}

extern "C" int tb_gated_rmsnorm(const float* o, int ldo, const float* w, const void* gate, int ldg, void* y, int ldy,
                                int dtype, int n_rows, int N, float eps, cudaStream_t stream) {
    TB_REQUIRE(n_rows > 0 && N > 0 && o && w && gate && y, "gated_rmsnorm: sizes must be positive (rows=%d N=%d)", n_rows, N);
    if (dtype == TB_F32) launch_gated_rmsnorm<float>(o, ldo, w, (const float*)gate, ldg, (float*)y, ldy, n_rows, N, eps, stream);
    else if (dtype == TB_BF16) launch_gated_rmsnorm<__nv_bfloat16>(o, ldo, w, (const __nv_bfloat16*)gate, ldg, (__nv_bfloat16*)y, ldy, n_rows, N, eps, stream);
    else TB_REQUIRE(false, "gated_rmsnorm: unknown dtype %d", dtype);
    TB_CHECK_LAUNCH("gated_rmsnorm");
    return 0;
}

extern "C" int tb_rotary_rows(float* x, int stride, const int* pos_of, int n_rows, int heads, int hd, const TbRotary* rope, int scale_from,
                              float scale, cudaStream_t stream) {
    TB_REQUIRE(x && pos_of && rope && n_rows > 0 && heads > 0 && hd > 0 && stride >= heads * hd, "rotary_rows: rows of heads are wanted");
    TB_REQUIRE(rope->inv_freq && rope->rot > 0 && rope->rot % 2 == 0 && rope->rot <= hd, "rotary_rows: %d rotated dimensions of a head of %d", rope->rot, hd);
    tb_launch(rotary_rows_kernel, n_rows, 128, (size_t)rope->rot * sizeof(float), stream, x, stride, pos_of, heads, hd, *rope, scale_from, scale);
    TB_CHECK_LAUNCH("rotary_rows");
    return 0;
}
