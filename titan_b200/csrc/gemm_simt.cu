// Plain matrix product on the CUDA cores: out = X[M,K] . W[N,K]^T with float32 accumulation.
//
// This is the true 32-bit path (T = float: FFMA only, no tensor-core or reduced-precision mode)
// and the plain twin of the tensor-core kernel for bfloat16 operands; it takes every M, N, K.
// berniehans/titan's counterpart is its warp-per-column kernels
// (engine/engine-cuda/kernels/gemm_quant.cu:2331-2363 gemm_f32_kernel, :3365-3499 batched), which
// fuse the residual into the epilogue (:3489-3493) and SwiGLU into gate/up (:2589).
//
// One order of sums for every kernel here but one (gemm_heads_kernel), whatever M: in each run of SUM_RUN neighbouring k the products at even and those at
// odd k are added one after the other (fused multiply-adds from zero), then the two sums, and the runs' sums one after the
// other.  A row's result is then the same bits alone and beside any other rows, in a decode step as in a prompt.  Even
// and odd, because the two are neighbours in memory and one two-element instruction (fma.rn.f32x2) works on both.
//
// Epilogues:
//   TB_EPI_STORE   out[m][n] = acc                      (compute dtype), or an activation of it (activation.h)
//   TB_EPI_F32     out[m][n] = acc                      (float32: logits)
//   TB_EPI_ADD     out[m][n] += acc                     (float32 residual stream, in place)
//   TB_EPI_SWIGLU  out[m][j] = gate(acc[2j], acc[2j+1]) (rows of W interleaved gate, up; N even); the gate is
//                  silu(g) * u unless the launch names another (activation.h)
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "gemm.h"
#include "tma.cuh"

namespace {

// N elements of a row as one load (16 or 8 bytes) and as floats.
template <typename T, int N> struct Vec;
template <> struct Vec<float, 4> {
    float4 r;
    __device__ __forceinline__ void load(const float* p) { r = *reinterpret_cast<const float4*>(p); }
    __device__ __forceinline__ void get(float* o) const { o[0] = r.x; o[1] = r.y; o[2] = r.z; o[3] = r.w; }
};
template <> struct Vec<__nv_bfloat16, 4> {
    uint2 r;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { r = *reinterpret_cast<const uint2*>(p); }
    __device__ __forceinline__ void get(float* o) const {
        o[0] = __uint_as_float(r.x << 16); o[1] = __uint_as_float(r.x & 0xffff0000u);
        o[2] = __uint_as_float(r.y << 16); o[3] = __uint_as_float(r.y & 0xffff0000u);
    }
};
template <> struct Vec<__nv_bfloat16, 8> {
    uint4 r;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { r = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ void get(float* o) const {
        const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { o[2 * i] = __uint_as_float(w[i] << 16); o[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
    }
};
// Loads of activations that the compiler cannot take for loads of constants (as it may through a __restrict__ pointer to const): such a load could
// move above the wait for the kernel that writes them.  load_l2: rows that an SM reads once; load_row: rows that several of its warps read.
template <typename V> __device__ __forceinline__ V load_l2(const void* p);
template <> __device__ __forceinline__ float load_l2<float>(const void* p) {
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
template <> __device__ __forceinline__ __nv_bfloat16 load_l2<__nv_bfloat16>(const void* p) {
    unsigned short v;
    asm volatile("ld.global.cg.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
    return __ushort_as_bfloat16(v);
}
template <> __device__ __forceinline__ float4 load_l2<float4>(const void* p) {
    float4 v;
    asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}
template <> __device__ __forceinline__ uint2 load_l2<uint2>(const void* p) {
    uint2 v;
    asm volatile("ld.global.cg.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
    return v;
}
template <typename V> __device__ __forceinline__ V load_row(const void* p);
template <> __device__ __forceinline__ float load_row<float>(const void* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
template <> __device__ __forceinline__ __nv_bfloat16 load_row<__nv_bfloat16>(const void* p) {
    unsigned short v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
    return __ushort_as_bfloat16(v);
}
template <> __device__ __forceinline__ float4 load_row<float4>(const void* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}
template <> __device__ __forceinline__ uint4 load_row<uint4>(const void* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

// acc = a * b + acc on two neighbouring float32 at once, each rounded as fmaf rounds it (one instruction of sm_100a).
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pair_of(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float both(unsigned long long v) {      // the sum of the two
    return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}
__device__ __forceinline__ void copy16(void* to, const void* from, bool real = true) {      // zeros if not real
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from), "r"(real ? 16 : 0) : "memory");
}

constexpr int SUM_RUN = 32;

// ---------------------------------------------------------------- many rows: tiles
// Tiles of 64 x 64, K in steps of one run of sums, RI x 4 sums a thread: 4 x 4 (256 threads), or 8 x 4 (128 threads, fewer loads from
// shared memory a product) where there are tiles enough for three blocks an SM all the same.  Operands lie along K in shared memory (a row 16 bytes behind a whole
// number of banks: sixteen neighbouring rows do not collide), three steps deep; float32 rows come by cp.async and stay in flight for
// two steps.  Bound by the FMA pipes; several blocks an SM hide what is left of the latencies.  1,125 rows
// of K = 1,024: 5,632 columns 357 us (36 TFLOP/s), 1,024 columns 79 us; K = 2,816, 1,024 columns: 203 us (a kernel of 4 x 4 sums that
// waited for each step's operands took 445, 230 and 640 us).
constexpr int BM = 64, BN = 64, LDK = SUM_RUN + 4, TILE_STAGES = 3;
constexpr size_t TILE_SMEM = (size_t)TILE_STAGES * (BM + BN) * LDK * sizeof(float);

template <typename T, int EPI, int RI, bool VEC>
__global__ void __launch_bounds__(1024 / RI, RI == 4 ? 2 : 3)
gemm_simt_kernel(const T* X, const T* W, void* out_,
                 int M, int N, int K, int ldx, int ldo, long long sx, long long sw, long long so, int act, float limit) {
    constexpr int THREADS = 1024 / RI;
    pdl_launch_dependents();
    // blockIdx.z: one of a batch of products of equal shape (the heads of a mixer, say), each at its own offset
    X += (size_t)blockIdx.z * sx;
    W += (size_t)blockIdx.z * sw;
    void* out = (EPI == TB_EPI_STORE || EPI == TB_EPI_SWIGLU) ? (void*)((T*)out_ + (size_t)blockIdx.z * so)
                                                              : (void*)((float*)out_ + (size_t)blockIdx.z * so);
    extern __shared__ __align__(16) float tile_sm[];       // [TILE_STAGES][BM rows of X, BN rows of W][LDK]
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN, steps = (K + SUM_RUN - 1) / SUM_RUN;
    // Row r of the W area holds column 2 (r % 16) + r / 16 % 2 + 32 (r / 32) of the tile, so that the four a thread reads, sixteen rows
    // apart, are two pairs of neighbouring columns.
    auto stage = [&](bool weights, int step) {
        float* area = tile_sm + (size_t)((step % TILE_STAGES) * (BM + BN) + (weights ? BM : 0)) * LDK;
#pragma unroll
        for (int u = 0; u < BM * SUM_RUN / 4 / THREADS; ++u) {
            const int e = tid + THREADS * u, r = e / (SUM_RUN / 4), c = e % (SUM_RUN / 4) * 4, k = step * SUM_RUN + c;
            const int row = weights ? n0 + 2 * (r % 16) + r / 16 % 2 + 32 * (r / 32) : m0 + r;
            const bool real = row < (weights ? N : M) && k < K;
            const T* from = (weights ? W + (size_t)row * K : X + (size_t)row * ldx) + k;
            float* to = area + r * LDK + c;
            if constexpr (VEC && sizeof(T) == 4) {          // K is a multiple of four: a unit is inside or outside
                copy16(to, real ? from : X, real);
            } else if constexpr (VEC) {
                Vec<T, 4> v;
                float f[4] = {0.f, 0.f, 0.f, 0.f};
                if (real) { v.r = load_l2<decltype(v.r)>(from); v.get(f); }
                *reinterpret_cast<float4*>(to) = make_float4(f[0], f[1], f[2], f[3]);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    to[i] = 0.f;
                    if (real && k + i < K) { const T v = load_l2<T>(from + i); to[i] = ldf(&v); }
                }
            }
        }
    };
    float total[RI][4];
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) total[i][j] = 0.f;
    stage(true, 0);                                        // no kernel writes weights
    if (steps > 1) stage(true, 1);
    pdl_wait();
    stage(false, 0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (steps > 1) stage(false, 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                   // this step's rows are there; the step before has been read
        if (step + 2 < steps) { stage(true, step + 2); stage(false, step + 2); }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* xs = tile_sm + (size_t)(step % TILE_STAGES) * (BM + BN) * LDK + ty * LDK;
        const float* ws = tile_sm + (size_t)((step % TILE_STAGES) * (BM + BN) + BM + tx) * LDK;
        unsigned long long acc[RI][4] = {};
#pragma unroll 2
        for (int k = 0; k < SUM_RUN; k += 4) {
            ulonglong2 b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(ws + 16 * j * LDK + k);
#pragma unroll
            for (int i = 0; i < RI; ++i) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(xs + (64 / RI) * i * LDK + k);
#pragma unroll
                for (int j = 0; j < 4; ++j) { fma2(acc[i][j], a.x, b[j].x); fma2(acc[i][j], a.y, b[j].y); }
            }
        }
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) total[i][j] += both(acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        const int m = m0 + ty + (64 / RI) * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            const int n = n0 + 2 * tx + 16 * j;
            if (EPI == TB_EPI_SWIGLU) {
                if (n + 1 < N) stf((T*)out + (size_t)m * ldo + n / 2, tb_gated(act, limit, total[i][j], total[i][j + 1]));
                continue;
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (n + e >= N) continue;
                const size_t at = (size_t)m * ldo + n + e;
                const float v = total[i][j + e];
                if (EPI == TB_EPI_STORE) stf((T*)out + at, tb_unary(act, v));
                if (EPI == TB_EPI_F32) ((float*)out)[at] = v;
                if (EPI == TB_EPI_ADD) ((float*)out)[at] = load_l2<float>((float*)out + at) + v;
            }
        }
    }
}

// ---------------------------------------------------------------- few rows: weights streamed once
// A step of a few tokens is bound by the weights' bytes, and in 64 x 64 tiles most of the chip idles: 16 blocks for
// 1,024 columns, each walking all of K.  Here a block takes eight columns (COLS) at a time and up to MR rows, and its 256 threads the runs of
// SUM_RUN along K, a thread one column and one run.  A unit of work is eight columns and ``pass`` runs; its weights come into shared
// memory as one bulk copy a column, up to three units ahead, those of the first units before the wait for the kernel before (no
// kernel writes weights); the rows of X by cp.async, once a block where K is one pass.  A column of weights lies 16 bytes behind a whole
// number of banks and a run of X likewise, so that a warp's eight columns and four runs do not collide.  The run sums meet in shared
// memory and are added in order by a thread an output.  Each weight is read from memory once for MR rows; rows beyond
// are further blocks, which find the weights in L2.  Three rows: 1,024 columns
// of K = 2,816 in 6.4 us, 5,632 of K = 1,024 in 10.0, 32,768 in 30.5 (64 x 64 tiles: 189, 87 and 204 us; with copies of sixteen bytes a
// thread, and one warp that issued, added and waited in turn: 7.1, 12.9 and 59).
template <typename T> constexpr int few_run() { return SUM_RUN + 16 / (int)sizeof(T); }           // elements from a run to the next in shared memory
template <typename T> __host__ __device__ constexpr int few_col(int pass) { return pass * SUM_RUN + 16 / (int)sizeof(T); }      // a column of weights
template <typename T> __host__ __device__ constexpr int few_row(int pass) { return pass * few_run<T>(); }                         // a row of X
// Shared memory: the barriers; per stage [COLS] columns of ``pass`` runs and, where K takes several passes, [MR] rows; else the rows
// once, behind the stages; then two areas of run sums.
template <typename T, int MR, int COLS> size_t few_smem(int pass, int stages, bool one_pass) {
    return 64 + (size_t)stages * COLS * few_col<T>(pass) * sizeof(T) + (size_t)(one_pass ? 1 : stages) * MR * few_row<T>(pass) * sizeof(T) +
           (size_t)2 * pass * MR * COLS * sizeof(float);
}
__device__ unsigned int g_few_error = 0;

template <typename T, int EPI, int MR, int COLS, bool VEC>
__global__ void __launch_bounds__(256)
gemm_few_kernel(const T* X, const T* W, void* out_, int M, int N, int K, int ldx, int ldo, long long sx, long long sw, long long so,
                int pass, int stages, int act, float limit) {
    constexpr int RS = few_run<T>(), PER = 16 / (int)sizeof(T), UNITS = SUM_RUN / PER;
    pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char few_sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * MR, z = blockIdx.z;
    const int runs = (K + SUM_RUN - 1) / SUM_RUN, passes = (runs + pass - 1) / pass, groups = (N + COLS - 1) / COLS;
    const int cs = few_col<T>(pass), rs = few_row<T>(pass), stage_elems = COLS * cs + (passes > 1 ? MR * rs : 0);
    uint64_t* const landed = reinterpret_cast<uint64_t*>(few_sm);        // [stages]
    T* const stage0 = reinterpret_cast<T*>(few_sm + 64);   // [stages][COLS][cs] ([MR][rs])
    T* const x0 = stage0 + (passes > 1 ? COLS * cs : stages * stage_elems);        // rows of X: in every stage, or once
    float* const sums0 = reinterpret_cast<float*>(stage0 + stages * stage_elems + (passes > 1 ? 0 : MR * rs));      // [2][pass][MR][COLS]
    // ``here`` runs of one row from run ``first`` on into shared memory, by ``step`` threads; elements beyond K are zero
    auto stage = [&](T* to, int run, const T* row, int first, int here, int at, int step) {
        for (int u = at; u < here * UNITS; u += step) {
            T* dst = to + u / UNITS * run + u % UNITS * PER;
            const int k = first * SUM_RUN + u * PER;
            if (VEC && k < K) { copy16(dst, row + k); continue; }
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                T e = T(0.f);
                if (!VEC && k + i < K) e = load_l2<T>(row + k + i);
                dst[i] = e;
            }
        }
    };
    // unit u of this block: group blockIdx.x + (u / passes) * gridDim.x, pass u % passes
    const int my_groups = groups > (int)blockIdx.x ? (groups - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0, units = my_groups * passes;
    auto stage_w = [&](int u) {                            // columns outside: any valid one
        const int n0 = (blockIdx.x + u / passes * gridDim.x) * COLS, first = u % passes * pass, here = min(pass, runs - first);
        T* to = stage0 + (u % stages) * stage_elems;
        const T* from = W + (size_t)z * sw;
        if (VEC) {
            if (lane < COLS / 8) {                         // every warp its columns: one thread for all would be what a unit waits for
                const uint32_t bytes = (uint32_t)(min(here * SUM_RUN, K - first * SUM_RUN) * sizeof(T));
                const int c = warp * (COLS / 8) + lane;
                tbtma::mbar_expect_tx(landed + u % stages, bytes);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(tbtma::smem_u32(to + c * cs)),
                             "l"(from + (size_t)min(n0 + c, N - 1) * K + first * SUM_RUN), "r"(bytes), "r"(tbtma::smem_u32(landed + u % stages)) : "memory");
            }
        } else {
            for (int c = warp; c < COLS; c += 8) stage(to + c * cs, SUM_RUN, from + (size_t)min(n0 + c, N - 1) * K, first, here, lane, 32);
        }
    };
    auto stage_x = [&](int u) {                            // rows outside: any valid one
        const int first = u % passes * pass;
        for (int m = 0; m < MR; ++m)
            stage(x0 + (passes > 1 ? (u % stages) * stage_elems : 0) + m * rs, RS, X + (size_t)z * sx + (size_t)min(m0 + m, M - 1) * ldx, first,
                  min(pass, runs - first), tid, 256);
    };
    if (VEC) {
        if (tid == 0) {
            for (int s = 0; s < stages; ++s) tbtma::mbar_init(landed + s, COLS);
            tbtma::mbar_fence_init();
        }
        __syncthreads();
    }
    const int om = tid / COLS, on = tid % COLS;   // a thread's output, if it has one
    const int col = tid % COLS;
    float total = 0.f;
    // the rows of unit u arrive with copy group u: the first ``stages`` - 1 units together in group 0, empty groups after it
    for (int u = 0; u < min(units, max(1, stages - 1)); ++u) stage_w(u);
    pdl_wait();
    for (int u = 0; u < (passes > 1 ? min(units, max(1, stages - 1)) : 1); ++u) stage_x(u);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int u = 1; u < stages - 1; ++u) asm volatile("cp.async.commit_group;" ::: "memory");
    for (int u = 0; u < units; ++u) {
        if (stages > 1 && u + stages - 1 < units) {
            stage_w(u + stages - 1);
            if (passes > 1) stage_x(u + stages - 1);
        }
        if (stages > 1) asm volatile("cp.async.commit_group;" ::: "memory");
        if (stages == 4) asm volatile("cp.async.wait_group 3;" ::: "memory");
        else if (stages == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
        else if (stages == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (VEC) tbtma::mbar_wait(landed + u % stages, (u / stages) & 1, &g_few_error, 1);
        const int here = min(pass, runs - u % passes * pass);
        float* sums = sums0 + (u & 1) * pass * MR * COLS;
        const T* st = stage0 + (u % stages) * stage_elems;
        const T* sx_ = x0 + (passes > 1 ? (u % stages) * stage_elems : 0);
        for (int r = tid / COLS; r < here; r += 256 / COLS) {
            unsigned long long acc[MR];
#pragma unroll
            for (int m = 0; m < MR; ++m) acc[m] = 0ull;
            const T* wr = st + col * cs + r * SUM_RUN;
            const T* xr = sx_ + r * RS;
            const int k0 = (u % passes * pass + r) * SUM_RUN;
            auto unit = [&](int i) {
                Vec<T, PER> v;
                float wf[PER], xf[PER];
                v.load(wr + i * PER);
                v.get(wf);
#pragma unroll
                for (int m = 0; m < MR; ++m) {
                    v.load(xr + m * rs + i * PER);
                    v.get(xf);
#pragma unroll
                    for (int e = 0; e < PER; e += 2) fma2(acc[m], pair_of(xf[e], xf[e + 1]), pair_of(wf[e], wf[e + 1]));
                }
            };
            if (!VEC || k0 + SUM_RUN <= K) {
#pragma unroll
                for (int i = 0; i < UNITS; ++i) unit(i);
            } else {                                       // the last run, cut short: nothing was copied behind K, a multiple of PER
                for (int i = 0; k0 + i * PER < K; ++i) unit(i);
            }
#pragma unroll
            for (int m = 0; m < MR; ++m) sums[(r * MR + m) * COLS + col] = both(acc[m]);
        }
        __syncthreads();
        if (tid >= MR * COLS) continue;
        {
            const float* mine = sums + om * COLS + on;
            int r = 0;
            for (; r + 16 <= here; r += 16) {              // all loads first
                float v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = mine[(r + i) * MR * COLS];
#pragma unroll
                for (int i = 0; i < 16; ++i) total += v[i];
            }
            for (; r < here; ++r) total += mine[r * MR * COLS];
        }
        if (u % passes != passes - 1) continue;
        const int m = m0 + om, n = (blockIdx.x + u / passes * gridDim.x) * COLS + on;
        // the gate of a pair: its second column is the neighbouring thread's
        const float right = __shfl_down_sync(MR * COLS >= 32 ? 0xffffffffu : (1u << (MR * COLS % 32)) - 1u, total, 1);
        if (m < M && n < N) {
            const size_t at = (size_t)z * so + (size_t)m * ldo + n;
            if (EPI == TB_EPI_SWIGLU) { if (n % 2 == 0) stf((T*)out_ + (size_t)z * so + (size_t)m * ldo + n / 2, tb_gated(act, limit, total, right)); }
            if (EPI == TB_EPI_STORE) stf((T*)out_ + at, tb_unary(act, total));
            if (EPI == TB_EPI_F32) ((float*)out_)[at] = total;
            if (EPI == TB_EPI_ADD) ((float*)out_)[at] = load_l2<float>((float*)out_ + at) + total;
        }
        total = 0.f;
    }
}

// ---------------------------------------------------------------- small products: operands straight into registers
// The kernel above pays for its rows in shared memory in every block and for two or three barriers before the first sum: a router of
// 128 columns of K = 4,096 in bfloat16 took 9.7 us for eight rows.  Here a thread has one column and one run of SUM_RUN at a time, ``lanes`` of
// a block's threads along K, and a block one row: it loads both operands of the run itself (neighbouring threads have
// neighbouring columns of the same run, a row's loads are shared by the warp) and leaves the run's sum in shared memory, where a
// thread a column adds them in order: one barrier, 5.1 us for the router.  The weights of the first run come before the wait.  Bound by latency;
// weights are read once a row through L2 (two and four rows a block were slower wherever this kernel is the fastest).
template <typename T, bool VEC>
__global__ void __launch_bounds__(256)
gemm_small_kernel(const T* X, const T* W, void* out_, int N, int K, int ldx, int ldo, long long sx, long long sw, long long so,
                  int lanes, int pass, int epi, int act, float limit) {
    constexpr int PER = 16 / (int)sizeof(T), UNITS = SUM_RUN / PER;
    pdl_launch_dependents();
    extern __shared__ float small_sm[];                    // [pass][columns]
    const int tid = threadIdx.x, cols = (int)blockDim.x / lanes, col = tid % cols, lane = tid / cols, n = blockIdx.x * cols + col, runs = (K + SUM_RUN - 1) / SUM_RUN;
    const T* w = W + (size_t)blockIdx.z * sw + (size_t)n * K;
    const T* x = X + (size_t)blockIdx.z * sx + (size_t)blockIdx.y * ldx;
    float wf[SUM_RUN];
    auto load_w = [&](int k) {                             // (VEC: K is a multiple of a unit; places beyond it take the row's first)
        if constexpr (VEC) {
            Vec<T, PER> v[UNITS];
#pragma unroll
            for (int i = 0; i < UNITS; ++i) v[i].load(w + (k + i * PER < K ? k + i * PER : 0));
#pragma unroll
            for (int i = 0; i < UNITS; ++i) v[i].get(wf + i * PER);
        } else {
#pragma unroll
            for (int e = 0; e < SUM_RUN; ++e) wf[e] = k + e < K ? ldf(w + k + e) : 0.f;
        }
    };
    if (lane < runs && n < N) load_w(lane * SUM_RUN);
    pdl_wait();
    float total = 0.f;
    for (int p0 = 0; p0 < runs; p0 += pass) {
        const int here = min(pass, runs - p0);
        for (int r = p0 + lane; r < p0 + here && n < N; r += lanes) {
            const int k = r * SUM_RUN;
            if (r >= lanes) load_w(k);
            unsigned long long acc = 0ull;
            if constexpr (VEC) {
                Vec<T, PER> v[UNITS];
#pragma unroll
                for (int i = 0; i < UNITS; ++i) v[i].r = load_row<decltype(v[i].r)>(x + (k + i * PER < K ? k + i * PER : 0));
#pragma unroll
                for (int i = 0; i < UNITS; ++i) {
                    float xf[PER];
                    v[i].get(xf);
                    if (k + i * PER < K)
#pragma unroll
                        for (int e = 0; e < PER; e += 2) fma2(acc, pair_of(xf[e], xf[e + 1]), pair_of(wf[i * PER + e], wf[i * PER + e + 1]));
                }
            } else {
                float xf[SUM_RUN];
#pragma unroll
                for (int e = 0; e < SUM_RUN; ++e) {
                    xf[e] = 0.f;
                    if (k + e < K) { const T v = load_row<T>(x + k + e); xf[e] = ldf(&v); }
                }
#pragma unroll
                for (int e = 0; e < SUM_RUN; e += 2) fma2(acc, pair_of(xf[e], xf[e + 1]), pair_of(wf[e], wf[e + 1]));
            }
            small_sm[(r - p0) * cols + col] = both(acc);
        }
        __syncthreads();
        if (tid < cols && n < N) {
            const float* mine = small_sm + col;
            int r = 0;
            for (; r + 16 <= here; r += 16) {              // all loads first
                float v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = mine[(r + i) * cols];
#pragma unroll
                for (int i = 0; i < 16; ++i) total += v[i];
            }
            for (; r < here; ++r) total += mine[r * cols];
        }
        if (p0 + pass < runs) __syncthreads();
    }
    // the gate of a pair: its second column is the neighbouring thread's (an even number of columns a block)
    const float right = __shfl_down_sync(0xffffffffu, total, 1);
    if (tid >= cols || n >= N) return;
    const size_t row = (size_t)blockIdx.z * so + (size_t)blockIdx.y * ldo;
    if (epi == TB_EPI_SWIGLU) { if (n % 2 == 0) stf((T*)out_ + row + n / 2, tb_gated(act, limit, total, right)); }
    else if (epi == TB_EPI_STORE) stf((T*)out_ + row + n, tb_unary(act, total));
    else if (epi == TB_EPI_F32) ((float*)out_)[row + n] = total;
    else ((float*)out_)[row + n] = load_l2<float>((float*)out_ + row + n) + total;
}

// ---------------------------------------------------------------- heads' products of a decode step in bfloat16: a warp an output
// Products of a batch (STORE epilogue) whose rows are few: lanes along K with 16-byte loads of whole rows, so that weights stream at the
// best rate of all kernels here, once for each row.  The one kernel with an order of sums of its own: what it makes is rounded to
// bfloat16, and the products around it do not keep one order either; float32 takes the kernels above.
__global__ void __launch_bounds__(256)
gemm_heads_kernel(const __nv_bfloat16* __restrict__ X, const __nv_bfloat16* __restrict__ W, __nv_bfloat16* __restrict__ out_, int N, int K, int ldx, int ldo,
                  long long sx, long long sw, long long so, int act) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = blockIdx.x * 8 + warp;
    if (n >= N) return;
    const __nv_bfloat16* x = X + (size_t)blockIdx.z * sx + (size_t)blockIdx.y * ldx;
    const __nv_bfloat16* w = W + (size_t)blockIdx.z * sw + (size_t)n * K;
    float acc = 0.f;
    if (K % 8 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0) {
        for (int k = lane * 8; k < K; k += 256) {
            const uint4 a = *reinterpret_cast<const uint4*>(x + k), b = *reinterpret_cast<const uint4*>(w + k);
            const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc = fmaf(__uint_as_float(aw[i] << 16), __uint_as_float(bw[i] << 16), acc);
                acc = fmaf(__uint_as_float(aw[i] & 0xffff0000u), __uint_as_float(bw[i] & 0xffff0000u), acc);
            }
        }
    } else {
        for (int k = lane; k < K; k += 32) acc = fmaf(ldf(x + k), ldf(w + k), acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) stf(out_ + (size_t)blockIdx.z * so + (size_t)blockIdx.y * ldo + n, tb_unary(act, acc));
}

int sm_count() {
    static std::atomic<int> count[64];                     // a device each
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && (n = count[dev].load()) > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    if (dev < 64) count[dev].store(n);
    return n;
}

// Shared memory beyond 48 KB is asked for once a device and kernel, for the largest launch there is: a limit that each launch set for itself
// would be lowered under the launch of another thread.
template <auto Kernel>
int allow_smem(size_t most) {
    static std::atomic<bool> allowed[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && allowed[dev].load()) return 0;
    const cudaError_t e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    TB_REQUIRE(e == cudaSuccess, "gemm: cannot reserve %zu bytes of shared memory: %s", most, cudaGetErrorString(e));
    if (dev < 64) allowed[dev].store(true);
    return 0;
}

struct Product {
    const void* X; const void* W; void* out;
    int M, N, K, ldx, ldo, batch;
    long long sx, sw, so;
    int act; float limit;
    cudaStream_t stream;
};

// 16-byte loads of the few-rows kernel, four-element loads of the tiles: every row of every product starts on such a boundary.
template <typename T>
bool aligned(const Product& p, int per) {
    const size_t bytes = per * sizeof(T);
    return p.K % per == 0 && p.ldx % per == 0 && (uintptr_t)p.X % bytes == 0 && (uintptr_t)p.W % bytes == 0 &&
           (p.batch == 1 || (p.sx % per == 0 && p.sw % per == 0));
}

constexpr size_t FEW_SMEM = 220 * 1024;

template <typename T, int EPI, int MR, int COLS, bool VEC>
int few_launch(const Product& p) {
    const int SMS = sm_count();
    const int runs = (p.K + SUM_RUN - 1) / SUM_RUN, groups = (p.N + COLS - 1) / COLS, others = (p.M + MR - 1) / MR * p.batch;
    // One unit a block while the blocks fit the chip once: all of K at once.  Else passes of 32 runs (one a thread) and equal shares of the
    // column groups, for two blocks an SM with two stages each where their memory fits (one computes while the other waits), or
    // one block with up to four.
    const bool once = (long long)groups * others <= SMS;
    int pass = once ? 96 : 32;
    if (pass > runs) pass = runs;
    while (few_smem<T, MR, COLS>(pass, 1, pass >= runs) > 200 * 1024) --pass;
    const int passes = (runs + pass - 1) / pass, two = few_smem<T, MR, COLS>(pass, 2, passes == 1) <= 112 * 1024;
    const int room = (two ? 2 : 1) * SMS / others > 0 ? (two ? 2 : 1) * SMS / others : 1, each = (groups + room - 1) / room, x = (groups + each - 1) / each;
    const long long units = (long long)((groups + x - 1) / x) * passes;
    int stages = units < (two ? 2 : 4) ? (int)units : (two ? 2 : 4);
    while (stages > 1 && few_smem<T, MR, COLS>(pass, stages, passes == 1) > FEW_SMEM) --stages;
    if (stages == 1 && units > 1) { stages = 2; while (few_smem<T, MR, COLS>(pass, stages, false) > FEW_SMEM) --pass; }
    const size_t smem = few_smem<T, MR, COLS>(pass, stages, (runs + pass - 1) / pass == 1);
    const dim3 grid(x, (p.M + MR - 1) / MR, p.batch);
    if (smem > 48 * 1024 && allow_smem<gemm_few_kernel<T, EPI, MR, COLS, VEC>>(FEW_SMEM)) return 1;
    tb_launch(gemm_few_kernel<T, EPI, MR, COLS, VEC>, grid, 256, smem, p.stream, (const T*)p.X, (const T*)p.W, p.out, p.M, p.N, p.K, p.ldx, p.ldo,
              p.sx, p.sw, p.so, pass, stages, p.act, p.limit);
    return 0;
}
template <typename T, int EPI, int MR>
int few_rows(const Product& p) {
    // 32 columns a unit where a column has at most eight runs (with eight columns most of the block would have no run: sixteen heads'
    // products of 8 rows, 576 columns of K = 128, bfloat16: 9.4 -> 4.7 us)
    if (!aligned<T>(p, 16 / (int)sizeof(T))) return few_launch<T, EPI, MR, 8, false>(p);
    if (p.K <= 8 * SUM_RUN) return few_launch<T, EPI, MR, 32, true>(p);
    return few_launch<T, EPI, MR, 8, true>(p);
}

template <typename T, bool VEC>
int small_launch(const Product& p, int epi) {
    const int runs = (p.K + SUM_RUN - 1) / SUM_RUN;
    int lanes = 1, threads = 256;
    while (lanes < runs && lanes < 128) lanes *= 2;
    // smaller blocks while there are fewer than two an SM: a warp's columns are as many lines of the L1, which one SM would take one by one
    while (threads > 64 && threads / 2 >= 2 * lanes && (long long)p.N * lanes / threads * p.M * p.batch < 2 * sm_count()) threads /= 2;
    const int pass = runs < 16 * lanes ? runs : 16 * lanes, cols = threads / lanes;
    const dim3 grid((p.N + cols - 1) / cols, p.M, p.batch);
    tb_launch(gemm_small_kernel<T, VEC>, grid, threads, (size_t)pass * cols * sizeof(float), p.stream, (const T*)p.X, (const T*)p.W, p.out, p.N, p.K,
              p.ldx, p.ldo, p.sx, p.sw, p.so, lanes, pass, epi, p.act, p.limit);
    return 0;
}

template <typename T, int EPI, int RI, bool VEC>
int tiles(const Product& p) {
    const dim3 grid((p.N + BN - 1) / BN, (p.M + BM - 1) / BM, p.batch);
    if (allow_smem<gemm_simt_kernel<T, EPI, RI, VEC>>(TILE_SMEM)) return 1;
    tb_launch(gemm_simt_kernel<T, EPI, RI, VEC>, grid, 1024 / RI, TILE_SMEM, p.stream, (const T*)p.X, (const T*)p.W, p.out, p.M, p.N, p.K, p.ldx, p.ldo,
              p.sx, p.sw, p.so, p.act, p.limit);
    return 0;
}

// Which kernel.  All but the warp an output add in the one order, so that these lines, measured in us, decide about time alone.
enum Kind { SMALL, HEADS, FEW, TILES };
template <typename T>
Kind kind_of(const Product& p, int epi) {
    const int M = p.M, K = p.K, groups = (M + 7) / 8;
    const long long columns = (long long)p.N * p.batch, products = columns * M * K;
    const bool wide = aligned<T>(p, 16 / (int)sizeof(T));
    // Heads in bfloat16, warp an output / small / few / tiles: 128 heads of 128 columns, K = 512: 1 row 4.6 / 8.9 / 15 / 42, 8 rows 22 / 58 / 21 / 42;
    // four of 2,048, K = 2,048: 8 rows 24 / 85 / 30 / 157, 16 rows 45 / 165 / 51 / 157; 64 of 576, K = 128: 1 row 6.6 / 5.6 / 10 / 21, 4 rows 21 / 17 /
    // 13 / 21; 16 of 576, K = 128: 2 rows 3.5 / 2.6 / 2.6 / 10, 8 rows 11 / 8 / 4.1 / 10; four of 64, K = 64: 8 rows 1.5 / 1.6 / 3.0 / 3.5.
    if (sizeof(T) == 2 && p.batch > 1 && epi == TB_EPI_STORE && M <= 16) {
        if (M <= 2 && K <= 128 && wide) return SMALL;
        if (M <= 2 || K >= 1024 || (K >= 512 && M <= 12 && !(M == 8 && columns >= 16384)) || columns * M <= 12288) return HEADS;
    }
    // Small / few: up to half a million products the few-rows kernel's fixed cost decides (512 columns of K = 1,024, float32: 1 row 2.3 / 2.3, 2 rows
    // 2.8 / 2.5; 1,024 of K = 36, bfloat16: 8 rows 3.1 / 5.5); with few columns or short ones later (128 of K = 2,048: 8 rows 3.8 / 5.0, 16 rows
    // 5.9 / 5.0; eight heads of 100, K = 96: 8 rows 2.4 / 3.3), with long ones, whose rows it would take through shared memory in every block, later still (64 of K = 8,192: 8 rows 11 / 23,
    // 32 rows 26 / 23), and in bfloat16, whose loads are half as many, at four times the size (1,024 of K = 1,024: 2 rows 2.6 / 3.1, 4 rows 5.1 / 3.8).
    const int most = (columns <= 256 || K <= 64 || (K <= 128 && columns <= 1024) || (sizeof(T) == 2 && columns <= 4096)) ? (K > 2048 && columns <= 256 ? 6 << 20 : 2 << 20) : 1 << 19;
    // Rows that 16-byte loads cannot take: only short ones (1,024 of K = 1,023, bfloat16, 1 row: 5.9 / 3.2).
    if (products <= most && M <= 64 && (wide || K <= 128)) return SMALL;
    if (M == 1 && p.batch >= 32 && columns >= 16384) return SMALL;      // (one row of many heads, float32: 128 of 512 columns, K = 128: 11 / 16)
    if (M > 64) return TILES;
    // Few / tiles: every group of eight rows is a pass over the weights, which tiles read once for 64.  One group is always few (float32, K = 1,024: 8 rows
    // of 32,768 columns 56 / 140, of 151,936 247 / 538), two up to 32,768 columns (108 / 140; of 151,936, K = 2,560: 1,786 / 1,345), more while all groups'
    // columns stay below a bound (5,632 columns: 48 rows 58 / 67, 64 rows 77 / 69; 8,192: 32 rows 55 / 69, 48 rows 83 / 69), which is lower where K is
    // short, as the tiles then are (8,192 of K = 128: 16 rows 7.2 / 9.7, 32 rows 13 / 10; 40,000 of K = 32: 8 rows 13 / 7.1).
    if (K <= 64 && columns > 32768) return TILES;
    // Rows that 16-byte loads cannot take: 5,000 columns of K = 100, bfloat16: 4 rows 8.6 / 9.0, 8 rows 12.7 / 9.1; 3,000 of K = 1,001: 48 rows 80 / 85,
    // 64 rows 102 / 87 (float32).
    if (!wide && K <= 128 && M > 4) return TILES;
    if (!wide && groups > 1) return groups * columns <= 20480 ? FEW : TILES;
    if (groups == 1 || (groups == 2 && K > 128 && columns <= 32768)) return FEW;
    return groups * columns <= (K > 128 ? 36864 : 28672) ? FEW : TILES;
}

template <typename T, int EPI>
int product(const Product& p) {
    switch (kind_of<T>(p, EPI)) {
        case SMALL: return aligned<T>(p, 16 / (int)sizeof(T)) ? small_launch<T, true>(p, EPI) : small_launch<T, false>(p, EPI);
        case HEADS:
            if constexpr (sizeof(T) == 2)
                tb_launch(gemm_heads_kernel, dim3((p.N + 7) / 8, p.M, p.batch), 256, 0, p.stream, (const T*)p.X, (const T*)p.W, (T*)p.out, p.N, p.K, p.ldx, p.ldo,
                          p.sx, p.sw, p.so, p.act);
            return 0;
        case FEW:
            if (p.M == 1) return few_rows<T, EPI, 1>(p);
            if (p.M == 2) return few_rows<T, EPI, 2>(p);
            if (p.M <= 4) return few_rows<T, EPI, 4>(p);
            return few_rows<T, EPI, 8>(p);
        case TILES: break;
    }
    // 8 x 4 sums a thread from four tiles an SM on (5,632 columns of K = 1,024: 1,125 rows 389 -> 357 us, 3,000 rows 980 -> 888 us);
    // below, twice the warps are worth more (1,125 rows, 1,024 columns of K = 2,816: 294 -> 203 us)
    const long long count = (long long)((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN) * p.batch;
    if (!aligned<T>(p, 4)) return tiles<T, EPI, 4, false>(p);
    if (count >= 4 * sm_count()) return tiles<T, EPI, 8, true>(p);
    return tiles<T, EPI, 4, true>(p);
}

template <typename T>
int run(const Product& p, int epi) {
    switch (epi) {
        case TB_EPI_STORE: return product<T, TB_EPI_STORE>(p);
        case TB_EPI_F32: return product<T, TB_EPI_F32>(p);
        case TB_EPI_ADD: return product<T, TB_EPI_ADD>(p);
        case TB_EPI_SWIGLU: return product<T, TB_EPI_SWIGLU>(p);
    }
    tb_set_error("gemm: unknown epilogue %d", epi);
    return 1;
}

}  // namespace

// Clears and returns the code of a bounded wait that gave up (0: none): the results since the last call are then invalid.
extern "C" int tb_gemm_few_error() {
    unsigned int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_few_error, sizeof v) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_few_error, &zero, sizeof zero);
    return (int)v;
}

// ldx: row stride of X in elements; ldo: row stride of out in elements.  ``batch`` products of the same shape in one
// launch: product z reads X + z * sx and W + z * sw and writes out + z * so (offsets in elements).
// act, limit: the gate of the SWIGLU epilogue, or the activation of the STORE epilogue (activation.h).
extern "C" int tb_gemm_simt_gated(const void* X, const void* W, void* out, int dtype, int M, int N, int K, int ldx,
                                  int ldo, int epi, int batch, long long sx, long long sw, long long so, int act, float limit,
                                  cudaStream_t stream) {
    TB_REQUIRE(act >= 0 && act < (epi == TB_EPI_STORE ? TB_UNARY_KINDS : TB_ACT_KINDS), "gemm: unknown gate or activation %d", act);
    TB_REQUIRE(M > 0 && N > 0 && K > 0, "gemm: sizes must be positive (M=%d N=%d K=%d)", M, N, K);
    TB_REQUIRE(batch > 0 && batch <= 65535, "gemm: a batch of %d products", batch);
    TB_REQUIRE(ldx >= K, "gemm: row stride %d of X is shorter than K=%d", ldx, K);
    TB_REQUIRE(epi != TB_EPI_SWIGLU || N % 2 == 0, "gemm: the SwiGLU epilogue needs an even N, found %d", N);
    TB_REQUIRE((M + 63) / 64 <= 65535, "gemm: M=%d is too large for one launch", M);
    const Product p{X, W, out, M, N, K, ldx, ldo, batch, sx, sw, so, act, limit, stream};
    int rc;
    if (dtype == TB_F32) rc = run<float>(p, epi);
    else if (dtype == TB_BF16) rc = run<__nv_bfloat16>(p, epi);
    else { tb_set_error("gemm: unknown dtype %d", dtype); return 1; }
    if (rc) return rc;
    TB_CHECK_LAUNCH("gemm_simt");
    return 0;
}

extern "C" int tb_gemm_simt_batched(const void* X, const void* W, void* out, int dtype, int M, int N, int K, int ldx,
                                    int ldo, int epi, int batch, long long sx, long long sw, long long so, cudaStream_t stream) {
    return tb_gemm_simt_gated(X, W, out, dtype, M, N, K, ldx, ldo, epi, batch, sx, sw, so, TB_ACT_SILU, 0.f, stream);
}

extern "C" int tb_gemm_simt(const void* X, const void* W, void* out, int dtype, int M, int N, int K, int ldx,
                            int ldo, int epi, cudaStream_t stream) {
    return tb_gemm_simt_batched(X, W, out, dtype, M, N, K, ldx, ldo, epi, 1, 0, 0, 0, stream);
}

// ``act``: the activation of the STORE epilogue (activation.h).
// out (epilogue store, float32 or add) = X[M,K] . W[N,K]^T: the products of a decode step whose matrices are too small to pay for a
// tensor-core launch (a router, a narrow gate).
extern "C" int tb_gemm_rows(const void* X, const void* W, void* out, int dtype, int M, int N, int K, int ldx, int ldo, int epi,
                            int act, cudaStream_t stream) {
    TB_REQUIRE(epi == TB_EPI_STORE ? act >= 0 && act < TB_UNARY_KINDS : act == 0, "gemm_rows: unknown activation %d", act);
    TB_REQUIRE(M > 0 && N > 0 && K > 0 && M <= 65535, "gemm_rows: sizes (M=%d N=%d K=%d)", M, N, K);
    TB_REQUIRE(ldx >= K, "gemm_rows: row stride %d of X is shorter than K=%d", ldx, K);
    TB_REQUIRE(epi != TB_EPI_SWIGLU, "gemm_rows: epilogue %d is not one of store, float32, add", epi);
    const Product p{X, W, out, M, N, K, ldx, ldo, 1, 0, 0, 0, act, 0.f, stream};
    int rc;
    if (dtype == TB_F32) rc = run<float>(p, epi);
    else if (dtype == TB_BF16) rc = run<__nv_bfloat16>(p, epi);
    else { tb_set_error("gemm_rows: unknown dtype %d", dtype); return 1; }
    if (rc) return rc;
    TB_CHECK_LAUNCH("gemm_rows");
    return 0;
}
