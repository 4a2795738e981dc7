// out[M, N] = x[M, K] . w[N, K]^T in true 32-bit: plain FMA on CUDA cores, no tensor cores, no reduced-precision mode.
// (The reference's exact path is the CPU integer matmul of src/detllm/backends.py:95-96; this is its float counterpart.)
//
// One order of summation.  The inner axis is cut into segments of 128, dealt to eight classes in turn (class c: segments c,
// c + 8, ...).  A class is one chain of FMAs in ascending k; an output is ((c0 + c1) + c2) + c3 plus ((c4 + c5) + c6) + c7.
// Both kernels below do exactly that for every output, so its value does not depend on M, on the tile it falls in, on the
// kernel, or on what else is in the batch.  Classes are what lets a step of few tokens spread the inner axis over the
// warps of a block and a tile of outputs be worked by two halves of a block, without a second order of summation; chains
// of an eighth of the length also round less (1.5e-7 against 4e-7 relative at 1 024 .. 3 072 k).
//
// The kernels.
//   gemm_f32_few_kernel    few tokens: bound by the weight's bytes.  A block owns 8 or 16 output features and up to 32
//                          tokens; each of its eight warps runs one class through a cp.async ring of its own.
//                          A head of 151936 x 1024: 131 us with 1 token (4.7 TB/s), 184 us with 8; 1024 x 3072 with 8:
//                          14 us (some 7 of which are the measurement's).  A tile kernel of 64 x 64 with scalar loads and one
//                          chain over k, which it replaces, took 300 us for these products whatever the tokens.
//   gemm_f32_tile_kernel   many tokens: bound by the FMA rate (58 TFLOP/s is what FMAs from registers alone reach here).  Tiles
//                          of 64 x 64 outputs, 64 per thread.  2 048 tokens: 4096 x 1024 432 us (39.8 TFLOP/s), 1024 x 3072
//                          388 us (33.2).  Packed FMAs (fma.rn.f32x2) over even and odd k gave the same rate: twice the
//                          accumulators leave 32 outputs a thread and more shared-memory reads per FMA.
#include "common.cuh"

#define GF_SEG 128         // k per segment
#define GF_CLASSES 8

// 16 bytes of a row from element k on into shared memory, zeros behind the row's end (`rows_ok`: the row exists).  VEC: rows
// start on 16-byte borders; else element by element.
template <bool VEC>
__device__ __forceinline__ void copy_piece(float* dst, const float* row, int k, int K, bool row_ok) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if (VEC) {
        const bool in = row_ok && k < K;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(in ? row + k : row), "r"(in ? 16 : 0));
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const bool in = row_ok && k + e < K;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4 * e), "l"(in ? row + k + e : row), "r"(in ? 4 : 0));
        }
    }
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;"); }
template <int LEFT> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// ------------------------------------------------------------------------------------------------------ few tokens
#define GF_WARPS GF_CLASSES
#define GF_CHUNK 32                    // k per stage of a warp's ring
#define GF_ROW (GF_CHUNK + 4)          // a row of a stage in floats: eight rows' 16-byte reads meet in eight different places
template <int NG, int MT, int STAGES>
struct FewSmem {
    static constexpr int STAGE = (NG + MT) * GF_ROW;                          // floats of a warp's stage
    static constexpr int TABLE = GF_WARPS * MT * NG;                          // a feature group's class sums
    static constexpr int BYTES = (GF_WARPS * STAGES * STAGE + 2 * TABLE) * 4;
};

// Warp c runs class c of the block's features; behind a barrier, the thread that owns an output adds the eight chains (two
// tables in turn, so one barrier per feature group).  A warp's ring runs on across feature groups.
template <int NG, int MT, int STAGES, bool VEC>
__global__ void __launch_bounds__(GF_WARPS * 32) gemm_f32_few_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                     float* __restrict__ out, int M, int N, int K, int n_groups) {
    using S = FewSmem<NG, MT, STAGES>;
    constexpr int NI = NG / 8, MI = MT / 4;
    extern __shared__ __align__(16) float smem[];
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ln = lane & 7, lm = lane >> 3;                                  // features ln + 8 i, tokens lm + 4 j
    float* ring = smem + warp * STAGES * S::STAGE;
    float* tables = smem + GF_WARPS * STAGES * S::STAGE;
    const int m0 = blockIdx.y * MT, k_first = warp * GF_SEG;
    const int segs = (K + GF_SEG - 1) / GF_SEG, my_segs = warp < segs ? (segs - 1 - warp) / GF_CLASSES + 1 : 0;
    const int per_group = my_segs * (GF_SEG / GF_CHUNK);                      // chunks of this warp in a feature group
    const int total = per_group * ((n_groups - 1 - (int)blockIdx.x) / (int)gridDim.x + 1);
    int ask_group = blockIdx.x, ask_k = k_first, ask_c = 0;                   // the chunk that is asked for next
    auto step_ask = [&]() {
        ask_k += GF_CHUNK;
        if (ask_k % GF_SEG == 0) ask_k += (GF_CLASSES - 1) * GF_SEG;
        if (++ask_c == per_group) { ask_c = 0; ask_k = k_first; ask_group += gridDim.x; }
    };
    auto copy_w = [&](int slot) {
        float* dst = ring + slot * S::STAGE;
#pragma unroll
        for (int i = 0; i < NG / 4; ++i) {
            const int r = i * 4 + (lane >> 3), n = ask_group * NG + r, k = ask_k + (lane & 7) * 4;
            copy_piece<VEC>(dst + r * GF_ROW + (lane & 7) * 4, w + (size_t)min(n, N - 1) * K, k, K, n < N);
        }
    };
    auto copy_x = [&](int slot) {
        float* dst = ring + slot * S::STAGE + NG * GF_ROW;
#pragma unroll
        for (int i = 0; i < MT / 4; ++i) {
            const int r = i * 4 + (lane >> 3), m = m0 + r, k = ask_k + (lane & 7) * 4;
            copy_piece<VEC>(dst + r * GF_ROW + (lane & 7) * 4, x + (size_t)min(m, M - 1) * K, k, K, m < M);
        }
    };
    // the weight's first chunks are asked for before the kernel before has ended (no kernel writes a weight)
    for (int q = 0; q < STAGES - 1 && q < total; ++q) { copy_w(q); step_ask(); }
    pdl_wait();
    ask_group = blockIdx.x; ask_k = k_first; ask_c = 0;
    for (int q = 0; q < STAGES - 1; ++q) {
        if (q < total) { copy_x(q); step_ask(); }
        copies_commit();
    }
    int q = 0, slot = 0, turn = 0;
    for (int g = blockIdx.x; g < n_groups; g += gridDim.x, turn ^= 1) {
        float acc[NI][MI];
#pragma unroll
        for (int i = 0; i < NI; ++i)
#pragma unroll
            for (int j = 0; j < MI; ++j) acc[i][j] = 0.f;
        for (int c = 0; c < per_group; ++c, ++q) {
            copies_wait<STAGES - 2>();
            __syncwarp();
            if (q + STAGES - 1 < total) {
                const int to = slot == 0 ? STAGES - 1 : slot - 1;            // the stage that was read last
                copy_w(to); copy_x(to); step_ask();
            }
            copies_commit();
            const float* ws = ring + slot * S::STAGE + ln * GF_ROW;
            const float* xs = ring + slot * S::STAGE + (NG + lm) * GF_ROW;
            slot = slot == STAGES - 1 ? 0 : slot + 1;
#pragma unroll
            for (int k = 0; k < GF_CHUNK; k += 4) {
                float4 a[NI];
#pragma unroll
                for (int i = 0; i < NI; ++i) a[i] = *reinterpret_cast<const float4*>(ws + i * 8 * GF_ROW + k);
#pragma unroll
                for (int j = 0; j < MI; ++j) {
                    const float4 b = *reinterpret_cast<const float4*>(xs + j * 4 * GF_ROW + k);
#pragma unroll
                    for (int i = 0; i < NI; ++i) {
                        acc[i][j] = fmaf(b.x, a[i].x, acc[i][j]);
                        acc[i][j] = fmaf(b.y, a[i].y, acc[i][j]);
                        acc[i][j] = fmaf(b.z, a[i].z, acc[i][j]);
                        acc[i][j] = fmaf(b.w, a[i].w, acc[i][j]);
                    }
                }
            }
        }
        float* table = tables + turn * S::TABLE;
#pragma unroll
        for (int i = 0; i < NI; ++i)
#pragma unroll
            for (int j = 0; j < MI; ++j) table[(warp * MT + lm + 4 * j) * NG + ln + 8 * i] = acc[i][j];
        __syncthreads();
        for (int at = threadIdx.x; at < MT * NG; at += GF_WARPS * 32) {
            const int m = m0 + at / NG, n = g * NG + at % NG;
            const float* c = table + at;
            constexpr int D = MT * NG;
            const float low = ((c[0] + c[D]) + c[2 * D]) + c[3 * D], high = ((c[4 * D] + c[5 * D]) + c[6 * D]) + c[7 * D];
            if (m < M && n < N) out[(size_t)m * N + n] = low + high;
        }
    }
}

// ------------------------------------------------------------------------------------------------------ many tokens
#define GF_TILE 64
#define GF_BK 16
#define GF_BROW (GF_BK + 4)            // a row of a stage in floats (eight rows' 16-byte reads in eight different places)
#define GF_TSTAGES 2
#define GF_HALF 64                     // threads of a half of the block
#define GF_STAGE (2 * GF_TILE * GF_BROW)
#define GF_TILE_SMEM (2 * (GF_TSTAGES * GF_STAGE + 64 * GF_HALF) * 4)

// A block is two halves of two warps, a thread 8 x 8 outputs of the tile; half h runs classes 4 h .. 4 h + 3 through a ring of its
// own and adds them up in shared memory (64 more registers a thread would leave room for two blocks on an SM instead of
// three); the lower half's threads add the two halves' sums at the end.
template <bool VEC>
__global__ void __launch_bounds__(2 * GF_HALF, 3) gemm_f32_tile_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                       float* __restrict__ out, int M, int N, int K) {
    extern __shared__ __align__(16) float smem[];
    pdl_launch_dependents();
    pdl_wait();
    // a warp is 4 x 8 threads: four rows of x and eight of w per 16-byte read
    const int half = threadIdx.x / GF_HALF, ht = threadIdx.x % GF_HALF;
    const int tx = ht & 7, ty = ht >> 3;                                     // features tx + 8 j, tokens ty + 8 i
    const int m0 = blockIdx.y * GF_TILE, n0 = blockIdx.x * GF_TILE;
    float* ring = smem + half * GF_TSTAGES * GF_STAGE;
    float* sums = smem + 2 * GF_TSTAGES * GF_STAGE + half * 64 * GF_HALF + ht;   // [8 * 8][threads of a half]
    // a walk over this half's k: a class's segments, then the next class's
    struct Walk { int cls, k; };
    auto done = [&](const Walk& p) { return p.k >= K; };
    auto step = [&](Walk& p) {                                               // true behind a class's last piece
        p.k += GF_BK;
        if (p.k % GF_SEG == 0) p.k += (GF_CLASSES - 1) * GF_SEG;
        if (p.k < K) return false;
        ++p.cls;
        p.k = p.cls < 4 * half + 4 ? p.cls * GF_SEG : K;                     // (a class that starts behind K is empty, and so are those after it)
        return true;
    };
    // this thread's pieces of a stage: 16 bytes at column lk of rows lr, lr + 16, ... of the tile's x and w
    const int lr = ht >> 2, lk = (ht & 3) * 4;
    const float* px = x + (size_t)(m0 + lr) * K + lk;                        // (rows behind the end are not read: zeros go there)
    const float* pw = w + (size_t)(n0 + lr) * K + lk;
    const size_t step16 = (size_t)16 * K;
    auto copy_stage = [&](int slot, int k0) {
        float* dst = ring + slot * GF_STAGE + lr * GF_BROW + lk;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            copy_piece<VEC>(dst + i * 16 * GF_BROW, px + i * step16, k0, K - lk, m0 + lr + i * 16 < M);
            copy_piece<VEC>(dst + (GF_TILE + i * 16) * GF_BROW, pw + i * step16, k0, K - lk, n0 + lr + i * 16 < N);
        }
    };
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) { acc[i][j] = 0.f; sums[(i * 8 + j) * GF_HALF] = 0.f; }
    Walk ask{4 * half, 4 * half * GF_SEG}, at = ask;
    for (int s = 0; s < GF_TSTAGES - 1; ++s) {
        if (!done(ask)) { copy_stage(s, ask.k); step(ask); }
        copies_commit();
    }
    int slot = 0;
    while (!done(at)) {
        copies_wait<GF_TSTAGES - 2>();
        asm volatile("bar.sync %0, %1;" ::"r"(1 + half), "n"(GF_HALF) : "memory");
        if (!done(ask)) { copy_stage(slot == 0 ? GF_TSTAGES - 1 : slot - 1, ask.k); step(ask); }
        copies_commit();
        const float* xs = ring + slot * GF_STAGE + ty * GF_BROW;
        const float* ws = ring + slot * GF_STAGE + (GF_TILE + tx) * GF_BROW;
        slot = slot == GF_TSTAGES - 1 ? 0 : slot + 1;
#pragma unroll
        for (int k = 0; k < GF_BK; k += 4) {
            float4 a[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(xs + i * 8 * GF_BROW + k);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 b = *reinterpret_cast<const float4*>(ws + j * 8 * GF_BROW + k);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
            }
        }
        if (step(at)) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) { sums[(i * 8 + j) * GF_HALF] += acc[i][j]; acc[i][j] = 0.f; }
        }
    }
    __syncthreads();
    if (half == 1) return;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + ty + i * 8;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int n = n0 + tx + j * 8;
            if (n < N) out[(size_t)m * N + n] = sums[(i * 8 + j) * GF_HALF] + sums[(64 + i * 8 + j) * GF_HALF];
        }
    }
}

// ------------------------------------------------------------------------------------------------------ launches
// opt in to more than 48 KB of shared memory, once per kernel and device
template <typename F>
static int allow_smem(F kernel, int bytes, const char* what) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    IDM_REQUIRE(e == cudaSuccess, "%s: %d bytes of shared memory: %s", what, bytes, cudaGetErrorString(e));
    return 0;
}

template <int NG, int MT, int STAGES>
static int few_launch(const float* x, const float* w, float* out, int M, int N, int K, bool vec, int sms, cudaStream_t stream) {
    constexpr int BYTES = FewSmem<NG, MT, STAGES>::BYTES;
    auto kernel = vec ? gemm_f32_few_kernel<NG, MT, STAGES, true> : gemm_f32_few_kernel<NG, MT, STAGES, false>;
    if (int rc = allow_smem(kernel, BYTES, "gemm_f32")) return rc;
    const int n_groups = (N + NG - 1) / NG, per_sm = 227 * 1024 / (BYTES + 1024);
    idm_launch(kernel, dim3(min(n_groups, sms * per_sm), (M + MT - 1) / MT), dim3(GF_WARPS * 32), BYTES, stream, x, w, out, M, N,
               K, n_groups);
    return 0;
}

static int tile_launch(const float* x, const float* w, float* out, int M, int N, int K, bool vec, cudaStream_t stream) {
    auto kernel = vec ? gemm_f32_tile_kernel<true> : gemm_f32_tile_kernel<false>;
    if (int rc = allow_smem(kernel, GF_TILE_SMEM, "gemm_f32")) return rc;
    const dim3 grid((N + GF_TILE - 1) / GF_TILE, (M + GF_TILE - 1) / GF_TILE);
    IDM_REQUIRE(grid.y <= 65535, "gemm_f32: M=%d is too large for one launch", M);
    idm_launch(kernel, grid, dim3(2 * GF_HALF), GF_TILE_SMEM, stream, x, w, out, M, N, K);
    return 0;
}

// Which kernel: the same bits either way, so only time decides.  Measured (us, inputs out of the L2, few / tile), N x K: 1024 x 2048 with
// 613 tokens (160 tiles of 64 x 64) 114 / 140, with 1 024 (256 tiles) 185 / 143; 4096 x 1024 with 128 (128) 51 / 52, with
// 256 (256) 96 / 78; 6144 x 1024 with 128 (192) 75 / 80, with 256 (384) 138 / 101; a head of 151936 x 1024 with 32 tokens
// 412 / 506, with 64 807 / 521: from 200 tiles on the tiles fill the SMs, unless the step has so few tokens that half of
// every tile is padding.
#define GF_TILES_FROM 200
#define GF_FEW_UP_TO 32

extern "C" int idm_gemm_f32(const float* x, const float* w, float* out, int M, int N, int K, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    IDM_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    const bool vec = K % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
    int rc, dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
    const long long tiles = (long long)((M + GF_TILE - 1) / GF_TILE) * ((N + GF_TILE - 1) / GF_TILE);
    if (M > GF_FEW_UP_TO && tiles >= GF_TILES_FROM) {
        rc = tile_launch(x, w, out, M, N, K, vec, stream);
    } else if (N >= 16 * sms || M > 16) {
        // 16 features a block where that still gives every SM one (or a tile of 32 tokens has work enough for a block)
        rc = M <= 4 ? few_launch<16, 4, 4>(x, w, out, M, N, K, vec, sms, stream)
           : M <= 8 ? few_launch<16, 8, 3>(x, w, out, M, N, K, vec, sms, stream)
           : M <= 16 ? few_launch<16, 16, 3>(x, w, out, M, N, K, vec, sms, stream)
                     : few_launch<16, 32, 3>(x, w, out, M, N, K, vec, sms, stream);
    } else {
        rc = M <= 4 ? few_launch<8, 4, 6>(x, w, out, M, N, K, vec, sms, stream)
           : M <= 8 ? few_launch<8, 8, 6>(x, w, out, M, N, K, vec, sms, stream)
                    : few_launch<8, 16, 4>(x, w, out, M, N, K, vec, sms, stream);
    }
    if (rc) return rc;
    IDM_LAUNCH_CHECK("gemm_f32");
    return 0;
}
