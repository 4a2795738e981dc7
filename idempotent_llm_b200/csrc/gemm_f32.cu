// out[M, N] = x[M, K] . w[N, K]^T of 32-bit numbers to 32-bit precision, on the tensor cores.
// (The reference's exact path is the CPU integer matmul of src/detllm/backends.py:95-96; this is its float counterpart.)
//
// A 32-bit number is three bfloat16 parts, v = v1 + v2 + v3, to its last bit: v1 is v rounded to eight bits, v2 what that left out,
// v3 what both left out.  x . w is then the sum of nine products of parts; the three smallest (x2 w3, x3 w2, x3 w3) are below 2^-24
// of the largest and left out.  Products of bfloat16 numbers are exact in 32-bit, so what rounds is the adding, and that is kept
// short: a segment of 64 k is summed by the MMAs (x1 w1 in one accumulator, x2 w1 + x1 w2 in a second, x3 w1 + x2 w2 + x1 w3 in a
// third), and the segments are added up one after another by ordinary 32-bit adds.  Error against 64 bits, root mean square
// relative to the two rows' norms, at 64 / 128 / 1 024 / 3 072 / 8 192 k (one chain of 32-bit FMAs over k in brackets): normal
// numbers 0.9e-8 / 0.7e-8 / 0.3e-8 / 0.3e-8 / 0.2e-8 (1.8e-8 at all); all positive 0.6e-7 / 0.6e-7 / 0.6e-7 / 0.8e-7 / 1.2e-7
// (0.8e-7 / 1.1e-7 / 3.2e-7 / 4.7e-7 / 8.9e-7); magnitudes spread over e^(3 z) 1.5e-8 / 1.1e-8 / 0.4e-8 / 0.3e-8 / 0.2e-8
// (1.6e-8 / 1.5e-8 / 1.1e-8 / 0.9e-8 / 0.7e-8).  An output that is not finite is made again of plain FMAs (plain_sum): infinities
// and numbers at the very end of the range have no parts.
//
// One order of summation: an output's bits do not depend on M, on the tile it falls in, on how its segments were dealt out, or on
// what else is in the batch.
//
// A block has 128 features (the MMA's lanes) and 16, 32 or 64 tokens (its columns).  Sixteen warps read both operands from memory,
// a row's 256 bytes side by side, two segments ahead in registers, and lay the parts down in the swizzled rows that the MMA reads;
// the token parts lie one after another, so that w1 meets x1, x2 and x3 in one MMA, w2 meets x1 and x2 in one (shared memory is
// read twelve times a segment instead of 24).  One thread issues the MMAs; eight warps add the segments up from tensor memory, two
// of them in turn.  Where tiles are few, the blocks of a cluster deal a tile's segments out among them and send the sums to the
// block that adds up the feature's segments in order.  What bounds it is splitting and fetching, not the MMAs: 1.15 us a segment
// with 64 tokens, 0.95 with 16 or 32 (more than two stages leave the L1 too little room for the loads in flight: three take 1.3).
//   700 tokens: 4096 x 1024 64 us (92 TFLOP/s), 1024 x 3072 61 us (72); plain FMAs in tiles of 64 x 64 took 164 and 182.
//   8 tokens: 1024 x 3072 18 us, some 7 of which are the measurement's; a head of 151936 x 1024 145 us (4.3 TB/s).
// (A number that is split keeps its bits unless its third part leaves the exponent's range, below 2^-109 or so.)
#include "common.cuh"
#include "tcgen05.cuh"

#define GX_FEATURES 128                // features of a tile (the MMA's M axis)
#define GX_SEG 64                      // k per segment and stage: 64 bfloat16 = one swizzled row of 128 bytes
#define GX_ADD 256                     // threads that add segments up (a warp: a quarter of the features, half of the tokens),
#define GX_CONV 512                    // that split operands,
#define GX_THREADS (GX_ADD + GX_CONV + 32)   // and the warp that issues MMAs
#define GX_WARP_MMA ((GX_ADD + GX_CONV) / 32)
#define GX_SMEM (226 * 1024)           // dynamic shared memory that a block may ask for (a few bytes of its own beside it)

__device__ int g_gemm_f32_error = 0;

__device__ __forceinline__ void tc_ld8_issue(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}

template <int TN> struct SplitTile {                                           // 128 features, TN tokens
    static constexpr int A = GX_FEATURES * 128, B = TN * 128;                  // bytes of one part of a stage
    static constexpr int STAGE = 3 * (A + B);
    static constexpr int ROUNDS = 4 + (TN + 31) / 32;                   // rows of a thread that splits: features, then tokens
    static constexpr int COLS = TN == 64 ? 512 : 8 * TN;                       // tensor memory: three sums a segment, two segments in turn
};

// two numbers side by side: v - u
__device__ __forceinline__ float2 minus2(float2 v, float ux, float uy) {
    unsigned long long a, b, d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(ux), "f"(uy));
    asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(v.x), "f"(v.y));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(0xbf800000bf800000ull), "l"(b));       // u * -1 + v
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(d));
    return v;
}
// four numbers in three bfloat16 parts each, v = p1 + p2 + p3 (to the last bit unless p3 leaves the exponent's range)
__device__ __forceinline__ void split_four(float4 f, uint2 (&part)[3]) {
    float2 lo = make_float2(f.x, f.y), hi = make_float2(f.z, f.w);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const __nv_bfloat162 l = __floats2bfloat162_rn(lo.x, lo.y), h = __floats2bfloat162_rn(hi.x, hi.y);
        const uint32_t a = *reinterpret_cast<const uint32_t*>(&l), b = *reinterpret_cast<const uint32_t*>(&h);
        part[p] = make_uint2(a, b);
        if (p < 2) {
            lo = minus2(lo, __uint_as_float(a << 16), __uint_as_float(a & 0xffff0000u));
            hi = minus2(hi, __uint_as_float(b << 16), __uint_as_float(b & 0xffff0000u));
        }
    }
}

// An output that is not finite: infinities and numbers at the very end of the range have no parts (inf - inf), so its sum is made
// of plain FMAs, which stay not finite where the product is.
__device__ __noinline__ float plain_sum(const float* __restrict__ x, const float* __restrict__ w, int K) {
    float s = 0.f;
    for (int k = 0; k < K && !isnan(s); ++k) s = fmaf(x[k], w[k], s);
    return s;
}

// A block of a cluster whose wait has run out tells the others before they meet: none of them may add up sums that were not sent.
// (The thread whose wait it was sees its own flag.)
__device__ __forceinline__ void tell_cluster(int* abort_mem, int blocks) {
    if (*(volatile int*)abort_mem == 0) return;
    for (int r = 0; r < blocks; ++r) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(mapa_u32(smem_u32(abort_mem), r)), "r"(1) : "memory");
}

template <int TN, int ROWS>
__global__ void __launch_bounds__(GX_THREADS, 1) gemm_f32_split_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                       float* __restrict__ out, int M, int N, int K, int token_tiles, int tiles) {
    using S = SplitTile<TN>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) unsigned long long bars_mem[8];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_mem;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, bars = smem_u32(bars_mem);
    uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
    float* recv = reinterpret_cast<float*>(gen + 2 * S::STAGE);             // [segment][this block's features][TN]
    auto full = [&](int b) { return bars + 8u * b; };
    auto empty = [&](int b) { return bars + 8u * (2 + b); };
    auto acc_full = [&](int b) { return bars + 8u * (4 + b); };
    auto acc_empty = [&](int b) { return bars + 8u * (6 + b); };
    volatile int* abort_flag = &abort_mem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split = gridDim.z, rank = blockIdx.z;                            // blocks of a cluster deal a tile's segments out in turn
    const int segs = (K + GX_SEG - 1) / GX_SEG;
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; ++b) {
            mbar_init(full(b), GX_CONV / 32); mbar_init(empty(b), 1);
            mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), GX_ADD / 32);
        }
        abort_mem = 0;
        mbar_init_fence();
    }
    if (warp == GX_WARP_MMA) tmem_alloc(smem_u32(&tmem_slot), S::COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();               // (behind the allocation: a block of the next kernel cannot hold what this one waits for)
    if (split > 1) cluster_sync_all();     // every block of the cluster is there before one writes to another

    if (warp >= GX_ADD / 32 && warp < GX_WARP_MMA) {
        // ------------------------------------------------------------ operands: 32-bit from memory, three parts into the stage
        // a thread has four k of rows row, row + 32, ...: sixteen threads read a row's 256 bytes side by side
        const int ct = threadIdx.x - GX_ADD, row = ct >> 4, piece = ct & 15;
        float4 raw[2][S::ROUNDS];
        // rows behind the end are the last one again: their outputs are dropped
        struct Where { int tile, seg; const float *w, *x; int dw[3], dx; };     // (dw, dx: rows from there to this thread's others)
        auto place = [&](Where& p, int tile) {
            p.tile = tile; p.seg = rank;
            const int f = tile / token_tiles * GX_FEATURES + row, m = tile % token_tiles * TN + row, k = rank * GX_SEG + piece * 4;
            p.w = w + (size_t)min(f, N - 1) * K + k;
            p.x = x + (size_t)min(m, M - 1) * K + k;
#pragma unroll
            for (int i = 0; i < 3; ++i) p.dw[i] = min(f + 32 * (i + 1), N - 1) - min(f, N - 1);
            p.dx = min(m + 32, M - 1) - min(m, M - 1);
        };
        auto step = [&](Where& p) {                                            // false behind the block's last segment
            p.seg += split;
            if (p.seg < segs) { p.w += split * GX_SEG; p.x += split * GX_SEG; return true; }
            if (p.tile + (int)gridDim.x >= tiles) return false;
            place(p, p.tile + gridDim.x);
            return true;
        };
        auto load4k = [&](const float* p, int seg) {
            const int left = K - seg * GX_SEG - piece * 4;                     // elements of the row from here on
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (ROWS == 2) return __ldcg(reinterpret_cast<const float4*>(p));  // (K in whole segments)
            if (ROWS == 1) {
                if (left > 0) v = __ldcg(reinterpret_cast<const float4*>(p));
            } else {
                if (left > 0) v.x = p[0];
                if (left > 1) v.y = p[1];
                if (left > 2) v.z = p[2];
                if (left > 3) v.w = p[3];
            }
            return v;
        };
        auto load_w = [&](float4 (&v)[S::ROUNDS], const Where& p) {
            v[0] = load4k(p.w, p.seg);
#pragma unroll
            for (int i = 0; i < 3; ++i) v[i + 1] = load4k(p.w + (long long)p.dw[i] * K, p.seg);
        };
        auto load_x = [&](float4 (&v)[S::ROUNDS], const Where& p) {
            if (TN >= 32 || row < TN) v[4] = load4k(p.x, p.seg);
            if (TN > 32) v[S::ROUNDS - 1] = load4k(p.x + (long long)p.dx * K, p.seg);
        };
        if (blockIdx.x < tiles && rank < segs) {
            Where at;
            // the weight's first pieces are asked for before the kernel before has ended (no kernel writes a weight)
            place(at, blockIdx.x);
            load_w(raw[0], at);
            if (step(at)) load_w(raw[1], at);
            pdl_wait();
            place(at, blockIdx.x);
            int have = 1;                                                      // segments asked for
            load_x(raw[0], at);
            bool more = step(at);
            if (more) { load_x(raw[1], at); more = step(at); have = 2; }
            const uint32_t off = (uint32_t)(row * 128 + (((piece >> 1) ^ (row & 7)) << 4) + (piece & 1) * 8);   // (row + 32 i: the same place in its swizzle atom)
            for (int turn = 0; have > 0; turn ^= 1) {
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    if (have == 0) break;
                    if (!mbar_wait(empty(b), turn ^ 1, abort_flag, &g_gemm_f32_error)) { have = 0; break; }
                    uint8_t* stage = gen + b * S::STAGE + off;
#pragma unroll
                    for (int i = 0; i < S::ROUNDS; ++i) {
                        if (i >= 4 && TN < 32 && row >= TN) break;
                        uint2 part[3];
                        split_four(raw[b][i], part);
#pragma unroll
                        for (int p = 0; p < 3; ++p)
                            *reinterpret_cast<uint2*>(stage + (i < 4 ? p * S::A + i * 4096 : 3 * S::A + p * S::B + (i - 4) * 4096)) = part[p];
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full(b));                       // (one arrival a warp: they queue up at the barrier)
                    if (more) {
                        load_w(raw[b], at); load_x(raw[b], at);
                        more = step(at);
                    } else --have;
                }
            }
        }
    } else if (warp == GX_WARP_MMA) {
        // ------------------------------------------------------------ MMAs: products of parts, by size into three sums
        if (lane == 0) {
            const uint32_t three = umma_idesc(GX_FEATURES, 3 * TN), two = umma_idesc(GX_FEATURES, 2 * TN), one = umma_idesc(GX_FEATURES, TN);
            int it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x)
                for (int seg = rank; ok && seg < segs; seg += split, ++it) {
                    const int b = it & 1, turn = (it >> 1) & 1;
                    const uint32_t d = tmem + b * 3 * TN;
                    ok = mbar_wait(acc_empty(b), turn ^ 1, abort_flag, &g_gemm_f32_error) &&
                         mbar_wait(full(b), turn, abort_flag, &g_gemm_f32_error);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t a = base + b * S::STAGE;
                    const uint64_t a1 = umma_desc_kmajor(a), a2 = umma_desc_kmajor(a + S::A), a3 = umma_desc_kmajor(a + 2 * S::A);
                    const uint64_t t = umma_desc_kmajor(a + 3 * S::A);         // the token parts' rows one after another
                    tc_mma_bf16_kblock(d, a1, t, three, 0);                    // w1 x1 | w1 x2 | w1 x3
                    tc_mma_bf16_kblock(d + TN, a2, t, two, 1);                 //       + w2 x1 | w2 x2
                    tc_mma_bf16_kblock(d + 2 * TN, a3, t, one, 1);             //               + w3 x1
                    tc_commit(empty(b));
                    tc_commit(acc_full(b));
                }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ segments, one after another
        constexpr int COLS = TN / 2;
        float tot[COLS];
        int it = 0;
        bool ok = true;
        const int per = (GX_FEATURES + split - 1) / split, mine = (warp & 3) * 32 + lane, owner = mine / per, spot = mine % per, c0 = (warp >> 2) * COLS;
        pdl_wait();                        // (the kernel before may still read what is written here)
        for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
#pragma unroll
            for (int j = 0; j < COLS; ++j) tot[j] = 0.f;
            for (int seg = rank; seg < segs; seg += split, ++it) {
                ok = mbar_wait(acc_full(it & 1), (it >> 1) & 1, abort_flag, &g_gemm_f32_error);
                if (!ok) break;
                tc_fence_after();
                const uint32_t big = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (it & 1) * 3 * TN + c0;
#pragma unroll
                for (int c = 0; c < COLS; c += 8) {
                    uint32_t u[8], v[8], z[8];
                    tc_ld8_issue(big + c, u); tc_ld8_issue(big + TN + c, v); tc_ld8_issue(big + 2 * TN + c, z);
                    tc_ld_wait();
                    float sum[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) sum[j] = __uint_as_float(u[j]) + (__uint_as_float(v[j]) + __uint_as_float(z[j]));
                    if (split == 1) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) tot[c + j] += sum[j];
                    } else {
                        const uint32_t to = mapa_u32(smem_u32(recv + ((size_t)seg * per + spot) * TN + c0 + c), owner);
#pragma unroll
                        for (int j = 0; j < 8; j += 4)
                            asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to + 4 * j), "f"(sum[j]), "f"(sum[j + 1]), "f"(sum[j + 2]), "f"(sum[j + 3]) : "memory");
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty(it & 1));
            }
            if (split == 1 && ok) {
                const int f = tile / token_tiles * GX_FEATURES + mine, m0 = tile % token_tiles * TN + c0;
                if (f < N)
#pragma unroll
                    for (int j = 0; j < COLS; ++j)
                        if (m0 + j < M) {
                            float s = tot[j];
                            if (!isfinite(s)) s = plain_sum(x + (size_t)(m0 + j) * K, w + (size_t)f * K, K);
                            out[(size_t)(m0 + j) * N + f] = s;
                        }
            }
        }
    }
    __syncwarp();
    if (split > 1) {
        pdl_wait();
        tell_cluster(&abort_mem, split);
        cluster_sync_all();                // all segments' sums are here
        const int per = (GX_FEATURES + split - 1) / split, tile = blockIdx.x;
        const int f0 = tile / token_tiles * GX_FEATURES + rank * per, m0 = tile % token_tiles * TN, have = min(per, GX_FEATURES - rank * per);
        if (abort_mem == 0)
            for (int at = threadIdx.x; at < have * TN; at += GX_THREADS) {
                const int spot = at % have, f = f0 + spot, m = m0 + at / have;
                if (f >= N || m >= M) continue;
                float s = 0.f;
#pragma unroll 8
                for (int seg = 0; seg < segs; ++seg) s += recv[((size_t)seg * per + spot) * TN + at / have];
                if (!isfinite(s)) s = plain_sum(x + (size_t)m * K, w + (size_t)f * K, K);
                out[(size_t)m * N + f] = s;
            }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == GX_WARP_MMA) tmem_dealloc(tmem, S::COLS);
    if (abort_mem != 0) {                  // a wait ran out: none of the block's outputs passes for a number
        const int per = (GX_FEATURES + split - 1) / split, have = min(per, GX_FEATURES - rank * per);
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
            for (int at = threadIdx.x; at < have * TN; at += GX_THREADS) {
                const int f = tile / token_tiles * GX_FEATURES + rank * per + at % have, m = tile % token_tiles * TN + at / have;
                if (f < N && m < M) out[(size_t)m * N + f] = __int_as_float(0x7fffffff);
            }
    }
}

// ------------------------------------------------------------------------------------------------------ many tokens
// The same sums where there are tokens enough: the tokens' parts are made once, by a kernel in front, for all the feature tiles that meet them,
// and come as tiles by TMA; a block has 128 features and SUBS times 64 tokens, so that a split weight meets all of them.  A segment's
// 64 tokens are an accumulator's, as above: with SUBS of 2 the two take turns in tensor memory, with 1 neighbouring segments do.
// Eight warps split the weight, eight add up 64 tokens, one thread issues the MMAs and one the copies.
// Bound by shared memory: a segment's 128 tokens move 192 KB into the MMAs, 48 in from the weight's split and 48 from the copies, 1.2 of
// the 1.4 us it takes (64 tokens: 0.95 us, of which some 0.7).  700 tokens, with the kernel
// in front and inputs out of the L2: 4096 x 1024 58 us (split by every tile 68), 6144 x 1024 60 (86), 1024 x 3072 58 (64); 1 400 tokens: 83 (107),
// 108 (162), 85 (118).
#define GW_CONV 256
template <int SUBS> struct WideTile {
    static constexpr int ADD = SUBS * GX_ADD, THREADS = ADD + GW_CONV + 64, WARP_MMA = (ADD + GW_CONV) / 32;
    static constexpr int AHEAD = SUBS == 1 ? 2 : 1;                            // segments of the weight on their way in registers
    static constexpr int A = GX_FEATURES * 128, PART = 64 * 128, B = 3 * PART;     // bytes: one part of the weight, of 64 tokens; 64 tokens' parts
    static constexpr int STAGE = 3 * A + SUBS * B;
};

// parts [3][M][Kp] of x [M][K], zeros from K to Kp (a multiple of 64)
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ parts, int M, int K, int Kp, int vec) {
    pdl_launch_dependents();
    pdl_wait();
    const int quads = Kp / 4;
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= (long long)M * quads) return;
    const int m = (int)(i / quads), k = (int)(i - (long long)m * quads) * 4;
    const float* p = x + (size_t)m * K + k;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec) {
        if (k < K) v = *reinterpret_cast<const float4*>(p);
    } else {
        if (k < K) v.x = p[0];
        if (k + 1 < K) v.y = p[1];
        if (k + 2 < K) v.z = p[2];
        if (k + 3 < K) v.w = p[3];
    }
    uint2 part[3];
    split_four(v, part);
#pragma unroll
    for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(parts + ((size_t)j * M + m) * Kp + k) = part[j];
}

template <int SUBS, int ROWS>
__global__ void __launch_bounds__(WideTile<SUBS>::THREADS, 1) gemm_f32_wide_kernel(const __grid_constant__ CUtensorMap map_x, const float* __restrict__ x,
                                                                      const float* __restrict__ w, float* __restrict__ out, int M, int N, int K,
                                                                      int token_tiles, int tiles) {
    using S = WideTile<SUBS>;
    constexpr int TN = 64;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) unsigned long long bars_mem[8];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_mem;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, bars = smem_u32(bars_mem);
    uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
    auto full = [&](int b) { return bars + 8u * b; };
    auto empty = [&](int b) { return bars + 8u * (2 + b); };
    auto acc_full = [&](int b) { return bars + 8u * (4 + b); };
    auto acc_empty = [&](int b) { return bars + 8u * (6 + b); };
    volatile int* abort_flag = &abort_mem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, segs = (K + GX_SEG - 1) / GX_SEG;
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; ++b) {
            mbar_init(full(b), GW_CONV / 32 + 1); mbar_init(empty(b), 1);
            mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), GX_ADD / 32);
        }
        abort_mem = 0;
        mbar_init_fence();
    }
    if (warp == S::WARP_MMA) tmem_alloc(smem_u32(&tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();               // (behind the allocation: a block of the next kernel cannot hold what this one waits for)
    // the n-th segment of a block (over all its tiles) is in stage n & 1; its tokens' sums in accumulator (SUBS == 2 ? which 64 of them : n & 1)
    auto acc_of = [&](int n, int sub) { return SUBS == 2 ? sub : n & 1; };
    auto acc_turn = [&](int n) { return (SUBS == 2 ? n : n >> 1) & 1; };

    if (warp >= S::ADD / 32 && warp < S::WARP_MMA) {
        // ------------------------------------------------------------ the weight: 32-bit from memory, three parts into the stage
        // a thread has four k of rows row, row + 16, ...: sixteen threads read a row's 256 bytes side by side
        constexpr int ROUNDS = GX_FEATURES / 16;
        const int ct = threadIdx.x - S::ADD, row = ct >> 4, piece = ct & 15;
        float4 raw[S::AHEAD][ROUNDS];
        auto load = [&](float4 (&v)[ROUNDS], int tile, int seg) {              // (rows behind the end are the last one again: their outputs are dropped)
            const int f = tile / token_tiles * GX_FEATURES + row, k = seg * GX_SEG + piece * 4, left = K - k;
#pragma unroll
            for (int i = 0; i < ROUNDS; ++i) {
                const float* p = w + (size_t)min(f + 16 * i, N - 1) * K + k;
                if (ROWS == 2) v[i] = __ldcg(reinterpret_cast<const float4*>(p));
                else if (ROWS == 1) v[i] = left > 0 ? __ldcg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
                else v[i] = make_float4(left > 0 ? p[0] : 0.f, left > 1 ? p[1] : 0.f, left > 2 ? p[2] : 0.f, left > 3 ? p[3] : 0.f);
            }
        };
        int tile = blockIdx.x, seg = 0, have = 0;                              // the next segment to ask for, and how many have been
        auto ask = [&](float4 (&v)[ROUNDS]) {
            if (tile >= tiles) return;
            load(v, tile, seg);
            ++have;
            if (++seg == segs) { seg = 0; tile += gridDim.x; }
        };
        ask(raw[0]);                       // (no kernel writes a weight: nothing to wait for)
        if (S::AHEAD == 2) ask(raw[S::AHEAD - 1]);
        const uint32_t off = (uint32_t)(row * 128 + (((piece >> 1) ^ (row & 7)) << 4) + (piece & 1) * 8);   // (row + 16 i: the same place in its swizzle atom)
        for (int turn = 0; have > 0; turn ^= 1) {
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                if (have == 0) break;
                if (!mbar_wait(empty(b), turn ^ 1, abort_flag, &g_gemm_f32_error)) { have = 0; break; }
                uint8_t* stage = gen + b * S::STAGE + off;
#pragma unroll
                for (int i = 0; i < ROUNDS; ++i) {
                    uint2 part[3];
                    split_four(raw[b % S::AHEAD][i], part);
#pragma unroll
                    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(stage + p * S::A + i * 2048) = part[p];
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(full(b));
                --have;
                ask(raw[b % S::AHEAD]);
            }
        }
    } else if (warp == S::WARP_MMA + 1) {
        // ------------------------------------------------------------ the tokens' parts, by TMA
        pdl_wait();
        if (lane == 0) {
            int n = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x)
                for (int seg = 0; ok && seg < segs; ++seg, ++n) {
                    const int b = n & 1;
                    ok = mbar_wait(empty(b), ((n >> 1) & 1) ^ 1, abort_flag, &g_gemm_f32_error);
                    if (!ok) break;
                    mbar_expect_tx(full(b), SUBS * S::B);
#pragma unroll
                    for (int i = 0; i < 3 * SUBS; ++i)
                        tma_load_3d(base + b * S::STAGE + 3 * S::A + i * S::PART, &map_x, seg * GX_SEG,
                                    tile % token_tiles * (TN * SUBS) + i / 3 * TN, i % 3, full(b));
                }
        }
        __syncwarp();
    } else if (warp == S::WARP_MMA) {
        // ------------------------------------------------------------ MMAs: products of parts, by size into three sums
        if (lane == 0) {
            const uint32_t three = umma_idesc(GX_FEATURES, 3 * TN), two = umma_idesc(GX_FEATURES, 2 * TN), one = umma_idesc(GX_FEATURES, TN);
            int n = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x)
                for (int seg = 0; ok && seg < segs; ++seg, ++n) {
                    const int b = n & 1;
                    ok = mbar_wait(full(b), (n >> 1) & 1, abort_flag, &g_gemm_f32_error);
                    const uint32_t a = base + b * S::STAGE;
                    const uint64_t a1 = umma_desc_kmajor(a), a2 = umma_desc_kmajor(a + S::A), a3 = umma_desc_kmajor(a + 2 * S::A);
                    for (int sub = 0; ok && sub < SUBS; ++sub) {
                        const int acc = acc_of(n, sub);
                        ok = mbar_wait(acc_empty(acc), acc_turn(n) ^ 1, abort_flag, &g_gemm_f32_error);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t d = tmem + acc * 3 * TN;
                        const uint64_t t = umma_desc_kmajor(a + 3 * S::A + sub * S::B);   // the token parts' rows one after another
                        tc_mma_bf16_kblock(d, a1, t, three, 0);                // w1 x1 | w1 x2 | w1 x3
                        tc_mma_bf16_kblock(d + TN, a2, t, two, 1);             //       + w2 x1 | w2 x2
                        tc_mma_bf16_kblock(d + 2 * TN, a3, t, one, 1);         //               + w3 x1
                        if (sub == SUBS - 1) tc_commit(empty(b));
                        tc_commit(acc_full(acc));
                    }
                }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ segments, one after another
        // (with SUBS of 2 eight warps for each 64 tokens)
        constexpr int COLS = TN / 2;
        float tot[COLS];
        int n = 0;
        bool ok = true;
        const int sub = warp >> 3, mine = (warp & 3) * 32 + lane, c0 = (warp >> 2 & 1) * COLS;
        pdl_wait();                        // (the kernel before may still read what is written here)
        for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
#pragma unroll
            for (int j = 0; j < COLS; ++j) tot[j] = 0.f;
            for (int seg = 0; seg < segs; ++seg, ++n) {
                const int acc = acc_of(n, sub);
                ok = mbar_wait(acc_full(acc), acc_turn(n), abort_flag, &g_gemm_f32_error);
                if (!ok) break;
                tc_fence_after();
                const uint32_t big = tmem + ((uint32_t)((warp & 3) * 32) << 16) + acc * 3 * TN + c0;
#pragma unroll
                for (int c = 0; c < COLS; c += 8) {
                    uint32_t u[8], v[8], z[8];
                    tc_ld8_issue(big + c, u); tc_ld8_issue(big + TN + c, v); tc_ld8_issue(big + 2 * TN + c, z);
                    tc_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; ++j) tot[c + j] += __uint_as_float(u[j]) + (__uint_as_float(v[j]) + __uint_as_float(z[j]));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty(acc));
            }
            const int f = tile / token_tiles * GX_FEATURES + mine, m0 = tile % token_tiles * (TN * SUBS) + sub * TN + c0;
            if (ok && f < N)
#pragma unroll
                for (int j = 0; j < COLS; ++j)
                    if (m0 + j < M) {
                        float s = tot[j];
                        if (!isfinite(s)) s = plain_sum(x + (size_t)(m0 + j) * K, w + (size_t)f * K, K);
                        out[(size_t)(m0 + j) * N + f] = s;
                    }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == S::WARP_MMA) tmem_dealloc(tmem, 512);
    if (abort_mem != 0)                    // a wait ran out: none of the block's outputs passes for a number
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
            for (int at = threadIdx.x; at < GX_FEATURES * TN * SUBS; at += S::THREADS) {
                const int f = tile / token_tiles * GX_FEATURES + at % GX_FEATURES, m = tile % token_tiles * (TN * SUBS) + at / GX_FEATURES;
                if (f < N && m < M) out[(size_t)m * N + f] = __int_as_float(0x7fffffff);
            }
}

// ------------------------------------------------------------------------------------------------------ launches
template <int TN> static long long split_smem(int K, int split) {
    const long long segs = (K + GX_SEG - 1) / GX_SEG, per = (GX_FEATURES + split - 1) / split;
    return 1024 + 2 * SplitTile<TN>::STAGE + (split > 1 ? segs * per * TN * 4 : 0);
}

template <int TN>
static int split_launch(const float* x, const float* w, float* out, int M, int N, int K, int rows, int split, int sms, cudaStream_t stream) {
    const int bytes = (int)split_smem<TN>(K, split);
    auto kernel = rows == 0 ? gemm_f32_split_kernel<TN, 0> : rows == 1 ? gemm_f32_split_kernel<TN, 1> : gemm_f32_split_kernel<TN, 2>;
    // (the same limit from every call: a smaller one from another thread would have this launch refused)
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GX_SMEM);
    IDM_REQUIRE(e == cudaSuccess, "gemm_f32: %d bytes of shared memory: %s", GX_SMEM, cudaGetErrorString(e));
    const int token_tiles = (M + TN - 1) / TN;
    const long long tiles = (long long)token_tiles * ((N + GX_FEATURES - 1) / GX_FEATURES);
    IDM_REQUIRE(tiles < (1ll << 30), "gemm_f32: M=%d N=%d are too large for one launch", M, N);
    if (split > 1)
        idm_launch_cluster(kernel, dim3((unsigned)tiles, 1, split), dim3(GX_THREADS), bytes, stream, split, x, w, out, M, N, K, token_tiles, (int)tiles);
    else
        idm_launch(kernel, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(GX_THREADS), bytes, stream, x, w, out, M, N, K, token_tiles, (int)tiles);
    return 0;
}

// Tokens per tile and blocks per tile: the same bits whichever, so only time decides.  A block's time is its segments, one after
// another: 0.95 us with 16 or 32 tokens, 1.15 with 64, and about 3 us more where a tile is split (the cluster's barriers, and the sums
// sent).  Measured (us, inputs out of the L2): 1024 x 3072 with 8 tokens split 1 / 4 / 8: 49 / 29 / 18; 4096 x 1024 split
// 1 / 2 / 4: 25 / 20 / 16; with 700 tokens, tiles of 32 / 64 tokens: 4096 x 1024 78 / 64, 1024 x 3072 90 / 61; with 64 tokens
// 6144 x 1024 25 / 37.  A split needs room for all segments' sums of the features that a block adds up.
template <int TN> static void split_cost(int M, int N, int K, int sms, float per_segment, int& best_tn, int& best_split, float& best) {
    const long long tiles = (long long)((M + TN - 1) / TN) * ((N + GX_FEATURES - 1) / GX_FEATURES), segs = (K + GX_SEG - 1) / GX_SEG;
    for (const int split : {1, 2, 3, 4, 6, 8}) {                                 // (sizes of which the SMs of a cluster's reach hold whole numbers)
        if (split > segs || (split > 1 && tiles * split > sms)) break;
        if (split_smem<TN>(K, split) > GX_SMEM) continue;
        const float t = (split == 1 ? (float)((tiles + sms - 1) / sms * segs) : (float)((segs + split - 1) / split)) * per_segment + (split > 1 ? 3.f : 0.f);
        if (t < best) { best = t; best_tn = TN; best_split = split; }
    }
}

struct F32Choice { int tn, split, subs, sms; };               // subs > 0: gemm_f32_wide_kernel with so many times 64 tokens
static F32Choice f32_choice(int M, int N, int K) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
    F32Choice c{64, 1, 0, sms};
    float best = 1e30f;
    if (M <= 16) {
        split_cost<16>(M, N, K, sms, 0.95f, c.tn, c.split, best);
        return c;
    }
    split_cost<32>(M, N, K, sms, 0.95f, c.tn, c.split, best);
    split_cost<64>(M, N, K, sms, 1.15f, c.tn, c.split, best);
    // measured: 1.0 us a segment of 64 tokens and 1.4 of 128 with all SMs at it, and 5 us for the kernel in front and the start (us of tiles that
    // split both operands / 64 / 128 tokens: 180 x 4096 x 1024 28.7 / 27.6 / 35.8, 350 48.1 / 44.0 / 35.8, 700 67.6 / 60.4 / 58.4; 700 x 1024 x 3072
    // 63.5 / 58.4 / 80.9; 577 x 4200 x 1101 96.3 / 82.9 / 74.8; 1 400 x 2048 x 1024 67.6 / 60.4 / 60.4; inputs out of the L2)
    const long long features = (N + GX_FEATURES - 1) / GX_FEATURES, segs = (K + GX_SEG - 1) / GX_SEG;
    for (int subs = 1; subs <= 2; ++subs) {
        const long long tiles = features * ((M + 64 * subs - 1) / (64 * subs));
        const float t = (float)((tiles + sms - 1) / sms * segs) * (subs == 1 ? 1.0f : 1.4f) + 5.f;
        if (t < best) { best = t; c.subs = subs; }
    }
    return c;
}

// Bytes of scratch that a product wants: the parts of x, or 0
extern "C" long long idm_gemm_f32_scratch_bytes(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0 || f32_choice(M, N, K).subs == 0) return 0;
    return 3ll * M * ((K + GX_SEG - 1) / GX_SEG * GX_SEG) * 2;
}

template <int SUBS>
static int wide_launch(const float* x, const float* w, float* out, int M, int N, int K, int rows, void* scratch, int sms, cudaStream_t stream) {
    const int Kp = (K + GX_SEG - 1) / GX_SEG * GX_SEG, bytes = 1024 + 2 * WideTile<SUBS>::STAGE;
    auto kernel = rows == 0 ? gemm_f32_wide_kernel<SUBS, 0> : rows == 1 ? gemm_f32_wide_kernel<SUBS, 1> : gemm_f32_wide_kernel<SUBS, 2>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    IDM_REQUIRE(e == cudaSuccess, "gemm_f32: %d bytes of shared memory: %s", bytes, cudaGetErrorString(e));
    const int token_tiles = (M + 64 * SUBS - 1) / (64 * SUBS);
    const long long tiles = (long long)token_tiles * ((N + GX_FEATURES - 1) / GX_FEATURES), pieces = (long long)M * (Kp / 4);
    IDM_REQUIRE(tiles < (1ll << 30) && pieces < (1ll << 38), "gemm_f32: M=%d N=%d K=%d are too large for one launch", M, N, K);
    CUtensorMap map;
    const cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)M, 3}, strides[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)M * Kp * 2};
    const cuuint32_t box[3] = {GX_SEG, 64, 1};
    const int rc = tc_make_map_bf16(&map, scratch, 3, dims, strides, box);
    IDM_REQUIRE(rc == 0, "gemm_f32: no tensor map for %d x %d parts (%d)", M, Kp, rc);
    idm_launch(split_rows_kernel, dim3((unsigned)((pieces + 255) / 256)), dim3(256), 0, stream, x, (__nv_bfloat16*)scratch, M, K, Kp,
               (int)(K % 4 == 0 && ((uintptr_t)x & 15) == 0));
    idm_launch(kernel, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(WideTile<SUBS>::THREADS), bytes, stream, map, x, w, out, M, N, K, token_tiles, (int)tiles);
    return 0;
}

// scratch: idm_gemm_f32_scratch_bytes, on a 16-byte border
extern "C" int idm_gemm_f32(const float* x, const float* w, float* out, int M, int N, int K, void* scratch, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    IDM_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    const F32Choice c = f32_choice(M, N, K);
    int rc;
    if (c.subs) {
        IDM_REQUIRE(scratch != nullptr && ((uintptr_t)scratch & 15) == 0, "gemm_f32: scratch at %p", scratch);
        const int rows = K % 4 == 0 && ((uintptr_t)w & 15) == 0 ? (K % GX_SEG == 0 ? 2 : 1) : 0;
        rc = c.subs == 1 ? wide_launch<1>(x, w, out, M, N, K, rows, scratch, c.sms, stream) : wide_launch<2>(x, w, out, M, N, K, rows, scratch, c.sms, stream);
    } else {
        const int rows = K % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0 ? (K % GX_SEG == 0 ? 2 : 1) : 0;
        rc = c.tn == 16 ? split_launch<16>(x, w, out, M, N, K, rows, c.split, c.sms, stream)
           : c.tn == 32 ? split_launch<32>(x, w, out, M, N, K, rows, c.split, c.sms, stream)
                        : split_launch<64>(x, w, out, M, N, K, rows, c.split, c.sms, stream);
    }
    if (rc) return rc;
    IDM_LAUNCH_CHECK("gemm_f32");
    return 0;
}

#if defined(IDM_F32)
// The bounded wait in a cluster, by itself: block `late` waits on a barrier that nothing arrives at, for `limit_cycles` (late < 0: no block
// does); out[r]: whether block r knows when they have met.  The kernel ends normally either way.
#define GX_PROBE_BLOCKS 4
__global__ void __launch_bounds__(64) gemm_f32_wait_probe_kernel(long long limit_cycles, int late, int* out) {
    __shared__ __align__(8) unsigned long long bar_mem;
    __shared__ int abort_mem;
    const uint32_t bar = smem_u32(&bar_mem);
    if (threadIdx.x == 0) { mbar_init(bar, 1); abort_mem = 0; mbar_init_fence(); }
    __syncthreads();
    cluster_sync_all();
    if ((int)blockIdx.z == late && threadIdx.x == 32) mbar_wait_limit(bar, 0, (volatile int*)&abort_mem, &g_gemm_f32_error, limit_cycles);
    __syncwarp();
    tell_cluster(&abort_mem, GX_PROBE_BLOCKS);
    cluster_sync_all();
    if (threadIdx.x == 0) out[blockIdx.z] = abort_mem;
}
extern "C" int idm_gemm_f32_wait_probe(long long limit_cycles, int late, int* out, cudaStream_t stream) {
    IDM_REQUIRE(limit_cycles > 0 && limit_cycles <= 2000000000ll, "wait_probe: limit of %lld cycles (1 .. 2e9)", limit_cycles);
    IDM_REQUIRE(out != nullptr && late < GX_PROBE_BLOCKS, "wait_probe: block %d of %d", late, GX_PROBE_BLOCKS);
    idm_launch_cluster(gemm_f32_wait_probe_kernel, dim3(1, 1, GX_PROBE_BLOCKS), dim3(64), 0, stream, GX_PROBE_BLOCKS, limit_cycles, late, out);
    IDM_LAUNCH_CHECK("wait_probe");
    return 0;
}

// 0, or 1 if any block's bounded wait ran out since the last call (reads the flag: synchronises)
extern "C" int idm_gemm_status() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_gemm_f32_error, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_gemm_f32_error, &zero, sizeof(int));
    return v;
}
#endif
