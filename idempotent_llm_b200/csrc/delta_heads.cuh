// The delta rule over portions of many tokens where a head has ONE decay (not one per key channel), keys of up to 128.
//
// Chunks of C = 32 tokens.  With G_t the product of the decays up to and including token t of the chunk, E_s that of the ones behind s,
// F(t, s) = d_(s+1) .. d_t, and S the state before the chunk,
//
//   u_t = beta_t (v_t - G_t S^T k_t - sum_(s<t) A_ts u_s),   A_ts = F(t, s) k_s . k_t
//   o_t = G_t S^T q_t + sum_(s<=t) B_ts u_s,                 B_ts = F(t, s) k_s . q_t
//   S  <- G_C S + sum_s E_s k_s u_s^T
//
// The products k . k and k . q are the same for the heads that share a key: delta_heads_chunk_kernel has (chunk, key head), makes them once
// and weighs them for each head, and solves the triangular system for the right-hand sides G_t k_t and v_t (u = X_v - X_k S), a thread a
// right-hand side, all chunks side by side.  (F: products of the decays between, in ascending order; one that underflows ends at 0.)
// What is left is a chain, delta_heads_walk_kernel: a block has (sequence, head, 16 columns of S) and takes its chunks one after another,
// as products on the tensor cores of operands in three bfloat16 parts (split_mma.cuh) with S in registers as the products leave it.
//
// A token that is not a number reaches no earlier one: A and B are selected, the system runs forward, and a number of u or S that has no
// parts is 0 in the products; what meets it (a column from its token on) is made again of plain FMAs over the tokens a row may see.
//
// A prompt of 2 048 tokens, 32 heads of 128 x 64 over 8 keys: 51 us the chunks (their system's chains, two blocks of six warps an SM), 132 the walk:
// 2.06 us a chunk, of which the tensor instructions' pipe is busy for 0.7; the block's warps wait for instructions with fixed latencies and for one
// another (three barriers a chunk), L1 at half its rate, the 88 KB that a block takes in a chunk at 8 % of the L2's.  With operands
// split where they are used, 32-bit in scratch, the two took 39 and 186; decays per channel 258 and 230.
//
// A chunk of 32 heads over 8 keys leaves 1.8 MB.  So that a call's scratch does not grow with the prompt, places of chunks (a sequence's one
// after another, sequence after sequence) go through a window: chunks, walk, the next places' chunks, their walk; the state in between is the
// sequence's own in memory, in the 32 bits that the registers hold.  Layers of 64 heads, all places at once / windows of 32 M floats / 18 M: 2 048 tokens
// 576 / 577 / 612 us, 4 x 1 500 and fewer 1 290 / 1 389 / 1 437; 32 heads 261 / 260 / 267 and 596 / 620 / 621.
#pragma once
#include "split_mma.cuh"

#define DH_C 32
#define DH_DK 128                                               // channels of a key's row, rounded up
#define DH_COLS 16                                              // columns of S of a block of the walk
#define DH_HEADS 4                                              // heads that a block of the chunks weighs at a time, a warp each
#define DH_THREADS 192                                          // its threads: two heads of 128 channels and 64 columns, two right-hand sides a thread
#define DH_SCRATCH (32ll << 20)                                 // floats of scratch at most, whatever the prompt: about what the L2 holds
struct DeltaHeadsScan {
    const float* c; int c_stride, c_q, c_k, c_v;                // rows of packed tokens: q, k [Hk, dk], v [H, dv]
    const float* g;                                             // [n, H] decays
    const float* beta;                                          // [n, H]
    float* state; long long state_stride;                       // state + slot * stride : [H][dv][dk]
    float* o; int o_stride;                                     // o[t, h * dv + j]
    const int* cu_q; const int* slots;
    int n_seqs, H, Hk, dk, dv;
    char* scratch;
    int first, window;                                          // of the chunks' places: those of this launch
};
// What the chunks leave for the walk, in bytes.  Operands as the walk's products read them: three planes of bfloat16 parts, rows as they lie in
// its shared memory.  Of a chunk and key head: q and k [C][channels].  Of a chunk and head: X_k [C][channels], B [t][s], G and E [C] in 32-bit,
// then X_v in 32-bit by groups of 16 columns [C][16].
#define DH_LDW 136                                              // rows of 128 channels (an odd number of 16-byte pieces)
#define DH_LDB 40                                               // rows of 32 tokens
#define DH_WIDE (3 * DH_C * DH_LDW * 2)
#define DH_PAIRS (3 * DH_C * DH_LDB * 2)
#define DH_XV (DH_C * DH_COLS * 4)
#define DH_HEAD (DH_WIDE + DH_PAIRS + 2 * DH_C * 4)
__host__ __device__ __forceinline__ long long delta_heads_head_bytes(int dv) { return DH_HEAD + (dv + DH_COLS - 1) / DH_COLS * DH_XV; }
__host__ __device__ __forceinline__ long long delta_heads_chunk_bytes(int H, int Hk, int dv) { return (long long)Hk * 2 * DH_WIDE + H * delta_heads_head_bytes(dv); }
// the place of a sequence's first chunk: chunks of sequence s are no more than the tokens' places from there to the next one's
__host__ __device__ __forceinline__ long long delta_heads_slot(int cu_q, int s) { return (cu_q >> 5) + s; }
static_assert(DH_C == 32, "the places count tokens by 32");
// the last sequence whose place is at or before this one
__device__ __forceinline__ int delta_heads_sequence(const int* cu_q, int n_seqs, int slot) {
    int lo = 0, hi = n_seqs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (delta_heads_slot(cu_q[mid], mid) <= slot) lo = mid; else hi = mid - 1;
    }
    return lo;
}

#define DH_LD (DH_DK + 4)
#define DH_LDP 36
struct DeltaHeadsChunkSmem {
    float k[DH_C * DH_LD], q[DH_C * DH_LD];
    float kk[DH_C * DH_LDP], qk[DH_C * DH_LDP];
    float A[DH_HEADS][DH_C * DH_LDP];                           // [t][s], 0 from the diagonal on
    float beta[DH_HEADS][DH_C], G[DH_HEADS][DH_C];
};

__global__ void __launch_bounds__(DH_THREADS, 2) delta_heads_chunk_kernel(DeltaHeadsScan a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) char dh_sm[];
    DeltaHeadsChunkSmem& sm = *reinterpret_cast<DeltaHeadsChunkSmem*>(dh_sm);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, hk = blockIdx.y, slot = a.first + blockIdx.x;
    const int lo = delta_heads_sequence(a.cu_q, a.n_seqs, slot);
    const int t1 = a.cu_q[lo + 1], tb = a.cu_q[lo] + (slot - (int)delta_heads_slot(a.cu_q[lo], lo)) * DH_C;
    if (tb >= t1) return;
    const int n = min(DH_C, t1 - tb), per = a.H / a.Hk;
    char* mine = a.scratch + blockIdx.x * delta_heads_chunk_bytes(a.H, a.Hk, a.dv);

    // missing tokens and channels: k = q = 0, beta = 0, d = 1
    {
        constexpr int ALL = 2 * DH_C * DH_DK / 4, TURNS = (ALL + DH_THREADS - 1) / DH_THREADS;
        float4 x[TURNS];
#pragma unroll
        for (int i = 0; i < TURNS; ++i) {
            const int e = tid + i * DH_THREADS, t = e >> 5 & 31, d = (e & 31) * 4;
            x[i] = e < ALL && t < n && d < a.dk ? *reinterpret_cast<const float4*>(a.c + (size_t)(tb + t) * a.c_stride + (e < ALL / 2 ? a.c_k : a.c_q) + hk * a.dk + d)
                                                : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < TURNS; ++i) {
            const int e = tid + i * DH_THREADS, t = e >> 5 & 31, d = (e & 31) * 4;
            if (e >= ALL) break;
            *reinterpret_cast<float4*>((e < ALL / 2 ? sm.k : sm.q) + t * DH_LD + d) = x[i];
            store_split4(reinterpret_cast<__nv_bfloat16*>(mine + (2 * hk + (e < ALL / 2 ? 1 : 0)) * DH_WIDE) + t * DH_LDW + d, DH_C * DH_LDW, x[i]);
        }
    }
    __syncthreads();
    if (tid < 128) {   // 64 rows (keys, then queries) x 32 keys: eight rows and two keys a thread
        const int r0 = (tid >> 4) * 8, c0 = tid & 15;
        const float* rows = (r0 < DH_C ? sm.k + r0 * DH_LD : sm.q + (r0 - DH_C) * DH_LD);
        float2 acc[8][2] = {};                                  // even and odd channels
#pragma unroll 2
        for (int d = 0; d < DH_DK; d += 4) {
            float4 y[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) y[j] = *reinterpret_cast<const float4*>(sm.k + (c0 + 16 * j) * DH_LD + d);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 x = *reinterpret_cast<const float4*>(rows + i * DH_LD + d);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    acc[i][j] = __ffma2_rn(make_float2(x.x, x.y), make_float2(y[j].x, y[j].y), acc[i][j]);
                    acc[i][j] = __ffma2_rn(make_float2(x.z, x.w), make_float2(y[j].z, y[j].w), acc[i][j]);
                }
            }
        }
        float* to = r0 < DH_C ? sm.kk + r0 * DH_LDP : sm.qk + (r0 - DH_C) * DH_LDP;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) to[i * DH_LDP + c0 + 16 * j] = acc[i][j].x + acc[i][j].y;
    }
    // pairs of right-hand sides: channels of G k, then columns of v, a warp's of one head
    const int sides = DH_DK / 2 + (a.dv + 63) / 64 * 32;
    const long long bytes = delta_heads_head_bytes(a.dv);
    for (int h0 = 0; h0 < per; h0 += DH_HEADS) {
        const int heads = min(DH_HEADS, per - h0), first = hk * per + h0;
        char* out = mine + (long long)a.Hk * 2 * DH_WIDE + first * bytes;
        __syncthreads();                                        // the products are there; everyone is through with the heads before
        if (warp < heads) {                                     // a lane a token s
            const size_t at = (size_t)(tb + lane) * a.H + first + warp;
            const float d = lane < n ? a.g[at] : 1.f;
            sm.beta[warp][lane] = lane < n ? a.beta[at] : 0.f;
            float G = d, E = __shfl_down_sync(0xffffffffu, d, 1);
            if (lane == 31) E = 1.f;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float u = __shfl_up_sync(0xffffffffu, G, o), w = __shfl_down_sync(0xffffffffu, E, o);
                if (lane >= o) G *= u;
                if (lane + o < 32) E *= w;
            }
            sm.G[warp][lane] = G;
            float* ge = reinterpret_cast<float*>(out + warp * bytes + DH_WIDE + DH_PAIRS);
            ge[lane] = G;
            ge[DH_C + lane] = E;
            __nv_bfloat16* b = reinterpret_cast<__nv_bfloat16*>(out + warp * bytes + DH_WIDE);
            const bool upper = lane & 1;
            float F = 1.f;
#pragma unroll 4
            for (int t = 0; t < DH_C; t += 2) {
                float B[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float dt = __shfl_sync(0xffffffffu, d, t + i);
                    if (t + i > lane) F *= dt;
                    sm.A[warp][(t + i) * DH_LDP + lane] = t + i > lane ? F * sm.kk[(t + i) * DH_LDP + lane] : 0.f;
                    B[i] = t + i >= lane ? F * sm.qk[(t + i) * DH_LDP + lane] : 0.f;
                }
                // two lanes lay down a row each: tokens s, s + 1 of row t, and of row t + 1
                const float theirs = __shfl_xor_sync(0xffffffffu, upper ? B[0] : B[1], 1);
                uint32_t p[3];
                split3(upper ? theirs : B[0], upper ? B[1] : theirs, p[0], p[1], p[2]);
#pragma unroll
                for (int m = 0; m < 3; ++m) *reinterpret_cast<uint32_t*>(b + (m * DH_C + t + (upper ? 1 : 0)) * DH_LDB + (lane & ~1)) = p[m];
            }
        }
        __syncthreads();
        for (int i = tid; i < heads * sides; i += DH_THREADS) {
            const int hh = i / sides, col = (i - hh * sides) * 2, j = col - DH_DK;
            const float* A = sm.A[hh];
            float x[DH_C], y[DH_C];
            if (j < 0) {
#pragma unroll
                for (int t = 0; t < DH_C; ++t) {
                    const float2 k = *reinterpret_cast<const float2*>(sm.k + t * DH_LD + col);
                    x[t] = sm.G[hh][t] * k.x; y[t] = sm.G[hh][t] * k.y;
                }
            } else {
                const float* v = a.c + (size_t)tb * a.c_stride + a.c_v + (first + hh) * a.dv + j;
#pragma unroll
                for (int t = 0; t < DH_C; ++t) {
                    x[t] = t < n && j < a.dv ? v[(size_t)t * a.c_stride] : 0.f;
                    y[t] = t < n && j + 1 < a.dv ? v[(size_t)t * a.c_stride + 1] : 0.f;
                }
            }
#pragma unroll
            for (int t = 0; t < DH_C; ++t) {
                float sx[2] = {0.f, 0.f}, sy[2] = {0.f, 0.f};
#pragma unroll
                for (int s = 0; s < t; s += 4) {                // (entries from t on are 0, their x are not made yet)
                    const float4 c4 = *reinterpret_cast<const float4*>(A + t * DH_LDP + s);
                    sx[0] = fmaf(c4.x, x[s], sx[0]); sy[0] = fmaf(c4.x, y[s], sy[0]);
                    if (s + 1 < t) { sx[1] = fmaf(c4.y, x[s + 1], sx[1]); sy[1] = fmaf(c4.y, y[s + 1], sy[1]); }
                    if (s + 2 < t) { sx[0] = fmaf(c4.z, x[s + 2], sx[0]); sy[0] = fmaf(c4.z, y[s + 2], sy[0]); }
                    if (s + 3 < t) { sx[1] = fmaf(c4.w, x[s + 3], sx[1]); sy[1] = fmaf(c4.w, y[s + 3], sy[1]); }
                }
                x[t] = sm.beta[hh][t] * (x[t] - (sx[0] + sx[1]));
                y[t] = sm.beta[hh][t] * (y[t] - (sy[0] + sy[1]));
            }
            if (j < 0) {
                __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(out + hh * bytes) + col;
#pragma unroll
                for (int t = 0; t < DH_C; ++t) {
                    uint32_t p[3];
                    split3(x[t], y[t], p[0], p[1], p[2]);
#pragma unroll
                    for (int m = 0; m < 3; ++m) *reinterpret_cast<uint32_t*>(to + (m * DH_C + t) * DH_LDW) = p[m];
                }
            } else if (j < (a.dv + DH_COLS - 1) / DH_COLS * DH_COLS) {   // (the walk takes whole groups: zeros behind the last column)
                float* to = reinterpret_cast<float*>(out + hh * bytes + DH_HEAD + j / DH_COLS * DH_XV) + j % DH_COLS;
#pragma unroll
                for (int t = 0; t < DH_C; ++t) *reinterpret_cast<float2*>(to + t * DH_COLS) = make_float2(x[t], y[t]);
            }
        }
    }
}

#define DH_LDU 24                                               // rows of 16 columns
struct DeltaHeadsStage {                                        // as in scratch
    __nv_bfloat16 X[3][DH_C * DH_LDW];
    __nv_bfloat16 B[3][DH_C * DH_LDB];
    float G[DH_C], E[DH_C];
    float V[DH_C * DH_COLS];
    __nv_bfloat16 q[3][DH_C * DH_LDW];
    __nv_bfloat16 k[3][DH_C * DH_LDW];
};
struct DeltaHeadsWalkSmem {
    DeltaHeadsStage stage[2];                                   // a chunk and the next
    __nv_bfloat16 S[3][DH_DK * DH_LDU];                         // [channels][columns]
    __nv_bfloat16 u[3][DH_C * DH_LDU], Eu[3][DH_C * DH_LDU];    // [tokens][columns]; times E
    float S32[DH_DK * (DH_COLS + 1)];                           // where columns are made again of plain FMAs: S and u, and
    float u32[DH_C * (DH_COLS + 1)];
    float4 half[2][128];                                        // the products over the upper channels
    int first[DH_COLS];                                         // the first token from which on a column is
};
static_assert(sizeof(DeltaHeadsStage) == DH_HEAD + DH_XV + 2 * DH_WIDE, "the stage is laid out as the scratch is");

// a number of three planes
__device__ __forceinline__ float whole(const __nv_bfloat16* p, int plane, int at) {
    return __bfloat162float(p[at]) + __bfloat162float(p[plane + at]) + __bfloat162float(p[2 * plane + at]);
}

__global__ void __launch_bounds__(256, 1) delta_heads_walk_kernel(DeltaHeadsScan a) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) char dh_sm[];
    DeltaHeadsWalkSmem& sm = *reinterpret_cast<DeltaHeadsWalkSmem*>(dh_sm);
    constexpr int WIDE = DH_C * DH_LDW;                         // elements of a plane
    const int h = blockIdx.y, grp = blockIdx.x, hk = h / (a.H / a.Hk), j0 = grp * DH_COLS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane & 3, row = lane >> 2;
    pdl_wait();
    // the sequences from the one that the window's first place belongs to on; of a sequence the chunks that have their places there
    const int s = (a.first ? delta_heads_sequence(a.cu_q, a.n_seqs, a.first) : 0) + blockIdx.z;
    if (s >= a.n_seqs) return;
    const int t1 = a.cu_q[s + 1], slot0 = (int)delta_heads_slot(a.cu_q[s], s), c0 = max(a.first - slot0, 0), t0 = a.cu_q[s] + c0 * DH_C;
    const int chunks = min((t1 - t0 + DH_C - 1) / DH_C, a.first + a.window - slot0 - c0);
    if (t0 >= t1 || chunks <= 0) return;
    const long long chunk_bytes = delta_heads_chunk_bytes(a.H, a.Hk, a.dv);
    const char* from = a.scratch + (slot0 + c0 - a.first) * chunk_bytes;
    const char* shared = from + (long long)hk * 2 * DH_WIDE;                   // q and k
    const char* head = from + (long long)a.Hk * 2 * DH_WIDE + h * delta_heads_head_bytes(a.dv);
    // (by the upper four warps, while the others make u)
    auto copy = [&](char* dst, const char* src, int n) {        // n bytes, 16 a thread and turn
        const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
        for (int e = (tid - 128) * 16; e < n; e += 128 * 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(to + e), "l"(src + e) : "memory");
    };
    auto issue = [&](int ch) {
        if (ch < chunks) {
            DeltaHeadsStage& st = sm.stage[ch & 1];
            copy(reinterpret_cast<char*>(&st), head + ch * chunk_bytes, DH_HEAD);
            copy(reinterpret_cast<char*>(st.V), head + ch * chunk_bytes + DH_HEAD + grp * DH_XV, DH_XV);
            copy(reinterpret_cast<char*>(st.q), shared + ch * chunk_bytes, 2 * DH_WIDE);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    if (warp >= 4) issue(0);
    // S: a warp has 16 channels; a lane channels d, d + 8 and columns 2 q, 2 q + 1, and 8 on
    const int d0 = warp * 16 + row;
    float* sp = a.state + (size_t)a.slots[s] * a.state_stride + ((size_t)h * a.dv + j0) * a.dk;
    float S[2][4];
    auto state_at = [&](int j, int i, int& d, int& col) { d = d0 + (i >> 1) * 8; col = 8 * j + 2 * q + (i & 1); return d < a.dk && j0 + col < a.dv; };
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int d, col;
            const bool in = state_at(j, i, d, col);
            S[j][i] = in ? sp[(size_t)col * a.dk + d] : 0.f;
        }
    bool odd = false;                                           // some number of S here has no parts
    auto parts_or_0 = [](float x, float y, uint32_t (&p)[3]) {
        const bool a = magnitude(x) >= SPLIT_FINITE, b = magnitude(y) >= SPLIT_FINITE;
        split3(a ? 0.f : x, b ? 0.f : y, p[0], p[1], p[2]);
        return a || b;
    };
    auto lay_state = [&]() {
        odd = false;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint32_t p[3];
                odd |= parts_or_0(S[j][2 * i], S[j][2 * i + 1], p);
#pragma unroll
                for (int m = 0; m < 3; ++m) *reinterpret_cast<uint32_t*>(sm.S[m] + (d0 + 8 * i) * DH_LDU + 8 * j + 2 * q) = p[m];
            }
    };
    lay_state();
    const bool pairs = a.o_stride % 2 == 0 && a.dv % 2 == 0 && ((uintptr_t)a.o & 7) == 0;
    for (int ch = 0; ch < chunks; ++ch) {
        const DeltaHeadsStage& st = sm.stage[ch & 1];
        const int tb = t0 + ch * DH_C, n = min(DH_C, t1 - tb);
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();                                        // the chunk's numbers and S are there
        // X_k S (warps 0, 1 and 4, 5) and q S: the lower channels by warps 0 to 3, the upper by 4 to 7
        float out[2][4];
        bool bad = odd;
        {
            const __nv_bfloat16* mine = (warp & 2 ? st.q[0] : st.X[0]) + (warp & 1) * 16 * DH_LDW;
            SplitSum3<2> sum;
            sum.clear();
#pragma unroll
            for (int i = 0; i < 64; i += 16) {
                const int kk = (warp >> 2) * 64 + i;
                SplitA A;
                SplitB B;
                A.load(mine + kk, WIDE, DH_LDW, lane);
                B.load_t(sm.S[0] + kk * DH_LDU, DH_DK * DH_LDU, DH_LDU, lane);
                sum.add(0, A, B);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) out[j][i] = sum.sum(j, i);
        }
        if (warp >= 4) {
#pragma unroll
            for (int j = 0; j < 2; ++j) sm.half[j][tid - 128] = make_float4(out[j][0], out[j][1], out[j][2], out[j][3]);
        }
        __syncthreads();                                        // the upper channels' products are there
        if (warp >= 4) {
            issue(ch + 1);
        } else {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float4 x = sm.half[j][tid];
                out[j][0] += x.x; out[j][1] += x.y; out[j][2] += x.z; out[j][3] += x.w;
            }
            if (warp < 2) {
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int t = warp * 16 + row + 8 * i, col = 8 * j + 2 * q;
                        const float2 v = *reinterpret_cast<const float2*>(st.V + t * DH_COLS + col);
                        const float e = st.E[t], x = out[j][2 * i] = v.x - out[j][2 * i], y = out[j][2 * i + 1] = v.y - out[j][2 * i + 1];
                        uint32_t p[3], w[3];
                        bad |= parts_or_0(x, y, p);
                        parts_or_0(x * e, y * e, w);
#pragma unroll
                        for (int m = 0; m < 3; ++m) {
                            *reinterpret_cast<uint32_t*>(sm.u[m] + t * DH_LDU + col) = p[m];
                            *reinterpret_cast<uint32_t*>(sm.Eu[m] + t * DH_LDU + col) = w[m];
                        }
                    }
            }
        }
        bad = __syncthreads_or(bad);                            // u is there
        const float gc = st.G[DH_C - 1];
        constexpr int LD = DH_COLS + 1;
        if (bad) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int col = 8 * j + 2 * q + (i & 1);
                    sm.S32[(d0 + (i >> 1) * 8) * LD + col] = S[j][i];
                    if (warp < 2) sm.u32[(warp * 16 + row + (i >> 1) * 8) * LD + col] = out[j][i];
                }
            __syncthreads();
            if (tid < DH_COLS) {
                int t = 0;
                for (int d = 0; d < a.dk; ++d)
                    if (magnitude(sm.S32[d * LD + tid]) >= SPLIT_FINITE) t = -1;
                if (t == 0)
                    while (t < DH_C && magnitude(sm.u32[t * LD + tid]) < SPLIT_FINITE) ++t;
                sm.first[tid] = max(t, 0);
            }
            __syncthreads();
            for (int e = tid; e < DH_C * DH_COLS; e += 256) {
                const int t = e / DH_COLS, j = e % DH_COLS;
                if (t < sm.first[j]) continue;
                float x = st.V[e];
                for (int d = 0; d < a.dk; ++d) x = fmaf(-whole(st.X[0], WIDE, t * DH_LDW + d), sm.S32[d * LD + j], x);
                sm.u32[t * LD + j] = x;
            }
        }
        if (warp == 2 || warp == 3) {
            SplitSum3<2> sum;
            sum.clear();
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
                if (kk > warp - 2) continue;                // (tokens behind all of this warp's)
                SplitA A;
                SplitB B;
                A.load(st.B[0] + (warp - 2) * 16 * DH_LDB + 16 * kk, DH_C * DH_LDB, DH_LDB, lane);
                B.load_t(sm.u[0] + 16 * kk * DH_LDU, DH_C * DH_LDU, DH_LDU, lane);
                sum.add(0, A, B);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int t = (warp - 2) * 16 + row + 8 * i;
                if (t >= n) continue;
                const float g = st.G[t];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int left = a.dv - j0 - 8 * j - 2 * q;
                    float* dst = a.o + (size_t)(tb + t) * a.o_stride + h * a.dv + j0 + 8 * j + 2 * q;
                    const float x = fmaf(g, out[j][2 * i], sum.sum(j, 2 * i)), y = fmaf(g, out[j][2 * i + 1], sum.sum(j, 2 * i + 1));
                    if (pairs && left >= 2) *reinterpret_cast<float2*>(dst) = make_float2(x, y);
                    else {
                        if (left > 0) dst[0] = x;
                        if (left > 1) dst[1] = y;
                    }
                }
            }
        }
        SplitSum3<2> sum;
        sum.clear();
#pragma unroll
        for (int kk = 0; kk < DH_C; kk += 16) {
            SplitA A;
            SplitB B;
            A.load_t(st.k[0] + kk * DH_LDW + warp * 16, WIDE, DH_LDW, lane);
            B.load_t(sm.Eu[0] + kk * DH_LDU, DH_C * DH_LDU, DH_LDU, lane);
            sum.add(0, A, B);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) S[j][i] = fmaf(gc, S[j][i], sum.sum(j, i));
        if (bad) {
            __syncthreads();                                    // (the read-outs that are made again are written after the others)
            for (int e = tid; e < n * DH_COLS; e += 256) {
                const int t = e / DH_COLS, j = e % DH_COLS;
                if (j0 + j >= a.dv || t < sm.first[j]) continue;
                float x = 0.f;
                for (int d = 0; d < a.dk; ++d) x = fmaf(whole(st.q[0], WIDE, t * DH_LDW + d), sm.S32[d * LD + j], x);
                x *= st.G[t];
                for (int i = 0; i <= t; ++i) x = fmaf(whole(st.B[0], DH_C * DH_LDB, t * DH_LDB + i), sm.u32[i * LD + j], x);
                a.o[(size_t)(tb + t) * a.o_stride + h * a.dv + j0 + j] = x;
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int d = d0 + (i >> 1) * 8, col = 8 * j + 2 * q + (i & 1);
                    if (sm.first[col] == DH_C) continue;
                    float x = gc * sm.S32[d * LD + col];
                    for (int t = 0; t < n; ++t) x = fmaf(whole(st.k[0], WIDE, t * DH_LDW + d) * st.E[t], sm.u32[t * LD + col], x);
                    S[j][i] = x;
                }
        }
        lay_state();
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int d, col;
            if (state_at(j, i, d, col)) sp[(size_t)col * a.dk + d] = S[j][i];
        }
}
