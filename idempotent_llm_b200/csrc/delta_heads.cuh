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
// A prompt of 2 048 tokens, 32 heads of 128 x 64 over 8 keys: 39 us the chunks (shared memory's reads for the system bound them), 186 the walk
// (instructions of the splits, and the chain of a chunk's three barriers); decays per channel took 258 and 230.
#pragma once
#include "split_mma.cuh"

#define DH_C 32
#define DH_DK 128                                               // channels of a key's row, rounded up
#define DH_COLS 16                                              // columns of S of a block of the walk
#define DH_HEADS 8                                              // heads that a block of the chunks weighs at a time, a warp each
#define DH_MOST (128ll << 20)                                   // floats of scratch
struct DeltaHeadsScan {
    const float* c; int c_stride, c_q, c_k, c_v;                // rows of packed tokens: q, k [Hk, dk], v [H, dv]
    const float* g;                                             // [n, H] decays
    const float* beta;                                          // [n, H]
    float* state; long long state_stride;                       // state + slot * stride : [H][dv][dk]
    float* o; int o_stride;                                     // o[t, h * dv + j]
    const int* cu_q; const int* slots;
    int n_seqs, H, Hk, dk, dv;
    float* scratch;
};
// a chunk's numbers of one head in scratch: X_k [C][DH_DK], B [C][C], G [C], E [C], then X_v by groups of 16 columns [C][16]
#define DH_B (DH_C * DH_DK)
#define DH_G (DH_B + DH_C * DH_C)
#define DH_E (DH_G + DH_C)
#define DH_XV (DH_E + DH_C)
__host__ __device__ __forceinline__ int delta_heads_floats(int dv) { return DH_XV + (dv + DH_COLS - 1) / DH_COLS * DH_C * DH_COLS; }
// the place of a sequence's first chunk: chunks of sequence s are no more than the tokens' places from there to the next one's
__host__ __device__ __forceinline__ long long delta_heads_slot(int cu_q, int s) { return (cu_q >> 5) + s; }
static_assert(DH_C == 32, "the places count tokens by 32");

#define DH_LD (DH_DK + 4)
#define DH_LDP 36
struct DeltaHeadsChunkSmem {
    float k[DH_C * DH_LD], q[DH_C * DH_LD];
    float kk[DH_C * DH_LDP], qk[DH_C * DH_LDP];
    float A[DH_HEADS][DH_C * DH_LDP];                           // [t][s], 0 from the diagonal on
    float d[DH_HEADS][DH_C], beta[DH_HEADS][DH_C], G[DH_HEADS][DH_C];
};

__global__ void __launch_bounds__(256, 2) delta_heads_chunk_kernel(DeltaHeadsScan a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) char dh_sm[];
    DeltaHeadsChunkSmem& sm = *reinterpret_cast<DeltaHeadsChunkSmem*>(dh_sm);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, hk = blockIdx.y, slot = blockIdx.x;
    int lo = 0, hi = a.n_seqs - 1;                              // the last sequence whose place is at or before this one
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (delta_heads_slot(a.cu_q[mid], mid) <= slot) lo = mid; else hi = mid - 1;
    }
    const int t1 = a.cu_q[lo + 1], tb = a.cu_q[lo] + (slot - (int)delta_heads_slot(a.cu_q[lo], lo)) * DH_C;
    if (tb >= t1) return;
    const int n = min(DH_C, t1 - tb), per = a.H / a.Hk;

    // missing tokens and channels: k = q = 0, beta = 0, d = 1
    {
        float4 x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int e = tid + (i & 3) * 256, t = e >> 5, d = (e & 31) * 4;
            x[i] = t < n && d < a.dk ? *reinterpret_cast<const float4*>(a.c + (size_t)(tb + t) * a.c_stride + (i < 4 ? a.c_k : a.c_q) + hk * a.dk + d)
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int e = tid + (i & 3) * 256, t = e >> 5, d = (e & 31) * 4;
            *reinterpret_cast<float4*>((i < 4 ? sm.k : sm.q) + t * DH_LD + d) = x[i];
        }
    }
    __syncthreads();
    {   // 64 rows (keys, then queries) x 32 keys: four rows and two keys a thread
        const int r0 = (tid >> 4) * 4, c0 = tid & 15;
        const float* rows = (r0 < DH_C ? sm.k + r0 * DH_LD : sm.q + (r0 - DH_C) * DH_LD);
        float2 acc[4][2] = {};                                  // even and odd channels
#pragma unroll 4
        for (int d = 0; d < DH_DK; d += 4) {
            float4 y[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) y[j] = *reinterpret_cast<const float4*>(sm.k + (c0 + 16 * j) * DH_LD + d);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
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
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) to[i * DH_LDP + c0 + 16 * j] = acc[i][j].x + acc[i][j].y;
    }
    const int vcols = (a.dv + 31) / 32 * 32, sides = DH_DK + vcols, floats = delta_heads_floats(a.dv);
    for (int h0 = 0; h0 < per; h0 += DH_HEADS) {
        const int heads = min(DH_HEADS, per - h0), first = hk * per + h0;
        float* out = a.scratch + ((size_t)slot * a.H + first) * floats;
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
            float* mine = out + (size_t)warp * floats;
            mine[DH_G + lane] = G;
            mine[DH_E + lane] = E;
            float F = 1.f;
#pragma unroll 8
            for (int t = 0; t < DH_C; ++t) {
                const float dt = __shfl_sync(0xffffffffu, d, t);
                if (t > lane) F *= dt;
                sm.A[warp][t * DH_LDP + lane] = t > lane ? F * sm.kk[t * DH_LDP + lane] : 0.f;
                mine[DH_B + t * DH_C + lane] = t >= lane ? F * sm.qk[t * DH_LDP + lane] : 0.f;
            }
        }
        __syncthreads();
        // the system, a thread per right-hand side (a warp's are of one head): channels of G k, then columns of v
        for (int i = tid; i < heads * sides; i += 256) {
            const int hh = i / sides, col = i - hh * sides, j = col - DH_DK;
            const float* A = sm.A[hh];
            float x[DH_C];
            if (j < 0) {
#pragma unroll
                for (int t = 0; t < DH_C; ++t) x[t] = sm.G[hh][t] * sm.k[t * DH_LD + col];
            } else {
                const float* v = a.c + (size_t)tb * a.c_stride + a.c_v + (first + hh) * a.dv + j;
#pragma unroll
                for (int t = 0; t < DH_C; ++t) x[t] = t < n && j < a.dv ? v[(size_t)t * a.c_stride] : 0.f;
            }
#pragma unroll
            for (int t = 0; t < DH_C; ++t) {
                float sum[2] = {0.f, 0.f};
#pragma unroll
                for (int s = 0; s < t; s += 4) {                // (entries from t on are 0, their x are not made yet)
                    const float4 c4 = *reinterpret_cast<const float4*>(A + t * DH_LDP + s);
                    sum[0] = fmaf(c4.x, x[s], sum[0]);
                    if (s + 1 < t) sum[1] = fmaf(c4.y, x[s + 1], sum[1]);
                    if (s + 2 < t) sum[0] = fmaf(c4.z, x[s + 2], sum[0]);
                    if (s + 3 < t) sum[1] = fmaf(c4.w, x[s + 3], sum[1]);
                }
                x[t] = sm.beta[hh][t] * (x[t] - (sum[0] + sum[1]));
            }
            float* to = out + (size_t)hh * floats + (j < 0 ? col : DH_XV + j / DH_COLS * (DH_C * DH_COLS) + j % DH_COLS);
            const int step = j < 0 ? DH_DK : DH_COLS;
            if (j < 0 || j / DH_COLS * DH_COLS < a.dv)
#pragma unroll
                for (int t = 0; t < DH_C; ++t) to[t * step] = x[t];
        }
    }
}

#define DH_LDW 136                                              // rows of 128 channels, bfloat16 (an odd number of 16-byte pieces)
#define DH_LDB 40                                               // rows of 32 tokens
#define DH_LDU 24                                               // rows of 16 columns
struct DeltaHeadsWalkSmem {
    float raw[2][3 * DH_C * DH_DK + DH_C * DH_C + 2 * DH_C + DH_C * DH_COLS];   // X_k, q, k, B, G, E, X_v of a chunk and the next
    __nv_bfloat16 xq[3][2 * DH_C * DH_LDW];                     // X_k, then q: [rows][channels]
    __nv_bfloat16 k[3][DH_C * DH_LDW];                          // E k: [tokens][channels]
    __nv_bfloat16 B[3][DH_C * DH_LDB];                          // [tokens t][tokens s]
    __nv_bfloat16 S[3][DH_DK * DH_LDU];                         // [channels][columns]
    __nv_bfloat16 u[3][DH_C * DH_LDU];                          // [tokens][columns]
    float plain[DH_C * (DH_COLS + 1)];                          // u, where columns are made again of plain FMAs:
    int first[DH_COLS];                                         // the first token from which on a column is
};

__global__ void __launch_bounds__(256, 1) delta_heads_walk_kernel(DeltaHeadsScan a) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) char dh_sm[];
    DeltaHeadsWalkSmem& sm = *reinterpret_cast<DeltaHeadsWalkSmem*>(dh_sm);
    constexpr int T = DH_C * DH_DK, Q_AT = T, K_AT = 2 * T, B_AT = 3 * T, G_AT = B_AT + DH_C * DH_C, E_AT = G_AT + DH_C, V_AT = E_AT + DH_C;
    const int s = blockIdx.z, h = blockIdx.y, grp = blockIdx.x, hk = h / (a.H / a.Hk), j0 = grp * DH_COLS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane & 3, row = lane >> 2;
    pdl_wait();
    const int t0 = a.cu_q[s], t1 = a.cu_q[s + 1], chunks = (t1 - t0 + DH_C - 1) / DH_C;
    if (chunks <= 0) return;
    const int floats = delta_heads_floats(a.dv);
    const float* src = a.scratch + ((size_t)delta_heads_slot(t0, s) * a.H + h) * floats;
    auto copy16 = [](float* dst, const float* from) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(from) : "memory");
    };
    // what a thread brings of X_k, q and k it also splits, behind its own wait: X_k and q by all, k and B by the upper half
    auto issue = [&](int ch) {
        if (ch < chunks) {
            const float* from = src + (size_t)ch * a.H * floats;
            float* to = sm.raw[ch & 1];
            const int tb = t0 + ch * DH_C, n = min(DH_C, t1 - tb);
            const float* rows = a.c + (size_t)tb * a.c_stride + hk * a.dk;
            auto token_rows = [&](float* dst, const float* from, int e) {
                const int t = e >> 5, d = (e & 31) * 4;
                if (t < n && d < a.dk) copy16(dst + e * 4, from + (size_t)t * a.c_stride + d);
                else *reinterpret_cast<float4*>(dst + e * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
            };
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int e = tid + i * 256;
                copy16(to + e * 4, from + e * 4);
                token_rows(to + Q_AT, rows + a.c_q, e);
            }
            if (tid >= 128) {
#pragma unroll
                for (int i = 0; i < 8; ++i) token_rows(to + K_AT, rows + a.c_k, tid - 128 + i * 128);
#pragma unroll
                for (int i = 0; i < 2; ++i) copy16(to + B_AT + (tid - 128 + i * 128) * 4, from + DH_B + (tid - 128 + i * 128) * 4);
            } else {
                copy16(to + V_AT + tid * 4, from + DH_XV + grp * (DH_C * DH_COLS) + tid * 4);
                if (tid < 16) copy16(to + G_AT + tid * 4, from + DH_G + tid * 4);   // (E behind G)
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    issue(0);
    issue(1);
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
        const float* raw = sm.raw[ch & 1];
        const int tb = t0 + ch * DH_C, n = min(DH_C, t1 - tb);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
#pragma unroll
        for (int i = 0; i < 8; ++i) {                           // X_k and q (q lies right behind X_k)
            const int e = (tid + (i & 3) * 256) + (i >> 2) * (T / 4);
            store_split4(sm.xq[0] + (e >> 5) * DH_LDW + (e & 31) * 4, 2 * DH_C * DH_LDW, *reinterpret_cast<const float4*>(raw + e * 4));
        }
        __syncthreads();                                        // the chunk's numbers, X_k, q and S are there
        float out[2][4] = {};
        bool bad = odd;
        if (warp < 4) {                                         // X_k S (warps 0, 1) and q S (2, 3)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                SplitSum<2> sum;
                sum.clear();
#pragma unroll
                for (int kk = 64 * half; kk < 64 * half + 64; kk += 16) {
                    SplitA A;
                    SplitB B;
                    A.load(sm.xq[0] + warp * 16 * DH_LDW + kk, 2 * DH_C * DH_LDW, DH_LDW, lane);
                    B.load_t(sm.S[0] + kk * DH_LDU, DH_DK * DH_LDU, DH_LDU, lane);
                    sum.add(0, A, B);
                }
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) out[j][i] += sum.sum(j, i);
            }
            if (warp < 2) {
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int t = warp * 16 + row + 8 * i, col = 8 * j + 2 * q;
                        const float2 v = *reinterpret_cast<const float2*>(raw + V_AT + t * DH_COLS + col);
                        out[j][2 * i] = v.x - out[j][2 * i];
                        out[j][2 * i + 1] = v.y - out[j][2 * i + 1];
                        uint32_t p[3];
                        bad |= parts_or_0(out[j][2 * i], out[j][2 * i + 1], p);
#pragma unroll
                        for (int m = 0; m < 3; ++m) *reinterpret_cast<uint32_t*>(sm.u[m] + t * DH_LDU + col) = p[m];
                    }
            }
        } else {                                                // meanwhile E k and B
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int e = tid - 128 + i * 128;
                const float f = raw[E_AT + (e >> 5)];
                const float4 x = *reinterpret_cast<const float4*>(raw + K_AT + e * 4);
                store_split4(sm.k[0] + (e >> 5) * DH_LDW + (e & 31) * 4, DH_C * DH_LDW, make_float4(x.x * f, x.y * f, x.z * f, x.w * f));
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int e = tid - 128 + i * 128;
                store_split4(sm.B[0] + (e >> 3) * DH_LDB + (e & 7) * 4, DH_C * DH_LDB, *reinterpret_cast<const float4*>(raw + B_AT + e * 4));
            }
        }
        bad = __syncthreads_or(bad);                            // u, E k and B are there
        const float gc = raw[G_AT + DH_C - 1];
        constexpr int LD = DH_COLS + 1;
        float* sS = reinterpret_cast<float*>(sm.xq[0]);         // (the parts of X_k and q have been read)
        if (bad) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int col = 8 * j + 2 * q + (i & 1);
                    sS[(d0 + (i >> 1) * 8) * LD + col] = S[j][i];
                    if (warp < 2) sm.plain[(warp * 16 + row + (i >> 1) * 8) * LD + col] = out[j][i];
                }
            __syncthreads();
            if (tid < DH_COLS) {
                int t = 0;
                for (int d = 0; d < a.dk; ++d)
                    if (magnitude(sS[d * LD + tid]) >= SPLIT_FINITE) t = -1;
                if (t == 0)
                    while (t < DH_C && magnitude(sm.plain[t * LD + tid]) < SPLIT_FINITE) ++t;
                sm.first[tid] = max(t, 0);
            }
            __syncthreads();
            for (int e = tid; e < DH_C * DH_COLS; e += 256) {
                const int t = e / DH_COLS, j = e % DH_COLS;
                if (t < sm.first[j]) continue;
                float x = raw[V_AT + e];
                for (int d = 0; d < a.dk; ++d) x = fmaf(-raw[t * DH_DK + d], sS[d * LD + j], x);
                sm.plain[t * LD + j] = x;
            }
        }
        if (warp == 2 || warp == 3) {
            SplitSum<2> sum;
            sum.clear();
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
                if (kk > warp - 2) continue;                // (tokens behind all of this warp's)
                SplitA A;
                SplitB B;
                A.load(sm.B[0] + (warp - 2) * 16 * DH_LDB + 16 * kk, DH_C * DH_LDB, DH_LDB, lane);
                B.load_t(sm.u[0] + 16 * kk * DH_LDU, DH_C * DH_LDU, DH_LDU, lane);
                sum.add(0, A, B);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int t = (warp - 2) * 16 + row + 8 * i;
                if (t >= n) continue;
                const float g = raw[G_AT + t];
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
        SplitSum<2> sum;
        sum.clear();
#pragma unroll
        for (int kk = 0; kk < DH_C; kk += 16) {
            SplitA A;
            SplitB B;
            A.load_t(sm.k[0] + kk * DH_LDW + warp * 16, DH_C * DH_LDW, DH_LDW, lane);
            B.load_t(sm.u[0] + kk * DH_LDU, DH_C * DH_LDU, DH_LDU, lane);
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
                for (int d = 0; d < a.dk; ++d) x = fmaf(raw[Q_AT + t * DH_DK + d], sS[d * LD + j], x);
                x *= raw[G_AT + t];
                for (int i = 0; i <= t; ++i) x = fmaf(raw[B_AT + t * DH_C + i], sm.plain[i * LD + j], x);
                a.o[(size_t)(tb + t) * a.o_stride + h * a.dv + j0 + j] = x;
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int d = d0 + (i >> 1) * 8, col = 8 * j + 2 * q + (i & 1);
                    if (sm.first[col] == DH_C) continue;
                    float x = gc * sS[d * LD + col];
                    for (int t = 0; t < n; ++t) x = fmaf(raw[K_AT + t * DH_DK + d] * raw[E_AT + t], sm.plain[t * LD + col], x);
                    S[j][i] = x;
                }
        }
        lay_state();
        __syncthreads();                                        // everyone is through with the chunk's numbers and parts
        issue(ch + 2);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int d, col;
            if (state_at(j, i, d, col)) sp[(size_t)col * a.dk + d] = S[j][i];
        }
}
