// Linear recurrences over long portions, as products of tiles.  Per head, with a state S [dk, dv],
//
//   S_t = f_t S_(t-1) + a_t k_t v_t^T,      o_t = S_t^T q_t
//
// (f_t, a_t numbers; q and k shared by the heads of a group).  A portion is cut into chunks of CP_C tokens that run side by
// side.  Over a chunk that starts from S_in, with n tokens counted from 0 and F(t, s) = f_(s+1) ... f_t,
//
//   o_t   = F(t, -1) S_in^T q_t + sum_(s<=t) F(t, s) a_s (k_s . q_t) v_s
//   S_out = F(n-1, -1) S_in + sum_s F(n-1, s) a_s k_s v_s^T
//
// so the work is what a chunk adds to the state (chunk_state_kernel), the chunks' states one after another
// (chunk_carry_kernel: S_in of every chunk, from and to the sequence's state), and the read-outs (chunk_out_kernel).  The
// sums are those of the token by token walk in another order; everything is 32-bit, multiply-adds in the read-outs, which is what bounds them.
//
// A thread block has (chunk, group) and some of the group's panels (chunk_cut): a panel is 64 columns of one head's values.  What a
// panel does not depend on is done once for all of them: the keys' tile, the queries' tile and the pair scores k_s . q_t
// (a thread keeps its 4 x 4 of them in registers, and lays them down weighed for each head).  A panel's slices of the
// state and its values come by asynchronous copies, one slice ahead.
//
// A recurrence brings its numbers as a policy W (a kernel argument):
//   struct W::Head                               what a head's numbers over a chunk take in shared memory
//   prepare(Head&, head, t0, n)                  made by the whole block (it may synchronise; the caller synchronises behind it)
//   state(Head&, t) = F(t, -1);  pair(Head&, t, s) = F(t, s) a_s;  end(Head&, n, s) = F(n-1, s) a_s
//   store_end(Head&, chunk, head, n), end_factor(chunk, head, n)     F(n-1, -1), stored by chunk_state_kernel, read by the carry
//   finish(t, head, j, o, v)                     what goes out for column j of a head's read-out o, given the token's v
#pragma once
#include "split_mma.cuh"

#define CP_C 64                 // tokens of a chunk
#define CP_LD 68                // row stride of a tile of 64 columns in shared memory (16-byte rows, banks spread)
#define CP_TILE (64 * CP_LD)
#define CP_MAX_DK 256
#define CP_THREADS 256

struct ChunkArgs {
    const float* q; const float* k; const float* v;          // rows of packed tokens: q + t * q_stride + group * dk, v + t * v_stride + head * dv
    int q_stride, k_stride, v_stride;
    float* o; int o_stride;                                  // o[t, head * dv + j]
    float* state; long long state_stride;                    // state + slot * stride : [heads][dk][dv]
    const int* slots;
    const int* chunk_t0; const int* seq_chunk0;              // the chunks' first packed tokens [n_chunks + 1], each sequence's first chunk
    float* chunk_state;                                      // [n_chunks][heads][dk][dv]
    int groups, heads, dk, dv;
    int panels;                                              // of a block
    int vec;                                                 // tiles may be read and written in 16-byte pieces
};

// a tile of 64 rows of `width` (a multiple of 64) floats into shared memory: rows r < n_rows at src + r * ld, columns c < n_cols;
// zeros elsewhere.  16-byte copies are asynchronous.
template <int THREADS>
__device__ __forceinline__ void cp_tile(float* dst, int dst_ld, int width, const float* __restrict__ src, size_t ld, int n_rows, int n_cols, int vec) {
    if (vec) {
        const int per = width / 4;
        for (int e = threadIdx.x; e < 64 * per; e += THREADS) {
            const int r = e / per, c = (e - r * per) * 4;
            float* to = dst + r * dst_ld + c;
            if (r < n_rows && c < n_cols)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(src + (size_t)r * ld + c) : "memory");
            else *reinterpret_cast<float4*>(to) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    } else {
        for (int e = threadIdx.x; e < 64 * width; e += THREADS) {
            const int r = e / width, c = e - r * width;
            dst[r * dst_ld + c] = (r < n_rows && c < n_cols) ? src[(size_t)r * ld + c] : 0.f;
        }
    }
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(LEFT) : "memory"); }

// panel p of a group: its head and first column
__device__ __forceinline__ void panel_place(const ChunkArgs& a, int group, int p, int& head, int& j0) {
    const int across = (a.dv + 63) / 64;
    head = group * (a.heads / a.groups) + p / across;
    j0 = p % across * 64;
}
__device__ __forceinline__ int panel_count(const ChunkArgs& a) { return a.heads / a.groups * ((a.dv + 63) / 64); }

__device__ __forceinline__ void store_row4(float* p, const float* x, int left, int vec) {
    if (vec && left >= 4) { *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]); return; }
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (k < left) p[k] = x[k];
}

#define CS_LD 72                // row stride of a tile of 64 columns in three planes, bfloat16 (an odd number of 16-byte pieces)
#define CS_LDK 136              // of a tile of 128 columns
#define CS_PLANE (64 * CS_LD)
#define CS_PLANE_K (64 * CS_LDK)
// A tile of 64 x 64 numbers on its way: rows r < n_rows at src + r * ld, columns c < n_cols, zeros elsewhere.  A thread brings 16 of them as
// they are into a place of its own by asynchronous copies (issue), and later, behind its own wait alone, lays their parts down (split).
struct TileFrom { const float* src; size_t ld; int n_rows, n_cols; };
__device__ __forceinline__ void cs_issue(float* raw, const TileFrom& f, int vec) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int e = threadIdx.x + u * CP_THREADS, r = e >> 4, c = (e & 15) * 4;
        float* to = raw + e * 4;
        const float* from = f.src + (size_t)r * f.ld + c;
        const int left = r < f.n_rows ? f.n_cols - c : 0;
        if (vec) {                                           // (whole pieces are there or not)
            if (left > 0) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from) : "memory");
            else *reinterpret_cast<float4*>(to) = make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) to[i] = i < left ? from[i] : 0.f;
        }
    }
}
// dst: the first of three planes of 64 rows, LD apart.  SCALE: times scale[row]
template <int LD, bool SCALE>
__device__ __forceinline__ void cs_split(__nv_bfloat16* dst, const float* raw, const float* scale) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int e = threadIdx.x + u * CP_THREADS, r = e >> 4, c = (e & 15) * 4;
        float4 x = *reinterpret_cast<const float4*>(raw + e * 4);
        if (SCALE) { const float f = scale[r]; x = make_float4(x.x * f, x.y * f, x.z * f, x.w * f); }
        store_split4(dst + r * LD + c, 64 * LD, x);
    }
}
// planes of 64 x 128 and of 64 x 64 numbers, and two tiles on their way.  Two blocks an SM.
struct ChunkStateSmem {
    __nv_bfloat16 wide[3 * CS_PLANE_K];
    __nv_bfloat16 tile[3 * CS_PLANE];
    float raw[2][64 * 64];
};

// chunk_state[c, head, d, j] = sum_s end(s) k_s[d] v_s[j], 128 dims at a time, of which a warp has 32, and 32 columns: products of operands in three
// bfloat16 parts on the tensor cores (split_mma.cuh).  76 chunks of 32 heads of 128 x 64 87 us, 28 of 8 of 128 x 256 33 (by FMAs, 8 x 4 outputs a
// thread, 119 and 39).  Bound by a block's three barriers a panel and the splitting; two blocks an SM.
template <typename W>
__global__ void __launch_bounds__(CP_THREADS, 2) chunk_state_kernel(ChunkArgs a, W w) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) char cp_sm[];
    ChunkStateSmem& sm = *reinterpret_cast<ChunkStateSmem*>(cp_sm);          // wide: [tokens][128 dims]; tile: [tokens][columns], weighed
    __shared__ typename W::Head hd;
    __shared__ float weight[CP_C];
    const int c = blockIdx.x, g = blockIdx.y, t0 = a.chunk_t0[c], n = a.chunk_t0[c + 1] - t0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3, row = lane >> 2;
    const int p0 = blockIdx.z * a.panels, p1 = min(p0 + a.panels, panel_count(a)), col = (warp >> 2) * 32, wide = (a.dk + 127) / 128;
    // 128 dims' two tiles of keys, then the panels' values; and again for the other dims
    const int per = 2 + p1 - p0, steps = wide * per;
    auto issue = [&](int step) {
        if (step < steps) {
            const int d0 = step / per * 128, i = step % per;
            TileFrom f;
            if (i < 2) f = TileFrom{a.k + (size_t)t0 * a.k_stride + g * a.dk + d0 + i * 64, (size_t)a.k_stride, n, a.dk - d0 - i * 64};
            else {
                int head, j0;
                panel_place(a, g, p0 + i - 2, head, j0);
                f = TileFrom{a.v + (size_t)t0 * a.v_stride + head * a.dv + j0, (size_t)a.v_stride, n, a.dv - j0};
            }
            cs_issue(sm.raw[step & 1], f, a.vec);
        }
        cp_commit();
    };
    issue(0);
    issue(1);
    int last = -1;
    for (int step = 0; step < steps; ++step) {
        const int d0 = step / per * 128, i = step % per;
        int head = 0, j0 = 0;
        if (i >= 2) {
            panel_place(a, g, p0 + i - 2, head, j0);
            if (head != last) {
                __syncthreads();
                w.prepare(hd, head, t0, n);
                __syncthreads();
                if (threadIdx.x < CP_C) weight[threadIdx.x] = threadIdx.x < n ? w.end(hd, n, threadIdx.x) : 0.f;
                if (threadIdx.x == 0) w.store_end(hd, c, head, n);
                last = head;
            }
        }
        cp_wait<1>();
        __syncthreads();                                     // the weights are there, everyone is through with the planes before
        if (i < 2) cs_split<CS_LDK, false>(sm.wide + i * 64, sm.raw[step & 1], nullptr);
        else cs_split<CS_LD, true>(sm.tile, sm.raw[step & 1], weight);
        issue(step + 2);
        if (i < 2) continue;
        __syncthreads();
        const int m0 = (warp & 3) * 32;
        if (d0 + m0 >= a.dk) continue;
        SplitSum<4> sum[2];
        sum[0].clear();
        sum[1].clear();
#pragma unroll 1
        for (int kk = 0; kk < n; kk += 16) {                 // 16 tokens
            SplitA A[2];
#pragma unroll
            for (int m = 0; m < 2; ++m) A[m].load_t(sm.wide + kk * CS_LDK + m0 + 16 * m, CS_PLANE_K, CS_LDK, lane);
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                SplitB B;
                B.load_t(sm.tile + kk * CS_LD + col + 8 * j, CS_PLANE, CS_LD, lane);
                sum[0].add(j, A[0], B);
                sum[1].add(j, A[1], B);
            }
        }
        float* dst = a.chunk_state + ((size_t)c * a.heads + head) * a.dk * a.dv + j0;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int d = d0 + m0 + 16 * m + row + 8 * h;
                if (d >= a.dk) continue;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int jj = col + 8 * j + 2 * q, left = a.dv - j0 - jj;
                    float y[2] = {sum[m].sum(j, 2 * h), sum[m].sum(j, 2 * h + 1)};
                    if (!isfinite(y[0] + y[1]))              // (a number that has no parts): made again of plain FMAs
                        for (int u = 0; u < min(left, 2); ++u) {
                            if (isfinite(y[u])) continue;
                            const float* kd = a.k + (size_t)t0 * a.k_stride + g * a.dk + d;
                            const float* vd = a.v + (size_t)t0 * a.v_stride + head * a.dv + j0 + jj + u;
                            float s = 0.f;
                            for (int t = 0; t < n; ++t) s = fmaf(kd[(size_t)t * a.k_stride], vd[(size_t)t * a.v_stride] * weight[t], s);
                            y[u] = s;
                        }
                    float* to = dst + (size_t)d * a.dv + jj;
                    if (a.vec && left >= 2) *reinterpret_cast<float2*>(to) = make_float2(y[0], y[1]);
                    else {
                        if (left > 0) to[0] = y[0];
                        if (left > 1) to[1] = y[1];
                    }
                }
            }
    }
}

// chunk after chunk: what a chunk starts from takes the place of what it adds, and the state moves on.  A thread has V
// elements side by side; the chunks of a batch are on their way together, only the sums are a chain.
#define CP_BATCH 8
template <int V, typename W>
__global__ void __launch_bounds__(128) chunk_carry_kernel(ChunkArgs a, W w) {
    pdl_launch_dependents();
    pdl_wait();
    const int s = blockIdx.z, h = blockIdx.y;
    const size_t per = (size_t)a.dk * a.dv, e = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (e >= per) return;                                    // (V == 4: dv is a multiple of 4)
    const int c0 = a.seq_chunk0[s], c1 = a.seq_chunk0[s + 1];
    float* st = a.state + (size_t)a.slots[s] * a.state_stride + (size_t)h * per + e;
    float* cs = a.chunk_state + ((size_t)c0 * a.heads + h) * per + e;
    const size_t step = (size_t)a.heads * per;
    float S[V];
#pragma unroll
    for (int i = 0; i < V; ++i) S[i] = st[i];
    for (int b = c0; b < c1; b += CP_BATCH, cs += CP_BATCH * step) {
        float add[CP_BATCH][V], f[CP_BATCH];
#pragma unroll
        for (int u = 0; u < CP_BATCH; ++u)
            if (b + u < c1) {
                if constexpr (V == 4) {
                    const float4 x = *reinterpret_cast<const float4*>(cs + u * step);
                    add[u][0] = x.x; add[u][1] = x.y; add[u][2] = x.z; add[u][3] = x.w;
                } else add[u][0] = cs[u * step];
                f[u] = w.end_factor(b + u, h, a.chunk_t0[b + u + 1] - a.chunk_t0[b + u]);
            }
#pragma unroll
        for (int u = 0; u < CP_BATCH; ++u)
            if (b + u < c1) {
                if constexpr (V == 4) *reinterpret_cast<float4*>(cs + u * step) = make_float4(S[0], S[1], S[2], S[3]);
                else cs[u * step] = S[0];
#pragma unroll
                for (int i = 0; i < V; ++i) S[i] = fmaf(f[u], S[i], add[u][i]);
            }
    }
#pragma unroll
    for (int i = 0; i < V; ++i) st[i] = S[i];
}

// four tokens' weighed scores times their values for four rows; OWN: the rows' own tokens, of which row i sees the first i + 1
template <bool OWN>
__device__ __forceinline__ void add_values(float (&out)[4][4], const float* pr, const float* vc) {
    float4 p4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) p4[i] = *reinterpret_cast<const float4*>(pr + i * CP_LD);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float4 v4 = *reinterpret_cast<const float4*>(vc + e * CP_LD);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (OWN && i < e) continue;
            const float x = e == 0 ? p4[i].x : e == 1 ? p4[i].y : e == 2 ? p4[i].z : p4[i].w;
            out[i][0] = fmaf(x, v4.x, out[i][0]); out[i][1] = fmaf(x, v4.y, out[i][1]);
            out[i][2] = fmaf(x, v4.z, out[i][2]); out[i][3] = fmaf(x, v4.w, out[i][3]);
        }
    }
}

// read-outs: pair scores once, then panel after panel: q S_in over the dims (slices of 64), times state(t), plus the masked
// and weighed scores times v.  A thread has 4 tokens x 4 columns.
__host__ __device__ __forceinline__ int cp_q_ld(int dk) { return (dk + 63) / 64 * 64 + 4; }
static int chunk_out_smem(int dk) { return (64 * cp_q_ld(dk) + 4 * CP_TILE) * (int)sizeof(float); }
template <typename W>
__global__ void __launch_bounds__(CP_THREADS) chunk_out_kernel(ChunkArgs a, W w) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    __shared__ typename W::Head hd;
    const int ldq = cp_q_ld(a.dk), slices = (a.dk + 63) / 64;
    float* sq = sm;                                          // [tokens][dims]
    float* ss = sq + 64 * ldq;                               // two slices of the state [64 dims][columns]; the keys' tiles before that
    float* sv = ss + 2 * CP_TILE;                            // [tokens][columns]
    float* sp = sv + CP_TILE;                                // [t][s]: the head's weighed scores
    const int c = blockIdx.x, g = blockIdx.y, t0 = a.chunk_t0[c], n = a.chunk_t0[c + 1] - t0;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;  // tokens 4 ty .., columns 4 tx ..
    const int p0 = blockIdx.z * a.panels, p1 = min(p0 + a.panels, panel_count(a));
    const int nk = (4 * (ty | 1) + 3) / 16 + 1;              // groups of 16 tokens that a warp's rows (two ty) may see
    const float* kbase = a.k + (size_t)t0 * a.k_stride + g * a.dk;

    // pair[i][k]: tokens t = 4 ty + i, s = tx + 16 k
    float pair[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) pair[i][k] = 0.f;
    cp_tile<CP_THREADS>(sq, ldq, ldq - 4, a.q + (size_t)t0 * a.q_stride + g * a.dk, a.q_stride, n, a.dk, a.vec);
    cp_tile<CP_THREADS>(ss, CP_LD, 64, kbase, a.k_stride, n, a.dk, a.vec);
    cp_commit();
    for (int i = 0; i < slices; ++i) {
        if (i + 1 < slices)
            cp_tile<CP_THREADS>(ss + ((i + 1) & 1) * CP_TILE, CP_LD, 64, kbase + (i + 1) * 64, a.k_stride, n, a.dk - (i + 1) * 64, a.vec);
        cp_commit();
        cp_wait<1>();
        __syncthreads();
        const float* sk = ss + (i & 1) * CP_TILE;
#pragma unroll 2
        for (int d = 0; d < 64; d += 4) {
            float4 q4[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) q4[u] = *reinterpret_cast<const float4*>(sq + (4 * ty + u) * ldq + i * 64 + d);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k >= nk) break;                          // (a warp's rows all lie before these tokens)
                const float4 k4 = *reinterpret_cast<const float4*>(sk + (tx + 16 * k) * CP_LD + d);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    pair[u][k] = fmaf(q4[u].x, k4.x, pair[u][k]); pair[u][k] = fmaf(q4[u].y, k4.y, pair[u][k]);
                    pair[u][k] = fmaf(q4[u].z, k4.z, pair[u][k]); pair[u][k] = fmaf(q4[u].w, k4.w, pair[u][k]);
                }
            }
        }
        __syncthreads();                                     // the tile's place is free
    }

    // the steps of the panels, slice after slice; a panel's values come with its first slice
    auto copy_slice = [&](int step) {
        int head, j0;
        const int p = p0 + step / slices, i = step % slices;
        panel_place(a, g, p, head, j0);
        cp_tile<CP_THREADS>(ss + (step & 1) * CP_TILE, CP_LD, 64, a.chunk_state + (((size_t)c * a.heads + head) * a.dk + i * 64) * a.dv + j0, a.dv,
                                a.dk - i * 64, a.dv - j0, a.vec);
    };
    auto copy_values = [&](int p) {
        int head, j0;
        panel_place(a, g, p, head, j0);
        cp_tile<CP_THREADS>(sv, CP_LD, 64, a.v + (size_t)t0 * a.v_stride + head * a.dv + j0, a.v_stride, n, a.dv - j0, a.vec);
    };
    const int steps = (p1 - p0) * slices;
    copy_slice(0);
    copy_values(p0);
    cp_commit();
    int last = -1;
    for (int p = p0, step = 0; p < p1; ++p) {
        int head, j0;
        panel_place(a, g, p, head, j0);
        if (head != last) {
            w.prepare(hd, head, t0, n);
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int t = 4 * ty + i, s = tx + 16 * k;
                    sp[t * CP_LD + s] = s <= t && t < n ? pair[i][k] * w.pair(hd, t, s) : 0.f;
                }
            last = head;
        }
        float out[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) out[i][k] = 0.f;
        for (int i = 0; i < slices; ++i, ++step) {
            if (step + 1 < steps) copy_slice(step + 1);
            cp_commit();
            cp_wait<1>();
            __syncthreads();
            const float* st = ss + (step & 1) * CP_TILE + 4 * tx;
            const float* qr = sq + 4 * ty * ldq + i * 64;
#pragma unroll 2
            for (int d = 0; d < 64; d += 4) {
                float4 q4[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) q4[u] = *reinterpret_cast<const float4*>(qr + u * ldq + d);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float4 s4 = *reinterpret_cast<const float4*>(st + (d + e) * CP_LD);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float q = e == 0 ? q4[u].x : e == 1 ? q4[u].y : e == 2 ? q4[u].z : q4[u].w;
                        out[u][0] = fmaf(q, s4.x, out[u][0]); out[u][1] = fmaf(q, s4.y, out[u][1]);
                        out[u][2] = fmaf(q, s4.z, out[u][2]); out[u][3] = fmaf(q, s4.w, out[u][3]);
                    }
                }
            }
            __syncthreads();                                 // the slice's place is free
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float f = 4 * ty + i < n ? w.state(hd, 4 * ty + i) : 0.f;
#pragma unroll
            for (int k = 0; k < 4; ++k) out[i][k] *= f;
        }
        const float* pr = sp + 4 * ty * CP_LD;
        const float* vc = sv + 4 * tx;
#pragma unroll 2
        for (int s = 0; s < 4 * ty; s += 4) add_values<false>(out, pr + s, vc + s * CP_LD);
        add_values<true>(out, pr + 4 * ty, vc + 4 * ty * CP_LD);   // (the tokens behind a row's own are not touched, whatever they hold)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = 4 * ty + i, left = a.dv - j0 - 4 * tx;
            if (t >= n || left <= 0) continue;
            const float4 v4 = *reinterpret_cast<const float4*>(sv + t * CP_LD + 4 * tx);
            const float vx[4] = {v4.x, v4.y, v4.z, v4.w};
            w.finish(t0 + t, head, j0 + 4 * tx, out[i], vx, min(left, 4), a.vec);
            store_row4(a.o + (size_t)(t0 + t) * a.o_stride + head * a.dv + j0 + 4 * tx, out[i], left, a.vec);
        }
        __syncthreads();                                     // everyone is through with the values and the scores
        if (p + 1 < p1) copy_values(p + 1);                  // (its slice is on its way already: both are waited for together)
        cp_commit();
    }
}

// The same for one panel a block: a slice of q meets the keys' slice and the state's at once, so that only slices are in shared memory and
// three blocks share an SM.  The same sums in the same order.
static int chunk_out_one_smem() { return 4 * CP_TILE * (int)sizeof(float); }
template <typename W>
__global__ void __launch_bounds__(CP_THREADS, 3) chunk_out_one_kernel(ChunkArgs a, W w) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    __shared__ typename W::Head hd;
    float* sq = sm;                                          // [tokens][dims of the slice]; the weighed scores [t][s] behind the last
    float* sk = sq + CP_TILE;                                // [tokens][dims of the slice]
    float* ss = sk + CP_TILE;                                // [dims of the slice][columns]
    float* sv = ss + CP_TILE;                                // [tokens][columns]
    const int c = blockIdx.x, g = blockIdx.y, t0 = a.chunk_t0[c], n = a.chunk_t0[c + 1] - t0, slices = (a.dk + 63) / 64;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const int nk = (4 * (ty | 1) + 3) / 16 + 1;
    int head, j0;
    panel_place(a, g, blockIdx.z, head, j0);
    w.prepare(hd, head, t0, n);
    cp_tile<CP_THREADS>(sv, CP_LD, 64, a.v + (size_t)t0 * a.v_stride + head * a.dv + j0, a.v_stride, n, a.dv - j0, a.vec);
    float pair[4][4], out[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) pair[i][k] = out[i][k] = 0.f;
    for (int i = 0; i < slices; ++i) {
        const int d0 = i * 64, nd = a.dk - d0;
        if (i) __syncthreads();                              // everyone is through with the slice before
        cp_tile<CP_THREADS>(sq, CP_LD, 64, a.q + (size_t)t0 * a.q_stride + g * a.dk + d0, a.q_stride, n, nd, a.vec);
        cp_tile<CP_THREADS>(sk, CP_LD, 64, a.k + (size_t)t0 * a.k_stride + g * a.dk + d0, a.k_stride, n, nd, a.vec);
        cp_tile<CP_THREADS>(ss, CP_LD, 64, a.chunk_state + (((size_t)c * a.heads + head) * a.dk + d0) * a.dv + j0, a.dv, nd, a.dv - j0, a.vec);
        cp_commit();
        cp_wait<0>();
        __syncthreads();
#pragma unroll 2
        for (int d = 0; d < 64; d += 4) {
            float4 q4[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) q4[u] = *reinterpret_cast<const float4*>(sq + (4 * ty + u) * CP_LD + d);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k >= nk) break;                          // (a warp's rows all lie before these tokens)
                const float4 k4 = *reinterpret_cast<const float4*>(sk + (tx + 16 * k) * CP_LD + d);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    pair[u][k] = fmaf(q4[u].x, k4.x, pair[u][k]); pair[u][k] = fmaf(q4[u].y, k4.y, pair[u][k]);
                    pair[u][k] = fmaf(q4[u].z, k4.z, pair[u][k]); pair[u][k] = fmaf(q4[u].w, k4.w, pair[u][k]);
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float4 s4 = *reinterpret_cast<const float4*>(ss + (d + e) * CP_LD + 4 * tx);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float q = e == 0 ? q4[u].x : e == 1 ? q4[u].y : e == 2 ? q4[u].z : q4[u].w;
                    out[u][0] = fmaf(q, s4.x, out[u][0]); out[u][1] = fmaf(q, s4.y, out[u][1]);
                    out[u][2] = fmaf(q, s4.z, out[u][2]); out[u][3] = fmaf(q, s4.w, out[u][3]);
                }
            }
        }
    }
    __syncthreads();                                         // everyone is through with q: the scores take its place
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = 4 * ty + i;
        const float f = t < n ? w.state(hd, t) : 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int s = tx + 16 * k;
            sq[t * CP_LD + s] = s <= t && t < n ? pair[i][k] * w.pair(hd, t, s) : 0.f;
            out[i][k] *= f;
        }
    }
    __syncthreads();
    const float* pr = sq + 4 * ty * CP_LD;
    const float* vc = sv + 4 * tx;
#pragma unroll 2
    for (int s = 0; s < 4 * ty; s += 4) add_values<false>(out, pr + s, vc + s * CP_LD);
    add_values<true>(out, pr + 4 * ty, vc + 4 * ty * CP_LD);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = 4 * ty + i, left = a.dv - j0 - 4 * tx;
        if (t >= n || left <= 0) continue;
        const float4 v4 = *reinterpret_cast<const float4*>(sv + t * CP_LD + 4 * tx);
        const float vx[4] = {v4.x, v4.y, v4.z, v4.w};
        w.finish(t0 + t, head, j0 + 4 * tx, out[i], vx, min(left, 4), a.vec);
        store_row4(a.o + (size_t)(t0 + t) * a.o_stride + head * a.dv + j0 + 4 * tx, out[i], left, a.vec);
    }
}

// How many of a group's panels a block takes (the pair scores and the keys are then read once for them): all that still leave two blocks an
// SM, which is what an SM has room for; more where that leaves a round of a few blocks behind the others and a larger number fills one round.
// Where the blocks are a few more than a round (up to 2.4 an SM), a block takes one panel and the read-outs are chunk_out_one_kernel's,
// three blocks an SM.  Measured, us of a retention of 8 heads of 128 x 256 (32 of 128 x 128):
//   tokens                                    300    500    700   1 000   1 400   8 x 700
//   this rule                             45 (58)  47 (79)  59 (101)  75 (153)  99 (189)  337 (703)
//   always one panel, three an SM         51 (58)  52 (86)  59 (101)  84 (144)  99 (194)  350 (709)
//   one panel, two an SM                  44 (67)  47 (89)  67 (111)  88 (162) 109 (209)  386 (789)
// (The panels' blocks with 8 x 4 outputs a thread in four warps instead of 4 x 4 in eight took 71 (115) at 700 tokens and 348 (718) at 8 x 700.)
struct ChunkCut { int panels; bool one; };
static ChunkCut chunk_cut(int n_chunks, int groups, int panels) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long pairs = (long long)n_chunks * groups;
    auto blocks = [&](int p) { return pairs * ((panels + p - 1) / p); };
    const long long z = (2ll * sms + pairs - 1) / pairs;
    int p = z >= panels ? 1 : (int)((panels + z - 1) / z);
    if (5 * blocks(p) > 12ll * sms)
        for (int q = p + 1; q <= panels; ++q)
            if (blocks(q) <= 2ll * sms && 10 * blocks(q) >= 17ll * sms) { p = q; break; }
    const bool one = blocks(p) > 2ll * sms && 5 * blocks(p) <= 12ll * sms;
    return ChunkCut{one ? 1 : p, one};
}

// The same for what the chunks add to the state (chunk_state_kernel, two blocks an SM, in which a panel counts 5 and the keys' split 2): as few
// rounds of blocks times a block's length as there can be.  76 chunks of 8 groups of 4 panels: four a block 97 us, two 87.
static int chunk_state_panels(int n_chunks, int groups, int panels) {
    int dev = 0, sms = 0, best = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long long least = 0;
    for (int p = 1; p <= panels; ++p) {
        const long long blocks = (long long)n_chunks * groups * ((panels + p - 1) / p), cost = (blocks + 2 * sms - 1) / (2 * sms) * (5 * p + 2);
        if (p == 1 || cost < least) { best = p; least = cost; }
    }
    return best;
}

template <typename W>
static int chunk_products(ChunkArgs a, const W& w, int n_chunks, int n_seqs, const char* what, cudaStream_t stream) {
    const int panels = a.heads / a.groups * ((a.dv + 63) / 64), out_smem = chunk_out_smem(a.dk), out_most = chunk_out_smem(CP_MAX_DK);
    IDM_REQUIRE(n_chunks > 0 && a.heads % a.groups == 0 && a.dk <= CP_MAX_DK && a.groups <= 65535 && n_seqs <= 65535, "%s: %d chunks, %d heads in %d groups, keys of %d",
                what, n_chunks, a.heads, a.groups, a.dk);
    cudaError_t e = cudaFuncSetAttribute(chunk_state_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ChunkStateSmem));
    // (the same limit from every call: a smaller one from another thread would have this launch refused)
    if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_out_one_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, chunk_out_one_smem());
    if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_out_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, out_most);
    IDM_REQUIRE(e == cudaSuccess, "%s: %d bytes of shared memory were refused (%s)", what, out_most, cudaGetErrorString(e));
    a.panels = chunk_state_panels(n_chunks, a.groups, panels);
    idm_launch(chunk_state_kernel<W>, dim3(n_chunks, a.groups, (panels + a.panels - 1) / a.panels), dim3(CP_THREADS), (int)sizeof(ChunkStateSmem), stream, a, w);
    const ChunkCut cut = chunk_cut(n_chunks, a.groups, panels);
    a.panels = cut.panels;
    const dim3 grid(n_chunks, a.groups, (panels + a.panels - 1) / a.panels);
    const size_t per = (size_t)a.dk * a.dv;
    if (a.vec) idm_launch(chunk_carry_kernel<4, W>, dim3((unsigned)((per / 4 + 127) / 128), a.heads, n_seqs), dim3(128), 0, stream, a, w);
    else idm_launch(chunk_carry_kernel<1, W>, dim3((unsigned)((per + 127) / 128), a.heads, n_seqs), dim3(128), 0, stream, a, w);
    if (cut.one) idm_launch(chunk_out_one_kernel<W>, grid, dim3(CP_THREADS), chunk_out_one_smem(), stream, a, w);
    else idm_launch(chunk_out_kernel<W>, grid, dim3(CP_THREADS), out_smem, stream, a, w);
    IDM_LAUNCH_CHECK(what);
    return 0;
}
