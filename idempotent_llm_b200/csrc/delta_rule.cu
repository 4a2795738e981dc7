// The gated delta rule: a recurrent mixer whose state S [dk, dv] per head is decayed row by row, corrected
// towards the token's value at the token's key, and read with the token's query:
//
//   S <- diag(g_t) S;   u = beta_t (v_t - S^T k_t);   S <- S + k_t u^T;   o_t = S^T q_t
//
// q, k [Hk, dk] are unit vectors per head (q also times dk^-1/2), v [H, dv], beta [H] in (0, 1), g [H, dk] in (0, 1];
// head h reads q/k head h / (H / Hk).  Everything here is 32-bit: the state, the decays and their logarithms, the
// unit norms, the gates.  S lives per sequence as [H][dv][dk] (a column's dk numbers side by side) and is carried
// from step to step.  Steps of up to 4 tokens a sequence walk them one by one, and a token's bits do not depend on how its
// sequence was cut into such steps; when any sequence of a step brings more, all of the step's run in chunks, and a token's
// result is the same sums in another order.
//
// The read-out is computed from the decayed state before the write: o = (g S)^T q + u (k . q), the same number
// as S_new^T q, so that one round of shuffles per token serves both sums.
#include "common.cuh"
#include "delta_heads.cuh"

// ------------------------------------------------------------------ columns of a 32-bit buffer as a matrix operand
// out[t, c] = in[t, col0 + c] for c < width, 0 for width <= c < out_width, in the storage type
__global__ void __launch_bounds__(256) cols_cast_kernel(const float* __restrict__ in, int stride, int col0, int width,
                                                        T* __restrict__ out, int out_width, int n) {
    pdl_launch_dependents();
    pdl_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)n * out_width) return;
    const int t = (int)(i / out_width), c = (int)(i % out_width);
    from_f32(out[i], c < width ? in[(size_t)t * stride + col0 + c] : 0.f);
}

extern "C" int idm_cols_cast(const float* in, int stride, int col0, int width, void* out, int out_width, int n_tokens,
                             cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    IDM_REQUIRE(col0 >= 0 && width > 0 && col0 + width <= stride && out_width >= width,
                "cols_cast: columns %d..%d of rows of %d into rows of %d", col0, col0 + width, stride, out_width);
    const long long total = (long long)n_tokens * out_width;
    idm_launch(cols_cast_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, stream, in, stride, col0, width,
               (T*)out, out_width, n_tokens);
    IDM_LAUNCH_CHECK("cols_cast");
    return 0;
}

// ------------------------------------------------------------------ what the recurrence reads, made in place
// c [N, c_stride]: filtered and activated q (Hk x dk at c_q), k (at c_k); both become unit vectors per head,
// x / sqrt(sum x^2 + 1e-6), q also times dk^-1/2.  a [N, a_stride]: columns [a_col, a_col + H dk) hold the decay's
// projection and become g = exp(-exp(A_log[h]) * softplus(a + dt_bias)).  beta[t, h] = sigmoid(proj[t, b_col + h]).
// With one decay per head (head_col >= 0) the projection is proj[t, head_col + h], dt_bias has H entries, and the
// head's decay is written to all dk of its columns of `a`, which the recurrence reads as it reads decays per channel, or (a_dk == 1) to
// column a_col + h alone.
struct DeltaPrepArgs {
    float* c; int c_stride, c_q, c_k;
    float* a; int a_stride, a_col;
    const float* proj; int p_stride, b_col, head_col;
    const float* dt_bias; const float* a_log;
    float* beta;
    int H, Hk, dk, a_dk;                            // a_dk: columns of a head's decays
};

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }

__global__ void __launch_bounds__(128) delta_prep_kernel(DeltaPrepArgs p) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* row = p.c + (size_t)t * p.c_stride;
    const float q_scale = 1.0f / sqrtf((float)p.dk);
    for (int i = blockIdx.y * 4 + warp; i < 2 * p.Hk; i += gridDim.y * 4) {
        const bool is_q = i < p.Hk;
        float* x = row + (is_q ? p.c_q + i * p.dk : p.c_k + (i - p.Hk) * p.dk);
        float ss = 0.f;
        for (int d = lane; d < p.dk; d += 32) ss += x[d] * x[d];
        const float inv = (is_q ? q_scale : 1.f) / sqrtf(warp_sum(ss) + 1e-6f);
        for (int d = lane; d < p.dk; d += 32) x[d] *= inv;
    }
    float* arow = p.a + (size_t)t * p.a_stride + p.a_col;
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < p.H * p.a_dk; i += gridDim.y * blockDim.x) {
        const int hh = i / p.a_dk;
        const float rate = expf(p.a_log[hh]);
        const float z = p.head_col >= 0 ? p.proj[(size_t)t * p.p_stride + p.head_col + hh] + p.dt_bias[hh] : arow[i] + p.dt_bias[i];
        arow[i] = expf(-rate * softplus_f(z));
    }
    for (int h = blockIdx.y * blockDim.x + threadIdx.x; h < p.H; h += gridDim.y * blockDim.x)
        p.beta[(size_t)t * p.H + h] = 1.0f / (1.0f + expf(-p.proj[(size_t)t * p.p_stride + p.b_col + h]));
}

// The same with heads of up to 128 channels in pieces of four on their borders: a warp has four heads' rows on their way at a time, a
// decay per head is made once a token and spread from shared memory.  Bound by the bytes of the decays.
#define DP_HEADS 256
__global__ void __launch_bounds__(128) delta_prep_vec_kernel(DeltaPrepArgs p) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float decay[DP_HEADS];
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, d = lane * 4;
    float* row = p.c + (size_t)t * p.c_stride;
    const float q_scale = 1.0f / sqrtf((float)p.dk);
    if (p.head_col >= 0)
        for (int h = threadIdx.x; h < p.H; h += 128)
            decay[h] = expf(-expf(p.a_log[h]) * softplus_f(p.proj[(size_t)t * p.p_stride + p.head_col + h] + p.dt_bias[h]));
    for (int i0 = (blockIdx.y * 4 + warp) * 4; i0 < 2 * p.Hk; i0 += gridDim.y * 16) {
        float4 x[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = i0 + j;
            float* at = row + (i < p.Hk ? p.c_q + i * p.dk : p.c_k + (i - p.Hk) * p.dk) + d;
            x[j] = i < 2 * p.Hk && d < p.dk ? *reinterpret_cast<const float4*>(at) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = i0 + j;
            const float ss = warp_sum(fmaf(x[j].w, x[j].w, fmaf(x[j].z, x[j].z, fmaf(x[j].y, x[j].y, x[j].x * x[j].x))));
            const float inv = (i < p.Hk ? q_scale : 1.f) / sqrtf(ss + 1e-6f);
            float* at = row + (i < p.Hk ? p.c_q + i * p.dk : p.c_k + (i - p.Hk) * p.dk) + d;
            if (i < 2 * p.Hk && d < p.dk) *reinterpret_cast<float4*>(at) = make_float4(x[j].x * inv, x[j].y * inv, x[j].z * inv, x[j].w * inv);
        }
    }
    __syncthreads();
    float* arow = p.a + (size_t)t * p.a_stride + p.a_col;
    if (p.a_dk == 1)
        for (int h = blockIdx.y * 128 + threadIdx.x; h < p.H; h += gridDim.y * 128) arow[h] = decay[h];
    const int quads = p.a_dk / 4;
    for (int i = blockIdx.y * 128 + threadIdx.x; i < p.H * quads; i += gridDim.y * 128) {
        const int h = i / quads;
        float4* at = reinterpret_cast<float4*>(arow) + i;
        if (p.head_col >= 0) { const float g = decay[h]; *at = make_float4(g, g, g, g); continue; }
        const float rate = expf(p.a_log[h]);
        const float4 z = *at, b = *reinterpret_cast<const float4*>(p.dt_bias + 4 * i);
        *at = make_float4(expf(-rate * softplus_f(z.x + b.x)), expf(-rate * softplus_f(z.y + b.y)),
                          expf(-rate * softplus_f(z.z + b.z)), expf(-rate * softplus_f(z.w + b.w)));
    }
    for (int h = blockIdx.y * 128 + threadIdx.x; h < p.H; h += gridDim.y * 128)
        p.beta[(size_t)t * p.H + h] = 1.0f / (1.0f + expf(-p.proj[(size_t)t * p.p_stride + p.b_col + h]));
}

extern "C" int idm_delta_prep(float* c, int c_stride, int c_q, int c_k, float* a, int a_stride, int a_col,
                              const float* proj, int p_stride, int b_col, int head_col, const float* dt_bias, const float* a_log,
                              float* beta, int H, int Hk, int dk, int a_dk, int n_tokens, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    IDM_REQUIRE(H > 0 && Hk > 0 && H % Hk == 0 && dk > 0, "delta_prep: %d heads over %d key heads of %d", H, Hk, dk);
    IDM_REQUIRE(a_dk == dk || (a_dk == 1 && head_col >= 0), "delta_prep: %d decays of a head, keys of %d", a_dk, dk);
    DeltaPrepArgs p{c, c_stride, c_q, c_k, a, a_stride, a_col, proj, p_stride, b_col, head_col, dt_bias, a_log, beta, H, Hk, dk, a_dk};
    int split = (296 + n_tokens - 1) / n_tokens;
    const int most = (H * dk + 127) / 128;
    if (split > most) split = most;
    if (split < 1) split = 1;
    const bool vec = dk % 4 == 0 && dk <= 128 && H <= DP_HEADS && c_stride % 4 == 0 && c_q % 4 == 0 && c_k % 4 == 0 &&
                     (a_dk == 1 || (a_stride % 4 == 0 && a_col % 4 == 0 && ((uintptr_t)a & 15) == 0)) && ((uintptr_t)c & 15) == 0 && (head_col >= 0 || ((uintptr_t)dt_bias & 15) == 0);
    idm_launch(vec ? delta_prep_vec_kernel : delta_prep_kernel, dim3(n_tokens, split), dim3(128), 0, stream, p);
    IDM_LAUNCH_CHECK("delta_prep");
    return 0;
}

// ------------------------------------------------------------------ the recurrence
// A block owns (sequence, head, 16 columns of S).  Eight threads share a column: thread r of them keeps rows
// [r RP, (r + 1) RP) of it in registers, and the eight add their parts of a column's sums by three shuffles.  The
// next token's q, k, g are loaded while this token's sums are on their way.
struct DeltaScanArgs {
    const float* c; int c_stride, c_q, c_k, c_v;      // q, k unit vectors [Hk, dk]; v [H, dv]
    const float* g; int g_stride, g_col;              // decays [H, dk]
    const float* beta;                                // [N, H]
    float* state; long long state_stride;             // state + slot * state_stride : [H][dv][dk]
    float* o; int o_stride;                           // o[t, h * dv + j]
    const int* cu_q; const int* slots;
    int H, Hk, dk, dv;
};

#define DS_COLS 16

template <int RP>
__global__ void __launch_bounds__(DS_COLS * 8) delta_scan_kernel(DeltaScanArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    const int s = blockIdx.z, h = blockIdx.y, hk = h / (a.H / a.Hk);
    const int r = threadIdx.x & 7, j = blockIdx.x * DS_COLS + (threadIdx.x >> 3);
    const bool col = j < a.dv;
    const int row0 = r * RP;
    const int t0 = a.cu_q[s], t1 = a.cu_q[s + 1];
    float* sp = a.state + (size_t)a.slots[s] * a.state_stride + ((size_t)h * a.dv + (col ? j : 0)) * a.dk + row0;
    float S[RP], kq[3][RP];                           // (k, q, g of the token at hand)
    const bool vec = a.dk % 4 == 0 && ((uintptr_t)sp & 15) == 0;      // a thread's rows as 16-byte pieces
#pragma unroll
    for (int i = 0; i < RP; i += 4) {
        if (vec) {
            const float4 x = (col && row0 + i < a.dk) ? *reinterpret_cast<const float4*>(sp + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            S[i] = x.x; S[i + 1] = x.y; S[i + 2] = x.z; S[i + 3] = x.w;
        } else {
#pragma unroll
            for (int e = i; e < i + 4; ++e) S[e] = (col && row0 + e < a.dk) ? sp[e] : 0.f;
        }
    }

    auto load = [&](int t, float (&dst)[3][RP]) {
        const float* kp = a.c + (size_t)t * a.c_stride + a.c_k + hk * a.dk + row0;
        const float* qp = a.c + (size_t)t * a.c_stride + a.c_q + hk * a.dk + row0;
        const float* gp = a.g + (size_t)t * a.g_stride + a.g_col + h * a.dk + row0;
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            const bool live = row0 + i < a.dk;
            dst[0][i] = live ? kp[i] : 0.f;
            dst[1][i] = live ? qp[i] : 0.f;
            dst[2][i] = live ? gp[i] : 1.f;
        }
    };
    if (t0 < t1) load(t0, kq);
    for (int t = t0; t < t1; ++t) {
        float nx[3][RP];
        if (t + 1 < t1) load(t + 1, nx);
        const float v = col ? a.c[(size_t)t * a.c_stride + a.c_v + h * a.dv + j] : 0.f;
        const float beta = a.beta[(size_t)t * a.H + h];
        float sk = 0.f, sq = 0.f, kk = 0.f;
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            S[i] *= kq[2][i];
            sk = fmaf(S[i], kq[0][i], sk);
            sq = fmaf(S[i], kq[1][i], sq);
            kk = fmaf(kq[0][i], kq[1][i], kk);
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            sk += __shfl_xor_sync(0xffffffffu, sk, o);
            sq += __shfl_xor_sync(0xffffffffu, sq, o);
            kk += __shfl_xor_sync(0xffffffffu, kk, o);
        }
        const float u = beta * (v - sk);
#pragma unroll
        for (int i = 0; i < RP; ++i) S[i] = fmaf(kq[0][i], u, S[i]);
        if (col && r == 0) a.o[(size_t)t * a.o_stride + h * a.dv + j] = fmaf(u, kk, sq);
        if (t + 1 < t1) {
#pragma unroll
            for (int i = 0; i < RP; ++i) { kq[0][i] = nx[0][i]; kq[1][i] = nx[1][i]; kq[2][i] = nx[2][i]; }
        }
    }
    if (col) {
#pragma unroll
        for (int i = 0; i < RP; i += 4) {
            if (vec) {
                if (row0 + i < a.dk) *reinterpret_cast<float4*>(sp + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
            } else {
#pragma unroll
                for (int e = i; e < i + 4; ++e)
                    if (row0 + e < a.dk) sp[e] = S[e];
            }
        }
    }
}

// The same recurrence for portions of many tokens.  Walking a portion token by token from global memory pays a
// load's latency per token; here a block brings DS_TOK tokens' q, k, g, its 16 columns of v and beta into shared
// memory with asynchronous copies, two stages deep, and the walk reads them from there.  Element d = r RP + i of a
// head's q, k or g lies at ((i / 4) 8 + r) 4 + i % 4 of its row, so that the eight threads of a column read 128
// bytes side by side.  The arithmetic and its order are those of the kernel above: both give the same bits.
__device__ __forceinline__ void cp_async_4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

template <int RP>
struct DeltaStage {
    static constexpr int DKP = RP * 8;                          // a head's key size, rounded up to the threads' rows
    static constexpr int TOK = RP <= 16 ? 16 : 8;               // tokens per stage
    static constexpr int ROW = 3 * DKP + DS_COLS + 4;           // k, q, g, v of the block's columns, beta (and 3 unused)
    static constexpr int FLOATS = 2 * TOK * ROW;
};

template <int RP, bool VEC>
__global__ void __launch_bounds__(DS_COLS * 8) delta_scan_staged_kernel(DeltaScanArgs a) {
    using St = DeltaStage<RP>;
    extern __shared__ __align__(16) float ds_smem[];
    pdl_launch_dependents();
    const int s = blockIdx.z, h = blockIdx.y, hk = h / (a.H / a.Hk);
    const int tid = threadIdx.x, r = tid & 7, jl = tid >> 3, j0 = blockIdx.x * DS_COLS, j = j0 + jl;
    const bool col = j < a.dv;
    const int row0 = r * RP;
    // rows past dk are never copied: k = q = 0 and g = 1 there, once for both stages
    for (int e = tid; e < 2 * St::TOK * St::DKP; e += DS_COLS * 8) {
        const int row = e / St::DKP, p = e % St::DKP;
        const int d = (p >> 2 & 7) * RP + (p >> 5) * 4 + (p & 3);
        if (d >= a.dk) {
            float* base = ds_smem + row * St::ROW;
            base[p] = 0.f; base[St::DKP + p] = 0.f; base[2 * St::DKP + p] = 1.f;
        }
    }
    pdl_wait();
    const int t0 = a.cu_q[s], t1 = a.cu_q[s + 1];
    float* sp = a.state + (size_t)a.slots[s] * a.state_stride + ((size_t)h * a.dv + (col ? j : 0)) * a.dk + row0;
    float S[RP];
#pragma unroll
    for (int i = 0; i < RP; ++i) S[i] = (col && row0 + i < a.dk) ? sp[i] : 0.f;

    const int cols = min(DS_COLS, a.dv - j0);
    auto issue = [&](int tb, int stage) {
        const int n = min(St::TOK, t1 - tb);
        float* st = ds_smem + stage * St::TOK * St::ROW;
        if (VEC) {
            const int per = a.dk >> 2, total = n * 3 * per;
            for (int e = tid; e < total; e += DS_COLS * 8) {
                const int tt = e / (3 * per), w = e % (3 * per), which = w / per, d = (w % per) << 2;
                const float* src = which == 2 ? a.g + (size_t)(tb + tt) * a.g_stride + a.g_col + h * a.dk + d
                                              : a.c + (size_t)(tb + tt) * a.c_stride + (which ? a.c_q : a.c_k) + hk * a.dk + d;
                const int rr = d / RP, i = d % RP;
                cp_async_16(st + tt * St::ROW + which * St::DKP + (((i >> 2) * 8 + rr) << 2), src);
            }
        } else {
            const int total = n * 3 * a.dk;
            for (int e = tid; e < total; e += DS_COLS * 8) {
                const int tt = e / (3 * a.dk), w = e % (3 * a.dk), which = w / a.dk, d = w % a.dk;
                const float* src = which == 2 ? a.g + (size_t)(tb + tt) * a.g_stride + a.g_col + h * a.dk + d
                                              : a.c + (size_t)(tb + tt) * a.c_stride + (which ? a.c_q : a.c_k) + hk * a.dk + d;
                const int rr = d / RP, i = d % RP;
                cp_async_4(st + tt * St::ROW + which * St::DKP + (((i >> 2) * 8 + rr) << 2) + (i & 3), src);
            }
        }
        for (int e = tid; e < n * (cols + 1); e += DS_COLS * 8) {
            const int tt = e / (cols + 1), c = e % (cols + 1);
            const float* src = c < cols ? a.c + (size_t)(tb + tt) * a.c_stride + a.c_v + h * a.dv + j0 + c
                                        : a.beta + (size_t)(tb + tt) * a.H + h;
            cp_async_4(st + tt * St::ROW + 3 * St::DKP + (c < cols ? c : DS_COLS), src);
        }
        cp_async_commit();
    };

    const int n_chunks = (t1 - t0 + St::TOK - 1) / St::TOK;
    if (n_chunks > 0) issue(t0, 0);
    for (int ch = 0; ch < n_chunks; ++ch) {
        const int tb = t0 + ch * St::TOK;
        if (ch + 1 < n_chunks) { issue(tb + St::TOK, (ch + 1) & 1); cp_async_wait<1>(); }
        else cp_async_wait<0>();
        __syncthreads();
        const float* st = ds_smem + (ch & 1) * St::TOK * St::ROW;
        const int n = min(St::TOK, t1 - tb);
        for (int tt = 0; tt < n; ++tt) {
            const float* row = st + tt * St::ROW;
            const float v = row[3 * St::DKP + jl], beta = row[3 * St::DKP + DS_COLS];
            float kr[RP];
            float sk = 0.f, sq = 0.f, kk = 0.f;
#pragma unroll
            for (int m = 0; m < RP / 4; ++m) {
                const float4 k4 = *reinterpret_cast<const float4*>(row + ((m * 8 + r) << 2));
                const float4 q4 = *reinterpret_cast<const float4*>(row + St::DKP + ((m * 8 + r) << 2));
                const float4 g4 = *reinterpret_cast<const float4*>(row + 2 * St::DKP + ((m * 8 + r) << 2));
                const float kx[4] = {k4.x, k4.y, k4.z, k4.w}, qx[4] = {q4.x, q4.y, q4.z, q4.w}, gx[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float& Sv = S[m * 4 + i];
                    Sv *= gx[i];
                    sk = fmaf(Sv, kx[i], sk);
                    sq = fmaf(Sv, qx[i], sq);
                    kk = fmaf(kx[i], qx[i], kk);
                    kr[m * 4 + i] = kx[i];
                }
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                sk += __shfl_xor_sync(0xffffffffu, sk, o);
                sq += __shfl_xor_sync(0xffffffffu, sq, o);
                kk += __shfl_xor_sync(0xffffffffu, kk, o);
            }
            const float u = beta * (v - sk);
#pragma unroll
            for (int i = 0; i < RP; ++i) S[i] = fmaf(kr[i], u, S[i]);
            if (col && r == 0) a.o[(size_t)(tb + tt) * a.o_stride + h * a.dv + j] = fmaf(u, kk, sq);
        }
        __syncthreads();
    }
    if (col) {
#pragma unroll
        for (int i = 0; i < RP; ++i)
            if (row0 + i < a.dk) sp[i] = S[i];
    }
}

template <int RP>
static int delta_scan_staged(const DeltaScanArgs& a, dim3 grid, cudaStream_t stream) {
    const size_t smem = (size_t)DeltaStage<RP>::FLOATS * sizeof(float);
    const bool vec = a.dk % 4 == 0 && a.c_stride % 4 == 0 && a.c_q % 4 == 0 && a.c_k % 4 == 0 && a.g_stride % 4 == 0 &&
                     a.g_col % 4 == 0 && ((uintptr_t)a.c & 15) == 0 && ((uintptr_t)a.g & 15) == 0;
    static bool set[2] = {false, false};
    if (!set[vec]) {
        cudaError_t e = vec ? cudaFuncSetAttribute(delta_scan_staged_kernel<RP, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
                            : cudaFuncSetAttribute(delta_scan_staged_kernel<RP, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        IDM_REQUIRE(e == cudaSuccess, "delta_scan: %zu bytes of shared memory were refused (%s)", smem, cudaGetErrorString(e));
        set[vec] = true;
    }
    if (vec) idm_launch(delta_scan_staged_kernel<RP, true>, grid, dim3(DS_COLS * 8), smem, stream, a);
    else idm_launch(delta_scan_staged_kernel<RP, false>, grid, dim3(DS_COLS * 8), smem, stream, a);
    return 0;
}

__device__ __forceinline__ float dot4(float s, float4 a, float4 b) {
    s = fmaf(a.x, b.x, s); s = fmaf(a.y, b.y, s); s = fmaf(a.z, b.z, s);
    return fmaf(a.w, b.w, s);
}

// Few tokens per sequence (single tokens above all), keys of up to 128 in whole pieces of four: bound by the bytes of the state, so a
// thread has eight 16-byte pieces of it on their way.  L lanes have a column (4 L channels) and add its two sums up by a butterfly.
// 64 single tokens, 32 heads of 128 x 64 (134 MB in and out): 22 us, 6.1 TB/s (55 us by the general walk).
// A warp has COLS columns (times 32 / L): eight keep enough bytes on their way where the blocks fill the SMs, two where sequences
// are few and it is the chain of loads, sums and stores that counts; a column's sums are the same either way.  A layer's step with
// 1 / 4 / 16 single tokens takes 23.3 / 24.5 / 32.8 us (by the general walk 23.9 / 28.0 / 40.8).
#define DT_COLS 8
#define DT_FILL 296                    // blocks of eight columns a warp: two an SM
template <int L, int COLS>
__global__ void __launch_bounds__(128, 5) delta_token_kernel(DeltaScanArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int SIDE = 32 / L;                                // columns side by side
    const int s = blockIdx.z, h = blockIdx.y, hk = h / (a.H / a.Hk), lane = threadIdx.x & 31, ln = lane % L;
    const int j0 = (blockIdx.x * 4 + (threadIdx.x >> 5)) * COLS * SIDE + lane / L, d = ln * 4;
    const bool in = d < a.dk;
    const int t0 = a.cu_q[s], t1 = a.cu_q[s + 1];
    float* sp = a.state + (size_t)a.slots[s] * a.state_stride + (size_t)h * a.dv * a.dk + d;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 S[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
        const int j = j0 + i * SIDE;
        S[i] = in && j < a.dv ? *reinterpret_cast<const float4*>(sp + (size_t)j * a.dk) : zero;
    }
    for (int t = t0; t < t1; ++t) {
        const float* row = a.c + (size_t)t * a.c_stride;
        const float4 k = in ? *reinterpret_cast<const float4*>(row + a.c_k + hk * a.dk + d) : zero;
        const float4 q = in ? *reinterpret_cast<const float4*>(row + a.c_q + hk * a.dk + d) : zero;
        const float4 g = in ? *reinterpret_cast<const float4*>(a.g + (size_t)t * a.g_stride + a.g_col + h * a.dk + d) : zero;
        const float beta = a.beta[(size_t)t * a.H + h];
        float v[COLS], ks[COLS], qs[COLS], kq = dot4(0.f, k, q);
#pragma unroll
        for (int i = 0; i < COLS; ++i) {
            const int j = j0 + i * SIDE;
            v[i] = j < a.dv ? row[a.c_v + h * a.dv + j] : 0.f;
            S[i] = make_float4(g.x * S[i].x, g.y * S[i].y, g.z * S[i].z, g.w * S[i].w);
            ks[i] = dot4(0.f, k, S[i]);
            qs[i] = dot4(0.f, q, S[i]);
        }
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) {
            kq += __shfl_xor_sync(0xffffffffu, kq, o);
#pragma unroll
            for (int i = 0; i < COLS; ++i) {
                ks[i] += __shfl_xor_sync(0xffffffffu, ks[i], o);
                qs[i] += __shfl_xor_sync(0xffffffffu, qs[i], o);
            }
        }
        float mine = 0.f;                                       // lane i of a column's lanes stores column i's read-out
#pragma unroll
        for (int i = 0; i < COLS; ++i) {
            const float u = beta * (v[i] - ks[i]);
            S[i] = make_float4(fmaf(k.x, u, S[i].x), fmaf(k.y, u, S[i].y), fmaf(k.z, u, S[i].z), fmaf(k.w, u, S[i].w));
            if (ln == i) mine = fmaf(u, kq, qs[i]);
        }
        const int j = j0 + ln * SIDE;
        if (ln < COLS && j < a.dv) a.o[(size_t)t * a.o_stride + h * a.dv + j] = mine;
    }
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
        const int j = j0 + i * SIDE;
        if (in && j < a.dv) *reinterpret_cast<float4*>(sp + (size_t)j * a.dk) = S[i];
    }
}
template <int L, int COLS>
static void delta_token_launch(const DeltaScanArgs& a, int n_seqs, cudaStream_t stream) {
    constexpr int BLOCK = 4 * COLS * (32 / L);
    idm_launch(delta_token_kernel<L, COLS>, dim3((a.dv + BLOCK - 1) / BLOCK, a.H, n_seqs), dim3(128), 0, stream, a);
}
template <int L>
static void delta_token(const DeltaScanArgs& a, int n_seqs, cudaStream_t stream) {
    constexpr int BLOCK = 4 * DT_COLS * (32 / L);
    if ((long long)((a.dv + BLOCK - 1) / BLOCK) * a.H * n_seqs >= DT_FILL) delta_token_launch<L, DT_COLS>(a, n_seqs, stream);
    else delta_token_launch<L, 2>(a, n_seqs, stream);
}

// ------------------------------------------------------------------ the recurrence in chunks
// Over a chunk of C tokens that starts from the state S0, with G_t the product of the decays up to and including
// token t (per key channel), the walk above unrolls to
//
//   u_t  = beta_t (v_t - S0^T (G_t k_t) - sum_{s<t} A_ts u_s),      A_ts = sum_d k_s[d] k_t[d] G_t[d] / G_s[d]
//   o_t  = S0^T (G_t q_t) + sum_{s<=t} B_ts u_s,                    B_ts = sum_d k_s[d] q_t[d] G_t[d] / G_s[d]
//   S_C  = G_C S0 + sum_s (k_s G_C / G_s) u_s^T
//
// so that the work against the state becomes three products with C independent sums each instead of a chain of C dependent
// steps.  The quotients G_t / G_s are never divided out: they are products of the decays between s and t, in (0, 1], so a
// decay that underflows ends at 0 and nothing overflows.  All of it is 32-bit; the numbers are those of the walk up to the
// order of the sums.  There are two forms (delta_split says which a step takes).

// ---- chunks of 16, one chain: A and B belong to (chunk, head) and not to a column, so a pass of its own makes them for all
// chunks side by side; the triangular system (the u_t, 16 unknowns per column) is solved on the chain's way, in registers.
// It works on the tokens that are there, and its blocks of 65 KB share an SM: the form for steps that fill the SMs.
#define CH_C 16                                                 // tokens per chunk

// ab[(t H + h) 2C ..]: for token s of a chunk, -A_ts for the chunk's tokens t > s (0 elsewhere), then B_ts for t >= s
__global__ void __launch_bounds__(128) delta_pairs_kernel(DeltaScanArgs a, float* __restrict__ ab) {
    __shared__ float sm[3][CH_C][128];
    pdl_launch_dependents();
    pdl_wait();
    const int s = blockIdx.z, h = blockIdx.y, hk = h / (a.H / a.Hk), tid = threadIdx.x;
    const int t0 = a.cu_q[s], t1 = a.cu_q[s + 1], tb = t0 + blockIdx.x * CH_C;
    if (tb >= t1) return;
    const int n = min(CH_C, t1 - tb);
    for (int e = tid; e < n * a.dk; e += 128) {
        const int tt = e / a.dk, d = e % a.dk;
        const float* row = a.c + (size_t)(tb + tt) * a.c_stride + hk * a.dk + d;
        sm[0][tt][d] = row[a.c_k];
        sm[1][tt][d] = row[a.c_q];
        sm[2][tt][d] = a.g[(size_t)(tb + tt) * a.g_stride + a.g_col + h * a.dk + d];
    }
    for (int e = tid; e < n * 2 * CH_C; e += 128)
        ab[((size_t)(tb + e / (2 * CH_C)) * a.H + h) * (2 * CH_C) + e % (2 * CH_C)] = 0.f;
    __syncthreads();
    // a warp takes four tokens s whose rows together are as long as every other warp's; its lanes split the channels
    const int warp = tid >> 5, lane = tid & 31;
#pragma unroll 1
    for (int pass = 0; pass < 4; ++pass) {
        const int ts = pass == 0 ? warp : pass == 1 ? 7 - warp : pass == 2 ? 8 + warp : 15 - warp;
        if (ts >= n) continue;
        float kr[4];                                            // k_s times the decays from s up to the token at hand
#pragma unroll
        for (int i = 0; i < 4; ++i) kr[i] = lane + 32 * i < a.dk ? sm[0][ts][lane + 32 * i] : 0.f;
        float* out = ab + ((size_t)(tb + ts) * a.H + h) * (2 * CH_C);
        for (int t = ts; t < n; ++t) {
            float pa = 0.f, pb = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int d = lane + 32 * i;
                if (d < a.dk) {
                    if (t > ts) kr[i] *= sm[2][t][d];
                    pa = fmaf(sm[0][t][d], kr[i], pa);
                    pb = fmaf(sm[1][t][d], kr[i], pb);
                }
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                pa += __shfl_xor_sync(0xffffffffu, pa, o);
                pb += __shfl_xor_sync(0xffffffffu, pb, o);
            }
            if (lane == 0) {
                if (t > ts) out[t] = -pa;
                out[CH_C + t] = pb;
            }
        }
    }
}

// The chain: a block owns (sequence, head, 16 columns of S), a warp four of the columns, lane L rows
// [L RP, (L + 1) RP) of each.  Four columns a warp, because what a warp reads from shared memory (a token's scaled k or
// q) then serves four sums, and four independent chains keep one warp per scheduler busy.  Per chunk: (1) the threads
// turn the staged k, q, g in place into k G_C / G_t, q G_t, k G_t, a thread per channel and group of tokens, the
// groups' products joined through shared memory; (2) the warp lays its columns of S0 into shared memory, and lane t
// sums S0^T (G_t k_t) for token t's correction, lane 16 + t S0^T (G_t q_t) for its read-out; (3) the triangular system
// runs down the lanes: u_s goes from lane s to all, lane L adds row s's entry L of [-A | B] times u_s to its sum; (4)
// lanes 16.. store the read-outs, all lanes bring their rows of S behind the chunk.
#define CH_NC 4                                                 // columns per warp
template <int RP>
struct DeltaChain {
    static constexpr int DKP = RP * 32, NT = DS_COLS / CH_NC * 32;
    static constexpr int NG = NT / DKP < 1 ? 1 : NT / DKP;      // groups of tokens in step (1)
    static constexpr int V_AT = 3 * DKP, BETA_AT = V_AT + DS_COLS, AB_AT = BETA_AT + 4;
    static constexpr int ROW = AB_AT + 2 * CH_C;                // k, q, g, v of the block's columns, beta, -A and B
    static constexpr int GC_AT = 2 * CH_C * ROW;                // the chunk's whole decay, behind the two stages
    static constexpr int GP_AT = GC_AT + DKP;                   // the token groups' decays
    static constexpr int SW_AT = GP_AT + NG * DKP;              // the block's columns of S
    static constexpr int FLOATS = SW_AT + DS_COLS * DKP;
    static_assert(DKP <= NT && CH_C % NG == 0, "a thread per channel, whole groups of tokens");
};

template <int RP>
__device__ __forceinline__ void load_rows(const float* p, float (&x)[RP]) {
    if constexpr (RP == 4) { const float4 v = *reinterpret_cast<const float4*>(p); x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w; }
    else if constexpr (RP == 2) { const float2 v = *reinterpret_cast<const float2*>(p); x[0] = v.x; x[1] = v.y; }
    else x[0] = *p;
}

template <int RP, bool VEC>
__global__ void __launch_bounds__(DeltaChain<RP>::NT) delta_chain_kernel(DeltaScanArgs a, const float* __restrict__ ab) {
    using L = DeltaChain<RP>;
    constexpr int C = CH_C, NT = L::NT, NC = CH_NC, NW = NT / 32;
    extern __shared__ __align__(16) float ds_smem[];
    pdl_launch_dependents();
    const int s = blockIdx.z, h = blockIdx.y, hk = h / (a.H / a.Hk);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, j0 = blockIdx.x * DS_COLS, jw = warp * NC;
    const int row0 = lane * RP;
    for (int e = tid; e < 2 * C * L::DKP; e += NT) {            // channels past dk: k = q = 0, g = 1, never copied
        const int row = e / L::DKP, p = e % L::DKP;
        if (p >= a.dk) {
            float* base = ds_smem + row * L::ROW;
            base[p] = 0.f; base[L::DKP + p] = 0.f; base[2 * L::DKP + p] = 1.f;
        }
    }
    pdl_wait();
    const int t0 = a.cu_q[s], t1 = a.cu_q[s + 1];
    float* sp = a.state + (size_t)a.slots[s] * a.state_stride + ((size_t)h * a.dv + j0 + jw) * a.dk + row0;
    float S[NC][RP];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int i = 0; i < RP; ++i) S[c][i] = (j0 + jw + c < a.dv && row0 + i < a.dk) ? sp[(size_t)c * a.dk + i] : 0.f;

    const int cols = min(DS_COLS, a.dv - j0);
    auto issue = [&](int tb, int stage) {
        const int n = min(C, t1 - tb);
        for (int tt = warp; tt < n; tt += NW) {
            const int t = tb + tt;
            float* row = ds_smem + (stage * C + tt) * L::ROW;
            const float* kp = a.c + (size_t)t * a.c_stride + hk * a.dk;
            const float* gp = a.g + (size_t)t * a.g_stride + a.g_col + h * a.dk;
            if (VEC) {
                for (int d = lane * 4; d < a.dk; d += 128) {
                    cp_async_16(row + d, kp + a.c_k + d);
                    cp_async_16(row + L::DKP + d, kp + a.c_q + d);
                    cp_async_16(row + 2 * L::DKP + d, gp + d);
                }
            } else {
                for (int d = lane; d < a.dk; d += 32) {
                    cp_async_4(row + d, kp + a.c_k + d);
                    cp_async_4(row + L::DKP + d, kp + a.c_q + d);
                    cp_async_4(row + 2 * L::DKP + d, gp + d);
                }
            }
            if (lane < cols) cp_async_4(row + L::V_AT + lane, a.c + (size_t)t * a.c_stride + a.c_v + h * a.dv + j0 + lane);
            else if (lane == 16) cp_async_4(row + L::BETA_AT, a.beta + (size_t)t * a.H + h);
            else if (lane >= 24) cp_async_16(row + L::AB_AT + (lane - 24) * 4, ab + ((size_t)t * a.H + h) * (2 * C) + (lane - 24) * 4);
        }
        cp_async_commit();
    };

    const int n_chunks = (t1 - t0 + C - 1) / C;
    if (n_chunks > 0) issue(t0, 0);
    for (int ch = 0; ch < n_chunks; ++ch) {
        const int tb = t0 + ch * C;
        if (ch + 1 < n_chunks) { issue(tb + C, (ch + 1) & 1); cp_async_wait<1>(); }
        else cp_async_wait<0>();
        float* st = ds_smem + (ch & 1) * C * L::ROW;
        const int n = min(C, t1 - tb);
        // a last chunk of fewer tokens: the missing ones write nothing (k = 0, beta = 0) and decay nothing (g = 1)
        for (int e = tid; e < (C - n) * L::ROW; e += NT) {
            const int c = e % L::ROW;
            st[(n + e / L::ROW) * L::ROW + c] = (c >= 2 * L::DKP && c < 3 * L::DKP) ? 1.f : 0.f;
        }
        __syncthreads();
        // (1) in place, per channel: k -> k G_C / G_t, q -> q G_t, g -> k G_t; and G_C.  Thread (channel, group of tokens).
        {
            constexpr int TPG = C / L::NG;
            const int p = tid % L::DKP, grp = tid / L::DKP;
            float gg[TPG], kk[TPG], qq[TPG];
            if (grp < L::NG) {
                float prod = 1.f;
#pragma unroll
                for (int i = 0; i < TPG; ++i) {
                    const float* row = st + (TPG * grp + i) * L::ROW;
                    gg[i] = row[2 * L::DKP + p]; kk[i] = row[p]; qq[i] = row[L::DKP + p];
                    prod *= gg[i];
                }
                if (L::NG > 1) ds_smem[L::GP_AT + grp * L::DKP + p] = prod;
            }
            if (L::NG > 1) __syncthreads();
            if (grp < L::NG) {
                float G = 1.f, suf = 1.f;
                if (L::NG > 1) {
#pragma unroll
                    for (int o = 0; o < L::NG; ++o) {
                        const float x = ds_smem[L::GP_AT + o * L::DKP + p];
                        if (o < grp) G *= x;
                        if (o > grp) suf *= x;
                    }
                }
#pragma unroll
                for (int i = 0; i < TPG; ++i) {
                    float* row = st + (TPG * grp + i) * L::ROW;
                    G *= gg[i];
                    row[2 * L::DKP + p] = kk[i] * G;
                    row[L::DKP + p] = qq[i] * G;
                }
                if (grp == L::NG - 1) ds_smem[L::GC_AT + p] = G;
#pragma unroll
                for (int i = TPG - 1; i >= 0; --i) {
                    st[(TPG * grp + i) * L::ROW + p] = kk[i] * suf;
                    suf *= gg[i];
                }
            }
        }
        __syncthreads();
        // (2) what the state before the chunk gives token t's correction (lane t) and read-out (lane 16 + t): the columns
        // go through shared memory, and a lane walks all of them against its token's G_t k_t or G_t q_t
        float x[NC];
        {
            float* sw = ds_smem + L::SW_AT + jw * L::DKP;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if constexpr (RP == 4) *reinterpret_cast<float4*>(sw + c * L::DKP + row0) = make_float4(S[c][0], S[c][1], S[c][2], S[c][3]);
                else if constexpr (RP == 2) *reinterpret_cast<float2*>(sw + c * L::DKP + row0) = make_float2(S[c][0], S[c][1]);
                else sw[c * L::DKP + row0] = S[c][0];
            }
            __syncwarp();
            const float* xr = st + (lane & 15) * L::ROW + (lane < 16 ? 2 * L::DKP : L::DKP);
            float acc[NC][4];
#pragma unroll
            for (int c = 0; c < NC; ++c) acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.f;
#pragma unroll 8
            for (int m = 0; m < L::DKP / 4; ++m) {
                const float4 xv = *reinterpret_cast<const float4*>(xr + 4 * m);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const float4 sv = *reinterpret_cast<const float4*>(sw + c * L::DKP + 4 * m);
                    acc[c][0] = fmaf(xv.x, sv.x, acc[c][0]); acc[c][1] = fmaf(xv.y, sv.y, acc[c][1]);
                    acc[c][2] = fmaf(xv.z, sv.z, acc[c][2]); acc[c][3] = fmaf(xv.w, sv.w, acc[c][3]);
                }
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) x[c] = (acc[c][0] + acc[c][1]) + (acc[c][2] + acc[c][3]);
        }
        // (3) lane t < 16: v_t minus the sum, times beta_t when its turn comes; lane 16 + t: the read-out so far
        float u[NC][C];
        const float* mine = st + (lane & 15) * L::ROW;
        const float beta = lane < 16 ? mine[L::BETA_AT] : 0.f;
        if (lane < 16) {
#pragma unroll
            for (int c = 0; c < NC; ++c) x[c] = (j0 + jw + c < a.dv ? mine[L::V_AT + jw + c] : 0.f) - x[c];
        }
#pragma unroll
        for (int q = 0; q < C; ++q) {
            const float coef = st[q * L::ROW + L::AB_AT + lane];
            const bool behind = lane < 16 ? lane > q : lane - 16 >= q;      // (the tokens before q are not touched, whatever u_q is)
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                u[c][q] = __shfl_sync(0xffffffffu, beta * x[c], q);
                if (behind) x[c] = fmaf(coef, u[c][q], x[c]);
            }
        }
        if (lane >= 16 && lane - 16 < n) {
            float* dst = a.o + (size_t)(tb + lane - 16) * a.o_stride + h * a.dv + j0 + jw;
#pragma unroll
            for (int c = 0; c < NC; ++c)
                if (j0 + jw + c < a.dv) dst[c] = x[c];
        }
        // (4) the state behind the chunk
        {
            float gc[RP];
            load_rows<RP>(ds_smem + L::GC_AT + row0, gc);
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int i = 0; i < RP; ++i) S[c][i] *= gc[i];
        }
#pragma unroll
        for (int t = 0; t < C; ++t) {
            float kt[RP];
            load_rows<RP>(st + t * L::ROW + row0, kt);
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int i = 0; i < RP; ++i) S[c][i] = fmaf(kt[i], u[c][t], S[c][i]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int i = 0; i < RP; ++i)
            if (j0 + jw + c < a.dv && row0 + i < a.dk) sp[(size_t)c * a.dk + i] = S[c][i];
}

template <int RP>
static int delta_scan_chain(const DeltaScanArgs& a, float* ab, dim3 grid, int max_tokens, cudaStream_t stream) {
    const size_t smem = (size_t)DeltaChain<RP>::FLOATS * sizeof(float);
    const bool vec = a.dk % 4 == 0 && a.c_stride % 4 == 0 && a.c_q % 4 == 0 && a.c_k % 4 == 0 && a.g_stride % 4 == 0 &&
                     a.g_col % 4 == 0 && ((uintptr_t)a.c & 15) == 0 && ((uintptr_t)a.g & 15) == 0;
    const cudaError_t e = vec ? cudaFuncSetAttribute(delta_chain_kernel<RP, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
                              : cudaFuncSetAttribute(delta_chain_kernel<RP, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    IDM_REQUIRE(e == cudaSuccess, "delta_scan: %zu bytes of shared memory were refused (%s)", smem, cudaGetErrorString(e));
    idm_launch(delta_pairs_kernel, dim3((max_tokens + CH_C - 1) / CH_C, grid.y, grid.z), dim3(128), 0, stream, a, ab);
    if (vec) idm_launch(delta_chain_kernel<RP, true>, grid, dim3(DeltaChain<RP>::NT), smem, stream, a, (const float*)ab);
    else idm_launch(delta_chain_kernel<RP, false>, grid, dim3(DeltaChain<RP>::NT), smem, stream, a, (const float*)ab);
    return 0;
}

// ---- chunks of 32, split: the u_t are a triangular system whose right-hand sides are v_t and, row by row of S0, G_t k_t: with X
// the solutions for those, u = X_v - X_k S0.  So everything but S0 belongs to (chunk, head) and not to a column or to what came
// before: delta_chunk_kernel makes it for all chunks side by side (X_k, X_v, G_t q_t, k_s G_C / G_s, B, G_C), and the chain that is
// left (delta_walk_kernel) is products with S0 and with u.  (The decays between s and t: inside half a chunk multiplied up from s,
// across its middle the product up to the middle times the product from there.)  A walk's block has an SM to itself.
//
// A prompt of 2 048 tokens, 32 heads of 128 x 64: 257 us the chunks (two windows), 230 the walk; the chain of chunks of 16 takes
// 408 + 75 for its pairs.
#define DC_C 32                                                 // tokens per chunk
#define DC_H (DC_C / 2)
#define DC_THREADS 256
#define DC_DKP 128                                              // channels of a key's row, rounded up (keys of 65 to 128)
#define DC_ROW 36                                               // a row of C numbers in shared memory and scratch
struct DeltaChunk {
    static constexpr int LD = DC_DKP + 4;                          // a row of channels: eight rows' 16-byte reads in different places
    // a chunk's numbers in scratch, in floats: X_k, G q, k G_C / G (each [C][LD]), B [C][DC_ROW], G_C, then X_v by groups of 16 columns
    static constexpr int TILE = DC_C * LD;
    static constexpr int B_AT = 3 * TILE, GC_AT = B_AT + DC_C * DC_ROW, XV_AT = GC_AT + DC_DKP;
    static constexpr int XV = DC_C * DS_COLS;
    static constexpr int BUF = XV_AT + XV;                      // a stage of the walk: one group of columns
    static constexpr int CHUNK_SMEM = (3 * TILE + 2 * DC_C * DC_ROW + 2 * DC_DKP + DC_C) * 4;
    static constexpr int WALK_SMEM = (2 * BUF + DS_COLS * LD + DC_C * (DS_COLS + 4)) * 4;
};
__host__ __device__ __forceinline__ int delta_chunk_floats(int dv) {
    return 3 * DC_C * (DC_DKP + 4) + DC_C * DC_ROW + DC_DKP + (dv + DS_COLS - 1) / DS_COLS * DC_C * DS_COLS;
}

// Chunks first, first + 1, ... (gridDim.x of them) of every sequence and head; chunk c of sequence s goes to scratch + (s * gridDim.x + c -
// first) * H + h.
__global__ void __launch_bounds__(DC_THREADS, 2) delta_chunk_kernel(DeltaScanArgs a, float* __restrict__ scratch, int first) {
    using L = DeltaChunk;
    constexpr int C = DC_C, LD = L::LD;
    extern __shared__ __align__(16) float ds_smem[];
    pdl_launch_dependents();
    pdl_wait();
    float* sk = ds_smem;                                        // k; then k times the decays behind it in its half
    float* sq = sk + L::TILE;                                   // q; then q times the decays up to it in its half
    float* sg = sq + L::TILE;                                   // the decays; then k times the decays up to it in its half
    float* sA = sg + L::TILE;                                   // [t][s]
    float* sB = sA + C * DC_ROW;
    float* sG = sB + C * DC_ROW;                                // the halves' whole decays [2][DC_DKP]
    float* sbeta = sG + 2 * DC_DKP;
    const int s = blockIdx.z, h = blockIdx.y, hk = h / (a.H / a.Hk), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int t1 = a.cu_q[s + 1], tb = a.cu_q[s] + (first + (int)blockIdx.x) * C;
    if (tb >= t1) return;
    const int n = min(C, t1 - tb);
    float* out = scratch + (((size_t)s * gridDim.x + blockIdx.x) * a.H + h) * delta_chunk_floats(a.dv);

    // missing tokens and channels write nothing (k = q = 0, beta = 0) and decay nothing (g = 1)
#pragma unroll 4
    for (int e = tid; e < C * DC_DKP; e += DC_THREADS) {
        const int t = e / DC_DKP, d = e % DC_DKP;
        const bool in = t < n && d < a.dk;
        const float* row = a.c + (size_t)(tb + t) * a.c_stride + hk * a.dk + d;
        sk[t * LD + d] = in ? row[a.c_k] : 0.f;
        sq[t * LD + d] = in ? row[a.c_q] : 0.f;
        sg[t * LD + d] = in ? a.g[(size_t)(tb + t) * a.g_stride + a.g_col + h * a.dk + d] : 1.f;
    }
    if (tid < C) sbeta[tid] = tid < n ? a.beta[(size_t)(tb + tid) * a.H + h] : 0.f;
    for (int e = tid; e < 2 * C * DC_ROW; e += DC_THREADS) sA[e] = 0.f;                // (and B behind it)
    __syncthreads();

    // pairs inside a half: a warp has tokens s = w and 15 - w of both halves, its lanes the channels; k_s times the decays from s on
    // meets k_t and q_t
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const int base = (i & 1) * DC_H, ts = base + (i < 2 ? warp : DC_H - 1 - warp);
        constexpr int PER = DC_DKP / 32;
        float kr[PER];
#pragma unroll
        for (int m = 0; m < PER; ++m) kr[m] = sk[ts * LD + lane + 32 * m];
        for (int t = ts; t < base + DC_H; ++t) {
            float pa = 0.f, pb = 0.f;
#pragma unroll
            for (int m = 0; m < PER; ++m) {
                const int d = lane + 32 * m;
                if (t > ts) kr[m] *= sg[t * LD + d];
                pa = fmaf(kr[m], sk[t * LD + d], pa);
                pb = fmaf(kr[m], sq[t * LD + d], pb);
            }
            pa = warp_sum(pa); pb = warp_sum(pb);
            if (lane == 0) {
                if (t > ts) sA[t * DC_ROW + ts] = pa;
                sB[t * DC_ROW + ts] = pb;
            }
        }
    }
    __syncthreads();
    // in place, a thread per channel and half: k behind, q and k up to a token
    for (int e = tid; e < 2 * DC_DKP; e += DC_THREADS) {
        const int p = e % DC_DKP, t0 = e / DC_DKP * DC_H;
        float g[DC_H], k[DC_H], G = 1.f, suf = 1.f;
#pragma unroll
        for (int i = 0; i < DC_H; ++i) {
            g[i] = sg[(t0 + i) * LD + p]; k[i] = sk[(t0 + i) * LD + p];
            G *= g[i];
            sg[(t0 + i) * LD + p] = k[i] * G;
            sq[(t0 + i) * LD + p] *= G;
        }
        sG[e] = G;
#pragma unroll
        for (int i = DC_H - 1; i >= 0; --i) { sk[(t0 + i) * LD + p] = k[i] * suf; suf *= g[i]; }
    }
    __syncthreads();
    // pairs across the middle: 64 tiles of 2 x 2, four threads a tile with a quarter of the channels' pieces each
    {
        const int tile = tid >> 2, kg = tid & 3, tr = DC_H + (tile >> 3) * 2, sr = (tile & 7) * 2;
        float pa[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, pb[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 4
        for (int d = kg * 4; d < DC_DKP; d += 16) {
            float4 k4[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) k4[j] = *reinterpret_cast<const float4*>(sk + (sr + j) * LD + d);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float4 kt = *reinterpret_cast<const float4*>(sg + (tr + i) * LD + d);
                const float4 qt = *reinterpret_cast<const float4*>(sq + (tr + i) * LD + d);
#pragma unroll
                for (int j = 0; j < 2; ++j) { pa[i][j] = dot4(pa[i][j], kt, k4[j]); pb[i][j] = dot4(pb[i][j], qt, k4[j]); }
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
#pragma unroll
                for (int m = 1; m < 4; m <<= 1) {
                    pa[i][j] += __shfl_xor_sync(0xffffffffu, pa[i][j], m);
                    pb[i][j] += __shfl_xor_sync(0xffffffffu, pb[i][j], m);
                }
                if (kg == 0) { sA[(tr + i) * DC_ROW + sr + j] = pa[i][j]; sB[(tr + i) * DC_ROW + sr + j] = pb[i][j]; }
            }
    }
    __syncthreads();
    // what needs no solving goes out: G q, k G_C / G, B, G_C
    for (int e = tid; e < C * DC_DKP; e += DC_THREADS) {
        const int t = e / DC_DKP, d = e % DC_DKP;
        out[L::TILE + t * LD + d] = sq[t * LD + d] * (t < DC_H ? 1.f : sG[d]);
        out[2 * L::TILE + t * LD + d] = sk[t * LD + d] * (t < DC_H ? sG[DC_DKP + d] : 1.f);
    }
    for (int e = tid; e < C * DC_ROW; e += DC_THREADS) out[L::B_AT + e] = sB[e];
    for (int e = tid; e < DC_DKP; e += DC_THREADS) out[L::GC_AT + e] = sG[e] * sG[DC_DKP + e];
    // the triangular system, a thread per right-hand side: channels of G k, then columns of v
    const int vcols = (a.dv + DS_COLS - 1) / DS_COLS * DS_COLS;
    for (int col = tid; col < DC_DKP + vcols; col += DC_THREADS) {
        const int j = col - DC_DKP;
        float x[C];
#pragma unroll
        for (int t = 0; t < C; ++t) {
            float r;
            if (col < DC_DKP) r = sg[t * LD + col] * (t < DC_H ? 1.f : sG[col]);
            else r = t < n && j < a.dv ? a.c[(size_t)(tb + t) * a.c_stride + a.c_v + h * a.dv + j] : 0.f;
            float sum[2] = {0.f, 0.f};
#pragma unroll
            for (int i = 0; i < t; i += 4) {                    // (entries from t on are 0, their x are not made yet)
                const float4 c4 = *reinterpret_cast<const float4*>(sA + t * DC_ROW + i);
                sum[0] = fmaf(c4.x, x[i], sum[0]);
                if (i + 1 < t) sum[1] = fmaf(c4.y, x[i + 1], sum[1]);
                if (i + 2 < t) sum[0] = fmaf(c4.z, x[i + 2], sum[0]);
                if (i + 3 < t) sum[1] = fmaf(c4.w, x[i + 3], sum[1]);
            }
            x[t] = sbeta[t] * (r - (sum[0] + sum[1]));
        }
        float* dst = col < DC_DKP ? out + col : out + L::XV_AT + j / DS_COLS * L::XV + j % DS_COLS;
        const int step = col < DC_DKP ? LD : DS_COLS;
#pragma unroll
        for (int t = 0; t < C; ++t) dst[t * step] = x[t];
    }
}

// The chain: a block owns (sequence, head, 16 columns of S) and walks the chunks of one launch from and to the state.  S lies
// transposed in shared memory, a chunk's numbers come by asynchronous copies one chunk ahead.  Per chunk: (1) X_k S0 and (G q) S0, 64 x
// 16 sums in tiles of 4 x 4, four threads a tile with every fourth piece of four channels; u = X_v - X_k S0 to shared memory; (2) half of
// the block brings S behind the chunk, the other half adds B u to its read-outs and stores them.
__global__ void __launch_bounds__(DC_THREADS) delta_walk_kernel(DeltaScanArgs a, const float* __restrict__ scratch, int first, int count) {
    using L = DeltaChunk;
    constexpr int C = DC_C, LD = L::LD, LU = DS_COLS + 4;
    extern __shared__ __align__(16) float ds_smem[];
    pdl_launch_dependents();
    float* sS = ds_smem + 2 * L::BUF;                           // [16 columns][LD]
    float* sU = sS + DS_COLS * LD;                              // [C][LU]
    const int s = blockIdx.z, h = blockIdx.y, grp = blockIdx.x, j0 = grp * DS_COLS, tid = threadIdx.x;
    pdl_wait();
    const int t0 = a.cu_q[s], t1 = a.cu_q[s + 1];
    const int chunks = min(count, (t1 - t0 + C - 1) / C - first);
    if (chunks <= 0) return;
    const size_t per = delta_chunk_floats(a.dv);
    const float* src = scratch + ((size_t)s * count * a.H + h) * per;
    auto issue = [&](int ch) {
        const float* from = src + (size_t)ch * a.H * per;
        float* to = ds_smem + (ch & 1) * L::BUF;
        for (int e = tid * 4; e < L::BUF; e += DC_THREADS * 4)  // (the columns' part of X_v lies further on)
            cp_async_16(to + e, e < L::XV_AT ? from + e : from + e + (size_t)grp * L::XV);
        cp_async_commit();
    };
    issue(0);
    float* sp = a.state + (size_t)a.slots[s] * a.state_stride + ((size_t)h * a.dv + j0) * a.dk;
    const int cols = min(DS_COLS, a.dv - j0);
    for (int e = tid; e < DS_COLS * DC_DKP; e += DC_THREADS) {
        const int j = e / DC_DKP, d = e % DC_DKP;
        sS[j * LD + d] = j < cols && d < a.dk ? sp[(size_t)j * a.dk + d] : 0.f;
    }
    const int tile = tid >> 2, kg = tid & 3, row = (tile >> 2) * 4, col = (tile & 3) * 4;     // rows 0..31 of X_k, 32..63 of G q
    for (int ch = 0; ch < chunks; ++ch) {
        if (ch + 1 < chunks) { issue(ch + 1); cp_async_wait<1>(); }
        else cp_async_wait<0>();
        __syncthreads();                                        // the chunk's numbers and S are there
        const float* st = ds_smem + (ch & 1) * L::BUF;
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 4
        for (int d = kg * 4; d < DC_DKP; d += 16) {
            float4 x4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) x4[i] = *reinterpret_cast<const float4*>(st + (row + i) * LD + d);   // (G q lies right behind X_k)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 s4 = *reinterpret_cast<const float4*>(sS + (col + j) * LD + d);
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[i][j] = dot4(acc[i][j], x4[i], s4);
            }
        }
#pragma unroll
        for (int m = 1; m < 4; m <<= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] += __shfl_xor_sync(0xffffffffu, acc[i][j], m);
        float mine[4];                                          // row kg of the tile
#pragma unroll
        for (int j = 0; j < 4; ++j) mine[j] = kg == 0 ? acc[0][j] : kg == 1 ? acc[1][j] : kg == 2 ? acc[2][j] : acc[3][j];
        const int t = (row + kg) % C;
        if (row < C) {
            const float4 v = *reinterpret_cast<const float4*>(st + L::XV_AT + t * DS_COLS + col);
            *reinterpret_cast<float4*>(sU + t * LU + col) = make_float4(v.x - mine[0], v.y - mine[1], v.z - mine[2], v.w - mine[3]);
        }
        __syncthreads();                                        // u is there, everyone has read S
        if (row < C) {
            // S <- G_C S + (k G_C / G)^T u: four channels and DC_DKP / 32 columns a thread
            constexpr int NC = DC_DKP / 32;
            const int d = tid % (DC_DKP / 4) * 4, c0 = tid / (DC_DKP / 4) * NC;
            float4 n4[NC];
            const float4 gc = *reinterpret_cast<const float4*>(st + L::GC_AT + d);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float4 o = *reinterpret_cast<const float4*>(sS + (c0 + c) * LD + d);
                n4[c] = make_float4(o.x * gc.x, o.y * gc.y, o.z * gc.z, o.w * gc.w);
            }
#pragma unroll 8
            for (int i = 0; i < C; ++i) {
                const float4 k4 = *reinterpret_cast<const float4*>(st + 2 * L::TILE + i * LD + d);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const float u = sU[i * LU + c0 + c];
                    n4[c].x = fmaf(k4.x, u, n4[c].x); n4[c].y = fmaf(k4.y, u, n4[c].y);
                    n4[c].z = fmaf(k4.z, u, n4[c].z); n4[c].w = fmaf(k4.w, u, n4[c].w);
                }
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) *reinterpret_cast<float4*>(sS + (c0 + c) * LD + d) = n4[c];
        } else {
            const float* br = st + L::B_AT + t * DC_ROW;
            for (int i = 0; i <= t; i += 4) {                   // (entries behind t are 0, their u are numbers of later tokens: left out)
                const float4 b4 = *reinterpret_cast<const float4*>(br + i);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (i + e > t) break;
                    const float b = e == 0 ? b4.x : e == 1 ? b4.y : e == 2 ? b4.z : b4.w;
                    const float4 u = *reinterpret_cast<const float4*>(sU + (i + e) * LU + col);
                    mine[0] = fmaf(b, u.x, mine[0]); mine[1] = fmaf(b, u.y, mine[1]);
                    mine[2] = fmaf(b, u.z, mine[2]); mine[3] = fmaf(b, u.w, mine[3]);
                }
            }
            const int tt = t0 + (first + ch) * C + t;
            if (tt < t1) {
                float* dst = a.o + (size_t)tt * a.o_stride + h * a.dv + j0 + col;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (col + j < cols) dst[j] = mine[j];
            }
        }
        __syncthreads();                                        // S is behind the chunk; its numbers' place is free
    }
    for (int e = tid; e < DS_COLS * DC_DKP; e += DC_THREADS) {
        const int j = e / DC_DKP, d = e % DC_DKP;
        if (j < cols && d < a.dk) sp[(size_t)j * a.dk + d] = sS[j * LD + d];
    }
}

// Which form a step of more than 4 tokens takes: split where the walk's blocks (an SM each) all run at once, the longest portion has more
// than four chunks of 32, and the keys are wider than 64; else the chain.  Measured, us of the chain / split, keys of 128, values of 64:
//   one sequence, 32 heads (128 blocks): 32 tokens 24 / 31, 64 30 / 34, 128 47 / 42, 256 92 / 57, 1 024 245 / 246, 2 048 538 / 487, 8 192
//   1 914 / 1 889; 4 heads: 64 28 / 31, 128 41 / 38, 256 66 / 51, 2 048 425 / 245, 8 192 1 670 / 1 002;
//   more blocks than SMs: 48 heads (192 blocks) 512 tokens 181 / 215, 64 heads 215 / 250, 2 048 769 / 974; 3 x 1 500 tokens of 64 heads
//   1 394 / 2 263; 8 x 40 120 / 276; 2 048 tokens of 32 heads among 60 single tokens 921 / 3 756;
//   keys of 64, 32 heads: 512 tokens 171 / 117, 1 024 198 / 241, 4 096 772 / 1 032.
static bool delta_split(int n_seqs, int H, int dk, int dv, int max_tokens) {
    if (dk <= 64 || max_tokens <= 4 * DC_C) return false;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (long long)n_seqs * H * ((dv + DS_COLS - 1) / DS_COLS) <= sms;
}

// Chunks of a launch: as many of every sequence as fit 18 M floats of scratch (a chunk of one head of 128 x 64 is 64 KB, so that a long
// prompt's numbers are read again while they are in the L2), at least one (delta_split: sequences times heads are no more than the SMs).
// The state carries over from launch to launch.
#define DC_SCRATCH (18ll << 20)
static int delta_window(int n_seqs, int H, int dv, int max_tokens) {
    const long long fit = DC_SCRATCH / ((long long)n_seqs * H * delta_chunk_floats(dv)), all = (max_tokens + DC_C - 1) / DC_C;
    return (int)(fit < 1 ? 1 : fit < all ? fit : all);
}

static int delta_scan_split(const DeltaScanArgs& a, float* scratch, int n_seqs, int max_tokens, cudaStream_t stream) {
    using L = DeltaChunk;
    cudaError_t e = cudaFuncSetAttribute(delta_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::CHUNK_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::WALK_SMEM);
    IDM_REQUIRE(e == cudaSuccess, "delta_scan: %d bytes of shared memory were refused (%s)", L::WALK_SMEM, cudaGetErrorString(e));
    const int window = delta_window(n_seqs, a.H, a.dv, max_tokens), groups = (a.dv + DS_COLS - 1) / DS_COLS;
    for (int first = 0; first * DC_C < max_tokens; first += window) {
        idm_launch(delta_chunk_kernel, dim3(window, a.H, n_seqs), dim3(DC_THREADS), L::CHUNK_SMEM, stream, a, scratch, first);
        idm_launch(delta_walk_kernel, dim3(groups, a.H, n_seqs), dim3(DC_THREADS), L::WALK_SMEM, stream, a, (const float*)scratch, first, window);
    }
    return 0;
}

// Floats of scratch that a step of `n_seqs` sequences and `n_tokens` tokens, at most `max_tokens` of one sequence, wants (0: none).
extern "C" long long idm_delta_scan_scratch_floats(int n_seqs, int n_tokens, int H, int dk, int dv, int max_tokens) {
    if (max_tokens <= 4 || dk <= 0 || dk > 128 || dv <= 0 || n_seqs <= 0 || H <= 0) return 0;
    if (!delta_split(n_seqs, H, dk, dv, max_tokens)) return (long long)n_tokens * H * 2 * CH_C;
    return (long long)n_seqs * H * delta_window(n_seqs, H, dv, max_tokens) * delta_chunk_floats(dv);
}

// `max_tokens`: the most tokens any sequence brings to this step; steps of a few tokens walk them straight from
// global memory, longer portions run in chunks (keys of at most 128, with `scratch` of
// idm_delta_scan_scratch_floats) or walk through shared memory.
extern "C" int idm_delta_scan(const float* c, int c_stride, int c_q, int c_k, int c_v, const float* g, int g_stride,
                              int g_col, const float* beta, float* state, long long state_stride, float* o,
                              int o_stride, const int* cu_q, const int* slots, int n_seqs, int H, int Hk, int dk,
                              int dv, int max_tokens, float* scratch, cudaStream_t stream) {
    if (n_seqs == 0) return 0;
    IDM_REQUIRE(H > 0 && Hk > 0 && H % Hk == 0 && dk > 0 && dk <= 256 && dv > 0, "delta_scan: %d heads over %d key heads, "
                "keys of %d (at most 256), values of %d", H, Hk, dk, dv);
    IDM_REQUIRE(state != nullptr && state_stride >= (long long)H * dk * dv, "delta_scan: a slot's state must hold %d x %d x %d floats",
                H, dv, dk);
    IDM_REQUIRE(n_seqs <= 65535 && H <= 65535, "delta_scan: %d sequences, %d heads in one launch", n_seqs, H);
    DeltaScanArgs a{c, c_stride, c_q, c_k, c_v, g, g_stride, g_col, beta, state, state_stride, o, o_stride, cu_q, slots,
                    H, Hk, dk, dv};
    const dim3 grid((dv + DS_COLS - 1) / DS_COLS, H, n_seqs), block(DS_COLS * 8);
    if (max_tokens > 4 && dk <= 128 && scratch != nullptr) {
        IDM_REQUIRE(((uintptr_t)scratch & 15) == 0, "delta_scan: scratch at %p", (void*)scratch);
        const int rc = delta_split(n_seqs, H, dk, dv, max_tokens) ? delta_scan_split(a, scratch, n_seqs, max_tokens, stream)
                     : dk <= 32 ? delta_scan_chain<1>(a, scratch, grid, max_tokens, stream)
                     : dk <= 64 ? delta_scan_chain<2>(a, scratch, grid, max_tokens, stream) : delta_scan_chain<4>(a, scratch, grid, max_tokens, stream);
        if (rc) return rc;
    } else if (max_tokens > 4) {
        int rc;
        if (dk <= 32) rc = delta_scan_staged<4>(a, grid, stream);
        else if (dk <= 64) rc = delta_scan_staged<8>(a, grid, stream);
        else if (dk <= 128) rc = delta_scan_staged<16>(a, grid, stream);
        else rc = delta_scan_staged<32>(a, grid, stream);
        if (rc) return rc;
    } else if (dk <= 128 && dk % 4 == 0 && c_stride % 4 == 0 && c_q % 4 == 0 && c_k % 4 == 0 && g_stride % 4 == 0 && g_col % 4 == 0 &&
               state_stride % 4 == 0 && (((uintptr_t)c | (uintptr_t)g | (uintptr_t)state) & 15) == 0) {
        if (dk <= 32) delta_token<8>(a, n_seqs, stream);
        else if (dk <= 64) delta_token<16>(a, n_seqs, stream);
        else delta_token<32>(a, n_seqs, stream);
    } else if (dk <= 32) idm_launch(delta_scan_kernel<4>, grid, block, 0, stream, a);
    else if (dk <= 64) idm_launch(delta_scan_kernel<8>, grid, block, 0, stream, a);
    else if (dk <= 128) idm_launch(delta_scan_kernel<16>, grid, block, 0, stream, a);
    else idm_launch(delta_scan_kernel<32>, grid, block, 0, stream, a);
    IDM_LAUNCH_CHECK("delta_scan");
    return 0;
}

// ------------------------------------------------------------------ a decay per head, chunks of 32
static int delta_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// Places of a launch, as in delta_window: what fits the scratch (0: not one), in whole rounds of the chunks' blocks (two an SM) where there are more
// launches than one.  The state carries over from launch to launch.
static long long delta_heads_window(int n_seqs, int n_tokens, int H, int Hk, int dv) {
    const long long fit = DH_SCRATCH * 4 / delta_heads_chunk_bytes(H, Hk, dv), all = (long long)n_tokens / DH_C + n_seqs;
    if (fit >= all) return all;
    const long long round = 2 * delta_sms() / Hk;
    return round > 0 && fit > round ? fit / round * round : fit;
}

#define DH_PORTION 48
// Floats of scratch that a step of `n_seqs` sequences and `n_tokens` tokens, at most `max_tokens` of one sequence, wants; 0: the step's
// decays are wanted per channel (idm_delta_scan).  Keys of 65 to 128 channels in rows of whole 16-byte pieces, portions of more than DH_PORTION tokens, and of 24
// tokens a sequence on average (16 where a sequence's blocks of the walk are no more than the SMs: 32 heads): a sequence of one token costs a block of
// the walk, an SM each, as much as one of 32.
// Measured, us of a layer with 64 heads (32 heads), this form / the chain of chunks of 16: 8 x 12 tokens 146 / 115 (91 / 93), 8 x 40 195 / 193
// (101 / 107), 2 x 60 117 / 121 (92 / 103), 8 x 130 386 / 493 (195 / 254), 3 x 1 000 826 / 1 296 (391 / 598).  One portion among single tokens:
// 2 048 among 60 1 158 / 1 645 (538 / 1 018), 1 000 among 31 609 / 729 (282 / 456), 700 among 31 526 / 535 (252 / 342), 400 among 20 331 / 325 (172 / 200), 300 among 15
// 286 / 263 (141 / 177), 200 among 15 259 / 219 (131 / 131), 60 among 15 214 / 164 (111 / 97), 300 among 63 674 / 519 (352 / 250), 64 among 60 573 / 353 (302 / 194).
extern "C" int idm_delta_heads_portion() { return DH_PORTION; }
extern "C" long long idm_delta_heads_scratch_floats(int n_seqs, int n_tokens, int H, int Hk, int dk, int dv, int max_tokens, int c_stride, int c_q, int c_k) {
    if (max_tokens <= DH_PORTION || n_seqs <= 0 || H <= 0 || Hk <= 0 || H % Hk || dk <= 64 || dk > DH_DK || dv <= 0) return 0;
    if (dk % 4 || c_stride % 4 || c_q % 4 || c_k % 4 || H > 65535 || n_seqs > 65535 || Hk > 65535) return 0;
    const bool at_once = (long long)H * ((dv + DH_COLS - 1) / DH_COLS) <= delta_sms();
    if (n_tokens < (at_once ? 16ll : 24ll) * n_seqs) return 0;
    return delta_heads_window(n_seqs, n_tokens, H, Hk, dv) * (delta_heads_chunk_bytes(H, Hk, dv) / 4);
}

// The delta rule with a decay per head, g [n_tokens, H]; scratch of idm_delta_heads_scratch_floats.
extern "C" int idm_delta_heads(const float* c, int c_stride, int c_q, int c_k, int c_v, const float* g, const float* beta, float* state,
                               long long state_stride, float* o, int o_stride, const int* cu_q, const int* slots, int n_seqs, int n_tokens, int H,
                               int Hk, int dk, int dv, int max_tokens, float* scratch, cudaStream_t stream) {
    if (n_seqs == 0 || n_tokens == 0) return 0;
    IDM_REQUIRE(idm_delta_heads_scratch_floats(n_seqs, n_tokens, H, Hk, dk, dv, max_tokens, c_stride, c_q, c_k) > 0,
                "delta_heads: %d heads over %d key heads, keys of %d, values of %d, %d tokens of %d sequences, columns %d and %d of rows of %d", H, Hk,
                dk, dv, n_tokens, n_seqs, c_q, c_k, c_stride);
    IDM_REQUIRE(state != nullptr && state_stride >= (long long)H * dk * dv, "delta_heads: a slot's state must hold %d x %d x %d floats", H, dv, dk);
    IDM_REQUIRE(scratch != nullptr && (((uintptr_t)scratch | (uintptr_t)c) & 15) == 0, "delta_heads: scratch at %p, rows at %p", (void*)scratch, (const void*)c);
    const int all = n_tokens / DH_C + n_seqs, window = (int)delta_heads_window(n_seqs, n_tokens, H, Hk, dv);
    DeltaHeadsScan a{c, c_stride, c_q, c_k, c_v, g, beta, state, state_stride, o, o_stride, cu_q, slots, n_seqs, H, Hk, dk, dv, (char*)scratch, 0, window};
    constexpr int chunk_smem = (int)sizeof(DeltaHeadsChunkSmem), walk_smem = (int)sizeof(DeltaHeadsWalkSmem);
    cudaError_t e = cudaFuncSetAttribute(delta_heads_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, chunk_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_heads_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, walk_smem);
    IDM_REQUIRE(e == cudaSuccess, "delta_heads: %d bytes of shared memory were refused (%s)", walk_smem, cudaGetErrorString(e));
    for (; a.first < all; a.first += window) {                  // (a window's places are those of no more sequences)
        idm_launch(delta_heads_chunk_kernel, dim3(window < all - a.first ? window : all - a.first, Hk), dim3(DH_THREADS), chunk_smem, stream, a);
        idm_launch(delta_heads_walk_kernel, dim3((dv + DH_COLS - 1) / DH_COLS, H, n_seqs < window ? n_seqs : window), dim3(256), walk_smem, stream, a);
    }
    IDM_LAUNCH_CHECK("delta_heads");
    return 0;
}

// ------------------------------------------------------------------ behind the recurrence
// out[t, out_col + h dv + j] = o[t, h, j] / sqrt(mean_j o^2 + eps) * w[j] * act(gate[t, gate_col + h dv + j]) * scale (w
// null: ones), act = sigmoid (gate_act 0) or silu (gate_act 1); one warp per (token, head)
__global__ void __launch_bounds__(128) delta_out_kernel(const float* __restrict__ o, int o_stride, const float* __restrict__ w,
                                                        float eps, const float* __restrict__ gate, int gate_stride,
                                                        int gate_col, int gate_act, float scale, T* __restrict__ out,
                                                        int out_stride, int out_col, int n_tokens, int H, int dv) {
    pdl_launch_dependents();
    pdl_wait();
    const long long i = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= (long long)n_tokens * H) return;
    const int t = (int)(i / H), h = (int)(i % H);
    const float* x = o + (size_t)t * o_stride + (size_t)h * dv;
    float ss = 0.f;
    for (int d = lane; d < dv; d += 32) ss += x[d] * x[d];
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)dv + eps);
    const float* gr = gate + (size_t)t * gate_stride + gate_col + (size_t)h * dv;
    T* dst = out + (size_t)t * out_stride + out_col + (size_t)h * dv;
    for (int d = lane; d < dv; d += 32) {
        const float z = gr[d], sg = 1.0f / (1.0f + expf(-z));
        const float y = w ? x[d] * inv * w[d] : x[d] * inv;
        from_f32(dst[d], gate_act == 1 ? y * (z * sg) * scale : y / (1.0f + expf(-z)) * scale);
    }
}

// The same with four elements a lane and load: LANES lanes have a head of up to 4 LANES NV elements, everything a head needs is on its
// way before its sum is made.  Bound by the bytes of o and the gate.
template <int LANES, int NV>
__global__ void __launch_bounds__(128) delta_out_vec_kernel(const float* __restrict__ o, int o_stride, const float* __restrict__ w,
                                                            float eps, const float* __restrict__ gate, int gate_stride,
                                                            int gate_col, int gate_act, float scale, T* __restrict__ out,
                                                            int out_stride, int out_col, int n_tokens, int H, int dv) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = (int)blockIdx.x * (128 / LANES) + threadIdx.x / LANES, lane = threadIdx.x % LANES;
    const bool live = i < n_tokens * H;                          // (no lane leaves: the sums are over whole warps)
    const int t = live ? i / H : 0, h = live ? i % H : 0;
    const float* x = o + (size_t)t * o_stride + (size_t)h * dv;
    const float* gr = gate + (size_t)t * gate_stride + gate_col + (size_t)h * dv;
    float4 v[NV], z[NV];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int d = (k * LANES + lane) * 4;
        v[k] = z[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (live && d < dv) { v[k] = *reinterpret_cast<const float4*>(x + d); z[k] = *reinterpret_cast<const float4*>(gr + d); }
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) { ss = fmaf(v[k].x, v[k].x, ss); ss = fmaf(v[k].y, v[k].y, ss); ss = fmaf(v[k].z, v[k].z, ss); ss = fmaf(v[k].w, v[k].w, ss); }
#pragma unroll
    for (int m = LANES / 2; m > 0; m >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, m);
    const float inv = 1.0f / sqrtf(ss / (float)dv + eps);
    T* dst = out + (size_t)t * out_stride + out_col + (size_t)h * dv;
    auto one = [&](float xv, float zv, float wv) {
        const float y = w ? xv * inv * wv : xv * inv, den = 1.0f + expf(-zv);
        return gate_act == 1 ? y * (zv * (1.0f / den)) * scale : y / den * scale;
    };
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int d = (k * LANES + lane) * 4;
        if (!live || d >= dv) continue;
        const float4 wv = w ? *reinterpret_cast<const float4*>(w + d) : make_float4(1.f, 1.f, 1.f, 1.f);
        store4(dst + d, one(v[k].x, z[k].x, wv.x), one(v[k].y, z[k].y, wv.y), one(v[k].z, z[k].z, wv.z), one(v[k].w, z[k].w, wv.w));
    }
}

extern "C" int idm_delta_out(const float* o, int o_stride, const float* w, float eps, const float* gate, int gate_stride,
                             int gate_col, int gate_act, float scale, void* out, int out_stride, int out_col, int n_tokens, int H,
                             int dv, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    IDM_REQUIRE(H > 0 && dv > 0 && out_col >= 0 && out_col + H * dv <= out_stride, "delta_out: columns %d..%d of rows of %d",
                out_col, out_col + H * dv, out_stride);
    const long long warps = (long long)n_tokens * H;
    // heads whose rows are whole pieces of four elements on their borders (a prompt of 2 048 tokens, 32 heads of 64: 13 us, element by element 31): others
    // element by element
    const bool vec = dv % 4 == 0 && dv <= 512 && o_stride % 4 == 0 && gate_stride % 4 == 0 && gate_col % 4 == 0 && out_stride % 4 == 0 &&
                     out_col % 4 == 0 && (((uintptr_t)o | (uintptr_t)gate | (uintptr_t)w | (uintptr_t)out) & 15) == 0 && warps < (1ll << 31);
    if (vec) {
#define DELTA_OUT(LANES_, NV_) idm_launch(delta_out_vec_kernel<LANES_, NV_>, dim3((unsigned)((warps + 128 / LANES_ - 1) / (128 / LANES_))), dim3(128), 0, \
                                          stream, o, o_stride, w, eps, gate, gate_stride, gate_col, gate_act, scale, (T*)out, out_stride, out_col, n_tokens, H, dv)
        if (dv <= 32) DELTA_OUT(8, 1);
        else if (dv <= 64) DELTA_OUT(16, 1);
        else if (dv <= 128) DELTA_OUT(32, 1);
        else if (dv <= 256) DELTA_OUT(32, 2);
        else DELTA_OUT(32, 4);
#undef DELTA_OUT
        IDM_LAUNCH_CHECK("delta_out");
        return 0;
    }
    idm_launch(delta_out_kernel, dim3((unsigned)((warps + 3) / 4)), dim3(128), 0, stream, o, o_stride, w, eps, gate,
               gate_stride, gate_col, gate_act, scale, (T*)out, out_stride, out_col, n_tokens, H, dv);
    IDM_LAUNCH_CHECK("delta_out");
    return 0;
}
