// Retention: a linear recurrence whose heads fade at constant rates g_h,
//
//   S_t = g_h S_(t-1) + k_t v_t^T       (S: [dk, dv] per head),       o_t = S_t^T q_t
//
// q and k are columns of a 32-bit projection, the first 2 * half dims of each head turned by the token's position (dim i
// with dim i + half), k then times a constant; v other columns of it.  Everything here is 32-bit.  The state lives per
// sequence as [H][dk][dv] and is carried from step to step.
//
// Steps of a few tokens per sequence walk them one by one (retention_walk_kernel).  Longer portions are cut into chunks that
// run side by side as products of tiles (chunk_products.cuh, with f_t = g_h and a_t = 1); in front of them
// retention_turn_kernel turns q and k in place, once.  A prompt of 1 777 tokens, 8 heads of 128 x 256: 134 us.
#include "chunk_products.cuh"

struct RetentionArgs {
    float* proj; int stride, col_q, col_k, col_v;
    const float2* cs; int half;                     // [N, half] (cos, sin)
    float k_scale;
    const float* decay;                             // [H]
    float* state; long long state_stride;           // state + slot * stride : [H][dk][dv]
    float* o; int o_stride;                         // o[t, h * dv + j]
    const int* cu_q; const int* slots;
    int H, dk, dv;
};

// element d of a head's row x, turned by the token's row of the table
__device__ __forceinline__ float retention_turned(const float* __restrict__ x, int d, int half, const float2* __restrict__ cs) {
    if (d >= 2 * half) return x[d];
    const bool first = d < half;
    const float2 a = cs[first ? d : d - half];
    return first ? x[d] * a.x - x[d + half] * a.y : x[d] * a.x + x[d - half] * a.y;
}

// ------------------------------------------------------------------ few tokens per sequence: one after another
// A block has (sequence, head, 32 columns of S): warp w holds rows w, w + 8, .. of them in registers, a lane a column.
template <int RP>
__global__ void __launch_bounds__(256) retention_walk_kernel(RetentionArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float qk[2][8 * RP];
    __shared__ float part[8][32];
    const int s = blockIdx.z, h = blockIdx.y, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = blockIdx.x * 32 + lane;
    const bool col = j < a.dv;
    const int t0 = a.cu_q[s], t1 = a.cu_q[s + 1];
    float* sp = a.state + (size_t)a.slots[s] * a.state_stride + (size_t)h * a.dk * a.dv + (col ? j : 0);
    const float g = a.decay[h];
    float S[RP];
#pragma unroll
    for (int i = 0; i < RP; ++i) S[i] = (col && w + 8 * i < a.dk) ? sp[(size_t)(w + 8 * i) * a.dv] : 0.f;
    for (int t = t0; t < t1; ++t) {
        const float* row = a.proj + (size_t)t * a.stride;
        const float2* cs = a.cs + (size_t)t * a.half;
        const float v = col ? row[a.col_v + h * a.dv + j] : 0.f;
        for (int e = threadIdx.x; e < 2 * 8 * RP; e += 256) {
            const int which = e / (8 * RP), d = e % (8 * RP);
            float x = 0.f;
            if (d < a.dk) {
                x = retention_turned(row + (which ? a.col_k : a.col_q) + h * a.dk, d, a.half, cs);
                if (which) x *= a.k_scale;
            }
            qk[which][d] = x;
        }
        __syncthreads();
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < RP; ++i) {
            S[i] = fmaf(qk[1][w + 8 * i], v, g * S[i]);
            acc = fmaf(S[i], qk[0][w + 8 * i], acc);
        }
        part[w][lane] = acc;
        __syncthreads();
        if (w == 0 && col) {
            float y = 0.f;
#pragma unroll
            for (int p = 0; p < 8; ++p) y += part[p][lane];
            a.o[(size_t)t * a.o_stride + h * a.dv + j] = y;
        }
    }
#pragma unroll
    for (int i = 0; i < RP; ++i)
        if (col && w + 8 * i < a.dk) sp[(size_t)(w + 8 * i) * a.dv] = S[i];
}

// ------------------------------------------------------------------ long portions
// q and k turned in place, k times its constant: a thread per pair (or untouched dim) of a head
__global__ void __launch_bounds__(256) retention_turn_kernel(RetentionArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, per = a.dk - a.half;
    float* row = a.proj + (size_t)t * a.stride;
    for (int e = blockIdx.y * blockDim.x + threadIdx.x; e < 2 * a.H * per; e += gridDim.y * blockDim.x) {
        const int which = e / (a.H * per), h = e % (a.H * per) / per, i = e % per;
        float* x = row + (which ? a.col_k : a.col_q) + h * a.dk;
        const float f = which ? a.k_scale : 1.f;
        if (i < a.half) {
            const float2 cs = a.cs[(size_t)t * a.half + i];
            const float u = x[i], v = x[i + a.half];
            x[i] = (u * cs.x - v * cs.y) * f;
            x[i + a.half] = (v * cs.x + u * cs.y) * f;
        } else if (which) {
            x[i + a.half] *= f;
        }
    }
}

// a head's powers over a chunk
struct RetentionWeights {
    const float* decay;
    struct Head { float pw[CP_C + 1]; };
    __device__ __forceinline__ void prepare(Head& hd, int head, int, int) const {
        if (threadIdx.x <= CP_C) hd.pw[threadIdx.x] = powf(decay[head], (float)threadIdx.x);
    }
    __device__ __forceinline__ float state(const Head& hd, int t) const { return hd.pw[t + 1]; }
    __device__ __forceinline__ float pair(const Head& hd, int t, int s) const { return hd.pw[t - s]; }
    __device__ __forceinline__ float end(const Head& hd, int n, int s) const { return hd.pw[n - 1 - s]; }
    __device__ __forceinline__ void store_end(const Head&, int, int, int) const {}
    __device__ __forceinline__ float end_factor(int, int head, int n) const { return powf(decay[head], (float)n); }
    __device__ __forceinline__ void finish(int, int, int, float*, const float*, int, int) const {}
};

extern "C" int idm_retention_chunk_tokens() { return CP_C; }
// floats of scratch for a step of so many chunks
extern "C" long long idm_retention_scratch_floats(int n_chunks, int H, int dk, int dv) { return (long long)n_chunks * H * dk * dv; }

// chunk_t0 [n_chunks + 1], seq_chunk0 [n_seqs + 1] as for the other chunked recurrence (a chunk ends where the next
// begins, chunks hold CP_C tokens, a sequence's last one up to so many, and never cross a sequence's border); n_chunks == 0: every sequence token by
// token.  In chunks, the step's q and k columns of `proj` are turned in place.
extern "C" int idm_retention(float* proj, int stride, int col_q, int col_k, int col_v, const float* cs, int half, float k_scale,
                             const float* decay, float* state, long long state_stride, float* o, int o_stride, const int* cu_q,
                             const int* slots, int n_seqs, int H, int dk, int dv, const int* chunk_t0, const int* seq_chunk0,
                             int n_chunks, float* scratch, int n_tokens, cudaStream_t stream) {
    if (n_seqs == 0 || n_tokens == 0) return 0;
    IDM_REQUIRE(H > 0 && dk > 0 && dk <= 256 && dv > 0, "retention: %d heads, keys of %d (at most 256), values of %d", H, dk, dv);
    IDM_REQUIRE(half >= 0 && 2 * half <= dk && (half == 0 || cs != nullptr), "retention: %d turning pairs in heads of %d", half, dk);
    IDM_REQUIRE(col_q >= 0 && col_k >= 0 && col_v >= 0 && col_q + H * dk <= stride && col_k + H * dk <= stride && col_v + H * dv <= stride,
                "retention: columns beyond rows of %d", stride);
    IDM_REQUIRE(state != nullptr && state_stride >= (long long)H * dk * dv, "retention: a slot's state must hold %d x %d x %d floats", H, dk, dv);
    IDM_REQUIRE(n_seqs <= 65535 && H <= 65535, "retention: %d sequences, %d heads in one launch", n_seqs, H);
    IDM_REQUIRE(n_chunks == 0 || (chunk_t0 && seq_chunk0 && scratch), "retention: chunks need their lists and scratch");
    RetentionArgs a;
    a.proj = proj; a.stride = stride; a.col_q = col_q; a.col_k = col_k; a.col_v = col_v; a.cs = (const float2*)cs; a.half = half;
    a.k_scale = k_scale; a.decay = decay; a.state = state; a.state_stride = state_stride; a.o = o; a.o_stride = o_stride;
    a.cu_q = cu_q; a.slots = slots; a.H = H; a.dk = dk; a.dv = dv;
    if (n_chunks == 0) {
        const dim3 grid((dv + 31) / 32, H, n_seqs);
        if (dk <= 32) idm_launch(retention_walk_kernel<4>, grid, dim3(256), 0, stream, a);
        else if (dk <= 64) idm_launch(retention_walk_kernel<8>, grid, dim3(256), 0, stream, a);
        else if (dk <= 128) idm_launch(retention_walk_kernel<16>, grid, dim3(256), 0, stream, a);
        else idm_launch(retention_walk_kernel<32>, grid, dim3(256), 0, stream, a);
        IDM_LAUNCH_CHECK("retention_walk");
        return 0;
    }
    const int items = 2 * H * (dk - half);
    idm_launch(retention_turn_kernel, dim3(n_tokens, min(8, (items + 255) / 256)), dim3(256), 0, stream, a);
    IDM_LAUNCH_CHECK("retention_turn");
    ChunkArgs c;
    c.q = proj + col_q; c.k = proj + col_k; c.v = proj + col_v; c.q_stride = c.k_stride = c.v_stride = stride;
    c.o = o; c.o_stride = o_stride; c.state = state; c.state_stride = state_stride; c.slots = slots;
    c.chunk_t0 = chunk_t0; c.seq_chunk0 = seq_chunk0; c.chunk_state = scratch;
    c.groups = c.heads = H; c.dk = dk; c.dv = dv;
    c.vec = dk % 4 == 0 && dv % 4 == 0 && stride % 4 == 0 && col_q % 4 == 0 && col_k % 4 == 0 && col_v % 4 == 0 && o_stride % 4 == 0 &&
            (((uintptr_t)proj | (uintptr_t)scratch | (uintptr_t)o) & 15) == 0;
    return chunk_products(c, RetentionWeights{decay}, n_chunks, n_seqs, "retention", stream);
}
