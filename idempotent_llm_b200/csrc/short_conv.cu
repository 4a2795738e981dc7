// Short causal convolutions over time with per-sequence state, for mixers that filter their
// projections channel by channel:
//
//   y[t, c] = sum_j w[c, j] * u[t - taps + 1 + j, c]      (j = 0 .. taps - 1; zeros before the sequence's start)
//
// u are columns [col0, col0 + channels) of a 32-bit projection [N, in_stride] of the step's packed tokens.
// Inputs before the step's first token come from the sequence's state: `taps - 1` rows of `channels`
// floats per slot, holding the inputs at positions q_start - taps + 1 .. q_start - 1.  The sum runs in
// ascending j in 32-bit whatever the step looks like, so a token's result does not depend on how its
// sequence was cut into steps.
//
// State is moved on behind the reads: a sequence that brings one token has its rows shifted by the thread
// that owns the channel (it has read all of them); sequences that bring more are moved on by
// conv_state_update_kernel, launched after every reader of the old state.
#include "common.cuh"

#define CONV_MAX_TAPS 8

struct ConvSeg {
    const float* in; int in_stride; int col0;       // projection of the step [N, in_stride], first column
    int channels, taps;
    const float* w;                                 // [channels, taps]
    const float* bias;                              // [channels] or null
    float* state; long long state_stride;           // state + slot * state_stride : [taps - 1, channels]
};

struct ConvStep {
    const int* token_seq; const int* positions; const int* slots; const int* q_start; const int* cu_q;
};

// what a token's filters need to know of its sequence: looked up once per thread (or block)
struct ConvToken {
    int pos;        // the token's position
    int avail;      // tokens of this step before it in its sequence: inputs further back come from the state
    int slot;
    int single;     // its sequence brings this token only: the filter moves the state on itself
};
__device__ __forceinline__ ConvToken conv_token(const ConvStep& st, int t) {
    const int s = st.token_seq[t];
    ConvToken m;
    m.pos = st.positions[t];
    m.avail = m.pos - st.q_start[s];
    m.slot = st.slots[s];
    m.single = st.cu_q[s + 1] - st.cu_q[s] == 1;
    return m;
}

// Tokens per thread: 8, or up to CONV_ROUNDS times 8 one after another, where that still leaves blocks enough for the SMs (a thread's weights
// and state then serve all its outputs, and looking up places and addresses, most of the instructions, is done once), else one, so that
// a few single tokens spread over as many threads as they have channels (conv_at).  Channels per thread: two where pairs lie on 8-byte
// borders.  Bound by latencies and instructions, not yet by memory (which would take 13 to 18 us of the last two).  Measured: short_conv of 4 096
// channels x 4 taps, 2 048 tokens, 13.7 us (one channel and 8 tokens a thread 18.6, one token 47), 4 876 tokens 35 us (45); conv_qkv_cache of
// 4 096 channels x 3 taps, 4 876 tokens, 53 us (112 us with each token's turn read from memory behind the stores of the one before,
// 70 us in pairs without rounds); three blocks an SM instead of two spill and take 54.  At
// 6 to 8 taps pairs spill some registers and are the faster form all the same: 3 584 channels, 4 876 tokens, 4 / 6 / 7 / 8 taps into the cache
// 42 / 46 / 49 / 55 us (one channel and 8 tokens a thread 84 / 103 / 130 / 152), short_conv 25 / 31 / 36 / 38 (36 / 37 / 41 / 48).  With few tokens the looking up of a token's place, then
// loads, is the shortest chain: asked for in ConvChannel's order, 1 / 8 / 64 single tokens take 2.85 / 3.18 / 6.86 us in conv_qkv_cache
// (20 heads of 64) against 2.40 / 2.77 / 6.36.
#define CONV_TOKENS 8
#define CONV_BLOCKS 1184               // eight blocks of 256 threads an SM
#define CONV_ROUNDS 4
#define CONV_TABLE 40960               // bytes of shared memory for the turns' table

// the convolution of token t, channel c (the number of taps known at compile time: the loops unroll to straight
// code); moves the state on if t is its sequence's only token
template <int TAPS>
__device__ __forceinline__ float conv_at(const ConvSeg& g, const ConvToken& m, int t, int c) {
    constexpr int H = TAPS - 1;
    const float* base = g.in + (size_t)t * g.in_stride + g.col0 + c;
    float* srow = g.state + (size_t)m.slot * g.state_stride + c;
    float u[TAPS];
#pragma unroll
    for (int j = 0; j < TAPS; ++j) {
        const int back = H - j;                                    // the input `back` positions before the token
        float v = 0.f;
        if (back <= m.avail) v = base[-(ptrdiff_t)back * g.in_stride];
        else if (back <= m.pos) v = srow[(size_t)(H - (back - m.avail)) * g.channels];
        u[j] = v;
    }
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < TAPS; ++j) acc = fmaf(g.w[(size_t)c * TAPS + j], u[j], acc);
    if (g.bias) acc += g.bias[c];
    if (m.single) {
#pragma unroll
        for (int j = 1; j < TAPS; ++j) srow[(size_t)(j - 1) * g.channels] = u[j];
    }
    return acc;
}

// Channels c .. c + V - 1 of tokens t0 .. t0 + n - 1 (n <= CONV_TOKENS; the number of taps is known at compile time, so that the loops
// unroll to straight code).  A thread keeps its channels' inputs and taps in registers: every input is read once for all the
// outputs it takes part in.  load() asks for everything that does not depend on the tokens' places, the rows in front of t0 among it
// (they count only if they are the same sequence's), so that one wait covers these loads and the looking up of the places.
template <int V> struct ConvLoad;
template <> struct ConvLoad<1> { static __device__ __forceinline__ void at(const float* p, float* v) { v[0] = *p; } };
template <> struct ConvLoad<2> {
    static __device__ __forceinline__ void at(const float* p, float* v) { const float2 x = *reinterpret_cast<const float2*>(p); v[0] = x.x; v[1] = x.y; }
};
template <int TAPS, int V>
struct ConvChannel {
    static constexpr int H = TAPS - 1, TB = CONV_TOKENS;
    float x[H + TB][V], w[V][TAPS], bias[V];
    __device__ __forceinline__ void rows(const ConvSeg& g, int t0, int n, int c) {
        const float* base = g.in + (size_t)t0 * g.in_stride + g.col0 + c;
#pragma unroll
        for (int i = 0; i < TB; ++i) {
            if (i < n) ConvLoad<V>::at(base + (ptrdiff_t)i * g.in_stride, x[H + i]);
            else
#pragma unroll
                for (int e = 0; e < V; ++e) x[H + i][e] = 0.f;
        }
    }
    // the next eight tokens: the last inputs of these are in front of them
    __device__ __forceinline__ void next(const ConvSeg& g, int t0, int n, int c) {
#pragma unroll
        for (int i = 0; i < H; ++i)
#pragma unroll
            for (int e = 0; e < V; ++e) x[i][e] = x[TB + i][e];
        rows(g, t0, n, c);
    }
    __device__ __forceinline__ void load(const ConvSeg& g, int t0, int n, int c) {
        rows(g, t0, n, c);
        const float* base = g.in + (size_t)t0 * g.in_stride + g.col0 + c;
#pragma unroll
        for (int i = 0; i < H; ++i) {
            if (t0 >= H - i) ConvLoad<V>::at(base + (ptrdiff_t)(i - H) * g.in_stride, x[i]);
            else
#pragma unroll
                for (int e = 0; e < V; ++e) x[i][e] = 0.f;
        }
#pragma unroll
        for (int e = 0; e < V * TAPS; e += V) ConvLoad<V>::at(g.w + (size_t)c * TAPS + e, &w[0][0] + e);
#pragma unroll
        for (int e = 0; e < V; ++e) bias[e] = g.bias ? g.bias[c + e] : 0.f;
    }
    __device__ __forceinline__ void sums(const ConvSeg& g, const float (&u)[TAPS][V], float (&y)[V]) const {
#pragma unroll
        for (int e = 0; e < V; ++e) {
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < TAPS; ++j) acc = fmaf(w[e][j], u[j][e], acc);
            y[e] = g.bias ? acc + bias[e] : acc;
        }
    }
    // token i's outputs; m: the tokens' places (in shared memory).  PLAIN: it and the tokens before it whose inputs it takes are all of one
    // sequence and in the step.  Else moves the state on for a token that is its sequence's only one
    template <bool PLAIN>
    __device__ __forceinline__ void at(const ConvSeg& g, const ConvToken* m, int i, int c, float (&y)[V]) const {
        float u[TAPS][V];
#pragma unroll
        for (int j = 0; j < TAPS; ++j)
#pragma unroll
            for (int e = 0; e < V; ++e) u[j][e] = x[i + j][e];
        if constexpr (!PLAIN) {
            const int avail = m[i].avail, pos = m[i].pos;
            float* srow = g.state + (size_t)m[i].slot * g.state_stride + c;
#pragma unroll
            for (int j = 0; j < H; ++j) {
                const int back = H - j;                                // the input `back` positions before the token
                if (back <= avail) continue;
#pragma unroll
                for (int e = 0; e < V; ++e) u[j][e] = back <= pos ? srow[(size_t)(H - (back - avail)) * g.channels + e] : 0.f;
            }
            if (m[i].single)
#pragma unroll
                for (int j = 1; j < TAPS; ++j)
#pragma unroll
                    for (int e = 0; e < V; ++e) srow[(size_t)(j - 1) * g.channels + e] = u[j][e];
        }
        sums(g, u, y);
    }
    // whether that holds for eight tokens of a block
    static __device__ __forceinline__ bool plain(const ConvToken* m, int n) { return n == TB && m[0].avail >= H && m[TB - 1].avail == m[0].avail + TB - 1; }
};
__device__ __forceinline__ void conv_store(float* p, const float (&y)[1]) { *p = y[0]; }
__device__ __forceinline__ void conv_store(float* p, const float (&y)[2]) { *reinterpret_cast<float2*>(p) = make_float2(y[0], y[1]); }
__device__ __forceinline__ void conv_store(__nv_bfloat16* p, const float (&y)[1]) { from_f32(*p, y[0]); }
__device__ __forceinline__ void conv_store(__nv_bfloat16* p, const float (&y)[2]) {
    *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(y[0], y[1]);
}

// silu of a filter's output: exact in the 32-bit library; with the hardware exponential and division where the
// result is rounded to bfloat16 operands anyway (relative error ~1e-6)
__device__ __forceinline__ float silu_exact(float v) {
#if defined(IDM_F32)
    return v / (1.0f + expf(-v));
#else
    return __fdividef(v, 1.0f + __expf(-v));
#endif
}

// out [N, channels] 32-bit; act: 0 none, 1 silu
template <int TAPS>
__global__ void __launch_bounds__(256) short_conv_kernel(ConvSeg g, ConvStep st, float* __restrict__ out, int act) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ ConvToken token;                     // (one token per block: looked up by one thread)
    const int c = blockIdx.y * blockDim.x + threadIdx.x, t = blockIdx.x;
    if (threadIdx.x == 0) token = conv_token(st, t);
    __syncthreads();
    if (c >= g.channels) return;
    const float v = conv_at<TAPS>(g, token, t, c);
    out[(size_t)t * g.channels + c] = act == 1 ? silu_exact(v) : v;
}

// the same, V channels and `rounds` times eight tokens a thread
template <int TAPS, int V>
__global__ void __launch_bounds__(256) short_conv_tokens_kernel(ConvSeg g, ConvStep st, float* __restrict__ out, int act, int n_tokens, int rounds) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int TB = CONV_TOKENS;
    __shared__ ConvToken places[TB * CONV_ROUNDS];  // looked up by one thread each
    const int c = (blockIdx.y * blockDim.x + threadIdx.x) * V;
    int t0 = blockIdx.x * TB * rounds;
    const int t1 = min(t0 + TB * rounds, n_tokens);
    ConvChannel<TAPS, V> ch;
    if (c < g.channels) ch.load(g, t0, min(TB, t1 - t0), c);
    if (threadIdx.x < t1 - t0) places[threadIdx.x] = conv_token(st, t0 + threadIdx.x);
    __syncthreads();
    if (c >= g.channels) return;
    float* dst = out + (size_t)t0 * g.channels + c;
    auto finish = [&](float (&y)[V]) {
        if (act == 1)
#pragma unroll
            for (int e = 0; e < V; ++e) y[e] = silu_exact(y[e]);
        conv_store(dst, y);
        dst += g.channels;
    };
    for (const ConvToken* token = places;; token += TB) {
        const int n = min(TB, t1 - t0);
        if (ch.plain(token, n)) {
#pragma unroll
            for (int i = 0; i < TB; ++i) {
                float y[V];
                ch.template at<true>(g, token, i, c, y);
                finish(y);
            }
        } else {
#pragma unroll
            for (int i = 0; i < TB; ++i) {
                if (i >= n) break;
                float y[V];
                ch.template at<false>(g, token, i, c, y);
                finish(y);
            }
        }
        t0 += TB;
        if (t0 >= t1) break;
        ch.next(g, t0, min(TB, t1 - t0), c);
    }
}

// The attention side: q, k and v channels [n_q * dk | n_kv * dk | n_kv * dv] are filtered, the first
// 2 * half dims of every q and k head turned by the token's position (dim i with dim i + half; (u, v) ->
// (u cos - v sin, v cos + u sin), table cs [N, half] of (cos, sin)), q stored [N, n_q, dk] and k, v written
// to the token's place in the cache (pools [pages, n_kv, PAGE, dk] and [pages, n_kv, PAGE, dv]).
// With `maps` > 1 a q or k head is that many parts side by side, each turned like a head of dk / maps dims, and q goes out as
// one row per part, [N, n_q * maps, dk], zero outside its part: against the same key rows each such row scores its part
// alone.
// (u, v) turned by (cos, sin): one order of rounding in both kernels
__device__ __forceinline__ float2 conv_turned(float u, float v, float2 cs) {
    return make_float2(fmaf(u, cs.x, -__fmul_rn(v, cs.y)), fmaf(v, cs.x, __fmul_rn(u, cs.y)));
}
struct ConvQkvArgs {
    ConvSeg seg; ConvStep st;
    int n_q, n_kv, dk, dv, half;
    int maps;                       // parts of a q or k head that are turned each on its own (dk / maps dims each)
    const float2* cs;
    T* q_out; T* k_pool; T* v_pool;
    const int* table; int table_stride;
    int n_tokens;
};

template <int TAPS>
__global__ void __launch_bounds__(256) conv_qkv_cache_kernel(ConvQkvArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    const ConvToken m = conv_token(a.st, t);                       // (one token per block: every thread the same)
    const size_t page = a.table[(size_t)m.slot * a.table_stride + m.pos / IDM_PAGE], prow = m.pos % IDM_PAGE;
    const int qk_heads = a.n_q + a.n_kv;
    const int part = a.dk / a.maps, per = part - a.half;  // work items of a part: pairs, then single dims
    const int rest = a.maps * per;                        // work items of a q or k head
    const int qk_items = qk_heads * rest, v_items = a.n_kv * a.dv;
    // (steps of few tokens spread a token's items over several blocks: gridDim.y)
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < qk_items + v_items; i += gridDim.y * blockDim.x) {
        if (i < qk_items) {
            const int head = i / rest, mp = i % rest / per, r = i % per, d0 = mp * part;
            const bool is_q = head < a.n_q;
            T* row = is_q ? a.q_out + ((size_t)t * a.n_q + head) * a.maps * a.dk
                          : a.k_pool + ((page * a.n_kv + (head - a.n_q)) * IDM_PAGE + prow) * (size_t)a.dk;
            T* dst = row + (is_q ? mp * a.dk : 0) + d0;
            const int other = r < a.half ? r + a.half : -1, d = r < a.half ? r : r + a.half;
            if (other >= 0) {
                const float u = conv_at<TAPS>(a.seg, m, t, head * a.dk + d0 + d);
                const float v = conv_at<TAPS>(a.seg, m, t, head * a.dk + d0 + other);
                const float2 cs = a.cs[(size_t)t * a.half + r];
                const float2 y = conv_turned(u, v, cs);
                from_f32(dst[d], y.x);
                from_f32(dst[other], y.y);
            } else {
                from_f32(dst[d], conv_at<TAPS>(a.seg, m, t, head * a.dk + d0 + d));
            }
            if (is_q)
                for (int z = 0; z < a.maps; ++z)
                    if (z != mp) {
                        from_f32(row[z * a.dk + d0 + d], 0.f);
                        if (other >= 0) from_f32(row[z * a.dk + d0 + other], 0.f);
                    }
        } else {
            const int j = i - qk_items, g = j / a.dv, d = j % a.dv;
            T* dst = a.v_pool + ((page * a.n_kv + g) * IDM_PAGE + prow) * (size_t)a.dv;
            from_f32(dst[d], conv_at<TAPS>(a.seg, m, t, qk_heads * a.dk + j));
        }
    }
}

// the same, V channels (pairs of them in what is turned) and `rounds` times eight tokens a thread: first all that is turned, then what is
// left of the q and k heads, then the values, so that a warp's threads do the same.  The tokens' (cos, sin) rows lie in shared memory: behind the
// stores of the tokens before, a load of them would be a wait of its own for every token.
template <int TAPS, int V>
__global__ void __launch_bounds__(256, 2) conv_qkv_cache_tokens_kernel(ConvQkvArgs a, int rounds) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int TB = CONV_TOKENS;
    extern __shared__ __align__(16) float2 conv_cs[];               // [TB rounds][half]
    __shared__ ConvToken places[TB * CONV_ROUNDS];
    __shared__ unsigned place[TB * CONV_ROUNDS];    // a token's row among all rows of a kv-head's first page: + head * PAGE
    int t0 = blockIdx.x * TB * rounds;
    const int t1 = min(t0 + TB * rounds, a.n_tokens);
    const int parts = (a.n_q + a.n_kv) * a.maps, part = a.dk / a.maps, rest = part - 2 * a.half;
    const int turned = parts * (a.half / V), straight = turned + parts * (rest / V), items = straight + a.n_kv * a.dv / V;
    const int i = blockIdx.y * blockDim.x + threadIdx.x;
    const bool turn = i < turned, value = i >= straight;
    const int across = turn ? a.half / V : value ? a.dv / V : rest / V, j = i - (turn ? 0 : value ? straight : turned);
    const int unit = j / across, r = (j - unit * across) * V, d = r + (turn || value ? 0 : 2 * a.half);   // (unit: part of a q or k head, or kv-head)
    const int c = value ? parts * part + unit * a.dv + d : unit * part + d;
    ConvChannel<TAPS, V> one, two;
    if (i < items) {
        one.load(a.seg, t0, min(TB, t1 - t0), c);
        if (turn) two.load(a.seg, t0, min(TB, t1 - t0), c + a.half);
    }
    if (threadIdx.x < t1 - t0) {
        const ConvToken m = conv_token(a.st, t0 + threadIdx.x);
        places[threadIdx.x] = m;
        place[threadIdx.x] = (unsigned)a.table[(size_t)m.slot * a.table_stride + m.pos / IDM_PAGE] * a.n_kv * IDM_PAGE + m.pos % IDM_PAGE;
    }
    for (int e = threadIdx.x; e < (t1 - t0) * a.half; e += blockDim.x) conv_cs[e] = a.cs[(size_t)t0 * a.half + e];
    __syncthreads();
    if (i >= items) return;
    const int head = unit / a.maps, mp = unit - head * a.maps, at = value ? d : mp * part + d;
    const bool is_q = !value && head < a.n_q;
    // where a token goes: rows of q one after another, of a cache by the token's place
    T* base = value ? a.v_pool + (size_t)unit * IDM_PAGE * a.dv + at
              : is_q ? a.q_out + ((size_t)t0 * a.n_q + head) * a.maps * a.dk + mp * a.dk + at
                     : a.k_pool + (size_t)(head - a.n_q) * IDM_PAGE * a.dk + at;
    const unsigned row = value ? a.dv : is_q ? a.n_q * a.maps * a.dk : a.dk;
    for (int k0 = 0;; k0 += TB) {
        const ConvToken* token = places + k0;
        const int n = min(TB, t1 - t0);
        auto finish = [&](int k, float (&u)[V], float (&v)[V]) {
            T* dst = base + (unsigned long long)row * (is_q ? k0 + k : place[k0 + k]);
            if (turn) {
                const float2* cs = conv_cs + (k0 + k) * a.half + r;
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const float2 y = conv_turned(u[e], v[e], cs[e]);
                    u[e] = y.x;
                    v[e] = y.y;
                }
                conv_store(dst + a.half, v);
            }
            conv_store(dst, u);
            if (is_q)
                for (int z = 0; z < a.maps; ++z)
                    if (z != mp) {
                        const float zero[V] = {};
                        conv_store(dst + (z - mp) * a.dk, zero);
                        if (turn) conv_store(dst + (z - mp) * a.dk + a.half, zero);
                    }
        };
        if (one.plain(token, n)) {
#pragma unroll
            for (int k = 0; k < TB; ++k) {
                float u[V], v[V];
                one.template at<true>(a.seg, token, k, c, u);
                if (turn) two.template at<true>(a.seg, token, k, c + a.half, v);
                finish(k, u, v);
            }
        } else {
#pragma unroll
            for (int k = 0; k < TB; ++k) {
                if (k >= n) break;
                float u[V], v[V];
                one.template at<false>(a.seg, token, k, c, u);
                if (turn) two.template at<false>(a.seg, token, k, c + a.half, v);
                finish(k, u, v);
            }
        }
        t0 += TB;
        if (t0 >= t1) break;
        one.next(a.seg, t0, min(TB, t1 - t0), c);
        if (turn) two.next(a.seg, t0, min(TB, t1 - t0), c + a.half);
    }
}

// After every reader: the state of sequences that brought more than one token becomes the inputs at their
// last taps - 1 positions.  One thread per (sequence, channel) reads its rows, then writes them.
__global__ void __launch_bounds__(256) conv_state_update_kernel(ConvSeg g, ConvStep st, const int* __restrict__ kv_len) {
    pdl_launch_dependents();
    pdl_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x, s = blockIdx.y;
    if (c >= g.channels) return;
    const int n_new = st.cu_q[s + 1] - st.cu_q[s];
    if (n_new <= 1) return;                          // (one token: moved on by the convolution itself)
    const int start = st.q_start[s], end = kv_len[s], hist = g.taps - 1;
    float* srow = g.state + (size_t)st.slots[s] * g.state_stride + c;
    float u[CONV_MAX_TAPS];
#pragma unroll
    for (int r = 0; r < CONV_MAX_TAPS - 1; ++r) {
        if (r >= hist) break;
        const int p = end - hist + r;
        float v = 0.f;
        if (p >= start) v = g.in[(size_t)(st.cu_q[s] + p - start) * g.in_stride + g.col0 + c];
        else if (p >= 0) v = srow[(size_t)(p - (start - hist)) * g.channels];
        u[r] = v;
    }
#pragma unroll
    for (int r = 0; r < CONV_MAX_TAPS - 1; ++r) {
        if (r >= hist) break;
        srow[(size_t)r * g.channels] = u[r];
    }
}

static int conv_seg(ConvSeg& g, const char* what, const float* in, int in_stride, int col0, int channels, int taps,
                    const float* w, const float* bias, float* state, long long state_stride) {
    IDM_REQUIRE(channels > 0 && taps >= 1 && taps <= CONV_MAX_TAPS, "%s: %d channels, %d taps (at most %d)", what, channels,
                taps, CONV_MAX_TAPS);
    IDM_REQUIRE(col0 >= 0 && col0 + channels <= in_stride, "%s: columns %d..%d of rows of %d", what, col0, col0 + channels, in_stride);
    IDM_REQUIRE(taps == 1 || (state != nullptr && state_stride >= (long long)(taps - 1) * channels),
                "%s: the state of a slot must hold %d rows of %d floats", what, taps - 1, channels);
    g.in = in; g.in_stride = in_stride; g.col0 = col0; g.channels = channels; g.taps = taps; g.w = w; g.bias = bias;
    g.state = state; g.state_stride = state_stride;
    return 0;
}

// whether two neighbouring channels lie on 8-byte borders in the projection's rows, in the taps and among the channels
static bool conv_pairs(const ConvSeg& g) {
    return g.channels % 2 == 0 && g.in_stride % 2 == 0 && g.col0 % 2 == 0 && (((uintptr_t)g.in | (uintptr_t)g.w) & 7) == 0;
}

// A block of the kernels of eight tokens a thread goes on with the next eight, up to CONV_ROUNDS times, where that leaves the SMs
// enough blocks: looking up places and addresses is most of what a thread does for eight.  (`most`: as many as there is room for.)
static dim3 conv_cut(int n_tokens, int across, int most, int& rounds) {
    const long long blocks = (long long)((n_tokens + CONV_TOKENS - 1) / CONV_TOKENS) * across;
    rounds = (int)(blocks / 592);
    rounds = rounds > most ? most : rounds;
    rounds = rounds < 1 ? 1 : rounds > CONV_ROUNDS ? CONV_ROUNDS : rounds;
    return dim3((n_tokens + CONV_TOKENS * rounds - 1) / (CONV_TOKENS * rounds), across);
}

extern "C" int idm_short_conv(const float* in, int in_stride, int col0, int channels, int taps, const float* w,
                              const float* bias, int act, float* state, long long state_stride, float* out,
                              const int* token_seq, const int* positions, const int* slots, const int* q_start,
                              const int* cu_q, int n_tokens, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    ConvSeg g;
    if (conv_seg(g, "short_conv", in, in_stride, col0, channels, taps, w, bias, state, state_stride)) return 1;
    ConvStep st{token_seq, positions, slots, q_start, cu_q};
    const int across = (channels + 255) / 256;
    const bool many = (long long)(n_tokens / CONV_TOKENS) * across >= CONV_BLOCKS;
    const dim3 grid(n_tokens, across);
    const bool pairs = conv_pairs(g) && ((uintptr_t)out & 7) == 0;
    int rounds;
    const dim3 cut = conv_cut(n_tokens, pairs ? (channels + 511) / 512 : across, CONV_ROUNDS, rounds);
#define CONV_GO(TAPS_) case TAPS_: idm_launch(short_conv_kernel<TAPS_>, grid, dim3(256), 0, stream, g, st, out, act); break;
#define CONV_MANY(TAPS_) case TAPS_: \
        if (pairs) idm_launch(short_conv_tokens_kernel<TAPS_, 2>, cut, dim3(256), 0, stream, g, st, out, act, n_tokens, rounds); \
        else idm_launch(short_conv_tokens_kernel<TAPS_, 1>, cut, dim3(256), 0, stream, g, st, out, act, n_tokens, rounds); \
        break;
    if (many) switch (taps) { CONV_MANY(1) CONV_MANY(2) CONV_MANY(3) CONV_MANY(4) CONV_MANY(5) CONV_MANY(6) CONV_MANY(7) CONV_MANY(8) }
    else switch (taps) { CONV_GO(1) CONV_GO(2) CONV_GO(3) CONV_GO(4) CONV_GO(5) CONV_GO(6) CONV_GO(7) CONV_GO(8) }
#undef CONV_GO
#undef CONV_MANY
    IDM_LAUNCH_CHECK("short_conv");
    return 0;
}

extern "C" int idm_conv_qkv_cache(const float* in, int in_stride, int col0, int taps, const float* w, float* state,
                                  long long state_stride, int n_q, int n_kv, int dk, int dv, int half, int maps, const float* cs,
                                  void* q_out, void* k_pool, void* v_pool, const int* table, int table_stride,
                                  const int* token_seq, const int* positions, const int* slots, const int* q_start,
                                  const int* cu_q, int n_tokens, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    ConvQkvArgs a;
    const int channels = (n_q + n_kv) * dk + n_kv * dv;
    if (conv_seg(a.seg, "conv_qkv_cache", in, in_stride, col0, channels, taps, w, nullptr, state, state_stride)) return 1;
    IDM_REQUIRE(n_q > 0 && n_kv > 0 && dk > 0 && dv > 0 && maps >= 1 && dk % maps == 0 && half >= 0 && 2 * half <= dk / maps,
                "conv_qkv_cache: heads %d/%d, sizes %d/%d in %d parts, %d turning pairs", n_q, n_kv, dk, dv, maps, half);
    IDM_REQUIRE(half == 0 || cs != nullptr, "conv_qkv_cache: a rotation needs its table");
    a.st = ConvStep{token_seq, positions, slots, q_start, cu_q};
    a.n_q = n_q; a.n_kv = n_kv; a.dk = dk; a.dv = dv; a.half = half; a.maps = maps; a.cs = (const float2*)cs;
    a.q_out = (T*)q_out; a.k_pool = (T*)k_pool; a.v_pool = (T*)v_pool; a.table = table; a.table_stride = table_stride;
    a.n_tokens = n_tokens;
    // a thread per item and eight tokens; else a block per token, with few tokens several, so that two blocks' worth of work per SM is about
    const int items = (n_q + n_kv) * (dk - maps * half) + n_kv * dv, across = (items + 255) / 256;
    const size_t smem = (size_t)CONV_TOKENS * half * sizeof(float2);
    // (as many rounds as the table has room for: heads of 384, all turned, 4 000 tokens of 16 over 4, 89 us; a token a block 221, eight tokens
    // a thread without a table 162)
    const bool many = (long long)(n_tokens / CONV_TOKENS) * across >= CONV_BLOCKS && smem <= CONV_TABLE;
    const bool pairs = conv_pairs(a.seg) && half % 2 == 0 && (dk / maps) % 2 == 0 && dv % 2 == 0 &&
                       (((uintptr_t)q_out | (uintptr_t)k_pool | (uintptr_t)v_pool) & 7) == 0;
    int rounds;
    const dim3 cut = conv_cut(n_tokens, pairs ? (items + 511) / 512 : across, smem ? (int)(CONV_TABLE / smem) : CONV_ROUNDS, rounds);
    int split = (296 + n_tokens - 1) / n_tokens;
    if (split > across) split = across;
    if (split < 1) split = 1;
    const dim3 grid(n_tokens, split);
#define CONV_GO(TAPS_) case TAPS_: idm_launch(conv_qkv_cache_kernel<TAPS_>, grid, dim3(256), 0, stream, a); break;
#define CONV_MANY(TAPS_) case TAPS_: \
        if (pairs) idm_launch(conv_qkv_cache_tokens_kernel<TAPS_, 2>, cut, dim3(256), smem * rounds, stream, a, rounds); \
        else idm_launch(conv_qkv_cache_tokens_kernel<TAPS_, 1>, cut, dim3(256), smem * rounds, stream, a, rounds); \
        break;
    if (many) switch (taps) { CONV_MANY(1) CONV_MANY(2) CONV_MANY(3) CONV_MANY(4) CONV_MANY(5) CONV_MANY(6) CONV_MANY(7) CONV_MANY(8) }
    else switch (taps) { CONV_GO(1) CONV_GO(2) CONV_GO(3) CONV_GO(4) CONV_GO(5) CONV_GO(6) CONV_GO(7) CONV_GO(8) }
#undef CONV_GO
#undef CONV_MANY
    IDM_LAUNCH_CHECK("conv_qkv_cache");
    return 0;
}

extern "C" int idm_conv_state_update(const float* in, int in_stride, int col0, int channels, int taps, float* state,
                                     long long state_stride, const int* slots, const int* q_start, const int* cu_q,
                                     const int* kv_len, int n_seqs, cudaStream_t stream) {
    if (n_seqs == 0 || taps <= 1) return 0;
    ConvSeg g;
    if (conv_seg(g, "conv_state_update", in, in_stride, col0, channels, taps, nullptr, nullptr, state, state_stride)) return 1;
    IDM_REQUIRE(n_seqs <= 65535, "conv_state_update: %d sequences in one launch", n_seqs);
    ConvStep st{nullptr, nullptr, slots, q_start, cu_q};
    idm_launch(conv_state_update_kernel, dim3((channels + 255) / 256, n_seqs), dim3(256), 0, stream, g, st, kv_len);
    IDM_LAUNCH_CHECK("conv_state_update");
    return 0;
}
