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

// Tokens per thread: 8 where that still leaves blocks enough for the SMs (a thread's weights and state then serve eight outputs;
// ConvChannel), else one, so that a few single tokens spread over as many threads as they have channels (conv_at).  Measured, short_conv of 4 096
// channels x 4 taps: 2 048 tokens 18.6 us (one token a thread: 47), 6 000 tokens 45 us (113); conv_qkv_cache of 6 000 tokens x 6 144
// channels 112 us (127).  With few tokens the looking up of a token's place, then loads, is the shortest chain: asked for in
// ConvChannel's order, 1 / 8 / 64 single tokens take 2.85 / 3.18 / 6.86 us in conv_qkv_cache (20 heads of 64) against 2.40 / 2.77 / 6.36.
#define CONV_TOKENS 8
#define CONV_BLOCKS 1184               // eight blocks of 256 threads an SM

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

// Channel c of tokens t0 .. t0 + n - 1 (n <= CONV_TOKENS; the number of taps is known at compile time, so that the loops unroll to
// straight code).  A thread keeps the channel's last inputs and its taps in registers: every input is read once for all the
// outputs it takes part in.  load() asks for everything that does not depend on the tokens' places, the rows in front of t0 among it
// (they count only if they are the same sequence's), so that one wait covers these loads and the looking up of the places.
template <int TAPS>
struct ConvChannel {
    static constexpr int H = TAPS - 1, TB = CONV_TOKENS;
    float front[TAPS], v[TB], w[TAPS], bias;
    __device__ __forceinline__ void load(const ConvSeg& g, int t0, int n, int c) {
        const float* base = g.in + (size_t)t0 * g.in_stride + g.col0 + c;
#pragma unroll
        for (int i = 0; i < TB; ++i) v[i] = i < n ? base[(size_t)i * g.in_stride] : 0.f;
#pragma unroll
        for (int j = 0; j < H; ++j) front[j] = t0 >= H - j ? base[-(ptrdiff_t)(H - j) * g.in_stride] : 0.f;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) w[j] = g.w[(size_t)c * TAPS + j];
        bias = g.bias ? g.bias[c] : 0.f;
    }
    // the outputs; m: the tokens' places (in shared memory).  Moves the state on for a token that is its sequence's only one
    __device__ __forceinline__ void run(const ConvSeg& g, const ConvToken* m, int t0, int n, int c, float (&y)[TB]) const {
        float u[TAPS];
#pragma unroll
        for (int i = 0; i < TB; ++i) {
            if (i >= n) break;
            if (i == 0 || m[i].avail == 0) {                           // the inputs before a first token: from the step, or from the state
                const float* srow = g.state + (size_t)m[i].slot * g.state_stride + c;
#pragma unroll
                for (int j = 0; j < H; ++j) {
                    const int back = H - j;                            // the input `back` positions before the token
                    u[j] = back <= m[i].avail ? front[j]
                         : back <= m[i].pos ? srow[(size_t)(H - (back - m[i].avail)) * g.channels] : 0.f;
                }
            } else {
#pragma unroll
                for (int j = 0; j < H; ++j) u[j] = u[j + 1];
            }
            u[H] = v[i];
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < TAPS; ++j) acc = fmaf(w[j], u[j], acc);
            y[i] = g.bias ? acc + bias : acc;
            if (m[i].single) {
                float* srow = g.state + (size_t)m[i].slot * g.state_stride + c;
#pragma unroll
                for (int j = 1; j < TAPS; ++j) srow[(size_t)(j - 1) * g.channels] = u[j];
            }
        }
    }
};

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

// the same, eight tokens a thread
template <int TAPS>
__global__ void __launch_bounds__(256) short_conv_tokens_kernel(ConvSeg g, ConvStep st, float* __restrict__ out, int act, int n_tokens) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int TB = CONV_TOKENS;
    __shared__ ConvToken token[TB];                 // looked up by one thread each
    const int c = blockIdx.y * blockDim.x + threadIdx.x, t0 = blockIdx.x * TB, n = min(TB, n_tokens - t0);
    ConvChannel<TAPS> ch;
    if (c < g.channels) ch.load(g, t0, n, c);
    if (threadIdx.x < n) token[threadIdx.x] = conv_token(st, t0 + threadIdx.x);
    __syncthreads();
    if (c >= g.channels) return;
    float y[TB];
    ch.run(g, token, t0, n, c, y);
#pragma unroll
    for (int i = 0; i < TB; ++i)
        if (i < n) out[(size_t)(t0 + i) * g.channels + c] = act == 1 ? silu_exact(y[i]) : y[i];
}

// The attention side: q, k and v channels [n_q * dk | n_kv * dk | n_kv * dv] are filtered, the first
// 2 * half dims of every q and k head turned by the token's position (dim i with dim i + half; (u, v) ->
// (u cos - v sin, v cos + u sin), table cs [N, half] of (cos, sin)), q stored [N, n_q, dk] and k, v written
// to the token's place in the cache (pools [pages, n_kv, PAGE, dk] and [pages, n_kv, PAGE, dv]).
// With `maps` > 1 a q or k head is that many parts side by side, each turned like a head of dk / maps dims, and q goes out as
// one row per part, [N, n_q * maps, dk], zero outside its part: against the same key rows each such row scores its part
// alone.
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
                from_f32(dst[d], u * cs.x - v * cs.y);
                from_f32(dst[other], v * cs.x + u * cs.y);
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

// the same, eight tokens a thread
template <int TAPS>
__global__ void __launch_bounds__(256, 3) conv_qkv_cache_tokens_kernel(ConvQkvArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int TB = CONV_TOKENS;
    __shared__ ConvToken token[TB];
    __shared__ size_t place[TB];                    // a token's row among all rows of a kv-head's first page: + head * PAGE
    const int t0 = blockIdx.x * TB, n = min(TB, a.n_tokens - t0);
    const int qk_heads = a.n_q + a.n_kv;
    const int part = a.dk / a.maps, per = part - a.half;  // work items of a part: pairs, then single dims
    const int rest = a.maps * per;                        // work items of a q or k head
    const int qk_items = qk_heads * rest, items = qk_items + a.n_kv * a.dv;
    bool known = false;
    // (every thread comes to the barrier)
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; !known || i < items; i += gridDim.y * blockDim.x) {
        const bool value = i >= qk_items;
        const int j = value ? i - qk_items : i, head = value ? j / a.dv : j / rest;
        const int mp = value ? 0 : j % rest / per, r = value ? j % a.dv : j % per, d0 = mp * part;
        const bool is_q = !value && head < a.n_q, turned = !value && r < a.half;
        const int d = value || turned ? r : r + a.half, other = r + a.half;
        const int c = value ? qk_heads * a.dk + j : head * a.dk + d0 + d;
        ConvChannel<TAPS> one, two;
        if (i < items) {
            one.load(a.seg, t0, n, c);
            if (turned) two.load(a.seg, t0, n, c + a.half);
        }
        if (!known) {
            if (threadIdx.x < n) {
                const ConvToken m = conv_token(a.st, t0 + threadIdx.x);
                token[threadIdx.x] = m;
                place[threadIdx.x] = (size_t)a.table[(size_t)m.slot * a.table_stride + m.pos / IDM_PAGE] * a.n_kv * IDM_PAGE + m.pos % IDM_PAGE;
            }
            __syncthreads();
            known = true;
            if (i >= items) break;
        }
        float u[TB], v[TB];
        one.run(a.seg, token, t0, n, c, u);
        if (turned) two.run(a.seg, token, t0, n, c + a.half, v);
#pragma unroll
        for (int k = 0; k < TB; ++k) {
            if (k >= n) break;
            if (value) {
                from_f32(a.v_pool[(place[k] + (size_t)head * IDM_PAGE) * a.dv + d], u[k]);
                continue;
            }
            T* row = is_q ? a.q_out + ((size_t)(t0 + k) * a.n_q + head) * a.maps * a.dk
                          : a.k_pool + (place[k] + (size_t)(head - a.n_q) * IDM_PAGE) * a.dk;
            T* dst = row + (is_q ? mp * a.dk : 0) + d0;
            if (turned) {
                const float2 cs = a.cs[(size_t)(t0 + k) * a.half + r];
                from_f32(dst[d], u[k] * cs.x - v[k] * cs.y);
                from_f32(dst[other], v[k] * cs.x + u[k] * cs.y);
            } else {
                from_f32(dst[d], u[k]);
            }
            if (is_q)
                for (int z = 0; z < a.maps; ++z)
                    if (z != mp) {
                        from_f32(row[z * a.dk + d0 + d], 0.f);
                        if (turned) from_f32(row[z * a.dk + d0 + other], 0.f);
                    }
        }
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
    const dim3 grid(many ? (n_tokens + CONV_TOKENS - 1) / CONV_TOKENS : n_tokens, across);
#define CONV_GO(TAPS_) case TAPS_: idm_launch(short_conv_kernel<TAPS_>, grid, dim3(256), 0, stream, g, st, out, act); break;
#define CONV_MANY(TAPS_) case TAPS_: idm_launch(short_conv_tokens_kernel<TAPS_>, grid, dim3(256), 0, stream, g, st, out, act, n_tokens); break;
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
    const bool many = (long long)(n_tokens / CONV_TOKENS) * across >= CONV_BLOCKS;
    int split = many ? across : (296 + n_tokens - 1) / n_tokens;
    if (split > across) split = across;
    if (split < 1) split = 1;
    const dim3 grid(many ? (n_tokens + CONV_TOKENS - 1) / CONV_TOKENS : n_tokens, split);
#define CONV_GO(TAPS_) case TAPS_: idm_launch(conv_qkv_cache_kernel<TAPS_>, grid, dim3(256), 0, stream, a); break;
#define CONV_MANY(TAPS_) case TAPS_: idm_launch(conv_qkv_cache_tokens_kernel<TAPS_>, grid, dim3(256), 0, stream, a); break;
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
