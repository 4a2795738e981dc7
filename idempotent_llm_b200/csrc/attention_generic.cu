// Attention over the cache for any head size up to 256, any number of heads and groups, with or without a window, for prompts
// and for single tokens; all arithmetic in 32-bit on the FMA units.
//
// A query at position p of sequence s sees keys j with max(0, p - window + 1) <= j <= p
// (window <= 0: all j <= p), the slot-causal rule of src/detllm/model.py:259-266; with keep_first > 0 also the
// keys j < keep_first, however far back they lie (the blocks that hold them are walked first, then the
// window's).  With chunk > 0 it sees the keys of its own chunk only, p - p % chunk <= j <= p (chunks counted from the
// sequence's start).  softcap > 0 bounds a score: cap * tanh(score / cap), after the scale and before the softmax.
// With score_bias there is no softmax: a visible key's weight is sigmoid(score + score_bias[head]) and nothing is divided.
//
// One order of summation.  Keys lie in blocks of 64 and runs of two blocks, both at absolute positions.  A score is one chain of
// FMAs over the head's dims.  Inside a run (max, sum, context) start from nothing and are rescaled block by block; a block's
// weights are added 16 apart and then by a butterfly, its values by one chain over its keys; the runs are folded in ascending
// order (a run whose scores all lie below a 32-bit number's range adds nothing).  A key that a row does not see takes no part in anything (the float analogue of the reference's integer sentinel,
// src/detllm/ops/di_softmax.py:45-58): it is left out of the maximum and its value is not touched, whatever it holds.  So a
// row's bits depend on its position and its visible keys alone, not on the step's batch, on the tile it falls in, on how
// the sequence was cut into steps, or on whether one thread block walks its runs or several do.
//
// A thread block takes a tile of 4, 16 or 32 rows (tokens x q-heads of one kv-head): keys and values of a block of 64 are read once
// for all of them, through shared memory; with 32 rows a thread has 2 rows x 4 keys of the scores and x 4 columns (per 64) of the
// context.
// What bounds it: for prompts the FMA rate and the shared-memory reads behind it, for single tokens the bytes of the cache
// and, with few sequences, the walk itself, so that steps with too few tiles for the SMs give every run's result to scratch
// (attention_runs_fold_kernel).  A layer of 16 heads (8 kv-heads) of 128 in 32-bit: 8 single tokens over 400 keys 19 us, over 2 000
// keys 48 us, 64 over 2 000 keys 337 us (3.1 TB/s), prompts of 350 and 263 tokens 83 us; with a warp per (token, q-head), which
// this replaces, the first took 490 us and the last 484 us.  Runs of 64 keys were faster over 400 keys (16 us) and slower over
// 2 000 (60 us).
//
// Keys of the current step may come from packed buffers k_new/v_new instead of the
// cache (windowed layers, whose ring cannot hold a whole prompt).
#include "common.cuh"

struct AttnArgs {
    const T* q; T* out;
    KVAddr cache;
    const T* k_new; const T* v_new;
    const int* positions; const int* slots; const int* q_start; const int* cu_q;
    int n_tokens, n_q, n_kv, hd;
    float scale; int window;
    // beyond plain attention (all off in idm_attention_generic):
    int dv;                       // width of a value row (keys have hd)
    const float* sink;            // [n_q] or null: exp(sink[head]) joins the softmax's denominator, with no key and no value
    const float* gate; int gate_stride;   // or null: out *= sigmoid(gate[t * gate_stride + head * dv + d])
    int out_stride, out_col;      // out[t * out_stride + out_col + head * dv + d]
    float out_scale;
    const float* slopes;          // [n_q] or null: slopes[head] * (p - j) is taken off the score of key j
    int gate_per_head;            // the gate is one number per head: gate[t * gate_stride + head]
    float softcap;                // > 0: score <- softcap * tanh(score / softcap)
    int keep_first;               // > 0: keys j < keep_first are seen from any distance
    int chunk;                    // > 0: only keys of the query's own chunk of so many positions are seen
    const float* score_bias;      // [n_q] or null: the weights are sigmoid(score + score_bias[head]), not a softmax
    int n_seqs;
    // the launch's cut: q-heads of a kv-head in a tile and how many such parts a kv-head has, tokens per tile, and whether
    // every sequence is one tile
    int tile_heads, head_parts, tile_tokens, tile_per_seq;
    float* scratch; int max_runs; // or null: one thread block walks all of a tile's runs
};

#define AG_THREADS 256
#define AG_KEYS 64                // keys of a block: one page of the cache (a ring is whole pages)
#define AG_RUN 128                // keys of a run
#define AG_PROW (AG_KEYS + 4)     // a row of weights in shared memory
// what a run's maximum starts from: the lowest finite number, so that scores of minus infinity (below a 32-bit number's range) weigh
// exp(-inf) = 0 where a run has no others
#define AG_LOWEST (-3.402823466e38f)
static_assert(AG_KEYS == IDM_PAGE, "a block of keys lies in one page");

__host__ __device__ __forceinline__ int pad4(int n) { return (n + 3) & ~3; }
// floats of a row's result of one run in scratch: maximum, sum, two unused, context
__host__ __device__ __forceinline__ int run_floats(int dv) { return pad4(dv) + 4; }

// one row from global memory to 32-bit numbers in shared memory by one warp, zeros up to a multiple of 4 elements.  32-bit rows on
// 16-byte borders go asynchronously (wait with copies_wait, then a barrier); others are there after the barrier, four elements at
// a time where the row starts on a border of four
__device__ __forceinline__ void copy_row(float* dst, const float* src, int width, int lane) {
    if ((width & 3) == 0 && ((uintptr_t)src & 15) == 0) {
        for (int d = lane * 4; d < width; d += 128)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + d)), "l"(src + d));
    } else {
        for (int d = lane; d < pad4(width); d += 32) dst[d] = d < width ? src[d] : 0.f;
    }
}
__device__ __forceinline__ void copy_row(float* dst, const __nv_bfloat16* src, int width, int lane) {
    if ((width & 3) == 0 && ((uintptr_t)src & 7) == 0) {
        for (int d = lane * 4; d < width; d += 128) {
            const uint2 u = *reinterpret_cast<const uint2*>(src + d);
            *reinterpret_cast<float4*>(dst + d) = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u),
                                                              __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
        }
    } else {
        for (int d = lane; d < pad4(width); d += 32) dst[d] = d < width ? to_f32(src[d]) : 0.f;
    }
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;"); }
template <int LEFT> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

__device__ __forceinline__ float sum16(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float max16(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// what a row has summed up so far, and a run's result onto it; the context's factors for both
struct RowSum { float m, l; };
__device__ __forceinline__ void fold_run(RowSum& t, float m, float l, float& keep, float& add) {
    const float mn = fmaxf(t.m, m);
    keep = expf(t.m - mn);
    add = expf(m - mn);
    t.l = fmaf(l, add, t.l * keep);
    t.m = mn;
}
__device__ __forceinline__ float fold_value(float o, float r, float keep, float add) { return fmaf(r, add, o * keep); }

// the first key a query at `pos` sees, and how many first keys of the sequence it sees besides
__device__ __forceinline__ int first_key(const AttnArgs& a, int pos) {
    return a.chunk > 0 ? pos - pos % a.chunk : a.window > 0 ? max(0, pos - a.window + 1) : 0;
}
__device__ __forceinline__ int kept_keys(const AttnArgs& a, int lo) { return a.window > 0 ? min(a.keep_first, lo) : 0; }
__device__ __forceinline__ bool sees_any(int pos, int lo, int keep, int j0, int j1) {     // of keys j0 .. j1 - 1
    return j0 <= pos && (j1 > lo || j0 < keep);
}

// one chain over four dims
__device__ __forceinline__ float dot4(float s, float4 q, float4 k) {
    s = fmaf(q.x, k.x, s); s = fmaf(q.y, k.y, s); s = fmaf(q.z, k.z, s);
    return fmaf(q.w, k.w, s);
}

// a finished element of the context: over the sum, gated, scaled, stored
__device__ __forceinline__ void finish_element(const AttnArgs& a, int t, int head, int d, float o, float inv, float head_gate) {
    o = o * inv * head_gate;
    if (a.gate && !a.gate_per_head) o = o / (1.0f + expf(-a.gate[(size_t)t * a.gate_stride + (size_t)head * a.dv + d]));
    if (a.out_scale != 1.f) o *= a.out_scale;
    from_f32(a.out[(size_t)t * a.out_stride + a.out_col + (size_t)head * a.dv + d], o);
}
__device__ __forceinline__ float gate_of_head(const AttnArgs& a, int t, int head) {
    return a.gate && a.gate_per_head ? 1.0f / (1.0f + expf(-a.gate[(size_t)t * a.gate_stride + head])) : 1.f;
}

static int attention_smem_bytes(int rows, int dc, int hd) {
    return 4 * ((rows + AG_KEYS) * (pad4(hd) + 4) + AG_KEYS * 64 * dc + rows * AG_PROW);
}

// a block's weights times its values onto the context; MASKED: some weights are -1, their values are not touched (a weight that is
// not a number is no -1)
template <int RI, int DC, bool MASKED>
__device__ __forceinline__ void add_values(float (&o)[RI][4 * DC], const float* pr, const float* vc) {
#pragma unroll 2
    for (int k = 0; k < AG_KEYS; k += 4) {
        float4 p4[RI];
#pragma unroll
        for (int i = 0; i < RI; ++i) p4[i] = *reinterpret_cast<const float4*>(pr + i * 16 * AG_PROW + k);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
#pragma unroll
            for (int c = 0; c < DC; ++c) {
                const float4 v4 = *reinterpret_cast<const float4*>(vc + (k + e) * 64 * DC + 64 * c);
#pragma unroll
                for (int i = 0; i < RI; ++i) {
                    const float w = e == 0 ? p4[i].x : e == 1 ? p4[i].y : e == 2 ? p4[i].z : p4[i].w;
                    if (MASKED && w < 0.f) continue;
                    o[i][4 * c] = fmaf(w, v4.x, o[i][4 * c]);
                    o[i][4 * c + 1] = fmaf(w, v4.y, o[i][4 * c + 1]);
                    o[i][4 * c + 2] = fmaf(w, v4.z, o[i][4 * c + 2]);
                    o[i][4 * c + 3] = fmaf(w, v4.w, o[i][4 * c + 3]);
                }
            }
        }
    }
}

// A thread block's tile: its sequence, tokens [t0, t1), heads and keys; and the walk over the keys' blocks
struct Tile {
    int s, t0, t1, g, head0, heads, slot, first_new, tok0, pos_first, pos_last, lo_last, main0, kept_end;

    // which tile of which sequence: 32 sequences at a time, one per lane of the first warp; false: none
    __device__ __forceinline__ bool find(const AttnArgs& a, int (&place)[2]) {
        if (a.tile_per_seq) {
            s = blockIdx.x; t0 = a.cu_q[s];
            if (t0 >= a.cu_q[s + 1]) return false;
        } else {
            const int lane = threadIdx.x & 31;
            if (threadIdx.x < 32) {
                int before = 0, seq = -1, first = 0;
                for (int s0 = 0; s0 < a.n_seqs && seq < 0; s0 += 32) {
                    const int i = s0 + lane, at = i < a.n_seqs ? a.cu_q[i] : 0;
                    const int tiles = i < a.n_seqs ? (a.cu_q[i + 1] - at + a.tile_tokens - 1) / a.tile_tokens : 0;
                    int upto = tiles;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += u; }
                    const int mine = (int)blockIdx.x - before - (upto - tiles);
                    const unsigned hit = __ballot_sync(0xffffffffu, mine >= 0 && mine < tiles);
                    if (hit) {
                        const int src = __ffs(hit) - 1;
                        seq = s0 + src;
                        first = __shfl_sync(0xffffffffu, at + mine * a.tile_tokens, src);
                    }
                    before += __shfl_sync(0xffffffffu, upto, 31);
                }
                if (lane == 0) { place[0] = seq; place[1] = first; }
            }
            __syncthreads();
            s = place[0]; t0 = place[1];
            if (s < 0) return false;
        }
        g = blockIdx.y / a.head_parts;
        const int part = blockIdx.y % a.head_parts, group = a.n_q / a.n_kv;
        head0 = g * group + part * a.tile_heads;
        heads = min(a.tile_heads, group - part * a.tile_heads);
        t1 = min(t0 + a.tile_tokens, a.cu_q[s + 1]);
        slot = a.slots[s]; first_new = a.k_new ? a.q_start[s] : 0x7fffffff; tok0 = a.cu_q[s];
        pos_first = a.positions[t0]; pos_last = a.positions[t1 - 1];
        const int lo_first = first_key(a, pos_first);
        lo_last = first_key(a, pos_last);
        main0 = lo_first / AG_KEYS * AG_KEYS;
        kept_end = min(kept_keys(a, lo_last), main0);
        return true;
    }
    __device__ __forceinline__ bool live(const AttnArgs& a, int r) const {
        return r < a.tile_tokens * a.tile_heads && t0 + r / a.tile_heads < t1 && r % a.tile_heads < heads;
    }
    // the first block to walk at or behind j (a block's start), or past the end: in ascending order those of the kept first keys,
    // then from the first row's first key on; with scratch, of this thread block's runs only
    __device__ __forceinline__ int next_block(const AttnArgs& a, int j) const {
        for (;;) {
            if (j < main0 && j >= kept_end) j = main0;
            if (j > pos_last) return 0x7fffffff;
            if (!a.scratch || (j / AG_RUN) % gridDim.z == blockIdx.z) return j;
            j = (j / AG_RUN + 1) * AG_RUN;
        }
    }
    // the queries of the tile's rows, zeros for rows that are not live
    __device__ __forceinline__ void copy_queries(const AttnArgs& a, float* qs, int rows, int row_f) const {
        const int lane = threadIdx.x & 31;
        for (int r = threadIdx.x >> 5; r < rows; r += AG_THREADS / 32) {
            if (live(a, r)) copy_row(qs + r * row_f, a.q + ((size_t)(t0 + r / a.tile_heads) * a.n_q + head0 + r % a.tile_heads) * a.hd, a.hd, lane);
            else for (int d = lane; d < row_f; d += 32) qs[r * row_f + d] = 0.f;
        }
    }
    // the keys (or values) of the block from j0 on, up to the last one a row sees
    __device__ __forceinline__ void copy_keys(const AttnArgs& a, int j0, float* dst, int row_f, bool values) const {
        const size_t page_row = j0 < first_new ? kv_row(a.cache, slot, j0, g) : 0;
        const int width = values ? a.dv : a.hd;
        const T* old = values ? a.cache.v : a.cache.k;
        const T* fresh = values ? a.v_new : a.k_new;
        for (int i = threadIdx.x >> 5; i < AG_KEYS; i += AG_THREADS / 32) {
            const int j = j0 + i;
            if (j > pos_last) break;
            const T* src = j >= first_new ? fresh + ((size_t)(tok0 + j - first_new) * a.n_kv + g) * width : old + (page_row + i) * width;
            copy_row(dst + i * row_f, src, width, threadIdx.x & 31);
        }
    }
};

// a row of queries as the kernels know it
struct Row {
    int pos, lo, keep, t, head;
    float slope, bias;
    __device__ __forceinline__ void set(const AttnArgs& a, const Tile& tile, int r) {
        t = tile.t0 + r / a.tile_heads; head = tile.head0 + r % a.tile_heads;
        const bool live = tile.live(a, r);
        pos = live ? a.positions[t] : -1;
        lo = live ? first_key(a, pos) : 0;
        keep = kept_keys(a, lo);
        slope = live && a.slopes ? a.slopes[head] : 0.f;
        bias = live && a.score_bias ? a.score_bias[head] : 0.f;
    }
    // a sink is a key of score sink[head] (not scaled) whose value is zero: the sums start from it
    __device__ __forceinline__ RowSum start(const AttnArgs& a) const {
        return RowSum{pos >= 0 && a.sink ? a.sink[head] : -INFINITY, a.sink ? 1.f : 0.f};
    }
};

// where a row's result of a run goes: maximum, sum, two unused, context
__device__ __forceinline__ float* run_result(const AttnArgs& a, const Row& row, int run) {
    return a.scratch + (((size_t)row.t * a.n_q + row.head) * a.max_runs + run) * run_floats(a.dv);
}

// Four scores of a row (keys j0 + tx + 16 j) become weights, -1 where the row does not see the key; the run's maximum and sum move on;
// returns what the run's context is multiplied by first.  Called by the 16 threads of a row side by side.
__device__ __forceinline__ float block_weights(const AttnArgs& a, const Row& row, int j0, int tx, float (&sc)[4], float& m_run, float& l_run) {
    bool seen[4];
    float top = AG_LOWEST;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int key = j0 + tx + 16 * j;
        float x = sc[j] * a.scale;
        if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
        if (a.slopes) x -= row.slope * (float)(row.pos - key);
        seen[j] = key <= row.pos && (key >= row.lo || key < row.keep);
        sc[j] = x;
        if (seen[j]) top = fmaxf(top, x);
    }
    top = fmaxf(m_run, max16(top));
    if (a.score_bias) {
#pragma unroll
        for (int j = 0; j < 4; ++j) sc[j] = seen[j] ? 1.0f / (1.0f + expf(-(sc[j] + row.bias))) : -1.f;
        return 1.f;
    }
    // (a row that sees nothing of the block stays as it is)
    const float alpha = sees_any(row.pos, row.lo, row.keep, j0, j0 + AG_KEYS) ? expf(m_run - top) : 1.f;
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        sc[j] = seen[j] ? expf(sc[j] - top) : -1.f;
        sum += seen[j] ? sc[j] : 0.f;
    }
    l_run = fmaf(l_run, alpha, sum16(sum));
    m_run = top;
    return alpha;
}

// Many rows.  RI: rows per thread (a tile has 16 RI); DC: value columns in pieces of 64
template <int RI, int DC>
__global__ void __launch_bounds__(AG_THREADS) attention_tile_kernel(AttnArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    __shared__ int place[2];
    constexpr int ROWS = 16 * RI, VROW = 64 * DC;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int qrow_f = pad4(a.hd) + 4;
    float* qs = smem;                                           // [ROWS][qrow_f]
    float* ks = qs + ROWS * qrow_f;                             // [AG_KEYS][qrow_f]
    float* vs = ks + AG_KEYS * qrow_f;                          // [AG_KEYS][VROW]
    float* ps = vs + AG_KEYS * VROW;                            // [ROWS][AG_PROW]: weights, -1 where a row does not see the key
    Tile tile;
    if (!tile.find(a, place)) return;
    Row row[RI];
    RowSum total[RI];
    float m_run[RI], l_run[RI], o_tot[RI][4 * DC], o_run[RI][4 * DC];
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        row[i].set(a, tile, ty + 16 * i);
        total[i] = row[i].start(a);
        m_run[i] = AG_LOWEST; l_run[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 4 * DC; ++c) o_tot[i][c] = o_run[i][c] = 0.f;
    }
    int j0 = tile.next_block(a, 0);
    if (j0 > tile.pos_last) return;
    tile.copy_queries(a, qs, ROWS, qrow_f);
    tile.copy_keys(a, j0, ks, qrow_f, false); copies_commit();
    tile.copy_keys(a, j0, vs, VROW, true); copies_commit();
    while (j0 <= tile.pos_last) {
        const int after = tile.next_block(a, j0 + AG_KEYS);
        copies_wait<1>();
        __syncthreads();                                        // this block's keys (and the queries) are there
        float sc[RI][4];
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) sc[i][j] = 0.f;
        const float* qr = qs + ty * qrow_f;
        const float* kr = ks + tx * qrow_f;
#pragma unroll 4
        for (int d = 0; d < a.hd; d += 4) {
            float4 q4[RI];
#pragma unroll
            for (int i = 0; i < RI; ++i) q4[i] = *reinterpret_cast<const float4*>(qr + i * 16 * qrow_f + d);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 k4 = *reinterpret_cast<const float4*>(kr + j * 16 * qrow_f + d);
#pragma unroll
                for (int i = 0; i < RI; ++i) sc[i][j] = dot4(sc[i][j], q4[i], k4);
            }
        }
        __syncthreads();                                        // everyone has read the keys
        if (after <= tile.pos_last) tile.copy_keys(a, after, ks, qrow_f, false);
        copies_commit();
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const float alpha = block_weights(a, row[i], j0, tx, sc[i], m_run[i], l_run[i]);
#pragma unroll
            for (int c = 0; c < 4 * DC; ++c) o_run[i][c] *= alpha;
#pragma unroll
            for (int j = 0; j < 4; ++j) ps[(ty + 16 * i) * AG_PROW + tx + 16 * j] = sc[i][j];
        }
        copies_wait<1>();
        __syncthreads();                                        // this block's values and everyone's weights are there
        // (whether every live row sees every key of the block)
        if (j0 + AG_KEYS - 1 <= tile.pos_first && j0 >= tile.lo_last) add_values<RI, DC, false>(o_run, ps + ty * AG_PROW, vs + tx * 4);
        else add_values<RI, DC, true>(o_run, ps + ty * AG_PROW, vs + tx * 4);
        if (after > tile.pos_last || after / AG_RUN != j0 / AG_RUN) {                // the run's end
            const int run = j0 / AG_RUN;
#pragma unroll
            for (int i = 0; i < RI; ++i) {
                if (sees_any(row[i].pos, row[i].lo, row[i].keep, run * AG_RUN, (run + 1) * AG_RUN)) {
                    if (a.scratch) {
                        float* dst = run_result(a, row[i], run);
                        if (tx == 0) { dst[0] = m_run[i]; dst[1] = l_run[i]; }
#pragma unroll
                        for (int c = 0; c < 4 * DC; ++c) {
                            const int d = tx * 4 + (c >> 2) * 64 + (c & 3);
                            if (d < a.dv) dst[4 + d] = o_run[i][c];
                        }
                    } else {
                        float kept = 1.f, add = 1.f;
                        if (!a.score_bias) fold_run(total[i], m_run[i], l_run[i], kept, add);
#pragma unroll
                        for (int c = 0; c < 4 * DC; ++c) o_tot[i][c] = fold_value(o_tot[i][c], o_run[i][c], kept, add);
                    }
                }
                m_run[i] = AG_LOWEST; l_run[i] = 0.f;
#pragma unroll
                for (int c = 0; c < 4 * DC; ++c) o_run[i][c] = 0.f;
            }
        }
        __syncthreads();                                        // everyone has read the values and the weights
        if (after <= tile.pos_last) tile.copy_keys(a, after, vs, VROW, true);
        copies_commit();
        j0 = after;
    }
    if (a.scratch) return;
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        if (row[i].pos < 0) continue;
        const float inv = a.score_bias ? 1.0f : 1.0f / total[i].l, hg = gate_of_head(a, row[i].t, row[i].head);
#pragma unroll
        for (int c = 0; c < 4 * DC; ++c) {
            const int d = tx * 4 + (c >> 2) * 64 + (c & 3);
            if (d < a.dv) finish_element(a, row[i].t, row[i].head, d, o_tot[i][c], inv, hg);
        }
    }
}

// Few rows (up to 16: single tokens): the same sums with the work cut otherwise.  In the kernel above a row belongs to 16 threads, so two
// rows would keep one warp busy; here a thread takes (row, key) pairs for the scores and (row, column) pairs for the context, and
// only the weights are made 16 threads a row.  R: the most rows; DC: value columns in pieces of 64.
template <int R, int DC>
__global__ void __launch_bounds__(AG_THREADS) attention_rows_kernel(AttnArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    __shared__ float row_alpha[R], row_m[R], row_l[R];
    __shared__ int place[2];
    constexpr int VROW = 64 * DC, PASS = AG_THREADS / VROW, ITEMS = (R + PASS - 1) / PASS;   // rows of a pass over the columns
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int qrow_f = pad4(a.hd) + 4;
    float* qs = smem;                                           // [R][qrow_f]
    float* ks = qs + R * qrow_f;
    float* vs = ks + AG_KEYS * qrow_f;
    float* ps = vs + AG_KEYS * VROW;                            // [R][AG_PROW]: scores, then weights
    Tile tile;
    if (!tile.find(a, place)) return;
    int j0 = tile.next_block(a, 0);
    if (j0 > tile.pos_last) return;
    tile.copy_queries(a, qs, R, qrow_f);
    tile.copy_keys(a, j0, ks, qrow_f, false); copies_commit();
    tile.copy_keys(a, j0, vs, VROW, true); copies_commit();
    const int live = (tile.t1 - tile.t0) * a.tile_heads;        // rows (a part with fewer heads has some that see nothing)
    Row mine;                                                   // of the weights
    mine.set(a, tile, ty);
    float m_run = AG_LOWEST, l_run = 0.f;
    const int col = threadIdx.x % VROW, row0 = threadIdx.x / VROW;
    Row item[ITEMS];
    RowSum total[ITEMS];
    float o_tot[ITEMS], o_run[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        item[i].set(a, tile, row0 + i * PASS);
        total[i] = item[i].start(a);
        o_tot[i] = o_run[i] = 0.f;
    }
    while (j0 <= tile.pos_last) {
        const int after = tile.next_block(a, j0 + AG_KEYS);
        copies_wait<1>();
        __syncthreads();                                        // this block's keys (and the queries) are there
        for (int p = threadIdx.x; p < live * AG_KEYS; p += AG_THREADS) {
            const int r = p / AG_KEYS, k = p % AG_KEYS;
            const float* qr = qs + r * qrow_f;
            const float* kr = ks + k * qrow_f;
            float dot = 0.f;
#pragma unroll 8
            for (int d = 0; d < a.hd; d += 4) dot = dot4(dot, *reinterpret_cast<const float4*>(qr + d), *reinterpret_cast<const float4*>(kr + d));
            ps[r * AG_PROW + k] = dot;
        }
        __syncthreads();                                        // everyone has read the keys; the scores are there
        if (after <= tile.pos_last) tile.copy_keys(a, after, ks, qrow_f, false);
        copies_commit();
        if (threadIdx.x < (live * 16 + 31) / 32 * 32 && ty < R) {                    // whole warps
            float sc[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) sc[j] = ps[ty * AG_PROW + tx + 16 * j];
            const float alpha = block_weights(a, mine, j0, tx, sc, m_run, l_run);
#pragma unroll
            for (int j = 0; j < 4; ++j) ps[ty * AG_PROW + tx + 16 * j] = sc[j];
            if (tx == 0) { row_alpha[ty] = alpha; row_m[ty] = m_run; row_l[ty] = l_run; }
        }
        copies_wait<1>();
        __syncthreads();                                        // this block's values and the weights are there
        const bool whole = j0 + AG_KEYS - 1 <= tile.pos_first && j0 >= tile.lo_last;
        const bool run_ends = after > tile.pos_last || after / AG_RUN != j0 / AG_RUN;
        const int run = j0 / AG_RUN;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int r = row0 + i * PASS;
            if (r >= live) continue;
            float o = o_run[i] * row_alpha[r];
            const float* pr = ps + r * AG_PROW;
            const float* vc = vs + col;
#pragma unroll 4
            for (int k = 0; k < AG_KEYS; k += 4) {
                const float4 w = *reinterpret_cast<const float4*>(pr + k);
                const float v0 = vc[k * VROW], v1 = vc[(k + 1) * VROW], v2 = vc[(k + 2) * VROW], v3 = vc[(k + 3) * VROW];
                o = whole || !(w.x < 0.f) ? fmaf(w.x, v0, o) : o;
                o = whole || !(w.y < 0.f) ? fmaf(w.y, v1, o) : o;
                o = whole || !(w.z < 0.f) ? fmaf(w.z, v2, o) : o;
                o = whole || !(w.w < 0.f) ? fmaf(w.w, v3, o) : o;
            }
            o_run[i] = o;
            if (run_ends) {
                if (sees_any(item[i].pos, item[i].lo, item[i].keep, run * AG_RUN, (run + 1) * AG_RUN)) {
                    const float m = row_m[r], l = row_l[r];
                    if (a.scratch) {
                        float* dst = run_result(a, item[i], run);
                        if (col == 0) { dst[0] = m; dst[1] = l; }
                        if (col < a.dv) dst[4 + col] = o;
                    } else {
                        float kept = 1.f, add = 1.f;
                        if (!a.score_bias) fold_run(total[i], m, l, kept, add);
                        o_tot[i] = fold_value(o_tot[i], o, kept, add);
                    }
                }
                o_run[i] = 0.f;
            }
        }
        if (run_ends) { m_run = AG_LOWEST; l_run = 0.f; }
        __syncthreads();                                        // everyone has read the values and the weights
        if (after <= tile.pos_last) tile.copy_keys(a, after, vs, VROW, true);
        copies_commit();
        j0 = after;
    }
    if (a.scratch) return;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        if (row0 + i * PASS >= live || item[i].pos < 0 || col >= a.dv) continue;
        finish_element(a, item[i].t, item[i].head, col, o_tot[i], a.score_bias ? 1.0f : 1.0f / total[i].l,
                       gate_of_head(a, item[i].t, item[i].head));
    }
}

// One row a warp, for single tokens whose tiles would have a row or two (attention_by_warps): a lane has two keys of a block for the
// scores and every 32nd column for the context, keys and values come straight from memory.  The same sums in the same order: four
// weights 16 apart lie in lanes 16 apart.  NC: columns of a lane.
template <int NC>
__global__ void __launch_bounds__(AG_THREADS) attention_warp_kernel(AttnArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31;
    const long long id = (long long)blockIdx.x * (AG_THREADS / 32) + (threadIdx.x >> 5);
    if (id >= (long long)a.n_tokens * a.n_q) return;            // (warps leave whole; there is no block barrier)
    const int t = (int)(id / a.n_q), head = (int)(id % a.n_q), g = head / (a.n_q / a.n_kv);
    const int pos = a.positions[t], slot = a.slots[t];          // (every sequence has one token: sequence t)
    const int first_new = a.k_new ? a.q_start[t] : 0x7fffffff;
    const int lo = first_key(a, pos), keep = kept_keys(a, lo), main0 = lo / AG_KEYS * AG_KEYS, kept_end = min(keep, main0);
    float* qs = smem + (threadIdx.x >> 5) * pad4(a.hd);
    for (int d = lane; d < a.hd; d += 32) qs[d] = to_f32(a.q[((size_t)t * a.n_q + head) * a.hd + d]);
    __syncwarp();
    const float slope = a.slopes ? a.slopes[head] : 0.f, bias = a.score_bias ? a.score_bias[head] : 0.f;
    RowSum total{a.sink ? a.sink[head] : -INFINITY, a.sink ? 1.f : 0.f};
    float m_run = AG_LOWEST, l_run = 0.f, o_tot[NC], o_run[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) o_tot[i] = o_run[i] = 0.f;
    for (int j0 = kept_end > 0 ? 0 : main0; j0 <= pos;) {
        int after = j0 + AG_KEYS;
        if (after < main0 && after >= kept_end) after = main0;
        const size_t page_row = j0 < first_new ? kv_row(a.cache, slot, j0, g) : 0;
        auto row_of = [&](const T* old, const T* fresh, int width, int key) {
            return key >= first_new ? fresh + ((size_t)(t + key - first_new) * a.n_kv + g) * width : old + (page_row + (key - j0)) * width;
        };
        float w[2];
        bool seen[2];
        float top = AG_LOWEST;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int key = j0 + lane + 32 * u;
            seen[u] = key <= pos && (key >= lo || key < keep);
            w[u] = 0.f;
            if (!seen[u]) continue;
            const T* kr = row_of(a.cache.k, a.k_new, a.hd, key);
            float dot = 0.f;
            if (a.hd % Vec16<T>::N == 0) {
                for (int d = 0; d < a.hd; d += Vec16<T>::N) {
                    Vec16<T> kv; kv.load(kr + d);
#pragma unroll
                    for (int e = 0; e < Vec16<T>::N; ++e) dot = fmaf(qs[d + e], kv.get(e), dot);
                }
            } else {                                            // rows that do not start on 16-byte borders
                for (int d = 0; d < a.hd; ++d) dot = fmaf(qs[d], to_f32(kr[d]), dot);
            }
            float x = dot * a.scale;
            if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
            if (a.slopes) x -= slope * (float)(pos - key);
            w[u] = x;
            top = fmaxf(top, x);
        }
        float alpha = 1.f;
        if (a.score_bias) {
#pragma unroll
            for (int u = 0; u < 2; ++u) w[u] = 1.0f / (1.0f + expf(-(w[u] + bias)));
        } else {
            top = fmaxf(m_run, warp_max(top));
            alpha = expf(m_run - top);
            float mine[2], other[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                w[u] = expf(w[u] - top);
                mine[u] = seen[u] ? w[u] : 0.f;
                other[u] = __shfl_xor_sync(0xffffffffu, mine[u], 16);
            }
            const bool low = lane < 16;                         // keys 0, 16, 32, 48 from the lane's sixteenth on, in this order
            float sum = 0.f;
            sum += low ? mine[0] : other[0]; sum += low ? other[0] : mine[0];
            sum += low ? mine[1] : other[1]; sum += low ? other[1] : mine[1];
            l_run = fmaf(l_run, alpha, sum16(sum));
            m_run = top;
        }
#pragma unroll
        for (int i = 0; i < NC; ++i) o_run[i] *= alpha;
        const unsigned live[2] = {__ballot_sync(0xffffffffu, seen[0]), __ballot_sync(0xffffffffu, seen[1])};
#pragma unroll
        for (int u = 0; u < 2; ++u)
            for (int k0 = 0; k0 < 32 && live[u] >> k0; k0 += 8) {                // eight rows' loads at a time, up to the last one seen
                float v[8][NC];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const bool in = (live[u] >> (k0 + k)) & 1u;
                    const T* vr = in ? row_of(a.cache.v, a.v_new, a.dv, j0 + 32 * u + k0 + k) : nullptr;
#pragma unroll
                    for (int i = 0; i < NC; ++i) v[k][i] = in && lane + 32 * i < a.dv ? to_f32(vr[lane + 32 * i]) : 0.f;
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float wk = __shfl_sync(0xffffffffu, w[u], k0 + k);
                    if (!((live[u] >> (k0 + k)) & 1u)) continue;
#pragma unroll
                    for (int i = 0; i < NC; ++i) o_run[i] = fmaf(wk, v[k][i], o_run[i]);
                }
            }
        if (after > pos || after / AG_RUN != j0 / AG_RUN) {     // the run's end
            float kept = 1.f, add = 1.f;
            if (!a.score_bias) fold_run(total, m_run, l_run, kept, add);
#pragma unroll
            for (int i = 0; i < NC; ++i) { o_tot[i] = fold_value(o_tot[i], o_run[i], kept, add); o_run[i] = 0.f; }
            m_run = AG_LOWEST; l_run = 0.f;
        }
        j0 = after;
    }
    const float inv = a.score_bias ? 1.0f : 1.0f / total.l, hg = gate_of_head(a, t, head);
#pragma unroll
    for (int i = 0; i < NC; ++i)
        if (lane + 32 * i < a.dv) finish_element(a, t, head, lane + 32 * i, o_tot[i], inv, hg);
}

// the runs' results of a row (a thread block) from scratch, in ascending order; a thread per column.  (Only layers without a window or
// chunks come here: a row sees something of every run up to its own.)
__global__ void __launch_bounds__(256) attention_runs_fold_kernel(AttnArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x / a.n_q, head = blockIdx.x % a.n_q, d = threadIdx.x;
    const int runs = a.positions[t] / AG_RUN + 1;
    const float* src = a.scratch + ((size_t)t * a.n_q + head) * a.max_runs * run_floats(a.dv);
    RowSum total{a.sink ? a.sink[head] : -INFINITY, a.sink ? 1.f : 0.f};
    float o = 0.f;
    for (int r0 = 0; r0 < runs; r0 += 8) {                      // eight runs' loads at a time
        float m[8], l[8], v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (r0 + i < runs) {
                const float* p = src + (size_t)(r0 + i) * run_floats(a.dv);
                m[i] = p[0]; l[i] = p[1]; v[i] = d < a.dv ? p[4 + d] : 0.f;
            }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (r0 + i < runs) {
                float kept = 1.f, add = 1.f;
                if (!a.score_bias) fold_run(total, m[i], l[i], kept, add);
                o = fold_value(o, v[i], kept, add);
            }
    }
    if (d < a.dv) finish_element(a, t, head, d, o, a.score_bias ? 1.0f : 1.0f / total.l, gate_of_head(a, t, head));
}

// How a step is cut.  Tiles of 4 or 16 rows where no sequence brings more than that for a kv-head (single tokens), else of 32.  Runs go
// through scratch where the tiles would leave SMs without one, the layer has no bound on its keys (a window's walk is
// short), and the results take at most 64 MB.  Measured at 16 heads (8 kv-heads) of 128, us with runs apart / walked by one thread
// block: 1 sequence of 400 keys 15 / 34, of 4 000 keys 26 / 294; 8 of 2 000 48 / 155; 32 of 400 38 / 46 (256 tiles); 64 fill
// the SMs.  As many thread blocks share a tile's runs as make four blocks an SM.
#define AG_SCRATCH_MOST (16ll << 20)
struct AttnCut { int rows, tile_heads, head_parts, tile_tokens, tiles, runs_z, max_runs; long long scratch; };
static AttnCut attention_cut(int n_tokens, int n_seqs, int max_q_len, int max_kv_len, int n_q, int n_kv, int dv, bool bounded) {
    AttnCut c;
    const int group = n_q / n_kv;
    const long long most = (long long)max_q_len * group;
    c.rows = most <= 4 ? 4 : most <= 16 ? 16 : 32;
    c.tile_heads = group < c.rows ? group : c.rows;
    c.head_parts = (group + c.tile_heads - 1) / c.tile_heads;
    c.tile_tokens = c.rows / c.tile_heads;
    c.tiles = max_q_len <= c.tile_tokens ? n_seqs : n_tokens / c.tile_tokens + n_seqs;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long blocks = (long long)c.tiles * n_kv * c.head_parts;
    c.max_runs = (max_kv_len + AG_RUN - 1) / AG_RUN;
    c.scratch = (long long)n_tokens * n_q * c.max_runs * run_floats(dv);
    if (bounded || c.max_runs <= 1 || blocks >= 2 * sms || c.scratch > AG_SCRATCH_MOST) c.scratch = 0;
    const long long z = (4ll * sms + blocks - 1) / blocks;
    c.runs_z = c.scratch == 0 ? 1 : z < c.max_runs ? (int)z : c.max_runs;
    return c;
}

// floats of scratch a step's runs take (0: none; `bounded`: the layer has a window or chunks)
extern "C" long long idm_attention_generic_scratch_floats(int n_tokens, int n_seqs, int max_q_len, int max_kv_len, int n_q, int n_kv,
                                                          int dv, int bounded) {
    if (n_tokens <= 0 || n_kv <= 0 || n_q < n_kv) return 0;
    return attention_cut(n_tokens, n_seqs, max_q_len, max_kv_len, n_q, n_kv, dv, bounded != 0).scratch;
}

// (`most`: what the kernel's widest heads take.  The same limit from every call: a smaller one from another thread would have this
// launch refused.)
template <typename Kernel>
static int attention_launch(Kernel kernel, const AttnArgs& a, dim3 grid, int bytes, int most, cudaStream_t stream) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    IDM_REQUIRE(e == cudaSuccess, "attention: %d bytes of shared memory: %s", most, cudaGetErrorString(e));
    idm_launch(kernel, grid, dim3(AG_THREADS), bytes, stream, a);
    return 0;
}
template <int DC>
static int attention_launch_rows(int rows, const AttnArgs& a, dim3 grid, cudaStream_t stream) {
    const int bytes = attention_smem_bytes(rows, DC, a.hd), most = attention_smem_bytes(rows, DC, IDM_MAX_HEAD_DIM);
    return rows == 4 ? attention_launch(attention_rows_kernel<4, DC>, a, grid, bytes, most, stream)
         : rows == 16 ? attention_launch(attention_rows_kernel<16, DC>, a, grid, bytes, most, stream)
                      : attention_launch(attention_tile_kernel<2, DC>, a, grid, bytes, most, stream);
}

// Single tokens a warp a row, from 512 rows on: where a tile would hold one row (as many kv-heads as q-heads) in bfloat16, whose rows a tile's
// block cannot copy asynchronously, and where a window or chunks leave a short walk (bfloat16: up to three q-heads a kv-head).  Measured, us
// by warps / in tiles, 32 heads of 64 (16 of 32) in bfloat16: 64 tokens behind 100 keys 46 / 101 (31 / 56), behind 700 420 / 885 (285 / 396),
// 200 behind 300 391 / 1 235 (163 / 607), a window of 64 35 / 132 (23 / 64; in 32-bit 30 / 84, 16 / 48; 24 heads over 8 of 96 32 / 42);
// 8 tokens behind 30 13 / 9 (256 rows).  Without a window in 32-bit, or with two q-heads a kv-head in either type, tiles are faster
// (16 heads over 8 of 128, 64 tokens behind 700 keys: 276, a warp a row 643).
static bool attention_by_warps(const AttnArgs& a, const AttnCut& c, int n_seqs, int max_q_len) {
    const int group = a.n_q / a.n_kv;
    const bool bounded = a.window > 0 || a.chunk > 0, wide = sizeof(T) == 4;
    return c.scratch == 0 && max_q_len == 1 && a.n_tokens == n_seqs && (long long)a.n_tokens * a.n_q >= 512 && (wide ? bounded && group == 1 : group == 1 || (bounded && group <= 3));
}

static int attention_generic_launch(AttnArgs& a, int n_seqs, int max_q_len, int max_kv_len, float* scratch, cudaStream_t stream) {
    IDM_REQUIRE(n_seqs > 0 && max_q_len > 0 && max_kv_len > 0, "attention: %d sequences, at most %d tokens, %d keys", n_seqs, max_q_len, max_kv_len);
    IDM_REQUIRE(a.cache.ring % AG_KEYS == 0, "attention: a ring of %d keys is no multiple of %d", a.cache.ring, AG_KEYS);
    const AttnCut c = attention_cut(a.n_tokens, n_seqs, max_q_len, max_kv_len, a.n_q, a.n_kv, a.dv, a.window > 0 || a.chunk > 0);
    IDM_REQUIRE(c.scratch == 0 || scratch, "attention: the step's runs need scratch");
    IDM_REQUIRE((long long)a.n_kv * c.head_parts <= 65535, "attention: %d kv-heads", a.n_kv);
    a.n_seqs = n_seqs; a.tile_heads = c.tile_heads; a.head_parts = c.head_parts; a.tile_tokens = c.tile_tokens;
    a.scratch = c.scratch ? scratch : nullptr; a.max_runs = c.max_runs;
    if (attention_by_warps(a, c, n_seqs, max_q_len)) {
        const dim3 rows((unsigned)(((long long)a.n_tokens * a.n_q + AG_THREADS / 32 - 1) / (AG_THREADS / 32)));
        const size_t bytes = sizeof(float) * (AG_THREADS / 32) * pad4(a.hd);
        idm_launch(a.dv <= 32 ? attention_warp_kernel<1> : a.dv <= 64 ? attention_warp_kernel<2> : a.dv <= 128 ? attention_warp_kernel<4> : attention_warp_kernel<8>,
                   rows, dim3(AG_THREADS), bytes, stream, a);
        IDM_LAUNCH_CHECK("attention_generic");
        return 0;
    }
    const dim3 grid(c.tiles, a.n_kv * c.head_parts, c.runs_z);
    a.tile_per_seq = max_q_len <= c.tile_tokens;
    const int rc = a.dv <= 64 ? attention_launch_rows<1>(c.rows, a, grid, stream)
                 : a.dv <= 128 ? attention_launch_rows<2>(c.rows, a, grid, stream) : attention_launch_rows<4>(c.rows, a, grid, stream);
    if (rc) return rc;
    if (a.scratch) idm_launch(attention_runs_fold_kernel, dim3(a.n_tokens * a.n_q), dim3((a.dv + 31) / 32 * 32), 0, stream, a);
    IDM_LAUNCH_CHECK("attention_generic");
    return 0;
}

extern "C" int idm_attention_generic(const void* q, void* out, void* k_pool, void* v_pool, const int* table,
                                     int table_stride, int ring, const void* k_new, const void* v_new,
                                     const int* positions, const int* slots, const int* q_start, const int* cu_q, int n_tokens, int n_seqs, int max_q_len,
                                     int max_kv_len, float* scratch, int n_q, int n_kv,
                                     int hd, float scale, int window, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    IDM_REQUIRE(hd > 0 && hd % Vec16<T>::N == 0 && hd <= IDM_MAX_HEAD_DIM,
                "attention: head_dim=%d must be a multiple of %d and at most %d", hd, Vec16<T>::N,
                IDM_MAX_HEAD_DIM);
    IDM_REQUIRE(n_kv > 0 && n_q % n_kv == 0, "attention: %d q-heads are no multiple of %d kv-heads", n_q, n_kv);
    IDM_REQUIRE((k_new == nullptr) == (v_new == nullptr), "attention: k_new and v_new come together");
    AttnArgs a;
    a.q = (const T*)q; a.out = (T*)out;
    a.cache = KVAddr{(T*)k_pool, (T*)v_pool, table, table_stride, ring, n_kv, hd};
    a.k_new = (const T*)k_new; a.v_new = (const T*)v_new;
    a.positions = positions; a.slots = slots; a.q_start = q_start; a.cu_q = cu_q;
    a.n_tokens = n_tokens; a.n_q = n_q; a.n_kv = n_kv; a.hd = hd; a.scale = scale; a.window = window;
    a.dv = hd; a.sink = nullptr; a.gate = nullptr; a.gate_stride = 0; a.out_stride = n_q * hd; a.out_col = 0; a.out_scale = 1.f;
    a.slopes = nullptr; a.gate_per_head = 0; a.softcap = 0.f; a.keep_first = 0; a.chunk = 0; a.score_bias = nullptr;
    return attention_generic_launch(a, n_seqs, max_q_len, max_kv_len, scratch, stream);
}

// The same walk over the cache with what a gated attention with a sink adds: value rows of their own width
// `dv`, a learned score per head that joins the softmax's denominator without a key or a value, and the
// result times sigmoid(gate) times a constant, stored at a column offset of a wider buffer (gate: 32-bit
// [N, gate_stride], columns head * dv + d).  All keys come from the cache.
extern "C" int idm_attention_sink(const void* q, void* out, int out_stride, int out_col, float out_scale,
                                  void* k_pool, void* v_pool, const int* table, int table_stride,
                                  const float* sink, const float* gate, int gate_stride,
                                  const int* positions, const int* slots, const int* q_start, const int* cu_q, int n_tokens, int n_seqs, int max_q_len,
                                     int max_kv_len, float* scratch, int n_q, int n_kv,
                                  int hd, int dv, float scale, int window, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    IDM_REQUIRE(hd > 0 && hd <= IDM_MAX_HEAD_DIM && dv > 0 && dv <= IDM_MAX_HEAD_DIM,
                "attention: key and value sizes %d, %d must be at most %d", hd, dv, IDM_MAX_HEAD_DIM);
    IDM_REQUIRE(n_kv > 0 && n_q % n_kv == 0, "attention: %d q-heads are no multiple of %d kv-heads", n_q, n_kv);
    IDM_REQUIRE(out_col >= 0 && out_col + n_q * dv <= out_stride, "attention: columns %d..%d of rows of %d", out_col,
                out_col + n_q * dv, out_stride);
    AttnArgs a;
    a.q = (const T*)q; a.out = (T*)out;
    a.cache = KVAddr{(T*)k_pool, (T*)v_pool, table, table_stride, 0, n_kv, hd};
    a.k_new = nullptr; a.v_new = nullptr;
    a.positions = positions; a.slots = slots; a.q_start = q_start; a.cu_q = cu_q;
    a.n_tokens = n_tokens; a.n_q = n_q; a.n_kv = n_kv; a.hd = hd; a.scale = scale; a.window = window;
    a.dv = dv; a.sink = sink; a.gate = gate; a.gate_stride = gate_stride; a.out_stride = out_stride; a.out_col = out_col;
    a.out_scale = out_scale;
    a.slopes = nullptr; a.gate_per_head = 0; a.softcap = 0.f; a.keep_first = 0; a.chunk = 0; a.score_bias = nullptr;
    return attention_generic_launch(a, n_seqs, max_q_len, max_kv_len, scratch, stream);
}

// The same walk once more with every option this kernel has: a window over a cache that keeps all keys (ring 0) or
// a ring, a sink, a slope per head whose product with the distance p - j is taken off the score, a gate that is
// one number per head (gate_per_head) or one per channel, a cap on the scores and first keys that every query sees
// (keep_first; not with a ring, which does not keep them), chunks instead of a window, and sigmoid weights
// (score_bias; there is no denominator then, so no sink).
extern "C" int idm_attention_biased(const void* q, void* out, int out_stride, int out_col, float out_scale,
                                    void* k_pool, void* v_pool, const int* table, int table_stride, int ring,
                                    const float* sink, const float* slopes, const float* gate, int gate_stride,
                                    int gate_per_head, const int* positions, const int* slots,
                                    const int* q_start, const int* cu_q, int n_tokens, int n_seqs, int max_q_len,
                                     int max_kv_len, float* scratch, int n_q, int n_kv,
                                    int hd, int dv, float scale, int window, float softcap, int keep_first, int chunk,
                                    const float* score_bias, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    IDM_REQUIRE(hd > 0 && hd <= IDM_MAX_HEAD_DIM && dv > 0 && dv <= IDM_MAX_HEAD_DIM,
                "attention: key and value sizes %d, %d must be at most %d", hd, dv, IDM_MAX_HEAD_DIM);
    IDM_REQUIRE(n_kv > 0 && n_q % n_kv == 0, "attention: %d q-heads are no multiple of %d kv-heads", n_q, n_kv);
    IDM_REQUIRE(out_col >= 0 && out_col + n_q * dv <= out_stride, "attention: columns %d..%d of rows of %d", out_col,
                out_col + n_q * dv, out_stride);
    IDM_REQUIRE(keep_first >= 0 && softcap >= 0.f && (keep_first == 0 || ring == 0),
                "attention: keep_first=%d softcap=%g ring=%d (a ring does not keep a sequence's first keys)", keep_first, softcap, ring);
    IDM_REQUIRE(chunk >= 0 && (chunk == 0 || (window <= 0 && ring == 0)), "attention: chunks of %d with a window of %d, ring %d", chunk, window, ring);
    IDM_REQUIRE(score_bias == nullptr || sink == nullptr, "attention: sigmoid weights have no denominator for a sink to join");
    AttnArgs a;
    a.q = (const T*)q; a.out = (T*)out;
    a.cache = KVAddr{(T*)k_pool, (T*)v_pool, table, table_stride, ring, n_kv, hd};
    a.k_new = nullptr; a.v_new = nullptr;
    a.positions = positions; a.slots = slots; a.q_start = q_start; a.cu_q = cu_q;
    a.n_tokens = n_tokens; a.n_q = n_q; a.n_kv = n_kv; a.hd = hd; a.scale = scale; a.window = window;
    a.dv = dv; a.sink = sink; a.gate = gate; a.gate_stride = gate_stride; a.out_stride = out_stride; a.out_col = out_col;
    a.out_scale = out_scale; a.slopes = slopes; a.gate_per_head = gate_per_head;
    a.softcap = softcap; a.keep_first = keep_first; a.chunk = chunk; a.score_bias = score_bias;
    return attention_generic_launch(a, n_seqs, max_q_len, max_kv_len, scratch, stream);
}
