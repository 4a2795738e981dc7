// Feed-forward experts chosen per token: out[t] = weight * sum_k down_e (act(gate_e x_t) * up_e x_t), e = the
// k-th expert of token t = table[token id of t, k] (a table of integers [vocabulary, top]).  These kernels serve steps of few tokens (single tokens above all): every (token,
// choice) streams its expert's matrices once, a warp per output row, sums in 32-bit in a fixed order, so a
// token's result does not depend on what else the step holds.  Steps of many tokens group their rows by expert: in bfloat16 on
// the device, with one product over all experts (idm_experts_by_expert); in 32-bit on the host, with one product per expert
// between rows_gather and experts_combine, which adds the experts' outputs back in the order of a token's choices.
//
// A learned router names a token's experts on the device: then `tokens` holds the step's row numbers and `table` the
// step's choices [rows, top], and `pair_w` [rows, top] (null: 1) is the weight of every (token, choice) beside the
// constant `weight`.  Where an expert's activations are 32-bit numbers of these kernels' own, the pair's weight is
// multiplied into them (the down product is linear); where the library's products make them, the weight is applied
// when the experts' outputs are added.  With `weight_in` the pair's weight belongs on the expert's INPUT instead: gate and
// up are linear, so both of a pair's pre-activations are multiplied by it, in 32-bit, wherever they are made, and the
// outputs are added as they are.
#include "common.cuh"

// a pair's activation: the weight on what the activation gives, or (weight_in) on both of its arguments
__device__ __forceinline__ float pair_act(float g, float u, float pw, int weight_in, int act) {
    return weight_in ? gated_act(g * pw, u * pw, act) : gated_act(g, u, act) * pw;
}

// s + sum over a 16-byte piece of a row of its elements times x's, in ascending order; x (in shared memory, on a 16-byte
// border) is read four numbers at a time: element by element, a warp's lanes would meet in the same banks
__device__ __forceinline__ float piece_dot(const Vec16<T>& w, const float* __restrict__ x, float s) {
#pragma unroll
    for (int e = 0; e < Vec16<T>::N; e += 4) {
        const float4 v = *reinterpret_cast<const float4*>(x + e);
        s = fmaf(v.x, w.get(e), s); s = fmaf(v.y, w.get(e + 1), s); s = fmaf(v.z, w.get(e + 2), s); s = fmaf(v.w, w.get(e + 3), s);
    }
    return s;
}

__device__ __forceinline__ float row_dot(const T* __restrict__ w, const float* __restrict__ xs, int K, int lane, bool vec) {
    float s = 0.f;
    if (vec) {
        constexpr int VN = Vec16<T>::N;
        for (int d = lane * VN; d < K; d += 32 * VN) {
            Vec16<T> wv; wv.load(w + d);
            s = piece_dot(wv, xs + d, s);
        }
    } else {
        for (int d = lane; d < K; d += 32) s = fmaf(xs[d], to_f32(w[d]), s);
    }
    return warp_sum(s);
}

// two rows against two vectors at once: eight (long rows) or four 16-byte loads of a lane are in flight before the
// first is used; a sum's order depends on the row's length alone
__device__ __forceinline__ void row_dot2(const T* __restrict__ w0, const T* __restrict__ w1, const float* __restrict__ x0,
                                         const float* __restrict__ x1, int K, int lane, bool vec, float& r0, float& r1) {
    float s0 = 0.f, s1 = 0.f;
    if (vec) {
        constexpr int VN = Vec16<T>::N;
        int d = lane * VN;
        for (; d + 96 * VN < K; d += 128 * VN) {             // four pieces of each row: eight loads before the first use
            Vec16<T> a[4], b[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) { a[c].load(w0 + d + c * 32 * VN); b[c].load(w1 + d + c * 32 * VN); }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                s0 = piece_dot(a[c], x0 + d + c * 32 * VN, s0);
                s1 = piece_dot(b[c], x1 + d + c * 32 * VN, s1);
            }
        }
        for (; d + 32 * VN < K; d += 64 * VN) {
            Vec16<T> a0, a1, b0, b1;
            a0.load(w0 + d); b0.load(w1 + d); a1.load(w0 + d + 32 * VN); b1.load(w1 + d + 32 * VN);
            s0 = piece_dot(a0, x0 + d, s0); s1 = piece_dot(b0, x1 + d, s1);
            s0 = piece_dot(a1, x0 + d + 32 * VN, s0); s1 = piece_dot(b1, x1 + d + 32 * VN, s1);
        }
        for (; d < K; d += 32 * VN) {
            Vec16<T> a0, b0;
            a0.load(w0 + d); b0.load(w1 + d);
            s0 = piece_dot(a0, x0 + d, s0); s1 = piece_dot(b0, x1 + d, s1);
        }
    } else {
        for (int d = lane; d < K; d += 32) { s0 = fmaf(x0[d], to_f32(w0[d]), s0); s1 = fmaf(x1[d], to_f32(w1[d]), s1); }
    }
    r0 = warp_sum(s0); r1 = warp_sum(s1);
}

// a[t, k, f] = act(gate_e[f] . x_t) * (up_e[f] . x_t), 32-bit.  Gate and up rows of an expert lie in one array:
// row f of expert e starts at e * expert_stride + f * row_stride (gate) and up_off behind that (up), which serves both
// "gate rows, then up rows" and "gate and up rows alternating" (the layout a gated product's epilogue reads).
// A block has one (token, choice) and 8 rows f per pass of its warps.
__global__ void __launch_bounds__(256) experts_gate_up_kernel(const T* __restrict__ x, const int* __restrict__ tokens,
                                                              const int* __restrict__ table, const float* __restrict__ pair_w,
                                                              const T* __restrict__ gate_up, long long expert_stride,
                                                              long long row_stride, long long up_off,
                                                              float* __restrict__ a, int width, int ff, int top, int n_experts,
                                                              int act, int weight_in) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float xs[];
    const int tk = blockIdx.x;
    const int t = tk / top;
    const int e = table[(size_t)tokens[t] * top + tk % top];       // the token's id names its experts
    for (int d = threadIdx.x; d < width; d += blockDim.x) xs[d] = to_f32(x[(size_t)t * width + d]);
    __syncthreads();
    if (e < 0 || e >= n_experts) return;                     // (a table entry outside the experts: contributes nothing)
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool vec = (width * (int)sizeof(T)) % 16 == 0;
    const float pw = pair_w ? pair_w[tk] : 1.f;
    for (int f = blockIdx.y * 8 + wib; f < ff; f += gridDim.y * 8) {
        const T* row = gate_up + (size_t)e * expert_stride + (size_t)f * row_stride;
        float g, u;
        row_dot2(row, row + up_off, xs, xs, width, lane, vec, g, u);
        if (lane == 0) a[(size_t)tk * ff + f] = pair_w ? pair_act(g, u, pw, weight_in, act) : gated_act(g, u, act);
    }
}

// h[t, w] += weight * sum_k down_e[w] . a[t, k];  down: [E, width, ff]; a block has one token, a warp an output row
__global__ void __launch_bounds__(256) experts_down_kernel(const float* __restrict__ a, const int* __restrict__ tokens,
                                                           const int* __restrict__ table,
                                                           const T* __restrict__ down, float* __restrict__ h, int width,
                                                           int ff, int top, int n_experts, float weight) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float as[];                             // [top][ff]
    const int t = blockIdx.x;
    for (int d = threadIdx.x; d < top * ff; d += blockDim.x) as[d] = a[(size_t)t * top * ff + d];
    __syncthreads();
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool vec = (ff * (int)sizeof(T)) % 16 == 0;
    for (int w = blockIdx.y * 8 + wib; w < width; w += gridDim.y * 8) {
        float s = 0.f;
        int k = 0;
        for (; k + 1 < top; k += 2) {                       // two choices' rows at once (their loads side by side)
            const int e0 = table[(size_t)tokens[t] * top + k], e1 = table[(size_t)tokens[t] * top + k + 1];
            const bool ok0 = e0 >= 0 && e0 < n_experts, ok1 = e1 >= 0 && e1 < n_experts;
            if (ok0 && ok1) {
                float r0, r1;
                row_dot2(down + ((size_t)e0 * width + w) * ff, down + ((size_t)e1 * width + w) * ff, as + k * ff, as + (k + 1) * ff,
                         ff, lane, vec, r0, r1);
                s += r0; s += r1;
            } else {
                if (ok0) s += row_dot(down + ((size_t)e0 * width + w) * ff, as + k * ff, ff, lane, vec);
                if (ok1) s += row_dot(down + ((size_t)e1 * width + w) * ff, as + (k + 1) * ff, ff, lane, vec);
            }
        }
        for (; k < top; ++k) {
            const int e = table[(size_t)tokens[t] * top + k];
            if (e < 0 || e >= n_experts) continue;
            s += row_dot(down + ((size_t)e * width + w) * ff, as + k * ff, ff, lane, vec);
        }
        if (lane == 0) h[(size_t)t * width + w] += s * weight;
    }
}

extern "C" int idm_experts_few(const void* x, const int* tokens, const int* table, const float* pair_w, const void* gate_up, long long expert_stride,
                               long long row_stride, long long up_off, const void* down,
                               float* a, float* h, int n_tokens, int width, int ff, int top, int n_experts, int act,
                               float weight, int weight_in, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    IDM_REQUIRE(width > 0 && ff > 0 && top > 0 && n_experts > 0 && (act >= 0 && act <= 2), "experts: width=%d ff=%d top=%d experts=%d act=%d",
                width, ff, top, n_experts, act);
    IDM_REQUIRE((size_t)width * 4 <= 160 * 1024 && (size_t)top * ff * 4 <= 160 * 1024, "experts: width=%d or top * ff=%d does not fit shared memory",
                width, top * ff);
    const size_t s1 = (size_t)width * 4, s2 = (size_t)top * ff * 4;
    if (s1 > 48 * 1024) cudaFuncSetAttribute(experts_gate_up_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1);
    if (s2 > 48 * 1024) cudaFuncSetAttribute(experts_down_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s2);
    // blocks along the rows: enough to fill the part for one token, fewer per token as tokens grow
    const int by1 = max(1, min((ff + 7) / 8, 592 / max(1, n_tokens * top)));
    const int by2 = max(1, min((width + 7) / 8, 592 / max(1, n_tokens)));
    idm_launch(experts_gate_up_kernel, dim3(n_tokens * top, by1), dim3(256), s1, stream, (const T*)x, tokens, table, pair_w, (const T*)gate_up,
               expert_stride, row_stride, up_off, a, width, ff, top, n_experts, act, weight_in);
    IDM_LAUNCH_CHECK("experts_gate_up");
    idm_launch(experts_down_kernel, dim3(n_tokens, by2), dim3(256), s2, stream, (const float*)a, tokens, table, (const T*)down, h, width,
               ff, top, n_experts, weight);
    IDM_LAUNCH_CHECK("experts_down");
    return 0;
}

// out[i, :] = x[src[i], :]  (rows of the storage type; a step's rows in the order of their experts)
__global__ void __launch_bounds__(256) rows_gather_kernel(const T* __restrict__ x, const int* __restrict__ src, T* __restrict__ out, int width) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t i = blockIdx.x;
    const T* r = x + (size_t)src[i] * width;
    for (int d = threadIdx.x; d < width; d += blockDim.x) out[i * width + d] = r[d];
}

extern "C" int idm_rows_gather(const void* x, const int* src, void* out, int n_rows, int width, cudaStream_t stream) {
    if (n_rows == 0) return 0;
    idm_launch(rows_gather_kernel, dim3(n_rows), dim3(256), 0, stream, (const T*)x, src, (T*)out, width);
    IDM_LAUNCH_CHECK("rows_gather");
    return 0;
}

// h[t, :] += weight * sum_k z[place[t, k], :] in ascending k  (z 32-bit: the experts' outputs, grouped rows), and with x then
// += x[t, :] * (the weights of t's pairs whose expert table[tokens[t], k] is n_real or more: experts that hand their input on).
// Four elements a thread where rows allow it, four pairs' loads at a time: bound by the bytes of z.
struct CombineArgs {
    const float* z; const int* place; const float* pair_w; float* h;
    int width, top; float weight;
    const T* x; const int* tokens; const int* table; int n_real;
};
template <int V>
__global__ void __launch_bounds__(256) experts_combine_kernel(CombineArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t t = blockIdx.x;
    const int top = a.top;
    float same = 0.f;                                                        // the identity experts' weight
    if (a.x)
        for (int k = 0; k < top; ++k)
            if (a.table[(a.tokens ? (size_t)a.tokens[t] : t) * top + k] >= a.n_real) same += a.pair_w[t * top + k];
    for (int d = threadIdx.x * V; d < a.width; d += blockDim.x * V) {
        float s[V];
#pragma unroll
        for (int i = 0; i < V; ++i) s[i] = 0.f;
        for (int k0 = 0; k0 < top; k0 += 4) {
            float v[4][V], pw[4];
            int r[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const size_t p = t * top + k0 + j;
                r[j] = k0 + j >= top ? -1 : a.place ? a.place[p] : (int)p;   // (no places: pair by pair as they lie)
                pw[j] = r[j] >= 0 && a.pair_w ? a.pair_w[p] : 1.f;
                if (r[j] < 0) continue;
                const float* z = a.z + (size_t)r[j] * a.width + d;
                if (V == 4) *reinterpret_cast<float4*>(v[j]) = *reinterpret_cast<const float4*>(z);
                else v[j][0] = *z;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (r[j] >= 0) {
#pragma unroll
                    for (int i = 0; i < V; ++i) s[i] = a.pair_w ? fmaf(pw[j], v[j][i], s[i]) : s[i] + v[j][i];
                }
        }
        float* h = a.h + t * a.width + d;
        float o[V];
        if (V == 4) *reinterpret_cast<float4*>(o) = *reinterpret_cast<const float4*>(h);
        else o[0] = *h;
#pragma unroll
        for (int i = 0; i < V; ++i) {
            o[i] += s[i] * a.weight;
            if (a.x && same != 0.f) o[i] = fmaf(same, to_f32(a.x[t * a.width + d + i]), o[i]);
        }
        if (V == 4) *reinterpret_cast<float4*>(h) = *reinterpret_cast<const float4*>(o);
        else *h = o[0];
    }
}

static int experts_combine(const CombineArgs& a, int n_tokens, cudaStream_t stream) {
    const bool vec = a.width % 4 == 0 && (((uintptr_t)a.z | (uintptr_t)a.h) & 15) == 0;
    const int threads = vec ? min(256, (a.width / 4 + 31) / 32 * 32) : 256;
    idm_launch(vec ? experts_combine_kernel<4> : experts_combine_kernel<1>, dim3(n_tokens), dim3(threads), 0, stream, a);
    IDM_LAUNCH_CHECK("experts_combine");
    return 0;
}

extern "C" int idm_experts_combine(const float* z, const int* place, const float* pair_w, float* h, int n_tokens, int width,
                                   int top, float weight, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    return experts_combine(CombineArgs{z, place, pair_w, h, width, top, weight, nullptr, nullptr, nullptr, 0}, n_tokens, stream);
}

// out[place[p]] = pair_w[p] for every (token, choice) p that has a grouped row
__global__ void __launch_bounds__(256) rows_weight_kernel(const float* __restrict__ pair_w, const int* __restrict__ place,
                                                          float* __restrict__ out, int n_pairs) {
    pdl_launch_dependents();
    pdl_wait();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n_pairs && place[p] >= 0) out[place[p]] = pair_w[p];
}

extern "C" int idm_rows_weight(const float* pair_w, const int* place, float* out, int n_pairs, cudaStream_t stream) {
    if (n_pairs == 0) return 0;
    idm_launch(rows_weight_kernel, dim3((n_pairs + 255) / 256), dim3(256), 0, stream, pair_w, place, out, n_pairs);
    IDM_LAUNCH_CHECK("rows_weight");
    return 0;
}

// ------------------------------------------------------------------ the same, expert by expert
// For steps of more than a few tokens whose ids exist on the device only: a block has one expert and a slice of its
// rows, finds the (token, choice) pairs that use the expert (in ascending order), and walks them eight at a time: the
// eight input vectors wait in shared memory, a warp streams a row of the expert's matrix once for all eight.  An expert
// is read from memory once a step however many tokens use it.  MODE 0: a[pair, f] = act(gate[f] . x_t) * (up[f] . x_t);
// MODE 1: z[pair, w] = down[w] . a[pair].  Sums in 32-bit, lanes over the inner axis, then a butterfly.
#define EX_TOKENS 8

template <int MODE>
__global__ void __launch_bounds__(256) experts_major_kernel(const T* __restrict__ x, const float* __restrict__ a_in,
                                                            const int* __restrict__ tokens, const int* __restrict__ table,
                                                            const float* __restrict__ pair_w,
                                                            const T* __restrict__ w, long long expert_stride, long long row_stride,
                                                            long long up_off, float* __restrict__ out, int n_tokens, int top,
                                                            int K, int rows, int act, int weight_in) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float sm[];
    float* xs = sm;                                              // [EX_TOKENS][K]
    int* pairs = reinterpret_cast<int*>(sm + EX_TOKENS * K);     // [n_tokens * top]
    __shared__ int count_s;
    const int e = blockIdx.x, wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (wib == 0) {                                              // the pairs of this expert, in ascending order
        int count = 0;
        for (int p0 = 0; p0 < n_tokens * top; p0 += 32) {
            const int p = p0 + lane;
            const bool mine = p < n_tokens * top && table[(size_t)tokens[p / top] * top + p % top] == e;
            const unsigned m = __ballot_sync(0xffffffffu, mine);
            if (mine) pairs[count + __popc(m & ((1u << lane) - 1u))] = p;
            count += __popc(m);
        }
        if (lane == 0) count_s = count;
    }
    __syncthreads();
    const int count = count_s;
    if (count == 0) return;
    const bool vec = (K * (int)sizeof(T)) % 16 == 0;
    const T* we = w + (size_t)e * expert_stride;
    for (int p0 = 0; p0 < count; p0 += EX_TOKENS) {
        const int np = min(EX_TOKENS, count - p0);
        __syncthreads();                                         // the last eight's readers are done
        for (int i = threadIdx.x; i < EX_TOKENS * K; i += blockDim.x) {
            const int tt = i / K, d = i % K;
            float v = 0.f;
            if (tt < np) {
                const int p = pairs[p0 + tt];
                v = MODE == 0 ? to_f32(x[(size_t)(p / top) * K + d]) : a_in[(size_t)p * K + d];
            }
            xs[i] = v;
        }
        __syncthreads();
        for (int r = blockIdx.y * 8 + wib; r < rows; r += gridDim.y * 8) {
            const T* w0 = we + (size_t)r * row_stride;
            float g[EX_TOKENS], u[EX_TOKENS];
#pragma unroll
            for (int tt = 0; tt < EX_TOKENS; ++tt) g[tt] = u[tt] = 0.f;
            if (vec) {
                constexpr int VN = Vec16<T>::N;
                // four 16-byte pieces of the row (and of its partner) per lane are requested before the first is used
                for (int d0 = lane * VN; d0 < K; d0 += 4 * 32 * VN) {
                    Vec16<T> wg[4], wu[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int d = d0 + c * 32 * VN;
                        if (d < K) {
                            wg[c].load(w0 + d);
                            if (MODE == 0) wu[c].load(w0 + up_off + d);
                        }
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int d = d0 + c * 32 * VN;
                        if (d < K) {
#pragma unroll
                            for (int tt = 0; tt < EX_TOKENS; ++tt) {
#pragma unroll
                                for (int q = 0; q < VN; q += 4) {
                                    const float4 xv = *reinterpret_cast<const float4*>(xs + tt * K + d + q);
                                    g[tt] = fmaf(xv.x, wg[c].get(q), g[tt]); g[tt] = fmaf(xv.y, wg[c].get(q + 1), g[tt]);
                                    g[tt] = fmaf(xv.z, wg[c].get(q + 2), g[tt]); g[tt] = fmaf(xv.w, wg[c].get(q + 3), g[tt]);
                                    if (MODE == 0) {
                                        u[tt] = fmaf(xv.x, wu[c].get(q), u[tt]); u[tt] = fmaf(xv.y, wu[c].get(q + 1), u[tt]);
                                        u[tt] = fmaf(xv.z, wu[c].get(q + 2), u[tt]); u[tt] = fmaf(xv.w, wu[c].get(q + 3), u[tt]);
                                    }
                                }
                            }
                        }
                    }
                }
            } else {
                for (int d = lane; d < K; d += 32) {
                    const float wg = to_f32(w0[d]), wu = MODE == 0 ? to_f32(w0[up_off + d]) : 0.f;
#pragma unroll
                    for (int tt = 0; tt < EX_TOKENS; ++tt) {
                        g[tt] = fmaf(xs[tt * K + d], wg, g[tt]);
                        if (MODE == 0) u[tt] = fmaf(xs[tt * K + d], wu, u[tt]);
                    }
                }
            }
#pragma unroll
            for (int tt = 0; tt < EX_TOKENS; ++tt) {
                g[tt] = warp_sum(g[tt]);
                if (MODE == 0) u[tt] = warp_sum(u[tt]);
            }
            if (lane == 0) {
#pragma unroll
                for (int tt = 0; tt < EX_TOKENS; ++tt)
                    if (tt < np) {
                        const int pr = pairs[p0 + tt];
                        out[(size_t)pr * rows + r] = MODE == 0 ? (pair_w ? pair_act(g[tt], u[tt], pair_w[pr], weight_in, act) : gated_act(g[tt], u[tt], act)) : g[tt];
                    }
            }
        }
    }
}

// z: [n_tokens * top, width] 32-bit scratch for the experts' outputs (then added to h pair by pair in ascending k)
extern "C" int idm_experts_major(const void* x, const int* tokens, const int* table, const float* pair_w, const void* gate_up,
                                 long long expert_stride, long long row_stride, long long up_off, const void* down,
                                 float* a, float* z, float* h, int n_tokens, int width, int ff, int top, int n_experts,
                                 int act, float weight, int weight_in, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    IDM_REQUIRE(width > 0 && ff > 0 && top > 0 && n_experts > 0 && (act >= 0 && act <= 2), "experts: width=%d ff=%d top=%d experts=%d act=%d",
                width, ff, top, n_experts, act);
    const size_t s1 = (size_t)EX_TOKENS * width * 4 + (size_t)n_tokens * top * 4, s2 = (size_t)EX_TOKENS * ff * 4 + (size_t)n_tokens * top * 4;
    IDM_REQUIRE(s1 <= 200 * 1024 && s2 <= 200 * 1024, "experts: width=%d or ff=%d with %d tokens does not fit shared memory", width, ff, n_tokens);
    if (s1 > 48 * 1024) cudaFuncSetAttribute(experts_major_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1);
    if (s2 > 48 * 1024) cudaFuncSetAttribute(experts_major_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s2);
    const int by1 = max(1, min((ff + 7) / 8, 592 / n_experts)), by2 = max(1, min((width + 7) / 8, 592 / n_experts));
    idm_launch(experts_major_kernel<0>, dim3(n_experts, by1), dim3(256), s1, stream, (const T*)x, (const float*)nullptr, tokens, table, pair_w,
               (const T*)gate_up, expert_stride, row_stride, up_off, a, n_tokens, top, width, ff, act, weight_in);
    IDM_LAUNCH_CHECK("experts_major gate/up");
    idm_launch(experts_major_kernel<1>, dim3(n_experts, by2), dim3(256), s2, stream, (const T*)nullptr, (const float*)a, tokens, table, (const float*)nullptr,
               (const T*)down, (long long)width * ff, (long long)ff, 0LL, z, n_tokens, top, ff, width, act, 0);
    IDM_LAUNCH_CHECK("experts_major down");
    return experts_combine(CombineArgs{z, nullptr, nullptr, h, width, top, weight, nullptr, nullptr, nullptr, 0}, n_tokens, stream);
}

#if defined(IDM_BF16)
// ------------------------------------------------------------------ steps of many (token, choice) pairs, grouped by expert
// The pairs in the order of their experts, ascending inside an expert: offsets [E + 1] (an expert's first row), place [N, top] (a
// pair's row, -1 for a pair that names no expert), xg [rows, width] (the pairs' input rows) and, if asked for, row_w [rows]
// (their weights).  A block has some tokens and counts for itself how many pairs of each expert lie before them (the pairs
// are a few hundred KB at most, in the L2), so one launch does it all, without a count from the host; then it copies
// its tokens' rows, each read once.  Bound by the bytes of xg.
#define EG_THREADS 512
#define EG_SMEM (200 * 1024)
struct GroupArgs {
    const T* x; const int* tokens; const int* table; const float* pair_w;
    int n_tokens, top, n_experts, width, block_tokens;
    int* place; int* offsets; float* row_w; T* xg;
};
__device__ __forceinline__ int pair_expert(const GroupArgs& a, int p) {      // of pair p = token * top + choice, or -1
    int e;
    if (a.tokens) { const int t = p / a.top; e = a.table[(size_t)a.tokens[t] * a.top + (p - t * a.top)]; }
    else e = a.table[p];                                                     // (the table's rows are the step's)
    return e >= 0 && e < a.n_experts ? e : -1;
}
__global__ void __launch_bounds__(EG_THREADS) experts_group_kernel(GroupArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ int group_sm[];
    int* total = group_sm;                                                         // pairs of an expert; then the expert's first row
    int* before = total + a.n_experts;                                       // those before this block's; then before the next pair
    int* at = before + a.n_experts;                                          // [block_tokens * top]: this block's pairs' rows
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = blockIdx.x * a.block_tokens, t1 = min(t0 + a.block_tokens, a.n_tokens);
    const int pairs = a.n_tokens * a.top, p0 = t0 * a.top, p1 = t1 * a.top;
    // this block's rows in 16-byte pieces (whole pieces, width % 8 == 0), the first four of a thread on their way while it counts
    const int pieces = a.width / Vec16<T>::N, all = (t1 - t0) * pieces;
    const uint4* src = reinterpret_cast<const uint4*>(a.x + (size_t)t0 * a.width);
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if ((int)threadIdx.x + j * EG_THREADS < all) v[j] = src[threadIdx.x + j * EG_THREADS];
    for (int e = threadIdx.x; e < a.n_experts; e += EG_THREADS) { total[e] = 0; before[e] = 0; }
    __syncthreads();
    for (int c0 = warp * 32; c0 < pairs; c0 += 8 * EG_THREADS) {             // eight looks at the table on their way at a time
        int named[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int p = c0 + j * EG_THREADS + lane;
            named[j] = p < pairs ? pair_expert(a, p) : -1;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int p = c0 + j * EG_THREADS + lane;
            if (p >= p0 && p < p1) at[p - p0] = named[j];
            if (named[j] >= 0) {
                atomicAdd(&total[named[j]], 1);
                if (p < p0) atomicAdd(&before[named[j]], 1);
            }
        }
    }
    __syncthreads();
    if (warp == 0) {
        int rows = 0;                                                        // of the experts so far
        for (int e0 = 0; e0 < a.n_experts; e0 += 32) {
            const int e = e0 + lane, n = e < a.n_experts ? total[e] : 0;
            int upto = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += u; }
            if (e < a.n_experts) {
                total[e] = rows + upto - n;
                if (blockIdx.x == 0) a.offsets[e] = rows + upto - n;
            }
            rows += __shfl_sync(0xffffffffu, upto, 31);
        }
        if (blockIdx.x == 0 && lane == 0) a.offsets[a.n_experts] = rows;
        __syncwarp();
        for (int c = p0; c < p1; c += 32) {
            const int p = c + lane, e = p < p1 ? at[p - p0] : -1;
            const unsigned same = __match_any_sync(0xffffffffu, e);
            const int row = e >= 0 ? total[e] + before[e] + __popc(same & ((1u << lane) - 1u)) : -1;
            __syncwarp();
            if (e >= 0 && lane == __ffs(same) - 1) before[e] += __popc(same);
            __syncwarp();
            if (p < p1) {
                at[p - p0] = row;
                a.place[p] = row;
                if (row >= 0 && a.row_w) a.row_w[row] = a.pair_w[p];
            }
        }
    }
    __syncthreads();
    uint4* dst = reinterpret_cast<uint4*>(a.xg);
    for (int i0 = threadIdx.x; i0 < all; i0 += 4 * EG_THREADS) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = i0 + j * EG_THREADS, t = i / pieces, piece = i - t * pieces;
            if (i >= all) break;
            for (int k = 0; k < a.top; ++k) {
                const int row = at[t * a.top + k];
                if (row >= 0) dst[(size_t)row * pieces + piece] = v[j];
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i0 + (4 + j) * EG_THREADS < all) v[j] = src[i0 + (4 + j) * EG_THREADS];
    }
}

int gemm_experts_store(const void* x, const void* w, float* out, const int* offsets, int n_experts, int n_rows, int N, int K, cudaStream_t stream);
int gemm_experts_gated(const void* x, const void* w_tiled, void* y, const int* offsets, int n_experts, int n_rows, int inter, int K, int act,
                       const float* row_w, cudaStream_t stream);

// h[t] += weight * sum_k ff_e(x_t), e = table[tokens[t], k] (tokens null: table[t, k]), with the pairs grouped by expert: one launch groups them, one makes every
// expert's gated product (gate_up [E, tiles * 128, width], gate and up rows alternating), one every expert's down product (down
// [E, width, ff]), one adds the outputs up in the order of a token's choices.  Nothing depends on the host: steps can be captured.
// pair_w [N, top] (or null: 1) weighs the outputs, or (weight_in) the inputs; `identity`: pairs that name expert E or more add
// their weight times x_t itself.  scratch: xg, y [N * top, width | ff], z 32-bit [N * top, width], ints [E + 1 + N * top], row_w [N * top].
extern "C" int idm_experts_by_expert(const void* x, const int* tokens, const int* table, const float* pair_w, int n_experts, const void* gate_up,
                                     const void* down, void* xg, void* y, float* z, int* ints, float* row_w, float* h, int n_tokens, int top,
                                     int width, int ff, int act, float weight, int weight_in, int identity, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    IDM_REQUIRE(width > 0 && ff > 0 && width % 8 == 0 && ff % 8 == 0, "experts_by_expert: width=%d ff=%d (multiples of 8)", width, ff);
    IDM_REQUIRE(n_experts > 0 && top > 0 && (long long)n_tokens * top < (1ll << 31), "experts_by_expert: %d experts, %d x %d pairs", n_experts, n_tokens, top);
    IDM_REQUIRE(!(weight_in || identity) || pair_w, "experts_by_expert: weights on the inputs, or identity experts, need the pairs' weights");
    IDM_REQUIRE(!(weight_in && identity), "experts_by_expert: weights on the inputs and identity experts do not come together");
    IDM_REQUIRE(!weight_in || row_w, "experts_by_expert: weights on the inputs need their scratch");
    IDM_REQUIRE(((uintptr_t)x & 15) == 0, "experts_by_expert: rows must start on 16-byte borders");
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    GroupArgs g;
    g.x = (const T*)x; g.tokens = tokens; g.table = table; g.pair_w = pair_w;
    g.n_tokens = n_tokens; g.top = top; g.n_experts = n_experts; g.width = width;
    // two blocks an SM, so that few blocks count all pairs; no more pairs a block than one warp places in a moment
    const int even = (n_tokens + 2 * sms - 1) / (2 * sms), most = 512 / top > 0 ? 512 / top : 1;
    g.block_tokens = even < most ? even : most;
    g.offsets = ints; g.place = ints + n_experts + 1; g.row_w = weight_in ? row_w : nullptr; g.xg = (T*)xg;
    const size_t smem = (size_t)(2 * n_experts + g.block_tokens * top) * sizeof(int);
    IDM_REQUIRE(smem <= EG_SMEM, "experts_by_expert: %d experts do not fit shared memory", n_experts);
    if (smem > 48 * 1024) cudaFuncSetAttribute(experts_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, EG_SMEM);   // (every call the same limit)
    idm_launch(experts_group_kernel, dim3((n_tokens + g.block_tokens - 1) / g.block_tokens), dim3(EG_THREADS), smem, stream, g);
    IDM_LAUNCH_CHECK("experts_group");
    const int rows = n_tokens * top;
    if (gemm_experts_gated(xg, gate_up, y, g.offsets, n_experts, rows, ff, width, act, g.row_w, stream)) return 1;
    if (gemm_experts_store(y, down, z, g.offsets, n_experts, rows, width, ff, stream)) return 1;
    CombineArgs c{z, g.place, weight_in ? nullptr : pair_w, h, width, top, weight, nullptr, nullptr, nullptr, n_experts};
    if (identity) { c.x = (const T*)x; c.tokens = tokens; c.table = table; }
    return experts_combine(c, n_tokens, stream);
}
#endif
