// 32-bit products on the tensor cores' warp-wide instruction: small tiles whose operands are 32-bit.
//
// An operand x is split into three bfloat16 parts x = p0 + p1 + p2 (8 bits of the 24 each: what is left behind a part is exact, so the
// three carry the number whole down to some 2^-109), and a product is six products of parts, those down to 2^-16 of the largest:
//
//   x y  ~  p0 q0  +  (p0 q1 + p1 q0 + p0 q2 + p1 q1 + p2 q0)
//
// The first goes into one 32-bit sum, the others into another, because an addition in the tensor core cuts what lies below the sum's
// last bits off instead of rounding.  Every 64 k the two are added up by ordinary 32-bit additions (SplitSum::sum).  Against 64 bits,
// relative error of 16 x 8 outputs of normal (positive normal) numbers: k of 64 0.70e-7 (0.90e-7), 128 0.76e-7 (0.90e-7), 256 0.81e-7
// (0.90e-7); a chain of 32-bit FMAs 1.5e-7 (1.2e-7), 2.0e-7 (1.7e-7), 2.9e-7 (2.5e-7).
//
// Rate: mma.sync m16n8k16 runs 1 024 multiply-adds a clock and SM on this part (8 clocks an instruction and scheduler, 21 from
// one to a dependent one), so 170 a clock of 32-bit ones, where FMAs in tiles from shared memory reached 35 to 45 of their 128.
// Two operands in 10-bit parts (tf32, three products at half the rate) cost the same and are less exact: 2.0e-7 (3.0e-7) at k of 64.
//
// A number that is not finite, or rounds to a part that is not, comes out as NaN: callers make such outputs again of plain FMAs.
#pragma once
#include "common.cuh"

// the parts of two neighbours, each packed as the fragments hold them (x in the low half)
__device__ __forceinline__ void split3(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p0) : "f"(y), "f"(x));
    x -= __uint_as_float(p0 << 16); y -= __uint_as_float(p0 & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p1) : "f"(y), "f"(x));
    x -= __uint_as_float(p1 << 16); y -= __uint_as_float(p1 & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p2) : "f"(y), "f"(x));
}
// the largest magnitude's bits; from SPLIT_FINITE on a first part may not be finite
#define SPLIT_FINITE 0x7f7f8000u
__device__ __forceinline__ uint32_t magnitude(float x) { return __float_as_uint(x) & 0x7fffffffu; }

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void ldmatrix4_t(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}

// 16 rows x 16 k of the left operand, as lanes hold them: p[part][i] are the pairs (row g, k 2q), (g + 8, 2q), (g, 2q + 8), (g + 8, 2q + 8) of
// lane 4 g + q
struct SplitA {
    uint32_t p[3][4];
    // planes of `plane` elements, rows `ld` apart with k side by side; at: row 0, k 0
    __device__ __forceinline__ void load(const __nv_bfloat16* at, int plane, int ld, int lane) {
        const __nv_bfloat16* mine = at + (lane & 15) * ld + (lane >> 4) * 8;
#pragma unroll
        for (int i = 0; i < 3; ++i) ldmatrix4(p[i], mine + i * plane);
    }
    // the transposed: rows are k, the operand's rows side by side; at: k 0, row 0
    __device__ __forceinline__ void load_t(const __nv_bfloat16* at, int plane, int ld, int lane) {
        const __nv_bfloat16* mine = at + ((lane >> 4) * 8 + (lane & 7)) * ld + (lane >> 3 & 1) * 8;
#pragma unroll
        for (int i = 0; i < 3; ++i) ldmatrix4_t(p[i], mine + i * plane);
    }
};
// 16 k x 16 columns of the right operand, two tiles of 8 columns
struct SplitB {
    uint32_t p[3][4];                                        // [part][tile 0: k 0.., k 8..; tile 1: k 0.., k 8..]
    // planes of `plane` elements: rows are k, columns (n) side by side; at: row k0, column n0
    __device__ __forceinline__ void load_t(const __nv_bfloat16* at, int plane, int ld, int lane) {
        const __nv_bfloat16* mine = at + ((lane >> 3 & 1) * 8 + (lane & 7)) * ld + (lane >> 4) * 8;
#pragma unroll
        for (int i = 0; i < 3; ++i) ldmatrix4_t(p[i], mine + i * plane);
    }
};
// 16 x 8 N sums: lane 4 g + q has (g, 8 j + 2q), (g, 8 j + 2q + 1), (g + 8, ..), (g + 8, ..) of tile j
template <int N>
struct SplitSum {
    float big[N][4], small[N][4];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) big[j][i] = small[j][i] = 0.f;
    }
    // tiles j and j + 1; neighbouring instructions go to different sums
    __device__ __forceinline__ void add(int j, const SplitA& a, const SplitB& b) {
        mma_bf16(small[j], a.p[0], b.p[2][0], b.p[2][1]);
        mma_bf16(small[j + 1], a.p[0], b.p[2][2], b.p[2][3]);
        mma_bf16(big[j], a.p[0], b.p[0][0], b.p[0][1]);
        mma_bf16(big[j + 1], a.p[0], b.p[0][2], b.p[0][3]);
        mma_bf16(small[j], a.p[1], b.p[1][0], b.p[1][1]);
        mma_bf16(small[j + 1], a.p[1], b.p[1][2], b.p[1][3]);
        mma_bf16(small[j], a.p[2], b.p[0][0], b.p[0][1]);
        mma_bf16(small[j + 1], a.p[2], b.p[0][2], b.p[0][3]);
        mma_bf16(small[j], a.p[0], b.p[1][0], b.p[1][1]);
        mma_bf16(small[j + 1], a.p[0], b.p[1][2], b.p[1][3]);
        mma_bf16(small[j], a.p[1], b.p[0][0], b.p[0][1]);
        mma_bf16(small[j + 1], a.p[1], b.p[0][2], b.p[0][3]);
    }
    __device__ __forceinline__ float sum(int j, int i) const { return big[j][i] + small[j][i]; }
};

// the same with three sums (by the products' sizes): no instruction waits for the one before it where a warp has few tiles
template <int N>
struct SplitSum3 {
    float big[N][4], mid[N][4], low[N][4];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) big[j][i] = mid[j][i] = low[j][i] = 0.f;
    }
    __device__ __forceinline__ void add(int j, const SplitA& a, const SplitB& b) {
        mma_bf16(big[j], a.p[0], b.p[0][0], b.p[0][1]);
        mma_bf16(big[j + 1], a.p[0], b.p[0][2], b.p[0][3]);
        mma_bf16(low[j], a.p[0], b.p[2][0], b.p[2][1]);
        mma_bf16(low[j + 1], a.p[0], b.p[2][2], b.p[2][3]);
        mma_bf16(mid[j], a.p[0], b.p[1][0], b.p[1][1]);
        mma_bf16(mid[j + 1], a.p[0], b.p[1][2], b.p[1][3]);
        mma_bf16(low[j], a.p[1], b.p[1][0], b.p[1][1]);
        mma_bf16(low[j + 1], a.p[1], b.p[1][2], b.p[1][3]);
        mma_bf16(mid[j], a.p[1], b.p[0][0], b.p[0][1]);
        mma_bf16(mid[j + 1], a.p[1], b.p[0][2], b.p[0][3]);
        mma_bf16(low[j], a.p[2], b.p[0][0], b.p[0][1]);
        mma_bf16(low[j + 1], a.p[2], b.p[0][2], b.p[0][3]);
    }
    __device__ __forceinline__ float sum(int j, int i) const { return big[j][i] + (mid[j][i] + low[j][i]); }
};

// four neighbours into the three planes (shared memory or scratch), at an 8-byte border
__device__ __forceinline__ void store_split4(__nv_bfloat16* at, int plane, float4 x) {
    uint32_t a[3], b[3];
    split3(x.x, x.y, a[0], a[1], a[2]);
    split3(x.z, x.w, b[0], b[1], b[2]);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(at + i * plane) = make_uint2(a[i], b[i]);
}
