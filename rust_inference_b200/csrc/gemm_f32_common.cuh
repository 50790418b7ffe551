// What the float32 products share: reads of weights, the epilogues, and the cutting of a float32 number into three bfloat16 ones.
#pragma once

#include "common.cuh"

namespace ri {
namespace f32 {

// weights: read once, kept out of L1 (a load that may stand before the wait for the kernel before)
__device__ __forceinline__ float4 load_weight(const float* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

struct Forms {          // the epilogue's constants, loaded once per thread
    GateForm gate;
    ActForm act;
    int silu_feats;
};
template <int MODE>
__device__ __forceinline__ Forms load_forms(const float* bias) {
    Forms f;
    f.gate = load_gate_form(MODE == 3 ? bias : nullptr);
    f.act = MODE == 4 ? load_act_form(bias) : ActForm{0.f, 0.f, 0.f};
    f.silu_feats = MODE == 5 ? (int)bias[0] : 0;
    return f;
}
template <int MODE>
__device__ __forceinline__ void finish(float* out, size_t o, int f, float v, float up, const float* __restrict__ bias,
                                       const Forms& forms) {
    if (MODE == 1) out[o] = bias != nullptr ? v + bias[f] : v;
    else if (MODE == 2) out[o] += v;
    else if (MODE == 3) out[o] = gated_f32(v, up, forms.gate);
    else if (MODE == 4) out[o] = act_f32(v, forms.act);
    else out[o] = f < forms.silu_feats ? silu_f32(v) : v;
}

// x * 2^16 as three bfloat16 numbers that add up to it exactly, each the upper half of a float32: the leading 8 significant
// bits, the next 8 and the rest.  The factor keeps the parts of every float32 number, the denormal ones too, among the numbers
// bfloat16 has (without it numbers below 2^-110 lose bits); the sums are divided by both operands' factors at the end.  From
// 2^112 on the parts become infinite or NaN, as those of an infinity or a NaN are.
constexpr float UP = 65536.f, DOWN = 1.f / (UP * UP);
__device__ __forceinline__ float2 two(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 leading(const float2& v) {
    return make_float2(__uint_as_float(__float_as_uint(v.x) & 0xffff0000u), __uint_as_float(__float_as_uint(v.y) & 0xffff0000u));
}
__device__ __forceinline__ uint32_t upper_halves(const float2& v) { return __byte_perm(__float_as_uint(v.x), __float_as_uint(v.y), 0x7632); }
__device__ __forceinline__ void cut(float2 v, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    v = __fmul2_rn(v, two(UP));
    hi = upper_halves(v);
    v = __ffma2_rn(leading(v), two(-1.f), v);
    mid = upper_halves(v);
    v = __ffma2_rn(leading(v), two(-1.f), v);
    lo = upper_halves(v);
}
__device__ __forceinline__ void store8(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
// four consecutive k of one row into the three parts
__device__ __forceinline__ void put(uint32_t addr, uint32_t part_bytes, const float4& v) {
    uint32_t h[2], m[2], l[2];
    cut(make_float2(v.x, v.y), h[0], m[0], l[0]);
    cut(make_float2(v.z, v.w), h[1], m[1], l[1]);
    store8(addr, h[0], h[1]);
    store8(addr + part_bytes, m[0], m[1]);
    store8(addr + 2 * part_bytes, l[0], l[1]);
}

constexpr float LARGEST = 3.402823466e38f;
// The sums of up to four rows of X (from t0 on) and 32 rows of W, at buf[i * ld + lane] for a warp: those that are infinite or NaN are computed
// again, as plain float32 sums over k_begin .. k_end; the others stay what they are.  `exists`: the lane's row of W does (zeros in its place
// may have met an infinity too); weight_row(r): the memory of row r.  The warp takes four rows of W at a time that are to be done for
// any of the rows of X, its lanes along K, so that both operands are read in whole lines and each once for four sums.
template <typename Row>
__device__ __forceinline__ void sum_again(float* buf, int ld, const float* X, int t0, int columns, bool exists, int K, int k_begin, int k_end,
                                          Row weight_row) {
    const int lane = threadIdx.x & 31;
    const float* x[4];
    uint32_t odd[4], todo = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x[i] = X + (size_t)(i < columns ? t0 + i : t0) * K;
        odd[i] = __ballot_sync(0xffffffffu, i < columns && exists && !(fabsf(buf[i * ld + lane]) <= LARGEST));
        todo |= odd[i];
    }
    while (todo != 0) {
        const float* w[4];
        int r[4];
        float sum[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {                                // fewer than four left: the first again
            r[j] = todo != 0 ? __ffs(todo) - 1 : r[0];
            w[j] = weight_row(r[j]);
            todo &= todo - 1;
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[i][j] = 0.f;
        }
#pragma unroll 2
        for (int k = k_begin + lane * 4; k < k_end; k += 128) {
            float4 a[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = load_written(x[i] + k);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 b = load_weight(w[j] + k);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    sum[i][j] = fmaf(a[i].w, b.w, fmaf(a[i].z, b.z, fmaf(a[i].y, b.y, fmaf(a[i].x, b.x, sum[i][j]))));
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float v = warp_sum(sum[i][j]);
                if (lane == 0 && ((odd[i] >> r[j]) & 1)) buf[i * ld + r[j]] = v;
            }
    }
    __syncwarp();
}

}  // namespace f32
}  // namespace ri
