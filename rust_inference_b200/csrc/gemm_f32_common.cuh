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

}  // namespace f32
}  // namespace ri
