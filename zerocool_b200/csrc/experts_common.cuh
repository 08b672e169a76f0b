// What the decode family's two expert kernels (experts_item.cu, experts_decode.cu) share: the FP16 tensor-core product, the code
// conversions and the conversion of token rows. Both kernels must feed the same values, so the arithmetic stands here once.
#pragma once
#include "common.cuh"

namespace zc {
namespace {

constexpr int ROW_PAD = 8;            // halves added to each staged row (keeps 16-byte reads conflict free)

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

// D(16x8, fp32) += A(16x16, fp16, row) * B(16x8, fp16, col). Lane (g = lane/4, c = lane%4) holds
//   a0: A[g][2c,2c+1]   a1: A[g+8][2c,2c+1]   a2: A[g][2c+8,2c+9]   a3: A[g+8][2c+8,2c+9]
//   b0: B[2c,2c+1][g]   b1: B[2c+8,2c+9][g]
//   d0,d1: D[g][2c,2c+1]   d2,d3: D[g+8][2c,2c+1]
__device__ __forceinline__ void mma_f16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Same product with the addend taken from c (the first MMA of a group starts from the folded offset).
__device__ __forceinline__ void mma_f16_16816_c(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1,
                                                float c0, float c1, float c2, float c3) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}

// (a & b) | c in one logic instruction.
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// Q4: one word -> four half2 (k0,k4) (k1,k5) (k2,k6) (k3,k7) of its 8 codes.
template <bool FOLD>
__device__ __forceinline__ void dequant_q4(uint32_t w, uint32_t (&p)[4]) {
    const uint32_t lo = 0x000f000fu, hi = 0x00f000f0u, magic = 0x64006400u;
    const uint32_t w8 = w >> 8;
    p[0] = and_or(w, lo, magic);
    p[1] = and_or(w, hi, magic);
    p[2] = and_or(w8, lo, magic);
    p[3] = and_or(w8, hi, magic);
    if (!FOLD) {
        const __half2 k1024 = __floats2half2_rn(1024.0f, 1024.0f), k16 = __floats2half2_rn(0.0625f, 0.0625f), k64 = __floats2half2_rn(-64.0f, -64.0f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            __half2 v = *reinterpret_cast<__half2*>(&p[i]);
            v = (i & 1) ? __hfma2(v, k16, k64) : __hsub2(v, k1024);
            p[i] = *reinterpret_cast<uint32_t*>(&v);
        }
    }
}
// Q8: one word -> two half2 (k0,k1) (k2,k3); every integer in [-128, 255] is exact in FP16.
__device__ __forceinline__ void dequant_q8(uint32_t w, bool is_signed, uint32_t (&p)[2]) {
    if (is_signed) w ^= 0x80808080u;
    const float off = is_signed ? 8388608.0f + 128.0f : 8388608.0f;
    float f[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = __uint_as_float(0x4b000000u | ((w >> (8 * i)) & 0xffu)) - off;
    const __half2 a = __floats2half2_rn(f[0], f[1]), b = __floats2half2_rn(f[2], f[3]);
    p[0] = *reinterpret_cast<const uint32_t*>(&a);
    p[1] = *reinterpret_cast<const uint32_t*>(&b);
}

// Eight consecutive elements of a row (zeros in a lane past its end) as FP16 operands (hi, and lo when SPLIT) in the k order the MMA fragments expect - Q4 order inside each block of
// 8: (0,4,1,5,2,6,3,7); Q8: natural order - with their sums over the 64-wide group, which all eight lanes of a group return:
//   sx = sum of x (REF: the reference's BF16 sum of four, qwen.metal:55), times 16 when FOLD;
//   sf = sum of the values as staged.
// Folded Q4 codes: the value that meets a "1024 + 16 q" slot must be 1/16 of its neighbours'. Even slots are staged x 16 rather
// than odd slots / 16, which keeps small activations out of FP16's subnormal range; the accumulated result is multiplied by 1/16
// (exact) when it is finished. The bias term multiplies the sum of the activations. Outside the reference arithmetic it uses the
// sum of the values the MMA really sees, so that a rounding of an activation to FP16 enters the result through the weight s q + b
// and not through s q alone. beyond: some value would become an FP16 infinity (reported, not hidden).
template <bool Q4ORDER, bool SPLIT, bool FOLD>
__device__ __forceinline__ void convert8(const float (&v)[8], bool ref, uint4& hi, uint4& lo, float& sx, float& sf, bool& beyond) {
    sx = sf = 0.0f;
    if (ref) sx = bf_round(bf_round(bf_round(v[0] + v[1]) + v[2]) + v[3]) + bf_round(bf_round(bf_round(v[4] + v[5]) + v[6]) + v[7]);
    constexpr float EVEN = (FOLD && Q4ORDER) ? 16.0f : 1.0f;
    constexpr int order_q4[8] = {0, 4, 1, 5, 2, 6, 3, 7};
    __half h[8], l[8];
    float sn = 0.0f;                       // sums of the values as fed to the MMA, k ascending: as staged (sf), and in natural scale
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float pre = (i & 1) ? v[i] : v[i] * EVEN;
        beyond |= fabsf(pre) > 65504.0f;
        h[i] = __float2half_rn(pre);
        float fed = __half2float(h[i]);
        if (SPLIT) { l[i] = __float2half_rn(pre - fed); fed += __half2float(l[i]); }
        sf += fed;
        sn += (i & 1) ? fed : fed * (1.0f / EVEN);
    }
    if (!ref) sx = sn;
#pragma unroll
    for (int off = 1; off <= 4; off <<= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, off);
        if (FOLD) sf += __shfl_xor_sync(0xffffffffu, sf, off);
    }
    if (FOLD && Q4ORDER) sx *= 16.0f;
    uint32_t ph[4], pl[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int a = Q4ORDER ? order_q4[2 * i] : 2 * i, b = Q4ORDER ? order_q4[2 * i + 1] : 2 * i + 1;
        ph[i] = uint32_t(__half_as_ushort(h[a])) | (uint32_t(__half_as_ushort(h[b])) << 16);
        if (SPLIT) pl[i] = uint32_t(__half_as_ushort(l[a])) | (uint32_t(__half_as_ushort(l[b])) << 16);
    }
    hi = make_uint4(ph[0], ph[1], ph[2], ph[3]);
    if (SPLIT) lo = make_uint4(pl[0], pl[1], pl[2], pl[3]);
}

}  // namespace
}  // namespace zc
