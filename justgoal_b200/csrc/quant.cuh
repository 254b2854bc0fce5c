// Activation quantiser: the step right before the MoE operator.  bf16 hidden states [T, H] ->
// e4m3 [T, H] plus one fp32 scale per (token, 128 columns), stored K-block major [H/128, T] - the
// layout the operator's hidden_states_scale argument has.  scale = amax / 448 (1.0 for an all-zero
// group), q = round-to-nearest-even(x / scale), IEEE fp32 divisions, so the result is bit-identical
// to the same statement in PyTorch on the host.  The reference corpus receives pre-quantised inputs
// from its harness (goal_full_shape/fable-5.1/moe_fp8_fwd/<def>/moe_host.cu:100-103) and has no such
// kernel; the arithmetic is the one its input contract states (1x128 groups, amax / 448).
//
// HBM-bound byte work: 2 bytes read and 1 byte written per element, as long as the instructions stay few: 8 lanes own one
// group of 128 columns (16 bf16 = one 32-byte load per lane, so the group's scale, its reciprocal and the maximum's
// shuffles are shared by 16 elements), two groups' loads in flight per lane, the maximum over packed bf16 pairs.  A CTA owns a block of tokens x groups, so that it can
// walk the block without divisions and keep the scales in shared memory until a K block's run of tokens leaves as one
// store (one 4-byte store per group into the [H/128, T] layout touched a sector each).
//
// Launched with programmatic stream serialization: the kernel's start hides under the tail of the one before it (often the one
// that writes x: nothing is read or written before the wait), and the layer that follows starts under this one.  With four tokens per CTA
// (the host's rule) in a row of calls of this kernel alone, where each starts under the one before it: 4096 x 7168 20.4 -> 17.6 us
// (5.0 TB/s), 2048: 12.3 -> 10.0, 14107: 55.3 -> 52.9; through the public entry point, with the copies of other work around it,
// 4096: 20.5 -> 19.0.
//
// The divisions.  Eight IEEE divisions per lane and 128 columns made the kernel instruction-bound (4096 x 7168: 30.8 us,
// 2.9 TB/s).  With y = fl(1/s) a quotient needs three operations (Markstein, "IA-64 and Elementary Functions", ch. 8):
// q0 = fl(x y), e = fl(q0 s - x), q = fl(q0 - e y).  q0 is off by at most two units in the last place, e carries a relative
// error of 2^-25, so q rounds a value within 2^-22 units of x/s and can only differ from fl(x/s) where x/s lies that close
// to the middle between two floats.  For the e4m3 byte to differ, one of the two must be a tie M of the e4m3 grid as well,
// x/s = (M + half a unit)(1 + 2^-46): with x an 8-bit and s a 24-bit integer times a power of two this asks for
// r n = c, n the odd part of M, 2^24 > c 2^(25 - bits(n)) >= 2^23, |r| <= 8, which only n = c = r = 1 solves - a scale whose
// mantissa is all ones, and the quotient of an 8-bit number by 448 never is.  (The test runs all pairs of mantissas.)
// Scales below 2^-90 or above 2^126, where e or y would lose bits to the exponent range, take the dividing path.
// Zeros: e is +0 for x = +-0 (a sum of zeros of opposite sign), so e times the NEGATIVE factor -y is -0, which leaves q0 = +-0
// its sign; with the residual the other way round, x - q0 s times y, -0 came out as +0.  x enters negated for that: a
// bf16 is unpacked and negated in one integer operation (4096 x 7168, not overlapped: 20.5 us with either form on inputs from memory, 15.9
// against 16.4 us on inputs that the L2 still holds).
#pragma once
#include <cuda_bf16.h>
#include "common.cuh"

namespace b200moe {

// The two bf16 of a word as floats of the opposite sign
__device__ __forceinline__ float2 unpack_negated(uint32_t w) {
    return make_float2(__uint_as_float(w * 0x10000u + 0x80000000u), __uint_as_float((w & 0xFFFF0000u) ^ 0x80000000u));
}

// Four quotients v / s of one lane, rounded to e4m3 (one byte each), from n0, n1 = -v and ny = -fl(1 / s)
__device__ __forceinline__ uint32_t quantize4(const float2 n0, const float2 n1, float s, float ny) {
    const float2 ss = make_float2(s, s), yy = make_float2(ny, ny);
    const float2 p0 = __fmul2_rn(n0, yy), p1 = __fmul2_rn(n1, yy);
    const float2 q0 = __ffma2_rn(__ffma2_rn(p0, ss, n0), yy, p0), q1 = __ffma2_rn(__ffma2_rn(p1, ss, n1), yy, p1);
    return (uint32_t)f32x2_to_e4m3x2(q0.x, q0.y) | ((uint32_t)f32x2_to_e4m3x2(q1.x, q1.y) << 16);
}

constexpr int QUANT_TOKENS = 8;         // tokens of a CTA: a sector of scales (fewer or more by the host's rule)
constexpr int QUANT_GROUPS = 64;        // most groups (128 columns) of a token in a CTA
constexpr int QUANT_THREADS = 256, QUANT_LANES = 8, QUANT_FLIGHT = 2;     // lanes of a group, groups per lane in flight
constexpr int QUANT_SCALES = QUANT_TOKENS * QUANT_GROUPS;                 // most scales of a CTA
constexpr int QUANT_TURN = QUANT_THREADS / QUANT_LANES * QUANT_FLIGHT;    // groups a CTA takes at a time

// CTA (x, y): tokens [x * tpc, ...), groups [y * gpc, ...), tpc = 2^tsh, tpc * gpc <= QUANT_SCALES.  WIDE: x is 32-byte and q 16-byte aligned (torch tensors are);
// otherwise two 16-byte loads and two 8-byte stores take their place.
template <bool WIDE>
__global__ void __launch_bounds__(QUANT_THREADS) quantize_1x128_kernel(const __nv_bfloat16* __restrict__ x, int T, int H, int tsh, int gpc,
                                                             uint8_t* __restrict__ q, float* __restrict__ scale) {
    __shared__ float s_scale[QUANT_SCALES];      // [group][token]
    const int groups = H >> 7;
    const int t0 = blockIdx.x << tsh, k0 = blockIdx.y * gpc;
    const int nt = min(1 << tsh, T - t0), nk = min(gpc, groups - k0);
    const int sub = threadIdx.x & 7;      // lane inside the group
    pdl_wait();
    pdl_launch();
    constexpr int GP = QUANT_THREADS / QUANT_LANES, U = QUANT_FLIGHT;
    const int total = nt * nk;
    int t = 0, k = threadIdx.x >> 3;      // this lane's next group inside the block
    int dt = 0, dk = GP;                  // ... and the way to the one after it
    if (nk <= GP) {
        t = k / nk; k -= t * nk;
        dt = GP / nk; dk = GP - dt * nk;
    }
    // the trip count is the same for all lanes (the shuffles below stay inside a group, but name the warp)
    for (int i0 = 0; i0 < total; i0 += U * GP) {
        alignas(16) uint32_t raw[U][8];
        int tt[U], kk[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            tt[u] = t; kk[u] = k;
#pragma unroll
            for (int i = 0; i < 8; ++i) raw[u][i] = 0u;
            const __nv_bfloat16* src = x + (size_t)(t0 + t) * H + (size_t)(k0 + k) * 128 + sub * 16;
            if (t < nt) {
                if (WIDE) {
                    ld_global_v8(src, raw[u]);
                } else {
                    *reinterpret_cast<uint4*>(&raw[u][0]) = __ldcs(reinterpret_cast<const uint4*>(src));
                    *reinterpret_cast<uint4*>(&raw[u][4]) = __ldcs(reinterpret_cast<const uint4*>(src) + 1);
                }
            }
            t += dt; k += dk;
            if (k >= nk) { k -= nk; ++t; }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(raw[u]);
            __nv_bfloat162 m = __habs2(h2[0]);
#pragma unroll
            for (int i = 1; i < 8; ++i) m = __hmax2(m, __habs2(h2[i]));
            float amax = fmaxf(__low2float(m), __high2float(m));
#pragma unroll
            for (int o = 4; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
            if (tt[u] >= nt) continue;
            const float s = amax > 0.f ? __fdiv_rn(amax, 448.0f) : 1.0f;
            const float y = __fdiv_rn(1.0f, s);
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = quantize4(unpack_negated(raw[u][2 * j]), unpack_negated(raw[u][2 * j + 1]), s, -y);
            if (!(s >= 0x1p-90f && y >= 0x1p-126f)) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 f0 = __bfloat1622float2(h2[2 * j]), f1 = __bfloat1622float2(h2[2 * j + 1]);
                    w[j] = (uint32_t)f32x2_to_e4m3x2(__fdiv_rn(f0.x, s), __fdiv_rn(f0.y, s)) |
                           ((uint32_t)f32x2_to_e4m3x2(__fdiv_rn(f1.x, s), __fdiv_rn(f1.y, s)) << 16);
                }
            }
            uint8_t* dst = q + (size_t)(t0 + tt[u]) * H + (size_t)(k0 + kk[u]) * 128 + sub * 16;
            if (WIDE) {
                *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
            } else {
                reinterpret_cast<uint2*>(dst)[0] = make_uint2(w[0], w[1]);
                reinterpret_cast<uint2*>(dst)[1] = make_uint2(w[2], w[3]);
            }
            if (sub == 0) s_scale[(kk[u] << tsh) + tt[u]] = s;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nk << tsh; i += QUANT_THREADS) {
        const int kb = i >> tsh, tl = i - (kb << tsh);
        if (tl < nt) scale[(size_t)(k0 + kb) * T + t0 + tl] = s_scale[i];
    }
}

}  // namespace b200moe
