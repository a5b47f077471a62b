// The coil sums of readout runs on the tensor cores, in float32 precision.
//
// A run is up to 128 samples of which sample p (from 0) of spin j is z_j q_j^p: z_j the spin's first sample (written by
// the propagation), q_j the complex factor of the segment that separates the samples. Coil c's sum is sum_j z_j q_j^p
// s_jc, a matrix product over the spins: [samples][2 x spins] x [2 x spins][16]. Both operands are scaled by a power
// of two (32 spins' largest value to 2^12; every coil by its own) and split into two half-precision values (11 + 11 bits:
// x = hi + lo to 2^-23 of x down to 2^-14 of the largest), and hi hi + hi lo + lo hi accumulate in float32
// (mma.sync.m16n8k16; the dropped lo lo is 2^-24) over 8 spins, then by rounded float32 adds over the warp's spins: the
// tensor cores cut a sum's bits off towards zero (Fasi, Higham, Mikaitis and Pranesh, "Numerical behavior of NVIDIA tensor
// cores", 2021), and with 32 spins in one accumulator all signals came out 1.8e-7 too small; now 5e-8, which RO_CUT makes
// up for. Relative error of the signal against float64 (float32 products and sums; 32 spins; 8 spins and RO_CUT):
// 256 spins 2.1e-7, 2.7e-7, 1.6e-7; 9,025 spins 2.5e-7, 3.0e-7, 2.0e-7; 524,288 spins x 2 TRs of four echoes 3.4e-8,
// 2.2e-7, 3.6e-8. The readout of 1,048,576 spins x 512 samples x 8 coils went from 0.658 to 0.673 ms. Measured, mma.sync issues
// every 8 cycles per SM quarter for half and tf32 alike, and half holds twice the spins: 1.5 instructions per sample
// of 32 spins at 8 coils, 12 cycles, beside about 14 other issue slots; the float32 sum on the FMA pipe took 32
// multiply-adds and 14 other slots.
// tcgen05 is not used here: its 128-row tiles take the samples from shared or tensor memory, while the fragments of
// mma.sync are formed in registers: lane l holds row l / 4 and spins l % 4 of every four, so it starts from z q^(l / 4)
// and steps by q^8 to the rows 8 apart: four multiply-adds per sample and no data moved between lanes per sample.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "bloch_common.cuh"

// One cut costs half a unit in the last place of a float32 on average: 2^-24 / m of a sum with significand m in [1, 2),
// 2^-24 / (2 ln 2) over the usual distribution of significands.
#define RO_CUT (1.0 + 0.7213 / 16777216.0)
#define RO_ROWS 8          // rows of the sample table (a fragment's rows)
// Shared memory of a warp's 32 spins, laid out so that a lane's two spins of every eight (8 g + t and 8 g + 4 + t) come
// as the operands of paired instructions, without moves: a pair is 16 bytes, (re, re', im, im'), and the rows of the
// table of powers are 80 words apart (the rows a load phase takes lie on different banks). With a complex number per
// spin, and the imaginary sums' operand turned in registers, the ALU pipe was 58 % busy, then 48 %: 0.727 -> 0.665 ms for
// 1,048,576 spins x 512 samples x 8 coils, 3.11 -> 2.89 ms for 393,216 x 6,144.
#define RO_TAB_ROW 80  // floats per table row (16 pairs + 16 words)
__device__ __forceinline__ int pair_word(int spin) { return ((spin >> 3) * 4 + (spin & 3)) * 4 + ((spin >> 2) & 1); }

// Place of (spin, coil) in the warp's staged sensitivities ([32][8] of 16 bytes), swizzled so that a fragment's four
// spins fall on different banks.
__device__ __forceinline__ int sens_slot(int spin, int coil) { return spin * 8 + (coil ^ ((spin & 3) << 1)); }

// The power of two that takes the warp's largest finite magnitude to [2^12, 2^13), and its inverse, from the bits of a
// magnitude per lane (0 where there is none).
__device__ __forceinline__ void warp_scale(uint32_t bits, float& scale, float& inverse) {
    const uint32_t m = __reduce_max_sync(0xffffffffu, bits < 0x7f800000u ? bits : 0u);
    const uint32_t e = min(max(m >> 23, 13u), 253u);
    scale = __uint_as_float((m == 0u ? 127u : 266u - max(e, 12u)) << 23);
    inverse = __uint_as_float((m == 0u ? 127u : e - 12u) << 23);
}

__device__ __forceinline__ uint32_t half_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }

// (x, y) = hi + lo, each a pair of halves (x in the low half) rounded to nearest.
__device__ __forceinline__ void split_half(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x, y);
    hi = half_bits(h);
    lo = half_bits(__floats2half2_rn(x - __low2float(h), y - __high2float(h)));
}

// The same for two spins, a and b: the differences on paired instructions.
__device__ __forceinline__ void split_half2(const float2& x, const float2& y, uint32_t* hi, uint32_t* lo) {
    const __half2 ha = __floats2half2_rn(x.x, y.x), hb = __floats2half2_rn(x.y, y.y);
    const float2 dx = __fadd2_rn(x, make_float2(-__low2float(ha), -__low2float(hb)));
    const float2 dy = __fadd2_rn(y, make_float2(-__high2float(ha), -__high2float(hb)));
    hi[0] = half_bits(ha), hi[1] = half_bits(hb);
    lo[0] = half_bits(__floats2half2_rn(dx.x, dy.x)), lo[1] = half_bits(__floats2half2_rn(dx.y, dy.y));
}

// (re, -im) halves -> (im, re): the operand of the imaginary sums.
__device__ __forceinline__ uint32_t turn_half(uint32_t v) { return __byte_perm(v, 0u, 0x1032) ^ 0x00008000u; }

// A sensitivity as the tensor cores read it: the halves of (re, -im), high parts and low parts (a value that is not
// finite has no low part), and the same of (im, re), the operand of the imaginary sums.
__device__ __forceinline__ uint4 split_sens(float re, float im) {
    uint4 v;
    split_half(re, -im, v.x, v.y);
    if (!isfinite(re)) v.y &= 0xffff0000u;
    if (!isfinite(im)) v.y &= 0x0000ffffu;
    v.z = turn_half(v.x), v.w = turn_half(v.y);
    return v;
}

__device__ __forceinline__ void mma_half(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Complex numbers of two spins as pairs of real and imaginary parts; nim: the negated imaginary parts of b.
struct CPair {
    float2 re, im;
};

__device__ __forceinline__ CPair load_pair(const float* p) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    return CPair{make_float2(v.x, v.y), make_float2(v.z, v.w)};
}

__device__ __forceinline__ CPair cmul2(const CPair& a, const CPair& b, const float2& nim) {
    return CPair{__ffma2_rn(a.re, b.re, __fmul2_rn(a.im, nim)), __ffma2_rn(a.re, b.im, __fmul2_rn(a.im, b.re))};
}

// The factor q = (1 + e2)(c + i s) in float64.
__device__ __forceinline__ void factor64(const FreeFactors& f, double& x, double& y) {
    const double a = 1.0 + (double)f.e2;
    x = a * ((double)f.ch + (double)f.cl), y = a * ((double)f.sh + (double)f.sl);
}

// q^8 and q^32, in float64 and rounded once.
__device__ __forceinline__ void factor_powers(const FreeFactors& f, float2& q8, float2& q32) {
    double x, y;
    factor64(f, x, y);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const double t = fma(x, x, -y * y);
        y = 2.0 * x * y;
        x = t;
        if (i == 2) q8 = make_float2((float)x, (float)y);
    }
    q32 = make_float2((float)x, (float)y);
}

// a += b on paired instructions, rounded to nearest.
__device__ __forceinline__ void add4(float* a, const float* b) {
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
        const float2 s = __fadd2_rn(make_float2(a[i], a[i + 1]), make_float2(b[i], b[i + 1]));
        a[i] = s.x, a[i + 1] = s.y;
    }
}

// Two fragment rows' samples (z: this lane's row, zb: the row 8 below; two spins) times the spins' sensitivities s0 and
// s1, added to dr (real parts) and di (imaginary parts).
__device__ __forceinline__ void readout_mma(const CPair& z, const CPair& zb, const uint4& s0, const uint4& s1, float* dr,
                                            float* di) {
    uint32_t h[2], l[2], hb[2], lb[2];
    split_half2(z.re, z.im, h, l);
    split_half2(zb.re, zb.im, hb, lb);
    float tr[4] = {0.0f, 0.0f, 0.0f, 0.0f}, ti[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    mma_half(tr, l[0], lb[0], l[1], lb[1], s0.x, s1.x);  // the small terms first
    mma_half(ti, l[0], lb[0], l[1], lb[1], s0.z, s1.z);
    mma_half(tr, h[0], hb[0], h[1], hb[1], s0.y, s1.y);
    mma_half(ti, h[0], hb[0], h[1], hb[1], s0.w, s1.w);
    mma_half(tr, h[0], hb[0], h[1], hb[1], s0.x, s1.x);
    mma_half(ti, h[0], hb[0], h[1], hb[1], s0.z, s1.z);
    add4(dr, tr);
    add4(di, ti);
}
