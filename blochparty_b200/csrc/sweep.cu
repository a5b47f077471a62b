// The reverse sweep over runs of like segments (bp_sweep) and what the samples add to it (bp_cotangent).
//
// For the gradients that need no per-segment sums but the RF waveform's, a run of free segments and its samples have
// closed forms, and the sweep takes a run in one step where bp_adjoint takes every segment of it, twice:
//  * A run's samples are m_p = q^p z, z the first one (bp_propagate's runs; m and lambda as complex numbers x + i y). A
//    sample adds D_p = sum_c conj(s_c) H_pc to lambda there, so the run adds G0 = sum_p conj(q)^p D_p to lambda at its
//    first sample, and its later segments, each shared by the samples after it, add to the gradients of q's phase and
//    decay what G1 = sum_p p conj(q)^p D_p says: conj(z) G1. The coils' gradients are conj(z) T_c with
//    T_c = sum_p conj(q)^p H_pc, and G0 = sum_c conj(s_c) T_c. bp_cotangent_kernel forms T_c as a matrix product,
//    [spins][2 x samples] x [2 x samples][16], on the tensor cores in float32 precision, as the readout does
//    (readout.cuh: half-precision pairs, three products, float32 sums).
//  * Along free segments without samples lambda conj(m) keeps its value, so n segments add n times what one adds.
//  * A run of RF segments is integrated backward from the state after it (as bp_adjoint's sweep without per-spin
//    gradients does); K = 2 spins per thread run its arithmetic on paired instructions.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "packed.cuh"
#include "readout.cuh"
#include "../../include/blochparty_b200.h"

// ---- the samples' part ----

// A block is up to 32 samples of one run (subs: run, block). hs [rows][8 ncg]: the halves of (h0, -h1) of every row and
// coil, scaled by a power of two that takes the largest finite magnitude of the block and coil to 2^12; zero coils to pad;
// inverse [rows][8 ncg]: the scales' inverses, in the row of a block's first sample. (One scale for the whole sequence lost
// the gradients of late pulses where a loss weighs early samples 10^9 above late ones. With the turned halves too, as the
// readout's, bp_cotangent read twice the bytes: 0.83 -> 0.89 ms at 1,048,576 spins x 512 samples.)
#define HS_THREADS 256
__global__ void __launch_bounds__(HS_THREADS) bp_h_split_kernel(const float* __restrict__ h, int n_coils, int width,
                                                                const int4* __restrict__ runs,
                                                                const int2* __restrict__ subs, uint2* __restrict__ hs,
                                                                float* __restrict__ inverse) {
    const int lane = threadIdx.x & 31;
    const int2 sub = subs[blockIdx.x];
    const int4 run = runs[sub.x];
    const int64_t row0 = run.w + 32 * sub.y, row = row0 + lane;
    const bool there = lane < run.z - 32 * sub.y;
    for (int c = threadIdx.x >> 5; c < width; c += HS_THREADS / 32) {  // a warp per coil, a lane per sample
        float re = 0.0f, im = 0.0f, scale, inv;
        if (there && c < n_coils) re = h[row * 2 * n_coils + 2 * c], im = h[row * 2 * n_coils + 2 * c + 1];
        const uint32_t u = __float_as_uint(fabsf(re)), v = __float_as_uint(fabsf(im));
        warp_scale(max(u < 0x7f800000u ? u : 0u, v < 0x7f800000u ? v : 0u), scale, inv);
        const uint4 s = split_sens(re * scale, im * scale);
        if (there) hs[row * width + c] = make_uint2(s.x, s.y);
        if (lane == 0) inverse[row0 * width + c] = inv;
    }
}

#define CO_THREADS 128
#define CO_WARPS (CO_THREADS / 32)
#define CO_TAB_STRIDE 36  // float2 per row of the powers (32 spins + 4)
#define CO_ONE 1024.0f  // the powers' scale: a power of two that keeps their low halves normal, and 31 times them a half

struct CotArgs {
    const float* spins;
    const float* sens;
    const SegRec* segs;
    const double4* seg64;
    const int4* windows;
    int n, n_coils, wa, wb;
    const int4* runs;
    int n_runs;
    const uint2* hs;       // [rows][8 ncg]
    const float* inverse;  // the same: of the scales, by block
    float2* g0;            // [runs that start in the windows][n]
    float2* g1;            // null, or the same of G1
    const float2* z;       // with gc: the runs' first samples, [runs that start in the windows][n]
    float* gc;             // null, or [2C][n]: += the coils' gradients
};

// The first run that starts at segment s or later.
__device__ __forceinline__ int run_from(const int4* __restrict__ runs, int n_runs, int s) {
    int lo = 0, hi = n_runs;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (runs[mid].x < s)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// G1: whether the samples' numbers weigh a second sum. blockIdx.x: 128 spins, a warp 32 of them; blockIdx.y: every
// gridDim.y-th run (one part with coil gradients: they are summed over the runs, last to first).
template <bool WANT1>
__global__ void __launch_bounds__(CO_THREADS, WANT1 ? 3 : 4) bp_cotangent_kernel(CotArgs a) {
    __shared__ float2 tabs[CO_WARPS][RO_ROWS * CO_TAB_STRIDE];  // conj(q)^0 .. conj(q)^7 per spin
    __shared__ float2 steps[CO_WARPS][2][32];                   // conj(q)^8, conj(q)^32
    __shared__ float2 firsts[CO_WARPS][32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r = lane >> 2, t = lane & 3;
    const int n = a.n, j0 = ((int)blockIdx.x * CO_WARPS + warp) * 32;
    if (j0 >= n) return;
    float2* tab = tabs[warp];
    const int lo = run_from(a.runs, a.n_runs, a.windows[a.wa].x), hi = run_from(a.runs, a.n_runs, a.windows[a.wb - 1].y);
    const int ncg = (a.n_coils + 7) / 8, width = 8 * ncg;
    const int jl = min(j0 + lane, n - 1);
    const Spin sp = load_spin(a.spins, n, jl, true);
    const PropSpin p{(double)sp.px, (double)sp.py, (double)sp.pz, (double)sp.db0, sp.pd, sp.r1, sp.r2};
    int factors_of = -1;  // the segment whose factor's powers the table holds
    for (int run = hi - 1 - (int)blockIdx.y; run >= lo; run -= gridDim.y) {
        const int4 rr = a.runs[run];
        const int seg = rr.y >= 0 ? rr.y : rr.x;
        bool same = factors_of >= 0;
        if (same && seg != factors_of) {  // (uniform)
            const double4 x = a.seg64[factors_of], y = a.seg64[seg];
            same = a.segs[factors_of].dt == a.segs[seg].dt && x.x == y.x && x.y == y.y && x.z == y.z && x.w == y.w;
        }
        __syncwarp();
        if (!same) {
            FreeFactors f = prop_factors(a.segs[seg].dt, a.seg64[seg], p, 1);
            f.sh = -f.sh, f.sl = -f.sl;  // conj(q)
            float2 q8, q32;
            factor_powers(f, q8, q32);
            float zr = CO_ONE, zi = 0.0f;
            tab[lane] = make_float2(zr, zi);
#pragma unroll
            for (int i = 1; i < RO_ROWS; ++i) {
                readout_advance(f, zr, zi);
                tab[i * CO_TAB_STRIDE + lane] = make_float2(zr, zi);
            }
            steps[warp][0][lane] = q8;
            steps[warp][1][lane] = q32;
            factors_of = seg;
        }
        if (a.gc) firsts[warp][lane] = a.z[(size_t)(run - lo) * n + jl];
        __syncwarp();
        float2 g0[2][2], g1[2][2];  // 16 spins, row r and 8 below
#pragma unroll
        for (int i = 0; i < 4; ++i) g0[i >> 1][i & 1] = g1[i >> 1][i & 1] = make_float2(0.0f, 0.0f);
        for (int cg = 0; cg < ncg; ++cg) {
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                const int sa = 16 * mt + r, sb = sa + 8;
                float tr[4] = {0.f, 0.f, 0.f, 0.f}, ti[4] = {0.f, 0.f, 0.f, 0.f};
                float ur[4] = {0.f, 0.f, 0.f, 0.f}, ui[4] = {0.f, 0.f, 0.f, 0.f};
                // samples t and t + 4 of the block of 32, two spins; their steps by eight and by 32
                const float2 ta = tab[t * CO_TAB_STRIDE + sa], ta4 = tab[(t + 4) * CO_TAB_STRIDE + sa];
                const float2 tb = tab[t * CO_TAB_STRIDE + sb], tb4 = tab[(t + 4) * CO_TAB_STRIDE + sb];
                CPair wa{make_float2(ta.x, ta4.x), make_float2(ta.y, ta4.y)};
                CPair wb{make_float2(tb.x, tb4.x), make_float2(tb.y, tb4.y)};
                const float2 ea = steps[warp][0][sa], eb = steps[warp][0][sb];
                const CPair qa{make_float2(ea.x, ea.x), make_float2(ea.y, ea.y)};
                const CPair qb{make_float2(eb.x, eb.x), make_float2(eb.y, eb.y)};
                const float2 na = make_float2(-ea.y, -ea.y), nb = make_float2(-eb.y, -eb.y);
                for (int blk = 0; blk < rr.z; blk += 32) {
                    float dr[4] = {0.f, 0.f, 0.f, 0.f}, di[4] = {0.f, 0.f, 0.f, 0.f};
                    float er[4] = {0.f, 0.f, 0.f, 0.f}, ei[4] = {0.f, 0.f, 0.f, 0.f};
                    const float2 iv = *reinterpret_cast<const float2*>(a.inverse + (size_t)(rr.w + blk) * width + 8 * cg + 2 * t);
                    CPair xa = wa, xb = wb;
                    const int cnt = min(32, rr.z - blk);
                    for (int kb = 0; kb < cnt; kb += 8) {
                        const int p0 = kb + t, p1 = p0 + 4;
                        const uint2* hrow = a.hs + ((size_t)(rr.w + blk + p0) * width + 8 * cg + r);
                        const uint2 zero = make_uint2(0u, 0u);
                        const uint2 b0 = p0 < cnt ? hrow[0] : zero, b1 = p1 < cnt ? hrow[(size_t)4 * width] : zero;
                        const uint2 c0 = make_uint2(turn_half(b0.x), turn_half(b0.y));
                        const uint2 c1 = make_uint2(turn_half(b1.x), turn_half(b1.y));
                        uint32_t ha[2], la[2], hb[2], lb[2];
                        split_half2(xa.re, xa.im, ha, la);
                        split_half2(xb.re, xb.im, hb, lb);
                        mma_half(dr, la[0], lb[0], la[1], lb[1], b0.x, b1.x);
                        mma_half(di, la[0], lb[0], la[1], lb[1], c0.x, c1.x);
                        mma_half(dr, ha[0], hb[0], ha[1], hb[1], b0.y, b1.y);
                        mma_half(di, ha[0], hb[0], ha[1], hb[1], c0.y, c1.y);
                        mma_half(dr, ha[0], hb[0], ha[1], hb[1], b0.x, b1.x);
                        mma_half(di, ha[0], hb[0], ha[1], hb[1], c0.x, c1.x);
                        if (WANT1) {  // the same weighed by the samples' numbers in the block
                            const float2 num = make_float2((float)p0, (float)p1);
                            split_half2(__fmul2_rn(xa.re, num), __fmul2_rn(xa.im, num), ha, la);
                            split_half2(__fmul2_rn(xb.re, num), __fmul2_rn(xb.im, num), hb, lb);
                            mma_half(er, la[0], lb[0], la[1], lb[1], b0.x, b1.x);
                            mma_half(ei, la[0], lb[0], la[1], lb[1], c0.x, c1.x);
                            mma_half(er, ha[0], hb[0], ha[1], hb[1], b0.y, b1.y);
                            mma_half(ei, ha[0], hb[0], ha[1], hb[1], c0.y, c1.y);
                            mma_half(er, ha[0], hb[0], ha[1], hb[1], b0.x, b1.x);
                            mma_half(ei, ha[0], hb[0], ha[1], hb[1], c0.x, c1.x);
                        }
                        xa = cmul2(xa, qa, na);
                        xb = cmul2(xb, qb, nb);
                    }
                    const float2 inv = __fmul2_rn(iv, make_float2(1.0f / CO_ONE, 1.0f / CO_ONE));
                    const float2 from = make_float2((float)blk, (float)blk);
#pragma unroll
                    for (int i = 0; i < 4; i += 2) {  // (two coils on paired instructions)
                        const float2 x = __fmul2_rn(make_float2(dr[i], dr[i + 1]), inv);
                        const float2 y = __fmul2_rn(make_float2(di[i], di[i + 1]), inv);
                        float2 v = __fadd2_rn(make_float2(tr[i], tr[i + 1]), x);
                        tr[i] = v.x, tr[i + 1] = v.y;
                        v = __fadd2_rn(make_float2(ti[i], ti[i + 1]), y);
                        ti[i] = v.x, ti[i + 1] = v.y;
                        if (WANT1) {
                            v = __ffma2_rn(make_float2(er[i], er[i + 1]), inv, make_float2(ur[i], ur[i + 1]));
                            v = __ffma2_rn(from, x, v);
                            ur[i] = v.x, ur[i + 1] = v.y;
                            v = __ffma2_rn(make_float2(ei[i], ei[i + 1]), inv, make_float2(ui[i], ui[i + 1]));
                            v = __ffma2_rn(from, y, v);
                            ui[i] = v.x, ui[i + 1] = v.y;
                        }
                    }
                    if (blk + 32 < rr.z) {
                        const float2 fa = steps[warp][1][sa], fb = steps[warp][1][sb];
                        wa = cmul2(wa, CPair{make_float2(fa.x, fa.x), make_float2(fa.y, fa.y)}, make_float2(-fa.y, -fa.y));
                        wb = cmul2(wb, CPair{make_float2(fb.x, fb.x), make_float2(fb.y, fb.y)}, make_float2(-fb.y, -fb.y));
                    }
                }
                // T_c of spins sa (i = 0, 1) and sb (2, 3), coils 2 t and 2 t + 1
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int j = j0 + (h ? sb : sa);
                    const bool there = j < n;
                    const int jj = there ? j : n - 1;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int c = 8 * cg + 2 * t + i;
                        const float xr = tr[2 * h + i], xi = ti[2 * h + i];
                        const float sr = a.sens[(size_t)(2 * c) * n + jj], si = a.sens[(size_t)(2 * c + 1) * n + jj];
                        g0[mt][h].x = fmaf(sr, xr, fmaf(si, xi, g0[mt][h].x));
                        g0[mt][h].y = fmaf(sr, xi, fmaf(-si, xr, g0[mt][h].y));
                        if (WANT1) {
                            const float yr = ur[2 * h + i], yi = ui[2 * h + i];
                            g1[mt][h].x = fmaf(sr, yr, fmaf(si, yi, g1[mt][h].x));
                            g1[mt][h].y = fmaf(sr, yi, fmaf(-si, yr, g1[mt][h].y));
                        }
                        if (a.gc && there && c < a.n_coils) {  // conj(z) T_c
                            const float2 z = firsts[warp][h ? sb : sa];
                            float *gr = a.gc + (size_t)(2 * c) * n + j, *gi = gr + n;
                            *gr += fmaf(z.x, xr, z.y * xi);
                            *gi += fmaf(z.x, xi, -z.y * xr);
                        }
                    }
                }
            }
        }
        // over the four lanes of a spin's coils, then one lane writes it
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float2 v = g0[i >> 1][i & 1], w = g1[i >> 1][i & 1];
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                v.x += __shfl_xor_sync(0xffffffffu, v.x, o), v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
                if (WANT1) w.x += __shfl_xor_sync(0xffffffffu, w.x, o), w.y += __shfl_xor_sync(0xffffffffu, w.y, o);
            }
            const int j = j0 + 16 * (i >> 1) + 8 * (i & 1) + r;
            if (t == 0 && j < n) {
                a.g0[(size_t)(run - lo) * n + j] = v;
                if (WANT1) a.g1[(size_t)(run - lo) * n + j] = w;
            }
        }
    }
}

// ---- the sweep ----
#define SW_MAX 2048  // segments of an interval (its RF gradient is summed in shared memory)
#define SW_WIN BP_ADJ_WIN

struct SweepArgs {
    const float* spins;
    const SegRec* segs;
    const double4* seg64;
    const int4* windows;    // the adjoint's windows, each of RF segments or of free ones (SavedStates)
    int n, wa, wb;
    int seg0, seg_len;
    const float* wstates;   // per-spin gradients: [wb - wa + 1][6][n] state at every window start, then after the last
                            // window; else states by slot
    const int* wslot;       // null (per-spin gradients), or [n_windows + 1]: the slot of the state at a window's start
    float* chain;           // with wslot: [3][n], the state an RF run is integrated to, between calls
    int chain_in;
    const int4* runs;
    int n_runs;
    const float2* g0;       // [runs that start in the windows][n], or null: no samples
    const float2* g1;       // with per-spin gradients
    float* lam;             // [3][n] in, out
    float* gs;              // [8][n] += (px py pz db0 pd r1 r2 b1), or null
    float* gseg;            // [gridDim.x][seg_len][2]: the RF gradient's per-CTA sums, or null
    int* status;
};

// An RF segment backward for K spins, from its output state o (turned into its input) and lambda l (likewise), as
// bp_adjoint's rf_back, with the per-spin gradients of rf_reverse where SG. gx, gy: dL/d(-2 pi dt rf).
template <int K>
struct BackRun {
    Pk<K> a1, a2, ia1, ia2, pe;  // half-step factors and their inverses, pd expm1(-dt r1 / 2)
    Pk<K> wz, nwz, wz2;
};

template <bool SMALL, bool SG, int K>
__device__ __forceinline__ void rf_back_packed(const Pk<K>& wx0, const Pk<K>& wy0, const Pk<K>& b1, const Pk<K>& nb1,
                                               const BackRun<K>& r, const PropSpin* p, const SegRec& q, Pk<K>& ox,
                                               Pk<K>& oy, Pk<K>& oz, Pk<K>& lx, Pk<K>& ly, Pk<K>& lz, Pk<K>& gx,
                                               Pk<K>& gy, float* g) {
    const Pk<K> wx = pmul(wx0, b1), wy = pmul(wy0, b1), nwx = pmul(wx0, nb1), nwy = pmul(wy0, nb1);
    const Pk<K> p2 = pfma(wx, wx, pfma(wy, wy, r.wz2));
    Pk<K> s1, s2, s3;
    if (SMALL) {
        s1 = pfma(p2, pfma(p2, pfma(p2, pset<K>(-1.9841269841269841e-04f), pset<K>(8.3333333333333333e-03f)),
                           pset<K>(-1.6666666666666667e-01f)), pset<K>(1.0f));
        s2 = pfma(p2, pfma(p2, pfma(p2, pset<K>(-2.4801587301587302e-05f), pset<K>(1.3888888888888889e-03f)),
                           pset<K>(-4.1666666666666667e-02f)), pset<K>(0.5f));
        s3 = pfma(p2, pfma(p2, pfma(p2, pset<K>(-2.7557319223985893e-06f), pset<K>(1.9841269841269841e-04f)),
                           pset<K>(-8.3333333333333333e-03f)), pset<K>(1.6666666666666667e-01f));
    } else {
        float u[K], v[K], w[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const float x = p2.get(k);
            rodrigues_coeffs(x, u[k], v[k]);
            w[k] = x < 1.0f ? fmaf(x, fmaf(x, fmaf(x, fmaf(x, fmaf(x, -1.6059043836821615e-10f, 2.5052108385441720e-08f),
                                                           -2.7557319223985893e-06f), 1.9841269841269841e-04f),
                                           -8.3333333333333333e-03f), 1.6666666666666667e-01f)
                            : (1.0f - u[k]) / x;
        }
        s1 = pmake<K>(u), s2 = pmake<K>(v), s3 = pmake<K>(w);
    }
    const Pk<K> minus = pset<K>(-1.0f);
    const Pk<K> ns1 = pmul(s1, minus), ns2 = pmul(s2, minus), c = pfma(ns2, p2, pset<K>(1.0f));
    const Pk<K> nx = pmul(ox, r.ia2), ny = pmul(oy, r.ia2), nz = pmul(padd(oz, r.pe), r.ia1);
    const Pk<K> ax = pmul(lx, r.a2), ay = pmul(ly, r.a2), az = pmul(lz, r.a1);  // dL/dn
    const Pk<K> k2 = pmul(s2, pfma(wx, ax, pfma(wy, ay, pmul(r.wz, az))));
    const Pk<K> bx = pfma(c, ax, pfma(ns1, pfma(wy, az, pmul(r.nwz, ay)), pmul(k2, wx)));
    const Pk<K> by = pfma(c, ay, pfma(ns1, pfma(r.wz, ax, pmul(nwx, az)), pmul(k2, wy)));
    const Pk<K> bz = pfma(c, az, pfma(ns1, pfma(wx, ay, pmul(nwy, ax)), pmul(k2, r.wz)));
    const Pk<K> mx = pmul(nx, minus), my = pmul(ny, minus), mz = pmul(nz, minus);
    const Pk<K> ux = pfma(ny, az, pmul(mz, ay)), uy = pfma(nz, ax, pmul(mx, az)), uz = pfma(nx, ay, pmul(my, ax));
    const Pk<K> k3 = pmul(s3, pfma(wx, ux, pfma(wy, uy, pmul(r.wz, uz))));
    gx = pfma(s1, ux, pfma(ns2, pfma(wy, uz, pmul(r.nwz, uy)), pmul(k3, wx)));
    gy = pfma(s1, uy, pfma(ns2, pfma(r.wz, ux, pmul(nwx, uz)), pmul(k3, wy)));
    const Pk<K> k4 = pmul(s2, pfma(wx, nx, pfma(wy, ny, pmul(r.wz, nz))));
    const Pk<K> ix = pfma(c, nx, pfma(ns1, pfma(wy, nz, pmul(r.nwz, ny)), pmul(k4, wx)));
    const Pk<K> iy = pfma(c, ny, pfma(ns1, pfma(r.wz, nx, pmul(nwx, nz)), pmul(k4, wy)));
    const Pk<K> iz = pfma(c, nz, pfma(ns1, pfma(wx, ny, pmul(nwy, nx)), pmul(k4, r.wz)));
    const Pk<K> x0 = pmul(ix, r.ia2), y0 = pmul(iy, r.ia2), z0 = pmul(padd(iz, r.pe), r.ia1);
    if constexpr (SG) {
        static_assert(!SG || K == 1, "per-spin gradients: one spin per thread");
        const float gwz = fmaf(s1.f, uz.f, fmaf(ns2.f, fmaf(wx.f, uy.f, nwy.f * ux.f), k3.f * r.wz.f));
        const float h = 0.5f * q.dt, e1h = r.a1.f - 1.0f;
        const float gd2 = fmaf(bx.f, x0.f, fmaf(by.f, y0.f, fmaf(lx.f, nx.f, ly.f * ny.f)));
        const float gd1 = fmaf(bz.f, z0.f - p->pd, lz.f * (nz.f - p->pd));
        g[5] = fmaf(-gd1 * h, r.a1.f, g[5]);
        g[6] = fmaf(-gd2 * h, r.a2.f, g[6]);
        g[4] = fmaf(-(lz.f + bz.f), e1h, g[4]);
        g[7] = fmaf(gx.f, wx0.f, fmaf(gy.f, wy0.f, g[7]));
        const float gcyc = -BP_TWO_PI_F * gwz;
        g[0] = fmaf(gcyc, q.kx, g[0]), g[1] = fmaf(gcyc, q.ky, g[1]), g[2] = fmaf(gcyc, q.kz, g[2]);
        g[3] = fmaf(gcyc, q.dt, g[3]);
    }
    lx = pmul(bx, r.a2), ly = pmul(by, r.a2), lz = pmul(bz, r.a1);
    ox = x0, oy = y0, oz = z0;
}

template <int K, int NT, bool SG>
__global__ void __launch_bounds__(NT, NT == 32 ? 8 : 4) bp_sweep_kernel(SweepArgs a) {
    extern __shared__ __align__(16) float iacc[];  // [seg_len][2]: the RF gradient, summed over the CTA's tiles
    __shared__ float segacc[NT / 32][SW_WIN][2];
    __shared__ int4 win_s[32];     // of up to 32 windows: begin, end (begin: none to sweep), the last segment's flags
    __shared__ SegRec rec_s[32];   // and their first segments' records
    __shared__ double4 k64_s[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = a.n;
    constexpr int TILE = NT * K;
    const int n_tiles = (n + TILE - 1) / TILE;
    if (a.gseg)
        for (int i = tid; i < 2 * a.seg_len; i += NT) iacc[i] = 0.0f;
    __syncthreads();
    const int lo = a.g0 ? run_from(a.runs, a.n_runs, a.windows[a.wa].x) : 0;
    const int hi = a.g0 ? run_from(a.runs, a.n_runs, a.windows[a.wb - 1].y) : 0;

    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        PropSpin p[K];
        int jk[K];
        bool active[K];
        float in[6][K], bp[K], bn[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int j = tile * TILE + (warp * K + k) * 32 + lane;
            active[k] = j < n;
            jk[k] = active[k] ? j : 0;
            const Spin s = load_spin(a.spins, n, jk[k], active[k]);
            p[k] = PropSpin{(double)s.px, (double)s.py, (double)s.pz, (double)s.db0, s.pd, s.r1, s.r2};
            bp[k] = s.b1, bn[k] = -s.b1;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                in[i][k] = active[k] ? a.lam[(size_t)i * n + jk[k]] : 0.0f;
                in[3 + i][k] = !SG && a.chain_in && active[k] ? a.chain[(size_t)i * n + jk[k]] : 0.0f;
            }
        }
        const Pk<K> b1 = pmake<K>(bp), nb1 = pmake<K>(bn);
        Pk<K> lx = pmake<K>(in[0]), ly = pmake<K>(in[1]), lz = pmake<K>(in[2]);
        Pk<K> cx = pmake<K>(in[3]), cy = pmake<K>(in[4]), cz = pmake<K>(in[5]);  // !SG: the chain
        bool chained = !SG && a.chain_in != 0, lost = false;
        float g[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) g[i] = SG && active[0] ? a.gs[(size_t)i * n + jk[0]] : 0.0f;
        // the compensated state of a row set, rounded to one float32 per component
        auto load_state = [&](const float* st, Pk<K>& x, Pk<K>& y, Pk<K>& z) {
            float v[3][K];
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    v[i][k] = active[k] ? st[(size_t)i * n + jk[k]] + st[(size_t)(3 + i) * n + jk[k]] : 0.0f;
            x = pmake<K>(v[0]), y = pmake<K>(v[1]), z = pmake<K>(v[2]);
        };
        // the last run not yet met: its first segment and what its samples add, read as soon as the one after it is done
        int run, next;
        float2 add0[K], add1;
        SegRec rq{};
        auto meet = [&](int r) {
            run = r, next = -1;
            if (r < lo) return;
            const int4 rr = a.runs[r];
            next = rr.x;
#pragma unroll
            for (int k = 0; k < K; ++k)
                add0[k] = active[k] ? a.g0[(size_t)(r - lo) * n + jk[k]] : make_float2(0.0f, 0.0f);
            if constexpr (SG) {
                add1 = active[0] ? a.g1[(size_t)(r - lo) * n + jk[0]] : make_float2(0.0f, 0.0f);
                rq = a.segs[rr.y >= 0 ? rr.y : rr.x];  // (a single sample's add1 is 0)
            }
        };
        meet(hi - 1);
        // windows [blk, ...) are staged in `win_s` and the rest; the state at a window's start is read one window ahead
        float ahead[6];
        auto read_ahead = [&](int w) {
#pragma unroll
            for (int i = 0; i < 6; ++i) ahead[i] = 0.0f;
            if (SG && w >= a.wa && active[0]) {
                const float* st = a.wstates + (size_t)(w - a.wa) * 6 * n + jk[0];
#pragma unroll
                for (int i = 0; i < 6; ++i) ahead[i] = st[(size_t)i * n];
            }
        };
        Pk<K> x0 = pset<K>(0.0f), y0 = x0, z0 = x0;  // SG: the state at the start of the window after this one
        if (SG) load_state(a.wstates + (size_t)(a.wb - a.wa) * 6 * n, x0, y0, z0);
        read_ahead(a.wb - 1);
        int blk = a.wb;
        for (int w = a.wb - 1; w >= a.wa; --w) {
            if (w < blk) {  // the records of up to 32 windows at once: their loads' latency once
                blk = max(a.wa, w - 31);
                __syncthreads();
                if (tid < w - blk + 1) {
                    const int4 v = a.windows[blk + tid];
                    const bool fine = v.y > v.x && v.y - v.x <= SW_WIN && v.x >= a.seg0 && v.y <= a.seg0 + a.seg_len;
                    win_s[tid] = make_int4(v.x, fine ? v.y : v.x, fine ? a.segs[v.y - 1].flags : 0, 0);
                    if (fine) rec_s[tid] = a.segs[v.x], k64_s[tid] = a.seg64[v.x];
                }
                __syncthreads();
            }
            const int4 win = win_s[w - blk];
            const int nseg = win.y - win.x;
            // SG: this window's start state (read ahead), and the next one's on its way
            const Pk<K> ex = x0, ey = y0, ez = z0;  // the state after the window
            if constexpr (SG) {
                x0 = Pk<K>{ahead[0] + ahead[3]}, y0 = Pk<K>{ahead[1] + ahead[4]}, z0 = Pk<K>{ahead[2] + ahead[5]};
                read_ahead(w - 1);
            }
            if (nseg <= 0) {  // (uniform) not a window of this interval
                if (tid == 0) atomicOr(a.status, BP_ERR_BAD_WINDOW);
                continue;
            }
            const SegRec q = rec_s[w - blk];
            const int last = win.z;
            if (q.flags & BP_RF) {
                Pk<K> ox = cx, oy = cy, oz = cz;  // the state after the window
                if (SG) {
                    ox = ex, oy = ey, oz = ez;
                } else if (!chained) {
                    const int sl = a.wslot[w + 1];
                    if (sl < 0)
                        lost = true;  // (reported: the results are not valid)
                    else
                        load_state(a.wstates + (size_t)sl * 6 * n, ox, oy, oz);
                }
                BackRun<K> rb;
                float a1[K], a2[K], i1[K], i2[K], pe[K], wz[K], nwz[K], wz2[K];
                bool small = true;
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const float e1h = relax_expm1(-0.5f * q.dt * p[k].r1), e2h = relax_expm1(-0.5f * q.dt * p[k].r2);
                    a1[k] = 1.0f + e1h, a2[k] = 1.0f + e2h, i1[k] = 1.0f / a1[k], i2[k] = 1.0f / a2[k];
                    pe[k] = p[k].pd * e1h;
                    Spin s{};
                    s.px = (float)p[k].x, s.py = (float)p[k].y, s.pz = (float)p[k].z, s.db0 = (float)p[k].db0;
                    wz[k] = rf_wz(q, s), nwz[k] = -wz[k], wz2[k] = wz[k] * wz[k];
                }
                rb.a1 = pmake<K>(a1), rb.a2 = pmake<K>(a2), rb.ia1 = pmake<K>(i1), rb.ia2 = pmake<K>(i2);
                rb.pe = pmake<K>(pe);
                rb.wz = pmake<K>(wz), rb.nwz = pmake<K>(nwz), rb.wz2 = pmake<K>(wz2);
                // the window's RF, a segment per lane (its other values are the first segment's); every rotation small for
                // every spin of the warp: |w|^2 <= b1^2 max(wx0^2 + wy0^2) + wz^2
                float rfx = q.wx0, rfy = q.wy0;
                if (nseg > 1) {
                    const SegRec* qs = a.segs + min(win.x + lane, win.y - 1);
                    rfx = qs->wx0, rfy = qs->wy0;
                }
                {
                    const float v = fmaf(rfx, rfx, rfy * rfy);
                    const float top = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
#pragma unroll
                    for (int k = 0; k < K; ++k) small = small && fmaf(bp[k] * bp[k], top, wz2[k]) < 0.0624f;
                    small = __all_sync(0xffffffffu, small);
                }
                auto back = [&](auto tag) {
                    for (int s = nseg - 1; s >= 0; --s) {
                        Pk<K> gx, gy;
                        rf_back_packed<decltype(tag)::value, SG>(pset<K>(__shfl_sync(0xffffffffu, rfx, s)),
                                                                 pset<K>(__shfl_sync(0xffffffffu, rfy, s)), b1, nb1, rb, p,
                                                                 q, ox, oy, oz, lx, ly, lz, gx, gy, g);
                        if (a.gseg) {  // dL/d(-2 pi dt rf), summed over the warp: x into lane 0, y into lane 16
                            const Pk<K> vx = pmul(gx, b1), vy = pmul(gy, b1);
                            float v0 = active[0] ? vx.get(0) : 0.0f, v1 = active[0] ? vy.get(0) : 0.0f;
                            if (K > 1 && active[K - 1]) v0 += vx.get(K - 1), v1 += vy.get(K - 1);
                            const bool up = lane & 16;
                            float t = (up ? v1 : v0) + __shfl_xor_sync(0xffffffffu, up ? v0 : v1, 16);
#pragma unroll
                            for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                            if ((lane & 15) == 0) segacc[warp][s][up ? 1 : 0] = t;
                        }
                    }
                };
                if (small)
                    back(std::true_type{});
                else
                    back(std::false_type{});
                if (!SG) cx = ox, cy = oy, cz = oz, chained = true;
                if (a.gseg) {
                    __syncthreads();
                    for (int i = tid; i < 2 * nseg; i += NT) {
                        float t = 0.0f;
#pragma unroll
                        for (int ww = 0; ww < NT / 32; ++ww) t += segacc[ww][i >> 1][i & 1];
                        iacc[2 * (win.x - a.seg0) + i] += t;
                    }
                    __syncthreads();
                }
                continue;
            }
            chained = false;
            if (last & BP_SPOIL) lx = ly = pset<K>(0.0f);
            const double4 k64 = k64_s[w - blk];
            int cur = nseg;
            while (cur > 0) {
                // segments [from, cur) in one step: back to the last run that starts in the window, or to its start
                const bool at_run = next >= win.x;
                const int from = at_run ? next - win.x + 1 : 0, reps = cur - from;
                float v[3][K];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    v[0][k] = lx.get(k), v[1][k] = ly.get(k), v[2][k] = lz.get(k);
                    if (reps > 0) {
                        const FreeFactors f = prop_factors(q.dt, k64, p[k], reps);
                        const float x = v[0][k], y = v[1][k], z = v[2][k], e2 = 1.0f + f.e2;
                        v[0][k] = e2 * fmaf(f.ch, x, f.sh * y), v[1][k] = e2 * fmaf(-f.sh, x, f.ch * y);
                        v[2][k] = fmaf(z, f.e1, z);
                        if constexpr (SG) {
                            // the state after the step: the window's start state after `cur` segments
                            const FreeFactors u = from == 0 ? f : prop_factors(q.dt, k64, p[0], cur);
                            const float a2 = 1.0f + u.e2;
                            const float mx = a2 * fmaf(u.ch, x0.f, -u.sh * y0.f), my = a2 * fmaf(u.sh, x0.f, u.ch * y0.f);
                            const float zu = z0.f - p[0].pd;  // and Mz - pd before it
                            const float zf = from == 0 ? zu : fmaf(zu, relax_expm1(-__fmul_rn(q.dt, (float)from) * p[0].r1), zu);
                            const float dt = __fmul_rn(q.dt, (float)reps);
                            const float re = fmaf(x, mx, y * my), gcyc = -BP_TWO_PI_F * fmaf(y, mx, -x * my);
                            g[6] = fmaf(-dt, re, g[6]);
                            g[5] = fmaf(-dt * (1.0f + f.e1), z * zf, g[5]);
                            g[4] = fmaf(-z, f.e1, g[4]);
                            const float many = (float)reps;
                            g[0] = fmaf(gcyc, many * q.kx, g[0]), g[1] = fmaf(gcyc, many * q.ky, g[1]);
                            g[2] = fmaf(gcyc, many * q.kz, g[2]), g[3] = fmaf(gcyc, dt, g[3]);
                        }
                    }
                    if (at_run) {  // the run's samples
                        v[0][k] += add0[k].x, v[1][k] += add0[k].y;
                        if constexpr (SG) {  // and its later segments' phase and decay
                            const FreeFactors u = prop_factors(q.dt, k64, p[0], from);
                            const float a2 = 1.0f + u.e2;
                            const float mx = a2 * fmaf(u.ch, x0.f, -u.sh * y0.f), my = a2 * fmaf(u.sh, x0.f, u.ch * y0.f);
                            const float re = fmaf(add1.x, mx, add1.y * my);
                            const float gcyc = -BP_TWO_PI_F * fmaf(add1.y, mx, -add1.x * my);
                            g[6] = fmaf(-rq.dt, re, g[6]);
                            g[0] = fmaf(gcyc, rq.kx, g[0]), g[1] = fmaf(gcyc, rq.ky, g[1]);
                            g[2] = fmaf(gcyc, rq.kz, g[2]), g[3] = fmaf(gcyc, rq.dt, g[3]);
                        }
                    }
                }
                lx = pmake<K>(v[0]), ly = pmake<K>(v[1]), lz = pmake<K>(v[2]);
                cur = from;
                if (at_run) meet(run - 1);
            }
        }
        if (lost && lane == 0) atomicOr(a.status, BP_ERR_NO_STATE);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!active[k]) continue;
            a.lam[jk[k]] = lx.get(k), a.lam[(size_t)n + jk[k]] = ly.get(k), a.lam[2 * (size_t)n + jk[k]] = lz.get(k);
            if (!SG) {
                a.chain[jk[k]] = cx.get(k), a.chain[(size_t)n + jk[k]] = cy.get(k);
                a.chain[2 * (size_t)n + jk[k]] = cz.get(k);
            }
        }
        if (SG && active[0])
#pragma unroll
            for (int i = 0; i < 8; ++i) a.gs[(size_t)i * n + jk[0]] = g[i];
    }
    if (a.gseg) {
        __syncthreads();
        float* dst = a.gseg + (size_t)blockIdx.x * 2 * a.seg_len;
        for (int i = tid; i < 2 * a.seg_len; i += NT) dst[i] = iacc[i];
    }
}

// seg[seg0 + s][1, 2] += sum over CTAs of gseg[cta][s][0, 1] in float64: blockDim.y shares of the CTAs, each in order,
// then the shares in order
__global__ void bp_sweep_reduce_kernel(const float* __restrict__ gseg, int n_cta, int seg_len, int seg0,
                                       double* __restrict__ seg) {
    __shared__ double part[16][32];
    const int i = blockIdx.x * 32 + threadIdx.x;
    double t = 0.0;
    if (i < 2 * seg_len)
#pragma unroll 4
        for (int c = threadIdx.y; c < n_cta; c += 16) t += (double)gseg[(size_t)c * 2 * seg_len + i];
    part[threadIdx.y][threadIdx.x] = t;
    __syncthreads();
    if (threadIdx.y != 0 || i >= 2 * seg_len) return;
    for (int k = 1; k < 16; ++k) t += part[k][threadIdx.x];
    seg[(size_t)(seg0 + (i >> 1)) * 8 + 1 + (i & 1)] += t;
}

// ---- launchers ----
extern "C" int bp_cotangent_split(const float* h, int n_adc, int n_coils, const int* runs, int n_runs, const int* subs,
                                  int n_subs, void* hs, float* inverse, void* stream) {
    if (n_adc < 1 || n_coils < 1 || n_coils > BP_MAX_COILS || n_runs < 0 || n_subs < 0) return BP_E_ARG;
    if (n_runs == 0 || n_subs == 0) return BP_OK;
    if (!h || !runs || !subs || !hs || !inverse) return BP_E_ARG;
    if (((reinterpret_cast<uintptr_t>(hs) | reinterpret_cast<uintptr_t>(inverse)) & 7) != 0) return BP_E_ALIGN;
    bp_h_split_kernel<<<(unsigned)n_subs, HS_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
        h, n_coils, 8 * ((n_coils + 7) / 8), reinterpret_cast<const int4*>(runs), reinterpret_cast<const int2*>(subs),
        static_cast<uint2*>(hs), inverse);
    return cudaGetLastError() == cudaSuccess ? BP_OK : BP_E_LAUNCH;
}

extern "C" int bp_cotangent(const float* spins, const float* sens, int n, int n_coils, const void* segs,
                            const double* seg64, const int* windows, int wa, int wb, const int* runs, int n_runs,
                            const void* hs, const float* inverse, float* g0, float* g1, const float* z, float* gc,
                            void* stream) {
    if (n < 1 || n_coils < 1 || n_coils > BP_MAX_COILS || wa < 0 || wb < wa || n_runs < 0) return BP_E_ARG;
    if (wb == wa || n_runs == 0) return BP_OK;
    if (!spins || !sens || !segs || !seg64 || !windows || !runs || !hs || !inverse || !g0 || (gc && !z)) return BP_E_ARG;
    if (((reinterpret_cast<uintptr_t>(hs) | reinterpret_cast<uintptr_t>(inverse) | reinterpret_cast<uintptr_t>(g0) | reinterpret_cast<uintptr_t>(g1) |
          reinterpret_cast<uintptr_t>(z)) & 7) != 0)
        return BP_E_ALIGN;
    CotArgs a{};
    a.spins = spins, a.sens = sens;
    a.segs = static_cast<const SegRec*>(segs), a.seg64 = reinterpret_cast<const double4*>(seg64);
    a.windows = reinterpret_cast<const int4*>(windows);
    a.n = n, a.n_coils = n_coils, a.wa = wa, a.wb = wb;
    a.runs = reinterpret_cast<const int4*>(runs), a.n_runs = n_runs;
    a.hs = static_cast<const uint2*>(hs), a.inverse = inverse;
    a.g0 = reinterpret_cast<float2*>(g0), a.g1 = reinterpret_cast<float2*>(g1);
    a.z = reinterpret_cast<const float2*>(z), a.gc = gc;
    const int x = (n + CO_THREADS - 1) / CO_THREADS;
    // the runs divided among CTAs until the spins' CTAs fill the GPU about twice (not with coil gradients)
    int y = gc ? 1 : (2 * 4 * num_sms() + x - 1) / x;
    if (y > n_runs) y = n_runs;
    if (y > 1024) y = 1024;
    const dim3 grid((unsigned)x, (unsigned)(y < 1 ? 1 : y));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (g1)
        bp_cotangent_kernel<true><<<grid, CO_THREADS, 0, st>>>(a);
    else
        bp_cotangent_kernel<false><<<grid, CO_THREADS, 0, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? BP_OK : BP_E_LAUNCH;
}

template <int K, int NT, bool SG>
static int sweep_grid(int n, int seg_len) {
    const size_t smem = (size_t)2 * seg_len * sizeof(float);
    const int sms = num_sms();
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bp_sweep_kernel<K, NT, SG>, NT, smem) != cudaSuccess)
        return -1;
    const int tiles = (n + NT * K - 1) / (NT * K), room = sms * (per_sm > 0 ? per_sm : 1);
    return tiles < room ? tiles : room;
}

// one warp per CTA while the spins leave SM quarters with few warps (as bp_propagate)
static bool few(int n) { return n <= num_sms() * 4 * 32 * 2; }

extern "C" int bp_sweep_grid(int n, int seg_len, int spin_gradients) {
    if (n < 1 || seg_len < 0 || seg_len > SW_MAX) return -BP_E_ARG;
    const int g = spin_gradients ? (few(n) ? sweep_grid<1, 32, true>(n, seg_len) : sweep_grid<1, 128, true>(n, seg_len))
                                 : (few(n) ? sweep_grid<1, 32, false>(n, seg_len) : sweep_grid<2, 128, false>(n, seg_len));
    return g > 0 ? g : -BP_E_LAUNCH;
}

extern "C" int bp_sweep(const float* spins, int n, const void* segs, const double* seg64, const int* windows, int wa,
                        int wb, int seg0, int seg_len, const float* wstates, const int* wslot, float* chain,
                        int chain_in, const int* runs, int n_runs, const float* g0, const float* g1, float* lam,
                        float* gs, float* gseg, double* seg, int* status, void* stream) {
    if (n < 1 || wa < 0 || wb < wa || seg0 < 0 || seg_len < 0 || (gseg && seg_len > SW_MAX) || n_runs < 0) return BP_E_ARG;
    if (!spins || !segs || !seg64 || !windows || !wstates || !lam || !status || (g0 && !runs) || (gseg && !seg))
        return BP_E_ARG;
    if ((gs != nullptr) == (wslot != nullptr) || (wslot && !chain) || (gs && g0 && !g1)) return BP_E_ARG;
    if (wb == wa) return BP_OK;
    SweepArgs a{};
    a.spins = spins;
    a.segs = static_cast<const SegRec*>(segs), a.seg64 = reinterpret_cast<const double4*>(seg64);
    a.windows = reinterpret_cast<const int4*>(windows);
    a.n = n, a.wa = wa, a.wb = wb, a.seg0 = seg0, a.seg_len = seg_len;
    a.wstates = wstates, a.wslot = wslot, a.chain = chain, a.chain_in = chain_in;
    a.runs = reinterpret_cast<const int4*>(runs), a.n_runs = n_runs;
    a.g0 = reinterpret_cast<const float2*>(g0), a.g1 = reinterpret_cast<const float2*>(g1);
    a.lam = lam, a.gs = gs, a.gseg = gseg, a.status = status;
    const int grid = bp_sweep_grid(n, gseg ? seg_len : 0, gs != nullptr);
    if (grid < 1) return BP_E_LAUNCH;
    const size_t smem = gseg ? (size_t)2 * seg_len * sizeof(float) : 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (gs) {
        if (few(n))
            bp_sweep_kernel<1, 32, true><<<grid, 32, smem, st>>>(a);
        else
            bp_sweep_kernel<1, 128, true><<<grid, 128, smem, st>>>(a);
    } else {
        if (few(n))
            bp_sweep_kernel<1, 32, false><<<grid, 32, smem, st>>>(a);
        else
            bp_sweep_kernel<2, 128, false><<<grid, 128, smem, st>>>(a);
    }
    if (cudaGetLastError() != cudaSuccess) return BP_E_LAUNCH;
    if (gseg && seg_len > 0) {
        bp_sweep_reduce_kernel<<<(2 * seg_len + 31) / 32, dim3(32, 16), 0, st>>>(gseg, grid, seg_len, seg0, seg);
        if (cudaGetLastError() != cudaSuccess) return BP_E_LAUNCH;
    }
    return BP_OK;
}
