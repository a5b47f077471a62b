// K spins per thread as packed float32: K = 2 runs on the paired instructions of sm_100 (two float32 operations each,
// each rounded as one), K = 1 on the plain ones. The operations are the explicit round-to-nearest ones, so both give
// the same bits for a spin.
#pragma once
#include <cuda_runtime.h>

#include "bloch_common.cuh"

template <int K>
struct Pk;

template <>
struct Pk<1> {
    float f;
    __device__ __forceinline__ float get(int) const { return f; }
    __device__ __forceinline__ void set(int, float x) { f = x; }
};

// (the pair as one 64-bit register, so that the paired instructions need no moves around them)
template <>
struct Pk<2> {
    unsigned long long u;
    __device__ __forceinline__ float get(int k) const {
        float a, b;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(u));
        return k ? b : a;
    }
    __device__ __forceinline__ void set(int k, float x) {
        float a, b;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(u));
        if (k) b = x;
        else a = x;
        asm("mov.b64 %0, {%1, %2};" : "=l"(u) : "f"(a), "f"(b));
    }
};

__device__ __forceinline__ Pk<1> pfma(const Pk<1>& a, const Pk<1>& b, const Pk<1>& c) {
    return Pk<1>{__fmaf_rn(a.f, b.f, c.f)};
}
__device__ __forceinline__ Pk<1> pmul(const Pk<1>& a, const Pk<1>& b) { return Pk<1>{__fmul_rn(a.f, b.f)}; }
__device__ __forceinline__ Pk<1> padd(const Pk<1>& a, const Pk<1>& b) { return Pk<1>{__fadd_rn(a.f, b.f)}; }
__device__ __forceinline__ Pk<1> psub(const Pk<1>& a, const Pk<1>& b) { return Pk<1>{__fsub_rn(a.f, b.f)}; }
__device__ __forceinline__ Pk<2> pfma(const Pk<2>& a, const Pk<2>& b, const Pk<2>& c) {
    Pk<2> r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.u) : "l"(a.u), "l"(b.u), "l"(c.u));
    return r;
}
__device__ __forceinline__ Pk<2> pmul(const Pk<2>& a, const Pk<2>& b) {
    Pk<2> r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
    return r;
}
__device__ __forceinline__ Pk<2> padd(const Pk<2>& a, const Pk<2>& b) {
    Pk<2> r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
    return r;
}
template <int K>
__device__ __forceinline__ Pk<K> pset(float x);
template <>
__device__ __forceinline__ Pk<1> pset<1>(float x) {
    return Pk<1>{x};
}
template <>
__device__ __forceinline__ Pk<2> pset<2>(float x) {
    Pk<2> r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r.u) : "f"(x));
    return r;
}
__device__ __forceinline__ Pk<2> psub(const Pk<2>& a, const Pk<2>& b) {  // a - b, rounded once (b times -1 is exact)
    return pfma(b, pset<2>(-1.0f), a);
}
template <int K>
__device__ __forceinline__ Pk<K> pmake(const float* x) {
    Pk<K> r;
    if constexpr (K == 1)
        r.f = x[0];
    else
        asm("mov.b64 %0, {%1, %2};" : "=l"(r.u) : "f"(x[0]), "f"(x[1]));
    return r;
}

// hi + lo += d (d already holds lo): quick_two_sum's last steps.
template <int K>
__device__ __forceinline__ void quick_add(Pk<K>& hi, Pk<K>& lo, const Pk<K>& d) {
    const Pk<K> t = padd(hi, d);
    lo = psub(d, psub(t, hi));
    hi = t;
}

// A spin of the propagation: the coordinates its phase is formed from in float64 (exact copies of the float32 ones; a
// conversion takes the slow pipe and every free step would need four), the rest in float32.
struct PropSpin {
    double x, y, z, db0;
    float pd, r1, r2;
};

// expm1(x) of a relaxation for |x| <= 1/4: its Taylor series (the first term left out, x^7 / 7!, is below 4.9e-8 of x,
// under an ulp).
__device__ __forceinline__ float small_expm1(float x) {
    const float q = fmaf(x, fmaf(x, fmaf(x, fmaf(x, 1.0f / 720.0f, 1.0f / 120.0f), 1.0f / 24.0f), 1.0f / 6.0f), 0.5f);
    return fmaf(x * x, q, x);
}

__device__ __forceinline__ float relax_expm1(float x) { return fabsf(x) > 0.25f ? expm1f(x) : small_expm1(x); }

// What the steps of one RF run share, per spin: the half-step relaxation as RfRelax, the rotation about z.
template <int K>
struct RfRun {
    Pk<K> a1, a2, d1, d2, mpe, cz2;  // mpe = -pd expm1(-dt r1 / 2)
    Pk<K> wz, nwz, wz2;
};

template <int K>
__device__ __forceinline__ void rf_run_relax(RfRun<K>& r, float dt, const PropSpin* p) {
    float a1[K], a2[K], d1[K], d2[K], cz2[K], mpe[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const float e1h = relax_expm1(-0.5f * dt * p[k].r1), e2h = relax_expm1(-0.5f * dt * p[k].r2);
        a1[k] = 1.0f + e1h, a2[k] = 1.0f + e2h;
        d1[k] = e1h * (2.0f + e1h), d2[k] = e2h * (2.0f + e2h);
        cz2[k] = -(a1[k] + 1.0f) * p[k].pd * e1h;
        mpe[k] = -p[k].pd * e1h;
    }
    r.a1 = pmake<K>(a1), r.a2 = pmake<K>(a2), r.d1 = pmake<K>(d1), r.d2 = pmake<K>(d2), r.cz2 = pmake<K>(cz2);
    r.mpe = pmake<K>(mpe);
}

template <int K>
__device__ __forceinline__ void rf_run_offset(RfRun<K>& r, const SegRec& q, const PropSpin* p) {
    float wz[K], nwz[K], wz2[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        Spin s{};
        s.px = (float)p[k].x, s.py = (float)p[k].y, s.pz = (float)p[k].z, s.db0 = (float)p[k].db0;
        wz[k] = rf_wz(q, s);
        nwz[k] = -wz[k], wz2[k] = wz[k] * wz[k];
    }
    r.wz = pmake<K>(wz), r.nwz = pmake<K>(nwz), r.wz2 = pmake<K>(wz2);
}

template <int K>
struct State {
    Pk<K> x, y, z, lx, ly, lz;
};

// An RF segment (rf_step_wz's arithmetic, the increment's low part folded into its last multiply-adds): 49 packed
// operations for K spins. wx0, wy0: the record's RF, once per spin of the thread. SMALL: |w|^2 < 1/16 for every spin
// (the first tier of the Rodrigues factors, no tests).
template <bool SMALL, int K>
__device__ __forceinline__ void rf_step_packed(const Pk<K>& wx0, const Pk<K>& wy0, const Pk<K>& b1, const Pk<K>& nb1,
                                               const RfRun<K>& r, State<K>& m) {
    const Pk<K> wx = pmul(wx0, b1), wy = pmul(wy0, b1), nwx = pmul(wx0, nb1), nwy = pmul(wy0, nb1);
    const Pk<K> ux = pmul(m.x, r.a2), uy = pmul(m.y, r.a2), uz = pfma(m.z, r.a1, r.mpe);
    const Pk<K> p2 = pfma(wx, wx, pfma(wy, wy, r.wz2));
    Pk<K> s1, s2;
    if (SMALL) {
        s1 = pfma(p2, pfma(p2, pfma(p2, pset<K>(-1.9841269841269841e-04f), pset<K>(8.3333333333333333e-03f)),
                           pset<K>(-1.6666666666666667e-01f)), pset<K>(1.0f));
        s2 = pfma(p2, pfma(p2, pfma(p2, pset<K>(-2.4801587301587302e-05f), pset<K>(1.3888888888888889e-03f)),
                           pset<K>(-4.1666666666666667e-02f)), pset<K>(0.5f));
    } else {
        float a[K], b[K];
#pragma unroll
        for (int k = 0; k < K; ++k) rodrigues_coeffs(p2.get(k), a[k], b[k]);
        s1 = pmake<K>(a), s2 = pmake<K>(b);
    }
    const Pk<K> cx = pfma(wy, uz, pmul(r.nwz, uy)), cy = pfma(r.wz, ux, pmul(nwx, uz)), cz = pfma(wx, uy, pmul(nwy, ux));
    const Pk<K> dx = pfma(wy, cz, pmul(r.nwz, cy)), dy = pfma(r.wz, cx, pmul(nwx, cz)), dz = pfma(wx, cy, pmul(nwy, cx));
    const Pk<K> qx = pfma(s1, cx, pmul(s2, dx)), qy = pfma(s1, cy, pmul(s2, dy)), qz = pfma(s1, cz, pmul(s2, dz));
    quick_add(m.x, m.lx, pfma(r.a2, qx, pfma(r.d2, m.x, m.lx)));
    quick_add(m.y, m.ly, pfma(r.a2, qy, pfma(r.d2, m.y, m.ly)));
    quick_add(m.z, m.lz, pfma(r.a1, qz, pfma(r.d1, m.z, padd(m.lz, r.cz2))));
}

// The rotation by -2 pi t (t in turns, any size) as float-float pairs: c = ch + cl, s = sh + sl. t is reduced to a
// quarter turn and at most an eighth beside it, exactly; sine and cosine of the rest are their Taylor series in float64
// (|x| <= pi / 4: the first terms left out, x^17 / 17! and x^16 / 16!, are below 1.1e-15).
__device__ __forceinline__ void turn_factors(double t, float& ch, float& cl, float& sh, float& sl) {
    constexpr double kMagic = 6755399441055744.0;  // 1.5 x 2^52: adding it rounds to an integer in the low word
    const double tq = fma(t, 4.0, kMagic);
    const int quarter = __double2loint(tq);
    const double x = 6.283185307179586476925 * fma(tq - kMagic, -0.25, t);
    const double u = x * x;
    double s = fma(u, -1.0 / 1307674368000.0, 1.0 / 6227020800.0);
    s = fma(u, s, -1.0 / 39916800.0);
    s = fma(u, s, 1.0 / 362880.0);
    s = fma(u, s, -1.0 / 5040.0);
    s = fma(u, s, 1.0 / 120.0);
    s = fma(u, s, -1.0 / 6.0);
    s = fma(x * u, s, x);
    double c = fma(u, -1.0 / 87178291200.0, 1.0 / 479001600.0);
    c = fma(u, c, -1.0 / 3628800.0);
    c = fma(u, c, 1.0 / 40320.0);
    c = fma(u, c, -1.0 / 720.0);
    c = fma(u, c, 1.0 / 24.0);
    c = fma(u, c, -0.5);
    c = fma(u, c, 1.0);
    // each as a double whose low 29 bits are clear (a float32 value) and the rest
    const double c0 = __hiloint2double(__double2hiint(c), __double2loint(c) & 0xe0000000);
    const double s0 = __hiloint2double(__double2hiint(s), __double2loint(s) & 0xe0000000);
    const float a = (float)c0, al = (float)(c - c0), b = (float)s0, bl = (float)(s - s0);
    // cos and sin of -(quarter turns + x): the quarter swaps them and sets their signs
    const bool odd = quarter & 1;
    const unsigned cs = (unsigned)(quarter + 1) << 30 & 0x80000000u;  // cosine negative in quarters 1 and 2
    const unsigned ss = (unsigned)~quarter << 30 & 0x80000000u;       // minus sine negative in quarters 0 and 1
    ch = __uint_as_float(__float_as_uint(odd ? b : a) ^ cs), cl = __uint_as_float(__float_as_uint(odd ? bl : al) ^ cs);
    sh = __uint_as_float(__float_as_uint(odd ? a : b) ^ ss), sl = __uint_as_float(__float_as_uint(odd ? al : bl) ^ ss);
}

// The factors of `reps` copies of a free segment (free_factors_merged's quantities): the phase of all of them in
// float64, the relaxation over their duration t by its series, without branches (so that the factors of several steps
// overlap); finish_factors then replaces it where t r is too large for the series.
__device__ __forceinline__ FreeFactors start_factors(float dt, const double4& k64, const PropSpin& p, int reps,
                                                     float& t) {
    FreeFactors f;
    const double cyc = fma(k64.x, p.x, fma(k64.y, p.y, fma(k64.z, p.z, fma((double)dt, p.db0, k64.w))));
    turn_factors(cyc * (double)reps, f.ch, f.cl, f.sh, f.sl);
    t = __fmul_rn(dt, (float)reps);  // (one rounding: reps is small)
    f.e1 = small_expm1(-t * p.r1);
    f.e2 = small_expm1(-t * p.r2);
    return f;
}

__device__ __forceinline__ void finish_factors(FreeFactors& f, const PropSpin& p, float t) {
    if (fmaxf(fabsf(t * p.r1), fabsf(t * p.r2)) > 0.25f) {
        f.e1 = relax_expm1(-t * p.r1);
        f.e2 = relax_expm1(-t * p.r2);
    }
}

__device__ __forceinline__ FreeFactors prop_factors(float dt, const double4& k64, const PropSpin& p, int reps) {
    float t;
    FreeFactors f = start_factors(dt, k64, p, reps, t);
    finish_factors(f, p, t);
    return f;
}

// hi + lo = a + b exactly (Knuth's two-sum).
template <int K>
__device__ __forceinline__ void pair_sum(const Pk<K>& a, const Pk<K>& b, Pk<K>& hi, Pk<K>& lo) {
    hi = padd(a, b);
    const Pk<K> bb = psub(hi, a);
    lo = padd(psub(a, psub(hi, bb)), psub(b, bb));
}

// (ah + al) c + (bh + bl) s in float-float, not renormalised (na: -ah's product is formed with the factor nc = -c, ns
// likewise: the exact remainders of the products without a negation).
template <int K>
__device__ __forceinline__ void ff_turn(const Pk<K>& ah, const Pk<K>& al, const Pk<K>& bh, const Pk<K>& bl,
                                        const Pk<K>& c, const Pk<K>& nc, const Pk<K>& cl, const Pk<K>& s,
                                        const Pk<K>& ns, const Pk<K>& sl, Pk<K>& hi, Pk<K>& lo) {
    const Pk<K> p = pmul(c, ah), q = pmul(s, bh);
    const Pk<K> pe = pfma(c, ah, pmul(nc, ah)), qe = pfma(s, bh, pmul(ns, bh));
    Pk<K> e;
    pair_sum(p, q, hi, e);
    lo = padd(e, padd(pe, qe));
    lo = padd(lo, pfma(c, al, pmul(s, bl)));
    lo = padd(lo, pfma(cl, ah, pmul(sl, bh)));
}

// A free step for K spins (free_step's arithmetic): the state rotated and relaxed in float-float. The transverse
// relaxation's increment never outgrows its component (e2 > -1), so the fast sum keeps it.
template <int K>
__device__ __forceinline__ void free_step_packed(const FreeFactors* f, const PropSpin* p, State<K>& m) {
    float ch[K], cl[K], sh[K], sl[K], e1[K], e2[K], nch[K], nsh[K], nsl[K], pd[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        ch[k] = f[k].ch, cl[k] = f[k].cl, sh[k] = f[k].sh, sl[k] = f[k].sl, e1[k] = f[k].e1, e2[k] = f[k].e2;
        nch[k] = -f[k].ch, nsh[k] = -f[k].sh, nsl[k] = -f[k].sl, pd[k] = p[k].pd;
    }
    const Pk<K> c = pmake<K>(ch), nc = pmake<K>(nch), c1 = pmake<K>(cl), s = pmake<K>(sh), ns = pmake<K>(nsh);
    Pk<K> xh, xl, yh, yl;
    ff_turn(m.x, m.lx, m.y, m.ly, c, nc, c1, ns, s, pmake<K>(nsl), xh, xl);  // c x - s y
    ff_turn(m.y, m.ly, m.x, m.lx, c, nc, c1, s, ns, pmake<K>(sl), yh, yl);   // c y + s x
    const Pk<K> r2 = pmake<K>(e2);
    m.x = xh, m.y = yh;
    quick_add(m.x, m.lx, pfma(xh, r2, xl));
    quick_add(m.y, m.ly, pfma(yh, r2, yl));
    const Pk<K> z = m.z, d = pfma(psub(z, pmake<K>(pd)), pmake<K>(e1), m.lz);
    pair_sum(z, d, m.z, m.lz);
}
