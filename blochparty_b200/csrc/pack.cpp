// Host side of packing a case (blochparty_b200/engine.py): the segment records and flags in one pass over a sequence,
// and the spins' buffers converted by several threads into page-locked staging, each block copied to the device as soon
// as it is ready. Replaces the reference's packing in Python (engines/gpu/driver.py:291-440): what was numpy and torch
// here read every input several times on one core and copied from pageable memory (1,048,576 spins with 8 coils: 42 ms
// of conversions and 11 ms of copies).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <limits>
#include <thread>
#include <vector>

#include "../../include/blochparty_b200.h"

namespace {

constexpr double kTwoPi = 6.283185307179586;  // as Python's 2 * math.pi

enum { RF = 1, ADC = 2, SPOIL = 4, SAME_FREE = 8, SAME_RFDT = 16, SAME_OFF = 32, SMALL = 64 };

struct Record {
    float dt, wx, wy, kx, ky, kz, beta;
    int32_t flags;
};

// f(begin, end) over [0, n) on up to `most` threads (this one among them), at least `least` items each.
template <class F>
void parallel(int64_t n, int64_t least, int most, F f) {
    const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
    const int t = (int)std::max<int64_t>(1, std::min<int64_t>({(int64_t)cores, (int64_t)most, n / least}));
    std::vector<std::thread> extra;
    extra.reserve(t);
    for (int i = 1; i < t; ++i) {
        try {
            extra.emplace_back(f, n * i / t, n * (i + 1) / t);
        } catch (...) {  // no more threads: this one does the share
            f(n * i / t, n * (i + 1) / t);
        }
    }
    f((int64_t)0, n / t);
    for (auto& x : extra) x.join();
}

// The remainder with the sign of the divisor (Python's %), for a positive divisor.
inline double wrapped(double x, double period) {
    double r = std::fmod(x, period);
    if (r != 0.0) {
        if (r < 0.0) r += period;
    } else {
        r = 0.0;
    }
    return r;
}

inline double value(const void* p, int wide, int64_t i) {
    return wide ? static_cast<const double*>(p)[i] : (double)static_cast<const float*>(p)[i];
}

}  // namespace

extern "C" int bp_pack_segments(const double* dt, const double* rf, const double* grad, const double* b0,
                                const double* phase, const uint8_t* is_rf, const uint8_t* adc, const uint8_t* spoil,
                                int64_t n, const float* extent, void* records, double* seg64, int32_t* flags,
                                double* psi, int64_t* n_adc) {
    if (n < 0 || !n_adc || (n > 0 && (!dt || !rf || !grad || !phase || !is_rf || !adc || !spoil || !records || !seg64 ||
                                      !flags || !psi)))
        return BP_E_ARG;
    try {
    Record* rec = static_cast<Record*>(records);
    parallel(n, 1 << 13, 16, [&](int64_t a, int64_t b) {
        for (int64_t s = a; s < b; ++s) {
            const double w = -kTwoPi * dt[s], beta = (b0 ? b0[s] : 0.0) * dt[s];
            const double k[3] = {grad[3 * s] * dt[s], grad[3 * s + 1] * dt[s], grad[3 * s + 2] * dt[s]};
            Record& r = rec[s];
            r.dt = (float)dt[s];
            r.wx = (float)(w * rf[2 * s]), r.wy = (float)(w * rf[2 * s + 1]);
            r.kx = (float)k[0], r.ky = (float)k[1], r.kz = (float)k[2], r.beta = (float)beta;
            seg64[4 * s] = k[0], seg64[4 * s + 1] = k[1], seg64[4 * s + 2] = k[2], seg64[4 * s + 3] = beta;
            r.flags = (is_rf[s] ? RF : 0) | (adc[s] ? ADC : 0) | (spoil[s] ? SPOIL : 0);
        }
    });
    // what a segment shares with the one before it, and whether its rotation is small for every spin: extent holds the
    // largest |x| |y| |z| pd r1 r2 |dB0| |b1| (NULL: not marked)
    parallel(n, 1 << 13, 16, [&](int64_t a, int64_t b) {
        for (int64_t s = a; s < b; ++s) {
            Record& r = rec[s];
            int32_t f = r.flags & (RF | ADC | SPOIL);
            if (s > 0) {
                const Record& q = rec[s - 1];
                const double *u = seg64 + 4 * s, *v = u - 4;
                const bool rf0 = is_rf[s - 1] != 0, rf1 = is_rf[s] != 0, same_dt = r.dt == q.dt;
                if (!rf0 && !rf1 && same_dt && u[0] == v[0] && u[1] == v[1] && u[2] == v[2] && u[3] == v[3])
                    f |= SAME_FREE;
                if (rf0 && rf1 && same_dt) {
                    f |= SAME_RFDT;
                    if (r.kx == q.kx && r.ky == q.ky && r.kz == q.kz && r.beta == q.beta) f |= SAME_OFF;
                }
            }
            if (extent && (f & RF)) {
                const double wz = kTwoPi * (std::fabs((double)r.kx) * extent[0] + std::fabs((double)r.ky) * extent[1] +
                                            std::fabs((double)r.kz) * extent[2] + std::fabs((double)r.dt) * extent[6] +
                                            std::fabs((double)r.beta));
                const double b1 = extent[7], wx = r.wx, wy = r.wy;
                if (b1 * b1 * (wx * wx + wy * wy) + wz * wz < 0.0624) f |= SMALL;
            }
            flags[s] = f;
        }
    });
    int64_t rows = 0;
    for (int64_t s = 0; s < n; ++s) {
        rec[s].flags = flags[s];
        if (adc[s]) psi[rows++] = wrapped(phase[s], kTwoPi);
    }
    *n_adc = rows;
    return BP_OK;
    } catch (...) {  // (out of host memory: no exception leaves the library)
        return BP_E_SIZE;
    }
}

extern "C" int64_t bp_pack_spins_staging(int64_t n, int n_coils) {
    // one block per thread: 8 rows of the spins, 2C of the coils, 6 of the state
    const int64_t block = std::min<int64_t>(n, BP_PACK_BLOCK), blocks = (n + BP_PACK_BLOCK - 1) / BP_PACK_BLOCK;
    const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
    const int64_t threads = std::max<int64_t>(1, std::min<int64_t>({blocks, (int64_t)cores, 16}));
    return threads * (14 + 2 * (int64_t)n_coils) * block * (int64_t)sizeof(float);
}

extern "C" int bp_pack_spins(const BpHostSpins* in, int64_t n, int n_coils, float* spins, float* sens, float* state,
                             float* extent, void* staging, int64_t staging_bytes, void* stream) {
    if (!in || n < 1 || n_coils < 1 || n_coils > BP_MAX_COILS || !spins || !sens || !staging) return BP_E_ARG;
    if (!in->pos || !in->pd || !in->t1 || !in->t2 || !in->db0 || !in->coils) return BP_E_ARG;
    const int64_t block = std::min<int64_t>(n, BP_PACK_BLOCK), blocks = (n + BP_PACK_BLOCK - 1) / BP_PACK_BLOCK;
    const int64_t slot = (14 + 2 * (int64_t)n_coils) * block;
    const int64_t threads =
        std::max<int64_t>(1, std::min<int64_t>({blocks, staging_bytes / (slot * (int64_t)sizeof(float)), 16}));
    if (slot * (int64_t)sizeof(float) > staging_bytes) return BP_E_SIZE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return BP_E_LAUNCH;
    const int rows_padded = 16 * ((n_coils + 7) / 8);
    if (rows_padded > 2 * n_coils &&
        cudaMemsetAsync(sens + (size_t)2 * n_coils * n, 0, (size_t)(rows_padded - 2 * n_coils) * n * sizeof(float), st) !=
            cudaSuccess)
        return BP_E_LAUNCH;
    try {
    std::atomic<int64_t> next{0};
    std::atomic<int> code{BP_OK};
    std::vector<float> most(threads * 8, 0.0f);
    auto work = [&](int64_t t, int64_t) {
        float* base = static_cast<float*>(staging) + t * slot;
        float* ext = most.data() + 8 * t;
        cudaEvent_t done;
        if (cudaSetDevice(dev) != cudaSuccess || cudaEventCreateWithFlags(&done, cudaEventDisableTiming) != cudaSuccess) {
            code = BP_E_LAUNCH;
            return;
        }
        for (int64_t b; (b = next.fetch_add(1)) < blocks && code == BP_OK;) {
            const int64_t j0 = b * BP_PACK_BLOCK, m = std::min<int64_t>(BP_PACK_BLOCK, n - j0);
            float *sp = base, *co = base + 8 * m, *sv = co + 2 * (int64_t)n_coils * m;
            for (int64_t j = 0; j < m; ++j) {
                const int64_t i = j0 + j;
                sp[j] = (float)value(in->pos, in->wide[0], 3 * i);
                sp[m + j] = (float)value(in->pos, in->wide[0], 3 * i + 1);
                sp[2 * m + j] = (float)value(in->pos, in->wide[0], 3 * i + 2);
            }
            for (int64_t j = 0; j < m; ++j) sp[3 * m + j] = (float)value(in->pd, in->wide[1], j0 + j);
            for (int64_t j = 0; j < m; ++j) sp[4 * m + j] = (float)(1.0 / value(in->t1, in->wide[2], j0 + j));
            for (int64_t j = 0; j < m; ++j) sp[5 * m + j] = (float)(1.0 / value(in->t2, in->wide[3], j0 + j));
            for (int64_t j = 0; j < m; ++j) sp[6 * m + j] = (float)value(in->db0, in->wide[4], j0 + j);
            for (int64_t j = 0; j < m; ++j) sp[7 * m + j] = in->b1 ? (float)value(in->b1, in->wide[5], j0 + j) : 1.0f;
            for (int64_t j = 0; j < m; ++j)  // [spin][2C] -> [2C][spin], a block that stays in the cache
                for (int c = 0; c < 2 * n_coils; ++c)
                    co[c * m + j] = (float)value(in->coils, in->wide[6], (j0 + j) * 2 * n_coils + c);
            for (int r = 0; r < 8; ++r)  // (a NaN stays: no bound holds)
                for (int64_t j = 0; j < m && ext[r] == ext[r]; ++j) {
                    const float v = std::fabs(sp[r * m + j]);
                    if (!(v <= ext[r])) ext[r] = v;
                }
            auto copy = [&](float* dst, const float* src, int rows) {
                if (cudaMemcpy2DAsync(dst + j0, (size_t)n * sizeof(float), src, (size_t)m * sizeof(float),
                                      (size_t)m * sizeof(float), (size_t)rows, cudaMemcpyHostToDevice, st) != cudaSuccess)
                    code = BP_E_LAUNCH;
            };
            copy(spins, sp, 8);
            copy(sens, co, 2 * n_coils);
            if (state) {  // m0 in a float32 high part and its float32 remainder
                for (int c = 0; c < 3; ++c)
                    for (int64_t j = 0; j < m; ++j) {
                        const double v = in->m0   ? value(in->m0, in->wide[7], 3 * (j0 + j) + c)
                                         : c == 2 ? value(in->pd, in->wide[1], j0 + j)
                                                  : 0.0;
                        const float hi = (float)v;
                        sv[c * m + j] = hi;
                        sv[(3 + c) * m + j] = (float)(v - (double)hi);
                    }
                copy(state, sv, 6);
            }
            // the block's copies end before its staging is written again, or given back
            if (cudaEventRecord(done, st) != cudaSuccess || cudaEventSynchronize(done) != cudaSuccess) code = BP_E_LAUNCH;
        }
        cudaEventDestroy(done);
    };
    std::vector<std::thread> extra;
    extra.reserve(threads);
    for (int64_t t = 1; t < threads; ++t) {
        try {
            extra.emplace_back(work, t, 0);
        } catch (...) {
            break;  // fewer threads: the others take the blocks
        }
    }
    work(0, 0);
    for (auto& x : extra) x.join();
    if (extent) {
        for (int r = 0; r < 8; ++r) {
            extent[r] = 0.0f;
            for (int64_t t = 0; t < threads && extent[r] == extent[r]; ++t) {
                const float v = most[8 * t + r];
                if (!(v <= extent[r])) extent[r] = v;
            }
        }
    }
    return code;
    } catch (...) {
        return BP_E_SIZE;
    }
}
