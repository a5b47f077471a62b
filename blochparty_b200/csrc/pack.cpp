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

// f(the array as its own type).
template <class F>
void typed(const void* p, int wide, F f) {
    if (wide)
        f(static_cast<const double*>(p));
    else
        f(static_cast<const float*>(p));
}

inline void convert(const void* p, int wide, int64_t at, int64_t m, float* to) {
    typed(p, wide, [&](auto* x) {
        for (int64_t j = 0; j < m; ++j) to[j] = (float)(double)x[at + j];
    });
}

inline void convert_rate(const void* p, int wide, int64_t at, int64_t m, float* to) {
    typed(p, wide, [&](auto* x) {
        for (int64_t j = 0; j < m; ++j) to[j] = (float)(1.0 / (double)x[at + j]);
    });
}

// rows [at, at + m) of an array of `width` columns into one run of m per column
inline void transpose(const void* p, int wide, int64_t at, int64_t m, int width, float* to) {
    typed(p, wide, [&](auto* x) {
        x += at * width;
        for (int c0 = 0; c0 < width; c0 += 8) {
            const int w = std::min(8, width - c0);
            if (w == 8) {
                for (int64_t j = 0; j < m; ++j)
                    for (int c = 0; c < 8; ++c) to[(c0 + c) * m + j] = (float)(double)x[j * width + c0 + c];
            } else {
                for (int64_t j = 0; j < m; ++j)
                    for (int c = 0; c < w; ++c) to[(c0 + c) * m + j] = (float)(double)x[j * width + c0 + c];
            }
        }
    });
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
        // what a segment shares with the one before it, and whether its rotation is small for every spin: extent holds
        // the largest |x| |y| |z| pd r1 r2 |dB0| |b1| (NULL: not marked)
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
                    const double wz =
                        kTwoPi * (std::fabs((double)r.kx) * extent[0] + std::fabs((double)r.ky) * extent[1] +
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

// Blocks of spins converted by threads of their own (0: by the caller, which then needs no other thread) and the blocks
// the staging holds. Up to four blocks (half a millisecond) new threads cost more than they save.
static int64_t pack_threads(int64_t blocks) {
    if (blocks <= 4) return 0;
    const unsigned cores = std::max(2u, std::thread::hardware_concurrency());
    return std::min<int64_t>({blocks / 2, (int64_t)cores - 1, 15});
}

static int64_t pack_slots(int64_t blocks) {
    const int64_t t = pack_threads(blocks);
    return t ? std::min(blocks, 2 * t) : std::max<int64_t>(blocks, 1);
}

extern "C" int64_t bp_pack_spins_staging(int64_t n, int n_coils) {
    // a block: 8 rows of the spins, 2C of the coils, 6 of the state
    const int64_t block = std::min<int64_t>(n, BP_PACK_BLOCK), blocks = (n + BP_PACK_BLOCK - 1) / BP_PACK_BLOCK;
    return pack_slots(blocks) * (14 + 2 * (int64_t)n_coils) * block * (int64_t)sizeof(float);
}

extern "C" int bp_pack_spins(const BpHostSpins* in, int64_t n, int n_coils, float* spins, float* sens, float* state,
                             float* extent, void* staging, int64_t staging_bytes, void* stream) {
    if (!in || n < 1 || n_coils < 1 || n_coils > BP_MAX_COILS || !spins || !sens || !staging) return BP_E_ARG;
    if (!in->pos || !in->pd || !in->t1 || !in->t2 || !in->db0 || !in->coils) return BP_E_ARG;
    if (staging_bytes < bp_pack_spins_staging(n, n_coils)) return BP_E_SIZE;
    const int64_t block = std::min<int64_t>(n, BP_PACK_BLOCK), blocks = (n + BP_PACK_BLOCK - 1) / BP_PACK_BLOCK;
    const int64_t slot = (14 + 2 * (int64_t)n_coils) * block, slots = pack_slots(blocks), threads = pack_threads(blocks);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int rows_padded = 16 * ((n_coils + 7) / 8);
    if (rows_padded > 2 * n_coils &&
        cudaMemsetAsync(sens + (size_t)2 * n_coils * n, 0, (size_t)(rows_padded - 2 * n_coils) * n * sizeof(float), st) !=
            cudaSuccess)
        return BP_E_LAUNCH;
    // block b of the spins into its slot; ext: the largest magnitudes so far, as bits (a NaN's are above every number's)
    auto fill = [&](int64_t b, uint32_t* ext) {
        const int64_t j0 = b * BP_PACK_BLOCK, m = std::min<int64_t>(BP_PACK_BLOCK, n - j0);
        float* sp = static_cast<float*>(staging) + (b % slots) * slot;
        float *co = sp + 8 * m, *sv = co + 2 * (int64_t)n_coils * m;
        transpose(in->pos, in->wide[0], j0, m, 3, sp);
        convert(in->pd, in->wide[1], j0, m, sp + 3 * m);
        convert_rate(in->t1, in->wide[2], j0, m, sp + 4 * m);
        convert_rate(in->t2, in->wide[3], j0, m, sp + 5 * m);
        convert(in->db0, in->wide[4], j0, m, sp + 6 * m);
        if (in->b1)
            convert(in->b1, in->wide[5], j0, m, sp + 7 * m);
        else
            std::fill(sp + 7 * m, sp + 8 * m, 1.0f);
        transpose(in->coils, in->wide[6], j0, m, 2 * n_coils, co);
        for (int r = 0; r < 8; ++r)
            for (int64_t j = 0; j < m; ++j) {
                uint32_t bits;
                std::memcpy(&bits, sp + r * m + j, 4);
                ext[r] = std::max(ext[r], bits & 0x7fffffffu);
            }
        if (!state) return;
        std::fill(sv, sv + 6 * m, 0.0f);  // m0 in a float32 high part and its float32 remainder
        typed(in->m0 ? in->m0 : in->pd, in->m0 ? in->wide[7] : in->wide[1], [&](auto* x) {
            for (int c = in->m0 ? 0 : 2; c < 3; ++c)
                for (int64_t j = 0; j < m; ++j) {
                    const double v = (double)(in->m0 ? x[3 * (j0 + j) + c] : x[j0 + j]);
                    const float hi = (float)v;
                    sv[c * m + j] = hi;
                    sv[(3 + c) * m + j] = (float)(v - (double)hi);
                }
        });
    };
    auto send = [&](int64_t b) {
        const int64_t j0 = b * BP_PACK_BLOCK, m = std::min<int64_t>(BP_PACK_BLOCK, n - j0);
        const float* sp = static_cast<const float*>(staging) + (b % slots) * slot;
        auto copy = [&](float* dst, const float* src, int rows) {
            return cudaMemcpy2DAsync(dst + j0, (size_t)n * sizeof(float), src, (size_t)m * sizeof(float),
                                     (size_t)m * sizeof(float), (size_t)rows, cudaMemcpyHostToDevice, st) == cudaSuccess;
        };
        return copy(spins, sp, 8) && copy(sens, sp + 8 * m, 2 * n_coils) &&
               (!state || copy(state, sp + (8 + 2 * (int64_t)n_coils) * m, 6));
    };
    uint32_t most[8] = {0};
    bool ok = true;
    if (threads == 0) {
        for (int64_t b = 0; b < blocks; ++b) {
            fill(b, most);
            ok = send(b) && ok;
        }
        ok = cudaStreamSynchronize(st) == cudaSuccess && ok;  // the staging is the caller's again
    } else {
        // workers convert blocks as they come, waiting for a slot whose copies have ended; this thread copies them in
        // order and gives the slots back
        try {
            std::vector<std::atomic<int>> full(blocks);
            for (auto& f : full) f.store(0);
            std::atomic<int64_t> next{0}, given{slots};  // blocks below `given` may be converted
            std::vector<uint32_t> tops(threads * 8, 0u);
            std::vector<cudaEvent_t> events;
            events.reserve(slots);
            for (int64_t i = 0; i < slots && ok; ++i) {
                cudaEvent_t e;
                ok = cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
                if (ok) events.push_back(e);
            }
            auto work = [&](int64_t t) {
                for (int64_t b; (b = next.fetch_add(1)) < blocks;) {
                    while (given.load(std::memory_order_acquire) <= b) std::this_thread::yield();
                    fill(b, tops.data() + 8 * t);
                    full[b].store(1, std::memory_order_release);
                }
            };
            std::vector<std::thread> workers;
            workers.reserve(threads);
            for (int64_t t = 0; t < threads && ok; ++t) {
                try {
                    workers.emplace_back(work, t);
                } catch (...) {
                    break;  // fewer of them
                }
            }
            if (workers.empty()) {  // none: this thread does their work, a slot's worth at a time
                for (int64_t b = 0; b < blocks && ok; ++b) {
                    fill(b, most);
                    ok = send(b) && cudaStreamSynchronize(st) == cudaSuccess;
                }
            } else {
                int64_t back = 0;  // blocks whose slots have been given back
                for (int64_t b = 0; b < blocks; ++b) {
                    while (!full[b].load(std::memory_order_acquire)) std::this_thread::yield();
                    if (ok) ok = send(b) && cudaEventRecord(events[b % slots], st) == cudaSuccess;
                    for (; back <= b - slots / 2; ++back) {  // (after a failure the workers still get through)
                        if (ok) ok = cudaEventSynchronize(events[back % slots]) == cudaSuccess;
                        given.store(slots + back + 1, std::memory_order_release);
                    }
                }
                for (auto& w : workers) w.join();
            }
            ok = cudaStreamSynchronize(st) == cudaSuccess && ok;
            for (auto& e : events) cudaEventDestroy(e);
            for (int64_t i = 0; i < 8 * threads; ++i) most[i % 8] = std::max(most[i % 8], tops[i]);
        } catch (...) {  // (out of host memory before any worker ran: no exception leaves the library)
            return BP_E_SIZE;
        }
    }
    if (extent) std::memcpy(extent, most, sizeof(most));
    return ok ? BP_OK : BP_E_LAUNCH;
}
