// Forward propagation (bp_propagate) and the coil sums of the samples it meets (bp_readout): float32 readout.
//
// Replaces blochparty's bloch_chunk / bloch_chunk_mma (engines/gpu/cuda/kernels.cu.in:2-185) for static spins
// with PD, T1, T2, dB0, B1+, receive coils and b0_offset (the V=0 variant), driven by
// engines/gpu/driver.py:_forward (:197-756).
//
// The two halves of a forward have nothing in common but one complex number per spin and run of samples, so they are
// two kernels with a workspace z [runs][n] between them:
//  * bp_propagate_kernel: tile-major and persistent. A CTA takes tiles of NT K spins, K per thread, keeps the tile's
//    state in registers from the first window to the last (the start state is read once and the end state written
//    once), and streams the segment records through shared memory by TMA, one window ahead. Where a run of samples
//    starts it writes the spin's first sample to z. K = 2 runs an RF segment's arithmetic on paired instructions
//    (packed.cuh): one spin per thread left the RF steps bound by instruction issue.
//  * bp_readout_kernel: a CTA takes 128 samples (four times 32 of one run) and a range of spins, forms the samples in
//    registers and contracts them with the coil sensitivities on the tensor cores (readout.cuh), its sums in
//    registers over the whole range; then one float64 atomic per (sample, coil, re/im).
// One kernel for both had to go window by window through all tiles (the accumulators of a whole sequence fit nowhere):
// per window and tile it loaded spins, state and sensitivities and stored the state, which took a third of the time at
// 12 to 16 warps per SM, and with few spins every sample's work lay on the chain of segments.
//
// Measured against that kernel (bp_forward, which is still the faster one for short runs of samples: the rule and both
// sides' times are in blochparty_b200/engine.py; one B200): 8,388,608 spins x 8 TRs of the 4-echo head scan 143.0 -> 79.9
// ms, 1,048,576 spins x 24 TRs of the slab 3D GRE 18.1 -> 11.7 ms, the 393,216-spin TSE 185 -> 114 ms, 4,096 spins x 264 TRs
// of the 64 x 64 GRE 3.23 -> 0.79 ms. RF steps now take 61 cycles per 32 spins and SM quarter (the FMA pipe alone 54); with
// few spins the chain of steps bounds it (about 3 us per TR).
//
// Free segments with one set of factors, all samples or none, are one step within a block of BP_ADJ_WIN segments (the
// cuts depend on the sequence alone), the state from the merged factors, whose phase is taken in float64.
// Demodulation by exp(-i adc_phase) is the same for every spin and is applied after the sum, in float64
// (bp_signal_finish).
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "packed.cuh"
#include "readout.cuh"
#include "../../include/blochparty_b200.h"

// A run of samples: its first segment, the segment whose factor separates its samples (-1: a single sample), samples,
// and the ADC row of the first.
// (host: blochparty_b200/engine.py sample_runs)

struct PropArgs {
    const float* spins;    // [8][n]: px py pz pd r1 r2 db0 b1
    const SegRec* segs;    // [S]
    const double4* seg64;  // [S]: kx ky kz beta in float64
    const int4* windows;   // [n_windows]: first segment, end segment, first ADC row, samples
    int n;
    int w_begin, w_end;
    float* state;          // [6][n]: mx my mz and their low parts
    float* wstates;        // null, or [slots][6][n]: state at window starts
    int wstate_stride;
    const int* wslot;      // null, or [n_windows]: the slot of wstates that takes window w's start state (-1: none)
    const int4* runs;      // [n_runs], by first segment
    int n_runs;
    float2* z;             // [runs in the windows][n]: the first sample of every run, or null: no readout
    int z_cap;             // runs z holds
    int clip;              // BP_CLIP_BEGIN: a run the first window starts inside of begins there
    int* status;
};

// The first of [0, n) for which `before` does not hold (it holds up to there), by a warp: 32 probes a step.
template <class F>
__device__ __forceinline__ int warp_bound(int n, int lane, F before) {
    int lo = 0, len = n;
    while (len > 0) {
        const int step = (len + 31) / 32, i = lo + lane * step;
        const int k = __popc(__ballot_sync(0xffffffffu, i < lo + len && before(i)));
        if (k == 0) break;
        const int end = min(lo + k * step, lo + len);
        lo += (k - 1) * step + 1;
        len = end - lo;
    }
    return lo;
}

// The first run of windows that start at segment s: the first that starts there or later, or with BP_CLIP_BEGIN that
// ends after s. (warp)
__device__ __forceinline__ int windows_run(const int4* __restrict__ runs, int n_runs, int s, int clip, int lane) {
    return warp_bound(n_runs, lane, [&](int i) {
        const int4 r = runs[i];
        return r.x + ((clip & BP_CLIP_BEGIN) ? r.z - 1 : 0) < s;
    });
}

// The kernel's list of a chunk's steps: a first segment, its length, and what it is.
#define ST_LEN(e) (((e) >> 10) & 1023)
#define ST_SEG(e) ((e) & 1023)
#define ST_FREE (1 << 20)   // a piece of free segments (else RF)
#define ST_SMALL (1 << 21)  // RF: every step a small rotation (BP_SMALL)
#define ST_SAVE (1 << 22)   // the state at its start is saved

// HELP: steps whose factors are formed ahead. Eight left the first warp waiting longer at a chunk's start: 0.767 -> 0.735
// ms for 4,096 spins x 264 TRs (six 0.740), 0.434 -> 0.419 for 9,025 x 115; the same where help is off.
#define ST_BATCH 4

template <int CH, bool HELP>
__host__ __device__ constexpr size_t prop_smem() {
    return (size_t)CH * (2 * (sizeof(SegRec) + sizeof(double4)) + sizeof(float4) + 2 * sizeof(int)) +
           2 * sizeof(uint64_t) + (HELP ? 2 * ST_BATCH * 6 * 32 * sizeof(float) : 0);
}

// K: spins per thread; NT: threads per CTA; CH: segments per chunk (a multiple of 32). HELP: the CTA's first warp alone
// has spins (32), and the others form the factors of its next free steps: with few spins the chain of steps is the time,
// and the factors (about 350 of a step's 700 cycles, in float64) do not depend on the state.
template <int K, int NT, int CH, bool HELP>
__global__ void __launch_bounds__(NT, NT == 32 ? 8 : HELP ? 5 : 4) bp_propagate_kernel(PropArgs a) {
    static_assert(!HELP || (K == 1 && NT > 32), "helping warps");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    static_assert(CH % 32 == 0 && CH <= 512, "chunks are whole blocks of 32 segments");
    SegRec* segbuf = reinterpret_cast<SegRec*>(smem_raw);         // [2][CH]
    double4* k64buf = reinterpret_cast<double4*>(segbuf + 2 * CH);  // [2][CH]
    float4* rfx = reinterpret_cast<float4*>(k64buf + 2 * CH);     // [CH]: wx0, wx0, wy0, wy0
    int* list = reinterpret_cast<int*>(rfx + CH);                 // [CH]: the chunk's steps
    int* slots = list + CH;                                       // [CH]: the slot that takes the state at a segment
    uint64_t* bars = reinterpret_cast<uint64_t*>(slots + CH);
    float* ring = reinterpret_cast<float*>(bars + 2);             // HELP: [2][ST_BATCH][6][32] factors
    __shared__ int count[NT / 32 + 1];
    __shared__ int windows_in[2];  // windows that start in a chunk, by the chunk's parity
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = a.n;
    constexpr int TILE = (HELP ? 32 : NT) * K;
    const int n_tiles = (n + TILE - 1) / TILE;
    const int s_begin = a.windows[a.w_begin].x, s_end = a.windows[a.w_end - 1].y;
    if (s_begin < 0 || s_end < s_begin) {  // (uniform)
        if (tid == 0) atomicOr(a.status, BP_ERR_BAD_WINDOW);
        return;
    }
    if (s_end == s_begin) return;
    auto chunk_end = [&](int c) { return min(s_end, c - (c & 31) + CH); };  // chunks end at multiples of 32

    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
        windows_in[0] = windows_in[1] = 0;
    }
    __syncthreads();
    auto issue = [&](int c, int buf) {
        const uint32_t bytes = static_cast<uint32_t>(chunk_end(c) - c) * sizeof(SegRec);
        static_assert(sizeof(SegRec) == sizeof(double4), "one size for both copies");
        fence_proxy_async_smem();
        mbar_expect_tx(&bars[buf], 2 * bytes);
        tma_load_1d(segbuf + buf * CH, a.segs + c, bytes, &bars[buf]);
        tma_load_1d(k64buf + buf * CH, a.seg64 + c, bytes, &bars[buf]);
    };
    if (tid == 0 && (int)blockIdx.x < n_tiles) issue(s_begin, 0);
    const int run_lo = a.z ? windows_run(a.runs, a.n_runs, s_begin, a.clip, lane) : 0;

    int it = 0;  // chunks staged so far (buffer it & 1, its phase (it >> 1) & 1)
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        // the tile's spins (K per thread, 32 apart) and state
        PropSpin p[K];
        State<K> m;
        int jk[K];
        bool active[K];
        float v[6][K], bp[K], bn[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int j0 = tile * TILE + ((HELP ? 0 : warp) * K + k) * 32 + lane;
            active[k] = j0 < n;
            jk[k] = active[k] ? j0 : 0;
            const Spin s = load_spin(a.spins, n, jk[k], active[k]);
            p[k] = PropSpin{(double)s.px, (double)s.py, (double)s.pz, (double)s.db0, s.pd, s.r1, s.r2};
            bp[k] = s.b1, bn[k] = -s.b1;
#pragma unroll
            for (int i = 0; i < 6; ++i) v[i][k] = active[k] ? a.state[(size_t)i * n + jk[k]] : 0.0f;
        }
        m.x = pmake<K>(v[0]), m.y = pmake<K>(v[1]), m.z = pmake<K>(v[2]);
        m.lx = pmake<K>(v[3]), m.ly = pmake<K>(v[4]), m.lz = pmake<K>(v[5]);
        const Pk<K> b1 = pmake<K>(bp), nb1 = pmake<K>(bn);
        auto store_state = [&](float* dst) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                if (!active[k]) continue;
                float* st = dst + jk[k];
                st[0] = m.x.get(k), st[(size_t)n] = m.y.get(k), st[2 * (size_t)n] = m.z.get(k);
                st[3 * (size_t)n] = m.lx.get(k), st[4 * (size_t)n] = m.ly.get(k), st[5 * (size_t)n] = m.lz.get(k);
            }
        };
        int run = run_lo, next = 0x7fffffff;  // the next run and its first segment
        auto next_run = [&](int r) {
            run = r;
            next = a.z && r < a.n_runs && r - run_lo < a.z_cap ? max(a.runs[r].x, s_begin) : 0x7fffffff;
        };
        next_run(run_lo);
        auto write_z = [&](const float2* z) {
            float2* dst = a.z + (size_t)(run - run_lo) * n;
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (active[k]) dst[jk[k]] = z[k];
            next_run(run + 1);
        };
        auto sample = [&](float2* z) {
#pragma unroll
            for (int k = 0; k < K; ++k) z[k] = make_float2(m.x.get(k) + m.lx.get(k), m.y.get(k) + m.ly.get(k));
        };

        int w_at = a.w_begin;  // the first window that starts in the chunk or after it (with wstates)
        RfRun<K> rr;
        for (int c = s_begin; c < s_end; ++it) {
            const int buf = it & 1, c_end = chunk_end(c), nseg = c_end - c;
            const bool ok = mbar_wait_bounded(&bars[buf], (it >> 1) & 1);
            const SegRec* q0 = segbuf + buf * CH;
            const double4* k0 = k64buf + buf * CH;
            if (__syncthreads_or(!ok)) {  // (and every thread is done with the chunk before this one)
                if (tid == 0) atomicOr(a.status, BP_ERR_TMA_TIMEOUT);
                return;
            }
            if (tid == 0) {  // the next chunk, of this tile or the next one, after the check: nothing left in flight
                windows_in[(it + 1) & 1] = 0;  // (every thread has read the chunk before's, which the next one takes)
                if (c_end < s_end)
                    issue(c_end, buf ^ 1);
                else if (tile + (int)gridDim.x < n_tiles)
                    issue(s_begin, buf ^ 1);
            }
            if (a.wstates) {  // the segments whose state is saved
                for (int s = tid; s < nseg; s += NT) slots[s] = -1;
                __syncthreads();
                for (int w = w_at + tid; w < a.w_end; w += NT) {
                    const int x = a.windows[w].x - c;
                    if (x >= nseg) break;
                    const int i = w - a.w_begin;
                    if (x >= 0)
                        slots[x] = a.wslot ? a.wslot[w] : (i % a.wstate_stride) == 0 ? i / a.wstate_stride : -1;
                    atomicAdd(&windows_in[it & 1], 1);
                }
                __syncthreads();
            }
            // the chunk's steps: runs of RF segments that differ in the RF alone, all small rotations or not, without
            // samples or spoils (or one RF segment with them); and free pieces: the factors of the first, all samples
            // or none, a spoil at most on the last, within a block of BP_ADJ_WIN segments. Both start where a state
            // is saved. Every thread decides whether its segment starts one; the starts are compacted in order
            int steps = 0;
            for (int s0 = 0; s0 < nseg; s0 += NT) {
                const int s = s0 + tid;
                bool start = false;
                int kind = 0;
                if (s < nseg) {
                    const int f = q0[s].flags, g = s > 0 ? q0[s - 1].flags : 0;
                    rfx[s] = make_float4(q0[s].wx0, q0[s].wx0, q0[s].wy0, q0[s].wy0);
                    constexpr int kSame = BP_RF | BP_SAME_RFDT | BP_SAME_OFF;
                    if (f & BP_RF)
                        start = s == 0 || !(g & BP_RF) || (f & kSame) != kSame || ((f | g) & (BP_ADC | BP_SPOIL)) ||
                                ((f ^ g) & BP_SMALL);
                    else
                        start = s == 0 || (g & (BP_RF | BP_SPOIL)) || !(f & BP_SAME_FREE) || ((f ^ g) & BP_ADC) ||
                                ((c + s) & (BP_ADJ_WIN - 1)) == 0;
                    kind = (f & BP_RF) ? ((f & BP_SMALL) ? ST_SMALL : 0) : ST_FREE;
                    if (a.wstates && slots[s] >= 0) start = true, kind |= ST_SAVE;
                }
                const unsigned starts = __ballot_sync(0xffffffffu, start);
                int at = steps;
                if (NT > 32) {
                    if (lane == 0) count[warp] = __popc(starts);
                    __syncthreads();
#pragma unroll
                    for (int w = 0; w < NT / 32; ++w) {
                        if (w < warp) at += count[w];
                        steps += count[w];
                    }
                    __syncthreads();
                } else {
                    steps += __popc(starts);
                }
                if (start) list[at + __popc(starts & ((1u << lane) - 1u))] = s | kind;
            }
            __syncthreads();
            if (a.wstates) w_at += windows_in[it & 1];
            // a step ends where the next one starts
            auto entry = [&](int i) {
                const int e = list[i], to = i + 1 < steps ? ST_SEG(list[i + 1]) : nseg;
                return e | (to - ST_SEG(e)) << 10;
            };

            // HELP: the factors of steps [b0, b0 + ST_BATCH) into one half of the ring, by every warp but the first
            auto form = [&](int b0) {
                if (warp == 0) return;
                for (int i = b0 + warp - 1; i < min(b0 + ST_BATCH, steps); i += NT / 32 - 1) {
                    const int e = entry(i);
                    if (!(e & ST_FREE)) continue;
                    const FreeFactors f = prop_factors(q0[ST_SEG(e)].dt, k0[ST_SEG(e)], p[0], ST_LEN(e));
                    float* r = ring + (i % (2 * ST_BATCH)) * 6 * 32 + lane;
                    r[0] = f.ch, r[32] = f.cl, r[64] = f.sh, r[96] = f.sl, r[128] = f.e1, r[160] = f.e2;
                }
            };
            auto take = [&](int i) {  // step i
                const int e = entry(i), s = ST_SEG(e), len = ST_LEN(e), f = q0[s].flags;
                if (e & ST_SAVE) store_state(a.wstates + (size_t)slots[s] * 6 * n);
                if (!(e & ST_FREE)) {
                    if (s == 0 || !(f & BP_SAME_RFDT)) rf_run_relax(rr, q0[s].dt, p);
                    if (s == 0 || !(f & BP_SAME_OFF)) rf_run_offset(rr, q0[s], p);
                    auto step = [&](int t, auto tag) {
                        Pk<K> wx0, wy0;
                        if constexpr (K == 1) {
                            wx0.f = rfx[t].x, wy0.f = rfx[t].z;
                        } else {
                            const ulonglong2 w2 = *reinterpret_cast<const ulonglong2*>(rfx + t);
                            wx0.u = w2.x, wy0.u = w2.y;
                        }
                        rf_step_packed<decltype(tag)::value>(wx0, wy0, b1, nb1, rr, m);
                    };
                    if (e & ST_SMALL) {
#pragma unroll 4
                        for (int t = s; t < s + len; ++t) step(t, std::true_type{});
                    } else {
#pragma unroll 1
                        for (int t = s; t < s + len; ++t) step(t, std::false_type{});
                    }
                    if (f & (BP_ADC | BP_SPOIL)) {  // (a single step)
                        if ((f & BP_ADC) && c + s == next) {
                            float2 z[K];
                            sample(z);
                            write_z(z);
                        }
                        if (f & BP_SPOIL) m.x = m.y = m.lx = m.ly = pset<K>(0.0f);
                    }
                    return;
                }
                FreeFactors ff[K];
                if constexpr (HELP) {
                    const float* r = ring + (i % (2 * ST_BATCH)) * 6 * 32 + lane;
                    ff[0] = FreeFactors{r[0], r[32], r[64], r[96], r[128], r[160]};
                } else {
#pragma unroll
                    for (int k = 0; k < K; ++k) ff[k] = prop_factors(q0[s].dt, k0[s], p[k], len);
                }
                const bool starts = (f & BP_ADC) && c + s == next;  // a run's first sample
                float2 z[K];
                if (starts && len > 1) {
                    sample(z);
#pragma unroll
                    for (int k = 0; k < K; ++k)
                        readout_advance(prop_factors(q0[s].dt, k0[s], p[k], 1), z[k].x, z[k].y);
                }
                free_step_packed(ff, p, m);
                if (starts) {
                    if (len == 1) sample(z);
                    write_z(z);
                }
                if (q0[s + len - 1].flags & BP_SPOIL) m.x = m.y = m.lx = m.ly = pset<K>(0.0f);
            };
            if constexpr (HELP) {  // the first warp a batch behind the others
                form(0);
                __syncthreads();
                for (int b0 = 0; b0 < steps; b0 += ST_BATCH) {
                    form(b0 + ST_BATCH);
                    if (warp == 0)
                        for (int i = b0; i < min(b0 + ST_BATCH, steps); ++i) take(i);
                    __syncthreads();
                }
            } else {
                for (int i = 0; i < steps; ++i) take(i);
            }
            c = c_end;
        }
        if (!HELP || warp == 0) store_state(a.state);
    }
}

// ---- the coil sums ----
#define RO_THREADS 128
#define RO_WARPS (RO_THREADS / 32)
#define RO_SUBS 4          // blocks of 32 samples per CTA
#define RO_WARP_BYTES (RO_SUBS * 32 * 16 * 4)  // a warp's shared memory: its operands, then its sums
#define RO_FETCH 21        // float rows fetched per group of 32 spins: 16 sensitivities, x y z r2 db0

// One float per lane from global to shared memory, asynchronously (zero where there is none).
__device__ __forceinline__ void fetch4(void* dst, const void* src, bool there) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(there ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void fetch8(void* dst, const void* src, bool there) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(there ? 8 : 0)
                 : "memory");
}

struct ReadArgs {
    const float* spins;
    const float* sens;     // [16 ncg][n]: coil c real at row 2c, imaginary at 2c + 1, zero rows to pad
    const SegRec* segs;
    const double4* seg64;
    const int4* windows;
    int n, n_coils;
    int w_begin, w_end;
    const int4* runs;      // [n_runs]
    int n_runs;
    const int2* subs;      // [n_subs]: run, 32-sample block of it
    int n_subs;
    int first_y;           // the block of the grid's first row: the grid takes RO_SUBS blocks a row, from the windows' first
    const float2* z;
    int z_cap;
    int per_part;          // groups of 32 spins per blockIdx.x
    int clip;              // BP_CLIP_BEGIN, BP_CLIP_END: the windows' samples alone, of runs that reach beyond them
    double* raw;           // [n_adc][2C] raw coil sums (float64 atomics)
};

__global__ void __launch_bounds__(RO_THREADS, 3) bp_readout_kernel(ReadArgs a) {
    __shared__ __align__(16) unsigned char sm[RO_WARPS][RO_WARP_BYTES];
    __shared__ __align__(16) float fetched[RO_WARPS][RO_FETCH * 32];
    __shared__ __align__(16) float2 fetched_z[RO_WARPS][RO_SUBS * 32];
    __shared__ int4 sub[RO_SUBS];   // samples (0: none), slot of z, 32-sample block, first ADC row
    __shared__ int ratio[RO_SUBS];  // the segment of the factor; -1 where it is the block before's
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = a.n, cg = blockIdx.z;
    if (warp == 0) {
        const int s_begin = a.windows[a.w_begin].x, s_end = a.windows[a.w_end - 1].y;
        const int lo = windows_run(a.runs, a.n_runs, s_begin, a.clip, lane);
        const int hi = min(warp_bound(a.n_runs, lane, [&](int i) { return a.runs[i].x < s_end; }), lo + a.z_cap);
        const int from = warp_bound(a.n_subs, lane, [&](int i) { return a.subs[i].x < lo; }) +
                         (a.first_y + (int)blockIdx.y) * RO_SUBS;
        // a lane per block; then what each shares with the block before it
        int4 sb = make_int4(0, 0, 0, 0);
        int seg = -1;
        if (lane < RO_SUBS && from + lane < a.n_subs) {
            const int2 rb = a.subs[from + lane];
            if (rb.x >= lo && rb.x < hi) {
                const int4 r = a.runs[rb.x];
                const int begin = max(r.x, s_begin);  // (a run's samples lie on consecutive segments)
                const int end = (a.clip & BP_CLIP_END) ? min(r.x + r.z, s_end) : r.x + r.z;
                const int samples = min(32, end - begin - 32 * rb.y);
                if (samples > 0) {
                    sb = make_int4(samples, rb.x - lo, rb.y, r.w + begin - r.x + 32 * rb.y);
                    seg = r.y >= 0 ? r.y : r.x;
                }
            }
        }
        int before = -1;  // the factor's segment of the last block before this one that has samples
#pragma unroll
        for (int b = 0; b < RO_SUBS; ++b) {
            const int other = __shfl_sync(0xffffffffu, seg, b);
            if (b < lane && other >= 0) before = other;
        }
        if (lane < RO_SUBS) {
            bool same = before >= 0 && seg >= 0;
            if (same && seg != before) {
                const double4 x = a.seg64[before], y = a.seg64[seg];
                same = a.segs[before].dt == a.segs[seg].dt && x.x == y.x && x.y == y.y && x.z == y.z && x.w == y.w;
            }
            sub[lane] = sb;
            ratio[lane] = same ? -1 : seg;
        }
    }
    __syncthreads();
    if (sub[0].x == 0 && sub[1].x == 0 && sub[2].x == 0 && sub[3].x == 0) return;

    uint4* sens = reinterpret_cast<uint4*>(sm[warp]);              // [32][8], split and swizzled
    float* tab = reinterpret_cast<float*>(sens + 32 * 8);          // [RO_ROWS][RO_TAB_ROW]: q^0 .. q^7, in pairs of spins
    float* step8 = tab + RO_ROWS * RO_TAB_ROW;                     // [16][4]: q^8, in pairs
    float* first = step8 + 16 * 4;                                 // [16][4]: the block's first sample, scaled, in pairs
    float2* nstep = reinterpret_cast<float2*>(first + 16 * 4);     // [16]: -im of the pairs of step8
    float2* nfirst = nstep + 16;                                   // and of first
    const int pw = pair_word(lane);                                // this lane's spin's place in its pair
    const int r = lane >> 2, t = lane & 3;
    float acc[RO_SUBS][2][2][4];  // block, 16 samples, real and imaginary, fragment
#pragma unroll
    for (int b = 0; b < RO_SUBS; ++b)
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[b][i >> 3][(i >> 2) & 1][i & 3] = 0.0f;

    // a group's values are fetched one group ahead (the loads' latency was half of the time): every lane reads what it
    // fetched itself
    float* in = fetched[warp];
    float2* in_z = fetched_z[warp];
    const int groups = (n + 31) / 32;
    const int g_end = min(groups, ((int)blockIdx.x + 1) * a.per_part);
    auto fetch = [&](int grp) {
        const int j = grp * 32 + lane;
        const bool there = grp < g_end && j < n;
        const int jj = there ? j : 0;
        const float* s = a.sens + (size_t)(16 * cg) * n + jj;
#pragma unroll
        for (int c = 0; c < 16; ++c) fetch4(in + c * 32 + lane, s + (size_t)c * n, there);
        const float* q = a.spins + jj;
        fetch4(in + 16 * 32 + lane, q, there);
        fetch4(in + 17 * 32 + lane, q + (size_t)n, there);
        fetch4(in + 18 * 32 + lane, q + 2 * (size_t)n, there);
        fetch4(in + 19 * 32 + lane, q + 5 * (size_t)n, there);
        fetch4(in + 20 * 32 + lane, q + 6 * (size_t)n, there);
#pragma unroll
        for (int b = 0; b < RO_SUBS; ++b)
            if (sub[b].x > 0) fetch8(in_z + b * 32 + lane, a.z + (size_t)sub[b].y * n + jj, there);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int g0 = (int)blockIdx.x * a.per_part + warp;
    fetch(g0);
    for (int grp = g0; grp < g_end; grp += RO_WARPS) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        float sens_inv[2];  // of this lane's two coils
        PropSpin p{};
        float2 zin[RO_SUBS];
        {
            float v[16];
#pragma unroll
            for (int c = 0; c < 16; ++c) v[c] = in[c * 32 + lane];
            p.x = (double)in[16 * 32 + lane], p.y = (double)in[17 * 32 + lane], p.z = (double)in[18 * 32 + lane];
            p.r2 = in[19 * 32 + lane], p.db0 = (double)in[20 * 32 + lane];
#pragma unroll
            for (int b = 0; b < RO_SUBS; ++b) zin[b] = in_z[b * 32 + lane];
            fetch(grp + RO_WARPS);
#pragma unroll
            for (int c = 0; c < 8; ++c) {  // every coil by its own scale
                const uint32_t u = __float_as_uint(fabsf(v[2 * c])), w = __float_as_uint(fabsf(v[2 * c + 1]));
                float scale, inverse;
                warp_scale(max(u < 0x7f800000u ? u : 0u, w < 0x7f800000u ? w : 0u), scale, inverse);
                if (t == (c >> 1)) sens_inv[c & 1] = inverse;
                sens[sens_slot(lane, c)] = split_sens(v[2 * c] * scale, v[2 * c + 1] * scale);
            }
        }
        float2 q32 = make_float2(1.0f, 0.0f), z = make_float2(0.0f, 0.0f);
        int slot = -1, part = 0;  // the run z belongs to, and its 32-sample block
#pragma unroll
        for (int b = 0; b < RO_SUBS; ++b) {
            const int4 sb = sub[b];
            if (sb.x == 0) continue;
            if (ratio[b] >= 0) {  // (uniform) the factor's powers
                const FreeFactors f = prop_factors(a.segs[ratio[b]].dt, a.seg64[ratio[b]], p, 1);
                float2 q8;
                factor_powers(f, q8, q32);
                double x, y, zr = 1.0, zi = 0.0;  // (float64: one rounding, and no slower than a float32 recurrence)
                factor64(f, x, y);
#pragma unroll
                for (int i = 0; i < RO_ROWS; ++i) {
                    tab[i * RO_TAB_ROW + pw] = (float)zr, tab[i * RO_TAB_ROW + pw + 2] = (float)zi;
                    const double nr = fma(x, zr, -y * zi);
                    zi = fma(x, zi, y * zr), zr = nr;
                }
                step8[pw] = q8.x, step8[pw + 2] = q8.y;
                reinterpret_cast<float*>(nstep)[(pw >> 2) * 2 + (pw & 1)] = -q8.y;
            }
            if (slot != sb.y || part > sb.z) {
                z = zin[b];
                slot = sb.y, part = 0;
            }
            for (; part < sb.z; ++part)
                z = make_float2(fmaf(z.x, q32.x, -z.y * q32.y), fmaf(z.x, q32.y, z.y * q32.x));
            float scale, inverse;
            const uint32_t u = __float_as_uint(fmaxf(fabsf(z.x), fabsf(z.y)));
            warp_scale(u, scale, inverse);
            first[pw] = z.x * scale, first[pw + 2] = z.y * scale;
            reinterpret_cast<float*>(nfirst)[(pw >> 2) * 2 + (pw & 1)] = -(z.y * scale);
            __syncwarp();
            float dr[2][4], di[2][4];
#pragma unroll
            for (int i = 0; i < 8; ++i) dr[i >> 2][i & 3] = di[i >> 2][i & 3] = 0.0f;
#pragma unroll 2
            for (int g = 0; g < 4; ++g) {  // eight spins: 8 g + t and 8 g + 4 + t are this lane's
                const int pr = 4 * g + t;
                const uint4 sa = sens[sens_slot(8 * g + t, r)], sc = sens[sens_slot(8 * g + 4 + t, r)];
                const CPair step = load_pair(step8 + 4 * pr);
                const float2 nim = nstep[pr];
                const CPair z0 = cmul2(load_pair(tab + r * RO_TAB_ROW + 4 * pr), load_pair(first + 4 * pr), nfirst[pr]);
                const CPair z1 = cmul2(z0, step, nim);
                readout_mma(z0, z1, sa, sc, dr[0], di[0]);
                if (sb.x > 16) {
                    const CPair z2 = cmul2(z1, step, nim);
                    readout_mma(z2, cmul2(z2, step, nim), sa, sc, dr[1], di[1]);
                }
            }
            __syncwarp();  // the operands' reads have ended
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    acc[b][h][0][i] = fmaf(dr[h][i] * inverse, sens_inv[i & 1], acc[b][h][0][i]);
                    acc[b][h][1][i] = fmaf(di[h][i] * inverse, sens_inv[i & 1], acc[b][h][1][i]);
                }
        }
        __syncwarp();  // (a group whose blocks were all skipped)
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // the operands are done with: the warps' sums take their place
    float* out = reinterpret_cast<float*>(sm[warp]);  // [128][16]
#pragma unroll
    for (int b = 0; b < RO_SUBS; ++b)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int i = 0; i < 4; i += 2)
                    *reinterpret_cast<float2*>(out + (32 * b + 16 * h + r + 4 * i) * 16 + 8 * c + 2 * t) =
                        make_float2(acc[b][h][c][i], acc[b][h][c][i + 1]);
    __syncthreads();
    const int nv = 2 * a.n_coils;
    for (int k = tid; k < RO_SUBS * 32 * 16; k += RO_THREADS) {
        const int row = k >> 4, b = row >> 5, coil = 8 * cg + (k & 7), im = (k >> 3) & 1;
        if ((row & 31) >= sub[b].x || coil >= a.n_coils) continue;
        float s = 0.0f;  // the warps in fixed order: the CTA's sum does not depend on timing
#pragma unroll
        for (int w = 0; w < RO_WARPS; ++w) s += reinterpret_cast<const float*>(sm[w])[k];
        atomicAdd(a.raw + (size_t)(sub[b].w + (row & 31)) * nv + 2 * coil + im, (double)s * RO_CUT);
    }
}

// ---- launch helpers ----
template <int K, int NT, int CH, bool HELP>
static int launch_propagate(const PropArgs& a, int max_ctas, cudaStream_t stream) {
    constexpr size_t smem = prop_smem<CH, HELP>();
    static_assert(smem <= 48 * 1024, "no opt-in needed");
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bp_propagate_kernel<K, NT, CH, HELP>, NT, smem) !=
        cudaSuccess)
        return BP_E_LAUNCH;
    constexpr int TILE = (HELP ? 32 : NT) * K;
    const int n_tiles = (a.n + TILE - 1) / TILE;
    int grid = num_sms() * (per_sm > 0 ? per_sm : 1);
    if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
    if (grid > n_tiles) grid = n_tiles;
    bp_propagate_kernel<K, NT, CH, HELP><<<grid, NT, smem, stream>>>(a);
    return cudaGetLastError() == cudaSuccess ? BP_OK : BP_E_LAUNCH;
}

extern "C" int bp_propagate(const float* spins, int n, const void* segs, const double* seg64, const int* windows,
                            int w_begin, int w_end, float* state, float* wstates, int wstate_stride, const int* wslot,
                            const int* runs, int n_runs, float* z, int z_cap, int clip, int max_ctas,
                            int* status, void* stream) {
    if (n < 1 || w_begin < 0 || w_end < w_begin || n_runs < 0 || z_cap < 0) return BP_E_ARG;
    if (!spins || !segs || !seg64 || !windows || !state || !status || (z && !runs)) return BP_E_ARG;
    if (wstates && !wslot && wstate_stride < 1) return BP_E_ARG;
    if ((reinterpret_cast<uintptr_t>(segs) & 15) != 0 || (reinterpret_cast<uintptr_t>(seg64) & 15) != 0 ||
        (reinterpret_cast<uintptr_t>(z) & 7) != 0)
        return BP_E_ALIGN;
    if (w_end == w_begin) return BP_OK;
    PropArgs a{};
    a.spins = spins;
    a.segs = static_cast<const SegRec*>(segs);
    a.seg64 = reinterpret_cast<const double4*>(seg64);
    a.windows = reinterpret_cast<const int4*>(windows);
    a.n = n;
    a.w_begin = w_begin;
    a.w_end = w_end;
    a.state = state;
    a.wstates = wstates;
    a.wstate_stride = wstate_stride > 0 ? wstate_stride : 1;
    a.wslot = wslot;
    a.runs = reinterpret_cast<const int4*>(runs);
    a.n_runs = n_runs;
    a.z = reinterpret_cast<float2*>(z);
    a.z_cap = z_cap;
    a.clip = clip;
    a.status = status;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // while one warp of 32 spins per CTA and its three helpers fit the GPU at once (five CTAs per SM): those; then one
    // warp per CTA, so that few spins spread over the SMs; past twice four warps per SM two spins per thread
    const int sms = num_sms();
    if (n <= sms * 5 * 32) return launch_propagate<1, 128, 96, true>(a, max_ctas, st);
    if (n <= sms * 4 * 32 * 2) return launch_propagate<1, 32, 160, false>(a, max_ctas, st);
    return launch_propagate<2, 128, 256, false>(a, max_ctas, st);
}

extern "C" int bp_readout(const float* spins, const float* sens, int n, int n_coils, const void* segs,
                          const double* seg64, const int* windows, int w_begin, int w_end, const int* runs, int n_runs,
                          const int* subs, int n_subs, int most_subs, const float* z, int z_cap, int clip, double* raw,
                          void* stream) {
    if (n < 1 || n_coils < 1 || n_coils > BP_MAX_COILS || w_begin < 0 || w_end < w_begin || n_runs < 0 || n_subs < 0 ||
        most_subs < 0 || z_cap < 0)
        return BP_E_ARG;
    if (w_end == w_begin || n_subs == 0 || n_runs == 0) return BP_OK;
    if (!spins || !sens || !segs || !seg64 || !windows || !runs || !subs || !z || !raw) return BP_E_ARG;
    if ((reinterpret_cast<uintptr_t>(z) & 7) != 0) return BP_E_ALIGN;
    ReadArgs a{};
    a.spins = spins;
    a.sens = sens;
    a.segs = static_cast<const SegRec*>(segs);
    a.seg64 = reinterpret_cast<const double4*>(seg64);
    a.windows = reinterpret_cast<const int4*>(windows);
    a.n = n;
    a.n_coils = n_coils;
    a.w_begin = w_begin;
    a.w_end = w_end;
    a.runs = reinterpret_cast<const int4*>(runs);
    a.n_runs = n_runs;
    a.subs = reinterpret_cast<const int2*>(subs);
    a.n_subs = n_subs;
    a.z = reinterpret_cast<const float2*>(z);
    a.z_cap = z_cap;
    a.clip = clip;
    a.raw = raw;
    // the spins' split depends on their number and the device alone (so the sums' order does): parts of at least 1,024
    // spins, at most three per SM (the CTAs one holds, so that 128 samples alone fill the GPU)
    const int groups = (n + 31) / 32, most_parts = 3 * num_sms();
    int parts = (groups + 31) / 32;
    if (parts > most_parts) parts = most_parts;
    a.per_part = (groups + parts - 1) / parts;
    const int at_most = most_subs < n_subs ? most_subs : n_subs, rows = (at_most + RO_SUBS - 1) / RO_SUBS;
    const dim3 grid((unsigned)((groups + a.per_part - 1) / a.per_part), 1u, (unsigned)((n_coils + 7) / 8));
    for (int y = 0; y < rows; y += 65535) {  // (the most of a grid's second dimension)
        a.first_y = y;
        bp_readout_kernel<<<dim3(grid.x, (unsigned)(rows - y < 65535 ? rows - y : 65535), grid.z), RO_THREADS, 0,
                            static_cast<cudaStream_t>(stream)>>>(a);
    }
    return cudaGetLastError() == cudaSuccess ? BP_OK : BP_E_LAUNCH;
}

// ---- the magnetization from the state: [n][3], high and low parts added ----
__global__ void bp_final_m_kernel(const float* __restrict__ state, int n, float* __restrict__ m) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * (int64_t)n) return;
    const int64_t j = i / 3, c = i - 3 * j;
    m[i] = (float)((double)state[c * n + j] + (double)state[(3 + c) * n + j]);
}

extern "C" int bp_final_m(const float* state, int n, float* m, void* stream) {
    if (n < 0 || (n > 0 && (!state || !m))) return BP_E_ARG;
    if (n == 0) return BP_OK;
    const int64_t blocks = (3 * (int64_t)n + 255) / 256;
    bp_final_m_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(state, n, m);
    return cudaGetLastError() == cudaSuccess ? BP_OK : BP_E_LAUNCH;
}
