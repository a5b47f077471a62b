// Host-side launch loop of a forward whose recurring pulses are replaced (simulate(..., pulses="reuse") and
// pulses="surrogate"): the windows between occurrences through bp_propagate, with bp_readout over as many of them as the
// workspace z holds the sample runs of (without z through bp_forward), each occurrence through its map or network, all
// issued from host code in one call. The 408 pulses of the 393,216-spin TSE through float32 networks, whole call: 0.252 s
// with bp_forward for the windows, 0.216 s so. Replaces the per-occurrence dispatch of blochparty's driver
// (engines/gpu/driver.py:617-698 with the reuse branch of bloch_chunk_mma, engines/gpu/cuda/kernels.cu.in:141-165).
#include <cstddef>

#include "../../include/blochparty_b200.h"

static int forward_spans(const float* spins, const float* sens, int n, int n_coils, const void* segs,
                         const double* seg64, const int32_t* windows, const int32_t* ranges, int n_spans,
                         const BpSpan* spans, float* state, double* raw, int max_ctas, const int32_t* runs, int n_runs,
                         const int32_t* subs, int n_subs, int most_subs, const int32_t* run_at, float* z, int z_cap,
                         int32_t* status, void* stream) {
    if (!spins || !sens || !segs || !seg64 || !windows || !ranges || !state || !status || n < 1 || n_spans < 0 ||
        (n_spans > 0 && !spans))
        return BP_E_ARG;
    int w_first = 0, w_last = 0, base = 0;  // the windows since the last readout, and their first run
    auto read = [&]() {
        if (!z || w_last == w_first) return BP_OK;
        return bp_readout(spins, sens, n, n_coils, segs, seg64, windows, w_first, w_last, runs, n_runs, subs, n_subs,
                          most_subs, z, z_cap, 0, raw, stream);
    };
    auto step = [&](int r) {
        const int wa = ranges[2 * r], wb = ranges[2 * r + 1];
        if (wb < wa || wa < 0) return BP_E_ARG;
        if (wb == wa) return BP_OK;
        if (raw && !z)
            return bp_forward(spins, sens, n, n_coils, segs, seg64, windows, wa, wb, state, raw, nullptr, 1, max_ctas,
                              status, stream);
        int at = 0;  // the range's first run's place in z
        if (z) {
            if (run_at[r + 1] < run_at[r] || run_at[r + 1] - run_at[r] > z_cap) return BP_E_ARG;
            if (run_at[r + 1] - base > z_cap || w_last == w_first) {
                const int code = read();
                if (code != BP_OK) return code;
                w_first = wa, base = run_at[r];
            }
            w_last = wb, at = run_at[r] - base;
        }
        return bp_propagate(spins, n, segs, seg64, windows, wa, wb, state, nullptr, 1, nullptr, z ? runs : nullptr,
                            z ? n_runs : 0, z ? z + 2 * (size_t)n * at : nullptr, z ? z_cap - at : 0, 0, max_ctas,
                            status, stream);
    };
    for (int i = 0; i < n_spans; ++i) {
        int code = step(i);
        if (code != BP_OK) return code;
        const BpSpan& sp = spans[i];
        switch (sp.kind) {
            case BP_SPAN_MAP:
                code = bp_pulse_apply(sp.map, n, state, sp.phase, stream);
                break;
            case BP_SPAN_NET_MMA:
                code = bp_surrogate_pulse_mma(spins, state, n, sp.params, sp.wtiles, segs, sp.seg0, sp.k_steps, sp.T,
                                              sp.gz, sp.thickness, sp.z0, sp.phase, sp.b0off, sp.dom_df, sp.dom_b1,
                                              sp.dom_z, sp.counts, status, max_ctas, stream);
                break;
            case BP_SPAN_NET_F32:
                code = bp_surrogate_pulse(spins, state, n, sp.params, segs, sp.seg0, sp.k_steps, sp.T, sp.gz,
                                          sp.thickness, sp.z0, sp.phase, sp.b0off, sp.dom_df, sp.dom_b1, sp.dom_z,
                                          sp.counts, stream);
                break;
            default:
                code = BP_E_ARG;
        }
        if (code != BP_OK) return code;
    }
    const int code = step(n_spans);
    return code != BP_OK ? code : read();
}

extern "C" int bp_forward_spans(const float* spins, const float* sens, int n, int n_coils, const void* segs,
                                const double* seg64, const int32_t* windows, const int32_t* ranges, int n_spans,
                                const BpSpan* spans, float* state, double* raw, int max_ctas, int32_t* status,
                                void* stream) {
    return forward_spans(spins, sens, n, n_coils, segs, seg64, windows, ranges, n_spans, spans, state, raw, max_ctas,
                         nullptr, 0, nullptr, 0, 0, nullptr, nullptr, 0, status, stream);
}

extern "C" int bp_forward_spans_readout(const float* spins, const float* sens, int n, int n_coils, const void* segs,
                                        const double* seg64, const int32_t* windows, const int32_t* ranges, int n_spans,
                                        const BpSpan* spans, float* state, double* raw, int max_ctas,
                                        const int32_t* runs, int n_runs, const int32_t* subs, int n_subs, int most_subs,
                                        const int32_t* run_at, float* z, int z_cap, int32_t* status, void* stream) {
    if (!raw || !runs || !subs || !run_at || !z || n_runs < 0 || n_subs < 0 || most_subs < 0 || z_cap < 0) return BP_E_ARG;
    return forward_spans(spins, sens, n, n_coils, segs, seg64, windows, ranges, n_spans, spans, state, raw, max_ctas,
                         runs, n_runs, subs, n_subs, most_subs, run_at, z, z_cap, status, stream);
}
