// Host-side window planner of the C ABI (no GPU needed): see bp_plan_windows in include/blochparty_b200.h.
#include <cstdint>

#include "../../include/blochparty_b200.h"

extern "C" int bp_plan_windows(const int32_t* flags, int64_t n_segments, int seg_max, int samp_max,
                               const uint8_t* breaks, int32_t* windows, int64_t max_windows, int64_t* n_windows) {
    if (!flags || !windows || !n_windows || n_segments < 0 || seg_max < 1 || seg_max > BP_SEG_MAX || samp_max < 1)
        return BP_E_ARG;
    int64_t nw = 0, row = 0, s = 0;
    while (s < n_segments) {
        const int64_t start = s, row0 = row;
        int64_t samples = 0;
        bool limited = false;  // cut by seg_max or samp_max (not by a break or the sequence's end)
        while (s < n_segments) {
            if (s > start && breaks && breaks[s]) break;
            const bool adc = (flags[s] & 2) != 0;
            if (s - start == seg_max || (adc && samples == samp_max)) {
                limited = true;
                break;
            }
            samples += adc ? 1 : 0;
            ++s;
        }
        // a limit's cut moves back to a multiple of BP_ADJ_WIN segments when the window keeps one: the cuts then
        // fall on the same segments whatever the breaks before them
        const int64_t aligned = (s / BP_ADJ_WIN) * BP_ADJ_WIN;
        if (limited && aligned > start) {
            for (int64_t t = aligned; t < s; ++t) samples -= (flags[t] & 2) ? 1 : 0;
            s = aligned;
        }
        row += samples;
        if (nw >= max_windows) return BP_E_SIZE;
        windows[4 * nw] = static_cast<int32_t>(start);
        windows[4 * nw + 1] = static_cast<int32_t>(s);
        windows[4 * nw + 2] = static_cast<int32_t>(row0);
        windows[4 * nw + 3] = static_cast<int32_t>(samples);
        ++nw;
    }
    *n_windows = nw;
    return BP_OK;
}

// The runs of samples of bp_propagate and their 32-sample blocks (flags: 1 RF, 2 sample, 4 spoil, 8 the free segment
// before it has the same factors).
extern "C" int bp_sample_runs(const int32_t* flags, int64_t n, int run_max, int32_t* runs, int64_t max_runs,
                              int64_t* n_runs, int32_t* subs, int64_t max_subs, int64_t* n_subs) {
    if (n < 0 || run_max < 64 || !n_runs || !n_subs || (n > 0 && (!flags || !runs || !subs))) return BP_E_ARG;
    int64_t r = -1, row = 0;
    bool cut = false;  // the run is the rest of one that was too long: its first sample has its samples' factors
    for (int64_t s = 0; s < n; ++s) {
        const int32_t f = flags[s];
        if (!(f & 2)) continue;
        int32_t* u = runs + 4 * r;
        bool joins = false, full = false;
        if (r >= 0 && u[0] + u[2] == s && !(f & 1) && !(flags[s - 1] & 4)) {
            full = s % 32 == 0 && s - u[0] + 32 > run_max;
            joins = (u[2] == 1 && !cut) || ((f & 8) && !full);
        }
        if (joins) {
            u[1] = u[0] + 1;
            ++u[2];
        } else {
            cut = full && (f & 8) && u[2] > 1;
            if (++r >= max_runs) return BP_E_SIZE;
            u = runs + 4 * r;
            u[0] = (int32_t)s, u[1] = -1, u[2] = 1, u[3] = (int32_t)row;
        }
        ++row;
    }
    *n_runs = r + 1;
    int64_t m = 0;
    for (int64_t i = 0; i <= r; ++i)
        for (int32_t b = 0; b < (runs[4 * i + 2] + 31) / 32; ++b, ++m) {
            if (m >= max_subs) return BP_E_SIZE;
            subs[2 * m] = (int32_t)i, subs[2 * m + 1] = b;
        }
    *n_subs = m;
    return BP_OK;
}
