// Per-n schedule selection for the stage kernels.
//
// The reference specialises its kernel per (n, pairs per CTA, block size) with NVRTC
// and picks the block size by probing cuSolverDx or by a timing sweep
// (src/nvrtc/nvrtc_solver.cpp:205-240, 649-925, 1021-1042), caching the cubin in
// process and on disk (:392-597).  Here every kernel is compiled ahead of time for
// sm_100a and takes its CTA from n, so that of a schedule's eight fields two shape a launch: reduce_tc, and
// chain_threads for the pairs that inverse iteration gives up.  Suggested mode uses a built-in table;
// autotune mode times the stages on a synthetic batch, validates the schedule (every pair's info,
// eigenvalues against the built-in schedule's, host residuals of sampled columns), and memoises it in process and in a
// versioned, checksummed table file (atomic write-then-rename; a corrupt or foreign file is
// ignored and rewritten).
#pragma once

#include "kernels.cuh"

#include <string>

namespace sbg {

struct Schedule {
    int hetrd_threads = 256;    // what block_dim_x reports and force_block_dim_x sets (128 or 256); no kernel's
                                // CTA size depends on it
    int pair_warps = 2;         // 1, 2 or 4: what batches_per_block reports and sets for n <= 65; no kernel's
                                // shape depends on it
    int col_exact = 1;          // 0 or 1, kept from earlier tables: no kernel depends on it
    int back_lanes = 1;         // 1 or 2, kept from earlier tables: no kernel depends on it
    int back_qpass = 1;         // 1 or 2, likewise
    int reduce_tc = 0;          // n > 84: 1 = the tensor-core stages, 0 = csrc/bigsolve.cu's
    int ql_warps = 4;           // batches_per_block above n = 65, bounded by shared memory; no kernel's shape
                                // depends on it
    int chain_threads = 128;    // pairs (threads) per CTA of the QL scalar-chain kernel (n > 63, flagged pairs)
    LaunchShape shape() const {
        LaunchShape l;
        l.reduce_tc = reduce_tc;
        return l;
    }
    bool operator==(const Schedule& o) const {
        return hetrd_threads == o.hetrd_threads && pair_warps == o.pair_warps && col_exact == o.col_exact &&
               back_lanes == o.back_lanes && back_qpass == o.back_qpass && ql_warps == o.ql_warps &&
               chain_threads == o.chain_threads && reduce_tc == o.reduce_tc;
    }
};

struct TuneRequest {
    int n = 0;
    int device = 0;
    int precision = 0;
    int force_threads = 0;      // 0 = choose; else 128 or 256 (hetrd_threads)
    int force_bpb = 0;          // 0 = choose; else pairs per CTA (pair_warps for n <= 65, else ql_warps)
    bool autotune = false;
    int cache_mode = 0;         // SBG_CACHE_*
};

struct TuneResult {
    Schedule sched;
    bool autotuned = false;
    bool sweep_ran = false;
    const char* layer = "builtin";   // builtin | in-process | disk | measured
};

Schedule default_schedule(int n, int precision);
// Whether every kernel of the schedule fits the current device's shared memory for order n.
bool schedule_fits(int n, int precision, const Schedule& s);
TuneResult select_schedule(const TuneRequest& req);

// Table file helpers (exposed for tests through the C ABI in tuning_capi).
std::string tuning_cache_dir();
std::string tuning_table_path(int device);
void forget_in_process();
// Message returned by sbg_last_error() on this host thread.
void set_last_error(const std::string& msg);

}  // namespace sbg
