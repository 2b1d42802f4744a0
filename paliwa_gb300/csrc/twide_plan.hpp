// Host side of the TMA wide kernel (twide.cuh): which stages it takes, their
// jobs and tensor maps, and its launches.
#pragma once

#include <cudaTypedefs.h>

#include "plan.hpp"
#include "twide.cuh"

namespace pgb {

// Launch codes kTWide + a form code (twide_code).
constexpr int kTWide = 2048;

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against libcuda); nullptr where the driver lacks it.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder();

// The form code of the TMA wide launch that takes a stage planned on it
// (Stage::tma): the chunk size plus the form's offset, or kTWide32*; 0 for
// the other stages.
int twide_code(Stage const &st, int dtype);

// The stage's job, tensor maps (map[1], the halo buffer's, for windows only)
// and tiles; the job names them 0 and 1. False when it does not qualify
// (alignment, 2^30 tiles or more, or the encoder refuses a map); the stage
// then runs on its own kernel (Stage::R).
bool twide_job(Stage const &st, int dtype, TWideJob &job, CUtensorMap map[2],
               long long &tiles);

// Whether a launch of form `code` over `points` points in all is worth its
// start-up (mbarriers, the tensor map's first fetch).
bool twide_enough(int code, int dtype, long long points);

// Schedules of a caller's filters over the levels of dehierarchize_in and
// (+ 1) hierarchize_in, after the wavelets' 0 .. 5.
constexpr int kTableSched = 6;

// sched = 2 * wavelet + (forward ? 1 : 0), or kTableSched (+ 1) for FP32 and
// FP64 grids (then p.filters, and exact as from exact_scalers); code as from
// twide_code.
void launch_twide(int dtype, bool exact, int sched, int code,
                  TWideParams const &p, cudaStream_t s);
void launch_twide_f32(int sched, int code, TWideParams const &p,
                      cudaStream_t s);
void launch_twide_f32c(int sched, int code, TWideParams const &p,
                       cudaStream_t s);
void launch_twide_f64(int sched, int code, TWideParams const &p,
                      cudaStream_t s);
void launch_twide_table_f32(bool exact, int sched, int code,
                            TWideParams const &p, cudaStream_t s);
void launch_twide_table_f64(bool exact, int sched, int code,
                            TWideParams const &p, cudaStream_t s);

// Before a single-grid call on stream s queues anything: throws
// PALIWA_GB_TIMEOUT as check_stage_errors does (the call's grid is untouched),
// and returns the word that the call's bounded waits report to; nullptr where
// there is none, or no encoder: the call then runs without TMA launches.
unsigned *begin_stages(cudaStream_t s);
unsigned *stage_error_word(cudaStream_t s);

// Throws PALIWA_GB_TIMEOUT when a bounded wait of a single-grid launch gave
// up since the last report: one on stream s, or one that was captured (on any
// stream of the device). Clears the report.
void check_stage_errors(cudaStream_t s);

// Launches one stage of a single grid: on the TMA wide kernel when it is
// planned on it, qualifies and error (from begin_stages) is there, else on its
// own kernel. ws is the filters' wavelet schedule (or -1).
void launch_stage(int dtype, bool exact, bool symmetric, int ws,
                  LiftParams const &params, Stage const &st, unsigned *error,
                  cudaStream_t s);

} // namespace pgb
