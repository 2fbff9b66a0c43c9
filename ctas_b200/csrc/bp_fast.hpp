// bp_fast.hpp -- launch interface of the staged backprojection kernel.
#pragma once
#include <cuda_runtime.h>

#include <functional>
#include <tuple>

#include "fbp_kernels.hpp"

namespace ctas {
// True when the staged kernel can serve this launch (for the truncation rule
// the caller also checks that every sine of the angle table is >= 0).
bool bp_fast_supported(const BpLaunch &a);
// Number of tile configurations (ids 0 .. count-1).
int bp_fast_tile_count();
// Details of the last failure on this thread ("" if none).
const char *bp_fast_error_detail();
// Tile search: every shape with the arithmetic variant that is usually
// fastest, then every other variant of the winning shape (all_variants =
// float32 truncation launches; otherwise variant 0 only).  time_ms(tile)
// runs one candidate and returns its time, < 0 if it failed; each candidate
// runs twice and the second time counts.  Returns -1 if every one failed.
int bp_fast_search(const std::function<float(int)> &time_ms, bool all_variants);
// Launches that share the autotuner's choice: one device, geometry, kernel form and
// fill of the device.  The wide layout has kernels of its own, and the one or two slices
// that a stack leaves over (rest) do not decide for full launches: on nine slices of
// 1800 x 2560 the tile that two wide slices prefer (14) takes 14.8 ms, the full launch's
// own (15) 14.2.  Launches of few waves (up to eight 64 x 64 tiles per SM) are tuned for
// their number of slices: three full-turn slices of 700 x 700 prefer tile 18, with which
// five take 349 us, 222 with tile 14; eleven slices of 460 x 460 take 262 us with the
// tile of ten, 199 with their own.  Trial centres of one sinogram come in varying numbers
// from one search and share a choice.
using TuneKey = std::tuple<int, int, int, int, int, int, int, bool, bool, int>;
inline TuneKey bp_fast_tune_key(const BpLaunch &a, int device, bool rest, int sms = 148) {
  const int64_t tiles = (int64_t)((a.out_rows + 63) / 64) * ((a.out_cols + 63) / 64) * a.S;
  const int few = !a.centers && tiles <= 8 * (int64_t)sms ? a.S : 0;
  return TuneKey(device, a.W, a.N, a.store, a.interp, a.out_rows, a.out_cols, a.wide != 0, rest, few);
}
// Tile for this launch: `requested` if it is a valid id, else the
// CTAS_FBP_TILE environment override, else the autotuner's choice for the launch's
// TuneKey -- the first such launch runs bp_fast_search on a few of its slices
// (synchronising the stream).  While the stream is being captured nothing can be
// timed: a launch of a new key then takes a choice made for other slice counts, else the
// usually fastest tile, and it is not kept.
// rest: the launch is what a stack's four-slice groups leave over.
int bp_fast_choose_tile(const BpLaunch &a, cudaStream_t st, int requested, bool rest = false);
// True when CTAS_FBP_TILE names a tile.
bool bp_fast_tile_forced();
cudaError_t launch_bp_fast(const BpLaunch &a, cudaStream_t st, int tile);
// Same kernel with every shared-memory gather checked against its window
// (violations set bit 8 of *a.err and read 0); for tests.
cudaError_t launch_bp_fast_checked(const BpLaunch &a, cudaStream_t st, int tile);
// Rows x columns of a tile id's pixel tile, and its window length (samples).
void bp_fast_tile_shape(int tile, int *ty, int *tx);
int bp_fast_tile_window(int tile);
// Persistent backprojection of an uneven batch (float32 store, truncation
// rule, every sine >= 0): resident CTAs take (sinogram, tile) items from
// b.counter, which must be 0 at launch.
cudaError_t launch_bp_batch(const BatchLaunch &b, int tile, cudaStream_t st);
}  // namespace ctas
