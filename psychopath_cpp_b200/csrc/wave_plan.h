/*
 * How many paths a wave of a render holds, and whether two waves are in
 * flight (host).
 */
#ifndef PSY_WAVE_PLAN_H
#define PSY_WAVE_PLAN_H

#include <algorithm>
#include <cstdint>

namespace psy {

// Waves in flight.  A wave's launches each end with the longest of its rays
// or paths, on an ever emptier chip; two waves on two streams fill each
// other's ends (512x384x16 frame with 50,000 primitives 12.3 -> 11.3 ms,
// 320x240x16 1.95 -> 1.86, differentiable step 7.4 -> 7.1).  Below PAIR_MIN
// paths a wave is all latency and two halves of it gain nothing.
static constexpr uint64_t AUTO_PATHS = 1ull << 22;  // paths in flight unless the caller says
static constexpr uint64_t PAIR_MIN = 1ull << 17;

struct WavePlan {
	uint64_t paths;  // per wave
	bool pair;       // two waves in flight, not one after another
};

// The waves of `total` paths with `want` of them in flight.
inline WavePlan wave_plan(uint64_t total, uint64_t want, bool pair) {
	want = std::min(std::min<uint64_t>(want, 1ull << 26), total);
	pair = pair && want >= PAIR_MIN;
	return {pair ? (want + 1) / 2 : want, pair};
}

// The waves of a batch: the caller's `stream_paths`, one wave after another,
// else what the autotuner found or AUTO_PATHS, in flight.  Waves end on pixel
// boundaries, of at most `spp` paths a pixel, and two of them hold the paths
// wanted at least.
inline WavePlan batch_plan(uint64_t total, uint32_t spp, uint32_t stream_paths, uint32_t tuned) {
	WavePlan p = wave_plan(total, stream_paths ? stream_paths : tuned ? tuned : AUTO_PATHS, !stream_paths);
	p.paths = std::min(std::max<uint64_t>(p.paths + (p.pair ? spp : 0), spp), total);
	return p;
}

}  // namespace psy

#endif
