// Test harness: the wave plans (wave_plan.h) for a CPU test.
#include "wave_plan.h"

extern "C" int batch_wave(uint64_t total, uint32_t spp, uint32_t stream_paths, uint32_t tuned, uint64_t* paths) {
	const psy::WavePlan p = psy::batch_plan(total, spp, stream_paths, tuned);
	*paths = p.paths;
	return p.pair;
}
