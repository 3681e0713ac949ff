/*
 * The wave kernels of batched renders over flat scenes.
 */
#include "render_wave.cuh"

namespace psy {
template void launch_wave<BatchWave, FEAT_FLAT>(const BatchWave&, int, uint32_t, const HaltonDev&, const WaveRange&, const PathSoA&, const WaveBufs&, const WaveQueues&, unsigned*, int, size_t, cudaStream_t, uint32_t*, const LaunchTimer*);
}  // namespace psy
