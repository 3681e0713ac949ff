/*
 * The wave kernels of single renders over still-patch scenes.
 */
#include "render_wave.cuh"

namespace psy {
template void launch_wave<PlainWave, FEAT_STILL>(const PlainWave&, int, uint32_t, const HaltonDev&, const WaveRange&, const PathSoA&, const WaveBufs&, const WaveQueues&, unsigned*, int, size_t, cudaStream_t, uint32_t*, const LaunchTimer*);
}  // namespace psy
