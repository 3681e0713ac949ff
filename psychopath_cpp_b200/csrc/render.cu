/*
 * Host side of the wave renderer: the compiled variant of a scene, and the
 * batched light samples (psy_light_sample).
 */
#include "render_wave.cuh"

namespace psy {

extern template void launch_wave<PlainWave, FEAT_FLAT>(const PlainWave&, int, uint32_t, const HaltonDev&, const WaveRange&, const PathSoA&, const WaveBufs&, const WaveQueues&, unsigned*, int, size_t, cudaStream_t, uint32_t*, const LaunchTimer*);
extern template void launch_wave<PlainWave, FEAT_STILL_BICUBIC>(const PlainWave&, int, uint32_t, const HaltonDev&, const WaveRange&, const PathSoA&, const WaveBufs&, const WaveQueues&, unsigned*, int, size_t, cudaStream_t, uint32_t*, const LaunchTimer*);
extern template void launch_wave<PlainWave, FEAT_STILL>(const PlainWave&, int, uint32_t, const HaltonDev&, const WaveRange&, const PathSoA&, const WaveBufs&, const WaveQueues&, unsigned*, int, size_t, cudaStream_t, uint32_t*, const LaunchTimer*);
extern template void launch_wave<PlainWave, FEAT_ALL>(const PlainWave&, int, uint32_t, const HaltonDev&, const WaveRange&, const PathSoA&, const WaveBufs&, const WaveQueues&, unsigned*, int, size_t, cudaStream_t, uint32_t*, const LaunchTimer*);
extern template void launch_wave<BatchWave, FEAT_FLAT>(const BatchWave&, int, uint32_t, const HaltonDev&, const WaveRange&, const PathSoA&, const WaveBufs&, const WaveQueues&, unsigned*, int, size_t, cudaStream_t, uint32_t*, const LaunchTimer*);
extern template void launch_wave<BatchWave, FEAT_ALL>(const BatchWave&, int, uint32_t, const HaltonDev&, const WaveRange&, const PathSoA&, const WaveBufs&, const WaveQueues&, unsigned*, int, size_t, cudaStream_t, uint32_t*, const LaunchTimer*);

int render_counter_count(uint32_t path_length) { return wave_counter_count(path_length); }

static int valid_block(int block) { return (block == 64 || block == 128 || block == 256) ? block : 128; }

cudaError_t launch_render_wave(const DevScene& sc, const HaltonDev& hd, const RenderParams& rp, const WaveRange& wv,
                               const PathSoA& ps, const WaveBufs& wb, const WaveQueues& wq, unsigned* status,
                               int block, cudaStream_t st, uint32_t* launches, const LaunchTimer* timer) {
	PlainWave w;
	w.sc = sc;
	w.rp = rp;
	block = valid_block(block);
	const size_t gsmem = (rp.grad && rp.grad_in_smem) ? (rp.grad_in_smem == GRAD_SMEM64 ? sizeof(double) : sizeof(float)) * (size_t)rp.param_count : 0;
	const uint32_t L = rp.path_length;
	const int mode = shade_mode(sc.features, rp.grad != nullptr);
	switch (feature_variant(sc.features)) {
		case FEAT_FLAT: launch_wave<PlainWave, FEAT_FLAT>(w, mode, L, hd, wv, ps, wb, wq, status, block, gsmem, st, launches, timer); break;
		case FEAT_STILL_BICUBIC: launch_wave<PlainWave, FEAT_STILL_BICUBIC>(w, mode, L, hd, wv, ps, wb, wq, status, block, gsmem, st, launches, timer); break;
		case FEAT_STILL: launch_wave<PlainWave, FEAT_STILL>(w, mode, L, hd, wv, ps, wb, wq, status, block, gsmem, st, launches, timer); break;
		default: launch_wave<PlainWave, FEAT_ALL>(w, mode, L, hd, wv, ps, wb, wq, status, block, gsmem, st, launches, timer); break;
	}
	return cudaGetLastError();
}

cudaError_t launch_batch_wave(const DevScene* scenes, const RenderParams* renders, int count, unsigned features,
                              uint32_t max_path_length, const HaltonDev& hd, const WaveRange& wv, const PathSoA& ps,
                              const WaveBufs& wb, const WaveQueues& wq, unsigned* status, int block,
                              cudaStream_t st, uint32_t* launches) {
	BatchWave w;
	w.scenes = scenes;
	w.renders = renders;
	w.count = count;
	const int mode = shade_mode(features, false);
	block = valid_block(block);
	if (feature_variant(features) == FEAT_FLAT)
		launch_wave<BatchWave, FEAT_FLAT>(w, mode, max_path_length, hd, wv, ps, wb, wq, status, block, 0, st, launches, nullptr);
	else
		launch_wave<BatchWave, FEAT_ALL>(w, mode, max_path_length, hd, wv, ps, wb, wq, status, block, 0, st, launches, nullptr);
	return cudaGetLastError();
}

// ---------------------------------------------------------------------
// Batched LightTree::sample queries (psy_light_sample)
// ---------------------------------------------------------------------
// One LightTree::sample query of a Lambert surface.
__device__ __forceinline__ void light_query(const DevScene& sc, LightQuery* lq, float ident_inv) {
	lq->has_xform = false;
	lq->gtr = false;
	lq->id = 0;
	lq->selection_pdf = 1.0f;
	lq->light_sample_pdf = 1.0f;
	light_tree_pick<FEAT_ALL, false>(sc, lq);
	light_emit<FEAT_ALL>(sc, lq, ident_inv);
}

// Queries and samples as rows (psy_light_sample_rows).
__global__ void light_rows_kernel(DevScene sc, const float* __restrict__ rows, float* __restrict__ out,
                                  uint64_t* __restrict__ ids, uint32_t n, float ident_inv, unsigned* status) {
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const float* r = rows + 15 * (size_t)i;
	float* o = out + 14 * (size_t)i;
	LightQuery lq;
	lq.n = r[0];
	lq.u = r[1];
	lq.v = r[2];
	lq.pos = V3(r[3], r[4], r[5]);
	lq.nor = V3(r[6], r[7], r[8]);
	lq.d = V3(r[9], r[10], r[11]);
	lq.wavelength = r[12];
	lq.time = r[13];
	light_query(sc, &lq, ident_inv);
	if (!lq.valid) atomicOr(status, ERRF_NOLIGHT);
	// (a query without a sample ends the call with an error)
	o[0] = lq.valid ? lq.to_light.x : 0.0f;
	o[1] = lq.valid ? lq.to_light.y : 0.0f;
	o[2] = lq.valid ? lq.to_light.z : 0.0f;
	for (int k = 0; k < 4; ++k) o[3 + k] = lq.valid ? lq.spec.e[k] : 0.0f;
	o[7] = lq.wavelength;
	o[8] = lq.valid ? lq.selection_pdf : 0.0f;
	o[9] = lq.valid ? lq.light_sample_pdf : 0.0f;
	for (int k = 10; k < 14; ++k) o[k] = 0.0f;
	ids[i] = lq.valid ? lq.id : 0ull;
}

cudaError_t launch_light_rows(const DevScene& sc, const float* rows, float* out, uint64_t* ids, uint32_t n,
                              float ident_inv, unsigned* status, cudaStream_t st) {
	if (n == 0) return cudaSuccess;
	light_rows_kernel<<<(n + 127) / 128, 128, 0, st>>>(sc, rows, out, ids, n, ident_inv, status);
	return cudaGetLastError();
}

__global__ void light_sample_kernel(DevScene sc, LightQuerySoADev q, LightSampleSoADev o, uint32_t n, float ident_inv,
                                    unsigned* status) {
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	LightQuery lq;
	lq.n = q.n[i];
	lq.u = q.u[i];
	lq.v = q.v[i];
	lq.pos = V3(q.pos[3 * i], q.pos[3 * i + 1], q.pos[3 * i + 2]);
	lq.nor = V3(q.nor[3 * i], q.nor[3 * i + 1], q.nor[3 * i + 2]);
	lq.d = V3(q.d[3 * i], q.d[3 * i + 1], q.d[3 * i + 2]);
	lq.wavelength = q.wavelength[i];
	lq.time = q.time[i];
	light_query(sc, &lq, ident_inv);
	if (!lq.valid) {
		atomicOr(status, ERRF_NOLIGHT);
		return;
	}
	if (o.to_light) {
		o.to_light[3 * i] = lq.to_light.x;
		o.to_light[3 * i + 1] = lq.to_light.y;
		o.to_light[3 * i + 2] = lq.to_light.z;
	}
	if (o.spec)
		for (int k = 0; k < 4; ++k) o.spec[4 * i + k] = lq.spec.e[k];
	if (o.selection_pdf) o.selection_pdf[i] = lq.selection_pdf;
	if (o.light_pdf) o.light_pdf[i] = lq.light_sample_pdf;
	if (o.id) o.id[i] = lq.id;
}

cudaError_t launch_light_sample(const DevScene& sc, const LightQuerySoADev& q, const LightSampleSoADev& o, uint32_t n,
                                float ident_inv, unsigned* status, cudaStream_t st) {
	if (n == 0) return cudaSuccess;
	light_sample_kernel<<<(n + 127) / 128, 128, 0, st>>>(sc, q, o, n, ident_inv, status);
	return cudaGetLastError();
}

}  // namespace psy
