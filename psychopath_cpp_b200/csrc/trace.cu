/*
 * psy_trace kernel: Tracer::trace for a device ray stream
 * (reference tracer/tracer.cpp:38-121).  One thread per ray; rays are read
 * as SoA float streams and the requested Intersection fields are written as
 * SoA streams.
 */
#include "kernels.h"
#include "shade_geom.cuh"

namespace psy {

__device__ __forceinline__ V3 ld3(const float* p, uint32_t i) {
	return V3(__ldg(p + 3 * (size_t)i), __ldg(p + 3 * (size_t)i + 1), __ldg(p + 3 * (size_t)i + 2));
}
__device__ __forceinline__ void st3(float* p, uint32_t i, V3 v) {
	p[3 * (size_t)i] = v.x;
	p[3 * (size_t)i + 1] = v.y;
	p[3 * (size_t)i + 2] = v.z;
}

// A ray of the stream and the hit it ends with (Trav's IO).
struct StreamIO {
	const RaySoA* rays;
	HitRec* rec;
	HitPath* path;
	uint32_t i;
	__device__ __forceinline__ V3 origin() const { return ld3(rays->o, i); }
	__device__ __forceinline__ V3 direction() const { return ld3(rays->d, i); }
	__device__ __forceinline__ void differentials(V3* odx, V3* ody, V3* ddx, V3* ddy) const {
		*odx = ld3(rays->odx, i);
		*ody = ld3(rays->ody, i);
		*ddx = ld3(rays->ddx, i);
		*ddy = ld3(rays->ddy, i);
	}
	template <class T>
	__device__ __forceinline__ void hit(const T& tr, int inst, float t, float u, float v, float md) const {
		rec->t = t;
		rec->u = u;
		rec->v = v;
		rec->max_dim = md;
		rec->inst = inst;
		rec->place = tr.place;
		if (T::NESTED && tr.place < 0) {
			path->depth = tr.L + 1;
			for (int k = 1; k <= tr.L; ++k) path->path[k - 1] = tr.mem->lv_inst[k];
			path->path[tr.L] = inst;
		}
	}
};

// Register cap of the kernel: 64 for flat scenes (spheres, lights, bilinear
// patches in one level), where more resident warps hide the walk's memory
// latency (4M rays against the heightfield: 0.925 ms; 0.951 at 80 registers,
// 0.981 at 96, 1.085 at 128), 128 for the larger variants, whose bicubic
// bisection spills below that (300,000 mixed rays against instanced patches
// and spheres: 1.58 ms; 1.68 at 144, 1.63 at 168, 1.82 at 112, 1.85 at 96).
template <unsigned F>
struct TraceKernelRegs {
	static constexpr int value = F == FEAT_FLAT ? 64 : 128;
};

template <unsigned F>
__global__ void __maxnreg__(TraceKernelRegs<F>::value) trace_kernel(DevScene sc, RaySoA rays, HitSoA hits,
                                                                   uint32_t n, int lanes, unsigned* status) {
	// `lanes` rays a warp (a power of two)
	const int lane = threadIdx.x & 31;
	const uint32_t i = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (uint32_t)lanes + (uint32_t)lane;
	if (lane >= lanes || i >= n) return;
	HitRec rec;
	HitPath path;
	rec.inst = -1;
	WorldRayD wr;
	wr.o = ld3(rays.o, i);
	wr.d = ld3(rays.d, i);
	wr.time = __ldg(rays.time + i);
	wr.occl = rays.type ? (__ldg(rays.type + i) == 32) : false;
	unsigned err;
	{
		TravMem<F> mem;
		Trav<F, StreamIO> tr;
		tr.mem = &mem;
		tr.io.rays = &rays;
		tr.io.rec = &rec;
		tr.io.path = &path;
		tr.io.i = i;
		tr.init(sc, wr.o, wr.d, wr.time, wr.occl);
		tr.walk(sc);
		err = tr.err;
	}
	const bool hit = rec.inst >= 0;
	if (hits.hit) hits.hit[i] = hit ? 1 : 0;
	if (hits.id) hits.id[i] = hit ? hit_id(sc, rec, path) : 0ull;
	if (hits.t) hits.t[i] = (hit && !wr.occl) ? rec.t : INFINITY;
	if (hit && !wr.occl && hits.want_geometry) hit_surface(sc, &rec, path);
	if (hit && !wr.occl && hits.want_geometry == WANT_UV && (rec.kind == OBJ_BILINEAR || rec.kind == OBJ_BICUBIC)) {
		// a patch's u, v are the bisection's own: no geometry to evaluate
		hits.uv[2 * (size_t)i] = rec.u;
		hits.uv[2 * (size_t)i + 1] = rec.v;
	} else if (hit && !wr.occl && hits.want_geometry) {
		M44 space;
		const bool xf = hit_space<F>(sc, rec, path, wr.time, &space, &err);
		V3 lo = wr.o, ld = wr.d;
		if (xf) {
			lo = pos_to(space, wr.o);
			ld = dir_to(space, wr.d);
		} else {
			space = m44_identity();
		}
		HitInfo h;
		hit_geometry<true>(sc, rec, wr.time, lo, ld, hits.want_geometry != WANT_POINT, &h);
		if (hits.uv) {
			hits.uv[2 * (size_t)i] = h.geo.u;
			hits.uv[2 * (size_t)i + 1] = h.geo.v;
		}
		if (hits.p) st3(hits.p, i, h.geo.p);
		if (hits.n) st3(hits.n, i, h.geo.n);
		if (hits.dpdu) st3(hits.dpdu, i, h.geo.dpdu);
		if (hits.dpdv) st3(hits.dpdv, i, h.geo.dpdv);
		if (hits.dndu) st3(hits.dndu, i, h.geo.dndu);
		if (hits.dndv) st3(hits.dndv, i, h.geo.dndv);
		if (hits.backfacing) hits.backfacing[i] = h.backfacing ? 1 : 0;
		if (hits.light_pdf) hits.light_pdf[i] = h.light_pdf;
		if (hits.offset) st3(hits.offset, i, h.offset);
		if (hits.space)
			for (int k = 0; k < 16; ++k) hits.space[16 * (size_t)i + k] = space.m[k / 4][k % 4];
		if (hits.closure) hits.closure[i] = (uint8_t)h.closure;
		if (hits.closure_color) {
			hits.closure_color[3 * (size_t)i] = h.col[0];
			hits.closure_color[3 * (size_t)i + 1] = h.col[1];
			hits.closure_color[3 * (size_t)i + 2] = h.col[2];
		}
	} else if (hits.want_geometry) {
		if (hits.uv) {
			hits.uv[2 * (size_t)i] = 0.0f;
			hits.uv[2 * (size_t)i + 1] = 0.0f;
		}
		const V3 z(0.0f);
		if (hits.p) st3(hits.p, i, z);
		if (hits.n) st3(hits.n, i, z);
		if (hits.dpdu) st3(hits.dpdu, i, z);
		if (hits.dpdv) st3(hits.dpdv, i, z);
		if (hits.dndu) st3(hits.dndu, i, z);
		if (hits.dndv) st3(hits.dndv, i, z);
		if (hits.backfacing) hits.backfacing[i] = 0;
		if (hits.light_pdf) hits.light_pdf[i] = 9999.0f;
		if (hits.offset) st3(hits.offset, i, z);
		if (hits.space)
			for (int k = 0; k < 16; ++k) hits.space[16 * (size_t)i + k] = (k % 5 == 0) ? 1.0f : 0.0f;
		if (hits.closure) hits.closure[i] = 0;
		if (hits.closure_color) st3(hits.closure_color, i, z);
	}
	if (err) atomicOr(status, err);
}

cudaError_t launch_trace(const DevScene& sc, const RaySoA& rays, const HitSoA& hits, uint32_t n, unsigned* status,
                         cudaStream_t stream) {
	if (n == 0) return cudaSuccess;
	// A short stream is spread over the SMs, and its warps run on fewer lanes,
	// whose rays wait less for one another: at least 8 warps an SM as long as
	// there are rays (1021 rays against a flat scene: 51 us in 8 blocks of 128
	// threads, 20 so; 148 SMs).
	const int block = 128;
	const uint32_t warps = 8 * 148;
	int lanes = 32;
	while (lanes > 1 && n / (uint32_t)lanes < warps) lanes >>= 1;
	const uint32_t grid = (uint32_t)((((uint64_t)n + lanes - 1) / lanes * 32 + block - 1) / block);
	switch (feature_variant(sc.features)) {
		case FEAT_FLAT: trace_kernel<FEAT_FLAT><<<grid, block, 0, stream>>>(sc, rays, hits, n, lanes, status); break;
		case FEAT_STILL_BICUBIC: trace_kernel<FEAT_STILL_BICUBIC><<<grid, block, 0, stream>>>(sc, rays, hits, n, lanes, status); break;
		case FEAT_STILL: trace_kernel<FEAT_STILL><<<grid, block, 0, stream>>>(sc, rays, hits, n, lanes, status); break;
		default: trace_kernel<FEAT_ALL><<<grid, block, 0, stream>>>(sc, rays, hits, n, lanes, status); break;
	}
	return cudaGetLastError();
}

}  // namespace psy
