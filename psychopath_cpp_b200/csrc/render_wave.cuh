/*
 * Wavefront path tracer: PathTraceIntegrator::integrate restated for the
 * GPU (reference integrator/path_trace_integrator.cpp:91-384).
 *
 * The reference renders a bucket as a stream of paths and loops
 *   generate one ray per live path -> Tracer::trace -> update -> partition.
 * Here a wave of paths lives in HBM as SoA state and the loop is split into
 * kernels that each do one kind of work, so the traversal kernel carries no
 * shading state and the shading kernel no traversal state:
 *
 *   camera_gen   camera rays of every path of the wave
 *   trace        Tracer::trace of the closest-hit rays and of the shadow rays
 *                of the last vertex, in one launch
 *   shade        update_path with both results, then next_ray_for_path's two
 *                steps at the new vertex: light sample with its shadow ray,
 *                and the bounce ray; live paths are compacted into the next
 *                queue (ballot + popc, one atomic per warp)
 *   ... trace -> shade for path_length vertices, then the last shadow rays
 *   finish       their results, every sample's spectrum to XYZ, film sums
 *
 * The reference traces the shadow ray before it generates the bounce ray;
 * the bounce does not depend on the result (only the path's radiance does,
 * which is added to in the same order here), so both leave a vertex together
 * and nothing of the vertex is stored.  (As kernels of their own, hit and
 * shadow shading wrote and read 176 bytes of vertex a path and step, and a
 * small frame waited for twice as many launches: 80x60 preview 525 -> 443 us,
 * 320x240x16 render 2.55 -> 2.25 ms.)
 *
 * Rays and hits are stored by queue position (coalesced), path state by path
 * slot.  Finished paths leave their spectrum in the path state; a per-wave
 * reduction adds each pixel's samples (Color_XYZ(col) * XYZ_NORM_FAC) in
 * sample order.
 *
 * The same kernels serve two modes.  PlainWave renders one scene and takes
 * the scene and render parameters as kernel parameters.  BatchWave renders
 * many scenes at once: a wave covers consecutive global paths of several
 * renders, each path carries its render index, and scenes and parameters
 * are read from device arrays.
 *
 * Each (mode, feature variant) pair is compiled in a file of its own
 * (render_*.cu); render.cu picks the variant of a scene.
 */
#ifndef PSY_RENDER_WAVE_CUH
#define PSY_RENDER_WAVE_CUH

#include "kernels.h"
#include "render_device.cuh"

namespace psy {

__device__ __forceinline__ float4 f4(const Spec& s) { return make_float4(s.e[0], s.e[1], s.e[2], s.e[3]); }
__device__ __forceinline__ Spec sp(float4 v) {
	Spec s;
	s.e[0] = v.x; s.e[1] = v.y; s.e[2] = v.z; s.e[3] = v.w;
	return s;
}

// ---------------------------------------------------------------------
// Ray and hit records by queue position
// ---------------------------------------------------------------------
// Ray planes (5 x float4 per position):
//   0: o.xyz, time   1: d.xyz, odx.x   2: odx.yz, ody.xy   3: ody.z, ddx.xyz
//   4: ddy.xyz, tag = render index << 1 | 1 when there is no ray (the shadow
//      step found no light sample)
__device__ __forceinline__ void store_ray(float4* rb, int cap, int i, const WorldRayD& r, int tag) {
	rb[i] = make_float4(r.o.x, r.o.y, r.o.z, r.time);
	rb[cap + i] = make_float4(r.d.x, r.d.y, r.d.z, r.odx.x);
	rb[2 * cap + i] = make_float4(r.odx.y, r.odx.z, r.ody.x, r.ody.y);
	rb[3 * cap + i] = make_float4(r.ody.z, r.ddx.x, r.ddx.y, r.ddx.z);
	rb[4 * cap + i] = make_float4(r.ddy.x, r.ddy.y, r.ddy.z, __int_as_float(tag));
}
__device__ __forceinline__ int load_ray(const float4* rb, int cap, int i, WorldRayD* r) {
	const float4 a = rb[i], b = rb[cap + i], c = rb[2 * cap + i], d = rb[3 * cap + i], e = rb[4 * cap + i];
	r->o = V3(a.x, a.y, a.z);
	r->time = a.w;
	r->d = V3(b.x, b.y, b.z);
	r->odx = V3(b.w, c.x, c.y);
	r->ody = V3(c.z, c.w, d.x);
	r->ddx = V3(d.y, d.z, d.w);
	r->ddy = V3(e.x, e.y, e.z);
	return __float_as_int(e.w);
}

// Hit planes: 0: t, u, v, max_dim (float4)   1: instance, placement, depth,
// path[0]   2: path[1..4]   3: path[5..7] (int4).  The path is written and
// read in scenes without placements only, as far as the hit's depth.
__device__ __forceinline__ void load_rec(const WaveBufs& wb, int i, int4 a, float4 f, HitRec* h, HitPath* hp) {
	h->inst = a.x;
	if (a.x < 0) return;
	h->t = f.x; h->u = f.y; h->v = f.z; h->max_dim = f.w;
	h->place = a.y;
	hp->depth = 0;
	if (a.y >= 0) return;
	hp->depth = a.z;
	hp->path[0] = a.w;
	const int cap = wb.cap;
	if (hp->depth > 1) {
		const int4 b = wb.hit_i[cap + i];
		hp->path[1] = b.x; hp->path[2] = b.y; hp->path[3] = b.z; hp->path[4] = b.w;
	}
	if (hp->depth > 5) {
		const int4 c = wb.hit_i[2 * cap + i];
		hp->path[5] = c.x; hp->path[6] = c.y; hp->path[7] = c.z;
	}
}

// A ray of the wave's queue (Trav's IO).  Hits go straight to the ray's
// place in the hit planes: a lane carries nothing of them.
struct WaveIO {
	const float4* rb;
	const WaveBufs* wb;
	int i;  // queue position, -1 = no ray
	__device__ __forceinline__ V3 origin() const {
		const float4 a = rb[i];
		return V3(a.x, a.y, a.z);
	}
	__device__ __forceinline__ V3 direction() const {
		const float4 b = rb[wb->cap + i];
		return V3(b.x, b.y, b.z);
	}
	__device__ __forceinline__ void differentials(V3* odx, V3* ody, V3* ddx, V3* ddy) const {
		WorldRayD r;
		load_ray(rb, wb->cap, i, &r);
		*odx = r.odx;
		*ody = r.ody;
		*ddx = r.ddx;
		*ddy = r.ddy;
	}
	template <class T>
	__device__ __forceinline__ void hit(const T& tr, int inst, float t, float u, float v, float md) const {
		if (tr.flags & RAY_OCCL) return;
		wb->hit_f[i] = make_float4(t, u, v, md);
		if (!T::NESTED || tr.place >= 0) {
			wb->hit_i[i] = make_int4(inst, tr.place, 0, 0);
			return;
		}
		int p[PSY_MAX_LEVELS] = {};
		for (int k = 1; k <= tr.L; ++k) p[k - 1] = tr.mem->lv_inst[k];
		p[tr.L] = inst;
		const int cap = wb->cap;
		wb->hit_i[i] = make_int4(inst, -1, tr.L + 1, p[0]);
		if (tr.L > 0) wb->hit_i[cap + i] = make_int4(p[1], p[2], p[3], p[4]);
		if (tr.L > 4) wb->hit_i[2 * cap + i] = make_int4(p[5], p[6], p[7], 0);
	}
};

// World-space shading data of a path vertex (the PTState::inter and prev_ray
// of the reference).
struct Vertex {
	V3 p, n, off;       // geo.p, geo.n (after transformed_from), signed ray-origin offset
	V3 d;               // direction of the ray that met it
	V3 odx, ody;        // that ray's origin differentials transferred to the hit
	float bf;           // 1 when the hit was back-facing
	float col[3];       // closure colour (Lambert)
	int pid;            // differentiable renders: the shader's first albedo weight (>= 0), -2 - q when its
	                    // RGB albedo is scaled by params[q], or -1 (not parameterised)
	int gtr;            // the GTR shader of the hit, or -1 (Lambert)
};
// What the GTR closure reads besides: geo's derivatives in world space
// (transformed_from) and the direction differentials of the ray.
struct GtrVertex {
	V3 ddx, ddy, dpdu, dpdv, dndu, dndv;
};

// Intersection -> vertex: DifferentialGeometry::transformed_from(space)
// (basics/differential_geometry.hpp:20-40), the offset of
// path_trace_integrator.cpp:141-145 and the transferred differentials of
// propagate_differentials.
template <unsigned F, bool GTR>
__device__ __forceinline__ void make_vertex(const DevScene& sc, const HitRec& rec, const HitPath& path, const WorldRayD& wr, float ident_inv,
                                            Vertex* sh, GtrVertex* gv, int* closure, float* light_pdf, unsigned* err) {
	M44 space;
	const bool xf = hit_space<F>(sc, rec, path, wr.time, &space, err);
	V3 lo = wr.o, ld = wr.d;
	if (xf) {
		lo = pos_to(space, wr.o);
		ld = dir_to(space, wr.d);
	}
	HitInfo h;
	hit_geometry<GTR>(sc, rec, wr.time, lo, ld, false, &h);
	*closure = h.closure;
	sh->col[0] = h.col[0]; sh->col[1] = h.col[1]; sh->col[2] = h.col[2];
	*light_pdf = h.light_pdf;
	if (h.closure != CLOSURE_LAMBERT && !(GTR && h.closure == CLOSURE_GTR)) return;
	M44 inv;
	if (xf) {
		inv = m44_inverse_dev(space, sc.rcp);
	} else {
		inv = m44_identity();
		for (int i = 0; i < 4; ++i) inv.m[i][i] = ident_inv;
	}
	sh->p = pos_to(inv, h.geo.p);
	const M44 nx = xf ? space : m44_identity();
	const V3 n = nor_from(nx, h.geo.n);
	const float il = 1.0f / length(n);
	sh->n = n * il;
	sh->gtr = -1;
	if (GTR && h.closure == CLOSURE_GTR) {
		// the rest of DifferentialGeometry::transformed_from (basics/differential_geometry.hpp:20-40)
		sh->gtr = rec.shader;
		gv->dpdu = dir_to(inv, h.geo.dpdu);
		gv->dpdv = dir_to(inv, h.geo.dpdv);
		gv->dndu = nor_from(nx, h.geo.dndu) * il;
		gv->dndv = nor_from(nx, h.geo.dndv) * il;
		gv->ddx = wr.ddx;
		gv->ddy = wr.ddy;
	}
	V3 off = dir_to(inv, h.offset);
	if (h.backfacing) off = off * -1.0f;
	sh->off = off;
	sh->bf = h.backfacing ? 1.0f : 0.0f;
	sh->d = wr.d;
	const V3 nn = normalized(sh->n);
	sh->odx = transfer_origin_differential(rec.t, nn, wr.d, wr.odx, wr.ddx);
	sh->ody = transfer_origin_differential(rec.t, nn, wr.d, wr.ody, wr.ddy);
}

// The outgoing ray's differentials (LambertClosure::propagate_differentials,
// shading/surface_closure.hpp:306-320).
__device__ __forceinline__ void propagate_differentials(const Vertex& h, WorldRayD* out) {
	const float len = length(out->d);
	V3 x, y;
	coordinate_system(out->d, &x, &y);
	x = normalized(x);
	y = normalized(y);
	out->odx = h.odx;
	out->ody = h.ody;
	out->ddx = (x * 0.15f) / len;
	out->ddy = (y * 0.15f) / len;
}

// GTRClosure::propagate_differentials (shading/surface_closure.hpp:574-607):
// origin differentials transferred to the hit, normal differentials turned
// into half-vector differentials, direction differentials reflected about
// the half vector, then clamped (clamp_dd).
static __device__ __noinline__ void gtr_direction_differentials(const GtrVertex& g, V3 n, V3 d, V3 odx, V3 ody, V3 out,
                                                                V3* oddx, V3* oddy) {
	V3 nn = normalized(n);
	const V3 hh = normalized(normalized(d * -1.0f) + normalized(out));
	float dux, dvx, duy, dvy;
	uv_differentials(odx, g.dpdu, g.dpdv, &dux, &dvx);
	uv_differentials(ody, g.dpdu, g.dpdv, &duy, &dvy);
	V3 dndx = (g.dndu * dux) + (g.dndv * dvx);
	V3 dndy = (g.dndu * duy) + (g.dndv * dvy);
	if (dot(nn, hh) < 0.0f) {
		nn = nn * -1.0f;
		dndx = dndx * -1.0f;
		dndy = dndy * -1.0f;
	}
	const V3 axis = normalized(cross(nn, hh));
	const float angle = lm_acosf(clampf(dot(nn, hh), 0.0f, 1.0f));
	const M44 xf = axis_angle(axis, angle);
	const V3 dhdx = dir_to(xf, dndx);
	const V3 dhdy = dir_to(xf, dndy);
	V3 ddx = reflect_dd(hh, dhdx, d, g.ddx);
	V3 ddy = reflect_dd(hh, dhdy, d, g.ddy);
	const float len_d = length(out);
	const float len_dx = length(ddx);
	const float len_dy = length(ddy);
	if ((len_dx / len_d) > 0.9f) ddx = ddx * ((0.9f * len_d) / len_dx);
	if ((len_dy / len_d) > 0.9f) ddy = ddy * ((0.9f * len_d) / len_dy);
	*oddx = ddx;
	*oddy = ddy;
}
__device__ __forceinline__ void gtr_propagate_differentials(const Vertex& h, const GtrVertex& g, WorldRayD* out) {
	out->odx = h.odx;
	out->ody = h.ody;
	gtr_direction_differentials(g, h.n, h.d, h.odx, h.ody, out->d, &out->ddx, &out->ddy);
}

// ---------------------------------------------------------------------
// Wave modes: where a kernel finds the scene and parameters of render r
// ---------------------------------------------------------------------
struct PlainWave {
	static constexpr bool BATCH = false;
	DevScene sc;
	RenderParams rp;
	__device__ __forceinline__ const DevScene& scene(int) const { return sc; }
	__device__ __forceinline__ const RenderParams& render(int) const { return rp; }
	__device__ __forceinline__ int render_of_path(uint64_t) const { return 0; }
	__device__ __forceinline__ int render_of_pixel(uint64_t) const { return 0; }
};

struct BatchWave {
	static constexpr bool BATCH = true;
	const DevScene* scenes;
	const RenderParams* renders;
	int count;
	__device__ __forceinline__ const DevScene& scene(int r) const { return scenes[r]; }
	__device__ __forceinline__ const RenderParams& render(int r) const { return renders[r]; }
	// the last render whose first path (pixel) is at or before g
	__device__ __forceinline__ int render_of_path(uint64_t g) const {
		int lo = 0, hi = count - 1;
		while (lo < hi) {
			const int mid = (lo + hi + 1) >> 1;
			if (renders[mid].path_base <= g) lo = mid; else hi = mid - 1;
		}
		return lo;
	}
	__device__ __forceinline__ int render_of_pixel(uint64_t q) const {
		int lo = 0, hi = count - 1;
		while (lo < hi) {
			const int mid = (lo + hi + 1) >> 1;
			if (renders[mid].pixel_base <= q) lo = mid; else hi = mid - 1;
		}
		return lo;
	}
};

// ---------------------------------------------------------------------
// Differentiable rendering (no reference counterpart)
// ---------------------------------------------------------------------
// Emission scale parameter of object `obj`, or -1.
__device__ __forceinline__ int emission_param(const RenderParams& rp, int obj) {
	return (rp.params && obj >= 0) ? rp.object_param[obj] : -1;
}

// lambert_eval with the albedo taken from parameters when the stored hit's
// shader has them.
__device__ __forceinline__ Spec lambert_eval_p(const RenderParams& rp, const Vertex& sh, V3 out, float wl) {
	if (sh.pid == -1) return lambert_eval(sh.col, sh.d, out, sh.n, wl);
	if (sh.pid < -1) {
		Spec f = lambert_eval(sh.col, sh.d, out, sh.n, wl);
		const float q = rp.params[-2 - sh.pid];
		for (int k = 0; k < 4; ++k) f.e[k] *= q;
		return f;
	}
	const float c = lambert_cos(sh.d, out, sh.n);
	const Spec a = albedo_spec(rp.params + sh.pid, wl);
	Spec f;
	for (int k = 0; k < 4; ++k) f.e[k] = c * a.e[k];
	return f;
}

// Adjoint: adds u . dC/dparams for a radiance contribution C (hero
// wavelengths) whose albedo factors come from vertices 0..nv-1 of the path
// and whose emission is scaled by params[lp] (lp < 0: none).  C is the
// product of B (the contribution with every parameterised albedo and the
// emission scale left out), the parameterised vertices' albedos (each
// linear in its four weights) and the scale, so the derivative for one
// factor is the product of all the others: no division, so a factor that
// is zero (a black albedo, a light scaled to 0) still gets its gradient.
static __device__ void grad_add(const RenderParams& rp, float* sg, const PathSoA& ps, int slot, int nv, const Spec& B,
                         int lp, float wl) {
	const float4 u4 = ps.adj[slot];
	const float ub[4] = {u4.x * B.e[0], u4.y * B.e[1], u4.z * B.e[2], u4.w * B.e[3]};
	auto add = [&](int k, float v) {
		if (rp.grad_in_smem == GRAD_SMEM64) atomicAdd(reinterpret_cast<double*>(sg) + k, (double)v);
		else atomicAdd((rp.grad_in_smem ? sg : rp.grad) + k, v);
	};
	const float scale = lp >= 0 ? rp.params[lp] : 1.0f;
	if (nv > PSY_ADJ_MAX_VERTS) nv = PSY_ADJ_MAX_VERTS;
	float a[PSY_ADJ_MAX_VERTS][4];
	int pid[PSY_ADJ_MAX_VERTS];
	for (int v = 0; v < nv; ++v) {
		pid[v] = ps.vpid[slot * PSY_ADJ_MAX_VERTS + v];
		const float4 a4 = ps.valb[slot * PSY_ADJ_MAX_VERTS + v];
		a[v][0] = a4.x; a[v][1] = a4.y; a[v][2] = a4.z; a[v][3] = a4.w;
	}
	if (lp >= 0) {
		float d = 0.0f;
		for (int j = 0; j < 4; ++j) {
			float q = ub[j];
			for (int v = 0; v < nv; ++v)
				if (pid[v] != -1) q *= a[v][j];
			d += q;
		}
		add(lp, d);
	}
	for (int v = 0; v < nv; ++v) {
		if (pid[v] == -1) continue;
		float q[4];
		for (int j = 0; j < 4; ++j) {
			q[j] = ub[j] * scale;
			for (int o = 0; o < nv; ++o)
				if (o != v && pid[o] != -1) q[j] *= a[o][j];
		}
		if (pid[v] < -1) {
			// scaled RGB albedo: its derivative is the upsampled colour
			const float4 u = ps.vdsc[slot * PSY_ADJ_MAX_VERTS + v];
			add(-2 - pid[v], ((q[0] * u.x + q[1] * u.y) + q[2] * u.z) + q[3] * u.w);
			continue;
		}
		for (int k = 0; k < 4; ++k) {
			float d = 0.0f;
			for (int j = 0; j < 4; ++j) d += q[j] * albedo_basis(k, wavelength_n(wl, j));
			add(pid[v] + k, d);
		}
	}
}

// Per-block gradient accumulators: cleared at kernel start, added to the
// global gradient at the end.
__device__ __forceinline__ void grad_begin(const RenderParams& rp, float* sg) {
	if (!rp.grad || !rp.grad_in_smem) return;
	const int words = rp.param_count * (rp.grad_in_smem == GRAD_SMEM64 ? 2 : 1);
	for (int i = threadIdx.x; i < words; i += blockDim.x) sg[i] = 0.0f;
	__syncthreads();
}
__device__ __forceinline__ void grad_end(const RenderParams& rp, float* sg) {
	if (!rp.grad || !rp.grad_in_smem) return;
	__syncthreads();
	for (int i = threadIdx.x; i < rp.param_count; i += blockDim.x) {
		const float v = rp.grad_in_smem == GRAD_SMEM64 ? (float)reinterpret_cast<double*>(sg)[i] : sg[i];
		if (v != 0.0f) atomicAdd(rp.grad + i, v);
	}
}

// ---------------------------------------------------------------------
// Camera rays (next_ray_for_path, step 0: path_trace_integrator.cpp:109-125)
// ---------------------------------------------------------------------
template <class W>
__global__ void __launch_bounds__(256) camera_gen_kernel(W w, HaltonDev hd, WaveRange wv, PathSoA ps, WaveBufs wb) {
	const int slot = blockIdx.x * blockDim.x + threadIdx.x;
	if (slot >= wv.paths) return;
	const uint64_t gidx = wv.base + (uint64_t)slot;
	const int rid = w.render_of_path(gidx);
	const RenderParams& rp = w.render(rid);
	const uint64_t local = gidx - rp.path_base;
	const uint64_t pixel = local / rp.spp;
	const uint32_t px = (uint32_t)(pixel % rp.width);
	const uint32_t py = (uint32_t)(pixel / rp.width);
	const uint32_t s = (uint32_t)(local % rp.spp);
	const uint32_t smp = sampler_offset(px, py, s, rp.seed);
	uint32_t dim = 0;
	const float wl = (sampler_get(hd, smp, dim++) * (WAVELENGTH_MAX - WAVELENGTH_MIN)) + WAVELENGTH_MIN;
	const float samp_x = (fast_logit(sampler_get(hd, smp, dim++), 1.5f) + 0.5f + (float)px) / (float)rp.width;
	const float samp_y = (fast_logit(sampler_get(hd, smp, dim++), 1.5f) + 0.5f + (float)py) / (float)rp.height;
	const float rx = (float)(((double)samp_x - 0.5) * (double)(rp.max_x - rp.min_x));
	const float ry = (float)((0.5 - (double)samp_y) * (double)(rp.max_y - rp.min_y));
	const float dx = (rp.max_x - rp.min_x) / (float)rp.width;
	const float dy = (rp.max_y - rp.min_y) / (float)rp.height;
	const float samp_a = sampler_get(hd, smp, dim++);
	const float samp_b = sampler_get(hd, smp, dim++);
	const float samp_c = sampler_get(hd, smp, dim++);
	WorldRayD wr;
	camera_ray(w.scene(rid), rx, ry, dx, dy, samp_c, samp_a, samp_b, &wr);
	store_ray(wb.ray[0], wb.cap, slot, wr, rid << 1);
	ps.head[slot] = make_uint4(smp, dim, __float_as_uint(wl), __float_as_uint(0.0f));  // step 0
	if (!W::BATCH && rp.dl_dxyz) {
		// d(film sum)/d(col) of finish_path: XYZ_NORM_FAC / 4 * CIE(lambda_j)
		const float* g = rp.dl_dxyz + 3 * pixel;
		float u[4];
		for (int j = 0; j < 4; ++j) {
			const float lw = wavelength_n(wl, j);
			u[j] = ((g[0] * X_1931(lw) + g[1] * Y_1931(lw)) + g[2] * Z_1931(lw)) * (0.25f * XYZ_NORM_FAC);
		}
		ps.adj[slot] = make_float4(u[0], u[1], u[2], u[3]);
		ps.fexcl[slot] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
	}
}

// ---------------------------------------------------------------------
// Traversal of a ray buffer (Tracer::trace, tracer/tracer.cpp:38-121)
// ---------------------------------------------------------------------
// `parts`: TRACE_CLOSEST, TRACE_OCCL or both, n rays each (n_dev == nullptr:
// n_host), the closest-hit rays first.  A shadow ray's result (1 = blocked or
// no ray) goes to wb.occl by position.
//
// Persistent warps with per-lane ray replacement: a lane whose ray is
// finished takes the next ray of the queue between traversal steps instead
// of idling until the slowest ray of its warp is done.
//
// Registers: 128 a thread where a lane's step can be a bicubic split (96
// floats live); there more warps only push one another's stacks and cursors
// out of L1 (1280x720x4 many-light frame: 114.3 ms with 2 x 256 threads an
// SM, 121.7 with 5 x 128, 127.4 with 3 x 192, 130.6 with 3 x 256).  80 in flat
// scenes, where more warps hide the walk's latency (512x384x16 with 50,000
// primitives: 10.49 ms with 3 x 256, 10.62 with 4, 10.97 with 2).
// Idle lanes that trigger a refill: 2 of them 118.3 ms, 4 114.3, 8 109.2
// (instanced); 4 11.04, 8 10.70, 12 10.49 (flat).
template <unsigned F>
struct TraceCfg {
	static constexpr bool NESTED = (F & FEAT_NESTED) != 0;
	static constexpr int BLOCK = 256;                     // launch bound
	static constexpr int MIN_BLOCKS = NESTED ? 2 : 3;     // 128 and 80 registers a thread
	static constexpr int REFILL_MIN = NESTED ? 4 : 12;    // idle lanes that trigger a refill while rays remain
	static int launch_block(int render_block) { return NESTED ? BLOCK : render_block; }
};
// Each lane's traversal is cut into kinds of work: node visits (up to
// PSY_WALK_NODES at a time, stopping at a leaf), leaf visits of three
// classes (entering an assembly instance, testing a simple object, starting
// a patch bisection) and bisection iterations (PSY_PATCH_UNITS at a time).
// Each loop iteration of a warp runs the kind that most of its lanes have
// next, so that the lanes doing the same work run together instead of one
// lane's long bisection or transformed-instance entry holding up the others.
// (2, 4 or 8 node visits: within 1%; 16 bisection iterations: 2% better than
// 8 on the many-light frame, 32 another 1% in flat scenes.  Warps that follow one kind of work per block,
// which paid while a step's code and state did not fit the caches, cost 5%.)
#ifndef PSY_WALK_NODES
#define PSY_WALK_NODES 4
#endif
#ifndef PSY_PATCH_UNITS
#define PSY_PATCH_UNITS 32
#endif
// Kinds of work of a lane: idle, inner nodes, a leaf visit of one of three
// classes, a bisection in progress.  Leaf visits are told apart so that the
// lanes of a warp step run one branch together: assembly entries (ray
// transform), simple objects (spheres, sphere and rectangle lights), patches
// (root box, ray widths, bisection set-up).
enum : int { KIND_IDLE = 0, KIND_NODES, KIND_ENTER, KIND_SIMPLE, KIND_BEGIN, KIND_PATCH, KIND_COUNT };

enum : unsigned { TRACE_CLOSEST = 1u, TRACE_OCCL = 2u };

template <class W, unsigned F>
__global__ void __launch_bounds__(TraceCfg<F>::BLOCK, TraceCfg<F>::MIN_BLOCKS)
    trace_wave_kernel(W w, WaveBufs wb, const float4* __restrict__ rc, const float4* __restrict__ ro, const int* n_dev,
                      int n_host, unsigned parts, int* work, unsigned long long* counts, unsigned* status) {
	const int n = n_dev ? *n_dev : n_host;
	const int nc = (parts & TRACE_CLOSEST) ? n : 0;
	const unsigned total = (unsigned)nc + ((parts & TRACE_OCCL) ? (unsigned)n : 0u);
	// traversal counters of the block: closest-hit rays, occlusion rays
	__shared__ unsigned long long s_counts[2 * TC_COUNT];
	if (threadIdx.x < 2 * TC_COUNT) s_counts[threadIdx.x] = 0ull;
	__syncthreads();
	const int lane = threadIdx.x & 31;
	const unsigned lt_mask = (1u << lane) - 1u;
	unsigned err = 0;
	// per-lane work counters (TC_*), and the warp's own (lane 0 keeps them)
	unsigned rays = 0, c_nodes = 0, c_leaves = 0, c_iters = 0, c_warp = 0, c_lanes = 0;
	bool c_occl = nc == 0, w_occl = nc == 0;  // the kind of ray they are of
	auto flush = [&]() {
		unsigned long long* c = s_counts + (c_occl ? TC_COUNT : 0);
		if (rays) atomicAdd(c + TC_RAYS, (unsigned long long)rays);
		if (c_nodes) atomicAdd(c + TC_NODES, (unsigned long long)c_nodes);
		if (c_leaves) atomicAdd(c + TC_LEAVES, (unsigned long long)c_leaves);
		if (c_iters) atomicAdd(c + TC_PATCH_ITERS, (unsigned long long)c_iters);
		rays = c_nodes = c_leaves = c_iters = 0;
	};
	auto flush_warp = [&]() {
		unsigned long long* c = s_counts + (w_occl ? TC_COUNT : 0);
		if (lane == 0 && c_warp) {
			atomicAdd(c + TC_WARP_STEPS, (unsigned long long)c_warp);
			atomicAdd(c + TC_LANE_STEPS, (unsigned long long)c_lanes);
		}
		c_warp = c_lanes = 0;
	};
	TravMem<F> mem;
	Trav<F, WaveIO> tr;
	tr.mem = &mem;
	tr.io.rb = rc;
	tr.io.wb = &wb;
	tr.io.i = -1;
	tr.pmode = PM_NONE;
	tr.cur = REF_NONE;
	int rid = 0;
	bool more = true;  // the queue may still hold rays (warp-uniform)
	// a queue too short to fill every lane is spread over all warps: each
	// runs on fewer lanes, whose rays wait less for one another
	const unsigned warps = gridDim.x * (blockDim.x >> 5);
	const unsigned per = (total + warps - 1) / warps;
	const unsigned use = per < 32u ? (1u << per) - 1u : 0xffffffffu;
	const int refill = min(TraceCfg<F>::REFILL_MIN, __popc(use));
	while (true) {
		const unsigned idle = __ballot_sync(0xffffffffu, tr.io.i < 0) & use;
		if (more && (__popc(idle) >= refill || idle == use)) {
			unsigned base = 0;
			if (lane == 0) base = (unsigned)atomicAdd(work, __popc(idle));
			base = __shfl_sync(0xffffffffu, base, 0);
			if (base + __popc(idle) >= total) more = false;
			if (!w_occl && base >= (unsigned)nc) {
				flush_warp();
				w_occl = true;
			}
			if (tr.io.i < 0 && ((use >> lane) & 1u)) {
				const unsigned q = base + __popc(idle & lt_mask);
				if (q < total) {
					const bool occl = q >= (unsigned)nc;
					const int k = (int)(occl ? q - (unsigned)nc : q);
					const float4* rb = occl ? ro : rc;
					if (occl != c_occl) {
						flush();
						c_occl = occl;
					}
					const int tag = __float_as_int(rb[4 * (size_t)wb.cap + k].w);
					if (tag & 1) {
						// no ray: a shadow step without a light sample, or the
						// last vertex of a path
						if (occl) wb.occl[k] = 1;
					} else {
						rid = tag >> 1;
						tr.io.rb = rb;
						tr.io.i = k;
						const float4 a = rb[k], b = rb[(size_t)wb.cap + k];
						tr.init(w.scene(rid), V3(a.x, a.y, a.z), V3(b.x, b.y, b.z), a.w, occl);
						++rays;
						if (tr.cur == REF_EMPTY) {
							// an empty scene
							if (occl) wb.occl[k] = 0;
							else wb.hit_i[k] = make_int4(-1, 0, 0, 0);
							tr.io.i = -1;
						}
					}
				}
			}
		}
		// KIND_IDLE, KIND_NODES (inner nodes), a leaf visit of one of three
		// kinds, or KIND_PATCH (bisection)
		int kind = KIND_IDLE;
		if (tr.io.i >= 0) {
			const int cls = leaf_class(tr.cur);
			kind = tr.pmode != PM_NONE ? KIND_PATCH : tr.cur >= 0 ? KIND_NODES
			     : cls == LEAF_ENTER ? KIND_ENTER : cls == LEAF_PATCH ? KIND_BEGIN : KIND_SIMPLE;
		}
		unsigned m[KIND_COUNT];
#pragma unroll
		for (int k = KIND_NODES; k < KIND_COUNT; ++k) m[k] = __ballot_sync(0xffffffffu, kind == k);
		if ((m[KIND_NODES] | m[KIND_ENTER] | m[KIND_SIMPLE] | m[KIND_BEGIN] | m[KIND_PATCH]) == 0u) {
			if (!more) break;
			continue;
		}
		// the kind most of the lanes have next (later kinds win ties)
		int run = KIND_NODES;
		int best = __popc(m[KIND_NODES]);
#pragma unroll
		for (int k = KIND_ENTER; k < KIND_COUNT; ++k) {
			const int c = __popc(m[k]);
			if (c >= best && c > 0) {
				best = c;
				run = k;
			}
		}
		++c_warp;
		c_lanes += best;
		if (kind == run) {
			const DevScene& sc = w.scene(rid);
			bool live = true;
			if (run == KIND_NODES) {
#pragma unroll 1
				for (int k = 0; k < PSY_WALK_NODES; ++k) {
					++c_nodes;
					live = tr.node_step(sc) && tr.pop(sc);
					if (!live || tr.cur < 0) break;
				}
			} else {
				if (run == KIND_PATCH) {
					int left = PSY_PATCH_UNITS;
					live = tr.patch_step(sc, left);
					c_iters += PSY_PATCH_UNITS - left;
				} else {
					++c_leaves;
					if (TraceCfg<F>::NESTED && run == KIND_ENTER) live = tr.enter(sc);
					else if ((F & (FEAT_BILINEAR | FEAT_BICUBIC)) && run == KIND_BEGIN) live = tr.template patch_leaf<false>(sc);
					else live = leaf_class(tr.cur) == LEAF_SPHERE ? tr.sphere_leaf(sc) : tr.simple_leaf(sc);
				}
				if (live && tr.pmode == PM_NONE) live = tr.pop(sc);
			}
			if (!live) {
				err |= tr.err;
				if (tr.flags & RAY_OCCL) wb.occl[tr.io.i] = (tr.flags & RAY_HIT) ? 1 : 0;
				else if (!(tr.flags & RAY_HIT)) wb.hit_i[tr.io.i] = make_int4(-1, 0, 0, 0);
				tr.io.i = -1;
			}
		}
	}
	flush();
	flush_warp();
	__syncthreads();
	if (threadIdx.x < 2 * TC_COUNT && s_counts[threadIdx.x]) atomicAdd(counts + threadIdx.x, s_counts[threadIdx.x]);
	if (err) atomicOr(status, err);
}

// ---------------------------------------------------------------------
// A path's step from vertex to vertex: update_path with the shadow ray's
// result of the last vertex (path_trace_integrator.cpp:235-249) and with the
// camera (CAMERA) or bounce ray's (251-272, 273-302), then next_ray_for_path's
// shadow step (126-184) and bounce step (185-223) at the vertex met.
//
// The block works in phases that its warps enter together: surface, light
// tree walk, light sample and shadow ray, bounce.  The kernel's code is some
// hundred KB, and warps spread over all of it miss in the instruction cache
// (25 of 35 stall cycles an instruction, with 64 warps an SM each on its
// own); in phase they share the lines.
// ---------------------------------------------------------------------
//
// 512 threads, 2 blocks an SM (64 registers; the spills stay in L1), or 3 (40)
// in the adjoint pass, which keeps more of a vertex.  Fewer threads a block
// lose the phases' order: while hit and shadow shading had just been joined,
// the 512x384x16 frame with 50,000 primitives took 13.98 ms with 3 x 512,
// 14.23 with 2, 14.30 with 4, 14.81 with 4 x 256, 17.49 with 8 x 128.  Without
// the GTR code 2 and 3 blocks take 12.4 ms, the GTR frame 0.75 and 0.79, the
// differentiable step 7.63 and 7.37.
#define PSY_SHADE_BLOCK 512
constexpr int shade_min_blocks(unsigned mode) { return (mode & 2u) ? 3 : 2; }

enum : unsigned { SHADE_GTR = 1u, SHADE_ADJOINT = 2u };

template <class W, bool CAMERA, unsigned F, unsigned MODE>
__global__ void __launch_bounds__(PSY_SHADE_BLOCK, shade_min_blocks(MODE))
    shade_kernel(W w, HaltonDev hd, PathSoA ps, WaveBufs wb, const float4* __restrict__ rin, float4* __restrict__ rout,
                 float4* __restrict__ rshadow, const int* __restrict__ q_in, const int* n_dev, int n_host, int* q_out,
                 int* n_out, unsigned* status) {
	extern __shared__ __align__(16) float sgrad[];
	constexpr bool GTR = (MODE & SHADE_GTR) != 0, ADJOINT = !W::BATCH && (MODE & SHADE_ADJOINT) != 0;
	if (ADJOINT) grad_begin(w.render(0), sgrad);
	const int lane = threadIdx.x & 31;
	const int n = n_dev ? *n_dev : n_host;
	unsigned err = 0;
	for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
		const int i = base + (int)threadIdx.x;
		bool live = false, gtr = false, delta = false;
		int slot = 0, rid = 0;
		uint32_t smp = 0, dim = 0, step = 0;
		float wl = 0.0f, time = 0.0f;
		Vertex sh;
		GtrVertex gv;
		// ---- the results of the last vertex's rays
		if (i < n) {
			// (everything that is read by position or slot is asked for first:
			// one wait for memory instead of one after another.  The hit of an
			// entry without a ray is not used.)
			slot = CAMERA ? i : q_in[i];
			WorldRayD wr;
			const int tag = load_ray(rin, wb.cap, i, &wr);
			HitRec rec;
			HitPath path;
			const int4 hi = wb.hit_i[i];
			const float4 hf = wb.hit_f[i];
			const uint4 head = ps.head[slot];
			const float4 col4 = CAMERA ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : ps.col[slot];
			const float4 lcol4 = CAMERA ? col4 : ps.lcol[slot];
			const float4 fcol4 = CAMERA ? make_float4(1.0f, 1.0f, 1.0f, 1.0f) : ps.fcol[slot];
			const uint8_t blocked = CAMERA ? (uint8_t)1 : wb.occl[i];
			rid = tag >> 1;
			const DevScene& sc = w.scene(rid);
			const RenderParams& rp = w.render(rid);
			smp = head.x;
			dim = head.y & 0xffffu;
			step = head.y >> 16;
			wl = __uint_as_float(head.z);
			const float last_pdf = __uint_as_float(head.w);
			Spec col = sp(col4);
			if (!CAMERA) {
				if (blocked == 0) {
					const Spec c = sp(lcol4);
					for (int k = 0; k < 4; ++k) col.e[k] += c.e[k];
					if (ADJOINT)
						grad_add(rp, sgrad, ps, slot, (int)(step >> 1), sp(ps.nee_base[slot]), ps.nee_param[slot], wl);
				}
			}
			if (!(tag & 1)) {  // (tag & 1): the last vertex sent no bounce ray
				time = wr.time;
				load_rec(wb, i, hi, hf, &rec, &path);
				const Spec fcol = sp(fcol4);
				if (rec.inst >= 0) {
					hit_surface(sc, &rec, path);
					int closure;
					float lpdf;
					make_vertex<F, GTR>(sc, rec, path, wr, rp.ident_inv, &sh, &gv, &closure, &lpdf, &err);
					const int vtx = (int)(step >> 1);  // index of this path vertex
					if (closure == CLOSURE_EMIT) {
						const Spec e0 = rgb_to_spec(sh.col, wl);
						Spec e = e0;
						const int lp = emission_param(rp, rec.obj);
						if (lp >= 0)
							for (int k = 0; k < 4; ++k) e.e[k] *= rp.params[lp];
						const bool mis = !CAMERA && last_pdf != 0.0f;
						const float mis_inv_pdf = mis ? power_heuristic(last_pdf, lpdf) / last_pdf : 0.0f;
						Spec C;
						for (int k = 0; k < 4; ++k)
							C.e[k] = mis ? ((fcol.e[k] * last_pdf) * e.e[k]) * mis_inv_pdf : fcol.e[k] * e.e[k];
						for (int k = 0; k < 4; ++k) col.e[k] += C.e[k];
						if (ADJOINT) {
							// the same contribution without its parameterised factors
							const Spec fx = sp(ps.fexcl[slot]);
							Spec B;
							for (int k = 0; k < 4; ++k)
								B.e[k] = mis ? ((fx.e[k] * last_pdf) * e0.e[k]) * mis_inv_pdf : fx.e[k] * e0.e[k];
							grad_add(rp, sgrad, ps, slot, vtx, B, lp, wl);
						}
					} else if (closure == CLOSURE_LAMBERT || (GTR && closure == CLOSURE_GTR)) {
						// (closures outside the supported set end the path)
						live = true;
						sh.pid = (rp.params && rec.shader >= 0) ? rp.shader_param[rec.shader] : -1;
						gtr = GTR && sh.gtr >= 0;
						delta = gtr && gtr_is_delta(gtr_of(sc.shaders[sh.gtr]));
						if (ADJOINT && vtx < PSY_ADJ_MAX_VERTS) {
							Spec a = Spec{};
							if (sh.pid >= 0) {
								a = albedo_spec(rp.params + sh.pid, wl);
							} else if (sh.pid < -1) {
								const Spec up = rgb_to_spec(sh.col, wl);
								const float q = rp.params[-2 - sh.pid];
								for (int k = 0; k < 4; ++k) a.e[k] = up.e[k] * q;
								ps.vdsc[slot * PSY_ADJ_MAX_VERTS + vtx] = f4(up);
							}
							ps.vpid[slot * PSY_ADJ_MAX_VERTS + vtx] = sh.pid;
							ps.valb[slot * PSY_ADJ_MAX_VERTS + vtx] = f4(a);
						}
					}
				} else {
					const Spec bg = rgb_to_spec(sc.background, wl);
					for (int k = 0; k < 4; ++k) col.e[k] += fcol.e[k] * bg.e[k];
				}
			}
			ps.col[slot] = f4(col);
		}
		// ---- the live paths' places in the next queue (ballot compaction)
		const unsigned m = __ballot_sync(0xffffffffu, live);
		int j = 0;
		if (lane == 0 && m) j = atomicAdd(n_out, __popc(m));
		j = __shfl_sync(0xffffffffu, j, 0) + __popc(m & ((1u << lane) - 1u));
		if (live) q_out[j] = slot;
		__syncthreads();
		// ---- light tree walk
		LightQuery q;
		q.obj = -1;
		q.valid = false;
		q.has_xform = false;
		if (live && !delta) {
			const DevScene& sc = w.scene(rid);
			q.n = sampler_get(hd, smp, dim);
			q.u = sampler_get(hd, smp, dim + 1);
			q.v = sampler_get(hd, smp, dim + 2);
			q.pos = sh.p;
			// lq_nor = geo.n, flipped for back-facing hits
			q.nor = (sh.bf != 0.0f) ? sh.n * -1.0f : sh.n;
			q.d = sh.d;
			q.wavelength = wl;
			q.time = time;
			q.id = 0;
			q.selection_pdf = 1.0f;
			q.light_sample_pdf = 1.0f;
			q.gtr = gtr;
			if (gtr) q.gp = gtr_of(sc.shaders[sh.gtr]);
			light_tree_pick<F, GTR>(sc, &q);
		}
		__syncthreads();
		// ---- light sample and shadow ray
		if (live) {
			const DevScene& sc = w.scene(rid);
			const RenderParams& rp = w.render(rid);
			float4 contrib = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
			if (delta) {
				// a delta closure takes no light sample and no sampler draws;
				// the reference traces the step's ray again, and its result
				// adds nothing (path_trace_integrator.cpp:131-184, 235-249)
				const size_t cap = wb.cap;
				for (int k = 0; k < 4; ++k) rshadow[k * cap + j] = rin[k * cap + i];
				float4 last = rin[4 * cap + i];
				last.w = __int_as_float(rid << 1);
				rshadow[4 * cap + j] = last;
				if (ADJOINT) {
					ps.nee_param[slot] = -1;
					ps.nee_base[slot] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
				}
			} else {
				light_emit<F>(sc, &q, rp.ident_inv);
				dim += 3;
				if (q.valid) {
					const float bsdf_pdf = gtr ? gtr_pdf(q.gp, sh.d, q.to_light, sh.n) : lambert_pdf(sh.d, q.to_light, sh.n);
					const float mis_inv_pdf = power_heuristic(q.light_sample_pdf, bsdf_pdf) / q.light_sample_pdf;
					const float lc = (float)rp.light_count;
					Spec lcol;
					for (int k = 0; k < 4; ++k) lcol.e[k] = ((q.spec.e[k] * mis_inv_pdf) * lc) / q.selection_pdf;
					const int lp = emission_param(rp, q.obj);
					if (lp >= 0)
						for (int k = 0; k < 4; ++k) lcol.e[k] *= rp.params[lp];
					if (ADJOINT) ps.nee_param[slot] = lp;
					WorldRayD sray;
					sray.o = sh.p + sh.off;
					sray.d = (q.to_light - sh.off) * 0.9995f;
					sray.time = time;
					if (gtr) gtr_propagate_differentials(sh, gv, &sray);
					else propagate_differentials(sh, &sray);
					store_ray(rshadow, wb.cap, j, sray, rid << 1);
					// the light's contribution if the shadow ray is not blocked
					// (update_path, shadow result: path_trace_integrator.cpp:235-249)
					const Spec fac = gtr ? gtr_eval(q.gp, sh.d, sray.d, sh.n, wl) : lambert_eval_p(rp, sh, sray.d, wl);
					const Spec fcol = CAMERA ? Spec{{1.0f, 1.0f, 1.0f, 1.0f}} : sp(ps.fcol[slot]);
					Spec c;
					for (int k = 0; k < 4; ++k) c.e[k] = (fcol.e[k] * lcol.e[k]) * fac.e[k];
					contrib = f4(c);
					if (ADJOINT) {
						// without the light's scale and the albedos of parameterised vertices
						const Spec fx = sp(ps.fexcl[slot]);
						const float cs = gtr ? 0.0f : lambert_cos(sh.d, sray.d, sh.n);
						const Spec f0 = sh.pid != -1 ? Spec{{cs, cs, cs, cs}} : fac;
						Spec b;
						for (int k = 0; k < 4; ++k)
							b.e[k] = (fx.e[k] * (((q.spec.e[k] * mis_inv_pdf) * lc) / q.selection_pdf)) * f0.e[k];
						ps.nee_base[slot] = f4(b);
					}
				} else {
					err |= ERRF_NOLIGHT;
					rshadow[4 * (size_t)wb.cap + j] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float((rid << 1) | 1));
				}
			}
			ps.lcol[slot] = contrib;
		}
		__syncthreads();
		// ---- bounce
		if (live) {
			const RenderParams& rp = w.render(rid);
			step += 2;
			float pdf = 0.0f;
			if (step == rp.path_length * 2) {
				// the path's last vertex: only its shadow ray is left
				rout[4 * (size_t)wb.cap + j] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float((rid << 1) | 1));
			} else {
				Spec fcol = CAMERA ? Spec{{1.0f, 1.0f, 1.0f, 1.0f}} : sp(ps.fcol[slot]);
				// The reference passes two sampler.next() calls as arguments; g++
				// evaluates them right to left, so the second draw is `si` and the
				// first `sj`.
				const float sj = sampler_get(hd, smp, dim++);
				const float si = sampler_get(hd, smp, dim++);
				WorldRayD wr;
				wr.o = sh.p + sh.off;
				wr.time = time;
				V3 out;
				Spec filter;
				if (gtr) {
					const Gtr gp = gtr_of(w.scene(rid).shaders[sh.gtr]);
					gtr_sample(gp, sh.d, sh.n, si, sj, wl, &out, &filter, &pdf);
					wr.d = out;
					gtr_propagate_differentials(sh, gv, &wr);
				} else {
					V3 nn = normalized(sh.n);
					if (dot(nn, sh.d) > 0.0f) nn = nn * -1.0f;
					const V3 dir = cosine_sample_hemisphere(si, sj);
					pdf = dir.z * (float)PSY_INV_PI_D;
					out = zup_to_vec(dir, nn);
					filter = lambert_eval_p(rp, sh, out, wl);
					wr.d = out;
					propagate_differentials(sh, &wr);
				}
				store_ray(rout, wb.cap, j, wr, rid << 1);
				if (!delta) {
					if (pdf < 0.00001f) pdf = 0.00001f;
					for (int k = 0; k < 4; ++k) fcol.e[k] *= filter.e[k] / pdf;
				} else {
					for (int k = 0; k < 4; ++k) fcol.e[k] *= filter.e[k];
				}
				if (ADJOINT) {
					// the path weight without the parameterised albedos
					Spec fx = sp(ps.fexcl[slot]);
					const float cs = gtr ? 0.0f : lambert_cos(sh.d, out, sh.n);
					for (int k = 0; k < 4; ++k) fx.e[k] *= (sh.pid != -1 ? cs : filter.e[k]) / (delta ? 1.0f : pdf);
					ps.fexcl[slot] = f4(fx);
				}
				if (delta) pdf = 0.0f;  // last_pdf 0: the next emitter hit takes no MIS weight
				ps.fcol[slot] = f4(fcol);
			}
			ps.head[slot] = make_uint4(smp, (dim & 0xffffu) | (step << 16), __float_as_uint(wl), __float_as_uint(pdf));
		}
		__syncthreads();
	}
	if (ADJOINT) grad_end(w.render(0), sgrad);
	if (err) atomicOr(status, err);
}

// The shadow rays of the wave's last vertices.
template <class W>
__global__ void __launch_bounds__(256) shade_last_kernel(W w, PathSoA ps, WaveBufs wb, const int* __restrict__ q_in,
                                                         const int* n_dev) {
	extern __shared__ __align__(16) float sgrad[];
	if (!W::BATCH) grad_begin(w.render(0), sgrad);
	const int n = *n_dev;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		if (wb.occl[i] != 0) continue;
		const int slot = q_in[i];
		Spec col = sp(ps.col[slot]);
		const Spec c = sp(ps.lcol[slot]);
		for (int k = 0; k < 4; ++k) col.e[k] += c.e[k];
		ps.col[slot] = f4(col);
		if (!W::BATCH && w.render(0).grad) {
			const uint4 head = ps.head[slot];
			grad_add(w.render(0), sgrad, ps, slot, (int)(head.y >> 17), sp(ps.nee_base[slot]), ps.nee_param[slot],
			         __uint_as_float(head.z));
		}
	}
	if (!W::BATCH) grad_end(w.render(0), sgrad);
}

// The finished paths' film samples: Color_XYZ(col) * XYZ_NORM_FAC.
static __global__ void __launch_bounds__(256) sample_xyz_kernel(PathSoA ps, int paths) {
	const int slot = blockIdx.x * blockDim.x + threadIdx.x;
	if (slot >= paths) return;
	float xyz[3];
	spec_to_xyz(sp(ps.col[slot]), __uint_as_float(ps.head[slot].z), xyz);
	float3 o;
	o.x = xyz[0] * XYZ_NORM_FAC;
	o.y = xyz[1] * XYZ_NORM_FAC;
	o.z = xyz[2] * XYZ_NORM_FAC;
	reinterpret_cast<float3*>(ps.sample)[slot] = o;
}

// Adds each pixel's samples, in sample order, to its render's film; rejects
// non-finite samples as Film::add_sample does (film/film.hpp:135-153).
template <class W>
__global__ void film_reduce_kernel(W w, WaveRange wv, PathSoA ps) {
	const int p = blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= wv.pixels) return;
	const uint64_t q = wv.pix_base + (uint64_t)p;
	const RenderParams& rp = w.render(w.render_of_pixel(q));
	const uint64_t pixel = q - rp.pixel_base;
	const uint64_t first = rp.path_base + pixel * rp.spp - wv.base;  // slot of the pixel's first sample
	const float3* s = reinterpret_cast<const float3*>(ps.sample) + first;
	float* xyz = rp.xyz;
	float ax = xyz[pixel * 3], ay = xyz[pixel * 3 + 1], az = xyz[pixel * 3 + 2];
	uint32_t c = 0;
	for (uint32_t k = 0; k < rp.spp; ++k) {
		const float3 v = s[k];
		if (!isfinite(v.x) || !isfinite(v.y) || !isfinite(v.z)) continue;
		ax += v.x;
		ay += v.y;
		az += v.z;
		++c;
	}
	xyz[pixel * 3] = ax;
	xyz[pixel * 3 + 1] = ay;
	xyz[pixel * 3 + 2] = az;
	if (rp.counts) rp.counts[pixel] += c;
}

// ---------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------
static int sm_count() {
	int dev = 0, sms = 1;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	return sms;
}

// Persistent grid: resident blocks of `kernel` at `block` threads x SMs.
template <typename K>
static int persistent_grid(K kernel, int block) {
	int dev = 0, sms = 0, b = 0;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, block, 0);
	return sms * (b < 1 ? 1 : b);
}

// The compiled shading modes: Lambert and emission only (the closures of most
// scenes: without the GTR code and its vertex data there is less to spill),
// all closures, and the adjoint pass.  One kernel for all three: 512x384x16
// frame with 50,000 primitives 13.7 ms, 12.4 so (together with
// light_tree_pick's cut caps).
static constexpr int SHADE_MODES = 3;
inline int shade_mode(unsigned features, bool adjoint) { return adjoint ? 2 : (features & FEAT_GTR) ? 1 : 0; }

struct WaveGrids {
	int block = 0;
	int trace_b = 0;  // traversal block size
	int trace, shade_c[SHADE_MODES], shade_b[SHADE_MODES], last, sms;
};

template <class W, unsigned F>
static const WaveGrids& grids_for(int block) {
	// one entry per block size, filled on first use (block sizes 64..256)
	static WaveGrids g[5];
	const int k = block == 64 ? 0 : block == 128 ? 1 : block == 256 ? 2 : 3;
	if (g[k].block != block) {
		WaveGrids n;
		n.block = block;
		n.trace_b = TraceCfg<F>::launch_block(block);
		n.trace = persistent_grid(trace_wave_kernel<W, F>, n.trace_b);
		n.shade_c[0] = persistent_grid(shade_kernel<W, true, F, 0u>, PSY_SHADE_BLOCK);
		n.shade_b[0] = persistent_grid(shade_kernel<W, false, F, 0u>, PSY_SHADE_BLOCK);
		n.shade_c[1] = persistent_grid(shade_kernel<W, true, F, SHADE_GTR>, PSY_SHADE_BLOCK);
		n.shade_b[1] = persistent_grid(shade_kernel<W, false, F, SHADE_GTR>, PSY_SHADE_BLOCK);
		if constexpr (!W::BATCH) {
			n.shade_c[2] = persistent_grid(shade_kernel<W, true, F, SHADE_GTR | SHADE_ADJOINT>, PSY_SHADE_BLOCK);
			n.shade_b[2] = persistent_grid(shade_kernel<W, false, F, SHADE_GTR | SHADE_ADJOINT>, PSY_SHADE_BLOCK);
		}
		n.last = persistent_grid(shade_last_kernel<W>, 256);
		n.sms = sm_count();
		g[k] = n;
	}
	return g[k];
}

// Counters per wave, two a stage (vertices 0 .. path_length, the last stage
// being the last shadow rays): traversal work, live paths after the stage.
inline int wave_counter_count(uint32_t path_length) { return 2 * ((int)path_length + 1); }

template <class W, unsigned F>
void launch_wave(const W& w, int mode, uint32_t path_length, const HaltonDev& hd, const WaveRange& wv,
                        const PathSoA& ps, const WaveBufs& wb, const WaveQueues& wq, unsigned* status, int block,
                        size_t gsmem, cudaStream_t st, uint32_t* launches, const LaunchTimer* tm) {
	const WaveGrids& g = grids_for<W, F>(block);
	auto tstart = [&]() {
		if (tm && *tm->used < tm->capacity) cudaEventRecord(tm->events[2 * *tm->used], st);
	};
	auto tstop = [&]() {
		if (tm && *tm->used < tm->capacity) cudaEventRecord(tm->events[2 * (*tm->used)++ + 1], st);
	};
	const int P = wv.paths;
	int* c = wq.counters;
	cudaMemsetAsync(c, 0, sizeof(int) * wave_counter_count(path_length), st);
	camera_gen_kernel<W><<<(P + block - 1) / block, block, 0, st>>>(w, hd, wv, ps, wb);
	const float4* rin = wb.ray[0];
	float4 *rout = wb.ray[2], *rshadow = wb.ray[1];
	int *q = nullptr, *n = nullptr;  // the stage's queue (null: every path of the wave)
	auto grid = [&](int full, int threads) {
		const int need = (P + threads - 1) / threads;
		return need < full ? need : full;
	};
	// shading blocks: smaller ones for waves that would leave SMs without any
	// (80x60 preview: 443 us with 512-thread blocks on 10 SMs, 338 with 64 and
	// the rays spread over all warps)
	int sb = PSY_SHADE_BLOCK;
	while (sb > 64 && (P + sb - 1) / sb < 2 * g.sms) sb >>= 1;
	const int per = PSY_SHADE_BLOCK / sb;
	for (uint32_t v = 0; v <= path_length; ++v, c += 2) {
		const unsigned parts = v == 0 ? TRACE_CLOSEST : v == path_length ? TRACE_OCCL : TRACE_CLOSEST | TRACE_OCCL;
		tstart();
		trace_wave_kernel<W, F><<<g.trace, g.trace_b, 0, st>>>(w, wb, rin, rshadow, n, P, parts, c, wq.rays, status);
		tstop();
		int* q2 = (q == wq.q0) ? wq.q1 : wq.q0;
		if (v == path_length)
			shade_last_kernel<W><<<grid(g.last, 256), 256, gsmem, st>>>(w, ps, wb, q, n);
		else {
			auto shade = [&](auto first, auto later) {
				if (v == 0)
					first<<<grid(g.shade_c[mode] * per, sb), sb, gsmem, st>>>(w, hd, ps, wb, rin, rout, rshadow, nullptr, nullptr,
					                                                         P, q2, c + 1, status);
				else
					later<<<grid(g.shade_b[mode] * per, sb), sb, gsmem, st>>>(w, hd, ps, wb, rin, rout, rshadow, q, n, 0, q2,
					                                                         c + 1, status);
			};
			if (mode == 0) shade(shade_kernel<W, true, F, 0u>, shade_kernel<W, false, F, 0u>);
			else if (mode == 1) shade(shade_kernel<W, true, F, SHADE_GTR>, shade_kernel<W, false, F, SHADE_GTR>);
			else if constexpr (!W::BATCH)
				shade(shade_kernel<W, true, F, SHADE_GTR | SHADE_ADJOINT>, shade_kernel<W, false, F, SHADE_GTR | SHADE_ADJOINT>);
		}
		float4* t = const_cast<float4*>(rin);
		rin = rout;
		rout = t;
		q = q2;
		n = c + 1;
	}
	sample_xyz_kernel<<<(P + 255) / 256, 256, 0, st>>>(ps, P);
	film_reduce_kernel<W><<<(wv.pixels + 127) / 128, 128, 0, st>>>(w, wv, ps);
	*launches += 5 + 2 * path_length;
}

}  // namespace psy

#endif
