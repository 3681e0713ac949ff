/*
 * Device-side ray traversal of the uploaded scene.
 *
 * The reference traces ray *streams* breadth-first (accel/bvh4.cpp:163-236,
 * object/patch_utils.hpp:18-200); every per-ray decision there depends only
 * on that ray's own state, so a depth-first per-ray walk that keeps the
 * reference's tests and its max_t updates returns the same closest hit.  The
 * one order-dependent case, two candidates at exactly the same t, resolves
 * to whichever is found first; child boxes are visited nearest-first here.
 *
 * What a lane carries from step to step is small and meant for registers:
 * the ray in the current space, the next tree reference (`cur`), the stack
 * depth and the placement it is in.  Everything an assembly instance adds
 * on the way down (merged motion transforms, the inherited shader, the
 * element id prefix: the reference's xform_stack, surface_shader_stack and
 * element_id, tracer/tracer.cpp:125-219) depends on the path of instances
 * alone and is laid out once per scene, one DevPlace per unrolled assembly
 * instance.  Scenes that unroll to more than PSY_MAX_PLACES keep a level
 * stack in local memory instead.  (With the merged frames, the hit
 * record, the level stack and a copy of the ray in a lane's local memory the
 * 1280x720x4 many-light frame took 254 ms; with this, 170.)
 */
#ifndef PSY_TRACE_DEVICE_CUH
#define PSY_TRACE_DEVICE_CUH

#include "psy_math.h"
#include "psy_scene.h"

namespace psy {

#define PSY_NODE_STACK 64
#define PSY_MAX_LEVELS 8
#define PSY_MAX_MOTION 4
#define PSY_SPLIT_STACK 64


struct WorldRayD {
	V3 o, d, odx, ody, ddx, ddy;
	float time;
	bool occl;
};

__device__ __forceinline__ M44 load_m44_dev(const float* p) {
	M44 m;
	const float4* q = reinterpret_cast<const float4*>(p);
#pragma unroll
	for (int r = 0; r < 4; ++r) {
		const float4 v = __ldg(q + r);
		m.m[r][0] = v.x;
		m.m[r][1] = v.y;
		m.m[r][2] = v.z;
		m.m[r][3] = v.w;
	}
	return m;
}

// A sequence of motion matrices (16 floats each, 16-byte aligned): a
// placement's merged frame, an instance's transforms or a frame in local
// memory.  count 0 = no transform (identity).
struct Frame {
	const float* m;
	int count;
};

__device__ __forceinline__ M44 load_m44(const float* p) {
	M44 m;
	const float4* q = reinterpret_cast<const float4*>(p);
#pragma unroll
	for (int r = 0; r < 4; ++r) {
		const float4 v = q[r];
		m.m[r][0] = v.x;
		m.m[r][1] = v.y;
		m.m[r][2] = v.z;
		m.m[r][3] = v.w;
	}
	return m;
}

__device__ __forceinline__ M44 frame_at(const Frame& f, float alpha) {
	const SeqPos sp = seq_pos(alpha, f.count);
	if (sp.single) return load_m44(f.m + 16 * sp.i0);
	return m44_lerp(sp.nalpha, load_m44(f.m + 16 * sp.i0), load_m44(f.m + 16 * (sp.i0 + 1)));
}

__device__ __forceinline__ M44 seq_lerp_global(const float* xs, int count, float alpha) {
	const SeqPos sp = seq_pos(alpha, count);
	if (sp.single) return load_m44_dev(xs + 16 * sp.i0);
	return m44_lerp(sp.nalpha, load_m44_dev(xs + 16 * sp.i0), load_m44_dev(xs + 16 * (sp.i0 + 1)));
}

// Room for one merged frame in local memory.
struct alignas(16) FrameBuf {
	float m[PSY_MAX_MOTION * 16];
};

// merge() of transform sequences (math/transform.hpp:241-272): parent `a`
// with instance transforms `b`, written into `dst`.  Returns the merged
// sequence; its count is -1 if it needs more than PSY_MAX_MOTION samples.
// The three cases of the reference (equal counts, more parent samples, more
// instance samples) share one loop with one matrix product.
// Not inlined: placements hold the merged frames of assembly instances, and
// what is left (transformed object instances, scenes past the placements'
// limit) would spread a thousand instructions over the walk's code.
static __device__ __noinline__ Frame frame_merge(Frame a, const float* b, int nb, FrameBuf* dst) {
	const int na = a.count;
	Frame out{dst->m, -1};
	if (na > PSY_MAX_MOTION || nb > PSY_MAX_MOTION) return out;
	const int n = na > nb ? na : nb;
	const float inv_s = n > 1 ? 1.0f / (float)(n - 1) : 0.0f;
#pragma unroll 1
	for (int i = 0; i < n; ++i) {
		M44 r;
		if (na == nb) {
			r = m44_mul(load_m44(a.m + 16 * i), load_m44_dev(b + 16 * i));
		} else if (na > nb) {
			if (nb == 0) r = load_m44(a.m + 16 * i);
			else r = m44_mul(load_m44(a.m + 16 * i), seq_lerp_global(b, nb, (float)i * inv_s));
		} else {
			// the reference multiplies instance * lerped-parent in this case
			if (na == 0) r = load_m44_dev(b + 16 * i);
			else r = m44_mul(load_m44_dev(b + 16 * i), frame_at(a, (float)i * inv_s));
		}
		for (int k = 0; k < 16; ++k) dst->m[16 * i + k] = r.m[k / 4][k % 4];
	}
	out.count = n;
	return out;
}

// ---------------------------------------------------------------------
// Sphere / sphere light intersection (object/sphere.cpp:67-189,
// lights/sphere_light.hpp:159-246): returns the hit t or -1.
// ---------------------------------------------------------------------
__device__ __forceinline__ float sphere_t(V3 ro, V3 rd, V3 cent, float radi, float max_t) {
	const V3 o = ro - cent;
	const V3 d = rd;
	const float a = length2(d);
	const float b = 2.0f * dot(d, o);
	const float c = length2(o) - radi * radi;
	float disc = b * b - 4.0f * a * c;
	if (disc < 0.0f) return -1.0f;
	disc = sqrtf(disc);
	float q;
	if (b < 0.0f) q = -0.5f * (b - disc);
	else q = -0.5f * (b + disc);
	float t0 = q / a;
	float t1;
	if (q != 0.0f) t1 = c / q;
	else t1 = max_t;
	if (t0 > t1) {
		const float tmp = t1;
		t1 = t0;
		t0 = tmp;
	}
	if (t0 >= max_t || t1 < 0.0001f) return -1.0f;
	if (t0 >= 0.0001f) return t0;
	if (t1 < max_t) return t1;
	return -1.0f;
}

__device__ __forceinline__ void sphere_at(const DevScene& sc, const DevObject& ob, float time, V3* cent, float* radi) {
	const float* p = sc.fpool + ob.data;
	const SeqPos sp = seq_pos(time, ob.n0);
	if (sp.single) {
		*cent = V3(p[sp.i0 * 4], p[sp.i0 * 4 + 1], p[sp.i0 * 4 + 2]);
		*radi = p[sp.i0 * 4 + 3];
	} else {
		const float* a = p + sp.i0 * 4;
		const float* b = a + 4;
		*cent = lerp3(sp.nalpha, V3(a[0], a[1], a[2]), V3(b[0], b[1], b[2]));
		*radi = lerp1(sp.nalpha, a[3], b[3]);
	}
}

__device__ __forceinline__ void light_at(const DevScene& sc, const DevObject& ob, float time, V3* pos, float* radi,
                                         float col[3]) {
	const float* p = sc.fpool + ob.data;
	{
		const SeqPos sp = seq_pos(time, ob.n0);
		const float* a = p + sp.i0 * 3;
		if (sp.single) *pos = V3(a[0], a[1], a[2]);
		else *pos = lerp3(sp.nalpha, V3(a[0], a[1], a[2]), V3(a[3], a[4], a[5]));
	}
	const float* rp = p + ob.n0 * 3;
	{
		const SeqPos sp = seq_pos(time, ob.n1);
		if (sp.single) *radi = rp[sp.i0];
		else *radi = lerp1(sp.nalpha, rp[sp.i0], rp[sp.i0 + 1]);
	}
	const float* cp = rp + ob.n1;
	{
		const SeqPos sp = seq_pos(time, ob.n2);
		const float* a = cp + sp.i0 * 3;
		if (sp.single) {
			col[0] = a[0]; col[1] = a[1]; col[2] = a[2];
		} else {
			const float ia = one_minus(sp.nalpha);
			for (int k = 0; k < 3; ++k) col[k] = (a[k] * ia) + (a[3 + k] * sp.nalpha);
		}
	}
}

// RectangleLight's dimensions and colour at `time` (lerp_seq over each
// sequence, lights/rectangle_light.hpp:44-46).
__device__ __forceinline__ void rect_light_at(const DevScene& sc, const DevObject& ob, float time, float* dx, float* dy,
                                              float col[3]) {
	const float* p = sc.fpool + ob.data;
	{
		const SeqPos sp = seq_pos(time, ob.n0);
		const float* a = p + sp.i0 * 2;
		if (sp.single) {
			*dx = a[0];
			*dy = a[1];
		} else {
			// std::pair's operator* takes a float: (1 - alpha) is narrowed first
			const float ia = one_minus(sp.nalpha);
			*dx = (a[0] * ia) + (a[2] * sp.nalpha);
			*dy = (a[1] * ia) + (a[3] * sp.nalpha);
		}
	}
	if (col) {
		const float* cp = p + ob.n0 * 2;
		const SeqPos sp = seq_pos(time, ob.n1);
		const float* a = cp + sp.i0 * 3;
		if (sp.single) {
			col[0] = a[0]; col[1] = a[1]; col[2] = a[2];
		} else {
			const float ia = one_minus(sp.nalpha);
			for (int k = 0; k < 3; ++k) col[k] = (a[k] * ia) + (a[3 + k] * sp.nalpha);
		}
	}
}

// RectangleLight::intersect_ray's hit test (lights/rectangle_light.hpp:
// 106-121): the plane z = 0 of the light's space, inside the rectangle.
// The upper y bound is dimension x / 2, as the reference has it.  Returns t
// or -1.
__device__ __forceinline__ float rect_light_t(V3 o, V3 d, V3 dinv, float dx, float dy, float max_t) {
	if (d.z == 0.0f) return -1.0f;
	const float t = -o.z * dinv.z;
	if (t <= 0.0f || t > max_t) return -1.0f;
	const float x = o.x + (d.x * t);
	const float y = o.y + (d.y * t);
	if (x >= (dx * -0.5f) && x <= (dx * 0.5f) && y >= (dy * -0.5f) && y <= (dx * 0.5f)) return t;
	return -1.0f;
}

// ---------------------------------------------------------------------
// Patches (object/bilinear.hpp, object/bicubic.hpp)
// ---------------------------------------------------------------------
template <int NV>
struct Patch {
	V3 p[NV];
};

__device__ __forceinline__ float patch_ulen(const Patch<4>& q) { return longest_axis(q.p[0] - q.p[1]); }
__device__ __forceinline__ float patch_vlen(const Patch<4>& q) { return longest_axis(q.p[0] - q.p[2]); }
__device__ __forceinline__ float patch_ulen(const Patch<16>& q) { return longest_axis(q.p[0] - q.p[3]); }
__device__ __forceinline__ float patch_vlen(const Patch<16>& q) { return longest_axis(q.p[0] - q.p[12]); }

template <int NV>
__device__ __forceinline__ void patch_load(const float* src, Patch<NV>* q) {
#pragma unroll
	for (int i = 0; i < NV; ++i) q->p[i] = V3(__ldg(src + i * 3), __ldg(src + i * 3 + 1), __ldg(src + i * 3 + 2));
}

// A split of a patch at the middle of its first direction (Bilinear::split_u,
// object/bilinear.hpp:59-82; Bicubic::split_u, de Casteljau at 0.5 per row,
// object/bicubic.hpp:74-108), with the reference's float operations: the
// second half is left in `p`, the first goes to `f`.  split_v is the same on
// the transposed patch.
__device__ __forceinline__ void patch_split(Patch<4>& p, Patch<4>& f) {
	const V3 m01 = (p.p[0] + p.p[1]) * 0.5f;
	const V3 m23 = (p.p[2] + p.p[3]) * 0.5f;
	f.p[0] = p.p[0];
	f.p[1] = m01;
	f.p[2] = p.p[2];
	f.p[3] = m23;
	p.p[0] = m01;
	p.p[2] = m23;
}

// One de Casteljau split at 0.5 of the control points a,b,c,d of a row: a..d
// become the second half, fa..fd the first.
__device__ __forceinline__ void bezier_split(V3& a, V3& b, V3& c, V3& d, V3& fa, V3& fb, V3& fc, V3& fd) {
	const V3 tmp = (b + c) * 0.5f;
	const V3 q2 = (d + c) * 0.5f;
	const V3 q1 = (tmp + q2) * 0.5f;
	const V3 a1 = (a + b) * 0.5f;
	const V3 a2 = (tmp + a1) * 0.5f;
	const V3 a3 = (a2 + q1) * 0.5f;
	fa = a;
	fb = a1;
	fc = a2;
	fd = a3;
	a = a3;
	b = q1;
	c = q2;
}
__device__ __forceinline__ void patch_split(Patch<16>& p, Patch<16>& f) {
#pragma unroll
	for (int r = 0; r < 4; ++r)
		bezier_split(p.p[r * 4], p.p[r * 4 + 1], p.p[r * 4 + 2], p.p[r * 4 + 3], f.p[r * 4], f.p[r * 4 + 1],
		             f.p[r * 4 + 2], f.p[r * 4 + 3]);
}

// Exchanges the patch's two directions where `t` says so, by selection.
__device__ __forceinline__ void swap_if(bool t, float& a, float& b) {
	const float x = t ? b : a, y = t ? a : b;
	a = x;
	b = y;
}
__device__ __forceinline__ void swap_if(bool t, V3& a, V3& b) {
	swap_if(t, a.x, b.x);
	swap_if(t, a.y, b.y);
	swap_if(t, a.z, b.z);
}
__device__ __forceinline__ void patch_transpose_if(bool t, Patch<4>& p) { swap_if(t, p.p[1], p.p[2]); }
__device__ __forceinline__ void patch_transpose_if(bool t, Patch<16>& p) {
#pragma unroll
	for (int r = 0; r < 4; ++r)
#pragma unroll
		for (int c = r + 1; c < 4; ++c) swap_if(t, p.p[r * 4 + c], p.p[c * 4 + r]);
}

// Four floats as two packed pairs.
struct Quad {
	unsigned long long a, b;
};
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
	unsigned long long r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
	return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& x, float& y) {
	asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
	unsigned long long r;
	asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
	unsigned long long r;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
__device__ __forceinline__ void load_axis(const char* p, Quad& lo, Quad& hi) {
	asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(lo.a), "=l"(lo.b), "=l"(hi.a), "=l"(hi.b) : "l"(p));
}
__device__ __forceinline__ void lerp_quad(Quad& a, const Quad& b, unsigned long long ia, unsigned long long al) {
	a.a = add2(mul2(a.a, ia), mul2(b.a, al));
	a.b = add2(mul2(a.b, ia), mul2(b.b, al));
}
__device__ __forceinline__ void planes(const Quad& q, float no, float di, float* t) {
	const unsigned long long n = pack2(no, no), d = pack2(di, di);
	unpack2(mul2(add2(q.a, n), d), t[0], t[1]);
	unpack2(mul2(add2(q.b, n), d), t[2], t[3]);
}

// ---------------------------------------------------------------------
// Slab tests
// ---------------------------------------------------------------------
// min and max of the bisection: the reference's orders (a op b ? a : b,
// std::min / std::max), or, for operands that are never NaN (clean patches
// and rays: RAY_ODD), single instructions.  Without NaN the two differ in
// the sign of a zero at most, which no comparison that follows can tell.
template <bool CLEAN>
struct MinMax {
	__device__ static __forceinline__ float vlo(float a, float b) { return CLEAN ? fminf(a, b) : vmin(a, b); }
	__device__ static __forceinline__ float vhi(float a, float b) { return CLEAN ? fmaxf(a, b) : vmax(a, b); }
	__device__ static __forceinline__ float slo(float a, float b) { return CLEAN ? fminf(a, b) : smin(a, b); }
	__device__ static __forceinline__ float shi(float a, float b) { return CLEAN ? fmaxf(a, b) : smax(a, b); }
	__device__ static __forceinline__ float axis(V3 v) { return shi(shi(fabsf(v.x), fabsf(v.y)), fabsf(v.z)); }
};

// How a sub-patch is tested.  Without NaN the reference's minima and maxima
// are single instructions.  A ray whose slab tests can meet NaN (RAY_ODD: a
// direction component of zero, the common one, gives 0 * inf on a box's face)
// takes the reference's own for its slab test alone; only a patch with huge
// coordinates takes them, in the patch's own order, for its bounds too.
enum : int { TEST_CLEAN = 0, TEST_ODD_RAY, TEST_ODD_PATCH };

template <int NV, bool CLEAN>
__device__ __forceinline__ Box patch_bound(const Patch<NV>& q) {
	typedef MinMax<CLEAN> M;
	Box b;
	b.lo = q.p[0];
	b.hi = q.p[0];
#pragma unroll
	for (int i = 1; i < NV; ++i) {
		b.lo = V3(M::vlo(b.lo.x, q.p[i].x), M::vlo(b.lo.y, q.p[i].y), M::vlo(b.lo.z, q.p[i].z));
		b.hi = V3(M::vhi(b.hi.x, q.p[i].x), M::vhi(b.hi.y, q.p[i].y), M::vhi(b.hi.z, q.p[i].z));
	}
	return b;
}

// Bounds of a sub-patch (each time sample) and the ray's test against them:
// the top of the loop of intersect_rays_with_patch (object/patch_utils.hpp).
template <int NV, int TSC, int TEST>
__device__ __forceinline__ bool patch_node_test(const Patch<NV> (&q)[TSC], float t_nalpha, V3 o, V3 dinv, float max_t,
                                                float* max_dim, float* h0, float* h1) {
	constexpr bool CLEAN_BOUND = TEST != TEST_ODD_PATCH;
	typedef MinMax<CLEAN_BOUND> M;
	Box bb[TSC];
	float md = 0.0f;
#pragma unroll
	for (int k = 0; k < TSC; ++k) {
		bb[k] = patch_bound<NV, CLEAN_BOUND>(q[k]);
		const float ld = M::axis(bb[k].hi - bb[k].lo);
		md = (k == 0) ? ld : M::shi(md, ld);
	}
	*max_dim = md;
	const Box b = (TSC == 1) ? bb[0] : box_lerp(t_nalpha, bb[0], bb[TSC - 1]);
	if (TEST != TEST_CLEAN) {
		const bool h = box_hit(b, o, dinv, max_t, h0, h1);
		// A NaN far distance comes from 0 * inf: the ray runs exactly along a
		// box face (a zero direction component, the origin on the face).  The
		// reference's std::min/max slab test then reports a hit with h0 = 0 and
		// h1 = NaN, and every sub-box is again NaN or a plain miss, so none of
		// the subtree's leaves can be taken (their t = (h0 + h1) / 2 is NaN)
		// while the reference still walks all of it, millions of nodes deep
		// for a camera ray through the image centre.  Treating it as a miss
		// gives the same hits.
		return h && !(*h1 != *h1);
	}
	const float x0 = (b.lo.x - o.x) * dinv.x, x1 = (b.hi.x - o.x) * dinv.x;
	const float y0 = (b.lo.y - o.y) * dinv.y, y1 = (b.hi.y - o.y) * dinv.y;
	const float z0 = (b.lo.z - o.z) * dinv.z, z1 = (b.hi.z - o.z) * dinv.z;
	*h0 = fmaxf(fmaxf(0.0f, fminf(z0, z1)), fmaxf(fminf(x0, x1), fminf(y0, y1)));
	*h1 = fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fmaxf(z0, z1)) * BBOX_MAXT_ADJUST;
	return *h0 <= fminf(max_t, *h1);
}

// ---------------------------------------------------------------------
// Patch bisection
// ---------------------------------------------------------------------
// Ray::min_width (basics/ray.hpp:132-153) with the parts that do not change
// along the ray taken out of the bisection: the two flip distances cost an
// IEEE division each.
struct RayFlip {
	float ax, ay;          // owx - fwx, owy - fwy
	float tflipx, tflipy;
	float dwx, dwy, fwx, fwy;
};

__device__ __forceinline__ RayFlip ray_flip(const RayWidth& w) {
	RayFlip f;
	f.ax = w.owx - w.fwx;
	f.ay = w.owy - w.fwy;
	f.tflipx = f.ax / w.dwx;
	f.tflipy = f.ay / w.dwy;
	f.dwx = w.dwx; f.dwy = w.dwy;
	f.fwx = w.fwx; f.fwy = w.fwy;
	return f;
}

__device__ __forceinline__ float flip_min_width(const RayFlip& w, float tnear, float tfar) {
	float minx, miny;
	if (tnear < w.tflipx && tfar > w.tflipx) minx = w.fwx;
	else minx = smin(fabsf(w.ax + (w.dwx * tnear)) + w.fwx, fabsf(w.ax + (w.dwx * tfar)) + w.fwx);
	if (tnear < w.tflipy && tfar > w.tflipy) miny = w.fwy;
	else miny = smin(fabsf(w.ay + (w.dwy * tnear)) + w.fwy, fabsf(w.ay + (w.dwy * tfar)) + w.fwy);
	return smin(minx, miny);
}

// Pending first halves a bisection can hold: at most one per second half
// on the path, and the path has at most PSY_SPLIT_STACK - 1 of those.
#define PSY_PATCH_PEND PSY_SPLIT_STACK

// A bisection ends with an error (ERRF_BISECT) after this many loop
// iterations.  The walk is finite (a leaf is forced at 63 second halves or
// depth 127), but a ray the reference would bisect for hours must not hold
// a wave: far above any bisection of a real scene.
#define PSY_PATCH_MAX_STEPS (1u << 24)

// Per-ray bisection of one patch with TSC time samples (TSC = 1 or 2):
// intersect_rays_with_patch for a single ray (object/patch_utils.hpp:18-200).
//
// The reference walks the split tree depth first with a stack of sub-patches:
// a split pushes the first half, then the second, and the second half is
// processed first.  Here both halves are tested against the ray when they
// are made.  The second half is entered if its box is hit; the first half
// is entered at once if only its box is hit, pushed on a stack of pending
// first halves (control points and uv range) if both are, and dropped if
// its box is missed (box_hit only gets stricter as the ray's max t
// shrinks, so the reference would find it missed later as well).  When a
// subtree ends, the last pending first half is popped and tested again
// with the current max t.  A node carries its depth and the number of
// second halves on its path: the reference's stack index, its forced leaf
// at 63.  Control points and uv ranges are those of the reference's walk, so
// the visiting order and the leaf results are the same.
//
// The bisection can stop after any number of loop iterations and resume
// later from its cursor (the node at the top of the loop, whose box the ray
// hits) and its stack, so that a lane can leave a long bisection to run
// with the other lanes of its warp.  patch_run works on a cursor the caller
// holds as a local (kept in registers) and copies back only when it stops
// short of the end.
//
// A node may be kept transposed (`tr`): a patch to be split along its second
// direction is transposed by selection first, so that the lanes of a warp
// split along either direction in one piece of code (300,000 mixed rays
// against bicubic ground: 1.91 -> 1.68 ms, 4M rays against the heightfield
// 1.02 -> 0.97).
template <int NV, int TSC>
struct PatchCursor {
	Patch<NV> cur[TSC];        // the node at the top of the loop
	float a0, a1, b0, b1;      // its range along its first and second direction (u and v, or v and u if tr)
	float max_dim, h0, h1;     // its test
	float t_nalpha;
	bool tr;
	int depth, seconds;        // splits from the root, second halves among them
	int sp;                    // pending first halves on the stack
	unsigned steps;            // loop iterations taken (bounded: PSY_PATCH_MAX_STEPS)
};

// The pending first halves.
template <int NV, int TSC>
struct PatchStore {
	Patch<NV> pend[PSY_PATCH_PEND][TSC];
	float4 ab[PSY_PATCH_PEND];
	int2 at[PSY_PATCH_PEND];   // depth * 2 + tr, second halves
};

// The root's test: sets up `pc` and returns true when the ray hits the
// patch's box.
template <int NV, int TSC, int TEST>
__device__ __forceinline__ bool patch_begin(PatchCursor<NV, TSC>& pc, const float* verts, float time, V3 o, V3 dinv,
                                            float max_t) {
#pragma unroll
	for (int k = 0; k < TSC; ++k) patch_load<NV>(verts + k * NV * 3, &pc.cur[k]);
	pc.t_nalpha = 0.0f;
	if (TSC > 1) {
		// bounds are lerped between the two samples; time == 1.0 would index
		// past the last sample in the reference (undefined) and gives the
		// first sample's bounds here
		const float t_time = time * (float)(TSC - 1);
		pc.t_nalpha = t_time - (float)(int)t_time;
	}
	if (!patch_node_test<NV, TSC, TEST>(pc.cur, pc.t_nalpha, o, dinv, max_t, &pc.max_dim, &pc.h0, &pc.h1)) return false;
	pc.a0 = pc.b0 = 0.0f;
	pc.a1 = pc.b1 = 1.0f;
	pc.tr = false;
	pc.depth = 0;
	pc.seconds = 0;
	pc.sp = 0;
	pc.steps = 0;
	return true;
}

enum : int { PATCH_MORE = 0, PATCH_DONE = 1, PATCH_BLOCKED = 2 };

// Runs up to `units` iterations of the bisection loop (a leaf test or a
// split, with the resume that follows it).  Returns PATCH_DONE when the
// bisection has ended, PATCH_BLOCKED when an occlusion ray took a leaf
// (that ends it), PATCH_MORE when `pc` is the node to carry on from.
// `leaf(t, u, v, max_dim)` is called for every leaf taken, each closer than
// the last, with *max_t lowered to it.  A bisection that exceeds
// PSY_PATCH_MAX_STEPS iterations ends and sets ERRF_BISECT in *err.
template <int NV, int TSC, int TEST, class LEAF>
__device__ __forceinline__ int patch_run(PatchCursor<NV, TSC>& pc, PatchStore<NV, TSC>& ps, V3 o, V3 dinv,
                                         const RayFlip& rw, float* max_t, bool occl, float dice_rate, float min_upoly,
                                         int& units, unsigned* err, LEAF leaf) {
	Patch<NV>(&cur)[TSC] = pc.cur;
	const float t_nalpha = pc.t_nalpha;
	float &max_dim = pc.max_dim, &h0 = pc.h0, &h1 = pc.h1;
	float &a0 = pc.a0, &a1 = pc.a1, &b0 = pc.b0, &b1 = pc.b1;
	// (where a coordinate can be NaN, the order of a bound's minima matters:
	// the patch's own)
	auto test = [&](const Patch<NV>(&q)[TSC], float* md, float* t0, float* t1) {
		if constexpr (TEST != TEST_ODD_PATCH) {
			return patch_node_test<NV, TSC, TEST>(q, t_nalpha, o, dinv, *max_t, md, t0, t1);
		} else {
			Patch<NV> own[TSC];
			for (int k = 0; k < TSC; ++k) {
				own[k] = q[k];
				patch_transpose_if(pc.tr, own[k]);
			}
			return patch_node_test<NV, TSC, TEST>(own, t_nalpha, o, dinv, *max_t, md, t0, t1);
		}
	};
	while (true) {
		if (units == 0) return PATCH_MORE;
		--units;
		if (++pc.steps > PSY_PATCH_MAX_STEPS) {
			*err |= ERRF_BISECT;
			return PATCH_DONE;
		}
		// `cur` is a node whose box the ray hits; max_dim, h0, h1 are its test
		// A NaN width (from NaN ray differentials: a grazing hit makes the
		// next ray's origin differentials 0/0 in transfer_ray_origin_
		// differential, basics/differential_geometry.hpp:85-98) survives the
		// reference's std::max, no sub-patch is ever small enough, and its
		// bisection does not end.  Here it counts as zero width: the leaves
		// stop at min_upoly, as for a ray with zero differentials.
		const float wm = flip_min_width(rw, h0, h1) * dice_rate;
		const float width = (wm != wm) ? min_upoly : smax(wm, min_upoly);
		if (max_dim <= width || pc.seconds == PSY_SPLIT_STACK - 1 || pc.depth == 127) {
			const float tt = (h0 + h1) * 0.5f;
			if (tt > 0.0f && tt < *max_t) {
				if (!occl) *max_t = tt;
				const float a = (a0 + a1) * 0.5f, b = (b0 + b1) * 0.5f;
				leaf(tt, pc.tr ? b : a, pc.tr ? a : b, max_dim);
				if (occl) return PATCH_BLOCKED;
			}
		} else {
			// the longer direction is split, the second one on a tie (split_u
			// only if u is strictly longer)
			const float la = patch_ulen(cur[0]), lb = patch_vlen(cur[0]);
			const bool turn = pc.tr ? la < lb : !(la > lb);
			pc.tr = pc.tr != turn;
			swap_if(turn, a0, b0);
			swap_if(turn, a1, b1);
			Patch<NV> first[TSC];
#pragma unroll
			for (int k = 0; k < TSC; ++k) {
				patch_transpose_if(turn, cur[k]);
				patch_split(cur[k], first[k]);
			}
			float smd, sh0, sh1, fmd, fh0, fh1;
			const bool s_hit = test(cur, &smd, &sh0, &sh1);
			const bool f_hit = test(first, &fmd, &fh0, &fh1);
			const float mid = (a0 + a1) * 0.5f;
			if (s_hit) {
				++pc.depth;
				if (f_hit) {
					// the first half waits on the stack
					const int q = pc.sp++;
#pragma unroll
					for (int k = 0; k < TSC; ++k) ps.pend[q][k] = first[k];
					ps.ab[q] = make_float4(a0, mid, b0, b1);
					ps.at[q] = make_int2(pc.depth * 2 + (pc.tr ? 1 : 0), pc.seconds);
				}
				++pc.seconds;
				a0 = mid;
				max_dim = smd;
				h0 = sh0;
				h1 = sh1;
				continue;
			}
			if (f_hit) {
				++pc.depth;
#pragma unroll
				for (int k = 0; k < TSC; ++k) cur[k] = first[k];
				a1 = mid;
				max_dim = fmd;
				h0 = fh0;
				h1 = fh1;
				continue;
			}
		}
		// resume at the last pending first half whose box is still hit
		while (true) {
			if (pc.sp == 0) return PATCH_DONE;
			const int q = --pc.sp;
#pragma unroll
			for (int k = 0; k < TSC; ++k) cur[k] = ps.pend[q][k];
			const float4 w = ps.ab[q];
			a0 = w.x; a1 = w.y; b0 = w.z; b1 = w.w;
			const int2 at = ps.at[q];
			pc.depth = at.x >> 1;
			pc.tr = (at.x & 1) != 0;
			pc.seconds = at.y;
			if (test(cur, &max_dim, &h0, &h1)) break;
		}
	}
}

// The leaf a whole bisection ended with.
struct PatchHit {
	float t, u, v, max_dim;
};

// patch_begin and patch_run on a cursor in memory, for rays and patches whose
// tests can meet NaN.  Not inlined: streams along an axis consist of such
// rays, but the code of all others must not hold theirs, nor have variables
// of theirs in memory because these functions want an address.
template <int NV, int TSC>
static __device__ __noinline__ bool patch_odd_begin(PatchCursor<NV, TSC>& at, const float* verts, float time, V3 o, V3 dinv,
                                                    float max_t, bool odd_patch) {
	PatchCursor<NV, TSC> pc;
	const bool in = odd_patch ? patch_begin<NV, TSC, TEST_ODD_PATCH>(pc, verts, time, o, dinv, max_t)
	                          : patch_begin<NV, TSC, TEST_ODD_RAY>(pc, verts, time, o, dinv, max_t);
	if (in) at = pc;
	return in;
}

// What patch_odd_run leaves: PATCH_*, whether a leaf was taken and the
// closest one, the iterations not used, errors.
struct OddRun {
	int state;
	bool took;
	PatchHit hit;
	int units;
	unsigned err;
};

template <int NV, int TSC>
static __device__ __noinline__ OddRun patch_odd_run(PatchCursor<NV, TSC>& at, PatchStore<NV, TSC>& ps, V3 o, V3 dinv,
                                                    const RayFlip& rw, float max_t, bool occl, float dice_rate,
                                                    float min_upoly, bool odd_patch, int units) {
	PatchCursor<NV, TSC> pc = at;
	const RayFlip w = rw;
	bool took = false;
	unsigned err = 0;
	PatchHit h;
	auto leaf = [&](float t, float u, float v, float md) {
		took = true;
		h = PatchHit{t, u, v, md};
	};
	const int r = odd_patch ? patch_run<NV, TSC, TEST_ODD_PATCH>(pc, ps, o, dinv, w, &max_t, occl, dice_rate, min_upoly, units, &err, leaf)
	                        : patch_run<NV, TSC, TEST_ODD_RAY>(pc, ps, o, dinv, w, &max_t, occl, dice_rate, min_upoly, units, &err, leaf);
	if (r == PATCH_MORE) at = pc;
	return OddRun{r, took, h, units, err};
}

// ---------------------------------------------------------------------
// Whole-scene traversal
// ---------------------------------------------------------------------
// The closest hit as the traversal leaves it.  Object, kind, shader and
// element id follow from the instance and where it was met: the placement,
// or (place < 0) the path of instances from the root.
struct HitRec {
	float t;
	float u, v, max_dim;
	int inst;                  // global instance index, -1 = miss
	int place;                 // its assembly's placement, -1 = scene without placements
	int obj, kind, shader;     // set by hit_surface
};
// The path to a hit without placement: global instance indices, root first.
struct HitPath {
	int depth;
	int path[PSY_MAX_LEVELS];
};

// Element id of the hit (Intersection::id): the local instance index of
// every level, pushed with that assembly's bits.
__device__ __forceinline__ uint64_t hit_id(const DevScene& sc, const HitRec& h, const HitPath& hp) {
	if (h.place >= 0) {
		const DevPlace& p = sc.places[h.place];
		return id_push(p.id, (uint64_t)(h.inst - p.inst_base), p.id_bits);
	}
	uint64_t id = 0;
	int asmb = 0;
	for (int k = 0; k < hp.depth; ++k) {
		id = id_push(id, (uint64_t)(hp.path[k] - sc.assemblies[asmb].inst_base), sc.assemblies[asmb].id_bits);
		asmb = sc.instances[hp.path[k]].data;
	}
	return id;
}

// The shader bound to the hit: the innermost one on the path.
__device__ __forceinline__ int hit_shader(const DevScene& sc, const HitRec& h, const HitPath& hp) {
	const int own = sc.instances[h.inst].shader;
	if (own >= 0) return own;
	if (h.place >= 0) return sc.places[h.place].shader;
	for (int k = hp.depth - 2; k >= 0; --k) {
		const int s = sc.instances[hp.path[k]].shader;
		if (s >= 0) return s;
	}
	return -1;
}

// The object hit, its kind and its shader.
__device__ __forceinline__ void hit_surface(const DevScene& sc, HitRec* h, const HitPath& hp) {
	h->obj = sc.instances[h->inst].data;
	h->kind = sc.objects[h->obj].kind;
	h->shader = hit_shader(sc, *h, hp);
}

// Transform from world space into the hit object's space at the ray time
// (the Intersection::space of the reference).  Returns false when the path
// carries no transform (identity).
template <unsigned F>
__device__ bool hit_space(const DevScene& sc, const HitRec& rec, const HitPath& hp, float time, M44* out, unsigned* err) {
	if (!(F & FEAT_XFORM)) return false;
	Frame f{nullptr, 0};
	FrameBuf buf[2];
	int b = 0;
	auto merge = [&](const DevInstance& inst) {
		if (inst.xform_count == 0) return true;
		f = frame_merge(f, sc.xforms + (size_t)inst.xform * 16, inst.xform_count, &buf[b]);
		b ^= 1;
		if (f.count < 0) {
			*err |= ERRF_MOTION;
			return false;
		}
		return true;
	};
	if (rec.place >= 0) {
		const DevPlace& p = sc.places[rec.place];
		f = Frame{sc.place_frames + (size_t)p.frame * 16, p.frame_count};
		if (!merge(sc.instances[rec.inst])) return false;
	} else {
		for (int k = 0; k < hp.depth; ++k)
			if (!merge(sc.instances[hp.path[k]])) return false;
	}
	if (f.count == 0) return false;
	*out = frame_at(f, time);
	return true;
}

// Patch kind of a bisection in progress: bilinear or bicubic, one or two
// time samples; and what its tests can meet (PM_ODD: NaN, PM_ODD_PATCH: from
// the patch's own coordinates).
enum : int { PM_NONE = 0, PM_BILINEAR1, PM_BILINEAR2, PM_BICUBIC1, PM_BICUBIC2, PM_KIND = 7, PM_ODD = 8, PM_ODD_PATCH = 16 };

// Bytes of the bisection state for the patch kinds of feature set F.
template <unsigned F>
struct PatchBuf {
	static constexpr int TS = (F & FEAT_PATCH_MOTION) ? 2 : 1;
	template <int NV>
	struct Work {
		PatchCursor<NV, TS> c;
		PatchStore<NV, TS> st;
	};
	static constexpr size_t b4 = (F & FEAT_BILINEAR) ? sizeof(Work<4>) : 0;
	static constexpr size_t b16 = (F & FEAT_BICUBIC) ? sizeof(Work<16>) : 0;
	static constexpr size_t m = b4 > b16 ? b4 : b16;
	static constexpr size_t bytes = m > 16 ? m : 16;
};

// References beyond those of the tree: the end of a level on the stack
// (REF_LEVEL, or REF_LEVEL_RAY when the enclosing level's ray is to be
// restored), and no reference (take the next one from the stack).
static constexpr int REF_LEVEL = (int)0xf0000000;
static constexpr int REF_LEVEL_RAY = (int)0xf0000001;
static constexpr int REF_NONE = REF_EMPTY;

enum : unsigned {
	RAY_OCCL = 1u,   // occlusion ray: ends at the first hit
	RAY_ODD = 2u,    // a slab test of the ray in its current space can meet NaN or inf - inf; or the ray's time lies
	                 // before the first sample, where the boxes of moving nodes are extrapolated and may be inverted
	RAY_HIT = 4u,    // a hit was recorded
	RAY_WIDTH = 8u   // the width parameters are those of the current space
};

// The parts of a ray's traversal state that are indexed at run time or too
// large for registers.  They are a variable of their own: one struct with
// the walk's scalars would keep those in local memory too, since the
// compiler does not take a variable with a run-time index apart (1280x720x4
// many-light frame 149 ms so, 141 apart).
template <unsigned F>
struct TravMem {
	uint2 stack[PSY_NODE_STACK + PSY_MAX_LEVELS];  // reference, distance of its box (as bits)
	RayFlip rw;                                    // width parameters of the current space (RAY_WIDTH)
	float lvr[PSY_MAX_LEVELS][9];                  // ray of each enclosing level (REF_LEVEL_RAY)
	// scenes without placements: the entered instances and merged frames
	int lv_inst[PSY_MAX_LEVELS], lv_frame[PSY_MAX_LEVELS], lv_count[PSY_MAX_LEVELS];
	FrameBuf frames[PSY_MAX_LEVELS];
	// the bisection in progress: its instance, ray and widths, its cursor and stack
	int p_inst;
	V3 p_o, p_dinv;
	RayFlip p_rw;
	alignas(16) unsigned char pbuf[PatchBuf<F>::bytes];
};

// Traversal state of one ray.  IO gives the world ray (origin, direction,
// differentials: read again where an instance or a patch needs them) and
// takes the hits.
template <unsigned F, class IO>
struct Trav {
	V3 o, d, dinv;      // the ray in the current space
	float max_t, time;
	int cur;            // next reference
	int sp, L;          // stack entries, assembly levels entered
	int place;          // current placement (scenes with placements)
	int pmode;          // bisection in progress (PM_*)
	unsigned flags, err;
	IO io;
	TravMem<F>* mem;

	static constexpr bool NESTED = (F & FEAT_NESTED) != 0;
	static constexpr bool XFORM = (F & FEAT_XFORM) != 0;
	static constexpr int TS = PatchBuf<F>::TS;

	template <int NV>
	__device__ __forceinline__ typename PatchBuf<F>::template Work<NV>& work() {
		return *reinterpret_cast<typename PatchBuf<F>::template Work<NV>*>(mem->pbuf);
	}

	// the same room as that of a patch with one time sample
	typedef PatchBuf<F & ~FEAT_PATCH_MOTION> Still;
	template <int NV>
	__device__ __forceinline__ typename Still::template Work<NV>& still_work() {
		return *reinterpret_cast<typename Still::template Work<NV>*>(mem->pbuf);
	}

	__device__ __forceinline__ static bool odd_ray(V3 o, V3 d, V3 dinv) {
		// zero direction components (infinite reciprocals), infinities and NaN
		const float s = (fabsf(o.x) + fabsf(o.y) + fabsf(o.z)) + (fabsf(d.x) + fabsf(d.y) + fabsf(d.z));
		const float r = fmaxf(fmaxf(fabsf(dinv.x), fabsf(dinv.y)), fabsf(dinv.z));
		return !(s < INFINITY) || !(r < INFINITY);
	}

	__device__ __forceinline__ void set_ray(V3 no, V3 nd) {
		o = no;
		d = nd;
		dinv = recip3(nd);
		flags &= ~(RAY_ODD | RAY_WIDTH);
		if (odd_ray(o, d, dinv) || !(time >= 0.0f)) flags |= RAY_ODD;
	}

	__device__ __forceinline__ void init(const DevScene& sc, V3 wo, V3 wd, float t, bool occl) {
		flags = occl ? RAY_OCCL : 0u;
		time = t;
		set_ray(wo, wd);
		max_t = occl ? 1.0f : INFINITY;
		cur = __ldg(sc.asmb_root);
		sp = 0;
		L = 0;
		place = 0;
		pmode = PM_NONE;
		err = 0;
		if (NESTED && !sc.places) {
			place = -1;
			mem->lv_frame[0] = -1;
			mem->lv_count[0] = 0;
		}
	}

	// The merged motion frame of the current level.
	__device__ __forceinline__ Frame level_frame(const DevScene& sc) const {
		if (place >= 0) {
			const int4 p = __ldg(reinterpret_cast<const int4*>(sc.places + place));
			return Frame{sc.place_frames + (size_t)p.z * 16, p.w};
		}
		return Frame{mem->lv_count[L] ? mem->frames[mem->lv_frame[L]].m : nullptr, mem->lv_count[L]};
	}

	// Records a hit on instance gi.  Returns false when the ray is finished
	// (an occlusion ray).
	__device__ __forceinline__ bool record(int gi, float t, float u, float v, float md) {
		flags |= RAY_HIT;
		io.hit(*this, gi, t, u, v, md);
		return (flags & RAY_OCCL) == 0;
	}

	// Takes the next reference from the stack into `cur`, leaving finished
	// levels on the way.  An inner node whose box begins beyond max_t is
	// passed over: none of its children could be hit.  Returns false when the
	// stack is empty (the ray is finished).
	__device__ __forceinline__ bool pop(const DevScene& sc) {
		while (cur == REF_NONE) {
			if (sp == 0) return false;
			const uint2 e = mem->stack[--sp];
			const int ref = (int)e.x;
			if (ref >= 0) {
				if (__uint_as_float(e.y) < max_t) cur = ref;
				continue;
			}
			if (NESTED && ref >= REF_LEVEL && ref <= REF_LEVEL_RAY) {
				--L;
				if (place >= 0) place = (int)e.y;
				if (XFORM && ref == REF_LEVEL_RAY) {
					o = V3(mem->lvr[L][0], mem->lvr[L][1], mem->lvr[L][2]);
					d = V3(mem->lvr[L][3], mem->lvr[L][4], mem->lvr[L][5]);
					dinv = V3(mem->lvr[L][6], mem->lvr[L][7], mem->lvr[L][8]);
					flags &= ~(RAY_ODD | RAY_WIDTH);
					if (odd_ray(o, d, dinv) || !(time >= 0.0f)) flags |= RAY_ODD;
				}
				continue;
			}
			cur = ref;
		}
		return true;
	}

	// The planes of a node's child boxes at the ray time.
	static __device__ __forceinline__ void load_node(const DevScene& sc, const DevNode* nd, int ref, float time, Quad& xl,
	                                                 Quad& xh, Quad& yl, Quad& yh, Quad& zl, Quad& zh) {
		const char* base = reinterpret_cast<const char*>(nd);
		load_axis(base, xl, xh);
		load_axis(base + 32, yl, yh);
		load_axis(base + 64, zl, zh);
		if (!(ref & REF_NODE_MOVING)) return;
		const int4 meta = __ldg(reinterpret_cast<const int4*>(&nd->nchild));
		const SeqPos q = seq_pos(time, meta.y);
		auto extra = [&](int k) { return reinterpret_cast<const char*>(sc.node_extra + (size_t)(meta.z + k - 1) * 24); };
		if (q.i0 != 0) {
			const char* e = extra(q.i0);
			load_axis(e, xl, xh);
			load_axis(e + 32, yl, yh);
			load_axis(e + 64, zl, zh);
		}
		if (q.single) return;
		const char* e = extra(q.i0 + 1);
		const unsigned long long al = pack2(q.nalpha, q.nalpha), ia = pack2(one_minus(q.nalpha), one_minus(q.nalpha));
		Quad a, b;
		load_axis(e, a, b);
		lerp_quad(xl, a, ia, al); lerp_quad(xh, b, ia, al);
		load_axis(e + 32, a, b);
		lerp_quad(yl, a, ia, al); lerp_quad(yh, b, ia, al);
		load_axis(e + 64, a, b);
		lerp_quad(zl, a, ia, al); lerp_quad(zh, b, ia, al);
	}

	// The distances of a node's four children in the reference's own order of
	// operations (BBox4::intersect_ray, basics/bbox.hpp:566-595, SSE min/max
	// semantics), infinity for a miss: rays and boxes with infinities or NaN,
	// inverted boxes.  0 for a hit before the first time sample: an
	// extrapolated box need not hold its children's, and its distance on the
	// stack would prune them.
	// The near and far planes are picked for all four children at once, by the
	// ray's sign, so this costs about as much as the plain test: streams along
	// an axis consist of rays that come here (1M rays straight down on 20,000
	// spheres 1,499 -> 1,045 us, on a 256x256 heightfield 730 -> 405, bisection
	// included; a loop over the children with scalar loads before).
	static __device__ __noinline__ float4 odd_node(const DevScene& sc, int ref, V3 o, V3 dinv, float time, float max_t) {
		const DevNode* nd = sc.nodes + (ref & REF_NODE_MASK);
		const int nchild = __ldg(&nd->nchild);
		Quad xl, xh, yl, yh, zl, zh;
		load_node(sc, nd, ref, time, xl, xh, yl, yh, zl, zh);
		float xn[4], xf[4], yn[4], yf[4], zn[4], zf[4];
		const bool sx = dinv.x < 0.0f, sy = dinv.y < 0.0f, sz = dinv.z < 0.0f;
		planes(sx ? xh : xl, -o.x, dinv.x, xn);
		planes(sx ? xl : xh, -o.x, dinv.x, xf);
		planes(sy ? yh : yl, -o.y, dinv.y, yn);
		planes(sy ? yl : yh, -o.y, dinv.y, yf);
		planes(sz ? zh : zl, -o.z, dinv.z, zn);
		planes(sz ? zl : zh, -o.z, dinv.z, zf);
		float t[4];
#pragma unroll
		for (int c = 0; c < 4; ++c) {
			const float mins = vmax(vmax(xn[c], yn[c]), vmax(zn[c], 0.0f));
			const float maxs = vmax(vmin(vmin(xf[c], yf[c]), zf[c]), -INFINITY) * BBOX_MAXT_ADJUST;
			t[c] = c < nchild && mins < max_t && mins <= maxs ? (time >= 0.0f ? mins : 0.0f) : INFINITY;
		}
		return make_float4(t[0], t[1], t[2], t[3]);
	}

	// An inner node (cur): tests the child boxes, leaves the nearest hit child
	// in `cur` (REF_NONE when none is hit) and the others on the stack,
	// nearest on top, ties in child order.  Returns false when the node stack
	// overflows (the ray ends with an error).
	__device__ __forceinline__ bool node_step(const DevScene& sc) {
		const int ref = cur;
		const DevNode* nd = sc.nodes + (ref & REF_NODE_MASK);
		float t0, t1, t2, t3;
		const int4 ch = __ldg(reinterpret_cast<const int4*>(nd->child));
		if ((flags & RAY_ODD) || (ref & REF_NODE_ODD)) {
			const float4 t = odd_node(sc, ref, o, dinv, time, max_t);
			t0 = t.x; t1 = t.y; t2 = t.z; t3 = t.w;
		} else {
			float tn[4], tf[4];
			{
				Quad xl, xh, yl, yh, zl, zh;
				load_node(sc, nd, ref, time, xl, xh, yl, yh, zl, zh);
				float l[4], h[4];
				planes(xl, -o.x, dinv.x, l); planes(xh, -o.x, dinv.x, h);
#pragma unroll
				for (int c = 0; c < 4; ++c) { tn[c] = fminf(l[c], h[c]); tf[c] = fmaxf(l[c], h[c]); }
				planes(yl, -o.y, dinv.y, l); planes(yh, -o.y, dinv.y, h);
#pragma unroll
				for (int c = 0; c < 4; ++c) { tn[c] = fmaxf(tn[c], fminf(l[c], h[c])); tf[c] = fminf(tf[c], fmaxf(l[c], h[c])); }
				planes(zl, -o.z, dinv.z, l); planes(zh, -o.z, dinv.z, h);
#pragma unroll
				for (int c = 0; c < 4; ++c) { tn[c] = fmaxf(fmaxf(tn[c], fminf(l[c], h[c])), 0.0f); tf[c] = fminf(tf[c], fmaxf(l[c], h[c])) * BBOX_MAXT_ADJUST; }
			}
			t0 = tn[0] < max_t && tn[0] <= tf[0] ? tn[0] : INFINITY;
			t1 = tn[1] < max_t && tn[1] <= tf[1] ? tn[1] : INFINITY;
			t2 = tn[2] < max_t && tn[2] <= tf[2] && ch.z != REF_EMPTY ? tn[2] : INFINITY;
			t3 = tn[3] < max_t && tn[3] <= tf[3] && ch.w != REF_EMPTY ? tn[3] : INFINITY;
		}
		const bool h0 = t0 < INFINITY, h1 = t1 < INFINITY, h2 = t2 < INFINITY, h3 = t3 < INFINITY;
		if (flags & RAY_OCCL) {
			// any blocker ends the ray: the order is that of the children, and
			// max_t does not shrink
			t0 = h0 ? 0.0f : t0;
			t1 = h1 ? 0.0f : t1;
			t2 = h2 ? 0.0f : t2;
			t3 = h3 ? 0.0f : t3;
		}
		const int nhit = (h0 ? 1 : 0) + (h1 ? 1 : 0) + (h2 ? 1 : 0) + (h3 ? 1 : 0);
		if (sp - L + nhit > PSY_NODE_STACK) {
			err |= ERRF_STACK;
			return false;
		}
		// each child's place in the order: how many come before it
		const int l01 = t1 < t0, l02 = t2 < t0, l03 = t3 < t0, l12 = t2 < t1, l13 = t3 < t1, l23 = t3 < t2;
		const int r0 = l01 + l02 + l03, r1 = 1 - l01 + l12 + l13, r2 = 2 - l02 - l12 + l23, r3 = 3 - l03 - l13 - l23;
		const int top = sp + nhit - 1;
		int next = REF_NONE;
		auto put = [&](bool h, int r, int ref_c, float t) {
			if (!h) return;
			if (r == 0) next = ref_c;
			else mem->stack[top - r] = make_uint2((unsigned)ref_c, __float_as_uint(t));
		};
		put(h0, r0, ch.x, t0);
		put(h1, r1, ch.y, t1);
		put(h2, r2, ch.z, t2);
		put(h3, r3, ch.w, t3);
		if (nhit > 0) sp = top;
		cur = next;
		return true;
	}

	// A leaf (cur) of class LEAF_ENTER: enters the assembly of the instance,
	// moves the ray into its space and goes to its root.  Returns false when
	// the node stack overflows.
	__device__ __forceinline__ bool enter(const DevScene& sc) {
		const int gi = cur & REF_LEAF_MASK;
		const int4 m = __ldg(reinterpret_cast<const int4*>(&sc.leaves[gi].data));  // rank, transforms, assembly
		cur = REF_NONE;
		Frame f;
		int child = -1, root;
		if (place >= 0) {
			child = __ldg(&sc.places[place].child_base) + m.x;
			const int4 p = __ldg(reinterpret_cast<const int4*>(sc.places + child));
			root = p.x;
			f = Frame{sc.place_frames + (size_t)p.z * 16, p.w};
			if (root != REF_EMPTY && f.count < 0) {
				err |= ERRF_MOTION;
				return true;
			}
		} else {
			root = __ldg(sc.asmb_root + m.z);
			if (root != REF_EMPTY) {
				const Frame parent = level_frame(sc);
				f = parent;
				mem->lv_inst[L + 1] = gi;
				mem->lv_frame[L + 1] = mem->lv_frame[L];
				if (XFORM && m.y > 0) {
					const DevInstance inst = sc.instances[gi];
					f = frame_merge(parent, sc.xforms + (size_t)inst.xform * 16, inst.xform_count, &mem->frames[L + 1]);
					if (f.count < 0) {
						err |= ERRF_MOTION;
						return true;
					}
					mem->lv_frame[L + 1] = L + 1;
				}
				mem->lv_count[L + 1] = f.count;
			}
		}
		if (root == REF_EMPTY) return true;
		if (sp - L + 1 > PSY_NODE_STACK) {
			err |= ERRF_STACK;
			return false;
		}
		const bool moved = XFORM && m.y > 0;
		mem->stack[sp++] = make_uint2((unsigned)(moved ? REF_LEVEL_RAY : REF_LEVEL), (unsigned)place);
		if (moved) {
			mem->lvr[L][0] = o.x; mem->lvr[L][1] = o.y; mem->lvr[L][2] = o.z;
			mem->lvr[L][3] = d.x; mem->lvr[L][4] = d.y; mem->lvr[L][5] = d.z;
			mem->lvr[L][6] = dinv.x; mem->lvr[L][7] = dinv.y; mem->lvr[L][8] = dinv.z;
			const M44 t = frame_at(f, time);
			set_ray(pos_to(t, io.origin()), dir_to(t, io.direction()));
		}
		++L;
		place = child;
		cur = root;
		return true;
	}

	// The transform of object instance gi, which carries its own, at the ray
	// time.  Returns false when it needs more motion samples than supported.
	static __device__ __noinline__ bool object_transform(const DevScene& sc, Frame parent, int gi, float time, M44* om) {
		FrameBuf buf;
		const DevInstance inst = sc.instances[gi];
		const Frame f = frame_merge(parent, sc.xforms + (size_t)inst.xform * 16, inst.xform_count, &buf);
		if (f.count < 0) return false;
		*om = frame_at(f, time);
		return true;
	}
	__device__ __forceinline__ bool object_frame(const DevScene& sc, int gi, M44* om) {
		if (object_transform(sc, level_frame(sc), gi, time, om)) return true;
		err |= ERRF_MOTION;
		return false;
	}

	// A leaf of class LEAF_SPHERE: a sphere or sphere light at rest in its
	// assembly's space, whole in its leaf record.
	__device__ __forceinline__ bool sphere_leaf(const DevScene& sc) {
		const int gi = cur & REF_LEAF_MASK;
		cur = REF_NONE;
		const float4 g = __ldg(reinterpret_cast<const float4*>(sc.leaves[gi].sphere));
		const float t = sphere_t(o, d, V3(g.x, g.y, g.z), g.w, max_t);
		if (!(t >= 0.0f)) return true;
		if (!(flags & RAY_OCCL)) max_t = t;
		return record(gi, t, 0.0f, 0.0f, 0.0f);
	}

	// A leaf of class LEAF_SIMPLE: moving or transformed spheres and sphere
	// lights, rectangle lights.
	__device__ __forceinline__ bool simple_leaf(const DevScene& sc) {
		const int gi = cur & REF_LEAF_MASK;
		cur = REF_NONE;
		const DevInstance inst = sc.instances[gi];
		const DevObject ob = sc.objects[inst.data];
		V3 lo = o, ld = d, li = dinv;
		if (XFORM && inst.xform_count > 0) {
			M44 om;
			if (!object_frame(sc, gi, &om)) return true;
			lo = pos_to(om, io.origin());
			ld = dir_to(om, io.direction());
			li = recip3(ld);
		}
		float t;
		if (ob.kind == OBJ_RECT_LIGHT) {
			float dx, dy;
			rect_light_at(sc, ob, time, &dx, &dy, nullptr);
			t = rect_light_t(lo, ld, li, dx, dy, max_t);
		} else {
			V3 cent;
			float radi;
			float col[3];
			if (ob.kind == OBJ_SPHERE) sphere_at(sc, ob, time, &cent, &radi);
			else light_at(sc, ob, time, &cent, &radi, col);
			t = sphere_t(lo, ld, cent, radi, max_t);
		}
		if (!(t >= 0.0f)) return true;
		if (!(flags & RAY_OCCL)) max_t = t;
		return record(gi, t, 0.0f, 0.0f, 0.0f);
	}

	// Width parameters for the patch of instance at transform `om` (oxf: its
	// own; else the level's, kept for the next patch in the same space).
	__device__ __forceinline__ RayFlip widths(const DevScene& sc, bool oxf, M44& om, V3 lo, V3 ld) {
		if (!oxf && (flags & RAY_WIDTH)) return mem->rw;
		V3 odx, ody, ddx, ddy;
		io.differentials(&odx, &ody, &ddx, &ddy);
		bool xf = oxf;
		if (XFORM && !oxf) {
			const Frame f = level_frame(sc);
			if (f.count > 0) {
				om = frame_at(f, time);
				xf = true;
			}
		}
		if (xf) {
			odx = dir_to(om, odx);
			ody = dir_to(om, ody);
			ddx = dir_to(om, ddx);
			ddy = dir_to(om, ddy);
		}
		const RayFlip w = ray_flip(ray_width_params(lo, ld, odx, ody, ddx, ddy));
		if (!oxf) {
			mem->rw = w;
			flags |= RAY_WIDTH;
		}
		return w;
	}

	// patch_odd_run on the bisection in progress (mem->p_*, its work `w`) for up
	// to `units` iterations.
	template <class WORK>
	__device__ __forceinline__ OddRun odd_run(const DevScene& sc, WORK& w, bool odd_patch, int units) {
		const OddRun r = patch_odd_run(w.c, w.st, mem->p_o, mem->p_dinv, mem->p_rw, max_t, (flags & RAY_OCCL) != 0,
		                               sc.dice_rate, sc.min_upoly_size, odd_patch, units);
		err |= r.err;
		if (r.took) {
			if (!(flags & RAY_OCCL)) max_t = r.hit.t;
			record(mem->p_inst, r.hit.t, r.hit.u, r.hit.v, r.hit.max_dim);
		}
		return r;
	}

	// A leaf of class LEAF_PATCH.  WHOLE: the bisection runs here, to its end.
	// Otherwise the patch's box is tested and its bisection set up (pmode) for
	// patch_step to carry on.  Returns false when the ray is finished.
	template <bool WHOLE>
	__device__ __forceinline__ bool patch_leaf(const DevScene& sc) {
		const int gi = cur & REF_LEAF_MASK;
		cur = REF_NONE;
		const int4 m = __ldg(reinterpret_cast<const int4*>(&sc.leaves[gi].data));  // vertices, transforms, -, kind
		V3 lo = o, ld = d, li = dinv;
		const bool odd_patch = (m.w & LEAF_PATCH_ODD) != 0;
		bool odd = (flags & RAY_ODD) != 0 || odd_patch;
		M44 om;
		const bool oxf = XFORM && m.y > 0;
		if (oxf) {
			if (!object_frame(sc, gi, &om)) return true;
			lo = pos_to(om, io.origin());
			ld = dir_to(om, io.direction());
			li = recip3(ld);
			odd = odd_ray(lo, ld, li) || odd_patch;
		}
		const float* v = sc.fpool + m.x;
		const int pm = m.w & PM_KIND;
		const bool occl = (flags & RAY_OCCL) != 0;
		const float dr = sc.dice_rate, mu = sc.min_upoly_size;
		bool live = true, in = false;
		// one patch kind: its bisection state and the number of its time samples
		auto one = [&](auto& w) {
			constexpr int NV = sizeof(w.c.cur[0]) / sizeof(V3), N = sizeof(w.c.cur) / sizeof(w.c.cur[0]);
			if (odd) {
				in = patch_odd_begin<NV, N>(w.c, v, time, lo, li, max_t, odd_patch);
				if (WHOLE && in) {
					mem->p_rw = widths(sc, oxf, om, lo, ld);
					mem->p_inst = gi;
					mem->p_o = lo;
					mem->p_dinv = li;
					live = odd_run(sc, w, odd_patch, 0x7fffffff).state != PATCH_BLOCKED;
				}
				return;
			}
			PatchCursor<NV, N> pc;
			in = patch_begin<NV, N, TEST_CLEAN>(pc, v, time, lo, li, max_t);
			if (!in) return;
			if constexpr (WHOLE) {
				const RayFlip f = widths(sc, oxf, om, lo, ld);
				int units = 0x7fffffff;
				live = patch_run<NV, N, TEST_CLEAN>(pc, w.st, lo, li, f, &max_t, occl, dr, mu, units, &err,
				                                    [&](float t, float u, float v2, float md) { record(gi, t, u, v2, md); }) !=
				       PATCH_BLOCKED;
			} else {
				w.c = pc;
			}
		};
		if constexpr ((F & FEAT_BILINEAR) != 0) {
			if (pm == PM_BILINEAR1) one(still_work<4>());
			else if (TS == 2 && pm == PM_BILINEAR2) one(work<4>());
		}
		if constexpr ((F & FEAT_BICUBIC) != 0) {
			if (pm == PM_BICUBIC1) one(still_work<16>());
			else if (TS == 2 && pm == PM_BICUBIC2) one(work<16>());
		}
		if (!WHOLE && in) {
			mem->p_rw = widths(sc, oxf, om, lo, ld);
			pmode = pm | (odd ? PM_ODD : 0) | (odd_patch ? PM_ODD_PATCH : 0);
			mem->p_inst = gi;
			mem->p_o = lo;
			mem->p_dinv = li;
		}
		return live;
	}

	// Carries the bisection in progress on for up to `units` iterations of its
	// loop (`units` is left at the iterations not used).  Returns false when
	// the ray is finished (an occlusion ray's hit).
	__device__ __forceinline__ bool patch_step(const DevScene& sc, int& units) {
		int r = PATCH_DONE;
		const int pm = pmode & PM_KIND;
		const bool occl = (flags & RAY_OCCL) != 0;
		const float dr = sc.dice_rate, mu = sc.min_upoly_size;
		const RayFlip w = mem->p_rw;
		const V3 lo = mem->p_o, li = mem->p_dinv;
		// the cursor runs as a local copy (registers) and goes back to the
		// state only when the bisection stops short of its end
		auto run = [&](auto& pw) {
			if (pmode & PM_ODD) {
				const OddRun o = odd_run(sc, pw, (pmode & PM_ODD_PATCH) != 0, units);
				r = o.state;
				units = o.units;
				return;
			}
			auto pc = pw.c;
			r = patch_run<sizeof(pc.cur[0]) / sizeof(V3), sizeof(pc.cur) / sizeof(pc.cur[0]), TEST_CLEAN>(
			    pc, pw.st, lo, li, w, &max_t, occl, dr, mu, units, &err,
			    [&](float t, float u, float v, float md) { record(mem->p_inst, t, u, v, md); });
			if (r == PATCH_MORE) pw.c = pc;
		};
		if constexpr ((F & FEAT_BILINEAR) != 0) {
			if (pm == PM_BILINEAR1) run(still_work<4>());
			else if (TS == 2 && pm == PM_BILINEAR2) run(work<4>());
		}
		if constexpr ((F & FEAT_BICUBIC) != 0) {
			if (pm == PM_BICUBIC1) run(still_work<16>());
			else if (TS == 2 && pm == PM_BICUBIC2) run(work<16>());
		}
		if (r == PATCH_MORE) return true;
		pmode = PM_NONE;
		return r != PATCH_BLOCKED;
	}

	// A lane that runs its ray alone: the whole walk.  The closest hit does
	// not depend on the order objects are tested in (a sub-patch's box lies
	// inside its parent's, so max_t pruning only drops leaves that could not
	// be closer), except for exact ties.
	__device__ __forceinline__ void walk(const DevScene& sc) {
		bool live = pop(sc);
		while (live) {
			while (live && cur >= 0) live = node_step(sc) && pop(sc);
			if (!live) return;
			const int cls = leaf_class(cur);
			if (NESTED && cls == LEAF_ENTER) live = enter(sc);
			else if (cls == LEAF_SPHERE) live = sphere_leaf(sc);
			else if ((F & (FEAT_BILINEAR | FEAT_BICUBIC)) && cls == LEAF_PATCH) live = patch_leaf<true>(sc);
			else live = simple_leaf(sc);
			live = live && pop(sc);
		}
	}
};

}  // namespace psy

#endif
