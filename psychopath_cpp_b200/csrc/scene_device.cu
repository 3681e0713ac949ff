/*
 * The last steps of a scene's upload, on the device: what the builders left
 * (host or device built) is put into the form the render reads.
 */
#include "kernels.h"

namespace psy {

// ---------------------------------------------------------------------
// Tree references and absent children (the traversal's node form)
// ---------------------------------------------------------------------
// Boxes that the traversal may test with minima and maxima of the two planes
// of an axis: finite, and not inverted (a sphere of negative radius has an
// inverted box; by the ray's sign, as the reference tests, no ray hits it).
__device__ bool plain_boxes(const float* b, int nchild) {
	for (int axis = 0; axis < 3; ++axis)
		for (int c = 0; c < nchild; ++c) {
			const float lo = b[8 * axis + c], hi = b[8 * axis + 4 + c];
			if (!(fabsf(lo) < 1e37f) || !(fabsf(hi) < 1e37f) || !(lo <= hi)) return false;
		}
	return true;
}

// A builder's reference in the traversal's form.  `flags` holds the nodes'
// REF_NODE_* bits.
__device__ int finished_ref(int ref, const DevLeaf* leaves, const int* flags) {
	if (ref == REF_EMPTY) return ref;
	if (ref >= 0) return ref | flags[ref];
	const int gi = leaf_instance(ref);
	return class_ref(leaves[gi].kind >> 4, gi);
}

__global__ void node_flags_kernel(DevNode* nodes, float* extra, int n, int* flags) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	DevNode& nd = nodes[i];
	// (the test of plain nodes takes the first two children for granted)
	bool plain = nd.nchild >= 2 && plain_boxes(nd.b, nd.nchild);
	for (int t = 1; t < nd.ts; ++t) plain = plain && plain_boxes(extra + (size_t)(nd.extra + t - 1) * 24, nd.nchild);
	flags[i] = (nd.ts > 1 ? REF_NODE_MOVING : 0) | (plain ? 0 : REF_NODE_ODD);
	for (int t = 0; t < nd.ts || t == 0; ++t) {
		float* b = t == 0 ? nd.b : extra + (size_t)(nd.extra + t - 1) * 24;
		for (int k = 0; k < 24; ++k)
			if ((k & 3) >= nd.nchild) b[k] = (k & 4) ? -ABSENT_PLANE : ABSENT_PLANE;
	}
}

__global__ void node_refs_kernel(DevNode* nodes, int n, const DevLeaf* leaves, const int* flags) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	for (int c = 0; c < 4; ++c) nodes[i].child[c] = finished_ref(nodes[i].child[c], leaves, flags);
}

// Root references: of every assembly, and of every placement.
__global__ void root_refs_kernel(const DevAssembly* assemblies, int n, DevPlace* places, int np, const DevLeaf* leaves,
                                 const int* flags, int* asmb_root) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) asmb_root[i] = finished_ref(assemblies[i].root, leaves, flags);
	if (i < np) places[i].root = finished_ref(assemblies[places[i].asmb].root, leaves, flags);
}

cudaError_t launch_finish_nodes(DevNode* nodes, float* extra, int n, const DevLeaf* leaves, const DevAssembly* assemblies,
                                int assembly_count, DevPlace* places, int place_count, int* flags, int* asmb_root,
                                cudaStream_t st) {
	if (n > 0) {
		node_flags_kernel<<<(n + 127) / 128, 128, 0, st>>>(nodes, extra, n, flags);
		node_refs_kernel<<<(n + 127) / 128, 128, 0, st>>>(nodes, n, leaves, flags);
	}
	const int m = assembly_count > place_count ? assembly_count : place_count;
	root_refs_kernel<<<(m + 127) / 128, 128, 0, st>>>(assemblies, assembly_count, places, place_count, leaves, flags,
	                                                  asmb_root);
	return cudaGetLastError();
}

// ---------------------------------------------------------------------
// The light trees' children side by side (DevLightPair), with the parts of
// node_prob that depend on the node alone, in its float operations.
// ---------------------------------------------------------------------
__global__ void light_pairs_kernel(const DevLightNode* __restrict__ nodes, int n, DevLightPair* __restrict__ pairs) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n || nodes[i].is_leaf) return;
	DevLightPair p = {};
	auto child = [&](int c, float* centre, float* r2, float* e, int* ref) {
		const DevLightNode nd = nodes[c];
		Box b;
		b.lo = V3(nd.lo[0], nd.lo[1], nd.lo[2]);
		b.hi = V3(nd.hi[0], nd.hi[1], nd.hi[2]);
		const V3 m = box_center(b);
		centre[0] = m.x; centre[1] = m.y; centre[2] = m.z;
		const float r = box_diagonal(b) * 0.5f;
		*r2 = r * r;
		*e = nd.energy * (1.0f / *r2);
		if (nd.ts > 1) *r2 = -1.0f;
		*ref = nd.is_leaf ? -(nd.c1 + 1) : c;
	};
	child(nodes[i].c1, p.c1, &p.r2_1, &p.e1, &p.ref1);
	child(nodes[i].c2, p.c2, &p.r2_2, &p.e2, &p.ref2);
	pairs[i] = p;
}

cudaError_t launch_light_pairs(const DevLightNode* nodes, int n, DevLightPair* pairs, cudaStream_t st) {
	if (n == 0) return cudaSuccess;
	light_pairs_kernel<<<(n + 255) / 256, 256, 0, st>>>(nodes, n, pairs);
	return cudaGetLastError();
}

}  // namespace psy
