/*
 * Device scene layout (host + device).
 *
 * One flat set of arrays per uploaded scene, resident in HBM:
 *   assemblies[]   per-assembly roots and table bases
 *   leaves[]       per instance: what the traversal reads of it
 *   places[]       the unrolled assembly instances (DevPlace)
 *   instances[]    global instance table (all assemblies, contiguous per assembly)
 *   objects[]      global object table; geometry in the float pool
 *   nodes[]        BVH4 inner nodes, 128-byte records: the 4 child boxes of
 *                  time sample 0 as BBox4 SoA (xmin[4] xmax[4] ymin[4] ymax[4]
 *                  zmin[4] zmax[4], the reference's BBox4 layout,
 *                  basics/bbox.hpp:432-448) + child refs; further time
 *                  samples in node_extra[]
 *   xforms[]       16-float matrices, per assembly
 *   light_nodes[]  light-tree nodes
 *   shaders[]      surface shaders
 */
#ifndef PSY_SCENE_H
#define PSY_SCENE_H

#include <cstdint>

#include "psy_math.h"

namespace psy {

enum : int { OBJ_SPHERE = 0, OBJ_BILINEAR = 1, OBJ_BICUBIC = 2, OBJ_SPHERE_LIGHT = 3, OBJ_RECT_LIGHT = 4 };
enum : int { INST_OBJECT = 0, INST_ASSEMBLY = 1 };
enum : int { SHADER_LAMBERT = 0, SHADER_EMIT = 1, SHADER_GTR = 2 };
enum : int { CLOSURE_NONE = 0, CLOSURE_LAMBERT = 1, CLOSURE_EMIT = 2, CLOSURE_GTR = 3 };

// Device error flags, OR-ed into the context's status word by kernels.
enum : unsigned { ERRF_STACK = 1u, ERRF_MOTION = 4u, ERRF_TIMEOUT = 8u, ERRF_NOLIGHT = 16u,
                  ERRF_BISECT = 32u /* a patch bisection exceeded its step bound */ };

// Scene features that select a compiled variant of the traversal kernels.
enum : unsigned {
	FEAT_NESTED = 1u,        // assembly instances (levels)
	FEAT_XFORM = 2u,         // instance transforms
	FEAT_BICUBIC = 4u,       // bicubic patches
	FEAT_PATCH_MOTION = 8u,  // patches with two time samples
	FEAT_BILINEAR = 16u,     // bilinear patches
	FEAT_GTR = 32u,          // GTR shaders (shading only)
	FEAT_FLAT = 16u,         // spheres, lights and bilinear patches in one level
	FEAT_STILL_BICUBIC = 7u, // levels, transforms, bicubic patches (no bilinear, no patch motion)
	FEAT_STILL = 23u,        // everything but patch motion
	FEAT_ALL = 31u
};

// The compiled variant that covers a scene's features (the smallest of
// FEAT_FLAT, FEAT_STILL_BICUBIC, FEAT_STILL, FEAT_ALL: smaller variants
// leave out the code of absent features).
inline unsigned feature_variant(unsigned f) {
	f &= (unsigned)FEAT_ALL;
	if ((f & ~FEAT_FLAT) == 0u) return FEAT_FLAT;
	if ((f & ~FEAT_STILL_BICUBIC) == 0u) return FEAT_STILL_BICUBIC;
	if ((f & ~FEAT_STILL) == 0u) return FEAT_STILL;
	return FEAT_ALL;
}

// A child reference in a BVH4 node or an assembly root, as the builders
// leave it:
//   >= 0          inner node index (global)
//   < 0, != EMPTY leaf: global instance index = -(ref + 1)
static constexpr int REF_EMPTY = (int)0x80000000;
PSY_HD int leaf_ref(int instance) { return -(instance + 1); }
PSY_HD int leaf_instance(int ref) { return -(ref + 1); }

// The form the traversal reads (finish_nodes, scene_device.cu): an inner
// node's index with what its test needs to know before the node is read, or
// a leaf's class and global instance index.
static constexpr int REF_NODE_MOVING = 1 << 30;  // more than one time sample
static constexpr int REF_NODE_ODD = 1 << 29;     // a box is not finite, or inverted; or there is one child only
static constexpr int REF_NODE_MASK = (1 << 29) - 1;
static constexpr int REF_LEAF_MASK = (1 << 28) - 1;
static constexpr int REF_MAX_NODES = 1 << 29, REF_MAX_INSTANCES = 1 << 28;
enum : int {
	LEAF_ENTER = 1,   // assembly instance
	LEAF_SPHERE = 2,  // sphere or sphere light at rest in its assembly's space
	LEAF_SIMPLE = 3,  // other spheres, sphere lights and rectangle lights
	LEAF_PATCH = 4    // bilinear and bicubic patches
};
PSY_HD int leaf_class(int ref) { return (int)(((unsigned)ref >> 28) & 7u); }
PSY_HD int class_ref(int cls, int instance) { return (int)(0x80000000u | ((unsigned)cls << 28) | (unsigned)instance); }

// The planes of an absent child's box: finite, so that interpolating them
// stays so.  They keep nothing out: an absent child is told by its reference
// (REF_EMPTY), and only children 2 and 3 may be absent in a node that is not
// REF_NODE_ODD.
static constexpr float ABSENT_PLANE = 3.0e38f;

struct alignas(16) DevNode {
	float b[24];      // time sample 0 child bounds, BBox4 SoA
	int child[4];     // child refs
	int nchild;       // 2..4
	int ts;           // time samples
	int extra;        // index of time sample 1 in node_extra (24 floats per sample)
	int pad;
};
static_assert(sizeof(DevNode) == 128, "DevNode must be 128 bytes");

struct alignas(16) DevInstance {
	int kind;         // INST_OBJECT / INST_ASSEMBLY
	int data;         // global object index or global assembly index
	int xform;        // global transform index of the first motion sample
	int xform_count;  // 0 = none
	int shader;       // -1 = none
	int pad[3];
};

// What the traversal reads of an instance, by its global index.
struct alignas(16) DevLeaf {
	float sphere[4];  // LEAF_SPHERE: centre, radius
	int data;         // patches: float pool offset; assemblies: rank among its assembly's assembly instances
	int xforms;       // the instance's own motion samples
	int asmb;         // assemblies: assembly index
	int kind;         // patches: PM_* | LEAF_PATCH_ODD; bits 4..6: LEAF_* class
};
static constexpr int LEAF_PATCH_ODD = 8;  // a coordinate so large that sums of two may overflow

// An assembly instance as the walk from the root meets it: one entry per
// path of assembly instances (entry 0 is the root assembly), children of an
// entry in a row.  Holds what the path gives the level: the merged motion
// frame (place_frames, 16 floats per sample), the inherited shader and the
// element id so far.
struct alignas(16) DevPlace {
	int root;         // root reference of its assembly
	int child_base;   // entry of its first assembly instance
	int frame;        // first matrix of the merged frame
	int frame_count;  // its motion samples: 0 = no transform, -1 = more than supported
	int asmb;
	int inst_base;    // of its assembly
	int shader;
	int id_bits;      // of its assembly
	uint64_t id;
	int pad[2];
};
static_assert(sizeof(DevPlace) == 48, "DevPlace must be 48 bytes");
// Scenes that unroll to more entries than this are traversed with a level
// stack per ray instead (12 MB of entries, and the frames of as many
// transformed ones; a scene's upload spends about 0.2 us of host time per
// entry, whatever the assemblies hold besides, and none on a scene past it).
#define PSY_MAX_PLACES (1 << 18)

struct alignas(16) DevObject {
	int kind;
	int n0, n1, n2;   // time-sample counts (sphere/patch: n0; light: positions, radii, colours)
	int data;         // float pool offset
	int pad[3];
};

struct alignas(16) DevAssembly {
	int root;         // BVH4 root ref
	int inst_base;    // first global instance
	int inst_count;
	int id_bits;      // Assembly::element_id_bits()
	int light_root;   // light-tree root node (global), -1 = no lights
	int light_count;  // LightTree::light_count()
	float light_energy;
	int pad;
};

struct alignas(16) DevLightNode {
	float lo[3], hi[3];  // bounds, time sample 0
	float energy;
	int ts;              // bounds time samples
	int extra;           // index of time sample 1 in light_extra (6 floats per sample)
	int is_leaf;
	int c1, c2;          // children (global) or, for leaves, c1 = local instance index
};

// The two children of an inner light node as the tree walk reads them, at the
// node's own index: box centre, half diagonal squared (-1: the bounds move,
// read the node), energy over that, and where the child leads (an inner
// node's index, or -(local instance + 1) of a leaf).  Filled on the device
// after the upload (light_pairs_kernel).
struct alignas(64) DevLightPair {
	float c1[3], r2_1;
	float c2[3], r2_2;
	float e1, e2;
	float pad0[2];
	int ref1, ref2;
	int pad1[2];
};
static_assert(sizeof(DevLightPair) == 64, "DevLightPair must be 64 bytes");

struct alignas(16) DevShader {
	int kind;
	float col[3];
	// GTR: the parameters as GTRClosure::validate leaves them
	// (shading/surface_closure.hpp:352-372), its normalisation factor, and
	// pow(roughness^2, 1 - tail_shape); both computed on the host with the
	// host's powf, as the reference computes them
	float roughness, tail_shape, fresnel, norm;
	float pow_r2_1mt;
	int pad[3];
};

// Device pointers of an uploaded scene, passed to kernels by value.
struct DevScene {
	const DevAssembly* assemblies;
	const DevInstance* instances;
	const DevLeaf* leaves;
	const DevPlace* places;        // null: more than PSY_MAX_PLACES
	const float* place_frames;
	const int* asmb_root;          // per assembly: root reference (traversal form)
	const DevObject* objects;
	const DevNode* nodes;
	const float* node_extra;
	const float* xforms;
	const float* fpool;
	const DevLightNode* light_nodes;
	const DevLightPair* light_pairs;  // one per light node (inner nodes' are set)
	const float* light_extra;
	const DevShader* shaders;
	int assembly_count;
	int max_depth;        // deepest assembly nesting (root = 1)
	unsigned features;    // FEAT_* present in the scene
	float dice_rate;
	float min_upoly_size;
	// camera
	const float* cam_xforms;
	const float* cam_tfovs;
	const float* cam_apertures;
	const float* cam_focus;
	int cam_xform_count, cam_tfov_count, cam_aperture_count, cam_focus_count;
	float background[3];
	int light_node_count;  // all assemblies' light nodes (bounds a tree walk)
	// the host CPU's approximate reciprocal (psy_math.h), for matrix inverses
	RcpTable rcp;
};

}  // namespace psy

#endif
