// Test harness: the traversal tables of a scene (scene_build.cpp, compiled for
// the host) with `placed` instances of one assembly of `objects` spheres.
#include <chrono>

#include "scene_build.h"

using namespace psy;

// Seconds that build_tables takes.  Sets the number of placements, and whether
// every entry is what its instance gives it.
extern "C" double place_tables(int objects, int placed, int limit, int* places, int* right) {
	BuiltScene b;
	b.fpool = {0.0f, 0.0f, 0.0f, 1.0f};
	DevObject ball{};
	ball.kind = OBJ_SPHERE;
	ball.n0 = 1;
	b.objects.push_back(ball);
	DevAssembly root{}, group{};
	root.inst_count = placed + 1;
	root.id_bits = 20;
	group.inst_base = placed + 1;
	group.inst_count = objects;
	group.id_bits = 16;
	b.assemblies = {root, group};
	DevInstance in{};
	in.kind = INST_OBJECT;
	in.shader = -1;
	b.instances.push_back(in);  // an object before the placed assemblies
	in.kind = INST_ASSEMBLY;
	in.data = 1;
	in.xform_count = 1;
	b.xforms.resize(16);
	for (int i = 0; i < 4; ++i) b.xforms[5 * i] = 1.0f;
	for (int k = 0; k < placed; ++k) {
		in.shader = k % 3 - 1;
		b.instances.push_back(in);
	}
	in = DevInstance{};
	in.kind = INST_OBJECT;
	in.shader = -1;
	b.instances.resize(placed + 1 + objects, in);
	SceneTables t;
	const auto t0 = std::chrono::steady_clock::now();
	build_tables(b, limit, &t);
	const double s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
	*places = (int)t.places.size();
	*right = t.leaves.size() == b.instances.size();
	if (!t.places.empty()) {
		*right = *right && t.places[0].child_base == 1 && (int)t.places.size() == placed + 1 && t.frames.size() == 16u * (size_t)placed;
		for (int k = 0; k < placed; ++k) {
			const DevPlace& p = t.places[k + 1];
			*right = *right && t.leaves[k + 1].data == k && p.asmb == 1 && p.inst_base == placed + 1 && p.frame == k &&
			         p.frame_count == 1 && p.shader == k % 3 - 1 && p.id_bits == 16 && p.id == id_push(0, (uint64_t)k + 1, 20);
		}
	}
	return s;
}
