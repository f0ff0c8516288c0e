// kdn_world_march: the march form of a cell's kept programs, run on the host
// by the same interpreter the trace kernel runs (program.cuh), a step at a
// time as its turns take them: what a step does not set itself or an earlier
// one store is not in its ray's column (here it is not a number).
#include "context.h"
#include "locate.cuh"
#include "program.cuh"

#include <limits>
#include <vector>

using kdn::Context;

extern "C" kdn_status kdn_world_march(kdn_ctx* handle, uint64_t i, const float* points, uint32_t n, float* values, size_t capacity, uint32_t* programs) {
	if (handle == nullptr || programs == nullptr || (n > 0 && (points == nullptr || values == nullptr))) return KDN_BAD_ARG;
	Context* ctx = reinterpret_cast<Context*>(handle);
	if (ctx->source != nullptr) ctx = ctx->source; // a sharing context reads its scene's world
	std::lock_guard<std::mutex> guard(ctx->lock);
	if (!ctx->built) return ctx->fail(KDN_NOT_READY, "kdn_world_march: no world built");
	if (ctx->flat.nodes.empty()) return ctx->fail(KDN_NOT_READY, "kdn_world_march: no device layout: " + ctx->flatError);
	const int64_t c = ctx->preorderCell(i);
	if (c < 0) return ctx->fail(KDN_BAD_ARG, "kdn_world_march: no such cell");
	const int32_t node = ctx->flat.nodes[size_t(c)];
	if (node >= 0) {
		*programs = 0; // an inner cell keeps no programs
		return KDN_OK;
	}
	const kdn::GpuLeaf& leaf = ctx->flat.leaves[size_t(~node)];
	*programs                = leaf.count;
	if (size_t(leaf.count) * n > capacity) return ctx->fail(KDN_BAD_ARG, "kdn_world_march: values too small");
	std::vector<float> slots(kdn::kMaxSlots, std::numeric_limits<float>::quiet_NaN());
	kdn::setConstants(slots.data(), 1);
	const float nowhere[3] = { slots[kdn::SlotX], slots[kdn::SlotX], slots[kdn::SlotX] };
	for (uint32_t k = 0; k < leaf.count; ++k) {
		const kdn::GpuProgram& g = ctx->flat.programs[leaf.first + k];
		const kdn::MarchStep* code = ctx->flat.march.data() + g.march;
		for (uint32_t j = 0; j < n; ++j) {
			float last = 0.0f;
			for (uint32_t at = 0; at < g.marchCount; at += kdn::unitsOf(code[at])) {
				kdn::setPoint(slots.data(), 1, nowhere);
				last = kdn::programStep(code[at], code + at + 1, slots.data(), 1, points + 3 * size_t(j), last);
			}
			values[size_t(k) * n + j] = last;
		}
	}
	return KDN_OK;
}

// kdn_world_locate: the leaf of each point by the trace kernel's locate()
// (grid, then descent) and by the descent from the root, on the host.
extern "C" kdn_status kdn_world_locate(kdn_ctx* handle, const float* points, uint32_t n, uint32_t* by_grid, uint32_t* by_descent) {
	if (handle == nullptr || (n > 0 && (points == nullptr || by_grid == nullptr || by_descent == nullptr))) return KDN_BAD_ARG;
	Context* ctx = reinterpret_cast<Context*>(handle);
	if (ctx->source != nullptr) ctx = ctx->source; // a sharing context reads its scene's world
	std::lock_guard<std::mutex> guard(ctx->lock);
	if (!ctx->built) return ctx->fail(KDN_NOT_READY, "kdn_world_locate: no world built");
	if (ctx->flat.nodes.empty()) return ctx->fail(KDN_NOT_READY, "kdn_world_locate: no device layout: " + ctx->flatError);
	kdn::DeviceWorld w {};
	w.nodes     = ctx->flat.nodes.data();
	w.grid      = ctx->gridCells.data();
	w.bricks    = ctx->bricks.data();
	w.walls     = ctx->walls.data();
	ctx->setLocating(w);
	for (uint32_t j = 0; j < n; ++j) {
		by_grid[j]    = kdn::locate(w, points + 3 * size_t(j));
		by_descent[j] = kdn::descendFromRoot(w, points + 3 * size_t(j));
	}
	return KDN_OK;
}
