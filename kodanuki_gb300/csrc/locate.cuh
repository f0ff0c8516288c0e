// Locating the octree leaf a point lies in, for the device and, to check it,
// the host.
#pragma once

#include "program.cuh"
#include "world.h"

namespace kdn {

// A read-only load: through the read-only data cache on the device.
template <typename T>
KDN_HD T loadOnce(const T* p) {
#ifdef __CUDA_ARCH__
	return __ldg(p);
#else
	return *p;
#endif
}

// The place below a coordinate's estimate; not a number is place 0.
KDN_HD int placeBelow(float x) {
#ifdef __CUDA_ARCH__
	return __float2int_rd(x);
#else
	return x >= 2147483648.0f ? 0x7FFFFFFF : x >= -2147483648.0f ? int(floorf(x)) : x < 0.0f ? int(0x80000000) : 0;
#endif
}

// A point's place among the tabled walls, the boundary's past the region.
KDN_HD void placeOf(const DeviceWorld& w, const float p[3], int place[3]) {
	const int n = 1 << w.fineLevel;
	for (int a = 0; a < 3; ++a) {
		int i = placeBelow(fmaf(p[a], w.scale[a], w.bias[a]));
		i     = i < 0 ? 0 : i > n - 1 ? n - 1 : i;
		if (p[a] >= loadOnce(w.walls + a * (n + 1) + i + 1)) ++i;
		place[a] = i > n - 1 ? n - 1 : i;
	}
}

// The entry at a place (world.h kEntryLeaf): a leaf, or below the finest
// tabled level an inner node.
KDN_HD uint32_t entryAt(const DeviceWorld& w, const int place[3]) {
	uint32_t s     = w.fineLevel - w.gridLevel;
	uint32_t entry = loadOnce(w.grid + ((size_t(place[2] >> s) << w.gridLevel | size_t(place[1] >> s)) << w.gridLevel | size_t(place[0] >> s)));
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
	while (!(entry & kEntryLeaf) && s > 0) {
		// the place's next two bits an axis (the last one alone where one is left)
		const int mask = s > 1 ? 3 : 1;
		s -= s > 1 ? 2 : 1;
		entry = loadOnce(w.bricks + size_t(entry) * kBrick + ((place[0] >> s & mask) | (place[1] >> s & mask) << 2 | (place[2] >> s & mask) << 4));
	}
	return entry;
}

// The leaf below an inner node of the finest tabled level, and its box.
KDN_HD int32_t descend(const DeviceWorld& w, const float p[3], int32_t node, float lo[3], float hi[3]) {
	for (int depth = 0; depth < 30 && node >= 0; ++depth) {
		int o = 0;
		for (int a = 0; a < 3; ++a) {
			const float mid = 0.5f * (lo[a] + hi[a]);
			if (p[a] >= mid) {
				o |= 1 << a;
				lo[a] = mid;
			} else {
				hi[a] = mid;
			}
		}
		node = loadOnce(w.nodes + node + o);
	}
	return node;
}

// The leaf a point lies in.
KDN_HD uint32_t locate(const DeviceWorld& w, const float p[3]) {
	int place[3];
	placeOf(w, p, place);
	const uint32_t entry = entryAt(w, place);
	if (entry & kEntryLeaf) return entry & kEntryIndex;
	float lo[3], hi[3];
	for (int a = 0; a < 3; ++a) {
		const float* walls = w.walls + a * ((1 << w.fineLevel) + 1) + place[a];
		lo[a]              = loadOnce(walls);
		hi[a]              = loadOnce(walls + 1);
	}
	return uint32_t(~descend(w, p, int32_t(entry), lo, hi));
}

// The descent from the root alone, the reference for locate().
KDN_HD uint32_t descendFromRoot(const DeviceWorld& w, const float p[3]) {
	float lo[3], hi[3];
	for (int a = 0; a < 3; ++a) {
		lo[a] = w.lower[a];
		hi[a] = w.lower[a] + w.size[a];
	}
	return uint32_t(~descend(w, p, loadOnce(&w.nodes[0]), lo, hi));
}

} // namespace kdn
