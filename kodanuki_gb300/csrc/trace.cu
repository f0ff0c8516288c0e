// The geometry kernels: sphere tracing through the cut octree.
//
// K-trace marches each ray (plugins/geometry/sphere_trace/sphere_trace.cpp:
// 203 sphereFromOutside, :188 sphereFromInside) by the field read from the
// kept programs of the octree leaf the point lies in: there the kept
// programs are exactly the objects that can be least (cut.cpp:442 deciding),
// so the step is the scene's field.  An empty leaf holds no surface, and
// the ray skips to where it leaves the cell.
// K-hit then evaluates the winning program once in duals for the normal and,
// of the same values, its source leaf (sphere_trace.cpp:115 sphereField).
#include "kernels.h"
#include "locate.cuh"
#include "program.cuh"

#include <cuda_runtime.h>

namespace kdn {

namespace {

constexpr int kTraceBlock = 128;
// Rays a warp holds.  With one a lane, 12 of 32 lanes work in a turn; with 64
// in hand 20 to 24 do (config 2's full frame 480 ms against 425 ms, a launch
// of 960 x 540 x 8 of its rays 3.57 against 2.80 ms).  48: 460 ms; 96 take
// the L1 the programs are read through: 480 ms.
constexpr uint32_t kPool = 64;
// A ray's register slots are a column of shared memory, one float a slot.
constexpr uint32_t kStride = kTraceBlock / 32 * kPool;
// rays of a warp that may wait at their ends before the warp sees to them (16
// and 32 measured within 2%)
constexpr uint32_t kWaiting = 24;
// steps a ray takes in a shaped cell (world.h LeafShape) a turn (1 to 8
// measured within 3%)
constexpr uint32_t kMovesPerTurn = 4;
// with kFew rays in hand or less (2, 4, 8, 16: a 256 x 256 frame of 16 samples
// 14.0, 10.1, 9.4, 9.3 ms), a ray takes up to kAlone steps a turn
constexpr uint32_t kFew = 8, kAlone = 256;
// steps worked out at once where a ray is seen to stay in its cell
constexpr uint32_t kRun = 8;

__device__ __forceinline__ float slopeOf(float part) {
	const float tiny = 1e-12f;
	return 1.0f / (fabsf(part) < tiny ? copysignf(tiny, part) : part);
}

__device__ __forceinline__ float tolerance(const float p[3]) {
	const float big = fmaxf(fabsf(p[0]), fmaxf(fabsf(p[1]), fabsf(p[2])));
	return 2e-6f * fmaxf(1.0f, big * 0.25f);
}

__device__ __forceinline__ float nudge(float t) { return fmaxf(1e-5f, fabsf(t) * 2e-6f); }

// Where a ray leaves the cell it is in: its walls ahead, one an axis.  A march
// only goes forward and p = o + d t rounds monotonically, so a ray in a cell
// leaves it by these walls alone and the three behind it are never looked at.
// They are kept as the ray sees them, with the sign of its direction taken off
// both sides: up an axis it is in the cell while p < upper, down an axis while
// p >= lower, which is -p < the next number above -lower.
__device__ __forceinline__ float forward(float p, float d) { return __uint_as_float(__float_as_uint(p) ^ (__float_as_uint(d) & 0x80000000u)); }

__device__ __forceinline__ bool inside(const float wall[3], const float p[3], const float d[3]) {
	return forward(p[0], d[0]) < wall[0] && forward(p[1], d[1]) < wall[1] && forward(p[2], d[2]) < wall[2];
}

// A cell ahead of a ray: its leaf, its walls, and the parameter the ray
// reaches them at (of an axis's two walls (w - o) * inv is never less at the
// one ahead).
struct Ahead {
	uint32_t leaf;
	float wall[3];
	float exit;
};

__device__ __forceinline__ void walledBy(Ahead& c, const float at[3], const float o[3], const float d[3], const float inv[3]) {
	c.exit = 3.0e38f;
	for (int a = 0; a < 3; ++a) {
		const float back  = 0.0f - at[a]; // +0 for a wall at 0
		const int32_t bit = __float_as_int(back);
		c.wall[a]         = __float_as_int(d[a]) < 0 ? __int_as_float(bit < 0 ? bit - 1 : bit + 1) : at[a];
		c.exit            = fminf(c.exit, (at[a] - o[a]) * inv[a]);
	}
}

// A leaf below the finest tabled level: the descent goes on by midpoints.
__device__ __noinline__ Ahead deepCell(const DeviceWorld& w, float3 point, int32_t node, int3 at, float3 origin, float3 along, float3 inverse) {
	const float p[3] = { point.x, point.y, point.z }, o[3] = { origin.x, origin.y, origin.z };
	const float d[3] = { along.x, along.y, along.z }, inv[3] = { inverse.x, inverse.y, inverse.z };
	const int place[3] = { at.x, at.y, at.z };
	float lo[3], hi[3];
	for (int a = 0; a < 3; ++a) {
		const float* walls = w.walls + a * ((1 << w.fineLevel) + 1) + place[a];
		lo[a]              = walls[0];
		hi[a]              = walls[1];
	}
	Ahead c;
	c.leaf = uint32_t(~descend(w, p, node, lo, hi));
	for (int a = 0; a < 3; ++a) lo[a] = __float_as_int(d[a]) < 0 ? lo[a] : hi[a];
	walledBy(c, lo, o, d, inv);
	return c;
}

// A program at a point, out of line: the turns' code below is what the
// instruction cache is for (config 2's full frame 400 ms, 430 with it inline).
__device__ __noinline__ float programValue(const MarchStep* code, uint32_t count, float* slots, float3 at) {
	const float p[3] = { at.x, at.y, at.z };
	return evalSlots(code, count, slots, kStride, p);
}

// A primitive step along one ray, with what does not change from a point to
// the next worked out: the ray's part along each term's axis, and the choices
// as masks.  The value is primitiveValue's to the bit but for a zero's sign (a
// value of zero lands, and is worked out again), for a ray of finite parts.
struct AlongRay {
	float from[3], by[3];   // the point's coordinate: from + by * t
	float c[3], h[3];       // the slabs
	float low[3];           // 0 where the term is squared by its positive part
	uint32_t keep[3], turn[3], has[3]; // |u|, -u and a term left out, as masks
	float r, e;
	uint32_t within;        // the inside term's mask
	bool fused1, fused2, single, plain, third;
};

__device__ __forceinline__ AlongRay alongRay(const MarchStep& s, const MarchParams& c, const MarchParams& h, const float o[3], const float d[3]) {
	AlongRay a;
	const uint32_t terms[3] = { s.a, s.b, s.c };
	for (uint32_t k = 0; k < 3; ++k) {
		const uint32_t axis = terms[k] & 3u, side = terms[k] >> kTermSideShift;
		a.from[k] = axis == 0 ? o[0] : axis == 1 ? o[1] : o[2];
		a.by[k]   = axis == 0 ? d[0] : axis == 1 ? d[1] : d[2];
		a.c[k]    = -c.v[k];
		a.h[k]    = -h.v[k];
		a.low[k]  = s.flags & SumPositive0 << k ? 0.0f : -__int_as_float(0x7F800000);
		a.keep[k] = side == SideAbs ? 0x7FFFFFFFu : 0xFFFFFFFFu;
		a.turn[k] = side == SideNegative ? 0x80000000u : 0u;
		a.has[k]  = s.flags & SumHas0 << k ? 0xFFFFFFFFu : 0u;
	}
	a.r      = h.v[3];
	a.e      = -c.v[3];
	a.within = s.m & PrimInside ? 0xFFFFFFFFu : 0u;
	a.fused1 = s.flags & SumFused1;
	a.fused2 = s.flags & SumFused2;
	a.single = s.m & PrimSingle;
	a.plain  = s.m & PrimPlain;
	a.third  = s.m & PrimThird;
	return a;
}

__device__ __forceinline__ float masked(float x, uint32_t mask) { return __uint_as_float(__float_as_uint(x) & mask); }

__device__ __forceinline__ float valueAlong(const AlongRay& a, float t) {
	float u[3], p[3];
	for (int k = 0; k < 3; ++k) {
		const float x = __fadd_rn(fmaf(a.by[k], t, a.from[k]), a.c[k]);
		u[k]          = __fadd_rn(__fadd_rn(__uint_as_float((__float_as_uint(x) & a.keep[k]) ^ a.turn[k]), a.h[k]), a.r);
		p[k]          = masked(fmaxf(u[k], a.low[k]), a.has[k]);
	}
	float sum = __fmul_rn(p[0], p[0]);
	sum       = a.fused1 ? fmaf(p[1], p[1], sum) : __fadd_rn(__fmul_rn(p[1], p[1]), sum);
	sum       = a.fused2 ? fmaf(p[2], p[2], sum) : __fadd_rn(__fmul_rn(p[2], p[2]), sum);
	float f   = marchSqrt(sum);
	f         = a.single ? fmaxf(p[0] + p[1] + p[2], 0.0f) : f; // one term, the others zero
	f         = a.plain ? u[0] : f;
	f         = __fadd_rn(f, masked(fminf(fmaxf(u[0], fmaxf(u[1], a.third ? u[2] : u[1])), 0.0f), a.within));
	return __fadd_rn(f, a.e);
}

struct Field {
	float least;    // least program value
	uint32_t index; // which kept program is least
	uint32_t count; // kept programs
	uint32_t first; // first GpuProgram of the leaf
};

// The field at p from the kept programs of its cell; no programs in an empty one.
__device__ __forceinline__ Field fieldAt(const DeviceWorld& w, const float p[3], float* slots, uint32_t& steps) {
	const GpuLeaf leaf = w.leaves[locate(w, p)];
	Field f { 3.0e38f, 0, leaf.shape == ShapeEmpty ? 0u : leaf.count, leaf.first };
	for (uint32_t k = 0; k < f.count; ++k) {
		const GpuProgram g = w.programs[f.first + k];
		const float v      = programValue(w.march + g.march, g.marchCount, slots, make_float3(p[0], p[1], p[2]));
		steps += g.marchSteps;
		if (v < f.least) {
			f.least = v;
			f.index = k;
		}
	}
	return f;
}

// The least value at p, and the index of the kept program that is least a
// little further along among those tied with it (sphere_trace.cpp:96).
__device__ __noinline__ uint32_t winnerAt(const DeviceWorld& w, float3 at, float3 along, const Field f, float* slots) {
	const float p[3] = { at.x, at.y, at.z };
	const float big  = fmaxf(fabsf(p[0]), fmaxf(fabsf(p[1]), fabsf(p[2])));
	const float band = 2e-6f * (1.0f + big);
	const float q[3] = { p[0] + along.x * 2e-5f, p[1] + along.y * 2e-5f, p[2] + along.z * 2e-5f };
	uint32_t winner  = f.index;
	float onWinner   = 3.0e38f;
	for (uint32_t k = 0; k < f.count; ++k) {
		const GpuProgram g = w.programs[f.first + k];
		if (!(programValue(w.march + g.march, g.marchCount, slots, make_float3(p[0], p[1], p[2])) - f.least <= band)) continue;
		const float on = programValue(w.march + g.march, g.marchCount, slots, make_float3(q[0], q[1], q[2]));
		if (on < onWinner) {
			onWinner = on;
			winner   = k;
		}
	}
	return winner;
}

// sphereFromInside at a point p within the tolerance of the nearest surface:
// read the field a little past it, at q.  kind 0: go on past (t += inset); 1:
// the ray leaves its solid here (winner among the cell's programs); 2: it
// meets a solid of another material (the program past the point).
struct InsideStop {
	uint32_t kind, first, index, steps;
};

__device__ __noinline__ InsideStop insideStop(const DeviceWorld& w, const uint32_t* objectMaterial, uint32_t medium, float3 p, float3 q, float3 along, const Field f, float* slots) {
	const float beyond[3] = { q.x, q.y, q.z };
	uint32_t steps        = 0;
	const Field past      = fieldAt(w, beyond, slots, steps);
	if (past.count == 0 || past.least > 0.0f) return InsideStop { 1, f.first, winnerAt(w, p, along, f, slots), steps };
	const GpuProgram g = w.programs[past.first + past.index];
	// a solid of another material than the one the ray is in: stop there
	if (objectMaterial != nullptr && objectMaterial[g.object] != medium) return InsideStop { 2, past.first, past.index, steps };
	return InsideStop { 0, 0, 0, steps };
}

// The march as a step machine.  A warp holds a pool of rays, more than it has
// lanes, in shared memory.  A ray waits to be located, or to step in a cell
// whose field its leaf record holds (empty, or a single slab or sphere: a few
// operations in registers), or for the programs of its cell, a step of theirs
// at a time; every turn the warp does the one thing most of its rays wait for,
// a lane a ray of those.  Rays that have landed or ended wait until there are
// several, and the ended take the next rays of the launch (one atomic a warp).
// A mode's number is its count's place in the warp's sum of them.
enum LaneMode : uint32_t { Locating = 1, Stepping = 1 << 8, Evaluating = 1 << 16, Fetch = 1 << 24, Landed = 3 << 24, Finished = 5 << 24 };

constexpr uint32_t kOwn = (kPool + 31) / 32; // rays of the pool whose modes a lane counts
constexpr uint32_t kWarps = kTraceBlock / 32;

// A warp's pool: each row a float4 or less of every ray.
struct Pool {
	float4 origin[kPool];    // o, up
	float4 direction[kPool]; // d, stepLimit | within << 31
	float4 inverse[kPool];   // 1 / d, the ray's index in the launch
	float4 at[kPool];        // t, step, the cell's exit and leaf
	float4 wall[kPool];      // the cell's walls; its shape and, from bit 8, what a step in it adds to the program step count
	// the field of a slab or a sphere.  In a cell of programs: what the ones
	// evaluated so far came to, the least value and the second least (from
	// inside a solid, the least magnitude), the last step's value, and pc
	float4 field[kPool];
	uint2 program[kPool];    // where the program in hand ends; which it is, of how many, and which was least (a byte each)
	uint32_t mode[kPool];
	uint32_t taken[32];      // the rays of this turn
};

// Four blocks an SM: 128 registers, 28 KB of shared memory and the slots'
// columns a block.  Five leave less L1 (config 2's full frame 453 against 431
// ms before a few rays were the whole warp's).
// What bounds it: the issue of instructions while the SMs are full (51% of the
// cycles, at 18 of 32 lanes), and in a launch by itself the last rays of it
// (the SMs stand idle for 41% of 2.67 ms, 960 x 540 x 8 rays of config 2).
__global__ void __launch_bounds__(kTraceBlock, 4) traceKernel(const __grid_constant__ TraceArgs args) {
	extern __shared__ float4 poolMemory[];
	const DeviceWorld& w = args.world;
	Pool& pool           = reinterpret_cast<Pool*>(poolMemory)[threadIdx.x / 32];
	// a ray's register slots: a column each
	float* const columns = reinterpret_cast<float*>(reinterpret_cast<Pool*>(poolMemory) + kWarps) + threadIdx.x / 32 * kPool;
	// a lane's capped rays in the low 16 bits, its carried ones in the high: one register
	uint32_t marchSteps = 0, programSteps = 0, traced = 0, cappedCarried = 0, longest = 0;
	// the steps a ray may take in this launch: a launch's budget, or the cap
	const uint32_t allowance = args.budget > 0 ? args.budget : kMarchSteps;
	// the rays: [0, n1) and, after them in the fetch order, [second, second + n2)
	const uint32_t n1 = args.count ? *args.count : args.n;
	const uint32_t n  = n1 + (args.secondCount ? *args.secondCount : 0u);
	const unsigned lane = threadIdx.x & 31u;

	if (blockIdx.x == 0 && threadIdx.x == 0) {
		if (args.left != nullptr && args.counters != nullptr && *args.left) atomicAdd(&args.counters[6], (unsigned long long) *args.left);
		for (uint32_t* c : { args.clear[0], args.clear[1] }) {
			if (c != nullptr) *c = 0;
		}
		if (args.reached != nullptr) {
			// the host's view of the frame: this launch has begun, and whether it has rays
			if (n == 0) args.reached[1] = args.chunk;
			__threadfence_system();
			args.reached[0] = args.turn;
		}
	}
	// a launch of few rays spreads them over its warps (a ray alone is marched
	// soonest, and nothing else waits for the lanes)
	const uint32_t warps = gridDim.x * kWarps;
	const uint32_t share = min(kPool, (n + warps - 1u) / warps);
	if (n == 0) return;
	for (uint32_t r = lane; r < kPool; r += 32u) {
		pool.mode[r] = r < share ? Fetch : Finished;
		setConstants(columns + r, kStride);
	}
	__syncwarp();

	// the ray in a lane's hands this turn
	uint32_t r    = 0, mode = 0;
	float o[3] = { 0.0f, 0.0f, 0.0f }, d[3] = { 0.0f, 0.0f, 0.0f };
	float t = 0.0f, up = 0.0f;
	bool within   = false; // the ray started inside a solid
	uint32_t step = 0;
	// where the ray's march stops in this launch: the cap, or sooner its budget
	uint32_t stepLimit = 0;
	uint32_t kind      = 0; // shape and cost
	Ahead cell { kNoLeaf, { 0.0f, 0.0f, 0.0f }, 0.0f };
	// a ray ends: its state, the step counts, and the next ray
	auto done = [&](HitState h) {
		args.states[__float_as_uint(pool.inverse[r].w)] = h;
		marchSteps += h.steps; // less the steps it had when taken (at the fetch)
		longest = max(longest, h.steps);
		cappedCarried += h.kind == kCarried ? 0x10000u : (h.steps >= args.maxSteps ? 1u : 0u);
		mode = Fetch;
	};
	// past the cap or the region: a miss, which keeps where its march stopped
	// (a held path resumes it); out of this launch's budget before either:
	// carried, the march's whole state being (t, step)
	auto over = [&]() {
		if (step < stepLimit && t <= up) return false;
		const bool carried = step < args.maxSteps && t <= up;
		done(HitState { carried ? kCarried : 0u, t, kNoLeaf, 0, step });
		return true;
	};
	// a ray goes on from t to on, its march step taken: to the end of its march,
	// on in its cell, or out of it.  A step too small to move it would be taken
	// again to the limit: cost, what one adds to the program step count.
	auto goOn = [&](float on, uint32_t stepCost) {
		if (on == t) {
			programSteps += (stepLimit - step) * stepCost;
			step = stepLimit;
		}
		t = on;
		if (over()) return;
		const float p[3] = { o[0] + d[0] * t, o[1] + d[1] * t, o[2] + d[2] * t };
		mode             = inside(cell.wall, p, d) ? Stepping : Locating;
	};
	// the ray of a turn, from the pool and back
	auto load = [&]() {
		const float4 a = pool.origin[r], b = pool.direction[r], c = pool.at[r], e = pool.wall[r];
		o[0] = a.x, o[1] = a.y, o[2] = a.z, up = a.w;
		d[0] = b.x, d[1] = b.y, d[2] = b.z;
		stepLimit    = __float_as_uint(b.w) & 0x7FFFFFFFu;
		within       = __float_as_uint(b.w) >> 31 != 0u;
		t            = c.x;
		step         = __float_as_uint(c.y);
		cell.exit    = c.z;
		cell.leaf    = __float_as_uint(c.w);
		cell.wall[0] = e.x, cell.wall[1] = e.y, cell.wall[2] = e.z;
		kind         = __float_as_uint(e.w);
	};
	auto keep = [&]() {
		pool.at[r]   = make_float4(t, __uint_as_float(step), cell.exit, __uint_as_float(cell.leaf));
		pool.mode[r] = mode;
	};
	// the rays in one mode, a lane each: how many (the others take none)
	uint32_t own[kOwn];
	auto modeAt = [&](uint32_t k) { return kPool % 32 == 0 || lane + k * 32u < kPool ? pool.mode[lane + k * 32u] : 0u; };
	auto take = [&](uint32_t which) {
		uint32_t first = 0;
		const unsigned before = (1u << lane) - 1u;
		for (uint32_t k = 0; k < kOwn; ++k) {
			const unsigned those = __ballot_sync(0xFFFFFFFFu, own[k] == which);
			const uint32_t place = first + uint32_t(__popc(those & before));
			if (own[k] == which && place < 32u) pool.taken[place] = lane + k * 32u;
			first += uint32_t(__popc(those));
		}
		__syncwarp();
		r = pool.taken[lane];
		return min(first, 32u);
	};
	uint32_t finished = kPool - share; // places without a ray, the launch's all taken

	for (;;) {
		uint32_t sum = 0;
		for (uint32_t k = 0; k < kOwn; ++k) {
			own[k] = modeAt(k);
			sum += own[k];
		}
		const uint32_t modes      = __reduce_add_sync(0xFFFFFFFFu, sum);
		const uint32_t locating   = modes & 0xFFu, stepping = modes >> 8 & 0xFFu, evaluating = modes >> 16 & 0xFFu;
		const uint32_t busy       = locating + stepping + evaluating;
		const uint32_t waiting    = kPool - busy - finished;
		if (waiting >= kWaiting || waiting > busy) {
			if (lane < take(Landed)) {
				load();
				mode = Landed;
				// field and order hold what the march step came to: the least of the
				// cell's programs, the second least (from inside, the least magnitude)
				// and the least's index
				const GpuLeaf leaf = w.leaves[cell.leaf];
				const float4 field = pool.field[r];
				float* slots       = columns + r;
				const float p[3]   = { o[0] + d[0] * t, o[1] + d[1] * t, o[2] + d[2] * t };
				const Field f { field.x, pool.program[r].y >> 16, leaf.count, leaf.first };
				const float3 at = make_float3(p[0], p[1], p[2]), along = make_float3(d[0], d[1], d[2]);
				if (!within) {
					const float big = fmaxf(fabsf(p[0]), fmaxf(fabsf(p[1]), fabsf(p[2])));
					const bool tied = field.y - field.x <= 2e-6f * (1.0f + big);
					const uint32_t winner = tied ? winnerAt(w, at, along, f, slots) : f.index;
					done(HitState { 1, t, f.first, winner, step });
				} else {
					// sphereFromInside: stand on the nearest surface and read the field past it
					const float inset = 2.0f * tolerance(p), past = t + inset;
					const InsideStop stop = insideStop(w, args.objectMaterial, args.rays[__float_as_uint(pool.inverse[r].w)].within, at,
					                                   make_float3(o[0] + d[0] * past, o[1] + d[1] * past, o[2] + d[2] * past), along, f, slots);
					programSteps += stop.steps;
					if (stop.kind == 0) {
						uint32_t each = stop.steps;
						if (past == t) {
							for (uint32_t k = 0; k < leaf.count; ++k) each += w.programs[leaf.first + k].marchSteps;
						}
						goOn(past, each);
						if (mode == Stepping) mode = Locating; // the cell's field is to be read again
					} else {
						done(HitState { stop.kind, t, stop.first, stop.index, step });
					}
				}
				keep();
			}
			__syncwarp();
			for (uint32_t k = 0; k < kOwn; ++k) own[k] = modeAt(k);
			// take new rays, one atomic a warp
			const uint32_t wanted = take(Fetch);
			if (wanted) {
				uint32_t base = 0;
				if (lane == 0) base = atomicAdd(args.fetch, wanted);
				base = __shfl_sync(0xFFFFFFFFu, base, 0);
				if (lane < wanted) {
					uint32_t ray = base + lane;
					if (ray >= n) {
						pool.mode[r] = Finished;
					} else {
						if (ray >= n1) ray = args.second + (ray - n1);
						const kdn_ray from = args.rays[ray];
						within             = from.inside != 0;
						float inv[3];
						for (int a = 0; a < 3; ++a) {
							o[a]   = from.origin[a];
							d[a]   = from.direction[a];
							inv[a] = slopeOf(d[a]);
						}
						float lo = 0.0f;
						up       = from.far;
						for (int a = 0; a < 3; ++a) {
							const float x = (w.lower[a] - o[a]) * inv[a];
							const float y = (w.lower[a] + w.size[a] - o[a]) * inv[a];
							lo            = fmaxf(lo, fminf(x, y));
							up            = fminf(up, fmaxf(x, y));
						}
						t    = lo;
						step = 0;
						// a carried ray goes on where its march stood
						if (args.carry != nullptr && (from.pad_[0] & kRayResumes)) {
							const uint2 c = args.carry[ray];
							t             = __uint_as_float(c.x);
							step          = c.y;
						} else {
							++traced; // a segment is counted once, in the launch that starts it
						}
						stepLimit = min(args.maxSteps, step + allowance);
						marchSteps -= step;
						pool.origin[r]    = make_float4(o[0], o[1], o[2], up);
						pool.direction[r] = make_float4(d[0], d[1], d[2], __uint_as_float(stepLimit | (within ? 0x80000000u : 0u)));
						pool.inverse[r]   = make_float4(inv[0], inv[1], inv[2], __uint_as_float(ray));
						if (up < lo) done(HitState { 0, t, kNoLeaf, 0, step });
						else if (!over()) mode = Locating;
						keep();
					}
				}
				__syncwarp();
			}
			finished = 0;
			for (uint32_t k = 0; k < kOwn; ++k) finished += uint32_t(__popc(__ballot_sync(0xFFFFFFFFu, modeAt(k) == Finished)));
			if (finished == kPool) break;
			continue;
		}
		if (evaluating >= locating && evaluating >= stepping) {
			const uint32_t count = take(Evaluating);
			if (busy <= kFew) {
				// few rays in hand: whole march steps at a time, a share of the lanes a
				// ray (a ray that skims a box takes thousands of steps, and nothing else
				// is left to wait for).  Where the cell's programs are primitives, each
				// joined to the one before, a lane works out one primitive from
				// registers; else a program, or every so many.  A step is bound by its
				// chain of instructions, some 300 ns of them; a lane a ray took 500 for
				// a primitive and 1400 for a program of three (a 256 x 256 frame of 16
				// samples 13.3 against 9.4 ms, the interactive one of 4096 primitives
				// 18 against 14, the preview 5.1 against 3.4).
				const uint32_t wide  = count == 1u ? 32u : count == 2u ? 16u : count <= 4u ? 8u : 4u; // lanes a ray
				const uint32_t place = lane / wide, mine = lane & (wide - 1u);
				const bool leads     = mine == 0u && place < count;
				r                    = pool.taken[place < count ? place : 0u];
				load();
				const GpuLeaf leaf = w.leaves[cell.leaf];
				// the lane's primitive; which of its program's it is, and if the last
				MarchStep s {};
				uint32_t unit = 0, total = 0, nth = 0, longestProgram = 0, each = 0;
				bool ends = false, plain = true;
#pragma unroll 1
				for (uint32_t k = 0; k < leaf.count; ++k) {
					uint32_t pc = leaf.march, end = leaf.march + leaf.marchCount, cost = leaf.marchSteps;
					if (k != 0u) {
						const GpuProgram g = w.programs[leaf.first + k];
						pc   = g.march;
						end  = g.march + g.marchCount;
						cost = g.marchSteps;
					}
					each += cost;
					uint32_t at = 0;
#pragma unroll 1
					while (plain && pc < end) {
						const MarchStep x   = w.march[pc];
						const uint32_t next = pc + unitsOf(x);
						plain = primitiveStep(x) && total < wide && (x.op == FormPrimitive || x.m & PrimPrevious || x.w == SlotImm);
						if (total == mine) {
							s    = x;
							unit = pc;
							nth  = at;
							ends = next == end;
						}
						++total;
						++at;
						pc = next;
					}
					longestProgram = max(longestProgram, at);
				}
				for (int a = 0; a < 3; ++a) plain = plain && fabsf(o[a]) < 3.0e38f && fabsf(d[a]) < 3.0e38f;
				plain = __all_sync(0xFFFFFFFFu, plain);
				MarchParams c { { 0.0f, 0.0f, 0.0f, 0.0f } }, h { { 0.0f, 0.0f, 0.0f, -0.0f } };
				const bool holds = plain && mine < total; // a lane with a primitive
				if (holds) c = paramsAt(w.march + unit + 1);
				if (holds && s.m & PrimSized) h = paramsAt(w.march + unit + 2);
				const AlongRay primitive = alongRay(s, c, h, o, d);
				const uint32_t post = s.op & kMarchPostMask;
				const uint32_t rounds = __reduce_max_sync(0xFFFFFFFFu, longestProgram), most = __reduce_max_sync(0xFFFFFFFFu, plain ? total : wide);
				// the programs begin again at the first, and are counted again
				if (leads) {
					for (uint32_t k = pool.program[r].y >> 8 & 0xFFu; k-- > 0;) programSteps -= w.programs[leaf.first + k].marchSteps;
				}
				float* slots   = columns + lane; // no ray is within a program now
				float p[3]     = { o[0] + d[0] * t, o[1] + d[1] * t, o[2] + d[2] * t };
				uint32_t taken = 0;
				// a ray's march: on in its cell, landed, ended, or out of the cell
				enum { On, Lands, Ends, Leaves } state = On;
#pragma unroll 1
				for (uint32_t turn = 1; turn <= kAlone; ++turn) {
					float v = 3.0e38f;
					if (plain) {
						const float f = valueAlong(primitive, t);
						float last    = nth == 0u && post != PostNone ? posted(post, f, s.value, s.value, s.quarter) : f;
#pragma unroll 1
						for (uint32_t k = 1; k < rounds; ++k) {
							const float prior = __shfl_up_sync(0xFFFFFFFFu, last, 1);
							if (nth == k && post != PostNone) last = posted(post, f, s.m & PrimPrevious ? prior : s.value, s.value, s.quarter);
						}
						if (holds && ends) v = fminf(3.0e38f, within ? fabsf(last) : last);
					} else {
#pragma unroll 1
						for (uint32_t q = mine; q < leaf.count; q += wide) {
							const GpuProgram g = w.programs[leaf.first + q];
							const float u      = programValue(w.march + g.march, g.marchCount, slots, make_float3(p[0], p[1], p[2]));
							v                  = fminf(v, within ? fabsf(u) : u);
						}
					}
					// the least of a ray's lanes (of those that hold any)
					for (uint32_t k = 1; k < most; k *= 2u) v = fminf(v, __shfl_xor_sync(0xFFFFFFFFu, v, int(k)));
					v = __shfl_sync(0xFFFFFFFFu, v, 0, int(wide));
					if (state == On) {
						const float on = fminf(t + v, fmaxf(cell.exit, t) + nudge(t));
						++step;
						++taken;
						if (v < tolerance(p)) {
							state = Lands;
						} else {
							if (on == t) {
								taken += stepLimit - step;
								step = stepLimit;
							}
							t = on;
							for (int a = 0; a < 3; ++a) p[a] = o[a] + d[a] * t;
							state = !(step < stepLimit && t <= up) ? Ends : inside(cell.wall, p, d) ? On : Leaves;
						}
					}
					// until all have done with their cells, and where one has, for some steps
					const unsigned on = __ballot_sync(0xFFFFFFFFu, state == On);
					if (on == 0u || (on != 0xFFFFFFFFu && turn >= kRun)) break;
				}
				if (leads) {
					programSteps += taken * each;
					pool.program[r] = make_uint2(leaf.march + leaf.marchCount, leaf.count);
					float4 field    = make_float4(3.0e38f, 3.0e38f, 0.0f, __uint_as_float(leaf.march));
					mode            = Evaluating;
					if (state == Lands) {
						// the least of the programs, the second (from inside, the least
						// magnitude) and the least's index
						uint32_t index = 0;
#pragma unroll 1
						for (uint32_t k = 0; k < leaf.count; ++k) {
							const GpuProgram g = w.programs[leaf.first + k];
							const float v      = programValue(w.march + g.march, g.marchCount, slots, make_float3(p[0], p[1], p[2]));
							const bool lesser  = v < field.x;
							field.y            = within ? fminf(field.y, fabsf(v)) : lesser ? field.x : fminf(field.y, v);
							field.x            = lesser ? v : field.x;
							index              = lesser ? k : index;
						}
						pool.program[r].y = index << 16;
						mode              = Landed;
					} else if (state == Leaves) {
						mode = Locating;
					} else {
						over();
					}
					keep();
					pool.field[r]  = field;
					pool.wall[r].w = __uint_as_float((kind & 0xFFu) | uint32_t(leaf.marchSteps) << 8);
				}
			} else if (lane < count) {
				load();
				mode          = Evaluating;
				float4 f      = pool.field[r];
				uint2 program = pool.program[r];
				float* slots  = columns + r;
				float last    = f.z;
				// the program in hand: its code from pc to end, its last step's value, and
				// which it is, of how many, and which was least (a byte each)
				uint32_t pc = __float_as_uint(f.w), end = program.x, order = program.y, cost = kind >> 8;
				const float p[3]      = { o[0] + d[0] * t, o[1] + d[1] * t, o[2] + d[2] * t };
				const MarchStep s     = w.march[pc];
				const MarchStep* unit = w.march + pc + 1;
				pc += unitsOf(s);
				last = programStep(s, unit, slots, kStride, p, last);
				if (pc == end) {
					programSteps += cost;
					uint32_t k         = order >> 8 & 0xFFu;
					const bool lesser  = last < f.x;
					f.y                = within ? fminf(f.y, fabsf(last)) : lesser ? f.x : fminf(f.y, last);
					f.x                = lesser ? last : f.x;
					const GpuLeaf leaf = w.leaves[cell.leaf];
					if (lesser) order = (order & 0x0000FFFFu) | k << 16;
					if (++k < (order & 0xFFu)) {
						const GpuProgram g = w.programs[leaf.first + k];
						pc    = g.march;
						end   = g.march + g.marchCount;
						order = (order & 0x00FF00FFu) | k << 8;
						cost  = g.marchSteps;
					} else {
						// stop on the surface or go on by the value
						const float go = within ? f.y : f.x;
						++step;
						if (go < tolerance(p)) {
							mode = Landed;
						} else {
							const float on = fminf(t + go, fmaxf(cell.exit, t) + nudge(t));
							uint32_t each  = 0;
							if (on == t) {
								for (uint32_t k = 0; k < leaf.count; ++k) each += w.programs[leaf.first + k].marchSteps;
							}
							goOn(on, each);
							pc    = leaf.march;
							end   = leaf.march + leaf.marchCount;
							order = leaf.count;
							cost  = leaf.marchSteps;
							f.x = f.y = 3.0e38f;
							if (mode == Stepping) mode = Evaluating;
						}
					}
				}
				keep();
				pool.wall[r].w  = __uint_as_float((kind & 0xFFu) | cost << 8);
				pool.field[r]   = make_float4(f.x, f.y, last, __uint_as_float(pc));
				pool.program[r] = make_uint2(end, order);
			}
		} else if (locating >= stepping) {
			if (lane < take(Locating)) {
				load();
				mode             = Locating;
				const float4 i   = pool.inverse[r];
				const float inv[3] = { i.x, i.y, i.z };
				// the cell of the point; an empty one is left at once
				const float p[3] = { o[0] + d[0] * t, o[1] + d[1] * t, o[2] + d[2] * t };
				int place[3];
				placeOf(w, p, place);
				const uint32_t entry = entryAt(w, place);
				bool empty           = entry & kEntryEmpty;
				if (entry & kEntryLeaf) {
					const uint32_t wide = w.fineLevel - (entry >> kEntryLevelShift & 15u), row = (1u << w.fineLevel) + 1u;
					float at[3];
					for (int a = 0; a < 3; ++a) at[a] = __ldg(w.walls + a * row + ((uint32_t(place[a]) >> wide) + (__float_as_int(d[a]) < 0 ? 0u : 1u) << wide));
					walledBy(cell, at, o, d, inv);
					cell.leaf = entry & kEntryIndex;
				} else {
					cell  = deepCell(w, make_float3(p[0], p[1], p[2]), int32_t(entry), make_int3(place[0], place[1], place[2]), make_float3(o[0], o[1], o[2]), make_float3(d[0], d[1], d[2]), make_float3(inv[0], inv[1], inv[2]));
					empty = w.leaves[cell.leaf].shape == ShapeEmpty;
				}
				if (empty) {
					t = fmaxf(cell.exit, t) + nudge(t);
					++step;
					over();
				} else {
					const GpuLeaf leaf = w.leaves[cell.leaf];
					mode               = Stepping;
					if (leaf.shape == ShapePrograms) {
						mode            = Evaluating;
						pool.field[r]   = make_float4(3.0e38f, 3.0e38f, 0.0f, __uint_as_float(leaf.march));
						pool.program[r] = make_uint2(leaf.march + leaf.marchCount, leaf.count);
					} else {
						pool.field[r] = make_float4(leaf.params[0], leaf.params[1], leaf.params[2], leaf.params[3]);
					}
					pool.wall[r] = make_float4(cell.wall[0], cell.wall[1], cell.wall[2], __uint_as_float(leaf.shape | uint32_t(leaf.marchSteps) << 8));
				}
				keep();
			}
		} else if (lane < take(Stepping)) {
			load();
			mode = Stepping;
			const float4 kept = pool.field[r];
			const MarchParams field { { kept.x, kept.y, kept.z, kept.w } };
			const uint32_t shape = kind & 0xFFu, cost = kind >> 8;
			// a ray that skims the ground takes tens of thousands of these steps,
			// alone in its warp, each waiting on the one before
			uint32_t turns      = busy <= kFew ? kAlone : kMovesPerTurn;
			const uint32_t axis = shape >> kShapeAxisShift & 3u, side = shape >> kShapeSideShift;
			const float oa = axis == 0 ? o[0] : axis == 1 ? o[1] : o[2], da = axis == 0 ? d[0] : axis == 1 ? d[1] : d[2];
#pragma unroll 1
			do {
				const float p[3] = { o[0] + d[0] * t, o[1] + d[1] * t, o[2] + d[2] * t };
				const bool ball  = shape == ShapeSphere;
				const float value = ball ? sphereValue(p[0], p[1], p[2], field) : axisValue(oa + da * t, side, field);
				const float go = within ? fabsf(value) : value, tol = tolerance(p);
				if (!ball && t + 24.0f * go < cell.exit && (da > -0.05f || go > 64.0f * tol)) {
					// the steps of a ray that stays in its cell: t + go each, as long as
					// none lands (their least above the tolerance, which is greatest at an
					// end) and the last is short of the cell's walls, the march's end and
					// its limit, and moves; all of it as step by step, or not at all
					float at = t, before = t, least = 3.0e38f;
#pragma unroll
					for (uint32_t k = 0; k < kRun; ++k) {
						const float v = axisValue(oa + da * at, side, field);
						least         = fminf(least, within ? fabsf(v) : v);
						before        = at;
						at            = at + fabsf(v);
					}
					const float q[3] = { o[0] + d[0] * at, o[1] + d[1] * at, o[2] + d[2] * at };
					if (least >= fmaxf(tol, tolerance(q)) && at <= cell.exit && at <= up && at != before && step + kRun < stepLimit && inside(cell.wall, q, d)) {
						t = at;
						step += kRun;
						programSteps += kRun * cost;
						continue;
					}
				}
				programSteps += cost;
				++step;
				if (go < tol) { // it lands: the one program's value, its own second
					pool.field[r]     = make_float4(value, within ? go : 3.0e38f, 0.0f, 0.0f);
					pool.program[r].y = 0u;
					mode              = Landed;
					break;
				}
				goOn(fminf(t + go, fmaxf(cell.exit, t) + nudge(t)), cost);
			} while (mode == Stepping && --turns != 0u);
			keep();
		}
		__syncwarp();
	}
	if (args.counters) {
		// one add per warp (whose counts together are past 16 bits)
		uint32_t capped = cappedCarried & 0xFFFFu, carried = cappedCarried >> 16;
		for (int o = 16; o > 0; o >>= 1) {
			marchSteps += __shfl_down_sync(0xFFFFFFFFu, marchSteps, o);
			programSteps += __shfl_down_sync(0xFFFFFFFFu, programSteps, o);
			traced += __shfl_down_sync(0xFFFFFFFFu, traced, o);
			capped += __shfl_down_sync(0xFFFFFFFFu, capped, o);
			carried += __shfl_down_sync(0xFFFFFFFFu, carried, o);
			longest = max(longest, __shfl_down_sync(0xFFFFFFFFu, longest, o));
		}
		if ((threadIdx.x & 31) == 0) {
			atomicAdd(&args.counters[0], (unsigned long long) marchSteps);
			atomicAdd(&args.counters[1], (unsigned long long) programSteps);
			atomicMax(&args.counters[2], (unsigned long long) longest);
			atomicAdd(&args.counters[3], (unsigned long long) capped);
			atomicAdd(&args.counters[4], (unsigned long long) traced);
			if (carried) atomicAdd(&args.counters[5], (unsigned long long) carried);
		}
	}
}

// A hit's normal and leaves: one walk over the winning program in duals, which
// keeps every step's value for the walk back to the leaf.  What bounds it is
// that a warp's hits are on different programs: the common operations are one
// stretch of code for all (config 2's full frame 400 against 381 ms, the city 78
// against 72.6, with a walk for the duals, one for the values and a switch).
__global__ void __launch_bounds__(kTraceBlock) hitKernel(HitArgs args) {
	const DeviceWorld& w = args.world;
	const uint32_t n     = args.count ? *args.count : args.n;
	if (args.fetch != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *args.fetch = 0;
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		const HitState h  = args.states[i];
		const kdn_ray ray = args.rays[i];
		kdn_hit out;
		out.kind = 0;
		out.pad0_[0] = out.pad0_[1] = out.pad0_[2] = 0;
		out.distance = 0.0f;
		for (int a = 0; a < 3; ++a) {
			out.point[a]  = 0.0f;
			out.normal[a] = 0.0f;
		}
		out.leaf      = kNoLeaf;
		out.other     = kNoLeaf;
		out.share     = 0.0f;
		out.loosened  = 0.0f;
		out.leaf_kind = 0;
		out.pad1_[0] = out.pad1_[1] = out.pad1_[2] = 0;
		out.cell      = kNoLeaf;
		if (h.kind == kCarried) {
			// the march goes on in a later launch: where it stands and its steps
			out.kind     = kHitCarried;
			out.distance = h.distance;
			out.cell     = h.steps;
		} else if (h.kind != 0) {
			const float d[3]  = { ray.direction[0], ray.direction[1], ray.direction[2] };
			const float t     = h.distance;
			const float p[3]  = { ray.origin[0] + d[0] * t, ray.origin[1] + d[1] * t, ray.origin[2] + d[2] * t };
			// For a crossing into another material the field is read past the point.
			const float inset = h.kind == 2 ? 2.0f * tolerance(p) : 0.0f;
			const float q[3]  = { p[0] + d[0] * inset, p[1] + d[1] * inset, p[2] + d[2] * inset };
			const GpuProgram g = w.programs[h.first + h.index];
			// every slot is written before a step reads it (the slots follow the SSA order)
			DualF dslots[kMaxSlots];
			float values[kMaxSsa];
			DualF v;
			const bool held = evalDual(w.steps + g.code, g.count, g.slot, dslots, values, q, v);
			uint32_t leaf, other;
			float share;
			sourceOf(held, w.steps + g.code, w.ssa + g.code, g.count, g.result, values, q, leaf, other, share);
			// sphereNormal (sphere_trace.cpp:140)
			float n[3];
			const float len = sqrtf(v.g0 * v.g0 + v.g1 * v.g1 + v.g2 * v.g2);
			if (!(len > 0.0f)) {
				for (int a = 0; a < 3; ++a) n[a] = -d[a];
			} else {
				n[0] = v.g0 / len;
				n[1] = v.g1 / len;
				n[2] = v.g2 / len;
				const float along = n[0] * d[0] + n[1] * d[1] + n[2] * d[2];
				if (ray.inside) {
					if (along < 0.0f) {
						for (int a = 0; a < 3; ++a) n[a] = -n[a];
					}
				} else if (along > 0.0f) {
					float gz[3];
					for (int a = 0; a < 3; ++a) gz[a] = n[a] - d[a] * (along + 0.02f);
					const float gl = sqrtf(gz[0] * gz[0] + gz[1] * gz[1] + gz[2] * gz[2]);
					for (int a = 0; a < 3; ++a) n[a] = gz[a] / gl;
				}
			}
			out.kind     = 1;
			out.distance = t;
			for (int a = 0; a < 3; ++a) {
				out.point[a]  = p[a];
				out.normal[a] = n[a];
			}
			out.leaf     = leaf;
			out.other    = other;
			out.share    = share;
			out.loosened = tolerance(p);
			out.cell     = g.object;
		}
		args.hits[i] = out;
	}
}

} // namespace

cudaError_t launchTrace(const TraceArgs& args, cudaStream_t stream, int smCount) {
	if (args.n == 0) return cudaSuccess;
	// the warps' pools and a ray's register slots, as many as the world's
	// largest march program uses: the rest of the SM's shared memory stays
	// L1 for the programs' code
	const size_t shared = sizeof(Pool) * kWarps + size_t(std::max<uint32_t>(kMarchFirstSlot, std::min(args.world.marchSlots, kMaxSlots))) * kStride * sizeof(float);
	// persistent blocks: as many as fit on the SMs at once, fewer for a small launch
	static thread_local size_t sizedFor = 0;
	static thread_local int resident    = 0;
	if (sizedFor != shared) {
		int perSm = 0;
		if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, traceKernel, kTraceBlock, shared) != cudaSuccess || perSm < 1) perSm = 1;
		resident = perSm;
		sizedFor = shared;
	}
	// a warp a ray where they are few: see the kernel's share
	const uint64_t wanted = (uint64_t(args.n) + kTraceBlock / 32 - 1) / (kTraceBlock / 32);
	const uint32_t blocks = uint32_t(std::max<uint64_t>(1, std::min<uint64_t>(wanted, uint64_t(smCount) * uint64_t(resident))));
	traceKernel<<<blocks, kTraceBlock, shared, stream>>>(args);
	return cudaGetLastError();
}

cudaError_t launchHits(const HitArgs& args, cudaStream_t stream, int smCount) {
	if (args.n == 0) return cudaSuccess;
	const uint32_t blocks = uint32_t(std::min<uint64_t>((uint64_t(args.n) + kTraceBlock - 1) / kTraceBlock, uint64_t(smCount) * 16));
	hitKernel<<<blocks, kTraceBlock, 0, stream>>>(args);
	return cudaGetLastError();
}

cudaError_t setTraceAttributes() {
	return cudaFuncSetAttribute(traceKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(Pool) * kWarps + kMaxSlots * kStride * sizeof(float)));
}

} // namespace kdn
