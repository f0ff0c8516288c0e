// Device evaluation of a leaf's kept programs (sdf/program.cpp:57 runStep),
// in single precision.
//
//  - evalSlots: the march's form.  Values live in register slots held in
//    shared memory, a column each for the rays of a block: slot s of ray r is at
//    slots[s * stride + r], so a warp's accesses to one slot hit the banks of
//    its rays' places.
//  - evalDual:  the value and gradient (forward mode, sdf/numbers.cpp:440
//    Dual) over the same slots, 4 floats a slot, and every step's value kept
//    by step number.
//  - sourceOf:  the walk back from the result that names the source leaf
//    (sdf/program.cpp:478).
#pragma once

#include "world.h"

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>

// The march form's interpreter compiles for the host too, where
// kdn_world_march runs it to check the march form against the programs.
#define KDN_HD __host__ __device__ __forceinline__

namespace kdn {

KDN_HD float floatOfBits(uint32_t bits) {
#ifdef __CUDA_ARCH__
	return __uint_as_float(bits);
#else
	float f;
	std::memcpy(&f, &bits, sizeof f);
	return f;
#endif
}

KDN_HD float smoothMinF(float a, float b, float r) {
	const float blend = fmaxf(r - fabsf(a - b), 0.0f) / r;
	return fminf(a, b) - blend * blend * r * 0.25f;
}

KDN_HD float truthF(bool b) { return b ? 1.0f : 0.0f; }

// The march's square root: the hardware's approximate one on the device
// (PTX sqrt.approx.f32, relative error within 2^-22), correctly rounded on
// the host.
KDN_HD float marchSqrt(float x) {
#ifdef __CUDA_ARCH__
	float r;
	asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
	return r;
#else
	return sqrtf(x);
#endif
}

KDN_HD float stepValue(uint8_t op, float a, float b, float c, float value, const float p[3]) {
	switch (op) {
		case OpConstant: return value;
		case OpArgument: return 0.0f;
		case OpPointX: return p[0];
		case OpPointY: return p[1];
		case OpPointZ: return p[2];
		case OpNormalX: case OpNormalY: case OpNormalZ: return 0.0f;
		case OpAdd: return a + b;
		case OpSubtract: return a - b;
		case OpMultiply: return a * b;
		case OpDivide: return a / b;
		case OpNegate: return -a;
		case OpSqrt: return sqrtf(a);
		case OpAbs: return fabsf(a);
		case OpFloor: return floorf(a);
		case OpSin: return sinf(a);
		case OpCos: return cosf(a);
		case OpSign: return a > 0.0f ? 1.0f : (a < 0.0f ? -1.0f : 0.0f);
		case OpAtan2: return atan2f(a, b);
		case OpPow: return powf(a, b);
		case OpMin: return b < a ? b : a;
		case OpMax: return a < b ? b : a;
		case OpSmin: return smoothMinF(a, b, c);
		case OpPosSq: {
			const float q = fmaxf(a, 0.0f);
			return q * q;
		}
		case OpLess: return truthF(a < b);
		case OpLessEq: return truthF(a <= b);
		case OpEqual: return truthF(a == b);
		case OpNotEqual: return truthF(a != b);
		case OpAnd: return truthF(a != 0.0f && b != 0.0f);
		case OpOr: return truthF(a != 0.0f || b != 0.0f);
		case OpNot: return truthF(a == 0.0f);
		case OpSelect: return a != 0.0f ? b : c;
		default: return 0.0f;
	}
}

// The reserved slots of a thread's column: 0, 1 and -1 once, the point at
// each new point.
KDN_HD void setConstants(float* slots, uint32_t stride) {
	slots[SlotZero * stride]     = 0.0f;
	slots[SlotOne * stride]      = 1.0f;
	slots[SlotMinusOne * stride] = -1.0f;
}

KDN_HD void setPoint(float* slots, uint32_t stride, const float p[3]) {
	slots[SlotX * stride] = p[0];
	slots[SlotY * stride] = p[1];
	slots[SlotZ * stride] = p[2];
}

// Sums and products that are rounded one by one: the device compiler would
// otherwise make a fused multiply-add of a product and the sum that reads it.
KDN_HD float mulAlone(float a, float b) {
#ifdef __CUDA_ARCH__
	return __fmul_rn(a, b);
#else
	return a * b;
#endif
}
KDN_HD float addAlone(float a, float b) {
#ifdef __CUDA_ARCH__
	return __fadd_rn(a, b);
#else
	return a + b;
#endif
}

// A coordinate's distance to a slab: side of p - c, then - h, + r (and - e).
KDN_HD float slabValue(float p, uint32_t side, float c, float h, float r) {
	float u = addAlone(p, -c);
	u       = side == SideAbs ? fabsf(u) : u;
	u       = side == SideNegative ? 0.0f - u : u;
	return addAlone(addAlone(u, -h), r);
}
KDN_HD float axisValue(float p, uint32_t side, const MarchParams& q) { return addAlone(slabValue(p, side, q.v[0], q.v[1], q.v[2]), -q.v[3]); }

// A point's distance to a sphere: centre and radius.
KDN_HD float sphereValue(float px, float py, float pz, const MarchParams& q) {
	const float x = addAlone(px, -q.v[0]), y = addAlone(py, -q.v[1]), z = addAlone(pz, -q.v[2]);
	return addAlone(marchSqrt(fmaf(z, z, fmaf(x, x, mulAlone(y, y)))), -q.v[3]);
}

// The sum of squares of a root's terms (world.h SumFlag); a term left out
// adds an exact zero.
KDN_HD float squaresOf(float a, float b, float c, uint32_t flags) {
	const float p = flags & SumHas0 ? (flags & SumPositive0 ? fmaxf(a, 0.0f) : a) : 0.0f;
	const float q = flags & SumHas1 ? (flags & SumPositive1 ? fmaxf(b, 0.0f) : b) : 0.0f;
	const float r = flags & SumHas2 ? (flags & SumPositive2 ? fmaxf(c, 0.0f) : c) : 0.0f;
	float sum     = mulAlone(p, p);
	sum           = flags & SumFused1 ? fmaf(q, q, sum) : addAlone(mulAlone(q, q), sum);
	return flags & SumFused2 ? fmaf(r, r, sum) : addAlone(mulAlone(r, r), sum);
}

KDN_HD float greaterOf(float f, float w) { return f < w ? w : f; } // PostMax
KDN_HD float belowZero(float m) { return 0.0f < m ? 0.0f : m; }    // PostMin with 0

// world.h FormPrimitive at a point.
KDN_HD float primitiveValue(const MarchStep& s, const MarchParams& c, const MarchParams& h, float px, float py, float pz) {
	const uint32_t terms[3] = { s.a, s.b, s.c };
	float u[3];
	for (int k = 0; k < 3; ++k) {
		const uint32_t axis = terms[k] & 3u;
		u[k]                = slabValue(axis == 0 ? px : axis == 1 ? py : pz, terms[k] >> kTermSideShift, c.v[k], h.v[k], h.v[3]);
	}
	float f = marchSqrt(squaresOf(u[0], u[1], u[2], s.flags));
	if (s.m & PrimSingle) f = greaterOf(s.flags & SumHas0 ? u[0] : s.flags & SumHas1 ? u[1] : u[2], 0.0f);
	if (s.m & PrimPlain) f = u[0];
	const float inside = belowZero(greaterOf(u[0], s.m & PrimThird ? greaterOf(u[1], u[2]) : u[1]));
	f                  = s.m & PrimInside ? addAlone(f, inside) : f;
	return addAlone(f, -c.v[3]);
}

// The post operation of a step's value f, worked out together and the step's
// picked, so the lanes of a warp on different posts do not split.
KDN_HD float posted(uint32_t post, float f, float w, float value, float quarter) {
	const float p = fmaxf(f, 0.0f);
	// the smooth minimum of radius r = value: min - max(r - |f - w|, 0)^2 * 0.25 / r
	const float m = fmaxf(value - fabsf(f - w), 0.0f);
	float r       = f;
	r             = post == PostSqrt ? marchSqrt(f) : r;
	r             = post == PostAbs ? fabsf(f) : r;
	r             = post == PostPosSq ? p * p : r;
	r             = post == PostMin ? (w < f ? w : f) : r;
	r             = post == PostMax ? (f < w ? w : f) : r;
	r             = post == PostSminK ? fminf(f, w) - m * m * quarter : r;
	return r;
}

// A rare step's reference operation; out of line on the device, where its
// sines and powers would otherwise be laid into every march loop.
#ifdef __CUDA_ARCH__
__device__ __noinline__
#else
inline
#endif
float rareValue(uint8_t op, float a, float b, float c, float value, float3 at) {
	const float p[3] = { at.x, at.y, at.z };
	return stepValue(op, a, b, c, value, p);
}

// The parameters of a fused step, a unit.
KDN_HD MarchParams paramsAt(const MarchStep* unit) {
#ifdef __CUDA_ARCH__
	const float4 v = *reinterpret_cast<const float4*>(unit);
	return { { v.x, v.y, v.z, v.w } };
#else
	MarchParams q;
	std::memcpy(&q, unit, sizeof q);
	return q;
#endif
}

// One step of the march form (world.h MarchStep) at a point but a primitive,
// over a ray's slots: r = post(form, w); a rare step runs the reference
// operation.  Writes the result to its slot and returns it.
KDN_HD float marchStep(const MarchStep& s, const MarchStep* unit, float* slots, uint32_t stride) {
	slots[SlotImm * stride] = s.value;
	float r;
	if (s.op >= kMarchRare) {
		const float a = slots[s.a * stride], b = slots[s.b * stride], c = slots[s.c * stride];
		r = rareValue(uint8_t(s.op - kMarchRare), a, b, c, s.value, make_float3(slots[SlotX * stride], slots[SlotY * stride], slots[SlotZ * stride]));
	} else {
		const uint32_t form = s.op & kMarchFormMask, post = s.op & kMarchPostMask;
		if (form == FormNorm) {
			r = marchSqrt(squaresOf(slots[s.a * stride], slots[s.b * stride], slots[s.c * stride], s.flags));
			if (s.m != kNoInside) r = addAlone(r, belowZero(slots[s.m * stride]));
			r = addAlone(r, -paramsAt(unit).v[0]);
		} else if (form == FormRepeat) {
			const float x = slots[s.a * stride];
			r             = addAlone(x, -mulAlone(s.value, floorf(addAlone(x / s.value, s.quarter))));
		} else {
			r = fmaf(slots[s.a * stride], slots[s.b * stride], slots[s.c * stride]);
		}
		if (post != PostNone) r = posted(post, r, slots[s.w * stride], s.value, s.quarter);
	}
	slots[s.dst * stride] = r;
	return r;
}

// The units of a step.
KDN_HD uint32_t unitsOf(const MarchStep& s) {
	const uint32_t form = s.op & kMarchFormMask;
	return s.op >= kMarchRare || form == FormFma || form == FormRepeat ? 1u : form == FormPrimitive && s.m & PrimSized ? 3u : 2u;
}
KDN_HD bool primitiveStep(const MarchStep& s) { return s.op < kMarchRare && (s.op & kMarchFormMask) == FormPrimitive; }

// A primitive step at a point; last is the step before's result.  A post
// operation's w is that, the immediate or a slot of the program's, never the
// point's (the lowering makes a coordinate a plane of its own).
KDN_HD float primitiveStepValue(const MarchStep& s, const MarchStep* unit, float* slots, uint32_t stride, float px, float py, float pz, float last) {
	const MarchParams c = paramsAt(unit);
	MarchParams h { { 0.0f, 0.0f, 0.0f, -0.0f } };
	if (s.m & PrimSized) h = paramsAt(unit + 1);
	float r             = primitiveValue(s, c, h, px, py, pz);
	const uint32_t post = s.op & kMarchPostMask;
	if (post != PostNone) {
		float w = last;
		if (!(s.m & PrimPrevious)) w = s.w == SlotImm ? s.value : slots[s.w * stride];
		r = posted(post, r, w, s.value, s.quarter);
	}
	if (s.m & PrimStored) slots[s.dst * stride] = r;
	return r;
}

// A step as a turn of the march takes it: between turns a ray's column holds
// the constants and what steps stored, but not the point.
KDN_HD float programStep(const MarchStep& s, const MarchStep* unit, float* slots, uint32_t stride, const float p[3], float last) {
	if (primitiveStep(s)) return primitiveStepValue(s, unit, slots, stride, p[0], p[1], p[2], last);
	setPoint(slots, stride, p);
	return marchStep(s, unit, slots, stride);
}

// One program at one point; slots is its ray's column (stride the
// block's rays), with the constants set.  Returns the program's value, which
// its last step makes.
KDN_HD float evalSlots(const MarchStep* __restrict__ code, uint32_t count, float* slots, uint32_t stride, const float p[3]) {
	setPoint(slots, stride, p);
	float last = 0.0f;
#pragma unroll 1
	for (uint32_t i = 0; i < count;) {
		const MarchStep s = code[i];
		if (primitiveStep(s)) last = primitiveStepValue(s, code + i + 1, slots, stride, p[0], p[1], p[2], last);
		else last = marchStep(s, code + i + 1, slots, stride);
		i += unitsOf(s);
	}
	return last;
}

struct DualF {
	float v, g0, g1, g2;
};

__device__ __forceinline__ DualF dualConst(float v) { return { v, 0.0f, 0.0f, 0.0f }; }
__device__ __forceinline__ DualF chain1(DualF a, float f, float d) { return { f, d * a.g0, d * a.g1, d * a.g2 }; }
__device__ __forceinline__ DualF chain2(DualF a, DualF b, float f, float fa, float fb) {
	return { f, fa * a.g0 + fb * b.g0, fa * a.g1 + fb * b.g1, fa * a.g2 + fb * b.g2 };
}

// sdf/numbers.cpp:440-590 the Dual operations.
__device__ __forceinline__ DualF dualStep(uint8_t op, DualF a, DualF b, DualF c, float value, const float p[3]) {
	switch (op) {
		case OpConstant: return dualConst(value);
		case OpPointX: return { p[0], 1.0f, 0.0f, 0.0f };
		case OpPointY: return { p[1], 0.0f, 1.0f, 0.0f };
		case OpPointZ: return { p[2], 0.0f, 0.0f, 1.0f };
		case OpAdd: return chain2(a, b, a.v + b.v, 1.0f, 1.0f);
		case OpSubtract: return chain2(a, b, a.v - b.v, 1.0f, -1.0f);
		case OpMultiply: return chain2(a, b, a.v * b.v, b.v, a.v);
		case OpDivide: return chain2(a, b, a.v / b.v, 1.0f / b.v, -a.v / (b.v * b.v));
		case OpNegate: return chain1(a, -a.v, -1.0f);
		case OpSqrt: {
			const float f = sqrtf(a.v);
			return chain1(a, f, f > 0.0f ? 0.5f / f : 0.0f);
		}
		case OpAbs: return a.v < 0.0f ? chain1(a, -a.v, -1.0f) : a;
		case OpFloor: return dualConst(floorf(a.v));
		case OpSin: return chain1(a, sinf(a.v), cosf(a.v));
		case OpCos: return chain1(a, cosf(a.v), -sinf(a.v));
		case OpSign: return dualConst(a.v > 0.0f ? 1.0f : (a.v < 0.0f ? -1.0f : 0.0f));
		case OpAtan2: {
			const float r = b.v * b.v + a.v * a.v;
			return chain2(a, b, atan2f(a.v, b.v), b.v / r, -a.v / r);
		}
		case OpPow: {
			const float f = powf(a.v, b.v);
			return chain2(a, b, f, b.v * powf(a.v, b.v - 1.0f), f * (a.v > 0.0f ? logf(a.v) : 0.0f));
		}
		case OpMin: return a.v <= b.v ? a : b;
		case OpMax: return a.v >= b.v ? a : b;
		case OpSmin: {
			const float fa = fminf(fmaxf((c.v - (a.v - b.v)) / (2.0f * c.v), 0.0f), 1.0f);
			return chain2(a, b, smoothMinF(a.v, b.v, c.v), fa, 1.0f - fa);
		}
		case OpPosSq: return chain1(a, fmaxf(a.v, 0.0f) * fmaxf(a.v, 0.0f), 2.0f * fmaxf(a.v, 0.0f));
		case OpSelect: return a.v != 0.0f ? b : c;
		default: return dualConst(stepValue(op, a.v, b.v, c.v, value, p));
	}
}

// A step of the operations that distances are made of, worked out together and
// the step's picked, so the lanes of a warp at different steps do not split;
// dualStep's to the bit but for a product's gradient, whose two terms may be
// fused the other way.  A gradient is fa * x.g, and + fb * b.g for a sum or a
// product, x being an operand or a coordinate's own.
__device__ __forceinline__ DualF commonDual(uint8_t op, DualF a, DualF b, float value, const float p[3]) {
	const bool lesser = a.v <= b.v, greater = a.v >= b.v, negative = a.v < 0.0f;
	const bool second = op == OpMin ? !lesser : op == OpMax && !greater;
	const bool sum = op == OpAdd || op == OpSubtract, product = op == OpMultiply, point = op >= OpPointX && op <= OpPointZ;
	const bool turns = op == OpNegate || (op == OpAbs && negative);
	const float m    = fmaxf(a.v, 0.0f);
	DualF x;
	x.v  = second ? b.v : op == OpConstant ? value : op == OpPointX ? p[0] : op == OpPointY ? p[1] : op == OpPointZ ? p[2] : a.v;
	x.g0 = point ? (op == OpPointX ? 1.0f : 0.0f) : op == OpConstant ? 0.0f : second ? b.g0 : a.g0;
	x.g1 = point ? (op == OpPointY ? 1.0f : 0.0f) : op == OpConstant ? 0.0f : second ? b.g1 : a.g1;
	x.g2 = point ? (op == OpPointZ ? 1.0f : 0.0f) : op == OpConstant ? 0.0f : second ? b.g2 : a.g2;
	const float fa = product ? b.v : op == OpPosSq ? 2.0f * m : turns ? -1.0f : 1.0f;
	const float fb = product ? a.v : op == OpSubtract ? -1.0f : 1.0f;
	const bool two = sum || product;
	DualF r;
	r.v  = op == OpAdd ? a.v + b.v : op == OpSubtract ? a.v - b.v : product ? a.v * b.v : op == OpPosSq ? m * m : turns ? -a.v : x.v;
	r.g0 = two ? fa * x.g0 + fb * b.g0 : fa * x.g0;
	r.g1 = two ? fa * x.g1 + fb * b.g1 : fa * x.g1;
	r.g2 = two ? fa * x.g2 + fb * b.g2 : fa * x.g2;
	return r;
}

__device__ __forceinline__ bool isCommon(uint8_t op) {
	constexpr uint64_t those = 1ull << OpConstant | 1ull << OpPointX | 1ull << OpPointY | 1ull << OpPointZ | 1ull << OpAdd | 1ull << OpSubtract | 1ull << OpMultiply | 1ull << OpNegate | 1ull << OpAbs | 1ull << OpMin | 1ull << OpMax | 1ull << OpPosSq;
	return op < 64 && those >> op & 1u;
}

// The value and gradient, and every step's value by step number in v (for
// sourceOf), but where one is not a number: then false, and v is to be made.
__device__ __forceinline__ bool evalDual(const GpuStep* __restrict__ code, uint32_t count, uint32_t resultSlot, DualF* slots, float* v, const float p[3], DualF& result) {
	bool numbers = true;
	for (uint32_t i = 0; i < count; ++i) {
		const GpuStep s = code[i];
		const DualF a = slots[s.a], b = slots[s.b];
		DualF r;
		if (isCommon(s.op)) r = commonDual(s.op, a, b, s.value, p);
		else r = dualStep(s.op, a, b, slots[s.c], s.value, p);
		slots[s.dst] = r;
		v[i]         = r.v;
		numbers      = numbers && r.v == r.v;
	}
	result = slots[resultSlot];
	return numbers;
}

__device__ __forceinline__ bool isJoin(uint8_t op) { return op == OpMin || op == OpSmin || op == OpMax || op == OpNegate || op == OpSelect; }

__device__ __forceinline__ uint32_t chosenOperand(uint8_t op, const SsaOps& o, const float* v) {
	const float a = v[o.a], b = v[o.b];
	switch (op) {
		case OpMin: case OpSmin: return a <= b ? o.a : o.b;
		case OpMax: return a >= b ? o.a : o.b;
		case OpSelect: return a != 0.0f ? o.b : o.c;
		default: return o.a;
	}
}

// Every step's value by step number (unless v holds them), then the walk back
// through the joins (sdf/program.cpp:478 laneSourceOf): the leaf that decides
// the value, the leaf across the first smooth band and its share.
__device__ __forceinline__ void sourceOf(bool held, const GpuStep* __restrict__ code, const SsaOps* __restrict__ ssa, uint32_t count, uint32_t result, float* v, const float p[3], uint32_t& leaf, uint32_t& other, float& share) {
	for (uint32_t i = 0; i < (held ? 0u : count); ++i) {
		const GpuStep s = code[i];
		const SsaOps o  = ssa[i];
		v[i]            = stepValue(s.op, v[o.a], v[o.b], v[o.c], s.value, p);
	}
	other    = kNoLeaf;
	share    = 0.0f;
	uint32_t at = result;
	for (uint32_t guard = 0; guard < count && isJoin(code[at].op); ++guard) {
		const SsaOps o      = ssa[at];
		const uint8_t op    = code[at].op;
		const uint32_t next = chosenOperand(op, o, v);
		float s             = 0.0f;
		if (op == OpSmin) {
			const float radius = v[o.c];
			const float apart  = fabsf(v[o.a] - v[o.b]);
			s                  = radius > 0.0f && apart < radius ? 0.5f * (radius - apart) / radius : 0.0f;
		}
		if (s > 0.0f && other == kNoLeaf) {
			uint32_t side = next == o.a ? o.b : o.a;
			for (uint32_t g = 0; g < count && isJoin(code[side].op); ++g) side = chosenOperand(code[side].op, ssa[side], v);
			other = code[side].leaf;
			share = s;
		}
		at = next;
	}
	leaf = code[at].leaf;
}

} // namespace kdn
