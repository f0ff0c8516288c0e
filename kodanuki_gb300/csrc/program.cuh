// Device evaluation of a leaf's kept programs (sdf/program.cpp:57 runStep),
// in single precision.
//
//  - evalSlots: the march's form.  Values live in register slots held in
//    shared memory, one column per thread: slot s of thread t is at
//    slots[s * blockDim.x + t], so a warp's accesses to one slot hit 32
//    consecutive banks.
//  - evalDual:  the value and gradient (forward mode, sdf/numbers.cpp:440
//    Dual) over the same slots, 4 floats a slot.
//  - evalSsa:   every step's value kept by step number, for the walk back from
//    the result that names the source leaf (sdf/program.cpp:478).
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

// world.h FormAxis: a coordinate's distance to a slab.
KDN_HD float axisValue(float p, uint32_t side, const MarchParams& q) {
	float u = addAlone(p, -q.v[0]);
	u       = side == SideAbs ? fabsf(u) : u;
	u       = side == SideNegative ? 0.0f - u : u;
	return addAlone(addAlone(addAlone(u, -q.v[1]), q.v[2]), -q.v[3]);
}

// world.h FormSphere.
KDN_HD float sphereValue(float px, float py, float pz, const MarchParams& q) {
	const float x = addAlone(px, -q.v[0]), y = addAlone(py, -q.v[1]), z = addAlone(pz, -q.v[2]);
	return addAlone(marchSqrt(fmaf(z, z, fmaf(x, x, mulAlone(y, y)))), -q.v[3]);
}

// world.h FormNorm over the values of its slots.
KDN_HD float normValue(float a, float b, float c, float m, uint32_t flags, float e) {
	const float p = flags & NormPositive0 ? fmaxf(a, 0.0f) : a;
	const float q = flags & NormPositive1 ? fmaxf(b, 0.0f) : b;
	const float r = flags & NormPositive2 ? fmaxf(c, 0.0f) : c;
	float sum     = mulAlone(p, p);
	sum           = flags & NormFused1 ? fmaf(q, q, sum) : addAlone(mulAlone(q, q), sum);
	const float s = flags & NormFused2 ? fmaf(r, r, sum) : addAlone(mulAlone(r, r), sum);
	float f       = marchSqrt(flags & NormThree ? s : sum);
	if (flags & NormInside) {
		if (flags & NormInsideMax) {
			m = flags & NormThree ? (b < c ? c : b) : b;
			m = a < m ? m : a;
		}
		f = addAlone(f, 0.0f < m ? 0.0f : m);
	}
	return addAlone(f, -e);
}

// One step of the march form (world.h MarchStep) and, of a fused step, its
// parameters: r = post(form, w), with the post operations worked out
// together and the step's picked, so the lanes of a warp on different posts
// do not split; a rare step runs the reference operation.  Writes the result
// to its slot.
KDN_HD void marchStep(const MarchStep& s, const MarchParams& q, float* slots, uint32_t stride) {
	float r;
	if (s.op >= kMarchRare) {
		slots[SlotImm * stride] = s.value;
		const float a = slots[s.a * stride], b = slots[s.b * stride], c = slots[s.c * stride];
		const float p[3] = { slots[SlotX * stride], slots[SlotY * stride], slots[SlotZ * stride] };
		r                = stepValue(uint8_t(s.op - kMarchRare), a, b, c, s.value, p);
	} else {
		const uint32_t form = s.op & kMarchFormMask, post = s.op & kMarchPostMask;
		float f;
		if (form == FormAxis) {
			f = axisValue(slots[s.a * stride], s.flags, q);
		} else if (form == FormSphere) {
			f = sphereValue(slots[SlotX * stride], slots[SlotY * stride], slots[SlotZ * stride], q);
		} else if (form == FormNorm) {
			f = normValue(slots[s.a * stride], slots[s.b * stride], slots[s.c * stride], slots[s.m * stride], s.flags, q.v[0]);
		} else {
			slots[SlotImm * stride] = s.value;
			f                       = fmaf(slots[s.a * stride], slots[s.b * stride], slots[s.c * stride]);
		}
		r = f;
		if (post != PostNone) {
			slots[SlotImm * stride] = s.value;
			const float w = slots[s.w * stride];
			const float p = fmaxf(f, 0.0f);
			// the smooth minimum of radius r = value: min - max(r - |f - w|, 0)^2 * 0.25 / r
			const float m = fmaxf(s.value - fabsf(f - w), 0.0f);
			r             = post == PostSqrt ? marchSqrt(f) : r;
			r             = post == PostAbs ? fabsf(f) : r;
			r             = post == PostPosSq ? p * p : r;
			r             = post == PostMin ? (w < f ? w : f) : r;
			r             = post == PostMax ? (f < w ? w : f) : r;
			r             = post == PostSminK ? fminf(f, w) - m * m * s.quarter : r;
		}
	}
	slots[s.dst * stride] = r;
}

// The parameters of a fused step, in the unit after it.
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

// Whether a step is a fused one.
KDN_HD bool fusedStep(const MarchStep& s) { return s.op < kMarchRare && (s.op & kMarchFormMask) != FormFma; }

// One program at one point; slots is this thread's column base (stride
// blockDim.x), with the constants set.  Returns the program's value.
KDN_HD float evalSlots(const MarchStep* __restrict__ code, uint32_t count, uint32_t resultSlot, float* slots, uint32_t stride, const float p[3]) {
	setPoint(slots, stride, p);
	for (uint32_t i = 0; i < count; ++i) {
		const MarchStep s = code[i];
		MarchParams q {};
		if (fusedStep(s)) q = paramsAt(code + ++i);
		marchStep(s, q, slots, stride);
	}
	return slots[resultSlot * stride];
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

__device__ __forceinline__ DualF evalDual(const GpuStep* __restrict__ code, uint32_t count, uint32_t resultSlot, DualF* slots, const float p[3]) {
	for (uint32_t i = 0; i < count; ++i) {
		const GpuStep s = code[i];
		slots[s.dst]    = dualStep(s.op, slots[s.a], slots[s.b], slots[s.c], s.value, p);
	}
	return slots[resultSlot];
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

// Every step's value by step number, then the walk back through the joins
// (sdf/program.cpp:478 laneSourceOf): the leaf that decides the value, the
// leaf across the first smooth band and its share.
__device__ __forceinline__ void sourceOf(const GpuStep* __restrict__ code, const SsaOps* __restrict__ ssa, uint32_t count, uint32_t result, float* v, const float p[3], uint32_t& leaf, uint32_t& other, float& share) {
	for (uint32_t i = 0; i < count; ++i) {
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
