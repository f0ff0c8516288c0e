// The SVGF-like denoiser on the device (plugins/reconstruction/atrous/
// atrous.cpp:513 denoisedFrame), six kernels over the frame:
//   K-prep     guides (camera-space point, normal, plane offset, 1/reach) and
//              the demodulated light with its history variance (:148);
//   K-var      a 7x7 spatial variance where the history is young (:376);
//   K-atrous   x4: a 3x3 prefilter of the variance, then the 5x5 B3 spline
//              at steps 1, 2, 4, 8 stopped by normal^128, plane distance and
//              luminance over the deviation (:411); the last times the albedo,
//              faded toward the history by its length (:461).
// Features come in as FP16 (distance, normal, albedo) beside FP32 light.  The
// filter is FP32, its taps in the reference's order, its products fused into
// the sums that read them.  What the reference works out in double (the
// guides, the history's variance, the last fade) is worked out in pairs of
// floats, 46 bits: this GPU's double rate is a 64th of its float rate, and
// these few operations a pixel took as long as the whole filter (prep 456 us
// and the fade 155 us at 1080p in double, 31 us and nothing now).
//
// The filter's passes are bound by FP32 issue (68% of its peak): 25 taps of
// some 45 instructions a pixel (112 before: no multiply-add fused, bounds and
// addresses worked out a tap, a fourth load), 94 to 103 us a 1080p pass where
// it was 171, the whole denoiser 0.5 ms where it was 1.3.  A block's taps all
// lie inside the frame but for the blocks at its edges, which run the checked
// form.
#include "denoise.h"

#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace kdn {

namespace {

constexpr int kBlockX = 32;
constexpr int kBlockY = 8;

// A number as an unevaluated sum of two floats, to about 46 bits (Dekker's
// sums and products, the products' errors by a fused multiply-add).
struct Pair {
	float h, l;
};
__device__ __forceinline__ Pair tidy(float a, float b) { // |a| >= |b|
	const float s = a + b;
	return { s, b - (s - a) };
}
__device__ __forceinline__ Pair sum(float a, float b) {
	const float s = a + b, t = s - a;
	return { s, (a - (s - t)) + (b - t) };
}
__device__ __forceinline__ Pair product(float a, float b) {
	const float p = a * b;
	return { p, fmaf(a, b, -p) };
}
__device__ __forceinline__ Pair add(Pair a, Pair b) {
	const Pair s = sum(a.h, b.h);
	return tidy(s.h, s.l + (a.l + b.l));
}
__device__ __forceinline__ Pair mul(Pair a, Pair b) {
	const Pair p = product(a.h, b.h);
	return tidy(p.h, p.l + fmaf(a.h, b.l, a.l * b.h));
}
__device__ __forceinline__ Pair mul(Pair a, float b) {
	const Pair p = product(a.h, b);
	return tidy(p.h, fmaf(a.l, b, p.l));
}
__device__ __forceinline__ Pair negative(Pair a) { return { -a.h, -a.l }; }
__device__ __forceinline__ Pair inverse(Pair a) {
	const float r = 1.0f / a.h;
	return tidy(r, r * (fmaf(-a.h, r, 1.0f) - a.l * r));
}
__device__ __forceinline__ Pair inverseRoot(Pair a) {
	const float r  = rsqrtf(a.h);
	const Pair one = mul(mul(a, r), r);
	return tidy(r, 0.5f * r * ((1.0f - one.h) - one.l));
}
// The nearest pair to a double, for constants and the lens.
__host__ __device__ constexpr Pair pairOf(double a) { return { float(a), float(a - double(float(a))) }; }
__device__ __forceinline__ float single(Pair a) { return a.h + a.l; }

// atrous.cpp:31 of -v, v >= 0: 2^(-v log2 e), the mantissa from a fitted
// quadratic.  The whole part by a sum with 1.5 * 2^23, whose low bits are
// then the number (floor and the conversion run at an eighth of the rate);
// at a whole power it may be one less, where the fit meets itself.
__device__ __forceinline__ float quickExp(float v) {
	const float t     = fminf(v, 30.0f) * -1.44269504f;
	const float moved = (t - 0.5f) + 12582912.0f;
	const float f     = t - (moved - 12582912.0f);
	const float power = fmaf(f, fmaf(f, 0.33977f, 0.66023f), 1.0f);
	const float value = __int_as_float(__float_as_int(power) + (__float_as_int(moved) << 23));
	return v < 30.0f ? value : 0.0f;
}

__device__ __forceinline__ float luma(float r, float g, float b) { return fmaf(0.0722f, b, fmaf(0.7152f, g, 0.2126f * r)); }
__device__ __forceinline__ Pair lumaPair(Pair r, Pair g, Pair b) { return add(add(mul(r, pairOf(0.2126)), mul(g, pairOf(0.7152))), mul(b, pairOf(0.0722))); }

// atrous.cpp divisorOf: what light is divided by, and times again
__device__ __forceinline__ float divisorOf(uint16_t albedo) {
	const float a = __half2float(__ushort_as_half(albedo));
	return a < 1e-3f ? 1.0f : a; // no FP16 number lies between 1e-3 and its float
}

// atrous.cpp:55 denoiseCamera: the heading through a pixel's centre, corner +
// across (x + 1/2) + down (y + 1/2), worked out in double on the host
struct Lens {
	Pair corner[3], across[3], down[3];
};

__global__ void __launch_bounds__(kBlockX * kBlockY) prepKernel(const __grid_constant__ DenoiseArgs a, const __grid_constant__ Lens lens) {
	const int x = blockIdx.x * blockDim.x + threadIdx.x;
	const int y = blockIdx.y * blockDim.y + threadIdx.y;
	if (x >= a.width || y >= a.height) return;
	const size_t p = size_t(y) * size_t(a.width) + size_t(x);
	const float distance = __half2float(__ushort_as_half(a.distance[p]));
	const bool sky       = a.leaf[p] == 0xFFFFFFFFu || !isfinite(distance) || !(distance > 0.0f);
	float4 g0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), g1 = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
	float near = 0.0f;
	if (!sky) {
		const float n[3] = { __half2float(__ushort_as_half(a.normal[3 * p])), __half2float(__ushort_as_half(a.normal[3 * p + 1])),
			                 __half2float(__ushort_as_half(a.normal[3 * p + 2])) };
		Pair h[3];
		for (int k = 0; k < 3; ++k) h[k] = add(add(lens.corner[k], mul(lens.across[k], float(x) + 0.5f)), mul(lens.down[k], float(y) + 0.5f));
		const Pair s = mul(inverseRoot(add(add(mul(h[0], h[0]), mul(h[1], h[1])), mul(h[2], h[2]))), distance);
		Pair offset { 0.0f, 0.0f };
		float at[3];
		for (int k = 0; k < 3; ++k) {
			const Pair q = mul(h[k], s);
			at[k]        = single(q);
			offset       = add(offset, mul(q, n[k]));
		}
		g0   = make_float4(at[0], at[1], at[2], single(offset));
		g1   = make_float4(n[0], n[1], n[2], 0.0f);
		near = single(inverse(mul(pairOf(0.02), distance)));
	}
	a.guideA[p] = g0;
	a.guideB[p] = g1;
	a.near[p]   = near;
	float dv[3] = { 1.0f, 1.0f, 1.0f };
	if (!a.demodulated) {
		for (int c = 0; c < 3; ++c) dv[c] = divisorOf(a.albedo[3 * p + c]);
	}
	const float cr = a.colour[3 * p], cg = a.colour[3 * p + 1], cb = a.colour[3 * p + 2];
	float variance = -1.0f;
	const float length = a.length[p];
	if (length >= 4.0f) {
		const Pair l      = lumaPair({ cr, 0.0f }, { cg, 0.0f }, { cb, 0.0f });
		const Pair scale  = lumaPair({ dv[0], 0.0f }, { dv[1], 0.0f }, { dv[2], 0.0f });
		const Pair spread = add({ a.moment[p], 0.0f }, negative(mul(l, l)));
		variance          = spread.h > 0.0f ? single(mul(spread, inverse(mul(mul(scale, scale), length)))) : 0.0f;
		// what a pair does not hold (an infinity, a square past FP32's range) is worked out in double
		if (!isfinite(variance) || !isfinite(a.moment[p])) {
			const double ld = 0.2126 * double(cr) + 0.7152 * double(cg) + 0.0722 * double(cb);
			const double sd = 0.2126 * double(dv[0]) + 0.7152 * double(dv[1]) + 0.0722 * double(dv[2]);
			const double apart = double(a.moment[p]) - ld * ld;
			variance           = float((apart > 0.0 ? apart : 0.0) / (double(length) * sd * sd));
		}
	}
	// a quotient of floats rounds as its double would, rounded
	a.lightA[p] = make_float4(cr / dv[0], cg / dv[1], cb / dv[2], variance);
}

// The weight of tap q for centre p (atrous.cpp:260-300); b.w is 1 in the sky.
__device__ __forceinline__ float tapWeight(float4 pa, float4 pb, float plum, float4 qa, float4 qb, float qlum, float invPlane, float invDev, float kernel) {
	const float facing = fmaf(pb.w, qb.w, fmaf(pb.z, qb.z, fmaf(pb.y, qb.y, pb.x * qb.x)));
	float power        = facing > 0.5f ? facing : 0.0f;
#pragma unroll
	for (int n = 0; n < 7; ++n) power *= power;
	const float along = fmaf(qa.z, pb.z, fmaf(qa.y, pb.y, qa.x * pb.x));
	const float plane = fabsf(along - pa.w) * invPlane;
	return kernel * power * quickExp(fmaf(fabsf(qlum - plum), invDev, plane));
}

// Whether a tap lies outside the frame; Inside: no tap of the block's does.
template <bool Inside>
__device__ __forceinline__ bool outside(const DenoiseArgs& a, int qx, int qy) {
	return !Inside && (qx < 0 || qx >= a.width || qy < 0 || qy >= a.height);
}

template <bool Inside>
__device__ __forceinline__ float spatialVariance(const DenoiseArgs& a, int x, int y, float4 lp) {
	const size_t p  = size_t(y) * size_t(a.width) + size_t(x);
	const float4 pa = a.guideA[p], pb = a.guideB[p];
	const float plum = luma(lp.x, lp.y, lp.z), invPlane = a.near[p];
	float sr = 0.0f, sg = 0.0f, sb = 0.0f, sq = 0.0f, sw = 0.0f;
#pragma unroll 1
	for (int j = -3; j <= 3; ++j) {
		const int row = (y + j) * a.width + x;
#pragma unroll
		for (int i = -3; i <= 3; ++i) {
			if (outside<Inside>(a, x + i, y + j)) continue;
			const int q     = row + i;
			const float4 lq = a.lightA[q];
			const float qlum = luma(lq.x, lq.y, lq.z);
			const float w    = tapWeight(pa, pb, plum, a.guideA[q], a.guideB[q], qlum, invPlane, 0.0f, 1.0f);
			sr = fmaf(w, lq.x, sr);
			sg = fmaf(w, lq.y, sg);
			sb = fmaf(w, lq.z, sb);
			sw += w;
			sq = fmaf(w * qlum, qlum, sq);
		}
	}
	if (!(sw > 0.0f)) return 0.0f;
	const float mean = luma(sr, sg, sb) / sw;
	const float v    = sq / sw - mean * mean;
	return v > 0.0f ? v : 0.0f;
}

__global__ void __launch_bounds__(kBlockX * kBlockY) varianceKernel(const __grid_constant__ DenoiseArgs a) {
	const int x = blockIdx.x * blockDim.x + threadIdx.x;
	const int y = blockIdx.y * blockDim.y + threadIdx.y;
	if (x >= a.width || y >= a.height) return;
	const size_t p = size_t(y) * size_t(a.width) + size_t(x);
	float4 l       = a.lightA[p];
	const int left = blockIdx.x * kBlockX, top = blockIdx.y * kBlockY;
	const bool in  = left >= 3 && top >= 3 && left + kBlockX + 3 <= a.width && top + kBlockY + 3 <= a.height;
	if (l.w < 0.0f) l.w = in ? spatialVariance<true>(a, x, y, l) : spatialVariance<false>(a, x, y, l);
	a.lightB[p] = l;
}

// A centre of the filter and what its taps come to.
struct Centre {
	float4 pa, pb, lp;
	float plum, invDev, invPlane;
	float sr = 0.0f, sg = 0.0f, sb = 0.0f, sv = 0.0f, sw = 0.0f;
};

template <int Step, bool Inside>
__device__ __forceinline__ void centreAt(Centre& c, const DenoiseArgs& a, const float4* __restrict__ in, int x, int y) {
	const float gauss[3] = { 0.25f, 0.5f, 0.25f };
	const int p = y * a.width + x;
	c.lp        = in[p];
	c.plum      = luma(c.lp.x, c.lp.y, c.lp.z);
	// prefilteredDeviation: the 3x3 Gaussian of the variance
	float vs = 0.0f, vw = 0.0f;
#pragma unroll
	for (int j = -1; j <= 1; ++j) {
#pragma unroll
		for (int i = -1; i <= 1; ++i) {
			if (outside<Inside>(a, x + i, y + j)) continue;
			const float k = gauss[i + 1] * gauss[j + 1];
			vs            = fmaf(k, in[p + j * a.width + i].w, vs);
			vw += k;
		}
	}
	c.invDev   = 1.0f / fmaf(4.0f, sqrtf(vs / vw), fmaf(1e-3f, c.plum, 1e-4f));
	c.pa       = a.guideA[p];
	c.pb       = a.guideB[p];
	c.invPlane = a.near[p] * (1.0f / float(Step));
}

// A thread filters kCentres pixels a step apart down the frame: their taps
// are the same but for a row at each end, so a tap's 48 bytes are loaded for
// all of them at once (a 1080p pass of one pixel a thread 97 to 117 us, of
// two 94 to 103, of three slower: registers).
constexpr int kCentres = 2;

// The topmost row of a slot of kCentres rows Step apart.
template <int Step>
__device__ __forceinline__ int rowOf(int slot) { return slot / Step * (kCentres * Step) + slot % Step; }

template <int Step, bool Inside>
__device__ __forceinline__ void filter(Centre (&c)[kCentres], const DenoiseArgs& a, const float4* __restrict__ in, int x, int y) {
	const float spline[5] = { 1.0f / 16, 1.0f / 4, 3.0f / 8, 1.0f / 4, 1.0f / 16 };
	for (int k = 0; k < kCentres; ++k) {
		if (Inside || y + k * Step < a.height) centreAt<Step, Inside>(c[k], a, in, x, y + k * Step);
	}
#pragma unroll
	for (int j = -2; j <= 1 + kCentres; ++j) {
		const int row = (y + j * Step) * a.width + x;
#pragma unroll
		for (int i = -2; i <= 2; ++i) {
			if (outside<Inside>(a, x + i * Step, y + j * Step)) continue;
			const int q     = row + i * Step;
			const float4 lq = in[q], qa = a.guideA[q], qb = a.guideB[q];
			const float qlum = luma(lq.x, lq.y, lq.z);
#pragma unroll
			for (int k = 0; k < kCentres; ++k) {
				if (j - k < -2 || j - k > 2) continue;
				const float w = tapWeight(c[k].pa, c[k].pb, c[k].plum, qa, qb, qlum, c[k].invPlane, c[k].invDev, spline[i + 2] * spline[j - k + 2]);
				c[k].sr = fmaf(w, lq.x, c[k].sr);
				c[k].sg = fmaf(w, lq.y, c[k].sg);
				c[k].sb = fmaf(w, lq.z, c[k].sb);
				c[k].sv = fmaf(w * w, lq.w, c[k].sv);
				c[k].sw += w;
			}
		}
	}
}

template <int Step, bool Last>
__global__ void __launch_bounds__(kBlockX * kBlockY) atrousKernel(const __grid_constant__ DenoiseArgs a, const float4* __restrict__ in, float4* __restrict__ out) {
	const int x = blockIdx.x * kBlockX + threadIdx.x;
	const int y = rowOf<Step>(blockIdx.y * kBlockY + threadIdx.y);
	if (x >= a.width || y >= a.height) return;
	const int left = blockIdx.x * kBlockX, top = rowOf<Step>(blockIdx.y * kBlockY), bottom = rowOf<Step>(blockIdx.y * kBlockY + kBlockY - 1) + (kCentres - 1) * Step;
	Centre c[kCentres] {};
	if (left >= 2 * Step && left + kBlockX + 2 * Step <= a.width && top >= 2 * Step && bottom + 2 * Step < a.height) filter<Step, true>(c, a, in, x, y);
	else filter<Step, false>(c, a, in, x, y);
	for (int k = 0; k < kCentres; ++k) {
		if (y + k * Step >= a.height) return;
		const size_t p = size_t(y + k * Step) * size_t(a.width) + size_t(x);
		float4 l       = c[k].lp;
		if (c[k].sw > 0.0f) {
			const float scale = 1.0f / c[k].sw;
			l = make_float4(c[k].sr * scale, c[k].sg * scale, c[k].sb * scale, c[k].sv * scale * scale);
		}
		if (!Last) {
			out[p] = l;
			continue;
		}
		// remodulatedImage: share = 1 / (1 + length / 8)
		const Pair share  = mul(inverse(sum(8.0f, a.length[p])), 8.0f);
		const Pair rest   = add({ 1.0f, 0.0f }, negative(share));
		const float f[3]  = { l.x, l.y, l.z };
		for (int ch = 0; ch < 3; ++ch) {
			const float dv    = divisorOf(a.albedo[3 * p + ch]);
			const Pair held   = a.demodulated ? product(a.colour[3 * p + ch], dv) : Pair { a.colour[3 * p + ch], 0.0f };
			float shown       = single(add(mul(product(f[ch], dv), share), mul(held, rest)));
			if (!isfinite(shown)) { // what a pair does not hold, in double
				const double sd = 1.0 / (1.0 + double(a.length[p]) / 8.0), cd = double(a.colour[3 * p + ch]);
				shown           = float(double(f[ch]) * double(dv) * sd + (a.demodulated ? cd * double(dv) : cd) * (1.0 - sd));
			}
			a.out[3 * p + ch] = shown;
		}
	}
}

} // namespace

cudaError_t launchDenoise(const DenoiseArgs& args, cudaStream_t stream) {
	const dim3 block(kBlockX, kBlockY);
	const dim3 grid((args.width + kBlockX - 1) / kBlockX, (args.height + kBlockY - 1) / kBlockY);
	const double* L       = args.lens;
	const double sideways = L[12] * L[13];
	Lens lens;
	for (int k = 0; k < 3; ++k) {
		lens.corner[k] = pairOf(L[3 + k] - L[6 + k] * sideways + L[9 + k] * L[12]);
		lens.across[k] = pairOf(L[6 + k] * (2.0 * sideways / double(args.width)));
		lens.down[k]   = pairOf(L[9 + k] * (-2.0 * L[12] / double(args.height)));
	}
	prepKernel<<<grid, block, 0, stream>>>(args, lens);
	varianceKernel<<<grid, block, 0, stream>>>(args);
	// the spatial variance lives in lightB; the passes ping-pong B -> A -> B ...
	const auto slots = [&](int step) {
		const int rows = (args.height + kCentres * step - 1) / (kCentres * step) * step;
		return dim3(grid.x, (rows + kBlockY - 1) / kBlockY);
	};
	atrousKernel<1, false><<<slots(1), block, 0, stream>>>(args, args.lightB, args.lightA);
	atrousKernel<2, false><<<slots(2), block, 0, stream>>>(args, args.lightA, args.lightB);
	atrousKernel<4, false><<<slots(4), block, 0, stream>>>(args, args.lightB, args.lightA);
	atrousKernel<8, true><<<slots(8), block, 0, stream>>>(args, args.lightA, nullptr);
	return cudaGetLastError();
}

} // namespace kdn
