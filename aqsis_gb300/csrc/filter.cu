// filter.cu -- pixel reconstruction filter, exposure and quantize.
//
// Replaces CqBucketProcessor::FilterBucket (non-separable path,
// libs/core/bucketprocessor.cpp:584-664, 686-707), ExposeBucket (766-806) and
// the quantize of CqDisplayRequest::FormatBucketForDisplay
// (ddmanager/ddmanager.cpp:1022-1119).  One thread per display pixel walks
// the (2*shift+1)^2 neighbouring pixels and their samples in the reference's
// loop order (fy, fx, sy, sx), so the float sums round identically.
#include <algorithm>
#include <type_traits>

#include "aqh_internal.h"
#include "hider_device.cuh"
#include "sample_common.cuh"

namespace aqh {

namespace {

// aqsis lround (math.h:67-70) in double: lfloor(x - 0.5) + 1
__device__ __forceinline__ double lround_d(double x) {
	const double y = x - 0.5;
	long long i = (long long)y;
	i -= (y < 0.0 && y != (double)i) ? 1 : 0;
	return (double)(i + 1);
}

// The 8-bit value of channel value `v` with dither term dith * s: lround of
// v * one + dith * s in double, clamped to [min, max] (ddmanager.cpp:1054-1114),
// for min >= 0 and max <= 255.  FP64 issues at 1/64 of the FP32 rate on this
// GPU, so the sum is taken in float first: with both terms below 512 its error
// and that of subtracting 1/2 are below 4 * 2^-15 = 2^-13, so where the result
// is further than 2^-12 from an integer its floor is the double one's.  The rest
// (one value in 2,000, anything large or NaN) takes the double form.  With
// the reciprocal below: 16 samples at 1080p 658 -> 618 us on the tile kernel.
// The double forms are calls: inlined four times at the end of a pixel they cost
// the loop over its samples its schedule (320x240, 16 samples: 37 us before the
// float form, 40 with the double one inlined, 31 called).
__device__ __noinline__ uint8_t quantize8_double(float v, float one, float dith, float s, float qmin, float qmax) {
	double value = lround_d(0.0 + (double)v * (double)(one - 0.0f) + ((double)dith * (double)s));
	value = value < (double)qmin ? (double)qmin : (value > (double)qmax ? (double)qmax : value);
	return (uint8_t)(int)value;
}
__device__ __forceinline__ uint8_t quantize8(float v, float one, float dith, float s, float qmin, float qmax) {
	const float a = v * one, b = dith * s;
	const float t = (a + b) - 0.5f;
	const float f = floorf(t), frac = t - f;
	if (fabsf(a) < 512.0f && fabsf(b) < 512.0f && frac > 0.000244140625f && frac < 1.0f - 0.000244140625f) {
		const float r = f + 1.0f;
		return (uint8_t)(int)(r < qmin ? qmin : (r > qmax ? qmax : r));
	}
	return quantize8_double(v, one, dith, s, qmin, qmax);
}

// x^y rounded to float exactly as (float)pow((double)x, (double)y), for the
// exposure of a channel.  FP64 issues at 1/64 of the FP32 rate here, and the
// three double powers of a pixel were 600 us of a 935x533 frame's
// filter (1,078 us of which are 425 + 23 now).  x^y =
// 2^(y log2 x) is formed in pairs of floats: x = 2^e m with m scaled near 1 by
// one of eight 8-bit factors c, ln(m c) = 2 atanh(s) with s = (m c - 1) / (m c
// + 1), |s| < 0.031, by the series of atanh, and the power of two by its
// nearest eighth and the exponential series of the rest, |g| < 0.044.  Terms
// above 2^-17 carry a second float; the error of the pair is below 2^-39 of
// it.  Where the rounding to float could still depend on 2^-36 of the value
// (one in 2,000), and outside 2^-30 < x < 2^30, 1/16 <= y <= 4, the double
// power decides.
__device__ __forceinline__ float pow_double(float x, float y) { return (float)pow((double)x, (double)y); }
__device__ __forceinline__ float pow_rounded(float x, float y) {
	// 8-bit factor, minus its log2 as two floats, per eighth of [1, 2)
	constexpr float kC[8] = {0.94140625f, 0.84375f, 0.76171875f, 0.6953125f, 0.640625f, 0.59375f, 0.55078125f, 0.515625f};
	constexpr float kLh[8] = {0.087110661f, 0.245112494f, 0.392669678f, 0.524266541f,
	                          0.642448008f, 0.752072513f, 0.860448658f, 0.955605865f};
	constexpr float kLl[8] = {2.79982726e-09f, 4.20230739e-09f, 8.51601456e-09f, 2.80294206e-08f,
	                          -1.26785391e-08f, -2.65470703e-08f, -1.08651328e-08f, 1.61167044e-08f};
	// 2^(k/8), k = -4 .. 3, as two floats
	constexpr float kEh[8] = {0.707106769f, 0.771105409f, 0.840896428f, 0.917004049f,
	                          1.0f,         1.09050775f,  1.18920708f,  1.29683959f};
	constexpr float kEl[8] = {1.21016175e-08f, 4.03545242e-09f,  -1.23776633e-08f, -5.61963898e-09f,
	                          0.0f,            -1.30775399e-08f, 3.79763527e-08f,  -4.01899953e-08f};
	constexpr float kInvLn2H = 1.442695022f, kInvLn2L = 1.925963033e-08f;
	constexpr float kLn2H = 0.6931471825f, kLn2L = -1.904654323e-09f;
	constexpr float kThirdH = 0.3333333433f, kThirdL = -9.934107481e-09f;
	if (x == 0.0f && __float_as_int(x) == 0 && y > 0.0f) return 0.0f;
	if (!(x > 9.31322575e-10f && x < 1073741824.0f && y >= 0.0625f && y <= 4.0f)) return pow_double(x, y);
	const int bits = __float_as_int(x);
	const float e = (float)((bits >> 23) - 127);
	const int j = (bits >> 20) & 7;
	const float m = __int_as_float((bits & 0x007fffff) | 0x3f800000);
	float c = kC[0], th = kLh[0], tl = kLl[0];
#pragma unroll
	for (int i = 1; i < 8; ++i)
		if (j == i) {
			c = kC[i];
			th = kLh[i];
			tl = kLl[i];
		}
	// s = (m c - 1) / (m c + 1)
	const float p = m * c, pl = fmaf(m, c, -p);
	const float num = p - 1.0f, den = p + 1.0f, dl = (p - (den - 1.0f)) + pl;
	const float sh = num / den;
	const float sl = ((fmaf(-sh, den, num) + pl) - sh * dl) / den;
	// ln(m c) = 2 s (1 + q/3 + q^2/5 + ...), q = s^2
	const float qh = sh * sh, ql = fmaf(sh, sh, -qh) + 2.0f * sh * sl;
	const float wh = qh * kThirdH, wl = fmaf(qh, kThirdH, -wh) + fmaf(qh, kThirdL, ql * kThirdH);
	const float z = (qh * qh) * fmaf(qh, fmaf(qh, 0.111111111f, 0.142857143f), 0.2f);
	const float uh = 1.0f + wh, ul = (wh - (uh - 1.0f)) + (wl + z);
	const float s2 = 2.0f * sh, lh = s2 * uh, ll = fmaf(s2, uh, -lh) + fmaf(s2, ul, 2.0f * sl * uh);
	// log2 x = e - log2 c + ln(m c) / ln 2
	const float ah = lh * kInvLn2H, al = fmaf(lh, kInvLn2H, -ah) + fmaf(lh, kInvLn2L, ll * kInvLn2H);
	auto two_sum = [](float a, float b, float& err) {
		const float s = a + b, t = s - a;
		err = (a - (s - t)) + (b - t);
		return s;
	};
	float e1, e2;
	const float b1 = two_sum(e, th, e1), b2 = two_sum(b1, ah, e2);
	const float low = ((e1 + e2) + tl) + al;
	const float Lh = b2 + low, Ll = low - (Lh - b2);
	// t = y log2 x = n + k/8 + r
	const float t = y * Lh, tlo = fmaf(y, Lh, -t) + y * Ll;
	const float n8 = rintf(t * 8.0f), r = t - n8 * 0.125f;
	const int i8 = (int)n8, n = (i8 + 4) >> 3, k = i8 - 8 * n + 4;
	const float g0 = r * kLn2H, g1 = fmaf(r, kLn2H, -g0) + fmaf(r, kLn2L, tlo * kLn2H);
	float gl;
	const float gh = two_sum(g0, g1, gl);
	// e^g - 1
	const float hh = 0.5f * gh, qa = hh * gh, qb = fmaf(hh, gh, -qa) + gh * gl;
	const float g3 = (gh * gh) * gh;
	const float tail = g3 * fmaf(gh, fmaf(gh, fmaf(gh, 0.00138888889f, 0.00833333333f), 0.0416666667f), 0.166666667f);
	const float xh = gh + qa, xl = (qa - (xh - gh)) + ((gl + qb) + tail);
	float eh = kEh[0], el = kEl[0];
#pragma unroll
	for (int i = 1; i < 8; ++i)
		if (k == i) {
			eh = kEh[i];
			el = kEl[i];
		}
	const float v = eh * xh, vl = (fmaf(eh, xh, -v) + fmaf(eh, xl, el * xh)) + el;
	const float rh = eh + v, rl = (v - (rh - eh)) + vl;
	const float d = rh * 1.45519152e-11f;  // 2^-36
	const float up = rh + (rl + d), dn = rh + (rl - d);
	if (up != dn) return pow_double(x, y);
	return __int_as_float(__float_as_int(up) + (n << 23));
}

// 1.0 / (double)g rounded to float.  A quotient of two floats rounded to
// double's 53 bits and then to float's 24 is the float quotient (53 >= 2 * 24 +
// 2), where neither overflows or loses bits to underflow.
__device__ __noinline__ float reciprocal_double(float g) { return (float)(1.0 / (double)g); }
__device__ __forceinline__ float reciprocal_rounded(float g) {
	const float m = fabsf(g);
	if (m > 1e-30f && m < 1e30f) return 1.0f / g;
	return reciprocal_double(g);
}

__device__ __forceinline__ void finish_pixel(const FrameParams& fp, const SamplerDev& smp, int spp, float gTot,
                                             int count, const float acc[7], float* __restrict__ chan,
                                             uint8_t* __restrict__ q8, int x, int y);
__device__ __forceinline__ void store_pixel(const FrameParams& fp, const SamplerDev& smp, const float c[9],
                                            float* __restrict__ chan, uint8_t* __restrict__ q8, int x, int y);

// One display pixel (x, y).  SPP > 0: samples per pixel known at compile
// time (the sample loop is unrolled by four so its loads issue together); 0:
// read from fp.
template <int SPP>
__device__ __forceinline__ void filter_pixel(const FrameParams& fp, const SamplerDev& smp, const SampleStore& st,
                                             const float* __restrict__ ftab, float* __restrict__ chan,
                                             uint8_t* __restrict__ q8, int x, int y) {
	const float xcent = x + 0.5f, ycent = y + 0.5f;
	const int xmax = fp.shiftX, ymax = fp.shiftY;
	const int spp = SPP > 0 ? SPP : fp.spp;
	float gTot = 0.0f;
	int count = 0;
	float acc[7] = {0, 0, 0, 0, 0, 0, 0};
	for (int fy = -ymax; fy <= ymax; fy++) {
		const int py = y + fy;
		for (int fx = -xmax; fx <= xmax; fx++) {
			const int px = x + fx;
			const long long pix = (long long)(py - fp.sy0) * fp.sw + (px - fp.sx0);
			const long long pat = (st.wmask || !smp.pos_index) ? pix : (long long)__ldg(smp.pos_index + pix);
			const int bit = (fy + ymax) * (2 * xmax + 1) + fx + xmax;
			const int index = bit * spp;
			const float fpx = (float)px, fpy = (float)py;
			// samples in groups of four: the window tests of a group first, then
			// the sample data of the samples inside it, so each group costs two
			// memory round trips; the sums still run in sample order
			for (int i0 = 0; i0 < spp; i0 += 4) {
				bool in[4];
				float gv[4];
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					const int i = i0 + j;
					const bool ok = (SPP > 0 && SPP % 4 == 0) || i < spp;
					const int ic = ok ? i : i0;
					if (st.wmask) {
						in[j] = ok && ((__ldg(st.wmask + store_index(pix, ic, spp)) >> bit) & 1u);
					} else {
						const float2 o = __ldg(smp.pos + pat * spp + ic);
						const float vx = (fpx + o.x) - xcent;
						const float vy = (fpy + o.y) - ycent;
						in[j] = ok && vx >= -fp.xfwo2 && vy >= -fp.yfwo2 && vx <= fp.xfwo2 && vy <= fp.yfwo2;
					}
					gv[j] = __ldg(ftab + index + ic);
				}
				float4 av[4], bv[4];
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					const long long si = store_index(pix, in[j] ? i0 + j : i0, spp);
					bv[j] = in[j] ? __ldg(st.b + si) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
					av[j] = in[j] ? __ldg(st.a + si) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
				}
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					if (in[j]) {
						const float gw = gv[j];
						gTot += gw;
						if (bv[j].w != 0.0f) {
							const float4 a = av[j], b = bv[j];
							acc[0] += a.x * gw;
							acc[1] += a.y * gw;
							acc[2] += a.z * gw;
							acc[3] += b.x * gw;
							acc[4] += b.y * gw;
							acc[5] += b.z * gw;
							acc[6] += a.w * gw;
							count++;
						}
					}
				}
			}
		}
	}
	finish_pixel(fp, smp, spp, gTot, count, acc, chan, q8, x, y);
}

// The end of FilterBucket for one display pixel from its sums: normalisation
// by the weight total (1/gTot in double, rounded to float), coverage and
// alpha; then the channel-buffer write and the frame's fused 8-bit r g b a
// display.  Frames with exposure go through expose_kernel afterwards.
__device__ __forceinline__ void finish_pixel(const FrameParams& fp, const SamplerDev& smp, int spp, float gTot,
                                             int count, const float acc[7], float* __restrict__ chan,
                                             uint8_t* __restrict__ q8, int x, int y) {
	float c[9];
	float coverage;
	if (count == 0) {
#pragma unroll
		for (int k = 0; k < 9; ++k) c[k] = 0.0f;
		c[7] = FLT_MAX;
		coverage = 0.0f;
	} else {
		const float inv = reciprocal_rounded(gTot);
		c[0] = acc[0] * inv; c[1] = acc[1] * inv; c[2] = acc[2] * inv;
		c[3] = acc[3] * inv; c[4] = acc[4] * inv; c[5] = acc[5] * inv;
		c[7] = acc[6] * inv;
		coverage = (count >= spp) ? 1.0f : (float)count / (float)spp;
	}
	const float a = (c[3] + c[4] + c[5]) / 3.0f;
	c[6] = a * coverage;
	c[8] = coverage;
	store_pixel(fp, smp, c, chan, q8, x, y);
}

// The channel-buffer write of one display pixel and the frame's fused 8-bit
// r g b a display.
__device__ __forceinline__ void store_pixel(const FrameParams& fp, const SamplerDev& smp, const float c[9],
                                            float* __restrict__ chan, uint8_t* __restrict__ q8, int x, int y) {
	const long long p = (long long)(y - fp.crop_y0) * (fp.crop_x1 - fp.crop_x0) + (x - fp.crop_x0);
	float* out = chan + p * 9;
#pragma unroll
	for (int k = 0; k < 9; ++k) out[k] = c[k];
	if (q8) {
		// the frame's own display, r g b a, quantized as quantize_u8_kernel does
		const float s = smp.dither ? __ldg(smp.dither + p) : 0.0f;
		const float src[4] = {c[0], c[1], c[2], c[6]};
		uchar4 q;
		unsigned char* qb = reinterpret_cast<unsigned char*>(&q);
#pragma unroll
		for (int k = 0; k < 4; ++k)
			qb[k] = fp.q_one != 0.0f ? quantize8(src[k], fp.q_one, fp.q_dither, s, fp.q_min, fp.q_max)
			                         : (uint8_t)(int)(double)src[k];
		reinterpret_cast<uchar4*>(q8)[p] = q;
	}
}

// 16x16-pixel tiles of the crop window in raster order, `gridDim.x` of them
// in flight at once.
template <int SPP>
__global__ void __launch_bounds__(256)
filter_kernel(FrameParams fp, SamplerDev smp, SampleStore st, const float* __restrict__ ftab,
              float* __restrict__ chan, uint8_t* __restrict__ q8) {
	const int ntx = (fp.crop_x1 - fp.crop_x0 + 15) >> 4, nty = (fp.crop_y1 - fp.crop_y0 + 15) >> 4;
	for (int tile = blockIdx.x; tile < ntx * nty; tile += gridDim.x) {
		const int x = fp.crop_x0 + (tile % ntx) * 16 + (threadIdx.x & 15);
		const int y = fp.crop_y0 + (tile / ntx) * 16 + (threadIdx.x >> 4);
		if (x < fp.crop_x1 && y < fp.crop_y1) filter_pixel<SPP>(fp, smp, st, ftab, chan, q8, x, y);
	}
}

// ---- windows of 3x3 and 5x5 pixels (filter widths in [2, 6)): a rolling window ----
//
// One thread owns a display column and a run of rows.  With SH the filter's
// shift (1 or 2) it reads each row of input pixels once and adds every sample
// to the 2 SH + 1 output rows whose windows hold that row, from the row SH
// below it (window row fy = -SH) to the row SH above (fy = +SH).  Output row y
// takes its terms of window row fy from input row y + fy; input rows ascend,
// and within an input row the columns ascend (fx = -SH .. SH) and then the
// samples -- the reference's (fy, fx, sy, sx) order, so every sum rounds
// exactly as in filter_pixel.  Each sample is loaded by 2 SH + 1 threads (the
// neighbouring columns) instead of (2 SH + 1)^2, once per run of rows plus the
// SH rows on either side of it.
//
// Two neighbouring lanes share a column: one sums r, g, b and depth (the
// store's first record), the other the opacity (the second), so each holds
// half the sums (2 SH + 1 rows of them are live) and twice as many warps fit:
// the pass waits on loads, not on bandwidth.  Samples are loaded whether or
// not a window holds them, so a group's records and window words make one
// round trip.  Where windows are tested at sample positions the two lanes test
// half of a group each (1400x1000, 49 samples, 2x2 filter: 2.42 ms with every
// test in both lanes, 1.89 here, 2.08 with a thread per column).  1920x1080,
// 64 samples, 3x3: 3.82 ms with a thread per column, 2.22 ms here (14 GB of L2
// misses at 6.3 TB/s); 16 samples 658 us on the tile kernel, 399 us here;
// 935x533, 15 samples, 5x5 with exposure 977 us on the tile kernel, 425 + 23
// us here.
struct FiltSum {
	float acc[4];
	float gTot;
	int count;
};
__device__ __forceinline__ void fsum_reset(FiltSum& f) {
#pragma unroll
	for (int k = 0; k < 4; ++k) f.acc[k] = 0.0f;
	f.gTot = 0.0f;
	f.count = 0;
}

constexpr int kRollThreads = 128;  // threads per CTA: half as many display columns
constexpr int kRollCols = kRollThreads / 2;

// Display rows per CTA: a longer run reads fewer rows twice, a shorter one
// makes more CTAs; the most rows that leave at least `least` of them.
// Measured (us, rows 1 / 2 / 4 / 8 / 16): 1920x1080, 16 samples, 3x3: 884 / 605
// / 486 / 436 / 399; 640x480: 137 / 96 / 77 / 94 / 157; 320x240, 4 samples: 15 /
// 15 / 20 / 32 / 56; 935x533, 15 samples, 5x5: 1152 / 702 / 507 / 425 / 499 and
// its three output variables 753 / 441 / 413 / 306 / 439 (half as many CTAs for
// the same rows: three per SM, the colours four).  5x5 windows read more rows
// twice, so that a CTA in 32 fewer is worth eight rows to them (640x480, 16
// samples: 307 us with four, 247 with the 600 CTAs of eight).
inline int roll_rows(int cols, int h, int least) {
	int rows = 16;
	while (rows > 1 && (long long)cols * ((h + rows - 1) / rows) < least) rows >>= 1;
	return rows;
}

// With every sample offset in [0, 1] and half-widths of at least SH + 1/2,
// every sample of the neighbourhood passes the window test in float: for fx =
// -SH, (px + o) >= px rounds to at least x - SH and x + 0.5 is exact below
// 2^22, so v >= -(SH + 1/2); for fx = +SH, px + o <= x + SH + 1, so v <= SH +
// 1/2; the others and the rows alike.  The test then decides nothing.
__device__ __forceinline__ bool rolling_allin(const FrameParams& fp, const SamplerDev& smp, int sh) {
	const int lim = 1 << 22;
	const float half = (float)sh + 0.5f;
	return smp.pos_unit && fp.xfwo2 >= half && fp.yfwo2 >= half && fp.sx0 > -lim && fp.sy0 > -lim &&
	       fp.sx0 + fp.sw < lim && fp.sy0 + fp.sh < lim;
}

// The weights in shared memory as [fx][sample][window row], window rows padded
// to WP, so that one sample's weights for every row are one or two loads.
template <int SH>
struct RollTab {
	static constexpr int W = 2 * SH + 1, WP = SH == 1 ? 4 : 8;
	__device__ static void load(float* tab, const float* __restrict__ ftab, int spp) {
		for (int i = threadIdx.x; i < W * W * spp; i += kRollThreads) {
			const int k = i / (W * spp), r = i - k * W * spp;  // window row, (fx, sample)
			tab[r * WP + k] = ftab[i];
		}
	}
	__device__ static void weights(const float* tab, int at, float gw[W]) {
		const float4 a = *reinterpret_cast<const float4*>(tab + at * WP);
		gw[0] = a.x;
		gw[1] = a.y;
		gw[2] = a.z;
		if (SH == 2) {
			gw[W - 2] = a.w;
			gw[W - 1] = tab[at * WP + W - 1];
		}
	}
};

// The windows sample (ic of pattern `pat`) of pixel (fpx, r) lies in: bit k for
// window row fy = k - SH.
template <int SH>
__device__ __forceinline__ uint32_t roll_inside(const FrameParams& fp, const float2 o, float fpx, float fpy,
                                                float xcent, int r) {
	constexpr int W = 2 * SH + 1;
	const float vx = (fpx + o.x) - xcent;
	if (!(vx >= -fp.xfwo2 && vx <= fp.xfwo2)) return 0u;
	uint32_t m = 0u;
#pragma unroll
	for (int k = 0; k < W; ++k) {
		const float v = (fpy + o.y) - ((float)(r - (k - SH)) + 0.5f);
		if (v >= -fp.yfwo2 && v <= fp.yfwo2) m |= 1u << k;
	}
	return m;
}
// The same from a window word: every W-th bit from fx + SH on.
template <int SH>
__device__ __forceinline__ uint32_t roll_bits(uint32_t word, int fx) {
	constexpr int W = 2 * SH + 1;
	const uint32_t w = word >> (fx + SH);
	uint32_t m = 0u;
#pragma unroll
	for (int k = 0; k < W; ++k) m |= ((w >> (k * W)) & 1u) << k;
	return m;
}

// Input row Q0 + Q (0 .. R + 2 SH - 1) of a run: r = y0 - SH + q feeds output
// rows y0 + q (window row k = 0) to y0 + q - 2 SH (k = 2 SH), which is then
// complete.  Slots rotate with the input row: output row y0 + n lives in S[n %
// W].  MASK: the frame has window words.  All lanes of a warp take part (x is
// clamped; `write` says whose pixel it is).
template <int SPP, int SH, bool MASK, int Q>
__device__ __forceinline__ void roll_steps(const FrameParams& fp, const SamplerDev& smp, const SampleStore& st,
                                           const float* tab, float* __restrict__ chan, uint8_t* __restrict__ q8, int x,
                                           int y0, int q0, int R, FiltSum (&S)[2 * SH + 1], bool allin, bool write) {
	constexpr int W = 2 * SH + 1;
	if constexpr (Q < W) {
		const int q = q0 + Q;
		if (q >= R + 2 * SH) return;
		const int spp = SPP > 0 ? SPP : fp.spp;
		const bool opac = threadIdx.x & 1;  // this lane sums the opacity record
		if (q < R) fsum_reset(S[Q]);
		uint32_t use = 0;
#pragma unroll
		for (int k = 0; k < W; ++k) use |= (q - k >= 0 && q - k < R) ? 1u << k : 0u;
		const int r = y0 - SH + q;
		const float xcent = x + 0.5f, fpy = (float)r;
		for (int fx = -SH; fx <= SH; ++fx) {
			const int px = x + fx;
			const long long pix = (long long)(r - fp.sy0) * fp.sw + (px - fp.sx0);
			const long long at = store_index(pix, 0, spp);
			const float4* __restrict__ rec = (opac ? st.b : st.a) + at;
			const uint32_t* __restrict__ words = MASK ? st.wmask + at : nullptr;
			const float2* __restrict__ pos =
			    (MASK || allin) ? nullptr : smp.pos + (smp.pos_index ? (long long)__ldg(smp.pos_index + pix) : pix) * spp;
			// samples in groups of four, whose loads are in flight together
			for (int i0 = 0; i0 < spp; i0 += 4) {
				float4 v[4];
				uint32_t in[4];
				bool valid[4];
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					const bool ok = (SPP > 0 && SPP % 4 == 0) || i0 + j < spp;
					const int i = ok ? i0 + j : i0;
					v[j] = __ldg(rec + i * 32);
					if (MASK) {
						const uint32_t w = __ldg(words + i * 32);
						valid[j] = (w & kMaskValid) != 0u;
						in[j] = ok ? w : 0u;
					} else {
						in[j] = ok ? (1u << W) - 1u : 0u;
					}
				}
				if (!MASK && !allin) {
					// the two lanes of a column test two of the four positions each
					uint32_t mine[2], theirs[2];
#pragma unroll
					for (int j = 0; j < 2; ++j) {
						const int i = i0 + (opac ? 2 : 0) + j;
						const bool ok = (SPP > 0 && SPP % 4 == 0) || i < spp;
						mine[j] = ok ? roll_inside<SH>(fp, __ldg(pos + i), (float)px, fpy, xcent, r) : 0u;
						theirs[j] = __shfl_xor_sync(0xffffffffu, mine[j], 1);
					}
#pragma unroll
					for (int j = 0; j < 2; ++j) {
						in[j] = opac ? theirs[j] : mine[j];
						in[2 + j] = opac ? mine[j] : theirs[j];
					}
				}
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					if (MASK) {
						in[j] = roll_bits<SH>(in[j], fx);
					} else {
						const float other = __shfl_xor_sync(0xffffffffu, v[j].w, 1);
						valid[j] = (opac ? v[j].w : other) != 0.0f;
					}
					in[j] &= use;
				}
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					float gw[W];
					RollTab<SH>::weights(tab, (fx + SH) * spp + ((SPP > 0 && SPP % 4 == 0) || i0 + j < spp ? i0 + j : i0), gw);
#pragma unroll
					for (int k = 0; k < W; ++k)
						if ((in[j] >> k) & 1u) {
							FiltSum& f = S[(Q + W - k) % W];
							f.gTot += gw[k];
							if (valid[j]) {
								f.acc[0] += v[j].x * gw[k];
								f.acc[1] += v[j].y * gw[k];
								f.acc[2] += v[j].z * gw[k];
								f.acc[3] += v[j].w * gw[k];  // depth (unused by the opacity lane)
								f.count++;
							}
						}
				}
			}
		}
		if (q >= 2 * SH) {
			const FiltSum& A = S[(Q + 1) % W];  // k = 2 SH
			float acc[7] = {A.acc[0], A.acc[1], A.acc[2], 0.0f, 0.0f, 0.0f, A.acc[3]};
#pragma unroll
			for (int c = 0; c < 3; ++c) acc[3 + c] = __shfl_xor_sync(0xffffffffu, A.acc[c], 1);
			if (write && !opac) finish_pixel(fp, smp, spp, A.gTot, A.count, acc, chan, q8, x, y0 + q - 2 * SH);
		}
		roll_steps<SPP, SH, MASK, Q + 1>(fp, smp, st, tab, chan, q8, x, y0, q0, R, S, allin, write);
	}
}

template <int SPP, int SH, bool MASK>
__global__ void __launch_bounds__(kRollThreads)
filter_roll_kernel(FrameParams fp, SamplerDev smp, SampleStore st, const float* __restrict__ ftab,
                   float* __restrict__ chan, uint8_t* __restrict__ q8, int rows) {
	constexpr int W = 2 * SH + 1;
	__shared__ __align__(16) float tab[kRollTaps / W * RollTab<SH>::WP + 4];
	RollTab<SH>::load(tab, ftab, SPP > 0 ? SPP : fp.spp);
	__syncthreads();
	const int x = fp.crop_x0 + blockIdx.x * kRollCols + (threadIdx.x >> 1);
	const int y0 = fp.crop_y0 + blockIdx.y * rows;
	const int R = min(rows, fp.crop_y1 - y0);
	const bool allin = !MASK && rolling_allin(fp, smp, SH);
	FiltSum S[W];
#pragma unroll
	for (int k = 0; k < W; ++k) fsum_reset(S[k]);
	for (int q0 = 0; q0 < R + 2 * SH; q0 += W)
		roll_steps<SPP, SH, MASK, 0>(fp, smp, st, tab, chan, q8, min(x, fp.crop_x1 - 1), y0, q0, R, S, allin,
		                             x < fp.crop_x1);
}

// The vertex whose output variables micropolygon `id` carries (its vertex A).
__device__ __forceinline__ long long aov_vertex_of(const GridsDev& g, int id) {
	const int gi = grid_of(g, id);
	const int cu = __ldg(g.cu + gi);
	const int m = id - (int)__ldg(g.mpbase + gi);
	const int iv = m / cu, iu = m - iv * cu;
	return __ldg(g.cbase + gi) + (long long)iv * (cu + 1) + iu;
}

// Replaces every sample's micropolygon by that vertex, once, so that the
// filter's passes over the samples do not each look its grid up.  The last
// block of pixels (store_index) has places no sample fills: they are left.
__global__ void __launch_bounds__(256) aov_vertex_kernel(GridsDev g, int32_t* src, long long npix, int spp) {
	const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	const long long pix = i / (32 * spp) * 32 + (i & 31);
	if (pix < npix && src[i] >= 0) src[i] = (int32_t)aov_vertex_of(g, src[i]);
}

// Output variables [k0, k0 + NA) through 3x3 and 5x5 windows, by the rolling
// window of filter_roll_kernel (the same rows, order and weights), a thread
// per column, over the samples' vertices.
template <int NA>
struct AovSum {
	float acc[NA];
	float gTot;
	int count;
};

template <int SH, int NA, bool MASK, int Q>
__device__ __forceinline__ void aov_steps(const FrameParams& fp, const SamplerDev& smp, const SampleStore& st,
                                          const GridsDev& g, const float* tab, float* __restrict__ out, int x, int y0,
                                          int q0, int R, int k0, AovSum<NA> (&S)[2 * SH + 1], bool allin) {
	constexpr int W = 2 * SH + 1;
	if constexpr (Q < W) {
		const int q = q0 + Q;
		if (q >= R + 2 * SH) return;
		if (q < R) {
#pragma unroll
			for (int c = 0; c < NA; ++c) S[Q].acc[c] = 0.0f;
			S[Q].gTot = 0.0f;
			S[Q].count = 0;
		}
		uint32_t use = 0;
#pragma unroll
		for (int k = 0; k < W; ++k) use |= (q - k >= 0 && q - k < R) ? 1u << k : 0u;
		const int r = y0 - SH + q, spp = fp.spp, naov = g.naov;
		const float xcent = x + 0.5f;
		for (int fx = -SH; fx <= SH; ++fx) {
			const int px = x + fx;
			const long long pix = (long long)(r - fp.sy0) * fp.sw + (px - fp.sx0);
			const long long at = store_index(pix, 0, spp);
			const float2* __restrict__ pos =
			    (MASK || allin) ? nullptr : smp.pos + (smp.pos_index ? (long long)__ldg(smp.pos_index + pix) : pix) * spp;
			for (int i0 = 0; i0 < spp; i0 += 4) {
				uint32_t in[4];
				bool valid[4];
				int id[4];
				float v[4][NA];
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					const bool ok = i0 + j < spp;
					const int i = ok ? i0 + j : i0;
					id[j] = __ldg(st.aovsrc + at + i * 32);
					if (MASK) {
						const uint32_t w = __ldg(st.wmask + at + i * 32);
						valid[j] = (w & kMaskValid) != 0u;
						in[j] = ok ? w : 0u;
					} else {
						valid[j] = __ldg(&st.b[at + i * 32].w) != 0.0f;
						in[j] = !ok ? 0u : (allin ? (1u << W) - 1u : roll_inside<SH>(fp, __ldg(pos + i), (float)px, (float)r, xcent, r));
					}
				}
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					if (MASK) in[j] = roll_bits<SH>(in[j], fx);
					in[j] &= use;
#pragma unroll
					for (int c = 0; c < NA; ++c)
						v[j][c] = (in[j] && valid[j] && id[j] >= 0) ? __ldg(g.aov + (long long)id[j] * naov + k0 + c) : 0.0f;
				}
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					float gw[W];
					RollTab<SH>::weights(tab, (fx + SH) * spp + (i0 + j < spp ? i0 + j : i0), gw);
#pragma unroll
					for (int k = 0; k < W; ++k)
						if ((in[j] >> k) & 1u) {
							AovSum<NA>& A = S[(Q + W - k) % W];
							A.gTot += gw[k];
							if (valid[j]) {
								A.count++;
								if (id[j] >= 0)
#pragma unroll
									for (int c = 0; c < NA; ++c) A.acc[c] += v[j][c] * gw[k];
							}
						}
				}
			}
		}
		if (q >= 2 * SH) {
			const AovSum<NA>& A = S[(Q + 1) % W];
			float* o = out + ((long long)(y0 + q - 2 * SH - fp.crop_y0) * (fp.crop_x1 - fp.crop_x0) + (x - fp.crop_x0)) * naov;
			const float inv = A.count == 0 ? 0.0f : reciprocal_rounded(A.gTot);
#pragma unroll
			for (int c = 0; c < NA; ++c) o[k0 + c] = A.count == 0 ? 0.0f : A.acc[c] * inv;
		}
		aov_steps<SH, NA, MASK, Q + 1>(fp, smp, st, g, tab, out, x, y0, q0, R, k0, S, allin);
	}
}

template <int SH, int NA>
__global__ void __launch_bounds__(kRollThreads)
filter_aov_roll_kernel(FrameParams fp, SamplerDev smp, SampleStore st, GridsDev g, const float* __restrict__ ftab,
                       float* __restrict__ out, int k0, int rows) {
	constexpr int W = 2 * SH + 1;
	__shared__ __align__(16) float tab[kRollTaps / W * RollTab<SH>::WP + 4];
	RollTab<SH>::load(tab, ftab, fp.spp);
	__syncthreads();
	const int x = fp.crop_x0 + blockIdx.x * kRollThreads + threadIdx.x;
	const int y0 = fp.crop_y0 + blockIdx.y * rows;
	const int R = min(rows, fp.crop_y1 - y0);
	if (x >= fp.crop_x1 || R <= 0) return;
	AovSum<NA> S[W];
	if (st.wmask) {
		for (int q0 = 0; q0 < R + 2 * SH; q0 += W)
			aov_steps<SH, NA, true, 0>(fp, smp, st, g, tab, out, x, y0, q0, R, k0, S, false);
	} else {
		const bool allin = rolling_allin(fp, smp, SH);
		for (int q0 = 0; q0 < R + 2 * SH; q0 += W)
			aov_steps<SH, NA, false, 0>(fp, smp, st, g, tab, out, x, y0, q0, R, k0, S, allin);
	}
}

// Output variables of one display pixel: FilterBucket's weighted sum over
// the same window, weights and order as filter_pixel (gTot included), of the
// vertex-A values of each valid sample's front micropolygon.
template <int SPP>
__global__ void __launch_bounds__(256)
filter_aov_kernel(FrameParams fp, SamplerDev smp, SampleStore st, GridsDev g, const float* __restrict__ ftab,
                  float* __restrict__ out) {
	const int ntx = (fp.crop_x1 - fp.crop_x0 + 15) >> 4, nty = (fp.crop_y1 - fp.crop_y0 + 15) >> 4;
	const int spp = SPP > 0 ? SPP : fp.spp;
	const int naov = g.naov;
	for (int tile = blockIdx.x; tile < ntx * nty; tile += gridDim.x) {
		const int x = fp.crop_x0 + (tile % ntx) * 16 + (threadIdx.x & 15);
		const int y = fp.crop_y0 + (tile / ntx) * 16 + (threadIdx.x >> 4);
		if (x >= fp.crop_x1 || y >= fp.crop_y1) continue;
		const float xcent = x + 0.5f, ycent = y + 0.5f;
		const int xmax = fp.shiftX, ymax = fp.shiftY;
		float gTot = 0.0f;
		int count = 0;
		float acc[AQH_MAX_AOV];
#pragma unroll
		for (int k = 0; k < AQH_MAX_AOV; ++k) acc[k] = 0.0f;
		for (int fy = -ymax; fy <= ymax; fy++) {
			const int py = y + fy;
			for (int fx = -xmax; fx <= xmax; fx++) {
				const int px = x + fx;
				const long long pix = (long long)(py - fp.sy0) * fp.sw + (px - fp.sx0);
				const long long pat = (st.wmask || !smp.pos_index) ? pix : (long long)__ldg(smp.pos_index + pix);
				const int bit = (fy + ymax) * (2 * xmax + 1) + fx + xmax;
				const int index = bit * spp;
				const float fpx = (float)px, fpy = (float)py;
				for (int i = 0; i < spp; ++i) {
					bool inside;
					if (st.wmask) {
						inside = (__ldg(st.wmask + store_index(pix, i, spp)) >> bit) & 1u;
					} else {
						const float2 o = __ldg(smp.pos + pat * spp + i);
						const float vx = (fpx + o.x) - xcent;
						const float vy = (fpy + o.y) - ycent;
						inside = vx >= -fp.xfwo2 && vy >= -fp.yfwo2 && vx <= fp.xfwo2 && vy <= fp.yfwo2;
					}
					if (!inside) continue;
					const float gw = __ldg(ftab + index + i);
					gTot += gw;
					const long long si = store_index(pix, i, spp);
					if (__ldg(st.b + si).w == 0.0f) continue;
					count++;
					const int id = __ldg(st.aovsrc + si);
					if (id < 0) continue;
					const float* v = g.aov + (st.aov_vertex ? (long long)id : aov_vertex_of(g, id)) * naov;
#pragma unroll
					for (int k = 0; k < AQH_MAX_AOV; ++k)
						if (k < naov) acc[k] += __ldg(v + k) * gw;
				}
			}
		}
		float* o = out + ((long long)(y - fp.crop_y0) * (fp.crop_x1 - fp.crop_x0) + (x - fp.crop_x0)) * naov;
		const float inv = count == 0 ? 0.0f : reciprocal_rounded(gTot);
#pragma unroll
		for (int k = 0; k < AQH_MAX_AOV; ++k)
			if (k < naov) o[k] = count == 0 ? 0.0f : acc[k] * inv;
	}
}


// ExposeBucket (bucketprocessor.cpp:766-806) on one display pixel's channels.
__device__ __forceinline__ void expose(const FrameParams& fp, float c[9]) {
	// ExposeBucket: color = (color * gain) ^ (1 / gamma)
	if (!(fp.gain == 1.0f && fp.gamma == 1.0f)) {
		const float oneovergamma = 1.0f / fp.gamma;
		if (fp.gain != 1.0f) { c[0] *= fp.gain; c[1] *= fp.gain; c[2] *= fp.gain; }
		if (fp.gamma != 1.0f) {
			c[0] = pow_rounded(c[0], oneovergamma);
			c[1] = pow_rounded(c[1], oneovergamma);
			c[2] = pow_rounded(c[2], oneovergamma);
		}
	}
}

// ExposeBucket and the 8-bit display of a frame the filter left unexposed.  A
// pass of its own: with the power inside, the filter kernels lost more than
// this reads and writes (16 samples at 1080p: 618 -> 811 us inlined, 827 us
// called), and here every lane of a warp has a pixel to raise.
__global__ void __launch_bounds__(256)
expose_kernel(FrameParams fp, SamplerDev smp, float* __restrict__ chan, uint8_t* __restrict__ q8) {
	const int w = fp.crop_x1 - fp.crop_x0;
	const long long npix = (long long)w * (fp.crop_y1 - fp.crop_y0);
	const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= npix) return;
	float c[9];
#pragma unroll
	for (int k = 0; k < 9; ++k) c[k] = chan[p * 9 + k];
	expose(fp, c);
	store_pixel(fp, smp, c, chan, q8, fp.crop_x0 + (int)(p % w), fp.crop_y0 + (int)(p / w));
}

// The imager's write-back (bucketprocessor.cpp:712-743): Ci and Oi of each
// display pixel from the imager shader's output (the shading VM runs on the
// host), alpha = the mean of that opacity (no coverage factor), then
// ExposeBucket and the 8-bit display as after the filter.
__global__ void imager_kernel(FrameParams fp, SamplerDev smp, const float* __restrict__ ci_oi,
                              float* __restrict__ chan, uint8_t* __restrict__ q8) {
	const int w = fp.crop_x1 - fp.crop_x0;
	const long long npix = (long long)w * (fp.crop_y1 - fp.crop_y0);
	const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= npix) return;
	float c[9];
#pragma unroll
	for (int k = 0; k < 9; ++k) c[k] = chan[p * 9 + k];
#pragma unroll
	for (int k = 0; k < 6; ++k) c[k] = ci_oi[p * 6 + k];
	c[6] = (c[3] + c[4] + c[5]) / 3.0f;
	expose(fp, c);
	store_pixel(fp, smp, c, chan, q8, fp.crop_x0 + (int)(p % w), fp.crop_y0 + (int)(p / w));
}

__global__ void quantize_u8_kernel(FrameParams fp, SamplerDev smp, const float* __restrict__ chan,
                                   const int* __restrict__ chans, int nchan, uint8_t* __restrict__ out) {
	const long long npix = (long long)(fp.crop_x1 - fp.crop_x0) * (fp.crop_y1 - fp.crop_y0);
	const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= npix) return;
	const double s = smp.dither ? (double)__ldg(smp.dither + p) : 0.0;
	for (int c = 0; c < nchan; ++c) {
		double value = chan[p * 9 + chans[c]];
		if (fp.q_one != 0.0f) {
			value = lround_d(0.0 + value * (double)(fp.q_one - 0.0f) + ((double)fp.q_dither * s));
			value = value < (double)fp.q_min ? (double)fp.q_min : (value > (double)fp.q_max ? (double)fp.q_max : value);
		}
		out[p * nchan + c] = (uint8_t)(int)value;
	}
}

// FormatBucketForDisplay (ddmanager.cpp:1054-1114) for one display request:
// element type T, the request's own quantize settings and dither values.
template <class T>
__global__ void display_kernel(FrameParams fp, QuantizeParams q, const float* __restrict__ dither,
                               const float* __restrict__ chan, const float* __restrict__ aov, int naov,
                               const int* __restrict__ chans, int nchan, T* __restrict__ out) {
	const long long npix = (long long)(fp.crop_x1 - fp.crop_x0) * (fp.crop_y1 - fp.crop_y0);
	const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= npix) return;
	const double s = dither ? (double)__ldg(dither + p) : 0.0;
	for (int c = 0; c < nchan; ++c) {
		const int ch = chans[c];
		double value = ch < 9 ? chan[p * 9 + ch] : aov[p * naov + (ch - 9)];
		if (q.one != 0.0f) {
			value = lround_d((double)q.zero + value * (double)(q.one - q.zero) + ((double)q.dither * s));
			value = value < (double)q.min ? (double)q.min : (value > (double)q.max ? (double)q.max : value);
		}
		T v;
		if constexpr (std::is_floating_point<T>::value) {
			v = (T)value;                                   // PkDspyFloat32
		} else if constexpr (sizeof(T) == 4) {
			// 32-bit integers are clamped to their range first (ddmanager.cpp:1075-1095)
			const double lo = T(-1) < T(0) ? -2147483648.0 : 0.0;
			const double hi = T(-1) < T(0) ? 2147483647.0 : 4294967295.0;
			value = value < lo ? lo : (value > hi ? hi : value);
			v = T(value == value ? (long long)value : 0);
		} else {
			// narrower types: the value is inside the quantize range; outside the
			// type's range the conversion wraps (through a 64-bit integer)
			value = value < -9.0e18 ? -9.0e18 : (value > 9.0e18 ? 9.0e18 : value);
			v = T(value == value ? (long long)value : 0);
		}
		out[p * nchan + c] = v;
	}
}

__global__ void test_invbilinear_kernel(const float* q, const float2* P, int n, float2* uv) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	V3f v[4] = {V3f{q[0], q[1], 0.0f}, V3f{q[2], q[3], 0.0f}, V3f{q[4], q[5], 0.0f}, V3f{q[6], q[7], 0.0f}};
	HitCoeffs h;
	hit_setup(v, 0, h);
	float u, w;
	inv_bilinear(h.ax, h.ay, h.e_x, h.e_y, h.f_x, h.f_y, h.g_x, h.g_y, h.linear, P[i].x, P[i].y, u, w);
	uv[i] = make_float2(u, w);
}

}  // namespace

static void launch_filter_sums(const FrameParams& fp, const SamplerDev& sm, const SampleStore& st, const float* ftab,
                               float* channels, uint8_t* q8, cudaStream_t s) {
	const int w = fp.crop_x1 - fp.crop_x0, h = fp.crop_y1 - fp.crop_y0;
	if (w <= 0 || h <= 0) return;
	const int ntiles = ((w + 15) / 16) * ((h + 15) / 16);
	int dev = 0, nsm = 0;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
	// tiles in flight per SM: by default as many as can be resident (the
	// filter is latency-bound: fewer tiles in flight, whose samples would stay
	// in L2 between the passes, measured slower)
	const int taps = (2 * fp.shiftX + 1) * (2 * fp.shiftY + 1) * fp.spp;
	const int cols = (w + kRollCols - 1) / kRollCols, rows = roll_rows(cols, h, (fp.shiftX == 2 ? 31 : 32) * nsm / 8);
	if (fp.shiftX == fp.shiftY && (fp.shiftX == 1 || fp.shiftX == 2) && taps <= kRollTaps &&
	    !(rows < 4 && fp.spp <= 16) && !(fp.shiftX == 2 && fp.spp == 4) && !filter_tiles_asked(fp)) {
		// 3x3 windows: the rolling window reads each sample three times, not
		// nine, 5x5 five instead of 25.  Runs of fewer than four rows (images
		// below about 400x400) lose that where pixels hold few samples
		// (320x240, 4 samples, 3x3: 12 us on the tile kernel, 15 here; 15
		// samples, 5x5: 127 and 178), and the tile kernel takes them; with more
		// samples they gain here too (480x300, 36 samples, 3x3: 332 us against
		// 129; 211x171, 42 samples, 5x5: 277 against 262).  5x5 windows of 4
		// samples stay there at any size, where the sample count is a constant
		// (1400x1000: 270 us there, 436 here; other counts gain here)
		const dim3 rg(cols, (h + rows - 1) / rows);
		auto go = [&](auto kernel) { kernel<<<rg, kRollThreads, 0, s>>>(fp, sm, st, ftab, channels, q8, rows); };
		if (fp.shiftX == 1) {
			if (st.wmask && fp.spp == 16) go(filter_roll_kernel<16, 1, true>);
			else if (st.wmask) go(filter_roll_kernel<0, 1, true>);
			else if (fp.spp == 64) go(filter_roll_kernel<64, 1, false>);
			else if (fp.spp == 36) go(filter_roll_kernel<36, 1, false>);
			else go(filter_roll_kernel<0, 1, false>);
		} else if (st.wmask) {
			if (fp.spp == 16) go(filter_roll_kernel<16, 2, true>);
			else go(filter_roll_kernel<0, 2, true>);
		} else {
			go(filter_roll_kernel<0, 2, false>);
		}
		return;
	}
	const int per_sm = fp.filter_ctas > 0 ? std::min(fp.filter_ctas, 8) : 8;
	const int grid = std::max(1, std::min(ntiles, nsm * per_sm));
	switch (fp.spp) {
	case 4: filter_kernel<4><<<grid, 256, 0, s>>>(fp, sm, st, ftab, channels, q8); break;
	case 16: filter_kernel<16><<<grid, 256, 0, s>>>(fp, sm, st, ftab, channels, q8); break;
	case 36: filter_kernel<36><<<grid, 256, 0, s>>>(fp, sm, st, ftab, channels, q8); break;
	case 64: filter_kernel<64><<<grid, 256, 0, s>>>(fp, sm, st, ftab, channels, q8); break;
	default: filter_kernel<0><<<grid, 256, 0, s>>>(fp, sm, st, ftab, channels, q8); break;
	}
}

void launch_filter(const FrameParams& fp, const SamplerDev& sm, const SampleStore& st, const float* ftab,
                   float* channels, uint8_t* q8, cudaStream_t s) {
	const bool exposed = !(fp.gain == 1.0f && fp.gamma == 1.0f);
	launch_filter_sums(fp, sm, st, ftab, channels, exposed ? nullptr : q8, s);
	const long long npix = (long long)(fp.crop_x1 - fp.crop_x0) * (fp.crop_y1 - fp.crop_y0);
	if (exposed && npix > 0) expose_kernel<<<(unsigned)((npix + 255) / 256), 256, 0, s>>>(fp, sm, channels, q8);
}

void launch_imager(const FrameParams& fp, const SamplerDev& sm, const float* ci_oi, float* channels, uint8_t* q8,
                   cudaStream_t s) {
	const long long npix = (long long)(fp.crop_x1 - fp.crop_x0) * (fp.crop_y1 - fp.crop_y0);
	if (npix <= 0) return;
	imager_kernel<<<(unsigned)((npix + 255) / 256), 256, 0, s>>>(fp, sm, ci_oi, channels, q8);
}

void launch_filter_aov(const FrameParams& fp, const SamplerDev& sm, const SampleStore& st, const GridsDev& g,
                       const float* ftab, float* aov_channels, cudaStream_t s) {
	const int w = fp.crop_x1 - fp.crop_x0, h = fp.crop_y1 - fp.crop_y0;
	if (w <= 0 || h <= 0 || g.naov <= 0 || !st.aovsrc) return;
	int dev = 0, nsm = 0;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
	if (st.aov_vertex) {
		const long long npix = (long long)fp.sw * fp.sh, n = (long long)store_size(npix, fp.spp);
		aov_vertex_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(g, st.aovsrc, npix, fp.spp);
		const int sh = fp.shiftX;
		if (sh == fp.shiftY && (sh == 1 || sh == 2) && (2 * sh + 1) * (2 * sh + 1) * fp.spp <= kRollTaps) {
			const int cols = (w + kRollThreads - 1) / kRollThreads, rows = roll_rows(cols, h, 3 * nsm);
			const dim3 rg(cols, (h + rows - 1) / rows);
			for (int k0 = 0; k0 < g.naov; k0 += 4) {
				const int na = std::min(4, g.naov - k0);
				auto go = [&](auto kernel) { kernel<<<rg, kRollThreads, 0, s>>>(fp, sm, st, g, ftab, aov_channels, k0, rows); };
				if (sh == 1) {
					if (na == 1) go(filter_aov_roll_kernel<1, 1>);
					else if (na == 2) go(filter_aov_roll_kernel<1, 2>);
					else if (na == 3) go(filter_aov_roll_kernel<1, 3>);
					else go(filter_aov_roll_kernel<1, 4>);
				} else {
					if (na == 1) go(filter_aov_roll_kernel<2, 1>);
					else if (na == 2) go(filter_aov_roll_kernel<2, 2>);
					else if (na == 3) go(filter_aov_roll_kernel<2, 3>);
					else go(filter_aov_roll_kernel<2, 4>);
				}
			}
			return;
		}
	}
	const int ntiles = ((w + 15) / 16) * ((h + 15) / 16);
	const int grid = std::max(1, std::min(ntiles, nsm * 8));
	switch (fp.spp) {
	case 16: filter_aov_kernel<16><<<grid, 256, 0, s>>>(fp, sm, st, g, ftab, aov_channels); break;
	default: filter_aov_kernel<0><<<grid, 256, 0, s>>>(fp, sm, st, g, ftab, aov_channels); break;
	}
}

void launch_quantize_u8(const FrameParams& fp, const SamplerDev& sm, const float* channels, const int* chans,
                        int nchan, uint8_t* out, cudaStream_t s) {
	const long long npix = (long long)(fp.crop_x1 - fp.crop_x0) * (fp.crop_y1 - fp.crop_y0);
	if (npix <= 0) return;
	quantize_u8_kernel<<<(unsigned)((npix + 255) / 256), 256, 0, s>>>(fp, sm, channels, chans, nchan, out);
}

void launch_display(const FrameParams& fp, const QuantizeParams& q, const float* dither, const float* channels,
                    const float* aov_channels, int naov, const int* chans, int nchan, int format, void* out,
                    cudaStream_t s) {
	const long long npix = (long long)(fp.crop_x1 - fp.crop_x0) * (fp.crop_y1 - fp.crop_y0);
	if (npix <= 0) return;
	const unsigned nb = (unsigned)((npix + 255) / 256);
	switch (format) {
	case AQH_DSPY_FLOAT32: display_kernel<float><<<nb, 256, 0, s>>>(fp, q, dither, channels, aov_channels, naov, chans, nchan, (float*)out); break;
	case AQH_DSPY_UNSIGNED32: display_kernel<uint32_t><<<nb, 256, 0, s>>>(fp, q, dither, channels, aov_channels, naov, chans, nchan, (uint32_t*)out); break;
	case AQH_DSPY_SIGNED32: display_kernel<int32_t><<<nb, 256, 0, s>>>(fp, q, dither, channels, aov_channels, naov, chans, nchan, (int32_t*)out); break;
	case AQH_DSPY_UNSIGNED16: display_kernel<uint16_t><<<nb, 256, 0, s>>>(fp, q, dither, channels, aov_channels, naov, chans, nchan, (uint16_t*)out); break;
	case AQH_DSPY_SIGNED16: display_kernel<int16_t><<<nb, 256, 0, s>>>(fp, q, dither, channels, aov_channels, naov, chans, nchan, (int16_t*)out); break;
	case AQH_DSPY_UNSIGNED8: display_kernel<uint8_t><<<nb, 256, 0, s>>>(fp, q, dither, channels, aov_channels, naov, chans, nchan, (uint8_t*)out); break;
	default: display_kernel<int8_t><<<nb, 256, 0, s>>>(fp, q, dither, channels, aov_channels, naov, chans, nchan, (int8_t*)out); break;
	}
}

void launch_test_invbilinear(const float* quad8, const float2* P, int n, float2* uv, cudaStream_t s) {
	if (n <= 0) return;
	test_invbilinear_kernel<<<(n + 127) / 128, 128, 0, s>>>(quad8, P, n, uv);
}

}  // namespace aqh
