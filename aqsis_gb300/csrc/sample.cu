// sample.cu -- the sampling stage: subpixel hit tests with depth and opacity
// compositing into the pixel sample store.
//
// Replaces CqBucketProcessor::RenderMicroPoly / RenderMPG_Static /
// RenderMPG_MBOrDof / StoreSample (libs/core/bucketprocessor.cpp:1067-1569),
// CqMicroPolygon::Sample / fContains (micropolygon.cpp:1295-1660, 1768-1914)
// and CqImagePixel::Combine (imagepixel.cpp:144-332).
//
// Layout.  One CTA (16 warps) owns a tile of the sample region holding at
// most 4096 samples (16x16 pixels at 16 samples per pixel).  It walks its
// super-tile's grid list and expands the grids touching the tile into
// micropolygons, a round of some hundred at a time:
//   phase A: one micropolygon per thread tests bound, crop cull and a
//     tile-wide early-z; survivors are compacted in list order, then every
//     thread builds one shared-memory record (vertex order, edge and
//     inverse-bilinear coefficients, pixel and sub-sample ranges);
//   phase B: the hit tests, in one of these forms:
//     sample_near_kernel: opaque frames, grids near to far; pixels whose
//       result could depend on the order go to a list;
//     sample_opaque_kernel: in insertion order, (micropolygon, sample) pairs
//       in parallel; that list, frames without a depth order, and (MIXED)
//       transparent frames with occluders;
//     sample_frag_kernel: frames in which every hit is a fragment;
//     sample_static_kernel: CSG solids, midpoint depths and samples that may
//       not be culled: a warp takes 32 samples, one per lane, and walks the
//       union of their pixels' candidate masks in insertion order, each lane
//       running the reference's per-sample sequence (sub-sample range,
//       inclusive bound test, early-z, edge tests, inverse bilinear, depth,
//       store).
// Each section says why its form keeps the reference's order-dependent early-z
// and its "first of equal depths wins" rule.  Colours are resolved once per
// sample at the end (the reference interpolates them at store time; the values
// are the same because they depend only on the winning micropolygon and (u,v)).
#include "aqh_internal.h"
#include "hider_device.cuh"
#include "sample_common.cuh"

namespace aqh {

namespace {

constexpr int kThreadsS = 512;                   // 16 warps
constexpr int kWarpsS = kThreadsS / 32;
constexpr int kSlotsS = 256;                     // records per pass
constexpr int kWordsS = kSlotsS / 32;
constexpr int kTilePixMax = 256;
constexpr int kTileSampMax = 4096;

// Shared-memory record of one candidate micropolygon (static path).
struct RecS {
	float bminx, bmaxx, bminy, bmaxy, bminz;
	int px0, px1, py0, py1;        // pixels RenderMPG_Static visits: [floor(bmin), lceil(bmax))
	int im, em, in_, en;           // sub-sample starts / ends on the first / last pixel
	float ym[4], xm[4], ex[4], ey[4];
	float ax, ay, e_x, e_y, f_x, f_y, g_x, g_y;
	float z[4];
	int id;                        // global micropolygon id
	int bits;                      // 1 linear, 2 occluding store
};  // 43 words: an odd stride spreads neighbouring records over the banks

// RecS::bits; the grid index sits from bit 6 up.  kRecCsg: a CSG solid's
// micropolygon, never occlusion-cullable; kRecTrim: marked trimmed.
constexpr int kRecLinear = 1, kRecOccluding = 2, kRecTriangular = 4, kRecLod = 8, kRecCsg = 16, kRecTrim = 32;
constexpr int kRecGridShift = 6;

// The tests after fContains that can still reject a static hit at (x, y),
// (u, v): the trim curves of a micropolygon marked trimmed, then the split
// line of a triangular grid (key 0).
__device__ __forceinline__ bool rec_keeps(const GridsDev& g, const BinBuffers& bb, int bits, int id, float x, float y,
                                          float u, float v) {
	if ((bits & kRecTrim) && trim_rejects(g, id, bits >> kRecGridShift, u, v)) return false;
	return !(bits & kRecTriangular) || triangle_keeps(__ldg(bb.tri + (size_t)(bits >> kRecGridShift) * kMaxKeys), x, y);
}

struct SmemS {
	RecS rec[kSlotsS];
	uint32_t mask[kTilePixMax][kWordsS];  // candidate bits per tile pixel
	int2 pend[kSlotsS];                   // (grid, micropolygon) of the staged candidates
	int qgrid[kThreadsS];                 // grids of the current list chunk that touch the tile
	int qcum[kThreadsS + 1];              // running micropolygon counts of those grids
	int qsub[kThreadsS];                  // their micropolygon sub-rectangles (see stage_candidates)
	int warp_tot[32];
	float warp_max[32];
	int first_reject;
	int qn;
	float pixmax[kTilePixMax];            // largest occluding depth over each pixel's samples
	float blkmax[16];                     // ... over each 4x4-pixel block of the tile
	float soz[kTileSampMax];              // occlZ per tile sample
	int swin[kTileSampMax];               // occluding micropolygon per tile sample (-1 none)
};

// Running maximum of occluding depths for the early-z culls.  A NaN depth
// never passes `bminz > occlZ`, so it must never cull: it counts as +inf.
__device__ __forceinline__ float max_depth(float mx, float d) { return (d != d) ? INFINITY : fmaxf(mx, d); }

__device__ __forceinline__ float warp_max_f(float v) {
	v = (v != v) ? INFINITY : v;
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
	return v;
}

// Record of micropolygon m of grid gi: bound (CalculateBound), vertex order
// (ComputeVertexOrder), point-in-polygon and inverse-bilinear coefficients
// (cachePointInPolyTest), opacity (CacheOutputInterpCoeffs*), and the pixel
// and sub-sample ranges RenderMPG_Static walks.
__device__ __forceinline__ void build_record(const FrameParams& fp, const GridsDev& g, int gi, int m, RecS& rec) {
	const int cu = __ldg(g.cu + gi);
	const long long pb = __ldg(g.pbase + gi);
	const int gflags = __ldg(g.flags + gi);
	const int iv = m / cu, iu = m - iv * cu;
	const int index = iv * (cu + 1) + iu;
	V3f v[4];
	v[0] = ld3(g.P, pb + index);
	v[1] = ld3(g.P, pb + index + 1);
	v[2] = ld3(g.P, pb + index + cu + 1);
	v[3] = ld3(g.P, pb + index + cu + 2);
	const float bminx = amin(amin(amin(v[0].x, v[1].x), v[3].x), v[2].x);
	const float bminy = amin(amin(amin(v[0].y, v[1].y), v[3].y), v[2].y);
	const float bminz = amin(amin(amin(v[0].z, v[1].z), v[3].z), v[2].z);
	const float bmaxx = amax(amax(amax(v[0].x, v[1].x), v[3].x), v[2].x);
	const float bmaxy = amax(amax(amax(v[0].y, v[1].y), v[3].y), v[2].y);
	HitCoeffs h;
	hit_setup(v, vertex_order(v), h);
	rec.bminx = bminx; rec.bmaxx = bmaxx; rec.bminy = bminy; rec.bmaxy = bmaxy; rec.bminz = bminz;
	// bucketprocessor.cpp:1119-1138 (the clip to the sample region does not
	// change the range of any pixel inside it)
	const int sX = (int)floorf(bminx), eX = lceil_f(bmaxx);
	const int sY = (int)floorf(bminy), eY = lceil_f(bmaxy);
	rec.px0 = sX; rec.px1 = eX; rec.py0 = sY; rec.py1 = eY;
	rec.im = (int)floorf((bminx - (float)sX) * (float)fp.xs);
	rec.in_ = (int)floorf((bminy - (float)sY) * (float)fp.ys);
	rec.em = lceil_f((bmaxx - (float)(eX - 1)) * (float)fp.xs);
	rec.en = lceil_f((bmaxy - (float)(eY - 1)) * (float)fp.ys);
#pragma unroll
	for (int k = 0; k < 4; ++k) {
		rec.ym[k] = h.ym[k]; rec.xm[k] = h.xm[k]; rec.ex[k] = h.ex[k]; rec.ey[k] = h.ey[k];
		rec.z[k] = h.z[k];
	}
	rec.ax = h.ax; rec.ay = h.ay; rec.e_x = h.e_x; rec.e_y = h.e_y;
	rec.f_x = h.f_x; rec.f_y = h.f_y; rec.g_x = h.g_x; rec.g_y = h.g_y;
	rec.id = (int)(__ldg(g.mpbase + gi) + m);
	// SqMpgSampleInfo::isOpaque (micropolygon.cpp:1477-1529)
	bool opaque = true;
	const bool smooth = (gflags & 1) != 0;
	if (!(gflags & 8) && g.Oi) {
		const long long cb = __ldg(g.cbase + gi);
		const float4 o0 = ld_colour(g, g.Oi, cb + index);
		opaque = o0.x >= 1.0f && o0.y >= 1.0f && o0.z >= 1.0f;
		if (smooth) {
			const float4 o1 = ld_colour(g, g.Oi, cb + index + 1);
			const float4 o2 = ld_colour(g, g.Oi, cb + index + cu + 1);
			const float4 o3 = ld_colour(g, g.Oi, cb + index + cu + 2);
			opaque = opaque && (o1.x >= 1.0f && o1.y >= 1.0f && o1.z >= 1.0f) &&
			         (o2.x >= 1.0f && o2.y >= 1.0f && o2.z >= 1.0f) && (o3.x >= 1.0f && o3.y >= 1.0f && o3.z >= 1.0f);
		}
	}
	int bits = h.linear ? kRecLinear : 0;
	if (opaque || (gflags & 4)) bits |= kRecOccluding;
	if (gflags & 16) bits |= kRecTriangular;
	if (lod_active(fp, g, gi)) bits |= kRecLod;
	if (csg_grid(g, gi)) bits = (bits & ~kRecOccluding) | kRecCsg;
	if (g.trim.nsets > 0 && __ldg(g.trim.mark + rec.id)) bits |= kRecTrim;
	bits |= gi << kRecGridShift;
	rec.bits = bits;
}

// Final value of one sample: the occluding hit's colour at its (u,v), or the
// Combine of its transparent fragments; written to the sample store.
template <bool TRANSP>
__device__ __forceinline__ bool resolve_sample(const FrameParams& fp, const GridsDev& g, const FragPool& pool,
                                               const SampleStore& st, long long sidx, long long aidx, float x,
                                               float y, float oz, int w, int head) {
	float occl[7] = {0, 0, 0, 0, 0, 0, 0};
	int occl_flags = 0;
	if (w >= 0) {
		// recompute (u,v) of the winner exactly as when it was stored
		const int wg = grid_of(g, w);
		const int cu = __ldg(g.cu + wg);
		const int m = w - (int)__ldg(g.mpbase + wg);
		const int iv = m / cu, iu = m - iv * cu;
		const int index = iv * (cu + 1) + iu;
		const long long pb = __ldg(g.pbase + wg);
		V3f v[4] = {ld3(g.P, pb + index), ld3(g.P, pb + index + 1), ld3(g.P, pb + index + cu + 1),
		            ld3(g.P, pb + index + cu + 2)};
		HitCoeffs h;
		hit_setup(v, vertex_order(v), h);
		float u, vv;
		inv_bilinear(h.ax, h.ay, h.e_x, h.e_y, h.f_x, h.f_y, h.g_x, h.g_y, h.linear, x, y, u, vv);
		hit_colour(g, wg, m, u, vv, occl, occl_flags);
		occl[6] = (TRANSP && fp.midpoint_store) ? st.hitz[sidx] : oz;
	}
	int nf = 0;
	bool valid = w >= 0;
	int src = w;
	if (TRANSP && head >= 0) {
		bool emptied = false;
		nf = combine_fragments(fp, g, pool, head, w >= 0, oz, occl, occl_flags, w, src, emptied);
		valid = !emptied;
	}
	if (nf == 0 && valid) {
		// imagepixel.cpp:303-330: opaque matte hits become transparent black;
		// the midpoint depth filter averages with occlZ
		if (occl_flags & 1)
			for (int q = 0; q < 6; ++q) occl[q] = 0.0f;
		if (fp.depth_filter == 1) occl[6] = (float)(0.5 * ((double)occl[6] + (double)oz));
	}
	st.a[aidx] = make_float4(occl[0], occl[1], occl[2], occl[6]);
	st.b[aidx] = make_float4(occl[3], occl[4], occl[5], valid ? 1.0f : 0.0f);
	if (st.aovsrc) st.aovsrc[aidx] = valid ? src : -1;
	if (st.winner) st.winner[sidx] = w;
	if (st.occlz) st.occlz[sidx] = oz;
	if (st.nfrag) st.nfrag[sidx] = nf;
	return valid;
}

// Micropolygon m of grid gid has a bounded depth slack (bin.cu).
__device__ __forceinline__ bool mp_regular(const BinBuffers& bb, int gid, int m) {
	return __ldg(bb.grid_nirr + gid) >= 0 &&
	       !((__ldg(bb.irregular + (long long)gid * kIrrWords + (m >> 5)) >> (m & 31)) & 1u);
}

// Phase A: stream the super-tile's grid list from the cursor (lp, r0,
// qtotal) and append the micropolygons that are candidates of the tile to
// sm.pend, in insertion order, until kSlots are staged or the list ends
// (returns true then).  One micropolygon per thread tests bound, crop cull
// and early-z against the largest occluding depth of every pixel it visits;
// whole grids behind every sample of the 4x4-pixel blocks they overlap are
// skipped.  Survivors are compacted with block scans, so the staged order is
// the insertion order.
// MAY_CSG: the calling kernel can see CSG grids (the opaque kernel never
// does: frames with solids always render with fragments).  NEAR: the list near
// to far; a regular micropolygon is behind a depth only with its slack, and of
// a grid behind every depth the irregular ones are still staged.
template <int kSlots, bool MAY_CSG = true, bool NEAR = false, class Smem>
__device__ __forceinline__ bool stage_candidates(const FrameParams& fp, const GridsDev& g, const BinBuffers& bb,
                                                 Smem& sm, int tpx0, int tpy0, int tpx1, int tpy1, int lend, int& lp,
                                                 int& r0, int& qtotal, int& npend) {
	const int t = threadIdx.x;
	const int cullable = fp.cullable;
	while (npend < kSlots) {
		if (r0 >= qtotal) {
			if (lp >= lend) return true;
			// grids of the next list chunk that touch the tile, in order
			const int li = lp + t;
			int gid = -1, nmp = 0, sub = -1;  // sub: first column, first row, width; -1 = whole grid
			bool f = false, few = false;  // few: only the irregular ones
			if (li < lend) {
				gid = NEAR ? bb.st_sorted[li] : bb.st_list[li];
				const int4 rc = bb.grid_rect[gid];
				f = rc.x < rc.y && rc.x < tpx1 && rc.y > tpx0 && rc.z < tpy1 && rc.w > tpy0;
				if (f && cullable && !(MAY_CSG && csg_grid(g, gid))) {
					// whole grid behind every sample of the 4x4-pixel blocks it overlaps
					const int bx0 = (max(rc.x, tpx0) - tpx0) >> 2, bx1 = (min(rc.y, tpx1) - 1 - tpx0) >> 2;
					const int by0 = (max(rc.z, tpy0) - tpy0) >> 2, by1 = (min(rc.w, tpy1) - 1 - tpy0) >> 2;
					const int nbx = (fp.tile_w + 3) >> 2;
					float mx = -FLT_MAX;
					for (int by = by0; by <= by1; ++by)
						for (int bx = bx0; bx <= bx1; ++bx) mx = fmaxf(mx, sm.blkmax[by * nbx + bx]);
					if (NEAR) {
						const int nirr = __ldg(bb.grid_nirr + gid);
						if (nirr >= 0 && __ldg(bb.grid_minz + gid) - __ldg(bb.grid_slack + gid) > mx) {
							f = nirr > 0;
							few = f;
							nmp = nirr;
							sub = -2;
						}
					} else if (__ldg(bb.grid_minz + gid) > mx) {
						f = false;
					}
				}
				if (f && !few) {
					const int cu = __ldg(g.cu + gid), cv = __ldg(g.cv + gid);
					nmp = cu * cv;
					if (bb.strips && __ldg(bb.strips + (long long)gid * 64 + 63)) {
						// the columns and rows of micropolygons that can meet the tile
						const uint32_t* S = bb.strips + (long long)gid * 64;
						int iu0 = 64, iu1 = -1, iv0 = 64, iv1 = -1;
						for (int k = 0; k < cu; ++k) {
							const uint32_t w = __ldg(S + k);
							if ((int)(int16_t)(w & 0xffffu) < tpx1 && (int)(int16_t)(w >> 16) > tpx0) {
								iu0 = min(iu0, k);
								iu1 = k;
							}
						}
						for (int k = 0; k < cv; ++k) {
							const uint32_t w = __ldg(S + 32 + k);
							if ((int)(int16_t)(w & 0xffffu) < tpy1 && (int)(int16_t)(w >> 16) > tpy0) {
								iv0 = min(iv0, k);
								iv1 = k;
							}
						}
						if (iu1 < 0 || iv1 < 0) {
							f = false;
							nmp = 0;
						} else {
							nmp = (iu1 - iu0 + 1) * (iv1 - iv0 + 1);
							sub = iu0 | (iv0 << 8) | ((iu1 - iu0 + 1) << 16);
						}
					}
				}
			}
			int total, sum;
			const int pos = block_excl_scan(sm.warp_tot, f, total);
			__syncthreads();
			// running micropolygon counts of the queued grids
			const int pre = block_excl_sum(sm.warp_tot, nmp, sum);
			if (f) {
				sm.qgrid[pos] = gid;
				sm.qcum[pos] = pre;
				sm.qsub[pos] = sub;
			}
			if (t == 0) {
				sm.qcum[total] = sum;
				sm.qn = total;
			}
			__syncthreads();
			qtotal = sm.qcum[sm.qn];
			r0 = 0;
			lp += kThreadsS;
			continue;
		}
		// one micropolygon of the stream per thread: is it a candidate of this
		// tile?  Its grid: lane 0 searches for the warp's first position, the
		// other lanes step on from there.
		const int p = r0 + t;
		int lo0 = 0;
		if ((t & 31) == 0 && p < qtotal) {
			int lo = 0, hi = sm.qn - 1;
			while (lo < hi) {
				const int mid = (lo + hi + 1) >> 1;
				if (sm.qcum[mid] <= p) lo = mid; else hi = mid - 1;
			}
			lo0 = lo;
		}
		lo0 = __shfl_sync(0xffffffffu, lo0, 0);
		bool active = false;
		int gid = 0, m = 0;
		if (p < qtotal) {
			const int lo = advance_item(sm.qcum, sm.qn, lo0, p);
			gid = sm.qgrid[lo];
			m = p - sm.qcum[lo];
			const int cu = __ldg(g.cu + gid);
			const int sub = sm.qsub[lo];
			if (sub >= 0) {
				const int w = sub >> 16, jv = m / w;
				m = ((sub >> 8) & 0xff) * cu + jv * cu + (sub & 0xff) + (m - jv * w);
			} else if (NEAR && sub == -2) {
				// the m-th irregular micropolygon
				const uint32_t* irr = bb.irregular + (long long)gid * kIrrWords;
				int wd = 0;
				uint32_t w = __ldg(irr);
				while (m >= __popc(w)) {
					m -= __popc(w);
					w = __ldg(irr + ++wd);
				}
				m = wd * 32 + (int)__fns(w, 0, m + 1);
			}
			const long long pb = __ldg(g.pbase + gid);
			const int iv = m / cu, iu = m - iv * cu;
			const int index = iv * (cu + 1) + iu;
			const V3f a = ld3(g.P, pb + index), b = ld3(g.P, pb + index + 1);
			const V3f c = ld3(g.P, pb + index + cu + 1), d = ld3(g.P, pb + index + cu + 2);
			const float bminx = amin(amin(amin(a.x, b.x), d.x), c.x);
			const float bminy = amin(amin(amin(a.y, b.y), d.y), c.y);
			const float bminz = amin(amin(amin(a.z, b.z), d.z), c.z);
			const float bmaxx = amax(amax(amax(a.x, b.x), d.x), c.x);
			const float bmaxy = amax(amax(amax(a.y, b.y), d.y), c.y);
			const bool culled = g.culled && g.culled[__ldg(g.mpbase + gid) + m];
			// AddMPG crop cull (imagebuffer.cpp:533-539)
			const bool cropped =
			    bmaxx < fp.cull_x0 || bmaxy < fp.cull_y0 || bminx > fp.cull_x1 || bminy > fp.cull_y1;
			const int sX = max((int)floorf(bminx), tpx0), eX = min(lceil_f(bmaxx), tpx1);
			const int sY = max((int)floorf(bminy), tpy0), eY = min(lceil_f(bmaxy), tpy1);
			active = !culled && !cropped && sX < eX && sY < eY;
			if (active && cullable && !(MAY_CSG && csg_grid(g, gid))) {
				// early-z for every pixel it visits: behind all their samples' occluding depths
				float mx = -FLT_MAX;
				for (int yy = sY; yy < eY; ++yy)
					for (int xx = sX; xx < eX; ++xx) mx = fmaxf(mx, sm.pixmax[(yy - tpy0) * fp.tile_w + (xx - tpx0)]);
				if (NEAR) {
					if (bminz - __ldg(bb.grid_slack + gid) > mx && mp_regular(bb, gid, m)) active = false;
				} else if (bminz > mx) {
					active = false;
				}
			}
		}
		int total;
		const int rank = block_excl_scan(sm.warp_tot, active, total);
		const int navail = kSlots - npend;
		if (t == 0) sm.first_reject = kThreadsS;
		__syncthreads();
		if (active && rank == navail) sm.first_reject = t;
		if (active && rank < navail) sm.pend[npend + rank] = make_int2(gid, m);
		__syncthreads();
		const int consumed = (total > navail) ? sm.first_reject : min(kThreadsS, qtotal - r0);
		npend += min(total, navail);
		r0 += consumed;
	}
	return false;
}

// PERSIST: a fixed grid of CTAs pulls tiles from a device work queue
// (`queue[0]` counts tiles handed out, `order` lists tiles costliest first);
// otherwise one CTA per tile.
template <bool TRANSP, bool PERSIST>
__global__ void __launch_bounds__(kThreadsS, 2)
sample_static_kernel(FrameParams fp, GridsDev g, SamplerDev smp, BinBuffers bb, SampleStore st, FragPool pool,
                     int* queue, const int* order) {
	// a fragment-only frame without occluders is rendered by sample_frag_kernel
	if (TRANSP && fp.frag_only && !(fp.cullable && *pool.occluders)) return;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	SmemS& sm = *reinterpret_cast<SmemS*>(smem_raw);
	int32_t* fhead = reinterpret_cast<int32_t*>(smem_raw + sizeof(SmemS));  // TRANSP: fragment lists
	__shared__ int next_tile;
	const int ntiles = fp.ntx * fp.nty;
	for (int job = 0;; ++job) {
	int tile;
	if (PERSIST) {
		__syncthreads();
		if (threadIdx.x == 0) next_tile = atomicAdd(queue, 1);
		__syncthreads();
		tile = next_tile;
		if (tile >= ntiles) break;
		if (order) tile = order[tile];
	} else {
		if (job > 0) break;
		tile = blockIdx.x;
	}
	const int tx = tile % fp.ntx, ty = tile / fp.ntx;
	const int tpx0 = fp.sx0 + tx * fp.tile_w, tpy0 = fp.sy0 + ty * fp.tile_h;
	const int tpx1 = min(tpx0 + fp.tile_w, fp.sx0 + fp.sw), tpy1 = min(tpy0 + fp.tile_h, fp.sy0 + fp.sh);
	const int st_idx = (ty / fp.st_tiles) * fp.nstx + (tx / fp.st_tiles);
	const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
	const int spp = fp.spp;
	const int tpix = fp.tile_w * fp.tile_h;
	const int tsamp = tpix * spp;
	const int ngroups = (tsamp + 31) >> 5;
	const int cullable = fp.cullable;

	for (int i = t; i < tsamp; i += kThreadsS) {
		sm.soz[i] = FLT_MAX;
		sm.swin[i] = -1;
		if (TRANSP) fhead[i] = -1;
	}
	for (int i = t; i < kTilePixMax * kWordsS; i += kThreadsS) (&sm.mask[0][0])[i] = 0u;
	for (int i = t; i < kTilePixMax; i += kThreadsS) sm.pixmax[i] = FLT_MAX;
	if (t < 16) sm.blkmax[t] = FLT_MAX;
	if (t == 0) {
		sm.qn = 0;
		sm.qcum[0] = 0;
	}
	__syncthreads();

	const int lbeg = bb.st_offset[st_idx * bb.nranges];
	const int lend = (int)min((long long)bb.st_offset[(st_idx + 1) * bb.nranges], (long long)bb.list_capacity);

	// Stream cursor (uniform over the block): next list chunk, position in
	// the micropolygon stream of the queued grids.
	int lp = lbeg, r0 = 0, qtotal = 0;
	int npend = 0;
	for (;;) {
		// ---- phase A ----
		const bool exhausted =
		    stage_candidates<kSlotsS>(fp, g, bb, sm, tpx0, tpy0, tpx1, tpy1, lend, lp, r0, qtotal, npend);
		if (npend == 0) break;

		// ---- build the staged records with every thread busy ----
		for (int slot = t; slot < npend; slot += kThreadsS) {
			const int2 e = sm.pend[slot];
			RecS& rec = sm.rec[slot];
			build_record(fp, g, e.x, e.y, rec);
			const int sX = max(rec.px0, tpx0), eX = min(rec.px1, tpx1);
			const int sY = max(rec.py0, tpy0), eY = min(rec.py1, tpy1);
			const uint32_t bit = 1u << (slot & 31);
			const int wd = slot >> 5;
			for (int yy = sY; yy < eY; ++yy)
				for (int xx = sX; xx < eX; ++xx)
					atomicOr(&sm.mask[(yy - tpy0) * fp.tile_w + (xx - tpx0)][wd], bit);
		}
		__syncthreads();

		// ---- phase B: a warp walks 32 samples' candidates in insertion order ----
		float wmax = -FLT_MAX;
		for (int gq = warp; gq < ngroups; gq += kWarpsS) {
			const int s = gq * 32 + lane;
			const int pl = s / spp;
			const int si = s - pl * spp;
			const int lx = pl % fp.tile_w, ly = pl / fp.tile_w;
			const int px = tpx0 + lx, py = tpy0 + ly;
			const bool valid = s < tsamp && px < tpx1 && py < tpy1;
			const int sn = si / fp.xs, smm = si - sn * fp.xs;
			float x = 0.0f, y = 0.0f, oz = -FLT_MAX;
			int w = -1, fh = -1;
			if (valid) {
				const long long pix = (long long)(py - fp.sy0) * fp.sw + (px - fp.sx0);
				const long long pat = smp.pos_index ? (long long)__ldg(smp.pos_index + pix) : pix;
				const float2 o = __ldg(smp.pos + pat * spp + si);
				x = (float)px + o.x;  // CqImagePixel::setSamples: offset + positions[i]
				y = (float)py + o.y;
				oz = sm.soz[s];
				w = sm.swin[s];
				if (TRANSP) fh = fhead[s];
			}
			float gmax = warp_max_f(oz);
#pragma unroll 1
			for (int wd = 0; wd < kWordsS; ++wd) {
				const uint32_t mine = sm.mask[valid ? pl : 0][wd];  // index stays in bounds for idle lanes
				uint32_t bits = __reduce_or_sync(0xffffffffu, valid ? mine : 0u);
				while (bits) {
					const int b = __ffs(bits) - 1;
					bits &= bits - 1u;
					const RecS& r = sm.rec[wd * 32 + b];
					const bool rcull = cullable && !(r.bits & kRecCsg);  // CSG: never occlusion-culled
					if (rcull && r.bminz > gmax) continue;  // hidden from all 32 samples
					bool ok = valid && px >= r.px0 && px < r.px1 && py >= r.py0 && py < r.py1;
					if (ok) {
						const int m_lo = (px == r.px0) ? r.im : 0;
						const int m_hi = (px == r.px1 - 1) ? r.em : fp.xs;
						const int n_lo = (py == r.py0) ? r.in_ : 0;
						const int n_hi = (py == r.py1 - 1) ? r.en : fp.ys;
						ok = smm >= m_lo && smm < m_hi && sn >= n_lo && sn < n_hi;
					}
					// CqBound::Contains2D (bound.h:144-151) and early-z (bucketprocessor.cpp:1179)
					ok = ok && !((x < r.bminx || x > r.bmaxx) || (y < r.bminy || y > r.bmaxy));
					ok = ok && !(rcull && r.bminz > oz);
					ok = ok && !((r.bits & kRecLod) && lod_rejects(fp, g, smp, r.bits >> kRecGridShift, px, py,
					                                               sn * fp.xs + smm));
					ok = ok && edges_inside(r.ym, r.xm, r.ex, r.ey, x, y);
					bool stored = false;
					if (ok) {
						float u, v;
						inv_bilinear(r.ax, r.ay, r.e_x, r.e_y, r.f_x, r.f_y, r.g_x, r.g_y,
						             (r.bits & kRecLinear) != 0, x, y, u, v);
						const float D = bilerp1(r.z[0], r.z[1], r.z[2], r.z[3], u, v);
						// StoreSample (bucketprocessor.cpp:1471-1569) for a hit the split line keeps
						if (rec_keeps(g, bb, r.bits, r.id, x, y, u, v) && !(rcull && oz <= D)) {
							if ((r.bits & kRecOccluding) && rcull) {
								if (TRANSP && fp.midpoint_store) {
									// midpoint filter with a z display (bucketprocessor.cpp:1502-1530):
									// occlZ follows the second-nearest opaque depth, the hit the nearest
									const long long hx =
									    ((long long)(py - fp.sy0) * fp.sw + (px - fp.sx0)) * spp + si;
									const float hp = (w >= 0) ? st.hitz[hx] : FLT_MAX;
									if (hp < D) {
										oz = D;
									} else {
										oz = hp;
										st.hitz[hx] = D;
										w = r.id;
									}
								} else {
									oz = D;
									w = r.id;
								}
								stored = true;
							} else if (TRANSP) {
								// append a fragment {depth, id, u, v}; lists are newest-first
								const unsigned act = __activemask();
								const int leader = __ffs(act) - 1;
								const int rank = __popc(act & ((1u << lane) - 1u));
								unsigned long long base = 0;
								if (lane == leader) base = atomicAdd(pool.count, (unsigned long long)__popc(act));
								base = __shfl_sync(act, base, leader);
								const long long idx = (long long)base + rank;
								if (idx < pool.capacity) {
									pool.frag[idx] = make_float4(D, __int_as_float(r.id), u, v);
									pool.next[idx] = fh;
									fh = (int)idx;
								} else {
									atomicOr(pool.overflow, 1);
								}
							}
						}
					}
					if (__any_sync(0xffffffffu, stored)) gmax = warp_max_f(oz);
				}
			}
			if (valid) {
				sm.soz[s] = oz;
				sm.swin[s] = w;
				if (TRANSP) fhead[s] = fh;
			}
			wmax = fmaxf(wmax, gmax);
		}
		(void)wmax;
		// largest occluding depth per pixel and per 4x4 block, then clear the masks
		__syncthreads();
		for (int pp = t; pp < tpix; pp += kThreadsS) {
			float mx = -FLT_MAX;
			for (int k = 0; k < spp; ++k) mx = max_depth(mx, sm.soz[pp * spp + k]);
			sm.pixmax[pp] = mx;
		}
		for (int i = t; i < kTilePixMax * kWordsS; i += kThreadsS) (&sm.mask[0][0])[i] = 0u;
		__syncthreads();
		if (t < 16) {
			const int nbx = (fp.tile_w + 3) >> 2;
			const int bx = t % nbx, by = t / nbx;
			float mx = -FLT_MAX;
			if (by * 4 < fp.tile_h)
				for (int yy = by * 4; yy < min(by * 4 + 4, fp.tile_h); ++yy)
					for (int xx = bx * 4; xx < min(bx * 4 + 4, fp.tile_w); ++xx) mx = fmaxf(mx, sm.pixmax[yy * fp.tile_w + xx]);
			sm.blkmax[t] = mx;
		}
		__syncthreads();
		npend = 0;
		if (exhausted) break;
	}

	// ---- resolve: colours of the occluding hits, Combine of fragment lists ----
	// (consecutive threads take the samples of one pixel, whose fragments the
	// same warp allocated together)
	for (int s = t; s < tsamp; s += kThreadsS) {
		const int pl = s / spp;
		const int si = s - pl * spp;
		const int px = tpx0 + pl % fp.tile_w, py = tpy0 + pl / fp.tile_w;
		if (px >= tpx1 || py >= tpy1) continue;
		const long long pix = (long long)(py - fp.sy0) * fp.sw + (px - fp.sx0);
		const long long pat = smp.pos_index ? (long long)__ldg(smp.pos_index + pix) : pix;
		const float2 o = __ldg(smp.pos + pat * spp + si);
		const bool has = resolve_sample<TRANSP>(fp, g, pool, st, pix * spp + si, store_index(pix, si, spp), (float)px + o.x,
		                                        (float)py + o.y, sm.soz[s], sm.swin[s], TRANSP ? fhead[s] : -1);
		if (st.wmask) st.wmask[store_index(pix, si, spp)] =
		    window_word(fp, px, py, (float)px + o.x, (float)py + o.y, has);
	}
	}  // tile loop
}


// ---- opaque frames: parallel hit tests with an ordered fallback ----------
//
// When every micropolygon is opaque, StoreSample's early-z and store rule
// (bucketprocessor.cpp:1179, 1475: skip if bound.min.z > occlZ, keep the hit
// only if D < occlZ) reduce, for every hit whose depth D is not below its own
// bound's minimum z, to "occlZ = min(occlZ, D), first of equal depths wins":
// such a hit skipped by early-z has D >= min.z > occlZ and would not have
// been kept anyway.  So the winner of a sample is the least (D, insertion
// order) over those hits, which does not depend on the order in which they
// are visited: (candidate, sample) pairs are tested in parallel and folded
// with a 64-bit shared-memory atomicMin on (ordered depth bits, id + 1).
// A hit with D below its bound's minimum (rounding or Newton error), a NaN
// or a zero depth (the signs of zero compare equal) may behave differently
// in order, so the sample is flagged and replayed in insertion order over
// the round's candidates from its state at the start of the round.  A
// sample whose occlZ becomes NaN or zero stays on the ordered replay for
// the rest of the tile.  Early-z in the parallel pass tests the depth at the
// start of the round, which is never below the depth the ordered sequence
// would see, so it only skips what the reference skips.
//
// Frames that mix opaque and transparent micropolygons (MIXED) run each
// round's tests in two passes: the occluding candidates as above, then the
// transparent ones.  The reference keeps a transparent hit when !(b > z) and
// !(z <= D), z the occlZ at its place in insertion order, which only occluding
// hits move: z lies between the round's start (prev) and, of a sample that no
// occluding hit flagged, the round's end (key).  Where the two bounds decide
// alike the hit is a fragment or not; where they differ (an occluding
// candidate of the same round covers the sample) it is none if the nearest
// occluder comes before it (ids ascend in insertion order, and then z is at
// most key's depth).  Else the lane takes z from the occluding candidates
// before the hit's own, found in the pixel's candidate mask: the least of prev
// and their hits' depths.  Those with b above prev are left out (the reference
// skips them, and their hits can round to below prev); of the others an
// unflagged sample has no hit below b, so one that early-z skips lies above z
// and does not change the least.  Flagged samples replay both kinds in order.
// Fragments go to the pool in any order (Combine sorts them), and Combine runs
// as its own kernel. The ordered kernel these frames took before (a warp walks
// the union of 32 samples' candidates one after another, then combines with
// little L1 left) took 4.56 ms of a 1280x720 frame of 16 samples, 2.5 opaque
// and 0.8 transparent layers, against 1.97 ms here and 0.95 ms for Combine.
constexpr int kSlotsO = 192;
constexpr int kSlotsMix = 160;  // fewer: the candidate masks share the same shared memory

// Division of k < 2^16 by 1 <= d < 2^16 with a multiply: m = ceil(2^32 / d)
// makes floor(k * m / 2^32) exact (the error k * (m - 2^32/d) / 2^32 < 2^-16 <
// 1/d); d = 1 has no 32-bit m and is passed through.
__device__ __forceinline__ uint32_t div_magic(int d) { return d > 1 ? 0xffffffffu / (uint32_t)d + 1u : 0u; }
__device__ __forceinline__ int div_small(int k, int d, uint32_t m) { return d > 1 ? (int)__umulhi((uint32_t)k, m) : k; }

__device__ __forceinline__ unsigned long long depth_key(float z, int w) {
	const uint32_t u = __float_as_uint(z);
	const uint32_t o = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
	return ((unsigned long long)o << 32) | (uint32_t)(w + 1);
}
__device__ __forceinline__ float key_depth(unsigned long long k) {
	const uint32_t o = (uint32_t)(k >> 32);
	return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
__device__ __forceinline__ int key_winner(unsigned long long k) { return (int)(uint32_t)k - 1; }

template <int SLOTS, bool MIXED>
struct SmemOT {
	unsigned long long key[kTileSampMax];   // occluding hit of each tile sample (depth_key)
	unsigned long long prev[kTileSampMax];  // ... at the start of the round
	RecS rec[SLOTS];
	int2 pend[SLOTS];
	int pref[SLOTS + 1];                  // running count of (candidate, sample) tests
	int rng[SLOTS][4];                    // tests in the first column, the first row, per row; divisor magic
	int qgrid[kThreadsS];
	int qcum[kThreadsS + 1];
	int qsub[kThreadsS];
	int patidx[kTilePixMax];                // sample pattern of each tile pixel
	int warp_tot[32];
	int first_reject;
	int qn;
	float pixmax[kTilePixMax];
	float blkmax[16];
	uint32_t flag[kTileSampMax / 32];       // samples replayed in order this round
	uint32_t sticky[kTileSampMax / 32];     // samples replayed in order for the rest of the tile
	uint32_t dirty[kTilePixMax / 32];       // pixels whose samples changed this round
	uint32_t mask[MIXED ? kTilePixMax : 1][SLOTS / 32];  // the occluding candidates of each tile pixel
};
using SmemO = SmemOT<kSlotsO, false>;
using SmemMix = SmemOT<kSlotsMix, true>;
static_assert(sizeof(SmemMix) <= (228 * 1024 - 2 * 1024) / 2, "two CTAs of the mixed sampler must fit on an SM");

// Position (x, y), sub-sample (sm, sn) and pixel (px, py) against candidate r:
// every test RenderMPG_Static makes but early-z.  D and (u, v) of a hit.  The
// caller divides the sample's index si = sn * xs + sm once: inside its loop over
// candidates the division was 1 instruction in 9 of the ordered replay (layers in
// one plane at 1920x1080, which replay nearly every sample: 20.6 ms, 18.3 now).
__device__ __forceinline__ bool static_hit(const FrameParams& fp, const GridsDev& g, const SamplerDev& smp,
                                           const BinBuffers& bb, const RecS& r, int px, int py, int si, int smm,
                                           int sn, float x, float y, float& D, float& u, float& v) {
	const int xs = fp.xs, ys = fp.ys;
	const int m_lo = (px == r.px0) ? r.im : 0, m_hi = (px == r.px1 - 1) ? r.em : xs;
	const int n_lo = (py == r.py0) ? r.in_ : 0, n_hi = (py == r.py1 - 1) ? r.en : ys;
	if (!(px >= r.px0 && px < r.px1 && py >= r.py0 && py < r.py1 && smm >= m_lo && smm < m_hi && sn >= n_lo &&
	      sn < n_hi && !((x < r.bminx || x > r.bmaxx) || (y < r.bminy || y > r.bmaxy)) &&
	      !((r.bits & kRecLod) && lod_rejects(fp, g, smp, r.bits >> kRecGridShift, px, py, si)) &&
	      edges_inside(r.ym, r.xm, r.ex, r.ey, x, y)))
		return false;
	inv_bilinear(r.ax, r.ay, r.e_x, r.e_y, r.f_x, r.f_y, r.g_x, r.g_y, (r.bits & kRecLinear) != 0, x, y, u, v);
	D = bilerp1(r.z[0], r.z[1], r.z[2], r.z[3], u, v);
	return rec_keeps(g, bb, r.bits, r.id, x, y, u, v);
}

// REDO (with PERSIST): the tiles and single pixels of bb.redo, which the near
// to far sampler left to the order of insertion.
template <bool PERSIST, int SLOTS, bool MIXED, bool REDO = false>
__global__ void __launch_bounds__(kThreadsS, 2)
sample_opaque_kernel(FrameParams fp, GridsDev g, SamplerDev smp, BinBuffers bb, SampleStore st, FragPool pool,
                     int* queue, const int* order) {
	if (MIXED && !*pool.occluders) return;  // sample_frag_kernel renders this frame
	const bool redo_all = REDO && *bb.nirr_total > bb.nirr_limit;
	if (REDO && !redo_all && *bb.redo == 0) return;
	using SmemO = SmemOT<SLOTS, MIXED>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	SmemO& sm = *reinterpret_cast<SmemO*>(smem_raw);
	__shared__ int next_tile;
	const int ntiles = REDO && !redo_all ? *bb.redo : fp.ntx * fp.nty;
	const FragPool nopool{};
	// MIXED: append the fragments of the lanes with `app` (one per lane, sample
	// index `at` in pool.heads) from pool slots this warp reserved (a run's rest
	// is used before the next run is reserved).
	FragRun run;
	const int run_len = frag_run(fp.tile_w * fp.tile_h * fp.spp);
	auto append = [&](bool app, long long at, float D, int id, float u, float v) {
		const unsigned bal = __ballot_sync(0xffffffffu, app);
		const int nh = __popc(bal), lane = threadIdx.x & 31;
		if (nh == 0) return;
		const unsigned long long base = run.reserve(pool, nh, run_len, lane);
		if (app) {
			const long long idx = run.slot(__popc(bal & ((1u << lane) - 1u)), base);
			if (idx < pool.capacity) {
				pool.frag[idx] = make_float4(D, __int_as_float(id), u, v);
				pool.next[idx] = atomicExch(pool.heads + at, (int)idx);
			} else {
				atomicOr(pool.overflow, 1);
			}
		}
		run.used(nh, run_len, base);
	};
	for (int job = 0;; ++job) {
	int tile;
	if (PERSIST) {
		__syncthreads();
		if (threadIdx.x == 0) next_tile = atomicAdd(queue, 1);
		__syncthreads();
		tile = next_tile;
		if (tile >= ntiles) break;
		if (REDO) tile = redo_all ? tile : bb.redo[1 + tile];
		else if (order) tile = order[tile];
	} else {
		if (job > 0) break;
		tile = blockIdx.x;
	}
	// a redo entry below zero is a pixel: a tile at the pixel, cut off after it
	const bool one = REDO && tile < 0;
	const int tx = one ? (~tile % fp.sw) / fp.tile_w : tile % fp.ntx, ty = one ? (~tile / fp.sw) / fp.tile_h : tile / fp.ntx;
	const int tpx0 = one ? fp.sx0 + ~tile % fp.sw : fp.sx0 + tx * fp.tile_w;
	const int tpy0 = one ? fp.sy0 + ~tile / fp.sw : fp.sy0 + ty * fp.tile_h;
	const int tpx1 = one ? tpx0 + 1 : min(tpx0 + fp.tile_w, fp.sx0 + fp.sw);
	const int tpy1 = one ? tpy0 + 1 : min(tpy0 + fp.tile_h, fp.sy0 + fp.sh);
	const int st_idx = (ty / fp.st_tiles) * fp.nstx + (tx / fp.st_tiles);
	const int t = threadIdx.x;
	const int spp = fp.spp, xs = fp.xs, ys = fp.ys;
	const uint32_t mxs = div_magic(xs), mys = div_magic(ys);
	const int tpix = fp.tile_w * fp.tile_h;
	const int tsamp = tpix * spp;
	const int nflagw = (tsamp + 31) >> 5;
	const unsigned long long kinit = depth_key(FLT_MAX, -1);

	// MIXED: place of tile sample s of pixel pl in the pixel-major arrays
	auto sample_at = [&](int pl, int s) -> long long {
		const int py = tpy0 + pl / fp.tile_w, px = tpx0 + pl % fp.tile_w;
		return ((long long)(py - fp.sy0) * fp.sw + (px - fp.sx0)) * spp + (s - pl * spp);
	};
	for (int i = t; i < tsamp; i += kThreadsS) {
		sm.key[i] = kinit;
		sm.prev[i] = kinit;
		if (MIXED) {
			const int pl = i / spp;
			if (tpx0 + pl % fp.tile_w < tpx1 && tpy0 + pl / fp.tile_w < tpy1) pool.heads[sample_at(pl, i)] = -1;
		}
	}
	if (MIXED)
		for (int i = t; i < kTilePixMax * (SLOTS / 32); i += kThreadsS) (&sm.mask[0][0])[i] = 0u;
	for (int i = t; i < kTileSampMax / 32; i += kThreadsS) {
		sm.flag[i] = 0u;
		sm.sticky[i] = 0u;
	}
	if (t < kTilePixMax / 32) sm.dirty[t] = 0u;
	for (int i = t; i < kTilePixMax; i += kThreadsS) {
		sm.pixmax[i] = one && i > 0 ? -FLT_MAX : FLT_MAX;
		const int px = tpx0 + i % fp.tile_w, py = tpy0 + i / fp.tile_w;
		int pat = 0;
		if (i < tpix && px < tpx1 && py < tpy1) {
			const long long pix = (long long)(py - fp.sy0) * fp.sw + (px - fp.sx0);
			pat = smp.pos_index ? (int)__ldg(smp.pos_index + pix) : (int)pix;
		}
		sm.patidx[i] = pat;
	}
	if (t < 16) sm.blkmax[t] = FLT_MAX;
	if (t == 0) {
		sm.qn = 0;
		sm.qcum[0] = 0;
	}
	__syncthreads();

	const int lbeg = bb.st_offset[st_idx * bb.nranges];
	const int lend = (int)min((long long)bb.st_offset[(st_idx + 1) * bb.nranges], (long long)bb.list_capacity);
	int lp = lbeg, r0 = 0, qtotal = 0, npend = 0;
	for (;;) {
		const bool exhausted =
		    stage_candidates<SLOTS, false>(fp, g, bb, sm, tpx0, tpy0, tpx1, tpy1, lend, lp, r0, qtotal, npend);
		if (npend == 0) break;

		// ---- records, and the (candidate, sample) tests RenderMPG_Static makes ----
		// The samples a candidate visits form a product set: columns of the
		// clipped pixel range with their sub-sample ranges (the first and last
		// pixel trimmed, bucketprocessor.cpp:1135-1153) times the same in y.
		int ntests = 0;
		bool occludes = true;
		if (t < npend) {
			const int2 e = sm.pend[t];
			RecS& r = sm.rec[t];
			build_record(fp, g, e.x, e.y, r);
			const int sX = max(r.px0, tpx0), eX = min(r.px1, tpx1);
			const int sY = max(r.py0, tpy0), eY = min(r.py1, tpy1);
			// per-axis counts: first pixel, then full pixels, the last one trimmed
			int cx0 = ((sX == r.px1 - 1) ? r.em : xs) - ((sX == r.px0) ? r.im : 0);
			int totx = cx0;
			if (eX - sX > 1) totx += (eX - sX - 2) * xs + ((eX - 1 == r.px1 - 1) ? r.em : xs);
			int cy0 = ((sY == r.py1 - 1) ? r.en : ys) - ((sY == r.py0) ? r.in_ : 0);
			int toty = cy0;
			if (eY - sY > 1) toty += (eY - sY - 2) * ys + ((eY - 1 == r.py1 - 1) ? r.en : ys);
			totx = max(totx, 0);
			toty = max(toty, 0);
			ntests = totx * toty;
			sm.rng[t][0] = cx0;
			sm.rng[t][1] = cy0;
			sm.rng[t][2] = totx;
			sm.rng[t][3] = (int)div_magic(totx);
			if (MIXED) {
				occludes = (r.bits & kRecOccluding) != 0;
				if (occludes)
					for (int yy = sY; yy < eY; ++yy)
						for (int xx = sX; xx < eX; ++xx)
							atomicOr(&sm.mask[(yy - tpy0) * fp.tile_w + (xx - tpx0)][t >> 5], 1u << (t & 31));
			}
		}
		for (int ph = 0; ph < (MIXED ? 2 : 1); ++ph) {  // occluding candidates, then transparent ones
		int total;
		const int pre = block_excl_sum(sm.warp_tot, occludes == (ph == 0) ? ntests : 0, total);
		if (t < npend) sm.pref[t] = pre;
		__syncthreads();

		// ---- parallel pass: one (candidate, sample) test per lane, each warp
		// walking a contiguous run of tests so a lane finds its candidate a
		// step or two on from where the warp's last lane stopped ----
		const int chunk = ((total + kThreadsS - 1) / kThreadsS) * 32;
		const int pw0 = (t >> 5) * chunk, pw1 = min(total, pw0 + chunk);
		int cur = 0;
		for (int p0 = pw0; p0 < pw1; p0 += 32) {
			const int p = p0 + (t & 31);
			const int lo = advance_item(sm.pref, npend, cur, min(p, pw1 - 1));
			cur = __shfl_sync(0xffffffffu, lo, 31);
			bool app = false;  // MIXED, second pass: a fragment
			long long at = 0;
			int id = 0;
			float D = 0.0f, u = 0.0f, v = 0.0f;
			// one test; the lambda's returns end it
			[&]() {
			if (p >= pw1) return;
			const RecS& r = sm.rec[lo];
			const int k = p - sm.pref[lo];
			const int cx0 = sm.rng[lo][0], cy0 = sm.rng[lo][1], totx = sm.rng[lo][2];
			const uint32_t mtot = (uint32_t)sm.rng[lo][3];
			const int sX = max(r.px0, tpx0), sY = max(r.py0, tpy0);
			const int ky = div_small(k, totx, mtot), kx = k - ky * totx;
			int px, m, py, n;
			if (kx < cx0) {
				px = sX;
				m = ((sX == r.px0) ? r.im : 0) + kx;
			} else {
				const int q = kx - cx0;
				const int qd = div_small(q, xs, mxs);
				px = sX + 1 + qd;
				m = q - qd * xs;
			}
			if (ky < cy0) {
				py = sY;
				n = ((sY == r.py0) ? r.in_ : 0) + ky;
			} else {
				const int q = ky - cy0;
				const int qd = div_small(q, ys, mys);
				py = sY + 1 + qd;
				n = q - qd * ys;
			}
			const int si = n * xs + m;
			const int pl = (py - tpy0) * fp.tile_w + (px - tpx0);
			const int s = pl * spp + si;
			if (sm.flag[s >> 5] & (1u << (s & 31))) return;  // replayed in order below
			const float2 o = __ldg(smp.pos + (long long)sm.patidx[pl] * spp + si);
			const float x = (float)px + o.x, y = (float)py + o.y;
			// CqBound::Contains2D (bound.h:144-151), early-z, fContains
			if ((x < r.bminx || x > r.bmaxx) || (y < r.bminy || y > r.bmaxy)) return;
			if (r.bminz > key_depth(sm.prev[s])) return;
			if ((r.bits & kRecLod) && lod_rejects(fp, g, smp, r.bits >> kRecGridShift, px, py, si)) return;
			if (!edges_inside(r.ym, r.xm, r.ex, r.ey, x, y)) return;
			inv_bilinear(r.ax, r.ay, r.e_x, r.e_y, r.f_x, r.f_y, r.g_x, r.g_y, (r.bits & kRecLinear) != 0, x, y, u,
			             v);
			D = bilerp1(r.z[0], r.z[1], r.z[2], r.z[3], u, v);
			if (!rec_keeps(g, bb, r.bits, r.id, x, y, u, v)) return;
			if (MIXED && ph == 1) {
				const unsigned long long kk = sm.key[s];
				const float zp = key_depth(sm.prev[s]), zk = key_depth(kk);
				if (zp <= D) return;
				app = !(r.bminz > zk) && !(zk <= D);
				if (!app && key_winner(kk) > r.id) {
					// z after the occluding candidates before this one (those
					// behind prev fail early-z there too, wherever they are hit)
					float z = zp;
					for (int wd = 0; wd <= (lo >> 5); ++wd) {
						uint32_t mb = sm.mask[pl][wd];
						if (wd == (lo >> 5)) mb &= (1u << (lo & 31)) - 1u;
						while (mb) {
							const int c = wd * 32 + __ffs(mb) - 1;
							mb &= mb - 1u;
							float Dc, uc, vc;
							if (!(sm.rec[c].bminz > zp) && static_hit(fp, g, smp, bb, sm.rec[c], px, py, si, m, n, x, y, Dc, uc, vc))
								z = fminf(z, Dc);
						}
					}
					app = !(r.bminz > z) && !(z <= D);
				}
				at = sample_at(pl, s);
				id = r.id;
			} else if (!(D >= r.bminz) || D == 0.0f) {
				atomicOr(&sm.flag[s >> 5], 1u << (s & 31));
			} else {
				const unsigned long long k = depth_key(D, r.id);
				if (k < atomicMin(&sm.key[s], k)) atomicOr(&sm.dirty[pl >> 5], 1u << (pl & 31));
			}
			}();
			if (MIXED && ph == 1) append(app, at, D, id, u, v);
		}
		__syncthreads();
		}  // occluding, transparent
		int anyf = 0;
		for (int i = t; i < nflagw; i += kThreadsS) anyf |= (int)(sm.flag[i] != 0u);

		// ---- ordered replay of flagged samples: a warp per sample ----
		// Lanes test 32 candidates at a time (the tests do not depend on
		// occlZ); lane order then applies early-z and the store rule in
		// insertion order.
		if (__syncthreads_or(anyf)) {
			const int lane = t & 31, warp = t >> 5;
			for (int wd = warp; wd < nflagw; wd += kWarpsS) {
				uint32_t fb = sm.flag[wd];
				while (fb) {
					const int s = wd * 32 + __ffs(fb) - 1;
					fb &= fb - 1u;
					const int pl = s / spp, si = s - pl * spp;
					const int px = tpx0 + pl % fp.tile_w, py = tpy0 + pl / fp.tile_w;
					if (px >= tpx1 || py >= tpy1) continue;
					const int sn = si / xs, smm = si - sn * xs;
					const float2 o = __ldg(smp.pos + (long long)sm.patidx[pl] * spp + si);
					const float x = (float)px + o.x, y = (float)py + o.y;
					float oz = key_depth(sm.prev[s]);
					int w = key_winner(sm.prev[s]);
					for (int c0 = 0; c0 < npend; c0 += 32) {
						const int c = c0 + lane;
						bool hit = false, occl = true;
						float D = 0.0f, bz = 0.0f, u = 0.0f, v = 0.0f;
						int id = 0;
						if (c < npend) {
							const RecS& r = sm.rec[c];
							hit = static_hit(fp, g, smp, bb, r, px, py, si, smm, sn, x, y, D, u, v);
							bz = r.bminz;
							id = r.id;
							if (MIXED) occl = (r.bits & kRecOccluding) != 0;
						}
						uint32_t hb = __ballot_sync(0xffffffffu, hit);
						while (hb) {
							const int b = __ffs(hb) - 1;
							hb &= hb - 1u;
							const float Db = __shfl_sync(0xffffffffu, D, b);
							const float bzb = __shfl_sync(0xffffffffu, bz, b);
							const int idb = __shfl_sync(0xffffffffu, id, b);
							if (bzb > oz || oz <= Db) continue;
							if (!MIXED || __shfl_sync(0xffffffffu, (int)occl, b)) {
								oz = Db;
								w = idb;
							} else {
								append(lane == b, sample_at(pl, s), Db, idb, u, v);
							}
						}
					}
					if (lane == 0) {
						sm.key[s] = depth_key(oz, w);
						atomicOr(&sm.dirty[pl >> 5], 1u << (pl & 31));
						if (oz != oz || oz == 0.0f) atomicOr(&sm.sticky[s >> 5], 1u << (s & 31));
					}
				}
			}
		}
		__syncthreads();

		// ---- end of round: state and largest occluding depth of the pixels
		// whose samples changed (two threads per pixel, even and odd samples;
		// the maximum does not depend on the order, NaN counting as +inf),
		// flags ----
		for (int u0 = 0; u0 < 2 * tpix; u0 += kThreadsS) {
			const int u = u0 + t, pp = u >> 1, half = u & 1;
			const bool act = pp < tpix && (sm.dirty[pp >> 5] & (1u << (pp & 31)));
			float mx = -FLT_MAX;
			if (act)
				for (int k = half; k < spp; k += 2) {
					const unsigned long long kk = sm.key[pp * spp + k];
					sm.prev[pp * spp + k] = kk;
					mx = max_depth(mx, key_depth(kk));
				}
			mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
			if (act && half == 0) sm.pixmax[pp] = mx;
		}
		for (int i = t; i < nflagw; i += kThreadsS) sm.flag[i] = sm.sticky[i];
		if (MIXED)
			for (int i = t; i < kTilePixMax * (SLOTS / 32); i += kThreadsS) (&sm.mask[0][0])[i] = 0u;
		__syncthreads();
		if (t < kTilePixMax / 32) sm.dirty[t] = 0u;
		if (t < 16 * 16) {
			// 4x4-pixel block t / 16, one pixel per thread
			const int b = t >> 4, j = t & 15;
			const int nbx = (fp.tile_w + 3) >> 2;
			const int bx = b % nbx, by = b / nbx;
			const int yy = by * 4 + (j >> 2), xx = bx * 4 + (j & 3);
			float mx = (yy < fp.tile_h && xx < fp.tile_w) ? sm.pixmax[yy * fp.tile_w + xx] : -FLT_MAX;
#pragma unroll
			for (int o = 1; o < 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
			if (j == 0) sm.blkmax[b] = mx;
		}
		__syncthreads();
		npend = 0;
		if (exhausted) break;
	}

	// ---- resolve: colours of the occluding hits ----
	if (MIXED) {
		// hand the occluding hits to resolve_mixed_kernel, beside the list heads
		for (int q = t; q < tsamp; q += kThreadsS) {
			const int pl = q / spp;
			if (tpx0 + pl % fp.tile_w >= tpx1 || tpy0 + pl / fp.tile_w >= tpy1) continue;
			const long long at = sample_at(pl, q);
			st.winner[at] = key_winner(sm.key[q]);
			st.occlz[at] = key_depth(sm.key[q]);
		}
		continue;
	}
	if (st.keys) {
		// hand the occluding hits to resolve_opaque_kernel, pixel-major
		// ([pixel][sample index]) like its threads
		for (int q = t; q < tsamp; q += kThreadsS) {
			const int pl = q / spp;
			const int si = q - pl * spp;
			const int px = tpx0 + pl % fp.tile_w, py = tpy0 + pl / fp.tile_w;
			if (px >= tpx1 || py >= tpy1) continue;
			st.keys[((long long)(py - fp.sy0) * fp.sw + (px - fp.sx0)) * spp + si] = sm.key[pl * spp + si];
		}
		continue;
	}
	// pixel-major: the lanes of a pixel's samples mostly resolve the same
	// winner, whose grid, vertex and colour loads then merge (measured faster
	// than sample-major order, whose store writes coalesce instead)
	for (int q = t; q < tsamp; q += kThreadsS) {
		const int pl = q / spp;
		const int si = q - pl * spp;
		const int px = tpx0 + pl % fp.tile_w, py = tpy0 + pl / fp.tile_w;
		if (px >= tpx1 || py >= tpy1) continue;
		const long long pix = (long long)(py - fp.sy0) * fp.sw + (px - fp.sx0);
		const float2 o = __ldg(smp.pos + (long long)sm.patidx[pl] * spp + si);
		const unsigned long long kk = sm.key[pl * spp + si];
		const bool has = resolve_sample<false>(fp, g, nopool, st, pix * spp + si, store_index(pix, si, spp),
		                                       (float)px + o.x, (float)py + o.y, key_depth(kk), key_winner(kk), -1);
		if (st.wmask) st.wmask[store_index(pix, si, spp)] =
		    window_word(fp, px, py, (float)px + o.x, (float)py + o.y, has);
	}
	}  // tile loop
	if (MIXED) count_holes(pool, run.left);
}

// ---- opaque frames sampled near to far ----
//
// The kernel above visits candidates in insertion order because a hit whose
// depth D lies below its bound's min z b (rounding, Newton error: an anomalous
// hit) may be skipped by early-z although D < occlZ, and one not visited could
// be such a hit.  Neither matters unless depths nearly meet.  Let M be the
// least (D, id) over all hits of a sample, m the hit.
//  * If D_m >= b_m, or no other hit has its depth in [M, b_m), the reference
//    ends with m: when it comes to m, occlZ is FLT_MAX or another hit's depth,
//    which is at least b_m, so m passes early-z, is stored (occlZ > D_m, or >=
//    with m first), and nothing later is nearer.
//  * A regular micropolygon's hits lie no further than its slack below b
//    (bin.cu), so one with b - slack > z has no hit at or below z.  It can be
//    skipped when z is the sample's least depth so far, or, where that hit is
//    anomalous, its b.
// So candidates come in any order -- near grids first, which hides most of the
// rest before a vertex of theirs is read -- irregular micropolygons are never
// skipped, and each sample keeps its least (D, id), a bit for an anomalous hit
// in the key, and the least depth z2 of all its other tested hits.  At the end
// a sample whose m is anomalous with z2 < b_m is not decided (a skipped hit
// within [M, b_m) implies it: what it was skipped for is then a tested hit
// below b_m), nor is one that met a NaN or zero depth: their pixels, or the
// tile once there are many, are sampled again by the kernel above (REDO).  So
// is the whole frame when an eighth of its micropolygons is irregular: testing
// those behind everything else costs more than the order saves (measured at a
// quarter, folded quads 25 layers deep: 13.5 against 11.3 ms).
//
// Sampling and binning, 16 samples, ordered -> near (ms): 1920x1080 at 25
// layers 9.1 -> 5.7, at 4 layers 4.5 -> 3.4, at 0.7 1.9 -> 1.8, 640x480 at 0.7
// 0.36 -> 0.29 (no replays, and 18 KB less shared memory per CTA leave the
// sample patterns twice the L1): every opaque static frame takes it.  Layers of
// flat grids at random depths, where rounding makes 40% of the hits anomalous,
// 15.0 -> 4.1; several layers in exactly one plane, which mostly go in order
// after all, 19.0 -> 19.8.
//
// That last figure was 21.2 with every tile tried.  A tile given up costs a
// tenth of its ordered time, so once 32 tiles and three quarters of those tried
// were given up, the others go to the list untried, except one in 32, which
// keeps the share current where the image changes.  Which tiles those are
// depends on timing; the results do not.  Frames of up to 512 tiles, most of
// which start before one is done, are not counted.
constexpr int kCountedTiles = 512;

struct RecZ : RecS {
	float zcull;  // b - slack; -inf: never skipped
	int pad;      // an odd number of words
};
static_assert(sizeof(RecZ) % 8 == 4, "an odd stride spreads neighbouring records over the banks");

struct SmemZ {
	unsigned long long key[kTileSampMax];   // least hit: (ordered depth, id + 1, anomalous)
	uint32_t z2[kTileSampMax];              // least depth (ordered) of the other hits
	RecZ rec[kSlotsO];
	int2 pend[kSlotsO];
	int pref[kSlotsO + 1];
	int rng[kSlotsO][4];
	int qgrid[kThreadsS];
	int qcum[kThreadsS + 1];
	int qsub[kThreadsS];
	int patidx[kTilePixMax];
	int warp_tot[32];
	int first_reject;
	int qn;
	float pixmax[kTilePixMax];
	float blkmax[16];
	uint32_t dirty[kTilePixMax / 32];
	uint32_t bad[kTilePixMax / 32];         // pixels to sample again in order
	int whole;                              // ... or all of them
};

// Min z of micropolygon `id` (CalculateBound).
__device__ __noinline__ float mp_minz(const GridsDev& g, int id) {
	const int gi = grid_of(g, id);
	const int cu = __ldg(g.cu + gi);
	const int m = id - (int)__ldg(g.mpbase + gi), iv = m / cu;
	const float4* P = g.P + __ldg(g.pbase + gi) + iv * (cu + 1) + (m - iv * cu);
	return amin(amin(amin(__ldg(P).z, __ldg(P + 1).z), __ldg(P + cu + 2).z), __ldg(P + cu + 1).z);
}

template <bool PERSIST>
__global__ void __launch_bounds__(kThreadsS, 2)
sample_near_kernel(FrameParams fp, const __grid_constant__ GridsDev g, SamplerDev smp, BinBuffers bb, SampleStore st,
                   int* queue) {
	if (*bb.nirr_total > bb.nirr_limit) return;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	SmemZ& sm = *reinterpret_cast<SmemZ*>(smem_raw);
	__shared__ int next_tile;
	const int ntiles = fp.ntx * fp.nty;
	const bool counted = ntiles > kCountedTiles;
	const FragPool nopool{};
	for (int job = 0;; ++job) {
	int tile;
	if (PERSIST) {
		__syncthreads();
		if (threadIdx.x == 0) next_tile = atomicAdd(queue, 1);
		__syncthreads();
		tile = next_tile;
		if (tile >= ntiles) break;
	} else {
		if (job > 0) break;
		tile = blockIdx.x;
	}
	const int tw = fp.tile_w, th = fp.tile_h;
	const int tx = tile % fp.ntx, ty = tile / fp.ntx;
	const int tpx0 = fp.sx0 + tx * tw, tpy0 = fp.sy0 + ty * th;
	const int tpx1 = min(tpx0 + tw, fp.sx0 + fp.sw), tpy1 = min(tpy0 + th, fp.sy0 + fp.sh);
	const int st_idx = (ty / fp.st_tiles) * fp.nstx + (tx / fp.st_tiles);
	const int t = threadIdx.x;
	const int spp = fp.spp, xs = fp.xs, ys = fp.ys;
	const uint32_t mxs = div_magic(xs), mys = div_magic(ys);
	const int tpix = tw * th;
	const int tsamp = tpix * spp;
	int given = 0, tried = 0;
	if (t == 0 && counted) {
		tried = *(volatile int32_t*)bb.near_tried;
		given = *(volatile int32_t*)(bb.near_tried + 1);
	}
	const unsigned long long kinit = near_key(FLT_MAX, -1, false);

	for (int i = t; i < tsamp; i += kThreadsS) {
		sm.key[i] = kinit;
		sm.z2[i] = ordered_bits(FLT_MAX);
	}
	if (t < kTilePixMax / 32) {
		sm.dirty[t] = 0u;
		sm.bad[t] = 0u;
	}
	for (int i = t; i < kTilePixMax; i += kThreadsS) {
		sm.pixmax[i] = FLT_MAX;
		const int px = tpx0 + i % tw, py = tpy0 + i / tw;
		int pat = 0;
		if (i < tpix && px < tpx1 && py < tpy1) {
			const long long pix = (long long)(py - fp.sy0) * fp.sw + (px - fp.sx0);
			pat = smp.pos_index ? (int)__ldg(smp.pos_index + pix) : (int)pix;
		}
		sm.patidx[i] = pat;
	}
	if (t < 16) sm.blkmax[t] = FLT_MAX;
	if (t == 0) {
		sm.qn = 0;
		sm.qcum[0] = 0;
		sm.whole = (tile & 31) != 0 && given >= 32 && given > tried - (tried >> 2);  // not worth trying
	}
	__syncthreads();
	if (sm.whole) {
		if (t == 0) bb.redo[1 + atomicAdd(bb.redo, 1)] = tile;
		if (!PERSIST) break;
		continue;
	}

	const int lbeg = bb.st_offset[st_idx * bb.nranges];
	const int lend = (int)min((long long)bb.st_offset[(st_idx + 1) * bb.nranges], (long long)bb.list_capacity);
	int lp = lbeg, r0 = 0, qtotal = 0, npend = 0, undecided = 0;
	for (;;) {
		const bool exhausted = stage_candidates<kSlotsO, false, true>(fp, g, bb, sm, tpx0, tpy0, tpx1, tpy1, lend, lp, r0,
		                                                              qtotal, npend);
		if (npend == 0) break;

		// records and the (candidate, sample) tests, as in the kernel above
		int ntests = 0;
		if (t < npend) {
			const int2 e = sm.pend[t];
			RecZ& r = sm.rec[t];
			build_record(fp, g, e.x, e.y, r);
			r.zcull = mp_regular(bb, e.x, e.y) ? r.bminz - __ldg(bb.grid_slack + e.x) : -INFINITY;
			const int sX = max(r.px0, tpx0), eX = min(r.px1, tpx1);
			const int sY = max(r.py0, tpy0), eY = min(r.py1, tpy1);
			int cx0 = ((sX == r.px1 - 1) ? r.em : xs) - ((sX == r.px0) ? r.im : 0);
			int totx = cx0;
			if (eX - sX > 1) totx += (eX - sX - 2) * xs + ((eX - 1 == r.px1 - 1) ? r.em : xs);
			int cy0 = ((sY == r.py1 - 1) ? r.en : ys) - ((sY == r.py0) ? r.in_ : 0);
			int toty = cy0;
			if (eY - sY > 1) toty += (eY - sY - 2) * ys + ((eY - 1 == r.py1 - 1) ? r.en : ys);
			totx = max(totx, 0);
			toty = max(toty, 0);
			ntests = totx * toty;
			sm.rng[t][0] = cx0;
			sm.rng[t][1] = cy0;
			sm.rng[t][2] = totx;
			sm.rng[t][3] = (int)div_magic(totx);
		}
		int total;
		const int pre = block_excl_sum(sm.warp_tot, ntests, total);
		if (t < npend) sm.pref[t] = pre;
		__syncthreads();

		const int chunk = ((total + kThreadsS - 1) / kThreadsS) * 32;
		const int pw0 = (t >> 5) * chunk, pw1 = min(total, pw0 + chunk);
		int cur = 0;
		for (int p0 = pw0; p0 < pw1; p0 += 32) {
			const int p = p0 + (t & 31);
			const int lo = advance_item(sm.pref, npend, cur, min(p, pw1 - 1));
			cur = __shfl_sync(0xffffffffu, lo, 31);
			if (p >= pw1) continue;
			const RecZ& r = sm.rec[lo];
			const int k = p - sm.pref[lo];
			const int cx0 = sm.rng[lo][0], cy0 = sm.rng[lo][1], totx = sm.rng[lo][2];
			const uint32_t mtot = (uint32_t)sm.rng[lo][3];
			const int sX = max(r.px0, tpx0), sY = max(r.py0, tpy0);
			const int ky = div_small(k, totx, mtot), kx = k - ky * totx;
			int px, m, py, n;
			if (kx < cx0) {
				px = sX;
				m = ((sX == r.px0) ? r.im : 0) + kx;
			} else {
				const int q = kx - cx0;
				const int qd = div_small(q, xs, mxs);
				px = sX + 1 + qd;
				m = q - qd * xs;
			}
			if (ky < cy0) {
				py = sY;
				n = ((sY == r.py0) ? r.in_ : 0) + ky;
			} else {
				const int q = ky - cy0;
				const int qd = div_small(q, ys, mys);
				py = sY + 1 + qd;
				n = q - qd * ys;
			}
			const int si = n * xs + m;
			const int pl = (py - tpy0) * tw + (px - tpx0);
			const int s = pl * spp + si;
			const unsigned long long have = sm.key[s];
			// behind the sample's least depth (early-z)
			if (r.zcull > key_depth(have) && !((uint32_t)have & 1u)) continue;
			const float2 o = __ldg(smp.pos + (long long)sm.patidx[pl] * spp + si);
			const float x = (float)px + o.x, y = (float)py + o.y;
			// CqBound::Contains2D (bound.h:144-151), fContains
			if ((x < r.bminx || x > r.bmaxx) || (y < r.bminy || y > r.bmaxy)) continue;
			if ((r.bits & kRecLod) && lod_rejects(fp, g, smp, r.bits >> kRecGridShift, px, py, si)) continue;
			if (!edges_inside(r.ym, r.xm, r.ex, r.ey, x, y)) continue;
			float u, v;
			inv_bilinear(r.ax, r.ay, r.e_x, r.e_y, r.f_x, r.f_y, r.g_x, r.g_y, (r.bits & kRecLinear) != 0, x, y, u,
			             v);
			const float D = bilerp1(r.z[0], r.z[1], r.z[2], r.z[3], u, v);
			if (!rec_keeps(g, bb, r.bits, r.id, x, y, u, v)) continue;
			if (D != D || D == 0.0f || r.bminz != r.bminz) {
				// (NaN: the tile, whose culling of whole grids leaves NaN depths out)
				if (D == 0.0f) atomicOr(&sm.bad[pl >> 5], 1u << (pl & 31));
				else sm.whole = 1;
				continue;
			}
			const unsigned long long mine = near_key(D, r.id, D < r.bminz);
			const unsigned long long was = atomicMin(&sm.key[s], mine);
			// of the two the farther depth is another hit's
			atomicMin(&sm.z2[s], max((uint32_t)(was >> 32), (uint32_t)(mine >> 32)));
			if (mine < was) atomicOr(&sm.dirty[pl >> 5], 1u << (pl & 31));
		}
		__syncthreads();

		// ---- end of round: what hides candidates at the pixels whose samples
		// changed (two threads per pixel), then the 4x4-pixel blocks ----
		for (int u0 = 0; u0 < 2 * tpix; u0 += kThreadsS) {
			const int u = u0 + t, pp = u >> 1, half = u & 1;
			const bool act = pp < tpix && (sm.dirty[pp >> 5] & (1u << (pp & 31)));
			float mx = -FLT_MAX;
			if (act)
				for (int k = half; k < spp; k += 2) {
					const unsigned long long kk = sm.key[pp * spp + k];
					float z = key_depth(kk);
					if ((uint32_t)kk & 1u) {
						z = mp_minz(g, near_winner(kk));
						if (sm.z2[pp * spp + k] < ordered_bits(z)) atomicOr(&sm.bad[pp >> 5], 1u << (pp & 31));
					}
					mx = fmaxf(mx, z);
				}
			mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
			if (act && half == 0) sm.pixmax[pp] = mx;
		}
		__syncthreads();
		if (t < kTilePixMax / 32) sm.dirty[t] = 0u;
		if (t < 16 * 16) {
			const int b = t >> 4, j = t & 15;
			const int nbx = (tw + 3) >> 2;
			const int bx = b % nbx, by = b / nbx;
			const int yy = by * 4 + (j >> 2), xx = bx * 4 + (j & 3);
			float mx = (yy < th && xx < tw) ? sm.pixmax[yy * tw + xx] : -FLT_MAX;
#pragma unroll
			for (int o = 1; o < 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
			if (j == 0) sm.blkmax[b] = mx;
		}
		__syncthreads();
		npend = 0;
		// surfaces that coincide: the tile will be sampled in order anyway
		undecided = sm.whole ? kRedoPerTile + 1 : 0;
		for (int i = 0; i < kTilePixMax / 32; ++i) undecided += __popc(sm.bad[i]);
		if (exhausted || undecided > kRedoPerTile) break;
	}
	if (t == 0 && counted) {
		atomicAdd(bb.near_tried, 1);
		if (undecided > kRedoPerTile) atomicAdd(bb.near_tried + 1, 1);
	}
	if (undecided > kRedoPerTile) {
		if (t == 0) bb.redo[1 + atomicAdd(bb.redo, 1)] = tile;
		if (!PERSIST) break;
		continue;
	}
	// every warp has counted sm.bad before one sets more bits below: the count
	// decides for the whole block which of its barriers come next
	__syncthreads();

	// ---- the samples, pixel-major: undecided ones are noted; the rest are
	// resolved, or handed to resolve_opaque_kernel ----
	for (int q = t; q < tsamp; q += kThreadsS) {
		const int pl = q / spp;
		const int si = q - pl * spp;
		const int px = tpx0 + pl % tw, py = tpy0 + pl / tw;
		if (px >= tpx1 || py >= tpy1) continue;
		const long long pix = (long long)(py - fp.sy0) * fp.sw + (px - fp.sx0);
		const unsigned long long kk = sm.key[q];
		const float D = key_depth(kk);
		const int w = near_winner(kk);
		if (((uint32_t)kk & 1u) && sm.z2[q] < ordered_bits(mp_minz(g, w))) atomicOr(&sm.bad[pl >> 5], 1u << (pl & 31));
		if (st.keys) {
			st.keys[pix * spp + si] = depth_key(D, w);
			continue;
		}
		const float2 o = __ldg(smp.pos + (long long)sm.patidx[pl] * spp + si);
		const bool has = resolve_sample<false>(fp, g, nopool, st, pix * spp + si, store_index(pix, si, spp),
		                                       (float)px + o.x, (float)py + o.y, D, w, -1);
		if (st.wmask)
			st.wmask[store_index(pix, si, spp)] = window_word(fp, px, py, (float)px + o.x, (float)py + o.y, has);
	}
	__syncthreads();
	if (t == 0) {
		int n = 0;
		for (int i = 0; i < kTilePixMax / 32; ++i) n += __popc(sm.bad[i]);
		if (n > kRedoPerTile) {
			bb.redo[1 + atomicAdd(bb.redo, 1)] = tile;
		} else if (n > 0) {
			int at = 1 + atomicAdd(bb.redo, n);
			for (int pl = 0; pl < tpix; ++pl)
				if ((sm.bad[pl >> 5] >> (pl & 31)) & 1u)
					bb.redo[at++] = ~((tpy0 + pl / tw - fp.sy0) * fp.sw + (tpx0 + pl % tw - fp.sx0));
		}
	}
	}  // tile loop
}

// Colours of the occluding hits of an opaque frame: one thread per sample,
// pixel-major (consecutive threads, the samples of one pixel, which mostly
// share a winner whose loads then merge).
__global__ void __launch_bounds__(256)
resolve_opaque_kernel(FrameParams fp, GridsDev g, SamplerDev smp, SampleStore st) {
	const long long npix = (long long)fp.sw * fp.sh;
	const long long q0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // pixel * spp + sample index
	if (q0 >= npix * fp.spp) return;
	const long long pix = q0 / fp.spp;
	const int si = (int)(q0 - pix * fp.spp);
	const long long q = store_index(pix, si, fp.spp);
	const int px = fp.sx0 + (int)(pix % fp.sw), py = fp.sy0 + (int)(pix / fp.sw);
	const long long pat = smp.pos_index ? (long long)__ldg(smp.pos_index + pix) : pix;
	const float2 o = __ldg(smp.pos + pat * fp.spp + si);
	const unsigned long long kk = st.keys[q0];
	const bool has = resolve_sample<false>(fp, g, FragPool{}, st, pix * fp.spp + si, q, (float)px + o.x, (float)py + o.y,
	                                       key_depth(kk), key_winner(kk), -1);
	if (st.wmask) st.wmask[q] =
	    window_word(fp, px, py, (float)px + o.x, (float)py + o.y, has);
}


// ---- fragment-only frames: parallel hit tests appending fragments --------
//
// When no micropolygon of a static frame can be occluding (none opaque, none
// matte alpha), or samples are not cullable (a z display with the max or
// average depth filter), StoreSample never sets an occluding hit: occlZ stays
// FLT_MAX, early-z skips only bounds with min.z > FLT_MAX, and every hit with
// !(cullable && FLT_MAX <= D) becomes a fragment (bucketprocessor.cpp:
// 1471-1569).  Which hits are kept then does not depend on order, and Combine
// orders fragments by (depth, micropolygon id), so (micropolygon, sample)
// tests run in parallel as on the opaque path and hits are appended to the
// fragment pool in any order: each block iteration reserves its hits' slots
// with one atomic and links them into per-sample lists in shared memory.
constexpr int kSlotsF = 256;
constexpr int kFragRun = 256;  // pool slots a warp reserves at a time

struct SmemF {
	RecS rec[kSlotsF];
	int2 pend[kSlotsF];
	int pref[kSlotsF + 1];
	int rng[kSlotsF][4];
	int qgrid[kThreadsS];
	int qcum[kThreadsS + 1];
	int qsub[kThreadsS];
	int patidx[kTilePixMax];
	int warp_tot[32];
	int first_reject;
	int qn;
	float pixmax[kTilePixMax];  // stay FLT_MAX: no occluding hits
	float blkmax[16];
	int32_t fhead[kTileSampMax];
};

template <bool PERSIST>
__global__ void __launch_bounds__(kThreadsS, 2)
sample_frag_kernel(FrameParams fp, GridsDev g, SamplerDev smp, BinBuffers bb, SampleStore st, FragPool pool,
                   int* queue, const int* order) {
	if (fp.cullable && *pool.occluders) return;  // the ordered kernel renders this frame
	extern __shared__ __align__(16) unsigned char smem_raw[];
	SmemF& sm = *reinterpret_cast<SmemF*>(smem_raw);
	__shared__ int next_tile;
	const int ntiles = fp.ntx * fp.nty;
	const int cullable = fp.cullable;
	unsigned long long rnext = 0, rend = 0;  // this warp's reserved pool slots [rnext, rend)
	for (int job = 0;; ++job) {
	int tile;
	if (PERSIST) {
		__syncthreads();
		if (threadIdx.x == 0) next_tile = atomicAdd(queue, 1);
		__syncthreads();
		tile = next_tile;
		if (tile >= ntiles) break;
		if (order) tile = order[tile];
	} else {
		if (job > 0) break;
		tile = blockIdx.x;
	}
	const int tx = tile % fp.ntx, ty = tile / fp.ntx;
	const int tpx0 = fp.sx0 + tx * fp.tile_w, tpy0 = fp.sy0 + ty * fp.tile_h;
	const int tpx1 = min(tpx0 + fp.tile_w, fp.sx0 + fp.sw), tpy1 = min(tpy0 + fp.tile_h, fp.sy0 + fp.sh);
	const int st_idx = (ty / fp.st_tiles) * fp.nstx + (tx / fp.st_tiles);
	const int t = threadIdx.x;
	const int spp = fp.spp, xs = fp.xs, ys = fp.ys;
	const uint32_t mxs = div_magic(xs), mys = div_magic(ys);
	const int tpix = fp.tile_w * fp.tile_h;
	const int tsamp = tpix * spp;

	for (int i = t; i < tsamp; i += kThreadsS) sm.fhead[i] = -1;
	for (int i = t; i < kTilePixMax; i += kThreadsS) {
		sm.pixmax[i] = FLT_MAX;
		const int px = tpx0 + i % fp.tile_w, py = tpy0 + i / fp.tile_w;
		int pat = 0;
		if (i < tpix && px < tpx1 && py < tpy1) {
			const long long pix = (long long)(py - fp.sy0) * fp.sw + (px - fp.sx0);
			pat = smp.pos_index ? (int)__ldg(smp.pos_index + pix) : (int)pix;
		}
		sm.patidx[i] = pat;
	}
	if (t < 16) sm.blkmax[t] = FLT_MAX;
	if (t == 0) {
		sm.qn = 0;
		sm.qcum[0] = 0;
	}
	__syncthreads();

	const int lbeg = bb.st_offset[st_idx * bb.nranges];
	const int lend = (int)min((long long)bb.st_offset[(st_idx + 1) * bb.nranges], (long long)bb.list_capacity);
	int lp = lbeg, r0 = 0, qtotal = 0, npend = 0;
	for (;;) {
		const bool exhausted =
		    stage_candidates<kSlotsF>(fp, g, bb, sm, tpx0, tpy0, tpx1, tpy1, lend, lp, r0, qtotal, npend);
		if (npend == 0) break;

		// records and the (candidate, sample) tests, as on the opaque path
		int ntests = 0;
		if (t < npend) {
			const int2 e = sm.pend[t];
			RecS& r = sm.rec[t];
			build_record(fp, g, e.x, e.y, r);
			const int sX = max(r.px0, tpx0), eX = min(r.px1, tpx1);
			const int sY = max(r.py0, tpy0), eY = min(r.py1, tpy1);
			int cx0 = ((sX == r.px1 - 1) ? r.em : xs) - ((sX == r.px0) ? r.im : 0);
			int totx = cx0;
			if (eX - sX > 1) totx += (eX - sX - 2) * xs + ((eX - 1 == r.px1 - 1) ? r.em : xs);
			int cy0 = ((sY == r.py1 - 1) ? r.en : ys) - ((sY == r.py0) ? r.in_ : 0);
			int toty = cy0;
			if (eY - sY > 1) toty += (eY - sY - 2) * ys + ((eY - 1 == r.py1 - 1) ? r.en : ys);
			totx = max(totx, 0);
			toty = max(toty, 0);
			ntests = totx * toty;
			sm.rng[t][0] = cx0;
			sm.rng[t][1] = cy0;
			sm.rng[t][2] = totx;
			sm.rng[t][3] = (int)div_magic(totx);
		}
		int total;
		const int pre = block_excl_sum(sm.warp_tot, ntests, total);
		if (t < npend) sm.pref[t] = pre;
		__syncthreads();

		// each warp walks a contiguous run of tests (a lane finds its candidate
		// a step or two on from where the warp's last lane stopped) and appends
		// its hits into pool slots it reserved in runs of kFragRun: one global
		// atomic per run, no block barrier per batch of tests.  Lists are
		// sorted by (depth, id) in Combine, so their order does not matter;
		// slots left in a warp's last run stay unused.
		{
			const int lane = t & 31;
			const int chunk = ((total + kThreadsS - 1) / kThreadsS) * 32;
			const int pw0 = (t >> 5) * chunk, pw1 = min(total, pw0 + chunk);
			int cur = 0;
			for (int p0 = pw0; p0 < pw1; p0 += 32) {
				const int p = p0 + lane;
				const int lo = advance_item(sm.pref, npend, cur, min(p, pw1 - 1));
				cur = __shfl_sync(0xffffffffu, lo, 31);
				bool hit = false;
				int s = 0, id = 0;
				float D = 0.0f, u = 0.0f, v = 0.0f;
				if (p < pw1) {
					const RecS& r = sm.rec[lo];
					const int k = p - sm.pref[lo];
					const int cx0 = sm.rng[lo][0], cy0 = sm.rng[lo][1], totx = sm.rng[lo][2];
					const uint32_t mtot = (uint32_t)sm.rng[lo][3];
					const int sX = max(r.px0, tpx0), sY = max(r.py0, tpy0);
					const int ky = div_small(k, totx, mtot), kx = k - ky * totx;
					int px, m, py, n;
					if (kx < cx0) {
						px = sX;
						m = ((sX == r.px0) ? r.im : 0) + kx;
					} else {
						const int q = kx - cx0;
						const int qd = div_small(q, xs, mxs);
						px = sX + 1 + qd;
						m = q - qd * xs;
					}
					if (ky < cy0) {
						py = sY;
						n = ((sY == r.py0) ? r.in_ : 0) + ky;
					} else {
						const int q = ky - cy0;
						const int qd = div_small(q, ys, mys);
						py = sY + 1 + qd;
						n = q - qd * ys;
					}
					const int si = n * xs + m;
					const int pl = (py - tpy0) * fp.tile_w + (px - tpx0);
					s = pl * spp + si;
					const float2 o = __ldg(smp.pos + (long long)sm.patidx[pl] * spp + si);
					const float x = (float)px + o.x, y = (float)py + o.y;
					// Contains2D, early-z against occlZ = FLT_MAX, fContains, StoreSample's test
					hit = !((x < r.bminx || x > r.bmaxx) || (y < r.bminy || y > r.bmaxy)) &&
					      !(cullable && !(r.bits & kRecCsg) && r.bminz > FLT_MAX) &&
					      !((r.bits & kRecLod) && lod_rejects(fp, g, smp, r.bits >> kRecGridShift, px, py, si)) &&
					      edges_inside(r.ym, r.xm, r.ex, r.ey, x, y);
					if (hit) {
						inv_bilinear(r.ax, r.ay, r.e_x, r.e_y, r.f_x, r.f_y, r.g_x, r.g_y, (r.bits & kRecLinear) != 0,
						             x, y, u, v);
						D = bilerp1(r.z[0], r.z[1], r.z[2], r.z[3], u, v);
						hit = rec_keeps(g, bb, r.bits, r.id, x, y, u, v) &&
						      !(cullable && !(r.bits & kRecCsg) && FLT_MAX <= D);
						id = r.id;
					}
				}
				const unsigned bal = __ballot_sync(0xffffffffu, hit);
				const int nh = __popc(bal);
				if (nh > 0) {
					if (rnext + nh > rend) {
						unsigned long long b = 0;
						if (lane == 0) b = atomicAdd(pool.count, (unsigned long long)kFragRun);
						rnext = __shfl_sync(0xffffffffu, b, 0);
						rend = rnext + kFragRun;
					}
					if (hit) {
						const long long idx = (long long)(rnext + __popc(bal & ((1u << lane) - 1u)));
						if (idx < pool.capacity) {
							pool.frag[idx] = make_float4(D, __int_as_float(id), u, v);
							pool.next[idx] = atomicExch(&sm.fhead[s], (int)idx);
						} else {
							atomicOr(pool.overflow, 1);
						}
					}
					rnext += nh;
				}
			}
		}
		__syncthreads();
		npend = 0;
		if (exhausted) break;
	}

	// ---- resolve: Combine of each sample's fragments (or the list heads
	// handed to resolve_frag_kernel) ----
	for (int s = t; s < tsamp; s += kThreadsS) {
		const int pl = s / spp;
		const int si = s - pl * spp;
		const int px = tpx0 + pl % fp.tile_w, py = tpy0 + pl / fp.tile_w;
		if (px >= tpx1 || py >= tpy1) continue;
		const long long pix = (long long)(py - fp.sy0) * fp.sw + (px - fp.sx0);
		if (pool.heads) {
			pool.heads[pix * spp + si] = sm.fhead[s];
			continue;
		}
		const float2 o = __ldg(smp.pos + (long long)sm.patidx[pl] * spp + si);
		const bool has = resolve_sample<true>(fp, g, pool, st, pix * spp + si, store_index(pix, si, spp), (float)px + o.x,
		                     (float)py + o.y, FLT_MAX, -1, sm.fhead[s]);
		if (st.wmask) st.wmask[store_index(pix, si, spp)] =
		    window_word(fp, px, py, (float)px + o.x, (float)py + o.y, has);
	}
	}  // tile loop
}

// Combine of a transparent frame's samples from the list heads the sampler
// left and, OCCL, the occluding hits in st.winner / st.occlz (frames of the
// mixed sampler): one thread per sample, pixel-major, so a warp walks lists
// whose fragments the sampler's warps allocated together.  The kernels hold no
// shared memory, so the sort's local memory stays in L1.  Both may be queued;
// each reads the occluder flag and the one the frame is not for returns at
// once -- the mixed one from a grid bounded by the SMs, since the half million
// empty blocks of a 1080p frame at 64 samples would cost 0.3 ms.  One kernel
// for both measured slower (the occluding hits' colours cost the fragment-only
// form registers: 8.7 ms against 8.1 at that size).
template <bool OCCL>
__device__ __forceinline__ void resolve_frag(const FrameParams& fp, const GridsDev& g, const SamplerDev& smp,
                                             const SampleStore& st, const FragPool& pool, long long q) {
	const long long pix = q / fp.spp;
	const int si = (int)(q - pix * fp.spp);
	const int px = fp.sx0 + (int)(pix % fp.sw), py = fp.sy0 + (int)(pix / fp.sw);
	const long long pat = smp.pos_index ? (long long)__ldg(smp.pos_index + pix) : pix;
	const float2 o = __ldg(smp.pos + pat * fp.spp + si);
	const bool has = resolve_sample<true>(fp, g, pool, st, q, store_index(pix, si, fp.spp), (float)px + o.x, (float)py + o.y,
	                     OCCL ? st.occlz[q] : FLT_MAX, OCCL ? st.winner[q] : -1, pool.heads[q]);
	if (st.wmask) st.wmask[store_index(pix, si, fp.spp)] =
	    window_word(fp, px, py, (float)px + o.x, (float)py + o.y, has);
}

__global__ void __launch_bounds__(256)
resolve_frag_kernel(FrameParams fp, GridsDev g, SamplerDev smp, SampleStore st, FragPool pool) {
	if (fp.cullable && *pool.occluders) return;
	const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // pixel * spp + sample index
	if (q < (long long)fp.sw * fp.sh * fp.spp) resolve_frag<false>(fp, g, smp, st, pool, q);
}

__global__ void __launch_bounds__(256, 4)
resolve_mixed_kernel(FrameParams fp, GridsDev g, SamplerDev smp, SampleStore st, FragPool pool) {
	if (!*pool.occluders) return;
	const long long n = (long long)fp.sw * fp.sh * fp.spp;
	for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
		resolve_frag<true>(fp, g, smp, st, pool, q);
}

// Whether any micropolygon of the frame may be occluding: a grid flagged
// opaque or matte alpha, no opacity array, or a vertex with every opacity
// channel at 1 or more (a superset of SqMpgSampleInfo::isOpaque).
__global__ void occluder_scan_kernel(GridsDev g, int32_t* flag) {
	const int gi = blockIdx.x;
	if (gi >= g.ngrids) return;
	const int gflags = __ldg(g.flags + gi);
	bool occ = (gflags & (8 | 4)) != 0 || g.Oi == nullptr;
	if (!occ) {
		const long long nv = (long long)(__ldg(g.cu + gi) + 1) * (__ldg(g.cv + gi) + 1);
		const long long cb = __ldg(g.cbase + gi);
		for (long long i = threadIdx.x; i < nv && !occ; i += blockDim.x) {
			const float4 o = ld_colour(g, g.Oi, cb + i);
			occ = o.x >= 1.0f && o.y >= 1.0f && o.z >= 1.0f;
		}
	}
	if (__syncthreads_or(occ) && threadIdx.x == 0) *flag = 1;
}

}  // namespace

void launch_resolve_opaque(const FrameParams& fp, const GridsDev& g, const SamplerDev& sm, SampleStore st,
                           cudaStream_t s) {
	const long long n = (long long)fp.sw * fp.sh * fp.spp;
	if (n > 0) resolve_opaque_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(fp, g, sm, st);
}

void static_tiling(FrameParams& fp, int tile_pixels) {
	int tpix = min(kTilePixMax, max(1, kTileSampMax / fp.spp));
	if (tile_pixels > 0) tpix = min(tpix, tile_pixels);
	int tw = 1;
	while ((tw + 1) * (tw + 1) <= tpix) ++tw;
	fp.tile_w = tw;
	fp.tile_h = min(16, tpix / tw);  // at most 4x4 blocks of 4x4 pixels (blkmax)
	fp.tpp = 1;
}

void launch_sample_tiles(const FrameParams& fp, const GridsDev& g, const SamplerDev& sm, const BinBuffers& b,
                         SampleStore st, FragPool pool, int32_t* err, cudaStream_t s, cudaEvent_t colours_ready,
                         unsigned wait_flags) {
	(void)err;
	launch_sample_tiles_q(fp, g, sm, b, st, pool, nullptr, nullptr, 0, s, colours_ready, wait_flags);
}

void launch_sample_tiles_q(const FrameParams& fp, const GridsDev& g, const SamplerDev& sm, const BinBuffers& b,
                           SampleStore st, FragPool pool, int* queue, const int* order, int nctas, cudaStream_t s,
                           cudaEvent_t colours_ready, unsigned wait_flags) {
	const int ntiles = fp.ntx * fp.nty;
	const size_t smem_transp = sizeof(SmemS) + sizeof(int32_t) * kTileSampMax;
	configure_sample_kernels();
	const bool transp = pool.capacity > 0;
	const bool split = !transp && st.keys;  // the resolve kernel is the first reader of Ci/Oi
	if (colours_ready && !split) cudaStreamWaitEvent(s, colours_ready, wait_flags);
	// transparent frames with one occlZ per sample and no solids: the mixed
	// sampler takes them when they have occluders, else the ordered kernel does
	const bool mixed = transp && fp.frag_only && fp.cullable && g.csg.nnodes == 0 && pool.heads;
	if (transp && fp.frag_only) {
		// both samplers are queued; each reads the occluder flag and one returns at once
		if (fp.cullable) {
			cudaMemsetAsync(pool.occluders, 0, sizeof(int32_t), s);
			if (g.ngrids > 0) occluder_scan_kernel<<<g.ngrids, 256, 0, s>>>(g, pool.occluders);
		}
		if (queue)
			sample_frag_kernel<true><<<nctas, kThreadsS, sizeof(SmemF), s>>>(fp, g, sm, b, st, pool, queue, order);
		else
			sample_frag_kernel<false><<<ntiles, kThreadsS, sizeof(SmemF), s>>>(fp, g, sm, b, st, pool, nullptr,
			                                                                  nullptr);
		if (pool.heads) {
			const long long n = (long long)fp.sw * fp.sh * fp.spp, nb = (n + 255) / 256;
			if (n > 0) resolve_frag_kernel<<<(unsigned)nb, 256, 0, s>>>(fp, g, sm, st, pool);
			if (mixed) {
				if (queue) {
					sample_opaque_kernel<true, kSlotsMix, true><<<nctas, kThreadsS, sizeof(SmemMix), s>>>(
					    fp, g, sm, b, st, pool, queue + 1, order);  // sample_frag_kernel may have drawn from the first
				} else {
					sample_opaque_kernel<false, kSlotsMix, true><<<ntiles, kThreadsS, sizeof(SmemMix), s>>>(
					    fp, g, sm, b, st, pool, nullptr, nullptr);
				}
				int dev = 0, nsm = 0;
				cudaGetDevice(&dev);
				cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
				if (n > 0)
					resolve_mixed_kernel<<<(unsigned)min(nb, (long long)nsm * 32), 256, 0, s>>>(fp, g, sm, st, pool);
			}
		}
	}
	if (mixed) return;
	if (!transp && b.st_sorted) {
		// near to far, then what that left to the order of insertion
		if (queue)
			sample_near_kernel<true><<<nctas, kThreadsS, sizeof(SmemZ), s>>>(fp, g, sm, b, st, queue);
		else
			sample_near_kernel<false><<<ntiles, kThreadsS, sizeof(SmemZ), s>>>(fp, g, sm, b, st, nullptr);
		int dev = 0, nsm = 0;
		cudaGetDevice(&dev);
		cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
		sample_opaque_kernel<true, kSlotsO, false, true><<<2 * nsm, kThreadsS, sizeof(SmemO), s>>>(
		    fp, g, sm, b, st, pool, b.redo_next, nullptr);
		if (split) {
			if (colours_ready) cudaStreamWaitEvent(s, colours_ready, wait_flags);
			launch_resolve_opaque(fp, g, sm, st, s);
		}
		return;
	}
	if (transp) {
		if (queue)
			sample_static_kernel<true, true><<<nctas, kThreadsS, smem_transp, s>>>(fp, g, sm, b, st, pool, queue, order);
		else
			sample_static_kernel<true, false><<<ntiles, kThreadsS, smem_transp, s>>>(fp, g, sm, b, st, pool, nullptr, nullptr);
		return;
	}
	// no depth order (the no-allocation form, frames without grids): in order
	sample_opaque_kernel<false, kSlotsO, false><<<ntiles, kThreadsS, sizeof(SmemO), s>>>(fp, g, sm, b, st, pool, nullptr,
	                                                                                   nullptr);
	if (split) {
		if (colours_ready) cudaStreamWaitEvent(s, colours_ready, wait_flags);
		launch_resolve_opaque(fp, g, sm, st, s);
	}
}

// Shared-memory limits of the sampling kernels; safe to call repeatedly, and
// done before any graph capture (context creation calls it).
bool first_use_on_device(std::mutex& mu, uint64_t& mask) {
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
	std::lock_guard<std::mutex> lock(mu);
	if (mask >> dev & 1) return false;
	mask |= uint64_t(1) << dev;
	return true;
}

void configure_sample_kernels() {
	static std::mutex mu;
	static uint64_t configured = 0;
	if (!first_use_on_device(mu, configured)) return;
	const int smem_transp = (int)(sizeof(SmemS) + sizeof(int32_t) * kTileSampMax);
	cudaFuncSetAttribute(sample_opaque_kernel<false, kSlotsO, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                     (int)sizeof(SmemO));
	cudaFuncSetAttribute(sample_opaque_kernel<true, kSlotsO, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                     (int)sizeof(SmemO));
	cudaFuncSetAttribute(sample_near_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemZ));
	cudaFuncSetAttribute(sample_near_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemZ));
	cudaFuncSetAttribute(sample_opaque_kernel<false, kSlotsMix, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                     (int)sizeof(SmemMix));
	cudaFuncSetAttribute(sample_opaque_kernel<true, kSlotsMix, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                     (int)sizeof(SmemMix));
	cudaFuncSetAttribute(sample_static_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_transp);
	cudaFuncSetAttribute(sample_static_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_transp);
	cudaFuncSetAttribute(sample_frag_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemF));
	cudaFuncSetAttribute(sample_frag_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemF));
	configure_sample_mb_kernels();
}

int sample_static_ctas_per_sm(bool transp) {
	int n = 0;
	if (transp)
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sample_static_kernel<true, true>, kThreadsS,
		                                              sizeof(SmemS) + sizeof(int32_t) * kTileSampMax);
	else
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sample_near_kernel<true>, kThreadsS, sizeof(SmemZ));
	return n > 0 ? n : 1;
}

}  // namespace aqh
