// bin.cu -- bound-and-bin stage: per-grid raster rectangles and ordered
// per-super-tile grid lists.
//
// Replaces CqImageBuffer::AddMPG's bucket assignment (libs/core/imagebuffer.cpp:
// 514-591) at grid granularity.  A grid is listed for every super-tile (a
// square of sampling tiles) its pixel rectangle touches, and each list keeps
// grid submission order, so a tile that walks its super-tile's list sees its
// micropolygons in the reference's insertion order (grid order, then iv, iu).
// The exact per-micropolygon tests (bound, AddMPG crop cull) run in the
// sampling kernel; this stage only needs conservative rectangles.
#include "aqh_internal.h"
#include "hider_device.cuh"

namespace aqh {

// One warp per grid: min/max of x, y, z over every vertex of every key, grown
// by the largest circle of confusion in the grid's depth range when depth of
// field is on, turned into the pixel rectangle [floor(min), ceil(max)] + 1
// clipped to the sample region.
// Pixel range [floor(mn), lceil(mx)) packed as two int16, widened to the
// whole int16 range where the floats are out of range or NaN.
__device__ __forceinline__ uint32_t pack_range(float mn, float mx, bool bad) {
	int lo = -32768, hi = 32767;
	if (!bad) {
		if (mn > -32768.0f) lo = (int)floorf(mn);
		if (mx < 32767.0f) hi = lceil_f(mx);
	}
	return (uint32_t)(lo & 0xffff) | ((uint32_t)hi << 16);
}

// Strips: the pixel ranges each micropolygon column and row of a grid can
// touch (x over vertex columns iu, iu+1; y over vertex rows iv, iv+1; every
// motion key), so the sampler streams only the micropolygons whose column and
// row both meet its tile -- a superset of those whose bound does.  In frames
// with motion blur or depth of field the ranges grow by `grow` (the grid's
// largest circle of confusion) and one pixel on each side, which covers the
// staging rectangles of the motion sampler.  Lane = vertex column.
template <int NK>  // NK = 1: one key (its loads pipeline across rows); 0: nk keys
__device__ __forceinline__ void grid_strips(const float4* P, int cu, int cv, int nk, float growx, float growy,
                                            bool margin, int lane, uint32_t* S) {
	if (NK == 1) nk = 1;
	const bool on = lane <= cu;
	const long long nvk = (long long)(cu + 1) * (cv + 1);
	float cmn = FLT_MAX, cmx = -FLT_MAX, pmn = FLT_MAX, pmx = -FLT_MAX;
	bool cbad = false, pbad = false;
	const float mg = margin ? 1.0f : 0.0f;
	for (int j = 0; j <= cv; ++j) {
		float ymn = FLT_MAX, ymx = -FLT_MAX;
		bool ybad = false;
		for (int k = 0; k < nk; ++k) {
			if (on) {
				const float4 p = __ldg(P + k * nvk + j * (cu + 1) + lane);
				cbad |= (p.x != p.x);
				cmn = fminf(cmn, p.x);
				cmx = fmaxf(cmx, p.x);
				ybad |= (p.y != p.y);
				ymn = fminf(ymn, p.y);
				ymx = fmaxf(ymx, p.y);
			}
		}
		if (margin && on) {
			ymn = (ymn - growy) - mg;
			ymx = (ymx + growy) + mg;
		}
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) {
			ymn = fminf(ymn, __shfl_xor_sync(0xffffffffu, ymn, o));
			ymx = fmaxf(ymx, __shfl_xor_sync(0xffffffffu, ymx, o));
		}
		ybad = __any_sync(0xffffffffu, ybad);
		if (j > 0 && lane == 0) S[32 + j - 1] = pack_range(fminf(pmn, ymn), fmaxf(pmx, ymx), pbad || ybad);
		pmn = ymn;
		pmx = ymx;
		pbad = ybad;
	}
	if (margin && on) {
		cmn = (cmn - growx) - mg;
		cmx = (cmx + growx) + mg;
	}
	const float nmn = __shfl_down_sync(0xffffffffu, cmn, 1), nmx = __shfl_down_sync(0xffffffffu, cmx, 1);
	const bool nbad = __shfl_down_sync(0xffffffffu, cbad, 1);
	if (lane < cu) S[lane] = pack_range(fminf(cmn, nmn), fmaxf(cmx, nmx), cbad || nbad);
}

__global__ void grid_rects_kernel(FrameParams fp, GridsDev g, int4* rect, float* minz, uint32_t* strips,
                                  float4* tri, int32_t* redo_head) {
	if (redo_head && blockIdx.x == 0 && threadIdx.x < kRedoHead) redo_head[threadIdx.x] = 0;
	const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int lane = threadIdx.x & 31;
	if (warp >= g.ngrids) return;
	const int cu = g.cu[warp], cv = g.cv[warp];
	const int nk = g.nkeys[warp];
	const long long nv = (long long)(cu + 1) * (cv + 1) * nk;
	const float4* P = g.P + g.pbase[warp];
	float mnx = FLT_MAX, mny = FLT_MAX, mnz = FLT_MAX, mxx = -FLT_MAX, mxy = -FLT_MAX, mxz = -FLT_MAX;
	// four loads in flight per lane (the pass is bound by loads in flight)
#pragma unroll 4
	for (long long i = lane; i < nv; i += 32) {
		float4 p = __ldg(P + i);
		mnx = fminf(mnx, p.x); mxx = fmaxf(mxx, p.x);
		mny = fminf(mny, p.y); mxy = fmaxf(mxy, p.y);
		mnz = fminf(mnz, p.z); mxz = fmaxf(mxz, p.z);
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		mnx = fminf(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
		mny = fminf(mny, __shfl_xor_sync(0xffffffffu, mny, o));
		mnz = fminf(mnz, __shfl_xor_sync(0xffffffffu, mnz, o));
		mxx = fmaxf(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
		mxy = fmaxf(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
		mxz = fmaxf(mxz, __shfl_xor_sync(0xffffffffu, mxz, o));
	}
	// depth of field: the largest blur AddMPG gives any of the grid's
	// micropolygons, max(CoC(bound min z), CoC(bound max z)) over its own
	// bound (imagebuffer.cpp:520-531).  The grid's depth ends do not bound it
	// when the depth range reaches z = 0, where the blur has its pole.
	float mcx = 0.0f, mcy = 0.0f;
	if (fp.use_dof) {
		const long long nvk = (long long)(cu + 1) * (cv + 1);
		for (int m = lane; m < cu * cv; m += 32) {
			const int iv = m / cu, iu = m - iv * cu;
			const long long idx = (long long)iv * (cu + 1) + iu;
			float zl = FLT_MAX, zh = -FLT_MAX;
			for (int k = 0; k < nk; ++k) {
				const float4* Pk = P + k * nvk;
				const float za = __ldg(Pk + idx).z, zb = __ldg(Pk + idx + 1).z;
				const float zc = __ldg(Pk + idx + cu + 1).z, zd = __ldg(Pk + idx + cu + 2).z;
				zl = amin(zl, amin(amin(amin(za, zb), zc), zd));
				zh = amax(zh, amax(amax(amax(za, zb), zc), zd));
			}
			const float2 c1 = coc(zl, fp.dof_mult, fp.dof_inv_fd, fp.dof_scale_x, fp.dof_scale_y);
			const float2 c2 = coc(zh, fp.dof_mult, fp.dof_inv_fd, fp.dof_scale_x, fp.dof_scale_y);
			mcx = fmaxf(mcx, fmaxf(c1.x, c2.x));
			mcy = fmaxf(mcy, fmaxf(c1.y, c2.y));
		}
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) {
			mcx = fmaxf(mcx, __shfl_xor_sync(0xffffffffu, mcx, o));
			mcy = fmaxf(mcy, __shfl_xor_sync(0xffffffffu, mcy, o));
		}
	}
	if (strips) {
		uint32_t* S = strips + (long long)warp * 64;
		const bool mbdof = fp.use_dof || fp.any_motion;
		const bool has = (nk == 1 || mbdof) && nk <= kMaxKeys && cu <= 31 && cv <= 31;
		if (has) {
			if (nk == 1) grid_strips<1>(P, cu, cv, 1, mcx, mcy, mbdof, lane, S);
			else grid_strips<0>(P, cu, cv, nk, mcx, mcy, mbdof, lane, S);
		}
		if (lane == 0) S[63] = has ? 1u : 0u;
	}
	if (lane != 0) return;
	minz[warp] = mnz;
	if (tri && (g.flags[warp] & 16)) {
		// triangle split line per key (micropolygon.cpp:703-719, 737-746): through
		// corners cu and cv*(cu+1), ordered so that the kept side is positive
		const float4* Pg = g.P + g.pbase[warp];
		for (int k = 0; k < nk && k < kMaxKeys; ++k) {
			const long long kb = (long long)k * (cu + 1) * (cv + 1);
			const float4 v0 = Pg[kb], v1 = Pg[kb + cu], v2 = Pg[kb + (long long)cv * (cu + 1)];
			const bool cw = ((v1.x - v0.x) * (v2.y - v0.y) - (v1.y - v0.y) * (v2.x - v0.x)) >= 0;
			tri[(long long)warp * kMaxKeys + k] = cw ? make_float4(v1.x, v1.y, v2.x, v2.y)
			                                         : make_float4(v2.x, v2.y, v1.x, v1.y);
		}
	}
	if (fp.use_dof) {
		float2 c1 = coc(mnz, fp.dof_mult, fp.dof_inv_fd, fp.dof_scale_x, fp.dof_scale_y);
		float2 c2 = coc(mxz, fp.dof_mult, fp.dof_inv_fd, fp.dof_scale_x, fp.dof_scale_y);
		const float cx = fmaxf(fmaxf(c1.x, c2.x), mcx), cy = fmaxf(fmaxf(c1.y, c2.y), mcy);
		mnx -= cx; mxx += cx; mny -= cy; mxy += cy;
	}
	int4 r;
	// one pixel of slack on every side keeps the rectangle conservative
	// against rounding in the per-micropolygon ranges
	float fx0 = floorf(mnx) - 1.0f, fy0 = floorf(mny) - 1.0f;
	float fx1 = ceilf(mxx) + 2.0f, fy1 = ceilf(mxy) + 2.0f;
	const float rx0 = (float)fp.sx0, ry0 = (float)fp.sy0;
	const float rx1 = (float)(fp.sx0 + fp.sw), ry1 = (float)(fp.sy0 + fp.sh);
	fx0 = fmaxf(fx0, rx0); fy0 = fmaxf(fy0, ry0);
	fx1 = fminf(fx1, rx1); fy1 = fminf(fy1, ry1);
	if (!(fx0 < fx1 && fy0 < fy1) || !(mnx <= mxx)) {
		r = make_int4(0, 0, 0, 0);  // empty (also catches NaN)
	} else {
		r = make_int4((int)fx0, (int)fx1, (int)fy0, (int)fy1);
	}
	rect[warp] = r;
}

__device__ __forceinline__ void st_rect(const FrameParams& fp, int st, int& x0, int& x1, int& y0, int& y1) {
	const int stx = st % fp.nstx, sty = st / fp.nstx;
	x0 = fp.sx0 + stx * fp.st_tiles * fp.tile_w;
	y0 = fp.sy0 + sty * fp.st_tiles * fp.tile_h;
	x1 = x0 + fp.st_tiles * fp.tile_w;
	y1 = y0 + fp.st_tiles * fp.tile_h;
}

__device__ __forceinline__ bool rect_hits(int4 r, int x0, int x1, int y0, int y1) {
	return r.x < r.y && r.x < x1 && r.y > x0 && r.z < y1 && r.w > y0;
}

// grid (blockIdx.x = super-tile, blockIdx.y = grid range): count the range's
// grids that touch the super-tile.
__global__ void st_count_kernel(FrameParams fp, int ngrids, const int4* rect, int nranges, int range_size,
                                int32_t* count) {
	const int st = blockIdx.x, r = blockIdx.y;
	int x0, x1, y0, y1;
	st_rect(fp, st, x0, x1, y0, y1);
	const int g0 = r * range_size, g1 = min(ngrids, g0 + range_size);
	int c = 0;
	for (int gi = g0 + threadIdx.x; gi < g1; gi += blockDim.x) c += rect_hits(rect[gi], x0, x1, y0, y1) ? 1 : 0;
	__shared__ int red[32];
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
	if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
	__syncthreads();
	if (threadIdx.x < 32) {
		int v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0;
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
		if (threadIdx.x == 0) count[st * nranges + r] = v;
	}
}

// Ordered compaction: write the range's touching grids at the super-tile's
// offset, in grid order.
__global__ void st_write_kernel(FrameParams fp, int ngrids, const int4* rect, int nranges, int range_size,
                                const int32_t* offset, int32_t* list, long long capacity) {
	const int st = blockIdx.x, r = blockIdx.y;
	int x0, x1, y0, y1;
	st_rect(fp, st, x0, x1, y0, y1);
	const int g0 = r * range_size, g1 = min(ngrids, g0 + range_size);
	__shared__ int warp_tot[32];
	__shared__ int base;
	if (threadIdx.x == 0) base = offset[st * nranges + r];
	__syncthreads();
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
	for (int c0 = g0; c0 < g1; c0 += blockDim.x) {
		const int gi = c0 + threadIdx.x;
		const bool f = gi < g1 && rect_hits(rect[gi], x0, x1, y0, y1);
		const unsigned bal = __ballot_sync(0xffffffffu, f);
		if (lane == 0) warp_tot[wid] = __popc(bal);
		__syncthreads();
		int pre = 0, tot = 0;
		for (int w = 0; w < nw; ++w) {
			int t = warp_tot[w];
			pre += (w < wid) ? t : 0;
			tot += t;
		}
		const long long idx = (long long)base + pre + __popc(bal & ((1u << lane) - 1u));
		if (f && idx < capacity) list[idx] = gi;  // a short list is detected by the host and re-binned
		__syncthreads();
		if (threadIdx.x == 0) base += tot;
		__syncthreads();
	}
}

// Single-block exclusive scan with the grand total appended at out[n].
__global__ void scan_i32_kernel(const int32_t* in, int32_t* out, int n) {
	__shared__ int warp_sum[32];
	__shared__ int carry;
	if (threadIdx.x == 0) carry = 0;
	__syncthreads();
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
	for (int c0 = 0; c0 < n; c0 += blockDim.x) {
		const int i = c0 + threadIdx.x;
		int v = i < n ? in[i] : 0;
		int x = v;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			int y = __shfl_up_sync(0xffffffffu, x, o);
			if (lane >= o) x += y;
		}
		if (lane == 31) warp_sum[wid] = x;
		__syncthreads();
		int pre = 0, tot = 0;
		for (int w = 0; w < nw; ++w) {
			pre += (w < wid) ? warp_sum[w] : 0;
			tot += warp_sum[w];
		}
		if (i < n) out[i] = carry + pre + x - v;
		__syncthreads();
		if (threadIdx.x == 0) carry += tot;
		__syncthreads();
	}
	if (threadIdx.x == 0) out[n] = carry;
}

// Lookup table from micropolygon id to grid: entry k is the grid holding id
// k * 256 (thread per grid writes the entries whose id falls in it).
__global__ void id_grid_kernel(GridsDev g, int64_t nmps, int32_t* table) {
	const int gi = blockIdx.x * blockDim.x + threadIdx.x;
	if (gi >= g.ngrids) return;
	const int64_t s = g.mpbase[gi];
	const int64_t e = (gi + 1 < g.ngrids) ? g.mpbase[gi + 1] : nmps;
	for (int64_t k = (s + 255) >> 8; (k << 8) < e; ++k) table[k] = gi;
}

// Split's projection for grids flagged AQH_GRID_CAMERA: block per grid, every
// key's points replaced in place by their hybrid raster form, then the flag
// cleared so a later pass over the same arrays leaves them alone.
__global__ void project_grids_kernel(GridsDev g, float4* P, int32_t* flags, CamMatrix M) {
	const int gi = blockIdx.x;
	if (!(__ldg(g.flags + gi) & AQH_GRID_CAMERA)) return;
	const int64_t nv = (int64_t)(__ldg(g.cu + gi) + 1) * (__ldg(g.cv + gi) + 1);
	const int64_t n = nv * __ldg(g.nkeys + gi);
	float4* p = P + __ldg(g.pbase + gi);
	for (int64_t i = threadIdx.x; i < n; i += blockDim.x) p[i] = project_point(M.m, p[i]);
	__syncthreads();
	if (threadIdx.x == 0) flags[gi] &= ~AQH_GRID_CAMERA;
}

void launch_project_grids(const GridsDev& g, float4* P, int32_t* flags, const CamMatrix& m, cudaStream_t s) {
	if (g.ngrids == 0) return;
	project_grids_kernel<<<g.ngrids, 256, 0, s>>>(g, P, flags, m);
}

// CqBasicVec3 dot product (vector3d.h:602-606) and the back-face test of one
// vertex (micropolygon.cpp:451-459, 1013-1017).
__device__ __forceinline__ bool back_facing(float4 p, const float* ng, const float* n) {
	const float gx = __ldg(ng), gy = __ldg(ng + 1), gz = __ldg(ng + 2);
	float s = 1.0f;
	if (n) s = ((__ldg(n) * gx + __ldg(n + 1) * gy) + __ldg(n + 2) * gz < 0.0f) ? -1.0f : 1.0f;
	return ((s * gx) * p.x + (s * gy) * p.y) + (s * gz) * p.z >= 0.0f;
}

// CqMicroPolyGrid::Shade's and CqMotionMicroPolyGrid::Split's culling, one
// block per flagged grid, on camera-space P before projection.
__global__ void cull_grids_kernel(GridsDev g, const float* Ng, const float* N, long long nng, int zthr_black,
                                  uint8_t* culled, int32_t* err) {
	__shared__ int last_visible;
	const int gi = blockIdx.x;
	const int flags = __ldg(g.flags + gi);
	if (!(flags & (AQH_GRID_CULL_BACKFACING | AQH_GRID_CULL_TRANSPARENT))) return;
	const int cu = __ldg(g.cu + gi), cv = __ldg(g.cv + gi), nk = __ldg(g.nkeys + gi);
	const int nv = (cu + 1) * (cv + 1);
	const long long pb = __ldg(g.pbase + gi), cb = __ldg(g.cbase + gi), mb = __ldg(g.mpbase + gi);
	// the back-face test needs camera-space P: a grid already projected (a
	// device-resident grid after its first frame) keeps the result of none
	const bool bf = (flags & AQH_GRID_CULL_BACKFACING) && (flags & AQH_GRID_CAMERA);
	if (bf && (!Ng || pb < 0 || pb + (long long)nk * nv > nng)) {
		if (threadIdx.x == 0) atomicOr(err, 1);
		return;
	}
	// the trailing run of black Oi starts after the last vertex that is not black
	const bool tr = nk == 1 && (flags & AQH_GRID_CULL_TRANSPARENT) && g.Oi && !zthr_black;
	if (threadIdx.x == 0) last_visible = -1;
	__syncthreads();
	if (tr) {
		int mx = -1;
		for (int i = threadIdx.x; i < nv; i += blockDim.x) {
			float r, gg, b;
			if (g.colour3) {
				const float* o = reinterpret_cast<const float*>(g.Oi) + 3 * (cb + i);
				r = __ldg(o); gg = __ldg(o + 1); b = __ldg(o + 2);
			} else {
				const float4 o = __ldg(g.Oi + cb + i);
				r = o.x; gg = o.y; b = o.z;
			}
			if (!(r == 0.0f && gg == 0.0f && b == 0.0f)) mx = i;
		}
		atomicMax(&last_visible, mx);
	}
	__syncthreads();
	const int run_start = tr ? last_visible + 1 : nv;
	for (int m = threadIdx.x; m < cu * cv; m += blockDim.x) {
		const int ia = (m / cu) * (cu + 1) + (m % cu);
		bool c = false;
		if (bf) {
			int facing_away = 0;
			for (int k = 0; k < nk; ++k) {
				const long long e = pb + (long long)k * nv + ia;
				facing_away += back_facing(__ldg(g.P + e), Ng + 3 * e, N ? N + 3 * e : nullptr) ? 1 : 0;
			}
			c = facing_away == nk;
		}
		c = c || ia >= run_start;
		if (c) culled[mb + m] = 1;
	}
}

void launch_cull_grids(const GridsDev& g, const float* Ng, const float* N, long long nng, int zthr_black,
                       uint8_t* culled, int32_t* err, cudaStream_t s) {
	if (g.ngrids == 0) return;
	cull_grids_kernel<<<g.ngrids, 256, 0, s>>>(g, Ng, N, nng, zthr_black, culled, err);
}

// CqMicroPolyGrid::Split / CqMotionMicroPolyGrid::Split trimming
// (micropolygon.cpp:754-835, 1056-1130), one block per grid: the corners'
// surface parameters (index, index+1, index+cu+2, index+cu+1) are classified
// against the grid's trim set, inverted for the "outside" sense; all four
// trimmed with no edge crossing a loop drops the micropolygon, any trimmed
// marks it for the per-hit test.
__global__ void trim_mark_kernel(GridsDev g, long long nuv, uint8_t* mark, uint8_t* culled, int32_t* err) {
	const int gi = blockIdx.x;
	const int set = __ldg(g.trim.grid_set + gi);
	if (set < 0) return;
	const int cu = __ldg(g.cu + gi), cv = __ldg(g.cv + gi);
	const long long cb = __ldg(g.cbase + gi);
	if (cb < 0 || cb + (long long)(cu + 1) * (cv + 1) > nuv) {
		if (threadIdx.x == 0) atomicOr(err, 1);
		return;
	}
	const bool outside = (__ldg(g.flags + gi) & 64) != 0;
	const int l0 = __ldg(g.trim.set_first + set), l1 = __ldg(g.trim.set_first + set + 1);
	const long long mb = __ldg(g.mpbase + gi);
	const int nm = cu * cv;
	for (int m = threadIdx.x; m < nm; m += blockDim.x) {
		if (culled[mb + m]) continue;
		const long long c = cb + (long long)(m / cu) * (cu + 1) + (m % cu);
		const float2 A = __ldg(g.trim.uv + c), B = __ldg(g.trim.uv + c + 1);
		const float2 C = __ldg(g.trim.uv + c + cu + 2), D = __ldg(g.trim.uv + c + cu + 1);
		const bool tA = trim_point(g.trim.pts, g.trim.loop_first, l0, l1, A.x, A.y) != outside;
		const bool tB = trim_point(g.trim.pts, g.trim.loop_first, l0, l1, B.x, B.y) != outside;
		const bool tC = trim_point(g.trim.pts, g.trim.loop_first, l0, l1, C.x, C.y) != outside;
		const bool tD = trim_point(g.trim.pts, g.trim.loop_first, l0, l1, D.x, D.y) != outside;
		if (tA && tB && tC && tD && !trim_line(g.trim.pts, g.trim.loop_first, l0, l1, A, B) &&
		    !trim_line(g.trim.pts, g.trim.loop_first, l0, l1, B, C) &&
		    !trim_line(g.trim.pts, g.trim.loop_first, l0, l1, C, D) &&
		    !trim_line(g.trim.pts, g.trim.loop_first, l0, l1, D, A)) {
			culled[mb + m] = 1;
			continue;
		}
		if (tA || tB || tC || tD) mark[mb + m] = 1;
	}
}

void launch_trim_mark(const GridsDev& g, long long nuv, uint8_t* mark, uint8_t* culled, int32_t* err, cudaStream_t s) {
	if (g.ngrids == 0) return;
	trim_mark_kernel<<<g.ngrids, 128, 0, s>>>(g, nuv, mark, culled, err);
}

void launch_id_grid(const GridsDev& g, int64_t nmps, int32_t* table, cudaStream_t s) {
	if (g.ngrids == 0) return;
	id_grid_kernel<<<(g.ngrids + 255) / 256, 256, 0, s>>>(g, nmps, table);
}

void launch_grid_rects(const FrameParams& fp, const GridsDev& g, const BinBuffers& b, cudaStream_t s) {
	if (g.ngrids == 0) return;
	const int wpb = kBlock / 32;
	grid_rects_kernel<<<(g.ngrids + wpb - 1) / wpb, kBlock, 0, s>>>(fp, g, b.grid_rect, b.grid_minz, b.strips, b.tri,
	                                                                     b.redo_next);
}

void launch_st_count(const FrameParams& fp, const GridsDev& g, BinBuffers& b, cudaStream_t s) {
	dim3 grid(fp.nstx * fp.nsty, b.nranges);
	st_count_kernel<<<grid, kBlock, 0, s>>>(fp, g.ngrids, b.grid_rect, b.nranges, b.range_size, b.st_count);
}

// How far below its min z a hit of a micropolygon can lie, or false where no
// bound is known (an irregular one).
//
// The depth of a hit is the bilinear mix of the corner depths at the (u, v) of
// two Newton steps from the centre C.  With M1 = E + G/2, M2 = F + G/2, area A
// = M1 x M2 and G = g1 M1 + g2 M2, the first step lands at (x, y) = (u - 1/2,
// v - 1/2) with M1 x + M2 y = P - C, affine in the sample position P: at the
// corners x = +-1/2 +- g1/4 and y = +-1/2 +- g2/4, so |x| <= X = 1/2 + |g1|/4
// and |y| <= Y over the corners' hull, which holds every point the edge tests
// accept.  The second step's determinant there is A (1 + g2 x + g1 y), also
// affine, so at least A kappa with kappa its least value at the corners, 1 +-
// (g1 + g2)/2 + g1 g2/2 and 1 +- (g1 - g2)/2 - g1 g2/2, and its step is -(g1,
// g2) x y / (det / A).  Hence |u - 1/2| <= U = X + |g1| X Y / kappa, V alike,
// the weights' absolute values sum to at most W = max(1, 2U) max(1, 2V), the
// negative ones to (W - 1)/2, and the depth is at least min z - (W - 1)/2 (max
// z - min z).  (The bound below charges W/2, half a depth range more than
// that.)  Rounding: positions carry 2^-20 of the coordinates into the steps
// (eta below; a step divides it by kappa), the edge tests accept points up to
// 2^-10 / c < 1/32 of a cell outside for quads with 32 A >= L^2 (L the extent)
// whose corners turn by at least c A, c = 1 - (|g1| + |g2|)/2 >= 0.05, and the
// mix itself rounds by 2^-19 W max|z|.  Quads with kappa < 0.05 or c < 0.05
// (folded, nearly singular: one in 2,000 of a grid of unit spacing and +-0.3
// jitter), thin ones and anything not finite are irregular.
//
// Corners that move (rho > 0) are within rho, per coordinate, of a translate of
// the given ones: E and F then move by 2 rho, G, M1 and M2 by 4 rho, and the
// areas by the products' worth of that, against which the bounds are taken.
__device__ __forceinline__ bool depth_slack(V3f a, V3f b, V3f c, V3f d, float mnz, float mxz, float rho, float far,
                                            float& slack) {
	const float mnx = fminf(fminf(a.x, b.x), fminf(c.x, d.x)), mxx = fmaxf(fmaxf(a.x, b.x), fmaxf(c.x, d.x));
	const float mny = fminf(fminf(a.y, b.y), fminf(c.y, d.y)), mxy = fmaxf(fmaxf(a.y, b.y), fmaxf(c.y, d.y));
	const float sum = ((a.x + b.x) + (c.x + d.x)) + ((a.y + b.y) + (c.y + d.y)) + ((a.z + b.z) + (c.z + d.z));
	const float L = (mxx - mnx) + (mxy - mny) + 4.0f * rho;
	const float ex = b.x - a.x, ey = b.y - a.y, fx = c.x - a.x, fy = c.y - a.y;
	const float gx = (d.x - c.x) - ex, gy = (d.y - c.y) - ey;
	const float m1x = ex + 0.5f * gx, m1y = ey + 0.5f * gy, m2x = fx + 0.5f * gx, m2y = fy + 0.5f * gy;
	const float r4 = 4.0f * rho, r32 = 2.0f * r4 * r4;
	const float n1 = fabsf(m1x) + fabsf(m1y), n2 = fabsf(m2x) + fabsf(m2y), ng = fabsf(gx) + fabsf(gy);
	const float cross = m1x * m2y - m1y * m2x;
	const float area = fabsf(cross) - (r4 * (n1 + n2) + r32);
	if (!(32.0f * area >= L * L && L > 1e-12f && L < 1e6f && fabsf(sum) < 1e30f)) return false;  // NaN too
	const float ia = 1.0f / area;
	// g1 and g2 of the given corners, and their magnitudes with the movement
	const float s1 = (gx * m2y - gy * m2x) / cross, s2 = (m1x * gy - m1y * gx) / cross;
	const float g1 = (fabsf(gx * m2y - gy * m2x) + (r4 * (ng + n2) + r32)) * ia;
	const float g2 = (fabsf(m1x * gy - m1y * gx) + (r4 * (ng + n1) + r32)) * ia;
	const float turn = 1.0f - 0.5f * (g1 + g2);
	const float cmax = fmaxf(fmaxf(fabsf(mnx), fabsf(mxx)), fmaxf(fabsf(mny), fabsf(mxy))) + far;
	const float eta = 9.5367432e-7f * (cmax + 4.0f * L) * L * ia;  // 2^-20
	const float out = 0.03125f + 2.0f * eta;
	const float X = 0.5f + 0.25f * g1 + out, Y = 0.5f + 0.25f * g2 + out;
	// the movement changes s1 by at most t1 = r (1 + |s1|), r the areas' relative
	// change, and the corner values by at most (t1 + t2)(1 + max g)/2 + t1 t2/2
	const float t1 = g1 - fabsf(s1) + 2.0f * (fabsf(cross) - area) * ia * fabsf(s1);
	const float t2 = g2 - fabsf(s2) + 2.0f * (fabsf(cross) - area) * ia * fabsf(s2);
	const float moved = 0.5f * (t1 + t2) * (1.0f + fmaxf(g1, g2)) + 0.5f * (t1 * t2);
	const float h = 0.5f * (s1 * s2);
	const float kappa = 1.0f + fminf(h - 0.5f * fabsf(s1 + s2), -h - 0.5f * fabsf(s1 - s2)) - moved -
	                    (g1 + g2) * out - 0.001f;
	if (!(kappa >= 0.05f && turn >= 0.05f)) return false;
	const float ik = 1.0f / kappa;
	const float U = X + (g1 * (X * Y) + 8.0f * eta) * ik, V = Y + (g2 * (X * Y) + 8.0f * eta) * ik;
	const float W = fmaxf(1.0f, 2.0f * U) * fmaxf(1.0f, 2.0f * V);
	slack = 0.501f * W * (mxz - mnz) + 1.9073486e-6f * W * fmaxf(fabsf(mnz), fabsf(mxz));  // 2^-19
	return slack < 1e30f;
}

// WPG warps per grid, 32 micropolygons a warp at a time: the grid's largest
// slack and which micropolygons are irregular.  Few grids spread theirs over a
// block (195 grids: 11 us with a warp each, 4 with eight); from some thousands
// on the warps of other grids fill the SMs and a block each costs more than
// it gives (200,000 grids: 318 us and 505).
constexpr int kSlackWarps = 8;
template <int WPG>
__global__ void __launch_bounds__(32 * kSlackWarps) grid_slack_kernel(GridsDev g, BinBuffers bb) {
	__shared__ float most_s[kSlackWarps];
	__shared__ int nirr_s[kSlackWarps];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wid = warp % WPG;
	const int gi = blockIdx.x * (kSlackWarps / WPG) + warp / WPG;
	if (gi >= g.ngrids) return;  // whole warps; with WPG > 1 the block
	const int cu = __ldg(g.cu + gi), cv = __ldg(g.cv + gi), n = cu * cv;
	const bool fits = cu <= 1024 && cv <= 1024 && n <= 32 * kIrrWords;
	const float4* P = g.P + __ldg(g.pbase + gi);
	float most = 0.0f;
	int nirr = 0;
	if (fits)
		for (int m0 = wid * 32; m0 < n; m0 += 32 * WPG) {
			const int m = m0 + lane;
			bool irr = false;
			if (m < n) {
				const int iv = m / cu, i = iv * (cu + 1) + (m - iv * cu);
				float slack = 0.0f;
				const V3f a = ld3(P, i), b = ld3(P, i + 1), c = ld3(P, i + cu + 1), d = ld3(P, i + cu + 2);
				irr = !depth_slack(a, b, c, d, fminf(fminf(a.z, b.z), fminf(c.z, d.z)),
				                   fmaxf(fmaxf(a.z, b.z), fmaxf(c.z, d.z)), 0.0f, 0.0f, slack);
				if (!irr) most = fmaxf(most, slack);
			}
			const uint32_t w = __ballot_sync(0xffffffffu, irr);
			if (lane == 0) bb.irregular[(long long)gi * kIrrWords + (m0 >> 5)] = w;
			nirr += __popc(w);
		}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
	if (WPG > 1) {
		static_assert(WPG == 1 || WPG == kSlackWarps, "a block holds one grid's warps");
		if (lane == 0) {
			most_s[wid] = most;
			nirr_s[wid] = nirr;
		}
		__syncthreads();
		if (wid == 0 && lane == 0)
			for (int w = 1; w < WPG; ++w) {
				most = fmaxf(most, most_s[w]);
				nirr += nirr_s[w];
			}
	}
	if (lane != 0 || wid != 0) return;
	bb.grid_slack[gi] = most;
	bb.grid_nirr[gi] = fits ? nirr : -1;
	if (!fits) nirr = n;
	if (nirr > 0) atomicAdd(bb.nirr_total, nirr);
}

// One block per super-tile: its grid list by nearest depth, in 1,024 buckets
// between the list's nearest and farthest (the order within a bucket is left
// open: no result depends on the order, only how early the near grids come).
constexpr int kDepthBuckets = 1024;
__global__ void __launch_bounds__(kDepthBuckets) depth_order_kernel(BinBuffers bb) {
	__shared__ int count[kDepthBuckets];
	__shared__ int warp_sum[32];
	__shared__ uint32_t lo_s, hi_s;
	const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
	const int beg = bb.st_offset[blockIdx.x * bb.nranges];
	const int end = (int)min((long long)bb.st_offset[(blockIdx.x + 1) * bb.nranges], (long long)bb.list_capacity);
	auto depth = [&](int i) -> uint32_t {  // ordered bits of the grid's nearest depth
		const uint32_t u = __float_as_uint(__ldg(bb.grid_minz + bb.st_list[i]));
		return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
	};
	count[t] = 0;
	if (t == 0) {
		lo_s = 0xffffffffu;
		hi_s = 0u;
	}
	__syncthreads();
	uint32_t lo = 0xffffffffu, hi = 0u;
	for (int i = beg + t; i < end; i += blockDim.x) {
		const uint32_t k = depth(i);
		lo = min(lo, k);
		hi = max(hi, k);
	}
	lo = __reduce_min_sync(0xffffffffu, lo);
	hi = __reduce_max_sync(0xffffffffu, hi);
	if (lane == 0) {
		atomicMin(&lo_s, lo);
		atomicMax(&hi_s, hi);
	}
	__syncthreads();
	lo = lo_s;
	const float scale = hi_s > lo ? (float)(kDepthBuckets - 1) / (float)(hi_s - lo) : 0.0f;
	auto bucket = [&](uint32_t k) -> int { return min(kDepthBuckets - 1, (int)((float)(k - lo) * scale)); };
	for (int i = beg + t; i < end; i += blockDim.x) atomicAdd(&count[bucket(depth(i))], 1);
	__syncthreads();
	// exclusive scan of the counts, a bucket per thread
	const int v = count[t];
	int x = v;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const int y = __shfl_up_sync(0xffffffffu, x, o);
		if (lane >= o) x += y;
	}
	if (lane == 31) warp_sum[wid] = x;
	__syncthreads();
	int pre = 0;
	for (int w = 0; w < wid; ++w) pre += warp_sum[w];
	count[t] = beg + pre + x - v;
	__syncthreads();
	for (int i = beg + t; i < end; i += blockDim.x)
		bb.st_sorted[atomicAdd(&count[bucket(depth(i))], 1)] = bb.st_list[i];
}

void launch_depth_order(const FrameParams& fp, const GridsDev& g, const BinBuffers& b, cudaStream_t s) {
	if (g.ngrids == 0) return;
	if (!b.grid_slack) {
		// moving frames: the slacks come with the staging bounds
	} else if (g.ngrids < 4096)
		grid_slack_kernel<kSlackWarps><<<g.ngrids, 32 * kSlackWarps, 0, s>>>(g, b);
	else
		grid_slack_kernel<1><<<(g.ngrids + kSlackWarps - 1) / kSlackWarps, 32 * kSlackWarps, 0, s>>>(g, b);
	depth_order_kernel<<<fp.nstx * fp.nsty, kDepthBuckets, 0, s>>>(b);
}

void launch_scan_i32(const int32_t* in, int32_t* out, int n, int32_t*, cudaStream_t s) {
	scan_i32_kernel<<<1, 1024, 0, s>>>(in, out, n);
}

void launch_st_write(const FrameParams& fp, const GridsDev& g, BinBuffers& b, cudaStream_t s) {
	dim3 grid(fp.nstx * fp.nsty, b.nranges);
	st_write_kernel<<<grid, kBlock, 0, s>>>(fp, g.ngrids, b.grid_rect, b.nranges, b.range_size, b.st_offset,
	                                        b.st_list, (long long)b.list_capacity);
}

// The least depth at which micropolygon m can be hit at any time and lens
// position, -inf where no bound is known (depth_slack): its corners at a time
// between two keys are a mix of theirs, so they stay within rho of a translate
// of key 0's, rho the most any corner's displacement differs from corner 0's
// plus, under depth of field, the spread of the circles of confusion over its
// depths (all in front of the eye) times the lens offset, at most 1.
__device__ __forceinline__ float mb_hit_depth(const FrameParams& fp, const GridsDev& g, int gid, int m,
                                              const MbStageBound& sb) {
	const int cu = __ldg(g.cu + gid), nk = __ldg(g.nkeys + gid);
	const long long nv = (long long)(cu + 1) * (__ldg(g.cv + gid) + 1);
	const float4* P = g.P + __ldg(g.pbase + gid) + (m / cu) * (cu + 1) + m % cu;
	const V3f a = ld3(P, 0), b = ld3(P, 1), c = ld3(P, cu + 1), d = ld3(P, cu + 2);
	float rho = 0.0f, far = 0.0f;
	for (int k = 1; k < nk; ++k) {
		const float4* Q = P + k * nv;
		const V3f a1 = ld3(Q, 0), b1 = ld3(Q, 1), c1 = ld3(Q, cu + 1), d1 = ld3(Q, cu + 2);
		const float dx = a1.x - a.x, dy = a1.y - a.y;
		far = fmaxf(far, fmaxf(fabsf(dx), fabsf(dy)));
		auto off = [&](V3f p, V3f q) { rho = fmaxf(rho, fmaxf(fabsf((q.x - p.x) - dx), fabsf((q.y - p.y) - dy))); };
		off(b, b1);
		off(c, c1);
		off(d, d1);
		// NaN drops out of the maxima
		if (!(fabsf((a1.x + a1.y + a1.z) + (b1.x + b1.y + b1.z) + (c1.x + c1.y + c1.z) + (d1.x + d1.y + d1.z)) < 1e30f))
			return -INFINITY;
	}
	if (fp.use_dof) {
		if (!(sb.mnz > 0.0f && sb.mxz < FLT_MAX)) return -INFINITY;
		const float2 c1 = coc(sb.mnz, fp.dof_mult, fp.dof_inv_fd, fp.dof_scale_x, fp.dof_scale_y);
		const float2 c2 = coc(sb.mxz, fp.dof_mult, fp.dof_inv_fd, fp.dof_scale_x, fp.dof_scale_y);
		const float cx = fmaxf(fabsf(c1.x), fabsf(c2.x)), cy = fmaxf(fabsf(c1.y), fabsf(c2.y));
		// 1/z - 1/focus keeps its sign over the depths, or the circle passes through 0
		const bool side = (1.0f / sb.mnz - fp.dof_inv_fd > 0.0f) == (1.0f / sb.mxz - fp.dof_inv_fd > 0.0f);
		const float lx = side ? fminf(fabsf(c1.x), fabsf(c2.x)) : 0.0f, ly = side ? fminf(fabsf(c1.y), fabsf(c2.y)) : 0.0f;
		const float spread = fmaxf(cx - lx, cy - ly) + 1e-6f * fmaxf(cx, cy);
		rho += 1.01f * spread;
		far += 1.01f * fmaxf(cx, cy);
		if (!(spread < 1e6f)) return -INFINITY;
	}
	// roundings of the corners' mix and shift
	rho += 4.7683716e-7f * (fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(d.x), fabsf(d.y))) + 2.0f * far);  // 2^-21
	float slack = 0.0f;
	if (!depth_slack(a, b, c, d, sb.mnz, sb.mxz, rho, far, slack)) return -INFINITY;
	return sb.mnz - slack;
}

// One warp per grid: the staging bound of each of its micropolygons, read by
// every motion sampling tile the micropolygon may reach instead of its key
// vertices.  stride 2: each bound is followed by the micropolygon's path.
// nirr_total: the frame is sampled near to far, and the bound's least depth is
// that of its hits (mb_hit_depth) instead of its vertices.
__global__ void mb_stage_bounds_kernel(FrameParams fp, GridsDev g, int4* out, int stride, int32_t* nirr_total) {
	const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int lane = threadIdx.x & 31;
	if (warp >= g.ngrids) return;
	const int n = __ldg(g.cu + warp) * __ldg(g.cv + warp);
	int4* o = out + __ldg(g.mpbase + warp) * stride;
	int nirr = 0;
	for (int m = lane; m < n; m += 32) {
		int4 path;
		MbStageBound b = mb_stage_bound(fp, g, warp, m, stride == 2 ? &path : nullptr);
		if (nirr_total) {
			b.mnz = mb_hit_depth(fp, g, warp, m, b);
			if (b.keep && b.mnz == -INFINITY) ++nirr;
		}
		o[(long long)m * stride] = pack_stage_bound(b);
		if (stride == 2) o[(long long)m * 2 + 1] = path;
	}
	if (nirr_total) {
		nirr = __reduce_add_sync(0xffffffffu, nirr);
		if (lane == 0 && nirr > 0) atomicAdd(nirr_total, nirr);
	}
}

void launch_mb_stage_bounds(const FrameParams& fp, const GridsDev& g, const BinBuffers& b, cudaStream_t s) {
	if (g.ngrids <= 0) return;
	const int wpb = kBlock / 32;
	mb_stage_bounds_kernel<<<(g.ngrids + wpb - 1) / wpb, kBlock, 0, s>>>(fp, g, b.mp_bounds, b.mp_stride,
	                                                                        b.redo ? b.nirr_total : nullptr);
}

}  // namespace aqh
