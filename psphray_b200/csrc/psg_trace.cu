// Ray traversal; replaces rt_trace() raytrace.c:153-210 and the per-ray
// sort of trace() loop.c:375-386.
//
// The traversal walks the level-order copy of the octree (the 8 children of
// a cell contiguous), one warp per ray with a stack of crossed cells in
// shared memory; the set of crossed cells and the hits are the reference's
// parent/sibling walk's, found in another order. Hits go to per-ray slabs in
// discovery order and are then sorted per ray by (d, ipar).
#include <cub/cub.cuh>

#include <stdlib.h>
#include <string.h>

#include <vector>

#include "psg_internal.cuh"
#include "psg_bsort.cuh"
#include "psg_scan.cuh"
#include "psg_solve.cuh"

namespace {

// A ray as the traversal uses it. up: the direction's component is positive.
// Mirrored along the axes where it is not, every ray goes up: sg is the
// axis's sign, os the mirrored start negated, ad the mirrored direction and
// reach the mirrored displacement to its end.
struct RayGeom {
	float s[3], dir[3];
	float sg[3], os[3], ad[3], reach[3];
	bool up[3];
	float margin;      // of line_test(), per squared distance
};

__device__ __forceinline__ RayGeom load_ray(const psg_ray *__restrict__ rays, size_t r) {
	RayGeom g;
	const psg_ray &ry = rays[r];
	const float dist = (float)ry.length;      // rt_trace() takes the length as float
	float dir2 = 0.0f;
#pragma unroll
	for (int a = 0; a < 3; a++) {
		g.s[a] = ry.s[a];
		g.dir[a] = ry.dir[a];
		g.up[a] = g.dir[a] > 0.0f;
		g.sg[a] = g.up[a] ? 1.0f : -1.0f;
		g.os[a] = -g.sg[a] * g.s[a];
		g.ad[a] = g.sg[a] * g.dir[a];
		g.reach[a] = g.sg[a] * rn_fmul(dist, g.dir[a]);
		dir2 += g.dir[a] * g.dir[a];
	}
	g.margin = 2e-6f * fmaxf(1.0f, dir2);
	return g;
}

// pluecker_() pluecker-sse.c:28-198. The reference's 8 hand-written sign
// classes are mirror images of one another, and mirroring changes no
// magnitude: each product and difference rounds once, in float, to the
// reference's value or its negative, and each comparison is the reference's
// or its mirror image. lo.w and hi.w are not looked at.
__device__ __forceinline__ bool segment_hits_box(const RayGeom &g, const float4 lo, const float4 hi) {
	const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
	float n[3], f[3];      // the near and the far face, seen from the start
	bool miss = false;
#pragma unroll
	for (int a = 0; a < 3; a++) {
		n[a] = __fmaf_rn(g.sg[a], g.up[a] ? l[a] : h[a], g.os[a]);      // (one rounding: the product is exact)
		f[a] = __fmaf_rn(g.sg[a], g.up[a] ? h[a] : l[a], g.os[a]);
		miss = miss | (f[a] < 0.0f) | (rn_fsub(n[a], g.reach[a]) > 0.0f);
	}
#pragma unroll
	for (int q = 0; q < 3; q++) {
		const int i = q == 2 ? 1 : 0;
		const int j = q == 0 ? 1 : 2;
		miss = miss | (rn_fmul(g.ad[i], f[j]) < rn_fmul(g.ad[j], n[i])) | (rn_fmul(g.ad[i], n[j]) > rn_fmul(g.ad[j], f[i]));
	}
	return !miss;
}

// The line test of raytrace.c:168-195: float differences and products,
// double sums (in the order the reference's build adds them: y and z
// first, then x; its -ffast-math lets the compiler reassociate the loop,
// which rounds differently in rare cases, by 1 ulp of d). d: the distance to
// the centre; r2: the squared distance to the line; a hit unless sml^2 < r2.
struct HitDist {
	double d, proj;
	__device__ __forceinline__ double r2() const { return rn_dmul(rn_dsub(d, proj), rn_dadd(d, proj)); }
};
__device__ __forceinline__ double hit_d(const float s[3], const float4 q) {
	const float dx = rn_fsub(q.x, s[0]), dy = rn_fsub(q.y, s[1]), dz = rn_fsub(q.z, s[2]);
	return __dsqrt_rn(rn_dadd((double)rn_fmul(dx, dx), rn_dadd((double)rn_fmul(dy, dy), (double)rn_fmul(dz, dz))));
}
__device__ __forceinline__ double hit_proj(const float s[3], const float dir[3], const float4 q) {
	const float dx = rn_fsub(q.x, s[0]), dy = rn_fsub(q.y, s[1]), dz = rn_fsub(q.z, s[2]);
	return rn_dadd((double)rn_fmul(dx, dir[0]), rn_dadd((double)rn_fmul(dy, dir[1]), (double)rn_fmul(dz, dir[2])));
}

// Whether the line meets the particle, decided in float where that is sure:
// r2f = fl(d2f - fl(pf^2)) differs from the exact test's r2 by at most 8
// roundings of 2^-24 of d2 max(1, |dir|^2) (two each in the sums of d2f and
// pf, whose terms are the exact test's own, doubled by the square, one each
// in the square and the difference): 4.8e-7. Beyond a margin of 2e-6 the
// exact test decides alike; within it (or with squares near the smallest
// floats, or a NaN, which marks flagged particles) the exact one is made.
__device__ __forceinline__ bool line_test(const RayGeom &g, const float4 q, int p, const uint32_t *__restrict__ lidx) {
	const float dx = rn_fsub(q.x, g.s[0]), dy = rn_fsub(q.y, g.s[1]), dz = rn_fsub(q.z, g.s[2]);
	const float pf = __fadd_rn(__fadd_rn(rn_fmul(dx, g.dir[0]), rn_fmul(dy, g.dir[1])), rn_fmul(dz, g.dir[2]));
	const float d2f = __fadd_rn(__fadd_rn(rn_fmul(dx, dx), rn_fmul(dy, dy)), rn_fmul(dz, dz));
	const float s2 = rn_fmul(q.w, q.w);
	const float over = __fsub_rn(__fsub_rn(d2f, rn_fmul(pf, pf)), s2);
	const float m = d2f > 1e-30f ? g.margin * d2f : __int_as_float(0x7f800000);
	if (over < -m) return true;
	if (over > m) return false;
	if (__ldg(&lidx[p]) & PSG_INVALID_BIT) return false;
	const HitDist h{hit_d(g.s, q), hit_proj(g.s, g.dir, q)};
	return !((double)s2 < h.r2());
}

// Candidates listed in shared memory (leaf-order particle positions), tested
// 32 at a time; the hits go to the ray's slab in order of discovery, as
// positions alone: their distances are computed by the sort, with every
// lane busy.
// With count (several warps share the ray) the slab's places are taken from it.
__device__ __forceinline__ void test_candidates(const RayGeom &g, const int *list, int total,
		const float4 *__restrict__ lpsml, const uint32_t *__restrict__ lidx, uint32_t *__restrict__ slab, size_t scap,
		uint32_t &nh, uint32_t *__restrict__ count, int lane, unsigned lt_mask) {
	for (int k0 = 0; k0 < total; k0 += 32) {
		const int k = k0 + lane;
		bool acc = false;
		int p = 0;
		if (k < total) {
			p = list[k];
			acc = line_test(g, __ldg(&lpsml[p]), p, lidx);
		}
		const unsigned bal = __ballot_sync(0xffffffffu, acc);
		if (count) {
			if (!bal) continue;
			if (lane == 0) nh = atomicAdd(count, (uint32_t)__popc(bal));
			nh = __shfl_sync(0xffffffffu, nh, 0);
		}
		const size_t q = nh + __popc(bal & lt_mask);
		if (acc && q < scap) slab[q] = (uint32_t)p;
		nh += __popc(bal);
	}
}

// One warp per ray over the level-order tree, whose 8 children of a cell are
// contiguous. The warp keeps a stack (shared memory) of crossed internal
// cells; each step pops up to 4 of them and tests their 32 children at once,
// one per lane, with the reference's segment-box test; crossed internal
// children are pushed, crossed leaves list their particles for the line
// test. The cells tested are exactly the children of crossed cells, as in
// the reference's walk (raytrace.c:160-208); only the order differs, and the
// per-ray sort makes the output independent of it. The stack cannot exceed
// 4 + 28 entries per tree level (592 at 21 levels); an overflow would raise
// PSG_ST_STACK instead of losing cells.
//
// Bound by instruction issue: on the 2M-particle field a ray of 690 hits
// takes 69 rounds of cells and 60 of candidates. So the box test is one
// branch-free form for all sign classes, the line test is FP32 but near its
// boundary (2 candidates a ray), hits are stored as positions (4 bytes, not
// 20), a leaf's place in the list comes from ballots and its particles are
// listed by predicated stores, and 48 registers leave 40 warps per
// multiprocessor. 65536 rays: 1.91 -> 1.39 ms; 65536 on 16.8M particles (1200
// hits each) 5.0 -> 3.2 ms; 102400 on 64^3 (123 each) 0.68 -> 0.51 ms.
// PPC: the leaves' capacity where it is 8 (the reference's), else 0 and the
// argument.
//
// SPLIT: with fewer rays than resident warps (a host's few rays) a ray's walk is a serial chain of L2 round
// trips on an idle machine, so it is divided among nstart warps, each from one
// cell of an upper level of the tree on (from index start0; plan_trace
// chooses the level, which the tree has in full, so that levels 1, 2 and 3
// start at cells 1, 9 and 73). 32 rays on 32^3: 47 -> 19 us; 1024 rays on
// 64^3: 162 -> 109 us.
#define TR_STACK 640
#define TR_REGS 48
#define TR_MAX_WARPS 16      // warps per block: ctx->tune.trace_warps, at most this

template <int PPC, bool SPLIT>
__global__ void __maxnreg__(TR_REGS) k_trace_stack(const psg_ray *__restrict__ rays, size_t nray,
		const float4 *__restrict__ wlo, const float4 *__restrict__ whi,
		const float4 *__restrict__ lpsml, const uint32_t *__restrict__ lidx, int ppc_any,
		uint32_t *__restrict__ count, size_t scap, uint32_t *__restrict__ slab_ipar,
		unsigned long long *__restrict__ next_ray, uint32_t *__restrict__ status, const unsigned *__restrict__ nlim,
		int start0, int nstart) {
	extern __shared__ int tr_smem[];
	const int ppc = PPC ? PPC : ppc_any;
	// rays past *nlim (when given: the recombination path's emitted count)
	// are not traced; their counts stay as zeroed
	if (nlim) nray = min(nray, (size_t)*nlim);
	const int lane = threadIdx.x & 31;
	const int wib = threadIdx.x >> 5;
	int *stack = tr_smem + wib * (TR_STACK + 32 * ppc + 32);
	int *list = stack + TR_STACK;      // candidates waiting for a full round of 32
	const unsigned lt_mask = (1u << lane) - 1u;
	// persistent warps: each takes the next ray from a shared counter, so a
	// block never idles behind its longest ray
	for (;;) {
	unsigned long long rr = 0;
	if (lane == 0) rr = atomicAdd(next_ray, 1ull);
	rr = __shfl_sync(0xffffffffu, rr, 0);
	if (rr >= (SPLIT ? nray * nstart : nray)) break;
	const size_t r = SPLIT ? (size_t)rr / (unsigned)nstart : (size_t)rr;
	const int root = SPLIT ? start0 + (int)((size_t)rr - r * (unsigned)nstart) : 0;
	const RayGeom g = load_ray(rays, r);
	uint32_t *slab = slab_ipar + r * scap;
	uint32_t *const shared_count = SPLIT ? count + r : nullptr;
	uint32_t nh = 0;
	int sp = 0, nbuf = 0;
	bool overflow = false;
	{
		const float4 lo = __ldg(&wlo[root]), hi = __ldg(&whi[root]);
		bool hit = segment_hits_box(g, lo, hi);
		if (SPLIT)      // and its ancestors, as the walk from the root tests them
			for (int c = root; c > 0 && hit;) {
				c = (c - 1) >> 3;
				hit = segment_hits_box(g, __ldg(&wlo[c]), __ldg(&whi[c]));
			}
		if (hit) {
			const int w = __float_as_int(lo.w);
			if (w >= 0) {
				if (lane == 0) stack[0] = w;
				sp = 1;
			} else {
				const int cnt = min(-1 - w, ppc), ps = __float_as_int(hi.w);
				for (int k = lane; k < cnt; k += 32) list[k] = ps + k;
				__syncwarp();
				test_candidates(g, list, cnt, lpsml, lidx, slab, scap, nh, shared_count, lane, lt_mask);
			}
		}
	}
	__syncwarp();
	while (sp > 0) {
		const int k = min(sp, 4);
		const int node = lane >> 3;
		const bool valid = node < k;
		const int c = valid ? stack[sp - k + node] + (lane & 7) : 0;
		__syncwarp();
		sp -= k;
		const float4 lo = __ldg(&wlo[c]), hi = __ldg(&whi[c]);
		const bool hit = valid & segment_hits_box(g, lo, hi);
		const int w = __float_as_int(lo.w);
		const unsigned bi = __ballot_sync(0xffffffffu, hit && w >= 0);
		if (hit && w >= 0) {
			const int pos = sp + __popc(bi & lt_mask);
			if (pos < TR_STACK) stack[pos] = w;
		}
		sp += __popc(bi);
		if (sp > TR_STACK) { overflow = true; sp = TR_STACK; }
		// the crossed leaves' particles behind those waiting: each leaf's
		// place from the ballots of its count's bits
		const int cnt = (hit && w < 0) ? min(-1 - w, ppc) : 0;
		int before = 0;
#pragma unroll
		for (int bit = 0; bit < (PPC ? 4 : 8); bit++)
			before += __popc(__ballot_sync(0xffffffffu, (cnt >> bit) & 1) & lt_mask) << bit;
		const int ps = __float_as_int(hi.w);
		int *const mine = list + nbuf + before;
		if (PPC) {
#pragma unroll
			for (int q = 0; q < PPC; q++)
				if (q < cnt) mine[q] = ps + q;
		} else {
			for (int q = 0; q < cnt; q++) mine[q] = ps + q;
		}
		nbuf += __shfl_sync(0xffffffffu, before + cnt, 31);
		__syncwarp();
		// line tests only in full rounds of 32; the rest waits in the list
		if (nbuf >= 32) {
			const int full = nbuf & ~31, rem = nbuf - full;
			test_candidates(g, list, full, lpsml, lidx, slab, scap, nh, shared_count, lane, lt_mask);
			__syncwarp();
			const int keep = lane < rem ? list[full + lane] : 0;
			__syncwarp();
			if (lane < rem) list[lane] = keep;
			nbuf = rem;
			__syncwarp();
		}
	}
	if (nbuf) test_candidates(g, list, nbuf, lpsml, lidx, slab, scap, nh, shared_count, lane, lt_mask);
	if (lane == 0) {
		if (!SPLIT) count[r] = nh;
		if (overflow) atomicOr(status, PSG_ST_STACK);
	}
	__syncwarp();
	}
}

// With cap (a call without host reads), a total above the hit buffers'
// capacity empties every list instead (nothing downstream reads past cap)
// and flags the status word for the host to redo the call; the call's
// largest total is kept in *tickmax.
__global__ void k_offsets64(const unsigned long long *__restrict__ scan, const uint32_t *__restrict__ count,
		size_t nray, int64_t *__restrict__ off64,
		unsigned long long *__restrict__ maxcount, size_t cap, unsigned long long *__restrict__ tickmax,
		uint32_t *__restrict__ status) {
	const size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
	if (r > nray) return;
	// scan holds the exclusive scan over nray+1 entries (count[nray] = 0)
	const bool over = cap && (size_t)scan[nray] > cap;
	off64[r] = over ? 0 : scan[r];
	if (r < nray) {
		atomicMax(maxcount, (unsigned long long)count[r]);
	} else {
		maxcount[1] = scan[r];       // the hit total, read with the longest list
		if (cap) {
			atomicMax(tickmax, (unsigned long long)scan[r]);
			if (over) atomicOr(status, PSG_ST_SLAB);
		}
	}
}

// The caller's index of internal particle i (order: null when the arrays
// are still in caller order); ties in d are broken by it.
__device__ __forceinline__ uint32_t caller_index(const uint32_t *__restrict__ order, uint32_t i) {
	return order ? order[i] : i;
}

// What a sort kernel reads and writes: the rays (of a replayed batch, from its
// per-call values), their slabs of hit positions and the sorted lists. With
// want_kern, in the ticks, b becomes the column-density factor
// sph_depth(b/h)/h^2 (loop.c:429-445) and the distances, which only order the
// hits there, are not stored.
struct SortIO {
	const psg_ray *rays;
	const PsgBatchDev *B;
	const int64_t *off;
	size_t scap, slab_r0;
	const uint32_t *slab;
	uint32_t *out_ipar;
	double *out_d, *out_b;
	int want_kern;
	const float4 *psml;
	const uint32_t *order;
	__device__ __forceinline__ void ray(size_t r, float s[3], float dir[3]) const {
		const psg_ray &ry = (B ? B->rays : rays)[r];
#pragma unroll
		for (int a = 0; a < 3; a++) {
			s[a] = ry.s[a];
			dir[a] = ry.dir[a];
		}
	}
};

// The hit on particle ip at distance d as the sorted list's entry h.
__device__ __forceinline__ void put_sorted_hit(const SortIO &io, const PhysParams &P, int64_t h, uint32_t ip, double d,
		const float s[3], const float dir[3]) {
	const float4 q = io.psml[ip];
	const HitDist hd{d, hit_proj(s, dir, q)};
	const double b = __dsqrt_rn(fabs(hd.r2()));
	io.out_ipar[h] = ip;
	if (io.want_kern) {
		const double inv = __ddiv_rn(1.0, (double)q.w);
		io.out_b[h] = rn_dmul(sph_depth(P, rn_dmul(b, inv)), rn_dmul(inv, inv));
	} else {
		io.out_d[h] = d;
		io.out_b[h] = b;
	}
}

// Per-ray sort by (d, ipar), one ray per block of TPR threads holding IPT
// hits each: a block radix sort (passes of 4 bits) on d mapped to KEY_BITS
// bits over the ray's own range of d (a monotone map) -- 12 bits for up to
// 1024 hits, 16 up to 4096, 20 beyond, so that about n^2 / 2^(bits+1) pairs
// share a key -- and the few runs of equal keys are then insertion-sorted
// on the exact (d, ipar) -- the reference's d
// order (loop.c:783-787) with ties broken by the caller's particle index.
// The distances are computed from the particles' positions (the slab holds
// no more than the hits' particles) and kept in shared memory.
template <int TPR, int IPT>
struct SortSmem {
	using Sort = cub::BlockRadixSort<uint32_t, TPR, IPT, uint32_t, 4>;
	static constexpr int NMAX = TPR * IPT;
	double d[NMAX];
	double lo[TPR / 32], hi[TPR / 32];
	union {
		typename Sort::TempStorage sort;
		struct {
			uint32_t key[NMAX], pos[NMAX];
		} s;
	} u;
};
template <int TPR, int IPT>
__global__ void __launch_bounds__(TPR) k_sort_block(const uint32_t *__restrict__ list,
		const unsigned long long *__restrict__ d_nlist, const SortIO io, PhysParams P) {
	using Smem = SortSmem<TPR, IPT>;
	constexpr int NMAX = Smem::NMAX;
	extern __shared__ __align__(16) char sort_smem[];
	Smem &sm = *reinterpret_cast<Smem *>(sort_smem);
	uint32_t *const key = sm.u.s.key, *const pos = sm.u.s.pos;
	// a persistent grid: the class's ray count is read here, so the launch
	// needs no count from the host
	const unsigned long long nlist = *d_nlist;
	for (unsigned long long li = blockIdx.x; li < nlist; li += gridDim.x) {
	const size_t r = list[li];
	const int64_t h0 = io.off[r];
	const int n = (int)(io.off[r + 1] - h0);
	const uint32_t *__restrict__ raw = io.slab + (r - io.slab_r0) * io.scap;
	float s[3], dir[3];
	io.ray(r, s, dir);
	double dlo = 1e300, dhi = -1e300;
	for (int i = threadIdx.x; i < n; i += TPR) {
		const double d = hit_d(s, io.psml[raw[i]]);
		sm.d[i] = d;
		dlo = fmin(dlo, d);
		dhi = fmax(dhi, d);
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		dlo = fmin(dlo, __shfl_xor_sync(0xffffffffu, dlo, o));
		dhi = fmax(dhi, __shfl_xor_sync(0xffffffffu, dhi, o));
	}
	if ((threadIdx.x & 31) == 0) {
		sm.lo[threadIdx.x >> 5] = dlo;
		sm.hi[threadIdx.x >> 5] = dhi;
	}
	__syncthreads();
#pragma unroll
	for (int w = 0; w < TPR / 32; w++) {
		dlo = fmin(dlo, sm.lo[w]);
		dhi = fmax(dhi, sm.hi[w]);
	}
	constexpr int KEY_BITS = NMAX <= 1024 ? 12 : (NMAX <= 4096 ? 16 : 20);
	constexpr uint32_t KEY_MAX = (1u << KEY_BITS) - 1u;
	const double scale = dhi > dlo ? (double)KEY_MAX / (dhi - dlo) : 0.0;
	uint32_t k[IPT], v[IPT];
#pragma unroll
	for (int u = 0; u < IPT; u++) {
		const int i = threadIdx.x * IPT + u;
		// padding takes the largest key; the sort is stable and padding
		// follows every real item, so it stays behind them
		k[u] = i < n ? min((uint32_t)((sm.d[i] - dlo) * scale), KEY_MAX) : KEY_MAX;
		v[u] = (uint32_t)i;
	}
	typename Smem::Sort(sm.u.sort).Sort(k, v, 0, KEY_BITS);
	__syncthreads();
#pragma unroll
	for (int u = 0; u < IPT; u++) {
		const int i = threadIdx.x * IPT + u;
		key[i] = k[u];
		pos[i] = v[u];
	}
	__syncthreads();
	// exact order inside runs of equal keys
	for (int i = threadIdx.x; i + 1 < n; i += TPR) {
		if (key[i] != key[i + 1] || (i > 0 && key[i - 1] == key[i])) continue;
		int e = i + 1;
		while (e + 1 < n && key[e + 1] == key[i]) e++;
		for (int a = i + 1; a <= e; a++) {
			const uint32_t pa = pos[a];
			const double da = sm.d[pa];
			int c = a;
			while (c > i) {
				const uint32_t pc = pos[c - 1];
				const double dc = sm.d[pc];
				if (dc < da || (dc == da && caller_index(io.order, raw[pc]) < caller_index(io.order, raw[pa]))) break;
				pos[c] = pc;
				c--;
			}
			pos[c] = pa;
		}
	}
	__syncthreads();
	for (int i = threadIdx.x; i < n; i += TPR) {
		const uint32_t p = pos[i];
		put_sorted_hit(io, P, h0 + i, raw[p], sm.d[p], s, dir);
	}
	__syncthreads();     // shared memory is reused by the next ray
	}
}

template <int TPR, int IPT>
size_t sort_smem_bytes() {
	return sizeof(SortSmem<TPR, IPT>);
}

// Rays with more hits than the largest class (PSG_SORT_MAX), a block of
// LONG_NT threads each, persistent over their list: the hits as (d, caller
// index << 32 | slab position) pairs in tmp (the two halves, at the ray's
// list offset), sorted by block_sort_global on exactly the order of the
// class sorts -- d, then the caller's index.
#define LONG_NT 1024
struct LongHit {
	double d;
	unsigned long long ck;
};
struct LongHitLess {
	__device__ __forceinline__ bool operator()(const LongHit &x, const LongHit &y) const {
		return x.d < y.d || (x.d == y.d && x.ck < y.ck);
	}
};
__global__ void __launch_bounds__(LONG_NT) k_sort_long(const uint32_t *__restrict__ list,
		const unsigned long long *__restrict__ d_nlist, const SortIO io, PhysParams P, LongHit *tmp, size_t hb) {
	__shared__ LongHit tile[2 * LONG_NT];
	const LongHit pad{__longlong_as_double(0x7ff0000000000000ll), ~0ull};
	const unsigned long long nlist = *d_nlist;
	for (unsigned long long li = blockIdx.x; li < nlist; li += gridDim.x) {
		const size_t r = list[li];
		const int64_t h0 = io.off[r];
		const int64_t n = io.off[r + 1] - h0;
		const uint32_t *raw = io.slab + (r - io.slab_r0) * io.scap;
		float s[3], dir[3];
		io.ray(r, s, dir);
		LongHit *a = tmp + h0;
		for (int64_t i = threadIdx.x; i < n; i += LONG_NT)
			a[i] = LongHit{hit_d(s, io.psml[raw[i]]),
					(unsigned long long)caller_index(io.order, raw[i]) << 32 | (unsigned long long)i};
		const LongHit *f = block_sort_global<LONG_NT>(a, tmp + hb + h0, n, tile, pad, LongHitLess());
		for (int64_t i = threadIdx.x; i < n; i += LONG_NT)
			put_sorted_hit(io, P, h0 + i, raw[(uint32_t)f[i].ck], f[i].d, s, dir);
		__syncthreads();
	}
}

// Size classes of the ray sort: class c holds rays with at most
// kSortClassMax[c] hits (and more than the previous class's bound).
// size classes of the per-ray sort (threads x items per thread):
// 32x2, 32x4, 64x4, 128x4, 128x8, 256x8, 256x16, 512x16
#define SORT_NCLS 8
__constant__ int kSortBounds[SORT_NCLS] = {64, 128, 256, 512, 1024, 2048, 4096, PSG_SORT_MAX};

// rays [r0, nray) into the size classes' lists
__global__ void k_sort_classify(size_t r0, size_t nray, const int64_t *__restrict__ off, uint32_t *__restrict__ lists,
		size_t stride, unsigned long long *__restrict__ nclass, unsigned long long *__restrict__ nlong) {
	const size_t r = r0 + blockIdx.x * (size_t)blockDim.x + threadIdx.x;
	if (r >= nray) return;
	const int64_t n = off[r + 1] - off[r];
	if (n == 0) return;
	if (n > PSG_SORT_MAX) {      // the long list, after the classes'
		const unsigned long long k = atomicAdd(nlong, 1ull);
		lists[SORT_NCLS * stride + k] = (uint32_t)r;
		return;
	}
	int c = 0;
	while (c < SORT_NCLS - 1 && n > kSortBounds[c]) c++;
	const unsigned long long k = atomicAdd(&nclass[c], 1ull);
	lists[c * stride + k] = (uint32_t)r;
}

inline unsigned blocks(size_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// S_COUNT during a traversal: the hit counts (nray + 1, u32), then their
// exclusive scan (nray + 2, u64) at the next 16-byte boundary
const void *trace_kernel(const psg_context *ctx) {
	return ctx->ppc == 8 ? (const void *)k_trace_stack<8, false> : (const void *)k_trace_stack<0, false>;
}
size_t trace_smem(const psg_context *ctx, int warps) {
	return sizeof(int) * (TR_STACK + 32 * (size_t)ctx->ppc + 32) * warps;
}
// The traversal's launch: its persistent grid, and where the rays are few the
// tree level whose cells divide each of them: the deepest of 1 to 3 that the
// tree has in full and that makes at most twice as many parts as there are
// resident warps (more would only be cells that miss). Recombination rays are
// not divided: a fifth of the box long, each lies in a cell or two of these
// levels (100 of them on 1M particles: 55 us whole, 64 us divided).
struct TracePlan {
	unsigned grid = 0;
	int warps = 1, start0 = 0, nstart = 0;
};
int plan_trace(psg_context *ctx, size_t nray, bool divide, TracePlan *t) {
	t->warps = std::max(1, std::min(TR_MAX_WARPS, ctx->tune.trace_warps));
	const size_t smem = trace_smem(ctx, t->warps);
	const void *kern[2] = {trace_kernel(ctx), ctx->ppc == 8 ? (const void *)k_trace_stack<8, true>
			: (const void *)k_trace_stack<0, true>};
	if (smem > 48 * 1024)
		for (const void *k : kern)
			PSG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
	int per_sm = 1;
	PSG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern[0], 32 * t->warps, smem));
	const size_t resident = (size_t)std::max(per_sm, 1) * ctx->sms;
	size_t units = nray;
	t->nstart = 0;
	for (int l = 1; l <= 3 && divide && ctx->level_start[l]; l++)
		if (nray << (3 * l) <= 2 * resident * t->warps) {
			t->start0 = ctx->level_start[l];
			t->nstart = 1 << (3 * l);
			units = nray << (3 * l);
		}
	t->grid = (unsigned)std::min<size_t>(blocks(units, t->warps), resident);
	return PSG_OK;
}
// (with t.nstart the rays' counts have to be zero)
void launch_trace(psg_context *ctx, const TracePlan &t, const psg_ray *rays, size_t nray, uint32_t *count,
		size_t scap, uint32_t *slab, unsigned long long *next_ray, const unsigned *nlim) {
	const size_t smem = trace_smem(ctx, t.warps);
	auto go = [&](auto kern) {
		kern<<<t.grid, 32 * t.warps, smem, ctx->stream>>>(rays, nray, ctx->d_wide_lo, ctx->d_wide_hi, ctx->d_leaf_psml,
				ctx->d_leaf_idx, ctx->ppc, count, scap, slab, next_ray, ctx->d_status, nlim, t.start0, t.nstart);
	};
	if (t.nstart) {
		if (ctx->ppc == 8) go(k_trace_stack<8, true>);
		else go(k_trace_stack<0, true>);
	} else {
		if (ctx->ppc == 8) go(k_trace_stack<8, false>);
		else go(k_trace_stack<0, false>);
	}
	ctx->launches++;
}
size_t count_bytes(size_t nray) { return 16 * ((sizeof(uint32_t) * (nray + 1) + 15) / 16) + 8 * (nray + 2) + 64; }
unsigned long long *count_scan(uint32_t *count, size_t nray) {
	return (unsigned long long *)((char *)count + 16 * ((sizeof(uint32_t) * (nray + 1) + 15) / 16));
}

}  // namespace

// Hit counts clamped to the slab capacity for the offsets (the slabs hold
// no more); the longest list of the call kept in *callmax, and a clamped list
// flagged in the status word (PSG_ST_SLAB) so the host redoes the call
// with larger slabs.
__global__ void k_count_clamp(size_t nray, size_t scap, uint32_t *__restrict__ count,
		unsigned long long *__restrict__ callmax, uint32_t *__restrict__ status) {
	const size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
	if (r >= nray) return;
	const uint32_t c = count[r];
	if (c > scap) {
		count[r] = (uint32_t)scap;
		atomicOr(status, PSG_ST_SLAB);
	}
	if (c) atomicMax(callmax, (unsigned long long)c);
}

namespace {
// The counts of a recombination tick after its traversal: the source rays'
// from the call's traced source rays (the tick is B->k of the call), the
// emitted rays' clamped to the slabs (as k_count_clamp).
__global__ void k_rec_counts(const PsgBatchDev *__restrict__ B, size_t R, const int64_t *__restrict__ src_off,
		size_t cap_rec, size_t scap, uint32_t *__restrict__ count, unsigned long long *__restrict__ callmax,
		uint32_t *__restrict__ status) {
	const int64_t base = B->k * (int64_t)R;
	for (size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x; r < R + cap_rec;
			r += (size_t)gridDim.x * blockDim.x) {
		if (r < R) {
			count[r] = (uint32_t)(src_off[base + (int64_t)r + 1] - src_off[base + (int64_t)r]);
			continue;
		}
		const uint32_t c = count[r];
		if (c > scap) {
			count[r] = (uint32_t)scap;
			atomicOr(status, PSG_ST_SLAB);
		}
		if (c) atomicMax(callmax, (unsigned long long)c);
	}
}
// their sorted hits into the tick's lists, a warp per ray (nothing when the
// tick's offsets were emptied for exceeding the capacity)
__global__ void k_copy_src_hits(const PsgBatchDev *__restrict__ B, size_t R, const int64_t *__restrict__ src_off,
		const uint32_t *__restrict__ src_ipar, const double *__restrict__ src_kern, const int64_t *__restrict__ off,
		uint32_t *__restrict__ hit_ipar, double *__restrict__ hit_kern) {
	const size_t r = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) / 32;
	const int lane = threadIdx.x & 31;
	if (r >= R) return;
	const int64_t base = B->k * (int64_t)R + (int64_t)r;
	const int64_t s0 = src_off[base];
	const int64_t n = min(src_off[base + 1] - s0, off[r + 1] - off[r]);
	const int64_t d0 = off[r];
	for (int64_t i = lane; i < n; i += 32) {
		hit_ipar[d0 + i] = src_ipar[s0 + i];
		hit_kern[d0 + i] = src_kern[s0 + i];
	}
}
}  // namespace

struct SrcHits {
	const int64_t *off;
	const uint32_t *ipar;
	const double *kern;
};
static SrcHits src_hits(psg_context *ctx) {
	char *m = (char *)ctx->scratch[S_SRCHIT].p;
	SrcHits h;
	h.off = (const int64_t *)m;
	h.kern = (const double *)(m + sizeof(int64_t) * (ctx->src_nray + 1));
	h.ipar = (const uint32_t *)(h.kern + ctx->src_nhit);
	return h;
}

// All source rays of a recombination call traced and sorted (with the
// column-density factor) before its ticks run; kept in S_SRCHIT. One host
// synchronisation (the traversal's).
int psg_trace_src_batch(psg_context *ctx, const psg_ray *d_rays, size_t nray) {
	PsgTraceFill tf;
	int rc = psg_trace_fill(ctx, d_rays, nray, &tf);
	if (!rc) rc = psg_trace_sort_prepare(ctx, nray, tf.nhit, tf.maxcount, 1);
	if (!rc) rc = psg_trace_sort_enqueue(ctx, d_rays, nullptr, nray, tf.maxcount, 1, 0);
	if (rc) return rc;
	// the layout depends on a grow-only capacity, not on this call's hit
	// total, so that calls of similar totals share one captured tick graph
	if (tf.nhit > ctx->src_nhit || nray != ctx->src_nray) {
		size_t c = std::max(tf.nhit + tf.nhit / 8, ctx->src_nhit);
		c = (c + 65535) & ~(size_t)65535;
		ctx->src_nhit = c;
	}
	char *m = (char *)psg_scratch(ctx, S_SRCHIT, sizeof(int64_t) * (nray + 1) + (sizeof(double) + sizeof(uint32_t)) *
			ctx->src_nhit);
	if (!m) return PSG_E_NOMEM;
	ctx->src_nray = nray;
	ctx->src_total = tf.nhit;
	const SrcHits h = src_hits(ctx);
	cudaStream_t st = ctx->stream;
	PSG_CUDA(cudaMemcpyAsync((void *)h.off, ctx->scratch[S_OFFSETS].p, sizeof(int64_t) * (nray + 1),
			cudaMemcpyDeviceToDevice, st));
	if (tf.nhit) {
		PSG_CUDA(cudaMemcpyAsync((void *)h.ipar, ctx->scratch[S_HIT_IPAR].p, sizeof(uint32_t) * tf.nhit,
				cudaMemcpyDeviceToDevice, st));
		PSG_CUDA(cudaMemcpyAsync((void *)h.kern, ctx->scratch[S_HIT_KERN].p, sizeof(double) * tf.nhit,
				cudaMemcpyDeviceToDevice, st));
	}
	return PSG_OK;
}

// The traversal of a recombination tick: the emitted rays buf[R, R + *nlim)
// traversed (slabs from index 0), the source rays' counts from S_SRCHIT,
// then the scan and the offsets over all R + cap_rec rays.
int psg_trace_rec_fill_enqueue(psg_context *ctx, const psg_ray *buf, size_t R, size_t cap_rec, const unsigned *nlim,
		size_t cap, const PsgBatchDev *B) {
	cudaStream_t st = ctx->stream;
	const size_t nray = R + cap_rec;
	uint32_t *count = (uint32_t *)ctx->scratch[S_COUNT].p;
	unsigned long long *scan = count_scan(count, nray);
	int64_t *off64 = (int64_t *)ctx->scratch[S_OFFSETS].p;
	unsigned long long *d_max = ctx->d_counters + 4;
	unsigned long long *next_ray = ctx->d_counters + 9;
	const size_t scap = ctx->slab_cap;
	uint32_t *slab_ipar = (uint32_t *)ctx->scratch[S_REC_U32].p;
	TracePlan t;
	const int rc = plan_trace(ctx, cap_rec, false, &t);
	if (rc) return rc;
	const SrcHits h = src_hits(ctx);
	PSG_CUDA(cudaMemsetAsync(count, 0, sizeof(uint32_t) * (nray + 1), st));
	PSG_CUDA(cudaMemsetAsync(d_max, 0, 2 * sizeof(unsigned long long), st));
	PSG_CUDA(cudaMemsetAsync(next_ray, 0, sizeof(unsigned long long), st));
	launch_trace(ctx, t, buf + R, cap_rec, count + R, scap, slab_ipar, next_ray, nlim);
	PSG_CHECK_LAUNCH();
	k_rec_counts<<<(unsigned)std::min<size_t>(blocks(nray, 256), 4 * (size_t)ctx->sms), 256, 0, st>>>(B, R, h.off,
			cap_rec, scap, count, ctx->d_counters + 3, ctx->d_status);
	PSG_CHECK_LAUNCH();
	PSG_CUDA(scan_enqueue(st, count, nray + 1, scan, (unsigned long long *)ctx->scratch[S_SCAN].p, Widen()));
	k_offsets64<<<blocks(nray + 1, 256), 256, 0, st>>>(scan, count, nray, off64, d_max, cap,
			ctx->d_counters + 24, ctx->d_status);
	PSG_CHECK_LAUNCH();
	ctx->launches += 2 + scan_launches(nray + 1);
	return PSG_OK;
}

// The per-ray order of a recombination tick: the source rays' sorted hits
// copied from S_SRCHIT, the emitted rays (from R on) sorted from their slabs.
int psg_trace_rec_sort_enqueue(psg_context *ctx, size_t R, size_t nray, unsigned long long maxcount,
		const PsgBatchDev *B) {
	const SrcHits h = src_hits(ctx);
	k_copy_src_hits<<<blocks(R * 32, 256), 256, 0, ctx->stream>>>(B, R, h.off, h.ipar, h.kern,
			(const int64_t *)ctx->scratch[S_OFFSETS].p, (uint32_t *)ctx->scratch[S_HIT_IPAR].p,
			(double *)ctx->scratch[S_HIT_KERN].p);
	PSG_CHECK_LAUNCH();
	ctx->launches++;
	return psg_trace_sort_enqueue(ctx, nullptr, B, nray, maxcount, 1, R);
}

// Sizes the buffers psg_trace_rec_fill_enqueue uses for nray rays (allocates;
// before a capture).
int psg_trace_fill_prepare(psg_context *ctx, size_t nray) {
	const size_t scap = ctx->slab_cap;
	const size_t slots = nray * scap;
	if (!psg_scratch(ctx, S_COUNT, count_bytes(nray)) ||
			!psg_scratch(ctx, S_SCAN, sizeof(unsigned long long) * (scan_tiles(nray + 1) + 1)) ||
			!psg_scratch(ctx, S_OFFSETS, sizeof(int64_t) * (nray + 1) + 256) ||
			!psg_scratch(ctx, S_REC_U32, sizeof(uint32_t) * (slots ? slots : 1)))
		return PSG_E_NOMEM;
	return PSG_OK;
}

// The traversal of nray device-resident rays into per-ray slabs, the hit
// counts' scan and the offsets (S_OFFSETS: int64 offsets[nray+1]). One host synchronisation reads the longest list,
// the status word and the hit total; a ray that outgrew its slab grows the
// slabs and reruns the traversal once.
int psg_trace_fill(psg_context *ctx, const psg_ray *d_rays, size_t nray, PsgTraceFill *tf) {
	if (!ctx->have_tree) return psg_fail(ctx, PSG_E_INVAL, "trace: no tree (psg_build_tree first)");
	cudaStream_t st = ctx->stream;
	uint32_t *count = (uint32_t *)psg_scratch(ctx, S_COUNT, count_bytes(nray));
	char *offmem = (char *)psg_scratch(ctx, S_OFFSETS, sizeof(int64_t) * (nray + 1) + 256);
	unsigned long long *tiles = (unsigned long long *)psg_scratch(ctx, S_SCAN,
			sizeof(unsigned long long) * (scan_tiles(nray + 1) + 1));
	if (!count || !offmem || !tiles) return PSG_E_NOMEM;
	unsigned long long *scan = count_scan(count, nray);
	int64_t *off64 = (int64_t *)offmem;
	unsigned long long *d_max = ctx->d_counters + 4;
	unsigned long long *next_ray = ctx->d_counters + 9;
	TracePlan tp;
	const int prc = plan_trace(ctx, nray, true, &tp);
	if (prc) return prc;
	size_t scap = 0;
	unsigned long long hdr[2] = {0, 0};      // longest list, hit total
	for (int attempt = 0; attempt < 2; attempt++) {
		scap = ctx->slab_cap ? ctx->slab_cap : 1024;
		const size_t slots = nray * scap;
		uint32_t *slab_ipar = (uint32_t *)psg_scratch(ctx, S_REC_U32, sizeof(uint32_t) * (slots ? slots : 1));
		if (!slab_ipar) return PSG_E_NOMEM;
		PSG_CUDA(cudaMemsetAsync(tp.nstart ? count : count + nray, 0, sizeof(uint32_t) * (tp.nstart ? nray + 1 : 1), st));
		PSG_CUDA(cudaMemsetAsync(d_max, 0, 2 * sizeof(unsigned long long), st));
		psg_mark_begin(ctx, PSG_K_TRACE_FILL);
		if (nray) {
			PSG_CUDA(cudaMemsetAsync(next_ray, 0, sizeof(unsigned long long), st));
			launch_trace(ctx, tp, d_rays, nray, count, scap, slab_ipar, next_ray, nullptr);
		}
		PSG_CHECK_LAUNCH();
		psg_mark_end(ctx);
		PSG_CUDA(scan_enqueue(st, count, nray + 1, scan, tiles, Widen()));
		k_offsets64<<<blocks(nray + 1, 256), 256, 0, st>>>(scan, count, nray, off64, d_max, 0, nullptr,
				nullptr);
		PSG_CHECK_LAUNCH();
		ctx->launches += 1 + scan_launches(nray + 1);
		PSG_CUDA(cudaMemcpyAsync(hdr, d_max, sizeof(hdr), cudaMemcpyDeviceToHost, st));
		uint32_t stw = 0;
		PSG_CUDA(cudaMemcpyAsync(&stw, ctx->d_status, sizeof(stw), cudaMemcpyDeviceToHost, st));
		PSG_CUDA(cudaStreamSynchronize(st));
		ctx->host_syncs++;
		if (stw & PSG_ST_STACK) {
			PSG_CUDA(cudaMemsetAsync(ctx->d_status, 0, sizeof(uint32_t), st));
			return psg_fail(ctx, PSG_E_OVERFLOW, "trace: traversal stack overflow (tree deeper than supported)");
		}
		if (hdr[0] <= scap) break;
		size_t want = 1024;
		while (want < hdr[0] + hdr[0] / 4) want <<= 1;
		ctx->slab_cap = want;
		if (attempt == 1) return psg_fail(ctx, PSG_E_OVERFLOW, "trace: hit lists grew between passes");
	}
	if (!ctx->slab_cap) ctx->slab_cap = scap;
	if (hdr[1] >= (unsigned long long)INT32_MAX)
		return psg_fail(ctx, PSG_E_OVERFLOW, "trace: %llu hits in one batch exceed 2^31", hdr[1]);
	tf->nhit = (size_t)hdr[1];
	tf->maxcount = hdr[0];
	tf->scap = scap;
	return PSG_OK;
}

// Buffers of the sorted hit lists for up to cap hits: S_HIT_IPAR, S_HIT_KERN
// (b, or with want_kern the column-density factor), without want_kern S_RAW_D
// (d), and the class lists. Allocates; call before a stream capture.
int psg_trace_sort_prepare(psg_context *ctx, size_t nray, size_t cap, unsigned long long maxcount, int want_kern) {
	const size_t hb = cap ? cap : 1;
	uint32_t *hit_ipar = (uint32_t *)psg_scratch(ctx, S_HIT_IPAR, sizeof(uint32_t) * hb);
	double *hit_d = want_kern ? nullptr : (double *)psg_scratch(ctx, S_RAW_D, sizeof(double) * hb);
	double *hit_b = (double *)psg_scratch(ctx, S_HIT_KERN, sizeof(double) * hb);
	uint32_t *lists = (uint32_t *)psg_scratch(ctx, S_RAYLIST, sizeof(uint32_t) * (SORT_NCLS + 1) * (nray + 1));
	if (!hit_ipar || (!want_kern && !hit_d) || !hit_b || !lists) return PSG_E_NOMEM;
	ctx->hit_cap = hb;
	// the long rays' two halves of (d, key) pairs, at their list offsets
	if (maxcount > PSG_SORT_MAX && !psg_scratch(ctx, S_KEYS, sizeof(LongHit) * 2 * hb)) return PSG_E_NOMEM;
	// shared-memory limits and resident blocks per multiprocessor of the
	// eight class kernels (their persistent grids), once per context
	if (!ctx->sort_grid[0]) {
		int c = 0;
#define PSG_SORT_ATTR(T, I)                                                                                    \
	{                                                                                                        \
		if (sort_smem_bytes<T, I>() > 48 * 1024)                                                             \
			PSG_CUDA(cudaFuncSetAttribute(k_sort_block<T, I>, cudaFuncAttributeMaxDynamicSharedMemorySize,    \
					(int)sort_smem_bytes<T, I>()));                                                          \
		int per_sm = 1;                                                                                      \
		PSG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sort_block<T, I>, T,               \
				sort_smem_bytes<T, I>()));                                                                   \
		ctx->sort_grid[c++] = (unsigned)std::max(per_sm, 1) * (unsigned)ctx->sms;                             \
	}
		PSG_SORT_ATTR(32, 2) PSG_SORT_ATTR(32, 4) PSG_SORT_ATTR(64, 4) PSG_SORT_ATTR(128, 4)
		PSG_SORT_ATTR(128, 8) PSG_SORT_ATTR(256, 8) PSG_SORT_ATTR(256, 16) PSG_SORT_ATTR(512, 16)
#undef PSG_SORT_ATTR
	}
	return PSG_OK;
}

// The size classes a call with lists up to maxcount long can fill.
int psg_sort_classes(unsigned long long maxcount) {
	static const unsigned long long lower[SORT_NCLS] = {0, 64, 128, 256, 512, 1024, 2048, 4096};
	int c = 0;
	while (c < SORT_NCLS && maxcount > lower[c]) c++;
	return c;
}

// The per-ray sort by (d, ipar) of the filled slabs into the CSR lists.
// Launch sizes are fixed by nray (the persistent class kernels read their
// ray counts on the device), so it can be captured in a graph; with
// maxcount above PSG_SORT_MAX the long rays' kernel runs too.
// B: the rays are read from it on the device (a captured batch), else rays.
int psg_trace_sort_enqueue(psg_context *ctx, const psg_ray *rays, const PsgBatchDev *B, size_t nray,
		unsigned long long maxcount, int want_kern, size_t r0) {
	cudaStream_t st = ctx->stream;
	const size_t hb = ctx->hit_cap;
	SortIO io;
	io.rays = rays;
	io.B = B;
	io.off = (const int64_t *)ctx->scratch[S_OFFSETS].p;
	io.scap = ctx->slab_cap;
	io.slab_r0 = r0;
	io.slab = (const uint32_t *)ctx->scratch[S_REC_U32].p;
	io.out_ipar = (uint32_t *)ctx->scratch[S_HIT_IPAR].p;
	io.out_d = want_kern ? nullptr : (double *)ctx->scratch[S_RAW_D].p;
	io.out_b = (double *)ctx->scratch[S_HIT_KERN].p;
	io.want_kern = want_kern;
	io.psml = ctx->d_psml;
	io.order = ctx->d_order;
	if (nray <= r0) return PSG_OK;
	psg_mark_begin(ctx, PSG_K_SORT);
	{
		uint32_t *lists = (uint32_t *)ctx->scratch[S_RAYLIST].p;
		unsigned long long *d_ncls = ctx->d_counters + 16, *d_nlong = ctx->d_counters + 25;
		PSG_CUDA(cudaMemsetAsync(d_ncls, 0, SORT_NCLS * sizeof(unsigned long long), st));
		PSG_CUDA(cudaMemsetAsync(d_nlong, 0, sizeof(unsigned long long), st));
		k_sort_classify<<<blocks(nray - r0, 256), 256, 0, st>>>(r0, nray, io.off, lists, nray + 1, d_ncls, d_nlong);
		PSG_CHECK_LAUNCH();
		const PhysParams PP = psg_phys_params(ctx);
		const size_t stride = nray + 1;
		// a class whose rays all have more hits than the call's longest list
		// is empty: not launched (psg_sort_classes; part of a graph's key)
		const int ncls = psg_sort_classes(maxcount);
		auto launch_block = [&](auto kern, int tpr, size_t smem, int c) -> int {
			if (c >= ncls) return PSG_OK;
			const unsigned grid = (unsigned)std::min<size_t>(nray - r0, (size_t)ctx->sort_grid[c]);
			kern<<<grid, tpr, smem, st>>>(lists + c * stride, d_ncls + c, io, PP);
			PSG_CHECK_LAUNCH();
			ctx->launches++;
			return PSG_OK;
		};
		int rcs = launch_block(k_sort_block<32, 2>, 32, sort_smem_bytes<32, 2>(), 0);
		if (!rcs) rcs = launch_block(k_sort_block<32, 4>, 32, sort_smem_bytes<32, 4>(), 1);
		if (!rcs) rcs = launch_block(k_sort_block<64, 4>, 64, sort_smem_bytes<64, 4>(), 2);
		if (!rcs) rcs = launch_block(k_sort_block<128, 4>, 128, sort_smem_bytes<128, 4>(), 3);
		if (!rcs) rcs = launch_block(k_sort_block<128, 8>, 128, sort_smem_bytes<128, 8>(), 4);
		if (!rcs) rcs = launch_block(k_sort_block<256, 8>, 256, sort_smem_bytes<256, 8>(), 5);
		if (!rcs) rcs = launch_block(k_sort_block<256, 16>, 256, sort_smem_bytes<256, 16>(), 6);
		if (!rcs) rcs = launch_block(k_sort_block<512, 16>, 512, sort_smem_bytes<512, 16>(), 7);
		if (rcs) return rcs;
		ctx->launches++;
		if (maxcount > PSG_SORT_MAX) {
			// rays longer than the shared-memory classes: a block each
			const unsigned grid = (unsigned)std::min<size_t>(nray - r0, (size_t)ctx->sms);
			k_sort_long<<<grid, LONG_NT, 0, st>>>(lists + SORT_NCLS * stride, d_nlong, io, PP,
					(LongHit *)ctx->scratch[S_KEYS].p, hb);
			PSG_CHECK_LAUNCH();
			ctx->launches++;
		}
	}
	psg_mark_end(ctx);
	return PSG_OK;
}

// Traces nray device-resident rays: fill, buffers sized to the hits, sort.
// Leaves in scratch: S_OFFSETS, S_HIT_IPAR (sorted leaf-order indices),
// S_RAW_D (sorted d, without want_kern) and S_HIT_KERN (sorted b, or with
// want_kern the column-density factor).
int psg_trace_internal(psg_context *ctx, const psg_ray *d_rays, size_t nray, int want_kern) {
	PsgTraceFill tf;
	int rc = psg_trace_fill(ctx, d_rays, nray, &tf);
	if (rc) return rc;
	rc = psg_trace_sort_prepare(ctx, nray, tf.nhit, tf.maxcount, want_kern);
	if (rc) return rc;
	return psg_trace_sort_enqueue(ctx, d_rays, nullptr, nray, tf.maxcount, want_kern, 0);
}

// The sorted hits as the caller's records (its particle index, d, b), so that
// one copy brings them to it (three copies and a host loop took 1024 rays of
// 120 hits 1.05 ms in all, this 0.49).
__global__ void k_pack_hits(size_t n, const uint32_t *__restrict__ ipar, const double *__restrict__ d,
		const double *__restrict__ b, const uint32_t *__restrict__ order, psg_xtype *__restrict__ out) {
	const size_t h = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
	if (h >= n) return;
	psg_xtype x;
	x.ipar = caller_index(order, ipar[h]);
	x.d = d[h];
	x.b = b[h];
	out[h] = x;
}

// copies the traced hit lists to host Xtype records
static int download_hits(psg_context *ctx, size_t nray, int64_t *offsets, psg_xtype **x, size_t *size,
		size_t *nhit_out) {
	cudaStream_t st = ctx->stream;
	int64_t *off64 = (int64_t *)ctx->scratch[S_OFFSETS].p;
	int64_t total = 0;      // (or the offsets' last)
	PSG_CUDA(cudaMemcpyAsync(offsets ? offsets : &total, offsets ? off64 : off64 + nray,
			sizeof(int64_t) * (offsets ? nray + 1 : 1), cudaMemcpyDeviceToHost, st));
	PSG_CUDA(cudaStreamSynchronize(st));
	const size_t nhit = (size_t)(offsets ? offsets[nray] : total);
	if (*x == nullptr || *size < nhit) {
		size_t want = *size ? *size : 1000;
		while (want < nhit) want *= 2;
		psg_xtype *nx = (psg_xtype *)realloc(*x, sizeof(psg_xtype) * want);
		if (!nx) return psg_fail(ctx, PSG_E_NOMEM, "trace: host allocation failed");
		*x = nx;
		*size = want;
	}
	if (nhit) {
		psg_xtype *packed = (psg_xtype *)psg_scratch(ctx, S_MAP, sizeof(psg_xtype) * nhit);
		if (!packed) return PSG_E_NOMEM;
		k_pack_hits<<<(unsigned)((nhit + 255) / 256), 256, 0, st>>>(nhit, (const uint32_t *)ctx->scratch[S_HIT_IPAR].p,
				(const double *)ctx->scratch[S_RAW_D].p, (const double *)ctx->scratch[S_HIT_KERN].p, ctx->d_order, packed);
		PSG_CHECK_LAUNCH();
		PSG_CUDA(cudaMemcpyAsync(*x, packed, sizeof(psg_xtype) * nhit, cudaMemcpyDeviceToHost, st));
		PSG_CUDA(cudaStreamSynchronize(st));
	}
	*nhit_out = nhit;
	return PSG_OK;
}

static int upload_rays(psg_context *ctx, const psg_ray *rays, size_t nray, psg_ray **d_rays) {
	psg_ray *d = (psg_ray *)psg_scratch(ctx, S_RAYS, sizeof(psg_ray) * (nray ? nray : 1));
	if (!d) return PSG_E_NOMEM;
	if (nray) PSG_CUDA(cudaMemcpyAsync(d, rays, sizeof(psg_ray) * nray, cudaMemcpyHostToDevice, ctx->stream));
	*d_rays = d;
	return PSG_OK;
}

extern "C" int psg_trace(psg_context *ctx, const psg_ray *rays, size_t nray, int64_t *offsets,
		psg_xtype **x, size_t *size) {
	if (!ctx) return PSG_E_INVAL;
	if ((nray && !rays) || !x || !size) return psg_fail(ctx, PSG_E_INVAL, "psg_trace: null argument");
	PSG_CUDA(cudaSetDevice(ctx->device));
	psg_ray *d_rays = nullptr;
	int rc = upload_rays(ctx, rays, nray, &d_rays);
	if (rc) return rc;
	rc = psg_trace_internal(ctx, d_rays, nray, 0);
	if (rc) return rc;
	size_t nhit = 0;
	return download_hits(ctx, nray, offsets, x, size, &nhit);
}

extern "C" size_t psg_rt_trace(psg_context *ctx, const float s[3], const float dir[3], const float dist,
		psg_xtype **x, size_t *size) {
	if (!ctx || !s || !dir || !x || !size) return (size_t)-1;
	psg_ray ray;
	memset(&ray, 0, sizeof(ray));
	for (int d = 0; d < 3; d++) { ray.s[d] = s[d]; ray.dir[d] = dir[d]; }
	ray.length = dist;
	if (cudaSetDevice(ctx->device) != cudaSuccess) return (size_t)-1;
	psg_ray *d_rays = nullptr;
	if (upload_rays(ctx, &ray, 1, &d_rays)) return (size_t)-1;
	if (psg_trace_internal(ctx, d_rays, 1, 0)) return (size_t)-1;
	size_t nhit = 0;
	if (download_hits(ctx, 1, nullptr, x, size, &nhit)) return (size_t)-1;
	return nhit;
}
