/*
 * Permuted, scaled element-wise block kernels of libxm-gb300.
 *
 * One launch covers a batch of block tasks (xmgd_ptask_t): xm_set,
 * xm_copy, xm_add, xm_mul, xm_div, xm_dot and the standalone
 * xm_tensor_unfold_block / xm_tensor_fold_block all reduce to "for every
 * element of an up-to-8-D box, dst[.] = f(dst[.], src[.])" with independent
 * destination and source strides.  This replaces the reference's per-block
 * unfold -> scale -> fold -> axpy host loops (tensor.c:436-639,
 * scalar.c:123-239, xm.c:28-508) with one HBM pass.
 *
 * Five schedules, chosen per task on the host after xmg_ptask_shape has
 * normalised the iteration space; each schedule is its own kernel, and a
 * batch launches one kernel per schedule present:
 *  - flat: one contiguous run on both sides (whole canonical blocks);
 *  - row: dimension 0 unit-stride on the destination side; a CTA covers
 *    ROW_ELEMS elements along dim 0 for as many outer rows as fit, with
 *    per-row outer offsets precomputed in shared memory (outer permutations,
 *    transposes of thin blocks);
 *  - slices: the source's unit-stride dimension is dim 1 and both extents
 *    are small: a CTA moves whole s0 x s1 slices through padded shared
 *    memory (loads along the source's runs, stores along the
 *    destination's): the gather-transpose of unfold/fold;
 *  - tile: the same for larger extents, a t0 x t1 tile per CTA;
 *  - slab: xm_copy's transposes when each s0 x s1 slice lies contiguously
 *    on both sides and consecutive slices follow one another (whole
 *    blocks whose permutation swaps the two leading dimensions): a CTA
 *    brings its slices in with one bulk copy into shared memory,
 *    transposes there and stores along the destination's run.
 */
#include <stdlib.h>
#include <string.h>
#include <algorithm>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "tc.cuh"

namespace xmg {

constexpr int PT_THREADS = 256;
constexpr int ROW_ELEMS = 4096;    /* elements per CTA in row mode */
constexpr int FLAT_ELEMS = 8192;   /* elements per CTA in flat mode, at most */
constexpr int FLAT_MIN = 1024;     /* ... and at least */
/* rows of at most this many elements whose source runs are longer than a
 * slice go by the row schedule: a tile would hold 32 of them in a CTA, 256
 * go in one there (dot of 2 x 1 000 000 floats 432 us as tiles, 73 as rows;
 * quotient of 12 x 200 001 doubles 62 and 31) */
constexpr int ROW_THIN = 16;
constexpr int SLICE_MAX = 48;      /* slices: extents at most */
constexpr int SLICE_MAXQ = 64;     /* slices per CTA at most */
/* slab: about SLAB_CHUNK bytes of slices per CTA (one slice at least), at
 * most SLAB_SMEM bytes of shared memory (the source's slices and the padded
 * tile) */
constexpr int64_t SLAB_CHUNK = 16384;
constexpr int64_t SLAB_SMEM = 64 * 1024;
constexpr int64_t SLAB_MIN = 32 << 20;   /* bytes of a batch's slabs */
/* tile: elements per CTA (eight per thread, four of the 16-byte types), and
 * the shared tile with the padding of its rows */
static constexpr int tile_elems(int dbytes, int sbytes)
{
	return dbytes <= 8 && sbytes <= 8 ? 2048 : 1024;
}
static constexpr int tile_cap(int n) { return n + 256; }
/* slices: the same (one slice of 48 x 48 or two of 33 x 33 of the 8-byte
 * types; sixteen elements per thread of the 4-byte one; copies between types
 * hold the source alone) */
static constexpr int slice_elems(int dbytes, int sbytes)
{
	return dbytes == 4 && sbytes == 4 ? 4096 :
	    sbytes <= 8 && (dbytes <= 8 || dbytes != sbytes) ? 2304 : 1024;
}
static constexpr int slice_cap(int n) { return n == 2304 ? 48 * 49 : n + 256; }
/* log2 of the lanes along a run of n <= 32 elements: 8 to 32 */
static inline int lanes_log2(int n) { return n <= 8 ? 3 : n <= 16 ? 4 : 5; }

struct task_meta {
	int64_t first_cta;
	int32_t mode;          /* 0 row, 1 tile, 2 flat, 3 slices, 4 slab */
	int32_t rows_per_cta;  /* row mode: outer rows per CTA; flat mode:
	                          elements per CTA; slices and slab: slices */
	int64_t nouter;        /* row: product of dims 1..; tile: dims 2.. */
	int32_t ctas_d0, ctas_d1;
	int32_t t0, t1;        /* tile mode: extents of a tile */
	int32_t l1, lb;        /* tile mode: log2 of the lanes along dim 1, of
	                          the 32-lane blocks along dim 0 */
};

/* A batch of up to PACK tasks travels in the kernel's parameters, which
 * spares a small call its host-to-device copy; larger batches are read
 * from device memory. */
constexpr int PACK = 13;
struct task_pack {
	xmgd_ptask_t t[PACK];
	task_meta m[PACK];
};
static_assert(sizeof(task_pack) <= 3584, "kernel parameters");

template <typename T>
constexpr bool is_cplx = std::is_same<T, cf>::value || std::is_same<T, cd>::value;

/* a task's scalars (als: alpha in the source's type) */
template <typename D, typename S>
struct scalars {
	D al, be;
	S als;
	__device__ __forceinline__ explicit scalars(const xmgd_ptask_t &t) :
	    al(num<D>::mk(t.alpha)), be(num<D>::mk(t.beta)), als(num<S>::mk(t.alpha)) {}
};

__device__ __forceinline__ bool finite(const cd &v)
{
	return (__double2hiint(v.x) & 0x7ff00000) != 0x7ff00000 &&
	    (__double2hiint(v.y) & 0x7ff00000) != 0x7ff00000;
}

/* the whole complex expression, out of line: Inf and NaN alone take it */
static __device__ __noinline__ cd axpy_any(cd al, cd x, cd be, cd y)
{
	return num<cd>::add(num<cd>::mul(al, x), num<cd>::mul(be, y));
}

static __device__ __noinline__ cd mul_any(cd a, cd b) { return num<cd>::mul(a, b); }

/* s * v; ONE: s is 1, left out for real types and for finite complex doubles;
 * Inf and NaN take the product, which spreads NaN to both parts (complex
 * floats: what is left of it) */
template <bool ONE, typename T>
__device__ __forceinline__ T unit(const T &s, const T &v)
{
	if constexpr (!ONE)
		return num<T>::mul(s, v);
	else if constexpr (std::is_same<T, cd>::value)
		return finite(v) ? v : mul_any(s, v);
	else if constexpr (std::is_same<T, cf>::value)
		return cf{fmaf(-v.y, 0.0f, v.x), fmaf(v.x, 0.0f, v.y)};
	else
		return v;
}

/* The new value of a destination element x from a source element y (dot:
 * its product added to the sums).  ONE: alpha is 1 (and a complex beta
 * real), so that products with 1 and 0 are left out: the FP64 pipe issues 2
 * instructions a cycle and SM against one 8-byte element a cycle from
 * memory, so that two of them per element (alpha x and + beta y), ten of a
 * complex one, already take the time of the traffic or more. */
template <int OP, bool ONE, typename D, typename S>
__device__ __forceinline__ D
combine(D x, S y, const scalars<D, S> &c, double &dre, double &dim_)
{
	if constexpr (OP == XMGD_OP_SET)
		return c.al;
	else if constexpr (OP == XMGD_OP_SCALE)
		return num<D>::mul(c.al, x);
	else if constexpr (OP == XMGD_OP_AXPY && ONE && std::is_same<D, cd>::value)
		return finite(x) && finite(y) ?
		    cd{::fma(c.be.x, y.x, x.x), ::fma(c.be.x, y.y, x.y)} :
		    axpy_any(c.al, x, c.be, y);
	else if constexpr (OP == XMGD_OP_AXPY)
		return num<D>::add(unit<ONE>(c.al, x), num<D>::mul(c.be, conv<D, S>(y)));
	else if constexpr (OP == XMGD_OP_COPY)
		return conv<D, S>(unit<ONE>(c.als, y));
	else if constexpr (OP == XMGD_OP_MUL)
		return num<D>::mul(unit<ONE>(c.al, x), conv<D, S>(y));
	else if constexpr (OP == XMGD_OP_DIV)
		return num<D>::div(x, unit<ONE>(c.al, conv<D, S>(y)));
	else {
		/* a complex product is formed before it is added: two fused steps
		 * into the sum would round the sum, not the product, twice, and the
		 * halves of a product that cancel (|x| |y| large, re or im small)
		 * would take the sum's low bits with them */
		const D pr = num<D>::mul(x, conv<D, S>(y));
		dre += num<D>::re(pr);
		if constexpr (is_cplx<D>)
			dim_ += num<D>::im(pr);
		return x;
	}
}

/* f.run<OP, ONE>() for a task's operation; scalar conversions exist for
 * xm_copy alone, and ONE is set apart where FP64 work bounds the kernel or
 * costs nothing to leave out */
template <typename D, typename S, typename F>
__device__ __forceinline__ void
with_op(const xmgd_ptask_t &t, F f)
{
	constexpr bool special = !std::is_same<D, cf>::value;
	/* by their bits: a compare would be an FP64 instruction */
	bool one = special && __double_as_longlong(t.alpha[0]) == 0x3ff0000000000000ll;
	if (std::is_same<D, cd>::value)
		one = one && __double_as_longlong(t.alpha[1]) == 0 &&
		    __double_as_longlong(t.beta[1]) == 0;
#define WITH(OP) case OP: \
	if (one) f.template run<OP, special>(); else f.template run<OP, false>(); break
	switch (t.op) {
	case XMGD_OP_SET: f.template run<XMGD_OP_SET, false>(); break;
	WITH(XMGD_OP_COPY);
	default:
		if constexpr (std::is_same<D, S>::value) {
			switch (t.op) {
			case XMGD_OP_SCALE: f.template run<XMGD_OP_SCALE, false>(); break;
			WITH(XMGD_OP_AXPY);
			WITH(XMGD_OP_MUL);
			WITH(XMGD_OP_DIV);
			case XMGD_OP_DOT: f.template run<XMGD_OP_DOT, false>(); break;
			}
		}
	}
#undef WITH
}

constexpr bool op_reads_dst(int op) { return op != XMGD_OP_COPY && op != XMGD_OP_SET; }
constexpr bool op_reads_src(int op) { return op != XMGD_OP_SET && op != XMGD_OP_SCALE; }

/*
 * Flat runs with 16-byte accesses where both runs start on a 16-byte
 * boundary (whole blocks do), else one element at a time.  Each thread
 * issues the loads of U vectors (of both runs) before any of its stores:
 * stores to dst may alias src as far as the compiler knows, so a plain loop
 * keeps one iteration's loads in flight at a time.
 */
template <typename D> struct alignas(16) vec16 { D v[16 / sizeof(D)]; };

template <typename D, typename S>
struct flat_run {
	D *dp;
	const S *sp;
	int n;
	const xmgd_ptask_t &t;
	double &dre, &dim_;

	template <int OP, bool ONE>
	__device__ __forceinline__ void run()
	{
		int e0 = 0;
		if constexpr (std::is_same<D, S>::value) {
			if (((reinterpret_cast<uintptr_t>(dp) |
			    reinterpret_cast<uintptr_t>(sp)) & 15) == 0)
				e0 = vectors<OP, ONE>();
		}
		const scalars<D, S> c(t);
#pragma unroll 4
		for (int e = e0 + threadIdx.x; e < n; e += PT_THREADS) {
			const S y = op_reads_src(OP) ? sp[e] : S();
			const D x = combine<OP, ONE>(op_reads_dst(OP) ? dp[e] : D(), y, c, dre,
			    dim_);
			if (OP != XMGD_OP_DOT)
				dp[e] = x;
		}
	}

	/* whole vectors; the number of elements done */
	template <int OP, bool ONE>
	__device__ __forceinline__ int vectors()
	{
		/* (an FP64 division needs the registers of two vectors more) */
		constexpr bool f64 = std::is_same<D, double>::value || std::is_same<D, cd>::value;
		constexpr int W = 16 / sizeof(D), U = OP == XMGD_OP_DIV && f64 ? 2 : 4;
		vec16<D> *dv = reinterpret_cast<vec16<D> *>(dp);
		const vec16<D> *sv = reinterpret_cast<const vec16<D> *>(sp);
		const int nv = n / W;
		const scalars<D, S> c(t);

		for (int e0 = threadIdx.x; e0 < nv; e0 += U * PT_THREADS) {
			vec16<D> x[U], y[U];
#pragma unroll
			for (int u = 0; u < U; u++) {
				const int e = e0 + u * PT_THREADS;
				if (e < nv) {
					if (op_reads_dst(OP))
						x[u] = dv[e];
					if (op_reads_src(OP))
						y[u] = sv[e];
				}
			}
#pragma unroll
			for (int u = 0; u < U; u++) {
				const int e = e0 + u * PT_THREADS;
				if (e >= nv)
					break;
#pragma unroll
				for (int w = 0; w < W; w++)
					x[u].v[w] = combine<OP, ONE>(x[u].v[w], y[u].v[w], c, dre,
					    dim_);
				if (OP != XMGD_OP_DOT)
					dv[e] = x[u];
			}
		}
		return nv * W;
	}
};

static __device__ inline void
outer_offsets(const xmgd_ptask_t &t, int first_dim, int64_t o, int64_t &od,
    int64_t &os)
{
	od = 0;
	os = 0;
	for (int d = first_dim; d < t.ndim; d++) {
		const uint32_t sz = (uint32_t)t.size[d];
		int64_t q;
		if ((uint64_t)o >> 32) {
			q = o % sz;
			o /= sz;
		} else {	/* a 64-bit division costs about a hundred instructions */
			q = (uint32_t)o % sz;
			o = (uint32_t)o / sz;
		}
		od += q * t.dst_stride[d];
		os += q * t.src_stride[d];
	}
}

/* e / d by one multiplication, exact for e, d < 2^16 */
struct fastdiv {
	uint32_t d, mg;
	__device__ __forceinline__ explicit fastdiv(uint32_t d_) : d(d_), mg(0xffffffffu / d_ + 1) {}
	__device__ __forceinline__ uint32_t operator()(uint32_t e) const
	{ return d == 1 ? e : __umulhi(e, mg); }
};

/*
 * Tile schedule: a w0 x w1 tile of dims 0 (the destination's smallest
 * stride) and 1 (unit stride in src, w1 <= 32).  Loads have 2^l1 lanes along
 * dim 1, stores a warp along dim 0 in 2^lb blocks; a thread's loads of both
 * sides are issued together, and the source goes through shared memory with
 * an odd row pitch.  The kernel is bound by instruction issue, then HBM: a
 * flattened walk (multiplications to find each element's place, 165 issue
 * slots per element in all) moved 2 x 0.76 GB in 440 us; with fixed lanes
 * places advance by additions.
 */
template <typename D, typename S>
struct tile_run {
	D *dst;
	const S *src;
	int w0, w1, l1, lb;
	int64_t ss0, ds0, ds1;
	S *tile;
	const xmgd_ptask_t &t;
	double &dre, &dim_;

	template <int OP, bool ONE>
	__device__ __forceinline__ void run()
	{
		constexpr int U = tile_elems(sizeof(D), sizeof(S)) / PT_THREADS;
		constexpr int NW = PT_THREADS / 32;
		const int ld = w0 | 1;
		const int lx = threadIdx.x & 31, wy = threadIdx.x >> 5;
		const int l = threadIdx.x & ((1 << l1) - 1), r0 = threadIdx.x >> l1;
		const int rs = PT_THREADS >> l1, mask = (1 << lb) - 1;
		S y[U];
		D x[U];
		{
			const S *p = src + r0 * ss0 + l;
			const int64_t step = rs * ss0;
#pragma unroll
			for (int u = 0; u < U; u++, p += step)
				if (r0 + u * rs < w0 && l < w1)
					y[u] = *p;
		}
		/* store steps: block u & mask of dim 0, then dim 1 by NW */
		const int64_t da = 32 * ds0, db = NW * ds1 - mask * da;
		D *dp = dst + wy * ds1 + lx * ds0;
		if (op_reads_dst(OP)) {
			const D *p = dp;
#pragma unroll
			for (int u = 0; u < U; u++) {
				if (wy + NW * (u >> lb) < w1 && lx + 32 * (u & mask) < w0)
					x[u] = *p;
				p += ((u + 1) & mask) ? da : db;
			}
		}
		{
			S *p = tile + l * ld + r0;
#pragma unroll
			for (int u = 0; u < U; u++, p += rs)
				if (r0 + u * rs < w0 && l < w1)
					*p = y[u];
		}
		__syncthreads();
		const scalars<D, S> c(t);
		const S *tp = tile + wy * ld + lx;
		const int ta = 32, tb = NW * ld - mask * 32;
#pragma unroll
		for (int u = 0; u < U; u++) {
			if (wy + NW * (u >> lb) < w1 && lx + 32 * (u & mask) < w0) {
				x[u] = combine<OP, ONE>(x[u], *tp, c, dre, dim_);
				if (OP != XMGD_OP_DOT)
					*dp = x[u];
			}
			const bool in = ((u + 1) & mask) != 0;
			dp += in ? da : db;
			tp += in ? ta : tb;
		}
	}
};

/*
 * Slices schedule: k whole s0 x s1 slices (dims as above, both extents
 * small), flattened over the threads: with 16 x 16 slices, fixed lanes along
 * either run would leave half of them idle.  Strides fit 32 bits (checked on
 * the host), so that an element's place in its slice does too.
 */
template <typename D, typename S>
struct slice_run {
	D *dst;
	const S *src;
	int w0, w1, total;
	int ss0, ds0, ds1;
	const int64_t (*so)[SLICE_MAXQ];     /* slice offsets: dst, src */
	S *tile;
	const xmgd_ptask_t &t;
	double &dre, &dim_;

	template <int OP, bool ONE>
	__device__ __forceinline__ void run()
	{
		constexpr int U = slice_elems(sizeof(D), sizeof(S)) / PT_THREADS;
		/* steps that no thread has an element in are left out (20 million
		 * floats added in 4 x 4 slices: 327 us, now 240); four steps of
		 * 16-byte elements cost less than the branches (1.06) */
		constexpr bool SKIP = sizeof(D) <= 8;
		const int n = w0 * w1, ld = w0 | 1;
		const fastdiv by_n(n), by_w1(w1), by_w0(w0);
		S y[U];
		D x[U];
		uint32_t e0 = threadIdx.x;
#pragma unroll
		for (int u = 0; u < U; u++) {
			if (SKIP && u * PT_THREADS >= total)
				break;
			const uint32_t e = e0 + u * PT_THREADS;
			if ((int)e < total) {
				const uint32_t q = by_n(e), r = e - q * n;
				const int i0 = by_w1(r), i1 = r - i0 * w1;
				y[u] = (src + so[1][q])[i0 * ss0 + i1];
			}
		}
		if (op_reads_dst(OP)) {
#pragma unroll
			for (int u = 0; u < U; u++) {
				if (SKIP && u * PT_THREADS >= total)
					break;
				const uint32_t e = e0 + u * PT_THREADS;
				if ((int)e < total) {
					const uint32_t q = by_n(e), r = e - q * n;
					const int i1 = by_w0(r), i0 = r - i1 * w0;
					x[u] = (dst + so[0][q])[i1 * ds1 + i0 * ds0];
				}
			}
		}
		/* the places are computed again below: kept from above they
		 * would not fit the registers */
		asm volatile("" : "+r"(e0));
#pragma unroll
		for (int u = 0; u < U; u++) {
			if (SKIP && u * PT_THREADS >= total)
				break;
			const uint32_t e = e0 + u * PT_THREADS;
			if ((int)e < total) {
				const uint32_t q = by_n(e), r = e - q * n;
				const int i0 = by_w1(r), i1 = r - i0 * w1;
				tile[(q * w1 + i1) * ld + i0] = y[u];
			}
		}
		__syncthreads();
		const scalars<D, S> c(t);
#pragma unroll
		for (int u = 0; u < U; u++) {
			if (SKIP && u * PT_THREADS >= total)
				break;
			const uint32_t e = e0 + u * PT_THREADS;
			if ((int)e < total) {
				const uint32_t g = by_w0(e), q = by_n(e);
				const int i0 = e - g * w0, i1 = g - q * w1;
				x[u] = combine<OP, ONE>(x[u], tile[g * ld + i0], c, dre, dim_);
				if (OP != XMGD_OP_DOT)
					(dst + so[0][q])[i1 * ds1 + i0 * ds0] = x[u];
			}
		}
	}
};

/* Row schedule: rows of w0 elements along dim 0, one after the other over
 * the CTA's threads; eight elements of a thread in flight at a time (four
 * of the 16-byte types). */
template <typename D, typename S>
struct row_run {
	D *dst;
	const S *src;
	int rows, w0;
	int64_t ds0, ss0;
	const int64_t (*so)[PT_THREADS];     /* row offsets: dst, src */
	const xmgd_ptask_t &t;
	double &dre, &dim_;

	template <int OP, bool ONE>
	__device__ __forceinline__ void run()
	{
		constexpr int U = sizeof(D) <= 8 && OP != XMGD_OP_DIV ? 8 : 4;
		const scalars<D, S> c(t);
		const int n = rows * w0;
		const fastdiv by_w0(w0);
		for (int e0 = threadIdx.x; e0 < n; e0 += U * PT_THREADS) {
			S y[U];
			D x[U];
#pragma unroll
			for (int u = 0; u < U; u++) {
				const uint32_t e = e0 + u * PT_THREADS;
				if ((int)e < n) {
					const uint32_t r = by_w0(e), i = e - r * w0;
					if (op_reads_src(OP))
						y[u] = src[so[1][r] + i * ss0];
					if (op_reads_dst(OP))
						x[u] = dst[so[0][r] + i * ds0];
				}
			}
#pragma unroll
			for (int u = 0; u < U; u++) {
				const uint32_t e = e0 + u * PT_THREADS;
				if ((int)e < n) {
					const uint32_t r = by_w0(e), i = e - r * w0;
					x[u] = combine<OP, ONE>(x[u], y[u], c, dre, dim_);
					if (OP != XMGD_OP_DOT)
						dst[so[0][r] + i * ds0] = x[u];
				}
			}
		}
	}
};

/* Four CTAs per SM for every schedule: with five (48 registers) flat runs
 * spill, and their sums and copies take 3 to 12 % longer. */
template <typename D, typename S, int MODE>
__global__ void __launch_bounds__(PT_THREADS, 4)
ptask_kernel(const __grid_constant__ task_pack pack,
    const xmgd_ptask_t *__restrict__ dtasks,
    const task_meta *__restrict__ dmeta, int ntasks, int64_t cta0,
    double *__restrict__ partial)
{
	constexpr int PARTS = is_cplx<D> ? 2 : 1;

	/* locate the task of this CTA */
	const int64_t cta = cta0 + blockIdx.x;
	const xmgd_ptask_t *tasks = dtasks ? dtasks : pack.t;
	const task_meta *meta = dtasks ? dmeta : pack.m;
	const int lo = last_at_most(ntasks, cta, [&](int i) { return meta[i].first_cta; });
	const xmgd_ptask_t &t = tasks[lo];
	const task_meta &m = meta[lo];
	int64_t local = cta - m.first_cta;
	D *dst = reinterpret_cast<D *>(t.dst);
	const S *src = reinterpret_cast<const S *>(t.src);
	const int op = t.op;
	double dre = 0, dim_ = 0;

	if constexpr (MODE == 2) {
		/* flat: consecutive threads take consecutive elements */
		const int chunk = m.rows_per_cta;
		const int64_t base = local * chunk;
		const int n = (int)(t.size[0] - base < chunk ? t.size[0] - base : chunk);
		with_op<D, S>(t, flat_run<D, S>{dst + base, src + base, n, t, dre, dim_});
	} else if constexpr (MODE == 0) {
		__shared__ int64_t so[2][PT_THREADS];
		int64_t s0 = t.size[0];
		int64_t c0 = local % m.ctas_d0;
		int64_t orow = (local / m.ctas_d0) * m.rows_per_cta;
		int64_t i0beg = c0 * ROW_ELEMS;
		int64_t w0 = s0 - i0beg < ROW_ELEMS ? s0 - i0beg : ROW_ELEMS;
		int rows = m.rows_per_cta;
		if (orow + rows > m.nouter)
			rows = (int)(m.nouter - orow);
		for (int r = threadIdx.x; r < rows; r += PT_THREADS) {
			int64_t od, os;
			outer_offsets(t, 1, orow + r, od, os);
			so[0][r] = od + i0beg * t.dst_stride[0];
			so[1][r] = os + i0beg * t.src_stride[0];
		}
		__syncthreads();
		with_op<D, S>(t, row_run<D, S>{dst, src, rows, (int)w0, t.dst_stride[0],
		    t.src_stride[0], so, t, dre, dim_});
	} else {
		__shared__ S tile[MODE == 1 ? tile_cap(tile_elems(sizeof(D), sizeof(S))) :
		    slice_cap(slice_elems(sizeof(D), sizeof(S)))];
		if constexpr (MODE == 1) {
			const uint32_t x = (uint32_t)local, d0 = m.ctas_d0, d1 = m.ctas_d1;
			const uint32_t y = x / d0, c0 = x - y * d0, o = y / d1, c1 = y - o * d1;
			const int b0 = c0 * m.t0, b1 = c1 * m.t1;
			int64_t od, os;
			outer_offsets(t, 2, o, od, os);
			od += b0 * t.dst_stride[0] + b1 * t.dst_stride[1];
			os += b0 * t.src_stride[0] + b1;
			with_op<D, S>(t, tile_run<D, S>{dst + od, src + os,
			    min(m.t0, t.size[0] - b0), min(m.t1, t.size[1] - b1), m.l1, m.lb,
			    t.src_stride[0], t.dst_stride[0], t.dst_stride[1], tile, t, dre,
			    dim_});
		} else {
			__shared__ int64_t so[2][SLICE_MAXQ];
			const int64_t o0 = local * m.rows_per_cta;
			const int k = (int)(m.nouter - o0 < m.rows_per_cta ? m.nouter - o0 :
			    m.rows_per_cta);
			if ((int)threadIdx.x < k)
				outer_offsets(t, 2, o0 + threadIdx.x, so[0][threadIdx.x],
				    so[1][threadIdx.x]);
			__syncthreads();
			with_op<D, S>(t, slice_run<D, S>{dst, src, t.size[0], t.size[1],
			    k * t.size[0] * t.size[1], (int)t.src_stride[0],
			    (int)t.dst_stride[0], (int)t.dst_stride[1], so, tile, t, dre, dim_});
		}
	}
	if (op == XMGD_OP_DOT) {
		/* the threads' sums: a warp per part adds eight of them to a lane,
		 * then its lanes.  A warp's addition takes 16 cycles of the FP64
		 * pipe, as long as 32 elements; a reduction in every warp took 88 of
		 * them, more than a CTA's 2304 products, and now 13 per part */
		__shared__ double s_red[PARTS][PT_THREADS];
		s_red[0][threadIdx.x] = dre;
		if (PARTS == 2)
			s_red[PARTS - 1][threadIdx.x] = dim_;
		__syncthreads();
		const int part = threadIdx.x >> 5, lane = threadIdx.x & 31;
		if (part < PARTS) {
			double a = s_red[part][lane];
#pragma unroll
			for (int w = 1; w < PT_THREADS / 32; w++)
				a += s_red[part][lane + 32 * w];
			for (int off = 16; off > 0; off >>= 1)
				a += __shfl_down_sync(0xffffffffu, a, off);
			if (lane == 0) {
				partial[2 * cta + part] = a;
				if (PARTS == 1)
					partial[2 * cta + 1] = 0;
			}
		}
	}
}

/* a bounded wait of the slab schedule gave up (set on the device, read
 * and cleared by the host after the launches) */
__device__ int g_slab_err;

/*
 * Slab schedule: rows_per_cta consecutive s0 x s1 slices per CTA, each
 * contiguous on both sides (source: dim 1 unit stride, dim 0 stride s1;
 * destination: dim 0 unit stride, dim 1 stride s0; slice q at q * s0 * s1
 * on both), 16-byte aligned.  One bulk copy brings the CTA's slices of the
 * source into shared memory (one instruction, where the slices schedule
 * issues a load per element); the source goes into a tile with an odd row
 * pitch, so that both the transposing pass (threads along the source's
 * run) and the storing pass (threads along the destination's run) touch
 * distinct banks; stores follow the destination's run.
 */
template <typename T>
__global__ void __launch_bounds__(PT_THREADS, 6)
slab_kernel(const __grid_constant__ task_pack pack,
    const xmgd_ptask_t *__restrict__ dtasks,
    const task_meta *__restrict__ dmeta, int ntasks, int64_t cta0)
{
	extern __shared__ __align__(16) unsigned char dsm[];
	__shared__ __align__(8) uint64_t bar;
	__shared__ int s_err;

	const int64_t cta = cta0 + blockIdx.x;
	const xmgd_ptask_t *tasks = dtasks ? dtasks : pack.t;
	const task_meta *meta = dtasks ? dmeta : pack.m;
	const int lo = last_at_most(ntasks, cta, [&](int i) { return meta[i].first_cta; });
	const xmgd_ptask_t &t = tasks[lo];
	const task_meta &m = meta[lo];
	const int s0 = t.size[0], s1 = t.size[1], n = s0 * s1;
	const int ld = s0 | 1;
	const int64_t o0 = (cta - m.first_cta) * m.rows_per_cta;
	const int k = (int)(m.nouter - o0 < m.rows_per_cta ? m.nouter - o0 :
	    m.rows_per_cta);
	const int kn = k * n;
	const uint32_t cbytes = (uint32_t)kn * (uint32_t)sizeof(T);
	const T *sb = reinterpret_cast<const T *>(dsm);
	T *tb = reinterpret_cast<T *>(dsm + cbytes);
	T *dst = reinterpret_cast<T *>(t.dst) + o0 * n;
	const T *src = reinterpret_cast<const T *>(t.src) + o0 * n;
	const T al = num<T>::mk(t.alpha);

	const uint32_t b = smem_u32(&bar);
	if (threadIdx.x == 0) {
		s_err = 0;
		mbar_init(b, 1);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		mbar_expect_tx(b, cbytes);
		bulk_g2s(smem_u32(dsm), src, cbytes, b);
	}
	const bool ok = mbar_wait(b, 0, &s_err, &g_slab_err, 1);
	/* every thread leaves together when the wait gave up */
	if (__syncthreads_or(!ok))
		return;
	/* source order e = q n + i0 s1 + i1 -> tile q s1 ld + i1 ld + i0 */
	{
		int q = threadIdx.x / n, r = threadIdx.x - q * n;
		int i0 = r / s1, i1 = r - i0 * s1;
		const int dq = PT_THREADS / n, dr = PT_THREADS - dq * n;
		const int d0 = dr / s1, d1 = dr - d0 * s1;
		for (int e = threadIdx.x; e < kn; e += PT_THREADS) {
			tb[(q * s1 + i1) * ld + i0] = sb[e];
			i1 += d1;
			if (i1 >= s1) { i1 -= s1; i0++; }
			i0 += d0;
			if (i0 >= s0) { i0 -= s0; q++; }
			q += dq;
		}
	}
	__syncthreads();
	/* destination order e = q n + i1 s0 + i0 */
	int q = threadIdx.x / n, r = threadIdx.x - q * n;
	int i1 = r / s0, i0 = r - i1 * s0;
	const int dq = PT_THREADS / n, dr = PT_THREADS - dq * n;
	const int d1 = dr / s0, d0 = dr - d1 * s0;
	for (int e = threadIdx.x; e < kn; e += PT_THREADS) {
		dst[e] = num<T>::mul(al, tb[(q * s1 + i1) * ld + i0]);
		i0 += d0;
		if (i0 >= s0) { i0 -= s0; i1++; }
		i1 += d1;
		if (i1 >= s1) { i1 -= s1; q++; }
		q += dq;
	}
}

/* the slab schedule for a task: slices per CTA (0 when the schedule does
 * not apply: xm_copy of one scalar type only), and the CTA's shared memory */
static int64_t
slab_shape(const xmgd_ptask_t &t, int dbytes, int sbytes, int64_t *smem)
{
	if (dbytes != sbytes || t.op != XMGD_OP_COPY || t.ndim < 2 || t.ndim > 3)
		return 0;
	const int64_t s0 = t.size[0], s1 = t.size[1], n = s0 * s1;
	const int64_t mt = sbytes <= 8 ? 48 : 32;
	if (s0 > mt || s1 > mt || s0 < 2 || s1 < 2 ||
	    t.dst_stride[0] != 1 || t.dst_stride[1] != s0 ||
	    t.src_stride[1] != 1 || t.src_stride[0] != s1 ||
	    (t.ndim == 3 && (t.dst_stride[2] != n || t.src_stride[2] != n)) ||
	    (n * sbytes) % 16 != 0 || ((t.dst | t.src) & 15) != 0)
		return 0;
	int64_t k = n * sbytes >= SLAB_CHUNK ? 1 : SLAB_CHUNK / (n * sbytes);
	const int64_t cap = t.ndim == 3 ? t.size[2] : 1;
	if (k > cap)
		k = cap;
	*smem = k * n * sbytes + k * s1 * (s0 | 1) * sbytes;
	return *smem <= SLAB_SMEM ? k : 0;
}

/*
 * Sums of the per-CTA partial dot products, per task (in the caller's order,
 * order[]): LANES threads stride over a task's CTAs, four loads in flight, so
 * the order of the additions depends on the batch alone.  A warp per task for
 * batches of short tasks; 1024 threads where a task has more than 256 CTAs: a
 * lone warp takes 360 us for the 37 000 partial sums of a 40-million-element
 * block, longer than its products.
 */
template <int LANES>
__global__ void __launch_bounds__(LANES == 32 ? 256 : LANES)
dot_sum_kernel(const __grid_constant__ task_pack pack,
    const task_meta *__restrict__ dmeta, const int *__restrict__ order, int ntasks,
    int64_t nctas, const double *__restrict__ partial, double *__restrict__ out)
{
	constexpr int U = 4;
	__shared__ double s_red[2][LANES / 32];
	const task_meta *meta = dmeta ? dmeta : pack.m;
	const int t = LANES == 32 ? blockIdx.x * 8 + threadIdx.x / 32 : blockIdx.x;
	const int lane = threadIdx.x % LANES;
	if (t >= ntasks)
		return;
	const int64_t end = t + 1 < ntasks ? meta[t + 1].first_cta : nctas;
	const double2 *p2 = reinterpret_cast<const double2 *>(partial);
	double a = 0, b = 0;
	for (int64_t c = meta[t].first_cta + lane; c < end; c += U * LANES) {
		double2 v[U];
#pragma unroll
		for (int u = 0; u < U; u++)
			v[u] = c + u * LANES < end ? p2[c + u * LANES] : make_double2(0, 0);
#pragma unroll
		for (int u = 0; u < U; u++) {
			a += v[u].x;
			b += v[u].y;
		}
	}
	for (int off = 16; off > 0; off >>= 1) {
		a += __shfl_down_sync(0xffffffffu, a, off);
		b += __shfl_down_sync(0xffffffffu, b, off);
	}
	if constexpr (LANES > 32) {
		if (lane % 32 == 0) {
			s_red[0][lane / 32] = a;
			s_red[1][lane / 32] = b;
		}
		__syncthreads();
		if (lane >= 32)
			return;
		a = lane < LANES / 32 ? s_red[0][lane] : 0;
		b = lane < LANES / 32 ? s_red[1][lane] : 0;
		for (int off = 16; off > 0; off >>= 1) {
			a += __shfl_down_sync(0xffffffffu, a, off);
			b += __shfl_down_sync(0xffffffffu, b, off);
		}
	}
	if (lane == 0) {
		const int o = order ? order[t] : t;
		out[2 * o] = a;
		out[2 * o + 1] = b;
	}
}

template <typename D, typename S>
static int
launch_slab(const task_pack &pack, const xmgd_ptask_t *dtasks, const task_meta *dmeta,
    int ntasks, int64_t cta0, int64_t n, int64_t smem)
{
	if constexpr (std::is_same<D, S>::value) {
		static bool attr = false;
		if (!attr) {
			XMG_CK(cudaFuncSetAttribute(slab_kernel<D>,
			    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SLAB_SMEM));
			attr = true;
		}
		slab_kernel<D><<<(unsigned)n, PT_THREADS, (size_t)smem, stream()>>>(
		    pack, dtasks, dmeta, ntasks, cta0);
		g_launches++;
		XMG_CK(cudaGetLastError());
		return XMG_OK;
	} else {
		return xmg_seterr(XMG_EINVAL, "slab schedule: scalar conversion");
	}
}

template <typename D, typename S>
static int
launch(const task_pack &pack, const xmgd_ptask_t *dtasks, const task_meta *dmeta,
    int ntasks, const int64_t *begin, int64_t slab_smem, double *dpartial)
{
	if (begin[5] > begin[4]) {
		int st = launch_slab<D, S>(pack, dtasks, dmeta, ntasks, begin[4],
		    begin[5] - begin[4], slab_smem);
		if (st)
			return st;
	}
	/* one launch per schedule, over that schedule's CTA range */
	for (int mode = 0; mode < 4; mode++) {
		const int64_t n = begin[mode + 1] - begin[mode];
		if (n <= 0)
			continue;
		switch (mode) {
		case 0: ptask_kernel<D, S, 0><<<(unsigned)n, PT_THREADS, 0, stream()>>>(
		    pack, dtasks, dmeta, ntasks, begin[mode], dpartial); break;
		case 1: ptask_kernel<D, S, 1><<<(unsigned)n, PT_THREADS, 0, stream()>>>(
		    pack, dtasks, dmeta, ntasks, begin[mode], dpartial); break;
		case 2: ptask_kernel<D, S, 2><<<(unsigned)n, PT_THREADS, 0, stream()>>>(
		    pack, dtasks, dmeta, ntasks, begin[mode], dpartial); break;
		case 3: ptask_kernel<D, S, 3><<<(unsigned)n, PT_THREADS, 0, stream()>>>(
		    pack, dtasks, dmeta, ntasks, begin[mode], dpartial); break;
		}
		g_launches++;
		XMG_CK(cudaGetLastError());
	}
	return XMG_OK;
}

static int
elem_bytes(int type)
{
	return type == 0 ? 4 : type == 3 ? 16 : 8;	/* float, cd; double, cf */
}

static bool
reads_src(const xmgd_ptask_t &t)
{
	return t.op != XMGD_OP_SET && t.op != XMGD_OP_SCALE;
}

/* the schedule of a task without slab (task_meta.mode); slice_n: elements of
 * a CTA's slices */
static int
schedule_of(const xmgd_ptask_t &t, int slice_n)
{
	const int64_t far = 1 << 24;

	if (t.ndim == 1 && t.dst_stride[0] == 1 && (!reads_src(t) || t.src_stride[0] == 1))
		return 2;
	if (t.ndim < 2 || t.src_stride[1] != 1 || t.src_stride[0] == 1 || !reads_src(t) ||
	    (t.size[0] <= ROW_THIN && t.size[1] > SLICE_MAX))
		return 0;
	return t.size[0] <= SLICE_MAX && t.size[1] <= SLICE_MAX &&
	    t.size[0] * t.size[1] <= slice_n && t.src_stride[0] < far &&
	    t.dst_stride[0] < far && t.dst_stride[1] < far ? 3 : 1;
}

/*
 * Schedule of every task of a batch.  Tasks are grouped by schedule (stable
 * within a group, order[] maps group position -> caller's index) so that
 * each schedule owns one contiguous CTA range [begin[m], begin[m+1]); meta
 * and the task copy follow the grouped order.
 */
static void
plan_tasks(const xmgd_ptask_t *tasks, int ntasks, int dtype, int stype,
    std::vector<xmgd_ptask_t> &sorted, std::vector<task_meta> &meta,
    std::vector<int> &order, int64_t begin[6], int64_t *slab_smem)
{
	std::vector<task_meta> m0((size_t)ntasks);
	std::vector<int64_t> cnt((size_t)ntasks);
	const int tile_n = tile_elems(elem_bytes(dtype), elem_bytes(stype));
	const int slice_n = slice_elems(elem_bytes(dtype), elem_bytes(stype));
	const char *e = getenv("XMG_PTASK_SLAB");
	const bool slab_on = !(e && strcmp(e, "0") == 0);

	/* slab beats slices on what does not stay in L2 (copies of 40 million
	 * elements in 16 x 16 slices: float 89 against 134 us, double 119 against
	 * 151; of 3 million 28 against 26, its flag's way to the host); with
	 * 16-byte elements only where slices leave a quarter of their CTAs empty
	 * or products with the scalar to do (20 million in 24 x 24: 167 against
	 * 190 us; in 20 x 20: 173 against 164, scaled 173 against 203) */
	const int esz = elem_bytes(stype);
	int64_t need = 0, whole = 0;
	auto slab_task = [&](const xmgd_ptask_t &t) {
		const int64_t k = slab_shape(t, elem_bytes(dtype), esz, &need);
		const int n = k > 0 ? t.size[0] * t.size[1] : 1;
		const bool one = t.alpha[0] == 1 && t.alpha[1] == 0;
		return esz == 16 && one && slice_n / n * n * 4 >= slice_n * 3 ? 0 : k;
	};
	for (int i = 0; i < ntasks && slab_on; i++)
		if (slab_task(tasks[i]) > 0)
			whole += (int64_t)tasks[i].size[0] * tasks[i].size[1] *
			    (tasks[i].ndim == 3 ? tasks[i].size[2] : 1) * esz;

	int64_t nflat = 0, nslice = 0;
	*slab_smem = 0;	/* the slab launch's: the largest of its CTAs' */
	for (int i = 0; i < ntasks; i++) {
		const xmgd_ptask_t &t = tasks[i];
		task_meta &m = m0[i];
		memset(&m, 0, sizeof m);
		const int64_t k = whole >= SLAB_MIN ? slab_task(t) : 0;
		if (k > 0) {
			m.mode = 4;
			m.nouter = t.ndim == 3 ? t.size[2] : 1;
			m.rows_per_cta = (int32_t)k;
			cnt[i] = (m.nouter + k - 1) / k;
			*slab_smem = std::max(*slab_smem, need);
			continue;
		}
		m.mode = schedule_of(t, slice_n);
		m.nouter = 1;
		if (m.mode == 2) {
			nflat += t.size[0];
		} else if (m.mode != 0) {
			const int s0 = t.size[0], s1 = t.size[1];
			for (int d = 2; d < t.ndim; d++)
				m.nouter *= t.size[d];
			if (m.mode == 3) {
				/* as many slices as the elements and the tile hold */
				const int q = std::min({slice_n / (s0 * s1),
				    slice_cap(slice_n) / (s1 * (s0 | 1)), SLICE_MAXQ});
				m.rows_per_cta = std::max(1, q);
				nslice += m.nouter * s0 * s1;
			} else {
				/* t1: the source's run in equal parts of at most 32;
				 * t0: what fills the steps of 2^l1 lanes, in whole
				 * 32-lane blocks */
				const int parts = (s1 + 31) / 32;
				m.t1 = (s1 + parts - 1) / parts;
				m.l1 = lanes_log2(m.t1);
				const int most = tile_n >> m.l1;
				m.t0 = std::min(s0, most);
				for (m.lb = 0; (32 << m.lb) < most; m.lb++)
					;
				m.ctas_d0 = (s0 + m.t0 - 1) / m.t0;
				m.ctas_d1 = (s1 + m.t1 - 1) / m.t1;
				cnt[i] = (int64_t)m.ctas_d0 * m.ctas_d1 * m.nouter;
			}
		} else {
			m.ctas_d0 = (t.size[0] + ROW_ELEMS - 1) / ROW_ELEMS;
			for (int d = 1; d < t.ndim; d++)
				m.nouter *= t.size[d];
			int64_t rows = t.size[0] >= ROW_ELEMS ? 1 :
			    ROW_ELEMS / t.size[0];
			if (rows > PT_THREADS)
				rows = PT_THREADS;
			m.rows_per_cta = (int32_t)rows;
			cnt[i] = (int64_t)m.ctas_d0 * ((m.nouter + rows - 1) / rows);
		}
	}
	/* flat CTAs of 8192 elements (4096 of 16 bytes: setting a block of 196
	 * million complex doubles 450 us with 8192, 430 with 4096), halved while
	 * they leave SMs without four of them (a small batch is bound by the
	 * latency of a CTA's passes: 33 000 elements divided in 6 CTAs took 52
	 * us) */
	int32_t chunk = elem_bytes(dtype) == 16 ? FLAT_ELEMS / 2 : FLAT_ELEMS;
	while (chunk > FLAT_MIN && nflat < (int64_t)chunk * 4 * num_sms())
		chunk /= 2;
	/* slices of a small batch: spread over two CTAs per SM in the same way */
	const int64_t each = std::max<int64_t>(PT_THREADS, nslice / (2 * num_sms()));
	for (int i = 0; i < ntasks; i++)
		if (m0[i].mode == 2) {
			m0[i].rows_per_cta = chunk;
			m0[i].ctas_d0 = (int32_t)((tasks[i].size[0] + chunk - 1) / chunk);
			cnt[i] = m0[i].ctas_d0;
		} else if (m0[i].mode == 3) {
			int32_t &q = m0[i].rows_per_cta;
			q = (int32_t)std::max<int64_t>(1, std::min<int64_t>(q, each /
			    (tasks[i].size[0] * tasks[i].size[1])));
			cnt[i] = (m0[i].nouter + q - 1) / q;
		}
	sorted.clear();
	meta.clear();
	order.clear();
	int64_t n = 0;
	for (int mode = 0; mode < 5; mode++) {
		begin[mode] = n;
		for (int i = 0; i < ntasks; i++)
			if (m0[i].mode == mode) {
				task_meta m = m0[i];
				m.first_cta = n;
				n += cnt[i];
				sorted.push_back(tasks[i]);
				meta.push_back(m);
				order.push_back(i);
			}
	}
	begin[5] = n;
}

static int
launch_types(int dtype, int stype, const task_pack &pack, const xmgd_ptask_t *dt, const task_meta *dm,
    int ntasks, const int64_t *begin, int64_t slab_smem, double *dp)
{
	int st;

#define L(D, S) st = launch<D, S>(pack, dt, dm, ntasks, begin, slab_smem, dp)
	if (dtype == stype) {
		switch (dtype) {
		case 0: L(float, float); break;
		case 1: L(cf, cf); break;
		case 2: L(double, double); break;
		case 3: L(cd, cd); break;
		default: st = xmg_seterr(XMG_EINVAL, "bad scalar type");
		}
	} else if (dtype == 2 && stype == 0) L(double, float);
	else if (dtype == 0 && stype == 2) L(float, double);
	else if (dtype == 3 && stype == 1) L(cd, cf);
	else if (dtype == 1 && stype == 3) L(cf, cd);
	else st = xmg_seterr(XMG_EINVAL, "unsupported scalar conversion");
#undef L
	return st;
}

static size_t
task_bytes(int ntasks)
{
	return ((size_t)ntasks * sizeof(xmgd_ptask_t) + 255) & ~(size_t)255;
}

} /* namespace xmg */

using namespace xmg;

extern "C" int
xmgd_ptask_stage(const xmgd_ptask_t *tasks, int ntasks, int stype,
    xmgd_ptask_batch_t *b)
{
	std::vector<xmgd_ptask_t> sorted;
	std::vector<task_meta> meta;
	std::vector<int> order;
	const size_t tb = task_bytes(ntasks);
	int st;

	memset(b, 0, sizeof *b);
	if (ntasks <= 0)
		return XMG_OK;
	/* batches staged for replay carry one type on both sides */
	plan_tasks(tasks, ntasks, stype, stype, sorted, meta, order, b->begin,
	    &b->slab_smem);
	if ((st = xmgd_alloc(tb + meta.size() * sizeof(task_meta), &b->dbuf)))
		return st;
	b->ntasks = ntasks;
	XMG_CK(cudaMemcpyAsync((void *)b->dbuf, sorted.data(), (size_t)ntasks *
	    sizeof(xmgd_ptask_t), cudaMemcpyHostToDevice, stream()));
	XMG_CK(cudaMemcpyAsync((void *)(b->dbuf + tb), meta.data(), meta.size() *
	    sizeof(task_meta), cudaMemcpyHostToDevice, stream()));
	/* the host copies are local: finish before returning */
	XMG_CK(cudaStreamSynchronize(stream()));
	return XMG_OK;
}

extern "C" int
xmgd_ptask_launch(int dtype, int stype, const xmgd_ptask_batch_t *b)
{
	if (b->ntasks <= 0)
		return XMG_OK;
	static const task_pack none = {};
	return launch_types(dtype, stype, none, (const xmgd_ptask_t *)b->dbuf,
	    (const task_meta *)(b->dbuf + task_bytes(b->ntasks)), b->ntasks,
	    b->begin, b->slab_smem, nullptr);
}

/* page-locked host memory of the element-wise calls: the batch on its way
 * to the device, the sums a dot product's last kernel writes, the slab
 * schedule's flag on its way back.  Grow-only; every call that uses it
 * waits for its kernels before it returns. */
static int
batch_pinned(size_t bytes, void **p)
{
	static void *buf;
	static size_t cap;

	if (cap < bytes) {
		if (buf)
			XMG_CK(cudaFreeHost(buf));
		buf = nullptr;
		cap = 0;
		XMG_CK(cudaMallocHost(&buf, bytes + bytes / 2 + 65536));
		cap = bytes + bytes / 2 + 65536;
	}
	*p = buf;
	return XMG_OK;
}

static int
run_batch(int dtype, int stype, const xmgd_ptask_t *tasks, int ntasks, double *dots)
{
	std::vector<xmgd_ptask_t> sorted;
	std::vector<task_meta> meta;
	std::vector<int> order;
	task_pack pack;
	int64_t begin[6], nctas, slab_smem;
	uint64_t dbuf = 0, dpart = 0;
	const task_meta *dmeta = nullptr;
	const int *dorder = nullptr;
	void *pin = nullptr;
	double *sums = nullptr;
	int *slab_err = nullptr;
	int st;

	if (ntasks <= 0)
		return XMG_OK;
	plan_tasks(tasks, ntasks, dtype, stype, sorted, meta, order, begin, &slab_smem);
	nctas = begin[5];
	const bool slab = begin[5] > begin[4];
	const size_t tb = task_bytes(ntasks);
	const size_t mb = ((size_t)ntasks * sizeof(task_meta) + 255) & ~(size_t)255;
	const size_t ob = ((size_t)ntasks * sizeof(int) + 255) & ~(size_t)255;
	const size_t db = dots ? 2 * (size_t)ntasks * sizeof(double) : 0;
	const bool small = ntasks <= PACK;
	bool inorder = true;
	for (int i = 0; i < ntasks; i++)
		inorder = inorder && order[i] == i;
	/* an out-of-order batch of dots needs its order on the device */
	const size_t up = small && (inorder || !dots) ? 0 : tb + mb + ob;
	/* (all memory before the first copy: from there on the page-locked buffer
	 * is in use until the wait below) */
	if ((up > 0 && (st = xmgd_scratch(2, up, &dbuf)) != XMG_OK) ||
	    (dots && (st = xmgd_scratch(3, (size_t)nctas * 2 * sizeof(double), &dpart)) !=
	    XMG_OK))
		return st;
	if (up + db + slab > 0) {
		if ((st = batch_pinned(up + db + 256, &pin)) != XMG_OK)
			return st;
		sums = (double *)((char *)pin + up);
		slab_err = (int *)((char *)pin + up + db);
	}
	if (up > 0) {
		char *h = (char *)pin;
		memcpy(h, sorted.data(), (size_t)ntasks * sizeof(xmgd_ptask_t));
		memcpy(h + tb, meta.data(), (size_t)ntasks * sizeof(task_meta));
		memcpy(h + tb + mb, order.data(), (size_t)ntasks * sizeof(int));
		XMG_CK(cudaMemcpyAsync((void *)dbuf, pin, up, cudaMemcpyHostToDevice,
		    stream()));
		dmeta = (const task_meta *)(dbuf + tb);
		dorder = (const int *)(dbuf + tb + mb);
	} else {
		memcpy(pack.t, sorted.data(), (size_t)ntasks * sizeof(xmgd_ptask_t));
		memcpy(pack.m, meta.data(), (size_t)ntasks * sizeof(task_meta));
	}
	st = launch_types(dtype, stype, pack, (const xmgd_ptask_t *)dbuf, dmeta, ntasks,
	    begin, slab_smem, (double *)dpart);
	if (st == XMG_OK && dots) {
		int64_t longest = 0;
		for (int i = 0; i < ntasks; i++)
			longest = std::max(longest, (i + 1 < ntasks ? meta[i + 1].first_cta : nctas) -
			    meta[i].first_cta);
		if (longest <= 256)
			dot_sum_kernel<32><<<(unsigned)((ntasks + 7) / 8), 256, 0, stream()>>>(pack,
			    dmeta, dorder, ntasks, nctas, (const double *)dpart, sums);
		else
			dot_sum_kernel<1024><<<(unsigned)ntasks, 1024, 0, stream()>>>(pack,
			    dmeta, dorder, ntasks, nctas, (const double *)dpart, sums);
		g_launches++;
		st = check(cudaGetLastError(), "dot_sum_kernel");
	}
	if (st == XMG_OK && slab)
		st = check(cudaMemcpyFromSymbolAsync(slab_err, g_slab_err, sizeof(int), 0,
		    cudaMemcpyDeviceToHost, stream()), "slab flag");
	/* the buffers are reused by the next batch: wait here */
	const int st2 = check(cudaStreamSynchronize(stream()), "ptask_kernel");
	if (st != XMG_OK || (st = st2) != XMG_OK)
		return st;
	if (slab && *slab_err) {
		const int zero = 0;
		XMG_CK(cudaMemcpyToSymbol(g_slab_err, &zero, sizeof zero));
		return xmg_seterr(XMG_ETIMEOUT, "slab schedule: a bulk copy did not complete "
		    "within the bounded wait");
	}
	if (dots)
		memcpy(dots, sums, db);
	return XMG_OK;
}

/* Whether a task would read elements that it may already have overwritten:
 * a permuted operation of a block onto itself, unless each CTA's slices, all
 * loaded before any is stored, map onto themselves. */
static bool
overtakes(const xmgd_ptask_t &t, int slice_n)
{
	bool same = true, outer = true;

	if (t.src != t.dst || !reads_src(t) || t.op == XMGD_OP_DOT)
		return false;
	for (int d = 0; d < t.ndim; d++) {
		const bool eq = t.size[d] == 1 || t.dst_stride[d] == t.src_stride[d];
		same = same && eq;
		outer = outer && (d < 2 || eq);
	}
	return !same && !(outer && schedule_of(t, slice_n) == 3 && t.dst_stride[0] == 1 &&
	    t.size[0] == t.size[1] && t.dst_stride[1] == t.src_stride[0]);
}

/* bytes from a task's first source element to the end of its last */
static size_t
src_bytes(const xmgd_ptask_t &t, int esz)
{
	size_t n = 1;

	for (int d = 0; d < t.ndim; d++)
		n += (size_t)(t.size[d] - 1) * (size_t)t.src_stride[d];
	return n * esz;
}

/* The tasks of a batch.  Those of a block onto itself whose stores could
 * overtake their loads read a copy of the block made before, of COPY_MAX
 * bytes of blocks at a time: as in the reference, which reads a block whole
 * before it writes it (xm.c:66-413), the block's old elements count. */
extern "C" int
xmgd_ptasks(int dtype, int stype, const xmgd_ptask_t *tasks, int ntasks,
    double *dots)
{
	constexpr size_t COPY_MAX = (size_t)256 << 20;
	const int esz = elem_bytes(stype), slice_n = slice_elems(elem_bytes(dtype), esz);
	std::vector<xmgd_ptask_t> now, copied;
	int st;

	for (int i = 0; i < ntasks; i++)
		if (overtakes(tasks[i], slice_n))
			copied.push_back(tasks[i]);
	if (copied.empty())
		return run_batch(dtype, stype, tasks, ntasks, dots);
	for (int i = 0; i < ntasks; i++)
		if (!overtakes(tasks[i], slice_n))
			now.push_back(tasks[i]);
	st = run_batch(dtype, stype, now.data(), (int)now.size(), dots);
	for (size_t first = 0, end; first < copied.size() && st == XMG_OK; first = end) {
		uint64_t mem, at;
		size_t n = 0;
		for (end = first; end < copied.size(); end++) {
			const size_t b = src_bytes(copied[end], esz);
			if (end > first && n + b > COPY_MAX)
				break;
			n += (b + 255) & ~(size_t)255;
		}
		if ((st = xmgd_alloc(n, &mem)) != XMG_OK)
			return st;
		at = mem;
		for (size_t i = first; i < end && st == XMG_OK; i++) {
			const size_t b = src_bytes(copied[i], esz);
			st = xmgd_d2d(at, copied[i].src, b);
			copied[i].src = at;
			at += (b + 255) & ~(size_t)255;
		}
		if (st == XMG_OK)
			st = run_batch(dtype, stype, &copied[first], (int)(end - first), nullptr);
		xmgd_free(mem);
	}
	return st;
}
