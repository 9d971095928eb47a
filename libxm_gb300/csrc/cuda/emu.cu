/*
 * Split-precision contraction on tcgen05 tensor cores.
 *
 * Replaces the reference's per-pair ?gemm_ calls (contract.c:193-218) for
 * every canonical output block whose merged pair factors are +-1 or +-2
 * (always the case for (anti)symmetric tensors).  Two schemes share the
 * code:
 *
 *   FP64 ("emulated FP64"): 6 signed 8-bit slices per element (47-bit
 *     fixed point), the 21 slice products with p + q <= 5; weight groups
 *     0, 1, 2 accumulate exactly, groups 3..5 form a rounded low band.
 *   FP32 ("compensated bf16 split"): 3 slices (23-bit fixed point), the 6
 *     products with p + q <= 2, all exact -- no FP32 rounding at all.
 *
 * Complex types use the real-GEMM decomposition: each complex operand view
 * is realified along K as [re | im] (each half padded to 16), and the
 * output is computed in two passes over the same slices,
 *     pass 0: re(C) = A_re B_re - A_im B_im   (second half drained negated)
 *     pass 1: im(C) = A_re B_im + A_im B_re   (B halves swapped)
 *
 * Kernels:
 *  1. emu_exp_kernel   - largest binary exponent of every free-index row of
 *     each operand view over all contracted elements (re and im), max-reduced
 *     into tables shared by all views with the same free block index, so
 *     every pair of an output block uses the same row/column scaling.
 *  2. emu_split_kernel - the unfold (permutation gather through the view's
 *     offset tables) fused with the split: each element becomes a fixed-
 *     point integer relative to its row exponent, cut into balanced base-256
 *     digits d_t in [-128, 128]; digit t is stored as bf16 d_t * 2^(-8t)
 *     (exact).  Integer and FP32 arithmetic only -- GB300's FP64 pipe runs at
 *     ~1 TFLOP/s.  The output is pre-tiled in the exact shared-memory image
 *     the MMA reads (no-swizzle K-major core matrices), so the GEMM loads a
 *     K step of a tile with one 1-D bulk copy per operand.
 *  3. emu_gemm_kernel  - persistent, items of (output blocks, 128 x <= 128
 *     tile, pass);
 *     warp 0 streams stages with cp.async.bulk, warp 1 issues the slice
 *     products per 16-wide K step with tcgen05.mma.kind::f16 (bf16 x bf16 ->
 *     fp32) into TMEM accumulators, warps 2..17 drain them every 256 K
 *     elements (groups 0 and 1 of FP32 every 512; the exact groups stay
 *     below 2^24, exact in fp32) into
 *     per-thread int64 fixed-point sums in units of 2^(-16-F), applying the
 *     pair factor exactly.  The epilogue is the only FP64 work:
 *     C = alpha * 2^(eA + eB - 2 * EXPOFF - 16 - F) * V + beta * C, scattered
 *     through the output block's fold tables.
 *
 * Every mbarrier wait is bounded (2 s of %globaltimer); on timeout the
 * kernel records an error, waits (bounded) for its own copies and MMAs,
 * frees TMEM and returns, and the host reports XMG_ETIMEOUT.
 */
#include <algorithm>
#include <map>
#include <math.h>
#include <stdlib.h>
#include <string.h>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "tc.cuh"

namespace xmg {

constexpr int EMU_TM = 128;              /* rows per tile, both operands */
constexpr int EMU_KS = 16;               /* K per stage = K per MMA */
constexpr int EMU_CHUNK = 16;            /* K steps per chunk, FP64 (256) */
constexpr int EMU_CHUNK32 = 16;          /* K steps per chunk, FP32 (256) */
constexpr int SLICE_BYTES = EMU_TM * EMU_KS * 2;          /* 4096 */
#ifndef EMU_DW
#define EMU_DW 16                        /* drain warps: 8 or 16 */
#endif
constexpr int STAGE_BUDGET = 196608;                      /* 192 KiB */

/* input element traits: slices, kept products, fixed-point bits */
template <typename T> struct fin;
template <> struct fin<double> {
	static constexpr int S = 6, KEEP = 5, T1 = 47, MANT = 52, EMAX = 0x7ff;
	static constexpr int EXPOFF = 47 + 1022 - 8 * (6 - 1);    /* 1029 */
	/* the 32-bit word that holds the exponent, and the exponent in it */
	__device__ static inline int eword(const double *p)
	{ return __ldg(reinterpret_cast<const int *>(p) + 1); }
	__device__ static inline int bexp(int w) { return (w >> 20) & 0x7ff; }
};
template <> struct fin<float> {
	static constexpr int S = 3, KEEP = 2, T1 = 23, MANT = 23, EMAX = 0xff;
	static constexpr int EXPOFF = 23 + 126 - 8 * (3 - 1);     /* 133 */
	__device__ static inline int eword(const float *p)
	{ return __ldg(reinterpret_cast<const int *>(p)); }
	__device__ static inline int bexp(int w) { return (w >> 23) & 0xff; }
};

/* One work item: up to EMU_MAXMEM output blocks (members mfirst ..
 * mfirst + mcount - 1) stacked along one side of a 128 x N tile that share
 * the other side; pr = pass (bit 0) | swap (bit 1) | M-stacked (bit 2) |
 * live N rows in all << 8 (a multiple of 16).  Without swap b's view is
 * the M side (TMEM lanes) and a's the N side (TMEM columns); swap
 * exchanges them.
 *   N-stacked: m0 is the shared M-side tile (rows m0 .. m0 + 127 of the
 *     M-side view); each member is an N-side tile of its block at TMEM
 *     columns off .. off + rows - 1 (rows a multiple of 16).
 *   M-stacked: m0 is the shared N-side tile; each member is an M-side
 *     tile of its block at TMEM lanes off .. off + rows - 1 (off and rows
 *     multiples of 32, so a drain warp's lanes lie in one member).
 * Members share the other side pair by pair: the same view and K at every
 * pair index. */
struct emu_item {
	int32_t m0, mfirst, mcount, pr;
	int32_t cfirst, ccount;      /* its chunks */
	int32_t p0, k0, steps;       /* first pair, first K step in it, K steps */
	int32_t slot, parts;         /* sums shared by this many items (below) */
};

/* Where a list leaves SMs idle, the K steps of an item are divided among
 * several (split_items).  Each adds its 64-bit sums to the slot's, warp by warp,
 * and the warp that finds itself the last one of its place runs the epilogue on
 * the total: integers, so that the order does not matter.  A slot: 16 warps x
 * 32 columns x 32 lanes of sums, then the warps' counters. */
constexpr size_t SLOT_SUMS = (size_t)EMU_DW * (128 / (EMU_DW / 4)) * 32;
constexpr size_t SLOT_BYTES = SLOT_SUMS * 8 + 256;

/* a member: output block, first row of its tile in that block's view on
 * the stacked side, live rows (rounded up), first TMEM column or lane */
struct emu_member {
	int32_t cblock, n0, rows, off;
};
constexpr int EMU_MAXMEM = 4;

struct view_meta {
	int64_t first_cta;
};

/* rows of the tile that starts at row r0 of a view with mn rows: the live
 * ones rounded up to 16, at most 128 */
__host__ __device__ __forceinline__ int tile_rows(int mn, int r0)
{
	const int r = (mn - r0 + 15) / 16 * 16;
	return r < EMU_TM ? r : EMU_TM;
}

/* the view of a CTA: the last one whose first CTA is <= cta */
__device__ __forceinline__ int find_view(const view_meta *m, int n, int64_t cta)
{
	return last_at_most(n, cta, [&](int i) { return m[i].first_cta; });
}

/* Place of the real (half 0) or imaginary part of the element at row + col of
 * a complex block, counted in parts: a block's elements number below 2^31, its
 * parts do not. */
__host__ __device__ __forceinline__ int64_t part_at(int32_t row, int32_t col, int half)
{
	return 2 * (int64_t)(row + col) + half;
}

/* Element (k', r) of a view: real views directly, complex views realified
 * along K as [re | im] with halves of w.khp (zero padding). */
template <typename T>
__device__ __forceinline__ T fetch(const T *X, const int32_t *rowt, int32_t co,
    const xmgd_view_t &w, int k)
{
	if (!w.cplx) {
		return k < w.k ? X[rowt[k] + co] : T(0);
	}
	const int half = k >= w.khp;
	const int kk = k - half * w.khp;
	return kk < w.k ? X[part_at(rowt[kk], co, half)] : T(0);
}

/* ------------------------------------------------------------------ */
/* 1. exponent tables                                                  */

/* CTA = (view, 128-row tile, K range of kr elements).  The kernel is bound
 * by HBM on large operands and by the latency of its loads on small ones,
 * so a thread's loads are issued in batches of eight before any of them is
 * used (only the word with the exponent is loaded), and the host halves kr
 * until the grid covers the chip.  Indices past the range are clamped: a
 * maximum may see an element twice. */
template <typename T>
__global__ void __launch_bounds__(256)
emu_exp_kernel(const xmgd_view_t *__restrict__ views,
    const view_meta *__restrict__ meta, int nviews, int kr,
    const int32_t *__restrict__ tabs, int32_t *__restrict__ E,
    int *__restrict__ flags)
{
	const int v = find_view(meta, nviews, blockIdx.x);
	const xmgd_view_t w = views[v];
	const int local = (int)(blockIdx.x - meta[v].first_cta);
	const int nkb = (w.k + kr - 1) / kr;
	const int rt = local / nkb, kb = local % nkb;
	const T *X = reinterpret_cast<const T *>(w.ptr);
	const int32_t *rowt = tabs + w.rowtab, *colt = tabs + w.coltab;
	const int k0 = kb * kr, klast = min(w.k, k0 + kr) - 1;
	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	int bad = 0;

	if (w.kfast) {
		/* K runs along memory: a warp walks K for four rows at a time,
		 * directly when K is one contiguous run */
		const bool direct = w.kcontig && !w.cplx;
		const T *base = X + rowt[0];
		for (int r0 = rt * EMU_TM + warp * 16; r0 < min(w.mn, rt * EMU_TM +
		    warp * 16 + 16); r0 += 4) {
			int32_t co[4];
			int e[4] = {0, 0, 0, 0};
#pragma unroll
			for (int j = 0; j < 4; j++)
				co[j] = colt[min(r0 + j, w.mn - 1)];
			for (int k = k0 + lane; k <= klast; k += 64) {
				const int ka = k, kc = min(k + 32, klast);
				int x[4][2];
				if (direct) {
#pragma unroll
					for (int j = 0; j < 4; j++) {
						x[j][0] = fin<T>::eword(base + co[j] + ka);
						x[j][1] = fin<T>::eword(base + co[j] + kc);
					}
				} else if (!w.cplx) {
					const int32_t ra = rowt[ka], rc = rowt[kc];
#pragma unroll
					for (int j = 0; j < 4; j++) {
						x[j][0] = fin<T>::eword(X + ra + co[j]);
						x[j][1] = fin<T>::eword(X + rc + co[j]);
					}
				} else {
					const int32_t ra = rowt[ka], rc = rowt[kc];
#pragma unroll
					for (int j = 0; j < 4; j++) {
						const T *pa = X + part_at(ra, co[j], 0), *pc = X + part_at(rc, co[j], 0);
						const int a = fin<T>::eword(pa), b = fin<T>::eword(pc);
						const int p = fin<T>::eword(pa + 1), q = fin<T>::eword(pc + 1);
						x[j][0] = fin<T>::bexp(a) > fin<T>::bexp(p) ? a : p;
						x[j][1] = fin<T>::bexp(b) > fin<T>::bexp(q) ? b : q;
					}
				}
#pragma unroll
				for (int j = 0; j < 4; j++)
					e[j] = max(e[j], max(fin<T>::bexp(x[j][0]),
					    fin<T>::bexp(x[j][1])));
			}
			int mine = 0;
#pragma unroll
			for (int j = 0; j < 4; j++) {
				const int m = __reduce_max_sync(0xffffffffu, e[j]);
				bad |= m == fin<T>::EMAX;
				mine = lane == j ? m : mine;
			}
			if (lane < 4 && r0 + lane < w.mn && mine > E[w.exptab + r0 + lane])
				atomicMax(&E[w.exptab + r0 + lane], mine);
		}
	} else {
		/* free index contiguous: a thread per row, two K halves */
		const int rr = threadIdx.x % EMU_TM, half = threadIdx.x / EMU_TM;
		const int r = rt * EMU_TM + rr;
		if (r < w.mn) {
			const T *xr = X + (w.cplx ? 2 : 1) * (int64_t)colt[r];
			int e = 0;
			for (int k = k0 + half; k <= klast; k += 16) {
				int x[8];
				if (!w.cplx) {
#pragma unroll
					for (int j = 0; j < 8; j++)
						x[j] = fin<T>::eword(xr + rowt[min(k + 2 * j, klast)]);
				} else {
#pragma unroll
					for (int j = 0; j < 8; j++) {
						const T *p = xr + 2 * (int64_t)rowt[min(k + 2 * j, klast)];
						const int a = fin<T>::eword(p), b = fin<T>::eword(p + 1);
						x[j] = fin<T>::bexp(a) > fin<T>::bexp(b) ? a : b;
					}
				}
#pragma unroll
				for (int j = 0; j < 8; j++)
					e = max(e, fin<T>::bexp(x[j]));
			}
			bad |= e == fin<T>::EMAX;
			if (e > 0 && e > E[w.exptab + r])
				atomicMax(&E[w.exptab + r], e);
		}
	}
	if (bad)
		atomicOr(flags, 1);	/* Inf/NaN: not representable by slices */
}

/* ------------------------------------------------------------------ */
/* 2. unfold + split                                                   */

/*
 * An element as digits: Z = X + 128 (1 + 2^8 + ... + 2^(8 (S - 1))), X =
 * round(m * 2^(eb - er - (MANT + 1 - T1))) with the element's sign, halves
 * away from zero, |X| <= 2^T1.  The bias turns X's balanced digits into the
 * bytes of Z (the top one may be 256): no carries between digits.  With y =
 * 2 |X| cut to an integer, X is floor((y + 1) / 2) or -floor((y + 1) / 2) =
 * floor(-y / 2), so one complement, one addition of the doubled bias and one
 * shift serve both signs and the rounding.
 */
struct digits64 { uint32_t lo, hi; };
__device__ __forceinline__ digits64 digits_of(double x, int er)
{
	const unsigned long long b = (unsigned long long)__double_as_longlong(x);
	const uint32_t lo = (uint32_t)b, hi = (uint32_t)(b >> 32);
	const uint32_t e = (hi >> 20) & 0x7ff;
	const uint32_t mh = (hi & 0xFFFFF) | (e ? 0x100000u : 0u);
	const uint32_t sh = min(er - (int)max(e, 1u) + (fin<double>::MANT - fin<double>::T1), 63);
	/* (a funnel shift clamps at 32) */
	const uint32_t yl = __funnelshift_rc(lo, mh, sh) >> max((int)sh - 32, 0);
	const uint32_t yh = __funnelshift_rc(mh, 0, sh);
	const uint32_t s = (uint32_t)((int)hi >> 31);
	const unsigned long long z = (((unsigned long long)(yh ^ s) << 32) | (yl ^ s)) +
	    0x1010101010101ull;
	return digits64{(uint32_t)(z >> 1), (uint32_t)(z >> 33)};
}

struct digits32 { uint32_t lo; };
__device__ __forceinline__ digits32 digits_of(float x, int er)
{
	const uint32_t b = __float_as_uint(x), e = (b >> 23) & 0xff;
	const uint32_t m2 = (b << 1 & 0xFFFFFE) | (e ? 0x1000000u : 0u);
	const uint32_t sh = min(er - (int)max(e, 1u) + 1, 31);
	return digits32{((m2 >> sh ^ (uint32_t)((int)b >> 31)) + 0x1010101u) >> 1};
}

/* digit t of S as the float d * 2^(-8 t): its byte below the magic number
 * whose last place is 2^(-8 t), less that number and the bias */
template <int S, int T, typename D>
__device__ __forceinline__ uint32_t digit_bits(const D &z)
{
	constexpr uint32_t magic = (uint32_t)(0x4B - 4 * T) << 24;
	constexpr int byte = S - 1 - T;
	uint32_t w;
	if constexpr (S == 3)
		w = T == 0 ? magic | z.lo >> 16 : __byte_perm(z.lo, magic, 0x7540 | byte);
	else if constexpr (T <= 1)
		w = T == 0 ? magic | z.hi >> 8 : __byte_perm(z.hi, magic, 0x7540);
	else
		w = __byte_perm(z.lo, magic, 0x7540 | byte);
	constexpr float c = (8388608.0f + 128.0f) / (float)(1ull << (8 * T));
	return __float_as_uint(__uint_as_float(w) - c);
}

template <int S, int T, typename D>
__device__ __forceinline__ void digit_pairs(const D &a, const D &b, uint32_t (&bits)[S][4],
    int q)
{
	if constexpr (T < S) {
		/* (bf16 is exact: the digits' upper halves) */
		bits[T][q] = __byte_perm(digit_bits<S, T>(a), digit_bits<S, T>(b), 0x7632);
		digit_pairs<S, T + 1>(a, b, bits, q);
	}
}

/* CTA = (view, 128-row tile, group of 4 K steps); thread = (row, K octet).
 * The bytes (8 read and 12 written per double, 4 and 6 per float) bound it;
 * the digits take some 40 and 25 instructions per element.  Where K is one
 * contiguous run and a thread's octet lies on a 16-byte boundary, it is
 * loaded as 16-byte words, a quarter to a half of the requests for the same
 * sectors.  With 64-bit shifts, a carry from digit to digit and 8-byte loads
 * (some 100 and 76 instructions) both kernels of this pass together took 587
 * us for the operands of a 53 x 187 ladder (0.87 GB read twice, 1.2 GB
 * written), 1807 us for a float32 ring term's (2.1 GB, 3.2 GB); now 475 and
 * 1418. */
template <typename T>
__global__ void __launch_bounds__(256, 5)
emu_split_kernel(const xmgd_view_t *__restrict__ views,
    const view_meta *__restrict__ meta, int nviews,
    const int32_t *__restrict__ tabs, const int32_t *__restrict__ E, int rowmajor)
{
	constexpr int S = fin<T>::S;
	constexpr int CHUNK_ELEMS = S * SLICE_BYTES / 2;
	const int v = find_view(meta, nviews, blockIdx.x);
	const xmgd_view_t w = views[v];
	const int64_t local = blockIdx.x - meta[v].first_cta;
	const int ngrp = (w.n_ks + 3) / 4;
	const int rt = (int)(local / ngrp), g = (int)(local % ngrp);
	const int rr = threadIdx.x % EMU_TM, oct = threadIdx.x / EMU_TM;
	const int r = rt * EMU_TM + rr, tr = tile_rows(w.mn, rt * EMU_TM);
	const T *X = reinterpret_cast<const T *>(w.ptr);
	const int32_t *rowt = tabs + w.rowtab, *colt = tabs + w.coltab;
	const bool live = r < w.mn;
	const int32_t co = live ? colt[r] : 0;
	const int er = live ? E[w.exptab + r] : 0;
	uint16_t *out = reinterpret_cast<uint16_t *>(w.slices);
	/* a contiguous K run: direct loads, no offset table */
	const bool direct = w.kcontig && !w.cplx;
	const T *Xr = X + co + (direct ? rowt[0] : 0);
	/* (an octet is 32 or 64 bytes: the row's alignment is every octet's) */
	const bool wide = live && direct && ((uintptr_t)Xr & 15) == 0;
	if (rr >= tr)
		return;

	for (int ks = g * 4; ks < min(w.n_ks, g * 4 + 4); ks++) {
		const int k0 = ks * EMU_KS + oct * 8;
		T x[8];
		if (wide && k0 + 8 <= w.k) {
			constexpr int NW = 8 * sizeof(T) / 16, PER = 16 / sizeof(T);
			const uint4 *p = reinterpret_cast<const uint4 *>(Xr + k0);
			uint4 u[NW];
#pragma unroll
			for (int i = 0; i < NW; i++)
				u[i] = __ldg(p + i);
#pragma unroll
			for (int e = 0; e < 8; e++) {
				const uint4 q = u[e / PER];
				if constexpr (sizeof(T) == 8)
					x[e] = e % 2 ? __hiloint2double((int)q.w, (int)q.z) :
					    __hiloint2double((int)q.y, (int)q.x);
				else
					x[e] = __uint_as_float(e % 4 == 0 ? q.x : e % 4 == 1 ? q.y :
					    e % 4 == 2 ? q.z : q.w);
			}
		} else {
#pragma unroll
			for (int e = 0; e < 8; e++)
				x[e] = !live ? T(0) : direct ? (k0 + e < w.k ? Xr[k0 + e] : T(0)) :
				    fetch(X, rowt, co, w, k0 + e);
		}
		uint32_t bits[S][4];
#pragma unroll
		for (int q = 0; q < 4; q++)
			digit_pairs<S, 0>(digits_of(x[2 * q], er), digits_of(x[2 * q + 1], er), bits, q);
		/* chunk of a tile's live rows, rounded up to 16, in core matrices
		 * of 8 rows x 16 B, two per row group and slice.  Slice-major,
		 * [slice][8-row group]: consecutive slices follow one another
		 * like the rows of one wider operand.  Row-major, [8-row
		 * group][slice]: members' chunks stack by plain concatenation */
		const size_t chunk = (size_t)rt * w.n_ks * CHUNK_ELEMS +
		    (size_t)ks * (tr * EMU_KS * S);
		const size_t within = (size_t)(rr >> 3) * (rowmajor ? S * 128 : 128) +
		    oct * 64 + (rr & 7) * 8;
		const int ts = rowmajor ? 128 : tr * EMU_KS;
#pragma unroll
		for (int t = 0; t < S; t++) {
			uint4 val = make_uint4(bits[t][0], bits[t][1], bits[t][2], bits[t][3]);
			*reinterpret_cast<uint4 *>(out + chunk + t * ts + within) = val;
		}
	}
}

/* ------------------------------------------------------------------ */
/* 3. grouped tcgen05 GEMM with exact drains and the fused fold        */

/* |V| shifted up until its top bit is bit 63 (0 stays 0): words and shift */
struct norm64 { uint32_t hi, lo; int sh; };
__device__ __forceinline__ norm64 normalize(long long V)
{
	const unsigned long long a = V < 0 ? 0ull - (unsigned long long)V :
	    (unsigned long long)V;
	uint32_t hi = (uint32_t)(a >> 32), lo = (uint32_t)a;
	const bool low = hi == 0;
	hi = low ? lo : hi;
	lo = low ? 0 : lo;
	const int z = __clz(hi);
	return norm64{__funnelshift_l(lo, hi, z), lo << (z & 31), low ? z + 32 : z};
}

/* V * 2^e (sign flipped by sx) as a double, assembled in integer
 * arithmetic: |V| rounded once to 53 bits (to nearest, ties to even), the
 * exponent added to the mantissa with its leading bit, so that a carry out of
 * the rounding lands in the exponent.  A result out of the normal range is
 * scaled there by one multiplication.  Bit-identical to ldexp((double)V, e).
 * GB300's FP64 pipe is ~1/64 of its FP32 rate, so the epilogue keeps the
 * conversion and the scaling off it. */
__device__ __forceinline__ double pack_f64(long long V, int e, unsigned long long sx)
{
	const norm64 n = normalize(V);
	const int be = 63 - n.sh + e + 1023, bc = min(max(be, 1), 2045);
	const uint32_t lo = __funnelshift_r(n.lo, n.hi, 11), hi = n.hi >> 11;
	const uint32_t up = (n.lo & 0x7ff) + (lo & 1) > 0x400;
	const unsigned long long b = (((unsigned long long)hi << 32) | lo) + up +
	    ((unsigned long long)(bc - 1) << 52);
	const double v = __longlong_as_double((long long)((V ? b : 0ull) |
	    ((V < 0 ? 1ull << 63 : 0ull) ^ sx)));
	if (be == bc)
		return v;
	return v * __longlong_as_double((long long)(1023 + min(max(be - bc, -1022), 1023)) << 52);
}

/* A pipeline stage holds KSTEPS consecutive 16-wide K steps (each the
 * M-side chunk then the N-side chunk).  Smaller stages come back to the
 * producer sooner and leave less of a chunk to its head and tail; the price
 * is a barrier wait, a commit and the copies' arrival per stage.  With the
 * producer and MMA warps in step (mma_bf16_split) a stage costs the MMAs
 * nothing, and four stages of 48 KiB are best in both forms: one step of
 * the 6-slice form (GEMM of a 24 x 64 ladder 118 us with two steps in two
 * stages, 107 with one in four; 1.72 and 1.68 ms at 53 x 187; equal at 96 x
 * 384), two steps of the 3-slice form (float32 ring term, 64 x 256: 19.9 ms
 * with one step in eight stages, 19.2 with two in four, 19.8 with three in
 * three). */
template <int S>
struct stage_cfg {
#ifndef EMU_KSTEPS32
#define EMU_KSTEPS32 2
#endif
#ifndef EMU_BUDGET32
#define EMU_BUDGET32 196608                   /* 4 stages of 48 KiB */
#endif
#ifndef EMU_KSTEPS64
#define EMU_KSTEPS64 1                        /* 4 stages of 48 KiB */
#endif
	static constexpr int KSTEPS = S == fin<float>::S ? EMU_KSTEPS32 : EMU_KSTEPS64;
	static constexpr int BUDGET = S == fin<float>::S ? EMU_BUDGET32 : STAGE_BUDGET;
	static constexpr int CHUNK_BYTES = S * SLICE_BYTES;
	static constexpr int STEP_BYTES = 2 * CHUNK_BYTES;
	static constexpr int STAGE_BYTES = KSTEPS * STEP_BYTES;
	static constexpr int NST = BUDGET / STAGE_BYTES > 8 ? 8 :
	    BUDGET / STAGE_BYTES;
	static constexpr int SMEM = NST * STAGE_BYTES + 1024;
};

/* the end of the K segment holding step k: the pair, or the re/im half
 * of a realified complex view */
__device__ __forceinline__ int segment_end(int k, int nks, int cplx)
{
	return (cplx && k < nks / 2) ? nks / 2 : nks;
}

/* the stage that starts at step k holds steps [k, super_end): KSTEPS of
 * them, never past the segment's end */
template <int S>
__device__ __forceinline__ int super_end(int k, int nks, int cplx)
{
	return min(segment_end(k, nks, cplx), k + stage_cfg<S>::KSTEPS);
}

/* stages per pair: each segment in stages of KSTEPS steps */
template <int S>
__device__ __forceinline__ int stages_of(int nks, int cplx)
{
	constexpr int KS = stage_cfg<S>::KSTEPS;
	if (!cplx)
		return (nks + KS - 1) / KS;
	const int nh = nks / 2;
	return (nh + KS - 1) / KS + (nks - nh + KS - 1) / KS;
}

/*
 * Chunks and runs.  Set X (see below) is drained after each chunk of K steps,
 * set Y after each run of chunks.  An exact group g accumulates at most 3
 * products of |d_p d_q| <= 2^14 per K element, whose integer sum is exact in
 * fp32 up to 2^24, 341 elements.
 *   FP64: chunks of 256 elements of one pair, or half of a realified pair
 * (XMG_EMU_CHUNK steps, at most 20), each a run: the rounded low band's error
 * grows with the chunk (96 x 384 ladder: 3.1e-13 at 160, 4.4e-13 at 224,
 * 6.2e-13 at 320, against GEMM times of 35.8, 34.2 and 33.2 ms; chunks over
 * several short pairs took 15 % off an adjoint contraction's GEMM and doubled
 * its error).
 *   FP32, all exact: chunks of 256 elements that go on from one pair, or half,
 * to the next if their factors differ by a sign at most, the same for every
 * member of a stacked tile (the MMAs negate the M side then).  Group 2 (set X,
 * with two copies) is drained after each chunk, groups 0 and 1 (one and two
 * products) after two of them, unless a factor is 2: D0 is then at most 2^23,
 * D1 2^24, and D0 + D1 2^-8 below 2^24.  The drain of Y, 2700 cycles, had been
 * in the way of each chunk (float32 ring term, 64 x 256: 19.3 ms, now 16.9).
 * The host lists the chunks (chunk_lists); the MMA warp, short of issue slots
 * while the drains work, took some 500 cycles to put one together.
 */
struct emu_chunk {
	int32_t head;                /* stages | flags << 8 | the run's factors << 16:
				      * two bits per member, negative and twice */
	uint32_t neg, part;          /* per stage: negated; of one step (of two) */
	int32_t pad;
};
enum { RUN_FIRST = 1, RUN_LAST = 2, ITEM_LAST = 4 };

/*
 * Accumulators and MMAs of one K step.  Weight groups p + q = 0, 1, 2 have
 * an accumulator each (exact), 3..KEEP form the rounded low band.  FP64: the
 * low band is set X, the exact groups set Y; FP32: group 2 is X, 0 and 1 are
 * Y.  A slice of the M side times w consecutive slices of the N side is one
 * MMA of w * N columns when the accumulators of its w groups lie side by
 * side, since the slices of the N side follow one another in shared memory.
 * An MMA costs max(cols / 2, 28 + cols / 6) cycles, so fewer, wider ones
 * win.  Operands are read from shared memory at 128 B per cycle; the MMAs of
 * one M-side slice (4 KiB) follow one another and keep it in the tensor
 * core's buffer (at N = 128 a step's reads and copies then take 1248 cycles
 * against the MMAs' 1344, 1728 if each MMA read it again).  A step of 21
 * products, measured without copies: 1344 cycles at N = 128, 1014 at 96, 747
 * at 64 as in class 2; issued from one lane alone, with a barrier wait per
 * step, 1524, 1419 and 1419.  By the width N of a tile:
 *   class 0 (N <= 80): six accumulators, up to three slices: 9 MMAs;
 *   class 1 (N = 96): five (groups 4 and 5 share one), two slices: 15;
 *   class 2 (N > 96): four (3, 4, 5 share one), two slices: 17 (19 where X
 *     and Y are issued apart);
 *   class 3 (FP32): three, two slices within Y: 5;
 *   class 4: single products: CTA pairs (half of the N side in each CTA)
 *     and stacked tiles, whose members' slices do not follow one another.
 */
enum { SET_Y, SET_X, SET_ALL };

template <int S, int KEEP, int CLS, int SET>
struct prod {
	static constexpr int YTOP = KEEP > 2 ? 2 : 1;
	static constexpr int GLO = SET == SET_X ? YTOP + 1 : 0;
	static constexpr int GHI = SET == SET_Y ? YTOP : KEEP;
	static constexpr int W = CLS == 0 ? 3 : CLS == 4 ? 1 : 2;
	static constexpr int TOP = KEEP == 2 ? 2 : CLS == 0 ? 5 : CLS == 1 ? 4 : 3;
	/* accumulator of weight group g */
	static constexpr int acc(int g) { return g < TOP ? g : TOP; }
	/* slices of the MMA that starts with product (p, q) */
	static constexpr int width(int p, int q)
	{
		int w = 1;
		while (w < W && p + q + w <= GHI && q + w < S &&
		    acc(p + q + w) == acc(p + q + w - 1) + 1)
			w++;
		return w;
	}
};

/* what the MMAs of an item have in common */
struct mma_item {
	uint32_t idesc[3];           /* of one, two, three slices */
	uint32_t sa, sb;             /* slice strides of the descriptors */
	uint32_t sbo;                /* bytes between 8-row groups */
	uint32_t n;                  /* columns per accumulator */
	uint32_t neg;                /* instruction bit: M side negated */
};

/* the products of a set for one K step whose stage step starts at base;
 * acc0: 0 where they start the set's accumulators */
template <int S, int KEEP, int CLS, int SET, bool PAIR, int P = 0, int Q = -1>
__device__ __forceinline__ void
issue_set(const mma_item &m, uint32_t el, uint32_t tmem, uint32_t xcol, uint32_t alo, uint32_t ahi,
    uint32_t blo, uint32_t bhi, uint32_t acc0)
{
	using R = prod<S, KEEP, CLS, SET>;
	if constexpr (Q < 0) {
		constexpr int q0 = R::GLO > P ? R::GLO - P : 0;
		if constexpr (P < S)
			issue_set<S, KEEP, CLS, SET, PAIR, P, q0>(m, el, tmem, xcol, alo, ahi, blo, bhi, acc0);
	} else if constexpr (Q >= S || P + Q > R::GHI) {
		issue_set<S, KEEP, CLS, SET, PAIR, P + 1, -1>(m, el, tmem, xcol, alo, ahi, blo, bhi, acc0);
	} else {
		constexpr int w = R::width(P, Q), a = R::acc(P + Q);
		/* the first product of its accumulators: slice 0 of the M side
		 * with the first slice of each accumulator */
		constexpr bool first = P == 0 && (Q == R::GLO || R::acc(Q) != R::acc(Q - 1));
		/* FP32 alternates X between two fixed places */
		const uint32_t d = tmem + (KEEP == 2 && !PAIR && a == 2 ? xcol : a * m.n);
		const uint32_t acc = first ? acc0 : 1u;
		/* slice P stays in the buffer over its row of MMAs */
		constexpr bool row0 = Q == (R::GLO > P ? R::GLO - P : 0);
		constexpr bool row1 = Q + w >= S || P + Q + w > R::GHI;
		constexpr int COL = row0 && row1 ? COL_NONE : row0 ? COL_KEEP :
		    row1 ? COL_LAST : COL_USE;
		if constexpr (PAIR)
			mma_bf16_pair<COL>(el, d, alo + P * m.sa, ahi, blo + Q * m.sb, bhi,
			    m.idesc[0] | m.neg, acc);
		else
			mma_bf16_split<COL>(el, d, alo + P * m.sa, ahi, blo + Q * m.sb, bhi,
			    m.idesc[w - 1] | m.neg, acc);
		issue_set<S, KEEP, CLS, SET, PAIR, P, Q + w>(m, el, tmem, xcol, alo, ahi, blo, bhi, acc0);
	}
}

/* K steps of a pair of contracted extent k */
__device__ __forceinline__ int pair_steps(int k, int cplx)
{
	return (cplx ? 2 : 1) * ((k + EMU_KS - 1) / EMU_KS);
}

/*
 * Drain arithmetic.  A value x is rounded to an integer by fp32 adds and a
 * bit read, not by the conversion pipe (1/8 of the FMA pipe's rate): the
 * bits of x + M, M = 1.5 * 2^23, are those of M plus rint(x) for |x| < 2^22.
 * The bits of M stay in the sums and are subtracted once at the end.  64-bit
 * sums take shifted words and carries; a 32 x 32 -> 64 multiply-add costs
 * four issue slots (set Y of a chunk at N = 115: 4057 cycles with it, 3206 as
 * below, 3598 with a conversion per group; FP32's set X 1879 -> 1168).
 */
constexpr float MAGICF = 12582912.0f;
constexpr int MAGIC = 0x4B400000;

/* PAIR: a cluster of two CTAs runs each 256-row tile with cta_group::2
 * MMAs issued by rank 0: each CTA stages its own 128 M-side rows and half
 * of the N side, rank 1 forwards its stage completions to rank 0, the
 * drains of both CTAs read their own TMEM and release it to rank 0. */
template <int S, int KEEP, bool LOW, typename TOUT, int DW, bool PAIR>
__global__ void __launch_bounds__(64 + 32 * DW, 1)
emu_gemm_kernel(const emu_item *__restrict__ items, int nitems,
    const emu_member *__restrict__ members,
    const xmgd_cblock_t *__restrict__ cbs, const xmgd_pair_t *__restrict__ prs,
    const xmgd_view_t *__restrict__ va, const xmgd_view_t *__restrict__ vb,
    const int32_t *__restrict__ tabs, const int32_t *__restrict__ EA,
    const int32_t *__restrict__ EB, const int32_t *__restrict__ cbF,
    const emu_chunk *__restrict__ chunks, double alpha, double beta, int expoff2, int cplx,
    int hmax, int rowmajor,
    unsigned char *__restrict__ slots, int *__restrict__ flags)
{
	using C = stage_cfg<S>;
	constexpr int NST = C::NST;
	extern __shared__ __align__(1024) uint8_t smem_raw[];
	uint8_t *stages = reinterpret_cast<uint8_t *>(
	    (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
	__shared__ __align__(8) uint64_t bar_full[NST], bar_empty[NST];
	/* FP32 keeps two copies of set X (its third accumulator leaves room),
	 * used by the chunks in turn */
	constexpr bool XDB = KEEP == 2 && !PAIR;
	constexpr uint32_t XCOL = 256;       /* their columns: 256, 384 */
	__shared__ __align__(8) uint64_t bar_xfull, bar_xempty[2], bar_yempty, bar_fin;
	/* a chunk's products are done: two, since the MMA warp may finish a chunk
	 * whose Y goes on before the drains have seen the end of the last one */
	__shared__ __align__(8) uint64_t bar_yfull[2];
	__shared__ __align__(8) uint64_t bar_ifull[2], bar_iempty[2];
	/* the MMA warp's chunk, for the drains: its head */
	__shared__ __align__(8) uint64_t bar_info[2];
	__shared__ int s_head[2];
	__shared__ __align__(8) uint64_t bar_pfull[PAIR ? NST : 1];
	__shared__ int s_item[2];
	__shared__ uint32_t s_tmem;
	__shared__ volatile int s_err;
	int *g_err = flags + 1, *g_next = flags + 2;

	/* operands with Inf/NaN (flag set by the exponent kernel): write
	 * nothing, the host recomputes these blocks on the FP64 path */
	if (*(volatile int *)flags & 1)
		return;
	const int warp = __shfl_sync(0xffffffffu, threadIdx.x / 32, 0), lane = threadIdx.x % 32;
	const uint32_t rank = PAIR ? cluster_rank() : 0;
	/* bounded waits; in a pair, with cluster-scope acquire */
	auto wait = [&](uint32_t bar, uint32_t parity, int code) -> bool {
		if constexpr (PAIR)
			return mbar_wait_cl(bar, parity, &s_err, g_err, code);
		else
			return mbar_wait(bar, parity, &s_err, g_err, code);
	};
	/* arrive on a barrier of rank 0 (locally there, remotely from rank 1) */
	auto arrive0 = [&](uint64_t *bar) {
		if (!PAIR || rank == 0)
			mbar_arrive(smem_u32(bar));
		else
			mbar_arrive_remote(map_shared(smem_u32(bar), 0));
	};
	auto commit = [&](uint64_t *bar) {
		if constexpr (PAIR)
			mma_commit_pair(smem_u32(bar));
		else
			mma_commit(smem_u32(bar));
	};

	if (threadIdx.x == 0) {
		for (int s = 0; s < NST; s++) {
			mbar_init(smem_u32(&bar_full[s]), 1);
			mbar_init(smem_u32(&bar_empty[s]), 1);
		}
		mbar_init(smem_u32(&bar_xfull), 1);
		for (int q = 0; q < 2; q++) {
			mbar_init(smem_u32(&bar_yfull[q]), 1);
			mbar_init(smem_u32(&bar_xempty[q]), PAIR ? 2 * DW : DW);
		}
		mbar_init(smem_u32(&bar_yempty), PAIR ? 2 * DW : DW);
		mbar_init(smem_u32(&bar_fin), 1);
		for (int q = 0; q < 2; q++) {
			mbar_init(smem_u32(&bar_ifull[q]), 1);
			mbar_init(smem_u32(&bar_info[q]), 1);
			/* pair: both CTAs' drains, rank 0's MMA warp, rank 1's
			 * producer and forwarder */
			mbar_init(smem_u32(&bar_iempty[q]), PAIR ? 2 * DW + 3 : 1 + DW);
		}
		if (PAIR)
			for (int q = 0; q < NST; q++)
				mbar_init(smem_u32(&bar_pfull[q]), 1);
		s_err = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == 1) {
		if constexpr (PAIR) {
			asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;"
			    :: "r"(smem_u32(&s_tmem)));
			asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
		} else {
			asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;"
			    :: "r"(smem_u32(&s_tmem)));
			asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
		}
	}
	tc_fence_before();
	__syncthreads();
	if constexpr (PAIR)
		cluster_sync();	/* peers' barriers exist before any remote arrive */
	tc_fence_after();
	const uint32_t tmem = s_tmem;

	/* for the roles whose warp runs in step: the issuing lane, a value of
	 * lane 0 as a uniform one, a wait with one verdict */
	const uint32_t el = elect_lane();
	auto uni = [](auto v) { return __shfl_sync(0xffffffffu, v, 0); };
	auto wwait = [&](uint64_t *bar, uint32_t parity, int code) -> bool {
		return __all_sync(0xffffffffu, wait(smem_u32(bar), parity, code));
	};

	/* persistent: the producer takes the next item of the cost-sorted list
	 * from a global counter and passes its index to the MMA and drain
	 * warps through a two-slot ring (-1 ends); the stage ring and the
	 * accumulator phases carry across items */
	if (warp == 0) {
		/* ---------------- producer ----------------
		 * (in step, as the MMA warp; one lane issues) */
		int s = 0;
		uint32_t ph = 0;
		int lastp[NST];
#pragma unroll
		for (int q = 0; q < NST; q++)
			lastp[q] = -1;
		uint32_t iph = 0;
		bool ok = true;
		for (int slot = 0; ok; ) {
			int t = 0;
			if (!PAIR || rank == 0) {
				/* fetch the next item and hand it to every role */
				if (!wwait(&bar_iempty[slot], iph ^ 1, 5))
					break;
				if (lane == 0) {
					t = atomicAdd(g_next, 1);
					t = t < nitems ? t : -1;
					s_item[slot] = t;
					if (PAIR) {
						st_remote_u32(map_shared(smem_u32(&s_item[slot]), 1), (uint32_t)t);
						mbar_arrive_remote(map_shared(smem_u32(&bar_ifull[slot]), 1));
					}
					mbar_arrive(smem_u32(&bar_ifull[slot]));
				}
			} else {
				if (!wwait(&bar_ifull[slot], iph, 5))
					break;
				if (lane == 0) {
					t = s_item[slot];
					arrive0(&bar_iempty[slot]);
				}
			}
			t = uni(t);
			if (++slot == 2) { slot = 0; iph ^= 1; }
			if (t < 0)
				break;
			const emu_item it = items[t];
			const xmgd_cblock_t cb = cbs[members[it.mfirst].cblock];
			const int nmem = uni(it.mcount), npairs = uni(cb.npairs), pair0 = uni(cb.first_pair);
			const int pr0 = uni(it.pr), m0 = uni(it.m0);
			const int pass = pr0 & 1, swp = (pr0 >> 1) & 1, mstk = (pr0 >> 2) & 1;
			constexpr uint32_t ROWB = S * EMU_KS * 2;  /* a row's slices */
			/* the shared side: the M side's tile (this CTA's of the two
			 * in a pair) or, M-stacked, the N side's */
			const int stile = m0 / EMU_TM + (mstk ? 0 : (int)rank);
			const int slen = uni(mstk == swp ? cb.n : cb.m);
			/* (a pair's second M tile may lie past the view: its rows
			 * are then never stored) */
			const uint32_t sby = stile * EMU_TM < slen ?
			    tile_rows(slen, stile * EMU_TM) * ROWB : 0;
			/* the members: bytes copied per K step, bytes of their
			 * tile's chunk, place in the stage; one member, unless the
			 * list is stacked (row-major chunks); a pair stages half of
			 * its rows in each CTA */
			int mfp[EMU_MAXMEM], mrt[EMU_MAXMEM];
			uint32_t mby[EMU_MAXMEM], mch[EMU_MAXMEM], mdo[EMU_MAXMEM], stb = 0;
#pragma unroll
			for (int j = 0; j < EMU_MAXMEM; j++) {
				const emu_member mb = members[it.mfirst + (j < nmem ? j : 0)];
				const xmgd_cblock_t cj = cbs[mb.cblock];
				mfp[j] = uni(cj.first_pair);
				mrt[j] = uni(mb.n0) / EMU_TM;
				/* the stacked side: the N side (without swap a's rows)
				 * or, M-stacked, the M side */
				mch[j] = uni(tile_rows(mstk == swp ? cj.m : cj.n, mb.n0)) * ROWB;
				mby[j] = PAIR ? mch[j] / 2 : mch[j];
				mdo[j] = (mstk ? 0u : C::CHUNK_BYTES) + (uint32_t)uni(mb.off) * ROWB;
				stb += j < nmem ? mby[j] : 0;
			}
			const uint32_t mso = PAIR ? rank * mby[0] : 0;
			/* shared side from a's views when it is a's side */
			const bool sha = (mstk ^ swp) != 0;
			/* a pair's operand chunks: the shared side's tile and each
			 * member's */
			struct pair_src {
				unsigned long long gs, gn[EMU_MAXMEM];
				int k;
			};
			auto load_pair = [&](int p, pair_src &o) {
				/* the members' pair lists run in step: pair p of
				 * every member has member 0's view and K on the
				 * shared side */
				const xmgd_pair_t pr = prs[pair0 + p];
				o.k = pr.k;
				o.gs = sha ? va[pr.aview].slices : vb[pr.bview].slices;
#pragma unroll
				for (int j = 0; j < EMU_MAXMEM; j++) {
					if (j >= nmem)
						break;
					const xmgd_pair_t pj = prs[mfp[j] + p];
					o.gn[j] = sha ? vb[pj.bview].slices : va[pj.aview].slices;
				}
			};
			/* a view's tile, for all of the warp */
			auto tile_at = [&](unsigned long long slices, int tile, int nks) {
				return reinterpret_cast<const uint8_t *>(uni(slices)) +
				    (size_t)tile * nks * C::CHUNK_BYTES;
			};
			/* K step ks of a pair: the shared side reads at its own
			 * K index (the M side's or the N side's), the members at
			 * the other; the imaginary pass swaps B's re/im halves */
			auto kidx = [&](int ks, int nks, int &ksh, int &kst) {
				const int nh = nks / 2;
				const int kb = (cplx && pass) ? (ks < nh ? ks + nh : ks - nh) : ks;
				const int km = swp ? ks : kb, kn = swp ? kb : ks;
				ksh = mstk ? kn : km;
				kst = mstk ? km : kn;
			};
			/* the next pair's operand addresses are loaded while this
			 * one's steps are staged (two dependent loads) */
			pair_src nxt;
			int p = uni(it.p0), ks = uni(it.k0), todo = uni(it.steps);
			load_pair(p, nxt);
			for (; todo > 0 && ok; p++, ks = 0) {
				const int nks = pair_steps(uni(nxt.k), cplx);
				const uint8_t *gs = tile_at(nxt.gs, stile, nks), *gn[EMU_MAXMEM];
#pragma unroll
				for (int j = 0; j < EMU_MAXMEM; j++)
					if (j < nmem)
						gn[j] = tile_at(nxt.gn[j], mrt[j], nks) + mso;
				if (p + 1 < npairs)
					load_pair(p + 1, nxt);
				while (ks < nks && todo > 0) {
					const int ke = super_end<S>(ks, nks, cplx);
					if (!(ok = wwait(&bar_empty[s], ph ^ 1, 1)))
						break;
					uint32_t dst = smem_u32(stages + (size_t)s * C::STAGE_BYTES);
					const uint32_t fb = smem_u32(&bar_full[s]);
					if (el)
						mbar_expect_tx(fb, (uint32_t)(ke - ks) * (sby + stb));
					__syncwarp();
					/* (a stage's steps lie in one half of a realified view,
					 * so that both operands' chunks follow one another) */
					int ksh, kst;
					kidx(ks, nks, ksh, kst);
					const uint8_t *g = gs + (size_t)ksh * sby;
					for (int k = ks; k < ke; k++, kst++) {
						if (!PAIR || sby)
							bulk_g2s_el(el, dst + (mstk ? C::CHUNK_BYTES : 0u), g, sby, fb);
#pragma unroll
						for (int j = 0; j < EMU_MAXMEM; j++)
							if (j < nmem)
								bulk_g2s_el(el, dst + mdo[j],
								    gn[j] + (size_t)kst * mch[j], mby[j], fb);
						dst += C::STEP_BYTES;
						g += sby;
					}
#pragma unroll
					for (int q = 0; q < NST; q++)
						if (q == s)
							lastp[q] = (int)ph;
					if (++s == NST) { s = 0; ph ^= 1; }
					todo -= ke - ks;
					ks = ke;
				}
			}
		}
		/* on failure, let this CTA's copies still in flight land
		 * before it exits (bounded): the last phase issued on each
		 * stage completes when its bytes have arrived */
		if (s_err) {
			uint64_t t0 = gtimer();
#pragma unroll
			for (int q = 0; q < NST; q++)
				if (lastp[q] >= 0)
					while (!mbar_try(smem_u32(&bar_full[q]), (uint32_t)lastp[q]) &&
					    gtimer() - t0 < WAIT_NS)
						;
		}
	} else if (warp == 1 && PAIR && rank == 1) {
		/* ---------- rank 1: forward stage completions to rank 0 ---------- */
		if (lane == 0) {
			int s = 0;
			uint32_t ph = 0, iph = 0;
			for (int slot = 0; !s_err; ) {
				if (!wait(smem_u32(&bar_ifull[slot]), iph, 6))
					break;
				const int t = s_item[slot];
				arrive0(&bar_iempty[slot]);
				if (++slot == 2) { slot = 0; iph ^= 1; }
				if (t < 0)
					break;
				const xmgd_cblock_t cb = cbs[members[items[t].mfirst].cblock];
				for (int p = 0; p < cb.npairs && !s_err; p++) {
					const int nst_p = stages_of<S>(pair_steps(prs[cb.first_pair + p].k, cplx), cplx);
					for (int q = 0; q < nst_p; q++) {
						if (!wait(smem_u32(&bar_full[s]), ph, 3))
							break;
						mbar_arrive_remote(map_shared(smem_u32(&bar_pfull[s]), 0));
						if (++s == NST) { s = 0; ph ^= 1; }
					}
				}
			}
			/* rank 0's last MMAs (they write this CTA's TMEM) are done
			 * once the final commit lands here */
			uint64_t t0 = gtimer();
			while (!mbar_try_cl(smem_u32(&bar_fin), 0) && gtimer() - t0 < WAIT_NS)
				;
		}
	} else if (warp == 1) {
		/* ---------------- MMA issuer ----------------
		 * The warp runs in step, one lane issues (mma_bf16_split); what
		 * comes from memory is broadcast from lane 0, so that the MMAs'
		 * operands are uniform. */
		{
			const uint32_t tm = uni(tmem);
			int s = 0, prevn = 0;
			bool first = true;
			uint32_t ph = 0, xph = 0, yph = 0, nch = 0;
			uint32_t iph = 0;
			/* a stage is ready once this CTA's copies (and, in a pair,
			 * the peer's, forwarded) have landed */
			auto ready = [&](int st_, uint32_t par) -> bool {
				if (!wwait(&bar_full[st_], par, 3))
					return false;
				if (PAIR && !wwait(&bar_pfull[st_], par, 10))
					return false;
				tc_fence_after();
				return true;
			};
			auto done = [&](uint64_t *bar) {
				if (el)
					commit(bar);
				__syncwarp();
			};
			/* one item of a width class: its columns, M-side slice stride,
			 * chunks; false on failure (s_err set) */
			auto item = [&](auto cls, int n, uint32_t sa, int cfirst, int ccount) -> bool {
				constexpr int CLS = decltype(cls)::value;
				constexpr int KS = C::KSTEPS;
				mma_item mi;
				mi.n = n;
				for (int w = 0; w < 3; w++)
					mi.idesc[w] = PAIR ? idesc_pair_n(mi.n) : idesc_n((w + 1) * mi.n);
				mi.sbo = rowmajor ? S * 256 : 256;
				mi.sa = sa;
				mi.sb = rowmajor ? 16 : 2 * mi.n;
				/* accumulators of another width than the last item's lie
				 * across them: wait for both sets' drains */
				bool both = !XDB && !first && (int)mi.n != prevn;
				prevn = mi.n;
				const int4 *cp = reinterpret_cast<const int4 *>(chunks) + cfirst;
				int4 next = __ldg(cp);
				uint32_t ay = 0;
				for (bool more = true; more; ) {
						/* (the next chunk is loaded during this one) */
						more = --ccount > 0;
						const int head = uni(next.x) | (more ? 0 : ITEM_LAST << 8);
						const int fl = head >> 8, nss = head & 0xff;
						const uint32_t neg = uni(next.y), part = KS == 1 ? 0u : uni(next.z);
						if (more)
							next = __ldg(++cp);
						const uint32_t xcol = XCOL + (nch & 1) * 128;
						/* every accumulator restarts each chunk or run: the
						 * exact groups for their 2^24 bound, the low band
						 * because the tensor core's fp32 accumulation error
						 * grows with the accumulation length (per-pair
						 * accumulation measured 10x larger error) */
						uint32_t ax = 0;
						if (fl & RUN_FIRST)
							ay = 0;
						/* the products of stage sj, the chunk's j-th: set X
						 * (1), set Y (2) or both (3) */
						auto issue = [&](int sj, int j, auto which) {
							constexpr int WH = decltype(which)::value;
							const uint32_t base = smem_u32(stages + (size_t)sj * C::STAGE_BYTES);
							const int nk = KS == 1 || (part >> j & 1) ? 1 : KS;
							mi.neg = (neg >> j & 1) << 13;
							for (int u = 0; u < nk; u++) {
								const uint32_t b0 = base + u * C::STEP_BYTES;
								const uint64_t da = sdesc(b0, mi.sbo);
								const uint64_t db = sdesc(b0 + C::CHUNK_BYTES, mi.sbo);
								const uint32_t alo = (uint32_t)da, ahi = (uint32_t)(da >> 32);
								const uint32_t blo = (uint32_t)db, bhi = (uint32_t)(db >> 32);
								if constexpr (WH == 3 && CLS == 2 && KEEP > 2) {
									/* (a middle stage: both sets have started) */
									issue_set<S, KEEP, CLS, SET_ALL, PAIR>(mi, el, tm, xcol, alo,
									    ahi, blo, bhi, 1u);
									continue;
								}
								if constexpr (WH & 2) {
									issue_set<S, KEEP, CLS, SET_Y, PAIR>(mi, el, tm, xcol, alo, ahi,
									    blo, bhi, ay);
									ay = 1;
								}
								if constexpr (WH & 1) {
									issue_set<S, KEEP, CLS, SET_X, PAIR>(mi, el, tm, xcol, alo, ahi,
									    blo, bhi, ax);
									ax = 1;
								}
							}
						};
						const std::integral_constant<int, 1> X{};
						const std::integral_constant<int, 2> Y{};
						const std::integral_constant<int, 3> XY{};
						/* head: the first H (staged) stages, while Y is read;
						 * tail: the last T stages; middle: the rest.  H, T <=
						 * hmax <= NST: the stages a head or tail holds are
						 * released only after its set-Y products, so hmax < NST
						 * leaves stages for the producer to prefetch the steps
						 * after them */
						const bool ywait = !first && !both && (fl & RUN_FIRST);
						const int H = XDB && !ywait ? 0 : min(hmax, nss);
						const int T = XDB ? 0 : min(hmax, nss - H);
						/* head, set X, as soon as the drain has read X of
						 * the previous chunk (of the one before it, where X
						 * has two copies) */
						if (XDB) {
							if (nch >= 2 && !wwait(&bar_xempty[nch & 1],
							    ((nch >> 1) - 1) & 1, 2))
								return false;
						} else if (!first) {
							if (!wwait(&bar_xempty[0], xph, 2))
								return false;
							xph ^= 1;
						}
						if (both) {
							if (!wwait(&bar_yempty, yph, 8))
								return false;
							yph ^= 1;
						}
						tc_fence_after();
						/* (the drains have read what this slot held) */
						if (lane == 0) {
							const int z = nch & 1;
							s_head[z] = head;
							mbar_arrive(smem_u32(&bar_info[z]));
							if (PAIR) {
								st_remote_u32(map_shared(smem_u32(&s_head[z]), 1), (uint32_t)head);
								mbar_arrive_remote(map_shared(smem_u32(&bar_info[z]), 1));
							}
						}
						__syncwarp();
						for (int j = 0; j < H; j++) {
							const int sj = s + j < NST ? s + j : s + j - NST;
							if (!ready(sj, s + j < NST ? ph : ph ^ 1))
								return false;
							issue(sj, j, X);
						}
						if (T == 0 && !XDB)
							done(&bar_xfull);
						/* head, set Y, once Y is read too */
						if (ywait) {
							if (!wwait(&bar_yempty, yph, 8))
								return false;
							yph ^= 1;
						}
						first = both = false;
						tc_fence_after();
						for (int j = 0; j < H; j++) {
							const int sj = s + j < NST ? s + j : s + j - NST;
							issue(sj, j, Y);
							done(&bar_empty[sj]);
						}
						s += H;
						if (s >= NST) { s -= NST; ph ^= 1; }
						/* middle: every product per stage */
						for (int j = H; j < nss - T; j++) {
							if (!ready(s, ph))
								return false;
							issue(s, j, XY);
							done(&bar_empty[s]);
							if (++s == NST) { s = 0; ph ^= 1; }
						}
						/* tail: set X of the last T stages, then X is
						 * complete and its drain can start while the
						 * tensor core still works on set Y */
						for (int j = 0; j < T; j++) {
							const int sj = s + j < NST ? s + j : s + j - NST;
							if (!ready(sj, s + j < NST ? ph : ph ^ 1))
								return false;
							issue(sj, nss - T + j, X);
						}
						if (T > 0) {
							done(&bar_xfull);
							for (int j = 0; j < T; j++) {
								const int sj = s + j < NST ? s + j : s + j - NST;
								issue(sj, nss - T + j, Y);
								done(&bar_empty[sj]);
							}
							s += T;
							if (s >= NST) { s -= NST; ph ^= 1; }
						}
						done(&bar_yfull[nch & 1]);
						nch++;
				}
				return true;
			};
			for (int slot = 0, ok = 1; ok; ) {
				if (!wwait(&bar_ifull[slot], iph, 6))
					break;
				const int t = uni(*(volatile int *)&s_item[slot]);
				if (lane == 0)
					mbar_arrive(smem_u32(&bar_iempty[slot]));
				__syncwarp();
				if (++slot == 2) { slot = 0; iph ^= 1; }
				if (t < 0)
					break;
				const emu_item it = items[t];
				const int n = uni(it.pr) >> 8, c0 = uni(it.cfirst), cn = uni(it.ccount);
				const uint32_t sa = rowmajor ? 16 : 2 * uni(tile_rows((it.pr >> 1) & 1 ?
				    cbs[members[it.mfirst].cblock].m : cbs[members[it.mfirst].cblock].n,
				    it.m0));
				auto run = [&](auto cls) { return item(cls, n, sa, c0, cn); };
				if (PAIR || rowmajor)
					ok = run(std::integral_constant<int, 4>{});
				else if constexpr (PAIR)
					;
				else if constexpr (KEEP == 2)
					ok = run(std::integral_constant<int, 3>{});
				else if (n <= 80)
					ok = run(std::integral_constant<int, 0>{});
				else if (n <= 96)
					ok = run(std::integral_constant<int, 1>{});
				else
					ok = run(std::integral_constant<int, 2>{});
			}
			/* every MMA issued by this CTA has completed once bar_fin
			 * fires; TMEM is released only after that */
			done(&bar_fin);
			uint64_t t0 = gtimer();
			while (lane == 0 && !(PAIR ? mbar_try_cl(smem_u32(&bar_fin), 0) :
			    mbar_try(smem_u32(&bar_fin), 0)) && gtimer() - t0 < WAIT_NS)
				;
		}
	} else {
		/* ------------- drain + epilogue (warps 2 .. DW+1) -------------
		 * warp w reads TMEM lanes 32 * (w % 4) .. +31 (the tcgen05.ld
		 * lane-quadrant rule) and owns NC of the 128 columns */
		constexpr int NC = 128 / (DW / 4);
		constexpr int NSEG = NC / 16;
		const int quad = warp & 3, half = (warp - 2) >> 2;
		const uint32_t trow = tmem + ((uint32_t)(quad * 32) << 16);
		uint32_t nch = 0;
		bool ok = true;
		uint32_t iph = 0;
		/* one lane waits, the warp follows its verdict, so the
		 * .sync.aligned TMEM loads stay convergent */
		auto wait_warp = [&](uint64_t *bar, uint32_t par, int code) -> bool {
			int w = 1;
			if (lane == 0)
				w = wait(smem_u32(bar), par, code);
			w = __shfl_sync(0xffffffffu, w, 0);
			tc_fence_after();
			return w != 0;
		};
		/* this warp has read a set: the MMA warp may overwrite it */
		auto release = [&](uint64_t *bar) {
			tc_fence_before();
			__syncwarp();
			if (lane == 0)
				arrive0(bar);
		};
		for (int slot = 0; ok; ) {
			int t = -1;
			if (lane == 0) {
				if (wait(smem_u32(&bar_ifull[slot]), iph, 7)) {
					t = s_item[slot];
					arrive0(&bar_iempty[slot]);
				} else
					t = -2;
			}
			t = __shfl_sync(0xffffffffu, t, 0);
			if (++slot == 2) { slot = 0; iph ^= 1; }
			if (t < 0)
				break;
			const emu_item it = items[t];
			const int pass = it.pr & 1, swp = (it.pr >> 1) & 1, rows = it.pr >> 8;
			const int mstk = (it.pr >> 2) & 1;
			/* this warp's columns: 32, or 16 where the tile has at most
			 * 64, so that every column group has work */
			const int cw = rows <= 64 && NC == 32 ? 16 : NC;
			const int col0 = half * cw;
			const int nacc3 = KEEP == 2 || PAIR || rowmajor ? 1 : rows <= 80 ? 3 : rows <= 96 ? 2 : 1;
			/* its columns fall into segments of 16, each inside one
			 * member's output block (N-stacked members hold
			 * multiples of 16 columns; M-stacked ones multiples of 32
			 * lanes, so one member holds all of this warp's lanes): per
			 * segment the output block, its member, its F and the
			 * N-side row of the segment's first column; and the M-side
			 * row of this warp's first lane */
			int scb[NSEG], sF[NSEG], sq0[NSEG], mrow0;
			uint32_t smj = 0;            /* (per segment: its factor's place) */
			if (mstk) {
				const int row0 = quad * 32;
				int j = 0;
				for (int jj = 1; jj < it.mcount; jj++)
					j += row0 >= members[it.mfirst + jj].off;
				const emu_member mb = members[it.mfirst + j];
#pragma unroll
				for (int g = 0; g < NSEG; g++) {
					scb[g] = mb.cblock;
					smj |= (uint32_t)(16 + 2 * j) << (8 * g);
					sF[g] = cbF[mb.cblock];
					sq0[g] = it.m0 + col0 + g * 16;
				}
				mrow0 = mb.n0 + row0 - mb.off;
			} else {
#pragma unroll
				for (int g = 0; g < NSEG; g++) {
					const int col = col0 + g * 16;
					int j = 0;
					for (int jj = 1; jj < it.mcount; jj++)
						j += col >= members[it.mfirst + jj].off;
					const emu_member mb = members[it.mfirst + j];
					scb[g] = mb.cblock;
					smj |= (uint32_t)(16 + 2 * j) << (8 * g);
					sF[g] = cbF[mb.cblock];
					sq0[g] = mb.n0 + col - mb.off;
				}
				mrow0 = it.m0 + (int)rank * EMU_TM + quad * 32;
			}
			uint64_t V[NC];                  /* two's complement */
#pragma unroll
			for (int c = 0; c < NC; c++)
				V[c] = 0;
			/* columns per TMEM load and wait (8 took 3 % off the FP64
			 * drains, 4 is 1 % faster in FP32) */
			constexpr int W = LOW ? 8 : 4;
			/* set X.  FP64: the low band, L in units of 2^-16 (|L| <
			 * 2^19: 15 products of 256 times 2^14 at 2^-24, with the pair
			 * factor's 2), to units of 2^(-16-F): V += 2^12 h + l, h =
			 * rint(2^(F-12) L), l = rint(2^F L - 2^12 h).  FP32: group 2,
			 * an integer */
			auto drain_x = [&](uint32_t at, const float *s0) {
#pragma unroll
				for (int b = 0; b < NC; b += W) {
					if (b >= cw || col0 + b >= rows)
						break;	/* warp-uniform: columns past the tile */
					const int g = b / 16;
					float ax[W];
					tmem_ld(trow + at + col0 + b, ax);
					if (LOW && nacc3 > 1) {
						/* groups 4 (and 5) have their own accumulators,
						 * in the same units */
						float a4[W], a5[W] = {};
						tmem_ld(trow + at + rows + col0 + b, a4);
						if (nacc3 > 2)
							tmem_ld(trow + at + 2 * rows + col0 + b, a5);
						tmem_wait_ld();
#pragma unroll
						for (int c = 0; c < W; c++)
							ax[c] += a4[c] + a5[c];
					} else
						tmem_wait_ld();
#pragma unroll
					for (int c = 0; c < W; c++) {
						const float sx = s0[g] * (LOW ?
						    __int_as_float((127 + 4 + sF[g]) << 23) : 65536.0f);
						if (LOW) {
							const float t = fmaf(ax[c], sx, MAGICF);
							const float r = fmaf(ax[c], sx, MAGICF - t);
							const float l = fmaf(r, 4096.0f, MAGICF);
							V[b + c] += ((uint64_t)__float_as_uint(t) << 12) +
							    __float_as_uint(l);
						} else
							V[b + c] += (long long)__float2int_rn(ax[c] * sx);
					}
				}
			};
			/* set Y: D0 2^16 + D1 2^8 (+ D2), the exact groups, read as
			 * D0, D1 2^-8, D2 2^-16.  With h = rint(D1 2^-8), the sum is
			 * 2^16 (D0 + h) + e, e = 2^8 (D1 - 2^8 h) + D2: both fit 24
			 * bits (|D0| <= 2^22, |h| <= 2^15, |D2| < 3 * 2^22, each
			 * twice that with the pair factor's 2, then even), so two
			 * conversions serve three groups, one serves two in FP32 */
			auto drain_y = [&](const float *s0) {
#pragma unroll
				for (int b = 0; b < NC; b += W) {
					if (b >= cw || col0 + b >= rows)
						break;
					const int g = b / 16, F = sF[g];
					float a0[W], a1[W], a2[W];
					tmem_ld(trow + col0 + b, a0);
					tmem_ld(trow + rows + col0 + b, a1);
					if (LOW)
						tmem_ld(trow + 2 * rows + col0 + b, a2);
					tmem_wait_ld();
#pragma unroll
					for (int c = 0; c < W; c++) {
						const float h = fmaf(a1[c], s0[g], MAGICF) - MAGICF;
						const float r = fmaf(a1[c], s0[g], -h);
						const int d = __float2int_rn(fmaf(a0[c], s0[g], h));
						if (LOW) {
							const int e = __float2int_rn(fmaf(a2[c], s0[g], r) * 65536.0f);
							/* d 2^(16+F) + e 2^F, 1 <= F <= 15 */
							const uint64_t dv = ((uint64_t)(uint32_t)(d >> (16 - F)) << 32) |
							    ((uint32_t)d << (16 + F));
							const uint64_t ev = ((uint64_t)(uint32_t)(e >> (32 - F)) << 32) |
							    ((uint32_t)e << F);
							V[b + c] += dv + ev;
						} else {
							const float l = fmaf(r, 65536.0f, MAGICF);
							const uint64_t dv = ((uint64_t)(uint32_t)(d >> 16) << 32) |
							    ((uint32_t)d << 16);
							V[b + c] += dv + __float_as_uint(l);
						}
					}
				}
			};
			/* values rounded by the magic number (FP64: in X, FP32: in Y) */
			int nround = 0;
			for (bool more = true; more; nch++) {
				const int z = nch & 1;
				if (!(ok = wwait(&bar_info[z], (nch >> 1) & 1, 11)))
					break;
				const int head = *(volatile int *)&s_head[z], fl = head >> 8;
				more = !(fl & ITEM_LAST);
				nround += LOW || (fl & RUN_LAST);
				/* each segment's factor, sign * 2^shift (shift 0 or 1,
				 * checked by the planner), rides on the exact fp32 -> int
				 * scales */
				float s0[NSEG];
#pragma unroll
				for (int g = 0; g < NSEG; g++) {
					const uint32_t q = (uint32_t)head >> (smj >> (8 * g) & 0xff);
					s0[g] = __uint_as_float((q & 1) << 31 | (127 + (q >> 1 & 1)) << 23);
				}
				if (XDB) {
					/* Y first: X's copy is not needed for a chunk yet */
					if (!(ok = wait_warp(&bar_yfull[z], (nch >> 1) & 1, 9)))
						break;
					if (fl & RUN_LAST) {
						drain_y(s0);
						release(&bar_yempty);
					}
					drain_x(XCOL + z * 128, s0);
					release(&bar_xempty[z]);
				} else {
					/* X first, then it is free for the next chunk's head;
					 * Y once its last products have landed */
					if (!(ok = wait_warp(&bar_xfull, nch & 1, 4)))
						break;
					drain_x((LOW ? 3 : 2) * rows, s0);
					release(&bar_xempty[0]);
					if (!(ok = wait_warp(&bar_yfull[z], (nch >> 1) & 1, 9)))
						break;
					if (LOW || (fl & RUN_LAST)) {
						drain_y(s0);
						release(&bar_yempty);
					}
				}
			}
			/* the magic numbers' bits out of the sums (modulo 2^64) */
#pragma unroll
			for (int c = 0; c < NC; c++)
				V[c] -= (uint64_t)nround * (LOW ?
				    ((uint64_t)MAGIC << 12) + MAGIC : (uint64_t)MAGIC);
			if (__any_sync(0xffffffffu, !ok || s_err))
				break;
			if (it.parts > 1) {
				unsigned long long *sum = reinterpret_cast<unsigned long long *>(slots +
				    it.slot * SLOT_BYTES) + (size_t)(warp - 2) * NC * 32 + lane;
				int *count = reinterpret_cast<int *>(slots + it.slot * SLOT_BYTES +
				    SLOT_SUMS * 8) + warp - 2;
#pragma unroll
				for (int c = 0; c < NC; c++)
					if (c < cw)
						atomicAdd(sum + c * 32, (unsigned long long)V[c]);
				__threadfence();
				__syncwarp();
				int before = 0;
				if (lane == 0)
					before = atomicAdd(count, 1);
				before = __shfl_sync(0xffffffffu, before, 0);
				if (before != it.parts - 1)
					continue;
				__threadfence();
#pragma unroll
				for (int c = 0; c < NC; c++)
					if (c < cw)
						V[c] = __ldcg(sum + c * 32);
			}
			/* epilogue (overlaps the next item's first chunk of MMAs):
			 * this thread's TMEM lane is one M-side row; its columns are
			 * N-side rows of the segments' output blocks.  Without swap
			 * the M side is b's free index (j), with swap a's (i). */
			const int ms = mrow0 + lane;
			const bool bz = beta == 0.0;
			const int cm = cplx ? 2 : 1;
			/* alpha a normal power of two folds into the exponent and
			 * sign; any other alpha costs one multiply */
			const long long ab = __double_as_longlong(alpha);
			const int aex = (int)((ab >> 52) & 0x7ff);
			const bool apow2 = (ab & 0xFFFFFFFFFFFFFll) == 0 && aex > 0 && aex < 0x7ff;
			const int esa = apow2 ? aex - 1023 : 0;
			const unsigned long long asx = apow2 ?
			    (unsigned long long)ab & (1ull << 63) : 0ull;
			/* a segment's 16 columns: their exponents and offsets are
			 * loaded once, a column per lane, and C's old values eight at a
			 * time, before any is stored: one by one, each waits for the
			 * last one's store and for memory (complex128 ring term, 21 x
			 * 75: 90600 cycles a CTA, now 62200 of 550000) */
#pragma unroll
			for (int g = 0; g < NSEG; g++) {
				if (g * 16 >= cw)
					break;
				const xmgd_cblock_t cb = cbs[scb[g]];
				const int flim = swp ? cb.m : cb.n, vlim = swp ? cb.n : cb.m;
				const int nq = min(min(vlim - sq0[g], rows - col0 - g * 16), 16);
				TOUT *Cp = reinterpret_cast<TOUT *>(cb.c_ptr) + pass;
				int ve = 0, vo = 0, fo = 0, fe = 0;
				if ((lane & 15) < nq) {
					const int q = sq0[g] + (lane & 15);
					ve = (swp ? EB + cb.eB : EA + cb.eA)[q];
					vo = tabs[(swp ? cb.ccol : cb.crow) + q];
				}
				const bool live = ms < flim;
				if (live) {
					fo = tabs[(swp ? cb.crow : cb.ccol) + ms];
					fe = (swp ? EA + cb.eA : EB + cb.eB)[ms];
				}
				const int e0 = fe - expoff2 - 16 - sF[g];
#pragma unroll
				for (int c0 = 0; c0 < 16; c0 += 8) {
					TOUT old[8];
					if (!bz) {
#pragma unroll
						for (int c = 0; c < 8; c++) {
							const int o = __shfl_sync(0xffffffffu, vo, c0 + c) + fo;
							old[c] = live && c0 + c < nq ? Cp[(size_t)cm * o] : TOUT(0);
						}
					}
#pragma unroll
					for (int c = 0; c < 8; c++) {
						const int e = __shfl_sync(0xffffffffu, ve, c0 + c) + e0;
						const int o = __shfl_sync(0xffffffffu, vo, c0 + c) + fo;
						if (live && c0 + c < nq) {
							const long long x = (long long)V[g * 16 + c0 + c];
							TOUT *cp = Cp + (size_t)cm * o;
							double v = pack_f64(x, e + esa, asx);
							if (!apow2)
								v *= alpha;
							*cp = bz ? (TOUT)v : (TOUT)fma(beta, (double)old[c], v);
						}
					}
				}
			}
		}
	}
	/* the forwarder role runs on lane 0 alone, waits may leave lanes apart: the
	 * warps reconverge first, because an aligned barrier counts a whole
	 * warp as arrived when any of its lanes arrives, and TMEM must stay
	 * allocated until the MMA lane has seen its last commit land */
	__syncwarp();
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	if (warp == 1) {
		if constexpr (PAIR)
			asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;"
			    :: "r"(tmem));
		else
			asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;"
			    :: "r"(tmem));
	}
	/* neither CTA of a pair leaves while the other may still arrive on
	 * its barriers */
	if constexpr (PAIR)
		cluster_sync();
}

/* ------------------------------------------------------------------ */
/* host side: a reusable plan with an online tile-orientation autotuner  */

/*
 * Work-list policies.  The M side of a tile is always 128 rows (TMEM
 * lanes); the N side is the live rows rounded up to 16, so which operand
 * lies on the N side sets the padded work, and the order of the items
 * sets which tiles run together (L2 reuse: output blocks with the same
 * M-side free block read the same M-side operand rows).  Three policies,
 * each a complete work list:
 *   0  per block the orientation with less padded MMA work; blocks by
 *      decreasing cost, each block's tiles together;
 *   1  the same orientation; blocks grouped by their M-side free block and
 *      the group run M tile by M tile across its blocks;
 *   2  grouped as 1, orientation by max(N / 2, 32 + N / 4) per tile, which
 *      prefers wide tiles (an MMA's cost does not fall below 28 cycles).
 * (and 6, the stacked form below).  The first runs of a plan replay each
 * distinct policy within a quarter of the modelled best once, in the model's
 * order (list_cycles), timed with events, then keep the fastest; the choice
 * is remembered per block-size histogram so later plans of the same shape
 * start tuned.
 */
enum { EMU_NPOLICY = 3 };

/* policy 6: policy 2's orientation and order, with the N-side tails of the
 * output blocks that share an M side (the same M-side view and K for every
 * pair index) stacked into common 128-column tiles: the MMAs of a K step
 * get wider, the shared-memory operand reads per flop fewer */
enum { EMU_POL_MERGED = 2 * EMU_NPOLICY };

static bool
pair_policy(int pol)
{
	return pol >= EMU_NPOLICY && pol < 2 * EMU_NPOLICY;
}

/* The operands' layout a policy's kernel form takes (emu_split_kernel):
 * row-major where a tile stacks members, and for pairs; slice-major where
 * every tile is one block's. */
static bool
row_major(int pol)
{
	return pair_policy(pol) || pol == EMU_POL_MERGED;
}

/* CTA pairs (256-row M tiles, cta_group::2): policies 3..5 repeat 0..2 in
 * that form; offered to the tuner when XMG_CTA_PAIR=1 */
static bool
pairs_enabled()
{
	const char *e = getenv("XMG_CTA_PAIR");
	return e && strcmp(e, "1") == 0;
}

static double
tile_cost(int mside, int nside, int policy, int mrows)
{
	double c = 0;
	const int mt = (mside + mrows - 1) / mrows;
	for (int n0 = 0; n0 < nside; n0 += EMU_TM) {
		const int w = std::min(EMU_TM, (nside - n0 + 15) / 16 * 16);
		c += policy == 2 ? std::max(w / 2.0, 32.0 + w / 4.0) : (double)w;
	}
	return c * mt;
}

static uint64_t
mix64(uint64_t h)
{
	h ^= h >> 33; h *= 0xff51afd7ed558ccdULL;
	h ^= h >> 33; h *= 0xc4ceb93fe53e6ccdULL;
	return h ^ (h >> 33);
}

struct tune_entry {
	uint64_t sig;
	int policy;
};
static std::vector<tune_entry> g_tuned;

struct emu_cand {
	int policy;
	uint64_t d_items, d_members;
	int nitems, grid, nslots;
	float ms;
};

struct emu_plan {
	int dtype, cplx;
	double alpha, beta;
	std::vector<xmgd_view_t> VA, VB;     /* slices: offsets in the workspace */
	std::vector<char> useA, useB;
	uint64_t d_va = 0, d_vb = 0, d_meta[2][2] = {{0, 0}, {0, 0}};
	int64_t nctas[2][2] = {{0, 0}, {0, 0}};
	int kr[2] = {256, 256};              /* exponent pass: K per CTA */
	uint64_t d_E = 0, d_F = 0, d_chunks = 0;
	uint64_t dbuf = 0;                   /* the allocation of all of these */
	std::vector<xmgd_view_t> vstage;     /* bound views on their way up */
	int64_t nE = 0;
	int32_t nexp_a = 0;
	size_t slice_bytes = 0, slot_bytes = 0;  /* slots follow the slices */
	uint64_t ws = 0;                     /* workspace the views point into */
	const xmgd_cblock_t *d_cbs;
	const xmgd_pair_t *d_prs;
	const int32_t *d_tabs;
	std::vector<emu_cand> cand;
	int cur = 0, tuned = 0;
	int hmax = 4;                        /* head/tail steps (<= stages) */
	int a_mode = 0;                      /* shared a side (xmgd_contract_t) */
	uint64_t a_slices = 0, a_E = 0, a_flag = 0;
	int kchunk = EMU_CHUNK;              /* FP64: K steps per chunk */
	uint64_t sig = 0;
	int *h_flags = nullptr;              /* pinned: Inf/NaN, timeout */
	int (*split)(emu_plan *) = nullptr;
	int (*gemm)(emu_plan *) = nullptr;
};

/* the exponent pass, or the unfold + split, of one side on a stream */
template <typename TIN>
static int
launch_side(emu_plan *e, int side, int kind, int32_t *E, int *flags, cudaStream_t st)
{
	const xmgd_view_t *dv = (const xmgd_view_t *)(side ? e->d_vb : e->d_va);
	const int nv = (int)(side ? e->VB.size() : e->VA.size());
	const view_meta *m = (const view_meta *)e->d_meta[side][kind];
	const unsigned n = (unsigned)e->nctas[side][kind];

	if (n == 0)
		return XMG_OK;
	if (kind == 0)
		emu_exp_kernel<TIN><<<n, 256, 0, st>>>(dv, m, nv, e->kr[side], e->d_tabs, E,
		    flags);
	else
		emu_split_kernel<TIN><<<n, 256, 0, st>>>(dv, m, nv, e->d_tabs, E,
		    row_major(e->cand[e->cur].policy));
	g_launches++;
	XMG_CK(cudaGetLastError());
	return XMG_OK;
}

/* the slots' place in the workspace */
static size_t
slot_offset(const emu_plan *e)
{
	return (e->slice_bytes + 255) & ~(size_t)255;
}

/* exponent tables, then unfold + split of every used view of both sides.
 * The two sides are independent chains of two kernels: a's runs on a second
 * stream beside b's (two branches of the captured graph), since on small
 * operands each kernel is shorter than the time its launch takes to fill
 * and drain the chip.  A shared a side (streamed batches) keeps one chain:
 * its flag is copied between the kernels. */
template <typename TIN>
static int
launch_split(emu_plan *e)
{
	int32_t *EA = (int32_t *)e->d_E, *EB = EA + e->nexp_a;
	int *flags = (int *)(EA + e->nE);
	int st;

	XMG_CK(cudaMemsetAsync((void *)e->d_E, 0, (e->nE + 64) * sizeof(int32_t),
	    stream()));
	if (e->cand[e->cur].nslots)
		XMG_CK(cudaMemsetAsync((void *)(e->ws + slot_offset(e)), 0,
		    e->cand[e->cur].nslots * SLOT_BYTES, stream()));
	if (!e->a_mode) {
		cudaStream_t aux;
		if ((st = fork_aux(&aux)))
			return st;
		if ((st = launch_side<TIN>(e, 0, 0, EA, flags, aux)) ||
		    (st = launch_side<TIN>(e, 0, 1, EA, flags, aux)) ||
		    (st = launch_side<TIN>(e, 1, 0, EB, flags, stream())) ||
		    (st = launch_side<TIN>(e, 1, 1, EB, flags, stream()))) {
			/* what the second stream got is waited for on the engine's */
			join_aux();
			return st;
		}
		return join_aux();
	}
	/* a shared a side: the preparing plan fills the shared exponent table
	 * and flag; every plan, the preparing one and the ones that use it,
	 * takes the flag's Inf/NaN bit into its own */
	EA = (int32_t *)e->a_E;
	int *aflags = (int *)e->a_flag;
	if (e->a_mode == 1) {
		XMG_CK(cudaMemsetAsync(EA, 0, e->nexp_a * sizeof(int32_t), stream()));
		XMG_CK(cudaMemsetAsync(aflags, 0, sizeof(int), stream()));
		if ((st = launch_side<TIN>(e, 0, 0, EA, aflags, stream())))
			return st;
	}
	XMG_CK(cudaMemcpyAsync(flags, aflags, sizeof(int), cudaMemcpyDeviceToDevice,
	    stream()));
	if ((st = launch_side<TIN>(e, 1, 0, EB, flags, stream())) ||
	    (e->a_mode == 1 && (st = launch_side<TIN>(e, 0, 1, EA, aflags, stream()))))
		return st;
	return launch_side<TIN>(e, 1, 1, EB, flags, stream());
}

/* the persistent grouped GEMM of the current candidate, then the flags */
template <typename TIN, typename TOUT>
static int
launch_gemm(emu_plan *e)
{
	constexpr int S = fin<TIN>::S, KEEP = fin<TIN>::KEEP;
	constexpr bool LOW = KEEP > 2;
	const emu_cand &c = e->cand[e->cur];
	int32_t *EA = (int32_t *)e->d_E, *EB = EA + e->nexp_a;
	int *flags = (int *)(EA + e->nE);
	if (e->a_mode)
		EA = (int32_t *)e->a_E;	/* the shared a side's table */

	unsigned char *slots = (unsigned char *)(e->ws + slot_offset(e));

	if (pair_policy(c.policy)) {
		/* clusters of two CTAs */
		cudaLaunchConfig_t cfg = {};
		cudaLaunchAttribute at[1];
		at[0].id = cudaLaunchAttributeClusterDimension;
		at[0].val.clusterDim.x = 2;
		at[0].val.clusterDim.y = 1;
		at[0].val.clusterDim.z = 1;
		cfg.gridDim = dim3((unsigned)c.grid);
		cfg.blockDim = dim3(64 + 32 * EMU_DW);
		cfg.dynamicSmemBytes = stage_cfg<S>::SMEM;
		cfg.stream = stream();
		cfg.attrs = at;
		cfg.numAttrs = 1;
		XMG_CK(cudaLaunchKernelEx(&cfg, emu_gemm_kernel<S, KEEP, LOW, TOUT, EMU_DW, true>,
		    (const emu_item *)c.d_items, c.nitems, (const emu_member *)c.d_members,
		    e->d_cbs, e->d_prs,
		    (const xmgd_view_t *)e->d_va, (const xmgd_view_t *)e->d_vb, e->d_tabs,
		    (const int32_t *)EA, (const int32_t *)EB, (const int32_t *)e->d_F,
		    (const emu_chunk *)e->d_chunks, e->alpha, e->beta, 2 * fin<TIN>::EXPOFF,
		    e->cplx, e->hmax,
		    (int)row_major(c.policy), slots, flags));
	} else {
		emu_gemm_kernel<S, KEEP, LOW, TOUT, EMU_DW, false><<<(unsigned)c.grid,
		    64 + 32 * EMU_DW, stage_cfg<S>::SMEM, stream()>>>(
		    (const emu_item *)c.d_items, c.nitems, (const emu_member *)c.d_members,
		    e->d_cbs, e->d_prs,
		    (const xmgd_view_t *)e->d_va, (const xmgd_view_t *)e->d_vb, e->d_tabs,
		    EA, EB, (const int32_t *)e->d_F, (const emu_chunk *)e->d_chunks, e->alpha,
		    e->beta, 2 * fin<TIN>::EXPOFF, e->cplx, e->hmax,
		    (int)row_major(c.policy), slots, flags);
	}
	g_launches++;
	XMG_CK(cudaGetLastError());
	XMG_CK(cudaMemcpyAsync(e->h_flags, flags, 2 * sizeof(int),
	    cudaMemcpyDeviceToHost, stream()));
	return XMG_OK;
}

template <typename TIN, typename TOUT>
static int
set_attrs()
{
	constexpr int S = fin<TIN>::S, KEEP = fin<TIN>::KEEP;
	static bool done = false;
	if (!done) {
		XMG_CK(cudaFuncSetAttribute(emu_gemm_kernel<S, KEEP, (KEEP > 2), TOUT, EMU_DW, false>,
		    cudaFuncAttributeMaxDynamicSharedMemorySize, stage_cfg<S>::SMEM));
		XMG_CK(cudaFuncSetAttribute(emu_gemm_kernel<S, KEEP, (KEEP > 2), TOUT, EMU_DW, true>,
		    cudaFuncAttributeMaxDynamicSharedMemorySize, stage_cfg<S>::SMEM));
		done = true;
	}
	return XMG_OK;
}

void
emu_free(emu_plan *e)
{
	if (!e)
		return;
	if (e->dbuf)
		xmgd_free(e->dbuf);
	flag_pair_release(e->h_flags);
	delete e;
}

/* work list of one policy (see above) */
static void
make_items(const xmgd_contract_t *p, const std::vector<int> &cblocks, int cplx,
    int policy, std::vector<emu_item> &items, std::vector<emu_member> &members)
{
	struct blk {
		int ci, swp, mlen, nlen;
		double cost;
		uint64_t key;
	};
	const bool merged = policy == EMU_POL_MERGED;
	const int base = merged ? 2 : policy % EMU_NPOLICY;
	const int mstep = pair_policy(policy) ? 2 * EMU_TM : EMU_TM;
	const int pol = base == 2 ? 2 : 0;
	std::vector<blk> bl;
	for (int ci : cblocks) {
		const xmgd_cblock_t &cb = p->cblocks[ci];
		double k = 0;
		for (int q = 0; q < cb.npairs; q++)
			k += p->pairs[cb.first_pair + q].k;
		blk b;
		b.ci = ci;
		b.swp = tile_cost(cb.m, cb.n, pol, mstep) < tile_cost(cb.n, cb.m, pol, mstep);
		b.mlen = b.swp ? cb.m : cb.n;
		b.nlen = b.swp ? cb.n : cb.m;
		b.cost = k * cb.m * (double)cb.n;
		/* the M-side free block (its exponent-table slot names it) */
		b.key = ((uint64_t)b.swp << 40) | (uint32_t)(b.swp ? cb.eA : cb.eB);
		bl.push_back(b);
	}
	/* one item per member list (every complex pass); N-stacked: m0 is the
	 * M tile and the members' rows add up to N; M-stacked: m0 is the N tile
	 * and ncols its live rows */
	auto push = [&](int m0, int swp, const std::vector<emu_member> &mem,
	    int mstk = 0, int ncols = 0) {
		int tot = 0;
		for (const emu_member &x : mem)
			tot += x.rows;
		if (mstk)
			tot = ncols;
		for (int ps = 0; ps < (cplx ? 2 : 1); ps++) {
			items.push_back(emu_item{m0, (int)members.size(), (int)mem.size(),
			    ps | (swp ? 2 : 0) | (mstk ? 4 : 0) | (tot << 8)});
			members.insert(members.end(), mem.begin(), mem.end());
		}
	};
	auto emit = [&](const blk &b, int m0) {
		for (int n0 = 0; n0 < b.nlen; n0 += EMU_TM) {
			const int rows = std::min(EMU_TM, (b.nlen - n0 + 15) / 16 * 16);
			push(m0, b.swp, {emu_member{b.ci, n0, rows, 0}});
		}
	};
	items.clear();
	members.clear();
	std::stable_sort(bl.begin(), bl.end(),
	    [](const blk &x, const blk &y) { return x.cost > y.cost; });
	if (base == 0) {
		for (const blk &b : bl)
			for (int m0 = 0; m0 < b.mlen; m0 += mstep)
				emit(b, m0);
		return;
	}
	/* grouped: blocks reading the same M-side rows together, M tile by
	 * M tile, groups by decreasing cost; merged: a group holds only
	 * blocks whose pair lists have the same M-side view and K at every
	 * index, so their tiles can share the M-side stages */
	std::vector<std::vector<int64_t>> gkey;
	std::vector<std::vector<int>> groups;
	std::vector<double> gcost;
	std::vector<int64_t> k;
	for (int i = 0; i < (int)bl.size(); i++) {
		k.assign(1, (int64_t)bl[i].key);
		if (merged) {
			const xmgd_cblock_t &cb = p->cblocks[bl[i].ci];
			k.push_back(bl[i].mlen);
			for (int q = 0; q < cb.npairs; q++) {
				const xmgd_pair_t &pr = p->pairs[cb.first_pair + q];
				k.push_back(((int64_t)(bl[i].swp ? pr.aview : pr.bview) << 32) | pr.k);
			}
		}
		size_t g = 0;
		while (g < groups.size() && gkey[g] != k)
			g++;
		if (g == groups.size()) {
			gkey.push_back(k);
			groups.push_back({});
			gcost.push_back(0);
		}
		groups[g].push_back(i);
		gcost[g] += bl[i].cost;
	}
	std::vector<int> go(groups.size());
	for (size_t g = 0; g < go.size(); g++)
		go[g] = (int)g;
	std::stable_sort(go.begin(), go.end(),
	    [&](int x, int y) { return gcost[x] > gcost[y]; });
	/* merged: partial M tiles wait for the M-stacking pass below */
	struct tail { int i, m0, n0, ncols; };
	std::vector<tail> tails;
	for (int g : go) {
		int mmax = 0;
		for (int i : groups[g])
			mmax = std::max(mmax, bl[i].mlen);
		for (int m0 = 0; m0 < mmax; m0 += mstep) {
			if (!merged) {
				for (int i : groups[g])
					if (m0 < bl[i].mlen)
						emit(bl[i], m0);
				continue;
			}
			if (mmax - m0 < EMU_TM) {
				for (int i : groups[g])
					for (int n0 = 0; n0 < bl[i].nlen; n0 += EMU_TM)
						tails.push_back(tail{i, m0, n0, std::min(EMU_TM,
						    (bl[i].nlen - n0 + 15) / 16 * 16)});
				continue;
			}
			/* full 128-row N tiles alone; the partial ones packed
			 * first-fit decreasing into tiles of <= 128 rows and
			 * <= EMU_MAXMEM members */
			std::vector<emu_member> part;
			for (int i : groups[g]) {
				const blk &b = bl[i];
				for (int n0 = 0; n0 < b.nlen; n0 += EMU_TM) {
					const int rows = std::min(EMU_TM, (b.nlen - n0 + 15) / 16 * 16);
					if (rows == EMU_TM)
						push(m0, b.swp, {emu_member{b.ci, n0, rows, 0}});
					else
						part.push_back(emu_member{b.ci, n0, rows, 0});
				}
			}
			std::stable_sort(part.begin(), part.end(),
			    [](const emu_member &x, const emu_member &y) { return x.rows > y.rows; });
			std::vector<std::vector<emu_member>> bins;
			std::vector<int> fill;
			for (const emu_member &x : part) {
				size_t b = 0;
				while (b < bins.size() && (fill[b] + x.rows > EMU_TM ||
				    (int)bins[b].size() == EMU_MAXMEM))
					b++;
				if (b == bins.size()) {
					bins.push_back({});
					fill.push_back(0);
				}
				emu_member y = x;
				y.off = fill[b];
				bins[b].push_back(y);
				fill[b] += x.rows;
			}
			for (const auto &mem : bins)
				push(m0, bl[groups[g][0]].swp, mem);
		}
	}
	if (!merged)
		return;
	/* M-stacking: the partial M tiles of blocks that share the N side (the
	 * same N-side view and K at every pair index, the same N tile) fill
	 * common 128-lane tiles, 32 lanes at a time; a tile left alone runs
	 * as an ordinary item */
	std::vector<std::vector<int64_t>> tkey;
	std::vector<std::vector<int>> tgrp;
	for (int x = 0; x < (int)tails.size(); x++) {
		const blk &b = bl[tails[x].i];
		const xmgd_cblock_t &cb = p->cblocks[b.ci];
		k.assign({(int64_t)b.swp, tails[x].n0, tails[x].ncols, b.nlen});
		for (int q = 0; q < cb.npairs; q++) {
			const xmgd_pair_t &pr = p->pairs[cb.first_pair + q];
			k.push_back(((int64_t)(b.swp ? pr.bview : pr.aview) << 32) | pr.k);
		}
		size_t g = 0;
		while (g < tkey.size() && tkey[g] != k)
			g++;
		if (g == tkey.size()) {
			tkey.push_back(k);
			tgrp.push_back({});
		}
		tgrp[g].push_back(x);
	}
	for (const std::vector<int> &tg : tgrp) {
		std::vector<emu_member> part;
		for (int x : tg) {
			const tail &tl = tails[x];
			const blk &b = bl[tl.i];
			part.push_back(emu_member{b.ci, tl.m0, (b.mlen - tl.m0 + 31) / 32 * 32, 0});
		}
		std::stable_sort(part.begin(), part.end(),
		    [](const emu_member &x, const emu_member &y) { return x.rows > y.rows; });
		std::vector<std::vector<emu_member>> bins;
		std::vector<int> fill;
		for (const emu_member &x : part) {
			size_t b = 0;
			while (b < bins.size() && (fill[b] + x.rows > EMU_TM ||
			    (int)bins[b].size() == EMU_MAXMEM))
				b++;
			if (b == bins.size()) {
				bins.push_back({});
				fill.push_back(0);
			}
			emu_member y = x;
			y.off = fill[b];
			bins[b].push_back(y);
			fill[b] += x.rows;
		}
		const tail &t0 = tails[tg[0]];
		const int swp = bl[t0.i].swp;
		for (const auto &mem : bins) {
			if (mem.size() == 1)
				push(mem[0].n0, swp, {emu_member{mem[0].cblock, t0.n0, t0.ncols, 0}});
			else
				push(t0.n0, swp, mem, 1, t0.ncols);
		}
	}
}

/*
 * The chunks of every item of a list (see emu_chunk): one list per set of
 * members and pass, shared by the items with the same ones (the index spans
 * the candidates of a plan).
 */
struct chunk_index {
	std::vector<int> one;                      /* [2 * block + pass], or -1 */
	std::map<std::vector<int>, int> stacked;   /* pass, blocks */
	std::vector<std::pair<int, int>> size;     /* chunks, steps of the list that
	                                            * starts there */
};

static void
chunk_lists(const xmgd_contract_t *p, int cplx, int kchunk, std::vector<emu_item> &items,
    const std::vector<emu_member> &members, chunk_index &seen, std::vector<emu_chunk> &out)
{
	const bool dbl = p->dtype >= 2;
	const int KS = dbl ? stage_cfg<fin<double>::S>::KSTEPS : stage_cfg<fin<float>::S>::KSTEPS;
	std::vector<int> key;

	seen.one.resize(2 * (size_t)p->ncblocks, -1);
	for (emu_item &it : items) {
		const int pass = it.pr & 1, nmem = it.mcount, signs = 0x55 >> (8 - 2 * nmem);
		key.assign(1, pass);
		for (int j = 0; j < nmem; j++)
			key.push_back(members[it.mfirst + j].cblock);
		int &slot = nmem == 1 ? seen.one[2 * (size_t)key[1] + pass] :
		    seen.stacked.insert(std::make_pair(key, -1)).first->second;
		it.p0 = it.k0 = it.slot = it.steps = 0;
		it.parts = 1;
		it.cfirst = slot;
		if (slot >= 0) {
			it.ccount = seen.size[slot].first;
			it.steps = seen.size[slot].second;
			continue;
		}
		it.cfirst = slot = (int)out.size();
		const xmgd_cblock_t &cb = p->cblocks[key[1]];
		emu_chunk c = {};
		int nss = 0, room = 0, code = 0, last = 0, neg = 0, run = 0;
		bool fresh = true;
		auto close = [&](int flags) {
			c.head = nss | (c.head | flags) << 8 | code << 16;
			out.push_back(c);
			fresh = flags & RUN_LAST;
			nss = room = 0;
		};
		for (int q = 0; q < cb.npairs; q++) {
			const int steps = (p->pairs[cb.first_pair + q].k + EMU_KS - 1) / EMU_KS;
			int pc = 0;
			it.steps += (cplx ? 2 : 1) * steps;
			for (int j = 0; j < nmem; j++) {
				const xmgd_pair_t &pr = p->pairs[p->cblocks[key[1 + j]].first_pair + q];
				pc |= ((pr.esign < 0) | (pr.eshift ? 2 : 0)) << (2 * j);
			}
			for (int h = 0; h < (cplx ? 2 : 1); h++) {
				/* this half's factors; after the last one's */
				const int fc = pc ^ (h && !pass ? signs : 0);
				if (q || h) {
					const int x = fc ^ last;
					if (x && x != signs) {
						if (nss)
							close(RUN_LAST);
						else if (!fresh) {
							out.back().head |= RUN_LAST << 8;
							fresh = true;
						}
					} else if (x)
						neg ^= 1;
				}
				last = fc;
				for (int of = 0; of < steps; ) {
					if (!nss) {
						c = emu_chunk{};
						if (fresh) {
							code = fc;
							neg = run = 0;
							c.head = RUN_FIRST;
							fresh = false;
						}
						room = dbl ? kchunk : EMU_CHUNK32;
					}
					/* a stage holds KS steps, fewer at a half's end */
					const int left = steps - of, take = left <= room ? left : room / KS * KS;
					const int n = (take + KS - 1) / KS;
					if (neg)
						c.neg |= ((1u << n) - 1) << nss;
					nss += n;
					if (KS == 2 && (take & 1))
						c.part |= 1u << (nss - 1);
					room -= take;
					of += take;
					if (room == 0 || take < left || (dbl && of == steps))
						close(dbl || ++run == 2 || (code & 0xAA) ? RUN_LAST : 0);
				}
			}
		}
		if (nss)
			close(RUN_LAST);
		out.back().head |= RUN_LAST << 8;
		it.ccount = (int)out.size() - slot;
		seen.size.resize(out.size());
		seen.size[slot] = std::make_pair(it.ccount, it.steps);
	}
}

/* The invariants the kernel's addressing relies on, checked on the host
 * before a work list is uploaded: member tiles inside their views and the
 * stage (rows multiples of 16, stacked without gaps, <= 128 in all), and
 * members that share the M side pair by pair. */
static bool
items_ok(const xmgd_contract_t *p, const std::vector<emu_item> &items,
    const std::vector<emu_member> &mem, bool pair)
{
	for (const emu_item &it : items) {
		if (it.mcount < 1 || it.mcount > (pair ? 1 : EMU_MAXMEM) || it.mfirst < 0 ||
		    (size_t)it.mfirst + it.mcount > mem.size())
			return false;
		const int swp = (it.pr >> 1) & 1, tot = it.pr >> 8;
		const xmgd_cblock_t &c0 = p->cblocks[mem[it.mfirst].cblock];
		if ((it.pr >> 2) & 1) {
			/* M-stacked: the shared N tile, then 32-lane members */
			const int nlen = swp ? c0.n : c0.m;
			if (pair || it.m0 < 0 || it.m0 % EMU_TM || it.m0 >= nlen ||
			    tot != std::min(EMU_TM, (nlen - it.m0 + 15) / 16 * 16))
				return false;
			int off = 0;
			for (int j = 0; j < it.mcount; j++) {
				const emu_member &m = mem[it.mfirst + j];
				if (m.cblock < 0 || m.cblock >= p->ncblocks)
					return false;
				const xmgd_cblock_t &cb = p->cblocks[m.cblock];
				const int ml = swp ? cb.m : cb.n;
				if ((swp ? cb.n : cb.m) != nlen || cb.npairs != c0.npairs ||
				    m.off != off || m.rows < 32 || m.rows % 32 || m.n0 < 0 ||
				    m.n0 % EMU_TM || m.n0 >= ml ||
				    m.rows != std::min(EMU_TM, (ml - m.n0 + 31) / 32 * 32))
					return false;
				for (int q = 0; q < cb.npairs; q++) {
					const xmgd_pair_t &a = p->pairs[c0.first_pair + q];
					const xmgd_pair_t &b = p->pairs[cb.first_pair + q];
					if (a.k != b.k || (swp ? a.bview != b.bview : a.aview != b.aview))
						return false;
				}
				off += m.rows;
			}
			if (off > EMU_TM)
				return false;
			continue;
		}
		const int mlen = swp ? c0.m : c0.n;
		if (it.m0 < 0 || it.m0 % EMU_TM || it.m0 >= mlen)
			return false;
		int off = 0;
		for (int j = 0; j < it.mcount; j++) {
			const emu_member &m = mem[it.mfirst + j];
			if (m.cblock < 0 || m.cblock >= p->ncblocks)
				return false;
			const xmgd_cblock_t &cb = p->cblocks[m.cblock];
			const int nlen = swp ? cb.n : cb.m;
			if ((swp ? cb.m : cb.n) != mlen || cb.npairs != c0.npairs ||
			    m.off != off || m.rows < 16 || m.rows % 16 || m.n0 < 0 ||
			    m.n0 % EMU_TM || m.n0 >= nlen ||
			    m.rows > std::min(EMU_TM, (nlen - m.n0 + 15) / 16 * 16))
				return false;
			for (int q = 0; q < cb.npairs; q++) {
				const xmgd_pair_t &a = p->pairs[c0.first_pair + q];
				const xmgd_pair_t &b = p->pairs[cb.first_pair + q];
				if (a.k != b.k || (swp ? a.aview != b.aview : a.bview != b.bview))
					return false;
			}
			off += m.rows;
		}
		if (off != tot || tot < 16 || tot > EMU_TM)
			return false;
	}
	return true;
}

/* Modelled cycles of one K step of a tile of n columns: its MMAs (issue_set)
 * at max(columns / 2, 28 + columns / 6) cycles each, or the shared memory's
 * traffic at 128 B per cycle if that takes longer: each M-side slice once,
 * an N-side slice per product, the copied bytes. */
static double
step_cycles(bool dbl, bool rowmajor, int n)
{
	const int S = dbl ? fin<double>::S : fin<float>::S, products = dbl ? 21 : 6;
	double c = 0;
	auto mma = [&](int slices, int count) {
		c += count * std::max(slices * n / 2.0, 28 + slices * n / 6.0);
	};
	if (rowmajor)
		mma(1, products);
	else if (!dbl) {
		mma(2, 1);
		mma(1, 4);
	} else if (n <= 80) {
		mma(3, 5);
		mma(2, 2);
		mma(1, 2);
	} else {
		mma(2, n <= 96 ? 6 : 4);
		mma(1, n <= 96 ? 9 : 13);
	}
	return std::max(c, (S * EMU_TM + products * n + S * (EMU_TM + n)) / 4.0);
}

/* modelled cycles of a work list on the chip: the SMs' share, at least the
 * longest item */
static double
list_cycles(const xmgd_contract_t *p, const std::vector<emu_item> &items,
    const std::vector<emu_member> &mem, int cplx, bool rowmajor)
{
	double sum = 0, top = 0;
	for (const emu_item &it : items) {
		const xmgd_cblock_t &cb = p->cblocks[mem[it.mfirst].cblock];
		double steps = 0;
		for (int q = 0; q < cb.npairs; q++)
			steps += (cplx ? 2 : 1) * ((p->pairs[cb.first_pair + q].k + EMU_KS - 1) / EMU_KS);
		const double c = steps * step_cycles(p->dtype >= 2, rowmajor, it.pr >> 8);
		sum += c;
		top = std::max(top, c);
	}
	return std::max(top, sum / std::max(1, num_sms()));
}

/*
 * Lists of a few items per SM: the longest ones first, in eight classes (the
 * order within a class, which shares operands, stays; not worth the host's 10
 * to 20 us for lists of less than 0.8 ms), and items divided along K where that
 * ends a list sooner by a model: the SMs' share and 0.6 of the
 * longest item, or the rounds of the longest; parts of at least four chunks and
 * about all, a half, a third or a quarter of an SM's share.  (Dividing lists of
 * a modelled 0.15 ms and less costs the host more than it gives: an adjoint of
 * new tensors, two such GEMMs, 1575 -> 1680 us with it.)  A part costs some 8000
 * cycles beside its steps (the pipeline's ends, the sums' way through L2).
 * GEMM of a 53 x 187 ladder (some 900 items, ordered) 1619 -> 1486 us, of a
 * complex128 ring term, 21 x 75 (divided) 428 -> 383 us; 16 items per SM and
 * more are even enough.  all: short lists too (XMG_EMU_DIVIDE=1, for tests).
 * Returns the number of slots.
 */
static int
split_items(const xmgd_contract_t *p, int cplx, bool rowmajor, size_t sms, bool all,
    const std::vector<emu_chunk> &chunks, const std::vector<emu_member> &members,
    std::vector<emu_item> &items)
{
	const double over = 8000;
	const int KS = p->dtype >= 2 ? stage_cfg<fin<double>::S>::KSTEPS :
	    stage_cfg<fin<float>::S>::KSTEPS;
	const size_t n = items.size();
	double width[EMU_TM / 16 + 1], sum = 0, top = 0;

	if (n >= 16 * sms)
		return 0;
	for (int w = 1; w <= EMU_TM / 16; w++)
		width[w] = step_cycles(p->dtype >= 2, rowmajor, 16 * w);
	std::vector<double> cost(n);
	for (size_t i = 0; i < n; i++) {
		cost[i] = over + items[i].steps * width[items[i].pr >> 12];
		sum += cost[i];
		top = std::max(top, cost[i]);
	}
	/* parts of an item at a target (none below a quarter above it) */
	auto parts = [&](size_t i, double target) {
		if (cost[i] <= 1.25 * target)
			return 1;
		return std::max(1, std::min(items[i].ccount / 4, (int)ceil(cost[i] / target - 0.25)));
	};
	auto model = [&](double total, double longest, size_t count) {
		const double rounds = (double)((count + sms - 1) / sms);
		return std::min(total / sms + 0.6 * longest, rounds * longest);
	};
	double best = 0.93 * model(sum, top, n), target = 0;
	const bool divide = n < 8 * sms && (sum / sms >= 2.8e5 || all);
	for (int w = 1; w <= 4 && divide; w++) {
		const double t = sum / sms / w;
		double total = 0, longest = 0;
		size_t count = 0;
		if (top <= 1.25 * t)
			continue;
		for (size_t i = 0; i < n; i++) {
			const int q = parts(i, t);
			const double c = q == 1 ? cost[i] : (cost[i] - over) / q + over;
			total += q * c;
			count += q;
			longest = std::max(longest, c);
		}
		if (model(total, longest, count) < best) {
			best = model(total, longest, count);
			target = t;
		}
	}
	if (target == 0 && sum / sms < 1.5e6)
		return 0;
	std::vector<emu_item> out;
	int slots = 0;
	out.reserve(n);
	std::vector<double> c2;
	for (size_t i = 0; i < n && target > 0; i++) {
		const emu_item &it = items[i];
		const int q = parts(i, target);
		const size_t at = out.size();
		if (q == 1) {
			out.push_back(it);
			c2.push_back(cost[i]);
			continue;
		}
		/* cut after the run in which each part's share of steps ends */
		const xmgd_cblock_t &cb = p->cblocks[members[it.mfirst].cblock];
		emu_item x = it;
		int done = 0, pair = 0, k = 0;
		x.slot = slots;
		x.steps = 0;
		for (int c = 0; c < it.ccount; c++) {
			const emu_chunk &ch = chunks[it.cfirst + c];
			const int mine = (int)(out.size() - at) + 1;
			x.steps += (ch.head & 0xff) * KS - __builtin_popcount(ch.part);
			if (c + 1 < it.ccount && (!(ch.head >> 8 & RUN_LAST) || mine == q ||
			    done + x.steps < (long long)it.steps * mine / q))
				continue;
			x.ccount = it.cfirst + c + 1 - x.cfirst;
			x.p0 = pair;
			x.k0 = k;
			out.push_back(x);
			c2.push_back((cost[i] - over) * x.steps / it.steps + over);
			done += x.steps;
			/* where the next part starts */
			for (k += x.steps; pair < cb.npairs; pair++) {
				const int nks = (cplx ? 2 : 1) *
				    ((p->pairs[cb.first_pair + pair].k + EMU_KS - 1) / EMU_KS);
				if (k < nks)
					break;
				k -= nks;
			}
			x.cfirst += x.ccount;
			x.steps = 0;
		}
		for (size_t y = at; y < out.size(); y++)
			out[y].parts = (int)(out.size() - at);
		slots += out.size() - at > 1;
	}
	if (target > 0) {
		items.swap(out);
		cost.swap(c2);
		top = 0;
		for (double c : cost)
			top = std::max(top, c);
	}
	/* by class, longest first */
	size_t first[10] = {};
	auto cls = [&](size_t i) { return 8 - (int)(8 * cost[i] / top); };
	for (size_t i = 0; i < items.size(); i++)
		first[cls(i) + 1]++;
	for (int c = 1; c < 10; c++)
		first[c] += first[c - 1];
	out.resize(items.size());
	for (size_t i = 0; i < items.size(); i++)
		out[first[cls(i)]++] = items[i];
	items.swap(out);
	return slots;
}

/* K steps of every block's pairs in all */
static std::vector<int>
block_steps(const xmgd_contract_t *p, int cplx)
{
	std::vector<int> steps(p->ncblocks, 0);
	for (int i = 0; i < p->ncblocks; i++)
		for (int q = 0; q < p->cblocks[i].npairs; q++)
			steps[i] += (cplx ? 2 : 1) *
			    ((p->pairs[p->cblocks[i].first_pair + q].k + EMU_KS - 1) / EMU_KS);
	return steps;
}

/* What the kernel takes from a list with its chunks and parts beyond
 * items_ok, in O(items): an item's chunks lie in the array; an undivided one
 * starts at its first step and holds all of them; the parts of a slot are as
 * many as each of them says, share tile and members, and follow one another
 * from the first step and chunk to the last. */
static bool
parts_ok(const xmgd_contract_t *p, int cplx, const std::vector<int> &steps_of,
    const std::vector<emu_item> &items, const std::vector<emu_member> &mem,
    const std::vector<emu_chunk> &chunks, int nslots)
{
	struct place { int steps, chunk, item; };
	std::vector<std::vector<place>> slot(nslots);
	for (size_t i = 0; i < items.size(); i++) {
		const emu_item &it = items[i];
		const int ci = mem[it.mfirst].cblock;
		const xmgd_cblock_t &cb = p->cblocks[ci];
		if (it.cfirst < 0 || it.ccount < 1 || it.steps < 1 ||
		    (size_t)it.cfirst + it.ccount > chunks.size() || it.p0 < 0 || it.k0 < 0 ||
		    it.p0 >= cb.npairs || it.parts < 1)
			return false;
		if (it.parts == 1) {
			if (it.p0 || it.k0 || it.steps != steps_of[ci])
				return false;
			continue;
		}
		if (it.slot < 0 || it.slot >= nslots)
			return false;
		int before = it.k0;
		for (int q = 0; q < it.p0; q++)
			before += (cplx ? 2 : 1) *
			    ((p->pairs[cb.first_pair + q].k + EMU_KS - 1) / EMU_KS);
		slot[it.slot].push_back(place{before, it.cfirst, (int)i});
	}
	for (std::vector<place> &v : slot) {
		std::sort(v.begin(), v.end(),
		    [](const place &x, const place &y) { return x.steps < y.steps; });
		int steps = 0, chunk = v.empty() ? 0 : v[0].chunk;
		for (const place &x : v) {
			const emu_item &it = items[x.item], &f = items[v[0].item];
			if (it.parts != (int)v.size() || x.steps != steps || x.chunk != chunk ||
			    it.m0 != f.m0 || it.pr != f.pr || it.mfirst != f.mfirst ||
			    it.mcount != f.mcount)
				return false;
			steps += it.steps;
			chunk += it.ccount;
		}
		if (v.size() < 2 || steps != steps_of[mem[items[v[0].item].mfirst].cblock])
			return false;
	}
	return true;
}

/* The same against the roles of the kernel, stage by stage: the stages the
 * producer fills from (p0, k0) on are the ones the chunks count, of one step
 * where they say so, with the members' factors; chunks and runs stay below
 * the accumulators' exact ranges (see emu_chunk).  As long as the list's K
 * steps: for the host checks. */
static bool
chunks_ok(const xmgd_contract_t *p, int cplx, int kchunk, const std::vector<emu_item> &items,
    const std::vector<emu_member> &mem, const std::vector<emu_chunk> &chunks)
{
	const bool dbl = p->dtype >= 2;
	const int KS = dbl ? stage_cfg<fin<double>::S>::KSTEPS : stage_cfg<fin<float>::S>::KSTEPS;

	for (const emu_item &it : items) {
		const int pass = it.pr & 1;
		const xmgd_cblock_t &cb = p->cblocks[mem[it.mfirst].cblock];
		int q = it.p0, k = it.k0, left = it.steps, run = 0, code = 0;
		for (int c = 0; c < it.ccount; c++) {
			const emu_chunk &ch = chunks[it.cfirst + c];
			const int nss = ch.head & 0xff, fl = ch.head >> 8 & 0xff;
			const bool last = c + 1 == it.ccount;
			int steps = 0, from = -1;
			if (nss < 1 || nss > 32 || (run == 0) != ((fl & RUN_FIRST) != 0) ||
			    (fl & ITEM_LAST) || (last && !(fl & RUN_LAST)))
				return false;
			if (run++ == 0)
				code = ch.head >> 16;
			if (ch.head >> 16 != code || code >> (2 * it.mcount))
				return false;
			for (int j = 0; j < nss; j++) {
				if (q >= cb.npairs)
					return false;
				const int nks = (cplx ? 2 : 1) *
				    ((p->pairs[cb.first_pair + q].k + EMU_KS - 1) / EMU_KS);
				const int half = cplx && k >= nks / 2;
				const int end = cplx && !half ? nks / 2 : nks, n = std::min(KS, end - k);
				if (n != (KS == 2 && !(ch.part >> j & 1) ? 2 : 1))
					return false;
				for (int m = 0; m < it.mcount; m++) {
					const xmgd_pair_t &pr =
					    p->pairs[p->cblocks[mem[it.mfirst + m].cblock].first_pair + q];
					const int neg = (pr.esign < 0) ^ (half && !pass);
					const int has = code >> (2 * m) & 3;
					if ((has & 1) != (neg ^ (int)(ch.neg >> j & 1)) ||
					    (has >> 1) != (pr.eshift ? 1 : 0))
						return false;
				}
				/* FP64: one segment, as the drains' error asks */
				if (dbl && from >= 0 && from != 2 * q + half)
					return false;
				from = 2 * q + half;
				steps += n;
				k += n;
				if (k == nks) {
					k = 0;
					q++;
				}
			}
			left -= steps;
			if (steps > (dbl ? kchunk : EMU_CHUNK32) ||
			    run > (dbl || (code & 0xAA) ? 1 : 2))
				return false;
			if (fl & RUN_LAST)
				run = 0;
		}
		if (left != 0)
			return false;
	}
	return true;
}

/* bytes of one K step of a view with mn rows: whole tiles, then the last
 * one's rows (tile_rows) */
static size_t
view_step_bytes(int mn, int chunk_bytes)
{
	const int full = (mn - 1) / EMU_TM;
	return (size_t)full * chunk_bytes +
	    (size_t)tile_rows(mn, full * EMU_TM) * chunk_bytes / EMU_TM;
}

int
emu_prepare(const xmgd_contract_t *p, const std::vector<int> &cblocks,
    const xmgd_cblock_t *d_cbs, const xmgd_pair_t *d_prs,
    const int32_t *d_tabs, emu_plan **out)
{
	const bool realab = p->alpha[1] == 0 && p->beta[1] == 0;
	int cplx, st;

	*out = nullptr;
	switch (p->dtype) {
	case 0: case 2: cplx = 0; break;
	case 1: case 3:
		/* two real passes need real alpha and beta */
		if (!realab)
			return xmg_seterr(XMG_ENOTSUP, "split-precision path: complex "
			    "alpha/beta");
		cplx = 1;
		break;
	default:
		return xmg_seterr(XMG_ENOTSUP, "split-precision path: scalar type");
	}
	const bool dbl = p->dtype >= 2;
	const int chunk_bytes = (dbl ? fin<double>::S : fin<float>::S) * SLICE_BYTES;
	emu_plan *e = new emu_plan();
	e->dtype = p->dtype;
	e->cplx = cplx;
	{
		const int nst = dbl ? stage_cfg<fin<double>::S>::NST : stage_cfg<fin<float>::S>::NST;
		/* head/tail length in stages */
		const char *h = getenv("XMG_EMU_HEAD");
		e->hmax = h ? atoi(h) : 3;
		e->hmax = std::max(1, std::min(nst, e->hmax));
		/* FP64 chunks in whole stages (they start at a segment's first
		 * step, as the stages do) */
		const char *kc = getenv("XMG_EMU_CHUNK");
		constexpr int KS64 = stage_cfg<fin<double>::S>::KSTEPS;
		e->kchunk = kc ? std::max(1, std::min(20, atoi(kc))) : EMU_CHUNK;
		e->kchunk = std::max(KS64, e->kchunk / KS64 * KS64);
	}
	e->alpha = p->alpha[0];
	e->beta = p->beta[0];
	e->d_cbs = d_cbs;
	e->d_prs = d_prs;
	e->d_tabs = d_tabs;
	e->VA.assign(p->views_a, p->views_a + p->nviews_a);
	e->VB.assign(p->views_b, p->views_b + p->nviews_b);
	/* the plan that prepares a shared a side splits every view of a */
	e->a_mode = p->a_mode;
	e->a_slices = p->a_slices;
	e->a_E = p->a_E;
	e->a_flag = p->a_flag;
	e->useA.assign(e->VA.size(), p->a_mode == 1);
	e->useB.assign(e->VB.size(), 0);
	e->split = dbl ? launch_split<double> : launch_split<float>;
	e->gemm = dbl ? launch_gemm<double, double> : launch_gemm<float, float>;
	if ((st = dbl ? set_attrs<double, double>() : set_attrs<float, float>()))
		goto fail;

	{
	/* operand views used by the emulated blocks, and the fixed-point
	 * scale F of every block (|V| <= K_eff * 2^(30+F) <= 2^62) */
	std::vector<int32_t> F(p->ncblocks, 0);
	std::vector<uint64_t> hist;
	for (int ci : cblocks) {
		const xmgd_cblock_t &cb = p->cblocks[ci];
		double keff = 0;
		int64_t ksum = 0;
		for (int q = 0; q < cb.npairs; q++) {
			const xmgd_pair_t &pr = p->pairs[cb.first_pair + q];
			e->useA[pr.aview] = e->useB[pr.bview] = 1;
			double kr = cplx ? 2.0 * 16 * ((pr.k + 15) / 16) : pr.k;
			keff += ldexp(1.0, std::max(pr.eshift, 0)) * kr;
			ksum += pr.k;
		}
		int lg = (int)ceil(log2(std::max(keff, 2.0)));
		if (lg > 31) {
			st = xmg_seterr(XMG_ENOTSUP, "split-precision path: K too large");
			goto fail;
		}
		/* (FP32 has no rounded terms to place below its integers) */
		F[ci] = dbl ? std::max(1, std::min(15, 31 - lg)) : 0;
		hist.push_back(mix64(((uint64_t)cb.m << 40) ^ ((uint64_t)cb.n << 20) ^
		    (uint64_t)ksum));
	}
	std::sort(hist.begin(), hist.end());
	uint64_t sig = mix64((uint64_t)p->dtype + 1);
	for (uint64_t h : hist)
		sig = mix64(sig ^ h);
	e->sig = sig;

	/* slice storage: offsets now, rebased onto the workspace at bind */
	size_t off = 0;
	auto tile = [&](std::vector<xmgd_view_t> &V, std::vector<char> &use,
	    const int64_t *ext) {
		for (size_t v = 0; v < V.size(); v++) {
			if (!use[v])
				continue;
			xmgd_view_t &w = V[v];
			w.n_rt = (w.mn + EMU_TM - 1) / EMU_TM;
			w.cplx = cplx;
			w.khp = EMU_KS * ((w.k + EMU_KS - 1) / EMU_KS);
			w.n_ks = (cplx ? 2 : 1) * (w.khp / EMU_KS);
			w.kfast = w.k > 1 && p->tabs[w.rowtab + 1] - p->tabs[w.rowtab] == 1;
			w.kcontig = w.kfast;
			for (int32_t k = 2; w.kcontig && k < w.k; k++)
				w.kcontig = p->tabs[w.rowtab + k] - p->tabs[w.rowtab] == k;
			if (ext) {	/* in the shared a side's buffer */
				w.slices = (uint64_t)ext[v];
				continue;
			}
			w.slices = off;
			off += (size_t)w.n_ks * view_step_bytes(w.mn, chunk_bytes);
		}
	};
	tile(e->VA, e->useA, p->a_mode ? p->a_off : nullptr);
	tile(e->VB, e->useB, nullptr);
	e->slice_bytes = off;

	upload_batch up;
	/* CTA ranges of the exponent and split launches of each side */
	for (int side = 0; side < 2; side++) {
		std::vector<xmgd_view_t> &V = side ? e->VB : e->VA;
		std::vector<char> &use = side ? e->useB : e->useA;
		/* the exponent pass: K ranges of 256 (one atomic per row and CTA
		 * from the fewest CTAs), halved down to 32 while the grid is
		 * below two CTAs per SM (24 x 64 ladder, exponent and split pass:
		 * 54 us with eight, 48 with four, 47 with two; more CTAs, whose
		 * warps' sums outweigh their loads) */
		for (int &kr = e->kr[side]; kr > 32; kr /= 2) {
			int64_t n = 0;
			for (size_t v = 0; v < V.size(); v++)
				if (use[v])
					n += (int64_t)V[v].n_rt * ((V[v].k + kr - 1) / kr);
			if (n >= 2 * num_sms())
				break;
		}
		for (int kind = 0; kind < 2; kind++) {
			std::vector<view_meta> meta(V.size());
			int64_t n = 0;
			for (size_t v = 0; v < V.size(); v++) {
				meta[v].first_cta = n;
				if (!use[v])
					continue;
				if (kind == 0)
					n += (int64_t)V[v].n_rt * ((V[v].k + e->kr[side] - 1) / e->kr[side]);
				else
					n += (int64_t)V[v].n_rt * ((V[v].n_ks + 3) / 4);
			}
			e->nctas[side][kind] = n;
			up.add(meta.data(), meta.size() * sizeof(view_meta), &e->d_meta[side][kind]);
		}
	}
	e->nexp_a = p->nexp_a;
	e->nE = (int64_t)p->nexp_a + p->nexp_b;
	up.add(nullptr, (e->nE + 64) * sizeof(int32_t), &e->d_E);
	up.add(F.data(), F.size() * sizeof(int32_t), &e->d_F);
	/* (the views go up when bound: one array, a's then b's) */
	up.add(nullptr, (e->VA.size() + e->VB.size()) * sizeof(xmgd_view_t) + 16, &e->d_va);

	/* work lists: a remembered policy for this histogram, else every
	 * distinct policy once */
	int known = -1;
	for (const tune_entry &t : g_tuned)
		if (t.sig == sig)
			known = t.policy;
	if (getenv("XMG_TUNE") && strcmp(getenv("XMG_TUNE"), "0") == 0)
		known = EMU_POL_MERGED;
	if (getenv("XMG_POLICY"))	/* one fixed work-list policy */
		known = atoi(getenv("XMG_POLICY"));
	/* a plan that runs once has no runs left to tune with: the list the
	 * model puts first */
	const bool first_only = p->one_shot && known < 0;
	std::vector<int> pols = {EMU_POL_MERGED, 0, 1, 2};
	if (pairs_enabled())
		pols.insert(pols.end(), {EMU_NPOLICY, EMU_NPOLICY + 1, EMU_NPOLICY + 2});
	/* batches that share a's operands agree on their layout */
	if (p->a_mode && !getenv("XMG_POLICY")) {
		known = known >= 0 && row_major(known) ? known : -1;
		pols.erase(std::remove_if(pols.begin(), pols.end(),
		    [](int q) { return !row_major(q); }), pols.end());
	}
	std::vector<std::vector<emu_item>> lists;
	std::vector<uint64_t> whole;
	std::vector<std::vector<emu_member>> mlists;
	std::vector<double> est;
	chunk_index seen;
	std::vector<emu_chunk> chunks;
	const char *div = getenv("XMG_EMU_DIVIDE");
	const bool divide_all = div && atoi(div) == 1;
	const std::vector<int> steps_of = block_steps(p, cplx);
	for (int pol : pols) {
		if (known >= 0 && pol != known)
			continue;
		std::vector<emu_item> items;
		std::vector<emu_member> mem;
		make_items(p, cblocks, cplx, pol, items, mem);
		/* a list that fails its checks is never uploaded; the others
		 * stand in for it */
		if (!items_ok(p, items, mem, pair_policy(pol)))
			continue;
		chunk_lists(p, cplx, e->kchunk, items, mem, seen, chunks);
		const double cycles = list_cycles(p, items, mem, cplx, row_major(pol));
		/* (lists are divided later: their sums tell them apart) */
		uint64_t sum = items.size();
		for (const emu_item &it : items)
			sum = (sum ^ ((uint64_t)(uint32_t)it.m0 << 32 | (uint32_t)it.pr) ^
			    (uint64_t)it.mfirst << 20) * 0x9e3779b97f4a7c15ull;
		bool dup = false;
		for (size_t l = 0; l < lists.size(); l++)
			dup |= row_major(e->cand[l].policy) == row_major(pol) &&
			    pair_policy(e->cand[l].policy) == pair_policy(pol) &&
			    whole[l] == sum && mlists[l].size() == mem.size() &&
			    memcmp(mlists[l].data(), mem.data(), mem.size() * sizeof(emu_member)) == 0;
		if (dup)
			continue;
		emu_cand c;
		c.policy = pol;
		c.nslots = pair_policy(pol) ? 0 : split_items(p, cplx, row_major(pol),
		    (size_t)num_sms(), divide_all, chunks, mem, items);
		if (!parts_ok(p, cplx, steps_of, items, mem, chunks, c.nslots))
			continue;
		whole.push_back(sum);
		e->slot_bytes = std::max(e->slot_bytes, c.nslots * SLOT_BYTES);
		c.nitems = (int)items.size();
		c.grid = pair_policy(pol) ? 2 * std::min(c.nitems, num_sms() / 2) :
		    std::min(c.nitems, num_sms());
		c.ms = -1;
		c.d_items = c.d_members = 0;
		est.push_back(cycles);
		e->cand.push_back(c);
		lists.push_back(std::move(items));
		mlists.push_back(std::move(mem));
	}
	/* in the model's order; lists a quarter above the best are not tried
	 * (measured spread of the model's ratios: +-10 %) */
	{
		std::vector<int> ord(e->cand.size());
		for (size_t i = 0; i < ord.size(); i++)
			ord[i] = (int)i;
		std::stable_sort(ord.begin(), ord.end(),
		    [&](int x, int y) { return est[x] < est[y]; });
		std::vector<emu_cand> keep;
		std::vector<int> kept;
		for (int i : ord)
			if (keep.empty() || !(first_only || est[i] > 1.25 * est[ord[0]])) {
				keep.push_back(e->cand[i]);
				kept.push_back(i);
			}
		e->cand = keep;
		for (size_t i = 0; i < kept.size(); i++) {
			const int l = kept[i];
			up.add(lists[l].data(), lists[l].size() * sizeof(emu_item),
			    &e->cand[i].d_items);
			up.add(mlists[l].data(), mlists[l].size() * sizeof(emu_member),
			    &e->cand[i].d_members);
		}
	}
	up.add(chunks.data(), chunks.size() * sizeof(emu_chunk), &e->d_chunks);
	if (e->cand.empty()) {
		st = xmg_seterr(XMG_EINVAL, "split-precision path: no work list "
		    "passed its checks");
		goto fail;
	}
	e->tuned = e->cand.size() <= 1;
	if ((st = flag_pair(&e->h_flags)) || (st = up.commit(&e->dbuf)) ||
	    (st = check(cudaStreamSynchronize(stream()), "plan upload")))
		goto fail;
	e->d_vb = e->d_va + e->VA.size() * sizeof(xmgd_view_t);
	e->h_flags[0] = e->h_flags[1] = 0;
	}
	*out = e;
	return XMG_OK;
fail:
	emu_free(e);
	return st;
}

/* Slice workspace and absolute view addresses; *moved when the views had
 * to be re-uploaded (a captured graph holding the old ones is stale). */
int
emu_bind(emu_plan *e, bool *moved)
{
	uint64_t ws;
	int st;

	*moved = false;
	if ((st = xmgd_scratch(8, slot_offset(e) + e->slot_bytes + 16, &ws)) != XMG_OK)
		return st;
	if (ws == e->ws)
		return XMG_OK;
	e->vstage = e->VA;
	e->vstage.insert(e->vstage.end(), e->VB.begin(), e->VB.end());
	for (size_t v = 0; v < e->vstage.size(); v++) {
		const bool isa = v < e->VA.size();
		if (isa ? e->useA[v] : e->useB[v - e->VA.size()])
			e->vstage[v].slices += isa && e->a_mode ? e->a_slices : ws;
	}
	/* (the staged copy lives as long as the plan) */
	XMG_CK(cudaMemcpyAsync((void *)e->d_va, e->vstage.data(), e->vstage.size() *
	    sizeof(xmgd_view_t), cudaMemcpyHostToDevice, stream()));
	e->ws = ws;
	*moved = true;
	return XMG_OK;
}

/* The work list of one policy, built and checked on the host (no device) as
 * emu_prepare uploads it.  sms: the SMs it is divided for (0: the device's;
 * below 0: not divided), with short lists if all; slots, chunks: its numbers
 * of both. */
static int
checked_list(const xmgd_contract_t *p, int policy, int sms, bool all,
    std::vector<emu_item> &items, std::vector<emu_member> &mem, int *slots, size_t *nchunks,
    bool *ok)
{
	int cplx;

	switch (p->dtype) {
	case 0: case 2: cplx = 0; break;
	case 1: case 3: cplx = 1; break;
	default:
		return xmg_seterr(XMG_EINVAL, "work list: scalar type");
	}
	if (policy < 0 || (policy >= EMU_NPOLICY && !pair_policy(policy) &&
	    policy != EMU_POL_MERGED))
		return xmg_seterr(XMG_EINVAL, "work list: no policy %d", policy);
	std::vector<int> cblocks;
	for (int i = 0; i < p->ncblocks; i++)
		if (p->cblocks[i].npairs > 0 && p->emulatable[i])
			cblocks.push_back(i);
	make_items(p, cblocks, cplx, policy, items, mem);
	chunk_index seen;
	std::vector<emu_chunk> chunks;
	*slots = 0;
	if ((*ok = items_ok(p, items, mem, pair_policy(policy)))) {
		chunk_lists(p, cplx, EMU_CHUNK, items, mem, seen, chunks);
		if (sms >= 0 && !pair_policy(policy))
			*slots = split_items(p, cplx, row_major(policy),
			    (size_t)(sms ? sms : std::max(1, num_sms())), all, chunks, mem, items);
		*ok = parts_ok(p, cplx, block_steps(p, cplx), items, mem, chunks, *slots) &&
		    chunks_ok(p, cplx, EMU_CHUNK, items, mem, chunks);
	}
	*nchunks = chunks.size();
	return XMG_OK;
}

extern "C" int
xmgd_work_list_check(const xmgd_contract_t *p, int policy, long long out[4])
{
	std::vector<emu_item> items;
	std::vector<emu_member> mem;
	size_t nchunks;
	int slots, st;
	bool ok;

	if ((st = checked_list(p, policy, -1, false, items, mem, &slots, &nchunks, &ok)) != XMG_OK)
		return st;
	long long stacked = 0;
	for (const emu_item &it : items)
		stacked += it.mcount > 1;
	out[0] = (long long)items.size();
	out[1] = (long long)mem.size();
	out[2] = stacked;
	out[3] = ok;
	return XMG_OK;
}

extern "C" int
xmgd_work_list_parts(const xmgd_contract_t *p, int policy, int sms, long long out[4])
{
	std::vector<emu_item> items;
	std::vector<emu_member> mem;
	size_t nchunks;
	int slots, st;
	bool ok;

	if ((st = checked_list(p, policy, std::max(0, sms), true, items, mem, &slots, &nchunks,
	    &ok)) != XMG_OK)
		return st;
	out[0] = (long long)items.size();
	out[1] = slots;
	out[2] = (long long)nchunks;
	out[3] = ok;
	return XMG_OK;
}

int emu_current(const emu_plan *e) { return e->cur; }
int emu_ncand(const emu_plan *e) { return (int)e->cand.size(); }
bool emu_tuned(const emu_plan *e) { return e->tuned != 0; }

int emu_record_split(emu_plan *e) { return e->split(e); }
int emu_record_gemm(emu_plan *e) { return e->gemm(e); }
int64_t emu_slice_bytes(const emu_plan *e) { return (int64_t)e->slice_bytes; }
int emu_a_mode(const emu_plan *e) { return e->a_mode; }

/* part_at on the host: what the kernels of the operand pass index with */
extern "C" int64_t
xmgd_emu_part_at(int32_t row, int32_t col, int half)
{
	return part_at(row, col, half);
}

/* the slice bytes tile() gives one view */
extern "C" int64_t
xmgd_emu_view_bytes(const xmgd_view_t *v, int dtype)
{
	if (dtype < 0 || dtype > 3)
		return 0;
	const bool cplx = dtype == 1 || dtype == 3;
	const int chunk_bytes = (dtype >= 2 ? fin<double>::S : fin<float>::S) *
	    SLICE_BYTES;
	const int64_t n_ks = (cplx ? 2 : 1) * ((v->k + EMU_KS - 1) / EMU_KS);
	return n_ks * (int64_t)view_step_bytes(v->mn, chunk_bytes);
}
int emu_items(const emu_plan *e) { return e->cand[e->cur].nitems; }
int emu_policy(const emu_plan *e) { return e->cand[e->cur].policy; }

/* after the stream has drained: flags, then one tuning step with the
 * measured GEMM time of the candidate that ran */
int
emu_finish(emu_plan *e, float gemm_ms, int *nan)
{
	*nan = e->h_flags[0] & 1;
	if (e->h_flags[1])
		return xmg_seterr(XMG_ETIMEOUT, "split-precision GEMM: bounded "
		    "wait %d timed out", e->h_flags[1]);
	if (!e->tuned && !*nan) {
		e->cand[e->cur].ms = gemm_ms;
		if (e->cur + 1 < (int)e->cand.size())
			e->cur++;
		else {
			int best = 0;
			for (int i = 1; i < (int)e->cand.size(); i++)
				if (e->cand[i].ms < e->cand[best].ms)
					best = i;
			e->cur = best;
			e->tuned = 1;
			g_tuned.push_back(tune_entry{e->sig, e->cand[best].policy});
		}
	}
	return XMG_OK;
}

} /* namespace xmg */
