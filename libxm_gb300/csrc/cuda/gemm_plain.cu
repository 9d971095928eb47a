/*
 * Plain grouped block-pair GEMM of libxm-gb300 (the FP64 form, and the
 * float / complex forms on the CUDA cores).
 *
 * One launch computes every canonical output block assigned to it:
 *     C = beta * C + sum_p al_p * A_p^T B_p
 * over the block's merged pairs (contract.c:193-218 issues one host BLAS
 * call per pair instead).  The unfold of A_p, B_p and the fold of C are
 * not separate passes: tile loads gather through the per-operand offset
 * tables (element (k, i) of A_p at a_ptr + arow[k] + acol[i]) and the
 * epilogue scatters C the same way, so operands are read once from their
 * canonical storage and C is written once.
 *
 * Work items (block, m-tile, n-tile) arrive sorted by cost.  The float forms
 * run 64 x 64 tiles, 256 threads with 4 x 4 accumulators each.  The double
 * forms are bound by the FP64 pipe (2 multiply-adds a cycle and SM: a warp's
 * takes 64 cycles of its scheduler), beside which loads, shared memory and
 * L2 traffic are free; what costs is work on padding and SMs left without
 * work, so they run small tiles on 128 threads (a warp per scheduler):
 * 16 x 16, or 32 x 32 where there are thousands of those; thread rows and
 * columns past the block are skipped.  Ladder o20/v57 (2.6 GFLOP in 30
 * blocks): 210 tiles of 64 x 64 on 152 SMs took 4.40 ms, 16 x 16 tiles 2.50
 * (2.46 at the pipe's rate).
 */
#include <type_traits>

#include "common.cuh"

namespace xmg {

constexpr int PG_BK = 16;

struct pg_item {
	int32_t cblock, m0, n0, pad;
};

/* TB x TB tile, TM x TN outputs per thread: rows tx + (TB / TM) i, columns
 * ty + (TB / TN) j */
template <typename T, int TB, int TM, int TN>
struct pg {
	static constexpr int NX = TB / TM, NY = TB / TN, THREADS = NX * NY;
	static constexpr int NL = TB * PG_BK / THREADS;	/* loads per operand */

	/* this thread's NL elements of the K x TB operand tile at (k0, c0):
	 * consecutive threads walk k where K runs along memory, else the free
	 * index */
	static __device__ __forceinline__ void
	fetch(T (&v)[NL], const T *__restrict__ base, const int32_t *__restrict__ rowt,
	    const int32_t *__restrict__ colt, int k0, int kmax, int c0, int cmax,
	    bool kfast)
	{
		const int t = threadIdx.x;
#pragma unroll
		for (int r = 0; r < NL; r++) {
			const int kk = kfast ? t % PG_BK : t / TB + r * (THREADS / TB);
			const int cc = kfast ? t / PG_BK + r * (THREADS / PG_BK) : t % TB;
			v[r] = k0 + kk < kmax && c0 + cc < cmax ?
			    base[rowt[k0 + kk] + colt[c0 + cc]] : num<T>::zero();
		}
	}

	static __device__ __forceinline__ void
	put(T (*S)[TB + 1], const T (&v)[NL], bool kfast, const T *scale)
	{
		const int t = threadIdx.x;
#pragma unroll
		for (int r = 0; r < NL; r++) {
			const int kk = kfast ? t % PG_BK : t / TB + r * (THREADS / TB);
			const int cc = kfast ? t / PG_BK + r * (THREADS / PG_BK) : t % TB;
			S[kk][cc] = scale ? num<T>::mul(*scale, v[r]) : v[r];
		}
	}
};

/* ALL (float lists whose tiles are not mostly empty): every thread computes
 * its TM x TN outputs, past the block too, and a tile is loaded when it is due.
 * A float's multiply-add costs less than the branches around it (1500 x 1500 x
 * 1500 in 25 blocks 398 us, 756 with them; 16 x 16 x 5000, one sixteenth of a
 * tile, 475 and 353); the next tile's loads in flight change little there
 * (402). */
template <typename T, int TB, int TM, int TN, bool ALL = false>
__global__ void __launch_bounds__(pg<T, TB, TM, TN>::THREADS)
plain_gemm_kernel(const pg_item *__restrict__ items,
    const xmgd_cblock_t *__restrict__ cbs, const xmgd_pair_t *__restrict__ prs,
    const int32_t *__restrict__ tabs, double2 beta2)
{
	using P = pg<T, TB, TM, TN>;
	__shared__ T As[PG_BK][TB + 1];
	__shared__ T Bs[PG_BK][TB + 1];

	const pg_item it = items[blockIdx.x];
	const xmgd_cblock_t cb = cbs[it.cblock];
	const int tx = threadIdx.x % P::NX, ty = threadIdx.x / P::NX;
	/* rows and columns of threads that reach into the block */
	const int mi = ALL ? TM : min(TM, (cb.m - it.m0 + P::NX - 1) / P::NX);
	const int nj = ALL ? TN : min(TN, (cb.n - it.n0 + P::NY - 1) / P::NY);
	T acc[TM][TN];
#pragma unroll
	for (int i = 0; i < TM; i++)
#pragma unroll
		for (int j = 0; j < TN; j++)
			acc[i][j] = num<T>::zero();

	for (int p = 0; p < cb.npairs; p++) {
		const xmgd_pair_t pr = prs[cb.first_pair + p];
		const T *A = reinterpret_cast<const T *>(pr.a_ptr);
		const T *B = reinterpret_cast<const T *>(pr.b_ptr);
		const int32_t *arow = tabs + pr.arow, *acol = tabs + pr.acol;
		const int32_t *brow = tabs + pr.brow, *bcol = tabs + pr.bcol;
		const bool akf = pr.k > 1 && arow[1] - arow[0] == 1;
		const bool bkf = pr.k > 1 && brow[1] - brow[0] == 1;
		const T al = num<T>::mk(pr.al);
		T va[P::NL], vb[P::NL];
		if (!ALL) {
			P::fetch(va, A, arow, acol, 0, pr.k, it.m0, cb.m, akf);
			P::fetch(vb, B, brow, bcol, 0, pr.k, it.n0, cb.n, bkf);
		}
		for (int k0 = 0; k0 < pr.k; k0 += PG_BK) {
			if (ALL) {
				P::fetch(va, A, arow, acol, k0, pr.k, it.m0, cb.m, akf);
				P::fetch(vb, B, brow, bcol, k0, pr.k, it.n0, cb.n, bkf);
			}
			__syncthreads();
			P::put(As, va, akf, &al);
			P::put(Bs, vb, bkf, nullptr);
			__syncthreads();
			if (!ALL && k0 + PG_BK < pr.k) {	/* the next tile, in flight below */
				P::fetch(va, A, arow, acol, k0 + PG_BK, pr.k, it.m0, cb.m, akf);
				P::fetch(vb, B, brow, bcol, k0 + PG_BK, pr.k, it.n0, cb.n, bkf);
			}
			const int kn = min(PG_BK, pr.k - k0);
#pragma unroll 4
			for (int kk = 0; kk < kn; kk++) {
				T a[TM], b[TN];
#pragma unroll
				for (int i = 0; i < TM; i++)
					a[i] = As[kk][tx + P::NX * i];
#pragma unroll
				for (int j = 0; j < TN; j++)
					b[j] = Bs[kk][ty + P::NY * j];
#pragma unroll
				for (int i = 0; i < TM; i++) {
					if (i >= mi)
						break;
#pragma unroll
					for (int j = 0; j < TN; j++)
						if (j < nj)
							acc[i][j] = num<T>::fma(a[i], b[j], acc[i][j]);
				}
			}
		}
	}
	/* fused fold: C = beta * C + acc, scattered through the C tables;
	 * beta == 0 never reads C (contract.c:155-156) */
	T *C = reinterpret_cast<T *>(cb.c_ptr);
	const int32_t *crow = tabs + cb.crow, *ccol = tabs + cb.ccol;
	const double bb[2] = {beta2.x, beta2.y};
	const T beta = num<T>::mk(bb);
	const bool bzero = beta2.x == 0 && beta2.y == 0;
#pragma unroll
	for (int j = 0; j < TN; j++) {
		int n = it.n0 + ty + P::NY * j;
		if (n >= cb.n)
			continue;
		if constexpr (ALL) {
			/* a column's old values together: each load would wait for the
			 * last one's store (4000 x 4000 x 8 floats, beta 1/2: 114 us one by
			 * one, now 95; the FP64 forms take longer with it, a 20 x 57
			 * ladder 2525 -> 2680 us) */
			T *cn = C + ccol[n], old[TM];
#pragma unroll
			for (int i = 0; i < TM; i++) {
				int m = it.m0 + tx + P::NX * i;
				old[i] = bzero || m >= cb.m ? num<T>::zero() : cn[crow[m]];
			}
#pragma unroll
			for (int i = 0; i < TM; i++) {
				int m = it.m0 + tx + P::NX * i;
				if (m >= cb.m)
					continue;
				cn[crow[m]] = bzero ? acc[i][j] : num<T>::fma(beta, old[i], acc[i][j]);
			}
		} else {
			int32_t co = ccol[n];
#pragma unroll
			for (int i = 0; i < TM; i++) {
				int m = it.m0 + tx + P::NX * i;
				if (m >= cb.m)
					continue;
				T *cp = C + crow[m] + co;
				*cp = bzero ? acc[i][j] : num<T>::fma(beta, *cp, acc[i][j]);
			}
		}
	}
}

/* Tile side for a scalar type and the number of 32 x 32 tiles of the work:
 * double types 16 while that is below 32 per SM, else 32. */
int
plain_tile(int dtype, int64_t tiles32)
{
	return dtype < 2 ? 64 : tiles32 < 32 * (int64_t)num_sms() ? 16 : 32;
}

template <typename T>
int
plain_gemm_launch(const void *items, int nitems, int tile, bool full,
    const xmgd_cblock_t *cbs, const xmgd_pair_t *prs, const int32_t *tabs, const double *beta)
{
	const pg_item *it = (const pg_item *)items;
	const double2 b2 = make_double2(beta[0], beta[1]);

	if (nitems == 0)
		return XMG_OK;
	if constexpr (std::is_same<T, double>::value || std::is_same<T, cd>::value) {
		if (tile == 16)
			plain_gemm_kernel<T, 16, 2, 1><<<nitems, 128, 0, stream()>>>(it, cbs, prs,
			    tabs, b2);
		else
			plain_gemm_kernel<T, 32, 4, 2><<<nitems, 128, 0, stream()>>>(it, cbs, prs,
			    tabs, b2);
	} else if (std::is_same<T, float>::value && full)
		plain_gemm_kernel<T, 64, 4, 4, std::is_same<T, float>::value><<<nitems, 256, 0,
		    stream()>>>(it, cbs, prs, tabs, b2);
	else
		plain_gemm_kernel<T, 64, 4, 4><<<nitems, 256, 0, stream()>>>(it, cbs, prs, tabs,
		    b2);
	g_launches++;
	return check(cudaGetLastError(), "plain_gemm_kernel launch");
}

template int plain_gemm_launch<float>(const void *, int, int, bool, const xmgd_cblock_t *,
    const xmgd_pair_t *, const int32_t *, const double *);
template int plain_gemm_launch<double>(const void *, int, int, bool, const xmgd_cblock_t *,
    const xmgd_pair_t *, const int32_t *, const double *);
template int plain_gemm_launch<cf>(const void *, int, int, bool, const xmgd_cblock_t *,
    const xmgd_pair_t *, const int32_t *, const double *);
template int plain_gemm_launch<cd>(const void *, int, int, bool, const xmgd_cblock_t *,
    const xmgd_pair_t *, const int32_t *, const double *);

} /* namespace xmg */
