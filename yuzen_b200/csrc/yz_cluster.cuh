// yz_cluster.cuh -- the BiCGStab run of a small system, and the coarse levels
// of a large one's V-cycle, in one launch each on one thread-block cluster.
//
// An iteration is a chain of some thirty short dependent phases (smoothing,
// residual, restriction, ... , SpMV, dot products).  As separate launches,
// each pays the gap between two kernels and a cold start: about 5 us a phase
// whatever the rows, 110-190 us an iteration from 4,600 to 266,000 rows, and
// a loop graph has to be made for every new hierarchy.  Sixteen blocks of
// one cluster pass from phase to phase over the hardware's cluster barrier
// instead, keep the scalars of the run in every block (each folds the same
// partial sums in the same order), and exchange the partial sums of the dot
// products through distributed shared memory.  An iteration at 4,624 rows
// takes 62 us instead of 125; a phase is the barrier (1,100 cycles, most of
// it its stores reaching L2) and two or three dependent reads from L2.  The
// vectors and matrices stay in global memory: keeping a block's rows of the
// matrices in its shared memory gave 5 % at 4,624 rows.
//
// Loops over a row fill every place of their register arrays (0 where the
// row has ended): an array filled only under a condition stays alive across
// the loop, and 128 registers then spill every load (62 us became 120).
//
// Every sum has the order of the separate kernels and of the oracle.
#pragma once

#include "yz_amg_kernels.cuh"
#include "yz_solver_impl.h"

#include <cooperative_groups.h>

namespace yz {

constexpr int kClT = 512;                    // threads a block
constexpr int kClGroups = kClT / kRT;        // chunks of the reduction a block holds at a time
constexpr int kClMaxLevels = 12;
constexpr int kClBatch = 8;                  // entries of a row loaded together
constexpr int kClMaxChunks = 512;            // chunks of 256 rows a run may have

template<class T>
struct ClLevel
{
	int n, direct, last;                     // last: smoothed only, nothing coarser
	const int *ptr, *col;
	const T *val, *M, *inv;
	const int *rptr, *rcol;
	const T *rval;
	const int *pptr, *pcol;
	const T *pval;
	T *f, *x, *t, *xt;
};

template<class T>
struct ClPlan
{
	int count, sweeps;                       // levels; the finest level's post-smoothing sweeps
	double root[8], ratio;                   // and, for more than one, their Chebyshev roots
	double weight[8];                        // and weights, taken at the kernel's start (ChebWeight)
	const double *lam;
	const int *so;                           // the finest level's SELL-32 slices
	Sten sn;
	ClLevel<T> lv[kClMaxLevels];             // lv[0].val, .col: SELL-32
};

//  the system and the Krylov vectors of a run
template<class V>
struct ClSystem
{
	int n;
	const int *ptr, *so, *col;
	Sten sn;
	const V *val;
	const double *m;                         // the diagonal preconditioner (null: the V-cycle)
	double *x, *r, *rh, *p, *v, *s, *ph, *sh, *t;
	Scal *sc;
};

__device__ __forceinline__ void ClBarrier()
{
	asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct ClWho
{
	int rank, size;                          // this block in its cluster
	int gw, warps;                           // this warp in the cluster, neighbours in other blocks
};

//  sum_k val_k X(col_k) over a row, in the row's order, W entries' loads
//  issued before the first addition.  X reads a vector that other blocks write.
template<int W, class V, class XF>
__device__ __forceinline__ auto ClRowSum(int st, int len, int sd, const int *col, const V *val, XF xf) -> decltype(xf(0))
{
	using T = decltype(xf(0));
	T s = T(0);
#pragma unroll 1
	for(int k0 = 0; k0 < len; k0 += W)
	{
		int c[W];
		T v[W], x[W];
#pragma unroll
		for(int j = 0; j < W; ++j)
		{
			const bool on = k0 + j < len;
			c[j] = on ? __ldg(col + st + (k0 + j) * sd) : 0;
			v[j] = on ? (T)__ldg(val + st + (k0 + j) * sd) : T(0);
		}
#pragma unroll
		for(int j = 0; j < W; ++j)
			x[j] = k0 + j < len ? xf(c[j]) : T(0);
#pragma unroll
		for(int j = 0; j < W; ++j)
			if(k0 + j < len) s = s + v[j] * x[j];
	}
	return s;
}

//  the same over row i of the finest level (SELL-32; a stencil slice's
//  columns computed)
template<class V, class XF>
__device__ __forceinline__ auto ClRowSumFine(const Sten &sn, int i, const int *ptr, const int *so, const int *col,
                                             const V *val, XF xf) -> decltype(xf(0))
{
	using T = decltype(xf(0));
	const int st = __ldg(so + (i >> 5)) + (i & 31);
	if(sn.slice && __ldg(sn.slice + (i >> 5)))
	{
		T s = T(0);
#pragma unroll 1
		for(int k0 = 0; k0 < sn.len; k0 += kClBatch)
		{
			T v[kClBatch], x[kClBatch];
#pragma unroll
			for(int j = 0; j < kClBatch; ++j)
			{
				const bool on = k0 + j < sn.len;
				v[j] = on ? (T)__ldg(val + st + 32 * (k0 + j)) : T(0);
				x[j] = on ? xf(i + sn.off[k0 + j]) : T(0);
			}
#pragma unroll
			for(int j = 0; j < kClBatch; ++j)
				if(k0 + j < sn.len) s = s + v[j] * x[j];
		}
		return s;
	}
	return ClRowSum<kClBatch>(st, __ldg(ptr + i + 1) - __ldg(ptr + i), 32, col, val, xf);
}

//  rows of the finest level: chunk c of 256 rows belongs to block c mod size,
//  its groups of 256 threads taking the block's chunks in turn
#define YZ_CL_FINE(i, n)                                                                             \
	for(int c_ = who.rank + who.size * (int)(threadIdx.x / kRT); c_ * kRT < (n); c_ += who.size * kClGroups) \
		if(const int i = c_ * kRT + (int)(threadIdx.x % kRT); i < (n))

//  rows of a coarse level: groups of 32 rows over the cluster's warps
#define YZ_CL_ROWS(i, n)                                                          \
	for(int g_ = who.gw; g_ * 32 < (n); g_ += who.warps)                          \
		if(const int i = g_ * 32 + (int)(threadIdx.x & 31); i < (n))

//--------------------------------------------------------------------------
//  the reductions: the tree of yz_common.cuh.  A chunk's 256 values fold
//  over off = 128, 64, 32 (warp w with w+4, w+2, w+1) and then over the
//  lanes; the chunk sums go to every block's table, and once the cluster has
//  met each block folds the table the same way.
//--------------------------------------------------------------------------
struct ClRed
{
	double lanes[kClGroups][2][8][32];       // a group's values, by warp
	double fold[2][8][32];
	double part[2][2][kClMaxChunks];         // two tables in turn, up to two sums each
};

__device__ __forceinline__ double ClTree8(const double (*a)[32], int lane)
{
	return ((a[0][lane] + a[4][lane]) + (a[2][lane] + a[6][lane])) + ((a[1][lane] + a[5][lane]) + (a[3][lane] + a[7][lane]));
}

__device__ __forceinline__ double ClTreeLanes(double v)
{
#pragma unroll
	for(int off = 16; off >= 1; off >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, off);
	return v;
}

//  a group's chunk c: value a[q] of every thread (0 past the end)
template<int Q>
__device__ __forceinline__ void ClChunk(ClRed &R, const ClWho &who, int table, int c, const double (&a)[Q])
{
	const int g = threadIdx.x / kRT, w = (threadIdx.x >> 5) & 7, lane = threadIdx.x & 31;
#pragma unroll
	for(int q = 0; q < Q; ++q) R.lanes[g][q][w][lane] = a[q];
	asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "r"(kRT) : "memory");
	if(w < Q)
	{
		const double v = ClTreeLanes(ClTree8(R.lanes[g][w], lane));
		if(lane < who.size)
		{
			double *dst = cooperative_groups::this_cluster().map_shared_rank(&R.part[table][w][c], lane);
			*dst = v;
		}
	}
	asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "r"(kRT) : "memory");
}

//  after the cluster's barrier: the totals, in every thread
template<int Q>
__device__ __forceinline__ void ClTotals(ClRed &R, int table, int n, double (&tot)[Q])
{
	const int chunks = (n + kRChunk - 1) / kRChunk;
	const int t = threadIdx.x, lane = t & 31;
	const int q = t / kRT, u = t % kRT;
	if(q < Q)
	{
		double s = 0.0;
		for(int j = u; j < chunks; j += kRT) s = s + R.part[table][q][j];
		R.fold[q][u >> 5][lane] = s;
	}
	__syncthreads();
#pragma unroll
	for(int k = 0; k < Q; ++k) tot[k] = ClTreeLanes(ClTree8(R.fold[k], lane));
	__syncthreads();
}

//--------------------------------------------------------------------------
//  the V-cycle's levels below the finest, from lv[1].f (already there, and
//  the cluster past its barrier) to lv[1].x (barrier included)
//--------------------------------------------------------------------------
template<class T>
__device__ __forceinline__ void ClRestrict(const ClWho &who, int nc, const ClLevel<T> &L, const T *t, T *fc)
{
	//  four lanes a row, as KRestrict
	const int lane = threadIdx.x & 31, q = lane & 3;
	for(int g = who.gw; g * 8 < nc; g += who.warps)
	{
		const int row = g * 8 + (lane >> 2);
		T p = T(0);
		if(row < nc)
		{
			const int st = __ldg(L.rptr + row), len = __ldg(L.rptr + row + 1) - st;
			for(int k0 = q; k0 < len; k0 += 32)
			{
				T v[8], x[8];
#pragma unroll
				for(int j = 0; j < 8; ++j)
				{
					const bool on = k0 + 4 * j < len;
					v[j] = on ? __ldg(L.rval + st + k0 + 4 * j) : T(0);
					x[j] = on ? t[__ldg(L.rcol + st + k0 + 4 * j)] : T(0);
				}
#pragma unroll
				for(int j = 0; j < 8; ++j)
					if(k0 + 4 * j < len) p = p + v[j] * x[j];
			}
		}
		p = p + __shfl_down_sync(0xffffffffu, p, 1);
		p = p + __shfl_down_sync(0xffffffffu, p, 2);
		if(row < nc && q == 0) fc[row] = p;
	}
}

template<class T, class TF, class TX>
__device__ __forceinline__ void ClDense(const ClWho &who, int n, const T *inv, const TF *f, TX *x)
{
	//  a warp a row, as KDenseMV
	const int lane = threadIdx.x & 31;
	for(int i = who.gw; i < n; i += who.warps)
	{
		const T *row = inv + (size_t)i * n;
		T s = T(0);
#pragma unroll 1
		for(int j0 = lane; j0 < n; j0 += 256)
		{
			T a[8], b[8];
#pragma unroll
			for(int u = 0; u < 8; ++u)
			{
				const bool on = j0 + 32 * u < n;
				a[u] = on ? __ldg(row + j0 + 32 * u) : T(0);
				b[u] = on ? (T)f[j0 + 32 * u] : T(0);
			}
#pragma unroll
			for(int u = 0; u < 8; ++u)
				if(j0 + 32 * u < n) s = s + a[u] * b[u];
		}
#pragma unroll
		for(int off = 16; off >= 1; off >>= 1) s = s + __shfl_down_sync(0xffffffffu, s, off);
		if(lane == 0) x[i] = (TX)s;
	}
}

//  xt = m f + P xc of the next level
template<class T, class TF>
__device__ __forceinline__ T ClProlongRow(const ClLevel<T> &L, int i, const TF *f, const T *xc)
{
	const int st = __ldg(L.pptr + i), len = __ldg(L.pptr + i + 1) - st;
	const T s = ClRowSum<4>(st, len, 1, L.pcol, L.pval, [&](int c) { return xc[c]; });
	return __ldg(L.M + i) * (T)f[i] + s;
}

template<class T>
__device__ __forceinline__ void ClCoarse(const ClWho &who, const ClPlan<T> &P)
{
	int l = 1;
	for(;; ++l)
	{
		const ClLevel<T> &L = P.lv[l];
		if(L.direct) { ClDense<T, T, T>(who, L.n, L.inv, L.f, L.x); ClBarrier(); break; }
		if(L.last)
		{
			YZ_CL_ROWS(i, L.n) L.xt[i] = __ldg(L.M + i) * L.f[i];
			ClBarrier();
			YZ_CL_ROWS(i, L.n)
			{
				const int st = __ldg(L.ptr + i), len = __ldg(L.ptr + i + 1) - st;
				const T s = ClRowSum<8>(st, len, 1, L.col, L.val, [&](int c) { return L.xt[c]; });
				L.x[i] = L.xt[i] + __ldg(L.M + i) * (L.f[i] - s);
			}
			ClBarrier();
			break;
		}
		YZ_CL_ROWS(i, L.n)
		{
			const int st = __ldg(L.ptr + i), len = __ldg(L.ptr + i + 1) - st;
			const T s = ClRowSum<8>(st, len, 1, L.col, L.val, [&](int c) { return __ldg(L.M + c) * L.f[c]; });
			L.t[i] = L.f[i] - s;
		}
		ClBarrier();
		ClRestrict<T>(who, P.lv[l + 1].n, L, L.t, P.lv[l + 1].f);
		ClBarrier();
	}
	for(--l; l >= 1; --l)
	{
		const ClLevel<T> &L = P.lv[l];
		const T *xc = P.lv[l + 1].x;
		YZ_CL_ROWS(i, L.n) L.xt[i] = ClProlongRow<T, T>(L, i, L.f, xc);
		ClBarrier();
		YZ_CL_ROWS(i, L.n)
		{
			const int st = __ldg(L.ptr + i), len = __ldg(L.ptr + i + 1) - st;
			const T s = ClRowSum<8>(st, len, 1, L.col, L.val, [&](int c) { return L.xt[c]; });
			L.x[i] = L.xt[i] + __ldg(L.M + i) * (L.f[i] - s);
		}
		ClBarrier();
	}
}

//  z = V r on the finest level; the cluster past a barrier after r was
//  written; ends with one
template<class T>
__device__ __forceinline__ void ClCycle(const ClWho &who, const ClPlan<T> &P, const double *r, double *z)
{
	const ClLevel<T> &L = P.lv[0];
	const int n = L.n;
	if(L.direct) { ClDense<T, double, double>(who, n, L.inv, r, z); ClBarrier(); return; }
	if(L.last) { YZ_CL_FINE(i, n) L.xt[i] = __ldg(L.M + i) * (T)r[i]; }
	else
	{
		YZ_CL_FINE(i, n)
		{
			const T s = ClRowSumFine(P.sn, i, L.ptr, P.so, L.col, L.val, [&](int c) { return __ldg(L.M + c) * (T)r[c]; });
			L.t[i] = (T)r[i] - s;
		}
		ClBarrier();
		ClRestrict<T>(who, P.lv[1].n, L, L.t, P.lv[1].f);
		ClBarrier();
		ClCoarse<T>(who, P);
		const T *xc = P.lv[1].x;
		YZ_CL_FINE(i, n) L.xt[i] = ClProlongRow<T, double>(L, i, r, xc);
	}
	ClBarrier();
	if(std::is_same<T, double>::value || P.sweeps == 1)
	{
		YZ_CL_FINE(i, n)
		{
			const T s = ClRowSumFine(P.sn, i, L.ptr, P.so, L.col, L.val, [&](int c) { return L.xt[c]; });
			z[i] = (double)(L.xt[i] + __ldg(L.M + i) * ((T)r[i] - s));
		}
		ClBarrier();
		return;
	}
	//  the sweeps on the correction (KSweepFirst, KSweepNext): the residual in
	//  t, the correction in x and f by turns
	T *e = L.x, *eo = L.f;
	{
		const T w = (T)P.weight[0];
		YZ_CL_FINE(i, n)
		{
			const T ri = (T)r[i] - ClRowSumFine(P.sn, i, L.ptr, P.so, L.col, L.val, [&](int c) { return L.xt[c]; });
			L.t[i] = ri;
			e[i] = w * __ldg(L.M + i) * ri;
		}
		ClBarrier();
	}
	for(int k = 1; k + 1 < P.sweeps; ++k)
	{
		const T w = (T)P.weight[k];
		YZ_CL_FINE(i, n)
		{
			const T s = ClRowSumFine(P.sn, i, L.ptr, P.so, L.col, L.val, [&](int c) { return e[c]; });
			eo[i] = e[i] + w * __ldg(L.M + i) * (L.t[i] - s);
		}
		ClBarrier();
		T *u = e; e = eo; eo = u;
	}
	const T w = (T)P.weight[P.sweeps - 1];
	YZ_CL_FINE(i, n)
	{
		const T s = ClRowSumFine(P.sn, i, L.ptr, P.so, L.col, L.val, [&](int c) { return e[c]; });
		z[i] = (double)(L.xt[i] + (e[i] + w * __ldg(L.M + i) * (L.t[i] - s)));
	}
	ClBarrier();
}

template<class A> __device__ __forceinline__ void ClCopy(A &to, const A &from)
{
	static_assert(sizeof(A) % 4 == 0, "whole words");
	for(int k = threadIdx.x; k < (int)(sizeof(A) / 4); k += kClT) reinterpret_cast<int *>(&to)[k] = reinterpret_cast<const int *>(&from)[k];
}

__device__ __forceinline__ ClWho ClSelf()
{
	const auto cl = cooperative_groups::this_cluster();
	ClWho w;
	w.rank = (int)cl.block_rank();
	w.size = (int)cl.num_blocks();
	w.gw = (int)(threadIdx.x >> 5) * w.size + w.rank;
	w.warps = (kClT / 32) * w.size;
	return w;
}

//  z = M r; once in the code, not inlined: both of an iteration's calls run
//  the same instructions
template<class V, class T>
__device__ __noinline__ void ClPrec(const ClWho who, const ClPlan<T> &P, const ClSystem<V> &S, const double *r, double *z)
{
	if(S.m)
	{
		const int n = S.n;
		const double *m = S.m;
		YZ_CL_FINE(i, n) z[i] = __ldg(m + i) * r[i];
		ClBarrier();
	}
	else ClCycle<T>(who, P, r, z);
}

//--------------------------------------------------------------------------
//  A whole BiCGStab run (the loop of Solver::EnqueueIteration, step by step)
//  from the state KCtlStart left.  V: the matrix of the SpMVs; T: the
//  cycle's arithmetic.
//--------------------------------------------------------------------------
template<class V, class T>
__global__ void __launch_bounds__(kClT, 1) KLoopCluster(const __grid_constant__ ClSystem<V> S0, const __grid_constant__ ClPlan<T> P0)
{
	__shared__ ClRed R;
	//  the parameters in shared memory, where the functions not inlined reach them
	__shared__ ClSystem<V> S;
	__shared__ ClPlan<T> P;
	ClCopy(S, S0);
	ClCopy(P, P0);
	__syncthreads();
	if(P.sweeps > 1 && (int)threadIdx.x < P.sweeps) P.weight[threadIdx.x] = ChebWeight(P.lam, P.root[threadIdx.x], P.ratio);
	__syncthreads();
	const ClWho who = ClSelf();
	const int n = S.n;
	Scal *sc = S.sc;
	if(sc->state != kRun) return;            // the same word for every block, written before the launch
	const double eps = sc->eps;
	const int maxIter = sc->maxIter;
	double rho = sc->rho, res = sc->res, beta = 0.0, alpha = 0.0, omega = 0.0;
	int it = 0, state = kRun, bodies = 0;
	ClBarrier();                             // every block is running before the first remote write
	auto chunks = [&](auto body) {
		for(int c = who.rank + who.size * (int)(threadIdx.x / kRT); c * kRT < n; c += who.size * kClGroups)
			body(c, c * kRT + (int)(threadIdx.x % kRT));
	};
	double *const vx = S.x, *const vr = S.r, *const rh = S.rh, *const vp = S.p, *const vv = S.v, *const vs = S.s, *const ph = S.ph,
	              *const sh = S.sh, *const vt = S.t;
	for(;;)
	{
		++bodies;
		if(it >= maxIter) { state = kCap; break; }
		if(rho == 0.0) { state = kBreak; break; }
		YZ_CL_FINE(i, n) vp[i] = it == 0 ? vr[i] : vr[i] + beta * (vp[i] - omega * vv[i]);
		ClBarrier();
		ClPrec<V, T>(who, P, S, vp, ph);
		chunks([&](int c, int i) {
			double a[1] = {0.0};
			if(i < n)
			{
				const double s = ClRowSumFine(S.sn, i, S.ptr, S.so, S.col, S.val, [&](int q) { return ph[q]; });
				vv[i] = s;
				a[0] = 0.0 + rh[i] * s;
			}
			ClChunk<1>(R, who, 0, c, a);
		});
		ClBarrier();
		double tot1[1];
		ClTotals<1>(R, 0, n, tot1);
		alpha = rho / tot1[0];
		chunks([&](int c, int i) {
			double a[1] = {0.0};
			if(i < n)
			{
				const double si = vr[i] - alpha * vv[i];
				vs[i] = si;
				a[0] = 0.0 + si * si;
			}
			ClChunk<1>(R, who, 1, c, a);
		});
		ClBarrier();
		ClTotals<1>(R, 1, n, tot1);
		res = sqrt(tot1[0]);
		if(res <= eps)
		{
			//  converged at the half step: x takes alpha ph and the iteration counts
			YZ_CL_FINE(i, n) vx[i] = vx[i] + alpha * ph[i];
			state = kConv;
			++it;
			break;
		}
		ClPrec<V, T>(who, P, S, vs, sh);
		chunks([&](int c, int i) {
			double a[2] = {0.0, 0.0};
			if(i < n)
			{
				const double u = ClRowSumFine(S.sn, i, S.ptr, S.so, S.col, S.val, [&](int q) { return sh[q]; });
				vt[i] = u;
				a[0] = 0.0 + u * u;
				a[1] = 0.0 + u * vs[i];
			}
			ClChunk<2>(R, who, 0, c, a);
		});
		ClBarrier();
		double tot2[2];
		ClTotals<2>(R, 0, n, tot2);
		omega = tot2[1] / tot2[0];
		chunks([&](int c, int i) {
			double a[2] = {0.0, 0.0};
			if(i < n)
			{
				vx[i] = (vx[i] + alpha * ph[i]) + omega * sh[i];
				const double ri = vs[i] - omega * vt[i];
				vr[i] = ri;
				a[0] = 0.0 + ri * ri;
				a[1] = 0.0 + rh[i] * ri;
			}
			ClChunk<2>(R, who, 1, c, a);
		});
		ClBarrier();
		ClTotals<2>(R, 1, n, tot2);
		res = sqrt(tot2[0]);
		const double rhoPrev = rho;
		rho = tot2[1];
		++it;
		if(res <= eps) { state = kConv; break; }
		if(!(res == res)) { state = kNaN; break; }
		beta = (rho / rhoPrev) * (alpha / omega);
	}
	ClBarrier();                             // no block leaves while another may still write to its tables
	if(who.rank == 0 && threadIdx.x == 0)
	{
		sc->state = state; sc->it = it; sc->bodies = bodies;
		sc->res = res; sc->rho = rho; sc->alpha = alpha; sc->omega = omega;
	}
}

//  the coarse levels of a V-cycle whose finest level runs on the whole chip
template<class T>
__global__ void __launch_bounds__(kClT, 1) KCoarseCluster(const int *halt, const __grid_constant__ ClPlan<T> P)
{
	if(halt && *halt) return;
	const ClWho who = ClSelf();
	ClRestrict<T>(who, P.lv[1].n, P.lv[0], P.lv[0].t, P.lv[1].f);
	ClBarrier();
	ClCoarse<T>(who, P);
}
#undef YZ_CL_FINE
#undef YZ_CL_ROWS

} // namespace yz
