// yz_amg_kernels.cuh -- device kernels of the smoothed-aggregation AMG set-up
// and V-cycle.  Every floating-point expression follows the oracle
// (oracle/solver/yzo_solver.cpp) operation for operation; the file is compiled
// with -fmad=false so that no product is fused into an addition.
#pragma once

#include "yz_common.cuh"

namespace yz {

enum : int { kOut = 0, kUndecided = 1, kIn = 2 };

__device__ __forceinline__ uint32_t Hash32(uint32_t x)
{
	x ^= x >> 16; x *= 0x85ebca6bu;
	x ^= x >> 13; x *= 0xc2b2ae35u;
	x ^= x >> 16;
	return x;
}

__device__ __forceinline__ unsigned long long PackKey(int state, int i)
{
	return ((unsigned long long)state << 62) |
	       ((unsigned long long)(Hash32((uint32_t)i) & 0x3fffffffu) << 32) |
	       (unsigned long long)(uint32_t)i;
}

//--------------------------------------------------------------------------
//  Row access of the finest level.  Its matrix is held twice: CSR for the
//  set-up, and sliced ELLPACK (slices of 32 rows, entry k of every row of a
//  slice side by side, SELL-32) for the kernels of the iterations, whose
//  loads a warp then makes as whole lines.  A row's entries are taken in
//  the same order either way (ascending column), so every sum is the same.
//  sellOff null: CSR.
//--------------------------------------------------------------------------
__device__ __forceinline__ void RowRange(const int *__restrict__ ptr, const int *__restrict__ sellOff, int i, int &start,
                                         int &len, int &stride)
{
	len = ptr[i + 1] - ptr[i];
	if(sellOff) { start = sellOff[i >> 5] + (i & 31); stride = 32; }
	else { start = ptr[i]; stride = 1; }
}

//  sum_k val[e_k] * X(col[e_k]) over a row (e_k = st + k stride), from 0 in
//  the row's order: the loads of R entries are issued together, the last
//  ones of a row under a predicate, and the products then added one after the
//  other, so the sum is the sequential one and a row waits for two loads in
//  turn per R entries.  (With the last len mod 4 entries one by one, the
//  13-entry rows of a film's edges waited 9 times and held up their blocks:
//  the smoother of 262,144 rows 7.8 us, now 6.8.)  T is the arithmetic (the
//  type of the values): double everywhere but in the FP32 V-cycle.
//  The values may be stored narrower than the arithmetic (float values in a
//  double sum: the FP32-matrix SpMV); the arithmetic is that of X.
template<class V, class XF>
__device__ __forceinline__ auto RowSum(int st, int len, int sd, const int *__restrict__ col, const V *__restrict__ val,
                                       XF xf) -> decltype(xf(0))
{
	using T = decltype(xf(0));
	constexpr int R = 4;
	T s = T(0);
	for(int k = 0, e = st; k < len; k += R, e += R * sd)
	{
		int c[R];
		V v[R];
		T x[R];
#pragma unroll
		for(int j = 0; j < R; ++j)
		{
			const bool on = k + j < len;
			c[j] = on ? col[e + j * sd] : 0;
			v[j] = on ? val[e + j * sd] : V(0);
		}
#pragma unroll
		for(int j = 0; j < R; ++j) x[j] = k + j < len ? xf(c[j]) : T(0);
#pragma unroll
		for(int j = 0; j < R; ++j)
			if(k + j < len) s = s + (T)v[j] * x[j];
	}
	return s;
}

//  RowSum of row i of a level; a stencil row's length and offsets come from
//  the kernel's parameters (the loop is unrolled to the 16 entries a stencil
//  may have, so every offset is read by a constant index), so that its values
//  and x hang on no other read than the slice's flag and place.  The sum is
//  the same sequential one.  Four entries at a time: eight take 40 to 64
//  registers for 32 and a third of the warps, which is slower from 262,144
//  rows (the smoother at 1,048,576 rows in float 18.2 for 17.1 us).
template<class V, class XF>
__device__ __forceinline__ auto RowSumSten(const Sten &sn, int i, const int *__restrict__ ptr,
                                           const int *__restrict__ sellOff, const int *__restrict__ col,
                                           const V *__restrict__ val, XF xf) -> decltype(xf(0))
{
	using T = decltype(xf(0));
	int st, len, sd;
	RowRange(ptr, sellOff, i, st, len, sd);
	if(sn.slice)
	{
		if(sn.slice[i >> 5])
		{
			const V *__restrict__ row = val + st;
			T s = T(0);
#pragma unroll
			for(int k0 = 0; k0 < 16; k0 += 4)
			{
				if(k0 >= sn.len) break;
				V v[4];
				T xv[4];
#pragma unroll
				for(int j = 0; j < 4; ++j)
					if(k0 + j < sn.len) { v[j] = row[32 * (k0 + j)]; xv[j] = xf(i + sn.off[k0 + j]); }
#pragma unroll
				for(int j = 0; j < 4; ++j)
					if(k0 + j < sn.len) s = s + (T)v[j] * xv[j];
			}
			return s;
		}
	}
	return RowSum(st, len, sd, col, val, xf);
}

//--------------------------------------------------------------------------
//  ScaleRows + gather into the sorted mirror (LinearSolverBackend.cpp:227-252),
//  into both layouts of the finest level
//--------------------------------------------------------------------------
__global__ void KScaleGather(int n, const int *__restrict__ rowptr, const int *__restrict__ ssrc,
                             const double *__restrict__ values, const double *__restrict__ rhs, int scaling,
                             double *__restrict__ val0, double *__restrict__ b, const int *__restrict__ sellOff,
                             double *__restrict__ sellVal, float *__restrict__ sellVal32)
{
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		const int st = rowptr[i], ed = rowptr[i + 1];
		const int so = sellOff[i >> 5] + (i & 31);
		const double d = scaling ? values[st] : 1.0;
		if(!scaling || fabs(d) < 1.0e-30)
		{
			for(int k = st; k < ed; ++k)
			{
				const double v = values[ssrc[k]];
				val0[k] = v;
				sellVal[so + 32 * (k - st)] = v;
				if(sellVal32) sellVal32[so + 32 * (k - st)] = (float)v;
			}
			b[i] = rhs[i];
			continue;
		}
		const double inv = 1.0 / d;
		for(int k = st; k < ed; ++k)
		{
			const double v = values[ssrc[k]] * inv;
			val0[k] = v;
			sellVal[so + 32 * (k - st)] = v;
			if(sellVal32) sellVal32[so + 32 * (k - st)] = (float)v;
		}
		b[i] = rhs[i] * inv;
	}
}

//--------------------------------------------------------------------------
//  strength of connection, aggregation
//--------------------------------------------------------------------------
__global__ void KDiag(int n, const int *__restrict__ ptr, const int *__restrict__ col,
                      const double *__restrict__ val, double *__restrict__ dia)
{
	PdlEntry();
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		double d = 0.0;
		for(int k = ptr[i]; k < ptr[i + 1]; ++k) if(col[k] == i) { d = val[k]; break; }
		dia[i] = d;
	}
}

//  strong[k]: entry k of A is a strong connection; cnt: of every row, its
//  strong connections either way (a row that both holds and is held counts
//  twice: every use of the lists is a max or a min over them)
__global__ void KStrength(int n, const int *__restrict__ ptr, const int *__restrict__ col,
                          const double *__restrict__ val, const double *__restrict__ dia, double eps2,
                          unsigned char *__restrict__ strong, int *__restrict__ cnt)
{
	PdlEntry();
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		const double e = eps2 * dia[i];
		int out = 0;
		for(int k = ptr[i]; k < ptr[i + 1]; ++k)
		{
			const int c = col[k];
			const double v = val[k];
			const bool s = (c != i) && (e * dia[c] < v * v);
			strong[k] = s ? 1 : 0;
			if(s) { ++out; atomicAdd(&cnt[c], 1); }
		}
		if(out) atomicAdd(&cnt[i], out);
	}
}

//  the strong neighbours of every row, held and holding, in one list (in any
//  order): the rounds and the aggregation then read one list instead of
//  scanning a row's flags beside a second one
__global__ void KFillIn(int n, const int *__restrict__ ptr, const int *__restrict__ col,
                        const unsigned char *__restrict__ strong, int *__restrict__ fill, int *__restrict__ nbr)
{
	PdlEntry();
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		int out = 0;
		for(int k = ptr[i]; k < ptr[i + 1]; ++k)
			if(strong[k]) { ++out; nbr[atomicAdd(&fill[col[k]], 1)] = i; }
		if(!out) continue;
		int at = atomicAdd(&fill[i], out);
		for(int k = ptr[i]; k < ptr[i + 1]; ++k)
			if(strong[k]) nbr[at++] = col[k];
	}
}

//  The rounds of the distance-2 independent set.  Round r reads the count of
//  undecided rows u[r & 1] (0: the set is complete, the round does nothing):
//  KMisMax takes the largest key next to each row and zeroes u[(r + 1) & 1],
//  KMisUpdate the largest within distance 2, decides the row, writes its key of
//  the next round and counts the rows still undecided into u[(r + 1) & 1].
__global__ void KMisInit(int n, const int *__restrict__ nptr, int *__restrict__ state, unsigned char *__restrict__ iso,
                         unsigned long long *__restrict__ T0, int *__restrict__ undecided)
{
	PdlEntry();
	int cnt = 0;
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		const bool any = nptr[i + 1] > nptr[i];
		iso[i] = any ? 0 : 1;
		state[i] = any ? kUndecided : kOut;
		T0[i] = PackKey(any ? kUndecided : kOut, i);
		cnt += any;
	}
	for(int off = 16; off >= 1; off >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, off);
	if((threadIdx.x & 31) == 0 && cnt) atomicAdd(undecided, cnt);
}

__device__ __forceinline__ unsigned long long MisMaxRow(int i, const int *__restrict__ nptr, const int *__restrict__ nbr,
                                                        const unsigned long long *__restrict__ T)
{
	unsigned long long m = T[i];
	const int ed = nptr[i + 1];
	for(int k = nptr[i]; k < ed; k += 4)
	{
		unsigned long long u[4];
#pragma unroll
		for(int j = 0; j < 4; ++j) u[j] = k + j < ed ? T[nbr[k + j]] : 0ull;
#pragma unroll
		for(int j = 0; j < 4; ++j) m = u[j] > m ? u[j] : m;
	}
	return m;
}

__global__ void KMisMax(int n, const int *__restrict__ nptr, const int *__restrict__ nbr,
                        const unsigned long long *__restrict__ Tin, unsigned long long *__restrict__ Tout,
                        const int *__restrict__ undecided, int *zero)
{
	PdlEntry();
	if(blockIdx.x == 0 && threadIdx.x == 0) *zero = 0;
	if(*undecided == 0) return;
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
		Tout[i] = MisMaxRow(i, nptr, nbr, Tin);
}

__global__ void KMisUpdate(int n, const int *__restrict__ nptr, const int *__restrict__ nbr,
                           const unsigned long long *__restrict__ T1, int *__restrict__ state,
                           unsigned long long *__restrict__ T0, const int *__restrict__ undecided, int *__restrict__ next)
{
	PdlEntry();
	if(*undecided == 0) return;
	int cnt = 0;
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		int st = state[i];
		if(st == kUndecided)
		{
			const unsigned long long t = MisMaxRow(i, nptr, nbr, T1);
			if((int)(uint32_t)(t & 0xffffffffull) == i) st = kIn;
			else if((int)(t >> 62) == kIn) st = kOut;
			if(st != kUndecided) { state[i] = st; T0[i] = PackKey(st, i); }
		}
		cnt += (st == kUndecided);
	}
	for(int off = 16; off >= 1; off >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, off);
	if((threadIdx.x & 31) == 0 && cnt) atomicAdd(next, cnt);
}

__global__ void KRootFlags(int n, const int *__restrict__ state, int *__restrict__ flag)
{
	PdlEntry();
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) flag[i] = state[i] == kIn ? 1 : 0;
}

__global__ void KAssignFirst(int n, const int *__restrict__ nptr, const int *__restrict__ nbr,
                             const int *__restrict__ state, const unsigned char *__restrict__ iso,
                             const int *__restrict__ rootId, int *__restrict__ first)
{
	PdlEntry();
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		if(state[i] == kIn) { first[i] = rootId[i]; continue; }
		if(iso[i]) { first[i] = -1; continue; }
		int best = -1;
		for(int k = nptr[i]; k < nptr[i + 1]; ++k)
		{ const int j = nbr[k]; if(state[j] == kIn && (best < 0 || rootId[j] < best)) best = rootId[j]; }
		first[i] = best;
	}
}

__global__ void KAssignSecond(int n, const int *__restrict__ nptr, const int *__restrict__ nbr,
                              const unsigned char *__restrict__ iso, const int *__restrict__ first, int *__restrict__ agg)
{
	PdlEntry();
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		if(first[i] >= 0 || iso[i]) { agg[i] = first[i]; continue; }
		int best = -1;
		for(int k = nptr[i]; k < nptr[i + 1]; ++k)
		{ const int f = first[nbr[k]]; if(f >= 0 && (best < 0 || f < best)) best = f; }
		agg[i] = best;
	}
}

//  M32: the float copy for the FP32 cycle (null: none).  lam (null: not
//  wanted): by their bits, lam[0] the largest |m_i| sum_j |a_ij|, a bound of
//  the spectral radius of M A, and lam[1] the least m_i sum_j a_ij (0 if
//  negative) of the rows that are not a ghost's two entries -- the value
//  of M A on the constant, the bottom of its spectrum where A is the identity
//  plus a difference operator; lam[0] zero, lam[1] all ones before
__global__ void KSpai0(int n, const int *__restrict__ ptr, const int *__restrict__ col,
                       const double *__restrict__ val, double *__restrict__ M, float *__restrict__ M32,
                       unsigned long long *lam)
{
	PdlEntry();
	unsigned long long most = 0, least = ~0ull;
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		const int st = ptr[i], ed = ptr[i + 1];
		double num = 0.0, den = 0.0, sum = 0.0, all = 0.0;
		for(int k = st; k < ed; ++k)
		{
			const double v = val[k];
			den = den + v * v;
			if(col[k] == i) num = num + v;
			sum = sum + fabs(v);
			all = all + v;
		}
		const double m = (1.0 / den) * num;
		M[i] = m;
		if(M32) M32[i] = (float)m;
		const unsigned long long b = (unsigned long long)__double_as_longlong(fabs(m * sum));
		most = b > most ? b : most;
		const unsigned long long a = (unsigned long long)__double_as_longlong(m * all > 0.0 ? m * all : 0.0);
		if(ed - st > 2) least = a < least ? a : least;
	}
	if(!lam) return;
	for(int off = 16; off >= 1; off >>= 1)
	{
		const unsigned long long u = __shfl_down_sync(0xffffffffu, most, off), d = __shfl_down_sync(0xffffffffu, least, off);
		most = u > most ? u : most;
		least = d < least ? d : least;
	}
	if((threadIdx.x & 31) == 0) { atomicMax(lam, most); atomicMin(lam + 1, least); }
}

//  The weight of a Chebyshev step on [max(lo, hi / r), hi]: ck the cosine of
//  the step's root, ir = 1 / r.  lam[2] not 0: the hierarchy takes sweeps of
//  weight 1 (KProbeChoose).
__device__ __forceinline__ double ChebWeight(const double *lam, double ck, double ir)
{
	//  the three read at once: a sweep of a small level waits for them
	const double hi = lam[0], lo0 = lam[1], plain = lam[2];
	double lo = hi * ir;
	if(lo0 > lo && lo0 < hi) lo = lo0;
	const double w = 1.0 / (0.5 * ((hi + lo) - (hi - lo) * ck));
	return plain != 0.0 ? 1.0 : w;
}

//  damped Jacobi as a preconditioner: m_i = 0.72 * (1 / a_ii)
__global__ void KDampedJacobi(int n, const double *__restrict__ dia, double *__restrict__ M)
{
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) M[i] = 0.72 * (1.0 / dia[i]);
}

//--------------------------------------------------------------------------
//  prolongation  P = (I - omega D_f^-1 A_f) P_tent
//--------------------------------------------------------------------------
constexpr int kRowCap = 256;	// distinct aggregates / columns a row may gather

//  CAP: the distinct aggregates a row may gather in this launch (a row of A
//  with more entries than CAP sets *overflow; the caller then launches the
//  kRowCap instance)
template<int CAP>
__global__ void KPCount(int n, const int *__restrict__ ptr, const int *__restrict__ col,
                        const unsigned char *__restrict__ strong, const int *__restrict__ agg,
                        int *__restrict__ cnt, int *__restrict__ overflow)
{
	PdlEntry();
	int lc[CAP];
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		int m = 0;
		for(int k = ptr[i]; k < ptr[i + 1]; ++k)
		{
			const int c = col[k];
			if(c != i && !strong[k]) continue;
			const int cp = agg[c];
			if(cp < 0) continue;
			int q = 0;
			while(q < m && lc[q] != cp) ++q;
			if(q == m) { if(m == CAP) { atomicExch(overflow, 1); break; } lc[m++] = cp; }
		}
		cnt[i] = m;
	}
}

template<int CAP>
__global__ void KPFill(int n, const int *__restrict__ ptr, const int *__restrict__ col,
                       const double *__restrict__ val, const unsigned char *__restrict__ strong,
                       const int *__restrict__ agg, const int *__restrict__ pptr,
                       int *__restrict__ pcol, double *__restrict__ pval)
{
	PdlEntry();
	const double omega = 2.0 / 3.0;
	int lc[CAP];
	double lv[CAP];
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		double dia = 0.0;
		for(int k = ptr[i]; k < ptr[i + 1]; ++k)
			if(col[k] == i || !strong[k]) dia = dia + val[k];
		const double ds = (-omega) * (1.0 / dia);
		int m = 0;
		for(int k = ptr[i]; k < ptr[i + 1]; ++k)
		{
			const int c = col[k];
			if(c != i && !strong[k]) continue;
			const int cp = agg[c];
			if(cp < 0) continue;
			const double va = (c == i) ? (1.0 - omega) : ds * val[k];
			int q = 0;
			while(q < m && lc[q] != cp) ++q;
			if(q == m) { if(m == CAP) break; lc[m] = cp; lv[m] = 0.0; ++m; }
			lv[q] = lv[q] + va;
		}
		//  insertion sort by column (columns are distinct)
		for(int a = 1; a < m; ++a)
		{
			const int kc = lc[a]; const double kv = lv[a];
			int b = a - 1;
			while(b >= 0 && lc[b] > kc) { lc[b + 1] = lc[b]; lv[b + 1] = lv[b]; --b; }
			lc[b + 1] = kc; lv[b + 1] = kv;
		}
		const int o = pptr[i];
		for(int q = 0; q < m; ++q) { pcol[o + q] = lc[q]; pval[o + q] = lv[q]; }
	}
}

//  R = P^T: counts per column, atomic fill, then each row sorted by fine row
__global__ void KColCount(const int *__restrict__ total, const int *__restrict__ pcol, int *__restrict__ cnt)
{
	PdlEntry();
	const int nnz = *total;
	for(int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += gridDim.x * blockDim.x) atomicAdd(&cnt[pcol[k]], 1);
}

__global__ void KTransposeFill(int n, const int *__restrict__ pptr, const int *__restrict__ pcol,
                               const double *__restrict__ pval, int *__restrict__ fill,
                               int *__restrict__ rcol, double *__restrict__ rval)
{
	PdlEntry();
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
		for(int k = pptr[i]; k < pptr[i + 1]; ++k)
		{
			const int d = atomicAdd(&fill[pcol[k]], 1);
			rcol[d] = i; rval[d] = pval[k];
		}
}

//  each row sorted by column (the columns of a row are distinct): one warp
//  per row, every entry placed at its rank among the row's columns (rows of
//  up to 64 entries), longer rows by insertion in place
__global__ void __launch_bounds__(256) KRowSort(int n, const int *__restrict__ ptr, int *__restrict__ col,
                                                double *__restrict__ val)
{
	PdlEntry();
	constexpr int L = 64, W = 8;
	__shared__ int sc[W][L];
	__shared__ double sv[W][L];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
	for(long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < n; row += warps)
	{
		const int i = (int)row;
		const int st = ptr[i], ed = ptr[i + 1], m = ed - st;
		if(m <= L)
		{
			for(int a2 = lane; a2 < m; a2 += 32) { sc[w][a2] = col[st + a2]; sv[w][a2] = val[st + a2]; }
			__syncwarp();
			for(int a2 = lane; a2 < m; a2 += 32)
			{
				const int cc = sc[w][a2];
				int r = 0;
				for(int b2 = 0; b2 < m; ++b2) r += (sc[w][b2] < cc);
				col[st + r] = cc; val[st + r] = sv[w][a2];
			}
			__syncwarp();
			continue;
		}
		if(lane != 0) continue;
		for(int a2 = st + 1; a2 < ed; ++a2)
		{
			const int kc = col[a2]; const double kv = val[a2];
			int b2 = a2 - 1;
			while(b2 >= st && col[b2] > kc) { col[b2 + 1] = col[b2]; val[b2 + 1] = val[b2]; --b2; }
			col[b2 + 1] = kc; val[b2 + 1] = kv;
		}
	}
}

//--------------------------------------------------------------------------
//  sparse product C = X Y with the oracle's summation order: per output
//  entry from 0.0, contributions in the order of X's row (ascending k)
//--------------------------------------------------------------------------
//  CAP bounds the distinct columns of one output row held in registers /
//  local memory; a row beyond it sets *overflow (the caller then runs the
//  product again with the larger capacity).
template<int CAP>
__global__ void KGemmCount(int nx, const int *__restrict__ xptr, const int *__restrict__ xcol,
                           const int *__restrict__ yptr, const int *__restrict__ ycol,
                           int *__restrict__ cnt, int *__restrict__ overflow)
{
	int lc[CAP];
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < nx; i += gridDim.x * blockDim.x)
	{
		int m = 0;
		bool over = false;
		for(int kx = xptr[i]; kx < xptr[i + 1] && !over; ++kx)
		{
			const int k = xcol[kx];
			for(int ky = yptr[k]; ky < yptr[k + 1]; ++ky)
			{
				const int j = ycol[ky];
				int lo = 0, hi = m;
				while(lo < hi) { const int mid = (lo + hi) >> 1; if(lc[mid] < j) lo = mid + 1; else hi = mid; }
				if(lo < m && lc[lo] == j) continue;
				if(m == CAP) { over = true; break; }
				for(int q = m; q > lo; --q) lc[q] = lc[q - 1];
				lc[lo] = j; ++m;
			}
		}
		if(over) atomicExch(overflow, 1);
		cnt[i] = m;
	}
}

template<int CAP>
__global__ void KGemmFill(int nx, const int *__restrict__ xptr, const int *__restrict__ xcol,
                          const double *__restrict__ xval, const int *__restrict__ yptr,
                          const int *__restrict__ ycol, const double *__restrict__ yval,
                          const int *__restrict__ cptr, int *__restrict__ ccol, double *__restrict__ cval)
{
	int lc[CAP];
	double lv[CAP];
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < nx; i += gridDim.x * blockDim.x)
	{
		int m = 0;
		for(int kx = xptr[i]; kx < xptr[i + 1]; ++kx)
		{
			const int k = xcol[kx];
			const double xv = xval[kx];
			for(int ky = yptr[k]; ky < yptr[k + 1]; ++ky)
			{
				const int j = ycol[ky];
				int lo = 0, hi = m;
				while(lo < hi) { const int mid = (lo + hi) >> 1; if(lc[mid] < j) lo = mid + 1; else hi = mid; }
				if(!(lo < m && lc[lo] == j))
				{
					if(m == CAP) continue;
					for(int q = m; q > lo; --q) { lc[q] = lc[q - 1]; lv[q] = lv[q - 1]; }
					lc[lo] = j; lv[lo] = 0.0; ++m;
				}
				lv[lo] = lv[lo] + xv * yval[ky];
			}
		}
		const int o = cptr[i];
		for(int q = 0; q < m; ++q) { ccol[o + q] = lc[q]; cval[o + q] = lv[q]; }
	}
}

//--------------------------------------------------------------------------
//  The same product with L lanes per output row and at most kGemmCap
//  distinct columns a row, staged: row i at i kGemmCap, sorted by column, with
//  its count in cnt[i] (KGemmCompact moves the rows once the counts are
//  scanned); a row beyond the cap sets *overflow and leaves 0.  ystage: Y's
//  rows are staged so too, row k with yptr[k] entries.
//
//  Bound by latency: a film's row takes 13 short Y rows one after the other,
//  for every sum gets its contributions in X's row order from 0.0, as the
//  thread-per-row kernels and the oracle give them (a Y row holds a column
//  once, so the lanes of one step never add into the same sum).  So four Y
//  rows are read at once ahead of their sums, and a column's sum is found by a
//  hash table of 128 places in shared memory (64 columns and one Y row's 32
//  more always leave it a free place) rather than by a walk over the columns
//  so far.  The rows of P hold 3 entries on average, so A P gives a row 8
//  lanes (with 32, instructions for idle lanes bound it); the rows of A P hold
//  20 to 25, so R (A P) gives 32.  The 18 products of a 512 x 512 step with
//  rows walked one by one 72 us on average, now 37; 224 x 224 44 and 24.
//--------------------------------------------------------------------------
constexpr int kGemmCap = 64, kGemmTab = 128, kGemmThreads = 128;

//  one entry a lane (j < 0: none) into the lanes' row's table; returns the
//  columns that are new to it (gm: the lanes of the row)
__device__ __forceinline__ int GemmAdd(int *tcol, double *tval, unsigned gm, int j, double p)
{
	bool fresh = false;
	if(j >= 0)
	{
		unsigned h = ((unsigned)j * 2654435761u) >> 25;
		for(;;)
		{
			int have = *(volatile int *)(tcol + h);
			if(have == -1) have = atomicCAS(tcol + h, -1, j);
			if(have == -1) { fresh = true; break; }
			if(have == j) break;
			h = (h + 1) & (kGemmTab - 1);
		}
		tval[h] = (fresh ? 0.0 : tval[h]) + p;
	}
	return __popc(__ballot_sync(0xffffffffu, fresh) & gm);
}

template<int L>
__global__ void __launch_bounds__(kGemmThreads) KGemmWarp(int nx, const int *__restrict__ xptr, const int *__restrict__ xcol,
                                                          const double *__restrict__ xval, const int *__restrict__ yptr,
                                                          const int *__restrict__ ycol, const double *__restrict__ yval,
                                                          int *__restrict__ cnt, int *__restrict__ ccol,
                                                          double *__restrict__ cval, int *__restrict__ overflow, bool ystage)
{
	PdlEntry();
	constexpr int G = kGemmThreads / L, B = 4;
	constexpr unsigned all = 0xffffffffu;
	__shared__ __align__(16) int scol[G][kGemmTab];
	__shared__ double sval[G][kGemmTab];
	const int lane = threadIdx.x & 31, l = lane & (L - 1), w = threadIdx.x / L;
	const unsigned gm = (L == 32 ? all : ((1u << (L & 31)) - 1u)) << (lane & ~(L - 1));
	const unsigned lt = gm & ((1u << lane) - 1u);
	int *tc = scol[w];
	double *tv = sval[w];
	//  every loop's bounds are the warp's, so that its rows keep together
	const long long rows = (long long)gridDim.x * G;
	for(long long r0 = (long long)blockIdx.x * G + (threadIdx.x >> 5) * (32 / L); r0 < nx; r0 += rows)
	{
		const long long i = r0 + (lane / L);
		const bool live = i < nx;
		const int xs = live ? xptr[i] : 0, xe = live ? xptr[i + 1] : 0;
		const int xl = __reduce_max_sync(all, xe - xs);
		int m = 0;
#pragma unroll
		for(int q = 4 * l; q < kGemmTab; q += 4 * L) *reinterpret_cast<int4 *>(tc + q) = make_int4(-1, -1, -1, -1);
		__syncwarp();
		//  X's row L entries at a time: each lane loads one entry and its Y
		//  row's bounds, which the row's lanes then take in order by shuffles
		for(int xo = 0; xo < xl; xo += L)
		{
			const int xk = xs + xo + l;
			const bool av = xk < xe;
			const int kk = av ? xcol[xk] : 0;
			const double xvv = av ? xval[xk] : 0.0;
			const int ys = !av ? 0 : ystage ? kk : yptr[kk], yl = !av ? 0 : ystage ? yptr[kk] : yptr[kk + 1] - ys;
			const int cntx = min(L, xl - xo);
			for(int j0 = 0; j0 < cntx; j0 += B)
			{
				int c[B], len[B];
				double v[B];
#pragma unroll
				for(int u = 0; u < B; ++u)
				{
					const int yr = __shfl_sync(all, ys, j0 + u, L);
					len[u] = __shfl_sync(all, yl, j0 + u, L);
					const long long y0 = ystage ? (long long)yr * kGemmCap : (long long)yr;
					const bool on = l < len[u];		// past the row's end: 0
					c[u] = on ? ycol[y0 + l] : -1;
					v[u] = on ? yval[y0 + l] : 0.0;
				}
#pragma unroll
				for(int u = 0; u < B; ++u)
				{
					const double xv = __shfl_sync(all, xvv, j0 + u, L);
					m += GemmAdd(tc, tv, gm, m <= kGemmCap ? c[u] : -1, xv * v[u]);
					__syncwarp();
					if(!__any_sync(all, len[u] > L)) continue;
					const int yr = __shfl_sync(all, ys, j0 + u, L), most = __reduce_max_sync(all, len[u]);
					const long long y0 = (ystage ? (long long)yr * kGemmCap : (long long)yr) + l;
					for(int k0 = L; k0 < most; k0 += L)
					{
						const bool on = k0 + l < len[u] && m <= kGemmCap;
						m += GemmAdd(tc, tv, gm, on ? ycol[y0 + k0] : -1, on ? xv * yval[y0 + k0] : 0.0);
						__syncwarp();
					}
				}
			}
		}
		const bool over = m > kGemmCap;
		if(live && l == 0)
		{
			if(over) { atomicExch(overflow, 1); cnt[i] = 0; }
			else cnt[i] = m;
		}
		if(over) m = 0;
		//  the row's entries together at the front of its table (an entry
		//  never moves up), then each at its rank among the columns
		int at = 0;
		for(int q = 0; q < kGemmTab; q += L)
		{
			const int c = tc[q + l];
			const double v = tv[q + l];
			const unsigned mask = __ballot_sync(all, c >= 0);
			__syncwarp();		// a lane's place may be where another has just read
			if(c >= 0) { const int to = at + __popc(mask & lt); tc[to] = c; tv[to] = v; }
			at += __popc(mask & gm);
			__syncwarp();
		}
		const int mw = __reduce_max_sync(all, m);
		for(int q = l; q < mw; q += L)
		{
			const int c = tc[q];
			int r = 0;
			for(int t = 0; t < m; ++t) r += tc[t] < c;
			if(q < m) { ccol[i * kGemmCap + r] = c; cval[i * kGemmCap + r] = tv[q]; }
		}
		__syncwarp();
	}
}

template<int CAP>
__global__ void KGemmCompact(int nx, const int *__restrict__ cptr, const int *__restrict__ tcol,
                             const double *__restrict__ tval, int *__restrict__ ccol, double *__restrict__ cval)
{
	PdlEntry();
	for(long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < (long long)nx * CAP;
	    e += (long long)gridDim.x * blockDim.x)
	{
		const int i = (int)(e / CAP), r = (int)(e % CAP);
		const int o = cptr[i];
		if(r < cptr[i + 1] - o) { ccol[o + r] = tcol[e]; cval[o + r] = tval[e]; }
	}
}

//--------------------------------------------------------------------------
//  V-cycle.  Every kernel of the solve's iteration takes halt, the state
//  word of its BiCGStab run (non-zero once it has stopped), and does nothing
//  when it is set: the iterations are queued ahead of the host's check.
//--------------------------------------------------------------------------
//  The kernels of the cycle are written for the arithmetic T of the cycle's
//  matrices and vectors (double; float in the FP32 V-cycle, whose matrices
//  are the FP64 set-up's rounded to float).  The right-hand side f of the
//  finest level and the result x written there are the Krylov vectors, of
//  type TF and TX: each value is converted to T where it is read and the
//  result to TX where it is written.  With T = TF = TX = double every
//  conversion is the identity and the arithmetic the oracle's.
//--------------------------------------------------------------------------
//  x = m .* f, t = f - A x (x of the neighbours recomputed as m_j * f_j)
template<class T, class TF, class TX>
__global__ void KPreSmoothResidual(const int *__restrict__ halt, int n, const int *__restrict__ ptr,
                                   const int *__restrict__ sellOff, const __grid_constant__ Sten sn, const int *__restrict__ col,
                                   const T *__restrict__ val, const T *__restrict__ M, const TF *__restrict__ f,
                                   TX *__restrict__ x, T *__restrict__ t)
{
	PdlEntry();
	if(halt && *halt) return;
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if(i < n)
	{
		const T s = RowSumSten(sn, i, ptr, sellOff, col, val, [&](int c) { return M[c] * (T)f[c]; });
		const T fi = (T)f[i];
		x[i] = (TX)(M[i] * fi);
		t[i] = fi - s;
	}
}

template<class T, class TF, class TX>
__global__ void KPreSmooth(const int *__restrict__ halt, int n, const T *__restrict__ M, const TF *__restrict__ f,
                           TX *__restrict__ x)
{
	PdlEntry();
	if(halt && *halt) return;
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) x[i] = (TX)(M[i] * (T)f[i]);
}

//  y = A x (from 0.0, stored order)
__global__ void KSpmv(const int *__restrict__ halt, int n, const int *__restrict__ ptr, const int *__restrict__ col,
                      const double *__restrict__ val, const double *__restrict__ x, double *__restrict__ y)
{
	if(halt && *halt) return;
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
		y[i] = RowSum(ptr[i], ptr[i + 1] - ptr[i], 1, col, val, [&](int c) { return x[c]; });
}

//  f_c = R t with four lanes per row: lane q sums the row's entries q, q+4,
//  ... from 0.0 and the four partials are folded (p0 + p1) + (p2 + p3) --
//  the oracle's Restrict -- so that the long rows of R (an aggregate and its
//  neighbours) are taken four entries at a time; eight rows a warp, the
//  loop alike for all its lanes
template<class T>
__global__ void KRestrict(const int *__restrict__ halt, int n, const int *__restrict__ ptr, const int *__restrict__ col,
                          const T *__restrict__ val, const T *__restrict__ t, T *__restrict__ y)
{
	PdlEntry();
	if(halt && *halt) return;
	const int lane = threadIdx.x & 31, q = lane & 3;
	const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
	for(long long base = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 8; base < n; base += warps * 8)
	{
		const long long row = base + (lane >> 2);
		const bool active = row < n;
		T p = T(0);
		if(active)
		{
			const int st = ptr[row], len = ptr[row + 1] - st;
			for(int k = q; k < len; k += 4) p = p + val[st + k] * t[col[st + k]];
		}
		p = p + __shfl_down_sync(0xffffffffu, p, 1);
		p = p + __shfl_down_sync(0xffffffffu, p, 2);
		if(active && q == 0) y[row] = p;
	}
}

//  xout = x + P xc
template<class T>
__global__ void KProlong(const int *__restrict__ halt, int n, const int *__restrict__ pptr, const int *__restrict__ pcol,
                         const T *__restrict__ pval, const T *__restrict__ xc, const T *__restrict__ x,
                         T *__restrict__ xout)
{
	PdlEntry();
	if(halt && *halt) return;
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		const T s = RowSum(pptr[i], pptr[i + 1] - pptr[i], 1, pcol, pval, [&](int c) { return xc[c]; });
		xout[i] = x[i] + s;
	}
}

//  xout = x + m .* (f - A x)
template<class T, class TF, class TX>
__global__ void KPostSmooth(const int *__restrict__ halt, int n, const int *__restrict__ ptr,
                            const int *__restrict__ sellOff, const __grid_constant__ Sten sn, const int *__restrict__ col,
                            const T *__restrict__ val, const T *__restrict__ M, const TF *__restrict__ f,
                            const T *__restrict__ x, TX *__restrict__ xout)
{
	PdlEntry();
	if(halt && *halt) return;
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if(i < n)
	{
		const T fi = (T)f[i], xi = x[i], mi = M[i];
		const T s = RowSumSten(sn, i, ptr, sellOff, col, val, [&](int c) { return x[c]; });
		xout[i] = (TX)(xi + mi * (fi - s));
	}
}

//  The finest level's sweeps of the FP32 cycle, on the correction: the
//  residual r = f - A x once, then e = w m r (KSweepFirst), e = e + w m (r -
//  A e) (KSweepNext), and x + e at the last (KSweepLast); w a step of the
//  Chebyshev iteration on the bounds KSpai0 left, or 1 (ChebWeight).  On x
//  itself every sweep rounds A x, which is small against x's smooth part, and
//  a step's weight is up to 9 times a plain sweep's.  (BiCGStab iterations a
//  step of the 256^2 ConcZ film, the same order of the weights: 715 and 716 on
//  x, 650 and 641 so; Solver::SweepRoot has the order's part.)
template<class T, class TF>
__global__ void KSweepFirst(const int *__restrict__ halt, int n, const int *__restrict__ ptr,
                            const int *__restrict__ sellOff, const __grid_constant__ Sten sn, const int *__restrict__ col,
                            const T *__restrict__ val, const T *__restrict__ M, const TF *__restrict__ f,
                            const T *__restrict__ x, T *__restrict__ r, T *__restrict__ e, const double *__restrict__ lam,
                            double ck, double ir)
{
	PdlEntry();
	if(halt && *halt) return;
	const T w = (T)ChebWeight(lam, ck, ir);
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if(i < n)
	{
		const T fi = (T)f[i], mi = M[i];
		const T ri = fi - RowSumSten(sn, i, ptr, sellOff, col, val, [&](int c) { return x[c]; });
		r[i] = ri;
		e[i] = w * mi * ri;
	}
}

template<class T, class TX, bool Last>
__global__ void KSweepNext(const int *__restrict__ halt, int n, const int *__restrict__ ptr,
                           const int *__restrict__ sellOff, const __grid_constant__ Sten sn, const int *__restrict__ col,
                           const T *__restrict__ val, const T *__restrict__ M, const T *__restrict__ r,
                           const T *__restrict__ e, const T *__restrict__ x, TX *__restrict__ out, const double *__restrict__ lam,
                           double ck, double ir)
{
	PdlEntry();
	if(halt && *halt) return;
	const T w = (T)ChebWeight(lam, ck, ir);
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if(i < n)
	{
		const T ri = r[i], ei = e[i], mi = M[i], xi = Last ? x[i] : T(0);
		const T s = RowSumSten(sn, i, ptr, sellOff, col, val, [&](int c) { return e[c]; });
		const T en = ei + w * mi * (ri - s);
		out[i] = (TX)(Last ? xi + en : en);
	}
}

//--------------------------------------------------------------------------
//  Which sweeps a hierarchy takes.  The Chebyshev weights are made for a real
//  spectrum; where advection gives M A eigenvalues with imaginary parts near
//  half of its bound they amplify what sweeps of weight 1 damp.  Neither the
//  bounds nor the entries tell (a film's rows are as unsymmetric where its
//  mobility changes), so both are tried on noise at every set-up: the error
//  after two rounds of either, x - w M A x, and the set that leaves less of it
//  is taken.  Restated in 64 bits on 67 systems (films of every kind, upwind
//  advection of Courant number 0.2 to 30 with and without a fourth-order term,
//  all over or in 0.3 to 30 % of the area) the set so chosen took at most two
//  BiCGStab iterations more than the other, and up to 250 fewer; one round of
//  sweeps missed advection in 1 % of the area.
//
//  Both errors go side by side (x: Chebyshev, y: weight 1), so that 16 sweeps
//  read the matrix 16 times and not 32: a 640^2 step of four set-ups took 75 us
//  a set-up more with a row sum each, 17 with one of pairs.
//--------------------------------------------------------------------------
struct __align__(8) ProbePair
{
	float x, y;
	ProbePair() = default;
	__device__ __forceinline__ explicit ProbePair(float a) : x(a), y(a) {}
	__device__ __forceinline__ ProbePair(float a, float b) : x(a), y(b) {}
};
__device__ __forceinline__ ProbePair operator*(ProbePair a, ProbePair b) { return ProbePair(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ ProbePair operator+(ProbePair a, ProbePair b) { return ProbePair(a.x + b.x, a.y + b.y); }

__global__ void KProbeStart(int n, ProbePair *__restrict__ x, double *lam)
{
	if(blockIdx.x == 0 && threadIdx.x == 0) lam[2] = 0.0;
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		unsigned u = (unsigned)i * 2654435761u;
		u = (u ^ (u >> 15)) * 2246822519u;
		u = (u ^ (u >> 13)) * 3266489917u;
		u ^= u >> 16;
		const float v = (float)(int)(u >> 8) * (1.0f / 8388608.0f) - 1.0f;
		x[i] = ProbePair(v);
	}
}

__global__ void KProbeSweep(int n, const int *__restrict__ ptr, const int *__restrict__ sellOff,
                            const __grid_constant__ Sten sn, const int *__restrict__ col, const float *__restrict__ val,
                            const float *__restrict__ M, const ProbePair *__restrict__ x, ProbePair *__restrict__ xout,
                            const double *__restrict__ lam, double ck, double ir)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if(i >= n) return;
	const float w = (float)ChebWeight(lam, ck, ir);
	const ProbePair s = RowSumSten(sn, i, ptr, sellOff, col, val, [&](int c) { return x[c]; }), xi = x[i];
	const float m = M[i];
	xout[i] = ProbePair(xi.x - w * m * s.x, xi.y - m * s.y);
}

//  What is left of either; a sum that is not finite counts as more than one
//  that is.  Chebyshev sweeps that leave less than a fiftieth of the noise (its
//  square n / 3) are good whatever the others leave: on a well conditioned
//  system both leave 1e-5, a hair's breadth apart, and a hierarchy kept from one
//  onto a stiffer film then took 24 iterations with plain sweeps, 13 with these.
__global__ void __launch_bounds__(kRT) KProbeChoose(int n, const ProbePair *__restrict__ x, RedScratch rs, double *lam)
{
	__shared__ double sh[2 * kRT];
	double a[2] = {0.0, 0.0}, tot[2];
	const int i = blockIdx.x * kRT + threadIdx.x;
	if(i < n)
	{
		const ProbePair v = x[i];
		a[0] = (double)v.x * (double)v.x;
		a[1] = (double)v.y * (double)v.y;
	}
	if(GridFold<2>(a, sh, rs, tot) && threadIdx.x == 0) lam[2] = (tot[0] <= tot[1] || tot[0] <= 4e-4 / 3.0 * n || !(tot[1] == tot[1])) ? 0.0 : 1.0;
}

//  x = inv f, inv row-major: one warp per row, lane l sums j = l, l+32, ...
//  from 0.0 (coalesced reads of the row), then a pairwise shuffle fold
template<class T, class TF, class TX>
__global__ void KDenseMV(const int *__restrict__ halt, int n, const T *__restrict__ inv, const TF *__restrict__ f,
                         TX *__restrict__ x)
{
	PdlEntry();
	if(halt && *halt) return;
	const int lane = threadIdx.x & 31;
	const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
	for(long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps)
	{
		const T *row = inv + (size_t)i * n;
		T s = T(0);
		for(int j = lane; j < n; j += 32) s = s + row[j] * (T)f[j];
#pragma unroll
		for(int off = 16; off >= 1; off >>= 1) s = s + __shfl_down_sync(0xffffffffu, s, off);
		if(lane == 0) x[i] = (TX)s;
	}
}

//--------------------------------------------------------------------------
//  The coarse levels of the FP32 cycle with L lanes per row (L = 2, 4, 8):
//  lane q sums the row's entries q, q + L, ... and the group folds its L
//  partials by shuffles.  The coarse rows (an aggregate's Galerkin row, 10
//  to 30 entries) are few, so one thread a row leaves most of the GPU idle;
//  the FP32 cycle's sums are not the oracle's to begin with, so their order
//  is free.  32 / L rows a warp, the loop alike for all its lanes.
//--------------------------------------------------------------------------
template<int L, class T, class XF>
__device__ __forceinline__ T RowSumLanes(const int *__restrict__ ptr, const int *__restrict__ col,
                                         const T *__restrict__ val, long long row, bool active, int q, XF xf)
{
	T p = T(0);
	if(active)
	{
		const int st = ptr[row], len = ptr[row + 1] - st;
		for(int k = q; k < len; k += L) p = p + val[st + k] * xf(col[st + k]);
	}
#pragma unroll
	for(int off = L / 2; off >= 1; off >>= 1) p = p + __shfl_down_sync(0xffffffffu, p, off);
	return p;
}

#define YZ_LANE_LOOP(L)                                                                              \
	const int lane_ = threadIdx.x & 31, q = lane_ % (L);                                             \
	const long long warps_ = ((long long)gridDim.x * blockDim.x) >> 5;                              \
	for(long long base_ = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (32 / (L));   \
	    base_ < n; base_ += warps_ * (32 / (L)))

//  x = m .* f, t = f - A x
template<int L, class T>
__global__ void KPreSmoothResidualL(const int *__restrict__ halt, int n, const int *__restrict__ ptr,
                                    const int *__restrict__ col, const T *__restrict__ val, const T *__restrict__ M,
                                    const T *__restrict__ f, T *__restrict__ x, T *__restrict__ t)
{
	PdlEntry();
	if(halt && *halt) return;
	YZ_LANE_LOOP(L)
	{
		const long long row = base_ + lane_ / L;
		const bool active = row < n;
		const T s = RowSumLanes<L>(ptr, col, val, row, active, q, [&](int c) { return M[c] * f[c]; });
		if(active && q == 0)
		{
			const T fi = f[row];
			x[row] = M[row] * fi;
			t[row] = fi - s;
		}
	}
}

//  xout = x + m .* (f - A x)
template<int L, class T>
__global__ void KPostSmoothL(const int *__restrict__ halt, int n, const int *__restrict__ ptr,
                             const int *__restrict__ col, const T *__restrict__ val, const T *__restrict__ M,
                             const T *__restrict__ f, const T *__restrict__ x, T *__restrict__ xout)
{
	PdlEntry();
	if(halt && *halt) return;
	YZ_LANE_LOOP(L)
	{
		const long long row = base_ + lane_ / L;
		const bool active = row < n;
		const T s = RowSumLanes<L>(ptr, col, val, row, active, q, [&](int c) { return x[c]; });
		if(active && q == 0) xout[row] = x[row] + M[row] * (f[row] - s);
	}
}

//  xout = x + P xc
template<int L, class T>
__global__ void KProlongL(const int *__restrict__ halt, int n, const int *__restrict__ pptr, const int *__restrict__ pcol,
                          const T *__restrict__ pval, const T *__restrict__ xc, const T *__restrict__ x,
                          T *__restrict__ xout)
{
	PdlEntry();
	if(halt && *halt) return;
	YZ_LANE_LOOP(L)
	{
		const long long row = base_ + lane_ / L;
		const bool active = row < n;
		const T s = RowSumLanes<L>(pptr, pcol, pval, row, active, q, [&](int c) { return xc[c]; });
		if(active && q == 0) xout[row] = x[row] + s;
	}
}

//--------------------------------------------------------------------------
//  A coarse level's way down and way up, each in one launch.  Below the
//  finest level the V-cycle's phases are short (a few thousand rows) and
//  each costs a kernel boundary more than its work; two of the four per
//  level go by recomputing what the separate kernels passed through memory:
//
//    down:  fc = R (f - A (m .* f))              (pre-smoothing from zero,
//           the residual and the restriction; t_j recomputed by every R row
//           that holds j)
//    up:    x = xt + m .* (f - A xt),  xt = m .* f + P xc
//           (prolongation and post-smoothing; xt_k recomputed by every row
//           whose A row holds k)
//
//  The same arithmetic as the separate kernels in another order: the FP32
//  cycle's sums are not the oracle's.  L lanes a row (the down kernel's rows
//  are the next level's), each lane a fixed share of the row's entries, the
//  partials folded by shuffles: deterministic.
//--------------------------------------------------------------------------
template<int L, class T>
__global__ void KDownFused(const int *__restrict__ halt, int n, const int *__restrict__ rptr,
                           const int *__restrict__ rcol, const T *__restrict__ rval, const int *__restrict__ ptr,
                           const int *__restrict__ col, const T *__restrict__ val, const T *__restrict__ M,
                           const T *__restrict__ f, T *__restrict__ fc)
{
	PdlEntry();
	if(halt && *halt) return;
	YZ_LANE_LOOP(L)
	{
		const long long row = base_ + lane_ / L;
		const bool active = row < n;
		const T s = RowSumLanes<L>(rptr, rcol, rval, row, active, q, [&](int j) {
			T a = T(0);
			const int st = ptr[j], en = ptr[j + 1];
			for(int e = st; e < en; ++e)
			{
				const int c = col[e];
				a = a + val[e] * (M[c] * f[c]);
			}
			return f[j] - a;
		});
		if(active && q == 0) fc[row] = s;
	}
}

template<int L, class T>
__global__ void KUpFused(const int *__restrict__ halt, int n, const int *__restrict__ ptr, const int *__restrict__ col,
                         const T *__restrict__ val, const T *__restrict__ M, const int *__restrict__ pptr,
                         const int *__restrict__ pcol, const T *__restrict__ pval, const T *__restrict__ f,
                         const T *__restrict__ xc, T *__restrict__ x)
{
	PdlEntry();
	if(halt && *halt) return;
	auto xt = [&](int k) {
		T s = T(0);
		for(int e = pptr[k], en = pptr[k + 1]; e < en; ++e) s = s + pval[e] * xc[pcol[e]];
		return M[k] * f[k] + s;
	};
	YZ_LANE_LOOP(L)
	{
		const long long row = base_ + lane_ / L;
		const bool active = row < n;
		const T s = RowSumLanes<L>(ptr, col, val, row, active, q, xt);
		if(active && q == 0) x[row] = xt((int)row) + M[row] * (f[row] - s);
	}
}
#undef YZ_LANE_LOOP

//  the FP32 copies of the V-cycle's matrices: dst_k[i] = (float)src_k[i] over
//  a list of arrays, one launch for all of them
struct RoundList
{
	enum { kMax = 64 };
	const double *src[kMax];
	float *dst[kMax];
	long long n[kMax];
	int count;
};

__global__ void KRoundToFloat(RoundList L)
{
	const long long stride = (long long)gridDim.x * blockDim.x;
	for(int k = 0; k < L.count; ++k)
	{
		const double *__restrict__ s = L.src[k];
		float *__restrict__ d = L.dst[k];
		for(long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < L.n[k]; i += stride) d[i] = (float)s[i];
	}
}

__global__ void KDiagApply(const int *__restrict__ halt, int n, const double *__restrict__ M, const double *__restrict__ r, double *__restrict__ z)
{
	if(halt && *halt) return;
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) z[i] = M[i] * r[i];
}

} // namespace yz
