// yz_gj.cuh -- the dense inverse of the direct level: Gauss-Jordan with
// partial pivoting, element for element the oracle's GaussJordanInverse
// (yzo_solver.cpp), which runs on [A | I].
//
// Step k of that algorithm swaps rows k and p_k (the pivot row), divides row
// k by the pivot and subtracts f_k(i) times it from every other row i, f_k
// being column k before the division.  Two facts make it cheaper without
// changing an operation on a value that can differ from 0 (a pivot that is 0
// or not finite aside, see the end):
//
//  * In place.  Column n + o of [A | I] stays the unit vector of row o's
//    present position until row o is taken as a pivot row (its entry in row
//    k is 0 until then, so every step leaves it as it is), and column k is
//    the unit vector e_k from step k on.  So slot k holds column k before
//    step k and column n + orig(k) after it, orig(k) being the row taken:
//    n columns instead of 2 n, half the operations and half the bytes.  The
//    slot's new column is 1 / piv in row k and 0 - f (1 / piv) elsewhere.
//  * Blocked.  B consecutive steps change a column outside the panel only
//    through their pivots, multipliers and swaps, so a panel of B slots is
//    run through its steps in one block's registers and every other column
//    then replays them, each element receiving the same operations in the
//    same order, from registers.
//
// One launch (KGjStep) applies panel q to every column and, in block 0,
// first to the slots of panel q + 1, which it then factors: the serial chain
// of the pivots overlaps with the wide update of the other blocks.  The
// chain is what bounds it at the sizes of a film's coarsest level (347-500
// rows): a thread a row, its B entries in registers, the pivot found by
// integer warp reductions of the bits of |a| (their order is that of the
// values), three block barriers a step.  At 1,000-3,000 rows (small films,
// whose only level this is) the panel is narrower, as its rows take more of the
// registers, and the update's bytes bound it.  Against a panel launch and an
// update launch on [A | I], 32 steps a panel: the set-up of a 1,936-row system
// 38.0 -> 7.5 ms, of a 92,416-row one (347 rows at the bottom) 3.2 -> 1.9.
//
// A multiplier of 0 leaves the element as it is even where the row is not
// finite; the wide update tests that only where a row of the step is not
// finite (a singular level).  On [A | I] a pivot of 0 makes 0 / 0 in row k of
// the columns not yet taken, which are not held here.  Their slots' own row k
// is divided by that 0 too, so row k ends without a finite entry, and so does
// every row with a multiplier other than 0, in either form; the other rows are
// not touched.  A place may hold an infinity here and a NaN there: a run's
// first half step makes a NaN of both.
#pragma once

#include "yz_common.cuh"

namespace yz {

constexpr int kGjThreads = 512;             // one block an SM, 128 registers a thread
constexpr int kGjMaxB = 16;                  // slots a panel, at most
constexpr int kGjCols = 16;                  // columns an update tile
constexpr int kGjRows = 2 * kGjMaxB;         // rows a panel's pivots and swaps touch, at most

//  what the columns outside a panel need of it, beside its multipliers
struct GjPanel
{
	int b, k0, rows;                         // steps, first slot, rows listed below
	int loc[kGjMaxB];                        // the place of each step's pivot row in the list
	int list[kGjRows];                       // the rows the steps divide or swap: k0.., then the others
	double val[kGjMaxB];                     // the pivots
};

//  slots a panel: 16 while a thread holds one row or two, 8 with four or six
inline int GjPanelWidth(int n) { return n <= 2 * kGjThreads ? 16 : 8; }

__global__ void KGjInit(int n, const int *__restrict__ ptr, const int *__restrict__ col,
                        const double *__restrict__ val, double *__restrict__ Mc, int *__restrict__ orig)
{
	PdlEntry();
	for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		orig[i] = i;
		for(int k = ptr[i]; k < ptr[i + 1]; ++k) Mc[(size_t)col[k] * n + i] = val[k];
	}
}

//  The larger |a| first, the smaller row among equals, over a warp: the
//  first row of the largest |a| (key 0: none, or a NaN, which is never taken)
__device__ __forceinline__ void GjWarpBest(unsigned &hi, unsigned &lo, int &idx)
{
	const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
	const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
	idx = (int)__reduce_min_sync(0xffffffffu, (hi == mh && lo == ml) ? (unsigned)idx : 0x7fffffffu);
	hi = mh; lo = ml;
}

//  |a|'s bits plus one (0 for a NaN): an order-preserving key
__device__ __forceinline__ unsigned long long GjKey(double a)
{
	const unsigned long long u = (unsigned long long)__double_as_longlong(fabs(a));
	return u > 0x7ff0000000000000ull ? 0ull : u + 1ull;
}

//  Panel `prev` (its record and multipliers F, a column of n a step) applied
//  to the columns of tile [j0, j0 + 16) outside [s0, s1) by the block
template<int B, int CG, int RP>
__device__ __forceinline__ void GjApply(int n, double *__restrict__ Mc, const GjPanel *__restrict__ prev,
                                        const double *__restrict__ F, int j0, int j1, int s0, int s1,
                                        double (*__restrict__ rowK)[kGjCols], const double (*__restrict__ Fs)[kGjRows],
                                        const unsigned *__restrict__ touched,
                                        int *__restrict__ bad)
{
	const int t = threadIdx.x, lane = t & 31, w = t >> 5;
	const int b = prev->b, rows = prev->rows, k0 = prev->k0;
	auto skip = [&](int j) { return j >= j1 || (j >= k0 && j < k0 + b) || (j >= s0 && j < s1); };
	//  the rows the steps divide or swap, a warp a column, a lane a row: the
	//  pivot rows' quotients are what every other row subtracts
	if(w < kGjCols)
	{
		const int j = j0 + w;
		if(!skip(j))
		{
			const bool on = lane < rows;
			double *cj = Mc + (size_t)j * n;
			const int i = on ? prev->list[lane] : 0;
			const int lpl = lane < b ? prev->loc[lane] : 0;
			const double pvl = lane < b ? prev->val[lane] : 1.0;
			double v = on ? cj[i] : 0.0;
#pragma unroll 1
			for(int c = 0; c < b; ++c)
			{
				const double f = Fs[c][lane];
				const int lp = __shfl_sync(0xffffffffu, lpl, c);
				const double colp = __shfl_sync(0xffffffffu, v, lp), colk = __shfl_sync(0xffffffffu, v, c);
				const double rk = colp / __shfl_sync(0xffffffffu, pvl, c);
				if(lane == lp) v = colk;
				v = (lane == c) ? rk : (f == 0.0) ? v : v - f * rk;
				if(lane == 0)
				{
					rowK[c][w] = rk;
					if(!(fabs(rk) <= 1.7976931348623157e308)) *bad = 1;
				}
			}
			if(on) cj[i] = v;
		}
		else if(lane < kGjMaxB) rowK[lane][w] = 0.0;
	}
	__syncthreads();
	const bool safe = *bad == 0;
	//  the other rows, kGjCols / CG columns a thread, RP rows at a time, the
	//  multipliers four steps ahead of their use
	constexpr int NC = kGjCols / CG, RT = kGjThreads / CG, G = 4;
	const int c0 = (t / RT) * NC;
	unsigned on = 0;
#pragma unroll
	for(int u = 0; u < NC; ++u) on |= skip(j0 + c0 + u) ? 0u : 1u << u;
	if(on)
#pragma unroll 1
		for(int i0 = t % RT; i0 < n; i0 += RP * RT)
		{
			double m[RP][NC], f[RP][G];
			bool row[RP];
#pragma unroll
			for(int r = 0; r < RP; ++r)
			{
				const int i = i0 + r * RT;
				row[r] = i < n && !((touched[i >> 5] >> (i & 31)) & 1u);
#pragma unroll
				for(int u = 0; u < NC; ++u) m[r][u] = (row[r] && (on >> u) & 1u) ? Mc[(size_t)(j0 + c0 + u) * n + i] : 0.0;
#pragma unroll
				for(int q = 0; q < G; ++q) f[r][q] = (row[r] && q < b) ? F[(size_t)q * n + i] : 0.0;
			}
#pragma unroll 1
			for(int cb = 0; cb < b; cb += G)
			{
				double fn[RP][G];
#pragma unroll
				for(int r = 0; r < RP; ++r)
#pragma unroll
					for(int q = 0; q < G; ++q)
						fn[r][q] = (row[r] && cb + G + q < b) ? F[(size_t)(cb + G + q) * n + i0 + r * RT] : 0.0;
#pragma unroll
				for(int q = 0; q < G; ++q)
				{
					if(cb + q >= b) break;
#pragma unroll
					for(int r = 0; r < RP; ++r)
#pragma unroll
						for(int u = 0; u < NC; ++u)
						{
							const double d = m[r][u] - f[r][q] * rowK[cb + q][c0 + u];
							m[r][u] = (safe || f[r][q] != 0.0) ? d : m[r][u];
						}
				}
#pragma unroll
				for(int r = 0; r < RP; ++r)
#pragma unroll
					for(int q = 0; q < G; ++q) f[r][q] = fn[r][q];
			}
#pragma unroll
			for(int r = 0; r < RP; ++r)
#pragma unroll
				for(int u = 0; u < NC; ++u)
					if(row[r] && (on >> u) & 1u) Mc[(size_t)(j0 + c0 + u) * n + i0 + r * RT] = m[r][u];
		}
	__syncthreads();
}

//  The panel of bN <= B slots from kN on, run through its steps: a thread
//  holds R rows, t + 512 r.  Records the pivots and the multipliers (the
//  column of step c after its swap, n a step) and leaves the slots' columns
//  of the inverse in Mc.
template<int B, int R>
__device__ __forceinline__ void GjFactor(int n, double *__restrict__ Mc, int kN, int bN, GjPanel *__restrict__ next,
                                         double *__restrict__ F, int *__restrict__ orig)
{
	__shared__ __align__(16) double rowk[2][B], rowp[B], rq[B];
	constexpr int NW = kGjThreads / 32;
	__shared__ unsigned whi[NW], wlo[NW];
	__shared__ int widx[NW], piv[B], list[kGjRows];
	const int t = threadIdx.x, lane = t & 31, w = t >> 5;
	double a[R][B];
#pragma unroll
	for(int r = 0; r < R; ++r)
#pragma unroll
		for(int j = 0; j < B; ++j)
		{
			const int i = t + r * kGjThreads;
			a[r][j] = (i < n && j < bN) ? Mc[(size_t)(kN + j) * n + i] : 0.0;
		}
#pragma unroll 1
	for(int c = 0; c < bN; ++c)
	{
		const int k = kN + c;
		//  the pivot: the first row of the largest |a| among rows k..
		unsigned long long key = 0;
		int idx = 0x7fffffff;
#pragma unroll
		for(int r = 0; r < R; ++r)
		{
			const int i = t + r * kGjThreads;
			if(i >= k && i < n)
			{
				const unsigned long long u = GjKey(a[r][0]);
				if(u > key) { key = u; idx = i; }
			}
			if(i == k)
			{
#pragma unroll
				for(int j = 0; j < B; ++j) rowk[c & 1][j] = a[r][j];
			}
		}
		unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
		GjWarpBest(hi, lo, idx);
		if(lane == 0) { whi[w] = hi; wlo[w] = lo; widx[w] = idx; }
		__syncthreads();
		hi = lane < NW ? whi[lane] : 0u; lo = lane < NW ? wlo[lane] : 0u; idx = lane < NW ? widx[lane] : 0x7fffffff;
		GjWarpBest(hi, lo, idx);
		const unsigned long long best = ((unsigned long long)hi << 32) | lo;
		//  taken only when larger than |a_kk| (never over a NaN there)
		const unsigned long long own = GjKey(rowk[c & 1][0]);
		const int p = (own != 0 && best > own) ? idx : k;
#pragma unroll
		for(int r = 0; r < R; ++r)
			if(t + r * kGjThreads == p)
			{
#pragma unroll
				for(int j = 0; j < B; ++j) rowp[j] = a[r][j];
			}
		__syncthreads();
		//  row k's new values; the slot itself turns into the inverse's column
		if(t < B) rq[t] = (t == 0 ? 1.0 : rowp[t]) / rowp[0];
		if(t == 0) { piv[c] = p; next->val[c] = rowp[0]; }
		__syncthreads();
#pragma unroll
		for(int r = 0; r < R; ++r)
		{
			const int i = t + r * kGjThreads;
			if(i >= n) continue;
			if(i == k)
			{
				F[(size_t)c * n + i] = rowp[0];
#pragma unroll
				for(int j = 0; j < B; ++j) a[r][j] = rq[(j + 1) % B];
				continue;
			}
			if(i == p)
			{
#pragma unroll
				for(int j = 0; j < B; ++j) a[r][j] = rowk[c & 1][j];
			}
			const double f = a[r][0];
			F[(size_t)c * n + i] = f;
			//  the slots move down a register a step, so that the step's own
			//  is always the first: one loop body, which stays in the
			//  instruction cache (unrolled over the steps the kernel waited for
			//  its instructions, 2,500 cycles a step)
			const double slot = f == 0.0 ? 0.0 : 0.0 - f * rq[0];
#pragma unroll
			for(int j = 0; j + 1 < B; ++j) a[r][j] = f == 0.0 ? a[r][j + 1] : a[r][j + 1] - f * rq[j + 1];
			a[r][B - 1] = slot;
		}
	}
	//  register j holds slot (j + bN) mod B now
#pragma unroll
	for(int r = 0; r < R; ++r)
#pragma unroll
		for(int j = 0; j < B; ++j)
		{
			const int i = t + r * kGjThreads, q = (j + bN) % B;
			if(i < n && q < bN) Mc[(size_t)(kN + q) * n + i] = a[r][j];
		}
	//  the rows the steps touched (the panel's, then the other pivot rows,
	//  each once) and which original row each of them now holds: one warp, a
	//  lane a step, then a lane a row
	__syncthreads();
	if(w != 0) return;
	const unsigned all = 0xffffffffu;
	const bool step = lane < bN;
	const int p = step ? piv[lane] : -1 - lane;
	const int first = __ffs(__match_any_sync(all, p)) - 1;
	const unsigned others = __ballot_sync(all, step && p >= kN + bN && first == lane);
	const int at = (p < kN + bN) ? p - kN : bN + __popc(others & ((1u << first) - 1u));
	const int m = bN + __popc(others);
	if(step)
	{
		list[lane] = kN + lane;
		if(p >= kN + bN && first == lane) list[at] = p;
		next->loc[lane] = at;
	}
	__syncwarp();
	const int row = lane < m ? list[lane] : 0;
	int o = lane < m ? orig[row] : 0;
	for(int c = 0; c < bN; ++c)
	{
		const int lp = __shfl_sync(all, at, c);
		const int ok = __shfl_sync(all, o, c), op = __shfl_sync(all, o, lp);
		if(lane == lp) o = ok;
		if(lane == c) o = op;
	}
	if(lane < m) { next->list[lane] = row; orig[row] = o; }
	if(lane == 0) { next->b = bN; next->k0 = kN; next->rows = m; }
}

//  prev null: the first panel is factored (one block); bN 0: the last panel
//  is applied.  CG: threads side by side on a row's columns in the update (2
//  while 256 rows fill the block).
template<int B, int R, int CG, int RP>
__global__ void __launch_bounds__(kGjThreads, 1) KGjStep(int n, double *__restrict__ Mc, const GjPanel *__restrict__ prev,
                                                         const double *__restrict__ F, GjPanel *__restrict__ next,
                                                         double *__restrict__ Fn, int kN, int bN,
                                                         int *__restrict__ orig)
{
	PdlEntry();
	__shared__ __align__(16) double rowK[kGjMaxB][kGjCols];
	__shared__ double Fs[kGjMaxB][kGjRows];  // the multipliers of the listed rows
	__shared__ unsigned touched[96];         // a bit a row: listed (n <= 3000)
	__shared__ int bad;
	const int t = threadIdx.x;
	if(blockIdx.x == 0 && bN == 0) return;
	if(prev)
	{
		if(t < 96) touched[t] = 0;
		if(t == 0) bad = 0;
		__syncthreads();
		if(t < prev->rows)
		{
			const int i = prev->list[t];
			atomicOr(&touched[i >> 5], 1u << (i & 31));
		}
		for(int e = t; e < prev->b * kGjRows; e += kGjThreads)
			if(e % kGjRows < prev->rows) Fs[e / kGjRows][e % kGjRows] = F[(size_t)(e / kGjRows) * n + prev->list[e % kGjRows]];
		__syncthreads();
		if(blockIdx.x == 0) GjApply<B, CG, RP>(n, Mc, prev, F, kN, kN + bN, 0, 0, rowK, Fs, touched, &bad);
		else
			for(int tile = blockIdx.x - 1; tile * kGjCols < n; tile += gridDim.x - 1)
			{
				GjApply<B, CG, RP>(n, Mc, prev, F, tile * kGjCols, n, kN, kN + bN, rowK, Fs, touched, &bad);
				if(t == 0) bad = 0;
				__syncthreads();
			}
	}
	if(blockIdx.x == 0) GjFactor<B, R>(n, Mc, kN, bN, next, Fn, orig);
}

//  slot k is the inverse's column orig(k): into row-major order, 32 x 32
//  tiles through shared memory
__global__ void __launch_bounds__(256) KGjExtract(int n, const double *__restrict__ Mc, const int *__restrict__ orig,
                                                  double *__restrict__ inv)
{
	PdlEntry();
	__shared__ double tile[32][33];
	const int nt = (n + 31) / 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
	for(int q = blockIdx.x; q < nt * nt; q += gridDim.x)
	{
		const int i0 = (q % nt) * 32, k0 = (q / nt) * 32;
		for(int r = ty; r < 32; r += 8)
			if(k0 + r < n && i0 + tx < n) tile[r][tx] = Mc[(size_t)(k0 + r) * n + i0 + tx];
		__syncthreads();
		const int o = (k0 + tx < n) ? orig[k0 + tx] : 0;
		for(int r = ty; r < 32; r += 8)
			if(k0 + tx < n && i0 + r < n) inv[(size_t)(i0 + r) * n + o] = tile[tx][r];
		__syncthreads();
	}
}

} // namespace yz
