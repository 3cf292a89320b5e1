// yz_common.cuh -- shared host/device utilities of the B200 implicit-step library.
//
// Built for sm_100a only.  The FP64 parity kernels are compiled with
// -fmad=false so that every a*b+c rounds twice, as the reference's host code
// does under -ffp-contract=off (CMakeLists.txt:33-46).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <vector>

namespace yz {

//--------------------------------------------------------------------------
//  errors and launch accounting
//--------------------------------------------------------------------------
struct CudaError : std::runtime_error
{
	explicit CudaError(const std::string &m) : std::runtime_error(m) {}
};
struct UsageError : std::runtime_error
{
	explicit UsageError(const std::string &m) : std::runtime_error(m) {}
};
//  a numerical failure of the time step (the reference's FatalError at the
//  step: dt below MinDt, ImplicitSolver.cpp:180-184; no convergence at a
//  fixed step, FailedFixedStep, ImplicitSolver.cpp:192-201)
struct StepFailed : std::runtime_error
{
	explicit StepFailed(const std::string &m) : std::runtime_error(m) {}
};

inline void Check(cudaError_t e, const char *what)
{
	if(e != cudaSuccess)
	{
		//  a failed call also leaves its error as the thread's last error:
		//  take it, so that the next launch's check does not report it again
		(void)cudaGetLastError();
		throw CudaError(std::string(what) + ": " + cudaGetErrorString(e));
	}
}
#define YZ_CUDA(call) ::yz::Check((call), #call)

//  Every kernel launch of the library goes through YZ_LAUNCH, which counts it,
//  and, for the one kernel named by yz_time_kernel(), brackets it with CUDA
//  events on its own stream (the per-launch device time of that kernel).
extern std::atomic<long long> g_launches;     // every launch of the process (yz_launch_count)
extern thread_local long long t_launches;     // this thread's: a context's counts are taken from it
//  count n launches (negative: take back launches that were captured, not run)
inline void CountLaunches(long long n)
{
	g_launches.fetch_add(n, std::memory_order_relaxed);
	t_launches += n;
}
bool TimedKernel(const char *name);
bool TimingActive();   // a kernel is selected for per-launch timing
void TimeBegin(cudaStream_t st);
void TimeEnd(cudaStream_t st);
long long TimeCount();            // timed launches recorded so far
void TimeDropLast(long long k);   // forget the last k of them

#define YZ_LAUNCH(kernel, grid, block, smem, stream, ...)                         \
	do {                                                                          \
		const bool yzTimed_ = ::yz::TimedKernel(#kernel);                         \
		if(yzTimed_) ::yz::TimeBegin(stream);                                     \
		kernel<<<(grid), (block), (smem), (stream)>>>(__VA_ARGS__);               \
		if(yzTimed_) ::yz::TimeEnd(stream);                                       \
		::yz::CountLaunches(1);                                                   \
		::yz::Check(cudaGetLastError(), #kernel);                                 \
	} while(0)

//  Programmatic dependent launch for chains of short kernels: a kernel
//  launched by YZ_LAUNCH_CHAIN (the AMG set-up) or YZ_LAUNCH_PDL (the BiCGStab
//  loop and the V-cycle) may be scheduled while the kernel before it on the
//  stream drains.  Such a kernel begins with PdlEntry(): griddepcontrol.wait
//  holds every thread until the kernels it depends on have completed and their
//  memory is visible (so its reads and writes are those of a plain launch),
//  then launch_dependents lets the next kernel be scheduled.  Without the
//  launch attribute both are no-ops.
//  The set-up's 70 kernels a hierarchy are queued on the stream, where it pays:
//  64^2 1.81 -> 1.42 ms, 224^2 3.95 -> 3.23, 301^2 4.4 -> 3.6, and the direct
//  level's 242 launches at 1,936 rows 7.7 -> 7.2.  The loop's lie in a graph,
//  where it does not (a 512^2 solve in 64 bits 7.7 without, 7.9 with), so there it
//  is off.  YZ_PDL=0 in the environment turns it off for both, YZ_PDL=1 on.
bool PdlOn();
bool ChainOn();
__device__ __forceinline__ void PdlEntry()
{
#if defined(__CUDA_ARCH__)
	asm volatile("griddepcontrol.wait;" ::: "memory");
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
}
#define YZ_LAUNCH_PDL(...) YZ_LAUNCH_PDL_IF(::yz::PdlOn(), __VA_ARGS__)
#define YZ_LAUNCH_CHAIN(...) YZ_LAUNCH_PDL_IF(::yz::ChainOn(), __VA_ARGS__)
#define YZ_LAUNCH_PDL_IF(pdl, kernel, grid, block, smem, strm, ...)             \
	do {                                                                          \
		const bool yzTimed_ = ::yz::TimedKernel(#kernel);                         \
		if(yzTimed_) ::yz::TimeBegin(strm);                                     \
		if(pdl)                                                                 \
		{                                                                         \
			cudaLaunchConfig_t yzCfg_ = {};                                       \
			yzCfg_.gridDim = dim3(grid);                                          \
			yzCfg_.blockDim = dim3(block);                                        \
			yzCfg_.dynamicSmemBytes = (smem);                                     \
			yzCfg_.stream = (strm);                                             \
			cudaLaunchAttribute yzAttr_[1];                                       \
			yzAttr_[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   \
			yzAttr_[0].val.programmaticStreamSerializationAllowed = 1;            \
			yzCfg_.attrs = yzAttr_;                                               \
			yzCfg_.numAttrs = 1;                                                  \
			::yz::Check(cudaLaunchKernelEx(&yzCfg_, kernel, __VA_ARGS__), #kernel); \
		}                                                                         \
		else                                                                      \
			kernel<<<(grid), (block), (smem), (strm)>>>(__VA_ARGS__);           \
		if(yzTimed_) ::yz::TimeEnd(strm);                                       \
		::yz::CountLaunches(1);                                                   \
		::yz::Check(cudaGetLastError(), #kernel);                                 \
	} while(0)

void SetLastError(const std::string &m);

//--------------------------------------------------------------------------
//  device buffer (grows, never shrinks; no allocation when large enough)
//--------------------------------------------------------------------------
//  The finest level's stencil: the slices of 32 rows (SELL-32) whose every
//  row has the pattern's most common column set relative to the row (the
//  interior rows of the film: columns i + off[k], ascending) are flagged;
//  their columns are computed, not loaded.  slice null: no flagged slices.
struct Sten
{
	const unsigned char *slice;
	int len;
	int off[16];
};

template<class T>
struct DBuf
{
	T *p = nullptr;
	size_t cap = 0;
	DBuf() = default;
	DBuf(const DBuf &) = delete;
	DBuf &operator=(const DBuf &) = delete;
	~DBuf() { if(p) cudaFree(p); }
	T *get() const { return p; }
	//  a buffer that must grow takes half as much again, so that sizes that
	//  creep up from solve to solve (the coarse levels of the hierarchy) do
	//  not free and allocate (each a device-wide synchronisation) every time
	void reserve(size_t n)
	{
		if(n <= cap) return;
		const size_t grown = cap ? cap + cap / 2 : 0;
		if(p) { cudaFree(p); p = nullptr; cap = 0; }
		size_t want = n < 16 ? 16 : n;
		if(grown > want) want = grown;
		YZ_CUDA(cudaMalloc(&p, want * sizeof(T)));
		cap = want;
	}
	void upload(const T *h, size_t n, cudaStream_t st)
	{
		reserve(n);
		if(n) YZ_CUDA(cudaMemcpyAsync(p, h, n * sizeof(T), cudaMemcpyHostToDevice, st));
	}
	void download(T *h, size_t n, cudaStream_t st) const
	{
		if(n) YZ_CUDA(cudaMemcpyAsync(h, p, n * sizeof(T), cudaMemcpyDeviceToHost, st));
	}
};

//--------------------------------------------------------------------------
//  the deterministic reduction tree (the oracle's DetSum, yzo_solver.cpp):
//  chunk b of 256 elements per block of 256 threads, thread t holds element
//  b*256 + t, pairwise fold over the block; the chunk sums are summed
//  strided by 256 threads (thread t: chunks t, t+256, ... from 0.0) and
//  folded the same way by the block that finishes last.  One element per
//  thread keeps every SM busy at the sizes of a film (n / 256 blocks).
//--------------------------------------------------------------------------
constexpr int kRT = 256;
constexpr int kRK = 1;
constexpr int kRPer = 8;		// blocks an SM of the reducing kernels
constexpr int kRChunk = kRT * kRK;

__host__ __device__ inline int RedChunks(int n) { return n > 0 ? (n + kRChunk - 1) / kRChunk : 1; }
inline int RedBlocks(int n) { return RedChunks(n); }

//  The blocks that share the chunks (ChunkFold): at most the 8 of 256 threads that an SM holds, and
//  of those as many as give each the same number of chunks.
inline int RedGrid(int n)
{
	const int nb = RedBlocks(n), per = (nb + 148 * kRPer - 1) / (148 * kRPer);
	return (nb + per - 1) / per;
}

//  The tree over 256 values v[0..255] in shared memory, by one warp: the folds
//  at 128, 64 and 32 of lane t read v[t + 32 w] of the 8 warps, so one warp
//  makes them without a barrier between (the same sums in the same order as
//  the pairwise fold).  Result valid in lane 0.
__device__ __forceinline__ double LaneTree(const double *v, int t)
{
	double u[8];
#pragma unroll
	for(int w = 0; w < 8; ++w) u[w] = v[t + 32 * w];
	double s = ((u[0] + u[4]) + (u[2] + u[6])) + ((u[1] + u[5]) + (u[3] + u[7]));
#pragma unroll
	for(int off = 16; off >= 1; off >>= 1) s = s + __shfl_down_sync(0xffffffffu, s, off);
	return s;
}

//  Fold Q values per thread over a block of 256 (same order as the
//  oracle's Tree256).
//  sh: Q*256 doubles of shared memory.  Result valid in thread 0.
template<int Q>
__device__ __forceinline__ void BlockTree(double (&a)[Q], double *sh)
{
	const int t = threadIdx.x;
#pragma unroll
	for(int q = 0; q < Q; ++q) sh[q * kRT + t] = a[q];
	__syncthreads();
	if(t < 32)
	{
#pragma unroll
		for(int q = 0; q < Q; ++q) a[q] = LaneTree(sh + q * kRT, t);
	}
}

//  Reduction scratch: Q partial arrays of `blocks` doubles and a counter.
struct RedScratch
{
	double *part;          // [Q][maxBlocks]
	unsigned int *counter; // one per reduction site
	int maxBlocks;
};

//  The end of a grid's reduction: every block calls it after its threads'
//  partials are written; the last block to arrive folds the `chunks` partials
//  of each q and returns true with the totals in tot[q] (valid in every
//  thread of it).  sh: Q*256 doubles that no thread reads any more after a
//  barrier.
template<int Q>
__device__ __forceinline__ bool GridLast(int chunks, double *sh, const RedScratch rs, double (&tot)[Q])
{
	__shared__ bool amLast;
	__shared__ double bc[Q];
	const int t = threadIdx.x;
	if(t == 0)
	{
		__threadfence();
		const unsigned prev = atomicAdd(rs.counter, 1u);
		amLast = (prev == gridDim.x - 1);
	}
	__syncthreads();
	if(!amLast) return false;
	__threadfence();
	double b[Q];
#pragma unroll
	for(int q = 0; q < Q; ++q)
	{
		//  eight loads in flight: the block is alone, so their latency is the time
		double s = 0.0;
		for(int j = t; j < chunks; j += 8 * kRT)
		{
			double p[8];
#pragma unroll
			for(int u = 0; u < 8; ++u) p[u] = j + u * kRT < chunks ? __ldcg(&rs.part[q * rs.maxBlocks + j + u * kRT]) : 0.0;
#pragma unroll
			for(int u = 0; u < 8; ++u)
				if(j + u * kRT < chunks) s = s + p[u];
		}
		b[q] = s;
	}
	BlockTree<Q>(b, sh);
	if(t == 0)
	{
#pragma unroll
		for(int q = 0; q < Q; ++q) bc[q] = b[q];
		*rs.counter = 0u;
	}
	__syncthreads();
#pragma unroll
	for(int q = 0; q < Q; ++q) tot[q] = bc[q];
	return true;
}

//  Called by every block of a grid of one block a chunk after its threads
//  hold their per-thread sums a[q]: writes the block's partials, then GridLast.
template<int Q>
__device__ __forceinline__ bool GridFold(double (&a)[Q], double *sh, const RedScratch rs, double (&tot)[Q])
{
	BlockTree<Q>(a, sh);
	if(threadIdx.x == 0)
	{
#pragma unroll
		for(int q = 0; q < Q; ++q) rs.part[q * rs.maxBlocks + blockIdx.x] = a[q];
	}
	return GridLast<Q>((int)gridDim.x, sh, rs, tot);
}

//  One chunk's sums in a kernel whose grid of RedGrid(n) blocks shares the
//  chunks (block b takes b, b + G, ...; c is the block's k-th): the block's
//  values a[q] into shared memory, in two halves by turns, and one warp, k mod
//  8, writes the chunk's partials while the others go on to the next chunk.
//  The sums are the same whatever G is.  One barrier a chunk, and one fence
//  and one atomic a block in GridLast (after a barrier) rather than one a
//  chunk: at 1,048,576 rows the update of x and r went from 16.7 to 12.5 us,
//  that of s from 12.4 to 9.4.  sh: 2*Q*256 doubles.
//  The products with the matrix keep a block a chunk (GridFold): in a loop
//  over chunks the compiler holds the row's 13 addresses across the turns,
//  which at 32 registers spills (262,144 rows: 12.2 against 8.4 us), and
//  fewer blocks an SM with more registers are slower too (10.4 to 11.2).
template<int Q>
__device__ __forceinline__ void ChunkFold(const double (&a)[Q], double *sh, int k, int c, const RedScratch rs)
{
	const int t = threadIdx.x;
	double *v = sh + (k & 1) * Q * kRT;
#pragma unroll
	for(int q = 0; q < Q; ++q) v[q * kRT + t] = a[q];
	__syncthreads();
	if((t >> 5) == (k & 7))
	{
#pragma unroll
		for(int q = 0; q < Q; ++q)
		{
			const double s = LaneTree(v + q * kRT, t & 31);
			if((t & 31) == 0) rs.part[q * rs.maxBlocks + c] = s;
		}
	}
}

//  the loop of such a kernel: row i of chunk c, the block's k-th
#define YZ_CHUNKS(n) for(int c_ = blockIdx.x, k_ = 0; c_ < RedChunks(n); c_ += gridDim.x, ++k_)
#define YZ_CHUNK_ROW (c_ * kRChunk + (int)threadIdx.x)

//--------------------------------------------------------------------------
//  exclusive scan of n ints into out[0..n] (out[n] = total); integer, so
//  the order of the additions does not matter.  Scratch: ScanScratchSize(n).
//--------------------------------------------------------------------------
size_t ScanScratchSize(int n);
void ScanExclusive(const int *in, int *out, int n, int *scratch, cudaStream_t st);

//  Grid size for a grid-stride kernel over n items.
inline int GridFor(long long n, int block, int cap = 148 * 16)
{
	long long g = (n + block - 1) / block;
	if(g < 1) g = 1;
	if(g > cap) g = cap;
	return (int)g;
}

} // namespace yz
