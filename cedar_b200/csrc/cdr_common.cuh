// cdr_common.cuh -- shared definitions for the cedar_b200 CUDA library.
//
// Device layout of a 2D level (same logical layout as Cedar's arrays,
// include/cedar/stencil_op_nd.h:41-78): one ghost ring, i fastest, every stencil
// direction in its own plane.  Rows are padded to a pitch (elements) so that
// row starts are 128/256-byte aligned; planes are pitch*jj elements apart.
// Index (i, j, k) with 0-based i in [0, nx+1], j in [0, ny+1] (ghosts at 0 and
// n+1) lives at p[k*pitch*jj + j*pitch + i].
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>

#include "../../include/cdr_gpu.h"

namespace cdrgpu {

// Stencil plane numbers (Cedar 2D enum, include/cedar/2d/base_types.h:4-14).
enum : int { PC = 0, PW = 1, PS = 2, PSW = 3, PNW = 4 };
// Interpolation planes (include/cedar/2d/prolong_op.h:14).
enum : int { IL = 0, IR = 1, IA = 2, IB = 3, ISW = 4, INW = 5, INE = 6, ISE = 7 };

struct Dims2 {
	int nx, ny;     // interior points
	int pitch;      // elements per row (>= nx + 2)
	// Batches of independent problems of this size: a launch covers nb of them
	// (grid z); entry z of the batch is problem z*bstep of the arrays, whose
	// problems lie back to back (an array of P planes holds P*plane() elements
	// per problem).  A single problem has nb = bstep = 1.
	int nb = 1, bstep = 1;
	__host__ __device__ int ii() const { return nx + 2; }
	__host__ __device__ int jj() const { return ny + 2; }
	__host__ __device__ size_t plane() const { return (size_t)pitch * (ny + 2); }
	__host__ __device__ size_t at(int i, int j) const { return (size_t)j * pitch + i; }
#ifdef __CUDACC__
	// element offset of this CTA's problem in an array of `per` elements per problem
	__device__ __forceinline__ size_t bofs(size_t per) const { return (size_t)blockIdx.z * (size_t)bstep * per; }
#endif
};

// Counts kernel launches issued by this library (graph replays add the
// launches of the captured cycle).
void count_launches(long long n);

// Records the first error of this thread; the C ABI returns it and
// cdr_gpu_last_error() reports its text.
void set_error(int code, const char *fmt, ...);

// Kernel launch.  Where it pays, the grid depends programmatically on the kernel
// before it in the stream: it becomes resident while that one drains, which hides
// the launch and the first instruction fetch of the many short kernels of a cycle.
// Every kernel launched here begins with await_previous(): it touches no memory
// before the kernels ahead of it have completed.
// The rule counts SMs' worth of blocks (threads or shared memory, whichever fills
// an SM first).  Blocks that become resident early settle on the SMs that are
// free first, so a grid that does not fill the chip piles up on a few SMs when a
// large kernel is draining (2047^2: an FCG iteration 718 -> 750 us), and so do
// blocks of more than an eighth of an SM (all grids early: 881 us).  Early
// therefore: grids of small blocks, up to about a wave, that either fill most of the
// chip or follow a kernel that left half of it free; a few large blocks always.
struct LaunchSize {
	double sms, block;  // SMs' worth of the grid; part of an SM one block takes
	double blocks;
};
inline LaunchSize launch_size(dim3 grid, dim3 block, size_t smem)
{
	LaunchSize z;
	z.blocks = (double)grid.x * grid.y * grid.z;
	const double th = (double)(block.x * block.y * block.z) / 2048.0, sm = (double)smem / (228.0 * 1024.0);
	z.block = th > sm ? th : sm;
	z.sms = z.blocks * z.block;
	return z;
}
inline bool launch_early(const LaunchSize &z, double before)
{
	if (z.blocks <= 16.0) return true;
	return z.block <= 0.126 && z.sms <= 185.0 && (z.sms >= 60.0 || before <= 74.0);
}
// SMs' worth of this thread's last launch (only weighs the choice above)
inline double &launch_before()
{
	static thread_local double sms = 0.0;
	return sms;
}

template <typename... P, typename... A>
inline void launch_as(bool may_be_early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                      A... args)
{
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[0].val.programmaticStreamSerializationAllowed = 1;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = grid;
	cfg.blockDim = block;
	cfg.dynamicSmemBytes = smem;
	cfg.stream = st;
	cfg.attrs = attr;
	const LaunchSize z = launch_size(grid, block, smem);
	cfg.numAttrs = may_be_early && launch_early(z, launch_before()) ? 1 : 0;
	launch_before() = z.sms;
	(void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);  // CDR_LAUNCH_CHECK reads the error
}
template <typename... P, typename... A>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
	launch_as(true, kernel, grid, block, smem, st, args...);
}

#ifdef __CUDACC__
// First statement of every kernel started by launch(): waits for the kernels
// ahead to complete, then lets the next one become resident (its own wait
// keeps it from running; one grid ahead at a time).
__device__ __forceinline__ void await_previous()
{
	asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}
// The wait alone: for launches of many short blocks, where letting the next kernel
// in costs each block more than it hides.  The next one follows when this is done.
__device__ __forceinline__ void await_previous_only()
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
}
#endif

#define CDR_CUDA_TRY(expr)                                                          \
	do {                                                                            \
		cudaError_t _e = (expr);                                                    \
		if (_e != cudaSuccess) {                                                    \
			::cdrgpu::set_error(CDR_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__, #expr, \
			                    cudaGetErrorString(_e));                            \
			return CDR_ERR_CUDA;                                                    \
		}                                                                           \
	} while (0)

#define CDR_LAUNCH_CHECK()                                                          \
	do {                                                                            \
		::cdrgpu::count_launches(1);                                                \
		cudaError_t _e = cudaGetLastError();                                        \
		if (_e != cudaSuccess) {                                                    \
			::cdrgpu::set_error(CDR_ERR_CUDA, "%s:%d launch: %s", __FILE__, __LINE__,  \
			                    cudaGetErrorString(_e));                            \
			return CDR_ERR_CUDA;                                                    \
		}                                                                           \
	} while (0)

#define CDR_TRY(expr)                                                               \
	do {                                                                            \
		int _s = (expr);                                                            \
		if (_s != CDR_OK) return _s;                                                \
	} while (0)

inline int ceil_div(long a, long b) { return (int)((a + b - 1) / b); }

}  // namespace cdrgpu
