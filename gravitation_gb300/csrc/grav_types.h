// grav_types.h -- internal constants shared by host and device code of libgravgb300.
#pragma once

#include <cuda_runtime.h>

#include "gravitation_gb300.h"

// Wall-clock bound of every device-side wait on a bulk copy (nanoseconds).
#define GRAV_WAIT_NS 2000000000ull

namespace grav {

// Modes with FP64 positions and slots.
__host__ __device__ inline bool fp64_mode(int mode)
{
	return mode == GRAV_MODE_FP64 || mode == GRAV_MODE_FP64U;
}

// Launch-time view of one stage-1 kernel instantiation.
struct Stage1Kernel {
	int mode, bpt, threads, jtile;
	const void* fn;       // __global__ function
	int smem_bytes;       // dynamic shared memory per CTA
	bool dependent;       // waits with grid_dep_wait(): may launch as a programmatic dependent
	int block = 0;        // threads per CTA where they are not the tile's (rows / bpt)
	int cta_threads() const { return block ? block : threads; }
};

// Let launches of `fn` on the current device take `bytes` of dynamic shared memory (above 48 KB
// of static plus dynamic the kernel's limit has to be raised).  Called before occupancy queries
// and launches (abi.cu).
cudaError_t ensure_smem(const void* fn, int bytes);

// Stage-2 kernel (stage2.cu).  dependent = true launches it with programmatic stream
// serialization (it reads only plan tables before its grid_dep_wait()); false launches
// it the ordinary way, for callers whose previous kernel wrote those tables.
cudaError_t launch_stage2(const grav_batch& b, int flags, cudaStream_t stream,
	bool dependent = true);

// Single-launch step of one small universe (fused.cu).
const void* find_fused(int mode, int threads);
cudaError_t launch_fused(const grav_batch& b, int flags, int threads, int rows, int32_t* sync,
	cudaStream_t stream);
int fused_occupancy(int mode, int64_t n, int threads, int rows, int* ctas_per_sm);

// K steps of one universe in one launch (steps.cu).
bool steps_supported(int mode, int n, int sms);
int64_t steps_scratch(int n);
cudaError_t launch_steps(const grav_batch& b, int flags, int steps, int64_t a_stride, void* scratch,
	int sms, cudaStream_t stream);

// K backward steps of one universe in one launch (adjoint_steps.cu).
bool adjoint_steps_supported(int n, int sms);
int64_t adjoint_steps_scratch(int n);
cudaError_t launch_adjoint_steps(const grav_batch& b, const grav_adjoint& a, int steps,
	int64_t a_stride, void* scratch, int sms, cudaStream_t stream);

// Kernel tables, one per translation unit (stage1_f32.cu, stage1_f64.cu).
int stage1_table_f32(const Stage1Kernel** out);
int stage1_table_f64(const Stage1Kernel** out);
int stage1_table_sym(const Stage1Kernel** out);

// Launch with programmatic stream serialization: the kernel may begin while the kernel
// before it in the stream finishes; it must call grid_dep_wait() (grav_device.cuh)
// before touching anything that kernel, or one before it, writes.
inline cudaError_t launch_dependent(const void* fn, unsigned grid, unsigned threads,
	size_t smem, cudaStream_t stream, void** args)
{
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(grid);
	cfg.blockDim = dim3(threads);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = stream;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[0].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	return cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace grav
