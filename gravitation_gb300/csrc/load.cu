// load.cu -- loading an engine's state from packed device arrays: the range of G m that the
// host needs before it accepts them, and the rows of r and v.
//
// A state that changes on every call (a rollout inside an optimiser) is loaded once per pass.
// As tensor operations that was fourteen launches and three waits for a scalar, 335 us of host
// time at 4096 bodies; as these two launches, a copy of 16 bytes and grav_prepare it is 134.
// Both kernels read and write each value once and are launch bound at any size an engine
// steps quickly.
#include "grav_device.cuh"

namespace grav {

int record_error(int code, const char* msg);

constexpr int LD_T = 256;

// out[0] = max(gm, 0), out[1] = 1.0 if some value is not finite or below zero; both zeroed
// before.  Non-negative doubles order as their bits do.
__global__ void __launch_bounds__(LD_T) gm_range_kernel(const double* __restrict__ gm, const int64_t n,
	unsigned long long* __restrict__ out)
{
	unsigned long long top = 0;
	bool bad = false;
	for (int64_t i = static_cast<int64_t>(blockIdx.x) * LD_T + threadIdx.x; i < n;
		i += static_cast<int64_t>(gridDim.x) * LD_T) {
		const double x = gm[i];
		if (!(x >= 0.0) || isinf(x)) bad = true;
		else if (x > 0.0) top = max(top, static_cast<unsigned long long>(__double_as_longlong(x)));
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
	bad = __any_sync(0xffffffffu, bad);
	if ((threadIdx.x & 31) == 0) {
		if (top) atomicMax(out, top);
		if (bad) atomicExch(out + 1, static_cast<unsigned long long>(__double_as_longlong(1.0)));
	}
}

__global__ void __launch_bounds__(LD_T) load_state_kernel(const double* __restrict__ r,
	const double* __restrict__ v, const double* __restrict__ gm, const int64_t n,
	double* __restrict__ r4, double* __restrict__ v4)
{
	const int64_t i = static_cast<int64_t>(blockIdx.x) * LD_T + threadIdx.x;   // one value of a row
	if (i >= 4 * n) return;
	const int64_t row = i >> 2;
	const int c = static_cast<int>(i & 3);
	r4[i] = c < 3 ? r[3 * row + c] : gm[row];
	v4[i] = c < 3 ? v[3 * row + c] : 0.0;
}

}  // namespace grav

extern "C" int grav_gm_range(const double* gm, int64_t n, double* out, void* stream)
{
	if (n < 0 || !out || (n > 0 && !gm)) return grav::record_error(GRAV_E_ARG, "NULL pointer or n < 0");
	cudaStream_t st = static_cast<cudaStream_t>(stream);
	cudaError_t e = cudaMemsetAsync(out, 0, 2 * sizeof(double), st);
	if (e == cudaSuccess && n > 0) {
		const int64_t blocks = (n + grav::LD_T - 1) / grav::LD_T;
		grav::gm_range_kernel<<<static_cast<unsigned>(blocks < 608 ? blocks : 608), grav::LD_T, 0, st>>>(gm, n,
			reinterpret_cast<unsigned long long*>(out));
		e = cudaGetLastError();
	}
	return e == cudaSuccess ? GRAV_OK : grav::record_error(GRAV_E_CUDA, cudaGetErrorString(e));
}

extern "C" int grav_load_state(const double* r, const double* v, const double* gm, int64_t n,
	double* r4, double* v4, void* stream)
{
	if (n < 0 || (n > 0 && (!r || !v || !gm || !r4 || !v4)))
		return grav::record_error(GRAV_E_ARG, "NULL pointer or n < 0");
	if (n == 0) return GRAV_OK;
	if (4 * n / grav::LD_T >= INT32_MAX) return grav::record_error(GRAV_E_SIZE, "too many bodies");
	const unsigned blocks = static_cast<unsigned>((4 * n + grav::LD_T - 1) / grav::LD_T);
	grav::load_state_kernel<<<blocks, grav::LD_T, 0, static_cast<cudaStream_t>(stream)>>>(r, v, gm, n, r4, v4);
	const cudaError_t e = cudaGetLastError();
	return e == cudaSuccess ? GRAV_OK : grav::record_error(GRAV_E_CUDA, cudaGetErrorString(e));
}
