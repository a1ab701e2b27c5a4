// exchange.cuh -- tagged 128-bit words between the CTAs of one launch (steps.cu,
// adjoint_steps.cu), and the launch that puts CTAs which wait on one another on the GPU
// together (those, and fused.cu).
#pragma once
#include "grav_device.cuh"

namespace grav {

constexpr unsigned EXCHANGE_CLUSTER_MAX = 16;      // CTAs of a cluster (non-portable size)
constexpr unsigned EXCHANGE_CLUSTER_PORTABLE = 8;

// Head of the scratch buffer; the words follow at EXCHANGE_HEAD_BYTES.
struct ExchangeHead {
	uint32_t epoch;     // tags used so far
	int32_t departed;   // CTAs done with the launch
};
constexpr int EXCHANGE_HEAD_BYTES = 128;

typedef unsigned __int128 u128;

__device__ __forceinline__ u128 load_word(const void* p)
{
	u128 v;
	asm volatile("ld.relaxed.gpu.global.b128 %0, [%1];" : "=q"(v) : "l"(p) : "memory");
	return v;
}

__device__ __forceinline__ void store_word(void* p, float x, float y, float z, uint32_t tag)
{
	const u64 lo = static_cast<u64>(__float_as_uint(y)) << 32 | __float_as_uint(x);
	const u64 hi = static_cast<u64>(tag) << 32 | __float_as_uint(z);
	const u128 v = static_cast<u128>(hi) << 64 | lo;
	asm volatile("st.relaxed.gpu.global.b128 [%0], %1;" ::"l"(p), "q"(v) : "memory");
}

__device__ __forceinline__ uint32_t word_tag(u128 v) { return static_cast<uint32_t>(v >> 96); }

__device__ __forceinline__ float4 word_position(u128 v)
{
	return make_float4(__uint_as_float(static_cast<uint32_t>(v)),
		__uint_as_float(static_cast<uint32_t>(v >> 32)),
		__uint_as_float(static_cast<uint32_t>(v >> 64)), 0.f);
}

// Poll one published position until its tag is `tag`; false when the bounded wait expired.  A
// caller that goes on after that gives a word of shared memory, zero at first: once a wait with
// it has expired, the CTA's others with it end at once.  (The position loops, which stop at
// their first expired wait, do without: the test costs them 2 % at 4096 bodies.)
__device__ __forceinline__ bool wait_word(const void* p, uint32_t tag, u128& v, int* expired = nullptr,
	uint64_t limit_ns = GRAV_WAIT_NS)
{
	if (word_tag(v) == tag) return true;
	const uint64_t t0 = global_ns();
	for (;;) {
		for (int k = 0; k < 64; ++k) {
			v = load_word(p);
			if (word_tag(v) == tag) return true;
		}
		if (expired && *const_cast<volatile int*>(expired)) return false;
		if (global_ns() - t0 > limit_ns) {
			if (expired) *const_cast<volatile int*>(expired) = 1;
			return false;
		}
	}
}

// Hardware cluster barrier, split: every thread of every CTA of the cluster arrives
// (release: its earlier loads and stores are ordered before) and later waits (acquire).
__device__ __forceinline__ void cluster_arrive()
{
	asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}

__device__ __forceinline__ void cluster_wait()
{
	asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// CTAs in this CTA's thread-block cluster (1 when launched without clusters)
__device__ __forceinline__ unsigned cluster_ctas()
{
	unsigned v;
	asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(v));
	return v;
}

// Launch `grid` CTAs that exchange words.  clustered: as one thread-block cluster (launched as
// a programmatic dependent) where one holds them all; waits: they wait on one another and are
// launched cooperatively where they do not fit one cluster.
inline cudaError_t launch_exchanging(const void* fn, unsigned grid, unsigned threads, int smem,
	bool clustered, bool waits, cudaStream_t stream, void** args)
{
	cudaError_t e = ensure_smem(fn, smem);
	if (e != cudaSuccess) return e;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(grid);
	cfg.blockDim = dim3(threads);
	cfg.dynamicSmemBytes = static_cast<size_t>(smem);
	cfg.stream = stream;
	cudaLaunchAttribute attr[2];
	cfg.attrs = attr;
	cfg.numAttrs = 0;
	bool cluster = clustered && grid <= EXCHANGE_CLUSTER_MAX;
	if (cluster) {
		attr[0].id = cudaLaunchAttributeClusterDimension;
		attr[0].val.clusterDim.x = grid;
		attr[0].val.clusterDim.y = 1;
		attr[0].val.clusterDim.z = 1;
		cfg.numAttrs = 1;
		if (grid > EXCHANGE_CLUSTER_PORTABLE) {
			int fits = 0;
			e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
			if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&fits, fn, &cfg);
			if (e != cudaSuccess) {
				cudaGetLastError();  // a refused query is not sticky: fall back
				fits = 0;
			}
			cluster = fits > 0;
			if (!cluster) cfg.numAttrs = 0;
		}
	}
	if (waits && !cluster) {
		attr[0].id = cudaLaunchAttributeCooperative;
		attr[0].val.cooperative = 1;
		cfg.numAttrs = 1;
	} else {
		attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
		attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
		++cfg.numAttrs;
	}
	return cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace grav
