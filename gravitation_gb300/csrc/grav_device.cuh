// grav_device.cuh -- device-side helpers shared by the GB300 n-body kernels.
//
// Inline PTX for the SFU reciprocal square root, mbarrier waits with a time limit,
// and 1-D bulk (TMA) copies global -> shared.  Every spin-wait here is bounded:
// when the limit is reached the caller records an error code in device memory and
// returns, so that a lost copy never hangs the GPU.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "grav_types.h"

namespace grav {

// SFU reciprocal square root (MUFU), flush-to-zero.  For r2 > 0 normal inputs the
// result is within a few ulp of 1/sqrt(r2); the kernels guard r2 >= eps2 > 0.
__device__ __forceinline__ float rsqrt_sfu(float x)
{
	float y;
	asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
	return y;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
	return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}

// Make the initialised barriers visible to the async (TMA) proxy.
__device__ __forceinline__ void fence_barrier_init()
{
	asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async()
{
	asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
		"r"(bytes)
		: "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
	uint32_t ok;
	asm volatile(
		"{\n\t.reg .pred p;\n\t"
		"mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
		"selp.u32 %0, 1, 0, p;\n\t}"
		: "=r"(ok)
		: "r"(smem_addr(bar)), "r"(parity)
		: "memory");
	return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns()
{
	uint64_t t;
	asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
	return t;
}

// Bounded wait on one phase of an mbarrier.  Returns false when the phase has not
// completed after GRAV_WAIT_NS nanoseconds of polling (the clock is read every 16
// polls, so the bound holds whatever each poll's hardware suspend time is).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity,
	uint64_t limit_ns = GRAV_WAIT_NS)
{
	if (mbar_try_wait(bar, parity)) return true;
	const uint64_t t0 = global_ns();
	for (;;) {
		for (int k = 0; k < 16; ++k)
			if (mbar_try_wait(bar, parity)) return true;
		if (global_ns() - t0 > limit_ns) return false;
	}
}

// 1-D bulk copy of `bytes` (multiple of 16, both addresses 16-byte aligned) from
// global to this CTA's shared memory, completing on `bar`.
__device__ __forceinline__ void bulk_g2s(void* dst_smem, const void* src_gmem, uint32_t bytes,
	uint64_t* bar)
{
	asm volatile(
		"cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
		::"r"(smem_addr(dst_smem)), "l"(src_gmem), "r"(bytes), "r"(smem_addr(bar))
		: "memory");
}

// Packed FP32 (sm_100 and later): two independent lanes' values in one aligned register
// pair, each half rounded as the scalar instruction rounds it.  fma/add/mul.f32x2 do the
// FMA pipe's work of two scalar instructions in one issue slot, which is what limits the
// pair loops.  Kept as 64-bit integers so that the halves stay in register pairs.
typedef unsigned long long u64;

__device__ __forceinline__ u64 pack2(float a, float b)
{
	u64 r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
	return r;
}

__device__ __forceinline__ void unpack2(u64 v, float& a, float& b)
{
	asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}

__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c)
{
	u64 r;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
	return r;
}

__device__ __forceinline__ u64 mul2(u64 a, u64 b)
{
	u64 r;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}

__device__ __forceinline__ u64 add2(u64 a, u64 b)
{
	u64 r;
	asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}

// A row's position by four 32-bit loads.  Values that two rows' packed pairs are made of
// must not come from one 128-bit load: the compiler then keeps the loaded quad and forms
// the pairs again by register moves at every step of the pair loop (4 moves per pair
// measured, 1.38 against 1.17 ms per stage 1 at 65536 bodies).
__device__ __forceinline__ float4 load_row(const float4* p)
{
	float4 r;
	asm volatile("ld.global.f32 %0, [%1];" : "=f"(r.x) : "l"(p));
	asm volatile("ld.global.f32 %0, [%1+4];" : "=f"(r.y) : "l"(p));
	asm volatile("ld.global.f32 %0, [%1+8];" : "=f"(r.z) : "l"(p));
	asm volatile("ld.global.f32 %0, [%1+12];" : "=f"(r.w) : "l"(p));
	return r;
}

// Compensated accumulation (Knuth's TwoSum, "The Art of Computer Programming" vol. 2,
// 4.2.2): hi + lo is the running sum; the rounding error of hi + x is kept exactly and
// added to lo.  Six FP32 additions; no FP64 (which runs at ~1/75 of the FP32 rate on
// this GPU).  Used to fold FP32 tile partials into a ~48-bit per-body sum.
__device__ __forceinline__ void two_sum_acc(float& hi, float& lo, float x)
{
	const float s = hi + x;
	const float bp = s - hi;
	const float e = (hi - (s - bp)) + (x - bp);
	hi = s;
	lo += e;
}

// r2^(-3/2) in FP64 without the library's reciprocal square root, for exponents of r2 in
// 2^-598 .. 2^1023 (else `in_range` is false and the result 0).  y, the SFU's approximation of
// r2^(-1/2) (rsqrt.approx.ftz.f64, computed from the high word, its low word zero), leaves e =
// 1 - r2 y^2 below 2^-19, formed with one rounding of its own size; r2^(-3/2) = y^3 (1 -
// e)^(-3/2) = y^3 (1 + 3/2 e + 15/8 e^2 + O(2^-56)), the binomial series: six FP64
// instructions, no branch.
__device__ __forceinline__ double inv_cube(double r2, bool& in_range)
{
	in_range = static_cast<uint32_t>(__double2hiint(r2)) - 0x1a900000u < 0x65500000u;
	double y;
	asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2));
	const double t = y * y;
	const double e = fma(-r2, t, 1.0);
	const double y3 = y * t;
	const double f = fma(y3 * e, fma(1.875, e, 1.5), y3);
	// selected as words: a floating-point select would be an FP64 instruction
	return __hiloint2double(in_range ? __double2hiint(f) : 0, in_range ? __double2loint(f) : 0);
}

// The same for any r2 >= 0 (0 at 0): outside the range by the library's function.
__device__ __forceinline__ double inv_cube(double r2)
{
	bool in_range;
	const double f = inv_cube(r2, in_range);
	if (in_range) return f;
	const double inv = r2 > 0.0 ? rsqrt(r2) : 0.0;
	return inv * inv * inv;
}

// r2^(-1/2), 0 at r2 = 0, by the same series: y (1 + 1/2 e + 3/8 e^2); five FP64 instructions.
__device__ __forceinline__ double inv_root(double r2)
{
	if (static_cast<uint32_t>(__double2hiint(r2)) - 0x1a900000u < 0x65500000u) {
		double y;
		asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2));
		const double e = fma(-r2, y * y, 1.0);
		return fma(y * e, fma(0.375, e, 0.5), y);
	}
	return r2 > 0.0 ? rsqrt(r2) : 0.0;
}

// Programmatic dependent launch.  A kernel launched with programmatic stream
// serialization may start while the kernel before it in the stream is still running:
// grid_dep_wait() blocks until that kernel has completed and its memory operations are
// visible, so everything before it may only read data no earlier kernel writes (plan
// tables, launch arguments).  grid_dep_launch() lets the next kernel in the stream
// start its own launch.  Both are no-ops for a kernel launched the ordinary way.
__device__ __forceinline__ void grid_dep_wait()
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ void grid_dep_launch()
{
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Near-pair correction (GRAV_MODE_FP32N / GRAV_MODE_FP32UN).  Rounding a coordinate x
// to FP32 moves it by up to 2^-24 |x|, so the FP32 separation of two bodies far from the
// origin but close to each other carries a relative error of order 2^-24 |x| / |d|.
// The near modes evaluate every pair with r2 < near_threshold() (|d| below
// max|x| / GRAV_NEAR_KAPPA, max|x| over the coordinates of the thread's rows) a second
// time from the double-single separation d_a = (hi_j - hi_i) + (lo_j - lo_i) and add the
// difference.  Beyond that distance the FP32 separation is within
// 2^-24 (sqrt(3) (2 kappa + 1) + 1) of the exact one (~4.5e-6 relative pair-force error
// at kappa = 20, a bound; measured body errors stay below 1e-6).
// Padding rows of the near modes sit at (FAR, FAR, FAR) with Gm = 0: no contribution, as at the
// origin, but never within a near radius.  At the origin one body near it met every padding
// column of its universe on the correction path (fp32n at 3600 bodies 31 us per step against
// 14).  A thread's radius leaves its padding rows out.
constexpr float FAR_PAD = 1e18f;

__device__ __forceinline__ float near_scale(float x, float y, float z)
{
	return fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z)));
}

__device__ __forceinline__ float near_threshold(float max_abs_coord)
{
	constexpr float inv_k2 = 1.0f / (GRAV_NEAR_KAPPA * GRAV_NEAR_KAPPA);
	return max_abs_coord * max_abs_coord * inv_k2;
}

// The scale (largest |coordinate|) whose near radius a thread's rows share, so that one minimum
// per step tests them all: the largest of the first `real` rows', unless half of them or more are
// nearer the origin than the outermost by a factor of 8 (of 16 with few rows, which meet 8 by
// chance).  With the radius of such a row, a body that escaped, the others would meet
// near pairs everywhere (fp32un at 65536 bodies, one of them 1000 times farther out: 7.8 ms a
// step against 1.3); it is left out and the warp tests every row against its own radius.  Given
// squares (radii squared), FACTOR is the factor's square.
template <int B, int FACTOR = B <= 4 ? 16 : 8>
__device__ __forceinline__ float common_scale(const float (&scale)[B], int real)
{
	constexpr float FAR = FACTOR;
	float xmax = 3e38f;
	for (int i = 0; i < B; ++i) {   // each round leaves one more row out
		float top = 0.f;
		int far = 0;
#pragma unroll
		for (int k = 0; k < B; ++k)
			if (scale[k] <= xmax) top = fmaxf(top, scale[k]);
		xmax = top;
#pragma unroll
		for (int k = 0; k < B; ++k) far += FAR * scale[k] > xmax;
		if (2 * far > real || far >= real || xmax == 0.f || i == B - 1) break;
		xmax *= 1.f / FAR;
	}
	return xmax;
}

// Three-input minimum (min.f32 with three operands, sm_100 and later).
__device__ __forceinline__ float min3f(float a, float b, float c)
{
	float r;
	asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
	return r;
}

// Running minimum of the r2 values of a thread's B rows for the near test, one
// three-input min per two rows: call with k = 0 .. B-1 in order; `prev` holds the previous
// row's r2 between calls.
template <int B>
__device__ __forceinline__ void near_min_step(int k, float r2, float& m, float& prev)
{
	if (k == 0) m = r2;
	else if ((k & 1) == 0) m = min3f(m, prev, r2);
	else if (k == B - 1) m = fminf(m, r2);
	prev = r2;
}

// (ex, ey, ez) = d_a |d_a|^-3 - d |d|^-3 for the pair whose FP32 separation is (dx, dy,
// dz) with r2 = |d|^2 + eps2 (as the main loop formed it), lj / li the low parts of the
// column and row bodies; zero unless `on`.  The caller adds Gm_j e to the row's sum and
// -Gm_i e to the column's, which replaces the FP32 pair term by the double-single one.
__device__ __forceinline__ void near_delta(float dx, float dy, float dz, float r2,
	const float4& lj, const float4& li, float eps2, bool on, float& ex, float& ey, float& ez)
{
	const float ax = dx + (lj.x - li.x);
	const float ay = dy + (lj.y - li.y);
	const float az = dz + (lj.z - li.z);
	const float ra2 = fmaf(az, az, fmaf(ay, ay, fmaf(ax, ax, eps2)));
	const float ia = rsqrt_sfu(ra2);
	const float ia3 = ia * (ia * ia);
	const float i1 = rsqrt_sfu(r2);
	const float i3 = i1 * (i1 * i1);
	ex = on ? fmaf(ax, ia3, -(dx * i3)) : 0.f;
	ey = on ? fmaf(ay, ia3, -(dy * i3)) : 0.f;
	ez = on ? fmaf(az, ia3, -(dz * i3)) : 0.f;
}

// One j-tile against a thread's B rows, every ordered pair, rows only: the inner loop
// of the all-pairs kernel (stage1_f32.cu); rowlo[k * T + tid] holds the rows' low parts and near
// radii squared.  NEAR adds the near test (one three-input min per two rows and a compare with
// thr, the radius the rows share; with SELF -- tiles that hold the thread block's own rows, and
// warps with rows of another radius -- a test per pair that also excludes r2 = eps2, so that
// self pairs do not count) whose result is a bit per step, and after every 32 steps a cold
// path over the steps where some lane of the warp met a near pair, all rows of all lanes side
// by side (a vote per row to skip those without is slower: fp32n 4/128/128 at 16384 bodies
// 148.8 -> 141.4 us, two Plummer spheres 361 -> 344 us a step).
template <int B, int JT, bool DS, bool NEAR, bool SELF>
__device__ __forceinline__ void rows_tile(const float4* __restrict__ sj,
	const float4* __restrict__ sjl, float eps2, float thr, const float (&xi)[B],
	const float (&yi)[B], const float (&zi)[B], const float (&xl)[B], const float (&yl)[B],
	const float (&zl)[B], float (&fx)[B], float (&fy)[B], float (&fz)[B],
	const float4* __restrict__ rowlo, int tid, int T)
{
	static_assert(JT % 32 == 0, "j-tiles of whole 32-body groups");
	float radius2[B];   // SELF: the rows' near radii squared
#pragma unroll
	for (int k = 0; k < B; ++k) radius2[k] = NEAR && SELF && B > 1 ? rowlo[k * T + tid].w : thr;
#pragma unroll 1
	for (int j0 = 0; j0 < JT; j0 += 32) {
		uint32_t nmask = 0;
#pragma unroll 4
		for (int jj = 0; jj < 32; ++jj) {
			const float4 pj = sj[j0 + jj];
			float4 lj = make_float4(0.f, 0.f, 0.f, 0.f);
			if (DS) lj = sjl[j0 + jj];
			float rmin = 0.f, rprev = 0.f;
			bool near = false;
#pragma unroll
			for (int k = 0; k < B; ++k) {
				float dx = pj.x - xi[k], dy = pj.y - yi[k], dz = pj.z - zi[k];
				if (DS) {
					dx = dx + (lj.x - xl[k]);
					dy = dy + (lj.y - yl[k]);
					dz = dz + (lj.z - zl[k]);
				}
				const float r2 = fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, eps2)));
				if (NEAR && SELF) near |= (r2 < radius2[k]) & (r2 > eps2);
				if (NEAR && !SELF) near_min_step<B>(k, r2, rmin, rprev);
				const float inv = rsqrt_sfu(r2);
				float w = pj.w * inv;
				w = w * (inv * inv);
				fx[k] = fmaf(dx, w, fx[k]);
				fy[k] = fmaf(dy, w, fy[k]);
				fz[k] = fmaf(dz, w, fz[k]);
			}
			if (NEAR && !SELF) near = rmin < thr;
			if (NEAR && near) nmask |= 1u << jj;
		}
		if (NEAR) {
			uint32_t todo = __reduce_or_sync(0xffffffffu, nmask);
			while (todo) {
				const int jj = __ffs(todo) - 1;
				todo &= todo - 1;
				const float4 pj = sj[j0 + jj];
				const float4 lj = sjl[j0 + jj];
#pragma unroll
				for (int k = 0; k < B; ++k) {
					const float dx = pj.x - xi[k], dy = pj.y - yi[k], dz = pj.z - zi[k];
					const float r2 = fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, eps2)));
					const float4 li = rowlo[k * T + tid];
					const bool nk = (r2 < (B > 1 ? li.w : thr)) & (r2 > eps2);
					float ex, ey, ez;
					near_delta(dx, dy, dz, r2, lj, li, eps2, nk, ex, ey, ez);
					fx[k] = fmaf(ex, pj.w, fx[k]);
					fy[k] = fmaf(ey, pj.w, fy[k]);
					fz[k] = fmaf(ez, pj.w, fz[k]);
				}
			}
		}
	}
}

// Combine the compensated FP32 sums (H, L) of the WIDTH lanes of an aligned lane group
// by an xor butterfly: H by TwoSum, L and the rounding error added.  Every lane ends
// with the same bits: TwoSum's error term is the exact rounding error of H_a + H_b in
// either operand order, and FP32 addition commutes.
template <int WIDTH>
__device__ __forceinline__ void group_sum_pair(float& H, float& L, unsigned mask)
{
#pragma unroll
	for (int o = 1; o < WIDTH; o <<= 1) {
		const float hb = __shfl_xor_sync(mask, H, o);
		const float lb = __shfl_xor_sync(mask, L, o);
		const float s = H + hb;
		const float bp = s - H;
		const float e = (H - (s - bp)) + (hb - bp);
		H = s;
		L = (L + lb) + e;
	}
}

// Record the first error code seen by any CTA.
__device__ __forceinline__ void set_error(int* err, int code)
{
	if (err) atomicCAS(err, 0, code);
}

// Index of the last plan segment whose unit_begin <= ub (unit_begin never decreases
// along the table and seg[0].unit_begin = 0 <= ub).  Each warp searches on its own:
// per round its 32 lanes probe 32 evenly spaced candidates and a ballot keeps the
// interval between the last candidate that qualifies and the next one, so the search
// takes ceil(log32(n_seg)) rounds of independent loads where a bisection takes
// log2(n_seg) dependent ones.  All 32 lanes of the warp must call it together.
__device__ __forceinline__ int find_segment(const grav_seg_desc* seg, int n_seg, int64_t ub)
{
	const unsigned full = 0xffffffffu;
	const int lane = threadIdx.x & 31;
	int lo = 0, hi = n_seg - 1;
	while (lo < hi) {
		const int span = hi - lo + 1;  // candidates left, >= 2
		const int idx = span <= 32 ? lo + min(lane, span - 1)
		                           : lo + static_cast<int>((static_cast<int64_t>(lane) * span) / 32);
		const unsigned ok = __ballot_sync(full, seg[idx].unit_begin <= ub);  // lane 0 qualifies
		const int top = 31 - __clz(ok);
		const int at = __shfl_sync(full, idx, top);
		const int after = __shfl_sync(full, idx, (top + 1) & 31);
		if (span <= 32) return at;
		hi = top < 31 ? after - 1 : hi;
		lo = at;
	}
	return lo;
}

}  // namespace grav
