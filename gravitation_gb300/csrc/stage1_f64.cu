// stage1_f64.cu -- stage 1 in GRAV_MODE_FP64 (ordered pairs) and GRAV_MODE_FP64U (unique
// pairs).
//
// Same persistent stream-K decomposition and bulk-copy pipeline as stage1_f32.cu and
// stage1_sym.cu, with FP64 positions (x, y, z, G*m) in the tiles and FP64 arithmetic
// throughout:
//     d = r_j - r_i ;  r2 = |d|^2 ;  w = Gm_j / r2^(3/2) (0 when r2 == 0) ;  a += w d
// which is the reference's law (np1.py:81-95, py1.py:57-64) in double precision.
//
// What bounds it: each of an SM's four FP64 pipes takes a warp instruction every ~67 cycles, so
// the number of FP64 instructions per pair is the time, one warp fills its pipe, and loads,
// shuffles and integer work are free beside them.  r2^(-3/2) takes six (inv_cube) on top of
// the SFU's approximation, a pair 16 in rows alone and 20 with both bodies' sums: 10 per
// interaction on unique pairs, against 18 with the library's reciprocal square root on
// ordered pairs.  The pipe is 89 % busy at 8191 bodies, whose step takes 1.25 ms (2.19 before);
// at 1000 bodies 84 -> 29 us, at 300 bodies 90 -> 12.5 us.
#include "grav_device.cuh"

namespace grav {

struct __align__(32) dpos4 {
	double x, y, z, w;
};

template <int B, int T, int J>
__global__ void __launch_bounds__(T) stage1_f64_kernel(const grav_batch b)
{
	constexpr int IT = B * T;
	constexpr uint32_t TILE_BYTES = J * sizeof(dpos4);
	extern __shared__ __align__(128) dpos4 smem_dtiles[];  // [2][J]
	__shared__ __align__(8) uint64_t bar[2];

	const int tid = threadIdx.x;
	const int64_t U = b.n_units;
	const int64_t G = gridDim.x;
	const int64_t c = blockIdx.x;
	int64_t ub = c * U / G;
	const int64_t ue = (c + 1) * U / G;
	if (ub >= ue) return;

	if (tid == 0) {
		mbar_init(&bar[0], 1);
		mbar_init(&bar[1], 1);
		fence_barrier_init();
	}
	__syncthreads();

	const dpos4* __restrict__ pos = static_cast<const dpos4*>(b.pos);

	int s = find_segment(b.seg, b.n_seg, ub);
	// positions and partial-sum slots belong to the kernels before this one
	grid_dep_wait();

	uint32_t gt = 0;
	bool timed_out = false;

	while (ub < ue && s < b.n_seg) {
		const grav_seg_desc S = b.seg[s];
		if (S.n_units == 0 || S.unit_begin + S.n_units <= ub) {
			++s;
			continue;
		}
		const grav_univ_desc Uu = b.univ[S.u];
		const int64_t jt0 = ub - S.unit_begin;
		const int64_t jt1 = min(ue - S.unit_begin, (int64_t)S.n_units);
		const int nt = static_cast<int>(jt1 - jt0);
		const int64_t ibase = Uu.pad_off + S.il0;
		const dpos4* __restrict__ jsrc = pos + Uu.pad_off;

		if (tid == 0) {
			const int bs = gt & 1;
			mbar_arrive_expect_tx(&bar[bs], TILE_BYTES);
			bulk_g2s(smem_dtiles + bs * J, jsrc + jt0 * J, TILE_BYTES, &bar[bs]);
		}

		double xi[B], yi[B], zi[B], ax[B], ay[B], az[B];
#pragma unroll
		for (int k = 0; k < B; ++k) {
			const dpos4 p = pos[ibase + tid + k * T];
			xi[k] = p.x;
			yi[k] = p.y;
			zi[k] = p.z;
			ax[k] = ay[k] = az[k] = 0.0;
		}

		for (int t = 0; t < nt; ++t, ++gt) {
			const int bs = gt & 1;
			const bool ok = mbar_wait_bounded(&bar[bs], (gt >> 1) & 1);
			if (__syncthreads_or(!ok)) {
				timed_out = true;
				break;
			}
			if (tid == 0 && t + 1 < nt) {
				const int bn = (gt + 1) & 1;
				mbar_arrive_expect_tx(&bar[bn], TILE_BYTES);
				bulk_g2s(smem_dtiles + bn * J, jsrc + (jt0 + t + 1) * J, TILE_BYTES, &bar[bn]);
			}
			const dpos4* __restrict__ sj = smem_dtiles + bs * J;
#pragma unroll 2
			for (int j = 0; j < J; ++j) {
				const dpos4 pj = sj[j];
#pragma unroll
				for (int k = 0; k < B; ++k) {
					const double dx = pj.x - xi[k];
					const double dy = pj.y - yi[k];
					const double dz = pj.z - zi[k];
					const double r2 = dx * dx + dy * dy + dz * dz;
					const double w = pj.w * inv_cube(r2);
					ax[k] += w * dx;
					ay[k] += w * dy;
					az[k] += w * dz;
				}
			}
		}
		if (timed_out) break;

		const int64_t slot = S.slot_base + (c - S.cta_first);
		double* __restrict__ out = b.part + slot * 3 * IT;
#pragma unroll
		for (int k = 0; k < B; ++k) {
			out[tid + k * T] = ax[k];
			out[IT + tid + k * T] = ay[k];
			out[2 * IT + tid + k * T] = az[k];
		}
		ub = S.unit_begin + jt1;
		++s;
	}

	// the next kernel in the stream may start launching now (it waits for this grid)
	grid_dep_launch();
	if (timed_out && tid == 0) {
		set_error(b.err, GRAV_DEV_TIMEOUT);
		mbar_wait_bounded(&bar[gt & 1], (gt >> 1) & 1);
	}
}

// Whether a pair takes the cold path: out of inv_cube's range and not at zero separation.
__device__ __forceinline__ bool out_of_range(double r2, bool in_range)
{
	return !in_range && (__double2hiint(r2) | __double2loint(r2)) != 0;
}

// Unique pairs (plan of grav_plan_pairs; the scheme of stage1_sym.cu): row blocks of R = 32,
// 64 or 128 rows and j-tiles of 32 bodies.  A CTA is four warps, one per FP64 pipe: warp w
// holds the 32 rows w mod (R / 32) of the block and takes an equal part of the 32 steps, so a
// 32-row block also keeps the whole SM busy (with one warp per 32 rows a unit of 32 x 32
// pairs took 22 us, here 5 us) and the units are fine enough to balance.  A tile of the block
// itself is done as ordered pairs, rows only; one of a later block on unique pairs, lane l
// meeting body (l + s) mod 32 at step s while the tile's column sums rotate one lane per
// step.  The warps' column sums are added in order and go, as FP64, to the column slot of
// (I, J); the step parts' row sums likewise at the end of a piece.
template <int RG>
__global__ void __launch_bounds__(128) stage1_f64_pairs_kernel(const grav_batch b)
{
	constexpr int W = 4, T = 32 * W, R = 32 * RG, TPB = RG, JT = 32;
	constexpr int PARTS = W / RG, STEPS = 32 / PARTS;   // step parts, steps per part
	constexpr uint32_t TILE_BYTES = JT * sizeof(dpos4);
	__shared__ __align__(128) dpos4 tiles[2][JT];
	__shared__ double colacc[W][3][JT];
	__shared__ double rowacc[PARTS][3][R];
	__shared__ __align__(8) uint64_t bar[2];

	const int tid = threadIdx.x;
	const int lane = tid & 31;
	const int warp = tid >> 5;
	const int row = (warp % RG) * 32 + lane;      // this thread's row of the block
	const int part = warp / RG, s0 = part * STEPS;
	const int64_t U = b.n_units;
	const int64_t G = gridDim.x;
	const int64_t c = blockIdx.x;
	int64_t ub = c * U / G;
	const int64_t ue = (c + 1) * U / G;
	if (ub >= ue) return;

	if (tid == 0) {
		mbar_init(&bar[0], 1);
		mbar_init(&bar[1], 1);
		fence_barrier_init();
	}
	__syncthreads();

	const dpos4* __restrict__ pos = static_cast<const dpos4*>(b.pos);
	int s = find_segment(b.seg, b.n_seg, ub);
	// positions and partial-sum slots belong to the kernels before this one
	grid_dep_wait();

	uint32_t gt = 0;
	bool timed_out = false;
	while (ub < ue && s < b.n_seg) {
		const grav_seg_desc S = b.seg[s];
		if (S.n_units == 0 || S.unit_begin + S.n_units <= ub) {
			++s;
			continue;
		}
		const grav_univ_desc Uu = b.univ[S.u];
		const int blkI = S.il0 / R;
		const int64_t t0 = ub - S.unit_begin;
		const int64_t t1 = min(ue - S.unit_begin, (int64_t)S.n_units);
		const int nt = static_cast<int>(t1 - t0);
		const int64_t jt_first = static_cast<int64_t>(blkI) * TPB + t0;
		const dpos4* __restrict__ jsrc = pos + Uu.pad_off;

		if (tid == 0) {
			const int bs = gt & 1;
			mbar_arrive_expect_tx(&bar[bs], TILE_BYTES);
			bulk_g2s(tiles[bs], jsrc + jt_first * JT, TILE_BYTES, &bar[bs]);
		}
		const dpos4 pi = pos[Uu.pad_off + S.il0 + row];
		double ax = 0.0, ay = 0.0, az = 0.0;

		for (int t = 0; t < nt; ++t, ++gt) {
			const int bs = gt & 1;
			const bool ok = mbar_wait_bounded(&bar[bs], (gt >> 1) & 1);
			if (__syncthreads_or(!ok)) {
				timed_out = true;
				break;
			}
			const int64_t jt = jt_first + t;
			if (tid == 0 && t + 1 < nt) {
				const int bn = (gt + 1) & 1;
				mbar_arrive_expect_tx(&bar[bn], TILE_BYTES);
				bulk_g2s(tiles[bn], jsrc + (jt + 1) * JT, TILE_BYTES, &bar[bn]);
			}
			const dpos4* __restrict__ sc = tiles[bs];
			const int blkJ = static_cast<int>(jt / TPB);
			uint32_t slow = 0;   // steps whose separation is out of the fast range
			if (blkJ == blkI) {
#pragma unroll 4
				for (int st = 0; st < STEPS; ++st) {
					const dpos4 pj = sc[s0 + st];
					const double dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
					const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
					bool in_range;
					const double w = pj.w * inv_cube(r2, in_range);
					slow |= out_of_range(r2, in_range) ? 1u << st : 0u;
					ax = fma(w, dx, ax);
					ay = fma(w, dy, ay);
					az = fma(w, dz, az);
				}
				for (; slow; slow &= slow - 1) {
					const dpos4 pj = sc[s0 + __ffs(slow) - 1];
					const double dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
					const double w = pj.w * inv_cube(fma(dz, dz, fma(dy, dy, dx * dx)));
					ax = fma(w, dx, ax);
					ay = fma(w, dy, ay);
					az = fma(w, dz, az);
				}
			} else {
				double cx = 0.0, cy = 0.0, cz = 0.0;   // of body (lane + s0 + st) mod 32
#pragma unroll 4
				for (int st = 0; st < STEPS; ++st) {
					const dpos4 pj = sc[(lane + s0 + st) & 31];
					const double dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
					const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
					bool in_range;
					const double inv3 = inv_cube(r2, in_range);
					slow |= out_of_range(r2, in_range) ? 1u << st : 0u;
					const double wj = pj.w * inv3, wi = pi.w * inv3;
					ax = fma(wj, dx, ax);
					ay = fma(wj, dy, ay);
					az = fma(wj, dz, az);
					cx = fma(-wi, dx, cx);
					cy = fma(-wi, dy, cy);
					cz = fma(-wi, dz, cz);
					const int src = (lane + 1) & 31;
					cx = __shfl_sync(0xffffffffu, cx, src);
					cy = __shfl_sync(0xffffffffu, cy, src);
					cz = __shfl_sync(0xffffffffu, cz, src);
				}
				// the pairs out of range, which contributed nothing above: step st met body
				// (lane + s0 + st) mod 32, whose sum lane (lane + st - STEPS) mod 32 now holds
				for (uint32_t todo = __reduce_or_sync(0xffffffffu, slow); todo; todo &= todo - 1) {
					const int st = __ffs(todo) - 1;
					const dpos4 pj = sc[(lane + s0 + st) & 31];
					const double dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
					const bool mine = slow >> st & 1u;
					const double inv3 = mine ? inv_cube(fma(dz, dz, fma(dy, dy, dx * dx))) : 0.0;
					const double wj = pj.w * inv3, wi = pi.w * inv3;
					if (mine) {
						ax = fma(wj, dx, ax);
						ay = fma(wj, dy, ay);
						az = fma(wj, dz, az);
					}
					const int from = (lane - st + STEPS) & 31;
					cx += __shfl_sync(0xffffffffu, mine ? -wi * dx : 0.0, from);
					cy += __shfl_sync(0xffffffffu, mine ? -wi * dy : 0.0, from);
					cz += __shfl_sync(0xffffffffu, mine ? -wi * dz : 0.0, from);
				}
				const int body = (lane + s0 + STEPS) & 31;
				colacc[warp][0][body] = cx;
				colacc[warp][1][body] = cy;
				colacc[warp][2][body] = cz;
				__syncthreads();
				const grav_seg_desc SJ = b.seg[s + (blkJ - blkI)];
				const int64_t slot = SJ.slot_base + SJ.nslots - (blkJ - blkI);
				double* __restrict__ out = b.part + slot * 3 * R + (jt * JT - static_cast<int64_t>(blkJ) * R);
				if (warp < 3) {
					double sum = colacc[0][warp][lane];
#pragma unroll
					for (int w = 1; w < W; ++w) sum += colacc[w][warp][lane];
					out[warp * R + lane] = sum;
				}
			}
		}
		if (timed_out) break;

		rowacc[part][0][row] = ax;
		rowacc[part][1][row] = ay;
		rowacc[part][2][row] = az;
		__syncthreads();
		const int64_t slot = S.slot_base + (c - S.cta_first);
		double* __restrict__ out = b.part + slot * 3 * R;
		for (int i = tid; i < 3 * R; i += T) {
			double sum = rowacc[0][i / R][i % R];
#pragma unroll
			for (int p = 1; p < PARTS; ++p) sum += rowacc[p][i / R][i % R];
			out[i] = sum;
		}
		ub = S.unit_begin + t1;
		++s;
	}

	// the next kernel in the stream may start launching now (it waits for this grid)
	grid_dep_launch();
	if (timed_out && tid == 0) {
		set_error(b.err, GRAV_DEV_TIMEOUT);
		mbar_wait_bounded(&bar[gt & 1], (gt >> 1) & 1);
	}
}

#define GRAV_F64_ENTRY(B, T, J) \
	{GRAV_MODE_FP64, B, T, J, reinterpret_cast<const void*>(&stage1_f64_kernel<B, T, J>), \
		2 * J * 32, true}
#define GRAV_F64U_ENTRY(RG) \
	{GRAV_MODE_FP64U, 1, 32 * RG, 32, reinterpret_cast<const void*>(&stage1_f64_pairs_kernel<RG>), \
		0, true, 128}

static const Stage1Kernel k_table_f64[] = {
	GRAV_F64_ENTRY(1, 128, 128),
	GRAV_F64_ENTRY(2, 128, 128),
	GRAV_F64_ENTRY(1, 256, 128),
	GRAV_F64_ENTRY(2, 256, 128),
	GRAV_F64U_ENTRY(1),
	GRAV_F64U_ENTRY(2),
	GRAV_F64U_ENTRY(4),
};

int stage1_table_f64(const Stage1Kernel** out)
{
	*out = k_table_f64;
	return static_cast<int>(sizeof(k_table_f64) / sizeof(k_table_f64[0]));
}

}  // namespace grav
