// stage1_sym.cu -- stage 1 over unique pairs (GRAV_MODE_FP32U, GRAV_MODE_FP32CU,
// GRAV_MODE_FP32UN).
//
// The reference's CPU kernels visit every unordered pair once and update both bodies
// (np1.py:81-95, _lib1_/lib.c:78-114, _lib4_/lib.c:244-317: a_i -= ..., a_j += ...).
// This kernel does the same on the GPU, which removes a third of the FMA-pipe work of
// the all-pairs kernel (16 instead of 2 x 12 FMA-pipe operations per pair).  Arithmetic
// per pair is the FP32 law of stage1_f32.cu:
//     d = r_j - r_i ; r2 = |d|^2 + eps2 ; inv3 = rsqrt(r2)^3
//     a_i += (Gm_j inv3) d ;  a_j -= (Gm_i inv3) d
//
// Decomposition (plan: grav_plan_pairs).  Each universe is cut into row blocks of R =
// 32 * W * B bodies (one segment each); the work units of row block I are the j-tiles
// (JT bodies) of blocks J >= I.  A j-tile inside block I itself is done "all pairs,
// rows only" (every ordered pair of the block once, like stage1_f32.cu); a j-tile of a
// block J > I is done on unique pairs: warp w holds 32 x B rows of block I, and for
// each 32-body chunk of the tile, lane l meets body (l + s) mod 32 of the chunk at step
// s while the chunk's column sums rotate one lane per step (shfl), so after 32 steps
// every row of the warp has met every body of the chunk once and each lane holds the
// complete column sum of "its" body.  Each warp writes its column sums to its own row of
// a shared-memory buffer, and the tile's column sums (the warps added in a fixed order)
// go into the column slot of (I, J): block J's segment lists its row slots first and then
// one column slot per block I < J (its last J slots), so stage 2 adds them like any
// partial sums (fixed order: the result does not depend on scheduling).
// Row sums are FP32 per tile, folded into compensated (TwoSum) FP32 hi+lo sums, as in
// stage1_f32.cu, and go out as FP32 (hi, lo) pairs; column sums are FP32 per tile and go
// out as FP32 (the first 3R floats of the slot), which stage 2 adds by TwoSum in FP32.
//
// What bounds it, and the packed loop.  With scalar FP32 instructions the loop issued 18
// (near-corrected 22) instructions per pair for 16 of the FMA pipe and ran at 25-26 cycles
// per pair and warp: issue slots and register-port conflicts, FMA pipe 67 % busy.  Two rows
// of a thread now share every FMA-pipe instruction (f32x2: one issue slot for the pipe work
// of two; a thread's rows come in packed pairs), the j-tile is expanded in shared memory to
// (x, x) pairs so that no register move builds them, and the chunk is stored twice in a row
// so that the rotated read needs no index arithmetic: 11 (12) instructions and 21.8 (24.4)
// cycles per pair, FMA pipe 79 % (66 %) busy.  What is left is the pipe itself (16 cycles),
// the SFU's reciprocal square root (it costs the scheduler ~2 more) and, in the near mode,
// the three-input minima, whose register reads compete with the packed operands'.
// Stage 1 at 65536 bodies, best tile, scalar loop -> this one: fp32u 1.335 -> 1.155 ms,
// fp32cu 2.07 -> 1.56 ms, fp32un 1.40 -> 1.32 ms; at 16384 bodies 98 -> 82, 129 -> 118,
// 106 -> 94 us.  One barrier per j-tile: a warp that is done with tile t expands its share
// of tile t + 1 and meets the others once; the column sums of tile t leave after that.
#include <type_traits>

#include "grav_device.cuh"

namespace grav {

// KIND selects the separations:
//   SYM_PLAIN (GRAV_MODE_FP32U): FP32 positions, d = hi_j - hi_i.
//   SYM_DS    (GRAV_MODE_FP32CU): FP32 hi and lo parts of the FP64 positions,
//             d = (hi_j - hi_i) + (lo_j - lo_i), exact to FP32 relative precision however
//             far from the origin the bodies are (+6 FADD per pair).
//   SYM_NEAR  (GRAV_MODE_FP32UN): the SYM_PLAIN loop plus a running minimum of r2 over the
//             thread's rows, compared with the near radius once per step (grav_device.cuh,
//             near_threshold) into a bit mask; the steps that met a near pair re-evaluate the
//             near pairs from the double-single separation and add the difference
//             (near_delta), after the chunk or, with rows of 8, after the j-tile.  Near pairs
//             are rare (~3e-5 of the pairs of the N = 65536 uniform cube), so this path is
//             cold; a warp that met many evaluates every pair of its next tile that way
//             (ds_column).
enum { SYM_PLAIN = 0, SYM_DS = 1, SYM_NEAR = 2 };

// Dynamic shared memory of one CTA, in this order (16-byte units throughout).
template <int B, int W, int JT, int KIND>
struct SymSmem {
	static constexpr int T = 32 * W, NP = KIND == SYM_PLAIN ? 1 : 2;
	static constexpr int EXA = KIND == SYM_DS ? 4 : 2;            // expanded rows per chunk
	static constexpr int EX_TILE = (JT / 32) * EXA * 64;         // ulonglong2 per expanded tile
	static constexpr int RAW = 0;                                 // [2][NP][JT] float4
	static constexpr int EX = RAW + 2 * NP * JT * 16;             // [2][JT / 32][EXA][64] ulonglong2
	static constexpr int CSUM = EX + 2 * EX_TILE * 16;            // [3][B][T] float2
	static constexpr int COL = CSUM + 3 * B * T * 8;              // [2][W][3][JT] float
	static constexpr int ROWLO = COL + 2 * W * 3 * JT * 4;        // [B][T] float4 (SYM_NEAR)
	// near pairs gone through once per j-tile, lane by lane, rather than once per chunk and step
	static constexpr bool BY_LANE = KIND == SYM_NEAR && B >= 8 && JT <= 128;
	static constexpr int MASK = ROWLO + (KIND == SYM_NEAR ? B * T * 16 : 0);   // [JT / 32][T] uint32 (BY_LANE)
	static constexpr int BYTES = MASK + (BY_LANE ? JT / 32 * T * 4 : 0);
};

// Column sums of the j-tile `jt` (block J > I) -> column slot of (I, J), the warps added in
// order.  They are FP32 sums, so they go out as FP32 (first half of the slot; stage 2 adds
// them by TwoSum in FP32): half the bytes of an FP64 slot.  s: the segment of block I.
template <int W, int T, int JT, int R>
__device__ __forceinline__ void flush_columns(const grav_batch& b, int s, int blkI, int blkJ,
	int64_t jt, const float* __restrict__ col, int tid)
{
	const grav_seg_desc SJ = b.seg[s + (blkJ - blkI)];
	const int64_t slot = SJ.slot_base + SJ.nslots - (blkJ - blkI);
	float* __restrict__ out = reinterpret_cast<float*>(b.part + slot * 3 * R) +
		(jt * JT - static_cast<int64_t>(blkJ) * R);
	for (int i = tid; i < JT; i += T) {
#pragma unroll
		for (int c = 0; c < 3; ++c) {
			float sum = col[c * JT + i];
#pragma unroll
			for (int w = 1; w < W; ++w) sum += col[(w * 3 + c) * JT + i];
			out[c * R + i] = sum;
		}
	}
}

// Fold a packed pair of row partials into the rows' compensated sums (entries sums[0] and
// sums[T]).
__device__ __forceinline__ void fold_pair(float2* sums, int T, u64 f)
{
	float f0, f1;
	unpack2(f, f0, f1);
	float2 a = sums[0], c = sums[T];
	two_sum_acc(a.x, a.y, f0);
	two_sum_acc(c.x, c.y, f1);
	sums[0] = a;
	sums[T] = c;
}

// The near correction of one column body (pj, low part lj) against a thread's rows: pairs
// closer than the near radius again, from the double-single separation, the difference
// added to the rows' sums f and (COLS) the rows' column terms, Gm_i e, to q.  Every lane of
// the warp calls it with a body of its own (on: it has one); a row's radius squared stands in
// rowlo's fourth component.
template <int H, int T, bool COLS>
__device__ __forceinline__ void near_rows(const float4& pj, const float4& lj, float eps2, bool on,
	const u64 (&nx)[H], const u64 (&ny)[H], const u64 (&nz)[H], const u64 (&g2)[H],
	const float4* __restrict__ rowlo, u64 (&fx)[H], u64 (&fy)[H], u64 (&fz)[H], float& qx,
	float& qy, float& qz)
{
	const u64 px = pack2(pj.x, pj.x), py = pack2(pj.y, pj.y), pz = pack2(pj.z, pj.z);
	const u64 pw = pack2(pj.w, pj.w), eps22 = pack2(eps2, eps2);
	uint32_t rows = 0;   // bit k: row k of this lane is near
#pragma unroll
	for (int h = 0; h < H; ++h) {
		const u64 dx = add2(px, nx[h]), dy = add2(py, ny[h]), dz = add2(pz, nz[h]);
		float ra, rb;
		unpack2(fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, eps22))), ra, rb);
		if (on & (ra < rowlo[(2 * h) * T].w) & (ra > eps2)) rows |= 1u << (2 * h);
		if (on & (rb < rowlo[(2 * h + 1) * T].w) & (rb > eps2)) rows |= 2u << (2 * h);
	}
	const uint32_t any = __reduce_or_sync(0xffffffffu, rows);
#pragma unroll
	for (int h = 0; h < H; ++h) {
		if (any >> (2 * h) & 3u) {
			const u64 dx = add2(px, nx[h]), dy = add2(py, ny[h]), dz = add2(pz, nz[h]);
			float ra, rb;
			unpack2(fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, eps22))), ra, rb);
			const bool na = rows >> (2 * h) & 1u, nb = rows >> (2 * h) & 2u;
			float x0, x1, y0, y1, z0, z1, ex0, ey0, ez0, ex1, ey1, ez1;
			unpack2(dx, x0, x1);
			unpack2(dy, y0, y1);
			unpack2(dz, z0, z1);
			near_delta(x0, y0, z0, ra, lj, rowlo[(2 * h) * T], eps2, na, ex0, ey0, ez0);
			near_delta(x1, y1, z1, rb, lj, rowlo[(2 * h + 1) * T], eps2, nb, ex1, ey1, ez1);
			fx[h] = fma2(pack2(ex0, ex1), pw, fx[h]);
			fy[h] = fma2(pack2(ey0, ey1), pw, fy[h]);
			fz[h] = fma2(pack2(ez0, ez1), pw, fz[h]);
			if (COLS) {
				float ga, gb;
				unpack2(g2[h], ga, gb);
				qx = fmaf(ex1, gb, fmaf(ex0, ga, qx));
				qy = fmaf(ey1, gb, fmaf(ey0, ga, qy));
				qz = fmaf(ez1, gb, fmaf(ez0, ga, qz));
			}
		}
	}
}

// A column body (p, low part l) against a thread's rows, every pair from its double-single
// separation, pairs whose FP32 separation is zero contributing nothing; COLS: the column's
// packed sums too.  Returns whether some row met it within its near radius.
template <int H, int T, bool COLS>
__device__ __forceinline__ bool ds_column(const float4& p, const float4& l, float eps2,
	const u64 (&nx)[H], const u64 (&ny)[H], const u64 (&nz)[H], const u64 (&g2)[H],
	const float4* __restrict__ rowlo, u64 (&fx)[H], u64 (&fy)[H], u64 (&fz)[H], u64& cx, u64& cy,
	u64& cz)
{
	const u64 px = pack2(p.x, p.x), py = pack2(p.y, p.y), pz = pack2(p.z, p.z);
	const u64 lx = pack2(l.x, l.x), ly = pack2(l.y, l.y), lz = pack2(l.z, l.z);
	const u64 pw = pack2(p.w, p.w), eps22 = pack2(eps2, eps2);
	bool near = false;
#pragma unroll
	for (int h = 0; h < H; ++h) {
		const float4 la = rowlo[(2 * h) * T], lb = rowlo[(2 * h + 1) * T];
		u64 dx = add2(px, nx[h]), dy = add2(py, ny[h]), dz = add2(pz, nz[h]);
		float xa, xb, ya, yb, za, zb, ra, rb;
		unpack2(dx, xa, xb);
		unpack2(dy, ya, yb);
		unpack2(dz, za, zb);
		const bool na = fabsf(xa) + fabsf(ya) + fabsf(za) > 0.f, nb = fabsf(xb) + fabsf(yb) + fabsf(zb) > 0.f;
		dx = add2(dx, add2(lx, pack2(-la.x, -lb.x)));
		dy = add2(dy, add2(ly, pack2(-la.y, -lb.y)));
		dz = add2(dz, add2(lz, pack2(-la.z, -lb.z)));
		unpack2(fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, eps22))), ra, rb);
		near |= (na & (ra < la.w)) | (nb & (rb < lb.w));
		const u64 inv = pack2(na ? rsqrt_sfu(ra) : 0.f, nb ? rsqrt_sfu(rb) : 0.f);
		const u64 inv3 = mul2(inv, mul2(inv, inv));
		const u64 wj = mul2(pw, inv3);
		fx[h] = fma2(dx, wj, fx[h]);
		fy[h] = fma2(dy, wj, fy[h]);
		fz[h] = fma2(dz, wj, fz[h]);
		if (COLS) {
			const u64 wi = mul2(g2[h], inv3);
			cx = fma2(dx, wi, cx);
			cy = fma2(dy, wi, cy);
			cz = fma2(dz, wi, cz);
		}
	}
	return near;
}

// This lane's next step with a near pair, taken out of its mask (bit 31 - st: step st).
__device__ __forceinline__ int next_step(uint32_t& mask)
{
	const int st = __clz(mask) & 31;
	mask &= ~(0x80000000u >> st);
	return st;
}

// Expand a j-tile for the packed loops: every coordinate twice in a 64-bit pair, (x, x | y, y)
// and (z, z | Gm, Gm), and the 32 bodies of a chunk twice in a row, so that lane l reads
// body (l + s) mod 32 at constant offset s.
template <int T, int JT, bool DS>
__device__ __forceinline__ void expand_tile(ulonglong2* __restrict__ ex,
	const float4* __restrict__ hi, const float4* __restrict__ lo, int tid)
{
	constexpr int EXA = DS ? 4 : 2;
	for (int i = tid; i < JT; i += T) {
		ulonglong2* __restrict__ q = ex + (i >> 5) * (EXA * 64) + (i & 31);
		const float4 p = hi[i];
		const ulonglong2 xy = make_ulonglong2(pack2(p.x, p.x), pack2(p.y, p.y));
		const ulonglong2 zw = make_ulonglong2(pack2(p.z, p.z), pack2(p.w, p.w));
		q[0] = q[32] = xy;
		q[64] = q[96] = zw;
		if (DS) {
			const float4 l = lo[i];
			const ulonglong2 lxy = make_ulonglong2(pack2(l.x, l.x), pack2(l.y, l.y));
			const ulonglong2 lz = make_ulonglong2(pack2(l.z, l.z), 0ull);
			q[128] = q[160] = lxy;
			q[192] = q[224] = lz;
		}
	}
}

// B rows per thread, W warps, j-tiles of JT bodies; MINB CTAs per SM (the register limit);
// COLPAIR: the even and odd rows' column sums rotate apart, a chain of 16 B terms each (two
// shuffles per component), or the rows of a step are added up before they join the rotating
// sum, a chain of 32 (one shuffle and two additions).  The shorter chain is the more exact
// one: rows of 4 keep the sums apart, rows of 8 add them (rms force error at 65536 bodies
// 5.6e-8 against 1.0e-7 and 1.3e-7 against 7e-8; within 3 % in time either way).  The plain
// mode, whose error is the rounding of the positions, adds them always (2 % faster).
template <int B, int W, int JT, int KIND, int UNROLL, int MINB, bool COLPAIR>
__global__ void __launch_bounds__(32 * W, MINB) stage1_sym_kernel(const grav_batch b)
{
	using L = SymSmem<B, W, JT, KIND>;
	constexpr int T = 32 * W;
	constexpr int R = T * B;            // rows per block (= itile)
	constexpr int H = B / 2;            // packed pairs of rows per thread
	constexpr int TPB = R / JT;         // j-tiles per block
	constexpr int NCH = JT / 32;        // 32-body chunks per j-tile
	constexpr uint32_t TILE_BYTES = JT * sizeof(float4);
	constexpr int NP = L::NP;                       // position arrays copied per j-tile
	constexpr bool DS = KIND == SYM_DS;             // double-single separations everywhere
	constexpr bool NEAR = KIND == SYM_NEAR;         // double-single for near pairs only
	constexpr bool BY_LANE = L::BY_LANE;
	static_assert(B % 2 == 0 && R % JT == 0 && JT % 32 == 0 && (NCH & (NCH - 1)) == 0, "tile shapes");
	extern __shared__ __align__(128) unsigned char sym_smem[];
	float4* const raw = reinterpret_cast<float4*>(sym_smem + L::RAW);
	ulonglong2* const ex = reinterpret_cast<ulonglong2*>(sym_smem + L::EX);
	// compensated row sums (hi, lo) of this thread's rows, touched once per j-tile
	float2* const csum = reinterpret_cast<float2*>(sym_smem + L::CSUM) + threadIdx.x;  // [c][k]: (c * B + k) * T
	// column sums of a j-tile, one row per warp: every warp writes each chunk of the tile
	// once, and the flush adds the warps in a fixed order (no shared-memory atomics, whose
	// order would depend on warp timing)
	float* const colacc = reinterpret_cast<float*>(sym_smem + L::COL);
	// low parts of this thread's rows and their near radii squared (NEAR), for the cold path
	float4* const rowlo = reinterpret_cast<float4*>(sym_smem + L::ROWLO) + threadIdx.x;  // [k]: k * T
	// steps of each chunk that met near pairs, this thread's (BY_LANE)
	uint32_t* const masks = reinterpret_cast<uint32_t*>(sym_smem + L::MASK) + threadIdx.x;  // [cc]: cc * T
	__shared__ __align__(8) uint64_t bar[2];

	const int tid = threadIdx.x;
	const int lane = tid & 31;
	const int warp = tid >> 5;
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

	const float4* __restrict__ pos = static_cast<const float4*>(b.pos);
	const float eps2 = b.eps2;
	const u64 eps22 = pack2(eps2, eps2);

	// Segment of unit ub by bisection, and no programmatic-launch instructions: a CTA runs
	// for 1e5-1e6 cycles, where a few microseconds of prologue do not matter.
	int s;
	{
		int lo = 0, hi = b.n_seg - 1;
		while (lo < hi) {
			const int mid = (lo + hi + 1) >> 1;
			if (b.seg[mid].unit_begin <= ub) lo = mid;
			else hi = mid - 1;
		}
		s = lo;
	}

	uint32_t gt = 0;   // tiles of this CTA before this piece (tile g: buffer g & 1, phase g >> 1)
	int in_flight = 0;  // copies in flight when a wait expired, the first one that of tile gt
	while (ub < ue && s < b.n_seg) {
		const grav_seg_desc S = b.seg[s];
		if (S.n_units == 0 || S.unit_begin + S.n_units <= ub) {
			++s;
			continue;
		}
		const grav_univ_desc Uu = b.univ[S.u];
		const int blkI = S.il0 / R;
		const int64_t t0 = ub - S.unit_begin;                              // local unit
		const int64_t t1 = min(ue - S.unit_begin, (int64_t)S.n_units);
		const int nt = static_cast<int>(t1 - t0);
		const int64_t jt_first = static_cast<int64_t>(blkI) * TPB + t0;  // global j-tile of unit t0
		const float4* __restrict__ jsrc = pos + Uu.pad_off;
		const float4* __restrict__ jsrclo = pos + b.n_pad_total + Uu.pad_off;
		const auto copy_tile = [&](int t) {   // tile t of this piece -> buffer (gt + t) & 1
			const int bs = (gt + t) & 1;
			mbar_arrive_expect_tx(&bar[bs], NP * TILE_BYTES);
			bulk_g2s(raw + bs * NP * JT, jsrc + (jt_first + t) * JT, TILE_BYTES, &bar[bs]);
			if (NP == 2)
				bulk_g2s(raw + (bs * NP + 1) * JT, jsrclo + (jt_first + t) * JT, TILE_BYTES, &bar[bs]);
		};
		// wait for tile t and expand this thread's share of it; false when the wait expired
		const auto expand = [&](int t) {
			const int bs = (gt + t) & 1;
			if (!mbar_wait_bounded(&bar[bs], ((gt + t) >> 1) & 1)) return false;
			expand_tile<T, JT, DS>(ex + bs * L::EX_TILE, raw + bs * NP * JT, raw + (bs * NP + 1) * JT, tid);
			return true;
		};
		if (tid == 0) {
			copy_tile(0);
			if (nt > 1) copy_tile(1);
		}

		// rows of this warp: w*32*B + k*32 + lane, packed (2h, 2h + 1), coordinates negated so
		// that a separation is one packed add
		const int64_t ibase = Uu.pad_off + S.il0 + warp * 32 * B + lane;
		u64 nx[H], ny[H], nz[H], g2[H], fx[H], fy[H], fz[H];
		u64 nxl[H], nyl[H], nzl[H];                      // low parts (DS)
		float scale[B];                                  // NEAR: largest |coordinate| of each row
#pragma unroll
		for (int h = 0; h < H; ++h) {
			const float4 p = load_row(pos + ibase + (2 * h) * 32);
			const float4 q = load_row(pos + ibase + (2 * h + 1) * 32);
			nx[h] = pack2(-p.x, -q.x);
			ny[h] = pack2(-p.y, -q.y);
			nz[h] = pack2(-p.z, -q.z);
			g2[h] = pack2(p.w, q.w);
			nxl[h] = nyl[h] = nzl[h] = 0ull;
			if (DS) {
				const float4 pl = load_row(pos + b.n_pad_total + ibase + (2 * h) * 32);
				const float4 ql = load_row(pos + b.n_pad_total + ibase + (2 * h + 1) * 32);
				nxl[h] = pack2(-pl.x, -ql.x);
				nyl[h] = pack2(-pl.y, -ql.y);
				nzl[h] = pack2(-pl.z, -ql.z);
			}
			if (NEAR) {
				const int row = S.il0 + warp * 32 * B + (2 * h) * 32 + lane;   // of the universe
				scale[2 * h] = row < Uu.n ? near_scale(p.x, p.y, p.z) : 0.f;
				scale[2 * h + 1] = row + 32 < Uu.n ? near_scale(q.x, q.y, q.z) : 0.f;
			}
			fx[h] = fy[h] = fz[h] = 0ull;
		}
#pragma unroll
		for (int e = 0; e < 3 * B; ++e) csum[e * T] = make_float2(0.f, 0.f);
		// NEAR: the near radius that the rows share; in a warp with rows that are left out of it
		// (apart) every row is tested against its own, rowlo's fourth component
		float thr = 0.f;
		bool apart = false;
		if (NEAR) {
			const int row = S.il0 + warp * 32 * B + lane;   // of the universe
			const float xmax = common_scale<B>(scale, min(B, (Uu.n - row + 31) / 32));
			thr = near_threshold(xmax);
			bool stray = false;
#pragma unroll
			for (int k = 0; k < B; ++k) {
				float4 lo = pos[b.n_pad_total + ibase + k * 32];
				lo.w = near_threshold(fmaxf(scale[k], xmax));
				rowlo[k * T] = lo;
				stray |= scale[k] > xmax;
			}
			apart = __any_sync(0xffffffffu, stray);
		}

		bool ok = expand(0);
		// NEAR: the tile (first: the chunk) before met so many near pairs (marks: this lane's
		// steps that met one) that double-single separations for all pairs of the next are
		// cheaper: two Plummer spheres of 16384 bodies, 8/64/64, 473 us a step without
		bool dense = false;
		int marks = 0;
		int blk_done = 0;   // block J of the previous tile when it left column sums, else 0
		for (int t = 0; t < nt; ++t) {
			// every warp has finished tile t - 1, its share of tile t is expanded, and its
			// column sums of tile t - 1 are in colacc
			if (__syncthreads_or(!ok)) {
				in_flight = t == 0 && nt > 1 ? 2 : 1;
				gt += t;
				break;
			}
			const int bs = (gt + t) & 1;
			if (t > 0) {
				if (tid == 0 && t + 1 < nt) copy_tile(t + 1);   // over tile t - 1
				if (blk_done)
					flush_columns<W, T, JT, R>(b, s, blkI, blk_done, jt_first + t - 1,
						colacc + (bs ^ 1) * W * 3 * JT, tid);
			}
			const int64_t jt = jt_first + t;   // j-tile index in the universe
			const float4* __restrict__ sj = raw + bs * NP * JT;
			const float4* __restrict__ sjl = sj + JT;   // low parts (NP == 2)
			const ulonglong2* __restrict__ et = ex + bs * L::EX_TILE;
			const int blkJ = static_cast<int>(jt / TPB);
			if (blkJ == blkI) {
				// diagonal block: every ordered pair of the block once, rows only.  In NEAR
				// mode a tile that holds this warp's own rows meets their self pairs (d = 0,
				// r2 = eps2): there the near test also requires r2 > eps2, so that self pairs
				// do not send the warp down the correction path
				const int jl0 = static_cast<int>(jt - static_cast<int64_t>(blkI) * TPB) * JT;
				const bool own = jl0 < (warp + 1) * 32 * B && jl0 + JT > warp * 32 * B;
#pragma unroll 1
				for (int ch = 0; ch < NCH; ++ch) {
					if (NEAR && dense) {
						u64 unused = 0ull;
#pragma unroll 1
						for (int j = ch * 32; j < ch * 32 + 32; ++j)
							marks += ds_column<H, T, false>(sj[j], sjl[j], eps2, nx, ny, nz, g2, rowlo, fx, fy, fz,
								unused, unused, unused);
						continue;
					}
					const ulonglong2* __restrict__ se = et + ch * (L::EXA * 64);
					uint32_t nmask = 0;
#pragma unroll 2
					for (int j = 0; j < 32; ++j) {
						const ulonglong2 pxy = se[j], pzw = se[64 + j];
						ulonglong2 lxy = make_ulonglong2(0ull, 0ull), lz = lxy;
						if (DS) {
							lxy = se[128 + j];
							lz = se[192 + j];
						}
						bool near = false;
#pragma unroll
						for (int h = 0; h < H; ++h) {
							u64 dx = add2(pxy.x, nx[h]), dy = add2(pxy.y, ny[h]), dz = add2(pzw.x, nz[h]);
							if (DS) {
								dx = add2(dx, add2(lxy.x, nxl[h]));
								dy = add2(dy, add2(lxy.y, nyl[h]));
								dz = add2(dz, add2(lz.x, nzl[h]));
							}
							float ra, rb;
							unpack2(fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, eps22))), ra, rb);
							if (NEAR) {
								float ta = thr, tb = thr;
								if (apart) {
									ta = rowlo[(2 * h) * T].w;
									tb = rowlo[(2 * h + 1) * T].w;
								}
								near |= own ? ((ra < ta) & (ra > eps2)) | ((rb < tb) & (rb > eps2))
								            : (ra < ta) | (rb < tb);
							}
							const u64 inv = pack2(rsqrt_sfu(ra), rsqrt_sfu(rb));
							const u64 w = mul2(mul2(pzw.y, inv), mul2(inv, inv));
							fx[h] = fma2(dx, w, fx[h]);
							fy[h] = fma2(dy, w, fy[h]);
							fz[h] = fma2(dz, w, fz[h]);
						}
						if (NEAR && near) nmask |= 0x80000000u >> j;
					}
					if (NEAR) marks += __popc(nmask);
					if (NEAR && t == 0 && ch == 0) dense = __any_sync(0xffffffffu, marks > 32 / 6);
					if (NEAR) {
						while (__any_sync(0xffffffffu, nmask != 0u)) {
							const bool on = nmask != 0u;
							const int j = ch * 32 + next_step(nmask);
							float qx = 0.f, qy = 0.f, qz = 0.f;
							near_rows<H, T, false>(sj[j], sjl[j], eps2, on, nx, ny, nz, g2, rowlo, fx, fy, fz, qx,
								qy, qz);
						}
					}
				}
				blk_done = 0;
			} else {
				// unique pairs with block J > I: rotate the chunk's column sums
				float* __restrict__ cw = colacc + (bs * W + warp) * 3 * JT;
				uint32_t met = 0;   // BY_LANE: this lane's steps with near pairs, any chunk
#pragma unroll 1
				for (int cc = 0; cc < NCH; ++cc) {
					const int ch = (cc + warp) & (NCH - 1);
					const ulonglong2* __restrict__ se = et + ch * (L::EXA * 64) + lane;
					u64 cx = 0ull, cy = 0ull, cz = 0ull;     // even and odd rows' column sums
					float sx = 0.f, sy = 0.f, sz = 0.f;
					uint32_t nmask = 0;   // NEAR: bit 31 - st of a step st that met a near pair
					// the column sums move on to the lane that meets their body next
					const auto rotate = [&]() {
						const int src = (lane + 1) & 31;
						float a0, a1;
						if (COLPAIR) {
							unpack2(cx, a0, a1);
							cx = pack2(__shfl_sync(0xffffffffu, a0, src), __shfl_sync(0xffffffffu, a1, src));
							unpack2(cy, a0, a1);
							cy = pack2(__shfl_sync(0xffffffffu, a0, src), __shfl_sync(0xffffffffu, a1, src));
							unpack2(cz, a0, a1);
							cz = pack2(__shfl_sync(0xffffffffu, a0, src), __shfl_sync(0xffffffffu, a1, src));
						} else {
							unpack2(cx, a0, a1);
							sx = __shfl_sync(0xffffffffu, sx + (a0 + a1), src);
							unpack2(cy, a0, a1);
							sy = __shfl_sync(0xffffffffu, sy + (a0 + a1), src);
							unpack2(cz, a0, a1);
							sz = __shfl_sync(0xffffffffu, sz + (a0 + a1), src);
						}
					};
					// one column against the rows; by_row: every row against its own near radius
					const auto step = [&](int st, auto by_row_t) {
						constexpr bool by_row = decltype(by_row_t)::value;
						const ulonglong2 pxy = se[st], pzw = se[64 + st];
						ulonglong2 lxy = make_ulonglong2(0ull, 0ull), lz = lxy;
						if (DS) {
							lxy = se[128 + st];
							lz = se[192 + st];
						}
						float rmin = 0.f;   // NEAR: smallest r2 of this step
						bool near = false;
						if (!COLPAIR) cx = cy = cz = 0ull;
#pragma unroll
						for (int h = 0; h < H; ++h) {
							u64 dx = add2(pxy.x, nx[h]), dy = add2(pxy.y, ny[h]), dz = add2(pzw.x, nz[h]);
							if (DS) {
								dx = add2(dx, add2(lxy.x, nxl[h]));
								dy = add2(dy, add2(lxy.y, nyl[h]));
								dz = add2(dz, add2(lz.x, nzl[h]));
							}
							float ra, rb;
							unpack2(fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, eps22))), ra, rb);
							if (NEAR && by_row)
								near |= (ra < rowlo[(2 * h) * T].w) | (rb < rowlo[(2 * h + 1) * T].w);
							else if (NEAR) rmin = h == 0 ? fminf(ra, rb) : min3f(rmin, ra, rb);
							const u64 inv = pack2(rsqrt_sfu(ra), rsqrt_sfu(rb));
							const u64 inv3 = mul2(inv, mul2(inv, inv));
							const u64 wj = mul2(pzw.y, inv3);
							const u64 wi = mul2(g2[h], inv3);
							fx[h] = fma2(dx, wj, fx[h]);
							fy[h] = fma2(dy, wj, fy[h]);
							fz[h] = fma2(dz, wj, fz[h]);
							if (!COLPAIR && h == 0) {
								cx = mul2(dx, wi);
								cy = mul2(dy, wi);
								cz = mul2(dz, wi);
							} else {
								cx = fma2(dx, wi, cx);
								cy = fma2(dy, wi, cy);
								cz = fma2(dz, wi, cz);
							}
						}
						// both are >= 0, so they compare as integers; the sign goes into the mask
						if (NEAR && by_row) nmask = nmask << 1 | (near ? 1u : 0u);
						else if (NEAR)
							nmask = __funnelshift_l(__float_as_uint(rmin) - __float_as_uint(thr), nmask, 1);
						rotate();
					};
					if (NEAR && dense) {
						// every pair from its double-single separation, hi-part separations of zero
						// contributing nothing; the near pairs are only counted
#pragma unroll 1
						for (int st = 0; st < 32; ++st) {
							const int j = ch * 32 + ((lane + st) & 31);
							if (!COLPAIR) cx = cy = cz = 0ull;
							marks += ds_column<H, T, true>(sj[j], sjl[j], eps2, nx, ny, nz, g2, rowlo, fx, fy, fz, cx, cy, cz);
							rotate();
						}
					} else if (NEAR && apart) {
#pragma unroll 1
						for (int st = 0; st < 32; ++st) step(st, std::true_type());
					} else {
#pragma unroll UNROLL
						for (int st = 0; st < 32; ++st) step(st, std::false_type());
					}
					if (COLPAIR) {
						float a0, a1;
						unpack2(cx, a0, a1);
						sx = a0 + a1;
						unpack2(cy, a0, a1);
						sy = a0 + a1;
						unpack2(cz, a0, a1);
						sz = a0 + a1;
					}
					if (NEAR) marks += __popc(nmask);
					if (NEAR && t == 0 && cc == 0) dense = __any_sync(0xffffffffu, marks > 32 / 6);
					if (BY_LANE) {
						masks[cc * T] = nmask;
						met |= nmask;
					} else if (NEAR) {
						// cold path: the steps that met near pairs again, every lane with the body it met
						// then; their column terms belong to that body, whose sum lane (lane + st) mod 32
						// now holds
						uint32_t todo = __reduce_or_sync(0xffffffffu, nmask);
						while (todo) {
							const int st = next_step(todo);
							const int j = ch * 32 + ((lane + st) & 31);
							float qx = 0.f, qy = 0.f, qz = 0.f;
							near_rows<H, T, true>(sj[j], sjl[j], eps2, true, nx, ny, nz, g2, rowlo, fx, fy, fz, qx,
								qy, qz);
							const int from = (lane - st) & 31;
							sx += __shfl_sync(0xffffffffu, qx, from);
							sy += __shfl_sync(0xffffffffu, qy, from);
							sz += __shfl_sync(0xffffffffu, qz, from);
						}
					}
					cw[ch * 32 + lane] = -sx;
					cw[JT + ch * 32 + lane] = -sy;
					cw[2 * JT + ch * 32 + lane] = -sz;
				}
				if (BY_LANE && __any_sync(0xffffffffu, met != 0u)) {
					// cold path, once per tile: each lane's own steps that met near pairs, all lanes
					// side by side; the column terms go to the body met, lanes that met the same one
					// in turn
					__syncwarp();
					int cc = 0;
					uint32_t mask = masks[0];
					for (;;) {
						while (!mask && cc + 1 < NCH) mask = masks[++cc * T];
						if (!__any_sync(0xffffffffu, mask != 0u)) break;
						const bool on = mask != 0u;
						const int j = ((cc + warp) & (NCH - 1)) * 32 + ((lane + next_step(mask)) & 31);
						float qx = 0.f, qy = 0.f, qz = 0.f;
						near_rows<H, T, true>(sj[j], sjl[j], eps2, on, nx, ny, nz, g2, rowlo, fx, fy, fz, qx, qy,
							qz);
						const uint32_t same = __match_any_sync(0xffffffffu, on ? j : JT + lane);
						const unsigned turn = __popc(same & ((1u << lane) - 1u));
						const unsigned turns = __reduce_max_sync(0xffffffffu, turn);
						for (unsigned i = 0; i <= turns; ++i) {
							if (turn == i && on) {
								cw[j] -= qx;
								cw[JT + j] -= qy;
								cw[2 * JT + j] -= qz;
							}
							__syncwarp();
						}
					}
				}
				blk_done = blkJ;
			}
			if (NEAR) {
				dense = __any_sync(0xffffffffu, marks > JT / 6);
				marks = 0;
			}
			// fold the tile's row partials into the compensated sums
#pragma unroll
			for (int h = 0; h < H; ++h) {
				fold_pair(csum + (0 * B + 2 * h) * T, T, fx[h]);
				fold_pair(csum + (1 * B + 2 * h) * T, T, fy[h]);
				fold_pair(csum + (2 * B + 2 * h) * T, T, fz[h]);
				fx[h] = fy[h] = fz[h] = 0ull;
			}
			ok = t + 1 < nt ? expand(t + 1) : true;
		}
		if (in_flight) break;
		__syncthreads();   // colacc of the last tile is complete; the buffers are free again
		if (blk_done)
			flush_columns<W, T, JT, R>(b, s, blkI, blk_done, jt_first + nt - 1,
				colacc + ((gt + nt - 1) & 1) * W * 3 * JT, tid);
		gt += nt;

		// row sums of this CTA's piece as FP32 (hi, lo) pairs, one 8-byte slot entry each
		const int64_t slot = S.slot_base + (c - S.cta_first);
		float2* __restrict__ out = reinterpret_cast<float2*>(b.part + slot * 3 * R) + warp * 32 * B + lane;
#pragma unroll
		for (int cpt = 0; cpt < 3; ++cpt)
#pragma unroll
			for (int k = 0; k < B; ++k) out[cpt * R + k * 32] = csum[(cpt * B + k) * T];
		ub = S.unit_begin + t1;
		++s;
	}

	if (in_flight && tid == 0) {
		set_error(b.err, GRAV_DEV_TIMEOUT);
		// give each copy in flight one more bounded wait, so that none lands in shared memory
		// after this CTA exits
		for (uint32_t g = gt; g < gt + in_flight; ++g) mbar_wait_bounded(&bar[g & 1], (g >> 1) & 1);
	}
}

// launched the ordinary way (not as a programmatic dependent): see the kernel's prologue
#define GRAV_SYM_KERNEL(MODE, KIND, B, W, J, UN, MINB, CP) \
	{MODE, B, 32 * W, J, \
		reinterpret_cast<const void*>(&stage1_sym_kernel<B, W, J, KIND, UN, MINB, CP>), \
		SymSmem<B, W, J, KIND>::BYTES, false}
#define GRAV_SYM_ENTRY(B, W, J, MINB) GRAV_SYM_KERNEL(GRAV_MODE_FP32U, SYM_PLAIN, B, W, J, 16, MINB, false)
#define GRAV_SYMC_ENTRY(B, W, J, UN, MINB) GRAV_SYM_KERNEL(GRAV_MODE_FP32CU, SYM_DS, B, W, J, UN, MINB, B < 8)
#define GRAV_SYMN_ENTRY(B, W, J, UN, MINB) GRAV_SYM_KERNEL(GRAV_MODE_FP32UN, SYM_NEAR, B, W, J, UN, MINB, B < 8)

// UN (unrolling of the step loop) and MINB (the occupancy that ptxas must leave room for) as
// measured per shape over 1 to 16 steps and the occupancies around each; no sum's order
// depends on them.  Stage 1 at 65536 bodies, unrolled by 4 at the higher occupancy and as
// compiled here:
//   fp32cu 8/64/64 1682 (6 CTAs, 165 registers) and 1580 us (4 CTAs, 194);
//   fp32u 8/128/64 1297 and 1225, 8/64/64 1210 and 1200, at 16384 bodies 88 and 82.
// Two warps per scheduler with every operand in registers beat three that reload some.  16
// rows per thread (fp32u) share a step's loads, shuffles and column additions: from 32768
// bodies on 2-3 % faster than 8 (131072 bodies 4746 -> 4604 us), below slower, their blocks of
// 1024 rows being too coarse.
//
// Near pairs (fp32un).  A chunk of 32 columns against a warp's rows of 8 holds 0.5 near pairs
// in a cube at rest and 1.2 in a Gaussian cloud.  Going through the chunk's steps that met any,
// the whole warp at each, is a chain of some 500 cycles that two warps per scheduler hide
// badly; once per j-tile with every lane at its own steps it runs once or twice per tile.
// Stage 1 at 65536 bodies, cube / cloud (without any near pass 1290 / 1290):
//   8/128/128 1329 / 1401 -> 1318 / 1354 us, 8/64/64 1352 / 1417 -> 1359 / 1387, and by lane
//   4/256/256 1323 / 1341 -> 1366 / 1394: rows of 4 meet half as many and keep the pass per
//   chunk, as does 8/128/256, whose second CTA per SM would not fit the masks.
// The separate loop for warps with rows far out costs the others nothing at the unrolling
// chosen with it; a step of 65536 bodies with one body 1000 times farther out than the others
// takes 1.33 ms (7.8 with one radius per thread), with twenty 1.46.  Tiles full of near pairs
// (dense clusters) go through ds_column: two Plummer spheres of 16384 bodies 172 us a step, of
// 65536 2.07 ms (marked steps corrected one by one, in the loop: 239 us and 3.25 ms).
static const Stage1Kernel k_table_sym[] = {
	GRAV_SYM_ENTRY(4, 4, 128, 4),
	GRAV_SYM_ENTRY(4, 8, 256, 2),
	GRAV_SYM_ENTRY(8, 4, 256, 2),
	GRAV_SYM_ENTRY(4, 4, 256, 3),
	GRAV_SYM_ENTRY(2, 8, 256, 2),
	GRAV_SYM_ENTRY(8, 8, 256, 1),
	GRAV_SYM_ENTRY(8, 4, 128, 3),
	GRAV_SYM_ENTRY(8, 4, 64, 3),
	GRAV_SYM_ENTRY(4, 2, 64, 8),
	GRAV_SYM_ENTRY(8, 2, 64, 4),
	GRAV_SYM_KERNEL(GRAV_MODE_FP32U, SYM_PLAIN, 16, 2, 64, 8, 4, false),
	GRAV_SYMC_ENTRY(4, 4, 128, 16, 3),
	GRAV_SYMC_ENTRY(8, 4, 256, 4, 1),
	GRAV_SYMC_ENTRY(4, 4, 256, 16, 2),
	GRAV_SYMC_ENTRY(4, 8, 256, 16, 1),
	GRAV_SYMC_ENTRY(8, 4, 128, 4, 2),
	GRAV_SYMC_ENTRY(4, 2, 64, 16, 5),
	GRAV_SYMC_ENTRY(8, 2, 64, 4, 4),
	GRAV_SYMN_ENTRY(4, 4, 128, 16, 3),
	GRAV_SYMN_ENTRY(8, 4, 256, 10, 2),
	GRAV_SYMN_ENTRY(8, 4, 128, 8, 2),
	GRAV_SYMN_ENTRY(8, 4, 64, 8, 2),
	GRAV_SYMN_ENTRY(4, 4, 256, 16, 2),
	GRAV_SYMN_ENTRY(4, 8, 256, 16, 1),
	GRAV_SYMN_ENTRY(4, 2, 64, 2, 7),
	GRAV_SYMN_ENTRY(8, 2, 64, 2, 4),
	GRAV_SYMN_ENTRY(8, 2, 128, 4, 4),
};

int stage1_table_sym(const Stage1Kernel** out)
{
	*out = k_table_sym;
	return static_cast<int>(sizeof(k_table_sym) / sizeof(k_table_sym[0]));
}

}  // namespace grav
