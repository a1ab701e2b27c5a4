// steps.cu -- K full steps (stage 1 + stage 2) of one universe in one launch
// (grav_steps).
//
// Up to about ten thousand bodies a step is a few microseconds of arithmetic, and two
// dependent launches per step (the persistent stage-1 grid, then stage 2 over its slots)
// spend most of it on launch, drain and memory latency: 8.8 us per step at 64 bodies, 9.2 us
// at 1000, 17.7 us at 4096 (fp32n, graph-replayed).  Here one grid of at most one CTA per SM
// stays for all K steps: 1.9, 3.6 and 11.8 us per step of 20.  Each CTA keeps the FP64 state
// of its R rows in registers and every body's FP32 position in shared memory; per step it
// completes its rows' accelerations over all columns, integrates the rows and exchanges the
// new positions with the other CTAs.  At 1000 bodies a step is ~1 us of pair work and ~0.5 us
// of the slowest warp's near pairs, ~0.8 us of FP64 update (a chain of eight FP64
// instructions of 67 cycles each to the new position, three more to its low part) and ~1.4 us of exchange; at 4096 the pair loop takes 7.8 us,
// 70 % of what its FMA-pipe instructions need.
//
// Exchange.  There is no grid barrier between steps.  A row's new position is published as
// a 128-bit word (x, y, z, tag) by one relaxed 128-bit store and read by one relaxed
// 128-bit load, which the memory model keeps whole; the tag is a step number that no
// earlier step (or launch) used, so a reader that polls until the tag matches has the
// position itself and needs no separate flag, fence or second round trip.  Two buffers
// alternate: a CTA overwrites step k's positions when it publishes step k + 2, which it
// does only after it has read every CTA's position of step k + 1, and a CTA publishes that
// only after it is done with step k's.  One CTA alone exchanges through its own shared
// memory.  The CTAs wait on one another, so they are co-scheduled: up to 16 as one
// thread-block cluster (launched as a programmatic dependent), more as a cooperative
// launch.  Every wait is bounded (GRAV_WAIT_NS) and a thread waits no more once one has expired:
// the CTA records GRAV_DEV_TIMEOUT and leaves without writing its rows.  A CTA whose words did
// arrive may have written its own, so the state is undefined then.
//
// Pair loop.  A CTA's rows come in groups of 4 and the columns in blocks of 64; a unit is one
// group against one block and the CTA's units are dealt evenly to its warps in order, so a
// few rows keep every warp busy.  Lane 16 q + c of a warp takes rows 2 q and 2 q + 1 of the
// group and the column pairs c and c + 16 of the block: the two columns of a pair are one
// packed FP32 pair (x0, x1), read from shared memory in that layout, the rows duplicated
// pairs.  12 packed FMA-pipe instructions and two reciprocal square roots per row and pair
// (24 + 4 cycles), one 128-bit shared load; with one row per lane and two loads the loads'
// return path was as long as the arithmetic.  Partials are FP32 over 16 blocks (32
// terms per lane and column parity) and added into a second FP32 level; the warps' pieces of
// a row are added by TwoSum (48 bits) in warp order: nothing depends on scheduling.
//
// Near pairs.  The loop keeps one bit per block and lane that met a pair within the near
// radius (each row's own, or one that the group shares: steps_kind); after every 32 blocks each
// lane goes through its own blocks' near pairs, all lanes side by side.  The CTAs run in step,
// so the warp with the most near pairs sets everyone's pace: with the warp going through the
// union of its lanes' blocks after every 16, a step took 4.5 us at 1000 bodies (2.9 without the
// near pairs) and 14.0 at 4096; so 3.8 and 11.8.  The low parts are not kept in shared memory
// (unless one CTA holds every row): the few that near pairs need come from the exchange buffer,
// and the exchange moves half the bytes (14.0 to 12.6 us at 4096).
#include "exchange.cuh"

namespace grav {

// Double-single separations everywhere; for near pairs, each row with a near radius of its own;
// for near pairs, the rows of a group sharing theirs (common_scale).
enum { STEPS_DS = 0, STEPS_NEAR = 1, STEPS_NEAR_SHARED = 2 };
constexpr int ST_T = 512;            // threads per CTA
constexpr int ST_W = ST_T / 32;
constexpr int ST_RG = 4;             // rows per group
constexpr int ST_CB = 64;            // columns per block
constexpr int ST_CHUNK = 16;         // blocks per first-level FP32 sum
constexpr int ST_SEG = 32;           // blocks between two passes over the near pairs met
constexpr int ST_RPW = 10;           // rows whose state one warp holds (3 lanes each)
constexpr int ST_MAX_ROWS = ST_RPW * ST_W;
constexpr int ST_SMEM_MAX = 227 * 1024 - 64;   // dynamic, less the kernel's own words

// Shared memory of one CTA for n bodies and R rows per CTA (byte offsets, 16-byte units).
struct StepsSmem {
	int cols;     // [blocks][2][32] ulonglong2: (x0, x1 | y0, y1), (z0, z1 | Gm0, Gm1)
	int colslo;   // the same for the low parts (DS, and NEAR with one CTA: lo_here)
	int rown;     // [rows][2] ulonglong2: (-x, -x | -y, -y), (-z, -z | near radius^2)
	int rownlo;   // the same for the low parts (DS, NEAR)
	int red;      // [groups + warps][ST_RG][3] float: the pieces' sums
	int bytes;
	bool lo_here;
	__host__ __device__ StepsSmem(int kind, int n, int rows)
	{
		const int nb = (n + ST_CB - 1) / ST_CB;
		const int ng = (rows + ST_RG - 1) / ST_RG;
		const int r4 = ng * ST_RG;
		lo_here = kind == STEPS_DS || rows >= n;
		cols = 0;
		colslo = cols + nb * 1024;
		rown = colslo + (lo_here ? nb * 1024 : 0);
		rownlo = rown + r4 * 32;
		red = rownlo + r4 * 32;
		bytes = (red + (ng + ST_W) * ST_RG * 3 * 4 + 15) / 16 * 16;
	}
};

// A row's duplicated, negated coordinates and, for its high parts, the near radius squared.
__device__ __forceinline__ void set_row(ulonglong2* p, float x, float y, float z, float thr)
{
	p[0] = make_ulonglong2(pack2(-x, -x), pack2(-y, -y));
	p[1] = make_ulonglong2(pack2(-z, -z), pack2(thr, 0.f));
}

// Two columns (2p, 2p + 1) of an expanded array; w given only where it is first written.
__device__ __forceinline__ void set_pair(ulonglong2* cols, int p, const float4& a, const float4& c)
{
	ulonglong2* q = cols + (p >> 5) * 64 + (p & 31);
	q[0] = make_ulonglong2(pack2(a.x, c.x), pack2(a.y, c.y));
	*reinterpret_cast<u64*>(q + 32) = pack2(a.z, c.z);
}

// One coordinate set of column j (one CTA: its rows are all the columns).
__device__ __forceinline__ void set_column(ulonglong2* cols, int j, float x, float y, float z)
{
	float* q = reinterpret_cast<float*>(cols + (j >> 6) * 64 + ((j >> 1) & 31)) + (j & 1);
	q[0] = x;
	q[2] = y;
	q[32 * 4] = z;
}

template <int KIND>
__global__ void __launch_bounds__(ST_T, 1) steps_kernel(const grav_batch b, const int flags,
	const int K, const int64_t a_stride, const int R, unsigned char* __restrict__ scratch)
{
	constexpr bool DS = KIND == STEPS_DS;
	constexpr bool NEAR = KIND != STEPS_DS;
	constexpr bool SHARED = KIND == STEPS_NEAR_SHARED;
	extern __shared__ __align__(16) unsigned char steps_smem[];
	__shared__ int expired;   // a wait of the near pass has run out (read after the first barrier)
	const int tid = threadIdx.x;
	const int lane = tid & 31;
	const int warp = tid >> 5;
	const int n = static_cast<int>(b.n_bodies);
	const int G = gridDim.x;
	const bool multi = G > 1;
	const bool clustered = multi && cluster_ctas() == static_cast<unsigned>(G);
	const int row0 = blockIdx.x * R;
	const int rows_here = max(0, min(R, n - row0));
	const int NB = (n + ST_CB - 1) / ST_CB;
	const int NG = (rows_here + ST_RG - 1) / ST_RG;
	const float eps2 = b.eps2;
	const u64 eps22 = pack2(eps2, eps2);
	const bool integrate = (flags & GRAV_S2_INTEGRATE) != 0;

	const StepsSmem L(KIND, n, R);
	ulonglong2* const cols = reinterpret_cast<ulonglong2*>(steps_smem + L.cols);
	ulonglong2* const colslo = reinterpret_cast<ulonglong2*>(steps_smem + L.colslo);
	ulonglong2* const rown = reinterpret_cast<ulonglong2*>(steps_smem + L.rown);
	ulonglong2* const rownlo = reinterpret_cast<ulonglong2*>(steps_smem + L.rownlo);
	float* const red = reinterpret_cast<float*>(steps_smem + L.red);
	const bool lo_here = L.lo_here;

	ExchangeHead* const head = reinterpret_cast<ExchangeHead*>(scratch);
	const int64_t words = static_cast<int64_t>(NB) * ST_CB;   // per array and buffer
	float4* const xbuf = reinterpret_cast<float4*>(scratch + EXCHANGE_HEAD_BYTES);  // [2][hi, lo][words]
	const double Tu = b.univ[0].T;

	// this warp's units [u0, u1) of the CTA's NG x NB
	const int U = NG * NB;
	const int Wn = max(1, min(ST_W, U));
	const int u0 = warp < Wn ? warp * U / Wn : U, u1 = warp < Wn ? (warp + 1) * U / Wn : U;
	const int g_first = u0 / NB;
	const int cb_first = u0 - g_first * NB;
	const int c16 = lane & 15;             // column lane; rows 2 (lane / 16) and the next one

	// three lanes per row, ten rows per warp: lane 3 i + c owns component c of its row's r and
	// v for the whole launch (FP64 instructions cost this GPU ~20 cycles per warp and SM
	// whatever their active lanes, so the rows' components share them)
	const int rl = warp * ST_RPW + lane / 3, rc = lane % 3;
	const bool mine = lane < 3 * ST_RPW && rl < rows_here;
	const bool warp_rows = warp * ST_RPW < rows_here;
	const int grow = rl / ST_RG;   // this lane's row group; the warps that hold its pieces
	int w_lo = 0, w_hi = -1;
	if (mine) {
		w_lo = ((grow * NB + 1) * Wn + U - 1) / U - 1;
		w_hi = ((grow + 1) * NB * Wn + U - 1) / U - 1;
	}

	if (tid == 0) expired = 0;
	// everything below belongs to the kernels before this one
	grid_dep_wait();
	const uint32_t tag0 = multi ? head->epoch + 1 : 0;   // tag of the positions step 0 makes
	double* const rd = b.r;
	double* const vd = b.v;
	const int64_t e = 4 * static_cast<int64_t>(row0 + rl) + rc;
	double rr = 0.0, vv = 0.0;
	const float4* __restrict__ pos = static_cast<const float4*>(b.pos);
	const float4* __restrict__ poslo = pos + b.n_pad_total;
	if (mine && integrate) {
		rr = rd[e];
		vv = vd[e];
	}

	// positions of every body; padding columns as FAR_PAD says
	for (int p = tid; p < NB * 32; p += ST_T) {
		const float4 far = make_float4(FAR_PAD, FAR_PAD, FAR_PAD, 0.f), z = make_float4(0.f, 0.f, 0.f, 0.f);
		const int j = 2 * p;
		const float4 a = j < n ? pos[j] : far, c = j + 1 < n ? pos[j + 1] : far;
		set_pair(cols, p, a, c);
		(cols + (p >> 5) * 64 + (p & 31) + 32)->y = pack2(a.w, c.w);
		if (lo_here) set_pair(colslo, p, j < n ? poslo[j] : z, j + 1 < n ? poslo[j + 1] : z);
	}
	// own rows, the last group padded with its last row (results unused)
	for (int i = tid; i < NG * ST_RG; i += ST_T) {
		const int64_t row = row0 + min(i, rows_here - 1);
		const float4 p = pos[row];
		set_row(rown + 2 * i, p.x, p.y, p.z, near_threshold(near_scale(p.x, p.y, p.z)));
		const float4 q = poslo[row];
		set_row(rownlo + 2 * i, q.x, q.y, q.z, 0.f);
	}

	const bool deferred = integrate && multi && !clustered && K == 1;
	bool ok = true;
	for (int k = 0; k < K; ++k) {
		if (__syncthreads_or(!ok)) {
			ok = false;
			break;
		}
		// ---- the rows' accelerations: this warp's pieces ----
		int u = u0, g = g_first, cb = cb_first;
		while (u < u1) {
			int left = min(NB - cb, u1 - u);   // blocks of this piece
			u += left;
			const ulonglong2* __restrict__ rp = rown + 2 * (g * ST_RG + (lane >> 4) * 2);
			const ulonglong2* __restrict__ rlp = rownlo + 2 * (g * ST_RG + (lane >> 4) * 2);
			u64 nx[2], ny[2], nz[2], lx[2], ly[2], lz[2];   // the rows; DS: their low parts
			u64 sx[2], sy[2], sz[2];                        // second-level sums
			// NEAR: r2 as an integer less eps2 + 1 is below `near_below` for near pairs; self
			// pairs and coincident bodies (r2 = eps2) wrap to the largest integers
			const uint32_t eps_bits = __float_as_uint(eps2) + 1u;
			uint32_t near_below[2];
			float thr[2];
			float common = 0.f;   // SHARED: the radius^2 that the group's rows share
			if (SHARED) {
				float own[ST_RG];
#pragma unroll
				for (int i = 0; i < ST_RG; ++i)
					own[i] = reinterpret_cast<const float*>(rown + 2 * (g * ST_RG + i) + 1)[2];
				common = common_scale<ST_RG, 256>(own, ST_RG);
			}
#pragma unroll
			for (int r = 0; r < 2; ++r) {
				const ulonglong2 xy = rp[2 * r], zt = rp[2 * r + 1];
				nx[r] = xy.x;
				ny[r] = xy.y;
				nz[r] = zt.x;
				if (DS) {
					const ulonglong2 lxy = rlp[2 * r], lzz = rlp[2 * r + 1];
					lx[r] = lxy.x;
					ly[r] = lxy.y;
					lz[r] = lzz.x;
				}
				if (NEAR) {
					float unused;
					unpack2(zt.y, thr[r], unused);
					if (SHARED) thr[r] = fmaxf(thr[r], common);
					const uint32_t t = __float_as_uint(thr[r]);
					near_below[r] = t > eps_bits ? t - eps_bits : 0u;
				}
				sx[r] = sy[r] = sz[r] = 0ull;
			}
			do {
				const int m = min(ST_SEG, left);
				const ulonglong2* __restrict__ cp = cols + cb * 64 + c16;
				const ulonglong2* __restrict__ cl = colslo + cb * 64 + c16;
				uint32_t nmask = 0;   // NEAR: bit q of a block q that holds a near pair
#pragma unroll 1
				for (int q0 = 0; q0 < m; q0 += ST_CHUNK) {
					const int q1 = min(m, q0 + ST_CHUNK);
					u64 fx[2], fy[2], fz[2];
#pragma unroll
					for (int r = 0; r < 2; ++r) fx[r] = fy[r] = fz[r] = 0ull;
#pragma unroll (NEAR ? 4 : 2)
					for (int q = q0; q < q1; ++q, cp += 64, cl += 64) {
						uint32_t rmin[2] = {0xffffffffu, 0xffffffffu};
#pragma unroll
						for (int i = 0; i < 2; ++i) {
							const ulonglong2 cxy = cp[16 * i], czw = cp[16 * i + 32];
							ulonglong2 dxy = make_ulonglong2(0ull, 0ull), dzz = dxy;
							if (DS) {
								dxy = cl[16 * i];
								dzz = cl[16 * i + 32];
							}
#pragma unroll
							for (int r = 0; r < 2; ++r) {
								u64 dx = add2(cxy.x, nx[r]), dy = add2(cxy.y, ny[r]), dz = add2(czw.x, nz[r]);
								if (DS) {
									dx = add2(dx, add2(dxy.x, lx[r]));
									dy = add2(dy, add2(dxy.y, ly[r]));
									dz = add2(dz, add2(dzz.x, lz[r]));
								}
								float ra, rb;
								unpack2(fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, eps22))), ra, rb);
								if (NEAR)
									rmin[r] = min(__float_as_uint(ra) - eps_bits,
										min(__float_as_uint(rb) - eps_bits, rmin[r]));
								const u64 inv = pack2(rsqrt_sfu(ra), rsqrt_sfu(rb));
								const u64 w = mul2(mul2(czw.y, inv), mul2(inv, inv));
								fx[r] = fma2(dx, w, fx[r]);
								fy[r] = fma2(dy, w, fy[r]);
								fz[r] = fma2(dz, w, fz[r]);
							}
						}
						if (NEAR && (rmin[0] < near_below[0] || rmin[1] < near_below[1])) nmask |= 1u << q;
					}
#pragma unroll
					for (int r = 0; r < 2; ++r) {
						sx[r] = add2(sx[r], fx[r]);
						sy[r] = add2(sy[r], fy[r]);
						sz[r] = add2(sz[r], fz[r]);
					}
				}
				if (SHARED && __reduce_add_sync(0xffffffffu, __popc(nmask)) > 2u * m) {
					// near pairs in more than one of 16 lanes' blocks: the rows' own radii from here on
#pragma unroll
					for (int r = 0; r < 2; ++r) {
						thr[r] = reinterpret_cast<const float*>(rp + 2 * r + 1)[2];
						const uint32_t t = __float_as_uint(thr[r]);
						near_below[r] = t > eps_bits ? t - eps_bits : 0u;
					}
				}
				if (NEAR) {
					// cold path: each lane goes through the blocks where it met a pair within the near
					// radius, one such pair at a time, all lanes side by side
					while (nmask) {
						const int at = (cb + __ffs(nmask) - 1) * 64 + c16;
						nmask &= nmask - 1;
						uint32_t found = 0;   // bit 4 i + 2 r + h: column h of pair i against row r
#pragma unroll
						for (int i = 0; i < 2; ++i) {
							const ulonglong2 cxy = cols[at + 16 * i], czw = cols[at + 16 * i + 32];
#pragma unroll
							for (int r = 0; r < 2; ++r) {
								const u64 dx = add2(cxy.x, nx[r]), dy = add2(cxy.y, ny[r]), dz = add2(czw.x, nz[r]);
								float ra, rb;
								unpack2(fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, eps22))), ra, rb);
								if ((ra < thr[r]) & (ra > eps2)) found |= 1u << (4 * i + 2 * r);
								if ((rb < thr[r]) & (rb > eps2)) found |= 2u << (4 * i + 2 * r);
							}
						}
						while (found) {
							const int bit = __ffs(found) - 1;
							found &= found - 1;
							const int i = bit >> 2, r = bit >> 1 & 1, h = bit & 1;
							const float* cf = reinterpret_cast<const float*>(cols + at + 16 * i) + h;
							const float* rf = reinterpret_cast<const float*>(rp + 2 * r);
							const float* lf = reinterpret_cast<const float*>(rlp + 2 * r);
							// the padding columns are near only a body that sits where they do
							const int j = min((at & ~63) + 2 * (16 * i + c16) + h, n - 1);
							float4 lj;
							if (lo_here) {
								const float* clf = reinterpret_cast<const float*>(colslo + at + 16 * i) + h;
								lj = make_float4(clf[0], clf[2], clf[128], 0.f);
							} else if (k == 0) {
								lj = poslo[j];
							} else {
								const float4* glo = xbuf + (((k - 1) & 1) * 2 + 1) * words + j;
								u128 w = load_word(glo);
								ok = wait_word(glo, tag0 + static_cast<uint32_t>(k) - 1, w, &expired) && ok;
								lj = word_position(w);
							}
							const float dx = cf[0] + rf[0], dy = cf[2] + rf[2], dz = cf[128] + rf[4];
							const float r2 = fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, eps2)));
							float ex, ey, ez;
							near_delta(dx, dy, dz, r2, lj, make_float4(-lf[0], -lf[2], -lf[4], 0.f), eps2,
								true, ex, ey, ez);
							const u64 gm = pack2(cf[130], 0.f);
							if (r) {
								sx[1] = fma2(pack2(ex, 0.f), gm, sx[1]);
								sy[1] = fma2(pack2(ey, 0.f), gm, sy[1]);
								sz[1] = fma2(pack2(ez, 0.f), gm, sz[1]);
							} else {
								sx[0] = fma2(pack2(ex, 0.f), gm, sx[0]);
								sy[0] = fma2(pack2(ey, 0.f), gm, sy[0]);
								sz[0] = fma2(pack2(ez, 0.f), gm, sz[0]);
							}
						}
					}
					__syncwarp();
				}
				left -= m;
				cb += m;
			} while (left > 0);
			// the rows' sums over their 16 lanes: after the first round lanes 8 q .. 8 q + 7 hold
			// row q's three components
			float v[2][3], t;
#pragma unroll
			for (int r = 0; r < 2; ++r) {
				unpack2(sx[r], v[r][0], t);
				v[r][0] += t;
				unpack2(sy[r], v[r][1], t);
				v[r][1] += t;
				unpack2(sz[r], v[r][2], t);
				v[r][2] += t;
			}
			const bool second = lane & 8;
#pragma unroll
			for (int i = 0; i < 3; ++i) {
				const float give = second ? v[0][i] : v[1][i], keep = second ? v[1][i] : v[0][i];
				v[0][i] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
			}
#pragma unroll
			for (int o = 4; o > 0; o >>= 1)
#pragma unroll
				for (int i = 0; i < 3; ++i) v[0][i] += __shfl_xor_sync(0xffffffffu, v[0][i], o);
			// pieces in (warp, group) order take distinct slots warp + group
			const int c8 = lane & 7;
			if (c8 < 3)
				red[(g + warp) * (ST_RG * 3) + (lane >> 3) * 3 + c8] =
					c8 == 0 ? v[0][0] : (c8 == 1 ? v[0][1] : v[0][2]);
			++g;
			cb = 0;
		}
		const bool last = k + 1 == K;
		if (last) {
			if (__syncthreads_or(!ok)) {
				ok = false;
				break;
			}
		} else {
			__syncthreads();
		}

		// a single-step launch writes the positions it read: in a cluster once every CTA is
		// done with them, else the last CTA out copies them over (with more steps, each CTA has
		// by now read every other CTA's later ones)
		const bool settle = integrate && clustered && K == 1;
		if (settle) cluster_arrive();

		// ---- stage 2 of this lane's row component ----
		if (warp_rows) {
			double a = 0.0;
			if (mine) {
				float h = 0.f, l = 0.f;
				for (int w = w_lo; w <= w_hi; ++w)
					two_sum_acc(h, l, red[(grow + w) * (ST_RG * 3) + (rl % ST_RG) * 3 + rc]);
				a = static_cast<double>(h) + static_cast<double>(l);
			}
			if (integrate) {
				// the base class's update with separately rounded products and sums
				// (_base_.py:58-62, np2.py:110-115), as stage2.cu applies it
				vv = __dadd_rn(__dmul_rn(a, Tu), vv);
				rr = __dadd_rn(__dmul_rn(vv, Tu), rr);
				const float hx = __double2float_rn(rr);
				const float hy = __shfl_down_sync(0xffffffffu, hx, 1);
				const float hz = __shfl_down_sync(0xffffffffu, hx, 2);
				const bool lead = mine && rc == 0;
				const bool publish = lead && multi && (!last || deferred);
				if (publish) store_word(xbuf + (k & 1) * 2 * words + row0 + rl, hx, hy, hz, tag0 + k);
				const float lx = __double2float_rn(__dsub_rn(rr, static_cast<double>(hx)));
				const float ly = __shfl_down_sync(0xffffffffu, lx, 1);
				const float lz = __shfl_down_sync(0xffffffffu, lx, 2);
				if (publish)
					store_word(xbuf + ((k & 1) * 2 + 1) * words + row0 + rl, lx, ly, lz, tag0 + k);
				if (last) {
					// ---- the launch's results: state and stage-1 positions ----
					if (settle) cluster_wait();
					if (mine) {
						rd[e] = rr;
						vd[e] = vv;
						if (!deferred) {
							float* const q = reinterpret_cast<float*>(b.pos) + e;
							*q = hx;
							q[4 * b.n_pad_total] = lx;
						}
					}
				} else if (lead) {
					// own rows for the next step; the last row also stands in for the padding rows
					const float thr = near_threshold(near_scale(hx, hy, hz));
					const int i1 = rl == rows_here - 1 ? NG * ST_RG : rl + 1;
					for (int i = rl; i < i1; ++i) {
						set_row(rown + 2 * i, hx, hy, hz, thr);
						set_row(rownlo + 2 * i, lx, ly, lz, 0.f);
					}
					if (!multi) {
						set_column(cols, rl, hx, hy, hz);
						if (lo_here) set_column(colslo, rl, lx, ly, lz);
					}
				}
			}
			if (mine && (flags & GRAV_S2_WRITE_A) && (last || a_stride)) {
				double* const ao = b.a_out + k * a_stride + e;
				__stcs(ao, a);
				if (rc == 2) __stcs(ao + 1, 0.0);
			}
		} else if (settle) {
			cluster_wait();
		}

		// ---- every body's new position ----
		if (multi && !last) {
			const float4* __restrict__ src = xbuf + (k & 1) * 2 * words;
			const uint32_t want = tag0 + k;
			for (int p = tid; 2 * p < n; p += ST_T) {
				const int j = 2 * p, j1 = min(j + 1, n - 1);
				u128 w0 = load_word(src + j), w1 = load_word(src + j1), l0 = 0, l1 = 0;
				if (lo_here) {
					l0 = load_word(src + words + j);
					l1 = load_word(src + words + j1);
				}
				ok = ok && wait_word(src + j, want, w0) && wait_word(src + j1, want, w1);
				float4 c = word_position(w1);
				if (j + 1 >= n) c = make_float4(FAR_PAD, FAR_PAD, FAR_PAD, 0.f);
				set_pair(cols, p, word_position(w0), c);
				if (lo_here) {
					ok = ok && wait_word(src + words + j, want, l0) && wait_word(src + words + j1, want, l1);
					c = word_position(l1);
					if (j + 1 >= n) c = make_float4(0.f, 0.f, 0.f, 0.f);
					set_pair(colslo, p, word_position(l0), c);
				}
			}
		}
	}

	if (!ok) set_error(b.err, GRAV_DEV_TIMEOUT);
	// the last CTA out hands the tags on for the next launch and, after a deferred single step,
	// moves the new positions into the stage-1 array that every CTA has now read
	if (multi) {
		__shared__ int last_out;
		__threadfence();
		__syncthreads();
		if (tid == 0) {
			last_out = atomicAdd(&head->departed, 1) == G - 1;
			__threadfence();
		}
		__syncthreads();
		if (last_out) {
			if (deferred) {
				float* const q = reinterpret_cast<float*>(b.pos);
				constexpr int IN_FLIGHT = 4;
				for (int j0 = tid; j0 < n; j0 += IN_FLIGHT * ST_T) {
					u128 h[IN_FLIGHT], l[IN_FLIGHT];
#pragma unroll
					for (int i = 0; i < IN_FLIGHT; ++i) {
						const int j = min(j0 + i * ST_T, n - 1);
						h[i] = load_word(xbuf + j);
						l[i] = load_word(xbuf + words + j);
					}
#pragma unroll
					for (int i = 0; i < IN_FLIGHT; ++i) {
						const int j = j0 + i * ST_T;
						if (j >= n) continue;
						const float4 p = word_position(h[i]);
						*reinterpret_cast<float2*>(q + 4 * j) = make_float2(p.x, p.y);
						q[4 * j + 2] = p.z;
						reinterpret_cast<float4*>(q)[b.n_pad_total + j] = word_position(l[i]);
					}
				}
			}
			if (tid == 0) {
				head->departed = 0;
				head->epoch = tag0 - 1 + static_cast<uint32_t>(K);
			}
		}
	}
	grid_dep_launch();
}

namespace {

// Rows share a near radius where the two-launch kernels' threads share one among their rows: 4
// or 8 of them on unique pairs; on all pairs two from ~4100 to ~7000 bodies, one elsewhere.
// Where they share, rows with radii of their own are less exact: rms force error at 6000
// bodies, cube / Gaussian cloud, 2.0e-7 / 1.7e-7 alone, 1.3e-7 / 0.9e-7 shared, 1.4e-7 / 1.0e-7
// with the unique-pair kernels, at 20.7 and 21.5 us a step (2500 bodies 6.9 and 7.4).  Where
// they do not, rows alone are as exact as theirs (4096 bodies 2.1e-7 / 1.8e-7 against 2.2e-7 /
// 1.9e-7, 9000 1.8e-7 / 1.5e-7 against 1.9e-7 / 1.5e-7) and 4 % faster.  A piece that meets
// near pairs in more than one of 16 lanes' blocks (of 8 pairs) goes on with the rows' own
// radii: two Plummer spheres of 6100 bodies take 58 us a step (own radii alone 55, shared to
// the end 146), bodies spread over four decades 32 (23, 120), in the error of which the pairs
// between the two radii show (norm 2.3e-7; 3.2e-7 own, 1.6e-7 shared).
int steps_kind(int mode, int n)
{
	switch (mode) {
	case GRAV_MODE_FP32C: case GRAV_MODE_FP32CU: return STEPS_DS;
	case GRAV_MODE_FP32N: return n > 4096 && n <= 7000 ? STEPS_NEAR_SHARED : STEPS_NEAR;
	case GRAV_MODE_FP32UN: return STEPS_NEAR_SHARED;
	default: return -1;
	}
}

const void* steps_fn(int kind)
{
	return kind == STEPS_DS     ? reinterpret_cast<const void*>(&steps_kernel<STEPS_DS>)
	       : kind == STEPS_NEAR ? reinterpret_cast<const void*>(&steps_kernel<STEPS_NEAR>)
	                            : reinterpret_cast<const void*>(&steps_kernel<STEPS_NEAR_SHARED>);
}

}  // namespace

// Rows per CTA: few bodies one CTA; up to 512 at most 16 CTAs (one cluster); above, one CTA per
// SM, whole groups of 4 rows.  One CTA needs no exchange, but from 41 rows on two warps of a
// scheduler share its FP64 unit: a step of a long launch takes 1.65 us at 17 bodies, 1.92 at 48
// and 2.19 at 64 in one CTA, 1.95 in a cluster at any of them.  A cluster's launch costs 1.4 us
// more, which eight steps of 64 bodies win back.
int steps_rows(int n, int sms, int steps)
{
	if (n <= 48 || (n <= 64 && steps < 8)) return 64;
	const int ctas = n <= 512 ? static_cast<int>(EXCHANGE_CLUSTER_MAX) : sms;
	return (n + ST_RG * ctas - 1) / (ST_RG * ctas) * ST_RG;
}

// Whether grav_steps can take n bodies of `mode` on a GPU of `sms` SMs: the positions and a
// CTA's rows fit its shared memory, and a CTA's rows its threads.
bool steps_supported(int mode, int n, int sms)
{
	const int kind = steps_kind(mode, n);
	if (kind < 0 || n < 1 || sms < 1 || n > ST_MAX_ROWS * sms) return false;
	const int R = steps_rows(n, sms, 1);
	return R <= ST_MAX_ROWS && StepsSmem(kind, n, R).bytes <= ST_SMEM_MAX;
}

int64_t steps_scratch(int n)
{
	const int64_t words = (static_cast<int64_t>(n) + ST_CB - 1) / ST_CB * ST_CB;
	return EXCHANGE_HEAD_BYTES + 4 * words * 16;
}

cudaError_t launch_steps(const grav_batch& b, int flags, int steps, int64_t a_stride, void* scratch,
	int sms, cudaStream_t stream)
{
	const int n = static_cast<int>(b.n_bodies);
	const int kind = steps_kind(b.mode, n);
	const void* fn = steps_fn(kind);
	int R = steps_rows(n, sms, steps);
	const int smem = StepsSmem(kind, n, R).bytes;
	const unsigned grid = static_cast<unsigned>((n + R - 1) / R);
	grav_batch copy = b;
	int f = flags, K = steps;
	unsigned char* s = static_cast<unsigned char*>(scratch);
	void* args[] = {&copy, &f, &K, &a_stride, &R, &s};
	const bool integrate = grid > 1 && (flags & GRAV_S2_INTEGRATE);
	return launch_exchanging(fn, grid, ST_T, smem, integrate, integrate && steps > 1, stream, args);
}

}  // namespace grav
