// adjoint_steps.cu -- K backward steps of one universe in one launch (grav_adjoint_steps).
//
// The transposed step of adjoint.cu (derivation there) with the forward's accelerations kept,
// in the scheme of steps.cu: one grid of at most one CTA per SM stays for all K steps, every
// CTA holds all bodies' FP32 positions and u in shared memory, completes h and g of its rows
// over all columns, updates the rows' FP64 state and exchanges what the next step needs.  The
// two launches per step it replaces (pair kernel, adjoint stage 2) were bound by launch, drain
// and the slots' way through memory up to some thousands of bodies: 13.3 us per step at 64
// bodies, 13.8 at 1000, 22.9 at 4096, 55 at 6900; here 2.2, 3.9, 20.0 and 52, of which the pair
// loop's FMA-pipe instructions need 11.3 and 32 at the last two.
//
// Exchange.  Tagged 128-bit words as in steps.cu: u of the next step once h is known, in two
// alternating buffers, and the reversed position.  The reversal r_k = r_{k+1} - T v_{k+1},
// v_k = v_{k+1} - T a_k needs no pair result, so a row's position of step k + 2 goes out
// while it waits for the others' u of step k + 1; its buffers are three: whoever writes step
// k + 2's has read every CTA's u of step k, which that CTA published after it had read
// step k - 1's positions.
//
// Pair loop.  Rows in groups of 4, columns in blocks of 64, two rows and two packed column
// pairs per lane as in steps.cu; 27 packed FMA-pipe instructions and two reciprocal square
// roots per row and pair of columns (54 cycles), in the notation of adjoint.cu, per row
//     P += inv3 u_j,  S += Gm_j inv3,  -Q += (Gm_j d.u_i - Gm_i d.u_j) inv2 inv3 d,
//     D += inv3 d.u_j,      h = Gm_i P - u_i S - 3 Q and g = D, formed every 16 blocks.
// Zero separations are selected away (inv = 0).  Partials are FP32 over 16 blocks (32 terms
// per lane and column parity), added into a second FP32 level; lanes and the warps' pieces of
// a row are added by TwoSum in a fixed order: nothing depends on scheduling.
#include "exchange.cuh"

namespace grav {

constexpr int AT_T = 512;            // threads per CTA
constexpr int AT_W = AT_T / 32;
constexpr int AT_RG = 4;             // rows per group
constexpr int AT_CB = 64;            // columns per block
constexpr int AT_CHUNK = 16;         // blocks per first-level FP32 sum
constexpr int AT_RPW = 8;            // rows whose state one warp holds (4 lanes each)
constexpr int AT_MAX_ROWS = AT_RPW * AT_W;
constexpr int AT_SMEM_MAX = 227 * 1024;

// Padding columns: no mass, no u, and at a distance whose powers stay finite.
constexpr float AT_PAD = 1e9f;

// Shared memory of one CTA for n bodies and R rows per CTA (byte offsets, 16-byte units).
struct AdjointStepsSmem {
	int rown;   // after cols, [blocks][4][32] ulonglong2: (x0, x1 | y0, y1), (z | Gm), (ux | uy), (uz |)
	int red;    // after rows, [rows][4] ulonglong2: (-x | -y), (-z | -Gm), (ux | uy), (uz |), doubled
	int bytes;  // red: [groups + warps][AT_RG][4] float2, the pieces' sums of -h and g (hi, lo)
	__host__ __device__ AdjointStepsSmem(int n, int rows)
	{
		const int nb = (n + AT_CB - 1) / AT_CB;
		const int ng = (rows + AT_RG - 1) / AT_RG;
		rown = nb * 2048;
		red = rown + ng * AT_RG * 64;
		bytes = red + (ng + AT_W) * AT_RG * 32;
	}
};

__device__ __forceinline__ u64 twice(float x) { return pack2(x, x); }

// A row's doubled entries; Gm stays as set_mass left it.
__device__ __forceinline__ void set_adjoint_row(ulonglong2* p, float x, float y, float z, float ux,
	float uy, float uz)
{
	p[0] = make_ulonglong2(twice(-x), twice(-y));
	p[1].x = twice(-z);
	p[2] = make_ulonglong2(twice(ux), twice(uy));
	p[3].x = twice(uz);
}

// Columns 2 p and 2 p + 1.
__device__ __forceinline__ void set_adjoint_pair(ulonglong2* cols, int p, const float4& a,
	const float4& c, const float4& ua, const float4& uc)
{
	ulonglong2* q = cols + (p >> 5) * 128 + (p & 31);
	q[0] = make_ulonglong2(pack2(a.x, c.x), pack2(a.y, c.y));
	q[32].x = pack2(a.z, c.z);
	q[64] = make_ulonglong2(pack2(ua.x, uc.x), pack2(ua.y, uc.y));
	q[96].x = pack2(ua.z, uc.z);
}

// 512 threads leave 128 registers each: 132 bytes are spilled (with the chunk's g sums kept over
// the whole piece 84, in the same time from 64 to 6900 bodies).
__global__ void __launch_bounds__(AT_T, 1) adjoint_steps_kernel(const grav_batch b,
	double* __restrict__ gr, double* __restrict__ gv, double* __restrict__ ggm, float4* upos,
	const double* __restrict__ a_in, const int64_t a_stride, const int K, const int R,
	unsigned char* __restrict__ scratch)
{
	extern __shared__ __align__(16) unsigned char adjoint_smem[];
	const int tid = threadIdx.x;
	const int lane = tid & 31;
	const int warp = tid >> 5;
	const int n = static_cast<int>(b.n_bodies);
	const int row0 = blockIdx.x * R;
	const int rows_here = max(0, min(R, n - row0));
	const int NB = (n + AT_CB - 1) / AT_CB;
	const int NG = (rows_here + AT_RG - 1) / AT_RG;
	const AdjointStepsSmem L(n, R);
	ulonglong2* const cols = reinterpret_cast<ulonglong2*>(adjoint_smem);
	ulonglong2* const rown = reinterpret_cast<ulonglong2*>(adjoint_smem + L.rown);
	float2* const red = reinterpret_cast<float2*>(adjoint_smem + L.red);

	ExchangeHead* const head = reinterpret_cast<ExchangeHead*>(scratch);
	const int64_t words = static_cast<int64_t>(NB) * AT_CB;
	float4* const pbuf = reinterpret_cast<float4*>(scratch + EXCHANGE_HEAD_BYTES);  // [3][words]
	float4* const ubuf = pbuf + 3 * words;                                          // [2][words]
	const double T = b.univ[0].T;

	// this warp's units [u0, u1) of the CTA's NG x NB
	const int U = NG * NB;
	const int Wn = max(1, min(AT_W, U));
	const int u0 = warp < Wn ? warp * U / Wn : U, u1 = warp < Wn ? (warp + 1) * U / Wn : U;
	const int g_first = u0 / NB;
	const int cb_first = u0 - g_first * NB;
	const int c16 = lane & 15;             // column lane; rows 2 (lane / 16) and the next one

	// four lanes per row, eight rows per warp: lane 4 i + c holds component c of r, v, gr and gv,
	// lane 4 i + 3 the mass gradient (in `grc`, whose update it shares: the pieces hold -h and g)
	const int rl = warp * AT_RPW + lane / 4, c = lane & 3;
	const bool mine = rl < rows_here;
	const bool warp_rows = warp * AT_RPW < rows_here;
	const int grow = rl / AT_RG;
	int w_lo = 0, w_hi = -1;
	if (mine) {
		w_lo = ((grow * NB + 1) * Wn + U - 1) / U - 1;
		w_hi = ((grow + 1) * NB * Wn + U - 1) / U - 1;
	}
	const bool lead = mine && c == 0;

	// everything below belongs to the kernels before this one
	grid_dep_wait();
	const uint32_t tag0 = head->epoch + 1;
	const float4* __restrict__ pos = static_cast<const float4*>(b.pos);
	const int64_t e = 4 * static_cast<int64_t>(row0 + rl) + c;
	double rc = 0.0, vc = 0.0, grc = 0.0, gvc = 0.0, ac = 0.0;
	if (mine) {
		if (c < 3) {
			rc = b.r[e];
			vc = b.v[e];
			grc = gr[e];
			gvc = gv[e];
			ac = __ldcs(a_in + e);   // read once: evict-first
		} else {
			grc = ggm[row0 + rl];
		}
	}
	for (int p = tid; p < NB * 32; p += AT_T) {
		const float4 pad = make_float4(AT_PAD, AT_PAD, AT_PAD, 0.f), z = make_float4(0.f, 0.f, 0.f, 0.f);
		const int j = 2 * p;
		const float4 a = j < n ? pos[j] : pad, d = j + 1 < n ? pos[j + 1] : pad;
		set_adjoint_pair(cols, p, a, d, j < n ? upos[j] : z, j + 1 < n ? upos[j + 1] : z);
		cols[(p >> 5) * 128 + (p & 31) + 32].y = pack2(a.w, d.w);
	}
	// own rows, the last group padded with its last row (results unused)
	for (int i = tid; i < NG * AT_RG; i += AT_T) {
		const int64_t row = row0 + min(i, rows_here - 1);
		const float4 p = pos[row], q = upos[row];
		set_adjoint_row(rown + 4 * i, p.x, p.y, p.z, q.x, q.y, q.z);
		rown[4 * i + 1].y = twice(-p.w);
	}

	// u of the step at hand, and the reversal of that step: r_k, v_k and the position that the
	// next step contracts at (FP32), published for it
	double uc = gvc + T * grc;
	float nextp = 0.f;
	auto reverse = [&](int k) {
		rc = __dsub_rn(rc, __dmul_rn(vc, T));
		vc = __dsub_rn(vc, __dmul_rn(ac, T));
		if (mine && c < 3 && k + 1 < K) ac = __ldcs(a_in + (k + 1) * a_stride + e);
		nextp = __double2float_rn(__dsub_rn(rc, __dmul_rn(vc, T)));
		const float y = __shfl_down_sync(0xffffffffu, nextp, 1);
		const float z = __shfl_down_sync(0xffffffffu, nextp, 2);
		if (lead && k + 1 < K)
			store_word(pbuf + (k + 1) % 3 * words + row0 + rl, nextp, y, z, tag0 + k + 1);
	};
	if (warp_rows) reverse(0);

	bool ok = true;
	for (int k = 0; k < K; ++k) {
		if (__syncthreads_or(!ok)) {
			ok = false;
			break;
		}
		// ---- -h and g of the rows: this warp's pieces ----
		int u = u0, g = g_first, cb = cb_first;
		while (u < u1) {
			int left = min(NB - cb, u1 - u);   // blocks of this piece
			u += left;
			const ulonglong2* __restrict__ rp = rown + 4 * (g * AT_RG + (lane >> 4) * 2);
			u64 nx[2], ny[2], nz[2], ng[2], ux[2], uy[2], uz[2];   // the rows
			u64 sh[2][3], sg[2];                                    // second-level sums
#pragma unroll
			for (int r = 0; r < 2; ++r) {
				const ulonglong2 xy = rp[4 * r], zg = rp[4 * r + 1], uxy = rp[4 * r + 2];
				nx[r] = xy.x;
				ny[r] = xy.y;
				nz[r] = zg.x;
				ng[r] = zg.y;
				ux[r] = uxy.x;
				uy[r] = uxy.y;
				uz[r] = rp[4 * r + 3].x;
				sh[r][0] = sh[r][1] = sh[r][2] = sg[r] = 0ull;
			}
			do {
				const int m = min(AT_CHUNK, left);
				const ulonglong2* __restrict__ cp = cols + cb * 128 + c16;
				u64 S[2], Px[2], Py[2], Pz[2], Qx[2], Qy[2], Qz[2], D[2];
#pragma unroll
				for (int r = 0; r < 2; ++r)
					S[r] = Px[r] = Py[r] = Pz[r] = Qx[r] = Qy[r] = Qz[r] = D[r] = 0ull;
#pragma unroll 1
				for (int q = 0; q < m; ++q, cp += 128) {
#pragma unroll
					for (int i = 0; i < 2; ++i) {
						const ulonglong2 cxy = cp[16 * i], czg = cp[16 * i + 32], cu = cp[16 * i + 64];
						const u64 cuz = cp[16 * i + 96].x;
#pragma unroll
						for (int r = 0; r < 2; ++r) {
							const u64 dx = add2(cxy.x, nx[r]), dy = add2(cxy.y, ny[r]), dz = add2(czg.x, nz[r]);
							float ra, rb;
							unpack2(fma2(dz, dz, fma2(dy, dy, mul2(dx, dx))), ra, rb);
							const u64 inv = pack2(ra > 0.f ? rsqrt_sfu(ra) : 0.f, rb > 0.f ? rsqrt_sfu(rb) : 0.f);
							const u64 inv2 = mul2(inv, inv);
							const u64 inv3 = mul2(inv2, inv);
							S[r] = fma2(czg.y, inv3, S[r]);
							Px[r] = fma2(cu.x, inv3, Px[r]);
							Py[r] = fma2(cu.y, inv3, Py[r]);
							Pz[r] = fma2(cuz, inv3, Pz[r]);
							const u64 duj = fma2(dz, cuz, fma2(dy, cu.y, mul2(dx, cu.x)));
							const u64 dui = fma2(dz, uz[r], fma2(dy, uy[r], mul2(dx, ux[r])));
							D[r] = fma2(duj, inv3, D[r]);
							const u64 t = mul2(mul2(fma2(czg.y, dui, mul2(ng[r], duj)), inv2), inv3);
							Qx[r] = fma2(t, dx, Qx[r]);
							Qy[r] = fma2(t, dy, Qy[r]);
							Qz[r] = fma2(t, dz, Qz[r]);
						}
					}
				}
				const u64 m3 = twice(-3.f);
#pragma unroll
				for (int r = 0; r < 2; ++r) {
					sh[r][0] = add2(sh[r][0], fma2(ng[r], Px[r], fma2(ux[r], S[r], mul2(m3, Qx[r]))));
					sh[r][1] = add2(sh[r][1], fma2(ng[r], Py[r], fma2(uy[r], S[r], mul2(m3, Qy[r]))));
					sh[r][2] = add2(sh[r][2], fma2(ng[r], Pz[r], fma2(uz[r], S[r], mul2(m3, Qz[r]))));
					sg[r] = add2(sg[r], D[r]);
				}
				left -= m;
				cb += m;
			} while (left > 0);
			// the rows' sums over their 16 lanes by TwoSum, values and lanes halved in turn: lane
			// pair 8 q + 2 i ends with component i of row q
			float v[8], vl[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
			for (int r = 0; r < 2; ++r)
#pragma unroll
				for (int i = 0; i < 4; ++i) {
					float x, y;
					unpack2(i < 3 ? sh[r][i < 3 ? i : 0] : sg[r], x, y);
					v[4 * r + i] = x + y;
				}
#pragma unroll
			for (int o = 8, w = 4; o > 0; o >>= 1, w >>= 1) {
				const bool upper = lane & o;
#pragma unroll
				for (int i = 0; i < max(w, 1); ++i) {
					const int i2 = w ? w + i : i;   // the last round sums, every value is taken
					const float give = upper ? v[i] : v[i2], gl = upper ? vl[i] : vl[i2];
					float keep = upper ? v[i2] : v[i], kl = upper ? vl[i2] : vl[i];
					if (o < 8) kl += __shfl_xor_sync(0xffffffffu, gl, o);
					two_sum_acc(keep, kl, __shfl_xor_sync(0xffffffffu, give, o));
					v[i] = keep;
					vl[i] = kl;
				}
			}
			// pieces in (warp, group) order take distinct slots warp + group
			if (!(lane & 1)) red[(g + warp) * (AT_RG * 4) + (lane >> 1)] = make_float2(v[0], vl[0]);
			++g;
			cb = 0;
		}
		const bool last = k + 1 == K;
		if (__syncthreads_or(last && !ok)) {
			ok = false;
			break;
		}

		// ---- adjoint stage 2 of this lane's row component ----
		if (warp_rows) {
			float h = 0.f, l = 0.f;
			for (int w = w_lo; w <= w_hi; ++w) {
				const float2 piece = red[(grow + w) * (AT_RG * 4) + (rl % AT_RG) * 4 + c];
				two_sum_acc(h, l, piece.x);
				l += piece.y;
			}
			const double s = static_cast<double>(h) + static_cast<double>(l);   // -h, or g
			grc -= T * s;   // gr += T h, ggm -= T g
			gvc = uc;
			uc = gvc + T * grc;
			const float nu = __double2float_rn(uc);
			const float uy = __shfl_down_sync(0xffffffffu, nu, 1);
			const float uz = __shfl_down_sync(0xffffffffu, nu, 2);
			const float py = __shfl_down_sync(0xffffffffu, nextp, 1);
			const float pz = __shfl_down_sync(0xffffffffu, nextp, 2);
			if (!last) {
				if (lead) {
					store_word(ubuf + ((k + 1) & 1) * words + row0 + rl, nu, uy, uz, tag0 + k + 1);
					// own rows for the next step; the last row also stands in for the padding rows
					const int i1 = rl == rows_here - 1 ? NG * AT_RG : rl + 1;
					for (int i = rl; i < i1; ++i) set_adjoint_row(rown + 4 * i, nextp, py, pz, nu, uy, uz);
				}
				reverse(k + 1);
			} else if (mine) {
				// ---- the launch's results, prepared for a step after it ----
				if (c < 3) {
					b.r[e] = rc;
					b.v[e] = vc;
					gr[e] = grc;
					gv[e] = gvc;
					reinterpret_cast<float*>(b.pos)[e] = nextp;
					reinterpret_cast<float*>(upos)[e] = nu;
				} else {
					ggm[row0 + rl] = grc;
				}
			}
		}

		// ---- every body's next position and u ----
		if (!last) {
			const uint32_t want = tag0 + k + 1;
			const float4* __restrict__ ps = pbuf + (k + 1) % 3 * words;
			const float4* __restrict__ us = ubuf + ((k + 1) & 1) * words;
			for (int p = tid; 2 * p < n; p += AT_T) {
				const int j = 2 * p, j1 = min(j + 1, n - 1);
				u128 p0 = load_word(ps + j), p1 = load_word(ps + j1);
				u128 q0 = load_word(us + j), q1 = load_word(us + j1);
				ok = ok && wait_word(ps + j, want, p0) && wait_word(ps + j1, want, p1) &&
					wait_word(us + j, want, q0) && wait_word(us + j1, want, q1);
				float4 a1 = word_position(p1), d1 = word_position(q1);
				if (j + 1 >= n) {
					a1 = make_float4(AT_PAD, AT_PAD, AT_PAD, 0.f);
					d1 = make_float4(0.f, 0.f, 0.f, 0.f);
				}
				set_adjoint_pair(cols, p, word_position(p0), a1, word_position(q0), d1);
			}
		}
	}

	if (!ok) set_error(b.err, GRAV_DEV_TIMEOUT);
	// the last CTA out hands the tags on for the next launch
	__threadfence();
	__syncthreads();
	if (tid == 0) {
		if (atomicAdd(&head->departed, 1) == static_cast<int>(gridDim.x) - 1) {
			__threadfence();
			head->departed = 0;
			head->epoch = tag0 - 1 + static_cast<uint32_t>(K);
		}
	}
	grid_dep_launch();
}

namespace {

// Rows per CTA: up to 512 bodies at most 16 CTAs (one cluster); above, one CTA per SM, whole
// groups of 4 rows.
int adjoint_steps_rows(int n, int sms)
{
	const int ctas = n <= 512 ? static_cast<int>(EXCHANGE_CLUSTER_MAX) : sms;
	return (n + AT_RG * ctas - 1) / (AT_RG * ctas) * AT_RG;
}

}  // namespace

// Whether grav_adjoint_steps can take n bodies on a GPU of `sms` SMs: the positions, u and a
// CTA's rows fit its shared memory, and a CTA's rows its threads.
bool adjoint_steps_supported(int n, int sms)
{
	if (n < 1 || sms < 1 || n > AT_MAX_ROWS * sms) return false;
	const int R = adjoint_steps_rows(n, sms);
	return R <= AT_MAX_ROWS && AdjointStepsSmem(n, R).bytes <= AT_SMEM_MAX;
}

int64_t adjoint_steps_scratch(int n)
{
	const int64_t words = (static_cast<int64_t>(n) + AT_CB - 1) / AT_CB * AT_CB;
	return EXCHANGE_HEAD_BYTES + 5 * words * 16;
}

cudaError_t launch_adjoint_steps(const grav_batch& b, const grav_adjoint& a, int steps,
	int64_t a_stride, void* scratch, int sms, cudaStream_t stream)
{
	const int n = static_cast<int>(b.n_bodies);
	int R = adjoint_steps_rows(n, sms), K = steps;
	const unsigned grid = static_cast<unsigned>((n + R - 1) / R);
	grav_batch copy = b;
	double *gr = a.gr, *gv = a.gv, *ggm = a.ggm;
	float4* upos = static_cast<float4*>(a.upos);
	const double* a_in = a.a_in;
	unsigned char* s = static_cast<unsigned char*>(scratch);
	void* args[] = {&copy, &gr, &gv, &ggm, &upos, &a_in, &a_stride, &K, &R, &s};
	return launch_exchanging(reinterpret_cast<const void*>(&adjoint_steps_kernel), grid, AT_T,
		AdjointStepsSmem(n, R).bytes, grid > 1, grid > 1, stream, args);
}

}  // namespace grav
