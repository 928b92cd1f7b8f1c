// Kernels of one EMC iteration for sm_100a (B200); layouts in emc_common.cuh.
// Included by emc_api.cu only (one definition of each kernel).
#pragma once

#include "emc_common.cuh"

namespace dfg {

// ---------------------------------------------------------------------------
// (a) slice generation: logW[tile][p][j] = log(W_r[p]) and u_r, r = tile * TILE + j
// ---------------------------------------------------------------------------
// The model as corner quads: quad[v] holds the model at voxel v and at its
// neighbours in the last two axes, (+0, +1, +S, +S + 1), zero past the end (no
// cell reaches there). A trilinear sample then is two 32-byte loads instead of eight
// of 8 bytes (a bilinear one a single load). The slices were bound by the L1
// wavefronts of those gathers (88 % of the L1 rate, FP64 pipe 32 %): a warp's 32
// neighbouring pixels touch as many lines with each load however narrow it is.
__global__ void __launch_bounds__(256) quad_kernel(const double *__restrict__ model, long long n, long long S,
                                                   double4 *__restrict__ quad) {
	const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	auto at = [&](long long v) { return v < n ? __ldg(model + v) : 0.; };
	quad[i] = make_double4(at(i), at(i + 1), at(i + S), at(i + S + 1));
}

// Block = OB consecutive orientations (OB divides TILE); it walks every pixel in
// chunks of CB, in pixel order. Eight warps compute W of a chunk into shared
// memory (consecutive threads take consecutive pixels of one orientation, so a
// warp reads neighbouring voxels) and, after a barrier among themselves, store log W as
// coalesced row segments (max_prob.c:94-97; with Wd given, for the
// background-aware path, W itself in FP64). Meanwhile a ninth warp adds the
// previous chunk's mask-0 values to u in pixel order -- one chain of additions
// per orientation, which keeps u_r bit-identical to the reference's sequential
// sum (max_prob.c:32-38) -- and fetches the next chunk's pixels (in the storing
// threads the sums held the whole block up). Bound by the L1 path of the
// gathers; times and block sizes at slice_block_for.
template <int OB>
struct SliceShape {
	static constexpr int SAMPLES = OB >= 32 ? 2048 : 1024;  // per chunk
	static constexpr int CB = SAMPLES / OB;                  // pixels per chunk
};
constexpr int SLICE_THREADS = 288;

template <int OB, int GEO>
__global__ void __launch_bounds__(SLICE_THREADS, 3) slice_u_kernel(
    const double *__restrict__ quats, int M, int R, const double *__restrict__ qvals,
    const double *__restrict__ corr, const uint8_t *__restrict__ mask, int P, const SliceModel model,
    long long S, long long V, float *__restrict__ logW, double *__restrict__ u, double *__restrict__ Wd) {
	static_assert(TILE % OB == 0, "orientation block must divide the tile");
	constexpr int CB = SliceShape<OB>::CB;
	static_assert(256 % CB == 0, "a thread keeps one pixel of the chunk");
	constexpr int NU = OB >= 32 ? OB / 32 : 1;   // sums per lane of the ninth warp
	__shared__ double s_rot[OB][9];
	__shared__ int s_mode[OB];
	__shared__ double s_w[2][CB][OB + 1];
	__shared__ double s_q[3][CB][4];
	__shared__ int s_m[3][CB];
	const int t = threadIdx.x, lane = t & 31, r0 = blockIdx.x * OB, rt = r0 / TILE, jj0 = r0 % TILE;
	const bool sums = t >= 256;
	for (int j = t; j < OB; j += blockDim.x) {
		const int r = r0 + j;
		const int rr = r < R ? r : 0;
		geo_setup<GEO>(quats, rr / M, s_rot[j]);
		s_mode[j] = rr % M;
	}
	auto fetch = [&](int c) {
		for (int k = lane; k < CB; k += 32) {
			const int p = c * CB + k;
			if (p < P) {
				s_q[c % 3][k][0] = qvals[3 * (size_t)p];
				s_q[c % 3][k][1] = qvals[3 * (size_t)p + 1];
				s_q[c % 3][k][2] = qvals[3 * (size_t)p + 2];
				s_q[c % 3][k][3] = corr[p];
				s_m[c % 3][k] = mask[p];
			} else {
				s_m[c % 3][k] = -1;
			}
		}
	};
	if (sums)
		fetch(0);
	__syncthreads();
	const double center = (double)(S / 2);
	const int nc = (P + CB - 1) / CB;
	double acc[NU];
#pragma unroll
	for (int k = 0; k < NU; ++k)
		acc[k] = 0.;
	for (int c = 0; c <= nc; ++c) {
		if (sums) {
			if (c + 1 < nc)
				fetch(c + 1);
			if (c > 0 && lane < OB) {
				const double(*w)[OB + 1] = s_w[(c - 1) & 1];
				const int *m = s_m[(c - 1) % 3];
#pragma unroll 8
				for (int k = 0; k < CB; ++k)
					if (m[k] == 0) {
#pragma unroll
						for (int h = 0; h < NU; ++h)
							acc[h] = dadd(acc[h], w[k][lane + 32 * h]);
					}
			}
		} else if (c < nc) {
			double(*w)[OB + 1] = s_w[c & 1];
			const int i = t % CB;
			if (s_m[c % 3][i] >= 0) {
				const double *q = s_q[c % 3][i];
				const double qx = q[0], qy = q[1], qz = q[2], cr = q[3];
#pragma unroll 2
				for (int j = t / CB; j < OB; j += 256 / CB)
					w[i][j] = quad_sample<GEO>(s_rot[j], qx, qy, qz, center, S, model, (long long)s_mode[j] * V, cr);
			}
			asm volatile("bar.sync 1, 256;" ::: "memory");
			const size_t row0 = (size_t)rt * (P + 1) + (size_t)c * CB;
			const int rows = min(CB, P - c * CB);
#pragma unroll 2
			for (int idx = t; idx < rows * OB; idx += 256) {
				const int row = idx / OB, col = idx % OB;
				const size_t at = (row0 + row) * TILE + jj0 + col;
				const double v = w[row][col];
				if (Wd != nullptr)
					Wd[at] = v;
				else
					logW[at] = (float)log(v);
			}
		}
		__syncthreads();
	}
	if (sums && lane < OB) {
#pragma unroll
		for (int h = 0; h < NU; ++h) {
			const int r = r0 + lane + 32 * h;
			if (r < R)
				u[r] = acc[h];
		}
	}
}

// log w_r per orientation, so that no pair evaluates a logarithm of its
// orientation weight (max_prob.c:122).
__global__ void logw_kernel(const double *__restrict__ quats, int M, int R, double *__restrict__ logw) {
	const int r = blockIdx.x * blockDim.x + threadIdx.x;
	if (r < R)
		logw[r] = log(quats[(r / M) * 5 + 4]);
}

// rescale = mean_count / sum_r w_r u_r * M, summed in orientation order
// (max_prob.c:40, 55-60): the block stages 256 products at a time in shared
// memory and one thread adds them in order.
__global__ void __launch_bounds__(256) rescale_kernel(const double *__restrict__ u, const double *__restrict__ quats,
                                                      int M, int R, double mean_count, double *__restrict__ scalars) {
	__shared__ double s_p[256];
	double total = 0.;
	for (int r0 = 0; r0 < R; r0 += 256) {
		const int r = r0 + threadIdx.x;
		s_p[threadIdx.x] = r < R ? dmul(quats[(r / M) * 5 + 4], u[r]) : 0.;
		__syncthreads();
		if (threadIdx.x == 0) {
			const int n = min(256, R - r0);
#pragma unroll 8
			for (int k = 0; k < n; ++k)
				total = dadd(total, s_p[k]);
		}
		__syncthreads();
	}
	if (threadIdx.x == 0)
		scalars[0] = mean_count / total * M;
}

// ---------------------------------------------------------------------------
// (b) E-step: pval[tile][d][j] = log w_r - u_r * s_d + sum_k c_k logW_r[p_k]
// ---------------------------------------------------------------------------
// One warp per (orientation tile, frame), tiles outermost so that resident
// warps share one tile's log-slices in L2. Each photon costs one coalesced
// row read (one LW-wide vector load per lane) and a compensated FP32
// addition per orientation (no conversion instructions in the loop); padded
// segments need no per-photon bounds test. The photon sum is formed in FP64
// once per pair. s_d = phi_d when need_scaling &&
// (iteration > 1 || known_scale), else the rescale factor (max_prob.c:122-128).
constexpr int ESTEP_MINB = LW == 2 ? 4 : 3;

// Coarse-to-fine refinement (param->refine, max_prob.c:110-120): frame d
// evaluates orientation r only when r's coarse cell qmap[r] is one of the
// frame's relevant coarse orientations, held as one bit per coarse
// orientation in rel[d * rwords ...]. A pair that is not evaluated never
// enters the frame's list; its log-likelihood is stored as -inf, which the
// normalisation neither keeps nor takes as a maximum. qmap == nullptr: every
// pair is evaluated.
struct RefineMask {
	const int *qmap;      // [R_pad] coarse cell per orientation, -1 past R
	const uint32_t *rel;  // [N][rwords]
	int rwords;
};

// Bit k set when orientation r0 + k (k < LW) is evaluated for frame d.
__device__ __forceinline__ unsigned refine_live(const RefineMask &rm, int d, int r0) {
	if (rm.qmap == nullptr)
		return (1u << LW) - 1u;
	const uint32_t *bits = rm.rel + (size_t)d * rm.rwords;
	unsigned live = 0;
#pragma unroll
	for (int k = 0; k < LW; ++k) {
		const int c = __ldg(rm.qmap + r0 + k);
		if (c >= 0 && (__ldg(bits + (c >> 5)) >> (c & 31) & 1u))
			live |= 1u << k;
	}
	return live;
}

// A (tile, frame) task with no evaluated pair: an empty tile maximum, which
// makes the normalisation treat the tile as dead without reading its
// log-likelihoods (so none are written).
__device__ __forceinline__ void refine_skip_tile(double *__restrict__ tmax, int *__restrict__ targ, int rt,
                                                 int Nc, int dl, int lane) {
	if (lane == 0) {
		tmax[(size_t)rt * Nc + dl] = MAX_EXP_START;
		targ[(size_t)rt * Nc + dl] = -1;
	}
}

template <bool REFINE, int MINB = ESTEP_MINB>
__global__ void __launch_bounds__(256, MINB) estep_kernel(
    const float *__restrict__ logW, const double *__restrict__ u, const double *__restrict__ logw, int R,
    const uint32_t *__restrict__ ph, const long long *__restrict__ ph_off, const long long *__restrict__ ph_mid,
    const double *__restrict__ scale, const uint8_t *__restrict__ blacklist, int d0, int Nc, int use_scale,
    const double *__restrict__ scalars, int P, int RT, double *__restrict__ pval, double *__restrict__ tmax,
    int *__restrict__ targ, RefineMask rm, int t0 = 0) {
	// RT tiles from tile t0 (orientation blocks: logW holds tiles t0 ..)
	const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int lane = threadIdx.x & 31;
	if (warp >= (long long)RT * Nc)
		return;
	const int rl = (int)(warp / Nc), dl = (int)(warp - (long long)rl * Nc), d = d0 + dl, rt = t0 + rl;
	if (blacklist[d])
		return;
	const int r0 = rt * TILE + lane * LW;
	unsigned live = (1u << LW) - 1u;
	if constexpr (REFINE) {
		live = refine_live(rm, d, r0);
		if (!__any_sync(FULL, live)) {
			refine_skip_tile(tmax, targ, rt, Nc, dl, lane);
			return;
		}
	}
	const float *L = logW + (size_t)rl * (P + 1) * TILE + lane * LW;
	const long long beg = ph_off[d], mid = ph_mid[d], end = ph_off[d + 1];
	// segments start at multiples of 8 words: two 16-byte loads, identical for
	// every lane (broadcast), bring 8 photon words
	const uint4 *w4 = reinterpret_cast<const uint4 *>(ph);
	float s[LW], c[LW];
#pragma unroll
	for (int k = 0; k < LW; ++k)
		s[k] = c[k] = 0.f;
	// the next 8 words are fetched while the current 8 rows are in flight
	uint4 a = make_uint4(P, P, P, P), b = a;
	if (beg < mid) {
		a = __ldg(w4 + (beg >> 2));
		b = __ldg(w4 + (beg >> 2) + 1);
	}
	for (long long j = beg; j < mid; j += 8) {
		float v[8][LW];
		ld_row(L + a.x * TILE, v[0]);
		ld_row(L + a.y * TILE, v[1]);
		ld_row(L + a.z * TILE, v[2]);
		ld_row(L + a.w * TILE, v[3]);
		ld_row(L + b.x * TILE, v[4]);
		ld_row(L + b.y * TILE, v[5]);
		ld_row(L + b.z * TILE, v[6]);
		ld_row(L + b.w * TILE, v[7]);
		if (j + 8 < mid) {
			a = __ldg(w4 + ((j + 8) >> 2));
			b = __ldg(w4 + ((j + 8) >> 2) + 1);
		}
#pragma unroll
		for (int q = 0; q < 8; ++q)
#pragma unroll
			for (int k = 0; k < LW; ++k)
				kahan_add(s[k], c[k], v[q][k]);
	}
	for (long long j = mid; j < end; j += 8) {
		const uint4 a = __ldg(w4 + (j >> 2)), b = __ldg(w4 + (j >> 2) + 1);
		const uint32_t e[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
		float v[8][LW];
#pragma unroll
		for (int q = 0; q < 8; ++q)
			ld_row(L + (e[q] & IDX_MASK) * TILE, v[q]);
#pragma unroll
		for (int q = 0; q < 8; ++q)
#pragma unroll
			for (int k = 0; k < LW; ++k)
				kahan_add_count(s[k], c[k], e[q] >> IDX_BITS, v[q][k]);
	}
	const double sd = use_scale ? scale[d] : scalars[0];
	double acc[LW];
	// tile maximum and its lowest orientation index (strict > in ascending r,
	// as the running maximum of max_prob.c:199-202)
	double m = MAX_EXP_START;
	int am = -1;
#pragma unroll
	for (int k = 0; k < LW; ++k) {
		const int r = r0 + k;
		acc[k] = 0.;
		if (r < R) {
			double ph_sum = kahan_value(s[k], c[k]);
			acc[k] = dadd(dsub(logw[r], dmul(u[r], sd)), ph_sum);
			if (REFINE && !(live >> k & 1u))
				acc[k] = -INFINITY;
			else if (acc[k] > m) {
				m = acc[k];
				am = r;
			}
		}
	}
	st_row(pval + ((size_t)rt * Nc + dl) * TILE + lane * LW, acc);
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		double om = __shfl_xor_sync(FULL, m, o);
		int oa = __shfl_xor_sync(FULL, am, o);
		if (om > m || (om == m && oa >= 0 && (am < 0 || oa < am))) {
			m = om;
			am = oa;
		}
	}
	if (lane == 0) {
		tmax[(size_t)rt * Nc + dl] = m;
		targ[(size_t)rt * Nc + dl] = am;
	}
}

// The E-step's end where the hot pixels' photon sums are already in pval
// (emc_hot.cuh): the other photons are gathered as in estep_kernel, and the
// log-likelihood formed. A tile marked special gathers all of its photons (full)
// instead. The lists are short (tens of rows), so what a warp spends outside
// the rows counts: the grid gives tile and frame without a division, the frame's
// partial sums and the orientations' constants come as one 32-byte load per lane,
// two orientations share each compensated addition, and the tile's maximum takes
// three integer reductions (15 shuffles and their comparisons before: E-step at
// 17220 x 40000, 23 words a frame, 8.03 -> 7.49 ms; 12960 x 20001 2.61 -> 2.40).
// Issue and the L2 path bound it about equally.
struct HotLists {
	const int *special;          // [RT]
	const uint32_t *ph;          // every photon's lists
	const long long *off, *mid;
};

// Tiles with an evaluated pair under refinement, over all frames (the share of
// the pairs that a gathering E-step would visit). One warp per (tile, frame) in
// turn; out += live tiles.
__global__ void __launch_bounds__(256) refine_count_kernel(RefineMask rm, int N, int RT,
                                                           unsigned long long *__restrict__ out) {
	const int rt = blockIdx.y, lane = threadIdx.x & 31;
	unsigned live = 0;
	for (int d = blockIdx.x * 8 + (threadIdx.x >> 5); d < N; d += gridDim.x * 8)
		live += __any_sync(FULL, refine_live(rm, d, rt * TILE + lane * LW)) ? 1u : 0u;
	if (lane == 0 && live)
		atomicAdd(out, (unsigned long long)live);
}

#if DFG_LANE_W == 4   // the products need 128-orientation tiles (hot_choose)
template <bool REFINE, int MINB>
__global__ void __launch_bounds__(256, MINB) estep_cold_kernel(
    const float *__restrict__ logW, const double *__restrict__ u, const double *__restrict__ logw, int R,
    const uint32_t *__restrict__ ph, const long long *__restrict__ ph_off, const long long *__restrict__ ph_mid,
    const double *__restrict__ scale, const uint8_t *__restrict__ blacklist, int d0, int Nc, int use_scale,
    const double *__restrict__ scalars, int P, double *pval, double *__restrict__ tmax, int *__restrict__ targ,
    HotLists full, RefineMask rm) {
	const int rt = blockIdx.y, dl = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, d = d0 + dl;
	if (dl >= Nc || blacklist[d])
		return;
	unsigned live = (1u << LW) - 1u;
	if constexpr (REFINE) {
		live = refine_live(rm, d, rt * TILE + lane * LW);
		if (!__any_sync(FULL, live)) {
			refine_skip_tile(tmax, targ, rt, Nc, dl, lane);
			return;
		}
	}
	const bool special = full.special[rt] != 0;
	if (special) {
		ph = full.ph;
		ph_off = full.off;
		ph_mid = full.mid;
	}
	const long long beg = ph_off[d], mid = ph_mid[d];
	const int n1 = (int)(mid - beg) >> 3, nm = (int)(ph_off[d + 1] - mid) >> 3;  // groups of 8 words
	const float *L = logW + (size_t)rt * (P + 1) * TILE + lane * LW;
	double *const row = pval + ((size_t)rt * Nc + dl) * TILE + lane * LW;
	const uint4 *w4 = reinterpret_cast<const uint4 *>(ph + beg);
	f32x2 s[NPAIR], c[NPAIR];
#pragma unroll
	for (int h = 0; h < NPAIR; ++h)
		s[h] = c[h] = 0ull;
	uint4 a = make_uint4(P, P, P, P), b = a;
	if (n1 > 0) {
		a = __ldg(w4);
		b = __ldg(w4 + 1);
	}
	for (int j = 0; j < n1; ++j) {
		f32x2 v[8][NPAIR];
		ld_pairs(L + a.x * TILE, v[0]);
		ld_pairs(L + a.y * TILE, v[1]);
		ld_pairs(L + a.z * TILE, v[2]);
		ld_pairs(L + a.w * TILE, v[3]);
		ld_pairs(L + b.x * TILE, v[4]);
		ld_pairs(L + b.y * TILE, v[5]);
		ld_pairs(L + b.z * TILE, v[6]);
		ld_pairs(L + b.w * TILE, v[7]);
		w4 += 2;
		if (j + 1 < n1) {
			a = __ldg(w4);
			b = __ldg(w4 + 1);
		}
#pragma unroll
		for (int q = 0; q < 8; ++q)
#pragma unroll
			for (int h = 0; h < NPAIR; ++h)
				kahan_add2(s[h], c[h], v[q][h]);
	}
	for (int j = 0; j < nm; ++j, w4 += 2) {
		const uint4 x = __ldg(w4), y = __ldg(w4 + 1);
		const uint32_t e[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
		f32x2 v[8][NPAIR];
#pragma unroll
		for (int q = 0; q < 8; ++q)
			ld_pairs(L + (e[q] & IDX_MASK) * TILE, v[q]);
#pragma unroll
		for (int q = 0; q < 8; ++q)
#pragma unroll
			for (int h = 0; h < NPAIR; ++h)
				kahan_add_count2(s[h], c[h], e[q] >> IDX_BITS, v[q][h]);
	}
	double hot[LW] = {0., 0., 0., 0.}, ur[LW], lw[LW], acc[LW];
	if (!special)
		asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
		             : "=d"(hot[0]), "=d"(hot[1]), "=d"(hot[2]), "=d"(hot[3])
		             : "l"(row));
	const int r0 = rt * TILE + lane * LW;
	ld_row32(u + r0, ur);
	ld_row32(logw + r0, lw);
	const double sd = use_scale ? scale[d] : scalars[0];
	double m = MAX_EXP_START;
	int am = -1;
#pragma unroll
	for (int k = 0; k < LW; ++k) {
		float slo, shi, clo, chi;
		f2_unpack(s[k / 2], slo, shi);
		f2_unpack(c[k / 2], clo, chi);
		double sum = k & 1 ? kahan_value(shi, chi) : kahan_value(slo, clo);
		if (!special)
			sum = dadd(sum, hot[k]);
		acc[k] = 0.;
		if (r0 + k < R) {
			acc[k] = dadd(dsub(lw[k], dmul(ur[k], sd)), sum);
			if (REFINE && !(live >> k & 1u)) {
				acc[k] = -INFINITY;
			} else if (acc[k] > m) {
				m = acc[k];
				am = r0 + k;
			}
		}
	}
	asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(row), "d"(acc[0]), "d"(acc[1]), "d"(acc[2]),
	             "d"(acc[3])
	             : "memory");
	// the tile's maximum and its lowest orientation, by three integer
	// reductions over keys that order as the doubles do (no NaN is ever a maximum)
	const long long bits = __double_as_longlong(m);
	const unsigned long long key = (unsigned long long)bits ^ (bits < 0 ? ~0ull : 1ull << 63);
	const unsigned hi = __reduce_max_sync(FULL, (unsigned)(key >> 32));
	const bool top = (unsigned)(key >> 32) == hi;
	const unsigned lo = __reduce_max_sync(FULL, top ? (unsigned)key : 0u);
	const bool best = top && (unsigned)key == lo;
	am = (int)__reduce_min_sync(FULL, best ? (unsigned)am : 0xffffffffu);   // -1 (none) stays -1
	const unsigned long long got = (unsigned long long)hi << 32 | lo;
	m = __longlong_as_double((long long)(got >> 63 ? got ^ 1ull << 63 : ~got));
	if (lane == 0) {
		tmax[(size_t)rt * Nc + dl] = m;
		targ[(size_t)rt * Nc + dl] = am;
	}
}
#endif

// Near ties of the most likely orientation. The products add the log-slices
// exactly, the gathers round once per photon word, so two orientations that agree
// to a few parts in 1e9 could change places with the form of the E-step (one frame
// of 40000 at 17220 orientations). Every orientation within the forms' rounding of
// its frame's maximum is therefore summed again as estep_kernel does (the frame's
// full lists, same order, same operations): where there are several, the
// maximum and its orientation are those of the gathers, bit for bit.
// Width: a compensated FP32 addition of x is off by at most 2u|x| (u = 2^-24, the
// roundings of x - comp and, where |s| < |x|, of t - s), a digit by 2^-27. For both
// forms and two orientations that is 8u sum|x| + n 2^-26 over n photons, and sum|x|
// <= |sum x| + 2 n 31 while no log-slice is above 31; near_tie_width is twice that.
// Between two in a thousand and one in a hundred frames have a second orientation there.
// Block = 32 frames, one per lane while the tile maxima are read (the warps share the
// tiles) and the widths formed; then each warp takes four frames and counts the near
// values in the row of their best tile. Only a frame with several, or with another
// near tile, is slow: its orientations are listed and summed, up to 32 at once, one per
// lane. Bound by latency, of the few frames with the longest lists: 9 us at 420 x 450,
// 15 at 3240 x 3000, 50 at 10860 x 30000, 99 at 6300 x 15000 with 1500 photons (with 8
// rows in flight and the widths formed frame by frame 13, 27, 76 and 155 us).
__device__ __forceinline__ double near_tie_width(double sum, int photons) {
	return 0x1p-20 * (fabs(sum) + 32. * photons);
}

constexpr int TIE_WARPS = 8, TIE_FRAMES = 32 / TIE_WARPS;

__global__ void __launch_bounds__(32 * TIE_WARPS) estep_ties_kernel(
    const float *__restrict__ logW, const double *__restrict__ u, const double *__restrict__ logw, int R,
    const uint32_t *__restrict__ ph, const long long *__restrict__ ph_off, const long long *__restrict__ ph_mid,
    const double *__restrict__ scale, const uint8_t *__restrict__ blacklist, const int *__restrict__ fcounts, int d0,
    int Nc, int RT, int use_scale, const double *__restrict__ scalars, int P, double *pval, double *tmax, int *targ) {
	// largest and second largest tile maximum of each frame and warp, the tile of the
	// largest; then the frame's tile (-1: none) and lowest near value
	__shared__ double s_m[TIE_WARPS][32], s_n[TIE_WARPS][32], s_low[32];
	__shared__ int s_t[TIE_WARPS][32], s_tile[32];
	__shared__ bool s_more[32];   // another tile is near
	__shared__ int s_list[TIE_WARPS][32 + TILE];
	const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, dl0 = blockIdx.x * 32;
	auto take = [](double v, int rt, double &m, double &m2, int &t) {
		if (v > m) {
			m2 = m;
			m = v;
			t = rt;
		} else if (v > m2) {
			m2 = v;
		}
	};
	double m = MAX_EXP_START, m2 = MAX_EXP_START;
	int best = -1;
	if (dl0 + lane < Nc && !blacklist[d0 + dl0 + lane])
#pragma unroll 8
		for (int rt = w; rt < RT; rt += TIE_WARPS)
			take(tmax[(size_t)rt * Nc + dl0 + lane], rt, m, m2, best);
	s_m[w][lane] = m;
	s_n[w][lane] = m2;
	s_t[w][lane] = best;
	__syncthreads();
	if (w == 0) {
#pragma unroll
		for (int k = 1; k < TIE_WARPS; ++k) {
			take(s_m[k][lane], s_t[k][lane], m, m2, best);
			m2 = fmax(m2, s_n[k][lane]);
		}
		double low = 0.;
		if (best >= 0) {
			const int d = d0 + dl0 + lane, r = targ[(size_t)best * Nc + dl0 + lane];
			const double sd = use_scale ? scale[d] : scalars[0];
			low = m - near_tie_width(m - (logw[r] - u[r] * sd), fcounts[d]);
		}
		s_low[lane] = low;
		s_tile[lane] = best;
		s_more[lane] = m2 >= low;
	}
	__syncthreads();
	unsigned todo = 0;   // of this warp's frames
	double x[TIE_FRAMES][LW];
#pragma unroll
	for (int i = 0; i < TIE_FRAMES; ++i) {
		const int f = w * TIE_FRAMES + i, rt = s_tile[f];
		if (rt >= 0) {
			const double *row = pval + ((size_t)rt * Nc + dl0 + f) * TILE + lane * LW;
#pragma unroll
			for (int k = 0; k < LW; ++k)
				x[i][k] = row[k];
		}
	}
#pragma unroll
	for (int i = 0; i < TIE_FRAMES; ++i) {
		const int f = w * TIE_FRAMES + i, rt = s_tile[f];
		if (rt >= 0) {
			int near = 0;
#pragma unroll
			for (int k = 0; k < LW; ++k)
				near += __popc(__ballot_sync(FULL, rt * TILE + lane * LW + k < R && x[i][k] >= s_low[f]));
			if (near > 1 || s_more[f])
				todo |= 1u << i;
		}
	}
	int *const list = s_list[w];
#pragma unroll 1
	for (; todo; todo &= todo - 1) {
		const int f = w * TIE_FRAMES + __ffs(todo) - 1, dl = dl0 + f, d = d0 + dl;
		const double low = s_low[f], sd = use_scale ? scale[d] : scalars[0];
		const long long beg = ph_off[d], mid = ph_mid[d], end = ph_off[d + 1];
		// n of the listed orientations, one per lane, as estep_kernel
		auto again = [&](int i0, int n) {
			__syncwarp();
			const int r = list[i0 + (lane < n ? lane : 0)], rt = r / TILE, j = r % TILE;
			const float *L = logW + (size_t)rt * (P + 1) * TILE + j;
			float s = 0.f, c = 0.f;
			// a count of 1 adds as estep_kernel's single photons do, bit for bit, and the
			// zero row past the end (as the lists' padding) leaves s - c as it is: one
			// form for all words
			uint32_t next = beg + lane < end ? __ldg(ph + beg + lane) : (uint32_t)P;
			for (long long q = beg; q < end; q += 32) {
				const uint32_t word = next;
				next = q + 32 + lane < end ? __ldg(ph + q + 32 + lane) : (uint32_t)P;
				const bool one = q + lane < mid;
				const uint32_t at = (one ? word : word & IDX_MASK) * TILE, count = one ? 1u : word >> IDX_BITS;
				float v[32];
#pragma unroll
				for (int k = 0; k < 32; ++k)
					v[k] = __ldg(L + __shfl_sync(FULL, at, k));
#pragma unroll
				for (int k = 0; k < 32; ++k)
					kahan_add_count(s, c, __shfl_sync(FULL, count, k), v[k]);
			}
			if (lane < n)
				pval[((size_t)rt * Nc + dl) * TILE + j] = dadd(dsub(logw[r], dmul(u[r], sd)), kahan_value(s, c));
			__syncwarp();
		};
		// calls f(rt, v) for every tile whose maximum is near, v its row's values of this lane
		auto near_tiles = [&](auto &&f) {
			for (int rt0 = 0; rt0 < RT; rt0 += 32) {
				const bool near = rt0 + lane < RT && tmax[(size_t)(rt0 + lane) * Nc + dl] >= low;
				for (unsigned tiles = __ballot_sync(FULL, near); tiles; tiles &= tiles - 1) {
					const int rt = rt0 + __ffs(tiles) - 1;
					const double *row = pval + ((size_t)rt * Nc + dl) * TILE + lane * LW;
					double v[LW];
#pragma unroll
					for (int k = 0; k < LW; ++k)
						v[k] = row[k];
					f(rt, v);
				}
			}
		};
		int n = 0;
		near_tiles([&](int rt, const double (&v)[LW]) {
#pragma unroll
			for (int k = 0; k < LW; ++k) {
				const int r = rt * TILE + lane * LW + k;
				const unsigned got = __ballot_sync(FULL, r < R && v[k] >= low);
				if (got >> lane & 1u)
					list[n + __popc(got & ((1u << lane) - 1u))] = r;
				n += __popc(got);
			}
			for (; n >= 32; n -= 32)
				again(n - 32, 32);
		});
		again(0, n);
		near_tiles([&](int rt, const double (&v)[LW]) {
			double tm = MAX_EXP_START;
			int ta = -1;
#pragma unroll
			for (int k = 0; k < LW; ++k) {
				const int r = rt * TILE + lane * LW + k;
				if (r < R && v[k] > tm) {
					tm = v[k];
					ta = r;
				}
			}
#pragma unroll
			for (int o = 16; o > 0; o >>= 1) {
				const double om = __shfl_xor_sync(FULL, tm, o);
				const int oa = __shfl_xor_sync(FULL, ta, o);
				if (om > tm || (om == tm && oa >= 0 && (ta < 0 || oa < ta))) {
					tm = om;
					ta = oa;
				}
			}
			if (lane == 0) {
				tmax[(size_t)rt * Nc + dl] = tm;
				targ[(size_t)rt * Nc + dl] = ta;
			}
		});
	}
}

// ---------------------------------------------------------------------------
// (c) per-frame maximum, pruning, normalisation and frame reductions
// ---------------------------------------------------------------------------
// Asynchronous 16-byte global -> shared copies (cp.async, L2 only). Each
// lane copies and later reads its own bytes, so completion of the lane's own
// groups (cp.async.wait_group) is all the synchronisation needed; the waits
// are hardware waits on copies already issued and always end.
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
	const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Rows of a frame's log-likelihoods in flight per warp in the normalisation
// (a ring of NORM_RING 1-KB rows in shared memory per warp).
constexpr int NORM_RING = 6;

// Streams rows 0 .. RT-1 of one lane's LW doubles (row k at src + k * stride)
// through the lane's slots of a shared-memory ring, NORM_RING - 1 rows ahead
// of the one being consumed, and calls f(rt, v) for each row in order.
template <typename F>
__device__ __forceinline__ void stream_rows(const double *__restrict__ src, size_t stride, int RT,
                                            double *ring, int lane, F &&f) {
	double *mine = ring + lane * LW;
	auto issue = [&](int rt) {
		const double *g = src + (size_t)rt * stride;
		double *d = mine + (rt % NORM_RING) * TILE;
#pragma unroll
		for (int k = 0; k < LW; k += 2)
			cp_async16(d + k, g + k);
	};
#pragma unroll
	for (int k = 0; k < NORM_RING - 1; ++k) {
		if (k < RT)
			issue(k);
		cp_async_commit();
	}
	for (int rt = 0; rt < RT; ++rt) {
		if (rt + NORM_RING - 1 < RT)
			issue(rt + NORM_RING - 1);
		cp_async_commit();
		cp_async_wait<NORM_RING - 1>();   // the group of row rt has landed
		double v[LW];
		const double *d = mine + (rt % NORM_RING) * TILE;
#pragma unroll
		for (int k = 0; k < LW; k += 2) {
			const double2 x = *reinterpret_cast<const double2 *>(d + k);
			v[k] = x.x;
			v[k + 1] = x.y;
		}
		f(rt, v);
	}
	cp_async_wait<0>();
}

// One warp per frame. The reference visits orientations in ascending order
// with a running maximum m (max_prob.c:184-203): a pair enters the kept list
// when pval + 14/beta > m and, when pval > m, the list is pruned to entries
// > pval - 14/beta. With one thread the final list is: every r up to the first
// maximiser r* with pval > max - 14/beta, and every r after r* with
// pval + 14/beta > max. The maximiser is the lowest index reaching the maximum;
// it comes from the per-tile maxima the E-step wrote (lanes take tiles lane,
// lane + 32, ...). P_dr = exp(beta (pval - max)) / p_norm (max_update.c:96-98),
// formed as a product with 1 / p_norm; likelihood, psum_d, info and quat_norm
// follow max_update.c:105-130, with log(P / w_r * M) written as
// beta (pval - max) - log p_norm + log M - log w_r so that no pair evaluates a
// logarithm. The two passes over a frame's log-likelihoods keep UNR tile rows
// in flight per lane. With Pd given (background-aware path) P is also stored
// in FP64, with the same sign convention as Pst.
#ifndef DFG_NORM_MINB
#define DFG_NORM_MINB 4
#endif
// ONE (without tile skipping or the FP64 copy): one exp per kept pair. The
// first pass stores E = exp(beta (pval - max)) in FP32 in Pst and sums, per
// frame and in FP64, E, E pval, E u_r, E (y - log w_r) and E per mode; the
// second pass reads E back, writes P = E / p_norm with the sign gate and takes
// the pairs with P < PROB_MIN (which info and quat_norm leave out) back out of
// those sums. Then likelihood = sum E pval / p_norm - sum_fact, psum_d =
// rescale sum E u_r / p_norm and info = (sum' E (y - log w_r) + (log M -
// log p_norm) sum' E) / p_norm over the pairs with P >= PROB_MIN -- the
// reference's per-pair sums (max_update.c:96-130), regrouped.
template <bool MULTI, bool SKIP, bool ONE = false>
__global__ void __launch_bounds__(256, DFG_NORM_MINB) norm_kernel(
    const double *__restrict__ pval, const double *__restrict__ tmax, const int *__restrict__ targ, int RT,
    int Nc, int d0, int R, int M, const double *__restrict__ logw, const double *__restrict__ u,
    const double *__restrict__ beta, const double *__restrict__ sum_fact, const uint8_t *__restrict__ blacklist,
    int psum_d_on, const double *__restrict__ scalars, float *__restrict__ Pst, int *__restrict__ rmax,
    double *__restrict__ max_exp, double *__restrict__ p_norm, double *__restrict__ info,
    double *__restrict__ likelihood, double *__restrict__ psum_d, double *__restrict__ quat_norm,
    int *__restrict__ num_prob, double *__restrict__ Pd, uint8_t *__restrict__ tlive, int zero_dead) {
	constexpr int UNR = 2;
	// without tile skipping every row of the frame is read, twice: both passes
	// stream them through a per-warp ring (stream_rows)
	__shared__ __align__(16) double s_ring[SKIP ? 1 : 8][SKIP ? 1 : NORM_RING * TILE];
	const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int lane = threadIdx.x & 31;
	const size_t tstride = (size_t)Nc * TILE, pstride = (size_t)(Nc + 1) * TILE;
	float zero[LW];
#pragma unroll
	for (int k = 0; k < LW; ++k)
		zero[k] = 0.f;
	double zerod[LW];
#pragma unroll
	for (int k = 0; k < LW; ++k)
		zerod[k] = 0.;
	const size_t lstride = (size_t)Nc + 1;  // tlive [RT][Nc + 1]
	if (warp == Nc) {  // the zero row that padding words of the M-step point at
		for (int rt = 0; rt < RT; ++rt) {
			st_row(Pst + rt * pstride + (size_t)Nc * TILE + lane * LW, zero);
			if (Pd != nullptr)
				st_row(Pd + rt * pstride + (size_t)Nc * TILE + lane * LW, zerod);
			if (SKIP && lane == 0)
				tlive[rt * lstride + Nc] = 0;
		}
		return;
	}
	if (warp > Nc)
		return;
	const int dl = warp, d = d0 + dl;
	const double *pv = pval + (size_t)dl * TILE + lane * LW;
	float *ps = Pst + (size_t)dl * TILE + lane * LW;
	const bool bl = blacklist[d] != 0;

	double m = MAX_EXP_START;
	int am = -1;
	if (!bl) {
		for (int rt = lane; rt < RT; rt += 32) {
			double v = tmax[(size_t)rt * Nc + dl];
			if (v > m) {
				m = v;
				am = targ[(size_t)rt * Nc + dl];
			}
		}
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		double om = __shfl_xor_sync(FULL, m, o);
		int oa = __shfl_xor_sync(FULL, am, o);
		if (om > m || (om == m && oa >= 0 && (am < 0 || oa < am))) {
			m = om;
			am = oa;
		}
	}
	if (bl || m == MAX_EXP_START) {
		for (int rt = 0; rt < RT; ++rt) {
			if (!SKIP || zero_dead) {
				st_row(ps + rt * pstride, zero);
				if (Pd != nullptr)
					st_row(Pd + (size_t)dl * TILE + lane * LW + rt * pstride, zerod);
			}
			if (SKIP && lane == 0)
				tlive[rt * lstride + dl] = 0;
		}
		if (lane == 0) {
			rmax[d] = -1;
			max_exp[d] = MAX_EXP_START;
			p_norm[d] = 0.;
			info[d] = 0.;
			likelihood[d] = 0.;
			psum_d[d] = 0.;
			num_prob[d] = 0;
		}
		if (MULTI && lane < M)
			quat_norm[(size_t)d * M + lane] = 0.;
		return;
	}
	const double b = beta[d];
	const double thr = PDIFF_THRESH / b;
	const double lo = dsub(m, thr);
	const int rstar = am;

	// a tile whose maximum can keep no pair is dead: its log-likelihoods are
	// not read, its probabilities are zero (written only with zero_dead), and
	// tlive tells the later phases to skip it
	auto dead = [&](int rt) {
		if constexpr (!SKIP)
			return false;
		const double t = tmax[(size_t)rt * Nc + dl];
		return !(t > lo) && !(dadd(t, thr) > m);
	};
	if constexpr (ONE) {
		static_assert(!SKIP, "the one-exp form reads every row");
		// MULTI: sums of E per mode in shared memory, one column per lane (with a
		// register per mode every kept pair issued MAX_MODES predicated additions:
		// 12960 x 20001 in four modes 3.02 -> 1.20 ms, 1800 x 20000 in ten 0.54 -> 0.21)
		extern __shared__ double s_modes[];   // [8 warps][M][32]
		double *const qe = MULTI ? s_modes + (size_t)(threadIdx.x >> 5) * M * 32 + lane : nullptr;
		if (MULTI)
			for (int k = 0; k < M; ++k)
				qe[k * 32] = 0.;
		// mode of the lane's first orientation of row rt, and of the e-th after it
		const int step = MULTI ? TILE % M : 0;
		int mode0 = MULTI ? lane * LW % M : 0;
		auto mode_at = [&](int e) {
			int m = mode0 + e;
			m = m >= M ? m - M : m;
			return m >= M ? m - M : m;
		};
		double s = 0., sx = 0., su = 0., sy = 0.;
		int cnt = 0;
		stream_rows(pv, tstride, RT, s_ring[threadIdx.x >> 5], lane, [&](int rt, const double (&v)[LW]) {
			float out[LW];
			// (32-byte loads: 17220 x 40000 3.03 -> 2.75 ms)
			double ur[LW], lw[LW];
			ld_row32(u + rt * TILE + lane * LW, ur);
			ld_row32(logw + rt * TILE + lane * LW, lw);
#pragma unroll
			for (int e = 0; e < LW; ++e) {
				const int r = rt * TILE + lane * LW + e;
				out[e] = 0.f;
				if (r < R) {
					const double x = v[e];
					const bool kept = (r <= rstar) ? (x > lo) : (dadd(x, thr) > m);
					if (kept) {
						const double y = dmul(b, dsub(x, m));
						const double E = exp(y);
						s += E;
						sx += E * x;
						if (psum_d_on)
							su += E * ur[e];
						sy += E * (y - lw[e]);
						if (MULTI)
							qe[mode_at(e) * 32] += E;
						cnt++;
						out[e] = (float)E;   // kept pairs have y > -14: a normal FP32 value
					}
				}
			}
			if (MULTI) {
				mode0 += step;
				mode0 = mode0 >= M ? mode0 - M : mode0;
			}
			st_row(ps + rt * pstride, out);
		});
		s = warp_sum(s);
		for (int o = 16; o > 0; o >>= 1)
			cnt += __shfl_xor_sync(FULL, cnt, o);
		const double inv_s = 1. / s;
		const float inv_sf = (float)inv_s;
		// second pass: this lane's own FP32 values of the first pass, four rows
		// in flight
		double ys = 0., es = 0.;
		constexpr int R2 = 4;
		for (int rt0 = 0; rt0 < RT; rt0 += R2) {
			float ev[R2][LW];
#pragma unroll
			for (int k = 0; k < R2; ++k)
				if (rt0 + k < RT)
					ld_row_rw(ps + (rt0 + k) * pstride, ev[k]);
#pragma unroll
			for (int k = 0; k < R2; ++k) {
				const int rt = rt0 + k;
				if (rt >= RT)
					break;
				float out[LW];
#pragma unroll
				for (int e = 0; e < LW; ++e) {
					const float E = ev[k][e];
					const float P = E * inv_sf;
					out[e] = (P > (float)PROB_MIN) ? P : -P;
					if (E > 0.f && (double)E * inv_s < PROB_MIN) {
						// a kept pair that info and quat_norm leave out
						const int r = rt * TILE + lane * LW + e;
						es += (double)E;
						ys += (double)E * ((double)logf(E) - logw[r]);
						if (MULTI)
							qe[r % M * 32] -= (double)E;
					}
				}
				st_row(ps + rt * pstride, out);
			}
		}
		sx = warp_sum(sx);
		su = warp_sum(su);
		sy = warp_sum(sy);
		ys = warp_sum(ys);
		es = warp_sum(es);
		const double rescale = scalars[0], sf = sum_fact[d];
		const double cinf = log((double)M) - log(s);
		if (MULTI) {
			for (int k = 0; k < M; ++k) {
				const double v = warp_sum(qe[k * 32]);
				if (lane == 0)
					quat_norm[(size_t)d * M + k] = v * inv_s;
			}
		}
		if (lane == 0) {
			rmax[d] = rstar;
			max_exp[d] = m;
			p_norm[d] = s;
			likelihood[d] = sx * inv_s - sf;
			info[d] = ((sy - ys) + cinf * (s - es)) * inv_s;
			psum_d[d] = psum_d_on ? rescale * su * inv_s : 0.;
			num_prob[d] = cnt;
		}
		return;
	}
	double s = 0.;
	int cnt = 0;
	if constexpr (!SKIP) {
		stream_rows(pv, tstride, RT, s_ring[threadIdx.x >> 5], lane, [&](int rt, const double (&v)[LW]) {
#pragma unroll
			for (int e = 0; e < LW; ++e) {
				const int r = rt * TILE + lane * LW + e;
				if (r < R) {
					bool kept = (r <= rstar) ? (v[e] > lo) : (dadd(v[e], thr) > m);
					if (kept) {
						s += exp(dmul(b, dsub(v[e], m)));
						cnt++;
					}
				}
			}
		});
	} else
	for (int rt0 = 0; rt0 < RT; rt0 += UNR) {
		double v[UNR][LW];
		bool dd[UNR];
#pragma unroll
		for (int k = 0; k < UNR; ++k) {
			if constexpr (SKIP) {
				dd[k] = rt0 + k >= RT || dead(rt0 + k);
				if (!dd[k])
					ld_row(pv + (rt0 + k) * tstride, v[k]);
			} else {
				dd[k] = false;
				if (rt0 + k < RT)
					ld_row(pv + (rt0 + k) * tstride, v[k]);
			}
		}
#pragma unroll
		for (int k = 0; k < UNR; ++k) {
			if (rt0 + k >= RT)
				break;
			if (SKIP && dd[k])
				continue;
#pragma unroll
			for (int e = 0; e < LW; ++e) {
				const int r = (rt0 + k) * TILE + lane * LW + e;
				if (r < R) {
					bool kept = (r <= rstar) ? (v[k][e] > lo) : (dadd(v[k][e], thr) > m);
					if (kept) {
						s += exp(dmul(b, dsub(v[k][e], m)));
						cnt++;
					}
				}
			}
		}
	}
	s = warp_sum(s);
	for (int o = 16; o > 0; o >>= 1)
		cnt += __shfl_xor_sync(FULL, cnt, o);

	const double rescale = scalars[0], sf = sum_fact[d];
	const double inv_s = 1. / s, cinf = log((double)M) - log(s);
	double ll = 0., pd = 0., inf = 0.;
	double qn[MULTI ? MAX_MODES : 1];
#pragma unroll
	for (int k = 0; k < (MULTI ? MAX_MODES : 1); ++k)
		qn[k] = 0.;
	// one kept or dropped pair of the second pass: P, the frame sums, and the
	// stored probability (sign = PROB_MIN gate)
	auto pair2 = [&](int r, double x, float &out, double &outd) {
		out = 0.f;
		outd = 0.;
		if (r < R) {
			bool kept = (r <= rstar) ? (x > lo) : (dadd(x, thr) > m);
			if (kept) {
				const double y = dmul(b, dsub(x, m));
				const double P = exp(y) * inv_s;
				ll += P * (x - sf);
				if (psum_d_on)
					pd += P * u[r] * rescale;
				if (!(P < PROB_MIN)) {
					inf += P * (y + cinf - logw[r]);
					if (MULTI) {
						int mode = r % M;
#pragma unroll
						for (int q = 0; q < (MULTI ? MAX_MODES : 1); ++q)
							if (q == mode)
								qn[q] += P;
					}
				}
				out = (P > PROB_MIN) ? (float)P : -(float)P;
				outd = (P > PROB_MIN) ? P : -P;
			}
		}
	};
	if constexpr (!SKIP) {
		stream_rows(pv, tstride, RT, s_ring[threadIdx.x >> 5], lane, [&](int rt, const double (&v)[LW]) {
			float out[LW];
			double outd[LW];
#pragma unroll
			for (int e = 0; e < LW; ++e)
				pair2(rt * TILE + lane * LW + e, v[e], out[e], outd[e]);
			st_row(ps + rt * pstride, out);
			if (Pd != nullptr)
				st_row(Pd + (size_t)dl * TILE + lane * LW + rt * pstride, outd);
		});
	} else
	for (int rt0 = 0; rt0 < RT; rt0 += UNR) {
		double v[UNR][LW];
		bool dd[UNR];
#pragma unroll
		for (int k = 0; k < UNR; ++k) {
			if constexpr (SKIP) {
				dd[k] = rt0 + k >= RT || dead(rt0 + k);
				if (!dd[k])
					ld_row(pv + (rt0 + k) * tstride, v[k]);
			} else {
				dd[k] = false;
				if (rt0 + k < RT)
					ld_row(pv + (rt0 + k) * tstride, v[k]);
			}
		}
#pragma unroll
		for (int k = 0; k < UNR; ++k) {
			const int rt = rt0 + k;
			if (rt >= RT)
				break;
			if (SKIP && lane == 0)
				tlive[rt * lstride + dl] = dd[k] ? 0 : 1;
			if (SKIP && dd[k]) {
				if (zero_dead) {
					st_row(ps + rt * pstride, zero);
					if (Pd != nullptr)
						st_row(Pd + (size_t)dl * TILE + lane * LW + rt * pstride, zerod);
				}
				continue;
			}
			float out[LW];
			double outd[LW];
#pragma unroll
			for (int e = 0; e < LW; ++e)
				pair2(rt * TILE + lane * LW + e, v[k][e], out[e], outd[e]);
			st_row(ps + rt * pstride, out);
			if (Pd != nullptr)
				st_row(Pd + (size_t)dl * TILE + lane * LW + rt * pstride, outd);
		}
	}
	ll = warp_sum(ll);
	pd = warp_sum(pd);
	inf = warp_sum(inf);
	if (MULTI) {
		for (int k = 0; k < M && k < MAX_MODES; ++k) {
			double v = warp_sum(qn[k]);
			if (lane == 0)
				quat_norm[(size_t)d * M + k] = v;
		}
	}
	if (lane == 0) {
		rmax[d] = rstar;
		max_exp[d] = m;
		p_norm[d] = s;
		likelihood[d] = ll;
		info[d] = inf;
		psum_d[d] = pd;
		num_prob[d] = cnt;
	}
}

// psum_r partials: sum over a frame range of |Pst| * (phi_d or 1)
// (max_update.c:108-116). Grid (RT, splits), 8 warps per block; fixed order.
// part_max (may be null): the largest Pst of each orientation in the range, the
// unit of the M-step's fixed-point products (emc_hot.cuh).
__global__ void __launch_bounds__(256) psum_r_kernel(const float *__restrict__ Pst, int Nc, int d0,
                                                      int frames_per_split, const double *__restrict__ scale,
                                                      int need_scaling, double *__restrict__ part, int R_pad,
                                                      const uint8_t *__restrict__ tlive,
                                                      float *__restrict__ part_max) {
	__shared__ double s[8][TILE];
	__shared__ float s_m[8][TILE];
	const int rt = blockIdx.x, split = blockIdx.y, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int beg = split * frames_per_split, end = min(Nc, beg + frames_per_split);
	double acc[LW];
	float top[LW];
#pragma unroll
	for (int k = 0; k < LW; ++k) {
		acc[k] = 0.;
		top[k] = 0.f;
	}
	const float *p = Pst + (size_t)rt * (Nc + 1) * TILE + lane * LW;
	const uint8_t *live = tlive ? tlive + (size_t)rt * (Nc + 1) : nullptr;
	constexpr int UNR = 4;  // rows in flight per warp
	for (int dl0 = beg + w; dl0 < end; dl0 += 8 * UNR) {
		float v[UNR][LW];
		double f[UNR];
#pragma unroll
		for (int q = 0; q < UNR; ++q) {
			const int dl = dl0 + 8 * q;
#pragma unroll
			for (int k = 0; k < LW; ++k)
				v[q][k] = 0.f;
			f[q] = 0.;
			// dead tile: no probability (norm_kernel with tile skipping)
			if (dl < end && (live == nullptr || live[dl])) {
				ld_row(p + (size_t)dl * TILE, v[q]);
				f[q] = need_scaling ? scale[d0 + dl] : 1.;
			}
		}
#pragma unroll
		for (int q = 0; q < UNR; ++q)
			if (dl0 + 8 * q < end && (live == nullptr || live[dl0 + 8 * q])) {
#pragma unroll
				for (int k = 0; k < LW; ++k) {
					acc[k] += need_scaling ? fabs((double)v[q][k]) * f[q] : fabs((double)v[q][k]);
					top[k] = fmaxf(top[k], v[q][k]);
				}
			}
	}
#pragma unroll
	for (int k = 0; k < LW; ++k) {
		s[w][lane * LW + k] = acc[k];
		s_m[w][lane * LW + k] = top[k];
	}
	__syncthreads();
	for (int j = threadIdx.x; j < TILE; j += blockDim.x) {
		double t = 0.;
		float m = 0.f;
#pragma unroll
		for (int k = 0; k < 8; ++k) {
			t += s[k][j];
			m = fmaxf(m, s_m[k][j]);
		}
		part[(size_t)split * R_pad + rt * TILE + j] = t;
		if (part_max != nullptr)
			part_max[(size_t)split * R_pad + rt * TILE + j] = m;
	}
}

__global__ void psum_r_reduce_kernel(const double *__restrict__ part, int nsplit, int R, int R_pad,
                                     double *__restrict__ psum_r, const float *__restrict__ part_max,
                                     float *__restrict__ rowmax) {
	int r = blockIdx.x * blockDim.x + threadIdx.x;
	if (part_max != nullptr && r < R_pad) {
		float m = 0.f;
		for (int k = 0; k < nsplit; ++k)
			m = fmaxf(m, part_max[(size_t)k * R_pad + r]);
		rowmax[r] = m;
	}
	if (r >= R)
		return;
	double s = 0.;
	for (int k = 0; k < nsplit; ++k)
		s += part[(size_t)k * R_pad + r];
	psum_r[r] += s;
}

// ---------------------------------------------------------------------------
// (e1) M-step back-projection: T[tile][p][j] += sum_(d,c) c * P_dr
// ---------------------------------------------------------------------------
// Gather form of update_tomogram_nobg (max_update.c:142-230): one warp per
// (orientation tile, pixel), walking the pixel's list of frames (pixels with
// mask < 2 only) and reading one row of P per entry (one LW-wide vector load
// per lane); count-1 and multi-photon segments as in the E-step, compensated
// FP32 sums, two orientations per paired FP32 instruction (this kernel is
// bound by instruction issue; the E-step, bound by L2, gains nothing from
// pairing). No atomics; pixels are visited heaviest first for balance.
constexpr int MSTEP_MINB = LW == 4 ? 4 : 6;

template <bool SKIP, int MINB = MSTEP_MINB>
__global__ void __launch_bounds__(256, MINB) mstep_kernel(const float *__restrict__ Pst, int Nc,
                                                     const uint32_t *__restrict__ cs,
                                                     const long long *__restrict__ cs_off,
                                                     const long long *__restrict__ cs_mid,
                                                     const int *__restrict__ pix, int npix, int P, int RT,
                                                     float *__restrict__ T, const uint8_t *__restrict__ tlive,
                                                     int t0 = 0) {
	// RT tiles from tile t0 (orientation blocks: T holds tiles t0 ..)
	const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int lane = threadIdx.x & 31;
	if (warp >= (long long)RT * npix)
		return;
	const int rl = (int)(warp / npix), kp = (int)(warp - (long long)rl * npix), rt = t0 + rl;
	const int p = pix[kp];
	const float *Pr = Pst + (size_t)rt * (Nc + 1) * TILE + lane * LW;
	// SKIP: frames whose tile is dead (norm_kernel) read the chunk's zero row
	// instead (cached), so their probability rows are never fetched
	const uint8_t *live = tlive + (size_t)rt * (Nc + 1);
	const uint32_t zrow = (uint32_t)Nc;
	auto lv = [&](uint32_t f) {
		if constexpr (SKIP)
			return live[f] ? f : zrow;
		else
			return f;
	};
	const long long beg = cs_off[p], mid = cs_mid[p], end = cs_off[p + 1];
	const uint4 *w4 = reinterpret_cast<const uint4 *>(cs);
	float s[LW], c[LW];
	// orientations in pairs: paired FP32 compensated additions; the next
	// 8 words are fetched while the current 8 rows are in flight
	constexpr int NP = NPAIR;
	f32x2 s2[NP], c2[NP];
#pragma unroll
	for (int h = 0; h < NP; ++h)
		s2[h] = c2[h] = 0ull;
	uint4 a = make_uint4(Nc, Nc, Nc, Nc), b = a;
	if (beg < mid) {
		a = __ldg(w4 + (beg >> 2));
		b = __ldg(w4 + (beg >> 2) + 1);
	}
	for (long long j = beg; j < mid; j += 8) {
		if constexpr (SKIP) {
			// a group of 8 frames without a live tile adds nothing
			if (!(live[a.x] | live[a.y] | live[a.z] | live[a.w] | live[b.x] | live[b.y] | live[b.z] |
			      live[b.w])) {
				if (j + 8 < mid) {
					a = __ldg(w4 + ((j + 8) >> 2));
					b = __ldg(w4 + ((j + 8) >> 2) + 1);
				}
				continue;
			}
		}
		f32x2 v[8][NP];
		ld_pairs(Pr + lv(a.x) * TILE, v[0]);
		ld_pairs(Pr + lv(a.y) * TILE, v[1]);
		ld_pairs(Pr + lv(a.z) * TILE, v[2]);
		ld_pairs(Pr + lv(a.w) * TILE, v[3]);
		ld_pairs(Pr + lv(b.x) * TILE, v[4]);
		ld_pairs(Pr + lv(b.y) * TILE, v[5]);
		ld_pairs(Pr + lv(b.z) * TILE, v[6]);
		ld_pairs(Pr + lv(b.w) * TILE, v[7]);
		if (j + 8 < mid) {
			a = __ldg(w4 + ((j + 8) >> 2));
			b = __ldg(w4 + ((j + 8) >> 2) + 1);
		}
#pragma unroll
		for (int q = 0; q < 8; ++q)
#pragma unroll
			for (int h = 0; h < NP; ++h) {
				float lo, hi;
				f2_unpack(v[q][h], lo, hi);
				kahan_add2(s2[h], c2[h], f2_pack(fmaxf(lo, 0.f), fmaxf(hi, 0.f)));
			}
	}
	for (long long j = mid; j < end; j += 8) {
		const uint4 a = __ldg(w4 + (j >> 2)), b = __ldg(w4 + (j >> 2) + 1);
		const uint32_t e[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
		if constexpr (SKIP) {
			uint32_t any = 0;
#pragma unroll
			for (int q = 0; q < 8; ++q)
				any |= live[e[q] & IDX_MASK];
			if (!any)
				continue;
		}
		f32x2 v[8][NP];
#pragma unroll
		for (int q = 0; q < 8; ++q)
			ld_pairs(Pr + lv(e[q] & IDX_MASK) * TILE, v[q]);
#pragma unroll
		for (int q = 0; q < 8; ++q)
#pragma unroll
			for (int h = 0; h < NP; ++h) {
				float lo, hi;
				f2_unpack(v[q][h], lo, hi);
				kahan_add_count2(s2[h], c2[h], e[q] >> IDX_BITS, f2_pack(fmaxf(lo, 0.f), fmaxf(hi, 0.f)));
			}
	}
#pragma unroll
	for (int h = 0; h < NP; ++h) {
		f2_unpack(s2[h], s[2 * h], s[2 * h + 1]);
		f2_unpack(c2[h], c[2 * h], c[2 * h + 1]);
	}
	float *out = T + ((size_t)rl * P + p) * TILE + lane * LW;
	float o[LW];
	ld_row_rw(out, o);
#pragma unroll
	for (int k = 0; k < LW; ++k) {
		double t = kahan_value(s[k], c[k]);
		o[k] = (float)((double)o[k] + t);
	}
	st_row(out, o);
}

// ---------------------------------------------------------------------------
// (e2) merge: slice_merge3d of tomo_r / psum_r for every r with psum_r > 0
// ---------------------------------------------------------------------------
// Every (pixel, orientation) with mask <= 1 and in bounds adds (f * w, f) to the
// corners of its cell (model.c:171-244, max_update.c:33-36). The accumulators are
// FP64: FP32 sums of thousands of contributions per voxel would carry ~1e-6
// relative error into the next iteration's likelihoods. They are two planes of n
// = M V sums, model then weights: the weight sum depends only on which
// orientations have psum_r > 0, so when that set is the one of a cached weight
// grid with_weight is 0 and the model plane alone is touched, and a zero
// tomogram value adds nothing. With views_final the tomograms already are the
// views (background-aware update) and are not divided by psum_r.
//
// The L2's atomic units take 190e9 additions a second on a grid that fits L2
// (33e9 on one that does not: at 201^3 one plane is 65 MB, two interleaved were
// 130), so the kernel sends as few as it can. A lane walks a run of ML
// neighbouring pixels and keeps the corner sums of the cell that it is in: pixels
// in the same cell add to them in registers, and on a step into the next
// cell across a face only the face left behind goes to memory, the other one
// becomes the new cell's. All 32 runs of a warp belong to one orientation and walk
// about the same way, so the corners are numbered along that way (bit 0 behind, 1
// ahead) and a step across one face is the same code for every lane; any other
// move (a gap, an edge of the detector) writes the whole cell out. Before, the
// lanes of a warp held 32 neighbouring pixels and summed equal cells by shuffles:
// the kernel was bound by those (L1 wavefronts 85 %).
// Block = 32 runs of ML pixels x 32 orientations, their tomogram values staged
// through shared memory; rows in run order so that neither side has bank conflicts.
// Runs of 8: the last cell of a run is written out whole, twice as often as with
// runs of 16, but three blocks of warps fit an SM (two with 16: 50100 x
// 66820 61.0 against 52.2 ms). Each pair of corners is one sector for the atomic
// units: see send.
// Merge in ms before / now: 50100 x 66820 84 / 52, 17220 x 9025 4.0 / 2.5, 6300 x
// 11817 1.93 / 1.19, 3240 x 4096 0.36 / 0.23, near the solution 10860 x 15625 2.0 /
// 1.5; without the pairs 62, 3.4, 1.6, 0.31 and 1.7.
constexpr int MO = 32;  // orientations per block
constexpr int ML = 8;   // pixels per run

struct MergeShared {
	float t[ML * 32][MO + 1];
	double q[4][ML][32];   // qx, qy, qz, 1 / corr
	double rot[MO][9];
	double ips[MO];        // 1 / psum_r, 0 where it is not positive
	int mode[MO];
	unsigned use[ML];      // per step: the lanes whose pixel is merged
};

// Cell and fractions of a pixel's position, and whether the cell is inside.
template <int GEO>
__device__ __forceinline__ bool locate_axes(const double *rot, double qx, double qy, double qz, double center, int S,
                                            int (&c)[3], double (&f)[3]) {
	if constexpr (GEO == MT_3D) {
		const Cell k = locate(rot, qx, qy, qz, center, S, c);
		f[0] = k.fx;
		f[1] = k.fy;
		f[2] = k.fz;
		return k.ok;
	} else {
		const Cell2 k = locate2d(rot, qx, qy, center, S);
		c[0] = (int)(k.i00 / S);
		c[1] = (int)(k.i00 - (long long)c[0] * S);
		f[0] = k.fx;
		f[1] = k.fy;
		return k.ok;
	}
}

template <int GEO>
__global__ void __launch_bounds__(256, 3) merge_runs_kernel(
    const float *__restrict__ T, const double *__restrict__ psum_r, const double *__restrict__ quats, int M, int R,
    const double *__restrict__ qvals, const double *__restrict__ corr, const uint8_t *__restrict__ mask, int P,
    long long S, long long V, long long n, double *__restrict__ accum, const int *__restrict__ weight_flag,
    int views_final) {
	constexpr int NA = GEO == MT_3D ? 3 : 2, NC = 1 << NA;  // axes, corners
	extern __shared__ __align__(16) unsigned char merge_smem[];
	MergeShared &sh = *reinterpret_cast<MergeShared *>(merge_smem);
	const int t = threadIdx.x, w = t >> 5, lane = t & 31;
	// grid: pixel chunks fastest, then the orientation blocks
	const int chunks = (P + 32 * ML - 1) / (32 * ML), ob = blockIdx.x / chunks;
	const int p0 = (blockIdx.x - ob * chunks) * (32 * ML), rt = ob / (TILE / MO), j0 = ob % (TILE / MO) * MO;
	const int with_weight = *weight_flag, Si = (int)S;
	if (t < MO) {
		const int r = rt * TILE + j0 + t;
		const int rr = r < R ? r : 0;
		geo_setup<GEO>(quats, rr / M, sh.rot[t]);
		sh.mode[t] = rr % M;
		const double ps = r < R ? psum_r[r] : 0.;
		sh.ips[t] = ps > 0. ? fmax(fmin(1. / ps, DBL_MAX), DBL_MIN) : 0.;
	}
	// pixel p0 + l * ML + s is step s of lane l's run: row s * 32 + l
	for (int i = w; i < 32 * ML; i += 8) {
		const int p = p0 + i, row = i % ML * 32 + i / ML;
		sh.t[row][lane] = p < P ? __ldcs(T + ((size_t)rt * P + p) * TILE + j0 + lane) : 0.f;
	}
	for (int s = w; s < ML; s += 8) {
		const int p = p0 + lane * ML + s;
		const bool use = p < P && mask[p] <= 1;
		sh.q[0][s][lane] = use ? qvals[3 * (size_t)p] : 0.;
		sh.q[1][s][lane] = use ? qvals[3 * (size_t)p + 1] : 0.;
		sh.q[2][s][lane] = use ? qvals[3 * (size_t)p + 2] : 0.;
		sh.q[3][s][lane] = use ? 1. / corr[p] : 0.;
		const unsigned u = __ballot_sync(FULL, use);
		if (lane == 0)
			sh.use[s] = u;
	}
	__syncthreads();
	const double center = (double)(S / 2);
	const int stride[3] = {GEO == MT_3D ? Si * Si : Si, GEO == MT_3D ? Si : 1, 1};
	const bool odd = lane & 1;
	for (int h = 0; h < (with_weight ? 2 : 1); ++h)
		for (int j = w; j < MO; j += 8) {
			const double ips = sh.ips[j];
			if (!(ips > 0.))
				continue;
			const double *rot = sh.rot[j];
			// the way of the warp's runs: the signs of one lane's first step (a
			// wrong guess costs whole cells, nothing else)
			bool back[NA];
			int off[NC];   // corner q from corner 0, the one behind on every axis
			{
				const unsigned both = sh.use[0] & sh.use[1];
				const int l0 = both ? __ffs(both) - 1 : 0;
				double d[3];
#pragma unroll
				for (int k = 0; k < 3; ++k)
					d[k] = sh.q[k][1][l0] - sh.q[k][0][l0];
#pragma unroll
				for (int q = 0; q < NC; ++q)
					off[q] = 0;
#pragma unroll
				for (int a = 0; a < NA; ++a) {
					const double m = GEO == MT_3D ? rot[3 * a] * d[0] + rot[3 * a + 1] * d[1] + rot[3 * a + 2] * d[2]
					                              : (a == 0 ? rot[0] * d[0] - rot[1] * d[1] : rot[1] * d[0] + rot[0] * d[1]);
					back[a] = m < 0.;
#pragma unroll
					for (int q = 0; q < NC; ++q)
						if (q >> (NA - 1 - a) & 1)
							off[q] += back[a] ? -stride[a] : stride[a];
				}
			}
			double *const grid = accum + (size_t)h * n + (size_t)sh.mode[j] * V;
			uint32_t at = 0;      // corner 0 of the lane's cell (a volume has fewer than 2^32 voxels)
			int cell[NA];
			bool open = false;    // the lane holds a cell
			double v[NC];
#pragma unroll
			for (int a = 0; a < NA; ++a)
				cell[a] = 0;
#pragma unroll
			for (int q = 0; q < NC; ++q)
				v[q] = 0.;
			// Adds the corners in the lane's bit set `out`. Corners q and q | 1 are
			// consecutive doubles: neighbouring lanes trade one of the two, so that each
			// of two instructions carries both of one lane in neighbouring lanes.
			auto send = [&](unsigned out) {
				const unsigned theirs = __shfl_xor_sync(FULL, out, 1);
				const uint32_t their_at = __shfl_xor_sync(FULL, at, 1);
				const unsigned first = odd ? theirs : out, second = odd ? out : theirs;  // even lane's, odd lane's
				const uint32_t at1 = odd ? their_at : at, at2 = odd ? at : their_at;
#pragma unroll
				for (int q = 0; q < NC; q += 2) {
					const double got = __shfl_xor_sync(FULL, odd ? v[q] : v[q | 1], 1);
					const int mine = odd ? q | 1 : q;          // the corner of either cell that this lane adds
					const uint32_t o = (uint32_t)(odd ? off[q | 1] : off[q]);
					if (first >> mine & 1u)
						atomicAdd(grid + (uint32_t)(at1 + o), odd ? got : v[q]);
					if (second >> mine & 1u)
						atomicAdd(grid + (uint32_t)(at2 + o), odd ? v[q | 1] : got);
				}
			};
#pragma unroll 1
			for (int s = 0; s < ML; ++s) {
				const float tv = sh.t[s * 32 + lane][j];
				const double icr = sh.q[3][s][lane];
				bool on = (sh.use[s] >> lane & 1u) && (h || tv != 0.f || isinf(icr));
				if (!__any_sync(FULL, on))
					continue;
				int c[3];
				double f[3];
				const bool in = locate_axes<GEO>(rot, sh.q[0][s][lane], sh.q[1][s][lane], sh.q[2][s][lane], center, Si, c, f);
				on = on && in;
				// the move from the lane's cell, along the runs' way: the axes
				// crossed into the next cell, or any other move
				int far = 0;
				unsigned cross = 0;
#pragma unroll
				for (int a = 0; a < NA; ++a) {
					const int d = back[a] ? cell[a] - c[a] : c[a] - cell[a];
					far |= d;
					cross |= (unsigned)(d & 1) << (NA - 1 - a);
				}
				const bool whole = on && (!open || (far & ~1));
				if (whole || !on)
					cross = 0;
				// corners left behind: q with a crossed axis where it is behind
				constexpr unsigned long long LEFT = NA == 3 ? 0x7f3f5f0f77335500ull : 0x07030500ull;
				const unsigned left = whole ? (open ? (1u << NC) - 1u : 0u) : (unsigned)(LEFT >> (8 * cross)) & 0xffu;
				if (__any_sync(FULL, left != 0u))
					send(left);
				if (__any_sync(FULL, whole)) {
					if (whole) {
#pragma unroll
						for (int q = 0; q < NC; ++q)
							v[q] = 0.;
						uint32_t x = 0;
#pragma unroll
						for (int a = 0; a < NA; ++a)
							x += (uint32_t)(c[a] + (back[a] ? 1 : 0)) * (uint32_t)stride[a];
						at = x;
						open = true;
					}
				}
#pragma unroll
				for (int a = 0; a < NA; ++a) {
					constexpr int top = NA - 1;
					const int bit = 1 << (top - a);
					if (cross & bit) {
#pragma unroll
						for (int q = 0; q < NC; ++q)
							if (!(q & bit)) {
								v[q] = v[q | bit];
								v[q | bit] = 0.;
							}
						at += (uint32_t)off[bit];
					}
				}
				if (on) {
#pragma unroll
					for (int a = 0; a < NA; ++a)
						cell[a] = c[a];
					const double wv = h ? 1. : (views_final ? (double)tv * icr : (double)tv * ips * icr);
					double w0[NA], w1[NA];   // weight behind, ahead
#pragma unroll
					for (int a = 0; a < NA; ++a) {
						const double g = dsub(1., f[a]);
						w0[a] = back[a] ? f[a] : g;
						w1[a] = back[a] ? g : f[a];
					}
					w0[0] *= wv;
					w1[0] *= wv;
#pragma unroll
					for (int q = 0; q < NC; q += 2) {
						double x = q >> (NA - 1) & 1 ? w1[0] : w0[0];
						if (NA == 3)
							x *= q >> 1 & 1 ? w1[1] : w0[1];
						v[q] = fma(x, w0[NA - 1], v[q]);
						v[q | 1] = fma(x, w1[NA - 1], v[q | 1]);
					}
				}
			}
			if (__any_sync(FULL, open))
				send(open ? (1u << NC) - 1u : 0u);
		}
}

// The merge of the pair lists (3-D): tomogram values are mostly zero and skipped,
// and the weights are a change to the cached grid: wsign[r] = +1 / -1 adds /
// subtracts orientation r's weights (its psum_r > 0 state changed, or +1 for every
// orientation with psum_r > 0 when no grid is cached), 0 adds none. Block =
// orientation tile x PB pixels, the tomogram rows staged through shared memory.
__global__ void __launch_bounds__(256, 3) merge_change_kernel(
    const float *__restrict__ T, const double *__restrict__ psum_r, const double *__restrict__ quats, int R,
    const double *__restrict__ qvals, const double *__restrict__ corr, const uint8_t *__restrict__ mask, int P,
    long long S, long long n, double *__restrict__ accum, const signed char *__restrict__ wsign) {
	__shared__ double s_rot[TILE][9];
	__shared__ double s_ps[TILE];
	__shared__ signed char s_sg[TILE];
	__shared__ float s_tile[PB][TILE + 1];
	const int t = threadIdx.x, rt = blockIdx.y, p0 = blockIdx.x * PB;
	for (int j = t; j < TILE; j += blockDim.x) {
		const int r = rt * TILE + j;
		rot_from_quat(quats + 5 * (size_t)(r < R ? r : 0), s_rot[j]);
		const double ps = r < R ? psum_r[r] : 0.;
		s_ps[j] = ps > 0. ? fmax(fmin(1. / ps, DBL_MAX), DBL_MIN) : 0.;  // 0: not merged
		s_sg[j] = r < R ? wsign[r] : 0;
	}
	{
		const int w = t >> 5, lane = t & 31;
		for (int row = w; row < PB; row += 8) {
			const int pp = p0 + row;
			float v[LW];
#pragma unroll
			for (int k = 0; k < LW; ++k)
				v[k] = 0.f;
			if (pp < P)
				ld_row_stream(T + ((size_t)rt * P + pp) * TILE + lane * LW, v);
#pragma unroll
			for (int k = 0; k < LW; ++k)
				s_tile[row][lane * LW + k] = v[k];
		}
	}
	__syncthreads();
	const int i = t & (PB - 1), g = t >> 6, p = p0 + i;
	if (p >= P || mask[p] > 1)
		return;
	const double qx = qvals[3 * (size_t)p], qy = qvals[3 * (size_t)p + 1], qz = qvals[3 * (size_t)p + 2];
	const double icr = 1. / corr[p];
	const double center = (double)(S / 2);
	long long o[8];
	corner_offsets(S, o);
	for (int k = 0; k < TILE / 4; ++k) {
		const int j = g + 4 * k, sg = s_sg[j];
		const double ips = s_ps[j];
		const bool model = ips > 0. && s_tile[i][j] != 0.f;
		if (!model && sg == 0)
			continue;
		const Cell c = locate(s_rot[j], qx, qy, qz, center, S);
		if (!c.ok)
			continue;
		double fw[8];
		corner_weights(c, fw);
		double *a = accum + c.i000;
		if (model) {
			const double wv = (double)s_tile[i][j] * ips * icr;
#pragma unroll
			for (int q = 0; q < 8; ++q)
				atomicAdd(a + o[q], fw[q] * wv);
		}
		if (sg != 0) {
#pragma unroll
			for (int q = 0; q < 8; ++q)
				atomicAdd(a + n + o[q], sg > 0 ? fw[q] : -fw[q]);
		}
	}
}

// ---------------------------------------------------------------------------
// model update (recon.pyx:112-149) and small per-frame kernels
// ---------------------------------------------------------------------------
// Whether the merge must accumulate weights: the set of orientations with
// psum_r > 0 (the only input of the weight grid once the geometry is fixed)
// differs from the one of the cached grid, or no grid is cached. flags[0] =
// accumulate weights, flags[1] = a grid is cached (cleared by the host when
// the geometry changes). One block; the pattern is updated in place.
__global__ void __launch_bounds__(1024) weight_pattern_kernel(const double *__restrict__ psum_r, int R,
                                                              uint8_t *__restrict__ pattern, int *__restrict__ flags) {
	int changed = 0;
	for (int r = threadIdx.x; r < R; r += blockDim.x) {
		const uint8_t p = psum_r[r] > 0. ? 1 : 0;
		if (p != pattern[r]) {
			pattern[r] = p;
			changed = 1;
		}
	}
	changed = __syncthreads_or(changed);
	if (threadIdx.x == 0) {
		flags[0] = (changed || flags[1] == 0) ? 1 : 0;
		flags[1] = 1;
	}
}

// Pair lists: the weight change of this merge. sign[r] = +1 for every
// orientation with psum_r > 0 when no grid is cached (flags[0] = 1), else
// the change of its psum_r > 0 state against the cached grid's (flags[0] =
// 2: the merge's weight sums are added to the cached grid). One block.
__global__ void __launch_bounds__(1024) weight_sign_kernel(const double *__restrict__ psum_r, int R,
                                                           uint8_t *__restrict__ pattern,
                                                           signed char *__restrict__ sign, int *__restrict__ flags) {
	const bool full = flags[1] == 0;
	for (int r = threadIdx.x; r < R; r += blockDim.x) {
		const uint8_t p = psum_r[r] > 0. ? 1 : 0;
		sign[r] = full ? (signed char)p : (signed char)((int)p - (int)pattern[r]);
		pattern[r] = p;
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		flags[0] = full ? 1 : 2;
		flags[1] = 1;
	}
}

// model2 / inter_weight from the accumulators; the weights come from this
// merge (flag 1), from weight_cache (flag 0) or from weight_cache plus this
// merge's change (flag 2); weight_cache keeps the result.
__global__ void unpack_accum_kernel(const double *__restrict__ accum, long long n, double *__restrict__ model2,
                                    double *__restrict__ weight, double *__restrict__ weight_cache,
                                    const int *__restrict__ weight_flag) {
	long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	const int with_weight = *weight_flag;
	model2[i] = accum[i];
	if (with_weight == 1) {
		const double w = accum[n + i];
		weight[i] = w;
		weight_cache[i] = w;
	} else if (with_weight == 2) {
		const double w = weight_cache[i] + accum[n + i];
		weight[i] = w;
		weight_cache[i] = w;
	} else {
		weight[i] = weight_cache[i];
	}
}

__device__ __forceinline__ double friedel_avg(double a1, double w1, double a2, double w2) {
	double a = dmul(0.5, dadd(dmul(a1, w1), dmul(a2, w2)));
	double ws = dmul(0.5, dadd(w1, w2));
	return ws > 0 ? a / ws : 0.;
}

// symmetrize_friedel (model.c:470-490) over every mode. The reference visits
// (x, y, z) for x, y in [lo, S), z in [lo, c] sequentially; pairs with z < c
// are touched once, pairs inside the z == c plane twice (the second visit
// starts from the first member's result with the roles swapped). Each thread
// owns one pair and replays exactly those visits.
__global__ void friedel_kernel(double *__restrict__ model2, const double *__restrict__ weight, int S, int M) {
	const int c = S / 2, lo = (S % 2 == 0) ? 1 : 0, n = S - lo, nz = c - lo + 1;
	const long long per_mode = (long long)n * n * nz;
	long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (id >= per_mode * M)
		return;
	const int mode = (int)(id / per_mode);
	long long k = id - (long long)mode * per_mode;
	const int z = lo + (int)(k % nz);
	k /= nz;
	const int y = lo + (int)(k % n);
	const int x = lo + (int)(k / n);
	const long long V = (long long)S * S * S;
	double *a = model2 + (size_t)mode * V;
	const double *w = weight + (size_t)mode * V;
	const long long v1 = ((long long)x * S + y) * S + z;
	const long long v2 = ((long long)(2 * c - x) * S + (2 * c - y)) * S + (2 * c - z);
	if (z < c) {
		double A = friedel_avg(a[v1], w[v1], a[v2], w[v2]);
		a[v1] = A;
		a[v2] = A;
		return;
	}
	// z == c: the member visited first owns the pair
	const int mx = 2 * c - x, my = 2 * c - y;
	const bool first = (x < mx) || (x == mx && y <= my);
	if (!first)
		return;
	double A = friedel_avg(a[v1], w[v1], a[v2], w[v2]);
	if (v1 != v2)
		A = friedel_avg(A, w[v2], A, w[v1]);
	a[v1] = A;
	a[v2] = A;
}

// symmetrize_friedel2d (model.c:495-515) over every layer: (y, z) and
// (2c - y, 2c - z) for y in [lo, S), z in [lo, c], visited as friedel_kernel
// visits its pairs (the z == c line holds the pairs touched twice).
__global__ void friedel2d_kernel(double *__restrict__ model2, const double *__restrict__ weight, int S, int M) {
	const int c = S / 2, lo = (S % 2 == 0) ? 1 : 0, n = S - lo, nz = c - lo + 1;
	const long long per_layer = (long long)n * nz;
	const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (id >= per_layer * M)
		return;
	const int layer = (int)(id / per_layer);
	const long long k = id - (long long)layer * per_layer;
	const int z = lo + (int)(k % nz), y = lo + (int)(k / nz);
	const long long A2 = (long long)S * S;
	double *a = model2 + (size_t)layer * A2;
	const double *w = weight + (size_t)layer * A2;
	const long long v1 = (long long)y * S + z, v2 = (long long)(2 * c - y) * S + (2 * c - z);
	if (z < c) {
		const double A = friedel_avg(a[v1], w[v1], a[v2], w[v2]);
		a[v1] = A;
		a[v2] = A;
		return;
	}
	// z == c: the member visited first owns the pair
	if (y > 2 * c - y)
		return;
	double A = friedel_avg(a[v1], w[v1], a[v2], w[v2]);
	if (v1 != v2)
		A = friedel_avg(A, w[v2], A, w[v1]);
	a[v1] = A;
	a[v2] = A;
}

// model2 /= weight where weight > 0; squared change against model1; model1
// <- model2 or the alpha mix (recon.pyx:136-147). Block partial sums of the
// squared change go to part[blockIdx.x] for a fixed-order reduction.
template <typename MT>
__global__ void __launch_bounds__(256) divide_update_kernel(double *__restrict__ model2,
                                                            const double *__restrict__ weight,
                                                            double *__restrict__ model1, MT *__restrict__ model1_copy,
                                                            long long n, double alpha, double *__restrict__ part) {
	__shared__ double s[8];
	long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	double d2 = 0.;
	if (i < n) {
		double m2 = model2[i];
		if (weight[i] > 0.)
			m2 = m2 / weight[i];
		model2[i] = m2;
		double m1 = model1[i];
		double diff = m2 - m1;
		d2 = diff * diff;
		double nm = alpha > 0. ? alpha * m1 + (1 - alpha) * m2 : m2;
		model1[i] = nm;
		if (model1_copy != nullptr)
			model1_copy[i] = (MT)nm;
	}
	d2 = warp_sum(d2);
	if ((threadIdx.x & 31) == 0)
		s[threadIdx.x >> 5] = d2;
	__syncthreads();
	if (threadIdx.x == 0) {
		double t = 0.;
		for (int k = 0; k < 8; ++k)
			t += s[k];
		part[blockIdx.x] = t;
	}
}

// Point-group and axial symmetrisation (symmetrize_octahedral /
// symmetrize_icosahedral / symmetrize_axial, model.c:527-757, with
// rotate_model_openmp :423-468): for every voxel v = (vx, vy, vz) - c with
// vx, vy, vz in [0, S-2], sum over the n rotations g, in list order, of the
// trilinear sample of model2 * weight and of weight at g v + c (samples
// outside [0, S-1) are skipped); out = (sum A, sum W). One thread per voxel,
// FP64 in the reference's operation order. The plane index S-1 stays zero,
// as in the reference.
__global__ void symmetrize_kernel(const double *__restrict__ model2, const double *__restrict__ weight, int S,
                                  const double *__restrict__ rots, int n, double2 *__restrict__ out) {
	const long long V = (long long)S * S * S;
	const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= V)
		return;
	const int iz = (int)(i % S), iy = (int)((i / S) % S), ix = (int)(i / ((long long)S * S));
	double sa = 0., sw = 0.;
	if (ix < S - 1 && iy < S - 1 && iz < S - 1) {
		const int c = S / 2;
		const double vx = (double)(ix - c), vy = (double)(iy - c), vz = (double)(iz - c), cd = (double)c;
		const long long SS = (long long)S * S;
		for (int g = 0; g < n; ++g) {
			const double *R = rots + 9 * g;
			double rv[3];
#pragma unroll
			for (int k = 0; k < 3; ++k)
				rv[k] = dadd(dadd(dadd(dmul(R[3 * k], vx), dmul(R[3 * k + 1], vy)), dmul(R[3 * k + 2], vz)), cd);
			if (rv[0] < 0. || rv[0] >= S - 1 || rv[1] < 0. || rv[1] >= S - 1 || rv[2] < 0. || rv[2] >= S - 1)
				continue;
			const int x = (int)rv[0], y = (int)rv[1], z = (int)rv[2];
			const double fx = dsub(rv[0], (double)x), fy = dsub(rv[1], (double)y), fz = dsub(rv[2], (double)z);
			const double cx = dsub(1., fx), cy = dsub(1., fy), cz = dsub(1., fz);
			const double wts[8] = {dmul(dmul(cx, cy), cz), dmul(dmul(cx, cy), fz), dmul(dmul(cx, fy), cz),
			                       dmul(dmul(cx, fy), fz), dmul(dmul(fx, cy), cz), dmul(dmul(fx, cy), fz),
			                       dmul(dmul(fx, fy), cz), dmul(dmul(fx, fy), fz)};
			const long long b = x * SS + (long long)y * S + z;
			const long long o[8] = {0, 1, S, S + 1, SS, SS + 1, SS + S, SS + S + 1};
			double ta = 0., tw = 0.;
#pragma unroll
			for (int q = 0; q < 8; ++q) {
				const double w = __ldg(weight + b + o[q]);
				const double a = dmul(__ldg(model2 + b + o[q]), w);
				ta = q == 0 ? dmul(wts[q], a) : dadd(ta, dmul(wts[q], a));
				tw = q == 0 ? dmul(wts[q], w) : dadd(tw, dmul(wts[q], w));
			}
			sa = dadd(sa, ta);
			sw = dadd(sw, tw);
		}
	}
	out[i] = make_double2(sa, sw);
}

// model2 = sum A / sum W where sum W > 0 (else 0), weight = sum W
// (model.c:553-569, 715-729, 751-756).
__global__ void symmetrize_finish_kernel(const double2 *__restrict__ in, long long n, double *__restrict__ model2,
                                         double *__restrict__ weight) {
	const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	const double2 v = in[i];
	model2[i] = v.y > 0. ? v.x / v.y : 0.;
	weight[i] = v.y;
}

// Fixed-order sum of n doubles by one block (second stage of reductions).
__global__ void __launch_bounds__(1024) sum_kernel(const double *__restrict__ x, long long n,
                                                   double *__restrict__ out) {
	__shared__ double s[32];
	double acc = 0.;
	for (long long i = threadIdx.x; i < n; i += blockDim.x)
		acc += x[i];
	acc = warp_sum(acc);
	if ((threadIdx.x & 31) == 0)
		s[threadIdx.x >> 5] = acc;
	__syncthreads();
	if (threadIdx.x < 32) {
		double v = threadIdx.x < (blockDim.x >> 5) ? s[threadIdx.x] : 0.;
		v = warp_sum(v);
		if (threadIdx.x == 0)
			*out = v;
	}
}

// Sums of info / likelihood over good frames, and count of good frames:
// out[0] = sum info, out[1] = sum likelihood (max_prob.c:367-371); one block.
__global__ void __launch_bounds__(1024) frame_totals_kernel(const double *__restrict__ info,
                                                            const double *__restrict__ ll,
                                                            const uint8_t *__restrict__ blacklist, int N,
                                                            double *__restrict__ out) {
	__shared__ double s[2][32];
	double a = 0., b = 0.;
	for (int d = threadIdx.x; d < N; d += blockDim.x)
		if (!blacklist[d]) {
			a += info[d];
			b += ll[d];
		}
	a = warp_sum(a);
	b = warp_sum(b);
	if ((threadIdx.x & 31) == 0) {
		s[0][threadIdx.x >> 5] = a;
		s[1][threadIdx.x >> 5] = b;
	}
	__syncthreads();
	if (threadIdx.x < 32) {
		int nw = blockDim.x >> 5;
		double x = threadIdx.x < nw ? s[0][threadIdx.x] : 0., y = threadIdx.x < nw ? s[1][threadIdx.x] : 0.;
		x = warp_sum(x);
		y = warp_sum(y);
		if (threadIdx.x == 0) {
			out[0] = x;
			out[1] = y;
		}
	}
}

// beta_d = min(1, beta_start_d * factor) for good frames (recon.pyx:165-171)
__global__ void beta_kernel(const double *__restrict__ beta_start, const uint8_t *__restrict__ blacklist,
                            int N, double factor, double *__restrict__ beta) {
	int d = blockIdx.x * blockDim.x + threadIdx.x;
	if (d >= N || blacklist[d] == 1)
		return;
	double b = beta_start[d] * factor;
	beta[d] = b > 1. ? 1. : b;
}

// phi_d = fcounts_d / psum_d for good frames (max_scale.c:13-15)
__global__ void scale_kernel(const int *__restrict__ fcounts, const double *__restrict__ psum_d,
                             const uint8_t *__restrict__ blacklist, int N, double *__restrict__ scale) {
	int d = blockIdx.x * blockDim.x + threadIdx.x;
	if (d >= N || blacklist[d])
		return;
	scale[d] = fcounts[d] / psum_d[d];
}

// Good-frame sum of phi and count, for normalize_scale (one block).
__global__ void __launch_bounds__(1024) scale_sum_kernel(const double *__restrict__ scale,
                                                         const uint8_t *__restrict__ blacklist, int N,
                                                         double *__restrict__ out) {
	__shared__ double s[2][32];
	double a = 0., c = 0.;
	for (int d = threadIdx.x; d < N; d += blockDim.x)
		if (!blacklist[d]) {
			a += scale[d];
			c += 1.;
		}
	a = warp_sum(a);
	c = warp_sum(c);
	if ((threadIdx.x & 31) == 0) {
		s[0][threadIdx.x >> 5] = a;
		s[1][threadIdx.x >> 5] = c;
	}
	__syncthreads();
	if (threadIdx.x < 32) {
		int nw = blockDim.x >> 5;
		double x = threadIdx.x < nw ? s[0][threadIdx.x] : 0., y = threadIdx.x < nw ? s[1][threadIdx.x] : 0.;
		x = warp_sum(x);
		y = warp_sum(y);
		if (threadIdx.x == 0) {
			out[0] = x;
			out[1] = y;
		}
	}
}

// a[i] += b[i]: one detector's merged sums into the shared model's.
__global__ void add_into_kernel(double *__restrict__ a, const double *__restrict__ b, long long n) {
	const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n)
		a[i] += b[i];
}

// phi /= mean for good frames; model1 of mode 0 *= mean (iterate.pyx:372-382);
// mean = sums[0] / sums[1] (sum and count of good frames' phi); nothing
// changes without good frames (the host reports that case).
__global__ void apply_scale_norm_kernel(double *__restrict__ scale, const uint8_t *__restrict__ blacklist,
                                        int N, double *__restrict__ model1, float *__restrict__ model1f,
                                        long long V, const double *__restrict__ sums) {
	long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (!(sums[1] > 0.))
		return;
	const double m = sums[0] / sums[1];
	if (i < V) {
		double v = model1[i] * m;
		model1[i] = v;
		if (model1f != nullptr)
			model1f[i] = (float)v;
	}
	if (i < N && !blacklist[i])
		scale[i] /= m;
}

// Captured probability mass of watched frames (learned proposals): for watched
// frame w (chunk-local frame wl[w]) the sum of |P| over the orientations whose
// coarse cell qmap[r] is among the frame's proposed cells (bits[w * rwords ..]),
// divided by the sum over all orientations. Dead tiles (tlive 0) hold no
// probability. One warp per watched frame of the chunk.
__global__ void __launch_bounds__(256) captured_mass_kernel(const float *__restrict__ Pst, int RT, int Nc,
                                                            const uint8_t *__restrict__ tlive,
                                                            const int *__restrict__ qmap, const int *__restrict__ wl,
                                                            int nw, const uint32_t *__restrict__ bits, int rwords,
                                                            double *__restrict__ mass) {
	const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
	if (w >= nw)
		return;
	const int dl = wl[w];
	const size_t pstride = (size_t)(Nc + 1) * TILE;
	const uint32_t *b = bits + (size_t)w * rwords;
	double in = 0., all = 0.;
	for (int rt = 0; rt < RT; ++rt) {
		if (tlive && !tlive[(size_t)rt * (Nc + 1) + dl])
			continue;
		float v[LW];
		ld_row(Pst + rt * pstride + (size_t)dl * TILE + lane * LW, v);
#pragma unroll
		for (int k = 0; k < LW; ++k) {
			const double p = fabs((double)v[k]);
			const int c = qmap[rt * TILE + lane * LW + k];
			all += p;
			if (c >= 0 && (b[c >> 5] >> (c & 31) & 1u))
				in += p;
		}
	}
	in = warp_sum(in);
	all = warp_sum(all);
	if (lane == 0)
		mass[w] = all > 0. ? in / all : 0.;
}

// Nearest coarse orientation of every fine one (voronoi_subset,
// quaternion.c:844-862): distance 1 - (q . q')^2 with the dot product summed
// in component order, first coarse index on ties (strict <). One thread per
// fine orientation; the coarse list is staged through shared memory.
__global__ void __launch_bounds__(256) voronoi_kernel(const double *__restrict__ coarse, int nc,
                                                      const double *__restrict__ fine, int nf,
                                                      int *__restrict__ nearest) {
	__shared__ double cq[256][4];
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	double q[4] = {0., 0., 0., 0.};
	if (i < nf)
		for (int k = 0; k < 4; ++k)
			q[k] = fine[(size_t)i * 5 + k];
	double dmin = 2.;
	int best = -1;
	for (int j0 = 0; j0 < nc; j0 += 256) {
		const int n = min(256, nc - j0);
		__syncthreads();
		if (threadIdx.x < n)
			for (int k = 0; k < 4; ++k)
				cq[threadIdx.x][k] = coarse[(size_t)(j0 + threadIdx.x) * 5 + k];
		__syncthreads();
		for (int j = 0; j < n; ++j) {
			double dot = 0.;
#pragma unroll
			for (int k = 0; k < 4; ++k)
				dot = dadd(dot, dmul(q[k], cq[j][k]));
			const double dist = dsub(1., dmul(dot, dot));
			if (dist < dmin) {
				dmin = dist;
				best = j0 + j;
			}
		}
	}
	if (i < nf)
		nearest[i] = best;
}

// One slice, un-logged (Model.slice_gen, model.c:11-59)
// (slice_gen2d / slice_genrz, model.c:65-150, for 2-D and RZ models: g holds
// the quaternion, or (cos, sin) of the angle, or the five RZ parameters)
// (by value: no upload before the launch)
struct OneOrientation {
	double v[8];
};

template <int GEO>
__global__ void slice_one_kernel(const OneOrientation g, int mode, const double *__restrict__ qvals,
                                 const double *__restrict__ corr, int P, const double *__restrict__ model,
                                 long long S, long long V, double *__restrict__ out) {
	int p = blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= P)
		return;
	double rot[9];
	if constexpr (GEO == MT_3D)
		rot_from_quat(g.v, rot);
	else
		for (int k = 0; k < 5; ++k)
			rot[k] = g.v[k];
	out[p] = geo_sample<GEO>(rot, qvals[3 * (size_t)p], qvals[3 * (size_t)p + 1], qvals[3 * (size_t)p + 2],
	                         (double)(S / 2), S, model + (size_t)mode * V, corr[p]);
}

// One merge in FP64 (Model.slice_merge, model.c:171-244)
// (slice_merge2d / slice_mergerz, model.c:254-340, for 2-D and RZ models)
template <int GEO>
__global__ void merge_one_kernel(const double *__restrict__ g, int mode, const double *__restrict__ view,
                                 const double *__restrict__ qvals, const double *__restrict__ corr,
                                 const uint8_t *__restrict__ mask, int P, long long S, long long V,
                                 double *__restrict__ model2, double *__restrict__ weight) {
	int p = blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= P || mask[p] > 1)
		return;
	const double qx = qvals[3 * (size_t)p], qy = qvals[3 * (size_t)p + 1], qz = qvals[3 * (size_t)p + 2];
	const double center = (double)(S / 2);
	double fw[8];
	long long o[8], base;
	int nc;
	if constexpr (GEO == MT_3D) {
		double rot[9];
		rot_from_quat(g, rot);
		Cell c = locate(rot, qx, qy, qz, center, S);
		if (!c.ok)
			return;
		corner_weights(c, fw);
		corner_offsets(S, o);
		base = c.i000;
		nc = 8;
	} else {
		Cell2 c = GEO == MT_2D ? locate2d(g, qx, qy, center, S) : locate_rz(g, qx, qy, center, S);
		if (!c.ok)
			return;
		corner_weights2(c, fw);
		o[0] = 0; o[1] = 1; o[2] = S; o[3] = S + 1;
		base = c.i00;
		nc = 4;
	}
	const double w = view[p] / corr[p];
	for (int q = 0; q < nc; ++q) {
		atomicAdd(weight + (size_t)mode * V + base + o[q], fw[q]);
		atomicAdd(model2 + (size_t)mode * V + base + o[q], fw[q] * w);
	}
}

// ---------------------------------------------------------------------------
// sparse probabilities and tomograms for the result getters
// ---------------------------------------------------------------------------
// Per frame of the chunk: the number of pairs with P > PROB_MIN (positive
// Pst), i.e. the length of the frame's list after resparsify
// (max_prob.c:321-325, 429-448). One warp per frame.
__global__ void __launch_bounds__(256) count_prob_kernel(const float *__restrict__ Pst, int RT, int Nc,
                                                         int *__restrict__ count) {
	const int dl = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
	if (dl >= Nc)
		return;
	const size_t pstride = (size_t)(Nc + 1) * TILE;
	int c = 0;
	for (int rt = 0; rt < RT; ++rt) {
		float v[LW];
		ld_row(Pst + rt * pstride + (size_t)dl * TILE + lane * LW, v);
#pragma unroll
		for (int e = 0; e < LW; ++e)
			c += v[e] > 0.f;
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1)
		c += __shfl_xor_sync(FULL, c, o);
	if (lane == 0)
		count[dl] = c;
}

// The frame's list in ascending orientation order, as the reference's
// combined and resparsified prob / place_prob (max_prob.c:306-325): P is
// formed again in FP64 from the log-likelihood exactly as the normalisation
// formed it. off [Nc + 1] holds the chunk-local list offsets. One warp per
// frame; lanes own LW consecutive orientations, so a warp-wide exclusive scan
// of the per-lane counts orders each row.
__global__ void __launch_bounds__(256) compact_prob_kernel(
    const double *__restrict__ pval, const float *__restrict__ Pst, int RT, int Nc, int d0,
    const double *__restrict__ beta, const double *__restrict__ max_exp, const double *__restrict__ p_norm,
    const long long *__restrict__ off, int *__restrict__ place, double *__restrict__ prob) {
	const int dl = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
	if (dl >= Nc)
		return;
	long long base = off[dl];
	if (off[dl + 1] == base)
		return;
	const int d = d0 + dl;
	const double m = max_exp[d], inv_s = 1. / p_norm[d], b = beta[d];
	const size_t pstride = (size_t)(Nc + 1) * TILE, tstride = (size_t)Nc * TILE;
	for (int rt = 0; rt < RT; ++rt) {
		float pv[LW];
		ld_row(Pst + rt * pstride + (size_t)dl * TILE + lane * LW, pv);
		int c = 0;
#pragma unroll
		for (int e = 0; e < LW; ++e)
			c += pv[e] > 0.f;
		int incl = c;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const int y = __shfl_up_sync(FULL, incl, o);
			if (lane >= o)
				incl += y;
		}
		const int total = __shfl_sync(FULL, incl, 31);
		if (c > 0) {
			double x[LW];
			ld_row(pval + rt * tstride + (size_t)dl * TILE + lane * LW, x);
			long long pos = base + incl - c;
#pragma unroll
			for (int e = 0; e < LW; ++e)
				if (pv[e] > 0.f) {
					place[pos] = rt * TILE + lane * LW + e;
					prob[pos] = exp(dmul(b, dsub(x[e], m))) * inv_s;
					++pos;
				}
		}
		base += total;
	}
}

// Tomograms of orientations r0 .. r0 + n - 1 divided by psum_r where it is
// positive (update_tomogram_nobg's final step, max_update.c:226-229), as
// out [n][P] FP64; with psum_r null (background path) T already holds them.
__global__ void tomogram_kernel(const float *__restrict__ T, const double *__restrict__ psum_r, int P, int r0,
                                int n, double *__restrict__ out) {
	const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (idx >= (long long)n * P)
		return;
	const int k = (int)(idx / P), p = (int)(idx - (long long)k * P), r = r0 + k;
	const double v = T[((size_t)(r / TILE) * P + p) * TILE + r % TILE];
	const double ps = psum_r != nullptr ? psum_r[r] : 0.;
	out[idx] = ps > 0. ? v / ps : v;
}

}  // namespace dfg
