// Hot pixels of the E-step and M-step as exact integer products on the
// 5th-generation tensor cores (sm_100a tcgen05 kind::i8 + TMA). Included by
// emc_api.cu only.
//
// The sparse gathers read one 512-byte row per (tile, frame, photon): their
// time follows the photons and is bound by the L2 path (20 TB/s of rows). A
// pixel that many frames share is cheaper as a column of a matrix product, whose
// time follows pixels x frames. Both phases are that product,
//     E-step  S[d][r] = sum_k count[d][k] logW[r][k]     (k: hot pixels)
//     M-step  T[p][r] = sum_d count[d][p] P[r][d]        (d: the chunk's frames)
// and it is formed without rounding, as the Ozaki scheme does on integer units
// (Ootomo, Ozaki and Yokota, "DGEMM on integer matrix multiplication unit"): counts are unsigned bytes, the FP32
// operand becomes a 32-bit fixed-point number cut into four bytes (signed for
// log-slices, unsigned for probabilities), each byte's product accumulates in an
// INT32 TMEM accumulator (exact below 2^24 counts per sum, 2^23 with unsigned
// digits), and the epilogue puts the four sums together in FP64. The
// FP32 log-slices are multiples of 2^-26 from |x| = 1/8 on (below it they are
// off by at most 2^-27), so the E-step's sum is the exact sum of the values that
// the gathers add; the probabilities are taken relative to their orientation's
// largest in the chunk (4.2e9 steps), 1.2e-10 of it, far below the FP32 rounding of
// the tomogram they end in. The remaining (cold) photons are gathered as before.
// Errors against 64 bits over those of the gathers alone (seven shapes, 16 seeds each):
// log-likelihoods 0.62 to 0.81, models 0.83 to 1.03, within their seeds' spread of
// 0.6 to 1.5; with |log W| small everywhere (one photon per pixel) 0.78 and 0.97.
//
// One CTA per SM walks tiles of 256 rows (frames or pixels) x 64 orientations:
//   warp 0      TMA producer: per 128-deep block the 256 x 128 count tile and
//               the 256 x 128 digit tile (4 digits x 64 orientations) into one of
//               three 64-KB stages (128-byte swizzle), running ahead into the
//               next tile while this one is in its epilogue;
//   warp 1      one lane issues tcgen05.mma (M 128, N 256, K 32), two row
//               blocks x 256 columns: all 512 TMEM columns;
//   warps 2-9   epilogue: digit sums -> FP64 -> log-likelihood partials
//               or tomogram rows.
// The 256 x 64 shape reads 512 operand bytes per 65536 multiply-adds; 128 x 128
// would read 640, and a shape that leaves room for a second accumulator 768:
// the L2 path, not the tensor pipe, would bound those.
// Measured: 3.75e15 operations/s on 50176 x 20000 x 8320 (18.0 ms; the tensor
// pipe's nominal dense INT8 rate is 4.5e15). At the production geometry (50100
// orientations, 60000 frames of 313 photon words, 72 % of them on 8320 hot pixels)
// the E-step went from 220.6 to 146.1 ms and the M-step from 206.0 to 142.8 ms;
// with 95 x 95 pixels (17220 x 40000) from 22.2 to 9.9 and 22.7 to 5.4 ms.
// Every wait gives up after wait_cycles clock cycles, sets the error flag and
// lets the CTA free its TMEM and exit, as in the dense form.
#pragma once

#include <cuda.h>

#include "emc_common.cuh"
#include "tcgen05.cuh"

namespace dfg {

constexpr int HM = 256;      // rows (frames or pixels) per tile
constexpr int HO = 64;       // orientations per tile (x 4 digits = UMMA N 256)
constexpr int HK = 128;      // reduction depth per stage: one 128-byte swizzle row
constexpr int HSTAGES = 3;
constexpr int HA_BYTES = HM * HK;
constexpr int HB_BYTES = 4 * HO * HK;
constexpr int HSTAGE_BYTES = HA_BYTES + HB_BYTES;  // 64 KB
constexpr int HOUT_BYTES = 32 * 128;                // one warp's 32 rows x 16 doubles on their way out
constexpr int HSMEM_BYTES = 1024 + HSTAGES * HSTAGE_BYTES + 8 * HOUT_BYTES + 128;
constexpr int HTHREADS = 320;
constexpr int HGROUP = 12;   // orientation tiles per rasterisation group: 12 x 12 resident tiles share operands in L2
constexpr float HE_SCALE = 67108864.f;  // log-slices in steps of 2^-26
constexpr float HE_LIMIT = 31.f;        // largest |log W| that the four digits hold (W from 3.4e-14)
constexpr double HP_STEPS = 4.2e9;      // steps of an orientation's largest probability (< 2^32)

// Instruction descriptor of kind::i8: S32 accumulator (bits 4-5 = 2), A
// unsigned (bits 7-9 = 0), B unsigned (bits 10-12 = 0) or signed bytes (1), both
// K-major, N >> 3 at bit 17, M >> 4 at bit 24.
constexpr uint32_t HIDESC = (2u << 4) | ((uint32_t)(4 * HO >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t HIDESC_SIGNED = HIDESC | (1u << 10);

template <uint32_t IDESC>
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
	asm volatile(
	    "{\n\t.reg .pred p;\n\t"
	    "setp.ne.b32 p, %4, 0;\n\t"
	    "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
	    "l"(adesc), "l"(bdesc), "r"(IDESC), "r"(accumulate)
	    : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
	asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// 8 TMEM columns of this thread's lane, without waiting for them.
__device__ __forceinline__ void tmem_ld8_issue(uint32_t taddr, uint32_t (&r)[8]) {
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
	             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
	             : "r"(taddr));
}
// Orders the uses of the loaded columns after the wait for them.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&a)[8], uint32_t (&b)[8], uint32_t (&c)[8],
                                             uint32_t (&d)[8]) {
	asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
	for (int k = 0; k < 8; ++k)
		asm volatile("" : "+r"(a[k]), "+r"(b[k]), "+r"(c[k]), "+r"(d[k]));
}

// An int32 in FP64 through the bits of 2^52 + 2^31 + x, without a conversion
// instruction (those run at a sixteenth of the FP64 rate).
__device__ __forceinline__ double i32_to_f64(uint32_t x) {
	return __dsub_rn(__hiloint2double(0x43300000, (int)(x ^ 0x80000000u)), 4503601774854144.0);
}

// d3 2^24 + d2 2^16 + d1 2^8 + d0, exact (below 2^53).
__device__ __forceinline__ double join_digits(uint32_t d0, uint32_t d1, uint32_t d2, uint32_t d3) {
	double v = fma(i32_to_f64(d3), 256., i32_to_f64(d2));
	v = fma(v, 256., i32_to_f64(d1));
	return fma(v, 256., i32_to_f64(d0));
}

// 3-D tiled TMA store from this CTA's shared memory, and the waits for the
// stores of this thread: until they have read it, until they are done.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, const void *src, int x, int y, int z) {
	asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
	                 (uint64_t)map),
	             "r"(smem_addr(src)), "r"(x), "r"(y), "r"(z)
	             : "memory");
	asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait_read() {
	asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Where a tile's sums go. MSTEP false: pval[tile][frame][128] (FP64 photon sums
// of the hot pixels; rows = frames), by TMA through map_out, whose rows past the
// chunk's frames are clipped; true: T[tile][pix[row]][128] += sum x
// rmax[r] / HP_STEPS (rows = hot pixels; overwritten for the first chunk,
// whose tomograms are zero).
struct HotOut {
	float *T;
	const int *pix;     // hot pixel of each row
	const float *rmax;  // [R_pad] largest probability of each orientation in the chunk
	int P, first;
};

template <bool MSTEP>
__global__ void __launch_bounds__(HTHREADS, 1) hot_product_kernel(
    const __grid_constant__ CUtensorMap map_cnt, const __grid_constant__ CUtensorMap map_dig,
    const __grid_constant__ CUtensorMap map_out, int num_kb, int OT, int FT, int nrows, HotOut out,
    const int *__restrict__ special, int *__restrict__ err, long long wait_cycles, int withhold_kb) {
	extern __shared__ uint8_t hsm_raw[];
	uint8_t *sm = (uint8_t *)(((uintptr_t)hsm_raw + 1023) & ~(uintptr_t)1023);
	uint8_t *outs = sm + HSTAGES * HSTAGE_BYTES;
	uint64_t *bars = (uint64_t *)(outs + 8 * HOUT_BYTES);
	uint64_t *full = bars, *empty = bars + HSTAGES, *tfull = bars + 2 * HSTAGES, *tempty = tfull + 1;
	uint32_t *tmem_slot = (uint32_t *)(tempty + 1);
	volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const long long tiles = (long long)OT * FT;
	const long long per_group = (long long)HGROUP * FT;

	if (threadIdx.x == 0) {
		for (int s = 0; s < HSTAGES; ++s) {
			mbar_init(&full[s], 1);
			mbar_init(&empty[s], 1);
		}
		mbar_init(tfull, 1);
		mbar_init(tempty, 8);
		*abort_flag = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == 1) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
		                 smem_addr(tmem_slot)),
		             "r"(512)
		             : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = *tmem_slot;

	// tile -> (orientation tile, row tile), HGROUP orientation tiles at a time
	auto locate_tile = [&](long long t, int &ot, int &ft) {
		const int grp = (int)(t / per_group);
		const int rem = (int)(t - grp * per_group);
		const int rows = min(HGROUP, OT - grp * HGROUP);
		ot = grp * HGROUP + rem % rows;
		ft = rem / rows;
	};

	// E-step tiles that gather all of their photons (hot_digits_kernel)
	auto skipped = [&](int ot) { return !MSTEP && __ldg(special + (ot >> 1)) != 0; };

	if (warp == 0) {
		if (lane == 0) {
			long long it = 0, issued = 0;  // stage counter over all tiles; stages whose copies were issued
			bool ok = true;
			for (long long t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
				int ot, ft;
				locate_tile(t, ot, ft);
				if (skipped(ot))
					continue;
				for (int kb = 0; kb < num_kb; ++kb, ++it) {
					const int s = (int)(it % HSTAGES);
					const uint32_t ph = (uint32_t)(it / HSTAGES) & 1u;
					if (*abort_flag || !mbar_wait(&empty[s], ph ^ 1u, wait_cycles)) {
						*abort_flag = 1;
						atomicExch(err, 1);
						ok = false;
						break;
					}
					if (kb == withhold_kb) {  // test hook: this stage's copies are never issued
						ok = false;
						break;
					}
					uint8_t *st = sm + s * HSTAGE_BYTES;
					mbar_expect_tx(&full[s], HSTAGE_BYTES);
					tma_load_2d(st, &map_cnt, &full[s], kb * HK, ft * HM);
					tma_load_2d(st + HA_BYTES, &map_dig, &full[s], kb * HK, ot * 4 * HO);
					issued = it + 1;
				}
			}
			// the copies in flight land before the CTA exits (after a give-up
			// some of them may not have been consumed)
			for (long long k = issued > HSTAGES ? issued - HSTAGES : 0; k < issued; ++k)
				mbar_wait(&full[k % HSTAGES], (uint32_t)(k / HSTAGES) & 1u, wait_cycles);
		}
		__syncwarp();
	} else if (warp == 1) {
		if (lane == 0) {
			long long it = 0;
			uint32_t n = 0;  // tiles done by this CTA
			bool ok = true;
			for (long long t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
				int ot, ft;
				locate_tile(t, ot, ft);
				if (skipped(ot))
					continue;
				// the epilogue has read the previous tile's sums
				if (*abort_flag || !mbar_wait(tempty, (n & 1u) ^ 1u, wait_cycles)) {
					*abort_flag = 1;
					atomicExch(err, 1);
					break;
				}
				tc_fence_after();
				for (int kb = 0; kb < num_kb; ++kb, ++it) {
					const int s = (int)(it % HSTAGES);
					const uint32_t ph = (uint32_t)(it / HSTAGES) & 1u;
					if (*abort_flag || !mbar_wait(&full[s], ph, wait_cycles)) {
						*abort_flag = 1;
						atomicExch(err, 1);
						ok = false;
						break;
					}
					tc_fence_after();
					const uint32_t a = smem_addr(sm + s * HSTAGE_BYTES), b = a + HA_BYTES;
#pragma unroll
					for (int k = 0; k < HK / 32; ++k) {
						const uint64_t db = sw128_desc(b + 32 * k);
						const uint32_t acc = (kb | k) != 0;
						constexpr uint32_t idesc = MSTEP ? HIDESC : HIDESC_SIGNED;
						umma_i8<idesc>(tmem, sw128_desc(a + 32 * k), db, acc);
						umma_i8<idesc>(tmem + 4 * HO, sw128_desc(a + 128 * HK + 32 * k), db, acc);
					}
					umma_commit(&empty[s]);
				}
				if (ok)
					umma_commit(tfull);
				++n;
			}
		}
		__syncwarp();
	} else {
		// warp w: row block (w - 2) / 4, TMEM lanes 32 (w % 4) .. + 31
		const int m = (warp - 2) >> 2, q = warp & 3, i = m * 128 + q * 32 + lane;
		const uint32_t base = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(m * 4 * HO);
		uint32_t n = 0;
		for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
			int ot, ft;
			locate_tile(t, ot, ft);
			if (skipped(ot))
				continue;
			// the flag may change between the lanes' reads: decide for the warp
			bool ok = mbar_wait(tfull, n & 1u, wait_cycles) && !*abort_flag;
			++n;
			ok = __all_sync(FULL, ok);
			if (!ok) {
				if (lane == 0) {
					*abort_flag = 1;
					atomicExch(err, 1);
				}
				break;
			}
			tc_fence_after();
			const int rt = ot >> 1, j0 = (ot & 1) * HO, row = ft * HM + i;
			const bool valid = row < nrows;
			float *const tp =
			    MSTEP ? out.T + ((size_t)rt * out.P + (valid ? out.pix[row] : 0)) * TILE + j0 : nullptr;
			// all sums into registers first, so that the next tile's products
			// run while this one's results are stored (the stores alone take about
			// 10000 cycles a tile, as long as the products over 1250 pixels)
			double v[HO];
#pragma unroll
			for (int c = 0; c < HO / 8; ++c) {
				uint32_t d0[8], d1[8], d2[8], d3[8];
				tmem_ld8_issue(base + c * 8, d0);
				tmem_ld8_issue(base + HO + c * 8, d1);
				tmem_ld8_issue(base + 2 * HO + c * 8, d2);
				tmem_ld8_issue(base + 3 * HO + c * 8, d3);
				tmem_ld_wait(d0, d1, d2, d3);
#pragma unroll
				for (int k = 0; k < 8; ++k)
					v[c * 8 + k] = join_digits(d0[k], d1[k], d2[k], d3[k]);
			}
			tc_fence_before();
			__syncwarp();
			if (lane == 0)
				mbar_arrive(tempty);
			if constexpr (MSTEP) {
				if (valid) {
					const float *rm = out.rmax + (size_t)rt * TILE + j0;
#pragma unroll
					for (int k = 0; k < HO; k += 4) {
						float4 *dst = reinterpret_cast<float4 *>(tp + k);
						const float4 r4 = __ldg(reinterpret_cast<const float4 *>(rm + k));
						const float rr[4] = {r4.x, r4.y, r4.z, r4.w};
						float4 o4 = make_float4(0.f, 0.f, 0.f, 0.f);
						if (!out.first)
							o4 = *dst;
						float o[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
						for (int e = 0; e < 4; ++e)
							o[e] = (float)((double)o[e] + v[k + e] * ((double)rr[e] * (1. / HP_STEPS)));
						*dst = make_float4(o[0], o[1], o[2], o[3]);
					}
				}
			} else {
				// rows are a KB apart: stored from the lanes, each instruction touched
				// 32 lines. 16 doubles of every row go to shared memory (128-byte
				// swizzle, as the tensor map has it) and leave as one TMA store.
				uint8_t *const mine = outs + (warp - 2) * HOUT_BYTES;
				const int row0 = ft * HM + m * 128 + q * 32;
				if (row0 < nrows) {
#pragma unroll
					for (int c = 0; c < HO / 16; ++c) {
						if (lane == 0)
							tma_store_wait_read();
						__syncwarp();
#pragma unroll
						for (int k = 0; k < 8; ++k)
							*reinterpret_cast<double2 *>(mine + lane * 128 + ((k ^ (lane & 7)) << 4)) =
							    make_double2(v[c * 16 + 2 * k] * (1. / HE_SCALE), v[c * 16 + 2 * k + 1] * (1. / HE_SCALE));
						asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
						__syncwarp();
						if (lane == 0)
							tma_store_3d(&map_out, mine, j0 + c * 16, row0, rt);
					}
				}
			}
			__syncwarp();
		}
		if (!MSTEP && lane == 0)
			tma_store_wait();
		__syncwarp();
	}
	tc_fence_before();
	__syncthreads();
	if (warp == 1) {
		tc_fence_after();
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
	}
}

// Fixed-point digits, K-major: dig[(tile-half * 4 + digit) * 64 + j][k] of
// 64-orientation halves of the 128-orientation tiles, k = hot pixels
// (MSTEP false; from logW [tile][P + 1][128]) or the chunk's frames (true; from
// Pst [tile][Nc + 1][128], max(P, 0) relative to the orientation's largest).
// Balanced digits: x = sum_g d_g 256^g with -128 <= d_g <= 127 (false), its bytes (true:
// twice the steps of signed ones; the model's error against 64 bits is 0.98 to 1.02
// of the gathers' over seven shapes, 0.98 to 1.04 with signed ones). K past the last
// pixel or frame is zero. A log-slice that the digits cannot hold (log 0, the
// value outside the model, NaN) sets special[tile]: the E-step then gathers
// that tile's photons all, and its products are left out (an empty one of several
// modes does that to every tile). live (true; may be null): [tile][Nc + 1] flags of
// the rows that hold probabilities (tile skipping), the others count as zero.
// Block = 128 reduction rows x 64 orientations,
// transposed through shared memory; the rotation by 4 (k / 16) keeps the
// column reads free of bank conflicts. Memory-bound: 4 bytes read, 4 written. The
// grid is flat, blocks of one 64-orientation half in turn (digit_blocks): from
// 32768 tiles on there are more halves than a grid's second extent takes.
template <bool MSTEP>
__global__ void __launch_bounds__(256) hot_digits_kernel(const float *__restrict__ src, size_t tile_stride,
                                                         const int *__restrict__ pix, int nk, int k_pitch,
                                                         const float *__restrict__ rmax, int8_t *__restrict__ dig,
                                                         int *__restrict__ special,
                                                         const uint8_t *__restrict__ live) {
	__shared__ int s[HK][HO + 1];
	__shared__ double s_scale[HO];
	const int kblocks = k_pitch / HK, ot = blockIdx.x / kblocks, kb = blockIdx.x - ot * kblocks, t = threadIdx.x;
	const int rt = ot >> 1, j0 = (ot & 1) * HO;
	if (MSTEP && t < HO) {
		const float m = rmax[(size_t)rt * TILE + j0 + t];
		s_scale[t] = m > 0.f ? HP_STEPS / (double)m : 0.;
	}
	if constexpr (MSTEP)
		__syncthreads();
	int bad = 0;
	for (int idx = t; idx < HK * (HO / 4); idx += 256) {
		const int k = idx / (HO / 4), o = (idx % (HO / 4)) * 4, kg = kb * HK + k;
		int v[4] = {0, 0, 0, 0};
		if (kg < nk && (live == nullptr || live[(size_t)rt * (nk + 1) + kg])) {
			const int row = MSTEP ? kg : pix[kg];
			const float4 x4 = __ldg(reinterpret_cast<const float4 *>(src + (size_t)rt * tile_stride +
			                                                          (size_t)row * TILE + j0 + o));
			const float x[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
			for (int e = 0; e < 4; ++e) {
				if constexpr (MSTEP) {
					v[e] = (int)__double2uint_rn((double)fmaxf(x[e], 0.f) * s_scale[o + e]);
				} else {
					const bool fits = fabsf(x[e]) < HE_LIMIT;  // false for NaN
					v[e] = fits ? __float2int_rn(x[e] * HE_SCALE) : 0;
					bad |= !fits;
				}
			}
		}
		int *d = &s[k][(o + 4 * (k >> 4)) & (HO - 1)];
#pragma unroll
		for (int e = 0; e < 4; ++e)
			d[e] = v[e];
	}
	bad = __syncthreads_or(bad);
	if (!MSTEP && bad && t == 0)
		special[rt] = 1;
	for (int idx = t; idx < HO * (HK / 16); idx += 256) {
		const int o = idx >> 3, a = idx & 7;  // 16 reduction rows a * 16 .. of orientation o
		uint32_t w[4][4];
#pragma unroll
		for (int g = 0; g < 4; ++g)
#pragma unroll
			for (int h = 0; h < 4; ++h)
				w[g][h] = 0u;
#pragma unroll
		for (int e = 0; e < 16; ++e) {
			int x = s[a * 16 + e][(o + 4 * a) & (HO - 1)];
#pragma unroll
			for (int g = 0; g < 4; ++g) {
				const int d = (int)(int8_t)(x & 0xff);
				w[g][e >> 2] |= (uint32_t)(uint8_t)d << (8 * (e & 3));
				x = MSTEP ? (int)((uint32_t)x >> 8) : (x - d) >> 8;
			}
		}
#pragma unroll
		for (int g = 0; g < 4; ++g)
			*reinterpret_cast<uint4 *>(dig + ((size_t)(ot * 4 + g) * HO + o) * k_pitch + (size_t)kb * HK + a * 16) =
			    make_uint4(w[g][0], w[g][1], w[g][2], w[g][3]);
	}
}

// A chunk's counts on the hot pixels as bytes, both ways round: by_frame
// [frames][h_pitch] and by_pixel [H][k_pitch] (zeroed before). One warp per hot pixel
// walks the chunk's list of it (counts <= 255, so one word per frame; padding
// words name frame Nc).
__global__ void __launch_bounds__(256) hot_counts_kernel(const uint32_t *__restrict__ cs,
                                                         const long long *__restrict__ cs_off,
                                                         const long long *__restrict__ cs_mid,
                                                         const int *__restrict__ pix, int H, int h_pitch, int Nc,
                                                         int k_pitch, uint8_t *__restrict__ by_frame,
                                                         uint8_t *__restrict__ by_pixel) {
	const int h = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
	if (h >= H)
		return;
	const int p = pix[h];
	const long long mid = cs_mid[p], end = cs_off[p + 1];
	for (long long j = cs_off[p] + lane; j < end; j += 32) {
		const uint32_t w = cs[j], f = j < mid ? w : (w & IDX_MASK);
		if (f >= (uint32_t)Nc)
			continue;
		const uint8_t c = (uint8_t)(j < mid ? 1u : (w >> IDX_BITS));
		by_frame[(size_t)f * h_pitch + h] = c;
		by_pixel[(size_t)h * k_pitch + f] = c;
	}
}

// The photon lists without the hot pixels, in two passes: the words of each
// list's two segments (counts), then the lists, each segment padded to 8 words
// with `pad`. A count of up to COLD_REPEAT becomes that many count-1 words: the
// few such photons of a cold pixel would take a segment of their own, padded to 8
// rows. (Each of them rounds by itself, where a counted word's product is exact; the
// errors at the head of this file include that.) One warp per list. BY_LIST false: lists of pixels per frame (E-step), hot
// words dropped; true: lists of frames per pixel (M-step), hot lists dropped.
// Words naming `limit` or above are padding.
constexpr uint32_t COLD_REPEAT = 4;

// (count-1 words, counted words) that word w of a list contributes
template <bool BY_LIST>
__device__ __forceinline__ int2 cold_words(uint32_t w, bool multi, uint32_t limit, const uint8_t *__restrict__ is_hot) {
	const uint32_t idx = multi ? (w & IDX_MASK) : w, c = multi ? (w >> IDX_BITS) : 1u;
	if (idx >= limit || (!BY_LIST && is_hot[idx]))
		return make_int2(0, 0);
	return c <= COLD_REPEAT ? make_int2((int)c, 0) : make_int2(0, 1);
}

template <bool BY_LIST>
__global__ void __launch_bounds__(256) cold_count_kernel(const uint32_t *__restrict__ words,
                                                         const long long *__restrict__ off,
                                                         const long long *__restrict__ mid, int n, uint32_t limit,
                                                         const uint8_t *__restrict__ is_hot, int2 *__restrict__ out) {
	const int d = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
	if (d >= n)
		return;
	int a = 0, b = 0;
	if (!BY_LIST || !is_hot[d])
		for (long long j = off[d] + lane; j < off[d + 1]; j += 32) {
			const int2 k = cold_words<BY_LIST>(words[j], j >= mid[d], limit, is_hot);
			a += k.x;
			b += k.y;
		}
	a = __reduce_add_sync(FULL, a);
	b = __reduce_add_sync(FULL, b);
	if (lane == 0)
		out[d] = make_int2(a, b);
}

__device__ __forceinline__ int warp_prefix(int x, int lane) {  // inclusive
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const int y = __shfl_up_sync(FULL, x, o);
		if (lane >= o)
			x += y;
	}
	return x;
}

template <bool BY_LIST>
__global__ void __launch_bounds__(256) cold_write_kernel(const uint32_t *__restrict__ words,
                                                         const long long *__restrict__ off,
                                                         const long long *__restrict__ mid, int n, uint32_t limit,
                                                         uint32_t pad, const uint8_t *__restrict__ is_hot,
                                                         const long long *__restrict__ coff,
                                                         const long long *__restrict__ cmid,
                                                         uint32_t *__restrict__ out) {
	const int d = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
	if (d >= n || coff[d + 1] == coff[d])
		return;
	long long at1 = coff[d], atm = cmid[d];
	for (long long j0 = off[d]; j0 < off[d + 1]; j0 += 32) {
		const long long j = j0 + lane;
		const bool multi = j >= mid[d];
		const uint32_t w = j < off[d + 1] ? words[j] : 0u;
		const int2 k = j < off[d + 1] ? cold_words<BY_LIST>(w, multi, limit, is_hot) : make_int2(0, 0);
		const int p1 = warp_prefix(k.x, lane), pm = warp_prefix(k.y, lane);
		for (int c = 0; c < k.x; ++c)
			out[at1 + p1 - k.x + c] = multi ? (w & IDX_MASK) : w;
		if (k.y)
			out[atm + pm - 1] = w;
		at1 += __shfl_sync(FULL, p1, 31);
		atm += __shfl_sync(FULL, pm, 31);
	}
	for (long long j = at1 + lane; j < cmid[d]; j += 32)
		out[j] = pad;
	for (long long j = atm + lane; j < coff[d + 1]; j += 32)
		out[j] = pad;
}

}  // namespace dfg
