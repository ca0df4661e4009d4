/*
 * tile.cu -- FP64 registers beyond the caches: more rotations per state
 * round trip than a pass holds.
 *
 * A pass holds what a thread's 32 amplitudes can take, rotations whose flip
 * masks span 5 dimensions: 5.5 qDRIFT draws.  At the HBM limit the FP64
 * pipe is then two thirds idle.  Here a block takes a tile of 2^12
 * amplitudes into shared memory, closed under rotations whose masks span 8
 * dimensions beside the 4 lowest qubits, 9 draws or more, and runs them as
 * sub-passes of 16 amplitudes a thread.  The FP64 update rounds every
 * product and sum of an amplitude by itself, so grouping does not change
 * the bits.
 *
 * The four low qubits are in every tile so that HBM is read and written in
 * runs of 256 bytes: tiles of 10 dimensions and 64-byte runs (two whole
 * passes) copy at 3.5 TB/s at 28 qubits, 8 and 256 bytes at 5.6, single
 * passes at 5.7 (the same copy kernel).
 *
 * Tile-local index: an amplitude's bits at the pivots (leading bits) of the
 * tile space's reduced echelon form, whose lowest rows are the unit vectors
 * of the low qubits.
 */
#include <cuda_runtime.h>

#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define LOG_SUBSYS "engine"
#include "log.h"

#include "p2_sub.cuh"
#include "tile_core.h"

#define P2_TILE_TPB (1 << (P2_TILE_BITS - P2_TILE_SPAN))
#define P2_TILE_TB (P2_TILE_BITS - P2_TILE_SPAN)
#define P2_TILE_SLOTS (1 << P2_TILE_SPAN)
#define P2_TILE_MIN_QB 20
#define P2_TILE_BYTES ((size_t)16 << P2_TILE_BITS)

#define P2_CASE_T(K)                                                           \
	case K:                                                                \
		p2_rot<P2_TILE_SPAN, ((K) >> 1), ((K)&1)>(re, im, q.c, q.s, sm,  \
			0u);                                                   \
		break;

__device__ __forceinline__ void p2_tile_apply(const struct p2_tile_rec &q,
	double (&re)[P2_TILE_SLOTS], double (&im)[P2_TILE_SLOTS], uint32_t sm)
{
	switch (q.key) {
		P2_CASE_T(0) P2_CASE_T(1) P2_CASE_T(2) P2_CASE_T(3)
		P2_CASE_T(4) P2_CASE_T(5) P2_CASE_T(6) P2_CASE_T(7)
		P2_CASE_T(8) P2_CASE_T(9) P2_CASE_T(10) P2_CASE_T(11)
		P2_CASE_T(12) P2_CASE_T(13) P2_CASE_T(14) P2_CASE_T(15)
		P2_CASE_T(16) P2_CASE_T(17) P2_CASE_T(18) P2_CASE_T(19)
		P2_CASE_T(20) P2_CASE_T(21) P2_CASE_T(22) P2_CASE_T(23)
		P2_CASE_T(24) P2_CASE_T(25) P2_CASE_T(26) P2_CASE_T(27)
		P2_CASE_T(28) P2_CASE_T(29) P2_CASE_T(30) P2_CASE_T(31)
	default:
		break;
	}
}
#undef P2_CASE_T

/* Tile number -> its representative: zeros at the tile's pivots. */
__device__ __forceinline__ uint64_t p2_tile_base(uint64_t t,
	const struct p2_tile &tl)
{
#pragma unroll
	for (int k = 0; k < P2_TILE_BITS; ++k) {
		const uint32_t q = tl.piv[k];
		t = ((t >> q) << (q + 1)) | (t & ((UINT64_C(1) << q) - 1));
	}
	return t;
}

/* Start the copy of a tile into shared memory; x: its base with the
 * thread's part of the local index (the low bits), pos that part's place. */
__device__ __forceinline__ void p2_tile_fetch(uint32_t sbase,
	const double2 *__restrict__ st, uint64_t x, uint32_t pos,
	const struct p2_tile &tl)
{
#pragma unroll
	for (int j = 0; j < P2_TILE_SLOTS; ++j) {
		uint64_t off = 0;
#pragma unroll
		for (int k = 0; k < P2_TILE_SPAN; ++k)
			if (j >> k & 1)
				off ^= tl.row[P2_TILE_TB + k];
		p2_cp16(sbase + 16 * (pos ^ p2_sub_swz((uint32_t)j
						  << P2_TILE_TB)),
			st + (x ^ off));
	}
	p2_cp_commit();
}

/*
 * Persistent: the next tile is copied in while the last sub-pass of the
 * current one, by then wholly in registers, is applied and stored.  A
 * record's sign bits take the tile's part of the parity once a tile.
 */
__global__ void __launch_bounds__(P2_TILE_TPB, 2) k_tile(
	double2 *__restrict__ st, uint64_t ntile,
	const __grid_constant__ struct p2_tile tl,
	const struct p2_tile_sub *__restrict__ subs,
	const struct p2_tile_rec *__restrict__ recs)
{
	extern __shared__ __align__(128) unsigned char p2_tile_dyn[];
	__shared__ struct p2_tile_rec srec[P2_TILE_ROTS];
	__shared__ struct p2_tile_sub hdr[P2_TILE_ROTS];
	/* two: threads still in a tile's last sub-pass read theirs */
	__shared__ uint16_t ssm_all[2][P2_TILE_ROTS];
	const uint32_t tid = threadIdx.x;
	const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(p2_tile_dyn);
	for (uint32_t r = tid; r < tl.nrot; r += P2_TILE_TPB)
		srec[r] = recs[tl.rot_off + r];
	for (uint32_t i = tid; i < tl.nsub; i += P2_TILE_TPB)
		hdr[i] = subs[tl.sub_off + i];
	uint64_t tin = 0, tout = 0; /* the thread's offsets: copy in, store */
#pragma unroll
	for (int k = 0; k < P2_TILE_TB; ++k) {
		const uint64_t m = 0u - (uint64_t)(tid >> k & 1);
		tin ^= m & tl.row[k];
		tout ^= m & tl.tout[k];
	}
	const uint32_t pin = p2_sub_swz(tid);
	p2_grid_wait();
	uint64_t t = blockIdx.x;
	uint64_t x0 = p2_tile_base(t, tl);
	if (t < ntile)
		p2_tile_fetch(sbase, st, x0 ^ tin, pin, tl);
	__syncthreads();
	for (uint32_t odd = 0; t < ntile; t += gridDim.x, odd ^= 1u) {
		uint16_t *const ssm = ssm_all[odd];
		for (uint32_t r = tid; r < tl.nrot; r += P2_TILE_TPB)
			ssm[r] = srec[r].sm ^ (uint16_t)(0u -
				(uint32_t)(__popcll(x0 & srec[r].z) & 1));
		p2_cp_wait<0>();
		__syncthreads();
		const uint64_t xn = p2_tile_base(t + gridDim.x, tl);
		for (uint32_t i = 0; i < tl.nsub; ++i) {
			const struct p2_tile_sub &h = hdr[i];
			uint32_t y = tid;
#pragma unroll
			for (int k = 0; k < P2_TILE_SPAN; ++k) {
				const uint32_t q = h.piv[k];
				y = ((y >> q) << (q + 1)) | (y & ((1u << q) - 1u));
			}
			const uint32_t a0 = 16 * p2_sub_swz(y);
			uint32_t sp[P2_TILE_SPAN];
#pragma unroll
			for (int k = 0; k < P2_TILE_SPAN; ++k)
				sp[k] = 16u * h.pslot[k];
			double re[P2_TILE_SLOTS], im[P2_TILE_SLOTS];
#pragma unroll
			for (int u = 0; u < P2_TILE_SLOTS; ++u) {
				uint32_t a = a0;
#pragma unroll
				for (int k = 0; k < P2_TILE_SPAN; ++k)
					if (u >> k & 1)
						a ^= sp[k];
				p2_res_ld<false>(sbase + a, re[u], im[u]);
			}
			const bool last = i + 1 == tl.nsub;
			if (last) {
				__syncthreads();
				if (t + gridDim.x < ntile)
					p2_tile_fetch(sbase, st, xn ^ tin, pin, tl);
			}
			const uint32_t r1 = h.rot0 + h.nrot;
			for (uint32_t r = h.rot0; r < r1; ++r) {
				const struct p2_tile_rec q = srec[r];
				p2_tile_apply(q, re, im, (uint32_t)ssm[r] ^
					(0u - p2_parity(y & (uint32_t)q.zl)));
			}
			if (last) {
				const uint64_t xs = p2_opaque(x0 ^ tout);
#pragma unroll
				for (int u = 0; u < P2_TILE_SLOTS; ++u) {
					uint64_t off = 0;
#pragma unroll
					for (int k = 0; k < P2_TILE_SPAN; ++k)
						if (u >> k & 1)
							off ^= tl.sout[k];
					st[xs ^ off] = make_double2(re[u], im[u]);
				}
			} else {
				const uint32_t as = p2_opaque(a0);
#pragma unroll
				for (int u = 0; u < P2_TILE_SLOTS; ++u) {
					uint32_t a = as;
#pragma unroll
					for (int k = 0; k < P2_TILE_SPAN; ++k)
						if (u >> k & 1)
							a ^= sp[k];
					p2_res_st<false>(sbase + a, re[u], im[u]);
				}
				__syncthreads();
			}
		}
		x0 = xn;
	}
}

/* ---- host ----------------------------------------------------------------- */

/*
 * Flushes of at most 10 rotations a planned pass, which the pass kernels run
 * at the memory's speed, from 20 qubits on (below: split.cu).  1e12
 * rotations x amplitudes a second at 20 / 24 / 28 / 30 qubits, pass kernels
 * in brackets: 5.5 draws a pass 0.88 (0.80) / 1.23 (1.04) / 1.31 (1.07) /
 * 1.30 (1.04), dense random strings 0.83 (0.74) / 1.16 (0.97) / 1.23 (0.98)
 * / 1.19 (0.96).  Beyond, both are bound by the FP64 operations and the
 * order varies: 14-18 strings a pass 1.49 (1.28) / 1.79 (1.74) / 1.91
 * (1.96) / 1.89 (1.97), 250 a pass 1.88 (1.90) / 2.22 (2.16) / 2.27 (2.17)
 * / 2.28 (2.17).  Runs of 128 bytes (9 dimensions beside 3 low qubits, 9.9
 * draws a trip) gave 0.86 / 1.15 / 1.16 / 1.14.
 *
 * A short flush whose runs are as many as its passes gains nothing by them
 * (us, pass kernels / tiles: 10 random strings, two passes, at 22, 24, 28
 * qubits 53 / 56, 183 / 209, 2849 / 3337; 5 strings 28 / 34, 95 / 102, 1367
 * / 1409), except one of few rotations with one mask, which a pass reads in
 * short runs (1 and 4 of them at 22 qubits 29 / 22, 29 / 26, at 24 97 / 95,
 * 98 / 98, at 28 1428 / 1426, 1439 / 1457), and one pass again at 20 qubits,
 * where the launch bounds it (16 / 10).  Long ones always gain.
 */
static bool short_gain(const struct phase2_pass *passes, size_t npass,
	const struct phase2_rot_rec *recs, size_t nrec)
{
	if (npass > 4 || p2_tile_count(passes, npass, recs) < npass)
		return true;
	if (npass > 1 || nrec > 6)
		return false;
	uint32_t mask = 0;
	for (size_t i = 0; i < nrec; i++) {
		if (mask && recs[i].U && recs[i].U != mask)
			return false;
		mask |= recs[i].U;
	}
	return true;
}

bool p2_tile_ok(const struct p2_dev *d, int form,
	const struct phase2_pass *passes, size_t npass,
	const struct phase2_rot_rec *recs, size_t nrec)
{
	return form == PHASE2_FORM_EXACT && d->tiles &&
		d->nqb >= P2_TILE_MIN_QB && nrec <= 10 * npass &&
		((npass == 1 && d->nqb == P2_TILE_MIN_QB) ||
			short_gain(passes, npass, recs, nrec));
}

int p2_tile_run(struct p2_dev *d, const struct p2_graph *g)
{
	static uint64_t done;
	unsigned per_sm;
	if (!p2_done(&done, d->context, &per_sm)) {
		int n = 0;
		CUDA_OK(cudaFuncSetAttribute(k_tile,
				cudaFuncAttributeMaxDynamicSharedMemorySize,
				(int)P2_TILE_BYTES),
			"tile kernel shared memory");
		CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_tile,
				P2_TILE_TPB, P2_TILE_BYTES),
			"tile kernel occupancy");
		per_sm = n > 0 ? (unsigned)n : 1;
		p2_set_done(&done, d->context, per_sm);
	}
	const uint64_t ntile = d->namp >> P2_TILE_BITS;
	uint64_t grid = (uint64_t)d->sm_count * per_sm;
	if (grid > ntile)
		grid = ntile;
	const struct p2_tile_rec *r = (const struct p2_tile_rec *)g->d_recs;
	const struct p2_tile_sub *s = (const struct p2_tile_sub *)(r + g->nrec);
	for (uint32_t i = 0; i < g->ntile; i++)
		CUDA_OK(p2_launch(k_tile, (unsigned)grid, P2_TILE_TPB,
				P2_TILE_BYTES, d->stream, (double2 *)d->state,
				ntile, g->tiles[i], s, r),
			"tile launch");
	return 0;
}
