/*
 * split.cu -- passes of registers of middle width, a coset shared by four
 * threads.
 *
 * The pass kernels give a thread a whole coset of 32 amplitudes.  A register
 * of 15 to 19 qubits then has at most one warp a scheduler, whose FP64
 * operations wait for one another through every rotation of the pass: 430-
 * 1000 ns a rotation whatever the width.  Here a block
 * of 128 threads holds a tile of 2^10 amplitudes (32 cosets of a span-5
 * pass) in shared memory and applies the pass as sub-passes of 8
 * amplitudes a thread (sub_core.h): four times the warps, and 16 cases of
 * 8 unrolled slots in place of 64 of 32.  Amplitudes stay doubles inside
 * the pass, so the bits are the pass kernels'.
 */
#include <cuda_runtime.h>

#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define LOG_SUBSYS "engine"
#include "log.h"

#include "p2_sub.cuh"

#define P2_SPLIT_MIN_QB 15 /* below: resident.cu */
#define P2_SPLIT_MAX_QB 19
#define P2_SPLIT_TPB (1 << (P2_SPLIT_BITS - P2_SUB_SPAN))
#define P2_SPLIT_SMEM                                                          \
	((16 << P2_SPLIT_BITS) + P2_MAX_ROTS_PER_PASS *                        \
		(sizeof(struct p2_sub_rec) + sizeof(struct p2_sub)))

/*
 * One pass of span M (3..5).  Tile-local index: representative number in
 * the low 10 - M bits, slot above.  Everything the pass does not read from
 * the state (records, headers) is staged before the wait for the previous
 * kernel, which may still be running when this one starts
 * (programmatic dependent launch).
 */
template <typename ST, bool X, int M>
__global__ void __launch_bounds__(P2_SPLIT_TPB, 7) k_pass_split(
	ST *__restrict__ st, const struct phase2_pass p,
	const struct p2_sub *__restrict__ subs, uint32_t nsub,
	const struct p2_sub_rec *__restrict__ recs)
{
	constexpr int LB = P2_SPLIT_BITS - M;
	constexpr int UL = 7 - LB; /* slot bits in the thread number */
	extern __shared__ __align__(16) unsigned char p2_split_dyn[];
	const uint32_t tid = threadIdx.x;
	struct p2_sub_rec *const srec =
		(struct p2_sub_rec *)(p2_split_dyn + (16 << P2_SPLIT_BITS));
	struct p2_sub *const hdr = (struct p2_sub *)(srec + p.nrot);
	const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(p2_split_dyn);
	const uint64_t t0 = (uint64_t)blockIdx.x << LB;
	const uint64_t xb = p2_rep<M>(t0, p);
	for (uint32_t k = tid; k < p.nrot; k += P2_SPLIT_TPB) {
		struct p2_sub_rec r = recs[p.rot_off + k];
		/* the tile's part of the sign parity (pad1: the phase mask) */
		r.sm ^= (uint8_t)(0u - (uint32_t)(__popcll(xb & r.pad1) & 1));
		srec[k] = r;
	}
	for (uint32_t k = tid; k < 4 * nsub; k += P2_SPLIT_TPB)
		((uint4 *)hdr)[k] = ((const uint4 *)subs)[k];
	uint64_t x = p2_rep<M>(t0 + (tid & ((1u << LB) - 1u)), p);
#pragma unroll
	for (int k = 0; k < UL; ++k)
		x ^= (0u - (uint64_t)(tid >> (LB + k) & 1)) & p.basis[k];
	p2_grid_wait();
#pragma unroll
	for (int i = 0; i < P2_RES_SLOTS; ++i) {
		uint64_t off = 0;
#pragma unroll
		for (int k = 0; k < 3; ++k)
			if (i >> k & 1)
				off ^= p.basis[UL + k];
		double re, im;
		p2_ld(st, x ^ off, re, im);
		p2_res_st<false>(sbase + 16 * p2_sub_swz(tid + 128u * i), re, im);
	}
	__syncthreads();
	for (uint32_t i = 0; i < nsub; ++i) {
		const struct p2_sub &h = hdr[i];
		const struct p2_sub_rec *const q0 = srec + (h.rot_off - p.rot_off);
		uint32_t y = tid;
#pragma unroll
		for (int k = 0; k < P2_SUB_SPAN; ++k) {
			const uint32_t q = h.piv[k];
			y = ((y >> q) << (q + 1)) | (y & ((1u << q) - 1u));
		}
		if constexpr (X) {
			const uint32_t y0 = y;
#pragma unroll
			for (int k = 0; k < P2_SUB_SPAN; ++k)
				y ^= (0u - p2_parity(y0 & h.orient[k])) & h.slot[k];
		}
		const uint32_t py = p2_sub_swz(y);
		uint32_t addr[P2_RES_SLOTS];
		double re[P2_RES_SLOTS], im[P2_RES_SLOTS];
#pragma unroll
		for (int u = 0; u < P2_RES_SLOTS; ++u) {
			uint32_t a = py;
#pragma unroll
			for (int k = 0; k < P2_SUB_SPAN; ++k)
				if (u >> k & 1)
					a ^= h.pslot[k];
			addr[u] = sbase + 16 * a;
			p2_res_ld<false>(addr[u], re[u], im[u]);
		}
		const uint32_t nrot = h.nrot;
		for (uint32_t r = 0; r < nrot; ++r) {
			const struct p2_sub_rec q = q0[r];
			p2_sub_apply<X>(q, re, im,
				(uint32_t)q.sm ^ (0u - p2_parity(y & q.z)));
		}
#pragma unroll
		for (int u = 0; u < P2_RES_SLOTS; ++u)
			p2_res_st<false>(addr[u], re[u], im[u]);
		__syncthreads();
	}
	/* late: blocks that wait for this kernel take places from its own */
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
	const uint32_t neg = X && p.scale < 0 ? 0x80000000u : 0u;
#pragma unroll
	for (int i = 0; i < P2_RES_SLOTS; ++i) {
		uint64_t off = 0;
#pragma unroll
		for (int k = 0; k < 3; ++k)
			if (i >> k & 1)
				off ^= p.basis[UL + k];
		double re, im;
		p2_res_ld<false>(sbase + 16 * p2_sub_swz(tid + 128u * i), re, im);
		if constexpr (X) {
			re = p2_sgn(re, neg);
			im = p2_sgn(im, neg);
		}
		p2_st(st, x ^ off, re, im);
	}
}

/* ---- host ----------------------------------------------------------------- */

/*
 * Up to 19 qubits: us a pass at 17 / 19 / 20 qubits, FP64 (the pass kernels
 * in brackets): 5.6 draws a pass 3.4 (5.8) / 5.8 (6.0) / 8.3 (7.5), 17
 * strings in lexicographic order 5.4 (9.8) / 9.6 (10.2) / 14.0 (13.1), 50
 * rotations sorted by flip mask 11.2 (21.6) / 18.1 (20.2) / 28.4 (28.2);
 * FP32 at 19: 5.0 (5.5), 8.7 (9.8), 16.9 (20.2).  From 20 qubits on every
 * scheduler has enough cosets, and the work a rotation costs beside its
 * FP64 operations counts per 8 amplitudes here, per 32 there.
 */
bool p2_split_ok(const struct p2_dev *d, int form)
{
	return d->nqb >= P2_SPLIT_MIN_QB && d->nqb <= P2_SPLIT_MAX_QB &&
		form != PHASE2_FORM_LIFTED_F32;
}

template <typename ST, bool X, int M>
static cudaError_t split_launch_m(struct p2_dev *d, const struct p2_split_pass &sp,
	const struct p2_sub *subs, const struct p2_sub_rec *recs)
{
	static uint64_t done;
	unsigned ok;
	if (!p2_done(&done, d->context, &ok)) {
		const cudaError_t e = cudaFuncSetAttribute(k_pass_split<ST, X, M>,
			cudaFuncAttributeMaxDynamicSharedMemorySize,
			(int)P2_SPLIT_SMEM);
		if (e != cudaSuccess)
			return e;
		p2_set_done(&done, d->context, 1);
	}
	return p2_launch(k_pass_split<ST, X, M>,
		(unsigned)(d->namp >> P2_SPLIT_BITS), P2_SPLIT_TPB,
		(16 << P2_SPLIT_BITS) + sp.pass.nrot * sizeof(struct p2_sub_rec) +
			sp.nsub * sizeof(struct p2_sub),
		d->stream, (ST *)d->state, sp.pass, subs + sp.sub_off, sp.nsub,
		recs);
}

template <typename ST, bool X>
static int split_launch(struct p2_dev *d, const struct p2_graph *g)
{
	const struct p2_sub_rec *recs = (const struct p2_sub_rec *)g->d_recs;
	const struct p2_sub *subs = (const struct p2_sub *)(recs + g->nrec);
	for (size_t i = 0; i < g->npass; i++) {
		const struct p2_split_pass &sp = g->split[i];
		CUDA_OK(sp.pass.span == 5
				? (split_launch_m<ST, X, 5>(d, sp, subs, recs))
				: sp.pass.span == 4
				? (split_launch_m<ST, X, 4>(d, sp, subs, recs))
				: (split_launch_m<ST, X, 3>(d, sp, subs, recs)),
			"split pass launch");
	}
	return 0;
}

int p2_split_run(struct p2_dev *d, const struct p2_graph *g)
{
	return d->prec == PHASE2_PREC_FP64 ? split_launch<double2, false>(d, g)
					   : split_launch<float2, true>(d, g);
}
