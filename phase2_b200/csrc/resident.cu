/*
 * resident.cu -- small registers held on chip: one launch runs a whole
 * flush.
 *
 * A register of up to 14 qubits is at most 256 KiB (as complex doubles): one
 * block, or one thread-block cluster, holds it in shared memory, so the
 * passes of a flush need no kernel boundary between them, only a barrier.
 * The pass kernels spend 5 us on such a pass of 5 random strings: a launch,
 * one or a few blocks of cold code (64 cases of 32 unrolled slots), and one
 * warp a scheduler whose FP64 operations wait for one another.  Here a
 * sub-pass of 3 strings takes 1 us, bound by latencies (ncu, 10 qubits: one
 * instruction in 4 cycles and scheduler, 1.7 of them fixed-latency waits;
 * 144 warp instructions a rotation, 48 of them FP64 products and sums).
 * ns a rotation, 10 / 12 / 14 qubits: random strings 322 / 608 / 921
 * (pass kernels 943 / 1122 / 1133), excitation groups of 8 strings 169 /
 * 204 / 234 (402 / 430 / 430).
 */
#include <cuda_runtime.h>

#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define LOG_SUBSYS "engine"
#include "log.h"

#include "p2_sub.cuh"
#include "tile_core.h"

#define P2_RES_MIN_QB 3
#define P2_RES_MIN_SHARE 5 /* log2 of a block's least share of a register */
#define P2_RES_MAX_QB 14
#define P2_RES_TPB 256
/* samples: many run at once, so a block may take a whole register */
#define P2_RES_SMP_TPB 1024
#define P2_RES_SMEM (16 << 13) /* the most amplitudes of a block, 2^13 */

/* ---- the kernel ---------------------------------------------------------- */

/* Sub-passes whose records are on their way or in use, and headers held:
 * a sub-pass can be shorter than the latency of a copy from L2. */
#define P2_RES_STAGES 4
#define P2_RES_HDRS 8

/* Start the copy of sub-pass j's records (one commit group a call). */
__device__ __forceinline__ void p2_res_stage(uint32_t j, uint32_t nsub,
	const struct p2_sub *hdr,
	struct p2_sub_rec (*srec)[P2_SUB_ROTS],
	const struct p2_sub_rec *__restrict__ recs, uint32_t tid, uint32_t nt)
{
	if (j < nsub) {
		const struct p2_sub &h = hdr[j % P2_RES_HDRS];
		const uint32_t dst = (uint32_t)__cvta_generic_to_shared(
			&srec[j % P2_RES_STAGES][0]);
		const unsigned char *const src =
			(const unsigned char *)(recs + h.rot_off);
		for (uint32_t k = tid; k < 2u * h.nrot; k += nt)
			p2_cp16(dst + 16 * k, src + 16 * k);
	}
	p2_cp_commit();
}

/* Per-block staging of k_resident's kernels. */
struct p2_res_stagebuf {
	struct p2_sub hdr[P2_RES_HDRS];
	struct p2_sub_rec rec[P2_RES_STAGES][P2_SUB_ROTS];
};

/*
 * The sub-passes subs[0..nsub) on the register held by the cluster (CL) or
 * block: blocks of 2^kc amplitudes each, thread t of all threads.  A
 * sub-pass is one trip of every amplitude through registers (8 a thread)
 * and one barrier; the records of later sub-passes and their headers are
 * copied to shared memory meanwhile.  The state is held as complex doubles
 * whatever its precision: FP32 states round at the end of each pass, where
 * the pass kernels do.  Every thread of the cluster calls it; the barrier
 * at its start orders the caller's stores to shared memory before it.
 */
template <bool X, bool CL>
__device__ __forceinline__ void p2_res_run(uint32_t nqb, uint32_t kc,
	uint32_t sbase, uint32_t t, const struct p2_sub *__restrict__ subs,
	uint32_t nsub, const struct p2_sub_rec *__restrict__ recs,
	struct p2_res_stagebuf &sb)
{
	const uint32_t tid = threadIdx.x, nt = blockDim.x;
	const bool active = t < (1u << (nqb - P2_SUB_SPAN));
	for (uint32_t k = tid; k < 4 * P2_RES_HDRS && k < 4 * nsub; k += nt)
		p2_cp16((uint32_t)__cvta_generic_to_shared(sb.hdr) + 16 * k,
			(const unsigned char *)subs + 16 * k);
	p2_cp_commit();
	p2_cp_wait<0>();
	__syncthreads();
	for (uint32_t j = 0; j < P2_RES_STAGES - 1; ++j)
		p2_res_stage(j, nsub, sb.hdr, sb.rec, recs, tid, nt);
	p2_cp_wait<P2_RES_STAGES - 2>();
	p2_res_barrier<CL>();

	for (uint32_t i = 0; i < nsub; ++i) {
		const struct p2_sub &h = sb.hdr[i % P2_RES_HDRS];
		const struct p2_sub_rec *const q0 = sb.rec[i % P2_RES_STAGES];
		/* the header whose records are staged P2_RES_STAGES - 1 rounds
		 * from now, into the place of the one just done */
		if (i > 0 && i + P2_RES_HDRS - 1 < nsub && tid < 4)
			p2_cp16((uint32_t)__cvta_generic_to_shared(
					&sb.hdr[(i - 1) % P2_RES_HDRS]) + 16 * tid,
				(const unsigned char *)(subs + i +
					P2_RES_HDRS - 1) + 16 * tid);
		p2_res_stage(i + P2_RES_STAGES - 1, nsub, sb.hdr, sb.rec, recs,
			tid, nt);
		if (active) {
			uint32_t x = t;
#pragma unroll
			for (int k = 0; k < P2_SUB_SPAN; ++k) {
				const uint32_t p = h.piv[k];
				x = ((x >> p) << (p + 1)) | (x & ((1u << p) - 1u));
			}
			if constexpr (X) {
				const uint32_t x0 = x;
#pragma unroll
				for (int k = 0; k < P2_SUB_SPAN; ++k)
					x ^= (0u - p2_parity(x0 & h.orient[k])) &
						h.slot[k];
			}
			const uint32_t px = p2_sub_swz(x);
			uint32_t addr[P2_RES_SLOTS];
			double re[P2_RES_SLOTS], im[P2_RES_SLOTS];
#pragma unroll
			for (int u = 0; u < P2_RES_SLOTS; ++u) {
				uint32_t p = px;
#pragma unroll
				for (int k = 0; k < P2_SUB_SPAN; ++k)
					if (u >> k & 1)
						p ^= h.pslot[k];
				addr[u] = p2_res_addr<CL>(sbase, p, kc);
				p2_res_ld<CL>(addr[u], re[u], im[u]);
			}
			const uint32_t nrot = h.nrot;
			for (uint32_t r = 0; r < nrot; ++r) {
				const struct p2_sub_rec q = q0[r];
				p2_sub_apply<X>(q, re, im,
					(uint32_t)q.sm ^ (0u - p2_parity(x & q.z)));
			}
			if (X && (h.flags & P2_SUB_LAST)) {
				const uint32_t neg = h.flags & P2_SUB_NEG
					? 0x80000000u : 0u;
#pragma unroll
				for (int u = 0; u < P2_RES_SLOTS; ++u) {
					re[u] = (double)__double2float_rn(
						p2_sgn(re[u], neg));
					im[u] = (double)__double2float_rn(
						p2_sgn(im[u], neg));
				}
			}
#pragma unroll
			for (int u = 0; u < P2_RES_SLOTS; ++u)
				p2_res_st<CL>(addr[u], re[u], im[u]);
		}
		p2_cp_wait<P2_RES_STAGES - 2>();
		p2_res_barrier<CL>();
	}
	p2_cp_wait<0>();
}

/* A register's flush: load, run, store. */
template <typename ST, bool X, bool CL>
__global__ void __launch_bounds__(P2_RES_TPB) k_resident(ST *__restrict__ st,
	uint32_t nqb, uint32_t kc, const struct p2_sub *__restrict__ subs,
	uint32_t nsub, const struct p2_sub_rec *__restrict__ recs)
{
	extern __shared__ __align__(16) unsigned char p2_res_dyn[];
	__shared__ __align__(16) struct p2_res_stagebuf sb;
	const uint32_t tid = threadIdx.x, nt = blockDim.x;
	const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(p2_res_dyn);
	const uint32_t rank = CL ? blockIdx.x : 0u;
	const uint32_t mine = 1u << kc, first = rank << kc;
	for (uint32_t i = tid; i < mine; i += nt) {
		double re, im;
		p2_ld(st, first + i, re, im);
		p2_res_st<false>(p2_res_addr<false>(sbase,
				 p2_sub_swz(first + i), kc), re, im);
	}
	p2_res_run<X, CL>(nqb, kc, sbase, rank * nt + tid, subs, nsub, recs, sb);
	for (uint32_t i = tid; i < mine; i += nt) {
		double re, im;
		p2_res_ld<false>(p2_res_addr<false>(sbase,
				 p2_sub_swz(first + i), kc), re, im);
		p2_st(st, first + i, re, im);
	}
}

/*
 * Samples of a sampled driver (sampling.cu), one cluster of 2^lb blocks
 * each, entirely on chip: zero, the trial state's determinants (in order:
 * later writes win), the sub-passes of every chunk, the determinants'
 * amplitudes out.  Only sample `keep` of the round stores its state.
 */
template <typename ST, bool X, bool CL>
__global__ void __launch_bounds__(P2_RES_SMP_TPB) k_resident_smp(
	const struct p2_res_samples a)
{
	extern __shared__ __align__(16) unsigned char p2_res_dyn[];
	__shared__ __align__(16) struct p2_res_stagebuf sb;
	const uint32_t tid = threadIdx.x, nt = blockDim.x;
	const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(p2_res_dyn);
	const uint32_t kc = a.nqb - a.lb, low = (1u << kc) - 1u;
	const uint64_t s = blockIdx.x >> a.lb;
	const uint32_t rank = CL ? blockIdx.x & ((1u << a.lb) - 1u) : 0u;
	const uint32_t mine = 1u << kc, first = rank << kc;
	for (uint32_t i = tid; i < mine; i += nt)
		p2_res_st<false>(sbase + 16 * i, 0.0, 0.0);
	__syncthreads();
	if (tid == 0)
		for (uint32_t e = 0; e < a.ndet; ++e) {
			const uint32_t g = (uint32_t)a.widx[e];
			if (g >> kc != rank)
				continue;
			double re = a.wval[2 * e], im = a.wval[2 * e + 1];
			if (sizeof(ST) == 8) {
				re = (double)__double2float_rn(re);
				im = (double)__double2float_rn(im);
			}
			p2_res_st<false>(sbase + 16 * (p2_sub_swz(g) & low), re,
				im);
		}
	const struct p2_sub_rec *const recs = a.recs + s * a.T;
	for (uint32_t c = 0; c < a.C; ++c)
		p2_res_run<X, CL>(a.nqb, kc, sbase, rank * nt + tid,
			a.subs + s * a.T + (uint64_t)c * P2_QUEUE_FLUSH,
			a.nsub[s * a.C + c], recs, sb);
	/* its last barrier (or, without sub-passes, its first) ordered every
	 * block's stores before these reads of the block's own part */
	for (uint32_t e = tid; e < a.ndet; e += nt) {
		const uint32_t g = (uint32_t)a.widx[e];
		if (g >> kc != rank)
			continue;
		double re, im;
		p2_res_ld<false>(sbase + 16 * (p2_sub_swz(g) & low), re, im);
		a.gout[s * a.ndet + e] = make_double2(re, im);
	}
	if (s == a.keep)
		for (uint32_t i = tid; i < mine; i += nt) {
			double re, im;
			p2_res_ld<false>(sbase + 16 *
					(p2_sub_swz(first + i) & low), re, im);
			p2_st((ST *)a.state, first + i, re, im);
		}
}

/*
 * A batch's programs (batch.cu), one cluster of 2^lb blocks each: the
 * register's state stays on chip from the first op to the last.  A register
 * too narrow to share out lies in the first block alone; the others keep the
 * barriers.
 */
template <typename ST, bool X, bool CL>
__global__ void __launch_bounds__(P2_RES_SMP_TPB) k_resident_prog(
	const struct p2_res_prog *__restrict__ progs, uint32_t lb,
	const uint64_t *__restrict__ widx, const double *__restrict__ wval,
	const uint64_t *__restrict__ gidx, double2 *__restrict__ gout,
	struct p2_bctl *__restrict__ ctl, unsigned long long *start)
{
	extern __shared__ __align__(16) unsigned char p2_res_dyn[];
	__shared__ __align__(16) struct p2_res_stagebuf sb;
	const uint32_t tid = threadIdx.x, nt = blockDim.x;
	const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(p2_res_dyn);
	const uint32_t rank = CL ? blockIdx.x & ((1u << lb) - 1u) : 0u;
	const uint32_t who = blockIdx.x >> lb;
	const struct p2_res_prog a = progs[who];
	const bool shared_out = CL && a.nqb >= lb + P2_RES_MIN_SHARE;
	const uint32_t kc = shared_out ? a.nqb - lb : a.nqb;
	const uint32_t low = (1u << kc) - 1u, first = rank << kc;
	const bool mine = shared_out || rank == 0;
	const uint32_t n = mine ? 1u << kc : 0u;
	/* threads of a block beyond its share of the register idle */
	const uint32_t share = 1u << (kc - P2_SUB_SPAN);
	const uint32_t t = mine && tid < share ? rank * share + tid : ~0u;
	if (blockIdx.x == 0 && tid == 0)
		atomicMax(start, ~p2_globaltimer());
	for (uint32_t i = tid; i < n; i += nt) {
		double re, im;
		p2_ld((const ST *)a.state, first + i, re, im);
		p2_res_st<false>(sbase + 16 * (p2_sub_swz(first + i) & low), re,
			im);
	}
	for (uint32_t o = 0; o < a.nops; ++o) {
		const struct p2_res_op op = a.ops[o];
		if (op.kind == P2_RES_RUN) {
			p2_res_run<X, CL>(a.nqb, kc, sbase, t, a.subs + op.a,
				op.b, a.recs, sb);
			continue;
		}
		/* between two runs a block touches only its own amplitudes */
		__syncthreads();
		if (op.kind == P2_OP_ZERO) {
			for (uint32_t i = tid; i < n; i += nt)
				p2_res_st<false>(sbase + 16 * i, 0.0, 0.0);
		} else if (op.kind == P2_OP_WRITE) {
			/* in order: later writes win */
			for (uint32_t e = op.a; tid == 0 && e < op.a + op.b; ++e) {
				const uint32_t g = (uint32_t)widx[e];
				if (!mine || g >> kc != rank)
					continue;
				double re = wval[2 * e], im = wval[2 * e + 1];
				if (sizeof(ST) == 8) {
					re = (double)__double2float_rn(re);
					im = (double)__double2float_rn(im);
				}
				p2_res_st<false>(sbase + 16 *
						(p2_sub_swz(g) & low), re, im);
			}
		} else {
			for (uint32_t e = op.a + tid; e < op.a + op.b; e += nt) {
				const uint32_t g = (uint32_t)gidx[e];
				if (!mine || g >> kc != rank)
					continue;
				double re, im;
				p2_res_ld<false>(sbase + 16 *
						(p2_sub_swz(g) & low), re, im);
				gout[e] = make_double2(re, im);
			}
		}
		__syncthreads();
	}
	for (uint32_t i = tid; i < n; i += nt) {
		double re, im;
		p2_res_ld<false>(sbase + 16 * (p2_sub_swz(first + i) & low), re,
			im);
		p2_st((ST *)a.state, first + i, re, im);
	}
	if (rank == 0 && tid == 0)
		ctl[who].end_ns = p2_globaltimer();
}

/* ---- host side ----------------------------------------------------------- */

/*
 * log2 of the blocks of a register's cluster: one block up to 11 qubits,
 * where a second block only adds the cluster barrier and remote shared
 * memory (11 qubits, random strings, ns a rotation: 399 on one block, 592
 * on two); 8 at 12 qubits (608; 645 on one, 731 on four), 16 at 13 and 14
 * (651 and 921; the pass kernels 1112 and 1133).  At 15 qubits the traffic
 * between the blocks bounds a sub-pass (1583) and the pass kernels are
 * faster (1122).
 */
static uint32_t res_log_blocks(uint32_t nqb)
{
	return nqb <= 11 ? 0 : nqb == 12 ? 3 : 4;
}

/* 64-bit words, four chains (n a multiple of 8). */
static uint64_t hash_words(uint64_t h, const void *p, size_t n)
{
	const unsigned char *b = (const unsigned char *)p;
	uint64_t c[4] = { h, ~h, h << 7, h >> 9 };
	size_t i = 0;
	for (; i + 32 <= n; i += 32) {
		uint64_t w[4];
		memcpy(w, b + i, 32);
		for (int k = 0; k < 4; k++) {
			c[k] = (c[k] ^ w[k]) * UINT64_C(0x9e3779b97f4a7c15);
			c[k] ^= c[k] >> 29;
		}
	}
	for (; i + 8 <= n; i += 8) {
		uint64_t w;
		memcpy(&w, b + i, 8);
		c[0] = (c[0] ^ w) * UINT64_C(0x9e3779b97f4a7c15);
		c[0] ^= c[0] >> 29;
	}
	for (int k = 1; k < 4; k++)
		c[0] = (c[0] ^ c[k]) * UINT64_C(0x9e3779b97f4a7c15) ^
			(c[k] >> 31);
	return c[0];
}

/*
 * The device copy of a flush's sub-passes: found among the last
 * P2_GRAPH_SLOTS plans of the register by plan id (the same flush again) or
 * by content, or built and uploaded into the least recently used slot
 * (stream order keeps the copy behind the launches that read the slot).
 * kind: sub-passes of the register (here), of each pass on tiles of its own
 * (split.cu), or tile runs (tile.cu).
 * *hit: found.  NULL on failure.
 */
struct p2_graph *p2_sub_plan(struct p2_dev *d,
	const struct phase2_pass *passes, size_t npass,
	const struct phase2_rot_rec *recs, size_t nrec, uint64_t plan_id,
	enum p2_plan_kind kind, bool *hit)
{
	struct p2_graph *lru = &d->graphs[0];
	d->graph_clock++;
	*hit = true;
	for (int k = 0; k < P2_GRAPH_SLOTS; k++) {
		struct p2_graph *g = &d->graphs[k];
		if (plan_id && g->nsub && g->plan_id == plan_id) {
			g->used = d->graph_clock;
			return g;
		}
	}
	uint64_t h = hash_words(UINT64_C(0xcbf29ce484222325), passes,
		npass * sizeof *passes);
	h = hash_words(h, recs, nrec * sizeof *recs);
	for (int k = 0; k < P2_GRAPH_SLOTS; k++) {
		struct p2_graph *g = &d->graphs[k];
		if (g->nsub && g->hash == h && g->npass == npass &&
			g->nrec == nrec &&
			!memcmp(g->passes, passes, npass * sizeof *passes) &&
			!memcmp(g->recs, recs, nrec * sizeof *recs)) {
			g->used = d->graph_clock;
			g->plan_id = plan_id;
			return g;
		}
		if (g->used < lru->used)
			lru = g;
	}
	*hit = false;
	if (lru->d_cap) {
		/* keep the device buffer of a resident plan */
		free(lru->passes);
		free(lru->recs);
		free(lru->split);
		free(lru->tiles);
		lru->split = NULL;
		lru->tiles = NULL;
		lru->nsub = lru->ntile = 0;
	} else {
		p2_graph_drop(d, lru);
	}
	lru->passes = (struct phase2_pass *)malloc(npass * sizeof *passes);
	lru->recs = (struct phase2_rot_rec *)malloc(nrec * sizeof *recs);
	lru->hash = h;
	lru->npass = npass;
	lru->nrec = nrec;
	lru->plan_id = 0;
	lru->used = 0;
	if (kind == P2_PLAN_SPLIT)
		lru->split = (struct p2_split_pass *)malloc(
			npass * sizeof *lru->split);
	if (kind == P2_PLAN_TILE)
		lru->tiles = (struct p2_tile *)malloc(
			nrec * sizeof *lru->tiles);
	if (!lru->passes || !lru->recs ||
		(kind == P2_PLAN_SPLIT && !lru->split) ||
		(kind == P2_PLAN_TILE && !lru->tiles))
		goto fail;
	memcpy(lru->passes, passes, npass * sizeof *passes);
	memcpy(lru->recs, recs, nrec * sizeof *recs);
	{
		/* staging: sub-passes from the end of the records' area on (at
		 * most one a rotation) */
		struct phase2_rot_rec *stage =
			p2_stage_reserve(d, 3 * nrec);
		if (!stage)
			goto fail;
		struct p2_sub_rec *const sr = (struct p2_sub_rec *)stage;
		struct p2_sub *const ss = (struct p2_sub *)(sr + nrec);
		uint32_t n = 0;
		size_t sub_bytes = sizeof *ss;
		if (kind == P2_PLAN_TILE) {
			lru->ntile = p2_tile_build(passes, npass, recs, nrec,
				lru->tiles, (struct p2_tile_sub *)ss,
				(struct p2_tile_rec *)sr, &n);
			sub_bytes = sizeof(struct p2_tile_sub);
			struct p2_tile *fit = (struct p2_tile *)realloc(
				lru->tiles, lru->ntile * sizeof *fit);
			if (fit)
				lru->tiles = fit;
		}
		for (size_t i = 0; i < npass && kind != P2_PLAN_TILE; i++)
			if (kind == P2_PLAN_SPLIT) {
				p2_split_build(d->nqb, &passes[i], recs,
					&lru->split[i], n, ss + n, sr);
				n += lru->split[i].nsub;
			} else {
				n += p2_sub_split(&passes[i],
					recs + passes[i].rot_off, d->nqb,
					passes[i].rot_off, ss + n,
					sr + passes[i].rot_off);
			}
		const size_t bytes = nrec * sizeof *sr + n * sub_bytes;
		if (bytes > lru->d_cap) {
			p2_scratch_free(lru->d_recs, d->stream);
			lru->d_recs = NULL;
			lru->d_cap = 0;
			if (p2_scratch_alloc((void **)&lru->d_recs, bytes,
				    d->stream) != cudaSuccess) {
				lru->d_recs = NULL;
				goto fail;
			}
			lru->d_cap = bytes;
		}
		if (p2_stage_upload(d, lru->d_recs, bytes) < 0)
			goto fail;
		lru->nsub = n;
	}
	lru->plan_id = plan_id;
	lru->used = d->graph_clock;
	return lru;
fail:
	log_warn("no room for a flush's sub-passes: pass kernels");
	cudaGetLastError();
	p2_graph_drop(d, lru);
	return NULL;
}

/* Largest cluster a kernel can be launched with on this device (blocks of
 * 128 threads and 16 KiB), once per kernel and context; 0 when it cannot be
 * configured. */
template <auto F>
static unsigned res_clusters(const struct p2_dev *d, bool clusters)
{
	static uint64_t done;
	unsigned best;
	if (p2_done(&done, d->context, &best))
		return best;
	best = 0;
	if (cudaFuncSetAttribute(F, cudaFuncAttributeMaxDynamicSharedMemorySize,
		    P2_RES_SMEM) == cudaSuccess) {
		best = 1;
		if (clusters && cudaFuncSetAttribute(F,
				cudaFuncAttributeNonPortableClusterSizeAllowed,
				1) != cudaSuccess)
			best = 0;
		for (unsigned c = 16; clusters && best == 1 && c > 1; c /= 2) {
			cudaLaunchConfig_t cfg;
			cudaLaunchAttribute at[1];
			memset(&cfg, 0, sizeof cfg);
			memset(at, 0, sizeof at);
			at[0].id = cudaLaunchAttributeClusterDimension;
			at[0].val.clusterDim.x = c;
			at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
			cfg.gridDim = dim3(c);
			cfg.blockDim = dim3(128);
			cfg.dynamicSmemBytes = 16 << 10;
			cfg.attrs = at;
			cfg.numAttrs = 1;
			int n = 0;
			if (cudaOccupancyMaxActiveClusters(&n, F, &cfg) ==
					cudaSuccess && n > 0)
				best = c;
		}
	}
	cudaGetLastError();
	p2_set_done(&done, d->context, best);
	return best;
}

/* A register width and form the kernels here take. */
static bool res_width_ok(const struct p2_dev *d, int form)
{
	return d->nqb >= P2_RES_MIN_QB && d->nqb <= P2_RES_MAX_QB &&
		form != PHASE2_FORM_LIFTED_F32;
}

bool p2_resident_ok(const struct p2_dev *d, int form)
{
	if (!res_width_ok(d, form))
		return false;
	const uint32_t lb = res_log_blocks(d->nqb);
	const unsigned most = d->prec == PHASE2_PREC_FP64
		? (lb ? res_clusters<k_resident<double2, false, true>>(d, true)
		      : res_clusters<k_resident<double2, false, false>>(d, false))
		: (lb ? res_clusters<k_resident<float2, true, true>>(d, true)
		      : res_clusters<k_resident<float2, true, false>>(d, false));
	return most >= (1u << lb);
}

/* Launch blocks of a register's (or sample's) share in clusters of 2^lb:
 * grid blocks, one thread for 8 amplitudes. */
template <typename F, typename... A>
static cudaError_t res_launch(F *fn, unsigned grid, uint32_t nqb, uint32_t lb,
	cudaStream_t stream, A... args)
{
	cudaLaunchConfig_t cfg;
	cudaLaunchAttribute at[1];
	uint32_t tpb = 1u << (nqb - P2_SUB_SPAN - lb);
	if (tpb < 32)
		tpb = 32;
	memset(&cfg, 0, sizeof cfg);
	memset(at, 0, sizeof at);
	cfg.gridDim = dim3(grid);
	cfg.blockDim = dim3(tpb);
	cfg.dynamicSmemBytes = (size_t)16 << (nqb - lb);
	cfg.stream = stream;
	if (lb) {
		at[0].id = cudaLaunchAttributeClusterDimension;
		at[0].val.clusterDim.x = 1u << lb;
		at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
		cfg.attrs = at;
		cfg.numAttrs = 1;
	}
	return cudaLaunchKernelEx(&cfg, fn, args...);
}

template <typename ST, bool X>
static int res_launch_flush(struct p2_dev *d, const struct p2_graph *g)
{
	const uint32_t lb = res_log_blocks(d->nqb);
	const struct p2_sub_rec *sr = (const struct p2_sub_rec *)g->d_recs;
	const struct p2_sub *subs = (const struct p2_sub *)(sr + g->nrec);
	CUDA_OK(res_launch(lb ? k_resident<ST, X, true>
			      : k_resident<ST, X, false>,
			1u << lb, d->nqb, lb, d->stream, (ST *)d->state, d->nqb,
			d->nqb - lb, subs, g->nsub, sr),
		"resident launch");
	return 0;
}

int p2_resident_run(struct p2_dev *d, const struct p2_graph *g)
{
	return d->prec == PHASE2_PREC_FP64
		? res_launch_flush<double2, false>(d, g)
		: res_launch_flush<float2, true>(d, g);
}

/* ---- samples -------------------------------------------------------------- */

/*
 * log2 of a sample's blocks in a round of g samples: more blocks shorten one
 * sample, but the traffic between them costs throughput, so only as many as
 * leave half of the SMs a block (1000 draws, us a call, blocks a sample 1 /
 * 2 / 4 / 8 / 16: 13 qubits, 8 samples 1534 / 1441 / 1353 / 1118 / 1150, 32
 * samples 1581 / 1512 / 1485 / 1577 / 1724, 128 samples 1812 / 2424 / 3651 /
 * 3964 / 4559).  A block holds 2^13 amplitudes at most.
 */
static uint32_t res_sample_blocks(uint32_t nqb, int sm_count, uint64_t g)
{
	const uint32_t least = nqb > 13 ? nqb - 13 : 0;
	uint32_t lb = res_log_blocks(nqb);
	while (lb > least && (g << lb) > (uint64_t)sm_count / 2)
		lb--;
	return lb;
}

bool p2_resident_samples_ok(const struct p2_dev *d, int form)
{
	if (!res_width_ok(d, form))
		return false;
	/* both kernels: the number of samples chooses between them */
	const unsigned need = 1u << res_log_blocks(d->nqb);
	return d->prec == PHASE2_PREC_FP64
		? res_clusters<k_resident_smp<double2, false, true>>(d, true) >=
				need &&
			res_clusters<k_resident_smp<double2, false, false>>(
				d, false) >= 1
		: res_clusters<k_resident_smp<float2, true, true>>(d, true) >=
				need &&
			res_clusters<k_resident_smp<float2, true, false>>(
				d, false) >= 1;
}

template <typename ST, bool X>
static cudaError_t res_launch_samples(struct p2_dev *d,
	const struct p2_res_samples &a, uint32_t g)
{
	return res_launch(a.lb ? k_resident_smp<ST, X, true>
			       : k_resident_smp<ST, X, false>,
		g << a.lb, a.nqb, a.lb, d->stream, a);
}

cudaError_t p2_resident_samples(struct p2_dev *d, struct p2_res_samples a,
	uint32_t g)
{
	a.nqb = d->nqb;
	a.lb = res_sample_blocks(d->nqb, d->sm_count, g);
	a.state = d->state;
	return d->prec == PHASE2_PREC_FP64
		? res_launch_samples<double2, false>(d, a, g)
		: res_launch_samples<float2, true>(d, a, g);
}

/* ---- batch programs ------------------------------------------------------- */

bool p2_resident_prog_ok(const struct p2_dev *d, int form)
{
	if (!res_width_ok(d, form))
		return false;
	/* any width's clusters: the batch's widest register chooses them */
	return d->prec == PHASE2_PREC_FP64
		? res_clusters<k_resident_prog<double2, false, true>>(d, true) >= 16 &&
			res_clusters<k_resident_prog<double2, false, false>>(
				d, false) >= 1
		: res_clusters<k_resident_prog<float2, true, true>>(d, true) >= 16 &&
			res_clusters<k_resident_prog<float2, true, false>>(
				d, false) >= 1;
}

template <typename ST, bool X>
static cudaError_t res_launch_progs(uint32_t nqb, uint32_t lb, uint32_t g,
	cudaStream_t stream, const struct p2_res_prog *progs,
	const uint64_t *widx, const double *wval, const uint64_t *gidx,
	double2 *gout, struct p2_bctl *ctl, unsigned long long *start)
{
	return res_launch(lb ? k_resident_prog<ST, X, true>
			     : k_resident_prog<ST, X, false>,
		g << lb, nqb, lb, stream, progs, lb, widx, wval, gidx, gout, ctl,
		start);
}

cudaError_t p2_resident_progs(const struct p2_dev *d, uint32_t nqb, uint32_t g,
	uint32_t even, const struct p2_res_prog *progs, const uint64_t *widx,
	const double *wval, const uint64_t *gidx, double2 *gout,
	struct p2_bctl *ctl, unsigned long long *start)
{
	uint32_t lb = res_sample_blocks(nqb, d->sm_count, even);
	/* at 14 qubits a program has two blocks in any case: four each, as
	 * long as an SM in eight stays free for the clusters to fit in */
	if (nqb == 14 && lb == 1 && (even << 2) <= (uint32_t)d->sm_count * 7 / 8)
		lb = 2;
	return d->prec == PHASE2_PREC_FP64
		? res_launch_progs<double2, false>(nqb, lb, g, d->stream, progs,
			  widx, wval, gidx, gout, ctl, start)
		: res_launch_progs<float2, true>(nqb, lb, g, d->stream, progs,
			  widx, wval, gidx, gout, ctl, start);
}
