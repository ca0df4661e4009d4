/*
 * onchip.cu -- many samples of registers of 12 to 14 qubits: one block or one
 * cluster a sample, whole passes on the state in shared memory.
 *
 * k_resident_smp moves every amplitude through registers twice or three
 * times a pass, as a complex double, and at 14 qubits half of them through
 * another block's shared memory: with tens of samples that traffic bounds it
 * (32 FP32 samples of 1000 draws, 14 qubits: 1.9 ms).  Here the register is
 * held as it is stored, and a thread takes a coset of 32 amplitudes through a
 * whole pass, as the pass kernels do: an eighth (FP64: a quarter) of the
 * bytes.  That takes 1.39 ms in one block a sample and 0.84 ms in four; two
 * warps or one a scheduler, so the latency of one warp's chain (loads, the
 * pass's rotations, stores, barrier) bounds it: of the cycles FP64 operations
 * issue in 29 % and conversions in 25 % (one block).
 */
#include <cuda_runtime.h>

#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define LOG_SUBSYS "engine"
#include "log.h"

#include "p2_kernels.cuh"
#include "p2_cluster.cuh"
#include "sub_core.h"

#define P2_OC_TPB 256
#define P2_OC_SMEM ((size_t)128 << 10) /* 2^14 complex floats, 2^13 doubles */

/* Place of index g: the bits of its bank (4 for 8-byte amplitudes, 3 for
 * 16-byte ones) take the XOR of the groups of as many bits above. */
template <typename ST> __device__ __forceinline__ uint32_t p2_oc_swz(uint32_t g)
{
	if (sizeof(ST) == 16)
		return p2_sub_swz(g);
	uint32_t f = g >> 4;
	f ^= f >> 8;
	f ^= f >> 4;
	return g ^ (f & 15u);
}

template <bool CL, typename ST>
__device__ __forceinline__ void p2_oc_ld(uint32_t a, double &re, double &im)
{
	if constexpr (sizeof(ST) == 16) {
		p2_res_ld<CL>(a, re, im);
	} else {
		float x, y;
		if constexpr (CL)
			asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];"
				: "=f"(x), "=f"(y) : "r"(a) : "memory");
		else
			asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];"
				: "=f"(x), "=f"(y) : "r"(a) : "memory");
		re = (double)x;
		im = (double)y;
	}
}

template <bool CL, typename ST>
__device__ __forceinline__ void p2_oc_st(uint32_t a, double re, double im)
{
	if constexpr (sizeof(ST) == 16) {
		p2_res_st<CL>(a, re, im);
	} else {
		const float x = __double2float_rn(re), y = __double2float_rn(im);
		if constexpr (CL)
			asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};"
				:: "r"(a), "f"(x), "f"(y) : "memory");
		else
			asm volatile("st.shared.v2.f32 [%0], {%1, %2};"
				:: "r"(a), "f"(x), "f"(y) : "memory");
	}
}

template <int M, typename ST, bool CL>
__device__ __forceinline__ void p2_oc_pass(uint32_t base, uint32_t kb,
	uint32_t rank, uint32_t nrank, uint32_t nqb, const struct phase2_pass &p,
	const struct phase2_rot_rec *srec)
{
	uint32_t sb[M];
#pragma unroll
	for (int k = 0; k < M; ++k)
		sb[k] = p2_oc_swz<ST>((uint32_t)p.basis[k]) *
			(uint32_t)sizeof(ST);
	const uint32_t neg = p.scale < 0 ? 0x80000000u : 0u;
	const uint32_t nrep = (1u << nqb) >> M, nrot = p.nrot;
	for (uint32_t t = rank * blockDim.x + threadIdx.x; t < nrep;
		t += nrank * blockDim.x) {
		const uint32_t x = p2_rep_t<M, uint32_t>(t, p);
		const uint32_t px = p2_oc_swz<ST>(x) * (uint32_t)sizeof(ST);
		double re[1 << M], im[1 << M];
#pragma unroll
		for (int u = 0; u < (1 << M); ++u) {
			uint32_t a = px;
#pragma unroll
			for (int k = 0; k < M; ++k)
				if (u >> k & 1)
					a ^= sb[k];
			p2_oc_ld<CL, ST>(p2_res_map<CL>(base, a, kb), re[u],
				im[u]);
		}
		for (uint32_t r = 0; r < nrot; ++r) {
			const uint32_t sm = srec[r].smask ^
				(0u - p2_parity(x & (uint32_t)srec[r].z));
			const uint32_t key =
				(uint32_t)srec[r].U << 1 | srec[r].odd;
			if constexpr (sizeof(ST) == 16)
				p2_apply<M>(key, re, im, srec[r].c, srec[r].s, sm,
					0u);
			else
				p2_apply_lift<M>(key, re, im, srec[r].c,
					srec[r].s, sm);
		}
		const uint32_t ps = p2_opaque(px);
#pragma unroll
		for (int u = 0; u < (1 << M); ++u) {
			uint32_t a = ps;
#pragma unroll
			for (int k = 0; k < M; ++k)
				if (u >> k & 1)
					a ^= sb[k];
			p2_oc_st<CL, ST>(p2_res_map<CL>(base, a, kb),
				p2_sgn(re[u], neg), p2_sgn(im[u], neg));
		}
	}
}

/* Copies of a pass header (9 words of 8 bytes) and of its records. */
__device__ __forceinline__ void p2_oc_header(struct phase2_pass *dst,
	const struct phase2_pass *src)
{
	static_assert(sizeof(struct phase2_pass) == 72, "pass header words");
	if (threadIdx.x < 9)
		asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(
				     (uint32_t)__cvta_generic_to_shared(dst) +
				     8 * threadIdx.x),
			"l"((const unsigned char *)src + 8 * threadIdx.x)
			: "memory");
}

__device__ __forceinline__ void p2_oc_records(struct phase2_rot_rec *dst,
	const struct phase2_rot_rec *recs, const struct phase2_pass &p)
{
	const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
	const unsigned char *const s = (const unsigned char *)(recs + p.rot_off);
	for (uint32_t k = threadIdx.x; k < 2 * p.nrot; k += blockDim.x)
		p2_cp16(d + 16 * k, s + 16 * k);
}

/* 2^lb blocks a sample, a cluster when more than one; a.passes and a.recs as
 * k_smp_plan leaves them.  The next pass's records and the headers after it
 * come in during a pass. */
template <typename ST, bool CL>
__global__ void __launch_bounds__(P2_OC_TPB, 1) k_onchip_smp(
	const struct p2_oc_samples a)
{
	extern __shared__ __align__(16) unsigned char p2_oc_dyn[];
	__shared__ __align__(16) struct phase2_rot_rec srec[2]
							   [P2_MAX_ROTS_PER_PASS];
	__shared__ __align__(16) struct phase2_pass hdr[4];
	ST *const st = (ST *)p2_oc_dyn;
	const uint64_t s = blockIdx.x >> a.lb;
	const uint32_t nrank = 1u << a.lb, rank = blockIdx.x & (nrank - 1);
	const uint32_t kc = a.nqb - a.lb, n = 1u << kc, tid = threadIdx.x;
	const uint32_t kb = kc + (sizeof(ST) == 16 ? 4 : 3);
	const uint32_t base = (uint32_t)__cvta_generic_to_shared(st);
	for (uint32_t i = tid; i < n; i += blockDim.x)
		p2_st(st, i, 0.0, 0.0);
	__syncthreads();
	/* in order: later writes win */
	for (uint32_t e = 0; tid == 0 && e < a.ndet; ++e) {
		const uint32_t at = p2_oc_swz<ST>((uint32_t)a.widx[e]);
		if (at >> kc == rank)
			p2_st(st, at & (n - 1), a.wval[2 * e],
				a.wval[2 * e + 1]);
	}
	for (uint32_t c = 0; c < a.C; ++c) {
		const struct phase2_pass *const ps =
			a.passes + s * a.T + (uint64_t)c * P2_QUEUE_FLUSH;
		const uint32_t np = a.npc[s * a.C + c];
		for (uint32_t j = 0; j < 3 && j < np; ++j)
			p2_oc_header(&hdr[j], ps + j);
		p2_cp_commit();
		p2_cp_wait<0>();
		__syncthreads();
		if (np)
			p2_oc_records(srec[0], a.recs, hdr[0]);
		p2_cp_commit();
		p2_cp_wait<0>();
		p2_res_barrier<CL>();
		for (uint32_t i = 0; i < np; ++i) {
			if (i + 1 < np)
				p2_oc_records(srec[(i + 1) & 1], a.recs,
					hdr[(i + 1) & 3]);
			if (i + 3 < np)
				p2_oc_header(&hdr[(i + 3) & 3], ps + i + 3);
			p2_cp_commit();
			const struct phase2_pass &p = hdr[i & 3];
			const struct phase2_rot_rec *const q = srec[i & 1];
			switch (p.span) {
			case 1:
				p2_oc_pass<1, ST, CL>(base, kb, rank, nrank,
					a.nqb, p, q);
				break;
			case 2:
				p2_oc_pass<2, ST, CL>(base, kb, rank, nrank,
					a.nqb, p, q);
				break;
			case 3:
				p2_oc_pass<3, ST, CL>(base, kb, rank, nrank,
					a.nqb, p, q);
				break;
			case 4:
				p2_oc_pass<4, ST, CL>(base, kb, rank, nrank,
					a.nqb, p, q);
				break;
			default:
				p2_oc_pass<5, ST, CL>(base, kb, rank, nrank,
					a.nqb, p, q);
				break;
			}
			p2_cp_wait<0>();
			p2_res_barrier<CL>();
		}
	}
	for (uint32_t e = tid; e < a.ndet; e += blockDim.x) {
		const uint32_t at = p2_oc_swz<ST>((uint32_t)a.widx[e]);
		double re, im;
		if (at >> kc != rank)
			continue;
		p2_ld(st, at & (n - 1), re, im);
		a.gout[s * a.ndet + e] = make_double2(re, im);
	}
	if (s == a.keep)
		for (uint32_t i = tid; i < n; i += blockDim.x)
			((ST *)a.state)[rank << kc | i] =
				st[p2_oc_swz<ST>(rank << kc | i) & (n - 1)];
}

/* 2^14 complex floats or 2^13 complex doubles in a block. */
static uint32_t onchip_least(const struct p2_dev *d)
{
	const uint32_t most = d->prec == PHASE2_PREC_FP64 ? 13 : 14;
	return d->nqb > most ? d->nqb - most : 0;
}

/*
 * log2 of a sample's blocks in a launch of g samples.  At 14 qubits one block
 * would take two cosets a thread: as many blocks, 8 at most, as leave each an
 * SM of its own.  Narrower samples hold a coset a thread in one block, and
 * more only send amplitudes between SMs (1000 draws, us a call, blocks a
 * sample 1 / 2 / 4 / 8.  FP32, 14 qubits: 8 samples 1762 / 1414 / 1229 /
 * 1170, 32 samples 1837 / 1466 / 1305 / 1299, 64 samples 1913 / 1541 / 1611
 * / 1641, 128 samples 2066 / 2702 / 2810 / 2926; 13 qubits: 8 samples 1104 /
 * 1101 / 1086 / 1077, 128 samples 1407 / 1539 / 1641 / 2480.  FP64, 14
 * qubits: 16 samples - / 1751 / 1625 / 1547, 64 samples - / 1907 / 2266 /
 * 2340).
 */
static uint32_t onchip_blocks(const struct p2_dev *d, uint64_t g)
{
	const uint32_t least = onchip_least(d);
	uint32_t lb = d->nqb == 14 ? 3 : 0;
	while (lb > least && (g << lb) > (uint64_t)d->sm_count)
		lb--;
	return lb;
}

template <auto F> static bool onchip_ready(const struct p2_dev *d)
{
	static uint64_t done;
	unsigned ok;
	if (!p2_done(&done, d->context, &ok)) {
		ok = cudaFuncSetAttribute(F,
			     cudaFuncAttributeMaxDynamicSharedMemorySize,
			     (int)P2_OC_SMEM) == cudaSuccess;
		cudaGetLastError();
		p2_set_done(&done, d->context, ok);
	}
	return ok;
}

/*
 * For launches of g samples.  FP32: from 4 samples at 12 qubits, 8 at 13, 1 at
 * 14 on; FP64: from 16 at 13, 8 at 14 (1000 draws, us a call, here /
 * k_resident_smp.  FP32, 12 qubits, 4 and 128 samples 893 / 1033, 1183 /
 * 1366; 13 qubits, 4, 8 and 128 samples 1095 / 1031, 1104 / 1113, 1407 /
 * 1818; 14 qubits, 1, 32 and 128 samples 1134 / 1263, 1305 / 2519, 2066 /
 * 4703.  FP64, 12 qubits, 4 and 128 samples 1000 / 997, 1330 / 1247; 13
 * qubits, 8, 16 and 128 samples 1196 / 1091, 1228 / 1310, 1514 / 1609; 14
 * qubits, 4, 8, 32 and 128 samples 1425 / 1227, 1435 / 1543, 1708 / 2434,
 * 3380 / 4541).
 */
bool p2_onchip_samples_ok(const struct p2_dev *d, int form, uint64_t g)
{
	if (form == PHASE2_FORM_LIFTED_F32)
		return false;
	if (d->prec == PHASE2_PREC_FP64)
		return ((d->nqb == 13 && g >= 16) ||
			       (d->nqb == 14 && g >= 8)) &&
			onchip_ready<k_onchip_smp<double2, true>>(d) &&
			onchip_ready<k_onchip_smp<double2, false>>(d);
	return ((d->nqb == 12 && g >= 4) || (d->nqb == 13 && g >= 8) ||
		       d->nqb == 14) &&
		onchip_ready<k_onchip_smp<float2, true>>(d) &&
		onchip_ready<k_onchip_smp<float2, false>>(d);
}

cudaError_t p2_onchip_samples(struct p2_dev *d, struct p2_oc_samples a,
	uint32_t g)
{
	cudaLaunchConfig_t cfg;
	cudaLaunchAttribute at[1];
	a.nqb = d->nqb;
	a.lb = onchip_blocks(d, g);
	a.state = d->state;
	const uint32_t kc = a.nqb - a.lb;
	memset(&cfg, 0, sizeof cfg);
	memset(at, 0, sizeof at);
	cfg.gridDim = dim3(g << a.lb);
	/* a coset of 32 a thread, as far as a block goes */
	cfg.blockDim = dim3(kc < 13 ? 1u << (kc - 5) : P2_OC_TPB);
	cfg.dynamicSmemBytes = d->elem << kc;
	cfg.stream = d->stream;
	if (a.lb) {
		at[0].id = cudaLaunchAttributeClusterDimension;
		at[0].val.clusterDim.x = 1u << a.lb;
		at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
		cfg.attrs = at;
		cfg.numAttrs = 1;
	}
	if (d->prec == PHASE2_PREC_FP64)
		return cudaLaunchKernelEx(&cfg,
			a.lb ? k_onchip_smp<double2, true>
			     : k_onchip_smp<double2, false>,
			a);
	return cudaLaunchKernelEx(&cfg,
		a.lb ? k_onchip_smp<float2, true> : k_onchip_smp<float2, false>,
		a);
}
