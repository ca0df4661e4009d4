/*
 * onchip.cu -- many samples of registers of 12 to 14 qubits (FP64: 13): a
 * block a sample, whole passes on the state in shared memory.
 *
 * k_resident_smp moves every amplitude through registers twice or three
 * times a pass, as a complex double, and at 14 qubits half of them through
 * another block's shared memory: with tens of samples that traffic bounds
 * it (32 FP32 samples of 1000 draws, 14 qubits: 1.9 ms).  Here a block holds
 * the register as it is stored, and a thread takes a coset of 32 amplitudes
 * through a whole pass, as the pass kernels do: an eighth (FP64: a quarter)
 * of the bytes, bound by the FP64 operations (1.43 ms).  A single sample
 * takes longer this way (one SM's FP64 units).
 */
#include <cuda_runtime.h>

#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define LOG_SUBSYS "engine"
#include "log.h"

#include "p2_kernels.cuh"
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

template <int M, typename ST>
__device__ __forceinline__ void p2_oc_pass(ST *st, uint32_t nqb,
	const struct phase2_pass &p, const struct phase2_rot_rec *srec)
{
	uint32_t sb[M];
#pragma unroll
	for (int k = 0; k < M; ++k)
		sb[k] = p2_oc_swz<ST>((uint32_t)p.basis[k]);
	const uint32_t neg = p.scale < 0 ? 0x80000000u : 0u;
	const uint32_t nrep = (1u << nqb) >> M, nrot = p.nrot;
	for (uint32_t t = threadIdx.x; t < nrep; t += P2_OC_TPB) {
		const uint32_t x = p2_rep_t<M, uint32_t>(t, p);
		const uint32_t px = p2_oc_swz<ST>(x);
		double re[1 << M], im[1 << M];
#pragma unroll
		for (int u = 0; u < (1 << M); ++u) {
			uint32_t a = px;
#pragma unroll
			for (int k = 0; k < M; ++k)
				if (u >> k & 1)
					a ^= sb[k];
			p2_ld(st, a, re[u], im[u]);
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
			p2_st(st, a, p2_sgn(re[u], neg), p2_sgn(im[u], neg));
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
	for (uint32_t k = threadIdx.x; k < 2 * p.nrot; k += P2_OC_TPB)
		p2_cp16(d + 16 * k, s + 16 * k);
}

/* One block a sample; a.passes and a.recs as k_smp_plan leaves them.  The
 * next pass's records and the headers after it come in during a pass. */
template <typename ST>
__global__ void __launch_bounds__(P2_OC_TPB, 1) k_onchip_smp(
	const struct p2_oc_samples a)
{
	extern __shared__ __align__(16) unsigned char p2_oc_dyn[];
	__shared__ __align__(16) struct phase2_rot_rec srec[2]
							   [P2_MAX_ROTS_PER_PASS];
	__shared__ __align__(16) struct phase2_pass hdr[4];
	ST *const st = (ST *)p2_oc_dyn;
	const uint64_t s = blockIdx.x;
	const uint32_t n = 1u << a.nqb, tid = threadIdx.x;
	for (uint32_t i = tid; i < n; i += P2_OC_TPB)
		p2_st(st, i, 0.0, 0.0);
	__syncthreads();
	/* in order: later writes win */
	for (uint32_t e = 0; tid == 0 && e < a.ndet; ++e)
		p2_st(st, p2_oc_swz<ST>((uint32_t)a.widx[e]), a.wval[2 * e],
			a.wval[2 * e + 1]);
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
		__syncthreads();
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
				p2_oc_pass<1, ST>(st, a.nqb, p, q);
				break;
			case 2:
				p2_oc_pass<2, ST>(st, a.nqb, p, q);
				break;
			case 3:
				p2_oc_pass<3, ST>(st, a.nqb, p, q);
				break;
			case 4:
				p2_oc_pass<4, ST>(st, a.nqb, p, q);
				break;
			default:
				p2_oc_pass<5, ST>(st, a.nqb, p, q);
				break;
			}
			p2_cp_wait<0>();
			__syncthreads();
		}
	}
	for (uint32_t e = tid; e < a.ndet; e += P2_OC_TPB) {
		double re, im;
		p2_ld(st, p2_oc_swz<ST>((uint32_t)a.widx[e]), re, im);
		a.gout[s * a.ndet + e] = make_double2(re, im);
	}
	if (s == a.keep)
		for (uint32_t i = tid; i < n; i += P2_OC_TPB)
			((ST *)a.state)[i] = st[p2_oc_swz<ST>(i)];
}

template <typename ST> static bool onchip_ready(void)
{
	static unsigned ready; /* 1 yes, 2 no */
	unsigned r = __atomic_load_n(&ready, __ATOMIC_ACQUIRE);
	if (!r) {
		r = cudaFuncSetAttribute(k_onchip_smp<ST>,
			    cudaFuncAttributeMaxDynamicSharedMemorySize,
			    (int)P2_OC_SMEM) == cudaSuccess
			? 1
			: 2;
		cudaGetLastError();
		__atomic_store_n(&ready, r, __ATOMIC_RELEASE);
	}
	return r == 1;
}

/*
 * FP32: from 4 samples at 12 qubits, 8 at 13, 12 at 14 on; FP64: from 16 at
 * 13 (1000 draws, us a call, here / k_resident_smp.  FP32, 12 qubits, 4 and
 * 128 samples 908 / 1009, 1174 / 1370; 13 qubits, 4, 8 and 128 samples 1108
 * / 1007, 1125 / 1125, 1400 / 1799; 14 qubits, 8, 16 and 128 samples 1787 /
 * 1627, 1813 / 2121, 2072 / 4686.  FP64, 12 qubits, 4 and 128 samples 1049
 * / 973, 1311 / 1239; 13 qubits, 8, 16 and 128 samples 1216 / 1091, 1226 /
 * 1308, 1499 / 1600).
 */
bool p2_onchip_samples_ok(const struct p2_dev *d, int form, uint64_t samples)
{
	if (form == PHASE2_FORM_LIFTED_F32)
		return false;
	if (d->prec == PHASE2_PREC_FP64)
		return d->nqb == 13 && samples >= 16 && onchip_ready<double2>();
	return d->nqb >= 12 && d->nqb <= 14 && samples >= 4 * (d->nqb - 11) &&
		onchip_ready<float2>();
}

cudaError_t p2_onchip_samples(struct p2_dev *d, struct p2_oc_samples a,
	uint32_t g)
{
	const size_t smem = d->elem << d->nqb;
	a.nqb = d->nqb;
	a.state = d->state;
	if (d->prec == PHASE2_PREC_FP64)
		k_onchip_smp<double2><<<g, P2_OC_TPB, smem, d->stream>>>(a);
	else
		k_onchip_smp<float2><<<g, P2_OC_TPB, smem, d->stream>>>(a);
	return cudaGetLastError();
}
