/*
 * p2_sub.cuh -- device code shared by the kernels that run sub-passes
 * (sub_core.h): complex doubles in shared memory (of the block, or CL of
 * any block of the cluster), and a rotation on a coset of 8 slots.
 */
#ifndef P2_SUB_CUH
#define P2_SUB_CUH

/* all four pairs of a coset step by step: few warps share a scheduler in
 * these kernels, so independent FP64 operations have to come from each */
#define P2_ROT_GROUP 4
#define P2_LIFT_GROUP 4
#include "p2_kernels.cuh"
#include "sub_core.h"

#define P2_RES_SLOTS (1 << P2_SUB_SPAN)

/* ---- shared memory of the cluster --------------------------------------- */

template <bool CL>
__device__ __forceinline__ uint32_t p2_res_addr(uint32_t base, uint32_t pos,
	uint32_t kc)
{
	uint32_t a = base + ((pos & ((1u << kc) - 1u)) << 4);
	if constexpr (CL) {
		const uint32_t rank = pos >> kc;
		asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a)
			: "r"(a), "r"(rank));
	}
	return a;
}

template <bool CL>
__device__ __forceinline__ void p2_res_ld(uint32_t a, double &re, double &im)
{
	if constexpr (CL)
		asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];"
			: "=d"(re), "=d"(im) : "r"(a) : "memory");
	else
		asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
			: "=d"(re), "=d"(im) : "r"(a) : "memory");
}

template <bool CL>
__device__ __forceinline__ void p2_res_st(uint32_t a, double re, double im)
{
	if constexpr (CL)
		asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};"
			:: "r"(a), "d"(re), "d"(im) : "memory");
	else
		asm volatile("st.shared.v2.f64 [%0], {%1, %2};"
			:: "r"(a), "d"(re), "d"(im) : "memory");
}

template <bool CL> __device__ __forceinline__ void p2_res_barrier()
{
	if constexpr (CL)
		asm volatile("barrier.cluster.arrive.release.aligned;\n"
			     "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
	else
		__syncthreads();
}

/* The rotation (key) on a coset of 8 slots: the exact FP64 update, or the
 * lifted one in FP64. */
template <bool X, int K>
__device__ __forceinline__ void p2_sub_rot(double (&re)[P2_RES_SLOTS],
	double (&im)[P2_RES_SLOTS], double c, double s, uint32_t sm)
{
	if constexpr (X)
		p2_rot_lift<P2_SUB_SPAN, (K >> 1), (K & 1)>(re, im, c, s, sm);
	else
		p2_rot<P2_SUB_SPAN, (K >> 1), (K & 1)>(re, im, c, s, sm, 0u);
}

#define P2_CASE_S(K)                                                           \
	case K:                                                                \
		p2_sub_rot<X, K>(re, im, q.c, q.s, sm);                        \
		break;

template <bool X>
__device__ __forceinline__ void p2_sub_apply(const struct p2_sub_rec &q,
	double (&re)[P2_RES_SLOTS], double (&im)[P2_RES_SLOTS], uint32_t sm)
{
	switch (q.key) {
		P2_CASE_S(0) P2_CASE_S(1) P2_CASE_S(2) P2_CASE_S(3)
		P2_CASE_S(4) P2_CASE_S(5) P2_CASE_S(6) P2_CASE_S(7)
		P2_CASE_S(8) P2_CASE_S(9) P2_CASE_S(10) P2_CASE_S(11)
		P2_CASE_S(12) P2_CASE_S(13) P2_CASE_S(14) P2_CASE_S(15)
	default:
		break;
	}
}
#undef P2_CASE_S

#endif /* P2_SUB_CUH */
