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
#include "p2_cluster.cuh"
#include "sub_core.h"

#define P2_RES_SLOTS (1 << P2_SUB_SPAN)

/* ---- slots ---------------------------------------------------------------- */

template <bool CL>
__device__ __forceinline__ uint32_t p2_res_addr(uint32_t base, uint32_t pos,
	uint32_t kc)
{
	return p2_res_map<CL>(base, pos << 4, kc + 4);
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
