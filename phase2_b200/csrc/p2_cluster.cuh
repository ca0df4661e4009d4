/*
 * p2_cluster.cuh -- amplitudes in the shared memory of a block, or (CL) of
 * the blocks of a cluster: a register's share of 2^kb bytes in each, at the
 * same address of every block.
 */
#ifndef P2_CLUSTER_CUH
#define P2_CLUSTER_CUH

#include <stdint.h>

/* Shared address of a byte offset into the register. */
template <bool CL>
__device__ __forceinline__ uint32_t p2_res_map(uint32_t base, uint32_t off,
	uint32_t kb)
{
	uint32_t a = base + (off & ((1u << kb) - 1u));
	if constexpr (CL)
		asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a)
			: "r"(a), "r"(off >> kb));
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

#endif /* P2_CLUSTER_CUH */
