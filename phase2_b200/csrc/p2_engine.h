/*
 * p2_engine.h -- internals shared by the CUDA sources of the engine:
 * engine.cu (registers, pass kernels, state I/O, reductions), batch.cu
 * (the persistent kernel), sampling.cu (device sampling) and sweep.cu
 * (sweeps).  Include after log.h.
 */
#ifndef P2_ENGINE_H
#define P2_ENGINE_H

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "phase2_b200.h"

#include "p2_internal.h"

#define P2_TPB 128

/* Registers below this many qubits run mixed-form passes on the FP64-
 * arithmetic kernels: a spread state of n qubits has components of
 * standard deviation 2^-(n+1)/2, which reach P2_HEAVY_MIN often below 24
 * qubits (at 22, a quarter of the cosets), and a heavy coset costs its
 * warp a serial FP64 run; at 24 the threshold is 5.7 deviations away. */
#define P2_MIXED_MIN_QB 24
#define P2_RED_TPB 256

/* Replay of repeated flushes: registers up to this width keep a small LRU
 * of captured pass sequences (launch overhead matters only there). */
#define P2_GRAPH_SLOTS 8
#define P2_GRAPH_MAX_QB 24

struct p2_graph {
	uint64_t hash;
	size_t npass, nrec;
	struct phase2_pass *passes;    /* host copies: exact comparison */
	struct phase2_rot_rec *recs;
	struct phase2_rot_rec *d_recs; /* records read by the graph */
	cudaGraphExec_t exec;
	size_t nlaunch; /* kernel launches in the graph */
	/* resident registers (resident.cu): d_recs holds the flush's repacked
	 * records and its nsub sub-passes, d_cap bytes from the pool */
	size_t d_cap;
	uint32_t nsub;
	struct p2_split_pass *split; /* per pass (split.cu), or NULL */
	struct p2_tile *tiles;       /* ntile runs (tile.cu), or NULL */
	uint32_t ntile;
	uint64_t plan_id; /* the caller's number of this plan (0: none) */
	int status;     /* the graph holds kernels that write d_status */
	uint64_t used;
};

struct p2_dev {
	uint32_t nqb;
	int prec;
	size_t elem;
	uint64_t namp;
	void *state;
	cudaStream_t stream;
	int sm_count;
	int tiles;        /* passes may be regrouped (p2d_set_tiles) */
	uint64_t last_plan; /* number of the last flush's plan */
	int device;       /* of the shell (engine.cu) */
	uint64_t context;

	struct phase2_rot_rec *d_recs;
	size_t d_recs_cap;
	struct phase2_rot_rec *h_recs[2];
	size_t h_recs_cap[2];
	cudaEvent_t h_ev[2];
	int h_ev_live[2];
	int ring;

	/* error word of kernels with bounded waits (lift_bulk.cu): set on
	 * the device, read at the next synchronisation (p2_status_check) */
	unsigned int *d_status;
	unsigned int *h_status;
	int status_pending;

	uint64_t *d_idx;
	double *d_val;
	uint64_t *h_idx;
	double *h_val;
	size_t io_cap;

	double *d_part;
	size_t part_cap;

	unsigned char *d_cm; /* coefficient-matrix tables */
	size_t cm_cap;

	int timing;
	cudaEvent_t t0, t1;

	uint64_t rotations, passes, launches, timed_passes;
	uint64_t sweeps, timed_sweeps; /* state round trips (pass or sweep
					* kernels) */
	uint64_t h2d_bytes, d2h_bytes;
	double pass_ms;

	struct p2_graph graphs[P2_GRAPH_SLOTS];
	uint64_t graph_clock;
	uint64_t graph_replays;
	int graphs_on;
};

#define CUDA_OK(call, what)                                                    \
	do {                                                                   \
		cudaError_t e_ = (call);                                       \
		if (e_ != cudaSuccess) {                                       \
			log_error("%s: %s", (what), cudaGetErrorString(e_));  \
			cudaGetLastError(); /* reported here only */           \
			return -1;                                             \
		}                                                              \
	} while (0)


static inline unsigned grid_for(const struct p2_dev *d, uint64_t work, unsigned tpb,
	unsigned per_sm)
{
	uint64_t b = (work + tpb - 1) / tpb;
	const uint64_t cap = (uint64_t)d->sm_count * per_sm;
	if (b > cap)
		b = cap;
	return b ? (unsigned)b : 1u;
}

#ifdef __CUDACC__
/*
 * A pass kernel's launch: it may start before the previous kernel of the
 * stream has ended (programmatic dependent launch), stages its records, and
 * waits (p2_grid_wait) before it touches the state.  A pass of a register
 * that fits the L2 cache takes 3-10 us, of which the launch gap was 2-3.
 * Records are uploaded by copies, which such a launch still waits for.
 */
template <typename... P, typename... A>
static cudaError_t p2_launch(void (*fn)(P...), unsigned grid, unsigned tpb,
	size_t smem, cudaStream_t stream, A... args)
{
	cudaLaunchConfig_t cfg;
	cudaLaunchAttribute at[1];
	memset(&cfg, 0, sizeof cfg);
	memset(at, 0, sizeof at);
	cfg.gridDim = dim3(grid);
	cfg.blockDim = dim3(tpb);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = stream;
	at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at[0].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = at;
	cfg.numAttrs = 1;
	return cudaLaunchKernelEx(&cfg, fn, P(args)...);
}

/* Wait for the previous kernel's end and its stores. */
__device__ __forceinline__ void p2_grid_wait()
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
}
#endif

/*
 * What is set on a kernel (shared memory, cluster size) belongs to the
 * device's context, and a device reset makes a new one: a "done" word holds
 * the context's number (p2_dev.context) above a byte of the answer, so one
 * of another context counts as unset.
 */
static inline bool p2_done(const uint64_t *word, uint64_t context,
	unsigned *answer)
{
	const uint64_t w = __atomic_load_n(word, __ATOMIC_ACQUIRE);
	*answer = (unsigned)(w & 0x7f);
	return (w & 0x80) && w >> 8 == context;
}

static inline void p2_set_done(uint64_t *word, uint64_t context,
	unsigned answer)
{
	__atomic_store_n(word, context << 8 | 0x80 | answer, __ATOMIC_RELEASE);
}

/* ---- cross-file entry points -------------------------------------------- */

/* engine.cu: transient device buffers of one call (a batch program, the
 * scratch of device sampling), stream-ordered from the device's default
 * memory pool, which keeps up to a sixteenth of the device's memory for the next call
 * instead of unmapping it at every synchronisation (a cudaFree of such a
 * buffer could take hundreds of milliseconds).  The pool is configured on
 * the first call, for the current device (one device per process). */
cudaError_t p2_scratch_alloc(void **p, size_t bytes, cudaStream_t stream);
void p2_scratch_free(void *p, cudaStream_t stream);

struct p2_binst;
struct p2_bctl;

/* Idle scheduling rounds (each sleeps ~1 us, and counting restarts
 * whenever any ticket moves) before a block of the persistent kernel gives
 * up. */
#define P2_BATCH_IDLE_LIMIT 2000000u

/* batch.cu: the persistent kernel for FP32 registers (FP32 arithmetic,
 * P2_BK_F32, or FP64 arithmetic, P2_BK_F32X) or FP64 registers
 * (P2_BK_F64): the instance for a precision and FP32 form, its function
 * (occupancy queries) and its launch.  status points to 16
 * zeroed bytes: status[0] is raised when a wait gives up, status[2..3]
 * receive the complement of the launch's start time (global timer).  cum
 * (device, one double per program, or NULL for round robin): running
 * totals of the programs' work, which spread the warps' home programs. */
enum { P2_BK_F32 = 0, P2_BK_F32X = 1, P2_BK_F64 = 2 };
int p2_batch_kind(int prec, int form);
const void *p2_batch_kernel(int kind);
void p2_batch_launch(int kind, unsigned grid, cudaStream_t stream,
	const struct p2_binst *inst, uint32_t ninst, const struct p2_op *ops,
	const struct phase2_pass *passes, const struct phase2_rot_rec *recs,
	const uint64_t *widx, const double *wval, const uint64_t *gidx,
	double2 *gout, struct p2_bctl *ctl, unsigned int *status,
	const double *cum);

/* engine.cu: pinned staging for `n` records of 32 bytes (double buffered;
 * NULL on failure), and the copy of its first `bytes` to device memory. */
struct phase2_rot_rec *p2_stage_reserve(struct p2_dev *d, size_t n);
int p2_stage_upload(struct p2_dev *d, void *dst, size_t bytes);

/* engine.cu: release a plan slot (graph or resident plan) and clear it. */
void p2_graph_drop(struct p2_dev *d, struct p2_graph *g);

/* resident.cu: whether a register's flush of this form runs as one launch
 * on the register held in shared memory, and that launch (the caller counts
 * it). */
bool p2_resident_ok(const struct p2_dev *d, int form);
int p2_resident_run(struct p2_dev *d, const struct p2_graph *g);

/* resident.cu: a register's plan slot for a flush, its sub-passes on the
 * device (see there); NULL where there is no room for them.  plan_id:
 * nonzero and the same for flushes with the same passes and records. */
enum p2_plan_kind { P2_PLAN_RESIDENT, P2_PLAN_SPLIT, P2_PLAN_TILE };
struct p2_graph *p2_sub_plan(struct p2_dev *d,
	const struct phase2_pass *passes, size_t npass,
	const struct phase2_rot_rec *recs, size_t nrec, uint64_t plan_id,
	enum p2_plan_kind kind, bool *hit);

/* split.cu: registers of middle width, a coset shared by four threads:
 * whether a register's flush of this form runs there, and its launches, as
 * p2_resident_run. */
bool p2_split_ok(const struct p2_dev *d, int form);
int p2_split_run(struct p2_dev *d, const struct p2_graph *g);

/*
 * resident.cu: a round of samples run on chip, one cluster each: sample s's
 * sub-passes of chunk c are subs[s * T + c * P2_QUEUE_FLUSH ..], nsub[s * C +
 * c] of them, records recs[s * T ..]; it starts from the determinants
 * (widx, wval) and leaves their amplitudes in gout[s * ndet ..]; sample
 * `keep` stores its state in the register.  nqb, lb and state are filled by
 * the launch.
 */
struct p2_sub;
struct p2_sub_rec;
struct p2_res_samples {
	uint32_t nqb, lb, ndet, C;
	uint64_t T, keep;
	const struct p2_sub *subs;
	const uint32_t *nsub;
	const struct p2_sub_rec *recs;
	const uint64_t *widx;
	const double *wval;
	double2 *gout;
	void *state;
};
bool p2_resident_samples_ok(const struct p2_dev *d, int form);
cudaError_t p2_resident_samples(struct p2_dev *d, struct p2_res_samples a,
	uint32_t g);

/* onchip.cu: the same for launches of g samples, 2^lb blocks each, by whole
 * passes: sample s's passes of chunk c are passes[s * T + c *
 * P2_QUEUE_FLUSH ..], npc[s * C + c] of them, their rot_off into recs. */
struct p2_oc_samples {
	uint32_t nqb, lb, ndet, C;
	uint64_t T, keep;
	const struct phase2_pass *passes;
	const uint32_t *npc;
	const struct phase2_rot_rec *recs;
	const uint64_t *widx;
	const double *wval;
	double2 *gout;
	void *state;
};
bool p2_onchip_samples_ok(const struct p2_dev *d, int form, uint64_t g);
cudaError_t p2_onchip_samples(struct p2_dev *d, struct p2_oc_samples a,
	uint32_t g);

/*
 * resident.cu: a batch whose registers all fit on chip.  A program's ops: a
 * run of sub-passes subs[a .. a + b) (records recs), or P2_OP_ZERO / WRITE /
 * GATHER with a, b as in struct p2_op.  Whether a register of this form can
 * be in such a batch, and the launch of g programs on d's stream (nqb: the
 * widest register; even: as many programs of the largest one's work as the
 * batch's work makes; ctl[i].end_ns and the complement of the start time in
 * *start as k_batch leaves them).
 */
#define P2_RES_RUN 0x100
struct p2_res_op {
	uint32_t kind, a, b;
};
struct p2_res_prog {
	void *state;
	const struct p2_res_op *ops;
	const struct p2_sub *subs;
	const struct p2_sub_rec *recs;
	uint32_t nqb, nops;
};
bool p2_resident_prog_ok(const struct p2_dev *d, int form);
cudaError_t p2_resident_progs(const struct p2_dev *d, uint32_t nqb, uint32_t g,
	uint32_t even, const struct p2_res_prog *progs, const uint64_t *widx,
	const double *wval, const uint64_t *gidx, double2 *gout,
	struct p2_bctl *ctl, unsigned long long *start);

/* tile.cu: FP64 registers beyond the caches: whether a flush's rotations run
 * regrouped into tile runs, and their launches, as p2_resident_run. */
bool p2_tile_ok(const struct p2_dev *d, int form,
	const struct phase2_pass *passes, size_t npass,
	const struct phase2_rot_rec *recs, size_t nrec);
int p2_tile_run(struct p2_dev *d, const struct p2_graph *g);

/* lift_bulk.cu: one FP32 pass of the FP64-arithmetic form on a kernel
 * whose next cosets are staged in shared memory, by bulk copies (variant
 * 1) or cp.async (variant 2); returns 1 when launched, 0 when the pass
 * does not qualify (the caller runs the direct kernel), -1 on error.
 * per_sm_cap: resident blocks per SM at most (0: occupancy). */
extern "C" int p2_lift_staged_launch(struct p2_dev *d,
	const struct phase2_pass *p, const struct phase2_rot_rec *recs,
	int variant, unsigned per_sm_cap);

/* engine.cu: read the error word of kernels with bounded waits if one ran
 * since the last check (synchronises the register's stream); -1 and a
 * logged error when a wait gave up. */
int p2_status_check(struct p2_dev *d);

/* slab.cu: 0 if [p, p + bytes) is device memory of the current device
 * inside one allocation; -1 (logged, prefixed by `what`) otherwise, also
 * when the allocation cannot be looked up.  Allocates nothing. */
int p2_check_device_range(const void *p, size_t bytes, const char *what);

/* sweep.cu: whether planned sweeps run as one kernel each on this
 * register, and the launch of the sweep starting at passes[i] (returns the
 * passes it covers, 1 when passes[i] should run alone, -1 on error). */
bool p2_sweeps_on(const struct p2_dev *d);
long p2_sweep_launch(struct p2_dev *d, const struct phase2_pass *passes,
	size_t npass, size_t i, const struct phase2_rot_rec *d_recs);

#endif /* P2_ENGINE_H */
