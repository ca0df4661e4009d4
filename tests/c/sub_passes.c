/*
 * Checks csrc/sub_core.h on the host: the sub-passes a plan is cut into
 * give the amplitudes of its passes bit for bit (the lifted update, whose
 * pairs are ordered), enumerate every amplitude once, cover every rotation
 * in order, and stay inside their staging limits; and the same for the
 * sub-passes on tiles of one pass (p2_split_build).  Prints "ok" and returns
 * 0, or names the first case that fails.
 */
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include "sub_core.h"

/* The rotation (U, odd, t, s) on the 2^m amplitudes a[idx[...]]: three
 * shears a pair, the slot with a zero at the top bit of U first. */
static void rotate(double *a, const uint32_t *idx, int m, uint32_t U, int odd,
	double t, double s, uint32_t sm)
{
	for (uint32_t u = 0; u < (1u << m); u++) {
		const double g = (sm >> u & 1) ? -1.0 : 1.0;
		const double st = g * t, ss = g * s;
		double *yu = a + 2 * idx[u];
		if (U == 0) {
			yu[0] = fma(-st, yu[1], yu[0]);
			yu[1] = fma(ss, yu[0], yu[1]);
			yu[0] = fma(-st, yu[1], yu[0]);
			continue;
		}
		if (u >> top_bit(U) & 1)
			continue;
		double *yw = a + 2 * idx[u ^ U];
		for (int k = 0; k < 3; k++) {
			double *to = k == 1 ? yw : yu, *from = k == 1 ? yu : yw;
			const double f = k == 1 ? ss : st;
			if (odd) {
				to[0] = fma(-f, from[1], to[0]);
				to[1] = fma(f, from[0], to[1]);
			} else {
				to[0] = fma(k == 1 ? -f : f, from[0], to[0]);
				to[1] = fma(k == 1 ? -f : f, from[1], to[1]);
			}
		}
	}
}

static uint32_t insert_zeros(uint32_t x, const uint32_t *piv, int n)
{
	for (int k = 0; k < n; k++)
		x = ((x >> piv[k]) << (piv[k] + 1)) | (x & ((1u << piv[k]) - 1));
	return x;
}

static void run_pass(double *a, uint32_t n, const struct phase2_pass *p,
	const struct phase2_rot_rec *recs)
{
	uint32_t piv[PHASE2_MAX_SPAN], idx[32];
	for (uint32_t k = 0; k < p->span; k++)
		piv[k] = p->piv[k];
	for (uint32_t t = 0; t < (1u << n) >> p->span; t++) {
		const uint32_t x = insert_zeros(t, piv, (int)p->span);
		for (uint32_t u = 0; u < (1u << p->span); u++) {
			idx[u] = x;
			for (uint32_t k = 0; k < p->span; k++)
				if (u >> k & 1)
					idx[u] ^= (uint32_t)p->basis[k];
		}
		for (uint32_t r = 0; r < p->nrot; r++) {
			const struct phase2_rot_rec *q = &recs[r];
			rotate(a, idx, (int)p->span, q->U, q->odd, q->c, q->s,
				q->smask ^ (0u - (uint32_t)parity64(x & q->z)));
		}
	}
	for (size_t i = 0; i < (size_t)2 << n; i++)
		a[i] = (float)(p->scale < 0 ? -a[i] : a[i]);
}

static const char *run_sub(double *a, uint32_t n, const struct p2_sub *h,
	const struct p2_sub_rec *recs, char *seen)
{
	memset(seen, 0, (size_t)1 << n);
	if (h->nrot == 0 || h->nrot > P2_SUB_ROTS)
		return "rotation count";
	for (uint32_t t = 0; t < (1u << n) >> P2_SUB_SPAN; t++) {
		uint32_t x = insert_zeros(t, h->piv, P2_SUB_SPAN), idx[8];
		const uint32_t x0 = x;
		for (int k = 0; k < P2_SUB_SPAN; k++)
			if (parity64(x0 & h->orient[k]))
				x ^= h->slot[k];
		for (uint32_t u = 0; u < 8; u++) {
			uint32_t g = x, pos = p2_sub_swz(x);
			for (int k = 0; k < P2_SUB_SPAN; k++)
				if (u >> k & 1) {
					g ^= h->slot[k];
					pos ^= h->pslot[k];
				}
			if (g >> n || seen[g]++ || pos != p2_sub_swz(g) || pos >> n)
				return "enumeration";
			idx[u] = g;
		}
		for (uint32_t r = 0; r < h->nrot; r++) {
			const struct p2_sub_rec *q = &recs[h->rot_off + r];
			if (q->key > 15)
				return "key";
			rotate(a, idx, P2_SUB_SPAN, q->key >> 1, q->key & 1, q->c,
				q->s, q->sm ^ (0u - (uint32_t)parity64(x & q->z)));
		}
	}
	if (h->flags & P2_SUB_LAST)
		for (size_t i = 0; i < (size_t)2 << n; i++)
			a[i] = (float)(h->flags & P2_SUB_NEG ? -a[i] : a[i]);
	return NULL;
}

/* One pass through its tiles, as k_pass_split walks them. */
static const char *run_split(double *a, uint32_t n,
	const struct p2_split_pass *sp, const struct p2_sub *subs,
	const struct p2_sub_rec *recs, char *seen)
{
	const struct phase2_pass *p = &sp->pass;
	const uint32_t M = p->span, LB = P2_SPLIT_BITS - M, UL = 7 - LB;
	uint32_t piv[PHASE2_MAX_SPAN], at[1 << P2_SPLIT_BITS];
	if (M < 3 || M > 5)
		return "split span";
	for (uint32_t k = 0; k < M; k++)
		piv[k] = p->piv[k];
	memset(seen, 0, (size_t)1 << n);
	for (uint32_t b = 0; b < (1u << n) >> P2_SPLIT_BITS; b++) {
		const uint32_t xb = insert_zeros(b << LB, piv, (int)M);
		for (uint32_t t = 0; t < 128; t++)
			for (uint32_t i = 0; i < 8; i++) {
				uint32_t g = insert_zeros((b << LB) +
						(t & ((1u << LB) - 1)),
					piv, (int)M);
				for (uint32_t k = 0; k < UL; k++)
					if (t >> (LB + k) & 1)
						g ^= (uint32_t)p->basis[k];
				for (uint32_t k = 0; k < 3; k++)
					if (i >> k & 1)
						g ^= (uint32_t)p->basis[UL + k];
				if (g >> n || seen[g]++)
					return "split enumeration";
				at[t + 128 * i] = g;
			}
		for (uint32_t i = 0; i < sp->nsub; i++) {
			const struct p2_sub *h = &subs[sp->sub_off + i];
			for (uint32_t t = 0; t < 128; t++) {
				uint32_t y = insert_zeros(t, h->piv, P2_SUB_SPAN);
				uint32_t idx[8];
				const uint32_t y0 = y;
				for (int k = 0; k < P2_SUB_SPAN; k++)
					if (parity64(y0 & h->orient[k]))
						y ^= h->slot[k];
				for (uint32_t u = 0; u < 8; u++) {
					uint32_t g = y;
					for (int k = 0; k < P2_SUB_SPAN; k++)
						if (u >> k & 1)
							g ^= h->slot[k];
					if (g >> P2_SPLIT_BITS)
						return "split slot";
					idx[u] = at[g];
				}
				for (uint32_t r = 0; r < h->nrot; r++) {
					const struct p2_sub_rec *q =
						&recs[h->rot_off + r];
					const int s = parity64(y & q->z) ^
						parity64(xb & q->pad1);
					rotate(a, idx, P2_SUB_SPAN, q->key >> 1,
						q->key & 1, q->c, q->s,
						q->sm ^ (0u - (uint32_t)s));
				}
			}
		}
	}
	for (size_t i = 0; i < (size_t)2 << n; i++)
		a[i] = (float)(p->scale < 0 ? -a[i] : a[i]);
	return NULL;
}

int main(void)
{
	enum { R = 400, N = 1 << 14 };
	static struct phase2_rot_in q[R];
	static struct phase2_pass ps[R];
	static struct phase2_rot_rec rc[R];
	static struct p2_sub ss[R];
	static struct p2_sub_rec sr[R];
	static double a[2 * N], b[2 * N], c[2 * N];
	static char seen[N];
	srand48(1);
	for (int trial = 0; trial < 300; trial++) {
		const uint32_t n = 3 + (uint32_t)trial % 12;
		const size_t nr = 1 + (size_t)lrand48() % R;
		const uint64_t m = (UINT64_C(1) << n) - 1;
		for (size_t i = 0; i < nr; i++) {
			/* dense strings, a few flips, or long equal groups */
			uint64_t f = (uint64_t)lrand48() & m;
			if (trial % 3 == 1)
				f = (UINT64_C(1) << lrand48() % n) ^
					(UINT64_C(1) << lrand48() % n);
			else if (trial % 3 == 2 && i % 90)
				f = q[i - 1].flip;
			q[i].flip = f;
			q[i].phase = (uint64_t)lrand48() & m;
			q[i].phi = drand48() * 8 - 4;
		}
		const int form = trial & 1 ? PHASE2_FORM_LIFTED
					   : PHASE2_FORM_LIFTED_MIXED;
		const long np = p2_plan_core(n, q, NULL, nr,
			1 + (int)(lrand48() % 5),
			lrand48() % 4 ? 0 : 1 + (int)(lrand48() % 9),
			P2_DEFAULT_PAD_SPAN, form, 0, 0, ps, rc);
		for (size_t i = 0; i < (size_t)2 << n; i++)
			a[i] = b[i] = c[i] = (float)(drand48() - 0.5);
		uint32_t ns = 0, covered = 0;
		for (long p = 0; p < np; p++) {
			run_pass(a, n, &ps[p], rc + ps[p].rot_off);
			ns += p2_sub_split(&ps[p], rc + ps[p].rot_off, n,
				ps[p].rot_off, ss + ns, sr + ps[p].rot_off);
		}
		const char *bad = np < 0 ? "plan" : NULL;
		for (uint32_t i = 0; i < ns && !bad; i++) {
			if (ss[i].rot_off != covered)
				bad = "order";
			else
				bad = run_sub(b, n, &ss[i], sr, seen);
			covered += ss[i].nrot;
		}
		if (!bad && covered != nr)
			bad = "coverage";
		if (!bad && memcmp(a, b, (size_t)16 << n))
			bad = "bits";
		ns = 0;
		for (long p = 0; p < np && !bad && n >= P2_SPLIT_BITS; p++) {
			struct p2_split_pass sp;
			p2_split_build(n, &ps[p], rc, &sp, ns, ss + ns, sr);
			ns += sp.nsub;
			bad = run_split(c, n, &sp, ss, sr, seen);
		}
		if (!bad && n >= P2_SPLIT_BITS &&
			memcmp(a, c, (size_t)16 << n))
			bad = "split bits";
		if (bad) {
			printf("trial %d, %u qubits: %s\n", trial, n, bad);
			return 1;
		}
	}
	puts("ok");
	return 0;
}
