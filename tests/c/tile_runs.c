/*
 * Checks csrc/tile_core.h on the host: tile runs give the amplitudes of the
 * rotations one by one, bit for bit (the exact update rounds every product
 * and sum of an amplitude by itself), enumerate every amplitude once, and
 * cover every rotation in order.  Prints "ok" and returns 0, or names the
 * first case that fails.
 */
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include "tile_core.h"

enum { R = 300, NQ = 16, N = 1 << NQ };

/* The rotation on the amplitude pairs (u, u ^ U) of a[idx[..]], sign bit u
 * of sm. */
static void rotate(double *a, const uint32_t *idx, uint32_t n, uint32_t U,
	int odd, double c, double s, const unsigned char *neg)
{
	for (uint32_t u = 0; u < n; u++) {
		const uint32_t w = u ^ U;
		if (w < u)
			continue;
		double *x = a + 2 * idx[u], *y = a + 2 * idx[w];
		const double x0 = x[0], x1 = x[1], y0 = y[0], y1 = y[1];
		const double su = neg[u] ? -s : s, sw = neg[w] ? -s : s;
		x[0] = c * x0 + (odd ? -su * y1 : su * y0);
		x[1] = c * x1 + (odd ? su * y0 : su * y1);
		if (w != u) {
			y[0] = c * y0 + (odd ? -sw * x1 : sw * x0);
			y[1] = c * y1 + (odd ? sw * x0 : sw * x1);
		}
	}
}

static uint32_t insert_zeros(uint32_t x, uint32_t p)
{
	return ((x >> p) << (p + 1)) | (x & ((1u << p) - 1));
}

/* One tile run, as k_tile walks it. */
static const char *run_tile(double *a, uint32_t n, const struct p2_tile *t,
	const struct p2_tile_sub *subs, const struct p2_tile_rec *recs,
	char *seen)
{
	const uint32_t T = 1u << P2_TILE_BITS, S = 1u << P2_TILE_SPAN;
	static uint32_t at[1 << P2_TILE_BITS];
	static char used[1 << P2_TILE_BITS];
	memset(seen, 0, (size_t)1 << n);
	for (uint32_t b = 0; b < (1u << n) / T; b++) {
		uint32_t x0 = b;
		for (int k = 0; k < P2_TILE_BITS; k++)
			x0 = insert_zeros(x0, t->piv[k]);
		for (uint32_t y = 0; y < T; y++) {
			uint32_t g = x0;
			for (int k = 0; k < P2_TILE_BITS; k++)
				if (y >> k & 1)
					g ^= (uint32_t)t->row[k];
			if (g >> n || seen[g]++)
				return "tile enumeration";
			at[y] = g;
		}
		for (uint32_t i = 0; i < t->nsub; i++) {
			const struct p2_tile_sub *h = &subs[t->sub_off + i];
			memset(used, 0, sizeof used);
			for (uint32_t th = 0; th < T / S; th++) {
				uint32_t y = th, idx[1 << P2_TILE_SPAN], out = x0;
				for (int k = 0; k < P2_TILE_SPAN; k++)
					y = insert_zeros(y, h->piv[k]);
				for (int k = 0; k < P2_TILE_BITS - P2_TILE_SPAN; k++)
					if (th >> k & 1)
						out ^= (uint32_t)t->tout[k];
				for (uint32_t u = 0; u < S; u++) {
					uint32_t pos = p2_sub_swz(y), o = out, v = 0;
					for (int k = 0; k < P2_TILE_SPAN; k++)
						if (u >> k & 1) {
							pos ^= h->pslot[k];
							o ^= (uint32_t)t->sout[k];
						}
					/* the swizzle is its own inverse */
					v = p2_sub_swz(pos);
					if (v >> P2_TILE_BITS || used[v]++)
						return "slot enumeration";
					idx[u] = at[v];
					if (i + 1 == t->nsub && o != at[v])
						return "store address";
				}
				for (uint32_t r = h->rot0; r < h->rot0 + h->nrot;
					r++) {
					const struct p2_tile_rec *q =
						&recs[t->rot_off + r];
					unsigned char neg[1 << P2_TILE_SPAN];
					const int par = parity64(y & q->zl) ^
						parity64(x0 & q->z);
					for (uint32_t u = 0; u < S; u++)
						neg[u] = (q->sm >> u & 1) ^ par;
					if (q->key >= 2 * S)
						return "key";
					rotate(a, idx, S, q->key >> 1, q->key & 1,
						q->c, q->s, neg);
				}
			}
		}
	}
	return NULL;
}

int main(void)
{
	static struct phase2_rot_in q[R];
	static struct phase2_pass ps[R];
	static struct phase2_rot_rec rc[R];
	static struct p2_tile tl[R];
	static struct p2_tile_sub ss[R];
	static struct p2_tile_rec tr[R];
	static double a[2 * N], b[2 * N];
	static uint32_t all[N];
	static unsigned char neg[N];
	static char seen[N];
	srand48(2);
	for (uint32_t g = 0; g < N; g++)
		all[g] = g;
	for (int trial = 0; trial < 24; trial++) {
		const uint32_t n = 13 + (uint32_t)trial % 4;
		const size_t nr = 1 + (size_t)lrand48() % R;
		const uint64_t m = (UINT64_C(1) << n) - 1;
		for (size_t i = 0; i < nr; i++) {
			uint64_t f = (uint64_t)lrand48() & m;
			if (trial % 3 == 1)
				f = (UINT64_C(1) << lrand48() % n) ^
					(UINT64_C(1) << lrand48() % n);
			else if (trial % 3 == 2 && i % 140)
				f = q[i - 1].flip;
			q[i].flip = f;
			q[i].phase = (uint64_t)lrand48() & m;
			q[i].phi = drand48() * 8 - 4;
		}
		const long np = p2_plan_core(n, q, NULL, nr, 5, 0,
			P2_DEFAULT_PAD_SPAN, PHASE2_FORM_EXACT, 0, 0, ps, rc);
		for (size_t i = 0; i < (size_t)2 << n; i++)
			a[i] = b[i] = drand48() - 0.5;
		for (size_t i = 0; i < nr; i++) {
			/* a_g <- c a_g + i s conj(z_g) a_(g ^ f) */
			const int k = (1 - __builtin_popcountll(q[i].flip &
						  q[i].phase)) & 3;
			for (uint32_t g = 0; g < 1u << n; g++)
				neg[g] = (unsigned char)(parity64(g & q[i].phase) ^
					(k >> 1));
			rotate(a, all, 1u << n, (uint32_t)q[i].flip, k & 1,
				cos(q[i].phi), sin(q[i].phi), neg);
		}
		uint32_t ns;
		const uint32_t nt = p2_tile_build(ps, (size_t)np, rc, nr, tl, ss,
			tr, &ns);
		const char *bad = np < 0 ? "plan" : NULL;
		uint32_t rot = 0, sub = 0;
		for (uint32_t i = 0; i < nt && !bad; i++) {
			if (tl[i].rot_off != rot || tl[i].sub_off != sub ||
				tl[i].nrot == 0 || tl[i].nrot > P2_TILE_ROTS)
				bad = "order";
			rot += tl[i].nrot;
			sub += tl[i].nsub;
			if (!bad)
				bad = run_tile(b, n, &tl[i], ss, tr, seen);
		}
		if (!bad && (rot != nr || sub != ns))
			bad = "coverage";
		if (!bad && memcmp(a, b, (size_t)16 << n))
			bad = "bits";
		if (bad) {
			printf("trial %d, %u qubits: %s\n", trial, n, bad);
			return 1;
		}
	}
	puts("ok");
	return 0;
}
