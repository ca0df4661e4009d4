/*
 * sub_core.h -- passes cut into sub-passes for the resident kernel
 * (resident.cu), on the host.
 *
 * A pass holds 2^span <= 32 amplitudes a thread; a register that fits on
 * chip has too few cosets of that size to fill an SM, and 32 unrolled slots
 * times 64 cases of rotations is more code than the instruction caches
 * hold.  A sub-pass is a run of a pass's rotations whose slot combinations
 * U span at most P2_SUB_SPAN dimensions: 8 amplitudes a thread, 16 cases.
 * Amplitudes between two sub-passes of a pass keep the precision they have
 * inside the pass, so the arithmetic of every amplitude is the pass's.
 *
 * The lifted (shear) update treats the two amplitudes of a pair
 * differently: the one whose slot has a zero at the top bit of U goes first.
 * Slots of a sub-pass are numbered along a reduced echelon basis of its
 * U's (slot bit k = coordinate of pivot k of the slot space), and its
 * representatives have coordinate 0 at those pivots, so the top bit of a
 * rotation's combination in the sub-pass marks the same amplitude.
 */
#ifndef P2_SUB_CORE_H
#define P2_SUB_CORE_H

#include <stdint.h>
#include <string.h>

#include "plan_core.h"

#define P2_SUB_SPAN 3
#define P2_SUB_ROTS 64 /* rotations of a sub-pass (one staging buffer) */

enum { P2_SUB_LAST = 1, P2_SUB_NEG = 2 };

/*
 * Thread number t -> index x: zeros inserted at piv (ascending), then
 * slot[k] XORed in where parity(x & orient[k]) is odd; slot u is x ^ (xor
 * of slot[k] over the bits of u).  pslot: slot after the shared-memory
 * swizzle.
 */
struct p2_sub {
	uint32_t rot_off;
	uint16_t nrot;
	uint16_t flags; /* P2_SUB_LAST: ends its pass (FP32 states round
			 * here), P2_SUB_NEG: negate there */
	uint32_t piv[P2_SUB_SPAN];
	uint32_t slot[P2_SUB_SPAN];
	uint32_t orient[P2_SUB_SPAN];
	uint32_t pslot[P2_SUB_SPAN];
	uint32_t pad[2];
};

/* One rotation of a sub-pass: c, s as in struct phase2_rot_rec; sm: sign
 * bit of slot u at bit u (before parity(x & z)); key = U << 1 | odd. */
struct p2_sub_rec {
	double c, s;
	uint32_t z;
	uint8_t sm, key;
	uint16_t pad0;
	uint64_t pad1;
};

/* Shared-memory position of index g: the low 3 bits (the 16-byte bank
 * groups) take the XOR of the 3-bit groups above, so that lanes that differ
 * in any bits fall on different banks as far as a linear map can. */
P2_HD uint32_t p2_sub_swz(uint32_t g)
{
	uint32_t f = g >> 3;
	f ^= f >> 12;
	f ^= f >> 6;
	f ^= f >> 3;
	return g ^ (f & 7u);
}

/* Header of a sub-pass whose reduced slot rows are row[0..d-1] with pivots
 * sp[0..d-1] ascending: index offsets, padding by unit vectors, pivots. */
P2_HD void p2_sub_header(const struct phase2_pass *ps, const uint32_t *h,
	uint32_t nqb, const uint32_t *row, const int *sp, int d,
	struct p2_sub *out)
{
	struct echelon e;
	uint32_t combo;
	memset(&e, 0, sizeof e);
	for (int k = 0; k < d; k++) {
		uint64_t v = 0;
		for (uint32_t j = 0; j < ps->span; j++)
			if (row[k] >> j & 1)
				v ^= ps->basis[j];
		out->slot[k] = (uint32_t)v;
		out->orient[k] = h[sp[k]];
		ech_insert(&e, ech_reduce(&e, v, &combo), 0);
	}
	for (uint32_t q = 0, k = (uint32_t)d; k < P2_SUB_SPAN && q < nqb; q++) {
		uint32_t v = UINT32_C(1) << q;
		const uint64_t rem = ech_reduce(&e, v, &combo);
		if (rem == 0)
			continue;
		/* a padding slot keeps the pairs' order: coordinate 0 at the
		 * slot pivots */
		const uint32_t v0 = v;
		for (int j = 0; j < d; j++)
			if (P2_POPC32(v0 & out->orient[j]) & 1)
				v ^= out->slot[j];
		out->slot[k] = v;
		out->orient[k] = 0;
		ech_insert(&e, rem, 0);
		k++;
	}
	for (int k = 0; k < P2_SUB_SPAN; k++) {
		out->piv[k] = (uint32_t)e.piv[P2_SUB_SPAN - 1 - k];
		out->pslot[k] = p2_sub_swz(out->slot[k]);
	}
}

/* Sub-passes of one pass (nqb >= 3); recs are the pass's records, their
 * repacked copies go to out[0..nrot), numbered from rec0.  Returns the
 * sub-passes written (at most nrot). */
P2_HD uint32_t p2_sub_split(const struct phase2_pass *ps,
	const struct phase2_rot_rec *recs, uint32_t nqb, uint32_t rec0,
	struct p2_sub *subs, struct p2_sub_rec *out)
{
	const int M = (int)ps->span;
	/* h[k]: mask with parity(g & h[k]) = slot coordinate k of index g
	 * (Gauss-Jordan on the basis bits at the pivots) */
	uint32_t a[PHASE2_MAX_SPAN], x[PHASE2_MAX_SPAN], h[PHASE2_MAX_SPAN];
	for (int i = 0; i < M; i++) {
		a[i] = 0;
		for (int k = 0; k < M; k++)
			a[i] |= (uint32_t)(ps->basis[k] >> ps->piv[i] & 1) << k;
		x[i] = UINT32_C(1) << ps->piv[i];
	}
	for (int k = 0; k < M; k++) {
		int r = k;
		while (r < M - 1 && !(a[r] >> k & 1))
			r++;
		uint32_t t = a[r];
		a[r] = a[k];
		a[k] = t;
		t = x[r];
		x[r] = x[k];
		x[k] = t;
		for (int i = 0; i < M; i++)
			if (i != k && (a[i] >> k & 1)) {
				a[i] ^= a[k];
				x[i] ^= x[k];
			}
	}
	for (int k = 0; k < M; k++)
		h[k] = x[k];

	uint32_t n = 0, r = 0;
	while (r < ps->nrot) {
		uint32_t row[P2_SUB_SPAN];
		int sp[P2_SUB_SPAN], d = 0;
		const uint32_t first = r;
		for (; r < ps->nrot && r - first < P2_SUB_ROTS; r++) {
			uint32_t v = recs[r].U;
			for (int j = 0; j < d; j++)
				if (v >> sp[j] & 1)
					v ^= row[j];
			if (v == 0)
				continue;
			if (d == P2_SUB_SPAN)
				break;
			const int p = top_bit(v);
			int at = d;
			for (int j = 0; j < d; j++)
				if (row[j] >> p & 1)
					row[j] ^= v;
			while (at > 0 && sp[at - 1] > p) {
				row[at] = row[at - 1];
				sp[at] = sp[at - 1];
				at--;
			}
			row[at] = v;
			sp[at] = p;
			d++;
		}
		struct p2_sub *s = &subs[n++];
		memset(s, 0, sizeof *s);
		s->rot_off = rec0 + first;
		s->nrot = (uint16_t)(r - first);
		p2_sub_header(ps, h, nqb, row, sp, d, s);
		for (uint32_t i = first; i < r; i++) {
			const struct phase2_rot_rec *q = &recs[i];
			struct p2_sub_rec o;
			memset(&o, 0, sizeof o);
			o.c = q->c;
			o.s = q->s;
			o.z = (uint32_t)q->z;
			uint32_t U = 0, W = 0, sm = 0;
			for (int k = 0; k < d; k++)
				U |= (uint32_t)(q->U >> sp[k] & 1) << k;
			for (int k = 0; k < P2_SUB_SPAN; k++)
				W |= (uint32_t)(P2_POPC32(s->slot[k] & o.z) & 1)
					<< k;
			for (uint32_t u = 0; u < (1u << P2_SUB_SPAN); u++)
				sm |= ((q->smask ^ (uint32_t)P2_POPC32(u & W)) &
					      1u) << u;
			o.sm = (uint8_t)sm;
			o.key = (uint8_t)(U << 1 | q->odd);
			out[i] = o;
		}
		if (r == ps->nrot)
			s->flags = (uint16_t)(P2_SUB_LAST |
				(ps->scale < 0 ? P2_SUB_NEG : 0));
	}
	return n;
}

/* ---- tiles of one pass (split.cu) --------------------------------------- */

#define P2_SPLIT_BITS 10 /* amplitudes of a tile, log2 */

/* A pass as k_pass_split takes it (span 3..5), and its sub-passes. */
struct p2_split_pass {
	struct phase2_pass pass;
	uint32_t sub_off, nsub;
};

/*
 * Sub-passes of pass `in` on tiles of 2^10 amplitudes: 2^(10 - span)
 * consecutive representatives (the tile-local index's low bits) and their
 * slots (its high bits).  The records' z are local, the pass's phase masks
 * are kept in pad1 (a tile adds its representatives' part of the parity).
 * recs, sr: the flush's records and their repacked copies.
 */
static inline void p2_split_build(uint32_t nqb, const struct phase2_pass *in,
	const struct phase2_rot_rec *recs, struct p2_split_pass *out,
	uint32_t sub_off, struct p2_sub *subs, struct p2_sub_rec *sr)
{
	struct phase2_pass *p = &out->pass;
	*p = *in;
	/* at least three dimensions: padding by unit vectors off the pivots,
	 * which leave the pairs' order as it is */
	for (uint32_t q = 0; p->span < P2_SUB_SPAN && q < nqb; q++) {
		uint32_t at = 0;
		while (at < p->span && p->piv[at] < q)
			at++;
		if (at < p->span && p->piv[at] == q)
			continue;
		for (uint32_t k = p->span; k > at; k--)
			p->piv[k] = p->piv[k - 1];
		p->piv[at] = (uint8_t)q;
		p->basis[p->span++] = UINT64_C(1) << q;
	}
	const uint32_t M = p->span, LB = P2_SPLIT_BITS - M;
	struct phase2_pass v;
	memset(&v, 0, sizeof v);
	v.span = M;
	v.nrot = p->nrot;
	v.rot_off = p->rot_off;
	v.scale = p->scale;
	for (uint32_t k = 0; k < M; k++) {
		v.basis[k] = UINT64_C(1) << (LB + k);
		v.piv[k] = (uint8_t)(LB + k);
	}
	uint64_t lane[P2_SPLIT_BITS];
	for (uint32_t j = 0; j < LB; j++) {
		lane[j] = UINT64_C(1) << j;
		for (uint32_t k = 0; k < M; k++) {
			const uint32_t q = p->piv[k];
			lane[j] = ((lane[j] >> q) << (q + 1)) |
				(lane[j] & ((UINT64_C(1) << q) - 1));
		}
	}
	struct phase2_rot_rec r[P2_MAX_ROTS_PER_PASS];
	for (uint32_t i = 0; i < p->nrot; i++) {
		r[i] = recs[p->rot_off + i];
		uint64_t z = 0;
		for (uint32_t j = 0; j < LB; j++)
			z |= (uint64_t)parity64(lane[j] & r[i].z) << j;
		for (uint32_t k = 0; k < M; k++)
			z |= (uint64_t)parity64(p->basis[k] & r[i].z)
				<< (LB + k);
		r[i].z = z;
	}
	out->sub_off = sub_off;
	out->nsub = p2_sub_split(&v, r, P2_SPLIT_BITS, p->rot_off, subs,
		sr + p->rot_off);
	for (uint32_t i = 0; i < p->nrot; i++)
		sr[p->rot_off + i].pad1 = recs[p->rot_off + i].z;
}

#endif /* P2_SUB_CORE_H */
