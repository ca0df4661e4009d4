/*
 * tile_core.h -- a flush of exact-form rotations cut into tiles (tile.cu),
 * on the host.
 */
#ifndef P2_TILE_CORE_H
#define P2_TILE_CORE_H

#include "sub_core.h"

#define P2_TILE_BITS 12 /* amplitudes of a tile, log2 */
#define P2_TILE_LOW 4   /* lowest qubits in every tile */
#define P2_TILE_SPAN 4  /* dimensions of a sub-pass */
#define P2_TILE_ROTS 128

/* One run of rotations on all tiles: index offsets of the local bits, their
 * pivots (ascending), its rotations and sub-passes, and of the last
 * sub-pass the index offsets of the thread-number and slot bits. */
struct p2_tile {
	uint64_t row[P2_TILE_BITS];
	uint64_t tout[P2_TILE_BITS - P2_TILE_SPAN];
	uint64_t sout[P2_TILE_SPAN];
	uint8_t piv[P2_TILE_BITS];
	uint32_t rot_off, nrot, sub_off, nsub;
};

/* Sub-pass: thread number -> local index by zeros inserted at piv; slot bit
 * k is the local vector whose place after the swizzle is pslot[k]. */
struct p2_tile_sub {
	uint16_t rot0, nrot; /* of the tile's rotations */
	uint16_t piv[P2_TILE_SPAN];
	uint16_t pslot[P2_TILE_SPAN];
	uint16_t pad[2];
};

/* One rotation: z phase mask, zl its local part (bit k: parity of row k);
 * sm: sign of slot u at bit u, before the parities of the tile's
 * representative with z and of the local index with zl. */
struct p2_tile_rec {
	double c, s;
	uint64_t z;
	uint16_t zl, sm;
	uint16_t key; /* U << 1 | odd */
	uint16_t pad;
};

/* Reduced echelon of up to P2_TILE_BITS rows, pivots descending. */
struct p2_tile_ech {
	int rows;
	uint64_t v[P2_TILE_BITS];
	int piv[P2_TILE_BITS];
};

static inline uint64_t p2_te_reduce(const struct p2_tile_ech *e, uint64_t v)
{
	for (int r = 0; r < e->rows; r++)
		if (v >> e->piv[r] & 1)
			v ^= e->v[r];
	return v;
}

/* Add v, already reduced and non-zero. */
static inline void p2_te_add(struct p2_tile_ech *e, uint64_t v)
{
	const int p = top_bit(v);
	int at = e->rows;
	for (int r = 0; r < e->rows; r++)
		if (e->v[r] >> p & 1)
			e->v[r] ^= v;
	while (at > 0 && e->piv[at - 1] < p) {
		e->v[at] = e->v[at - 1];
		e->piv[at] = e->piv[at - 1];
		at--;
	}
	e->v[at] = v;
	e->piv[at] = p;
	e->rows++;
}

/* Flip mask of a record of pass p. */
static inline uint64_t p2_rec_flip(const struct phase2_pass *p,
	const struct phase2_rot_rec *r)
{
	uint64_t f = 0;
	for (uint32_t k = 0; k < p->span; k++)
		if (r->U >> k & 1)
			f ^= p->basis[k];
	return f;
}

/* Local index of an offset in the tile space. */
static inline uint32_t p2_tile_local(const struct p2_tile *t, uint64_t v)
{
	uint32_t y = 0;
	for (int k = 0; k < P2_TILE_BITS; k++)
		y |= (uint32_t)(v >> t->piv[k] & 1) << k;
	return y;
}

/* Sub-passes of one tile whose rotations' local flips are fl[0..nrot);
 * completes out[]'s sm and key, returns their number. */
static inline uint32_t p2_tile_subs(struct p2_tile *t, const uint32_t *fl,
	struct p2_tile_sub *subs, struct p2_tile_rec *out)
{
	uint32_t n = 0, r = 0;
	while (r < t->nrot) {
		struct p2_tile_ech e;
		const uint32_t first = r;
		memset(&e, 0, sizeof e);
		for (; r < t->nrot; r++) {
			const uint64_t v = p2_te_reduce(&e, fl[r]);
			if (v == 0)
				continue;
			if (e.rows == P2_TILE_SPAN)
				break;
			p2_te_add(&e, v);
		}
		/* pad from the top, so that threads keep the low local bits */
		for (int q = P2_TILE_BITS - 1; e.rows < P2_TILE_SPAN; q--) {
			const uint64_t v = p2_te_reduce(&e, UINT64_C(1) << q);
			if (v)
				p2_te_add(&e, v);
		}
		struct p2_tile_sub *s = &subs[n++];
		memset(s, 0, sizeof *s);
		s->rot0 = (uint16_t)first;
		s->nrot = (uint16_t)(r - first);
		uint32_t pivs = 0, slot[P2_TILE_SPAN];
		for (int k = 0; k < P2_TILE_SPAN; k++) {
			slot[k] = (uint32_t)e.v[P2_TILE_SPAN - 1 - k];
			s->piv[k] = (uint16_t)e.piv[P2_TILE_SPAN - 1 - k];
			s->pslot[k] = (uint16_t)p2_sub_swz(slot[k]);
			pivs |= UINT32_C(1) << s->piv[k];
			t->sout[k] = 0;
			for (int j = 0; j < P2_TILE_BITS; j++)
				if (slot[k] >> j & 1)
					t->sout[k] ^= t->row[j];
		}
		for (int k = 0, j = 0; j < P2_TILE_BITS; j++)
			if (!(pivs >> j & 1))
				t->tout[k++] = t->row[j];
		for (uint32_t i = first; i < r; i++) {
			uint32_t U = 0, W = 0, sm = 0;
			for (int k = 0; k < P2_TILE_SPAN; k++) {
				U |= (fl[i] >> s->piv[k] & 1) << k;
				W |= (uint32_t)(P2_POPC32(slot[k] & out[i].zl) & 1)
					<< k;
			}
			for (uint32_t u = 0; u < (1u << P2_TILE_SPAN); u++)
				sm |= ((out[i].sm ^ (uint32_t)P2_POPC32(u & W)) &
					      1u) << u;
			out[i].sm = (uint16_t)sm;
			out[i].key = (uint16_t)(U << 1 | out[i].key);
		}
	}
	return n;
}

/* An empty run's echelon: the low qubits, which are in every tile. */
static inline void p2_tile_open(struct p2_tile_ech *e)
{
	memset(e, 0, sizeof *e);
	for (int q = 0; q < P2_TILE_LOW; q++)
		p2_te_add(e, UINT64_C(1) << q);
}

/* Add flip mask f to a run of n rotations: 0 if it is full. */
static inline int p2_tile_take(struct p2_tile_ech *e, uint32_t n, uint64_t f)
{
	if (n == P2_TILE_ROTS)
		return 0;
	const uint64_t v = p2_te_reduce(e, f);
	if (v) {
		if (e->rows == P2_TILE_BITS)
			return 0;
		p2_te_add(e, v);
	}
	return 1;
}

/* The runs that p2_tile_build makes of these passes. */
static inline size_t p2_tile_count(const struct phase2_pass *passes,
	size_t npass, const struct phase2_rot_rec *recs)
{
	struct p2_tile_ech e;
	size_t runs = 0;
	uint32_t n = 0;
	for (size_t p = 0; p < npass; p++)
		for (uint32_t r = 0; r < passes[p].nrot; r++) {
			const uint64_t f = p2_rec_flip(&passes[p],
				&recs[passes[p].rot_off + r]);
			if (runs == 0 || !p2_tile_take(&e, n, f)) {
				p2_tile_open(&e);
				p2_tile_take(&e, 0, f);
				runs++;
				n = 0;
			}
			n++;
		}
	return runs;
}

/*
 * The flush's rotations in order, greedily: a tile run takes rotations while
 * their flips span at most P2_TILE_BITS - P2_TILE_LOW dimensions beside the
 * low qubits.  Writes at most nrec tiles, sub-passes and (all) records;
 * *nsub gets the sub-passes; returns the tiles.
 */
static inline uint32_t p2_tile_build(const struct phase2_pass *passes,
	size_t npass, const struct phase2_rot_rec *recs, size_t nrec,
	struct p2_tile *tiles, struct p2_tile_sub *subs,
	struct p2_tile_rec *out, uint32_t *nsub)
{
	uint32_t nt = 0, ns = 0;
	size_t i = 0, p = 0;
	while (i < nrec) {
		struct p2_tile *t = &tiles[nt++];
		struct p2_tile_ech e;
		uint64_t flip[P2_TILE_ROTS];
		uint32_t fl[P2_TILE_ROTS];
		memset(t, 0, sizeof *t);
		p2_tile_open(&e);
		t->rot_off = (uint32_t)i;
		t->sub_off = ns;
		for (; i < nrec; i++) {
			while (p + 1 < npass && i >= passes[p + 1].rot_off)
				p++;
			const uint64_t f = p2_rec_flip(&passes[p], &recs[i]);
			if (!p2_tile_take(&e, t->nrot, f))
				break;
			flip[t->nrot++] = f;
		}
		for (int q = 0; e.rows < P2_TILE_BITS; q++) {
			const uint64_t v = p2_te_reduce(&e, UINT64_C(1) << q);
			if (v)
				p2_te_add(&e, v);
		}
		for (int k = 0; k < P2_TILE_BITS; k++) {
			t->row[k] = e.v[P2_TILE_BITS - 1 - k];
			t->piv[k] = (uint8_t)e.piv[P2_TILE_BITS - 1 - k];
		}
		for (uint32_t r = 0; r < t->nrot; r++) {
			const struct phase2_rot_rec *in = &recs[t->rot_off + r];
			struct p2_tile_rec *o = &out[t->rot_off + r];
			memset(o, 0, sizeof *o);
			o->c = in->c;
			o->s = in->s;
			o->z = in->z;
			for (int k = 0; k < P2_TILE_BITS; k++)
				o->zl |= (uint16_t)(parity64(t->row[k] & in->z)
					<< k);
			o->sm = (uint16_t)(in->smask & 1u);
			o->key = in->odd;
			fl[r] = p2_tile_local(t, flip[r]);
		}
		t->nsub = p2_tile_subs(t, fl, subs + ns, out + t->rot_off);
		ns += t->nsub;
	}
	*nsub = ns;
	return nt;
}

#endif /* P2_TILE_CORE_H */
