/*
 * Checks that p2_tile_count (csrc/tile_core.h) gives the number of runs that
 * p2_tile_build makes.  Prints "ok" and returns 0, or names the first case
 * that fails.
 */
#include <stdio.h>
#include <stdlib.h>

#include "tile_core.h"

enum { R = 400 };

int main(void)
{
	static struct phase2_rot_in q[R];
	static struct phase2_pass ps[R];
	static struct phase2_rot_rec rc[R];
	static struct p2_tile tl[R];
	static struct p2_tile_sub ss[R];
	static struct p2_tile_rec tr[R];
	srand48(3);
	for (int trial = 0; trial < 600; trial++) {
		const uint32_t n = 12 + (uint32_t)(trial % 19);
		const size_t nr = 1 + (size_t)lrand48() %
				(trial % 2 ? 16 : R);
		const uint64_t m = (UINT64_C(1) << n) - 1;
		for (size_t i = 0; i < nr; i++) {
			q[i].flip = (uint64_t)lrand48() & m;
			if (trial % 3 == 1)
				q[i].flip = (UINT64_C(1) << lrand48() % n) ^
					(UINT64_C(1) << lrand48() % n);
			else if (trial % 3 == 2 && i % 200)
				q[i].flip = q[i - 1].flip;
			q[i].phase = (uint64_t)lrand48() & m;
			q[i].phi = drand48();
		}
		const int span = 1 + trial / 3 % 5;
		const long np = p2_plan_core(n, q, NULL, nr, span, 0,
			P2_DEFAULT_PAD_SPAN, PHASE2_FORM_EXACT, 0, 0, ps, rc);
		uint32_t ns;
		if (np < 0 || p2_tile_count(ps, (size_t)np, rc) !=
				p2_tile_build(ps, (size_t)np, rc, nr, tl, ss,
					tr, &ns)) {
			printf("trial %d\n", trial);
			return 1;
		}
	}
	puts("ok");
	return 0;
}
