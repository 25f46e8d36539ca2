/*
 * Planner of factored sweeps (host C).
 *
 * Sweeps take their gates as in dk_plan.c: a tile of 2^m amplitudes over a
 * qubit set Q, any gate whose targets fit in Q and that commutes with the
 * gates left behind.  The gates of a sweep are grouped into passes over 4 tile
 * bits, and each pass is factored into real rotations, diagonal products and
 * relabellings of its 16 register amplitudes (dk_internal.h, "factored
 * sweeps").  A one-qubit unitary then costs 2 real multiply-adds per amplitude
 * and its phases are shared with the other gates of the pass, where an 8x8
 * complex product costs 24 per run of gates on 3 bits.  Sweeps that hold a
 * gate without such a factoring (dense gates on 2 and 3 qubits, one-qubit
 * matrices that are not a diagonal times a real rotation) are planned by
 * dk_plan.c.
 *
 * Planning runs while the device works (one step per call), so its cost per
 * gate matters: supports are computed once, a scan ends when every qubit is
 * blocked, and the search for a bank map runs only for sweeps that the fixed
 * residue map leaves with conflicts.  Nor may it fail there, between two sweeps
 * that change a register in place: a plan of factored sweeps only allocates nothing
 * once dk_fx_reserve has run, and any other plan, whose gates keep the matrices they
 * were given, can name the gates that it has not come to (dk_fx_left).
 */
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include "dk_internal.h"

#define FX_WINDOW 64 /* gates examined per pass */

enum { FX_NONE = 0, FX_DIAG, FX_PERM, FX_ROT };

/* A gate's factors are computed in extended precision; the diagonal products
 * of a stage, a few factors each, in double. */
typedef long double real;
typedef struct cpx {
	real x, y;
} cpx;
typedef struct cpd {
	double x, y;
} cpd;

static cpx cx(real x, real y)
{
	cpx r = { x, y };
	return r;
}
static cpx cmul(cpx a, cpx b) { return cx(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
/* a / b */
static cpx cdiv(cpx a, cpx b)
{
	const real d = b.x * b.x + b.y * b.y;
	return cx((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}
static int ceq(cpx a, cpx b) { return a.x == b.x && a.y == b.y; }
static int czero(cpx a) { return a.x == 0.0 && a.y == 0.0; }
static const cpx c_one = { 1.0, 0.0 };
static cpd cd(cpx a)
{
	cpd r = { (double)a.x, (double)a.y };
	return r;
}
static cpd dmul(cpd a, cpd b)
{
	cpd r = { a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x };
	return r;
}
static int deq(cpd a, cpd b) { return a.x == b.x && a.y == b.y; }
static const cpd d_one = { 1.0, 0.0 };

/* A gate with its factors: U = diag(l0, l1) [[1, -s], [t, 1]] diag(1, r1),
 * applied after an X when `flip` (FX_ROT); diag(l0, l1) after an X
 * (FX_PERM); diag(l0, l1) (FX_DIAG on one qubit). */
typedef struct fx_gate {
	uint64_t sup, tmask, ctl;
	int kind, flip;
	int unitary, is_x; /* one qubit: a multiple of a unitary; exactly X */
	int known; /* the factors below are those of its matrix */
	int gone; /* absorbed by a later gate */
	cpx l0, l1, r1;
	real s, t;
	cpd d0, d1, dr; /* l0, l1, r1 as the passes use them */
	double ds, dt;
} fx_gate;

static uint64_t tbit(unsigned q) { return UINT64_C(1) << q; }
static int popc(uint64_t x) { return __builtin_popcountll(x); }

static real cabs2(cpx a) { return a.x * a.x + a.y * a.y; }

/* What a factoring may leave out of a matrix, next to entries of size 1: of 20,000
 * random U3s in double it is 1.1e-15 at most, of products of three 1.7e-15. */
#define FX_DROP 4e-15L

/* a, b, c, d (a, d not zero) as diag(l0, l1) [[1, -s], [t, 1]] diag(1, r1);
 * 0 when s is not real.  r1 is a phase, so the factors stay as large as the
 * matrix.  s is real for every multiple of a unitary, up to the roundings of its
 * entries (products of several matrices among them, next to entries of size
 * 1); for other matrices it has to be real to a few roundings of itself.  The
 * phase of b c / (a d) that keeps s from being real is left out of all four
 * entries, in shares that leave the least error: a quarter of it from each where
 * they are alike, half from b and c where they are small. */
static int factor2(cpx a, cpx b, cpx c, cpx d, fx_gate *g)
{
	cpx r1 = c_one, l0 = a, l1 = d;
	real s = 0, t = 0;
	if (!czero(c)) {
		const cpx w = cdiv(c, d);
		t = sqrtl(cabs2(w));
		if (!(t > 0) || t > 1e6L)
			return 0;
		r1 = cx(w.x / t, -w.y / t);
		if (!czero(b)) {
			const cpx v = cmul(cdiv(b, a), cx(r1.x, -r1.y));
			s = -v.x;
			if (!(fabsl(v.y) <= (g->unitary ? FX_DROP : FX_DROP * fabsl(s))) ||
			    fabsl(s) > 1e6L)
				return 0;
			if (fabsl(v.y) <= 1e-8L * fabsl(s)) {
				/* v = -s exp(i e): e / 2 to r1; a and d turn by e / 2 times
				 * the part of b c in b c + a d */
				const real x = fabsl(s) * t, e = v.y / v.x;
				const cpx f = cx(1, e * x / (2 * (1 + x)));
				r1 = cmul(r1, cx(1, e / 2));
				l0 = cmul(a, f);
				l1 = cmul(d, f);
			}
		}
	} else if (!czero(b)) {
		const cpx v = cdiv(b, a);
		s = sqrtl(cabs2(v));
		if (!(s > 0) || s > 1e6L)
			return 0;
		r1 = cx(-v.x / s, -v.y / s);
	}
	g->l0 = l0;
	g->l1 = cmul(l1, cx(r1.x, -r1.y));
	g->r1 = r1;
	g->s = s;
	g->t = t;
	return isfinite(g->l0.x) && isfinite(g->l0.y) && isfinite(g->l1.x) && isfinite(g->l1.y);
}

/* The kind and factors of a one-qubit matrix m = (a, b, c, d). */
static void factor1(const cpx *m, fx_gate *g)
{
	const cpx a = m[0], b = m[1], c = m[2], d = m[3];
	g->kind = FX_NONE;
	g->flip = 0;
	if (czero(b) && czero(c)) {
		g->kind = FX_DIAG;
		g->l0 = a;
		g->l1 = d;
		return;
	}
	if (czero(a) && czero(d)) {
		g->kind = FX_PERM;
		g->l0 = b;
		g->l1 = c;
		return;
	}
	/* the larger of the two diagonals is factored out, so that s and t of
	 * a unitary stay within 1: an X first where it is the other one */
	g->flip = cabs2(b) * cabs2(c) > cabs2(a) * cabs2(d);
	if (g->flip ? (czero(b) || czero(c)) : (czero(a) || czero(d)))
		return;
	if (g->flip ? factor2(b, a, d, c, g) : factor2(a, b, c, d, g))
		g->kind = FX_ROT;
}

/* The kind of a one-qubit matrix; its factors too unless it is a rotation of a
 * unitary, whose factors (three divisions and a root) wait until the gate's last
 * matrix is known.  Its s is told real from b c / (a d) with half of factor2's
 * margin. */
static void classify1(const cpx *m, fx_gate *g)
{
	if (!g->unitary || czero(m[0]) || czero(m[1]) || czero(m[2]) || czero(m[3])) {
		factor1(m, g);
		g->known = 1;
		return;
	}
	const real na = cabs2(m[0]), nb = cabs2(m[1]), nc = cabs2(m[2]), nd = cabs2(m[3]);
	const cpx bc = cmul(m[1], m[2]), ad = cmul(m[0], m[3]);
	const real y = bc.y * ad.x - bc.x * ad.y;
	g->flip = nb * nc > na * nd;
	/* |Im s| = |y| / (|a|^2 |c| |d|), b for a and so on after an X */
	const real f = FX_DROP / 2 * (g->flip ? nb : na);
	g->kind = y * y <= f * f * nc * nd ? FX_ROT : FX_NONE;
	g->known = 0;
	if (g->kind == FX_NONE) {
		factor1(m, g);
		g->known = 1;
	}
}

static void load1(const dk_flat_op *op, cpx *m)
{
	for (int i = 0; i < 4; i++)
		m[i] = cx(op->gate->m[2 * i], op->gate->m[2 * i + 1]);
}

static void analyse(const dk_flat_op *op, fx_gate *g)
{
	g->tmask = 0;
	for (unsigned i = 0; i < op->k; i++)
		g->tmask |= tbit(op->tg[i]);
	g->ctl = op->cm | op->am;
	g->sup = g->tmask | g->ctl;
	g->kind = FX_NONE;
	g->flip = g->unitary = g->is_x = g->gone = 0;
	g->known = 1;
	if (op->k > DK_SWEEP_MAX_K)
		return;
	if (op->k > 1) {
		if (dk_gate_classify(op->gate) == DK_GK_DIAGK)
			g->kind = FX_DIAG;
		return;
	}
	cpx m[4];
	load1(op, m);
	/* columns of one length, orthogonal */
	const real n0 = cabs2(m[0]) + cabs2(m[2]), n1 = cabs2(m[1]) + cabs2(m[3]);
	const cpx x = cx(m[0].x * m[1].x + m[0].y * m[1].y + m[2].x * m[3].x + m[2].y * m[3].y,
			 m[0].x * m[1].y - m[0].y * m[1].x + m[2].x * m[3].y - m[2].y * m[3].x);
	g->unitary = n0 > 0 && fabsl(n0 - n1) <= 1e-14L * n0 && fabsl(x.x) + fabsl(x.y) <= 1e-14L * n0;
	classify1(m, g);
	g->is_x = g->kind == FX_PERM && ceq(m[1], c_one) && ceq(m[2], c_one);
}

/* ---- a sweep's program under construction -------------------------------- */

typedef struct fx_buf {
	dk_fx_op *op;
	int nop, cop;
	double *coef; /* doubles, whatever the program's precision */
	size_t ncoef, ccoef;
	dk_fx_list *list;
	int nlist, clist;
	dk_gate_cond cond[DK_FX_MAX_CONDS + DK_FX_COND];
	int ncond;
	int prec;
	size_t bytes; /* of the operations and their coefficients in the program */
	int oom;
} fx_buf;

struct dk_fx_plan {
	const dk_flat_op *ops;
	fx_gate *g;
	unsigned n;
	int prec;
	int nops; /* gates to plan */
	int ngone; /* gates absorbed by others, not yet counted in a step */
	int all; /* every gate has a factoring */
	dk_plan_limits lim;
	int *rem, head; /* gates left: rem[head .. nops) */
	int *take, *order, *win; /* a sweep's gates; in pass order; a pass's leftovers */
	dk_fx_pass *pass;
	uint32_t *need;
	uint8_t (*pbits)[DK_FX_BITS];
	uint32_t (*sp)[DK_FX_BITS]; /* slot offsets of a pass's bits */
	uint16_t (*range)[2]; /* gates of each pass, in `order` */
	int cpass;
	fx_buf b;
	unsigned char *prog;
	size_t cprog;
	/* steps of a sub-plan made by dk_plan.c */
	dk_plan sub;
	int sub_at, sub_n, *sub_ops;
	/* gates of the current sweep not yet emitted (its program was full) */
	int nleft;
	uint64_t leftQ;
};

static int grow(void **p, size_t elem, int *cap, int want)
{
	if (want <= *cap)
		return 0;
	int nc = *cap ? *cap : 64;
	while (nc < want)
		nc *= 2;
	void *np = realloc(*p, elem * (size_t)nc);
	if (!np)
		return -1;
	*p = np;
	*cap = nc;
	return 0;
}

/* Bytes of an operation's coefficients in the program. */
static size_t op_bytes(const dk_fx_op *o, int prec)
{
	if (o->code == DK_FX_STAGE)
		return 64u + (o->mask & 16u ? (prec == DK_C128 ? 256u : 128u) : 0u);
	if (o->code < DK_FX_PHASE)
		return 128;
	return o->code == DK_FX_PHASE ? 16 : 0;
}

static dk_fx_op *new_op(fx_buf *b, unsigned code, unsigned mask, uint32_t lc, uint32_t la)
{
	if (grow((void **)&b->op, sizeof(dk_fx_op), &b->cop, b->nop + 1)) {
		b->oom = 1;
		return NULL;
	}
	dk_fx_op *o = &b->op[b->nop++];
	o->code = (uint16_t)code;
	o->mask = (uint16_t)mask;
	o->coef = (uint32_t)b->ncoef;
	o->lc = lc;
	o->la = la;
	b->bytes += sizeof(*o) + op_bytes(o, b->prec);
	return o;
}

static double *new_coef(fx_buf *b, int count)
{
	if (b->ncoef + (size_t)count > b->ccoef) {
		size_t nc = b->ccoef ? b->ccoef : 4096;
		while (nc < b->ncoef + (size_t)count)
			nc *= 2;
		double *np = (double *)realloc(b->coef, sizeof(double) * nc);
		if (!np) {
			b->oom = 1;
			return NULL;
		}
		b->coef = np;
		b->ccoef = nc;
	}
	double *at = b->coef + b->ncoef;
	b->ncoef += (size_t)count;
	return at;
}

/* A stage of a pass: diag(din), then rotations along distinct directions,
 * then diag(dout), all in register space.  A stage grows while the next gate's
 * parts commute into it.  Sets of registers are 16-bit masks: M[j] holds the
 * registers whose pass index has bit j, dinm and doutm those whose factor may
 * differ from 1 (only these are stored). */
typedef struct fx_rotn {
	uint8_t dir, plain; /* plain: along a register bit, co[0] and co[1] for all */
	double co[16]; /* (x, y) of the 8 pairs */
} fx_rotn;

typedef struct fx_stage {
	cpd din[DK_FX_REGS], dout[DK_FX_REGS];
	uint32_t dinm, doutm, M[DK_FX_BITS];
	int nrot;
	fx_rotn rot[16];
} fx_stage;

#define ALL16 0xffffu
static const uint16_t low_regs[DK_FX_BITS] = { 0x5555, 0x3333, 0x0f0f, 0x00ff };

/* The set with every register p replaced by p ^ v. */
static uint32_t move16(uint32_t m, unsigned v)
{
	for (int j = 0; j < DK_FX_BITS; j++)
		if (v >> j & 1u)
			m = (m & low_regs[j]) << (1 << j) | (m >> (1 << j) & low_regs[j]);
	return m;
}

static unsigned label(const fx_stage *s, unsigned p)
{
	unsigned l = 0;
	for (int j = 0; j < DK_FX_BITS; j++)
		l |= (s->M[j] >> p & 1u) << j;
	return l;
}

/* The register that holds pass index l. */
static unsigned reg_of(const fx_stage *s, unsigned l)
{
	uint32_t m = ALL16;
	for (int j = 0; j < DK_FX_BITS; j++)
		m &= l >> j & 1u ? s->M[j] : ~s->M[j];
	return (unsigned)__builtin_ctz(m);
}

static unsigned direction(const fx_stage *s, int bit) { return reg_of(s, 0) ^ reg_of(s, 1u << bit); }

/* `cols`: the pass index that register 1 << j holds at the start (linear) */
static void stage_init(fx_stage *s, const uint8_t *cols)
{
	for (int j = 0; j < DK_FX_BITS; j++) {
		s->M[j] = 0;
		for (int i = 0; i < DK_FX_BITS; i++)
			if (cols[i] >> j & 1)
				s->M[j] ^= ALL16 & ~(uint32_t)low_regs[i];
	}
	s->dinm = s->doutm = 0;
	s->nrot = 0;
}

/* d[p] *= u for the registers of m */
static void mul_on(cpd *d, uint32_t *dm, uint32_t m, cpd u)
{
	if (deq(u, d_one))
		return;
	for (uint32_t x = m; x; x &= x - 1) {
		const int p = __builtin_ctz(x);
		d[p] = *dm >> p & 1u ? dmul(d[p], u) : u;
	}
	*dm |= m;
}

static void put_diag(fx_buf *b, const cpd *d, uint32_t dm)
{
	double *c = new_coef(b, 2 * DK_FX_REGS);
	for (int p = 0; c && p < DK_FX_REGS; p++) {
		const cpd v = dm >> p & 1u ? d[p] : d_one;
		c[2 * p] = v.x;
		c[2 * p + 1] = v.y;
	}
}

/* A diagonal product (1 outside dm) as one operation; a product of several
 * values is left to the caller's stage when `full` is given. */
static void emit_diag(fx_buf *b, const cpd *d, uint32_t dm, uint32_t lc, uint32_t la, int *full)
{
	cpd u = d_one;
	uint32_t mask = 0;
	int one = 1;
	if (full)
		*full = 0;
	for (uint32_t x = dm; x && one; x &= x - 1) {
		const int p = __builtin_ctz(x);
		if (deq(d[p], d_one))
			continue;
		if (!mask)
			u = d[p];
		one = deq(d[p], u);
		mask |= 1u << p;
	}
	if (one && !mask)
		return;
	if (one && u.x == -1 && u.y == 0) {
		new_op(b, DK_FX_NEG, mask, lc, la);
		return;
	}
	if (one && (popc(mask) <= DK_FX_REGS / 2 || !full)) {
		double *c;
		if (new_op(b, DK_FX_PHASE, mask, lc, la) && (c = new_coef(b, 2)) != NULL) {
			c[0] = u.x;
			c[1] = u.y;
		}
		return;
	}
	if (full) {
		*full = 1;
		return;
	}
	if (new_op(b, DK_FX_STAGE, 16, lc, la)) {
		double *c = new_coef(b, 8);
		if (c)
			memset(c, 0, 8 * sizeof(double));
		put_diag(b, d, dm);
	}
}

static void emit_rot(fx_buf *b, const fx_rotn *r, uint32_t lc, uint32_t la)
{
	if (!new_op(b, r->plain ? DK_FX_STAGE : DK_FX_ROT + r->dir, r->plain ? r->dir : 0, lc, la))
		return;
	double *c = new_coef(b, r->plain ? 8 : 16);
	for (int i = 0; c && i < (r->plain ? 8 : 16); i++)
		c[i] = !r->plain ? r->co[i] : i >> 1 == __builtin_ctz(r->dir) ? r->co[i & 1] : 0.0;
}

/* What a rotation adds to register p of register p ^ dir. */
static void rot_coefs(const fx_rotn *r, double *c)
{
	const unsigned dir = r->dir, low = dir & (0u - dir);
	int pr = 0;
	for (unsigned p = 0; p < DK_FX_REGS; p++) {
		if (p & low)
			continue;
		c[p] = r->co[r->plain ? 0 : 2 * pr];
		c[p ^ dir] = r->co[r->plain ? 1 : 2 * pr + 1];
		pr++;
	}
}

/* Two rotations commute where what each adds to a register is the same along the
 * other's direction.  (In one order register p gets a[p] b[p ^ dir a] of register
 * p ^ dir a ^ dir b, in the other b[p] a[p ^ dir b].)  Plain ones along two register
 * bits do; one along several bits, a CNOT's control and target, say, changes sides
 * under a plain one along either. */
static int rots_commute(const fx_rotn *a, const fx_rotn *b)
{
	if (a->plain && b->plain && a->dir != b->dir)
		return 1;
	double ca[DK_FX_REGS], cb[DK_FX_REGS];
	rot_coefs(a, ca);
	rot_coefs(b, cb);
	for (unsigned p = 0; p < DK_FX_REGS; p++)
		if (ca[p] != ca[p ^ b->dir] || cb[p] != cb[p ^ a->dir])
			return 0;
	return 1;
}

/* diag(din) and the stage's rotations: the plain ones that commute with those
 * before them in one operation with the product, the others in order. */
static void emit_stage(fx_buf *b, const fx_stage *s)
{
	int full, first[4] = { -1, -1, -1, -1 }, rest = 0;
	emit_diag(b, s->din, s->dinm, 0, 0, &full);
	unsigned mask = full ? 16u : 0u;
	for (int i = 0; i < s->nrot; i++) {
		const int j = __builtin_ctz(s->rot[i].dir);
		int ahead = s->rot[i].plain && first[j] < 0;
		for (int k = 0; k < i && ahead; k++)
			if (rest >> k & 1)
				ahead = rots_commute(&s->rot[k], &s->rot[i]);
		if (ahead) {
			first[j] = i;
			mask |= 1u << j;
		} else {
			rest |= 1 << i;
		}
	}
	if (mask && new_op(b, DK_FX_STAGE, mask, 0, 0)) {
		double *c = new_coef(b, 8);
		for (int i = 0; c && i < 8; i++)
			c[i] = first[i >> 1] >= 0 ? s->rot[first[i >> 1]].co[i & 1] : 0.0;
		if (full)
			put_diag(b, s->din, s->dinm);
	}
	for (int i = 0; i < s->nrot; i++)
		if (rest >> i & 1)
			emit_rot(b, &s->rot[i], 0, 0);
}

/* Emit din and the rotations; dout becomes the next stage's din. */
static void stage_flush(fx_buf *b, fx_stage *s)
{
	if (s->nrot) {
		emit_stage(b, s);
		s->nrot = 0;
		s->dinm = 0;
	}
	for (uint32_t x = s->doutm; x; x &= x - 1) {
		const int p = __builtin_ctz(x);
		s->din[p] = s->dinm >> p & 1u ? dmul(s->din[p], s->dout[p]) : s->dout[p];
	}
	s->dinm |= s->doutm;
	s->doutm = 0;
}

/* Emit everything pending: the registers hold the amplitudes themselves. */
static void stage_drain(fx_buf *b, fx_stage *s)
{
	stage_flush(b, s);
	emit_diag(b, s->din, s->dinm, 0, 0, NULL);
	s->dinm = 0;
}

/* The set of pairs (by number) of direction v whose registers are in `sel`. */
static uint32_t pairs_of(uint32_t sel, unsigned v)
{
	const unsigned low = v & (0u - v);
	uint32_t mask = 0;
	int pr = 0;
	for (unsigned p = 0; p < DK_FX_REGS; p++) {
		if (p & low)
			continue;
		mask |= (sel >> p & 1u) << pr;
		pr++;
	}
	return mask;
}

/* The registers of `sel` (closed under the direction of bit b) trade places
 * along it: a relabelling when that is affine, else an exchange. */
static void stage_x(fx_buf *b, fx_stage *s, int bit, uint32_t sel, int affine)
{
	if (affine) {
		s->M[bit] ^= sel;
		return;
	}
	stage_flush(b, s);
	const unsigned v = direction(s, bit), low = v & (0u - v);
	for (unsigned p = 0; p < DK_FX_REGS; p++) {
		if ((p & low) || !(sel >> p & 1u))
			continue;
		const uint32_t i = s->dinm >> p & 1u, j = s->dinm >> (p ^ v) & 1u;
		const cpd t = s->din[p];
		s->din[p] = s->din[p ^ v];
		s->din[p ^ v] = t;
		s->dinm = (s->dinm & ~(1u << p | 1u << (p ^ v))) | j << p | i << (p ^ v);
	}
	new_op(b, DK_FX_SWAP + v, pairs_of(sel, v), 0, 0);
}

/* The gate's rotation on the registers of `sel`. */
static void set_rot(fx_rotn *r, const fx_stage *s, const fx_gate *g, int bit, uint32_t sel, unsigned v)
{
	const unsigned low = v & (0u - v);
	r->dir = (uint8_t)v;
	r->plain = 0;
	if (v == low && sel == ALL16) {
		/* one bit, every register: plain when all pairs have the same of the
		 * two orders */
		const uint32_t first = low_regs[__builtin_ctz(v)], hi = s->M[bit] & first;
		if (hi == 0 || hi == first) {
			r->plain = 1;
			r->co[0] = hi ? g->dt : -g->ds;
			r->co[1] = hi ? -g->ds : g->dt;
			return;
		}
	}
	int pr = 0;
	for (unsigned p = 0; p < DK_FX_REGS; p++) {
		if (p & low)
			continue;
		const int on = sel >> p & 1u, hi = s->M[bit] >> p & 1u;
		r->co[2 * pr] = !on ? 0.0 : hi ? g->dt : -g->ds;
		r->co[2 * pr + 1] = !on ? 0.0 : hi ? -g->ds : g->dt;
		pr++;
	}
}

/* One gate into a pass's list.  treg: register bits of its targets; cr / ar:
 * its controls among the pass bits; lc / la: its controls on other tile
 * bits. */
static void add_gate(fx_buf *b, fx_stage *s, const dk_flat_op *op, const fx_gate *g,
		     const int *treg, uint32_t cr, uint32_t ar, uint32_t lc, uint32_t la)
{
	uint32_t sel = ALL16; /* registers whose controls hold */
	for (int j = 0; j < DK_FX_BITS; j++) {
		if (cr >> j & 1u)
			sel &= s->M[j];
		if (ar >> j & 1u)
			sel &= ~s->M[j];
	}
	const int bit = treg[0];
	if (g->kind == FX_DIAG) {
		cpd d[DK_FX_REGS], *to = s->dout;
		uint32_t dm = 0, *tom = &s->doutm;
		if (lc | la) {
			stage_flush(b, s);
			to = d;
			tom = &dm;
		}
		if (op->k == 1) {
			mul_on(to, tom, sel & ~s->M[bit], g->d0);
			mul_on(to, tom, sel & s->M[bit], g->d1);
		} else {
			const double *m = op->gate->m;
			const uint64_t dim = op->gate->dim;
			for (uint64_t e = 0; e < dim; e++) {
				uint32_t on = sel;
				for (unsigned t = 0; t < op->k; t++)
					on &= e >> t & 1u ? s->M[treg[t]] : ~s->M[treg[t]];
				mul_on(to, tom, on,
				       (cpd){ m[2 * (e * dim + e)], m[2 * (e * dim + e) + 1] });
			}
		}
		if (lc | la)
			emit_diag(b, d, dm, lc, la, NULL);
		return;
	}
	if (lc | la) {
		/* per thread: nothing may be left pending along the way */
		stage_drain(b, s);
		const unsigned v = direction(s, bit);
		cpd d[DK_FX_REGS];
		uint32_t dm = 0;
		if (g->kind == FX_PERM || g->flip)
			new_op(b, DK_FX_SWAP + v, pairs_of(sel, v), lc, la);
		if (g->kind == FX_ROT) {
			fx_rotn r;
			mul_on(d, &dm, sel & s->M[bit], g->dr);
			emit_diag(b, d, dm, lc, la, NULL);
			set_rot(&r, s, g, bit, sel, v);
			emit_rot(b, &r, lc, la);
			dm = 0;
		}
		mul_on(d, &dm, sel & ~s->M[bit], g->d0);
		mul_on(d, &dm, sel & s->M[bit], g->d1);
		emit_diag(b, d, dm, lc, la, NULL);
		return;
	}
	if (g->kind == FX_PERM || g->flip)
		stage_x(b, s, bit, sel, popc(cr | ar) <= 1);
	const uint32_t hi = sel & s->M[bit], lo = sel & ~s->M[bit];
	if (g->kind == FX_ROT) {
		const unsigned v = direction(s, bit);
		/* into the open stage when the right factor passes its rotations
		 * and the rotation its trailing product */
		int join = s->nrot > 0 && s->nrot < 16;
		if (join && s->doutm) {
			join = move16(s->doutm, v) == s->doutm;
			for (uint32_t x = s->doutm; join && x; x &= x - 1) {
				const int p = __builtin_ctz(x);
				join = deq(s->dout[p], s->dout[(unsigned)p ^ v]);
			}
		}
		for (int i = 0; join && i < s->nrot && !deq(g->dr, d_one); i++)
			join = move16(hi, s->rot[i].dir) == hi;
		if (!join)
			stage_flush(b, s);
		mul_on(s->din, &s->dinm, hi, g->dr);
		set_rot(&s->rot[s->nrot++], s, g, bit, sel, v);
	}
	/* a common factor goes in front of the rotations, to the product that
	 * is there in any case */
	if (sel == ALL16 && deq(g->d0, g->d1)) {
		mul_on(s->din, &s->dinm, ALL16, g->d0);
		return;
	}
	mul_on(s->dout, &s->doutm, lo, g->d0);
	mul_on(s->dout, &s->doutm, hi, g->d1);
}

/* ---- one sweep ------------------------------------------------------------ */

/* A gate of a pass. */
typedef struct listed {
	int id, cond; /* its tile condition among the pass's, -1: none */
	int treg[DK_SWEEP_MAX_K];
	uint32_t cr, ar, lc, la;
} listed;

/* At most DK_FX_COND past the program's limit, which the caller checks. */
static int find_cond(fx_buf *b, uint64_t gc, uint64_t ga)
{
	for (int i = 0; i < b->ncond; i++)
		if (b->cond[i].gc == gc && b->cond[i].ga == ga)
			return i;
	b->cond[b->ncond].gc = gc;
	b->cond[b->ncond].ga = ga;
	return b->ncond++;
}

/* tile bits of residue r mod sw, sw = 3 and 4 */
static const uint16_t residue[2][4] = { { 0x9249, 0x2492, 0x4924, 0 },
					{ 0x1111, 0x2222, 0x4444, 0x8888 } };

/* Thread bits of a pass: lanes first, the low ones on tile bits of distinct
 * residues mod sw where there are such, then the phase's warp bits. */
static int lane_order(uint32_t L, uint32_t W, int sw, uint8_t *lane)
{
	int nl = 0;
	uint32_t left = L;
	for (int r = 0; r < sw; r++) {
		const uint32_t x = left & residue[sw - 3][r];
		if (x) {
			lane[nl++] = (uint8_t)__builtin_ctz(x);
			left &= ~(x & (0u - x));
		}
	}
	const int distinct = nl;
	for (; left; left &= left - 1)
		lane[nl++] = (uint8_t)__builtin_ctz(left);
	for (; W; W &= W - 1)
		lane[nl++] = (uint8_t)__builtin_ctz(W);
	return distinct;
}

static int residues(uint32_t L, int sw)
{
	int n = 0;
	for (int r = 0; r < sw; r++)
		n += (L & residue[sw - 3][r]) != 0;
	return n;
}

/* Passes [p0, p1), whose target bits fit in m - wbits tile bits: complete
 * their bits, pick the warp bits they share, and lay out their threads. */
static void lay_out_phase(dk_fx_plan *P, int p0, int p1, int m, int wbits, int sw,
			  uint8_t (*lanes)[16], int *conflicts)
{
	const uint32_t all = (1u << m) - 1u;
	uint32_t F = 0;
	for (int i = p0; i < p1; i++)
		F |= P->need[i];
	for (int b = m - 1; popc(F) < DK_FX_BITS && b >= 0; b--)
		F |= 1u << b;
	for (int i = p0; i < p1; i++) {
		uint32_t B = P->need[i];
		for (int b = m - 1; popc(B) < DK_FX_BITS && b >= 0; b--)
			if (F >> b & 1u)
				B |= 1u << b;
		P->need[i] = B;
	}
	/* the last pass wants the lowest two tile bits on its lanes (a 64- or
	 * 32-byte run of the register): they stay out of the warp bits */
	uint32_t pool = all & ~F;
	if (popc(pool & ~3u) >= wbits)
		pool &= ~3u;
	uint32_t W = 0;
	int best = -1;
	for (uint32_t x = pool; best < sw * (p1 - p0); x = (x - 1) & pool) {
		if (popc(x) == wbits) {
			int sc = 0;
			for (int i = p0; i < p1; i++)
				sc += residues(all & ~P->need[i] & ~x, sw);
			if (sc > best) {
				best = sc;
				W = x;
			}
		}
		if (x == 0)
			break;
	}
	for (int i = p0; i < p1; i++) {
		dk_fx_pass *pd = &P->pass[i];
		const uint32_t B = P->need[i];
		int j = 0;
		for (int b = 0; b < m; b++)
			if (B >> b & 1u)
				P->pbits[i][j++] = (uint8_t)b;
		if (lane_order(all & ~B & ~W, W, sw, lanes[i]) < sw)
			*conflicts = 1;
		if (i + 1 < p1)
			pd->flags |= DK_PASS_WARP;
	}
}

static void pass_tables(dk_fx_pass *pd, uint32_t *sp, const uint8_t *pb, const uint8_t *lane,
			int m, const unsigned *F, unsigned amp)
{
	/* slot of a tile index: its bits above sw keep their place, the low ones
	 * take the bank directions; both are linear, so tables add up by XOR */
	uint32_t slot[16];
	for (int b = 0; b < m; b++)
		slot[b] = amp * (F[b] | (F[b] >> b & 1u ? 0u : 1u << b));
	for (int j = 0; j < DK_FX_BITS; j++) {
		pd->pm[j] = (uint16_t)(1u << pb[j]);
		sp[j] = slot[pb[j]];
	}
	const int nl = m - DK_FX_BITS;
	pd->rlo[0] = pd->slo[0] = pd->rhi[0] = pd->shi[0] = 0;
	for (uint32_t x = 1; x < 32; x++) {
		const int b = __builtin_ctz(x);
		pd->rlo[x] = (uint16_t)(pd->rlo[x & (x - 1)] | (b < nl ? 1u << lane[b] : 0u));
		pd->slo[x] = (uint16_t)(pd->slo[x & (x - 1)] ^ (b < nl ? slot[lane[b]] : 0u));
	}
	for (uint32_t x = 1; x < 8; x++) {
		const int b = 5 + __builtin_ctz(x);
		pd->rhi[x] = (uint16_t)(pd->rhi[x & (x - 1)] | (b < nl ? 1u << lane[b] : 0u));
		pd->shi[x] = (uint16_t)(pd->shi[x & (x - 1)] ^ (b < nl ? slot[lane[b]] : 0u));
	}
}

static size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

/* The coefficient tables in the program's precision, and the operations'
 * offsets into them in 16-byte units. */
static void put_coefs(fx_buf *b, int prec, unsigned char *dst)
{
	size_t at = 0;
	for (int i = 0; i < b->nop; i++) {
		dk_fx_op *o = &b->op[i];
		const size_t bytes = op_bytes(o, prec);
		if (!bytes) {
			o->coef = 0;
			continue;
		}
		const double *src = b->coef + o->coef;
		if (prec == DK_C128) {
			memcpy(dst + at, src, bytes);
		} else {
			/* reals twice, a diagonal's values as they are */
			float *f = (float *)(dst + at);
			int reals = 0, diag = 0;
			if (o->code == DK_FX_STAGE) {
				reals = 8;
				diag = o->mask & 16u ? 2 * DK_FX_REGS : 0;
			} else if (o->code == DK_FX_PHASE) {
				diag = 2;
				f[2] = f[3] = 0.0f;
			} else {
				reals = 16;
			}
			for (int j = 0; j < reals; j++)
				f[2 * j] = f[2 * j + 1] = (float)src[j];
			for (int j = 0; j < diag; j++)
				f[2 * reals + j] = (float)src[reals + j];
		}
		o->coef = (uint32_t)(at / 16);
		at += bytes;
	}
}

/* Columns of the inverse of a 4x4 matrix over GF(2) given by rows. */
static void invert4(const uint8_t *rows, uint8_t *cols)
{
	uint8_t a[4], inv[4]; /* inv: rows of the inverse */
	for (int j = 0; j < 4; j++) {
		a[j] = rows[j];
		inv[j] = (uint8_t)(1u << j);
	}
	for (int c = 0; c < 4; c++) {
		int p = c;
		while (!(a[p] >> c & 1))
			p++;
		uint8_t t = a[c];
		a[c] = a[p];
		a[p] = t;
		t = inv[c];
		inv[c] = inv[p];
		inv[p] = t;
		for (int r = 0; r < 4; r++)
			if (r != c && (a[r] >> c & 1)) {
				a[r] ^= a[c];
				inv[r] ^= inv[c];
			}
	}
	for (int j = 0; j < 4; j++) {
		cols[j] = 0;
		for (int r = 0; r < 4; r++)
			cols[j] |= (uint8_t)((inv[r] >> j & 1) << r);
	}
}

/* Bytes that a program may have. */
static size_t program_cap(unsigned n, int m)
{
	return n <= (unsigned)m + DK_FX_SMALL_TILES ? DK_FX_BYTES_SMALL : DK_FX_BYTES;
}

/* Emit the sweep of `cnt` gates (P->take) over Q; gates of passes that no
 * longer fit the program stay in P->take (P->nleft of them). */
static int emit(dk_fx_plan *P, int cnt, uint64_t Q, int m, dk_step *step,
		const unsigned char **prog)
{
	const unsigned n = P->n;
	const int sw = P->prec == DK_C64 ? 4 : 3;
	uint8_t qpos[16];
	int8_t loc[64];
	int nq = 0;
	memset(loc, -1, sizeof(loc));
	for (unsigned q = 0; q < n; q++)
		if (Q >> q & 1u) {
			loc[q] = (int8_t)nq;
			qpos[nq++] = (uint8_t)q;
		}
	/* group the gates into passes */
	int npass = 0, nord = 0, nrem = cnt;
	int *rem = P->take;
	while (nrem > 0) {
		if (npass == P->cpass)
			return DK_ERR_ALLOC;
		dk_fx_pass *pd = &P->pass[npass];
		memset(pd, 0, sizeof(*pd));
		uint32_t B = 0;
		uint64_t blocked = 0, gcs[DK_FX_COND], gas[DK_FX_COND];
		int nd = 0, i, nc = 0;
		P->range[npass][0] = (uint16_t)nord;
		for (i = 0; i < nrem && i < FX_WINDOW; i++) {
			const int id = rem[i];
			const fx_gate *g = &P->g[id];
			int ok = !(g->sup & blocked);
			if (ok) {
				uint32_t tl = 0, sl;
				for (uint64_t x = g->tmask; x; x &= x - 1)
					tl |= 1u << loc[__builtin_ctzll(x)];
				sl = tl;
				for (uint64_t x = g->ctl & Q; x; x &= x - 1)
					sl |= 1u << loc[__builtin_ctzll(x)];
				if (popc(sl) <= DK_FX_BITS)
					tl = sl;
				ok = popc(B | tl) <= DK_FX_BITS;
				const uint64_t gc = P->ops[id].cm & ~Q, ga = P->ops[id].am & ~Q;
				if (ok && (gc | ga)) {
					int c = 0;
					while (c < nc && (gcs[c] != gc || gas[c] != ga))
						c++;
					if (c == nc) {
						if (nc == DK_FX_COND) {
							ok = 0;
						} else {
							gcs[nc] = gc;
							gas[nc++] = ga;
						}
					}
				}
				if (ok)
					B |= tl;
			}
			if (ok) {
				P->order[nord++] = id;
			} else {
				rem[nd++] = id;
				blocked |= g->sup;
			}
		}
		if (i < nrem)
			memmove(rem + nd, rem + i, sizeof(int) * (size_t)(nrem - i));
		nrem = nd + nrem - i;
		P->range[npass][1] = (uint16_t)nord;
		P->need[npass] = B;
		npass++;
	}
	/* phases: passes that keep their warp bits need a warp barrier only */
	const int wbits = m > DK_FX_BITS + 5 ? m - DK_FX_BITS - 5 : 0;
	uint8_t lanes[DK_MAX_FX_PASSES][16];
	int conflicts = 0;
	for (int p0 = 0; p0 < npass;) {
		int p1 = p0 + 1;
		uint32_t U = P->need[p0];
		while (p1 < npass && popc(U | P->need[p1]) <= m - wbits)
			U |= P->need[p1++];
		lay_out_phase(P, p0, p1, m, wbits, sw, lanes, &conflicts);
		p0 = p1;
	}
	unsigned F[16];
	for (int b = 0; b < m; b++)
		F[b] = 1u << (b % sw);
	if (conflicts && n >= DK_FX_MAP_QUBITS) {
		/* some pass has no lanes on sw distinct residues: search a map */
		dk_bank_pat pat[DK_MAX_FX_PASSES];
		for (int i = 0; i < npass; i++) {
			pat[i].w = 1;
			pat[i].nb = sw;
			for (int j = 0; j < sw; j++)
				pat[i].b[j] = lanes[i][j];
		}
		dk_choose_bank_map(pat, npass, m, sw, F);
	}
	for (int i = 0; i < npass; i++)
		pass_tables(&P->pass[i], P->sp[i], P->pbits[i], lanes[i], m, F,
			    P->prec == DK_C64 ? 8u : 16u);

	/* operation lists, pass by pass while the program has room */
	fx_buf *b = &P->b;
	b->nop = b->nlist = b->ncond = b->oom = 0;
	b->bytes = 0;
	b->prec = P->prec;
	b->ncoef = 0;
	int all_touched = 0, done = 0;
	const size_t cap = program_cap(n, m);
	for (int i = 0; i < npass; i++) {
		dk_fx_pass *pd = &P->pass[i];
		const int nop0 = b->nop, nlist0 = b->nlist, ncond0 = b->ncond;
		const size_t ncoef0 = b->ncoef, bytes0 = b->bytes;
		int preg[16], touched = 0;
		memset(preg, -1, sizeof(preg));
		for (int r = 0; r < DK_FX_BITS; r++)
			preg[P->pbits[i][r]] = r;
		/* the pass's conditions */
		uint64_t gcs[DK_FX_COND], gas[DK_FX_COND];
		int nc = 0, np = 0;
		listed pg[FX_WINDOW]; /* its gates, with their register bits */
		pd->cond = 0;
		pd->list = (uint32_t)b->nlist;
		for (int k = P->range[i][0]; k < P->range[i][1]; k++) {
			const int id = P->order[k];
			const dk_flat_op *op = &P->ops[id];
			listed *e = &pg[np++];
			memset(e, 0, sizeof(*e));
			e->id = id;
			e->cond = -1;
			for (unsigned t = 0; t < op->k; t++)
				e->treg[t] = preg[loc[op->tg[t]]];
			for (uint64_t x = P->g[id].ctl & Q; x; x &= x - 1) {
				const int q = __builtin_ctzll(x), l = loc[q];
				const int anti = op->am >> q & 1u;
				if (preg[l] >= 0)
					*(anti ? &e->ar : &e->cr) |= 1u << preg[l];
				else
					*(anti ? &e->la : &e->lc) |= 1u << l;
			}
			if (e->lc | e->la)
				pd->flags |= DK_PASS_CTL;
			const uint64_t gc = op->cm & ~Q, ga = op->am & ~Q;
			int c = 0;
			if (!(gc | ga)) {
				touched = 1;
				continue;
			}
			while (c < nc && (gcs[c] != gc || gas[c] != ga))
				c++;
			if (c == nc) {
				gcs[nc] = gc;
				gas[nc] = ga;
				pd->cond |= (uint32_t)find_cond(b, gc, ga) << (5 * nc++);
			}
			e->cond = c;
		}
		pd->cond |= (uint32_t)nc << 15;
		if (grow((void **)&b->list, sizeof(dk_fx_list), &b->clist, b->nlist + (1 << nc)))
			return DK_ERR_ALLOC;
		for (int v = 0; v < 1 << nc; v++) {
			dk_fx_list *li = &b->list[b->nlist++];
			const listed *gl[FX_WINDOW];
			int ng = 0;
			for (int k = 0; k < np; k++)
				if (pg[k].cond < 0 || (v >> pg[k].cond & 1))
					gl[ng++] = &pg[k];
			/* CNOTs relabel the registers: the gather starts from the labels
			 * under which the most rotations run along a register bit.  rows:
			 * the linear part of register -> pass index so far, by rows */
			uint8_t rows[DK_FX_BITS], best[DK_FX_BITS], cols[DK_FX_BITS];
			for (int j = 0; j < DK_FX_BITS; j++)
				rows[j] = best[j] = cols[j] = (uint8_t)(1u << j);
			int cnt = 0, most = 0, moved = 0;
			for (int k = 0; k < ng; k++) {
				const fx_gate *g = &P->g[gl[k]->id];
				const uint32_t c = gl[k]->cr | gl[k]->ar;
				if (gl[k]->lc | gl[k]->la)
					continue;
				if ((g->kind == FX_PERM || (g->kind == FX_ROT && g->flip)) && popc(c) == 1) {
					if (cnt > most) {
						most = cnt;
						memcpy(best, rows, sizeof(best));
					}
					cnt = 0;
					rows[gl[k]->treg[0]] ^= rows[__builtin_ctz(c)];
					moved = 1;
				}
				cnt += g->kind == FX_ROT;
			}
			if (cnt > most)
				memcpy(best, rows, sizeof(best));
			if (moved)
				invert4(best, cols);
			fx_stage s;
			stage_init(&s, cols);
			uint32_t gt[DK_FX_BITS];
			for (int j = 0; j < DK_FX_BITS; j++) {
				gt[j] = 0;
				for (int x = 0; x < DK_FX_BITS; x++)
					if (cols[j] >> x & 1)
						gt[j] ^= P->sp[i][x];
			}
			li->pad = 0;
			li->op0 = (uint16_t)b->nop;
			for (int k = 0; k < ng; k++)
				add_gate(b, &s, &P->ops[gl[k]->id], &P->g[gl[k]->id], gl[k]->treg,
					 gl[k]->cr, gl[k]->ar, gl[k]->lc, gl[k]->la);
			stage_drain(b, &s);
			unsigned l0 = label(&s, 0), same = l0 == 0;
			li->lmap = (uint32_t)l0 << 16;
			li->sc = 0;
			for (int j = 0; j < DK_FX_BITS; j++) {
				const unsigned lj = label(&s, 1u << j) ^ l0;
				uint32_t st = 0;
				for (int x = 0; x < DK_FX_BITS; x++) {
					if (lj >> x & 1u)
						st ^= P->sp[i][x];
				}
				if (l0 >> j & 1u)
					li->sc ^= (uint16_t)P->sp[i][j];
				same &= st == gt[j];
				li->gt[j] = (uint16_t)gt[j];
				li->st[j] = (uint16_t)st;
				li->lmap |= (uint32_t)lj << (4 * j);
			}
			li->op1 = (uint16_t)b->nop;
			li->idle = same && li->op0 == li->op1;
		}
		const size_t bytes = sizeof(dk_sweep_hdr) + sizeof(dk_fx_pass) * (size_t)(i + 1) +
				     sizeof(dk_fx_list) * (size_t)b->nlist + b->bytes +
				     sizeof(dk_gate_cond) * (size_t)b->ncond;
		if (b->oom)
			return DK_ERR_ALLOC;
		if (bytes > cap || b->ncond > DK_FX_MAX_CONDS) {
			b->nop = nop0;
			b->nlist = nlist0;
			b->ncond = ncond0;
			b->ncoef = ncoef0;
			b->bytes = bytes0;
			const int k0 = P->range[i][0], k1 = P->range[i][1];
			if (i > 0 || k1 - k0 == 1)
				break; /* the other gates make another program */
			/* one pass too long for a program: its first half */
			P->range[i][1] = (uint16_t)(k0 + (k1 - k0) / 2);
			npass = 1;
			pd->flags = 0;
			i--;
			continue;
		}
		all_touched |= touched;
		done = i + 1;
	}
	if (done == 0)
		return DK_ERR_ARG; /* cannot happen: one gate's lists always fit */
	P->nleft = 0;
	for (int k = P->range[done - 1][1]; k < nord; k++)
		P->take[P->nleft++] = P->order[k];
	P->leftQ = Q;
	{
		dk_fx_pass *last = &P->pass[done - 1];
		uint32_t lb = 0;
		for (int j = 0; j < 5; j++)
			lb |= last->rlo[1u << j];
		last->flags &= ~(uint32_t)DK_PASS_WARP;
		if ((lb & 3u) == 3u)
			last->flags |= DK_FX_STORE;
	}

	const size_t pass_off = sizeof(dk_sweep_hdr);
	const size_t list_off = pass_off + sizeof(dk_fx_pass) * (size_t)done;
	const size_t gate_off = list_off + sizeof(dk_fx_list) * (size_t)b->nlist;
	const size_t cond_off = gate_off + sizeof(dk_fx_op) * (size_t)b->nop;
	const size_t mat_off = align16(cond_off + sizeof(dk_gate_cond) * (size_t)b->ncond);
	const size_t bytes = align16(mat_off + b->bytes - sizeof(dk_fx_op) * (size_t)b->nop);
	if (bytes > P->cprog) {
		unsigned char *np = (unsigned char *)realloc(P->prog, 2 * bytes);
		if (!np)
			return DK_ERR_ALLOC;
		P->prog = np;
		P->cprog = 2 * bytes;
	}
	dk_sweep_hdr *h = (dk_sweep_hdr *)P->prog;
	memset(h, 0, sizeof(*h));
	h->m = m;
	h->n = (int32_t)n;
	h->npass = done;
	h->ngate = b->nop;
	h->all_touched = all_touched;
	h->mode = DK_SWEEP_FACTORED;
	h->ntiles = UINT64_C(1) << (n - (unsigned)m);
	memcpy(h->qpos, qpos, (size_t)m);
	h->pass_off = (uint32_t)pass_off;
	h->gate_off = (uint32_t)gate_off;
	h->cond_off = (uint32_t)cond_off;
	h->mat_off = (uint32_t)mat_off;
	h->bytes = (uint32_t)bytes;
	h->ncond = (uint32_t)b->ncond;
	for (int i = sw; i < m; i++)
		h->bankv |= (uint64_t)F[i] << (4 * i);
	put_coefs(b, P->prec, P->prog + mat_off);
	memcpy(P->prog + pass_off, P->pass, sizeof(dk_fx_pass) * (size_t)done);
	memcpy(P->prog + list_off, b->list, sizeof(dk_fx_list) * (size_t)b->nlist);
	if (b->nop)
		memcpy(P->prog + gate_off, b->op, sizeof(dk_fx_op) * (size_t)b->nop);
	memcpy(P->prog + cond_off, b->cond, sizeof(dk_gate_cond) * (size_t)b->ncond);
	step->kind = 1;
	step->prog_off = 0;
	step->op_index = -1;
	step->ngates = P->range[done - 1][1] + P->ngone;
	P->ngone = 0;
	*prog = P->prog;
	return DK_OK;
}

/* What an uncontrolled one-qubit gate can hand on to the next such gate on
 * its qubit, given the gates in between. */
enum { PUSH_NONE = 0, PUSH_Z, PUSH_X, PUSH_ALL };

/* m as Rx(a) W with W = k [[1, -t], [t, 1]] diag(1, r1), |t| <= 1 (m a
 * multiple of a unitary).  With the first column (A, B): A + B and A - B are
 * multiples of exp(-i a) and exp(i a).  0 when t is not real (rx and *g are then
 * void). */
static int split_x(const cpx *m, cpx *rx, fx_gate *g)
{
	const cpx p = cx(m[0].x + m[2].x, m[0].y + m[2].y), q = cx(m[0].x - m[2].x, m[0].y - m[2].y);
	cpx z = cx(p.x * q.x + p.y * q.y, p.y * q.x - p.x * q.y), e = c_one; /* exp(-2 i a) */
	const real r = sqrtl(cabs2(z));
	if (r > 0) {
		z = cx(z.x / r, z.y / r);
		if (z.x >= 0) {
			e.x = sqrtl((1 + z.x) / 2);
			e.y = z.y / (2 * e.x);
		} else {
			e.y = sqrtl((1 - z.x) / 2);
			e.x = fabsl(z.y) / (2 * e.y);
			if (z.y < 0)
				e.y = -e.y;
		}
	}
	/* Rx(a) = [[c, -i s], [-i s, c]], exp(-i a) = c - i s = e */
	const cpx c = cx(e.x, 0), is = cx(0, e.y); /* -i s = i e.y */
	rx[0] = rx[3] = c;
	rx[1] = rx[2] = is;
	/* W = Rx(-a) m */
	cpx w[4];
	for (int j = 0; j < 2; j++) {
		const cpx u = cmul(cx(0, -e.y), m[2 + j]), v = cmul(cx(0, -e.y), m[j]);
		w[j] = cx(c.x * m[j].x + u.x, c.x * m[j].y + u.y);
		w[2 + j] = cx(v.x + c.x * m[2 + j].x, v.y + c.x * m[2 + j].y);
	}
	const cpx r1 = cdiv(w[3], w[0]);
	g->kind = FX_ROT;
	g->flip = 0;
	g->l0 = g->l1 = w[0];
	g->r1 = r1;
	const cpx t = cdiv(w[2], w[0]), s = cdiv(w[1], cmul(w[0], r1));
	g->t = t.x;
	g->s = -s.x;
	return fabsl(t.y) <= FX_DROP && fabsl(s.y) <= FX_DROP;
}

/* A factor on its way from a gate to a later one on the same qubit. */
typedef struct fx_pending {
	cpx w[4];
	int from; /* the gate that gave it, -1: none on its way */
	cpx whole[4]; /* that gate's matrix with the factor in it */
} fx_pending;

static void set_factors(fx_gate *g, const cpx *m)
{
	factor1(m, g);
	g->known = 1;
}

/* Moves factors of uncontrolled one-qubit gates to the next such gate on the
 * same qubit, where they join its matrix: the whole gate when nothing on the
 * qubit lies in between, its left phase through gates that are diagonal on the
 * qubit (controls among them), a left Rx through X and its controlled forms.
 * What stays is k [[1, -s], [t, 1]] diag(1, r1): one product in front of the
 * rotations of a stage and none behind them.
 *
 * Roundings add up along a run of gates, so a product of matrices that have a
 * factoring need not have one.  A factor is taken only by a gate whose product
 * with it has one; otherwise it goes back into the gate that gave it, and every
 * gate keeps a factoring throughout. */
static int move_factors(dk_fx_plan *P)
{
	uint8_t path[64];
	fx_pending *pend = (fx_pending *)malloc(sizeof(*pend) * P->n);
	if (!pend)
		return DK_ERR_ALLOC;
	memset(path, PUSH_NONE, sizeof(path));
	uint8_t *push = (uint8_t *)P->order; /* nops ints: free until the first sweep */
	for (int i = P->nops - 1; i >= 0; i--) {
		const fx_gate *g = &P->g[i];
		const dk_flat_op *op = &P->ops[i];
		push[i] = PUSH_NONE;
		if (op->k == 1 && !g->ctl) {
			const unsigned q = op->tg[0];
			uint8_t *w = &path[q];
			if (g->kind == FX_DIAG) {
				/* moves as a whole, or stays and stops what comes before it */
				if (g->unitary && (*w == PUSH_ALL || *w == PUSH_Z))
					push[i] = PUSH_ALL;
				else
					*w = PUSH_NONE;
				continue;
			}
			/* multiples of unitaries only: their products keep a factoring,
			 * up to roundings */
			push[i] = g->unitary ? *w : PUSH_NONE;
			*w = g->unitary ? PUSH_ALL : PUSH_NONE;
			continue;
		}
		uint64_t z = g->ctl; /* qubits this gate is diagonal on */
		if (op->k > 1 || g->kind == FX_DIAG) {
			z |= g->tmask;
		} else {
			uint8_t *w = &path[op->tg[0]];
			*w = g->is_x && (*w == PUSH_ALL || *w == PUSH_X) ? PUSH_X : PUSH_NONE;
		}
		for (; z; z &= z - 1) {
			uint8_t *w = &path[__builtin_ctzll(z)];
			*w = *w == PUSH_ALL || *w == PUSH_Z ? PUSH_Z : PUSH_NONE;
		}
	}
	for (unsigned q = 0; q < P->n; q++)
		pend[q].from = -1;
	for (int i = 0; i < P->nops; i++) {
		fx_gate *g = &P->g[i];
		if (P->ops[i].k != 1 || g->ctl)
			continue;
		fx_pending *pd = &pend[P->ops[i].tg[0]];
		if (pd->from < 0 && !push[i])
			continue;
		cpx m[4], *w = pd->w;
		load1(&P->ops[i], m);
		if (pd->from >= 0) {
			cpx t[4];
			for (int r = 0; r < 2; r++)
				for (int c = 0; c < 2; c++) {
					const cpx x = cmul(m[2 * r], w[c]), y = cmul(m[2 * r + 1], w[2 + c]);
					t[2 * r + c] = cx(x.x + y.x, x.y + y.y);
				}
			fx_gate f = *g;
			classify1(t, &f);
			if (f.kind != FX_NONE) {
				*g = f;
				memcpy(m, t, sizeof(m));
				if (!g->known && !push[i])
					set_factors(g, m);
			} else {
				P->g[pd->from].gone = 0;
				set_factors(&P->g[pd->from], pd->whole);
			}
			pd->from = -1;
		}
		if (push[i] == PUSH_NONE)
			continue;
		memcpy(pd->whole, m, sizeof(m));
		if (push[i] == PUSH_ALL) {
			memcpy(w, m, sizeof(m));
			g->gone = 1;
		} else if (push[i] == PUSH_X) {
			if (!split_x(m, w, g)) {
				set_factors(g, m);
				continue;
			}
			g->known = 1;
		} else {
			set_factors(g, m);
			w[0] = c_one;
			w[1] = w[2] = cx(0, 0);
			w[3] = cdiv(g->l1, g->l0);
			g->l1 = g->l0;
		}
		pd->from = i;
	}
	free(pend);
	return DK_OK;
}

/* ---- the plan ------------------------------------------------------------- */

/* Most operations and coefficients (doubles) of a gate in a list: a stage emitted
 * ahead of it (a product or a phase, the rotations along register bits, and one
 * operation for a rotation of its own), the product behind the stage, its exchange
 * and two products around its rotation; and of a list's end. */
#define FX_GATE_OPS 8
#define FX_GATE_COEFS 200
#define FX_LIST_OPS 4
#define FX_LIST_COEFS 90

/* Room for the longest program that the plan can come to: what fits a program, and
 * the pass that no longer does. */
int dk_fx_reserve(dk_fx_plan *P)
{
	fx_buf *b = &P->b;
	if (b->op || P->prog)
		return DK_OK; /* reserved before, or steps made without */
	const int m = P->lim.tile_bits;
	const int lists = P->n > (unsigned)m ? 1 << DK_FX_COND : 1; /* of a pass */
	const size_t cap = program_cap(P->n, m);
	const size_t gates = (size_t)(P->nops < DK_FX_MAX_GATES ? P->nops : DK_FX_MAX_GATES);
	const size_t window = gates < FX_WINDOW ? gates : FX_WINDOW;
	const size_t lops = FX_GATE_OPS * gates + FX_LIST_OPS * gates;
	const size_t lcoefs = FX_GATE_COEFS * gates + FX_LIST_COEFS * gates;
	/* a coefficient takes 4 bytes of a program or more */
	size_t nop = cap / sizeof(dk_fx_op), ncoef = cap / 4, nlist = cap / sizeof(dk_fx_list);
	if (nop > lops * (size_t)lists)
		nop = lops * (size_t)lists;
	if (ncoef > lcoefs * (size_t)lists)
		ncoef = lcoefs * (size_t)lists;
	if (nlist > gates * (size_t)lists)
		nlist = gates * (size_t)lists;
	size_t bytes = sizeof(dk_sweep_hdr) + sizeof(dk_fx_pass) * gates +
		       sizeof(dk_fx_list) * nlist + sizeof(dk_fx_op) * nop + 8 * ncoef +
		       sizeof(b->cond);
	if (bytes > cap)
		bytes = cap;
	nop += (FX_GATE_OPS * window + FX_LIST_OPS) * (size_t)lists;
	ncoef += (FX_GATE_COEFS * window + FX_LIST_COEFS) * (size_t)lists;
	nlist += (size_t)lists;
	b->op = (dk_fx_op *)malloc(sizeof(dk_fx_op) * nop);
	b->coef = (double *)malloc(sizeof(double) * ncoef);
	b->list = (dk_fx_list *)malloc(sizeof(dk_fx_list) * nlist);
	P->prog = (unsigned char *)malloc(bytes);
	if (!b->op || !b->coef || !b->list || !P->prog)
		return DK_ERR_ALLOC;
	b->cop = (int)nop;
	b->ccoef = ncoef;
	b->clist = (int)nlist;
	P->cprog = bytes;
	return DK_OK;
}

int dk_fx_begin(const dk_flat_op *ops, int nops, unsigned n, int prec,
		const dk_plan_limits *lim, dk_fx_plan **out)
{
	dk_fx_plan *P = (dk_fx_plan *)calloc(1, sizeof(*P));
	if (!P)
		return DK_ERR_ALLOC;
	P->ops = ops;
	P->nops = nops;
	P->n = n;
	P->prec = prec;
	P->lim = *lim;
	P->cpass = DK_MAX_FX_PASSES;
	const size_t cnt = (size_t)(nops > 0 ? nops : 1);
	P->g = (fx_gate *)calloc(cnt, sizeof(fx_gate));
	P->rem = (int *)malloc(sizeof(int) * cnt);
	P->take = (int *)malloc(sizeof(int) * cnt);
	P->order = (int *)malloc(sizeof(int) * cnt);
	P->sub_ops = (int *)malloc(sizeof(int) * cnt);
	P->pass = (dk_fx_pass *)malloc(sizeof(dk_fx_pass) * DK_MAX_FX_PASSES);
	P->need = (uint32_t *)malloc(sizeof(uint32_t) * DK_MAX_FX_PASSES);
	P->pbits = malloc(sizeof(*P->pbits) * DK_MAX_FX_PASSES);
	P->range = malloc(sizeof(*P->range) * DK_MAX_FX_PASSES);
	P->sp = malloc(sizeof(*P->sp) * DK_MAX_FX_PASSES);
	if (!P->g || !P->rem || !P->take || !P->order || !P->sub_ops || !P->pass || !P->need ||
	    !P->pbits || !P->range || !P->sp) {
		dk_fx_end(P);
		return DK_ERR_ALLOC;
	}
	int all = lim->tile_bits >= DK_FX_MIN_TILE;
	for (int i = 0; i < nops; i++) {
		analyse(&ops[i], &P->g[i]);
		all &= P->g[i].kind != FX_NONE;
	}
	/* gates that dk_plan.c plans from their matrices take no factor */
	P->all = all;
	if (all && move_factors(P)) {
		dk_fx_end(P);
		return DK_ERR_ALLOC;
	}
	P->nops = 0;
	for (int i = 0; i < nops; i++) {
		fx_gate *g = &P->g[i];
		if (g->gone) {
			P->ngone++;
			continue;
		}
		if (!g->known) {
			cpx mt[4];
			load1(&ops[i], mt);
			set_factors(g, mt);
		}
		g->d0 = cd(g->l0);
		g->d1 = cd(g->l1);
		g->dr = cd(g->r1);
		g->ds = (double)g->s;
		g->dt = (double)g->t;
		P->rem[P->nops++] = i;
	}
	*out = P;
	return DK_OK;
}

int dk_fx_all(const dk_fx_plan *P) { return P->all; }

int dk_fx_left(const dk_fx_plan *P, int *ids)
{
	if (P->all || P->nleft || P->sub_at < P->sub.nsteps)
		return -1;
	memcpy(ids, P->rem + P->head, sizeof(int) * (size_t)(P->nops - P->head));
	return P->nops - P->head;
}

void dk_fx_end(dk_fx_plan *P)
{
	if (!P)
		return;
	free(P->g);
	free(P->rem);
	free(P->take);
	free(P->order);
	free(P->sub_ops);
	free(P->pass);
	free(P->need);
	free(P->pbits);
	free(P->range);
	free(P->sp);
	free(P->b.op);
	free(P->b.coef);
	free(P->b.list);
	free(P->prog);
	dk_plan_free(&P->sub);
	free(P);
}

/* The steps of dk_plan.c for the gates P->take[0 .. cnt), which it gets as a
 * plan of their own. */
static int sub_plan(dk_fx_plan *P, int cnt)
{
	dk_flat_op *f = (dk_flat_op *)malloc(sizeof(dk_flat_op) * (size_t)cnt);
	if (!f)
		return DK_ERR_ALLOC;
	for (int i = 0; i < cnt; i++) {
		f[i] = P->ops[P->take[i]];
		P->sub_ops[i] = P->take[i];
	}
	dk_plan_limits lim = P->lim;
	dk_plan_free(&P->sub);
	P->sub_at = 0;
	const int rc = dk_plan_build(f, cnt, P->n, P->prec, &lim, &P->sub);
	free(f);
	return rc;
}

/* A sweep's gates. */
typedef struct fx_choice {
	uint64_t Q; /* their targets and the pinned low qubits */
	int nt, nd, end; /* P->take, P->order (passed over), the first not looked at */
	int factored;
} fx_choice;

static fx_choice choose(dk_fx_plan *P)
{
	const int m = P->lim.tile_bits;
	int low = P->lim.low_bits;
	if (low > m - DK_SWEEP_MAX_K)
		low = m - DK_SWEEP_MAX_K;
	uint64_t Q = (UINT64_C(1) << (low > 0 ? low : 0)) - 1u, blocked = 0;
	const uint64_t full = P->n >= 64 ? ~UINT64_C(0) : (UINT64_C(1) << P->n) - 1u;
	int nt = 0, nd = 0, factored = m >= DK_FX_MIN_TILE, i;
	int *defer = P->order; /* free until the sweep is emitted */
	for (i = P->head; i < P->nops && blocked != full && nt < DK_FX_MAX_GATES; i++) {
		const int id = P->rem[i];
		const fx_gate *g = &P->g[id];
		const uint64_t nq = Q | g->tmask;
		/* a gate that no sweep runs goes to dk_plan.c by itself */
		const int sweepable = P->ops[id].k <= DK_SWEEP_MAX_K && m >= DK_PASS_BITS;
		if (!sweepable && nt == 0 && nd == 0) {
			P->take[nt++] = id;
			factored = 0;
			i++;
			break;
		}
		if (sweepable && !(g->sup & blocked) && popc(nq) <= m) {
			Q = nq;
			P->take[nt++] = id;
			factored &= g->kind != FX_NONE;
		} else {
			defer[nd++] = id;
			blocked |= g->sup;
		}
	}
	const fx_choice c = { Q, nt, nd, i, factored };
	return c;
}

int dk_fx_next(dk_fx_plan *P, dk_step *step, const unsigned char **prog)
{
	const int m = P->lim.tile_bits;
	for (;;) {
		if (P->sub_at < P->sub.nsteps) {
			*step = P->sub.steps[P->sub_at++];
			*prog = NULL;
			if (step->kind == 1) {
				*prog = P->sub.blob + step->prog_off;
				step->prog_off = 0;
			} else {
				step->op_index = P->sub_ops[step->op_index];
			}
			return 1;
		}
		if (P->nleft) {
			const int rc = emit(P, P->nleft, P->leftQ, m, step, prog);
			return rc ? -rc : 1;
		}
		if (P->head >= P->nops)
			return 0;
		fx_choice c = choose(P);
		/* what was passed over comes right before what was not looked at */
		P->head = c.end - c.nd;
		memcpy(P->rem + P->head, P->order, sizeof(int) * (size_t)c.nd);
		if (!c.factored) {
			/* dk_plan.c sees the gates as they were given: not for a plan
			 * whose gates have taken factors of others */
			if (P->all)
				return -DK_ERR_ARG; /* cannot happen: every gate has a factoring */
			const int rc = sub_plan(P, c.nt);
			if (rc) {
				/* back in front of what was passed over */
				P->head -= c.nt;
				memcpy(P->rem + P->head, P->take, sizeof(int) * (size_t)c.nt);
				return -rc;
			}
			continue;
		}
		for (unsigned q = 0; popc(c.Q) < m && q < P->n; q++)
			c.Q |= tbit(q);
		const int rc = emit(P, c.nt, c.Q, m, step, prog);
		return rc ? -rc : 1;
	}
}
