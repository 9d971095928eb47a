/*
 * Element-wise tensor operations of libxm-gb300: set, copy, add, mul,
 * div, dot.  Each walks the canonical blocks of the output (for dot, every
 * nonzero block pair) in the reference's order (xm.c:28-508), maps each
 * block to the matching block of the second tensor through the index
 * strings, and turns the reference's unfold -> scale -> fold -> axpy chain
 * into one permuted, scaled CUDA pass over HBM (xmgd_ptasks).
 */
#include "xmg_host.h"
#include "hmap.h"

#define TASK_BATCH 4096

static int
check_pair(const xm_tensor_t *a, const xm_tensor_t *b, const char *idxa,
    const char *idxb, xm_dim_t *cidxa, xm_dim_t *cidxb, int same_type,
    const char *fn)
{
	size_t k;

	if (a->allocator != b->allocator)
		return xmg_seterr(XMG_EINVAL, "%s: tensors must use same "
		    "allocator", fn);
	if (same_type && a->type != b->type)
		return xmg_seterr(XMG_EINVAL, "%s: tensors must have same "
		    "scalar type", fn);
	if (strlen(idxa) != xm_block_space_get_ndims(a->bs))
		return xmg_seterr(XMG_EINVAL, "%s: idxa does not match tensor "
		    "dimensions", fn);
	if (strlen(idxb) != xm_block_space_get_ndims(b->bs))
		return xmg_seterr(XMG_EINVAL, "%s: idxb does not match tensor "
		    "dimensions", fn);
	xm_make_masks(idxa, idxb, cidxa, cidxb);
	if (cidxa->n != xm_block_space_get_ndims(a->bs) ||
	    cidxb->n != xm_block_space_get_ndims(b->bs))
		return xmg_seterr(XMG_EINVAL, "%s: index spaces do not match",
		    fn);
	for (k = 0; k < cidxa->n; k++)
		if (!xm_block_space_eq1(a->bs, cidxa->i[k], b->bs, cidxb->i[k]))
			return xmg_seterr(XMG_EINVAL, "%s: inconsistent "
			    "block-spaces", fn);
	return XMG_OK;
}

/*
 * Walk over the blocks of a (index 0 fastest) beside the matching blocks of
 * b: both linear positions advance by additions, so that a production
 * tensor's thousands of zero and derivative blocks cost a few instructions
 * each.
 */
typedef struct {
	size_t nd, n;			/* dimensions and blocks of a */
	size_t idx[XM_MAX_DIM], nb[XM_MAX_DIM];
	size_t step[XM_MAX_DIM];	/* b's linear step per a dimension */
	int bdim[XM_MAX_DIM];		/* b's dimension of each of a's */
	const size_t *split[XM_MAX_DIM];
	size_t la, lb;
} walk_t;

static void
walk_init(walk_t *w, const xm_tensor_t *a, const xm_tensor_t *b,
    const xm_dim_t *cidxa, const xm_dim_t *cidxb)
{
	xm_dim_t na = xm_block_space_get_nblocks(a->bs), nb;
	size_t k, j, st;

	memset(w, 0, sizeof *w);
	w->nd = na.n;
	w->n = a->nblocks_total;
	for (k = 0; k < na.n; k++) {
		w->nb[k] = na.i[k];
		w->split[k] = xmg_block_space_splits(a->bs, k);
	}
	if (b == NULL)
		return;
	nb = xm_block_space_get_nblocks(b->bs);
	for (k = 0; k < cidxa->n; k++) {
		for (st = 1, j = 0; j < cidxb->i[k]; j++)
			st *= nb.i[j];
		w->step[cidxa->i[k]] = st;
		w->bdim[cidxa->i[k]] = (int)cidxb->i[k];
	}
}

static inline void
walk_next(walk_t *w)
{
	size_t d;

	w->la++;
	for (d = 0; d < w->nd; d++) {
		w->lb += w->step[d];
		if (++w->idx[d] < w->nb[d])
			return;
		w->lb -= w->nb[d] * w->step[d];
		w->idx[d] = 0;
	}
}

/* dimensions of the current block of a; its number of elements */
static size_t
walk_dims(const walk_t *w, int64_t dims[XM_MAX_DIM])
{
	size_t d, n = 1;

	for (d = 0; d < w->nd; d++) {
		dims[d] = (int64_t)(w->split[d][w->idx[d] + 1] -
		    w->split[d][w->idx[d]]);
		n *= (size_t)dims[d];
	}
	return n;
}

/* element strides of a block of the given dims inside its source's data
 * (xmg_tensor_block_strides) */
static void
strides_of(const struct xmg_block *b, size_t nd, const int64_t *dims,
    int64_t *st)
{
	int64_t cd[XM_MAX_DIM], cs[XM_MAX_DIM], acc = 1;
	size_t k;

	/* dimension k of the block is dimension perm[k] of its source */
	for (k = 0; k < nd; k++)
		cd[b->perm.i[k]] = dims[k];
	for (k = 0; k < nd; k++) {
		cs[k] = acc;
		acc *= cd[k];
	}
	for (k = 0; k < nd; k++)
		st[k] = cs[b->perm.i[k]];
}

/* Fill t's iteration space "element of the current (canonical or
 * derivative) block ba of a <- matching element of block bb of b". */
static void
map_task(xmgd_ptask_t *t, const walk_t *w, const int64_t *dims,
    const struct xmg_block *ba, const struct xmg_block *bb)
{
	int64_t ds[XM_MAX_DIM], ss[XM_MAX_DIM], bst[XM_MAX_DIM], bd[XM_MAX_DIM];
	size_t k;

	for (k = 0; k < w->nd; k++)
		bd[w->bdim[k]] = dims[k];
	strides_of(ba, w->nd, dims, ds);
	strides_of(bb, w->nd, bd, bst);
	for (k = 0; k < w->nd; k++)
		ss[k] = bst[w->bdim[k]];
	xmg_ptask_shape(t, (int)w->nd, dims, ds, ss);
}

/* data handle of a nonzero block */
static uint64_t
handle_of(const xm_tensor_t *t, const struct xmg_block *b)
{
	return b->type == XM_BLOCK_TYPE_CANONICAL ? b->data :
	    t->blocks[b->data].data;
}

static uint64_t
dev_ptr(const xm_tensor_t *t, const struct xmg_block *b, size_t bytes)
{
	uint64_t d;

	xmg_die_on(xmg_alloc_device_view(t->allocator, handle_of(t, b), bytes,
	    &d));
	return d;
}

/* the staged output blocks of a batch outside GPU memory */
typedef struct {
	uint64_t h[TASK_BATCH];
	size_t bytes[TASK_BATCH];
	size_t n;
} outs_t;

/* Flush a batch; write staged outputs back. */
static int
flush(xmg_ptask_list_t *l, const xm_tensor_t *a, int dtype, int stype,
    outs_t *outs)
{
	size_t k;
	int st;

	if ((st = xmg_ptask_run(l, dtype, stype, NULL)) != XMG_OK)
		return st;
	l->n = 0;
	if (outs != NULL) {
		if ((st = xmgd_sync()) != XMG_OK)
			return st;
		for (k = 0; k < outs->n; k++)
			if ((st = xmg_alloc_commit_view(a->allocator, outs->h[k],
			    outs->bytes[k])) != XMG_OK)
				return st;
		outs->n = 0;
		xmg_alloc_release_views(a->allocator, 0);
	}
	return XMG_OK;
}

/* the output list of a batch: none for tensors in GPU memory */
static int
outs_create(const xm_tensor_t *a, outs_t **outs)
{
	*outs = NULL;
	if (!xmg_alloc_is_device(a->allocator) &&
	    (*outs = calloc(1, sizeof **outs)) == NULL)
		return xmg_seterr(XMG_ENOMEM, "out of memory");
	return XMG_OK;
}

static void
outs_push(outs_t *outs, uint64_t h, size_t bytes)
{
	if (outs != NULL) {
		outs->h[outs->n] = h;
		outs->bytes[outs->n++] = bytes;
	}
}

int
xmg_set(xm_tensor_t *a, xm_scalar_t x)
{
	xmg_ptask_list_t l = {0};
	size_t esz = xm_scalar_sizeof(a->type);
	xmgd_ptask_t *t;
	outs_t *outs;
	walk_t w;
	int64_t dims[XM_MAX_DIM], size;
	int st;

	if ((st = outs_create(a, &outs)) != XMG_OK)
		return st;
	walk_init(&w, a, NULL, NULL, NULL);
	for (; w.la < w.n && st == XMG_OK; walk_next(&w)) {
		struct xmg_block *ba = &a->blocks[w.la];
		if (ba->type != XM_BLOCK_TYPE_CANONICAL)
			continue;
		size = (int64_t)walk_dims(&w, dims);
		t = xmg_ptask_push(&l);
		t->op = XMGD_OP_SET;
		xmg_scalar_pack(x, t->alpha);
		t->dst = dev_ptr(a, ba, (size_t)size * esz);
		outs_push(outs, ba->data, (size_t)size * esz);
		xmg_ptask_shape(t, 1, &size, &(int64_t){1}, &(int64_t){0});
		if (l.n == TASK_BATCH)
			st = flush(&l, a, a->type, a->type, outs);
	}
	if (st == XMG_OK && l.n > 0)
		st = flush(&l, a, a->type, a->type, outs);
	if (st == XMG_OK)
		st = xmgd_sync();
	xmg_ptask_list_free(&l);
	free(outs);
	return st;
}

void
xm_set(xm_tensor_t *a, xm_scalar_t x)
{
	xmg_die_on(xmg_set(a, x));
}

/* Shared driver for copy / add / mul / div. */
enum { OPK_COPY, OPK_ADD, OPK_MUL, OPK_DIV };

static int
two_tensor(int kind, xm_scalar_t alpha, xm_tensor_t *a, xm_scalar_t beta,
    const xm_tensor_t *b, const char *idxa, const char *idxb, const char *fn)
{
	xm_dim_t cidxa, cidxb;
	xmg_ptask_list_t l = {0};
	xmgd_ptask_t *t;
	struct xmg_block *ba, *bb;
	outs_t *outs;
	walk_t w;
	xm_scalar_t s;
	int64_t dims[XM_MAX_DIM], size;
	size_t ea = xm_scalar_sizeof(a->type), eb = xm_scalar_sizeof(b->type);
	int st;

	if ((st = check_pair(a, b, idxa, idxb, &cidxa, &cidxb,
	    kind != OPK_COPY, fn)) != XMG_OK ||
	    (st = outs_create(a, &outs)) != XMG_OK)
		return st;
	walk_init(&w, a, b, &cidxa, &cidxb);
	for (; w.la < w.n && st == XMG_OK; walk_next(&w)) {
		ba = &a->blocks[w.la];
		if (ba->type != XM_BLOCK_TYPE_CANONICAL)
			continue;
		bb = &b->blocks[w.lb];
		size = (int64_t)walk_dims(&w, dims);
		t = xmg_ptask_push(&l);
		switch (kind) {
		case OPK_COPY:	/* xm.c:123-146 */
			if (alpha == 0 || bb->type == XM_BLOCK_TYPE_ZERO) {
				t->op = XMGD_OP_SET;
				break;
			}
			t->op = XMGD_OP_COPY;
			s = xm_scalar_mul(alpha, bb->scalar, b->type);
			xmg_scalar_pack(s, t->alpha);
			break;
		case OPK_ADD:	/* xm.c:212-240 */
			if (beta == 0 || bb->type == XM_BLOCK_TYPE_ZERO) {
				t->op = alpha == 0 ? XMGD_OP_SET : XMGD_OP_SCALE;
				xmg_scalar_pack(alpha == 0 ? 0 : alpha, t->alpha);
				break;
			}
			s = xm_scalar_mul(beta, bb->scalar, a->type);
			t->op = alpha == 0 ? XMGD_OP_COPY : XMGD_OP_AXPY;
			xmg_scalar_pack(alpha == 0 ? s : alpha, t->alpha);
			xmg_scalar_pack(s, t->beta);
			break;
		case OPK_MUL:	/* xm.c:304-323 */
			if (bb->type == XM_BLOCK_TYPE_ZERO) {
				t->op = XMGD_OP_SET;
				break;
			}
			t->op = XMGD_OP_MUL;
			xmg_scalar_pack(bb->scalar, t->alpha);
			break;
		case OPK_DIV:	/* xm.c:387-404 */
			if (bb->type == XM_BLOCK_TYPE_ZERO) {
				l.n--;
				st = xmg_seterr(XMG_EINVAL, "%s: division by zero",
				    fn);
				continue;
			}
			t->op = XMGD_OP_DIV;
			xmg_scalar_pack(bb->scalar, t->alpha);
			break;
		}
		t->dst = dev_ptr(a, ba, (size_t)size * ea);
		outs_push(outs, ba->data, (size_t)size * ea);
		if (t->op == XMGD_OP_SET || t->op == XMGD_OP_SCALE) {
			xmg_ptask_shape(t, 1, &size, &(int64_t){1},
			    &(int64_t){0});
		} else {
			t->src = dev_ptr(b, bb, (size_t)size * eb);
			map_task(t, &w, dims, ba, bb);
		}
		if (l.n == TASK_BATCH)
			st = flush(&l, a, a->type, b->type, outs);
	}
	if (st == XMG_OK && l.n > 0)
		st = flush(&l, a, a->type, b->type, outs);
	if (st == XMG_OK)
		st = xmgd_sync();
	if (!xmg_alloc_is_device(b->allocator))
		xmg_alloc_release_views(b->allocator, 0);
	xmg_ptask_list_free(&l);
	free(outs);
	return st;
}

void
xm_copy(xm_tensor_t *a, xm_scalar_t s, const xm_tensor_t *b, const char *idxa,
    const char *idxb)
{
	xmg_die_on(two_tensor(OPK_COPY, s, a, 0, b, idxa, idxb, __func__));
}

int
xmg_add(xm_scalar_t alpha, xm_tensor_t *a, xm_scalar_t beta,
    const xm_tensor_t *b, const char *idxa, const char *idxb)
{
	return two_tensor(OPK_ADD, alpha, a, beta, b, idxa, idxb, "xm_add");
}

void
xm_add(xm_scalar_t alpha, xm_tensor_t *a, xm_scalar_t beta,
    const xm_tensor_t *b, const char *idxa, const char *idxb)
{
	xmg_die_on(xmg_add(alpha, a, beta, b, idxa, idxb));
}

void
xm_mul(xm_tensor_t *a, const xm_tensor_t *b, const char *idxa,
    const char *idxb)
{
	xmg_die_on(two_tensor(OPK_MUL, 0, a, 0, b, idxa, idxb, __func__));
}

void
xm_div(xm_tensor_t *a, const xm_tensor_t *b, const char *idxa,
    const char *idxb)
{
	xmg_die_on(two_tensor(OPK_DIV, 0, a, 0, b, idxa, idxb, __func__));
}

/* The products of a pair of blocks: the data of both, and for each
 * dimension of a's source the dimension of b's source it runs along and its
 * extent.  Derivative blocks that agree in all of it have the same products,
 * whatever their own block indices. */
struct dot_key {
	uint64_t da, db, map;
	int64_t size[XM_MAX_DIM];
};

static void
dot_key(struct dot_key *q, const walk_t *w, const int64_t *dims,
    const xm_tensor_t *a, const struct xmg_block *ba, const xm_tensor_t *b,
    const struct xmg_block *bb)
{
	size_t k;

	memset(q, 0, sizeof *q);
	q->da = handle_of(a, ba);
	q->db = handle_of(b, bb);
	for (k = 0; k < w->nd; k++) {
		q->map |= (uint64_t)bb->perm.i[w->bdim[k]] << (4 * ba->perm.i[k]);
		q->size[ba->perm.i[k]] = dims[k];
	}
}

/* Sum over every block index of a where both blocks are nonzero of
 * (s_a * s_b) * <perm(a), perm(b)>  (xm.c:472-497), in the order of the
 * blocks.  Each distinct <,> -- the same data of a and of b, paired the
 * same way -- is computed once: for an antisymmetric pair of tensors that
 * is one block in four. */
xm_scalar_t
xm_dot(const xm_tensor_t *a, const xm_tensor_t *b, const char *idxa,
    const char *idxb)
{
	struct term { xm_scalar_t fac; size_t task; } *term = NULL;
	struct dot_key *key = NULL, q;
	xm_dim_t cidxa, cidxb;
	xmg_ptask_list_t l = {0};
	xmg_hmap_t seen;
	xmgd_ptask_t *t;
	xm_scalar_t dot = 0, part;
	double *dots = NULL;
	size_t i, nt = 0, cap = 0, esz = xm_scalar_sizeof(a->type);
	struct xmg_block *ba, *bb;
	int64_t dims[XM_MAX_DIM], size;
	uint64_t h, v;
	walk_t w;

	xmg_die_on(check_pair(a, b, idxa, idxb, &cidxa, &cidxb, 1, __func__));
	xmg_hmap_init(&seen);
	walk_init(&w, a, b, &cidxa, &cidxb);
	for (; w.la < w.n; walk_next(&w)) {
		ba = &a->blocks[w.la];
		bb = &b->blocks[w.lb];
		if (ba->type == XM_BLOCK_TYPE_ZERO ||
		    bb->type == XM_BLOCK_TYPE_ZERO)
			continue;
		if (nt == cap) {
			cap = cap ? 2 * cap : 256;
			if ((term = realloc(term, cap * sizeof *term)) == NULL ||
			    (key = realloc(key, cap * sizeof *key)) == NULL)
				xm_fatal("%s: out of memory", __func__);
		}
		term[nt].fac = xm_scalar_mul(ba->scalar, bb->scalar, a->type);
		size = (int64_t)walk_dims(&w, dims);
		dot_key(&q, &w, dims, a, ba, b, bb);
		h = xmg_hash64(q.da ^ xmg_hash64(q.db ^ xmg_hash64(q.map)));
		for (;; h = xmg_hash64(h + 1)) {
			if (h == XMG_HMAP_EMPTY)
				h--;
			if (!xmg_hmap_get(&seen, h, &v))
				break;
			if (memcmp(&key[v], &q, sizeof q) == 0)
				break;
		}
		if (xmg_hmap_get(&seen, h, &v)) {
			term[nt++].task = v;
			continue;
		}
		if (xmg_hmap_put(&seen, h, (uint64_t)l.n))
			xm_fatal("%s: out of memory", __func__);
		key[l.n] = q;
		term[nt++].task = (size_t)l.n;
		t = xmg_ptask_push(&l);
		t->op = XMGD_OP_DOT;
		t->dst = dev_ptr(a, ba, (size_t)size * esz);
		t->src = dev_ptr(b, bb, (size_t)size * esz);
		map_task(t, &w, dims, ba, bb);
	}
	if (nt > 0) {
		if ((dots = calloc(2 * (size_t)l.n, sizeof *dots)) == NULL)
			xm_fatal("%s: out of memory", __func__);
		xmg_die_on(xmg_ptask_run(&l, a->type, b->type, dots));
		xmg_die_on(xmgd_sync());
		for (i = 0; i < nt; i++) {
			part = dots[2 * term[i].task] +
			    dots[2 * term[i].task + 1] * I;
			part = xm_scalar_mul(term[i].fac, part, a->type);
			dot = xm_scalar_add(dot, part, a->type);
		}
	}
	if (!xmg_alloc_is_device(a->allocator))
		xmg_alloc_release_views(a->allocator, 0);
	xmg_hmap_free(&seen);
	xmg_ptask_list_free(&l);
	free(term);
	free(key);
	free(dots);
	return dot;
}

void
xm_print_banner(void)
{
	printf("Libxm Tensor Library (GB300 engine)\n");
	printf("libxm API on hand-written sm_103a CUDA kernels\n");
	printf("Reference algorithm: https://github.com/ilyak/libxm\n");
}
