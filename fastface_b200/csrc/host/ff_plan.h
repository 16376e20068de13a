/* ff_plan.h -- static layer plan derived from the FFW4 op list (C99 host side). */
#ifndef FF_PLAN_H
#define FF_PLAN_H

#include "ff_model.h"
#include "ff_cuda.h"

#ifdef __cplusplus
extern "C" {
#endif

typedef struct {
    int n_layers;
    ffcu_layer* layers;      /* arrays inside are owned by the plan (see pool) */
    int n_bufs;              /* activation buffers the plan needs */
    size_t bytes_per_face;   /* largest int8 activation tensor of one face */
    void** pool;             /* every allocation the layers point into */
    int pool_n, pool_cap;
} ff_plan;

/* Walks the op list the way the reference's driver loop does
 * (libfastface.c:243-269 shape pre-pass, :349-466 op loop), resolving at build
 * time which scale each kernel call would receive, and emits one ffcu_layer per
 * kernel launch.  0 on success. */
int  ff_plan_build(ff_plan* p, const ff_model* m);
void ff_plan_free(ff_plan* p);

/* The layers [0, return value) of l[0 .. n) that may run chunk by chunk, each chunk of faces through all of them before the
 * next one starts; at most `end`, at least 2 (the input's quantisation and the stem).  Tensors are laid out face after face
 * from their buffer's start, and a buffer holds tensors of different bytes per face, so face f of one may lie where
 * a lower face of another does: a head is only taken where no layer of it writes a buffer at fewer bytes per face than
 * the tensor that the rest of the network finds there (then chunk j writes behind all that chunks < j left).  with_next[k] != 0:
 * layers k and k + 1 go out as one launch and stay on one side. */
int  ff_plan_head_end(const ffcu_layer* l, int n, int end, const unsigned char* with_next);

/* May layers [first, first + count) of l[0 .. n) run face by face with only the last one's tensors in their buffers, and each
 * residual taken from outside or from the layer with a residual before it, whose result is kept until then?  Not where a layer
 * behind them reads another tensor of theirs.  from[i]: the layer, counted from `first`, whose result layer i adds; -1: a tensor
 * that was in its buffer before, or none.  1 / 0. */
int  ff_plan_stage(const ffcu_layer* l, int n, int first, int count, int* from);

#ifdef __cplusplus
}
#endif
#endif
