/* gb_bcg.h -- state shared by the block-CG sources (gb_bcg.cu, gb_bcg_persist.cu) */
#ifndef GB_BCG_H
#define GB_BCG_H

#include <stddef.h>

#include "gb_internal.h"

/* per-column scalars and block partials of a block-CG call, in its workspace */
struct bcg_state {
    double *rho1, *rho2, *err, *ptw, *part, *alpha, *beta, *sums;
    int *nact;
};

/* all FP64 rounds in one cooperative launch, on R (the initial residual) and X in
 * place; s->part: ceil(n / 128) doubles per column */
extern "C" int gb_bcg_persist64(gcge_gpu_ctx *ctx, const gcge_gpu_mat *A, const gb_bcg_args *b, const bcg_state *s,
                                double *R, long ldr, double *X, long ldx, double *P, double *W, long ld);

#endif
