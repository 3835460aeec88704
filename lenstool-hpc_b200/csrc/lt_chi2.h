/*
 * lt_chi2.h -- the device layout and the steps of one chi2 evaluation (lt_chi2.cu), shared
 * by the chi2 entry points and the serving loop's chi2 requests (lt_server.cpp).
 */
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <cuda_runtime.h>

#include "../../include/lt_b200.h"

struct lt_catalog;

namespace lt {

struct Chi2Dev {
    /* systems */
    int nsys, nimages;
    const int32_t *nimg, *first;        /* images per system, index of its first image */
    const double *ix, *iy, *dr;
    /* grid */
    int n;
    double xmin, ymin, dx, dy;
    const double *ax, *ay;              /* deflection grid, n x n */
    /* work and results: one block of each per model, model m's at m x its size */
    double *bx, *by;                    /* source per system */
    int32_t *hits, *keys;               /* hit count and hit keys (2 * cell + lower) per system */
    double *chi_terms;                  /* per observed image: its chi2 term */
    double *chi2;                       /* one word a model */
    int32_t *found;                     /* two words a model: predicted images; 1 if a source overflowed */
    int32_t *nfound;                    /* predicted images per system (<= LT_MAX_IMAGES) */
    double *fx, *fy;                    /* predicted images, nsys x LT_MAX_IMAGES */
};

/* Bytes of the device buffers of `nmodels` evaluations (systems, work and results of each
 * model, the n x n deflection planes, which the models take in turn); with `mem`, also lays them out there and fills `c` (grid from the frame:
 * dx = (xmax - xmin)/(n - 1), src/chi_CPU_barycenter.cpp:104-105). */
size_t chi2_layout(int nsys, int nimages, const lt_frame *f, int n, char *mem, Chi2Dev &c, int nmodels = 1);

/* Copy the systems (host arrays; `first` = index of each system's first image) into the
 * layout, stream-ordered; the host arrays must stay valid until the copies have run. */
cudaError_t chi2_upload_systems_async(const Chi2Dev &c, const int32_t *nimg, const int32_t *first, const double *x,
                                      const double *y, const double *dr, cudaStream_t s);

/* Steps 2-4 (sources, delensing, link and chi2) on a layout whose deflection planes hold
 * the grid, stream-ordered; results in c.chi2[0] and c.found[0..1]. */
int chi2_tail(lt_context *ctx, const lt_catalog *cat, const Chi2Dev &c, cudaStream_t s);

lt_status check_systems(lt_context *ctx, const lt_image_systems *sys);

} // namespace lt
