/*
 * The parts of the develop stage that are translation units (and so modules,
 * loaded by themselves) of their own; develop.cu calls them.
 */
#pragma once

#include <cuda_runtime.h>

#include "../kabi.h"

/* A bilinear or MHC frame (develop_linear.cu); 0 or -5. */
int craw_develop_linear(const CRAWKDevelop *k, const CRAWKDevelopIO *io, bool early, cudaStream_t s);

/* Loads those kernels on the current device; 0 or -5. */
int craw_develop_linear_prepare();

/* An RCD frame by 64x16 tiles and a per-pixel border (develop_rcd_tiles.cu);
 * 0 or -5. */
int craw_develop_rcd_tiles(const CRAWKDevelop *k, const CRAWKDevelopIO *io, cudaStream_t s);

/* Loads those kernels on the current device; 0 or -5. */
int craw_develop_rcd_tiles_prepare();
