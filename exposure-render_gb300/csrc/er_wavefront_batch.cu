/*
 * er_wavefront_batch.cu - the batch half of the wavefront stages (compiled
 * with --fmad=false): the kernels' variants that read each item's view from
 * the batch's table, apart from the one-view variants so that the two compile
 * in parallel.
 */
#define WF_BATCH_UNIT
#include "er_wavefront.cu"
