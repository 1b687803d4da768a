// Launch interface of the warp-per-sample k-hop kernel (nd_khop_rows.cu).
#pragma once

#include "nd_common.cuh"

bool nd_khop_rows_fits(const nd_sampler *s);   // the sample's row fits a CTA's shared memory
int nd_khop_rows_alloc(nd_sampler *s);
int nd_khop_rows_launch(nd_sampler *s);        // one whole job on the sampler's stream
