// Launch interface of the lane-per-walk kernels (nd_walk_rows.cu).
#pragma once

#include "nd_common.cuh"

int nd_walk_rows_alloc(nd_sampler *s);                    // per-graph layouts the kernels read
int nd_walk_rows_launch(nd_sampler *s, bool count_live);  // one whole job on the sampler's stream
