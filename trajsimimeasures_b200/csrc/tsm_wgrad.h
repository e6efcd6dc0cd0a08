// Encoder weight gradients on the tensor cores (tsm_wgrad.cu), called by the
// training backward (tsm_train.cu).
#pragma once

#include <cuda_runtime.h>

#include "tsm_train.h"

// d_ih[384][64] += sum over the batch's slots and trajectories of g (x) a,
// d_hh[384][128] += sum of g (x) h (the hidden-side n gradients for the n
// rows), from the BF16 hi/lo images of w.  Stream-ordered; a bounded wait that
// runs out ORs a bit into *status (device int) and its CTA adds nothing.
int tsm_wgrad_tc(const enc::TrainWs& w, int* status, float* d_ih, float* d_hh, cudaStream_t s);
