// Device set-up of channel bases (mq_solve.cu), for mq_grid.cpp. Not part of the public ABI.
#pragma once
#include "mq_grid.h"

// mq_channel_basis_ex on CUDA device `device`, with the host path's results bit for bit
mq_status mq_channel_basis_device(const mq_geom* g, int32_t basis, double tol, int32_t device, float* e4, double* phi_out,
                                  mq_solve_stats* stats);
