// Device set-up of channel bases (mq_solve.cu), for mq_grid.cpp. Not part of the public ABI.
#pragma once
#include "mq_grid.h"

// mq_channel_basis_ex on CUDA device `device`, with the host path's results bit for bit
mq_status mq_channel_basis_device(const mq_geom* g, int32_t basis, double tol, int32_t device, float* e4, double* phi_out,
                                  mq_solve_stats* stats);

// mq_laplace_solve_device, and with lists = 0 the way that it takes on grids of 2^32 nodes and more, whose node numbers
// do not fit the packed lists of free nodes: for tests of that way on grids of any size
extern "C" mq_status mq_laplace_solve_device_lists(int32_t nx, int32_t ny, int32_t nz, const uint8_t* mask, const double* fixed, double outer_bc,
                                                   double tol, int32_t device, int32_t lists, double* phi, mq_solve_stats* stats);
