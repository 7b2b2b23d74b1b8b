// Resident Jacobi-PCG kernel (resident.cu): the launch plan of a grid.
#pragma once

#include "pcg.hpp"

namespace rb200 {

// The shortest run whose bricks are at most `blocks` (0: the device's SMs).
int resident_setup(const GridDev& g, ResidentPlan* plan, int blocks = 0);
size_t resident_words(const ResidentPlan& plan);  // 64-bit words of the reductions, zeroed before each solve
cudaError_t launch_resident(const ResidentPlan& plan, const GridDev& g, SolveState* st, const double* b, double* p,
                            double* r, double* z, double* d0, double* d1, unsigned long long* words, GridBarrier* bar,
                            rb200_trace* trace, int budget, cudaStream_t s);

}  // namespace rb200
