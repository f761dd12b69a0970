// MINRES and conjugate residuals over natural-order slices (kernels_flow_more.cu).
#pragma once

#include "feec_system.h"

namespace feec {

struct FlowMoreArgs {
    int n, nslices;
    const int4* meta; const int* ci; const double* val;
    const double* b;
    double *x, *res;
    double* w[5];            // work vectors
    double* pub[2];          // published vectors, holding the sentinel in every slot
    double tol;              // max(precision * ||b||, 2^-26)
    int max_iter, print_modulo;
    double* partials;        // 8 per block
    DeviceStatus* st;
};

cudaError_t launch_flow_more(bool minres, const FlowForm& form, const FlowMoreArgs& a, cudaStream_t st);

}  // namespace feec
