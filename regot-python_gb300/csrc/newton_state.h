// Device-side state of the Newton systems (erot_newton.cu, newton_plan.cuh).
#pragma once

namespace regot {

struct NewtonState {
    int cg_done;
    int cg_it;
    int cg_max;
    int err;  // a barrier of a resident kernel gave up
    unsigned counter;
    double rz;       // r' z of the current CG residual
    double alpha;    // CG step
    double beta;     // CG direction update
    double thresh2;  // stop when ||r||^2 < thresh2
    double rnorm2;
    double f;        // objective at gamma
    double gnorm;
    double gtd;      // g' d
    double ad;       // a' d_alpha + b~' d_beta~
    double maxabs;   // bound on |gamma|, |d| for the hi/lo split
    unsigned long long t0;
};

}  // namespace regot
