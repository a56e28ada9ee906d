// cg.h -- CGNE propagator solver (congrad replacement).
#pragma once
#include "internal.h"

namespace chdwf {

template <class T> struct PcgWork;      // plane_cg.cuh

struct CgWork {
    PcgWork<double2>* w = nullptr;
    ~CgWork();
    void release();
};

// Solves M^dagger M x = Phi starting from x (in/out).  status 0 converged,
// 1 iteration cap (kthird*kvol), 2 non-finite.
cudaError_t cg_solve(CgWork& w, const Geom& g, const double2* phi, float res, const float* chif,
                     float am3, float hpin, int imass, int ibound, double2* x, int* itercg,
                     int* status, cudaStream_t st);

}  // namespace chdwf
