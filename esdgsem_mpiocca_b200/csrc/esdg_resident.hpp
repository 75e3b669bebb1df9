// Host interface of the chip-resident time loop (esdg_resident.cu).
#pragma once

#include <cuda_runtime.h>

#include "esdg_kernels.cuh"

namespace esdg {

struct ResWord;

// DevState::status of a wait that ran out (ST_OK and ST_NONFINITE: kernels.cuh,
// ST_TIMEOUT: the bulk copies, tma.cuh).
enum : int { ST_PEER_TIMEOUT = 3 };

struct ResArgs {
    int K, ne, ep;  // elements; elements per CTA (contiguous ranges) and per pass
    int fbase;      // first thread of the face warps, 0: every thread
    const double *Jinv, *Yxi, *Yeta, *Xxi, *Xeta, *Bx, *By, *D;
    double *q, *gRK;
    const int4 *ftab, *side;
    const double *nx, *ny, *scal, *bL, *bR;
    ResWord* tr;          // [2][K][4][3][ngl] exported traces
    ResWord* lam;         // [2][CTAs] wave-speed keys
    unsigned long long epoch;    // last epoch used before this launch
    DevState* st;
    PhysConst c;
    double rkA[8], rkB[8], rkC[8];
    int stages, ssp, numflux, ngl;
    int nsteps;                  // steps of this launch at most
    // positivity limiter and partial-dry treatment (the EXTRA instance)
    int PP;
    const double *EleSizes, *GLw;
    const int* dry_on;           // non-null: partial-dry treatment
    const double *B, *Dc, *Dup, *Ddn;
    long long wait_limit;        // clock cycles of a wait (0: the default)
};

// Launch shape for K elements on `sms` SMs: elements per CTA and per pass,
// CTAs (0 when the mesh does not fit the chip), threads, the kernel's block
// bound and the first thread of the face warps.
struct ResShape {
    int ne, ep, grid, threads, block, fbase;
    size_t smem;
};
ResShape resident_shape(int ngl, int K, int sms, bool extra, bool dry);
cudaError_t resident_setup(int ngl, const ResShape& s, bool extra);
cudaError_t resident_launch(const ResArgs& a, const ResShape& s, bool extra, cudaStream_t stream);

}  // namespace esdg
