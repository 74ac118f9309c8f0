// cuFFT plans kept by a context between calls.
#pragma once
#include <cufft.h>

#include "common.cuh"

namespace qsm {

// The 3-D plans one call uses, in its order of types, and their work area.
struct FftPlans {
    static constexpr int MAX = 4;
    cufftHandle h[MAX] = {};
    int slot[MAX] = {-1, -1, -1, -1};  // the context's entries
    void *work = nullptr;
};

// A plan of each of the n types over a volume (x fastest) on the context's stream:
// one the context has kept and no call is using, else a new one.  Making a plan
// uploads its tables (~0.5 ms each with the copies' synchronisations; V-SHARP takes
// four, the ADMM inversion two): kept, V-SHARP at 224 x 224 x 128 in FP64 takes 8.5 ms
// instead of 10.2, the ADMM inversion there 16.4 instead of 17.3.  A context keeps up
// to FFT_KEEP, the ones used last (tables of ~100 KB each at that size).  The
// work area, the large part, comes from the pool per call, one for all the plans:
// their transforms follow one another on the stream.  On failure nothing is held.
qsm_status fft_acquire(qsm_ctx *ctx, const Dims &d, const cufftType *type, int n, FftPlans *p);
// Gives the plans back (after the call's last transform is enqueued).
void fft_release(qsm_ctx *ctx, FftPlans *p);
// Destroys every plan of the context.
void fft_clear(qsm_ctx *ctx);

constexpr int FFT_KEEP = 12;

}  // namespace qsm
