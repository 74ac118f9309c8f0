// cuFFT plans kept by a context between calls (fft_plans.cuh).
#include <exception>
#include <mutex>
#include <vector>

#include "fft_plans.cuh"

namespace qsm {

namespace {
struct Entry {
    size_t n[3];
    cufftType type;
    cufftHandle h;
    size_t work;
    uint64_t used;
    bool busy, live;
};
}  // namespace

struct FftCache {
    std::mutex mu;  // calls of several threads on one context
    std::vector<Entry> e;
    uint64_t clock = 0;
};

static std::mutex g_make;

static FftCache *cache(qsm_ctx *ctx)
{
    std::lock_guard<std::mutex> lock(g_make);
    if (!ctx->fft) ctx->fft = new FftCache();
    return ctx->fft;
}

static qsm_status fail(qsm_ctx *ctx, const char *what, cufftResult r)
{
    set_error(ctx, "cuFFT: %s failed (%d)", what, (int)r);
    return r == CUFFT_ALLOC_FAILED ? QSM_ERR_NOMEM : QSM_ERR_CUDA;
}

static bool fits(const Entry &e, const Dims &d, cufftType type)
{
    return e.type == type && e.n[0] == d.nx && e.n[1] == d.ny && e.n[2] == d.nz;
}

// The entry to use for one type (made if none is free), or -1.
static int take(qsm_ctx *ctx, FftCache *c, const Dims &d, cufftType type, qsm_status *st)
{
    int s = -1;
    for (size_t k = 0; k < c->e.size() && s < 0; ++k)
        if (c->e[k].live && !c->e[k].busy && fits(c->e[k], d, type)) s = (int)k;
    if (s < 0) {
        for (size_t k = 0; k < c->e.size() && s < 0; ++k)
            if (!c->e[k].live) s = (int)k;
        if (s < 0) {
            c->e.push_back(Entry());
            s = (int)c->e.size() - 1;
        }
        Entry e{{d.nx, d.ny, d.nz}, type, 0, 0, 0, true, true};
        cufftResult r = cufftCreate(&e.h);
        if (r != CUFFT_SUCCESS) {
            *st = fail(ctx, "cufftCreate", r);
            return -1;
        }
        r = cufftSetAutoAllocation(e.h, 0);
        if (r == CUFFT_SUCCESS) r = cufftMakePlan3d(e.h, (int)d.nz, (int)d.ny, (int)d.nx, type, &e.work);
        if (r != CUFFT_SUCCESS) {
            cufftDestroy(e.h);
            *st = fail(ctx, "cufftMakePlan3d", r);
            return -1;
        }
        c->e[(size_t)s] = e;
    }
    c->e[(size_t)s].busy = true;
    c->e[(size_t)s].used = ++c->clock;
    return s;
}

qsm_status fft_acquire(qsm_ctx *ctx, const Dims &d, const cufftType *type, int n, FftPlans *p)
try {
    *p = FftPlans();
    qsm_status st = QSM_OK;
    size_t work = 0;
    FftCache *c = cache(ctx);
    {
        std::lock_guard<std::mutex> lock(c->mu);
        for (int k = 0; k < n && st == QSM_OK; ++k) {
            p->slot[k] = take(ctx, c, d, type[k], &st);
            if (p->slot[k] < 0) break;
            p->h[k] = c->e[(size_t)p->slot[k]].h;
            work = work > c->e[(size_t)p->slot[k]].work ? work : c->e[(size_t)p->slot[k]].work;
        }
    }
    if (st == QSM_OK) st = dalloc(ctx, &p->work, work);
    for (int k = 0; k < n && st == QSM_OK; ++k) {
        cufftResult r = cufftSetStream(p->h[k], ctx->stream);
        if (r == CUFFT_SUCCESS) r = cufftSetWorkArea(p->h[k], p->work);
        if (r != CUFFT_SUCCESS) st = fail(ctx, "cufftSetWorkArea", r);
    }
    if (st != QSM_OK) fft_release(ctx, p);
    return st;
} catch (const std::exception &) {  // host memory
    fft_release(ctx, p);
    set_error(ctx, "out of host memory");
    return QSM_ERR_NOMEM;
}

void fft_release(qsm_ctx *ctx, FftPlans *p)
{
    if (p->work) dfree(ctx, p->work);
    FftCache *c = ctx->fft;
    if (!c) return;
    std::lock_guard<std::mutex> lock(c->mu);
    for (int s : p->slot)
        if (s >= 0) c->e[(size_t)s].busy = false;
    *p = FftPlans();
    for (;;) {  // beyond the bound: the one used longest ago goes
        int n = 0, old = -1;
        for (size_t k = 0; k < c->e.size(); ++k) {
            if (!c->e[k].live) continue;
            ++n;
            if (!c->e[k].busy && (old < 0 || c->e[k].used < c->e[(size_t)old].used)) old = (int)k;
        }
        if (n <= FFT_KEEP || old < 0) break;
        cudaStreamSynchronize(ctx->stream);  // its transforms may still run
        cufftDestroy(c->e[(size_t)old].h);
        c->e[(size_t)old].live = false;
    }
}

void fft_clear(qsm_ctx *ctx)
{
    if (!ctx->fft) return;
    for (Entry &e : ctx->fft->e)
        if (e.live) cufftDestroy(e.h);
    delete ctx->fft;
    ctx->fft = nullptr;
}

}  // namespace qsm
