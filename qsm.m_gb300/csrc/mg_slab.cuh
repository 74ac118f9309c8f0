// Coarsest-level solver on one thread-block cluster of 1..16 CTAs
// (mgpcg_mex.c:265-275), included by mg.cu inside namespace qsm.
//
// The reference's coarsest loop is up to 1024 x (128 reverse + 128 forward
// red-black sweeps, residual, norm): thousands of short dependent colour
// passes, bound by the latency of one pass.  Here the level's G voxels, merged
// over both colours in index order, are cut into one chunk of equal length per
// CTA, so every CTA updates the same number of voxels whatever the mask's
// shape.  A CTA keeps its chunk's values in shared memory, each colour in its
// own array (consecutive voxels of a row are then consecutive words: no bank
// conflicts, where an x-fastest array has stride 2), between windows that
// receive the neighbouring chunks' values; a thread keeps its voxels' f and
// the six neighbour slots of each in registers, so a pass holds no index
// arithmetic.  A new value goes to each CTA that reads it with st.async, which
// counts its bytes on an mbarrier there: a CTA waits for the values it reads
// and for nothing else, instead of a cluster barrier per pass.
//
// Why no value is overwritten before it is read, and no phase is overrun: a
// voxel X in CTA a that CTA b reads is the neighbour of a voxel Y in b, and a
// reads Y.  a sends X's next value only after it has waited for Y's value of
// the pass in which b read X; and b's barrier for one colour is armed again
// two passes later, after b has waited for its previous phase.  The passes
// alternate strictly between the colours: where the last reverse pass and the
// first forward pass are of one colour, the former is left out, since the
// latter recomputes all it wrote from the same values of the other colour.
//
// A thread whose wait has run out neither waits nor sends any more, and where it is
// thread 0 its CTA arms no barrier.  The CTAs that read its values run out in turn.
// The passes left of the outer iteration run down, then the CTAs leave together after
// its cluster barrier, with the error word set.
//
// Results are those of every other coarsest solver bit for bit: a pass reads
// the other colour only, so its order is free, and the norm keeps the lane
// order.  What bounds a pass is latency: a barrier of the CTA's threads (205
// cycles for 128 of them, 360 for 1024, measured alone) and, on several CTAs,
// st.async and its wait (another ~340 cycles; a cluster barrier takes 625-935).
// Several voxels per thread on fewer warps measured slower than one (190^2 x
// 110 volume, 16 CTAs: 13.6 ms with one, 17.9 with two, 27.4 with four).
// Where the time lies against the other solvers: slab_ctas in mg.cu.

constexpr int SL_MAX_CTAS = 16;
constexpr int SL_MAX_THREADS = 1024;
constexpr int SL_MAX_PER = 2;                     // voxels of each colour per thread
constexpr unsigned SL_SOFT_MIN = 256;  // FP64 voxels per colour and CTA from which multiplies leave the FP64 pipe
constexpr unsigned SL_NONE = 0xFFFFFFFFu;         // pos of a voxel no pass updates
constexpr unsigned SL_TRY_NS = 2000;              // most one try of a wait is suspended
constexpr unsigned SL_TRIES = 1u << 20;           // tries before a wait gives up (seconds)
constexpr unsigned SL_SETTLE_NS = 200000;         // a stopped solver's time for the stores in flight

// meta word of a voxel: export list start (16 bits) and count (3), quirk flags,
// whether it reads a received value, neighbours read from global memory (6)
constexpr uint32_t SL_I1 = 1u << 19, SL_INX2 = 1u << 20, SL_HALO = 1u << 21, SL_ON = 1u << 22;
constexpr int SL_GLOB = 23;

// A level's chunks: pos[l] = index of voxel l in its colour list (SL_NONE
// outside the interior of G), cut as slab_cuts_k writes it.
struct SlabTab {
    unsigned *pos, *cut;
    int ctas;      // 1, 2, 4, 8 or 16; 0: not used
    int threads, per;
    bool soft;     // FP64: multiply on the integer pipes
    unsigned cap;  // most voxels of one colour in a chunk
    unsigned win;  // most voxels of one colour within one plane of indices
    size_t smem;
    unsigned tries, extra;  // a wait's tries; bytes it needs beyond those sent (0; 8 under QSM_DEBUG_WAIT_TIMEOUT)
};

// Shared-memory layout of one CTA (host and device agree on it).
struct SlabLayout {
    size_t v[2], blk, bc, exp[2], need, bytes;
    unsigned len;  // slots per colour: window, chunk, window, then one that holds 0
    __host__ __device__ SlabLayout(unsigned cap, unsigned win, int ctas, size_t es)
    {
        len = cap + 2 * win + 1;
        v[0] = 0;
        v[1] = v[0] + len * es;
        blk = (v[1] + len * es + 15) & ~(size_t)15;
        bc = blk + (size_t)RED_NBLK * es;
        exp[0] = (bc + 16 + 15) & ~(size_t)15;
        exp[1] = exp[0] + (ctas > 1 ? (size_t)6 * cap * sizeof(uint32_t) : 0);
        need = exp[1] + (ctas > 1 ? (size_t)6 * cap * sizeof(uint32_t) : 0);
        bytes = need + (ctas > 1 ? (size_t)2 * len : 0);
    }
};

__global__ void slab_pos_k(unsigned *pos, const uint32_t *__restrict__ l0, unsigned c0, const uint32_t *__restrict__ l1,
                           unsigned c1)
{
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < c0) pos[l0[t] & BL_IDX] = t;
    else if (t - c0 < c1) pos[l1[t - c0] & BL_IDX] = t - c0;
}

// The chunks of a level in sixteenths of its G voxels (both colours), cut at
// the segments (32 voxels of a row) that blist_seg_k counts: off is the scan of
// its counts.  out[2 c + q] = voxels of colour q before cut c; a solver of
// fewer CTAs takes every second, fourth, ... cut.
__global__ void slab_cuts_k(unsigned *out, const unsigned *__restrict__ off, const unsigned *__restrict__ tot,
                            unsigned nseg)
{
    const unsigned c = threadIdx.x, c0 = tot[2], c1 = tot[3];
    if (c > SL_MAX_CTAS) return;
    const unsigned b0 = off[2 * (size_t)nseg], b1 = off[3 * (size_t)nseg];
    const unsigned d = (unsigned)((unsigned long long)(c0 + c1) * c / SL_MAX_CTAS);
    unsigned lo = 0, hi = nseg;
    while (lo < hi) {  // first segment with d voxels or more before it
        const unsigned s = (lo + hi) / 2;
        if (off[2 * (size_t)nseg + s] - b0 + (off[3 * (size_t)nseg + s] - b1) < d) lo = s + 1;
        else hi = s;
    }
    out[2 * c] = lo < nseg ? off[2 * (size_t)nseg + lo] - b0 : c0;
    out[2 * c + 1] = lo < nseg ? off[3 * (size_t)nseg + lo] - b1 : c1;
}

__device__ __forceinline__ uint32_t sl_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t sl_mapa(uint32_t a, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void sl_send(uint32_t a, float v, uint32_t mb)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(a), "f"(v), "r"(mb)
                 : "memory");
}
__device__ __forceinline__ void sl_send(uint32_t a, double v, uint32_t mb)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(a), "d"(v), "r"(mb)
                 : "memory");
}
__device__ __forceinline__ void sl_arm(uint32_t mb, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
}
// waits for the phase of this parity; false once the tries, each of bounded time, have run out
__device__ __forceinline__ bool sl_wait(uint32_t mb, uint32_t parity, unsigned tries)
{
    for (unsigned k = 0; k < tries; ++k) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(mb), "r"(parity), "r"(SL_TRY_NS)
                     : "memory");
        if (ok) return true;
    }
    return false;
}

// Sets the stop word of every CTA.
__device__ __noinline__ void sl_stop(unsigned *stop)
{
    const uint32_t cn = cl_size();
    for (uint32_t r = 0; r < cn; ++r) cl_or(cl_map(stop, r), 1u);
}

// Time for the stores of a stopped solver to land, whose barriers no longer tell: none
// is sent any more, and one takes under a microsecond.  (The reads of the clock are
// bounded too.)
__device__ __noinline__ void sl_settle()
{
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (int k = 0; k < (1 << 16); ++k) {
        __nanosleep(1000);
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 >= SL_SETTLE_NS) break;
    }
}

// lane-order sum of src[e]^2 over e < n <= RED_LANES (src in global memory,
// written before the last cluster barrier), in every thread of the cluster
template <typename T>
__device__ T sl_lane_sum(const T *src, unsigned n, T *blk, T *bc, uint32_t c, uint32_t cn)
{
    const unsigned nw = blockDim.x / 32, w = threadIdx.x / 32, lane = threadIdx.x % 32;
    const unsigned nb = (n + RED_BLOCK - 1) / RED_BLOCK;
    for (unsigned b = c * nw + w; b < nb; b += cn * nw) {
        T x[RED_BLOCK / 32];
#pragma unroll
        for (int i = 0; i < RED_BLOCK / 32; ++i) {
            const unsigned e = b * RED_BLOCK + 32 * i + lane;
            x[i] = e < n ? __ldcg(src + e) : (T)0;
        }
#pragma unroll
        for (int i = 0; i < RED_BLOCK / 32; ++i) x[i] = x[i] * x[i];
        const T s = warp_halve(x);
        if (lane == 0) cl_st(cl_map(blk, 0) + (uint32_t)(b * sizeof(T)), s);
    }
    cl_sync();
    if (c == 0 && w == 0) {
        T x[RED_NBLK / 32];
#pragma unroll
        for (int i = 0; i < RED_NBLK / 32; ++i) x[i] = blk[32 * i + lane];  // b >= nb: +0, never written
        const T s = __shfl_sync(0xffffffffu, warp_halve(x), 0);
        if (lane < cn) cl_st(cl_map(bc, lane), s);
    }
    cl_sync();
    return bc[0];
}

__device__ __forceinline__ float sl_ld(uint32_t a, float)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ double sl_ld(uint32_t a, double)
{
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sl_st(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void sl_st(uint32_t a, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }

// A thread's voxels of one colour: the shared-memory addresses of their six
// neighbours (x-, x+, y-, y+, z-, z+), meta words and f.
template <typename T, int PER>
struct SlabShare {
    uint32_t a[PER][6], meta[PER];
    T f[PER];
};

// What one colour's passes need besides: where its values lie and go.
struct SlabCol {
    uint32_t own;         // address of the thread's first value
    uint32_t va, mb;      // this CTA's value array and barrier (mapped to a peer's when sending)
    const uint32_t *exp;  // targets: rank << 16 | slot
    const uint32_t *list;
};

// neighbours outside the chunk's lists that hold other than +0 (an initial
// guess outside G): read where they are, no pass changes them
template <typename T>
__device__ __forceinline__ void slab_globals(T (&x)[6], uint32_t g, const T *gv, size_t l, int nx, int nxny)
{
    if (g & 1u) x[0] = __ldcg(gv + l - 1);
    if (g & 2u) x[1] = __ldcg(gv + l + 1);
    if (g & 4u) x[2] = __ldcg(gv + l - nx);
    if (g & 8u) x[3] = __ldcg(gv + l + nx);
    if (g & 16u) x[4] = __ldcg(gv + l - nxny);
    if (g & 32u) x[5] = __ldcg(gv + l + nxny);
}

// One colour pass of the CTA.  Most voxels neither receive nor send a value:
// in FP32 their meta word, SL_ON alone, takes a short way.  FP64 has one way
// only: a warp with voxels of both kinds would issue the update twice, and an
// FP64 instruction costs its ~80 cycles whatever lanes it has.
template <typename T, int PER, typename GC, bool MULTI>
__device__ __forceinline__ void slab_pass(const SlabShare<T, PER> &S, const SlabCol &C, uint32_t skip, const GC &c,
                                          const T *gv, int nx, int nxny, uint32_t wait_mb, uint32_t wait_par, bool wait,
                                          unsigned tries, int &dead, int &arm)
{
    const uint32_t step = blockDim.x * (uint32_t)sizeof(T);
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const uint32_t meta = S.meta[u];
        if (sizeof(T) == 4 && meta == 0) continue;
        if (sizeof(T) == 4 && (meta & (~(SL_I1 | SL_INX2) | skip)) == SL_ON) {
            T x[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) x[k] = sl_ld(S.a[u][k], T());
            sl_st(C.own + u * step, c.hh * (S.f[u] + (c.hx * (x[0] + x[1]) + c.hy * (x[2] + x[3]) + c.hz * (x[4] + x[5]))));
            continue;
        }
        if (MULTI && wait && (meta & SL_HALO) && !dead && !sl_wait(wait_mb, wait_par, tries)) {
            dead = 1;
            arm = 0;
        }
        if (sizeof(T) == 8) {
            __syncwarp();  // (else compiled as two ways after all: 64^3 with two levels 34.4 instead of 28.5 ms)
            if (meta == 0) continue;
        }
        T val;
        if (meta & skip) {
            val = sl_ld(C.own + u * step, T());
        } else {
            T x[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) x[k] = sl_ld(S.a[u][k], T());
            if (meta >> SL_GLOB)
                slab_globals<T>(x, meta >> SL_GLOB, gv, C.list[threadIdx.x + u * blockDim.x] & BL_IDX, nx, nxny);
            val = c.hh * (S.f[u] + (c.hx * (x[0] + x[1]) + c.hy * (x[2] + x[3]) + c.hz * (x[4] + x[5])));
            sl_st(C.own + u * step, val);
        }
        const unsigned cnt = !MULTI || dead ? 0u : (meta >> 16) & 7u, s0 = meta & 0xffffu;
        for (unsigned k = 0; k < cnt; ++k) {
            const uint32_t t = C.exp[s0 + k];
            sl_send(sl_mapa(C.va, t >> 16) + (t & 0xffffu) * (uint32_t)sizeof(T), val, sl_mapa(C.mb, t >> 16));
        }
    }
    __syncthreads();
}

// MULTI: more than one CTA (one alone without the code of waits and sends: FP32 64^3 with
// four levels 2.05 instead of 2.17 ms)
template <typename T, int PER, typename GC, bool MULTI>
__global__ void __launch_bounds__(SL_MAX_THREADS) coarse_slab_k(T *gv, const T *__restrict__ gf, T *gr,
                                                                const uint32_t *__restrict__ l0,
                                                                const uint32_t *__restrict__ l1, SlabTab tab, Dims d,
                                                                GC gc, LapC<T> lc, double tol, int *err,
                                                                int *outer_out)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ __align__(8) unsigned long long mbar[2];
    __shared__ unsigned bnd[2 * (SL_MAX_CTAS + 1)], nexp[2], nrecv[2], cflag, stop;
    const SlabLayout lay(tab.cap, tab.win, tab.ctas, sizeof(T));
    const unsigned win = tab.win, len = lay.len;
    const uint32_t c = MULTI ? cl_rank() : 0u, cn = MULTI ? cl_size() : 1u;
    const int nx = (int)d.nx, nxny = (int)d.nxny();
    const unsigned n = (unsigned)d.n();
    const int tid = (int)threadIdx.x;
    T *v[2] = {(T *)(smraw + lay.v[0]), (T *)(smraw + lay.v[1])};
    T *blk = (T *)(smraw + lay.blk), *bc = (T *)(smraw + lay.bc);
    uint32_t *exp[2] = {(uint32_t *)(smraw + lay.exp[0]), (uint32_t *)(smraw + lay.exp[1])};
    uint8_t *need = smraw + lay.need;  // [colour][slot]: a received value some voxel of the chunk reads
    const uint32_t *list[2] = {l0, l1};
    chain_early();
    if (tid < 2) {
        nexp[tid] = 0;
        nrecv[tid] = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sl_addr(&mbar[tid])) : "memory");
    }
    if (tid == 0) {
        cflag = 0;
        stop = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int t = tid; t < RED_NBLK; t += blockDim.x) blk[t] = (T)0;
    for (unsigned t = tid; t < 2 * len; t += blockDim.x) v[0][t] = (T)0;  // both colours: the arrays are adjacent
    if (cn > 1)
        for (unsigned t = tid; t < 2 * len; t += blockDim.x) need[t] = 0;
    chain_wait();
    const int failed = *(const volatile int *)err;
    for (int t = tid; t < 2 * ((int)cn + 1); t += blockDim.x) bnd[t] = tab.cut[2 * (t / 2 * (SL_MAX_CTAS / (int)cn)) + t % 2];
    __syncthreads();
    if (failed) return;  // an earlier wait ran out (the whole cluster reads the same)
    const unsigned start[2] = {bnd[2 * c], bnd[2 * c + 1]};
    const unsigned cnt[2] = {bnd[2 * c + 2] - start[0], bnd[2 * c + 3] - start[1]};
    list[0] += start[0];
    list[1] += start[1];

    const uint32_t va[2] = {sl_addr(v[0]), sl_addr(v[1])};
    SlabShare<T, PER> S[2];
    int nzb = 0;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const unsigned e = (unsigned)tid + u * blockDim.x;
            S[q].meta[u] = 0;
            S[q].f[u] = (T)0;
#pragma unroll
            for (int k = 0; k < 6; ++k) S[q].a[u][k] = va[q ^ 1];
            if (e >= cnt[q]) continue;
            const uint32_t le = list[q][e];
            const uint32_t l = le & BL_IDX;
            const T fv = gf[l], vv = gv[l];
            S[q].f[u] = fv;
            v[q][win + e] = vv;
            nzb |= sizeof(T) == 8 ? (__double_as_longlong((double)fv) | __double_as_longlong((double)vv)) != 0
                                  : (__float_as_int((float)fv) | __float_as_int((float)vv)) != 0;
            uint32_t meta = SL_ON | (le & BL_I1 ? SL_I1 : 0u) | (le & BL_INX2 ? SL_INX2 : 0u);
            const int off[6] = {-1, 1, -nx, nx, -nxny, nxny};
            uint32_t slot[6], owner[6];
            const int qn = q ^ 1;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const uint32_t m = (uint32_t)((int)l + off[k]);
                const unsigned p = tab.pos[m];
                owner[k] = c;
                if (p == SL_NONE) {
                    slot[k] = len - 1;  // holds +0
                    const T x = gv[m];
                    const bool zero = sizeof(T) == 8 ? __double_as_longlong((double)x) == 0 : __float_as_int((float)x) == 0;
                    if (!zero) {
                        meta |= 1u << (SL_GLOB + k);
                        nzb = 1;
                    }
                    continue;
                }
                slot[k] = p + win - start[qn];
                if (p < start[qn] || p >= start[qn] + cnt[qn]) {  // another chunk's
                    uint32_t o = 0;
                    while (p >= bnd[2 * (o + 1) + qn]) ++o;
                    owner[k] = o;
                    meta |= SL_HALO;
                    v[qn][slot[k]] = gv[m];
                    need[qn * len + slot[k]] = 1;
                }
            }
#pragma unroll
            for (int k = 0; k < 6; ++k) S[q].a[u][k] = va[qn] + slot[k] * (uint32_t)sizeof(T);
            if (meta & SL_HALO) {
                // where this voxel's value goes: each chunk that holds a neighbour, once
                uint32_t tgt[6];
                int nt = 0;
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    bool isnew = owner[k] != c;
#pragma unroll
                    for (int j = 0; j < 6; ++j)
                        if (j < k && owner[j] == owner[k]) isnew = false;
                    if (isnew) tgt[nt++] = owner[k];
                }
                const unsigned at = atomicAdd(&nexp[q], (unsigned)nt);
                for (int j = 0; j < nt; ++j)
                    exp[q][at + j] = tgt[j] << 16 | (start[q] + e + win - bnd[2 * tgt[j] + q]);
                meta |= at | (uint32_t)nt << 16;
            }
            S[q].meta[u] = meta;
        }
    }
    const int any_nz = __syncthreads_or(nzb);
    if (cn > 1) {
        unsigned r0 = 0, r1 = 0;
        for (unsigned t = tid; t < len; t += blockDim.x) {
            r0 += need[t];
            r1 += need[len + t];
        }
        if (r0) atomicAdd(&nrecv[0], r0);
        if (r1) atomicAdd(&nrecv[1], r1);
    }
    // every chunk has loaded the values around it (and its barriers are set) before any is sent
    cl_sync();
    uint32_t bytes[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        bytes[q] = nrecv[q] ? nrecv[q] * (uint32_t)sizeof(T) + tab.extra : 0u;
        // thread 0 waits for every phase that bytes complete (SL_PASS says why); it has a
        // voxel then, as one of the other colour reads those
        if (tid == 0 && nrecv[q]) S[q ^ 1].meta[0] |= SL_HALO;
    }
    const uint32_t mb[2] = {sl_addr(&mbar[0]), sl_addr(&mbar[1])};
    const SlabCol col[2] = {{va[0] + (win + tid) * (uint32_t)sizeof(T), va[0], mb[0], exp[0], list[0]},
                            {va[1] + (win + tid) * (uint32_t)sizeof(T), va[1], mb[1], exp[1], list[1]}};
    // An idle solve: no voxel to update anywhere, or f and every value read +0.  Its
    // sweeps change nothing, so each outer iteration repeats the first exactly.
    if (tid < (int)cn) {
        const unsigned bits = (cnt[0] + cnt[1] > 0 ? 1u : 0u) | (any_nz ? 2u : 0u);
        if (bits) cl_or(cl_map(&cflag, (uint32_t)tid), bits);
    }
    const T ff = sl_lane_sum(gf, n, blk, bc, c, cn);
    const double fn = sizeof(T) == 4 ? (double)sqrtf((float)ff) : sqrt((double)ff);
    const double reltol = tol * fn;
    const bool idle = cflag != 3u;
    const bool r1first = ((nx + 1) & 1) != 0;  // reverse sweeps begin with colour 1
    unsigned done[2] = {0, 0};                 // passes of each colour so far
    int dead = 0, arm = cn > 1 && tid == 0;
    // one pass of colour Q: reads the other colour's values of its last pass.  Thread 0
    // arms the barrier of Q's values.  It has waited itself for that barrier's last phase,
    // in the pass before (SL_HALO is set for it): a phase still open must not be armed.
#define SL_PASS(Q, SKIP)                                                                                            \
    do {                                                                                                            \
        if (MULTI && arm) sl_arm(mb[Q], bytes[Q]);                                                                  \
        slab_pass<T, PER, GC, MULTI>(S[Q], col[Q], SKIP, gc, gv, nx, nxny, mb[1 - (Q)], (done[1 - (Q)] - 1) & 1u,              \
                          done[1 - (Q)] > 0, tab.tries, dead, arm);                                                 \
        ++done[Q];                                                                                                  \
    } while (0)
    int outer = 0;
    bool stopped = false;
    for (int it = 0; it < 1024; ++it) {
        outer = it + 1;
        if (r1first) {
            for (int s = 0; s < 127; ++s) {
                SL_PASS(1, 0u);
                SL_PASS(0, SL_INX2);
            }
            SL_PASS(1, 0u);  // the pass of colour 0 that would follow is the next one's
        } else {
            for (int s = 0; s < 128; ++s) {
                SL_PASS(0, 0u);
                SL_PASS(1, SL_INX2);
            }
        }
        for (int s = 0; s < 128; ++s) {
            SL_PASS(0, 0u);
            SL_PASS(1, SL_I1);
        }
        if (cn > 1 && !dead) {
            if (!sl_wait(mb[0], (done[0] - 1) & 1u, tab.tries) || !sl_wait(mb[1], (done[1] - 1) & 1u, tab.tries)) dead = 1;
        }
        if (dead) sl_stop(&stop);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                if (!(S[q].meta[u] & SL_ON)) continue;
                const unsigned e = (unsigned)tid + u * blockDim.x;
                const size_t l = list[q][e] & BL_IDX;
                T x[6];
#pragma unroll
                for (int k = 0; k < 6; ++k) x[k] = sl_ld(S[q].a[u][k], T());
                if (S[q].meta[u] >> SL_GLOB) slab_globals<T>(x, S[q].meta[u] >> SL_GLOB, gv, l, nx, nxny);
                gr[l] = S[q].f[u] + (lc.hh * v[q][win + e] + lc.hx * (x[0] + x[1]) + lc.hy * (x[2] + x[3]) +
                                     lc.hz * (x[4] + x[5]));
            }
        }
        cl_sync();
        if (cn > 1 && *(volatile unsigned *)&stop) {  // (the same in every CTA: set before its setter arrived)
            stopped = true;
            sl_settle();
            break;
        }
        const T rr = sl_lane_sum(gr, n, blk, bc, c, cn);
        const double rn = sizeof(T) == 4 ? (double)sqrtf((float)rr) : sqrt((double)rr);
        if (rn < reltol) break;
        if (idle) {
            outer = 1024;
            break;
        }
    }
#undef SL_PASS
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int u = 0; u < PER; ++u)
            if (S[q].meta[u] & SL_ON) {
                const unsigned e = (unsigned)tid + u * blockDim.x;
                gv[list[q][e] & BL_IDX] = v[q][win + e];
            }
    if (stopped && tid == 0) atomicExch(err, 1);
    if (c == 0 && tid == 0 && outer_out) *outer_out += outer;
    cl_sync();  // no CTA leaves while a peer may still address its shared memory
}
