// Coarsest-level solver over the whole GPU (mgpcg_mex.c:265-275), included by
// mg.cu inside namespace qsm: the form for passes of more voxels than one
// cluster's FP64 pipes take quickly (lbv's shallow hierarchies: ~5-16k FP64
// updates per colour).
//
// One CTA per SM (cooperative launch), each with an equal share of both colour
// lists in index order, so a voxel's x and most y neighbours lie in the CTA's
// shared memory and its z neighbours in other CTAs.  Values go between CTAs as
// packets in global memory: the value and the number of the pass that wrote it
// in one 16-byte (FP32: 8-byte) store, which the reader polls until the pass
// it needs is there.  No barrier joins the CTAs during the sweeps and nothing
// is fenced: a packet is one memory transaction.  The sum over the neighbours
// that lie in shared memory is formed before the poll.
//
// Why no packet is overwritten before it is read: a voxel's packet of pass p is
// read by its neighbours in pass p + 1 only, and it is written again in pass
// p + 2 at the earliest, after its thread has read those neighbours' packets of
// pass p + 1.  A voxel that a pass leaves as it is (the reference's quirk
// columns) publishes its value under the new pass number without waiting; a
// reader then may see a later number, with the same value.  So a reader takes
// any number from the one it needs on.  The passes alternate strictly between
// the colours (mg_slab.cuh says which pass that leaves out, and why).
//
// Every poll is bounded; one that runs out sets the error word, and the CTAs
// leave at the next grid barrier (there are three per outer iteration, around
// the residual and its norm).
//
// Bound by latency: a packet takes 700-1030 cycles from store to a successful
// poll (measured alone), then five dependent FP64 operations of 64 cycles each
// and the CTA's barrier; 1.2-1.5 us a pass against 2.6 us with a barrier of the
// grid.  Measured: see plan_coarse_grid.

constexpr int FL_THREADS = 512;  // most threads of a CTA, one voxel of each colour per thread
constexpr int FL_SPIN_LIMIT = 1 << 20;  // polls of a packet before a wait gives up (seconds)

// What the two passes of step s = 0 .. 255 of an outer iteration leave out: its
// 128 reverse and 128 forward sweeps as strictly alternating passes.  With
// reverse sweeps that begin with colour 1 the sequence is
// 1 0 1 0 ... 1 | 0 1 0 1 ... 0 1 (the last reverse pass of colour 0 left out),
// so the steps straddle the sweeps and the last one has its first pass only.
struct SweepSkip {
    uint32_t first, second;
    bool only_first;
};
__device__ __forceinline__ SweepSkip sweep_skip(bool r1first, int s, uint32_t i1, uint32_t inx2)
{
    if (r1first) return SweepSkip{s >= 128 ? i1 : 0u, s < 127 ? inx2 : 0u, s == 255};
    return SweepSkip{0u, s < 128 ? inx2 : i1, false};
}

template <typename T> struct FlowPkt;
template <> struct FlowPkt<double> { unsigned long long v, tag; };
template <> struct FlowPkt<float> { unsigned v, tag; };

__device__ __forceinline__ void fl_put(FlowPkt<double> *p, double v, unsigned tag)
{
    asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"((unsigned long long)tag)
                 : "memory");
}
__device__ __forceinline__ void fl_put(FlowPkt<float> *p, float v, unsigned tag)
{
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p),
                 "l"((unsigned long long)tag << 32 | (unsigned)__float_as_int(v))
                 : "memory");
}
__device__ __forceinline__ void fl_get(const FlowPkt<double> *p, double &v, unsigned &tag)
{
    unsigned long long a, b;
    asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
                 : "=l"(a), "=l"(b)
                 : "l"(p)
                 : "memory");
    v = __longlong_as_double((long long)a);
    tag = (unsigned)b;
}
__device__ __forceinline__ void fl_get(const FlowPkt<float> *p, float &v, unsigned &tag)
{
    unsigned long long a;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
    v = __int_as_float((int)(unsigned)a);
    tag = (unsigned)(a >> 32);
}

// 0, known only once x is computed
__device__ __forceinline__ uint32_t fl_after(double x)
{
    uint32_t r;
    asm volatile("{\n\t.reg .b32 h, l;\n\tmov.b64 {l, h}, %1;\n\tand.b32 %0, h, 0;\n\t}" : "=r"(r) : "d"(x));
    return r;
}
__device__ __forceinline__ uint32_t fl_after(float x)
{
    uint32_t r;
    asm volatile("and.b32 %0, %1, 0;" : "=r"(r) : "r"(__float_as_int(x)));
    return r;
}
// A thread's voxel of one colour.
template <typename T>
struct FlowVox {
    uint32_t a[6];  // a neighbour's shared-memory address (that of +0 outside G), or the entry in its list
    uint32_t l, p;  // its index, its entry in its list
    uint32_t meta;  // FL_ON, the quirk flags, neighbours to poll (bits 0-5), to read from v (bits 6-11)
    T f;
};
constexpr uint32_t FL_ON = 1u << 12, FL_I1 = 1u << 13, FL_INX2 = 1u << 14, FL_SEND = 1u << 15;
constexpr uint32_t FL_XYREM = 1u << 16;  // a voxel of the warp has an x or y neighbour in another CTA

// Neighbour k's value: in shared memory, or constant in gv (an initial guess outside G).
template <typename T>
__device__ __forceinline__ T flow_local(const FlowVox<T> &V, int k, const T *gv, int off)
{
    if (V.meta >> (6 + k) & 1u) return __ldcg(gv + (ptrdiff_t)V.l + off);
    return sl_ld(V.a[k], T());
}

// One colour pass of the CTA: the other colour's packets (pn) must be of pass
// `need` or later, this pass is number `tag`.  A warp whose x and y neighbours
// are all local forms their sum before it polls: a poll issued at once would
// find the pass before, and a second one costs another round trip (190^2 x 110
// FP64 solve: 76 ms polling first, 61 ms so).  The other warps, on whose packets
// the next CTAs wait, poll at once (a pause of 300 cycles there: 67 ms).
template <typename T>
__device__ __forceinline__ void flow_pass(const FlowVox<T> &V, uint32_t own, uint32_t skip, const GsC<T> &c, const T *gv,
                                          FlowPkt<T> *po, const FlowPkt<T> *pn, int nx, int nxny, unsigned need,
                                          unsigned tag, int polls, int &dead)
{
    if (V.meta & FL_ON) {
        T val;
        if (V.meta & skip) {
            val = sl_ld(own, T());
        } else {
            const int off[6] = {-1, 1, -nx, nx, -nxny, nxny};
            T x[6], y[6];
            unsigned tg[6];
#pragma unroll
            for (int k = 0; k < 6; ++k)
                if (!(V.meta >> k & 1u)) x[k] = flow_local<T>(V, k, gv, off[k]);
            T sum = (T)0;
            if (!(V.meta & FL_XYREM)) sum = c.hx * (x[0] + x[1]) + c.hy * (x[2] + x[3]);
            const uint32_t hold = fl_after(sum);
            uint32_t pend = V.meta & 63u;
#pragma unroll
            for (int k = 5; k >= 0; --k)
                if (V.meta >> k & 1u) fl_get(pn + (V.a[k] + hold), y[k], tg[k]);
            for (int tries = 0;;) {
#pragma unroll
                for (int k = 0; k < 6; ++k)
                    if ((pend >> k & 1u) && ((int)(tg[k] - need) >= 0 || dead)) {
                        x[k] = y[k];
                        pend &= ~(1u << k);
                    }
                if (!pend) break;
                if (++tries > polls) dead = 1;
#pragma unroll
                for (int k = 0; k < 6; ++k)
                    if (pend >> k & 1u) fl_get(pn + V.a[k], y[k], tg[k]);
            }
            if (V.meta & FL_XYREM) sum = c.hx * (x[0] + x[1]) + c.hy * (x[2] + x[3]);
            val = c.hh * (V.f + (sum + c.hz * (x[4] + x[5])));
        }
        if (V.meta & FL_SEND) fl_put(po + V.p, val, tag);
        sl_st(own, val);
    }
    __syncthreads();
}

// This CTA's share of colour q's list: entries [lo, hi).
__device__ __forceinline__ void flow_share(unsigned cnt, unsigned &lo, unsigned &hi)
{
    lo = (unsigned)((unsigned long long)cnt * blockIdx.x / gridDim.x);
    hi = (unsigned)((unsigned long long)cnt * (blockIdx.x + 1) / gridDim.x);
}

template <typename T>
__global__ void __launch_bounds__(FL_THREADS) coarse_flow_k(T *v, const T *__restrict__ f, T *r,
                                                            const uint32_t *__restrict__ l0, unsigned c0,
                                                            const uint32_t *__restrict__ l1, unsigned c1,
                                                            const unsigned *__restrict__ pos, FlowPkt<T> *pk, Dims d,
                                                            GsC<T> gc, LapC<T> lc, double tol, GridBar gb, T *part,
                                                            int *outer_out)
{
    __shared__ T val[2][FL_THREADS + 1];  // the CTA's values of each colour; the last one is +0
    __shared__ T tot;
    const int nx = (int)d.nx, nxny = (int)d.nxny();
    const size_t n = d.n();
    const int tid = (int)threadIdx.x;
    const uint32_t *list[2] = {l0, l1};
    const unsigned cnt[2] = {c0, c1};
    unsigned lo[2], hi[2];
    flow_share(c0, lo[0], hi[0]);
    flow_share(c1, lo[1], hi[1]);
    if (tid < 2) val[tid][FL_THREADS] = (T)0;
    const bool r1first = ((nx + 1) & 1) != 0;  // the sweeps begin with colour 1
    FlowVox<T> V[2];
#pragma unroll
    for (int z = 0; z < 2; ++z) {
        const int q = z ^ (r1first ? 1 : 0);
        const unsigned e = lo[q] + (unsigned)tid;
        V[z].meta = 0;
        if (e >= hi[q]) continue;
        const uint32_t le = list[q][e], l = le & BL_IDX;
        uint32_t meta = FL_ON | (le & BL_I1 ? FL_I1 : 0u) | (le & BL_INX2 ? FL_INX2 : 0u);
        const int off[6] = {-1, 1, -nx, nx, -nxny, nxny};
        const int qn = q ^ 1;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const uint32_t m = (uint32_t)((int)l + off[k]);
            const unsigned p = pos[m];
            unsigned slot = FL_THREADS;
            if (p == SL_NONE) {
                const T x = v[m];
                const bool zero = sizeof(T) == 8 ? __double_as_longlong((double)x) == 0 : __float_as_int((float)x) == 0;
                if (!zero) meta |= 1u << (6 + k);
            } else if (p >= lo[qn] && p < hi[qn]) {
                slot = p - lo[qn];
            } else {
                meta |= 1u << k | FL_SEND;  // a neighbour elsewhere: each reads the other
            }
            V[z].a[k] = meta >> k & 1u ? p : sl_addr(&val[qn][slot]);
        }
        V[z].l = l;
        V[z].p = e;
        V[z].f = f[l];
        V[z].meta = meta;
        val[q][tid] = v[l];
        if (meta & FL_SEND) fl_put(pk + (q ? c0 : 0u) + e, v[l], 0u);
    }
#pragma unroll
    for (int z = 0; z < 2; ++z)
        if (__any_sync(0xffffffffu, (V[z].meta & 15u) != 0)) V[z].meta |= V[z].meta ? FL_XYREM : 0u;
    const unsigned nb = (unsigned)lane_blocks(n);
    if (blockIdx.x == 0)
        for (unsigned b = nb + tid; b < RED_NBLK; b += blockDim.x) part[b] = (T)0;
    unsigned bk = 0;  // barriers passed
    T ff;
    // (its barrier also orders the packets of pass 0 before the first poll)
    if (!grid_lane_sum(f, n, part, &tot, gb, bk, &ff)) return;
    const double fn = sizeof(T) == 4 ? (double)sqrtf((float)ff) : sqrt((double)ff);
    const double reltol = tol * fn;
    // index 0: the colour the sweeps begin with (V and list are in that order)
    const uint32_t own[2] = {sl_addr(&val[r1first ? 1 : 0][tid]), sl_addr(&val[r1first ? 0 : 1][tid])};
    FlowPkt<T> *pk0 = pk + (r1first ? c0 : 0u), *pk1 = pk + (r1first ? 0u : c0);
    unsigned tag = 0, last0 = 0, last1 = 0;  // passes so far, the last one of each colour
    int dead = 0;
    int outer = 0;
    for (int it = 0; it < 1024; ++it) {
        outer = it + 1;
        for (int s = 0; s < 256; ++s) {
            const SweepSkip k = sweep_skip(r1first, s, FL_I1, FL_INX2);
            flow_pass<T>(V[0], own[0], k.first, gc, v, pk0, pk1, nx, nxny, last1 + gb.ahead, ++tag, gb.polls, dead);
            last0 = tag;
            if (k.only_first) break;
            flow_pass<T>(V[1], own[1], k.second, gc, v, pk1, pk0, nx, nxny, last0 + gb.ahead, ++tag, gb.polls, dead);
            last1 = tag;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (V[q].meta & FL_ON) v[V[q].l] = sl_ld(own[q], T());
        if (dead) atomicExch(gb.err, 1);
        if (!grid_bar(gb, bk)) return;
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (V[q].meta & FL_ON) {
                const size_t l = V[q].l;
                r[l] = V[q].f + (lc.hh * sl_ld(own[q], T()) + lc.hx * (__ldcg(v + l - 1) + __ldcg(v + l + 1)) +
                                 lc.hy * (__ldcg(v + l - nx) + __ldcg(v + l + nx)) +
                                 lc.hz * (__ldcg(v + l - nxny) + __ldcg(v + l + nxny)));
            }
        if (!grid_bar(gb, bk)) return;
        T rr;
        if (!grid_lane_sum(r, n, part, &tot, gb, bk, &rr)) return;
        const double rn = sizeof(T) == 4 ? (double)sqrtf((float)rr) : sqrt((double)rr);
        if (rn < reltol) break;
        if (cnt[0] + cnt[1] == 0) {  // no G voxel: every later outer iteration repeats this one exactly
            outer = 1024;
            break;
        }
    }
    if (blockIdx.x == 0 && tid == 0 && outer_out) *outer_out += outer;
}
