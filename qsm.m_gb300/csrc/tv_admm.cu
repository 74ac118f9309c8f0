// FFT total-variation inversion (ADMM) of src/inversion/tv.m:101-277 on the
// GPU: the data term's solve u = real(ifft3(iA .* (F + fft3(r)))) runs as a
// cuFFT R2C, one fused pointwise k-space kernel, and a cuFFT C2R; the
// gradient, shrinkage, multiplier update and residual norms are fused
// stencil kernels.  tv.m's stopping test and rho update (:226-268) run on the
// device (tv_ctl, FP64, the host's arithmetic), so iterations are queued
// without a host round trip; the host reads the control state every eighth
// iteration.
//
// k-space terms come from per-axis tables and two values stored per half-spectrum point:
//   D(k) = 1/3 - (k.b)^2/|k|^2, D(0) = 0, k_a = fftfreq(n_a, h_a)
//        (dipoleKernel.m:56-65, ifftshifted so DC is first), stored once per
//        solve in the working precision;
//   L(k) = sum_a (2/h_a^2)(1 - cos(2 pi i_a/n_a)), the symbol of the negated
//        7-point Laplacian (laplaceKernel.m, tv.m:140-142): the sum of three 1-D
//        tables' FP64 terms, stored beside D;
//   iA   = 1/(mu D^2 + rho L), 0 where not finite (tv.m:144-145), formed in
//        the k-space kernel, so a rho update costs nothing.
// No trigonometry and one division per point per iteration: FP64 arithmetic
// runs at a small fraction of the FP32 rate on this GPU.  u = real(ifft3(X))
// equals the C2R of the Hermitian part of X; the stored half spectrum
// therefore carries, on planes where index negation is not frequency
// negation (even-size Nyquist planes) and B0 is oblique, the average of the
// multipliers at k and at the negated index.
//
// FP64 (the MATLAB default class) or FP32 arithmetic by dtype; every
// reduction accumulates in FP64 with a fixed order (block partials folded
// in block order), so results are run-to-run deterministic.
#include <math.h>
#include <stdio.h>

#include <algorithm>

#include "common.cuh"
#include "fft_plans.cuh"

namespace qsm {

template <typename T> struct CxT;
template <> struct CxT<double> { using type = cufftDoubleComplex; };
template <> struct CxT<float> { using type = cufftComplex; };
template <typename T> struct alignas(2 * sizeof(T)) DL {
    T D, L;
};

constexpr int TV_BLOCK = 256;
// Grid-stride kernels run a fixed, fully resident grid (the block partials of the
// reductions then have a fixed count and order): 5 blocks of 256 threads per SM
// in FP32 (<= 51 registers), 3 in FP64 (<= 85 registers).
template <typename T> struct TvOcc { static constexpr int minb = sizeof(T) == 4 ? 5 : 3; };
template <typename T> constexpr int tv_grid() { return 152 * TvOcc<T>::minb; }
// grad_shrink_k needs more registers in FP32 (it spills at 48): 4 blocks per SM
template <typename T> struct TvOccGS { static constexpr int minb = sizeof(T) == 4 ? 4 : 3; };
constexpr int TV_GRID_MAX = 152 * 5;
constexpr int TV_NSUM = 5;         // nr, na, nb, ||s||^2, ||rho grad' l||^2
// ADMM control state on the device (doubles): rho and its inverse, the last
// iteration's residuals and tolerances, the rho-schedule flag, done, iteration
enum { C_RHO, C_IRHO, C_NR, C_NS, C_NA, C_NB, C_EP, C_ED, C_FLAG, C_DONE, C_IT, C_N };

struct TvK {
    int nx, ny, nz, nxh;   // real dims, half-spectrum x extent
    double hx, hy, hz;     // voxel size
    double bx, by, bz;     // unit B0 direction
    double mu;
    bool oblique;          // B0 has two or more non-zero components
};

struct Vox {
    size_t l, NX, NY, NZ;
    int i, j, k;
};

// The voxels of a grid-stride loop in order, with their (i, j, k) advanced by
// carries instead of a 64-bit division per voxel: the stride is split into
// (si, sj, sk) once per thread.
struct VoxWalk {
    Vox v;
    size_t S;
    int si, sj, sk, nx, ny;
    __device__ __forceinline__ VoxWalk(size_t l0, size_t stride, const Dims &d)
    {
        nx = (int)d.nx;
        ny = (int)d.ny;
        v.l = l0;
        v.i = (int)(l0 % d.nx);
        v.j = (int)((l0 / d.nx) % d.ny);
        v.k = (int)(l0 / d.nxny());
        v.NX = d.nx - 1;
        v.NY = d.nx * (d.ny - 1);
        v.NZ = d.nxny() * (d.nz - 1);
        S = stride;
        si = (int)(stride % d.nx);
        sj = (int)((stride / d.nx) % d.ny);
        sk = (int)(stride / d.nxny());
    }
    __device__ __forceinline__ void next()
    {
        v.l += S;
        v.i += si;
        int c = v.i >= nx;
        v.i -= c ? nx : 0;
        v.j += sj + c;
        c = v.j >= ny;
        v.j -= c ? ny : 0;
        v.k += sk + c;
    }
};

#define VOX_LOOP(W, D)                                                                                  \
    for (VoxWalk W((size_t)blockIdx.x * blockDim.x + threadIdx.x, (size_t)gridDim.x * blockDim.x, D); \
         W.v.l < (D).n(); W.next())

__device__ __forceinline__ double fftfreq(int i, int n, double h) { return (double)(i <= (n - 1) / 2 ? i : i - n) / (n * h); }

// per-axis tables: frequencies fx[nxh] fy[ny] fz[nz], then the Laplacian terms
// Lx[nxh] Ly[ny] Lz[nz] (FP64)
__global__ void ktab_k(double *tab, TvK K)
{
    const int na[3] = {K.nxh, K.ny, K.nz}, nn[3] = {K.nx, K.ny, K.nz};
    const double hh[3] = {K.hx, K.hy, K.hz};
    const int tot = K.nxh + K.ny + K.nz;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += gridDim.x * blockDim.x) {
        int a = 0, i = t;
        while (i >= na[a]) i -= na[a++];
        tab[t] = fftfreq(i, nn[a], hh[a]);
        tab[tot + t] = (2.0 / (hh[a] * hh[a])) * (1.0 - cospi(2.0 * i / nn[a]));
    }
}

__device__ __forceinline__ double dipole_at(const TvK &K, double fx, double fy, double fz)
{
    const double kb = K.bx * fx + K.by * fy + K.bz * fz;
    const double k2 = fx * fx + fy * fy + fz * fz;
    return 1.0 / 3.0 - (kb * kb) / k2;
}

// D and L on the half spectrum, rounded to the working precision (L's two FP64 sums
// per point in every kmul_k took that kernel to 24.3 us at 224 x 224 x 128 in FP32; with
// L from here 21.9, with two points a step 13.6)
template <typename T>
__global__ void dl_k(DL<T> *dl, const double *__restrict__ tab, TvK K)
{
    const size_t nh = (size_t)K.nxh * K.ny * K.nz;
    const int tot = K.nxh + K.ny + K.nz;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < nh; q += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(q % K.nxh), j = (int)((q / K.nxh) % K.ny), k = (int)(q / ((size_t)K.nxh * K.ny));
        DL<T> o;
        o.D = q == 0 ? (T)0 : (T)dipole_at(K, tab[i], tab[K.nxh + j], tab[K.nxh + K.ny + k]);
        o.L = (T)((tab[tot + i] + tab[tot + K.nxh + j]) + tab[tot + K.nxh + K.ny + k]);
        dl[q] = o;
    }
}

template <typename T>
__device__ __forceinline__ T inv_a(T K, T L, T rho)
{
    const T a = (T)1 / (K + rho * L);
    return isfinite(a) ? a : (T)0;
}

// X = iA .* (mu D .* fhat + R) / N in place of R (tv.m:172-175), in the working
// precision T
template <typename T>
__global__ void __launch_bounds__(TV_BLOCK, TvOcc<T>::minb) kmul_k(typename CxT<T>::type *R, const typename CxT<T>::type *__restrict__ fhat,
                       const DL<T> *__restrict__ dl, const double *__restrict__ tab, TvK K, const double *ctl, double invn_)
{
    const T mu = (T)K.mu, rho = (T)ctl[C_RHO], invn = (T)invn_;
    const Dims hd{(size_t)K.nxh, (size_t)K.ny, (size_t)K.nz};
    // two points a step, their loads first: one alone leaves HBM at 40 % (latency)
    using C = typename CxT<T>::type;
    const auto point = [&](const Vox &w, const DL<T> &e, const C &fh, const C &r) {
        const int i = w.i, j = w.j, k = w.k;
        const T D = e.D, L = e.L;
        T a = inv_a<T>(mu * D * D, L, rho), ad = a * (mu * D);
        if (K.oblique && ((2 * i == K.nx) || (2 * j == K.ny) || (2 * k == K.nz))) {
            // the negated index keeps Nyquist frequencies and flips the others
            const double fx = tab[i], fy = tab[K.nxh + j], fz = tab[K.nxh + K.ny + k];
            const double gx = 2 * i == K.nx ? fx : -fx, gy = 2 * j == K.ny ? fy : -fy, gz = 2 * k == K.nz ? fz : -fz;
            const T D2 = (T)dipole_at(K, gx, gy, gz);
            const T a2 = inv_a<T>(mu * D2 * D2, L, rho);
            ad = (T)0.5 * (ad + a2 * (mu * D2));
            a = (T)0.5 * (a + a2);
        }
        C o;
        o.x = (ad * fh.x + a * r.x) * invn;
        o.y = (ad * fh.y + a * r.y) * invn;
        R[w.l] = o;
    };
    const size_t n = hd.n();
    VOX_LOOP(wk, hd) {
        const Vox w = wk.v;
        const DL<T> e = dl[w.l];
        const C fh = fhat[w.l], r = R[w.l];
        wk.next();
        const bool two = wk.v.l < n;
        DL<T> e2{};
        C f2{}, r2{};
        if (two) {
            e2 = dl[wk.v.l];
            f2 = fhat[wk.v.l];
            r2 = R[wk.v.l];
        }
        point(w, e, fh, r);
        if (two) point(wk.v, e2, f2, r2);
    }
}


// gradfp_adj_mex.c:156-257 of the field g_c(l) (h holds -1/h), with the
// reference's association order of the three axis terms.
template <typename T, typename G>
__device__ __forceinline__ T adj_at(const Vox &v, const Dims &d, const T *ih, G g)
{
    const size_t l = v.l;
    const T a = ih[0] * (g(0, l) - g(0, v.i > 0 ? l - 1 : l + v.NX));
    const T b = ih[1] * (g(1, l) - g(1, v.j > 0 ? l - d.nx : l + v.NY));
    const T c = ih[2] * (g(2, l) - g(2, v.k > 0 ? l - d.nxny() : l + v.NZ));
    return v.k == 0 ? (a + b) + c : v.j == 0 ? (c + a) + b : (c + b) + a;
}

// Work of the column kernels below: a warp takes 32 columns in x times R rows in y
// and walks along z.  The backward values it needs come from the lane before (x),
// its own previous row (y) and its own previous plane (z); only at the tile's
// first column, row and plane are they loaded or formed again.  A block's warps take
// neighbouring tiles of one range of planes, so the planes' addresses are the
// block's and a lane holds one offset in the plane per row (O: in bytes, 32 bits
// where a plane is below 4 GB), and no branch lies between the loads of a plane.
struct Tiles {
    unsigned cx, cols, groups;  // tiles along x, in a plane, and blocks' shares of a plane
    unsigned zc, items;         // planes of a chunk; groups x chunks
};

static Tiles tiles_of(const Dims &d, int rows, unsigned blocks)
{
    // the chunk length whose last round leaves the fewest blocks idle; a chunk's
    // start costs about a quarter of a plane
    Tiles t{};
    t.cx = (unsigned)((d.nx + 31) / 32);
    t.cols = t.cx * (unsigned)((d.ny + rows - 1) / rows);
    t.groups = (t.cols + TV_BLOCK / 32 - 1) / (TV_BLOCK / 32);
    double best = 0.0;
    for (unsigned m = 1; m <= 8; ++m) {
        const size_t ch = std::min(std::max<size_t>(1, (size_t)m * blocks / t.groups), d.nz);
        const size_t zc = (d.nz + ch - 1) / ch, items = t.groups * ((d.nz + zc - 1) / zc);
        const double cost = (double)((items + blocks - 1) / blocks) * ((double)zc + 0.25);
        if (t.zc == 0 || cost < best) {
            best = cost;
            t.zc = (unsigned)zc;
            t.items = (unsigned)items;
        }
    }
    return t;
}

// A lane's part of a block's item: its column (clamped to the volume: on says whether it
// is inside), rows j0 .. j0 + nr - 1 (row[]: past the volume the last again), the row
// before the tile (rb) and, in lane q, the column before the tile in row q (re); offsets
// in a plane.  A warp without a tile takes the last one again, with nr = 0.
template <typename T, typename O, int R>
struct TileAt {
    int j0, nr, x, xb;
    O row[R], rb, re;
    bool on;
    __device__ __forceinline__ TileAt(const Tiles &t, unsigned group, const Dims &d)
    {
        const int lane = (int)(threadIdx.x & 31u), nx = (int)d.nx, ny = (int)d.ny;
        unsigned c = group * (TV_BLOCK / 32) + threadIdx.x / 32;
        const bool live = c < t.cols;
        c = live ? c : t.cols - 1;
        const int ty = (int)(c / t.cx), i0 = 32 * (int)(c - (unsigned)ty * t.cx);
        x = i0 + lane;
        on = x < nx && live;
        x = x < nx ? x : nx - 1;
        xb = i0 > 0 ? i0 - 1 : nx - 1;
        j0 = ty * R;
        const int n = ny - j0 < R ? ny - j0 : R;
#pragma unroll
        for (int q = 0; q < R; ++q) row[q] = at(x, j0 + (q < n ? q : n - 1), nx);
        rb = at(x, j0 > 0 ? j0 - 1 : ny - 1, nx);
        re = at(xb, j0 + (lane < n ? lane : 0), nx);
        nr = live ? n : 0;
    }
    static __device__ __forceinline__ O at(int i, int j, int nx) { return ((O)j * (O)nx + (O)i) * (O)sizeof(T); }
};

template <typename T, typename O> __device__ __forceinline__ T &off(T *p, O o) { return *(T *)((char *)p + o); }
template <typename T, typename O> __device__ __forceinline__ const T &off(const T *p, O o) { return *(const T *)((const char *)p + o); }

// adj_at's sum of the three axis terms
template <typename T>
__device__ __forceinline__ T adj_sum(T a, T b, T c, bool j0, bool k0)
{
    return k0 ? (a + b) + c : j0 ? (c + a) + b : (c + b) + a;
}

// r = gradfp_adj(rho v - l) (tv.m:166-170).  Iteration ii also keeps u when
// the control state says iteration ii - 1 converged: the iterations the host
// launched past convergence overwrite u.  Bound by HBM (7 arrays): 224 x 224 x 128
// in FP32 40.9 us with a thread per voxel (12 loads each), 36.1 us in columns (1, 2 or 3 rows
// a warp: 41.4, 38.3, 36.8).
template <typename T> struct AdjTile { static constexpr int R = sizeof(T) == 4 ? 4 : 2, minb = sizeof(T) == 4 ? 5 : 3; };
template <typename T, typename O>
__global__ void __launch_bounds__(TV_BLOCK, AdjTile<T>::minb) adj_rhs_k(T *r, const T *__restrict__ v, const T *__restrict__ lm, Dims d, Tiles tl, T nx_, T ny_, T nz_,
                                       const double *ctl, int ii, T *usave, const T *__restrict__ u)
{
    constexpr int R = AdjTile<T>::R;
    const size_t N = d.n(), nxny = d.nxny();
    const T rho = (T)ctl[C_RHO];
    const bool save = ctl[C_DONE] != 0.0 && ctl[C_IT] == (double)(ii - 1);
    const int lane = (int)(threadIdx.x & 31u);
    for (unsigned it = blockIdx.x; it < tl.items; it += gridDim.x) {
        const unsigned chunk = it / tl.groups;
        const TileAt<T, O, R> t(tl, it - chunk * tl.groups, d);
        const unsigned k0 = chunk * tl.zc, k1 = min(k0 + tl.zc, (unsigned)d.nz);
        T gz[R];
        {
            const size_t pb = nxny * (k0 > 0 ? k0 - 1 : d.nz - 1);
#pragma unroll
            for (int q = 0; q < R; ++q) gz[q] = rho * off(v + 2 * N + pb, t.row[q]) - off(lm + 2 * N + pb, t.row[q]);
        }
        for (unsigned k = k0; k < k1; ++k) {
            const size_t pk = nxny * k;
            const T *v0 = v + pk, *v1 = v + N + pk, *v2 = v + 2 * N + pk;
            const T *m0 = lm + pk, *m1 = lm + N + pk, *m2 = lm + 2 * N + pk;
            T va[R][3], la[R][3];
#pragma unroll
            for (int q = 0; q < R; ++q) {
                va[q][0] = off(v0, t.row[q]);
                va[q][1] = off(v1, t.row[q]);
                va[q][2] = off(v2, t.row[q]);
                la[q][0] = off(m0, t.row[q]);
                la[q][1] = off(m1, t.row[q]);
                la[q][2] = off(m2, t.row[q]);
            }
            const T vb = off(v1, t.rb), lb = off(m1, t.rb);
            T ve = 0, le = 0;
            if (lane < R) {
                ve = off(v0, t.re);
                le = off(m0, t.re);
            }
            T gy = rho * vb - lb;
            const T ge = rho * ve - le;
#pragma unroll
            for (int q = 0; q < R; ++q) {
                T a[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) a[c] = rho * va[q][c] - la[q][c];
                const T e = __shfl_sync(0xffffffffu, ge, q);
                T gx = __shfl_up_sync(0xffffffffu, a[0], 1);
                gx = lane == 0 ? e : gx;
                const T s = adj_sum<T>(nx_ * (a[0] - gx), ny_ * (a[1] - gy), nz_ * (a[2] - gz[q]), q == 0 && t.j0 == 0, k == 0);
                gy = a[1];
                gz[q] = a[2];
                if (t.on && q < t.nr) {
                    if (save) off(usave + pk, t.row[q]) = off(u + pk, t.row[q]);
                    off(r + pk, t.row[q]) = s;
                }
            }
        }
    }
}

template <int NS>
__device__ __forceinline__ void block_sums(double *part, double (&acc)[NS])
{
    __shared__ double red[NS][TV_BLOCK];
    const int t = threadIdx.x;
#pragma unroll
    for (int q = 0; q < NS; ++q) red[q][t] = acc[q];
    __syncthreads();
    for (int s = TV_BLOCK / 2; s > 0; s >>= 1) {
        if (t < s)
#pragma unroll
            for (int q = 0; q < NS; ++q) red[q][t] += red[q][t + s];
        __syncthreads();
    }
    if (t == 0)
#pragma unroll
        for (int q = 0; q < NS; ++q) part[q * gridDim.x + blockIdx.x] = red[q][0];
}

// tv.m's stopping test and rho schedule (tv.m:226-268) for iteration ii, in
// FP64 with the host's operations and order (no fused multiply-add on either
// side), from the five sums of the iteration.  Nothing changes once done.
struct TvCtlOpts {
    double rtol, atolp, atold, rtau, stau, gamma;
};

__device__ void tv_ctl(double *ctl, const double *sums, const TvCtlOpts &o, int ii)
{
    if (ctl[C_DONE] != 0.0) return;
    const double nrp = ctl[C_NR];
    const double nr = sums[0], na = sums[1], nb = sums[2], ns = sqrt(sums[3]);
    const double ep = o.atolp + o.rtol * (na < nb ? nb : na);
    const double ed = o.atold + o.rtol * sqrt(sums[4]);
    ctl[C_NR] = nr;
    ctl[C_NS] = ns;
    ctl[C_NA] = na;
    ctl[C_NB] = nb;
    ctl[C_EP] = ep;
    ctl[C_ED] = ed;
    ctl[C_IT] = (double)ii;
    if (nr < ep && ns < ed) {
        ctl[C_DONE] = 1.0;
        return;
    }
    double rho = ctl[C_RHO], flag = ctl[C_FLAG];
    if (nr > o.stau * ns || (nr > o.rtau * nrp && flag < 3.0)) {
        rho = o.gamma * rho;
        ctl[C_IRHO] = 1.0 / rho;
        if (flag > 5.0) flag = 0.0;
    } else if (nr < ns / o.stau) {
        rho = rho / (o.gamma * o.gamma);
        ctl[C_IRHO] = 1.0 / rho;
        flag = flag + 1.0;
    }
    ctl[C_RHO] = rho;
    ctl[C_FLAG] = flag;
}

// Block partials and what becomes of them: sums 0..ns1-1 have nblk1 partials each (at
// part), sums ns1..ns1+ns2-1 have nblk2 each (after them).
struct TvFold {
    double *part;
    int ns1, nblk1, ns2, nblk2;
    unsigned *count;  // blocks done (0 between kernels)
    TvCtlOpts o;
    int ii;
};

// Fold by one block of TV_BLOCK threads in a fixed order: thread t adds partials t,
// t + 256, ... of every sum in turn, then one shared-memory tree over all sums
// together.  Thread q returns sum q.
__device__ __forceinline__ double fold_sums(const TvFold &F)
{
    __shared__ double red[TV_NSUM][TV_BLOCK];
    const int t = threadIdx.x, ns = F.ns1 + F.ns2;
#pragma unroll
    for (int q = 0; q < TV_NSUM; ++q) {
        double s = 0.0;
        if (q < ns) {
            const double *p = q < F.ns1 ? F.part + q * F.nblk1 : F.part + F.ns1 * F.nblk1 + (q - F.ns1) * F.nblk2;
            const int nb = q < F.ns1 ? F.nblk1 : F.nblk2;
            for (int b = t; b < nb; b += TV_BLOCK) s += __ldcg(p + b);
        }
        red[q][t] = s;
    }
    __syncthreads();
    for (int h = TV_BLOCK / 2; h > 0; h >>= 1) {
        if (t < h)
#pragma unroll
            for (int q = 0; q < TV_NSUM; ++q) red[q][t] += red[q][t + h];
        __syncthreads();
    }
    return t < ns ? red[t][0] : 0.0;
}

// End of an iteration's last kernel: the block that finishes last folds the sums and
// brings the control state up to date (two launches of one block each, 16 us with
// their gaps, before).  The other blocks have read the state at their start.
__device__ __forceinline__ void fold_last(const TvFold &F, double *ctl)
{
    __shared__ double sums[TV_NSUM];
    __shared__ bool last;
    __threadfence();
    if (threadIdx.x == 0) last = atomicAdd(F.count, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const double s = fold_sums(F);
    if (threadIdx.x < TV_NSUM) sums[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        *F.count = 0;
        tv_ctl(ctl, sums, F.o, F.ii);
    }
}

// grad, over-relaxation, shrinkage, multiplier update and the primal
// residual sums of one ADMM iteration (tv.m:185-221, :227-234)
template <typename T, bool ISO>
__global__ void __launch_bounds__(TV_BLOCK, TvOccGS<T>::minb)
grad_shrink_k(T *vn, const T *__restrict__ vo, T *lm, const T *__restrict__ u, Dims d, T hx, T hy, T hz, T alpha,
              const double *ctl, double *part)
{
    const T rho = (T)ctl[C_RHO], irho = (T)ctl[C_IRHO];
    const size_t N = d.n();
    PartialSum<T> ps[3];  // nr, na, nb
    VOX_LOOP(wk, d) {
        const Vox &v = wk.v;
        const size_t l = v.l;
        const T u0 = u[l];
        T dd[3];
        dd[0] = hx * ((v.i + 1 < (int)d.nx ? u[l + 1] : u[l - v.NX]) - u0);
        dd[1] = hy * ((v.j + 1 < (int)d.ny ? u[l + d.nx] : u[l - v.NY]) - u0);
        dd[2] = hz * ((v.k + 1 < (int)d.nz ? u[l + d.nxny()] : u[l - v.NZ]) - u0);
        T d1[3], r[3], w[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            d1[c] = alpha * dd[c] + ((T)1 - alpha) * vo[c * N + l];
            r[c] = d1[c] + irho * lm[c * N + l];
        }
        if (ISO) {
            T s = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
            s = (s - irho) * (T)(s > irho) / s;
            if (!isfinite(s)) s = (T)0;
#pragma unroll
            for (int c = 0; c < 3; ++c) w[c] = r[c] * s;
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const T m = fabs(r[c]) - irho;
                const T sg = r[c] > (T)0 ? (T)1 : r[c] < (T)0 ? (T)-1 : (T)0;
                w[c] = (m > (T)0 ? m : (T)0) * sg;
            }
        }
        // per-voxel norms in the working precision (as MATLAB computes them in
        // the class of f), summed in FP64
        T e2 = 0, a2 = 0, b2 = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            vn[c * N + l] = w[c];
            lm[c * N + l] = lm[c * N + l] + rho * (d1[c] - w[c]);
            const T e = dd[c] - w[c];
            e2 += e * e;
            a2 += dd[c] * dd[c];
            b2 += w[c] * w[c];
        }
        ps[0].add(sqrt(e2));
        ps[1].add(sqrt(a2));
        ps[2].add(sqrt(b2));
    }
    double acc[3] = {ps[0].get(), ps[1].get(), ps[2].get()};
    block_sums<3>(part, acc);
}

// Anisotropic TV in FP32: grad_shrink_k and adj_norms_k in one pass, so the new v
// and l are not read back.  The adjoint's backward values w - vo and l of a
// neighbour are the ones its owner forms: handed on inside the warp's columns
// (Tiles), formed again at their edges by the same arithmetic (bit-identical).  l is
// double-buffered (lmo in, lmn out) because those edges read the old value.
// Bound by HBM (13 arrays): 224 x 224 x 128 92.3 us with a thread per voxel, every
// backward value formed again (19 loads and 6 shrinkages each), 84 us in columns with
// the fold (~5 us) and without its own two launches (11 us): 280 instead of ~350 issued
// instructions a voxel bound it, not HBM (45 %).  Rows a warp and blocks an SM: 4, 2
// 84 us; 3, 3 82; 2, 3 or 1, 4 91; 2, 4 (spills) 100.
struct ShrinkC {
    float alpha, rho, irho;
};
// component c: w - vo and the new l from the gradient dd, the old v and l
__device__ __forceinline__ void shrink1(const ShrinkC &k, float dd, float vo, float lo, float &w, float &dv, float &ln)
{
    const float d1 = k.alpha * dd + (1.f - k.alpha) * vo;
    const float r = d1 + k.irho * lo;
    w = copysignf(fmaxf(fabsf(r) - k.irho, 0.f), r);
    ln = lo + k.rho * (d1 - w);
    dv = w - vo;
}

constexpr int GSN_R = 4, GSN_MINB = 2;
template <typename O>
__global__ void __launch_bounds__(TV_BLOCK, GSN_MINB)
grad_shrink_norms_k(float *vn, const float *__restrict__ vo, float *__restrict__ lmn, const float *__restrict__ lmo,
                    const float *__restrict__ u, Dims d, Tiles tl, float hx, float hy, float hz, float alpha, double *ctl,
                    float nx_, float ny_, float nz_, TvFold F)
{
    constexpr int R = GSN_R;
    const ShrinkC K{alpha, (float)ctl[C_RHO], (float)ctl[C_IRHO]};
    const size_t N = d.n(), nxny = d.nxny();
    const int lane = (int)(threadIdx.x & 31u), nx = (int)d.nx, ny = (int)d.ny;
    PartialSum<float> ps[5];  // nr, na, nb, ||s||^2, ||rho grad' l||^2
    for (unsigned it = blockIdx.x; it < tl.items; it += gridDim.x) {
        const unsigned chunk = it / tl.groups;
        const TileAt<float, O, R> t(tl, it - chunk * tl.groups, d);
        const unsigned k0 = chunk * tl.zc, k1 = min(k0 + tl.zc, (unsigned)d.nz);
        const bool last_x = t.x + 1 == nx, edge_x = lane == 31 || last_x;
        // from a row to the column after (periodic); the row after the tile's last; in lane q row q's first column
        const O fx = (last_x ? (O)0 - (O)t.x : (O)1) * (O)sizeof(float);
        const int n = ny - t.j0 < R ? ny - t.j0 : R;
        const O rf = t.at(t.x, t.j0 + n < ny ? t.j0 + n : 0, nx);
        const O ri = t.at(t.xb + 1 == nx ? 0 : t.xb + 1, t.j0 + (lane < n ? lane : 0), nx);
        float u0[R], zd[R], zl[R];
        {
            const size_t pb = nxny * (k0 > 0 ? k0 - 1 : d.nz - 1);
#pragma unroll
            for (int q = 0; q < R; ++q) {
                u0[q] = off(u + nxny * k0, t.row[q]);
                float w;
                shrink1(K, hz * (u0[q] - off(u + pb, t.row[q])), off(vo + 2 * N + pb, t.row[q]), off(lmo + 2 * N + pb, t.row[q]), w, zd[q], zl[q]);
            }
        }
        for (unsigned k = k0; k < k1; ++k) {
            const size_t pk = nxny * k;
            const float *uk = u + pk, *uz = u + nxny * (k + 1 < d.nz ? k + 1 : 0);
            const float *v0 = vo + pk, *v1 = vo + N + pk, *v2 = vo + 2 * N + pk;
            const float *m0 = lmo + pk, *m1 = lmo + N + pk, *m2 = lmo + 2 * N + pk;
            float un[R], xr[R], va[R][3], la[R][3];
#pragma unroll
            for (int q = 0; q < R; ++q) {
                un[q] = off(uz, t.row[q]);
                va[q][0] = off(v0, t.row[q]);
                va[q][1] = off(v1, t.row[q]);
                va[q][2] = off(v2, t.row[q]);
                la[q][0] = off(m0, t.row[q]);
                la[q][1] = off(m1, t.row[q]);
                la[q][2] = off(m2, t.row[q]);
            }
            const float uh = off(uk, rf), ub = off(uk, t.rb), vb = off(v1, t.rb), lb = off(m1, t.rb);
            float ue = 0.f, ui = 0.f, ve = 0.f, le = 0.f;
            if (lane < R) {
                ue = off(uk, t.re);
                ui = off(uk, ri);
                ve = off(v0, t.re);
                le = off(m0, t.re);
            }
#pragma unroll
            for (int q = 0; q < R; ++q) xr[q] = 0.f;
            if (edge_x)
#pragma unroll
                for (int q = 0; q < R; ++q) xr[q] = off(uk, (O)(t.row[q] + fx));
            float yd, yl, xd, xl, w;
            shrink1(K, hy * (u0[0] - ub), vb, lb, w, yd, yl);
            shrink1(K, hx * (ui - ue), ve, le, w, xd, xl);
            float *o0 = vn + pk, *o1 = vn + N + pk, *o2 = vn + 2 * N + pk;
            float *p0 = lmn + pk, *p1 = lmn + N + pk, *p2 = lmn + 2 * N + pk;
#pragma unroll
            for (int q = 0; q < R; ++q) {
                float uf = __shfl_down_sync(0xffffffffu, u0[q], 1);
                uf = edge_x ? xr[q] : uf;
                const float uy = q + 1 < t.nr ? u0[q + 1 < R ? q + 1 : 0] : uh;
                const float dd[3] = {hx * (uf - u0[q]), hy * (uy - u0[q]), hz * (un[q] - u0[q])};
                float e2 = 0.f, a2 = 0.f, b2 = 0.f, wc[3], dv[3], ln[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    shrink1(K, dd[c], va[q][c], la[q][c], wc[c], dv[c], ln[c]);
                    const float e = dd[c] - wc[c];
                    e2 += e * e;
                    a2 += dd[c] * dd[c];
                    b2 += wc[c] * wc[c];
                }
                const float ed = __shfl_sync(0xffffffffu, xd, q), el = __shfl_sync(0xffffffffu, xl, q);
                float bd = __shfl_up_sync(0xffffffffu, dv[0], 1), bl = __shfl_up_sync(0xffffffffu, ln[0], 1);
                bd = lane == 0 ? ed : bd;
                bl = lane == 0 ? el : bl;
                const bool first = q == 0 && t.j0 == 0;
                const float sv = K.rho * adj_sum<float>(nx_ * (dv[0] - bd), ny_ * (dv[1] - yd), nz_ * (dv[2] - zd[q]), first, k == 0);
                const float tv = K.rho * adj_sum<float>(nx_ * (ln[0] - bl), ny_ * (ln[1] - yl), nz_ * (ln[2] - zl[q]), first, k == 0);
                yd = dv[1];
                yl = ln[1];
                zd[q] = dv[2];
                zl[q] = ln[2];
                u0[q] = un[q];
                const float se = sqrtf(e2), sa = sqrtf(a2), sb = sqrtf(b2);
                if (t.on && q < t.nr) {
                    off(o0, t.row[q]) = wc[0];
                    off(o1, t.row[q]) = wc[1];
                    off(o2, t.row[q]) = wc[2];
                    off(p0, t.row[q]) = ln[0];
                    off(p1, t.row[q]) = ln[1];
                    off(p2, t.row[q]) = ln[2];
                    ps[0].add(se);
                    ps[1].add(sa);
                    ps[2].add(sb);
                    ps[3].add(sv * sv);
                    ps[4].add(tv * tv);
                }
            }
        }
    }
    double acc[5] = {ps[0].get(), ps[1].get(), ps[2].get(), ps[3].get(), ps[4].get()};
    block_sums<5>(F.part, acc);
    fold_last(F, ctl);
}

// ||rho gradfp_adj(v - v_)||^2 and ||rho gradfp_adj(l)||^2 (tv.m:230, :239)
template <typename T>
__global__ void __launch_bounds__(TV_BLOCK, TvOcc<T>::minb)
adj_norms_k(const T *__restrict__ vn, const T *__restrict__ vo, const T *__restrict__ lm, Dims d, T nx_, T ny_, T nz_,
            double *ctl, TvFold F)
{
    const T rho = (T)ctl[C_RHO];
    const size_t N = d.n();
    const T ih[3] = {nx_, ny_, nz_};
    PartialSum<T> ps[2];
    VOX_LOOP(wk, d) {
        const T s = rho * adj_at<T>(wk.v, d, ih, [&](int c, size_t m) { return vn[c * N + m] - vo[c * N + m]; });
        const T t = rho * adj_at<T>(wk.v, d, ih, [&](int c, size_t m) { return lm[c * N + m]; });
        ps[0].add(s * s);
        ps[1].add(t * t);
    }
    double acc[2] = {ps[0].get(), ps[1].get()};
    block_sums<2>(F.part + F.ns1 * F.nblk1, acc);
    fold_last(F, ctl);
}

// initial v = grad(u), nr = sum |v| (tv.m:150-152)
template <typename T>
__global__ void __launch_bounds__(TV_BLOCK, TvOcc<T>::minb)
grad_init_k(T *v, const T *__restrict__ u, Dims d, T hx, T hy, T hz, double *part)
{
    const size_t N = d.n();
    PartialSum<T> ps;
    VOX_LOOP(wk, d) {
        const Vox &x = wk.v;
        const size_t l = x.l;
        const T u0 = u[l];
        const T a = hx * ((x.i + 1 < (int)d.nx ? u[l + 1] : u[l - x.NX]) - u0);
        const T b = hy * ((x.j + 1 < (int)d.ny ? u[l + d.nx] : u[l - x.NY]) - u0);
        const T c = hz * ((x.k + 1 < (int)d.nz ? u[l + d.nxny()] : u[l - x.NZ]) - u0);
        v[l] = a;
        v[N + l] = b;
        v[2 * N + l] = c;
        ps.add(sqrt(a * a + b * b + c * c));
    }
    double acc[1] = {ps.get()};
    block_sums<1>(part, acc);
}

__global__ void __launch_bounds__(TV_BLOCK) fold_k(double *out, TvFold F)
{
    const double s = fold_sums(F);
    if ((int)threadIdx.x < F.ns1 + F.ns2) out[threadIdx.x] = s;
}

template <typename T, typename S>
__global__ void cvt_in_k(T *o, const S *__restrict__ a, size_t n)
{
    for (size_t l = (size_t)blockIdx.x * blockDim.x + threadIdx.x; l < n; l += (size_t)gridDim.x * blockDim.x)
        o[l] = (T)a[l];
}

// x = mask .* u (tv.m:275)
template <typename T, typename S>
__global__ void mask_out_k(S *x, const T *__restrict__ u, const uint8_t *__restrict__ m, size_t n)
{
    for (size_t l = (size_t)blockIdx.x * blockDim.x + threadIdx.x; l < n; l += (size_t)gridDim.x * blockDim.x)
        x[l] = (S)((m[l] ? (T)1 : (T)0) * u[l]);
}

static const char *cufft_str(cufftResult r)
{
    switch (r) {
    case CUFFT_SUCCESS: return "CUFFT_SUCCESS";
    case CUFFT_ALLOC_FAILED: return "CUFFT_ALLOC_FAILED";
    case CUFFT_INVALID_VALUE: return "CUFFT_INVALID_VALUE";
    case CUFFT_INVALID_SIZE: return "CUFFT_INVALID_SIZE";
    case CUFFT_EXEC_FAILED: return "CUFFT_EXEC_FAILED";
    default: return "cuFFT error";
    }
}

#define QSM_FFT(call)                                                                           \
    do {                                                                                        \
        cufftResult r_ = (call);                                                                \
        if (r_ != CUFFT_SUCCESS) {                                                              \
            ::qsm::set_error(ctx, "%s:%d %s: %s", __FILE__, __LINE__, #call, cufft_str(r_));    \
            st = r_ == CUFFT_ALLOC_FAILED ? QSM_ERR_NOMEM : QSM_ERR_CUDA;                      \
            goto done;                                                                          \
        }                                                                                       \
    } while (0)

#define QSM_STEP(expr)           \
    do {                         \
        st = (expr);             \
        if (st != QSM_OK) goto done; \
    } while (0)

static qsm_status cuda_st(qsm_ctx *ctx, cudaError_t e, const char *what)
{
    if (e == cudaSuccess) return QSM_OK;
    set_error(ctx, "%s: %s", what, cudaGetErrorString(e));
    return QSM_ERR_CUDA;
}

struct TvOpts {
    double mu, rtol, atol, rho, alpha, rtau, stau, gamma;
    int tv, maxit, verbose;
};

template <typename T, typename S>
static qsm_status tv_run(qsm_ctx *ctx, const Dims &d, const S *f, const uint8_t *mask, const double *h,
                         const double *bdir, TvOpts o, S *xout, qsm_tv_info *info)
{
    using C = typename CxT<T>::type;
    const size_t N = d.n();
    const int nxh = (int)(d.nx / 2 + 1);
    const size_t nh = (size_t)nxh * d.ny * d.nz;
    // u, r, v[2] (3 components each, N apart), l (3); fhat, R; partials + sums
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t rb = al(N * sizeof(T)), vb = al(3 * N * sizeof(T)), cb = al(nh * sizeof(C));
    const size_t tb = al(2 * (size_t)(nxh + d.ny + d.nz) * sizeof(double)), db = al(nh * sizeof(DL<T>));
    const size_t bytes = 3 * rb + 4 * vb + 2 * cb + tb + db + (TV_NSUM * TV_GRID_MAX + 64 + C_N + 1) * sizeof(double);
    void *blk = nullptr;
    QSM_TRY(dalloc(ctx, &blk, bytes));
    char *c = (char *)blk;
    T *u = (T *)c; c += rb;
    T *r = (T *)c; c += rb;
    T *usave = (T *)c; c += rb;  // u of the converged iteration
    T *v[2];
    v[0] = (T *)c; c += vb;
    v[1] = (T *)c; c += vb;
    T *lmb[2];  // l, double-buffered where the fused FP32 pass reads the old value at neighbours
    lmb[0] = (T *)c; c += vb;
    lmb[1] = (T *)c; c += vb;
    int lc = 0;
    C *fhat = (C *)c; c += cb;
    C *R = (C *)c; c += cb;
    double *tab = (double *)c; c += tb;
    DL<T> *dl = (DL<T> *)c; c += db;
    double *part = (double *)c;
    double *sums = part + TV_NSUM * TV_GRID_MAX;
    double *ctl = sums + 64;
    unsigned *count = (unsigned *)(ctl + C_N);

    qsm_status st = QSM_OK;
    FftPlans plans;  // forward, inverse
    const cufftType types[2] = {sizeof(T) == 8 ? CUFFT_D2Z : CUFFT_R2C, sizeof(T) == 8 ? CUFFT_Z2D : CUFFT_C2R};
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    double hc[C_N] = {};
    int cur = 0;
    uint32_t it = 0;
    bool from_save = false;
    const double atolp = sqrt(3.0 * (double)N) * o.atol, atold = sqrt((double)N) * o.atol;
    TvK K;
    K.nx = (int)d.nx; K.ny = (int)d.ny; K.nz = (int)d.nz; K.nxh = nxh;
    K.hx = h[0]; K.hy = h[1]; K.hz = h[2];
    {
        const double bn = sqrt(bdir[0] * bdir[0] + bdir[1] * bdir[1] + bdir[2] * bdir[2]);
        K.bx = bdir[0] / bn; K.by = bdir[1] / bn; K.bz = bdir[2] / bn;
        K.oblique = ((bdir[0] != 0.0) + (bdir[1] != 0.0) + (bdir[2] != 0.0)) > 1;
    }
    K.mu = o.mu;
    const T ihx = (T)(1.0 / h[0]), ihy = (T)(1.0 / h[1]), ihz = (T)(1.0 / h[2]);
    const int TV_GRID = tv_grid<T>(), GS_GRID = 152 * TvOccGS<T>::minb, ADJ_GRID = 152 * AdjTile<T>::minb, GSN_GRID = 152 * GSN_MINB;
    const dim3 g(TV_GRID), gs(GS_GRID), b(TV_BLOCK);
    const Tiles ta = tiles_of(d, AdjTile<T>::R, (unsigned)ADJ_GRID), tg = tiles_of(d, GSN_R, (unsigned)GSN_GRID);
    const bool small = d.nxny() * sizeof(T) < (size_t)UINT32_MAX;  // a plane's offsets in 32 bits
    const auto adj_rhs = small ? adj_rhs_k<T, uint32_t> : adj_rhs_k<T, size_t>;
    const auto gsn = small ? grad_shrink_norms_k<uint32_t> : grad_shrink_norms_k<size_t>;
    const unsigned gk = (unsigned)std::min<size_t>((nh + TV_BLOCK - 1) / TV_BLOCK, (size_t)TV_GRID);

    QSM_STEP(cuda_st(ctx, cudaMemsetAsync(lmb[0], 0, 3 * N * sizeof(T), ctx->stream), "memset"));
    QSM_STEP(cuda_st(ctx, cudaMemsetAsync(count, 0, sizeof(unsigned), ctx->stream), "memset"));
    QSM_STEP(fft_acquire(ctx, d, types, 2, &plans));
    QSM_STEP(cuda_st(ctx, cudaEventCreate(&e0), "event"));
    QSM_STEP(cuda_st(ctx, cudaEventCreate(&e1), "event"));
    QSM_STEP(cuda_st(ctx, cudaEventRecord(e0, ctx->stream), "event"));

    // k-space tables and D (once per solve)
    ktab_k<<<1, 256, 0, ctx->stream>>>(tab, K);
    dl_k<T><<<gk, TV_BLOCK, 0, ctx->stream>>>(dl, tab, K);
    // u = f; fhat = fft3(f) (F = mu conj(D) fhat is formed in kmul_k)
    cvt_in_k<T, S><<<g, b, 0, ctx->stream>>>(u, f, N);
    if (sizeof(T) == 8) QSM_FFT(cufftExecD2Z(plans.h[0], (cufftDoubleReal *)u, (cufftDoubleComplex *)fhat));
    else QSM_FFT(cufftExecR2C(plans.h[0], (cufftReal *)u, (cufftComplex *)fhat));
    grad_init_k<T><<<g, b, 0, ctx->stream>>>(v[0], u, d, ihx, ihy, ihz, part);
    fold_k<<<1, TV_BLOCK, 0, ctx->stream>>>(sums, TvFold{part, 1, TV_GRID, 0, 0, nullptr, {}, 0});
    // control state: rho, 1/rho (as the host forms it), nr of the initial v, flag 0
    hc[C_RHO] = o.rho;
    hc[C_IRHO] = 1.0 / o.rho;
    QSM_STEP(cuda_st(ctx, cudaMemcpyAsync(ctl, hc, C_N * sizeof(double), cudaMemcpyHostToDevice, ctx->stream), "copy"));
    QSM_STEP(cuda_st(ctx, cudaMemcpyAsync(ctl + C_NR, sums, sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream), "copy"));
    if (o.verbose) printf("\niter\t\t||r||\t\teps_pri\t\t||s||\t\teps_dual\n");

    // Iterations are queued without waiting: tv_ctl applies the stopping
    // test and the rho schedule on the device, and the host reads the state
    // every `chunk` iterations (every iteration when printing).  Iterations
    // queued past convergence compute on with frozen rho; the converged u is
    // kept by the next adj_rhs_k, and the solve reports the converged state.
    {
        const TvCtlOpts co{o.rtol, atolp, atold, o.rtau, o.stau, o.gamma};
        const int chunk = o.verbose ? 1 : 8;
        int ii = 1, last = 0;
        bool done = false;
        while (ii <= o.maxit && !done) {
            const int end = std::min(o.maxit, ii + chunk - 1);
            for (; ii <= end; ++ii) {
                const int nxt = cur ^ 1;
                // u-subproblem
                adj_rhs<<<ADJ_GRID, b, 0, ctx->stream>>>(r, v[cur], lmb[lc], d, ta, -ihx, -ihy, -ihz, ctl, ii, usave, u);
                if (sizeof(T) == 8) QSM_FFT(cufftExecD2Z(plans.h[0], (cufftDoubleReal *)r, (cufftDoubleComplex *)R));
                else QSM_FFT(cufftExecR2C(plans.h[0], (cufftReal *)r, (cufftComplex *)R));
                kmul_k<T><<<gk, TV_BLOCK, 0, ctx->stream>>>(R, fhat, dl, tab, K, ctl, 1.0 / (double)N);
                if (sizeof(T) == 8) QSM_FFT(cufftExecZ2D(plans.h[1], (cufftDoubleComplex *)R, (cufftDoubleReal *)u));
                else QSM_FFT(cufftExecC2R(plans.h[1], (cufftComplex *)R, (cufftReal *)u));
                // v-subproblem, multipliers, residuals
                if constexpr (sizeof(T) == 4) if (o.tv == 1) {
                    gsn<<<GSN_GRID, b, 0, ctx->stream>>>(
                        v[nxt], v[cur], lmb[lc ^ 1], lmb[lc], u, d, tg, ihx, ihy, ihz, (float)o.alpha, ctl, -ihx, -ihy, -ihz,
                        TvFold{part, TV_NSUM, GSN_GRID, 0, 0, count, co, ii});
                    lc ^= 1;
                }
                if (sizeof(T) == 8 || o.tv != 1) {
                    if (o.tv == 1)
                        grad_shrink_k<T, false><<<gs, b, 0, ctx->stream>>>(v[nxt], v[cur], lmb[lc], u, d, ihx, ihy,
                                                                           ihz, (T)o.alpha, ctl, part);
                    else
                        grad_shrink_k<T, true><<<gs, b, 0, ctx->stream>>>(v[nxt], v[cur], lmb[lc], u, d, ihx, ihy,
                                                                          ihz, (T)o.alpha, ctl, part);
                    adj_norms_k<T><<<g, b, 0, ctx->stream>>>(v[nxt], v[cur], lmb[lc], d, -ihx, -ihy, -ihz, ctl,
                                                             TvFold{part, 3, GS_GRID, 2, TV_GRID, count, co, ii});
                }
                QSM_STEP(cuda_st(ctx, cudaGetLastError(), "launch"));
                cur = nxt;
            }
            last = ii - 1;
            QSM_STEP(cuda_st(ctx, cudaMemcpyAsync(hc, ctl, C_N * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream), "copy"));
            QSM_STEP(cuda_st(ctx, cudaStreamSynchronize(ctx->stream), "sync"));
            done = hc[C_DONE] != 0.0;
            if (o.verbose)
                printf("%3d/%d\t\t%.4e\t%.4e\t%.4e\t%.4e\n", (int)hc[C_IT], o.maxit, hc[C_NR], hc[C_EP], hc[C_NS],
                       hc[C_ED]);
        }
        it = done ? (uint32_t)hc[C_IT] : (uint32_t)last;
        from_save = done && (int)hc[C_IT] < last;
    }
    if (o.verbose) printf("\n");
    QSM_STEP(cuda_st(ctx, cudaEventRecord(e1, ctx->stream), "event"));
    mask_out_k<T, S><<<g, b, 0, ctx->stream>>>(xout, from_save ? usave : u, mask, N);
    QSM_STEP(cuda_st(ctx, cudaGetLastError(), "launch"));
    QSM_STEP(cuda_st(ctx, cudaStreamSynchronize(ctx->stream), "sync"));
    if (info) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        info->iters = it;
        info->rho = hc[C_RHO];
        info->nr = hc[C_NR];
        info->eps_pri = hc[C_EP];
        info->ns = hc[C_NS];
        info->eps_dual = hc[C_ED];
        info->seconds = ms * 1e-3;
    }
done:
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    fft_release(ctx, &plans);
    qsm_status st2 = dfree(ctx, blk);
    return st != QSM_OK ? st : st2;
}

}  // namespace qsm

using namespace qsm;

extern "C" qsm_status qsm_tv_admm(qsm_ctx *ctx, qsm_dtype dt, const size_t dims[3], const void *f, const uint8_t *mask,
                                  const double vsz[3], const double bdir[3], double mu, int32_t tv, double rtol,
                                  double atol, int32_t maxit, double rho, double alpha, double rtau, double stau,
                                  double gamma, int32_t verbose, void *x, qsm_tv_info *info)
{
    Range nvtx_range("tv_admm");
    if (!ctx || !dims || !f || !mask || !vsz || !bdir || !x) return QSM_ERR_ARG;
    if (dt != QSM_F32 && dt != QSM_F64) return QSM_ERR_DTYPE;
    if (tv != 1 && tv != 2) return QSM_ERR_ARG;
    if (maxit < 0 || !(rho > 0.0)) return QSM_ERR_ARG;
    if (bdir[0] == 0.0 && bdir[1] == 0.0 && bdir[2] == 0.0) return QSM_ERR_ARG;
    cudaSetDevice(ctx->device);
    const Dims d = make_dims(dims);
    if (d.nx < 3 || d.ny < 3 || d.nz < 3) {
        set_error(ctx, "tv: every dimension must be >= 3 (padarray of the 3x3x3 Laplace kernel)");
        return QSM_ERR_DIMS;
    }
    if (d.nx > 0x7fffffff || d.ny > 0x7fffffff || d.nz > 0x7fffffff) return QSM_ERR_DIMS;
    const size_t es = dt == QSM_F32 ? 4 : 8;
    Staged sf, sm, sx;
    QSM_TRY(stage_in(ctx, sf, f, d.n() * es, true));
    QSM_TRY(stage_in(ctx, sm, mask, d.n(), true));
    QSM_TRY(stage_in(ctx, sx, x, d.n() * es, false));
    TvOpts o{mu, rtol, atol, rho, alpha, rtau, stau, gamma, tv, maxit, verbose};
    qsm_status st;
    if (dt == QSM_F64)
        st = tv_run<double, double>(ctx, d, (const double *)sf.dev, (const uint8_t *)sm.dev, vsz, bdir, o,
                                    (double *)sx.dev, info);
    else
        st = tv_run<float, float>(ctx, d, (const float *)sf.dev, (const uint8_t *)sm.dev, vsz, bdir, o,
                                  (float *)sx.dev, info);
    stage_out(ctx, sf, false);
    stage_out(ctx, sm, false);
    if (st != QSM_OK) {
        stage_out(ctx, sx, false);
        return st;
    }
    return stage_out(ctx, sx, true);
}
