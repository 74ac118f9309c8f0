// Finite-difference operators: gradients (forward / backward / central,
// plain and masked, periodic), their adjoints, the masked Laplacian with
// one-sided boundary stencils and the Laplacian of a wrapped phase.
//
// One thread per voxel.  Every kernel evaluates the per-voxel rule of the
// reference loop nest it replaces with the same expression and association
// order; the file is compiled without fused multiply-add, so results are
// bit-identical to the reference C in FP32 and FP64.  In FP32 these are single
// sweeps bounded by HBM bandwidth: each reads its inputs once (neighbour
// re-reads hit L1/L2) and writes each output once.  In FP64 the FP64 pipe bounds
// them, so products with 1/h run on the integer pipes (fp64.cuh), a stencil's
// variants select its operands instead of computing each, and lapw_k forms each
// difference once.
#include "common.cuh"
#include "fp64.cuh"

namespace qsm {

#define VOXEL_PROLOGUE                                                        \
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;           \
    const size_t j = (size_t)blockIdx.y * blockDim.y + threadIdx.y;           \
    const size_t k = (size_t)blockIdx.z * blockDim.z + threadIdx.z;           \
    if (i >= d.nx || j >= d.ny || k >= d.nz) return;                          \
    const size_t nx = d.nx, ny = d.ny, nz = d.nz, nxny = nx * ny;             \
    const size_t l = i + nx * j + nxny * k;                                   \
    (void)ny; (void)nz;

template <typename T> struct H3 { KMul<T> x, y, z; };

// u[l + a] - u[l] (forward), else u[l] - u[l - a]
template <typename T>
__device__ __forceinline__ T diff(const T *__restrict__ u, size_t l, size_t a, bool fwd)
{
    return u[fwd ? l + a : l] - u[fwd ? l : l - a];
}

// ---- gradients ----------------------------------------------------------

// gradf_mex.c:149-245
template <typename T>
__global__ void gradf_k(T *dx, T *dy, T *dz, const T *__restrict__ u, H3<T> h, Dims d)
{
    VOXEL_PROLOGUE
    dx[l] = h.x * diff(u, l, 1, i + 1 < nx);
    dy[l] = h.y * diff(u, l, nx, j + 1 < ny);
    dz[l] = h.z * diff(u, l, nxny, k + 1 < nz);
}

// gradb_mex.c:142-229
template <typename T>
__global__ void gradb_k(T *dx, T *dy, T *dz, const T *__restrict__ u, H3<T> h, Dims d)
{
    VOXEL_PROLOGUE
    dx[l] = h.x * diff(u, l, 1, i == 0);
    dy[l] = h.y * diff(u, l, nx, j == 0);
    dz[l] = h.z * diff(u, l, nxny, k == 0);
}

// gradc_mex.c:309-563, including the k = 0 plane overwrite of its
// "i = nx-1, k = 0" loop (:396, j stepping by 1): every linear index
// l in [2nx-1, nx*ny-2] of that plane gets (backward, central, forward).
template <typename T>
__global__ void gradc_k(T *dx, T *dy, T *dz, const T *__restrict__ u, H3<T> h, H3<T> h2, Dims d)
{
    VOXEL_PROLOGUE
    if (k == 0 && l >= 2 * nx - 1 && l + 2 <= nxny) {
        dx[l] = h.x * (u[l] - u[l - 1]);
        dy[l] = h2.y * (u[l + nx] - u[l - nx]);
        dz[l] = h.z * (u[l + nxny] - u[l]);
        return;
    }
    dx[l] = i == 0 ? h.x * (u[l + 1] - u[l]) : i + 1 == nx ? h.x * (u[l] - u[l - 1]) : h2.x * (u[l + 1] - u[l - 1]);
    dy[l] = j == 0 ? h.y * (u[l + nx] - u[l]) : j + 1 == ny ? h.y * (u[l] - u[l - nx]) : h2.y * (u[l + nx] - u[l - nx]);
    dz[l] = k == 0 ? h.z * (u[l + nxny] - u[l]) : k + 1 == nz ? h.z * (u[l] - u[l - nxny]) : h2.z * (u[l + nxny] - u[l - nxny]);
}

// gradfm_mex.c:105-154
template <typename T>
__global__ void gradfm_k(T *dx, T *dy, T *dz, const T *__restrict__ u, const uint8_t *__restrict__ G, H3<T> h, Dims d)
{
    VOXEL_PROLOGUE
    if (!G[l]) return;
    const bool xf = i + 1 < nx && G[l + 1], yf = j + 1 < ny && G[l + nx], zf = k + 1 < nz && G[l + nxny];
    dx[l] = xf || (i > 0 && G[l - 1]) ? h.x * diff(u, l, 1, xf) : (T)0;
    dy[l] = yf || (j > 0 && G[l - nx]) ? h.y * diff(u, l, nx, yf) : (T)0;
    dz[l] = zf || (k > 0 && G[l - nxny]) ? h.z * diff(u, l, nxny, zf) : (T)0;
}

// gradbm_mex.c:106-154
template <typename T>
__global__ void gradbm_k(T *dx, T *dy, T *dz, const T *__restrict__ u, const uint8_t *__restrict__ G, H3<T> h, Dims d)
{
    VOXEL_PROLOGUE
    if (!G[l]) return;
    const bool xb = i > 0 && G[l - 1], yb = j > 0 && G[l - nx], zb = k > 0 && G[l - nxny];
    dx[l] = xb || (i + 1 < nx && G[l + 1]) ? h.x * diff(u, l, 1, !xb) : (T)0;
    dy[l] = yb || (j + 1 < ny && G[l + nx]) ? h.y * diff(u, l, nx, !yb) : (T)0;
    dz[l] = zb || (k + 1 < nz && G[l + nxny]) ? h.z * diff(u, l, nxny, !zb) : (T)0;
}

// gradcm_mex.c:122-186
template <typename T>
__global__ void gradcm_k(T *dx, T *dy, T *dz, const T *__restrict__ u, const uint8_t *__restrict__ G, H3<T> h, H3<T> h2, Dims d)
{
    VOXEL_PROLOGUE
    if (!G[l]) return;
    const bool xf = i + 1 < nx && G[l + 1], xb = i > 0 && G[l - 1];
    const bool yf = j + 1 < ny && G[l + nx], yb = j > 0 && G[l - nx];
    const bool zf = k + 1 < nz && G[l + nxny], zb = k > 0 && G[l - nxny];
    dx[l] = (xf && xb) ? h2.x * (u[l + 1] - u[l - 1]) : xf ? h.x * (u[l + 1] - u[l]) : xb ? h.x * (u[l] - u[l - 1]) : (T)0;
    dy[l] = (yf && yb) ? h2.y * (u[l + nx] - u[l - nx]) : yf ? h.y * (u[l + nx] - u[l]) : yb ? h.y * (u[l] - u[l - nx]) : (T)0;
    dz[l] = (zf && zb) ? h2.z * (u[l + nxny] - u[l - nxny]) : zf ? h.z * (u[l + nxny] - u[l]) : zb ? h.z * (u[l] - u[l - nxny]) : (T)0;
}

// gradfp_mex.c:147-242 (periodic)
template <typename T>
__global__ void gradfp_k(T *dx, T *dy, T *dz, const T *__restrict__ u, H3<T> h, Dims d)
{
    VOXEL_PROLOGUE
    const size_t NX = nx - 1, NY = nx * (ny - 1), NZ = nxny * (nz - 1);
    dx[l] = h.x * ((i + 1 < nx ? u[l + 1] : u[l - NX]) - u[l]);
    dy[l] = h.y * ((j + 1 < ny ? u[l + nx] : u[l - NY]) - u[l]);
    dz[l] = h.z * ((k + 1 < nz ? u[l + nxny] : u[l - NZ]) - u[l]);
}

// ---- adjoints -------------------------------------------------------------

// gradf_adj_mex.c:153-249 (h holds -1/h)
template <typename T>
__global__ void gradf_adj_k(T *du, const T *__restrict__ x, const T *__restrict__ y, const T *__restrict__ z, H3<T> h, Dims d)
{
    VOXEL_PROLOGUE
    const T a = diff(x, l, 1, i == 0), b = diff(y, l, nx, j == 0), c = diff(z, l, nxny, k == 0);
    du[l] = h.x * a + h.y * b + h.z * c;
}

// gradb_adj_mex.c:159-261
template <typename T>
__global__ void gradb_adj_k(T *du, const T *__restrict__ x, const T *__restrict__ y, const T *__restrict__ z, H3<T> h, Dims d)
{
    VOXEL_PROLOGUE
    const T a = diff(x, l, 1, i + 1 < nx), b = diff(y, l, nx, j + 1 < ny), c = diff(z, l, nxny, k + 1 < nz);
    du[l] = h.x * a + h.y * b + h.z * c;
}

// gradfm_adj_mex.c:110-162
template <typename T>
__global__ void gradfm_adj_k(T *du, const T *__restrict__ x, const T *__restrict__ y, const T *__restrict__ z,
                             const uint8_t *__restrict__ G, H3<T> h, Dims d)
{
    VOXEL_PROLOGUE
    if (!G[l]) return;
    const bool xb = i > 0 && G[l - 1], yb = j > 0 && G[l - nx], zb = k > 0 && G[l - nxny];
    const T c = zb || (k + 1 < nz && G[l + nxny]) ? h.z * diff(z, l, nxny, !zb) : (T)0;
    const T b = yb || (j + 1 < ny && G[l + nx]) ? h.y * diff(y, l, nx, !yb) : (T)0;
    const T a = xb || (i + 1 < nx && G[l + 1]) ? h.x * diff(x, l, 1, !xb) : (T)0;
    du[l] = a + b + c;
}

// gradbm_adj_mex.c:110-162
template <typename T>
__global__ void gradbm_adj_k(T *du, const T *__restrict__ x, const T *__restrict__ y, const T *__restrict__ z,
                             const uint8_t *__restrict__ G, H3<T> h, Dims d)
{
    VOXEL_PROLOGUE
    if (!G[l]) return;
    const bool xf = i + 1 < nx && G[l + 1], yf = j + 1 < ny && G[l + nx], zf = k + 1 < nz && G[l + nxny];
    const T a = xf || (i > 0 && G[l - 1]) ? h.x * diff(x, l, 1, xf) : (T)0;
    const T b = yf || (j > 0 && G[l - nx]) ? h.y * diff(y, l, nx, yf) : (T)0;
    const T c = zf || (k > 0 && G[l - nxny]) ? h.z * diff(z, l, nxny, zf) : (T)0;
    du[l] = a + b + c;
}

// gradfp_adj_mex.c:156-257: axis terms summed (x+y)+z on k = 0,
// (z+x)+y for k > 0, j = 0 and (z+y)+x for k > 0, j > 0.
template <typename T>
__global__ void gradfp_adj_k(T *du, const T *__restrict__ x, const T *__restrict__ y, const T *__restrict__ z, H3<T> h, Dims d)
{
    VOXEL_PROLOGUE
    const size_t NX = nx - 1, NY = nx * (ny - 1), NZ = nxny * (nz - 1);
    const T a = h.x * (x[l] - (i > 0 ? x[l - 1] : x[l + NX]));
    const T b = h.y * (y[l] - (j > 0 ? y[l - nx] : y[l + NY]));
    const T c = h.z * (z[l] - (k > 0 ? z[l - nxny] : z[l + NZ]));
    du[l] = k == 0 ? (a + b) + c : j == 0 ? (c + a) + b : (c + b) + a;
}

// ---- Laplacians -----------------------------------------------------------

// lap1_mex.c:208-315: one axis of the masked Laplacian.  sel = 3 central,
// 2 forward (4/3/2-point by availability), 1 backward, 0 none.
template <typename T>
__device__ __forceinline__ T lap_axis(const T *__restrict__ u, const uint8_t *__restrict__ G, size_t l, size_t a,
                                      size_t n, size_t i, int sel)
{
    switch (sel) {
    case 3: return u[l - a] - scale2<1>(u[l]) + u[l + a];
    case 2:
        if (i + 3 < n && G[l + 2 * a] && G[l + 3 * a])
            return scale2<1>(u[l]) - (T)5 * u[l + a] + scale2<2>(u[l + 2 * a]) - u[l + 3 * a];
        if (i + 2 < n && G[l + 2 * a]) return u[l] - scale2<1>(u[l + a]) + u[l + 2 * a];
        return u[l + a] - u[l];
    case 1:
        if (i >= 3 && G[l - 3 * a] && G[l - 2 * a])
            return -u[l - 3 * a] + scale2<2>(u[l - 2 * a]) - (T)5 * u[l - a] + scale2<1>(u[l]);
        if (i >= 2 && G[l - 2 * a]) return u[l - 2 * a] - scale2<1>(u[l - a]) + u[l];
        return u[l - a] - u[l];
    default: return (T)0;
    }
}

// lap1_mex.c:170-200: interior selector 2*G[+1] + G[-1]; faces forced.
__device__ __forceinline__ int lap_sel(const uint8_t *__restrict__ G, size_t l, size_t a, size_t i, size_t n)
{
    if (i >= 1 && i + 1 < n) return 2 * G[l + a] + G[l - a];
    return (i == 0) * 2 + (i + 1 == n);
}

// lap1_mex.c:136-205
template <typename T>
__global__ void lap1_k(T *du, const T *__restrict__ u, const uint8_t *__restrict__ G, H3<T> h, Dims d)
{
    VOXEL_PROLOGUE
    if (!G[l]) return;
    T v = h.x * lap_axis(u, G, l, 1, nx, i, lap_sel(G, l, 1, i, nx));
    v = v + h.y * lap_axis(u, G, l, nx, ny, j, lap_sel(G, l, nx, j, ny));
    v = v + h.z * lap_axis(u, G, l, nxny, nz, k, lap_sel(G, l, nxny, k, nz));
    du[l] = v;
}

// lapw_mex.c:10-11, :170-187: wrap into [-pi, pi] only when outside.  For |x| > 9
// as the reference has it; up to there fmod(x + pi, 2 pi) is x + pi itself (x <
// -pi: its magnitude is below 2 pi) or x + pi - 2 pi, exact since x + pi lies in
// [2 pi, 4 pi): adding pi to the one, subtracting it from the other is one
// rounding of x + pi + pi or x + pi - 3 pi, the fused multiply-add with 2 pi.
// FP64 tests run on the encodings, off the FP64 pipe; a NaN is
// outside no bound.
__device__ __forceinline__ bool beyond(float x, float b) { return fabsf(x) > b; }
__device__ __forceinline__ bool beyond(double x, double b)
{
    const long long m = __double_as_longlong(x) & 0x7fffffffffffffffll;
    return m > __double_as_longlong(b) && m <= 0x7ff0000000000000ll;
}

template <typename T>
__device__ __forceinline__ T wrap_pi(T x)
{
    const T pi = (T)3.14159265358979323846;
    const T tau = (T)(2 * 3.14159265358979323846);
    if (!beyond(x, pi)) return x;
    const bool neg = signbit(x), far = beyond(x, (T)9);
    x = x + pi;
    if (far) return x < (T)0 ? fmod(x, tau) + pi : fmod(x, tau) - pi;
    return fma(neg ? (T)0.5 : (T)-1.5, tau, x);
}

// lapw_mex.c:54-167 (interior only).  The six wrapped differences of a voxel are
// three of its own and three of its lower neighbours': a thread walks up z with
// LAPW_R rows, so z and most y differences are formed once, and takes the x one
// of the lane below (lane 0 forms only that: 31 voxels per warp).  FP64: ~8.5
// FP64 instructions per voxel and 3 per wrapped difference of a warp, against 26
// and more with six differences per voxel and tests on the FP64 pipe.
constexpr int LAPW_R = 4, LAPW_TY = 4;

// One voxel per thread, six wraps each: the form for volumes that do not fill the GPU
// with columns, where a column's chain is the time.  Below the line of lapw_small, kernel
// and launch in us over those of 3 x 3 x 3, voxels against columns: FP32 2 / 7 (33 x 31 x 29),
// 1 / 8 (64 x 64 x 40), 9 / 11 (96^3), 13 / 17 (128 x 128 x 80), above 19.8 / 19.2 (128^3), 33 / 32
// (181 x 217 x 91); FP64 10 / 17 (33 x 31 x 29), 19 / 20 (48^3), above 21 / 19 (64 x 64 x 40),
// 398 / 271 (181 x 217 x 91).
template <typename T> constexpr size_t lapw_small() { return sizeof(T) == 4 ? 2000000 : 130000; }
template <typename T>
__global__ void lapw_voxel_k(T *du, const T *__restrict__ u, H3<T> h, Dims d)
{
    VOXEL_PROLOGUE
    if (i == 0 || j == 0 || k == 0 || i + 1 >= nx || j + 1 >= ny || k + 1 >= nz) return;
    T v = h.x.w * (wrap_pi(u[l + 1] - u[l]) - wrap_pi(u[l] - u[l - 1]));
    v = v + h.y.w * (wrap_pi(u[l + nx] - u[l]) - wrap_pi(u[l] - u[l - nx]));
    v = v + h.z.w * (wrap_pi(u[l + nxny] - u[l]) - wrap_pi(u[l] - u[l - nxny]));
    du[l] = v;
}

template <typename T>
__global__ void __launch_bounds__(32 * LAPW_TY) lapw_k(T *du, const T *__restrict__ u, H3<T> h, Dims d, int kz)
{
    const size_t nx = d.nx, ny = d.ny, nz = d.nz, nxny = nx * ny;
    const size_t i = (size_t)blockIdx.x * 31 + threadIdx.x;
    const size_t j0 = 1 + ((size_t)blockIdx.y * LAPW_TY + threadIdx.y) * LAPW_R;
    const size_t k0 = 1 + (size_t)blockIdx.z * kz, k1 = min(k0 + (size_t)kz, nz - 1);
    if (j0 + 1 >= ny) return;  // (a whole warp)
    const bool on = i + 1 < nx, out = on && threadIdx.x > 0;
    const size_t ic = on ? i : nx - 1;  // lanes past the row read its last voxel
    const int rows = (int)min((size_t)LAPW_R, ny - 1 - j0);
    const T *p = u + ic + nx * (j0 - 1) + nxny * k0;
    T a[LAPW_R + 2], fz[LAPW_R];
#pragma unroll
    for (int r = 0; r < LAPW_R + 2; ++r) a[r] = r <= rows + 1 ? p[r * nx] : (T)0;
#pragma unroll
    for (int r = 0; r < LAPW_R; ++r) fz[r] = r < rows ? wrap_pi(a[r + 1] - p[(r + 1) * nx - nxny]) : (T)0;
    for (size_t k = k0; k < k1; ++k, p += nxny) {
        T n[LAPW_R + 2];
#pragma unroll
        for (int r = 0; r < LAPW_R + 2; ++r) n[r] = r <= rows + 1 ? p[r * nx + nxny] : (T)0;
        T fy = wrap_pi(a[1] - a[0]);
#pragma unroll
        for (int r = 0; r < LAPW_R; ++r) {
            if (r < rows) {  // uniform over the warp
                const T right = on ? p[(r + 1) * nx + 1] : a[r + 1];
                const T fx = wrap_pi(right - a[r + 1]);
                const T bx = __shfl_up_sync(0xffffffffu, fx, 1);
                const T gy = wrap_pi(a[r + 2] - a[r + 1]), gz = wrap_pi(n[r + 1] - a[r + 1]);
                T v = h.x * (fx - bx);
                v = v + h.y * (gy - fy);
                v = v + h.z * (gz - fz[r]);
                if (out) du[i + nx * (j0 + r) + nxny * k] = v;
                fy = gy;
                fz[r] = gz;
            }
        }
#pragma unroll
        for (int r = 0; r < LAPW_R + 2; ++r) a[r] = n[r];
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

template <typename T> static H3<T> inv_h(const double *h, double s)
{
    return H3<T>{make_kmul((T)(s / h[0])), make_kmul((T)(s / h[1])), make_kmul((T)(s / h[2]))};
}
template <typename T> static H3<T> inv_h2(const double *h)
{
    return H3<T>{make_kmul((T)(1.0 / (h[0] * h[0]))), make_kmul((T)(1.0 / (h[1] * h[1]))), make_kmul((T)(1.0 / (h[2] * h[2])))};
}

enum FdOp {
    OP_GRADF, OP_GRADB, OP_GRADC, OP_GRADFM, OP_GRADBM, OP_GRADCM, OP_GRADFP,
    OP_GRADF_ADJ, OP_GRADB_ADJ, OP_GRADFM_ADJ, OP_GRADBM_ADJ, OP_GRADFP_ADJ,
    OP_LAP1, OP_LAPW
};

template <typename T>
static qsm_status launch_fd(qsm_ctx *ctx, FdOp op, const Dims &d, void **a, const uint8_t *G, const double *h)
{
    const dim3 g = vox_grid(d), b = vox_block();
    cudaStream_t s = ctx->stream;
    T *o0 = (T *)a[0], *o1 = (T *)a[1], *o2 = (T *)a[2];
    const T *i0 = (const T *)a[3], *i1 = (const T *)a[1], *i2 = (const T *)a[2];
    switch (op) {
    case OP_GRADF: gradf_k<T><<<g, b, 0, s>>>(o0, o1, o2, i0, inv_h<T>(h, 1.0), d); break;
    case OP_GRADB: gradb_k<T><<<g, b, 0, s>>>(o0, o1, o2, i0, inv_h<T>(h, 1.0), d); break;
    case OP_GRADC: gradc_k<T><<<g, b, 0, s>>>(o0, o1, o2, i0, inv_h<T>(h, 1.0), inv_h<T>(h, 0.5), d); break;
    case OP_GRADFM: gradfm_k<T><<<g, b, 0, s>>>(o0, o1, o2, i0, G, inv_h<T>(h, 1.0), d); break;
    case OP_GRADBM: gradbm_k<T><<<g, b, 0, s>>>(o0, o1, o2, i0, G, inv_h<T>(h, 1.0), d); break;
    case OP_GRADCM: gradcm_k<T><<<g, b, 0, s>>>(o0, o1, o2, i0, G, inv_h<T>(h, 1.0), inv_h<T>(h, 0.5), d); break;
    case OP_GRADFP: gradfp_k<T><<<g, b, 0, s>>>(o0, o1, o2, i0, inv_h<T>(h, 1.0), d); break;
    // adjoints: a = {du, x, y, z}
    case OP_GRADF_ADJ: gradf_adj_k<T><<<g, b, 0, s>>>(o0, (const T *)a[1], (const T *)a[2], (const T *)a[3], inv_h<T>(h, -1.0), d); break;
    case OP_GRADB_ADJ: gradb_adj_k<T><<<g, b, 0, s>>>(o0, (const T *)a[1], (const T *)a[2], (const T *)a[3], inv_h<T>(h, -1.0), d); break;
    case OP_GRADFM_ADJ: gradfm_adj_k<T><<<g, b, 0, s>>>(o0, (const T *)a[1], (const T *)a[2], (const T *)a[3], G, inv_h<T>(h, -1.0), d); break;
    case OP_GRADBM_ADJ: gradbm_adj_k<T><<<g, b, 0, s>>>(o0, (const T *)a[1], (const T *)a[2], (const T *)a[3], G, inv_h<T>(h, -1.0), d); break;
    case OP_GRADFP_ADJ: gradfp_adj_k<T><<<g, b, 0, s>>>(o0, (const T *)a[1], (const T *)a[2], (const T *)a[3], inv_h<T>(h, -1.0), d); break;
    // Laplacians: a = {d2u, u}
    case OP_LAP1: lap1_k<T><<<g, b, 0, s>>>(o0, (const T *)a[1], G, inv_h2<T>(h), d); break;
    case OP_LAPW: {
        if (d.nx < 3 || d.ny < 3 || d.nz < 3) break;
        if (d.n() < lapw_small<T>()) {
            lapw_voxel_k<T><<<g, b, 0, s>>>(o0, (const T *)a[1], inv_h2<T>(h), d);
            break;
        }
        // columns of 16 planes; shorter ones where those would leave SMs without a few blocks each
        const unsigned gx = (unsigned)((d.nx - 2 + 30) / 31), gy = (unsigned)((d.ny - 2 + LAPW_R * LAPW_TY - 1) / (LAPW_R * LAPW_TY));
        int kz = 16;
        while (kz > 2 && (size_t)gx * gy * ((d.nz - 2 + kz - 1) / kz) < 1216) kz /= 2;
        lapw_k<T><<<dim3(gx, gy, (unsigned)((d.nz - 2 + kz - 1) / kz)), dim3(32, LAPW_TY), 0, s>>>(
            o0, (const T *)a[1], inv_h2<T>(h), d, kz);
        break;
    }
    }
    (void)i1; (void)i2;
    QSM_CUDA(cudaGetLastError());
    return QSM_OK;
}

// Stages `narr` arrays (the first `nout` are written), the optional mask,
// launches, copies outputs back and waits.
static qsm_status run_fd(qsm_ctx *ctx, qsm_dtype dt, const size_t *dims, FdOp op, int narr, int nout,
                         void **arrs, const uint8_t *G, bool need_G, const double *vsz, size_t min_dim)
{
    if (!ctx || !dims || !vsz) return QSM_ERR_ARG;
    if (dt != QSM_F32 && dt != QSM_F64) return QSM_ERR_DTYPE;
    for (int q = 0; q < narr; ++q)
        if (!arrs[q]) return QSM_ERR_ARG;
    if (need_G && !G) return QSM_ERR_ARG;
    for (int q = 0; q < 3; ++q)
        if (dims[q] < min_dim) {
            set_error(ctx, "every dimension must be >= %zu", min_dim);
            return QSM_ERR_DIMS;
        }
    cudaSetDevice(ctx->device);
    const Dims d = make_dims(dims);
    const size_t es = dt == QSM_F32 ? 4 : 8;
    Staged st[5];
    void *dev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    for (int q = 0; q < narr; ++q) {
        // outputs are in-place: masked operators leave untouched voxels as
        // the caller had them, so outputs are copied in as well
        QSM_TRY(stage_in(ctx, st[q], arrs[q], d.n() * es, true));
        dev[q] = st[q].dev;
    }
    Staged sg;
    const uint8_t *gdev = nullptr;
    if (need_G) {
        QSM_TRY(stage_in(ctx, sg, G, d.n(), true));
        gdev = (const uint8_t *)sg.dev;
    }
    qsm_status s = dt == QSM_F32 ? launch_fd<float>(ctx, op, d, dev, gdev, vsz)
                                 : launch_fd<double>(ctx, op, d, dev, gdev, vsz);
    for (int q = 0; q < narr; ++q) QSM_TRY(stage_out(ctx, st[q], q < nout));
    if (need_G) QSM_TRY(stage_out(ctx, sg, false));
    QSM_CUDA(cudaStreamSynchronize(ctx->stream));
    return s;
}

}  // namespace qsm

using namespace qsm;

extern "C" {

#define GRAD_API(name, OP, masked, mind)                                                               \
    qsm_status qsm_##name(qsm_ctx *ctx, qsm_dtype dt, const size_t dims[3], void *dx, void *dy,       \
                          void *dz, const void *u, const double vsz[3])                               \
    {                                                                                                  \
        void *a[4] = {dx, dy, dz, const_cast<void *>(u)};                                              \
        return run_fd(ctx, dt, dims, OP, 4, 3, a, nullptr, false, vsz, mind);                          \
    }

GRAD_API(gradf, OP_GRADF, 0, 2)
GRAD_API(gradb, OP_GRADB, 0, 2)
GRAD_API(gradc, OP_GRADC, 0, 2)
GRAD_API(gradfp, OP_GRADFP, 0, 1)

#define GRADM_API(name, OP)                                                                            \
    qsm_status qsm_##name(qsm_ctx *ctx, qsm_dtype dt, const size_t dims[3], void *dx, void *dy,       \
                          void *dz, const void *u, const uint8_t *G, const double vsz[3])             \
    {                                                                                                  \
        void *a[4] = {dx, dy, dz, const_cast<void *>(u)};                                              \
        return run_fd(ctx, dt, dims, OP, 4, 3, a, G, true, vsz, 1);                                    \
    }

GRADM_API(gradfm, OP_GRADFM)
GRADM_API(gradbm, OP_GRADBM)
GRADM_API(gradcm, OP_GRADCM)

#define ADJ_API(name, OP, mind)                                                                        \
    qsm_status qsm_##name(qsm_ctx *ctx, qsm_dtype dt, const size_t dims[3], void *du, const void *x,  \
                          const void *y, const void *z, const double vsz[3])                          \
    {                                                                                                  \
        void *a[4] = {du, const_cast<void *>(x), const_cast<void *>(y), const_cast<void *>(z)};        \
        return run_fd(ctx, dt, dims, OP, 4, 1, a, nullptr, false, vsz, mind);                          \
    }

ADJ_API(gradf_adj, OP_GRADF_ADJ, 2)
ADJ_API(gradb_adj, OP_GRADB_ADJ, 2)
ADJ_API(gradfp_adj, OP_GRADFP_ADJ, 1)

#define ADJM_API(name, OP)                                                                             \
    qsm_status qsm_##name(qsm_ctx *ctx, qsm_dtype dt, const size_t dims[3], void *du, const void *x,  \
                          const void *y, const void *z, const uint8_t *G, const double vsz[3])        \
    {                                                                                                  \
        void *a[4] = {du, const_cast<void *>(x), const_cast<void *>(y), const_cast<void *>(z)};        \
        return run_fd(ctx, dt, dims, OP, 4, 1, a, G, true, vsz, 1);                                    \
    }

ADJM_API(gradfm_adj, OP_GRADFM_ADJ)
ADJM_API(gradbm_adj, OP_GRADBM_ADJ)

qsm_status qsm_lap1(qsm_ctx *ctx, qsm_dtype dt, const size_t dims[3], void *d2u, const void *u, const uint8_t *G,
                    const double vsz[3])
{
    void *a[2] = {d2u, const_cast<void *>(u)};
    return run_fd(ctx, dt, dims, OP_LAP1, 2, 1, a, G, true, vsz, 2);
}

qsm_status qsm_lapw(qsm_ctx *ctx, qsm_dtype dt, const size_t dims[3], void *d2u, const void *u, const double vsz[3])
{
    void *a[2] = {d2u, const_cast<void *>(u)};
    return run_fd(ctx, dt, dims, OP_LAPW, 2, 1, a, nullptr, false, vsz, 1);
}

}  // extern "C"
