// Kernels of the barotropic step's general path (see general.h).  Compiled
// with --fmad=false: each expression below is written in the evaluation
// order of the Fortran line it cites (left to right through * / + - chains),
// so the rounding matches a non-contracting Fortran build.
#include "general.h"

#include <algorithm>

namespace inmsom {
namespace general {

namespace {

constexpr int BX = 32, BY = 8;

// Launch over the inclusive index range [m0,m1] x [n0,n1].
template <typename K, typename... A>
void launch2d(K k, int m0, int m1, int n0, int n1, cudaStream_t s, A... a)
{
    if (m1 < m0 || n1 < n0) return;
    dim3 blk(BX, BY);
    dim3 grd((m1 - m0 + BX) / BX, (n1 - n0 + BY) / BY);
    k<<<grd, blk, 0, s>>>(m0, m1, n0, n1, a...);
}

#define RANGE_GUARD                                   \
    const int m = m0 + blockIdx.x * BX + threadIdx.x; \
    const int n = n0 + blockIdx.y * BY + threadIdx.y; \
    if (m > m1 || n > n1) return;
#define X(m_, n_) ix(D, (m_), (n_))

__global__ void k_fill(int m0, int m1, int n0, int n1, Dom D, double *f, double v)
{
    RANGE_GUARD
    f[X(m, n)] = v;
}

// Service/oc_algorithms.f90:50-95 (wrap: ff(mmm-1)=ff(mm), ff(mm+1)=ff(mmm))
__global__ void k_cyclize_x(Dom D, double *f)
{
    const int n = D.bnd_y1 + blockIdx.x * blockDim.x + threadIdx.x;
    if (n > D.bnd_y2) return;
    double left = f[X(D.mm, n)], right = f[X(D.mmm, n)];
    f[X(D.mmm - 1, n)] = left;
    f[X(D.mm + 1, n)] = right;
}

// Service/oc_algorithms.f90:118-135
__global__ void k_cyclize_y(Dom D, double *f)
{
    const int m = D.bnd_x1 + blockIdx.x * blockDim.x + threadIdx.x;
    if (m > D.bnd_x2) return;
    f[X(m, D.nnn - 1)] = f[X(m, D.nn)];
    f[X(m, D.nn + 1)] = f[X(m, D.nnn)];
}

// ---- depth interpolation, Function/depth.f90:29-66 ----------------------
// hq(i): the depth on T points, element i of the layout (an array, or the
// rest depth plus a level)
struct HqArray {
    const double *hq;
    __device__ __forceinline__ double operator()(long long i) const { return hq[i]; }
};
struct HqOf {   // depth.f90:21-23, :121: h_r + sh*ffs
    const double *hr, *sh;
    double ffs;
    __device__ __forceinline__ double operator()(long long i) const { return hr[i] + sh[i] * ffs; }
};
struct HqRest {
    const double *hr;
    __device__ __forceinline__ double operator()(long long i) const { return hr[i]; }
};

template <class HQ>
__device__ __forceinline__ double h_on_u(const Dom &D, const GridDev &g, const HQ &hq, int m, int n)
{
    const float *lu = g.lu;
    double slu = (double)(lu[X(m, n)] + lu[X(m + 1, n)]);
    return (hq(X(m, n)) * g.dx[X(m, n)] * g.dy[X(m, n)] * (double)lu[X(m, n)]
            + hq(X(m + 1, n)) * g.dx[X(m + 1, n)] * g.dy[X(m + 1, n)] * (double)lu[X(m + 1, n)])
           / slu / g.dxt[X(m, n)] / g.dyh[X(m, n)];
}
template <class HQ>
__device__ __forceinline__ double h_on_v(const Dom &D, const GridDev &g, const HQ &hq, int m, int n)
{
    const float *lu = g.lu;
    double slu = (double)(lu[X(m, n)] + lu[X(m, n + 1)]);
    return (hq(X(m, n)) * g.dx[X(m, n)] * g.dy[X(m, n)] * (double)lu[X(m, n)]
            + hq(X(m, n + 1)) * g.dx[X(m, n + 1)] * g.dy[X(m, n + 1)] * (double)lu[X(m, n + 1)])
           / slu / g.dxh[X(m, n)] / g.dyt[X(m, n)];
}
template <class HQ>
__device__ __forceinline__ double h_on_h(const Dom &D, const GridDev &g, const HQ &hq, int m, int n)
{
    const float *lu = g.lu;
    double slu = (double)(lu[X(m, n)] + lu[X(m + 1, n)] + lu[X(m, n + 1)] + lu[X(m + 1, n + 1)]);
    return (hq(X(m, n)) * g.dx[X(m, n)] * g.dy[X(m, n)] * (double)lu[X(m, n)]
            + hq(X(m + 1, n)) * g.dx[X(m + 1, n)] * g.dy[X(m + 1, n)] * (double)lu[X(m + 1, n)]
            + hq(X(m, n + 1)) * g.dx[X(m, n + 1)] * g.dy[X(m, n + 1)] * (double)lu[X(m, n + 1)]
            + hq(X(m + 1, n + 1)) * g.dx[X(m + 1, n + 1)] * g.dy[X(m + 1, n + 1)] * (double)lu[X(m + 1, n + 1)])
           / slu / g.dxb[X(m, n)] / g.dyb[X(m, n)];
}

// hq = h_r + sh*ffs over the whole array (depth.f90:21-23, :121)
__global__ void k_hq_set(int m0, int m1, int n0, int n1, Dom D, const double *hr,
                         double *hq, const double *sh, double ffs, int use_sh)
{
    RANGE_GUARD
    hq[X(m, n)] = use_sh ? hr[X(m, n)] + sh[X(m, n)] * ffs : hr[X(m, n)];
}

// depth.f90:25-70 / :123-152 for one time level
__global__ void k_hh_interp(int m0, int m1, int n0, int n1, Dom D, GridDev g,
                            const double *hq, double *hu, double *hv, double *hh)
{
    RANGE_GUARD
    const HqArray q{hq};
    if (g.llu[X(m, n)] > 0.5f) hu[X(m, n)] = h_on_u(D, g, q, m, n);
    if (g.llv[X(m, n)] > 0.5f) hv[X(m, n)] = h_on_v(D, g, q, m, n);
    if (g.luh[X(m, n)] > 0.5f) hh[X(m, n)] = h_on_h(D, g, q, m, n);
}

__device__ __forceinline__ double asselin(double ts, double f, double fn, double fp, double div2, double ns)
{
    // f + ts*(fn - 2f + fp)/2/nstep, rounded as f + (((ts*((fn-2f)+fp))/2)/nstep)
    return f + ts * (fn - 2.0 * f + fp) / div2 / ns;
}

// ---- Function/mixing.f90:129-153 ---------------------------------------
__device__ __forceinline__ double tension(const Dom &D, const GridDev &g, const double *u, const double *v, int m, int n)
{
    const double *dx = g.dx, *dy = g.dy, *dxh = g.dxh, *dyh = g.dyh;
    return dy[X(m, n)] / dx[X(m, n)] * (u[X(m, n)] / dyh[X(m, n)] - u[X(m - 1, n)] / dyh[X(m - 1, n)])
           - dx[X(m, n)] / dy[X(m, n)] * (v[X(m, n)] / dxh[X(m, n)] - v[X(m, n - 1)] / dxh[X(m, n - 1)]);
}
__device__ __forceinline__ double shear(const Dom &D, const GridDev &g, const double *u, const double *v, int m, int n)
{
    const double *dxt = g.dxt, *dyt = g.dyt, *dxb = g.dxb, *dyb = g.dyb;
    return dxb[X(m, n)] / dyb[X(m, n)] * (u[X(m, n + 1)] / dxt[X(m, n + 1)] - u[X(m, n)] / dxt[X(m, n)])
           + dyb[X(m, n)] / dxb[X(m, n)] * (v[X(m + 1, n)] / dyt[X(m + 1, n)] - v[X(m, n)] / dyt[X(m, n)]);
}

// ---- Function/vel_ssh.f90:30-42 ------------------------------------------
__device__ __forceinline__ double vorticity(const Dom &D, const GridDev &g, const double *u, const double *v, int m, int n)
{
    const double *dxt = g.dxt, *dyt = g.dyt, *dxb = g.dxb, *dyb = g.dyb;
    return (v[X(m + 1, n)] * dyt[X(m + 1, n)] - v[X(m, n)] * dyt[X(m, n)])
           - (u[X(m, n + 1)] * dxt[X(m, n + 1)] - u[X(m, n)] * dxt[X(m, n)])
           - ((v[X(m + 1, n)] - v[X(m, n)]) * dyb[X(m, n)] - (u[X(m, n + 1)] - u[X(m, n)]) * dxb[X(m, n)]);
}

// ---- Function/vel_ssh.f90:54-109 -----------------------------------------
__device__ __forceinline__ double trans_x(const Dom &D, const GridDev &g, const double *u, const double *v,
                                          const double *vort, const double *hu, const double *hv, const double *hh,
                                          int m, int n)
{
    const double *dxh = g.dxh, *dyh = g.dyh;
    double fx_p = (u[X(m, n)] * dyh[X(m, n)] * hu[X(m, n)] + u[X(m + 1, n)] * dyh[X(m + 1, n)] * hu[X(m + 1, n)]) / 2.0
                  * (u[X(m, n)] + u[X(m + 1, n)]) / 2.0;
    double fx_m = (u[X(m, n)] * dyh[X(m, n)] * hu[X(m, n)] + u[X(m - 1, n)] * dyh[X(m - 1, n)] * hu[X(m - 1, n)]) / 2.0
                  * (u[X(m, n)] + u[X(m - 1, n)]) / 2.0;
    double fy_p = (v[X(m, n)] * dxh[X(m, n)] * hv[X(m, n)] + v[X(m + 1, n)] * dxh[X(m + 1, n)] * hv[X(m + 1, n)]) / 2.0
                  * (u[X(m, n + 1)] + u[X(m, n)]) / 2.0 * (double)g.luu[X(m, n)];
    double fy_m = (v[X(m, n - 1)] * dxh[X(m, n - 1)] * hv[X(m, n - 1)] + v[X(m + 1, n - 1)] * dxh[X(m + 1, n - 1)] * hv[X(m + 1, n - 1)]) / 2.0
                  * (u[X(m, n - 1)] + u[X(m, n)]) / 2.0 * (double)g.luu[X(m, n - 1)];
    return -(fx_p - fx_m + fy_p - fy_m)
           + (vort[X(m, n)] * hh[X(m, n)] * (v[X(m + 1, n)] + v[X(m, n)])
              + vort[X(m, n - 1)] * hh[X(m, n - 1)] * (v[X(m + 1, n - 1)] + v[X(m, n - 1)])) / 4.0;
}
__device__ __forceinline__ double trans_y(const Dom &D, const GridDev &g, const double *u, const double *v,
                                          const double *vort, const double *hu, const double *hv, const double *hh,
                                          int m, int n)
{
    const double *dxh = g.dxh, *dyh = g.dyh;
    double fy_p = (v[X(m, n)] * dxh[X(m, n)] * hv[X(m, n)] + v[X(m, n + 1)] * dxh[X(m, n + 1)] * hv[X(m, n + 1)]) / 2.0
                  * (v[X(m, n)] + v[X(m, n + 1)]) / 2.0;
    double fy_m = (v[X(m, n)] * dxh[X(m, n)] * hv[X(m, n)] + v[X(m, n - 1)] * dxh[X(m, n - 1)] * hv[X(m, n - 1)]) / 2.0
                  * (v[X(m, n)] + v[X(m, n - 1)]) / 2.0;
    double fx_p = (u[X(m, n)] * dyh[X(m, n)] * hu[X(m, n)] + u[X(m, n + 1)] * dyh[X(m, n + 1)] * hu[X(m, n + 1)]) / 2.0
                  * (v[X(m + 1, n)] + v[X(m, n)]) / 2.0;
    double fx_m = (u[X(m - 1, n)] * dyh[X(m - 1, n)] * hu[X(m - 1, n)] + u[X(m - 1, n + 1)] * dyh[X(m - 1, n + 1)] * hu[X(m - 1, n + 1)]) / 2.0
                  * (v[X(m - 1, n)] + v[X(m, n)]) / 2.0;
    return -(fx_p - fx_m + fy_p - fy_m)
           - (vort[X(m, n)] * hh[X(m, n)] * (u[X(m, n + 1)] + u[X(m, n)])
              + vort[X(m - 1, n)] * hh[X(m - 1, n)] * (u[X(m - 1, n + 1)] + u[X(m - 1, n)])) / 4.0;
}

// ---- stress divergence, Function/vel_ssh.f90:150-172 ---------------------
template <class HQ>
__device__ __forceinline__ double dif_xt(const Dom &D, const GridDev &g, const double *mu,
                                         const double *str_t, const HQ &hq, int m, int n)
{
    double dy1 = g.dy[X(m + 1, n)], dy0 = g.dy[X(m, n)];
    return (dy1 * dy1 * mu[X(m + 1, n)] * hq(X(m + 1, n)) * str_t[X(m + 1, n)]
            - dy0 * dy0 * mu[X(m, n)] * hq(X(m, n)) * str_t[X(m, n)]) / g.dyh[X(m, n)];
}
__device__ __forceinline__ double dif_xs(const Dom &D, const GridDev &g, const double *mu,
                                         const double *str_s, const double *hh, int m, int n)
{
    double muh_p = (mu[X(m, n)] + mu[X(m + 1, n)] + mu[X(m, n + 1)] + mu[X(m + 1, n + 1)]) / 4.0;
    double muh_m = (mu[X(m, n)] + mu[X(m + 1, n)] + mu[X(m, n - 1)] + mu[X(m + 1, n - 1)]) / 4.0;
    double b0 = g.dxb[X(m, n)], b1 = g.dxb[X(m, n - 1)];
    return (b0 * b0 * muh_p * hh[X(m, n)] * str_s[X(m, n)]
            - b1 * b1 * muh_m * hh[X(m, n - 1)] * str_s[X(m, n - 1)]) / g.dxt[X(m, n)];
}
template <class HQ>
__device__ __forceinline__ double dif_yt(const Dom &D, const GridDev &g, const double *mu,
                                         const double *str_t, const HQ &hq, int m, int n)
{
    double dx1 = g.dx[X(m, n + 1)], dx0 = g.dx[X(m, n)];
    return (dx1 * dx1 * mu[X(m, n + 1)] * hq(X(m, n + 1)) * str_t[X(m, n + 1)]
            - dx0 * dx0 * mu[X(m, n)] * hq(X(m, n)) * str_t[X(m, n)]) / g.dxh[X(m, n)];
}
__device__ __forceinline__ double dif_ys(const Dom &D, const GridDev &g, const double *mu,
                                         const double *str_s, const double *hh, int m, int n)
{
    double muh_p = (mu[X(m, n)] + mu[X(m + 1, n)] + mu[X(m, n + 1)] + mu[X(m + 1, n + 1)]) / 4.0;
    double muh_m = (mu[X(m, n)] + mu[X(m - 1, n)] + mu[X(m, n + 1)] + mu[X(m - 1, n + 1)]) / 4.0;
    double b0 = g.dyb[X(m, n)], b1 = g.dyb[X(m - 1, n)];
    return (b0 * b0 * muh_p * hh[X(m, n)] * str_s[X(m, n)]
            - b1 * b1 * muh_m * hh[X(m - 1, n)] * str_s[X(m - 1, n)]) / g.dyt[X(m, n)];
}

// ---- Function/vel_ssh.f90:707-719 (ssh_internal) --------------------------
__global__ void k_continuity(int m0, int m1, int n0, int n1, Dom D, GridDev g, Consts c,
                             double dt, double *sshn, const double *sshp, const double *u,
                             const double *v, const double *wflux)
{
    RANGE_GUARD
    if (g.lu[X(m, n)] > 0.5f) {
        const double *dxh = g.dxh, *dyh = g.dyh;
        const double div = u[X(m, n)] * dyh[X(m, n)] - u[X(m - 1, n)] * dyh[X(m - 1, n)]
                           + v[X(m, n)] * dxh[X(m, n)] - v[X(m, n - 1)] * dxh[X(m, n - 1)];
        sshn[X(m, n)] = sshp[X(m, n)] + 2.0 * dt * (wflux[X(m, n)] / c.rho * (double)c.ffs
                                                    - div / (g.dx[X(m, n)] * g.dy[X(m, n)]));
    }
}

// ---- Function/vel_ssh.f90:738-741 (ssh_internal) ---------------------------
__global__ void k_asselin_ssh(int m0, int m1, int n0, int n1, Dom D, GridDev g, double ts, double *ssh,
                              double *sshp, const double *sshn)
{
    RANGE_GUARD
    const long long i = X(m, n);
    if (g.lu[i] > 0.5f) { sshp[i] = asselin(ts, ssh[i], sshn[i], sshp[i], 2.0, 1.0); ssh[i] = sshn[i]; }
}

// ---- one substep, Function/vel_ssh.f90:484-615 -----------------------------
// The reference's loops in as few launches as their dependences allow: a
// loop that reads another's result at neighbouring points starts a new
// kernel (k_step_pre, [k_step_bih1, k_step_bih2,] k_step_main, k_step_shift),
// the rest is done by the thread that owns the point.  The loops' periodic
// wraps (cyclize8_x/_y after each) are part of the kernels: the thread of a
// wrap's target column or row evaluates the loop at its source point, whose
// value is what the wrap copies; points the loop does not compute never
// change during a call, so their wrap is done once before it (wrap_fields).
// One launch per loop took 153 us per substep on a 288 x 160 periodic band
// (36 launches) and 379 us on 1152 x 640; these three take 17 and 196 us,
// bound by the latency of a point's loads and divisions.
__device__ __forceinline__ int wrap_of(int i, int on, int lo, int hi)
{
    if (on) {
        if (i == lo - 1) return hi;
        if (i == hi + 1) return lo;
    }
    return i;
}

// the point whose loop value lands at (m, n), and the loops' ranges
struct Src {
    int m, n;
    bool interior, low, ring;   // nx_start.., nx_start-1..nx_end; (m, n) in the interior's one-point ring
    bool own;                   // the source is the point itself
    bool inner;                 // the point itself lies in the interior
};
__device__ __forceinline__ Src source(const Dom &D, int m, int n)
{
    Src s;
    s.m = wrap_of(m, D.px, D.mmm, D.mm);
    s.n = wrap_of(n, D.py, D.nnn, D.nn);
    s.low = s.m >= D.nx_start - 1 && s.m <= D.nx_end && s.n >= D.ny_start - 1 && s.n <= D.ny_end;
    s.interior = s.low && s.m >= D.nx_start && s.n >= D.ny_start;
    s.ring = m >= D.nx_start - 1 && m <= D.nx_end + 1 && n >= D.ny_start - 1 && n <= D.ny_end + 1;
    s.own = s.m == m && s.n == n;
    s.inner = m >= D.nx_start && m <= D.nx_end && n >= D.ny_start && n <= D.ny_end;
    return s;
}

// launched with programmatic stream serialisation: nothing is read before
// the previous kernel has completed (letting the next one's blocks in
// early, launch_dependents, cost 0.5-1 us of 12-18 per substep)
__device__ __forceinline__ void step_entry() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// NZ threads take a point (part 0 .. NZ-1), in neighbouring blocks, which
// then share their loads in L2
#define STEP_POINT(NZ)                                                  \
    step_entry();                                                       \
    const int part = blockIdx.x % (NZ);                                 \
    const int m = D.bnd_x1 + (int)(blockIdx.x / (NZ)) * SX + threadIdx.x; \
    const int n = D.bnd_y1 + blockIdx.y * SY + threadIdx.y;             \
    if (m > D.bnd_x2 || n > D.bnd_y2) return;                           \
    const Src q = source(D, m, n);                                      \
    const long long i = X(m, n), j = X(q.m, q.n);                       \
    (void)part, (void)j;

constexpr int SX = 32, SY = 4;

// In each kernel the loads of a point come before its stores, in one region
// per mask test, so that they are in flight together: with stores and
// nested mask tests between them the compiler keeps them in order and a
// point waits for some forty loads one after another (24 us per substep
// instead of 17 on 288 x 160 points).  The two components (or the continuity and the
// stresses) of a point are taken by two threads (parts).

// continuity (:487-499; part 0), stresses of the previous level
// (mixing.f90:129-153) and the metric vorticity (:30-42; part 1).
// DERIVE: the depths of the current level are hh_init's from ssh (every
// substep of a run after the first, :668-675), computed here and stored for
// k_step_main.
template <bool DERIVE>
__global__ void __launch_bounds__(SX *SY) k_step_pre(Dom D, GridDev g, Consts c, StepArgs a)
{
    STEP_POINT(2)
    if (!q.low) return;
    const int M = q.m, N = q.n;
    const HqOf hq{g.hrest, a.ssh, (double)c.ffs};
    if (part == 0) {
        if (!DERIVE && !q.interior) return;
        const Src tw = source(D, M - 1, N), ts = source(D, M, N - 1);
        const long long w = X(M - 1, N), so = X(M, N - 1);
        const bool wet = q.interior && g.lu[j] > 0.5f;
        const bool cu = DERIVE && g.llu[j] > 0.5f, cv = DERIVE && g.llv[j] > 0.5f;
        if (!DERIVE && !wet) return;
        // the depths on the four faces; a derived one where hh_init
        // computes it, through the wrap
        double hu0, hv0, huw = 0.0, hvs = 0.0;
        const bool cw = DERIVE && wet && tw.low && g.llu[X(tw.m, tw.n)] > 0.5f;
        const bool cs = DERIVE && wet && ts.low && g.llv[X(ts.m, ts.n)] > 0.5f;
        if (cu && cv && cw && cs) {
            hu0 = h_on_u(D, g, hq, M, N);
            hv0 = h_on_v(D, g, hq, M, N);
            huw = h_on_u(D, g, hq, tw.m, tw.n);
            hvs = h_on_v(D, g, hq, ts.m, ts.n);
        } else {
            hu0 = cu ? h_on_u(D, g, hq, M, N) : a.hu[j];
            hv0 = cv ? h_on_v(D, g, hq, M, N) : a.hv[j];
            if (wet) {
                huw = cw ? h_on_u(D, g, hq, tw.m, tw.n) : a.hu[w];
                hvs = cs ? h_on_v(D, g, hq, ts.m, ts.n) : a.hv[so];
            }
        }
        double sn = 0.0;
        if (wet) {
            const double *dxh = g.dxh, *dyh = g.dyh, *u = a.u, *v = a.v;
            const double div = u[j] * hu0 * dyh[j] - u[w] * huw * dyh[w] + v[j] * hv0 * dxh[j] - v[so] * hvs * dxh[so];
            sn = a.sshp[j] + 2.0 * a.ti * (a.wflux[j] / c.rho * (double)c.ffs - div / (g.dx[j] * g.dy[j]));
        }
        if (cu) a.hu[i] = hu0;
        if (cv) a.hv[i] = hv0;
        if (wet) a.sshn[i] = sn;
        return;
    }
    const bool t = q.interior && g.lu[j] > 0.5f, h = q.interior && g.luu[j] > 0.5f;
    const bool hd = DERIVE && g.luh[j] > 0.5f;
    double st = 0.0, ss = 0.0, vo = 0.0, hh = 0.0;
    if (t && h) {
        st = tension(D, g, a.up, a.vp, M, N);
        ss = shear(D, g, a.up, a.vp, M, N);
        vo = vorticity(D, g, a.u, a.v, M, N);
    } else if (t) {
        st = tension(D, g, a.up, a.vp, M, N);
    } else if (h) {
        ss = shear(D, g, a.up, a.vp, M, N);
        vo = vorticity(D, g, a.u, a.v, M, N);
    }
    if (hd) hh = h_on_h(D, g, hq, M, N);
    if (t) a.strt[i] = st;
    if (h) {
        a.strs[i] = ss;
        a.vort[i] = vo;
    }
    if (hd) a.hh[i] = hh;
}

// uv_diff2 (:141-179) and the first half of uv_diff4 (:216-257), the
// normalised harmonic operator; part the component.  uv_diff2's value
// travels to k_step_main in un (vn), which that kernel overwrites; at an
// interior wrap target its own value in difx (dify).
template <bool INSIDE>
__global__ void __launch_bounds__(SX *SY) k_step_bih1(Dom D, GridDev g, StepArgs a)
{
    STEP_POINT(2)
    const HqArray hq{a.hq};
    if (part == 0) {
        auto div = [&](const double *mu, int M, int N) {
            return dif_xt(D, g, mu, a.strt, hq, M, N) + dif_xs(D, g, mu, a.strs, a.hh, M, N);
        };
        if (INSIDE && q.inner && !q.own && g.lcu[i] > 0.5f) a.difx[i] = div(a.mu, m, n);
        if (!q.interior || !(g.lcu[j] > 0.5f)) return;
        const double f = div(a.mu4, q.m, q.n), d = div(a.mu, q.m, q.n);
        a.fx[i] = -f / a.hu[j] / g.dxt[j] / g.dyh[j];
        a.un[i] = d;
    } else {
        auto div = [&](const double *mu, int M, int N) {
            return -dif_yt(D, g, mu, a.strt, hq, M, N) + dif_ys(D, g, mu, a.strs, a.hh, M, N);
        };
        if (INSIDE && q.inner && !q.own && g.lcv[i] > 0.5f) a.dify[i] = div(a.mu, m, n);
        if (!q.interior || !(g.lcv[j] > 0.5f)) return;
        const double f = div(a.mu4, q.m, q.n), d = div(a.mu, q.m, q.n);
        a.fy[i] = -f / a.hv[j] / g.dxh[j] / g.dyt[j];
        a.vn[i] = d;
    }
}

// the stresses of (fx, fy), :259-272; part 0 tension, 1 shear
__global__ void __launch_bounds__(SX *SY) k_step_bih2(Dom D, GridDev g, StepArgs a)
{
    STEP_POINT(2)
    if (!q.interior) return;
    if (part == 0) {
        if (g.lu[j] > 0.5f) a.strt[i] = tension(D, g, a.fx, a.fy, q.m, q.n);
    } else {
        if (g.luu[j] > 0.5f) a.strs[i] = shear(D, g, a.fx, a.fy, q.m, q.n);
    }
}

// a component's new value, its terms and its parts of the time means
struct Momentum {
    double fn, adv, dif, mean, grad;
};

// the u equation at (M, N) (:536-552), its new depth hn and previous depth hp
template <bool DERIVE, bool MEANS, bool BIH>
__device__ __forceinline__ Momentum momentum_u(const Dom &D, const GridDev &g, const Consts &c, const StepArgs &a, int M,
                                               int N, double hn, double hp, double dif0)
{
    const double *dxt = g.dxt, *dyt = g.dyt, *dxh = g.dxh, *dyh = g.dyh;
    const double *dxb = g.dxb, *dyb = g.dyb, *rlh = g.rlh;
    (void)dxt, (void)dyt, (void)dxh, (void)dyh;
    const double grav = c.g, ti = a.ti;
    const long long k = X(M, N);
    const HqOf hqs{g.hrest, a.ssh, (double)c.ffs};
    const HqArray hqa{a.hq};
    const double hc = a.hu[k];
    Momentum r;
    if (BIH)
        r.dif = dif0 + dif_xt(D, g, a.mu4, a.strt, hqa, M, N) + dif_xs(D, g, a.mu4, a.strs, a.hh, M, N);
    else
        r.dif = (DERIVE ? dif_xt(D, g, a.mu, a.strt, hqs, M, N) : dif_xt(D, g, a.mu, a.strt, hqa, M, N)) +
                dif_xs(D, g, a.mu, a.strs, a.hh, M, N);
    r.adv = trans_x(D, g, a.u, a.v, a.vort, a.hu, a.hv, a.hh, M, N);
    const double bp = hn * dxt[k] * dyh[k] / 2.0 / ti;
    const double bp0 = hp * dxt[k] * dyh[k] / 2.0 / ti;
    const double sl = -grav * (a.ssh[X(M + 1, N)] - a.ssh[k]) * dyh[k] * hc;
    const double gr = a.rhsx[k] * a.rhs_scale + sl + r.dif + r.adv
                      - (a.rdis[k] + a.rdis[X(M + 1, N)]) / 2.0 * a.up[k] * dxt[k] * dyh[k] * hc
                      + (rlh[k] * a.hh[k] * dxb[k] * dyb[k] * (a.v[X(M + 1, N)] + a.v[k])
                         + rlh[X(M, N - 1)] * a.hh[X(M, N - 1)] * dxb[X(M, N - 1)] * dyb[X(M, N - 1)]
                           * (a.v[X(M + 1, N - 1)] + a.v[X(M, N - 1)])) / 4.0;
    r.fn = (a.up[k] * bp0 + gr) / bp;
    if (MEANS) {
        const double sln = -grav * (a.sshn[X(M + 1, N)] - a.sshn[k]) * dyh[k] * hn;
        r.mean = (a.u[k] * hc + r.fn * hn) / a.four_nstep;
        r.grad = (sl + sln) / a.four_nstep;
    }
    return r;
}

// the v equation at (M, N) (:554-571), its new depth hn and previous depth hp
template <bool DERIVE, bool MEANS, bool BIH>
__device__ __forceinline__ Momentum momentum_v(const Dom &D, const GridDev &g, const Consts &c, const StepArgs &a, int M,
                                               int N, double hn, double hp, double dif0)
{
    const double *dxt = g.dxt, *dyt = g.dyt, *dxh = g.dxh, *dyh = g.dyh;
    const double *dxb = g.dxb, *dyb = g.dyb, *rlh = g.rlh;
    (void)dxt, (void)dyt, (void)dxh, (void)dyh;
    const double grav = c.g, ti = a.ti;
    const long long k = X(M, N);
    const HqOf hqs{g.hrest, a.ssh, (double)c.ffs};
    const HqArray hqa{a.hq};
    const double hc = a.hv[k];
    Momentum r;
    if (BIH)
        r.dif = dif0 - dif_yt(D, g, a.mu4, a.strt, hqa, M, N) + dif_ys(D, g, a.mu4, a.strs, a.hh, M, N);
    else
        r.dif = -(DERIVE ? dif_yt(D, g, a.mu, a.strt, hqs, M, N) : dif_yt(D, g, a.mu, a.strt, hqa, M, N)) +
                dif_ys(D, g, a.mu, a.strs, a.hh, M, N);
    r.adv = trans_y(D, g, a.u, a.v, a.vort, a.hu, a.hv, a.hh, M, N);
    const double bp = hn * dyt[k] * dxh[k] / 2.0 / ti;
    const double bp0 = hp * dyt[k] * dxh[k] / 2.0 / ti;
    const double sl = -grav * (a.ssh[X(M, N + 1)] - a.ssh[k]) * dxh[k] * hc;
    const double gr = a.rhsy[k] * a.rhs_scale + sl + r.dif + r.adv
                      - (a.rdis[k] + a.rdis[X(M, N + 1)]) / 2.0 * a.vp[k] * dxh[k] * dyt[k] * hc
                      - (rlh[k] * a.hh[k] * dxb[k] * dyb[k] * (a.u[X(M, N + 1)] + a.u[k])
                         + rlh[X(M - 1, N)] * a.hh[X(M - 1, N)] * dxb[X(M - 1, N)] * dyb[X(M - 1, N)]
                           * (a.u[X(M - 1, N + 1)] + a.u[X(M - 1, N)])) / 4.0;
    r.fn = (a.vp[k] * bp0 + gr) / bp;
    if (MEANS) {
        const double sln = -grav * (a.sshn[X(M, N + 1)] - a.sshn[k]) * dxh[k] * hn;
        r.mean = (a.v[k] * hc + r.fn * hn) / a.four_nstep;
        r.grad = (sl + sln) / a.four_nstep;
    }
    return r;
}

// hh_update (depth.f90:108-170), uv_trans (:54-109), uv_diff2 or the second
// half of uv_diff4 (:274-312), the momentum equations and the time means
// (:531-573), part the component.  MEANS: a barotropic_dynamics substep,
// which carries the new depths on and adds to the time means; else a run's
// substep, which needs neither.  INSIDE: a wrap's target column or row lies
// in the interior.
template <bool DERIVE, bool MEANS, bool BIH, bool INSIDE>
__global__ void __launch_bounds__(SX *SY, 4) k_step_main(Dom D, GridDev g, Consts c, StepArgs a)
{
    STEP_POINT(2)
    const HqOf hqn{g.hrest, a.sshn, 1.0}, hqp{g.hrest, a.sshp, (double)c.ffs};
    const bool moving = c.ffs > 0;
    const bool here = q.low || (INSIDE && q.inner);
    if (part == 0) {
        if (MEANS && moving) a.hqn[i] = hqn(i);
        if (!here) return;
        const bool deep = g.llu[j] > 0.5f, ch = moving && q.low && deep, cp = DERIVE && q.low && deep;
        const bool wet = q.interior && g.lcu[j] > 0.5f;
        double hn = 0.0;
        Momentum r = {};
        if (wet && ch && (cp || !DERIVE)) {
            hn = h_on_u(D, g, hqn, q.m, q.n);
            const double hp = DERIVE ? h_on_u(D, g, hqp, q.m, q.n) : a.hup[j];
            r = momentum_u<DERIVE, MEANS, BIH>(D, g, c, a, q.m, q.n, hn, hp, BIH ? a.un[i] : 0.0);
        } else {
            if (ch && (MEANS || INSIDE)) hn = h_on_u(D, g, hqn, q.m, q.n);
            else hn = a.hun[j];
            if (wet) {
                const double hp = cp ? h_on_u(D, g, hqp, q.m, q.n) : a.hup[j];
                if (ch && !MEANS) hn = h_on_u(D, g, hqn, q.m, q.n);
                r = momentum_u<DERIVE, MEANS, BIH>(D, g, c, a, q.m, q.n, hn, hp, BIH ? a.un[i] : 0.0);
            }
        }
        if (wet) a.un[i] = r.fn;
        if (MEANS && ch) a.hun[i] = hn;
        bool mine = wet && q.own;
        if (INSIDE && !q.own && q.inner && g.lcu[i] > 0.5f) {
            // an interior point under a wrap: its own time means and terms
            const double hp = cp ? h_on_u(D, g, hqp, q.m, q.n) : a.hup[i];
            r = momentum_u<DERIVE, MEANS, BIH>(D, g, c, a, m, n, hn, hp, BIH ? a.difx[i] : 0.0);
            mine = true;
        }
        if (MEANS && mine) {
            a.ui[i] = a.ui[i] + r.mean;
            a.gx[i] = a.gx[i] + r.grad;
        }
        if (a.last && mine) {
            a.advx[i] = r.adv;
            a.difx[i] = r.dif;
        }
    } else {
        if (!here) return;
        if (MEANS && moving && q.low && g.luh[j] > 0.5f) a.hhn[i] = h_on_h(D, g, hqn, q.m, q.n);
        const bool deep = g.llv[j] > 0.5f, ch = moving && q.low && deep, cp = DERIVE && q.low && deep;
        const bool wet = q.interior && g.lcv[j] > 0.5f;
        double hn = 0.0;
        Momentum r = {};
        if (wet && ch && (cp || !DERIVE)) {
            hn = h_on_v(D, g, hqn, q.m, q.n);
            const double hp = DERIVE ? h_on_v(D, g, hqp, q.m, q.n) : a.hvp[j];
            r = momentum_v<DERIVE, MEANS, BIH>(D, g, c, a, q.m, q.n, hn, hp, BIH ? a.vn[i] : 0.0);
        } else {
            if (ch && (MEANS || INSIDE)) hn = h_on_v(D, g, hqn, q.m, q.n);
            else hn = a.hvn[j];
            if (wet) {
                const double hp = cp ? h_on_v(D, g, hqp, q.m, q.n) : a.hvp[j];
                if (ch && !MEANS) hn = h_on_v(D, g, hqn, q.m, q.n);
                r = momentum_v<DERIVE, MEANS, BIH>(D, g, c, a, q.m, q.n, hn, hp, BIH ? a.vn[i] : 0.0);
            }
        }
        if (wet) a.vn[i] = r.fn;
        if (MEANS && ch) a.hvn[i] = hn;
        bool mine = wet && q.own;
        if (INSIDE && !q.own && q.inner && g.lcv[i] > 0.5f) {
            // an interior point under a wrap: its own time means and terms
            const double hp = cp ? h_on_v(D, g, hqp, q.m, q.n) : a.hvp[i];
            r = momentum_v<DERIVE, MEANS, BIH>(D, g, c, a, m, n, hn, hp, BIH ? a.dify[i] : 0.0);
            mine = true;
        }
        if (MEANS && mine) {
            a.vi[i] = a.vi[i] + r.mean;
            a.gy[i] = a.gy[i] + r.grad;
        }
        if (a.last && mine) {
            a.advy[i] = r.adv;
            a.dify[i] = r.dif;
        }
    }
}

// the Robert-Asselin filter and shift on the interior and its ring
// (:589-612; part 0) and, with a free surface in barotropic_dynamics,
// hh_shift (depth.f90:191-217; part 1)
template <int NZ>
__global__ void __launch_bounds__(SX *SY) k_step_shift(Dom D, GridDev g, double ts, StepArgs a)
{
    STEP_POINT(NZ)
    if (!q.ring) return;
    // every load before the first store
    struct Three {
        double f, fn, fp;
    };
    auto load = [&](const double *f, const double *fn, const double *fp) { return Three{f[i], fn[i], fp[i]}; };
    auto store = [&](double *f, double *fp, const Three &x) {
        fp[i] = asselin(ts, x.f, x.fn, x.fp, 2.0, a.ns);
        f[i] = x.fn;
    };
    const bool t = g.lu[i] > 0.5f, cu = g.lcu[i] > 0.5f, cv = g.lcv[i] > 0.5f;
    if (part == 0) {
        const Three x = load(a.ssh, a.sshn, a.sshp), u = load(a.u, a.un, a.up), v = load(a.v, a.vn, a.vp);
        if (t) store(a.ssh, a.sshp, x);
        if (cu) store(a.u, a.up, u);
        if (cv) store(a.v, a.vp, v);
    } else {
        const bool du = g.llu[i] > 0.5f, dv = g.llv[i] > 0.5f, dh = g.luh[i] > 0.5f;
        const Three x = load(a.hq, a.hqn, a.hqp), u = load(a.hu, a.hun, a.hup), v = load(a.hv, a.hvn, a.hvp),
                    h = load(a.hh, a.hhn, a.hhp);
        if (du) store(a.hu, a.hup, u);
        if (dv) store(a.hv, a.hvp, v);
        if (t) store(a.hq, a.hqp, x);
        if (dh) store(a.hh, a.hhp, h);
    }
}

// hh_init (depth.f90:2-105), all twelve arrays with their wraps
struct Depths {
    double *p[12];   // hq hqp hqn hu hup hun hv hvp hvn hh hhp hhn
};
__global__ void __launch_bounds__(SX *SY) k_hh_init(Dom D, GridDev g, double ffs, const __grid_constant__ Depths h,
                                                    const double *sh, const double *shp)
{
    STEP_POINT(3)
    // part: the time level
    const int l = part;
    const HqOf hq{g.hrest, l == 0 ? sh : shp, ffs};
    const HqRest rest{g.hrest};
    const bool du = q.low && g.llu[j] > 0.5f, dv = q.low && g.llv[j] > 0.5f, dh = q.low && g.luh[j] > 0.5f;
    double hu = 0.0, hv = 0.0, hh = 0.0;
    auto faces = [&](const auto &f) {
        if (du && dv && dh) {
            hu = h_on_u(D, g, f, q.m, q.n);
            hv = h_on_v(D, g, f, q.m, q.n);
            hh = h_on_h(D, g, f, q.m, q.n);
            return;
        }
        if (du) hu = h_on_u(D, g, f, q.m, q.n);
        if (dv) hv = h_on_v(D, g, f, q.m, q.n);
        if (dh) hh = h_on_h(D, g, f, q.m, q.n);
    };
    double ht;
    if (l < 2) {
        ht = hq(i);
        faces(hq);
    } else {
        ht = rest(i);
        faces(rest);
    }
    h.p[l][i] = ht;
    if (du) h.p[3 + l][i] = hu;
    if (dv) h.p[6 + l][i] = hv;
    if (dh) h.p[9 + l][i] = hh;
}

// cyclize8_x then cyclize8_y of several fields (one per grid y)
struct Fields {
    double *p[12];
};
__global__ void k_wrap_fields(Dom D, Fields f)
{
    double *a = f.p[blockIdx.y];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int nya = D.bnd_y2 - D.bnd_y1 + 1, nxa = D.bnd_x2 - D.bnd_x1 + 1;
    // the y wrap runs last and reads x-wrapped columns: its rows take both
    if (D.px && t < nya) {
        const int n = D.bnd_y1 + t;
        if (!D.py || (n != D.nnn - 1 && n != D.nn + 1)) {
            const double left = a[X(D.mm, n)], right = a[X(D.mmm, n)];
            a[X(D.mmm - 1, n)] = left;
            a[X(D.mm + 1, n)] = right;
        }
    }
    if (D.py && t < nxa) {
        const int m = D.bnd_x1 + t, sm = wrap_of(m, D.px, D.mmm, D.mm);
        const double s = a[X(sm, D.nn)], nth = a[X(sm, D.nnn)];
        a[X(m, D.nnn - 1)] = s;
        a[X(m, D.nn + 1)] = nth;
    }
}

// dst[k] = src[k] (or 0 where src[k] is null) over the whole arrays, field
// k per grid z
__global__ void k_set_fields(int m0, int m1, int n0, int n1, Dom D, FieldSet f)
{
    RANGE_GUARD
    const double *src = f.src[blockIdx.z];
    f.dst[blockIdx.z][X(m, n)] = src ? src[X(m, n)] : 0.0;
}

// ---- Control/init_pars.f90:459-481 -----------------------------------------
__global__ void k_r_diss(int m0, int m1, int n0, int n1, Dom D, GridDev g, double r_fric, double *r)
{
    RANGE_GUARD
    if (g.lu[X(m, n)] > 0.5f) {
        const double *h = g.hrest, *dxt = g.dxt, *dyt = g.dyt;
        const float *lcu = g.lcu, *lcv = g.lcv;
        double a = (h[X(m + 1, n)] - h[X(m, n)]) / dxt[X(m, n)];
        double b = (h[X(m, n)] - h[X(m - 1, n)]) / dxt[X(m - 1, n)];
        double hx2 = (a * a * (double)lcu[X(m, n)] + b * b * (double)lcu[X(m - 1, n)])
                     / (double)(lcu[X(m, n)] + lcu[X(m - 1, n)]);
        double d = (h[X(m, n + 1)] - h[X(m, n)]) / dyt[X(m, n)];
        double e = (h[X(m, n)] - h[X(m, n - 1)]) / dyt[X(m, n - 1)];
        double hy2 = (d * d * (double)lcv[X(m, n)] + e * e * (double)lcv[X(m, n - 1)])
                     / (double)(lcv[X(m, n)] + lcv[X(m, n - 1)]);
        r[X(m, n)] = r_fric * sqrt(hx2 + hy2);
    }
}

// ---- Function/fluxes.f90:29-37 + Control/dyncall.f90:115-125 --------------
__global__ void k_wind(int m0, int m1, int n0, int n1, Dom D, GridDev g, double rho,
                       const double *taux, const double *tauy, double *rhsx, double *rhsy)
{
    RANGE_GUARD
    const long long i = X(m, n);
    const double *dx = g.dx, *dy = g.dy;
    if (g.lcu[i] > 0.5f) {
        double ss = (taux[i] * dx[i] * dy[i] + taux[X(m + 1, n)] * dx[X(m + 1, n)] * dy[X(m + 1, n)])
                    / rho / 2.0 / g.dxt[i] / g.dyh[i];
        // dyncall.f90:115-118 with the 3-D, bottom-stress and slpr terms zero
        rhsx[i] = rhsx[i] + ss * g.dxt[i] * g.dyh[i];
    }
    if (g.lcv[i] > 0.5f) {
        double ss = (tauy[i] * dx[i] * dy[i] + tauy[X(m, n + 1)] * dx[X(m, n + 1)] * dy[X(m, n + 1)])
                    / rho / 2.0 / g.dxh[i] / g.dyt[i];
        rhsy[i] = rhsy[i] + ss * g.dyt[i] * g.dxh[i];
    }
}

// ---- Control/dyncall.f90:110-130: the barotropic RHS, one term per launch
// in the reference's left-to-right order, so that every step rounds where
// the Fortran expression rounds (this file: --fmad=false, no reassociation):
// term 0: r - a; 1: r + a; 2: r + (a + b) * area; 3: r - dslpr * b * d / rho
__global__ void k_rhs2d_term(int m0, int m1, int n0, int n1, Dom D, GridDev g, double rho, int term,
                             double *rx, double *ry, const double *ax, const double *ay, const double *bx,
                             const double *by)
{
    RANGE_GUARD
    const long long i = X(m, n);
    if (g.lcu[i] > 0.5f) {
        double r = rx[i];
        if (term == 0) r = r - ax[i];
        else if (term == 1) r = r + ax[i];
        else if (term == 2) r = r + (ax[i] + bx[i]) * g.dxt[i] * g.dyh[i];
        else r = r - (ax[X(m + 1, n)] - ax[i]) * bx[i] * g.dyh[i] / rho;
        rx[i] = r;
    }
    if (g.lcv[i] > 0.5f) {
        double r = ry[i];
        if (term == 0) r = r - ay[i];
        else if (term == 1) r = r + ay[i];
        else if (term == 2) r = r + (ay[i] + by[i]) * g.dyt[i] * g.dxh[i];
        else r = r - (ay[X(m, n + 1)] - ay[i]) * by[i] * g.dxh[i] / rho;
        ry[i] = r;
    }
}

// ---- Control/dyncall.f90:188-201: corrected 2-D velocity and the slpr part
// of the time-mean pressure gradient (interior and its one-point ring)
__global__ void k_velocity2d(int m0, int m1, int n0, int n1, Dom D, GridDev g, double rho, double *uu2d,
                             double *vv2d, double *pgrx, double *pgry, const double *ubrtr_i,
                             const double *vbrtr_i, const double *slpr, const double *hhu, const double *hhv)
{
    RANGE_GUARD
    const long long i = X(m, n);
    if (g.lcu[i] > 0.5f) {
        uu2d[i] = ubrtr_i[i] / hhu[i];
        pgrx[i] = pgrx[i] - (slpr[X(m + 1, n)] - slpr[i]) * hhu[i] * g.dyh[i] / rho;
    }
    if (g.lcv[i] > 0.5f) {
        vv2d[i] = vbrtr_i[i] / hhv[i];
        pgry[i] = pgry[i] - (slpr[X(m, n + 1)] - slpr[i]) * hhv[i] * g.dxh[i] / rho;
    }
}

// ---- Service/grid_construction.f90:59-112 -----------------------------------
__global__ void k_gridcon(int m0, int m1, int n0, int n1, Dom D, const float *lu, float *luu,
                          float *luh, float *llu, float *llv, float *lcu, float *lcv)
{
    RANGE_GUARD
    float a = lu[X(m, n)], b = lu[X(m + 1, n)], cc = lu[X(m, n + 1)], d = lu[X(m + 1, n + 1)];
    if (a + b + cc + d > 0.5f) luh[X(m, n)] = 1.0f;
    if (a * b * cc * d > 0.5f) luu[X(m, n)] = 1.0f;
    if (a + b > 0.5f) llu[X(m, n)] = 1.0f;
    if (a + cc > 0.5f) llv[X(m, n)] = 1.0f;
    if (a * b > 0.5f) lcu[X(m, n)] = 1.0f;
    if (a * cc > 0.5f) lcv[X(m, n)] = 1.0f;
}

// ---- Control/dyncall.f90:452-516 ---------------------------------------------
__global__ void k_guard(int m0, int m1, int n0, int n1, Dom D, GridDev g, const double *ssh,
                        const double *u, const double *v, unsigned long long *nbad)
{
    const int m = m0 + blockIdx.x * BX + threadIdx.x;
    const int n = n0 + blockIdx.y * BY + threadIdx.y;
    unsigned bad = 0;
    if (m <= m1 && n <= n1) {
        const long long i = X(m, n);
        if (g.lu[i] > 0.5f && !(ssh[i] < 10.0 && ssh[i] > -10.0)) bad++;
        if (g.lcu[i] > 0.5f && !(u[i] < 100.0 && u[i] > -100.0)) bad++;
        if (g.lcv[i] > 0.5f && !(v[i] < 100.0 && v[i] > -100.0)) bad++;
    }
    // warp-aggregated count
    for (int o = 16; o > 0; o >>= 1) bad += __shfl_down_sync(0xffffffffu, bad, o);
    if ((threadIdx.x & 31) == 0 && bad) atomicAdd(nbad, (unsigned long long)bad);
}

// one block per interior row; fixed-order tree reduction -> deterministic
__global__ void k_diag_rows(Dom D, GridDev g, Consts c, const double *ssh, const double *u,
                            const double *v, const double *hu, const double *hv, double *rows)
{
    const int n = D.ny_start + blockIdx.x;
    const int nrows = D.ny_end - D.ny_start + 1;
    double vol = 0.0, en = 0.0;
    for (int m = D.nx_start + threadIdx.x; m <= D.nx_end; m += blockDim.x) {
        const long long i = X(m, n);
        if (g.lu[i] > 0.5f) {
            double a = g.dx[i] * g.dy[i];
            vol += (g.hrest[i] + ssh[i]) * a;
            en += 0.5 * c.g * ssh[i] * ssh[i] * a;
        }
        if (g.lcu[i] > 0.5f) en += 0.5 * hu[i] * u[i] * u[i] * g.dxt[i] * g.dyh[i];
        if (g.lcv[i] > 0.5f) en += 0.5 * hv[i] * v[i] * v[i] * g.dxh[i] * g.dyt[i];
    }
    for (int o = 16; o > 0; o >>= 1) {
        vol += __shfl_down_sync(0xffffffffu, vol, o);
        en += __shfl_down_sync(0xffffffffu, en, o);
    }
    __shared__ double sv[32], se[32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { sv[w] = vol; se[w] = en; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) { a += sv[k]; b += se[k]; }
        rows[blockIdx.x] = a;
        rows[nrows + blockIdx.x] = b;
    }
}

__global__ void k_diag_final(int nrows, const double *rows, double *out)
{
    // two warps sum the two columns of partials, each lane a fixed stride,
    // then a fixed shuffle tree: independent of timing
    const int col = threadIdx.x >> 5, l = threadIdx.x & 31;
    double s = 0.0;
    for (int k = l; k < nrows; k += 32) s += rows[col * nrows + k];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (l == 0) out[col] = s;
}

#undef X
#undef RANGE_GUARD

}  // namespace

// ===========================================================================
void fill(const Dom &d, double *f, double v, cudaStream_t s)
{
    launch2d(k_fill, d.bnd_x1, d.bnd_x2, d.bnd_y1, d.bnd_y2, s, d, f, v);
}

void halo(const Dom &d, double *f, cudaStream_t s)
{
    if (d.px) k_cyclize_x<<<(d.nya() + 127) / 128, 128, 0, s>>>(d, f);
    if (d.py) k_cyclize_y<<<(d.nxa() + 127) / 128, 128, 0, s>>>(d, f);
}

void wrap_fields(const Dom &d, std::initializer_list<double *> fields, cudaStream_t s)
{
    if (!d.px && !d.py) return;
    Fields f = {};
    int k = 0;
    for (double *p : fields) f.p[k++] = p;
    const int len = d.px && d.py ? std::max(d.nya(), d.nxa()) : (d.px ? d.nya() : d.nxa());
    k_wrap_fields<<<dim3((len + 127) / 128, k), 128, 0, s>>>(d, f);
}

void set_fields(const Dom &d, const FieldSet &f, cudaStream_t s)
{
    if (f.n < 1) return;
    const dim3 grid((d.nxa() + BX - 1) / BX, (d.nya() + BY - 1) / BY, f.n);
    k_set_fields<<<grid, dim3(BX, BY), 0, s>>>(d.bnd_x1, d.bnd_x2, d.bnd_y1, d.bnd_y2, d, f);
}

namespace {
// nz threads per point of the arrays; the kernel waits for its predecessor
// (programmatic stream serialisation), so that its launch overlaps it
template <typename... P, typename... A>
void step_launch(void (*k)(P...), int nz, const Dom &d, cudaStream_t s, A... a)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nz * ((d.nxa() + SX - 1) / SX), (d.nya() + SY - 1) / SY);
    cfg.blockDim = dim3(SX, SY);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, k, P(a)...);   // errors: cudaGetLastError
}
}  // namespace

void hh_init(const Dom &d, const GridDev &g, const Consts &c, double *const h[12], const double *sh,
             const double *shp, cudaStream_t s)
{
    Depths p;
    for (int k = 0; k < 12; k++) p.p[k] = h[k];
    step_launch(k_hh_init, 3, d, s, d, g, (double)c.ffs, p, sh, shp);
    wrap_fields(d, {h[3], h[4], h[5], h[6], h[7], h[8], h[9], h[10], h[11]}, s);
}

void hh_update(const Dom &d, const GridDev &g, double *hqn, double *hun,
               double *hvn, double *hhn, const double *sh, cudaStream_t s)
{
    launch2d(k_hq_set, d.bnd_x1, d.bnd_x2, d.bnd_y1, d.bnd_y2, s, d, g.hrest, hqn, sh, 1.0, 1);
    launch2d(k_hh_interp, d.nx_start - 1, d.nx_end, d.ny_start - 1, d.ny_end, s, d, g,
             (const double *)hqn, hun, hvn, hhn);
    halo(d, hun, s);
    halo(d, hvn, s);
    halo(d, hhn, s);
}

// a wrap's target column or row lies in the interior
static bool wrap_inside(const Dom &d)
{
    auto in = [](int i, int lo, int hi) { return i >= lo && i <= hi; };
    return (d.px && (in(d.mmm - 1, d.nx_start, d.nx_end) || in(d.mm + 1, d.nx_start, d.nx_end))) ||
           (d.py && (in(d.nnn - 1, d.ny_start, d.ny_end) || in(d.nn + 1, d.ny_start, d.ny_end)));
}

void substep(const Dom &d, const GridDev &g, const Consts &c, const StepArgs &a, bool means, bool derive, int ksw4,
             cudaStream_t s)
{
    const bool in = wrap_inside(d), bih = means && ksw4 > 0;
    step_launch(derive ? k_step_pre<true> : k_step_pre<false>, 2, d, s, d, g, c, a);
    if (bih) {
        step_launch(in ? k_step_bih1<true> : k_step_bih1<false>, 2, d, s, d, g, a);
        step_launch(k_step_bih2, 2, d, s, d, g, a);
    }
    auto *k = bih ? (in ? k_step_main<false, true, true, true> : k_step_main<false, true, true, false>)
              : means ? (in ? k_step_main<false, true, false, true> : k_step_main<false, true, false, false>)
              : derive ? (in ? k_step_main<true, false, false, true> : k_step_main<true, false, false, false>)
                       : (in ? k_step_main<false, false, false, true> : k_step_main<false, false, false, false>);
    step_launch(k, 2, d, s, d, g, c, a);
    const bool depths = means && c.ffs > 0;
    step_launch(depths ? k_step_shift<2> : k_step_shift<1>, depths ? 2 : 1, d, s, d, g, c.ts, a);
}

void continuity(const Dom &d, const GridDev &g, const Consts &c, double dt,
                double *sshn, const double *sshp, const double *u,
                const double *v, const double *wflux, cudaStream_t s)
{
    launch2d(k_continuity, d.nx_start, d.nx_end, d.ny_start, d.ny_end, s, d, g, c, dt, sshn,
             sshp, u, v, wflux);
}

void asselin_ssh(const Dom &d, const GridDev &g, const Consts &c, double *ssh, double *sshp, const double *sshn,
                 cudaStream_t s)
{
    // "/2.0d0" of vel_ssh.f90:743; the kernel divides by nstep = 1 as well (exact)
    launch2d(k_asselin_ssh, d.nx_start - 1, d.nx_end + 1, d.ny_start - 1, d.ny_end + 1, s, d, g, c.ts, ssh, sshp,
             sshn);
}

void r_diss(const Dom &d, const GridDev &g, double r_fric, double *r, cudaStream_t s)
{
    launch2d(k_r_diss, d.nx_start, d.nx_end, d.ny_start, d.ny_end, s, d, g, r_fric, r);
    halo(d, r, s);
}

void wind_forcing(const Dom &d, const GridDev &g, const Consts &c,
                  const double *taux, const double *tauy, double *rhsx,
                  double *rhsy, cudaStream_t s)
{
    launch2d(k_wind, d.nx_start, d.nx_end, d.ny_start, d.ny_end, s, d, g, c.rho, taux, tauy,
             rhsx, rhsy);
}

void velocity2d(const Dom &d, const GridDev &g, const Consts &c, double *uu2d, double *vv2d, double *pgrx,
                double *pgry, const double *ubrtr_i, const double *vbrtr_i, const double *slpr, const double *hhu,
                const double *hhv, cudaStream_t s)
{
    launch2d(k_velocity2d, d.nx_start - 1, d.nx_end + 1, d.ny_start - 1, d.ny_end + 1, s, d, g, c.rho, uu2d, vv2d,
             pgrx, pgry, ubrtr_i, vbrtr_i, slpr, hhu, hhv);
}

void rhs2d_term(const Dom &d, const GridDev &g, const Consts &c, int term, double *rx, double *ry,
                const double *ax, const double *ay, const double *bx, const double *by, cudaStream_t s)
{
    launch2d(k_rhs2d_term, d.nx_start, d.nx_end, d.ny_start, d.ny_end, s, d, g, c.rho, term, rx, ry, ax, ay,
             bx, by);
}

void gridcon(const Dom &d, const float *lu, float *luu, float *luh, float *llu,
             float *llv, float *lcu, float *lcv, cudaStream_t s)
{
    launch2d(k_gridcon, d.nx_start - 1, d.nx_end, d.ny_start - 1, d.ny_end, s, d, lu, luu,
             luh, llu, llv, lcu, lcv);
}

void guard(const Dom &d, const GridDev &g, const double *ssh, const double *u,
           const double *v, unsigned long long *nbad, cudaStream_t s)
{
    launch2d(k_guard, d.nx_start, d.nx_end, d.ny_start, d.ny_end, s, d, g, ssh, u, v, nbad);
}

void diag_rows(const Dom &d, const GridDev &g, const Consts &c,
               const double *ssh, const double *u, const double *v,
               const double *hu, const double *hv, double *rows, cudaStream_t s)
{
    const int nrows = d.ny_end - d.ny_start + 1;
    if (nrows <= 0) return;
    k_diag_rows<<<nrows, 256, 0, s>>>(d, g, c, ssh, u, v, hu, hv, rows);
}

void diag_final(int nrows, const double *rows, double *out, cudaStream_t s)
{
    k_diag_final<<<1, 64, 0, s>>>(nrows, rows, out);
}

}  // namespace general
}  // namespace inmsom
