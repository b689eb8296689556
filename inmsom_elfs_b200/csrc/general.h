// The barotropic step's general path.
//
// The reference's loops over the same index ranges, with the same masks and
// the same expression order, merged into the few kernels that their
// dependences allow; the file is compiled with --fmad=false, so every
// product and sum rounds where the Fortran expression rounds it.  This path
// handles everything the reference supports on one domain: 2-D metric
// arrays, periodic x/y wrap, the biharmonic option (ksw4) and ocean points
// in the halo ring.
#pragma once

#include <initializer_list>

#include "common.cuh"

namespace inmsom {
namespace general {

// whole-array helpers
void fill(const Dom &d, double *f, double v, cudaStream_t s);
// dst[k] = src[k], or 0 where src[k] is null, k < n, in one launch
struct FieldSet {
    double *dst[16];
    const double *src[16];
    int n;
    void add(double *d, const double *s) { dst[n] = d; src[n++] = s; }
};
void set_fields(const Dom &d, const FieldSet &f, cudaStream_t s);
// syncborder_real8 (a no-op on one domain) + cyclize8_x/_y
void halo(const Dom &d, double *f, cudaStream_t s);

// the same wraps of up to twelve fields in one launch (none: nothing)
void wrap_fields(const Dom &d, std::initializer_list<double *> fields, cudaStream_t s);

// Function/depth.f90:2-105; h: hq hqp hqn hu hup hun hv hvp hvn hh hhp hhn
void hh_init(const Dom &d, const GridDev &g, const Consts &c, double *const h[12], const double *sh,
             const double *shp, cudaStream_t s);
// Function/depth.f90:108-170
void hh_update(const Dom &d, const GridDev &g, double *hqn, double *hun,
               double *hvn, double *hhn, const double *sh, cudaStream_t s);

// One substep of the loop body of Function/vel_ssh.f90:484-615 on the work
// arrays.  means: a substep of barotropic_dynamics (time means, the new
// depths carried on and shifted by hh_shift); else one of a run, which ends
// with hh_init of the depths: derive takes the current and previous depths
// from ssh and sshp (every substep after a run's first) instead of the
// arrays.  last: store the advective and viscous terms (advx .. dify), which
// every substep of the reference overwrites.  Before the first substep
// sshn, un, vn (and fx, fy with ksw4 > 0) are zero and the wraps of vort,
// strt, strs (and hun, hvn, hhn) are done; before the first derived one
// those of hu, hv, hh.
struct StepArgs {
    double *u, *up, *un, *v, *vp, *vn, *ssh, *sshp, *sshn;
    double *hq, *hqp, *hqn, *hu, *hup, *hun, *hv, *hvp, *hvn, *hh, *hhp, *hhn;
    double *vort, *strt, *strs, *fx, *fy, *advx, *advy, *difx, *dify;
    double *ui, *vi, *gx, *gy;   // time means
    const double *rhsx, *rhsy, *wflux, *mu, *mu4, *rdis;
    double rhs_scale;            // RHSx/RHSy are used as RHSx*rhs_scale (x*1.0 == x)
    double ti, ns, four_nstep;   // inner step, nstep, 4*nstep
    int last;
};
void substep(const Dom &d, const GridDev &g, const Consts &c, const StepArgs &a, bool means, bool derive, int ksw4,
             cudaStream_t s);

// Function/vel_ssh.f90:707-719 and :738-741 (ssh_internal)
void continuity(const Dom &d, const GridDev &g, const Consts &c, double dt,
                double *sshn, const double *sshp, const double *u,
                const double *v, const double *wflux, cudaStream_t s);
void asselin_ssh(const Dom &d, const GridDev &g, const Consts &c, double *ssh, double *sshp, const double *sshn,
                 cudaStream_t s);

// Control/init_pars.f90:459-481
void r_diss(const Dom &d, const GridDev &g, double r_fric, double *r, cudaStream_t s);
// Function/fluxes.f90:29-37 followed by Control/dyncall.f90:110-130 (wind only)
void wind_forcing(const Dom &d, const GridDev &g, const Consts &c,
                  const double *taux, const double *tauy, double *rhsx,
                  double *rhsy, cudaStream_t s);
// Control/dyncall.f90:188-201: uu2d = ubrtr_i/hhu, pgrx -= slpr gradient (and v)
void velocity2d(const Dom &d, const GridDev &g, const Consts &c, double *uu2d, double *vv2d, double *pgrx,
                double *pgry, const double *ubrtr_i, const double *vbrtr_i, const double *slpr, const double *hhu,
                const double *hhv, cudaStream_t s);
// Control/dyncall.f90:110-130, one term of the barotropic RHS in the
// reference's order: 0 r -= a, 1 r += a, 2 r += (a + b) * (dxt*dyh | dyt*dxh),
// 3 r -= (a(next) - a) * b * (dyh | dxh) / rho (a = slpr, b = hhu | hhv)
void rhs2d_term(const Dom &d, const GridDev &g, const Consts &c, int term, double *rx, double *ry,
                const double *ax, const double *ay, const double *bx, const double *by, cudaStream_t s);
// Service/grid_construction.f90:59-112
void gridcon(const Dom &d, const float *lu, float *luu, float *luh, float *llu,
             float *llv, float *lcu, float *lcv, cudaStream_t s);
// Control/dyncall.f90:452-516 on (ssh, u, v); adds the count to *nbad
void guard(const Dom &d, const GridDev &g, const double *ssh, const double *u,
           const double *v, unsigned long long *nbad, cudaStream_t s);
// volume/energy partial sums per interior row (deterministic); rows holds
// 2*(ny_end-ny_start+1) doubles
void diag_rows(const Dom &d, const GridDev &g, const Consts &c,
               const double *ssh, const double *u, const double *v,
               const double *hu, const double *hv, double *rows, cudaStream_t s);
// sums the row partials in row order into out[0] (volume) and out[1] (energy)
void diag_final(int nrows, const double *rows, double *out, cudaStream_t s);

}  // namespace general
}  // namespace inmsom
