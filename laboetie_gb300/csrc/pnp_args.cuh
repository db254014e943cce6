// pnp_args.cuh -- arguments and node helpers shared by the Poisson-Nernst-Planck kernels: one launch
// per step (pnp.cu) and a resident loop (pnp_resident.cu).
#pragma once

#include "common.cuh"
#include "gridsync.cuh"
#include "lbgpu.h"
#include "pnp.h"

namespace lbg {

struct PnpArgs {
    const uint32_t *mask;
    const double *phi;
    double *phi_out;
    const double *cp, *cm;
    double *fp, *fm;
    double *partial;
    PnpCtl *ctl;
    long long N;
    int lx, ly, lz;
    double a0[3];
    double factor, omega, one_minus_omega;
    double eDp, eDm;
    double delta_axis, delta_diag;
    int color;        // multicolour SOR: the colour of this launch
    int ncolor;       // colours per sweep (the last colour's launch decides the stopping test)
    int gen;          // general colouring (some side odd): colour from k_sor_color_gen's rule
    int kx, ky, kz;   // colours per axis of the general colouring (1, 2 or 3)
    int loop_bug;     // just_eq_smolu.f90:68-70
};

__device__ __forceinline__ void coords(long long r, int lx, int ly, int &x, int &y, int &z)
{
    const unsigned nd = (unsigned)r;
    x = (int)(nd % (unsigned)lx);
    const unsigned yz = nd / (unsigned)lx;
    y = (int)(yz % (unsigned)ly);
    z = (int)(yz / (unsigned)ly);
}

// offset of (x + dx, y + dy, z + dz), periodic, dx.. in {-1,0,1}
__device__ __forceinline__ long long nb(int x, int y, int z, int dx, int dy, int dz, int lx, int ly, int lz)
{
    const int xx = dx > 0 ? wrap_plus(x, lx) : (dx < 0 ? wrap_minus(x, lx) : x);
    const int yy = dy > 0 ? wrap_plus(y, ly) : (dy < 0 ? wrap_minus(y, ly) : y);
    const int zz = dz > 0 ? wrap_plus(z, lz) : (dz < 0 ? wrap_minus(z, lz) : z);
    return xx + (long long)lx * (yy + (long long)ly * zz);
}

// Link flux of just_eq_smolu.f90:86-99 from site a (origin) to site b, from the sites' values.
__device__ __forceinline__ void link_flux_values(const PnpArgs &k, double phi_a, double cp_a, double cm_a, double phi_b,
                                                 double cp_b, double cm_b, double delta, double &Jp, double &Jm)
{
    const double e = exp(phi_b - phi_a);
    const double em = 1.0 / e;
    Jp = 0.5 * (1.0 + em) * (cp_b * e - cp_a);
    Jp = Jp * k.eDp / delta;
    Jm = 0.5 * (1.0 + e) * (cm_b * em - cm_a);
    Jm = Jm * k.eDm / delta;
}

// State of the resident loop between its launches.
struct PnpLoop {
    int iter, in_solve;      // sweeps of the solve under way (1: to be continued)
    int total;               // sum of the solves' sweep counts (iter - 1 each)
    int outer, equilibrium;  // outer iterations; the convergence test was met
    int converged, done;     // last solve converged; nothing left to do
    // The stopping value of a solve is a multiple of SUM(ABS(phi)) before it, which the reference adds up
    // in storage order.  Within a call the device's sum stands in for it, and where that could matter --
    // the residual as near the stopping value as the two sums may be -- the launch ends undecided and the
    // host, with the sum in storage order, decides for it.
    int limit_exact;         // the stopping value is of the sum in storage order
    int undecided, resume_conv;
    double limit, anormf0;   // stopping value of the solve under way, SUM(ABS(phi)) of the last one
    double residual, anorm;  // undecided: of the last sweep
    unsigned status;         // last: bits are added to it, the rest is stored by block 0
};

struct PnpResidentArgs {
    PnpArgs a;               // mask, N, sides, weights, factor, omega, eD, delta, loop_bug
    GridSync *sync;
    GridWait wait;
    PnpLoop *loop;
    double *phi, *cp, *cm;   // the state
    double *t0, *t1;         // w_axis phi by sweep parity
    double *bak[3];          // phi, c+, c- at the start of the outer iteration, between launches
    double *link;            // loop_bug: fluxes of the 9 lx links that start on the line, (J+, J-) each
    double *partial;         // pnp_resident_partials doubles
    double limit_factor;     // of anormf0
    int max_iter;            // sweeps per solve
    int max_outer;           // outer iterations, 0: one solve only
    int outer0;              // outer iterations before this launch
    int max_sweeps, outers_per_launch;
    double sigma, rho_ch, count_fluid;
};

}  // namespace lbg
