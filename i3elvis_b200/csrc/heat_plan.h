// heat_plan.h -- what one cycle of the heat solve does, from its coupling (plain C++, no CUDA).
//
// With q the ratio of a row's neighbour coefficients to its rho cp / dt, the Jacobi iteration matrix
// of level 0 has spectral radius mu <= q / (1 + q), and a red-black sweep with the damping factor w
// (t0koef) multiplies the error by the spectral radius of successive relaxation on a consistently
// ordered matrix (Young 1954): (w mu + sqrt(w^2 mu^2 - 4 (w - 1)))^2 / 4, or w - 1 where the root is
// imaginary; mu^2 for w = 1.
#pragma once
#include <algorithm>
#include <cmath>

namespace i3g {

// levels 0..last, two sweeps per leg and `sweeps` on the last
struct HeatPlan { int last, sweeps; };

constexpr int kHeatMaxSweeps = 16;

// The whole hierarchy, whatever the coupling.
inline HeatPlan heat_plan_full(int nlev) { return HeatPlan{nlev - 1, kHeatMaxSweeps}; }

// Error factor of one sweep; 1 where relaxation alone does not converge or q is not a number.
inline double heat_sweep_rate(double q, double w)
{
    if (!(q >= 0) || !(w > 0 && w < 2)) return 1.0;
    const double mu = std::isinf(q) ? 1.0 : q / (1.0 + q), b = w * mu, disc = b * b - 4.0 * (w - 1.0);
    if (disc < 0) return w - 1.0;
    const double s = 0.5 * (b + std::sqrt(disc));
    return std::min(1.0, s * s);
}

// sweeps that leave `left` of an error with coupling q; none of them would be enough: kHeatMaxSweeps
inline double heat_sweeps_for(double q, double w, double left)
{
    const double rate = heat_sweep_rate(q, w);
    return rate < 1.0 ? std::ceil(std::log(left) / std::log(std::max(1e-6, rate))) : kHeatMaxSweeps;
}

// What a solve's couplings ask for.  q[l]: of level l's cells without the outermost, which stay as
// narrow on every level as on level 0; qall[l] with them.  The last level used is the first one with q[l]
// <= 1 (or the coarsest).  Its sweeps reduce the error by 1e-3, or by the tolerance when it is level
// 0; at most 16, or 12 where coarser levels are left out, since the norm after a cycle costs as little
// there as one sweep.  A rate of 1 (rho cp / dt lost against the neighbour coefficients, or zero)
// takes all 16.  On a coarse level the narrow cells have to lose a quarter of their error too: with the
// few sweeps that the others ask for, a step of ten diffusion times on 65^3 stretched nodes and four
// coarse levels diverged, where 16 sweeps took 16 cycles.
// q comes from a bound on k / (rho cp) and the level's spacings (heat.cu, heat_coupling), so the plan
// is an estimate: a solve whose cycles fall behind it goes on with heat_plan_full.
inline HeatPlan heat_plan(const double *q, const double *qall, int nlev, double w, double rtol)
{
    HeatPlan P = heat_plan_full(nlev);
    int l = 0;
    while (l < nlev - 1 && !(q[l] <= 1.0)) l++;
    P.last = l;
    double need = heat_sweeps_for(q[l], w, l == 0 ? rtol : 1e-3);
    if (l > 0) need = std::max(need, heat_sweeps_for(qall[l], w, 0.75));
    const double most = l == 0 && nlev > 1 && q[0] <= 1.0 && heat_sweep_rate(q[0], w) < 1.0 ? 12.0 : kHeatMaxSweeps;
    P.sweeps = (int)std::min(most, std::max(2.0, need));
    return P;
}

// A solve goes on with the whole hierarchy when a cycle leaves more of the residual than this.  V-cycles
// leave 0.05 to 0.15 of it on uniform grids and up to 0.35 on stretched ones, where the whole hierarchy
// takes as many cycles of more sweeps: with 0.3 here a step of ten diffusion times on 65^3 stretched
// nodes took 4.9 ms instead of 4.4 (B200).
constexpr double kHeatPlanFactor = 0.5;

}  // namespace i3g
