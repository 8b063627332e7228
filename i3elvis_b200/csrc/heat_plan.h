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

// The last level used is the first one with coupling q[l] <= 1 (or the coarsest).  Its sweeps reduce
// the error by 1e-3, or by the tolerance when it is level 0; at most 16, or 12 where level 0 alone is
// weakly coupled, since the norm after a cycle costs as little there as one sweep.  A rate of 1 (rho
// cp / dt lost against the neighbour coefficients, or zero) takes all 16.
// q comes from a bound on k / (rho cp) and the level's spacings (heat.cu, heat_coupling), so the plan
// is an estimate: a solve whose cycles fall behind it goes on with heat_plan_full.
inline HeatPlan heat_plan(const double *q, int nlev, double w, double rtol)
{
    HeatPlan P = heat_plan_full(nlev);
    int l = 0;
    while (l < nlev - 1 && !(q[l] <= 1.0)) l++;
    P.last = l;
    const double rate = heat_sweep_rate(q[l], w);
    if (!(rate < 1.0)) return P;
    const double need = std::log(l == 0 ? rtol : 1e-3) / std::log(std::max(1e-6, rate));
    const double most = l == 0 && q[0] <= 1.0 ? 12.0 : kHeatMaxSweeps;
    P.sweeps = (int)std::min(most, std::max(2.0, std::ceil(need)));
    return P;
}

// A cycle of a plan that holds reduces the residual at least this much (a V-cycle of the full
// hierarchy: to 0.05 .. 0.15 of it).
constexpr double kHeatPlanFactor = 0.3;

}  // namespace i3g
