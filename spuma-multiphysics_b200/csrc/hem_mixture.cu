// Multi-species HEM UV flash on the device: a Peng-Robinson gas mixture of up
// to four species with up to two pure condensed liquids (the air / N2O /
// isopropanol model of the reference's production case). The independent
// evaluations of a cell's search (the two sides of every Jacobian column, a line
// search's trial fractions, the seeds) run on different lanes of a warp.
//
// The search restates the reference device flash
// (src/reactiveThermo/reactiveDeviceFlash.h) for models without solids, with its
// bounded finite-difference Newton Jacobian (an image's analyticJacobian flag
// selects the reference's analytic active-set Jacobian there, which is not
// restated: such images run on the finite differences and converge to the same
// solutions within the Newton tolerances), including its capillary form
// (recoverCapillary, :572-588: the phases at their own pressures across a fixed
// jump, the boundary search in every equilibrium batch, the frozen partition):
//   * phase sums of one evaluation at (p, T) with given liquid masses, the gas
//     phase from the remaining species and, on request, virtual liquids for the
//     chemical potentials (evaluate, :210-262);
//   * the all-gas partition: the scalar T-Newton at fixed density, else the
//     frozen (ln p, ln T) Newton with its halving line search (:264-326);
//   * the active-set Newton in (ln p, ln T, liquid fractions) or, in the
//     boundary recovery, (ln p, ln T, log vapour fractions), with the residual of
//     the volume, the scaled energy and each active liquid's chemical-potential
//     difference, the bounded central-difference Jacobian, the limiter, the
//     30-fraction line search with its coordinate rejection prefix, and the
//     equilibrium sound check (:327-448);
//   * the stability test: affinities against virtual liquids when gas is
//     present, the tangent plane of the liquid species otherwise (a 33-point scan
//     and 55 golden-section steps for two liquids) (:449-480);
//   * the candidate order, the seeds {previous, .5, .95, .1, .9999}, the first
//     maximum entropy among stable candidates, the restart temperatures at
//     {.02, .25, .5, .75} of the legal liquid interval, the optional
//     stableGasPrune policy, and the boundary recovery around nearly liquid cells
//     (:486-560, src/reactiveThermo/reactiveFlashSeeds.h:14-16).
// Phase properties come from the mixture evaluator of pr_mixture.cuh (pinned to
// the reference's evaluator). Every loop is bounded.
// One copy of each evaluator routine, loops rolled: a warp's tasks are seldom at the same
// instruction, so the searches are bound by instruction fetch (see mixture_residual.cuh).
#define RB200_MIX_FN static __noinline__
#define RB200_MIX_LOOP _Pragma("unroll 1")
#include "hem_mixture.h"
#include "pr_mixture.cuh"
#include "mixture_residual.cuh"
#include "common.cuh"

#include <algorithm>
#include <chrono>
#include <cstring>
#include <memory>
#include <type_traits>
#include <vector>

namespace rb200 {
namespace {

constexpr double kRu = 8314.46261815324;
constexpr int kNs = mix::kMaxNs;
constexpr int kLiq = 2;
constexpr int kBlock = 64;

// Phase sums of one evaluation (the state plus the derivatives the Newton
// iterations and the stability test use).
struct MixEval {
    ReactiveThermoState s;
    double volume, energy, entropyD, Vp, VT, Ep, ET, cpD;
    double muGas[kLiq], muLiq[kLiq], gasCond[kLiq];
    bool explicitGas;
};

struct Tally {
    unsigned long long phases = 0, residuals = 0, candidates = 0, stable = 0, failures = 0, fd = 0;
};

// One cell's recovery: its inputs, the search mode and, for a capillary batch,
// the interface color and the pressure jump sigma*kappa held fixed during the
// solve (src/reactiveThermo/reactiveDeviceFlash.h:146-153): the gas phase is
// evaluated at p - color*jump and the liquids at p + (1 - color)*jump, p the
// volume-averaged mechanical pressure.
struct MixCell {
    const ReactiveB200HemModel& m;
    double q[kNs];
    double energy;
    ReactiveThermoState guess;
    bool adaptive;
    Tally& n;
    double color = 0, jump = 0;
    // the reported-phase lines of the last gas composition and of the pure liquids:
    // forming one takes a mixing and a cubic solve at least, as much as the
    // evaluation it labels
    mix::PhaseLine gasLine{}, liquidLine[kLiq]{};
};

__device__ __forceinline__ bool fin(double x) { return x == x && fabs(x) <= 1.79769313486231570815e308; }
__device__ __forceinline__ double clampd(double a, double l, double h) { return fmin(fmax(a, l), h); }
__device__ __forceinline__ double maxAbs(const double* a, int n) {
    double r = 0;
    for (int i = 0; i < n; ++i) r = fmax(r, fabs(a[i]));
    return r;
}
__device__ __forceinline__ bool unavailable(int status) { return status == mix::UNAVAILABLE || status == mix::NO_ROOT; }

__device__ __forceinline__ double density(const MixCell& c) {
    double r = 0;
    for (int k = 0; k < c.m.ns; ++k) r += c.q[k];
    return r;
}
__device__ __forceinline__ bool inBounds(const ReactiveB200HemModel& m, double p, double T) {
    return fin(p) && fin(T) && p >= m.pmin && p <= m.pmax && T >= m.Tmin && T <= m.Tmax;
}
__device__ __forceinline__ bool isCondensable(const ReactiveB200HemModel& m, int k) {
    for (int i = 0; i < m.nl; ++i)
        if (m.condensable[i] == k) return true;
    return false;
}
__device__ __forceinline__ double energyScale(const MixEval& v) { return fmax(1e5 * v.s.rho, v.cpD * v.s.T); }
__device__ __forceinline__ double gasPressure(const MixCell& c, double p) { return p - c.color * c.jump; }
__device__ __forceinline__ double liquidPressure(const MixCell& c, double p) { return p + (1 - c.color) * c.jump; }

// The gas mixture at (p, T, Y) on its gas root; species outside their NASA
// range invalidate the state when the model enforces the ranges.
__device__ __noinline__ int gasPhase(MixCell& c, double p, double T, const double* Y, bool chem, mix::Props& out) {
    ++c.n.phases;
    if (!inBounds(c.m, p, T)) return mix::BAD_INPUT;
    if (c.m.enforceSpeciesTemperatureBounds)
        for (int k = 0; k < c.m.ns; ++k)
            if (Y[k] > 0) {
                const ReactiveB200Species& sp = c.m.phase[0].species[k];
                if (T < sp.regions[0].minimumTemperature || T > sp.regions[sp.regionCount - 1].maximumTemperature)
                    return mix::BAD_INPUT;
            }
    return mix::tp(c.m.phase[0], T, p, Y, mix::GAS, chem, out, &c.gasLine);
}

// The pure liquid of condensed phase i at (p, T) on its liquid root.
__device__ __noinline__ int liquidPhase(MixCell& c, int i, double p, double T, bool chem, mix::Props& out) {
    ++c.n.phases;
    if (!inBounds(c.m, p, T)) return mix::BAD_INPUT;
    if (T < c.m.liquidTmin[i]) return mix::BAD_INPUT;
    if (T >= c.m.liquidTc[i] * (1 - 1e-10)) return mix::UNAVAILABLE;
    const double pure[kNs] = {1, 0, 0, 0};
    return mix::tp(c.m.phase[i + 1], T, p, pure, mix::LIQUID, chem, out, &c.liquidLine[i]);
}

__device__ __forceinline__ void addPhase(MixEval& v, double mass, const mix::Props& p, double pressure) {
    const double volume = mass / p.rho, vp = -volume * p.kappaT, vt = volume * p.alpha;
    v.volume += volume;
    v.energy += mass * p.e;
    v.entropyD += mass * p.s;
    v.Vp += vp;
    v.VT += vt;
    v.Ep += -v.s.T * vt - pressure * vp;
    v.ET += mass * p.cp - pressure * vt;
    v.cpD += mass * p.cp;
}

// Phase sums at (p, T) with liquid masses `mass`; `vapor` (the boundary
// recovery) gives each condensable's gas amount explicitly; `virt` also
// evaluates absent liquids for the chemical potentials.
__device__ __noinline__ bool evaluate(MixCell& c, const double* mass, double p, double T, MixEval& v, bool virt,
                                      const double* vapor) {
    const ReactiveB200HemModel& m = c.m;
    v = MixEval{};
    if (!inBounds(m, p, T)) return false;
    ReactiveThermoState& s = v.s;
    s.p = p;
    s.T = T;
    s.rho = density(c);
    if (!(s.rho > 0)) return false;
    double gas[kNs] = {0, 0, 0, 0};
    for (int k = 0; k < m.ns; ++k) {
        if (!fin(c.q[k]) || c.q[k] < 0) return false;
        gas[k] = c.q[k];
    }
    for (int i = 0; i < m.nl; ++i) {
        const int k = m.condensable[i];
        if (!fin(mass[i]) || mass[i] < 0 || mass[i] > c.q[k]) return false;
        gas[k] = vapor ? vapor[i] : gas[k] - mass[i];
        if (!fin(gas[k]) || gas[k] < 0 || gas[k] > c.q[k]) return false;
    }
    for (int i = 0; i < m.nl; ++i) v.gasCond[i] = gas[m.condensable[i]];
    v.explicitGas = vapor != nullptr;
    double mg = 0;
    for (int k = 0; k < m.ns; ++k) mg += gas[k];
    s.gasMass = mg;
    const double pg = gasPressure(c, p), pl = liquidPressure(c, p);
    if (mg > 0) {
        for (int k = 0; k < m.ns; ++k) gas[k] /= mg;
        mix::Props prop;
        if (gasPhase(c, pg, T, gas, virt, prop) != mix::OK) return false;
        addPhase(v, mg, prop, pg);
        s.alphaGas = mg / prop.rho;
        s.rhoGas = prop.rho;
        if (virt)
            for (int i = 0; i < m.nl; ++i) v.muGas[i] = prop.mu[m.condensable[i]] / (kRu * T);
    }
    for (int i = 0; i < m.nl; ++i) {
        s.liquidMass[i] = mass[i];
        if (!(mass[i] > 0 || (virt && c.q[m.condensable[i]] > 0))) continue;
        mix::Props prop;
        const int status = liquidPhase(c, i, pl, T, virt, prop);
        if (status != mix::OK) {
            if (mass[i] > 0 || !unavailable(status)) return false;
            v.muLiq[i] = HUGE_VAL;
            continue;
        }
        if (virt) v.muLiq[i] = prop.mu[0] / (kRu * T);
        if (mass[i] > 0) {
            addPhase(v, mass[i], prop, pl);
            s.rhoLiquid[i] = prop.rho;
            s.alphaLiquid[i] = mass[i] / prop.rho;
            s.activeLiquids |= 1 << i;
        }
    }
    s.e = v.energy / s.rho;
    s.entropy = v.entropyD / s.rho;
    s.cp = v.cpD / s.rho;
    s.cv = (v.cpD + T * v.VT * v.VT / v.Vp) / s.rho;
    if (!fin(s.cv) || s.cv <= 0) return false;
    const double specific = v.volume / s.rho, vp = v.Vp / s.rho, vt = v.VT / s.rho;
    const double adiabatic = vp + T * vt * vt / s.cp;
    if (!(adiabatic < 0)) return false;
    s.soundFrozen = sqrt(-specific * specific / adiabatic);
    s.soundEquilibrium = s.soundFrozen;
    return fin(s.soundFrozen) && s.soundFrozen > 0;
}

// Dense solve with full pivoting (pivot search column by column, rows inside
// each column, first strict maximum) and the rank test pivot > largest * n * eps.
__device__ __noinline__ bool solveDense(const double a0[4][4], const double* rhs, int n, double* x) {
    double a[4][4], b[4], largest = 0;
    int column[4] = {0, 1, 2, 3};
    for (int i = 0; i < n; ++i) {
        b[i] = rhs[i];
        if (!fin(b[i])) return false;
        for (int j = 0; j < n; ++j) {
            a[i][j] = a0[i][j];
            if (!fin(a[i][j])) return false;
        }
    }
    for (int k = 0; k < n; ++k) {
        int row = k, col = k;
        double pivot = 0;
        for (int j = k; j < n; ++j)
            for (int i = k; i < n; ++i)
                if (fabs(a[i][j]) > pivot) { pivot = fabs(a[i][j]); row = i; col = j; }
        largest = fmax(largest, pivot);
        if (!(pivot > largest * n * 2.220446049250313e-16)) return false;
        if (row != k) {
            for (int j = 0; j < n; ++j) { const double t = a[k][j]; a[k][j] = a[row][j]; a[row][j] = t; }
            const double t = b[k]; b[k] = b[row]; b[row] = t;
        }
        if (col != k) {
            for (int i = 0; i < n; ++i) { const double t = a[i][k]; a[i][k] = a[i][col]; a[i][col] = t; }
            const int t = column[k]; column[k] = column[col]; column[col] = t;
        }
        for (int i = k + 1; i < n; ++i) {
            const double f = a[i][k] / a[k][k];
            a[i][k] = f;
            for (int j = k + 1; j < n; ++j) a[i][j] -= f * a[k][j];
            b[i] -= f * b[k];
        }
    }
    double z[4] = {0, 0, 0, 0};
    for (int i = n - 1; i >= 0; --i) {
        double v = b[i];
        for (int j = i + 1; j < n; ++j) v -= a[i][j] * z[j];
        z[i] = v / a[i][i];
        if (!fin(z[i])) return false;
    }
    for (int i = 0; i < n; ++i) x[column[i]] = z[i];
    return true;
}

// The scalar all-gas energy residual at (T, rho): properties at (T, rho), then
// the gas root at the resulting pressure must be that density. p is the
// mechanical pressure, the gas's plus color*jump.
__device__ __noinline__ bool gasProbe(MixCell& c, double T, double& F, double& cv, double& p, double* cp) {
    const double rho = density(c);
    double Y[kNs] = {0, 0, 0, 0};
    for (int k = 0; k < c.m.ns; ++k) Y[k] = c.q[k] / rho;
    ++c.n.phases;
    mix::Props prop;
    if (mix::trho(c.m.phase[0], T, rho, Y, false, prop, &c.gasLine) != mix::OK) return false;
    const double gasP = prop.p;
    p = gasP + c.color * c.jump;
    if (!inBounds(c.m, p, T)) return false;
    mix::Props gas;
    if (gasPhase(c, gasP, T, Y, false, gas) != mix::OK || fabs(gas.rho - rho) > 1e-8 * rho) return false;
    F = rho * prop.e - c.energy;
    cv = rho * prop.cv;
    if (cp) *cp = prop.cp;
    return fin(F) && fin(cv) && cv > 0;
}

__device__ __noinline__ bool scalarGas(MixCell& c, MixEval& result) {
    const ReactiveB200HemModel& m = c.m;
    const double rho = density(c);
    double T = clampd(c.guess.T, m.Tmin, m.Tmax), F, cv, p, cp;
    if (!gasProbe(c, T, F, cv, p, &cp)) return false;
    const double tol = m.etol * fmax(1e5 * rho, rho * cp * T);
    double lower = T, upper = T, fl = F, fh = F;
    if (fabs(F) > tol) {
        double radius = fmax(1., .01 * T);
        for (int j = 0; j < 24 && (fl > 0 || fh < 0); ++j, radius *= 2) {
            if (fl > 0) {
                double probe = fmax(m.Tmin, T - radius), value, dCv, dP;
                bool found = false;
                for (int retry = 0; retry < 8 && !found; ++retry) {
                    if (gasProbe(c, probe, value, dCv, dP, nullptr)) { fl = value; lower = probe; found = true; }
                    else probe = .5 * (lower + probe);
                }
                if (!found) return false;
            }
            if (fh < 0) {
                double probe = fmin(m.Tmax, T + radius), value, dCv, dP;
                bool found = false;
                for (int retry = 0; retry < 8 && !found; ++retry) {
                    if (gasProbe(c, probe, value, dCv, dP, nullptr)) { fh = value; upper = probe; found = true; }
                    else probe = .5 * (upper + probe);
                }
                if (!found) return false;
            }
            if (fabs(fl) <= tol) { T = lower; if (!gasProbe(c, T, F, cv, p, nullptr)) return false; break; }
            if (fabs(fh) <= tol) { T = upper; if (!gasProbe(c, T, F, cv, p, nullptr)) return false; break; }
            if (lower == m.Tmin && upper == m.Tmax) break;
        }
        if (!(fabs(F) <= tol || (fl <= 0 && fh >= 0 && upper > lower))) return false;
    }
    int it = 0;
    for (; it < 70 && fabs(F) > tol; ++it) {
        if (F > 0) upper = T; else lower = T;
        const double next = T - F / cv;
        T = fin(next) && next > lower && next < upper ? next : .5 * (lower + upper);
        if (!gasProbe(c, T, F, cv, p, nullptr)) return false;
    }
    if (fabs(F) > tol) return false;
    const double zero[kLiq] = {0, 0};
    if (!evaluate(c, zero, p, T, result, false, nullptr)) return false;
    result.s.volumeResidual = fabs(result.volume - 1);
    result.s.energyResidual = fabs(result.energy - c.energy) / energyScale(result);
    result.s.iterations = it;
    return result.s.volumeResidual <= m.vtol && result.s.energyResidual <= m.etol;
}

// Residual of an active set at x = (ln p, ln T, fractions): liquid fractions in
// [0, 1) or, in the boundary recovery, log vapour fractions <= 0.
__device__ __noinline__ bool activeResidual(MixCell& c, const int* active, int n, const double* x, double scale,
                                            double* f, MixEval& v) {
    ++c.n.residuals;
    const ReactiveB200HemModel& m = c.m;
    double mass[kLiq] = {0, 0}, vapor[kLiq] = {0, 0};
    for (int i = 0; i < m.nl; ++i) vapor[i] = c.q[m.condensable[i]];
    for (int j = 0; j < n; ++j) {
        const int i = active[j];
        const double q = c.q[m.condensable[i]];
        if (c.adaptive) {
            if (!fin(x[j + 2]) || x[j + 2] > 0) return false;
            vapor[i] = exp(x[j + 2]) * q;
            if (!(vapor[i] > 0)) return false;
            mass[i] = -expm1(x[j + 2]) * q;
        } else {
            if (!(x[j + 2] >= 0 && x[j + 2] < 1)) return false;
            mass[i] = x[j + 2] * q;
        }
    }
    if (!evaluate(c, mass, exp(x[0]), exp(x[1]), v, true, c.adaptive ? vapor : nullptr) || !(v.s.gasMass > 0))
        return false;
    f[0] = v.volume - 1;
    f[1] = (v.energy - c.energy) / scale;
    for (int j = 0; j < n; ++j) {
        f[2 + j] = v.muLiq[active[j]] - v.muGas[active[j]];
        if (!fin(f[2 + j])) return false;
    }
    return true;
}

__device__ __forceinline__ bool rejectedCoordinate(bool adaptive, double y) {
    return adaptive ? (!fin(y) || y > 0) : !(y >= 0 && y < 1);
}

// Gibbs energy of the gas mixture of the present liquids' species at mole
// fractions (fraction, 1 - fraction), less the liquids' chemical potentials:
// the tangent-plane distance (HUGE_VAL where the gas phase does not exist).
__device__ __noinline__ double tangent(MixCell& c, double p, double T, const int* present, int n, const double* mu,
                                       double fraction) {
    const ReactiveB200HemModel& m = c.m;
    double mole[kNs] = {0, 0, 0, 0}, Y[kNs] = {0, 0, 0, 0}, sum = 0;
    mole[m.condensable[present[0]]] = n == 1 ? 1 : fraction;
    if (n == 2) mole[m.condensable[present[1]]] = 1 - fraction;
    for (int k = 0; k < m.ns; ++k) { Y[k] = mole[k] * m.weights[k]; sum += Y[k]; }
    for (int k = 0; k < m.ns; ++k) Y[k] /= sum;
    mix::Props prop;
    const int status = gasPhase(c, gasPressure(c, p), T, Y, false, prop);
    if (status != mix::OK) return unavailable(status) ? HUGE_VAL : nan("");
    double reference = 0, W = 0;
    for (int i = 0; i < n; ++i) reference += mole[m.condensable[present[i]]] * mu[present[i]];
    for (int k = 0; k < m.ns; ++k) W += mole[k] * m.weights[k];
    return (prop.h - T * prop.s) * W / (kRu * T) - reference;
}

__device__ __noinline__ bool stableCandidate(MixCell& c, const MixEval& v) {
    const ReactiveB200HemModel& m = c.m;
    const double p = v.s.p, T = v.s.T;
    if (v.s.gasMass > 0) {
        const double mass[kLiq] = {v.s.liquidMass[0], v.s.liquidMass[1]};
        MixEval cmp;
        if (!evaluate(c, mass, p, T, cmp, true, v.explicitGas ? v.gasCond : nullptr)) return false;
        for (int i = 0; i < m.nl; ++i) {
            if (c.q[m.condensable[i]] == 0) continue;
            const double affinity = cmp.muLiq[i] - cmp.muGas[i];
            if (mass[i] > 0) {
                if (!fin(affinity) || fabs(affinity) > m.mutol * 2) return false;
            } else if (affinity < -m.mutol) return false;
        }
        return true;
    }
    int present[kLiq] = {0, 0}, np = 0;
    double mu[kLiq] = {0, 0};
    for (int i = 0; i < m.nl; ++i)
        if (v.s.liquidMass[i] > 0) {
            present[np++] = i;
            mix::Props prop;
            if (liquidPhase(c, i, liquidPressure(c, p), T, true, prop) != mix::OK) return false;
            mu[i] = prop.mu[0] / (kRu * T);
        }
    if (!np) return false;
    if (np == 1) return tangent(c, p, T, present, 1, mu, 1) >= -m.mutol;
    double best = HUGE_VAL;
    int location = 0;
    for (int j = 0; j <= 32; ++j) {
        const double t = tangent(c, p, T, present, np, mu, double(j) / 32);
        if (t != t) return false;
        if (t < best) { best = t; location = j; }
    }
    double left = fmax(0., double(location - 1) / 32), right = fmin(1., double(location + 1) / 32);
    for (int j = 0; j < 55; ++j) {
        const double a = left + (right - left) * .38196601125, b = left + (right - left) * .61803398875;
        const double ta = tangent(c, p, T, present, np, mu, a), tb = tangent(c, p, T, present, np, mu, b);
        if (ta != ta || tb != tb) return false;
        best = fmin(best, fmin(ta, tb));
        if (ta < tb) right = b; else left = a;
    }
    return best >= -m.mutol;
}

__device__ __forceinline__ bool prunable(const ReactiveB200HemModel& m) {
    return m.nl == 1 && m.condensedKind[0] == 0 && m.condensedKind[1] == 0;
}

// A candidate of the search: its state, entropy density and status (kInvalid: the
// cell's inputs are rejected; kNone: not converged).
enum : int { kInvalid = -1, kNone = 0, kUnstable = 1, kStable = 2 };
struct MixRecord {
    ReactiveThermoState s;
    double entropyD;
    int status, pad;
};

// Per-cell fixed-partition candidates, in the order they enter the selection: the
// all-gas one, the all-liquid one (cells without non-condensable gas) and, for
// models with stableGasPrune, the all-gas one without that policy's stall limit,
// which the boundary recovery's second search takes.
enum : int { kGasRecord = 0, kLiquidRecord = 1, kFullGasRecord = 2, kRecordKinds = 3 };

// One batch's device arrays. `order` (optional) names the cells: item i works on
// cell order[i], and every per-cell input is indexed by that cell; the records,
// the work list and its counters belong to the handle and are indexed by item.
struct MixBatch {
    const ReactiveB200HemModel* model;
    const MixTerms* terms;
    const double* q;
    const double* energy;
    size_t count;
    const ReactiveThermoState* seed;
    const ReactiveGpuHemCapillaryInputV2* capillary;
    const uint32_t* order;
    MixRecord* record[kRecordKinds];  // kFullGasRecord: null unless the model prunes
    unsigned* list;                   // Newton items: item * kRecordKinds + kind
    unsigned* counters;               // C_*
    unsigned long long* totals;
    ReactiveThermoState* out;
    int* success;
    ReactiveGpuHemOutputV1* outputs;
};
enum : int { C_LISTED, C_NEWTON, C_SEARCH, C_COUNT };

enum : int { M_PHASES, M_RESIDUALS, M_CANDIDATES, M_STABLE, M_FD, M_SUCCEEDED, M_COUNT };

__device__ __forceinline__ void flushTally(const Tally& n, unsigned long long* totals) {
    const unsigned long long v[5] = {n.phases, n.residuals, n.candidates, n.stable, n.fd};
    const int slot[5] = {M_PHASES, M_RESIDUALS, M_CANDIDATES, M_STABLE, M_FD};
    for (int i = 0; i < 5; ++i) {
        unsigned long long x = v[i];
        for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0 && x) atomicAdd(totals + slot[i], x);
    }
}

// A capillary cell input the reference's recoverCapillary accepts
// (src/reactiveThermo/reactiveDeviceFlash.h:572-588): a color in [0, 1], a
// finite jump, and a nonzero jump only with one pure liquid.
__device__ __forceinline__ bool capillaryAccepted(const ReactiveB200HemModel& m, double color, double jump) {
    return fin(color) && color >= 0 && color <= 1 && fin(jump) && (jump == 0 || (m.nl == 1 && m.condensedKind[0] == 0));
}

__device__ __forceinline__ void loadCell(const MixBatch& b, size_t item, MixCell& c) {
    const size_t cell = b.order ? size_t(b.order[item]) : item;
    for (int k = 0; k < kNs; ++k) c.q[k] = k < c.m.ns ? b.q[cell * size_t(c.m.ns) + k] : 0.0;
    c.energy = b.energy[cell];
    c.guess = b.seed[cell];
    c.color = b.capillary ? b.capillary[cell].color : 0.0;
    c.jump = b.capillary ? b.capillary[cell].pressureJump : 0.0;
    c.adaptive = false;
}
// A capillary item with the partition frozen at the seed's liquid masses.
__device__ __forceinline__ bool frozenItem(const MixBatch& b, size_t item) {
    return b.capillary && !b.capillary[b.order ? size_t(b.order[item]) : item].equilibrium;
}

__device__ __forceinline__ void storeRecord(MixRecord& r, const MixEval& v, int status) {
    r.s = v.s;
    r.entropyD = v.entropyD;
    r.status = status;
}

// The fixed-partition candidates' first part, one thread per item: the input
// checks, the scalar all-gas solve with its stability test, and the list of the
// partitions that need the (ln p, ln T) Newton.
__global__ void __launch_bounds__(kBlock) mixtureScalar(MixBatch b) {
    const ReactiveB200HemModel& m = *b.model;
    Tally n;
    MixCell c{m, {0, 0, 0, 0}, 0.0, ReactiveThermoState{}, false, n};
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < b.count; i += size_t(blockDim.x) * gridDim.x) {
        loadCell(b, i, c);
        const bool frozen = frozenItem(b, i);
        bool valid = !b.capillary || capillaryAccepted(m, c.color, c.jump);
        if (valid && !frozen) {
            valid = m.ns > 0 && m.ns <= kNs && m.nl >= 0 && m.nl <= kLiq && fin(c.energy) && density(c) > 0;
            for (int k = 0; k < m.ns && valid; ++k) valid = fin(c.q[k]) && c.q[k] >= 0;
        }
        b.record[kLiquidRecord][i].status = kNone;
        if (b.record[kFullGasRecord]) b.record[kFullGasRecord][i].status = kNone;
        MixRecord& gas = b.record[kGasRecord][i];
        gas.status = valid ? kNone : kInvalid;
        if (!valid || !fin(c.energy)) continue;
        const double mass0 = frozen ? c.guess.liquidMass[0] : 0.0, mass1 = frozen ? c.guess.liquidMass[1] : 0.0;
        MixEval v;
        if (m.scalarRecovery && mass0 == 0 && mass1 == 0 && scalarGas(c, v)) {
            const int status = frozen || stableCandidate(c, v) ? kStable : kUnstable;
            n.stable += !frozen && status == kStable;
            storeRecord(gas, v, status);
            if (b.record[kFullGasRecord]) storeRecord(b.record[kFullGasRecord][i], v, status);
        } else {
            b.list[atomicAdd(b.counters + C_LISTED, 1u)] = unsigned(i) * kRecordKinds + kGasRecord;
            if (!frozen && b.record[kFullGasRecord])
                b.list[atomicAdd(b.counters + C_LISTED, 1u)] = unsigned(i) * kRecordKinds + kFullGasRecord;
        }
        if (!frozen && m.nl) {
            double other = 0;
            for (int k = 0; k < m.ns; ++k)
                if (!isCondensable(m, k)) other += c.q[k];
            if (other == 0) b.list[atomicAdd(b.counters + C_LISTED, 1u)] = unsigned(i) * kRecordKinds + kLiquidRecord;
        }
    }
    __syncwarp();
    flushTally(n, b.totals);
}

// The frozen partitions (fixed liquid masses) the scalar solve left: Newton in
// (ln p, ln T) with the (0.7, 0.2) limiter and a halving line search; a stall limit
// ends the solve as a failure after that many consecutive steps accepted below a
// fraction of 1/32.
//
// Eight lanes per item: they evaluate eight consecutive fractions of a line search
// at once and the first acceptable one is taken, the fraction a serial search
// stops at. A partition that has no solution (a cold cell's all-gas one) halves
// deep in most of its 70 steps; serially one such cell's chain of evaluations,
// each of a few thousand dependent FP64 instructions, outlasted the batch.
constexpr int kNewtonLanes = 8;
constexpr int kSearchBlock = 128;
constexpr int kTrials = 30;  // fractions 1 .. 2^-29

__global__ void __launch_bounds__(kSearchBlock) mixtureNewton(MixBatch b) {
    const ReactiveB200HemModel& m = *b.model;
    const unsigned lane = threadIdx.x & 31u;
    const int base = int(lane) / kNewtonLanes * kNewtonLanes, r = int(lane) - base;
    const unsigned group = ((1u << kNewtonLanes) - 1u) << base;
    const unsigned total = b.counters[C_LISTED];
    Tally n;
    MixCell c{m, {0, 0, 0, 0}, 0.0, ReactiveThermoState{}, false, n};
    MixEval v;
    MixRecord* record = nullptr;
    double mass[kLiq] = {0, 0};
    bool active = false, exhausted = false, first = false, frozen = false;
    int stallLimit = 0, stalled = 0, it = 0, k = 0;
    double p = 0, T = 0, s0 = 0, s1 = 0, previous = 0, scale = 0;
    for (;;) {
        if (!active && !exhausted) {
            unsigned slot = 0;
            if (r == 0) slot = atomicAdd(b.counters + C_NEWTON, 1u);
            slot = __shfl_sync(group, slot, base);
            if (slot < total) {
                const unsigned entry = b.list[slot], item = entry / kRecordKinds;
                const int kind = int(entry % kRecordKinds);
                loadCell(b, item, c);
                frozen = frozenItem(b, item);
                record = b.record[kind] + item;
                for (int i = 0; i < kLiq; ++i)
                    mass[i] = frozen ? c.guess.liquidMass[i]
                                     : (kind == kLiquidRecord && i < m.nl ? c.q[m.condensable[i]] : 0.0);
                stallLimit = !frozen && kind == kGasRecord && m.stableGasPrune && prunable(m) ? 4 : 0;
                p = clampd(c.guess.p, m.pmin, m.pmax);
                T = clampd(c.guess.T, m.Tmin, m.Tmax);
                active = first = true;
                stalled = it = k = 0;
            } else exhausted = true;
        }
        __syncwarp();
        if (__all_sync(0xffffffffu, !active)) break;
        // every lane's evaluation at one call site
        double pe = p, te = T, fraction = 1;
        bool point = active && (first ? r == 0 : k + r < kTrials);
        if (active && !first) {
            fraction = ldexp(1.0, -(k + r));
            pe = p * exp(fraction * s0);
            te = T * exp(fraction * s1);
        }
        bool ok = false;
        if (point) ok = evaluate(c, mass, pe, te, v, false, nullptr);
        __syncwarp();
        if (!active) continue;
        if (!first && ok) {
            const double next = fmax(fabs(v.volume - 1), fabs(v.energy - c.energy) / scale);
            ok = next < previous * (1 - 1e-4 * fraction) || next < fmin(m.vtol, m.etol);
        }
        const unsigned accepted = __ballot_sync(group, ok);
        if (!accepted) {
            k += kNewtonLanes;
            if (first || k >= kTrials) active = false;  // the record stays kNone
            continue;
        }
        const int owner = __ffs(accepted) - 1;
        if (!first) {
            p = __shfl_sync(group, pe, owner);
            T = __shfl_sync(group, te, owner);
            stalled = k + owner - base > 5 ? stalled + 1 : 0;
            ++it;
        }
        // the owner of the accepted evaluation forms the next step
        int code = 0;  // 1 converged, -1 failed
        if (int(lane) == owner) {
            scale = energyScale(v);
            const double rv = v.volume - 1, re = (v.energy - c.energy) / scale;
            const bool within = fabs(rv) <= m.vtol && fabs(re) <= m.etol;
            if (stallLimit > 0 && stalled >= stallLimit
                && !(fabs(rv) <= m.vtol && fabs(v.energy - c.energy) / scale <= m.etol))
                code = -1;
            else if (it >= 70) code = -1;
            else if (within) {
                v.s.volumeResidual = fabs(rv);
                v.s.energyResidual = fabs(re);
                v.s.iterations = it;
                const int status = frozen || stableCandidate(c, v) ? kStable : kUnstable;
                n.stable += !frozen && status == kStable;
                storeRecord(*record, v, status);
                code = 1;
            } else {
                double jac[4][4] = {}, rhs[4] = {-rv, -re, 0, 0}, step[4] = {};
                jac[0][0] = v.Vp * p; jac[0][1] = v.VT * T;
                jac[1][0] = v.Ep * p / scale; jac[1][1] = v.ET * T / scale;
                if (!solveDense(jac, rhs, 2, step)) code = -1;
                const double limit = fmax(1., fmax(fabs(step[0]) / .7, fabs(step[1]) / .2));
                s0 = step[0] / limit;
                s1 = step[1] / limit;
                previous = fmax(fabs(rv), fabs(re));
            }
        }
        code = __shfl_sync(group, code, owner);
        scale = __shfl_sync(group, scale, owner);
        s0 = __shfl_sync(group, s0, owner);
        s1 = __shfl_sync(group, s1, owner);
        previous = __shfl_sync(group, previous, owner);
        first = false;
        k = 0;
        if (code) active = false;
    }
    flushTally(n, b.totals);
}

// The Newton candidates of one search: the active set, the fraction seed (< 0: the
// seed state's liquid fraction; -3 in the boundary recovery: a vapour fraction
// from the non-condensable inventory), the second liquid's seed (-2: the first's)
// and, in the restart search, the restart temperature (< 0: the seed state's).
struct MixTask {
    int active[kLiq], n;
    double seed, second, restartT;
};

// Task `index` of the search's task list in its selection order, false past its end:
// per active set (liquids present) the five seeds, in the boundary recovery the
// sixth and, with two liquids, their twelve unequal pairs; in the restart search
// the five seeds at each restart temperature of the set's legal interval.
__device__ __noinline__ bool nthTask(const MixCell& c, bool restarts, int index, MixTask& t) {
    const ReactiveB200HemModel& m = c.m;
    constexpr double seeds[5] = {-1, .5, .95, .1, .9999};
    constexpr double pairs[4] = {.1, .5, .95, .9999};
    constexpr double fractions[4] = {.02, .25, .5, .75};
    for (int mask = 1; mask < (1 << m.nl); ++mask) {
        bool possible = true;
        double lower = m.Tmin, upper = m.Tmax;
        t.n = 0;
        t.active[0] = t.active[1] = 0;
        for (int i = 0; i < m.nl; ++i)
            if (mask & (1 << i)) {
                if (c.q[m.condensable[i]] <= 0) possible = false;
                else {
                    t.active[t.n++] = i;
                    lower = fmax(lower, m.liquidTmin[i]);
                    upper = fmin(upper, m.liquidTc[i] * (1 - 1e-10));
                }
            }
        if (!possible || (restarts && !(upper > lower))) continue;
        const int tasks = restarts ? 20 : 5 + (c.adaptive ? (t.n == 2 ? 13 : 1) : 0);
        if (index >= tasks) {
            index -= tasks;
            continue;
        }
        t.second = -2;
        t.restartT = restarts ? lower + (upper - lower) * fractions[index / 5] : -1.0;
        if (restarts) t.seed = seeds[index % 5];
        else if (index < 5) t.seed = seeds[index];
        else if (index == 5) t.seed = -3;
        else {
            const int a = (index - 6) / 3, o = (index - 6) % 3;
            t.seed = pairs[a];
            t.second = pairs[o < a ? o : o + 1];
        }
        return true;
    }
    return false;
}

// The Newton start of a task, false when it has none.
__device__ __noinline__ bool taskStart(const MixCell& c, const MixTask& t, double* x, double& scale) {
    const ReactiveB200HemModel& m = c.m;
    const double rho = density(c), gT = t.restartT >= 0 ? t.restartT : c.guess.T;
    scale = fmax(1e5 * rho, fmax(fabs(c.energy), rho * 2000 * fmax(gT, m.Tmin)));
    x[0] = log(clampd(c.guess.p, m.pmin, m.pmax));
    x[1] = log(clampd(gT, m.Tmin, m.Tmax));
    x[2] = x[3] = 0;
    for (int j = 0; j < t.n; ++j) {
        const int i = t.active[j];
        const double selected = j == 1 && t.second != -2 ? t.second : t.seed;
        const double previous = c.guess.liquidMass[i] / c.q[m.condensable[i]];
        x[j + 2] = selected < 0 ? clampd(previous, 1e-8, 1 - 1e-8) : selected;
        if (c.adaptive) {
            double vapor = selected < 0 ? 1 - previous : 1 - selected;
            if (selected == -3 || (selected < 0 && vapor < 1e-6)) {
                double other = 0;
                for (int k = 0; k < m.ns; ++k) {
                    bool chosen = false;
                    for (int a = 0; a < t.n; ++a) chosen |= k == m.condensable[t.active[a]];
                    if (!chosen) other += c.q[k];
                }
                vapor = other > 0 ? fmin(1e-6, .01 * (other / c.q[m.condensable[i]])) : 1e-8;
            }
            if (!(vapor > 0 && fin(vapor))) return false;
            x[j + 2] = log(fmin(1., vapor));
        }
    }
    return true;
}

// The best stable candidate so far: the largest entropy density, the earliest in
// selection order on a tie (the first maximum, whatever order candidates finish in).
struct MixBest {
    bool have;
    double entropy;
    int order;
    __device__ bool takes(double e, int o) const { return !have || e > entropy || (e == entropy && o < order); }
};

// The tasks of one search over a warp. Groups of `width` lanes (two per Newton
// unknown: five groups of six with one liquid, four of eight with two) each run
// one task at a time and take the next when it ends; per round every lane makes
// at most one evaluation, all at one call site: the start, the two sides of every
// Jacobian column (bounded central differences: h = 2e-6 in ln p and ln T, 2e-5 in
// the fractions, halved up to 12 times when neither side evaluates, one-sided when
// only one does; the boundary recovery's coordinates step at least one ulp and
// weight the two sides by their actual steps), or `width` consecutive fractions of
// the line search, of which the first acceptable one is taken. The points, their
// order and the rule that accepts them are a serial search's; a Newton step takes
// two rounds instead of seven or more evaluations in a row. A point's residual is
// formed alone (mixture_residual.cuh) or, where that decides nothing, taken from the
// general evaluation, which differ by rounding.
//
// A point whose residual is within the tolerances is evaluated in full by its owner:
// the candidate's state, its reported residuals and the stability test (the chemical
// potentials of that same point) all come from this one evaluation, and the candidate
// has converged when its residual is within the tolerances too, else the Newton goes on
// from it. It stays in the owner's `v` while the last Jacobian is formed, so
// side points have a `side` of their own.
__device__ __noinline__ void runTasks(MixCell& c, const MixTerms& terms, bool restarts, MixRecord* bestRecord,
                                      MixBest& best) {
    const ReactiveB200HemModel& m = c.m;
    double q[kNs];
    bool alone = terms.valid;  // the residual formed alone (mixture_residual.cuh)
#pragma unroll
    for (int k = 0; k < kNs; ++k) {
        q[k] = c.q[k];
        alone = alone && q[k] >= 0 && fin(q[k]);
    }
    const double gasOffset = c.color * c.jump, liquidOffset = (1 - c.color) * c.jump;
    const unsigned lane = threadIdx.x & 31u;
    const int width = m.nl == 1 ? 6 : 8, groups = 32 / width;
    const int g = int(lane) / width;
    const bool inGroup = g < groups;
    const int base = g * width, r = int(lane) - base;
    const unsigned group = inGroup ? ((1u << width) - 1u) << base : 0u;
    const double rho = density(c);
    enum { IDLE, START, SIDES, TRIALS };
    int st = IDLE, task = 0, it = 0, k = 0, owner = base, attempt = 0, nextTask = 0;
    bool more = inGroup, converged = false, settled = false;
    MixTask t{{0, 0}, 0, 0, 0, 0};
    double x[4] = {}, f[4] = {}, step[4] = {}, column[4] = {}, scale = 1, previous = 0;
    MixEval v, side;
    for (;;) {
        // idle groups take the next tasks in order
        {
            const unsigned idle = __ballot_sync(0xffffffffu, inGroup && r == 0 && st == IDLE && more);
            if (inGroup && st == IDLE && more) {
                task = nextTask + __popc(idle & ((1u << base) - 1u));
                more = nthTask(c, restarts, task, t);
                if (more) {
                    if (r == 0) ++c.n.candidates;
                    if (taskStart(c, t, x, scale)) st = START;
                }
            }
            nextTask += __popc(idle);
        }
        if (__all_sync(0xffffffffu, st == IDLE)) {
            if (!__any_sync(0xffffffffu, more)) break;
            continue;
        }
        const int size = t.n + 2, j = r >> 1;
        double xe[4] = {x[0], x[1], x[2], x[3]}, fe[4] = {}, fraction = 1, hp = 0, hm = 0;
        bool point = false;
        if (st == START) point = r == 0;
        else if (st == SIDES) {
            if (j < size && !settled) {
                point = true;
                const double h = ldexp(j < 2 ? 2e-6 : 2e-5, -attempt);
                double xj = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) xj = i == j ? x[i] : xj;
                double xp = xj + h, xm = xj - h;
                if (c.adaptive) {
                    if (xp == xj) xp = nextafter(xj, HUGE_VAL);
                    if (xm == xj) xm = nextafter(xj, -HUGE_VAL);
                }
                hp = xp - xj;
                hm = xj - xm;
                if (!c.adaptive) hp = hm = h;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (i == j) xe[i] = (r & 1) ? xm : xp;
            }
        } else if (st == TRIALS && k + r < kTrials) {
            point = true;
            fraction = ldexp(1.0, -(k + r));
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < size) xe[i] = x[i] + fraction * step[i];
            for (int i = 0; i < t.n; ++i) point = point && !rejectedCoordinate(c.adaptive, xe[i + 2]);
        }
        bool ok = false;
        bool general = point && !alone;
        if (point && alone) {
            const int code = mixtureResidual(terms, q, c.energy, c.adaptive, gasOffset, liquidOffset, m.pmin, m.pmax, m.Tmin,
                                             m.Tmax, t.active, t.n, xe, scale, fe, c.n.phases);
            ok = code == RESIDUAL_OK;
            general = code == RESIDUAL_UNDECIDED;
            if (!general) ++c.n.residuals;
        }
        if (__any_sync(0xffffffffu, general)) {
            if (general) ok = activeResidual(c, t.active, t.n, xe, scale, fe, st == SIDES ? side : v);
        }
        __syncwarp();
        bool finished = false, stable = false, evaluated = false;  // evaluated: (x, f) is a new iterate
        if (st == SIDES) {
            const bool other = __shfl_xor_sync(group, ok, 1);
            double fo[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) fo[i] = __shfl_xor_sync(group, fe[i], 1);
            bool exhausted = false;
            if (j < size && !settled) {
                const bool upper = !(r & 1), plus = upper ? ok : other, minus = upper ? other : ok;
                if (plus || minus) {
                    double maximum = 0;
                    settled = true;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (i >= size) continue;
                        const double fp = upper ? fe[i] : fo[i], fm = upper ? fo[i] : fe[i];
                        double d;
                        if (c.adaptive)
                            d = plus && minus ? (hm / (hp + hm)) * ((fp - f[i]) / hp) + (hp / (hp + hm)) * ((f[i] - fm) / hm)
                                              : plus ? (fp - f[i]) / hp : (f[i] - fm) / hm;
                        else
                            d = plus && minus ? (fp - fm) / (2 * hp) : plus ? (fp - f[i]) / hp : (f[i] - fm) / hp;
                        column[i] = d;
                        maximum = fmax(maximum, fabs(d));
                        settled = settled && fin(d);
                    }
                    if (c.adaptive) settled = settled && maximum > 0;
                }
                if (!settled) exhausted = ++attempt >= 12;
            }
            const bool failed = __ballot_sync(group, exhausted) != 0;
            const bool whole = __ballot_sync(group, j < size && !settled) == 0;
            if (failed) finished = true;
            else if (whole) {
                double jac[4][4] = {}, rhs[4] = {}, answer[4] = {};
#pragma unroll
                for (int col = 0; col < 4; ++col)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const double d = __shfl_sync(group, column[i], base + (col < size ? 2 * col : 0));
                        if (i < size && col < size) jac[i][col] = d;
                    }
                if (converged) {
                    // the equilibrium sound speed of the converged point
                    const double vp = __shfl_sync(group, v.s.p, owner), vs = __shfl_sync(group, v.s.soundFrozen, owner);
                    rhs[0] = -1 / rho;
                    rhs[1] = vp / (rho * scale);
                    bool good = solveDense(jac, rhs, size, answer);
                    const double squared = vp * answer[0], sound = good ? sqrt(squared) : 0.0;
                    good = good && fin(squared) && squared > 0 && sound <= vs * (1 + 2e-3);
                    finished = true;
                    if (good && int(lane) == owner) {
                        v.s.volumeResidual = fabs(f[0]);
                        v.s.energyResidual = fabs(f[1]);
                        v.s.chemicalResidual = maxAbs(f + 2, t.n);
                        v.s.iterations = it;
                        v.s.soundEquilibrium = sound;
                        stable = true;
                        for (int i = 0; i < m.nl; ++i) {
                            if (c.q[m.condensable[i]] == 0) continue;
                            const double affinity = v.muLiq[i] - v.muGas[i];
                            stable = stable && (v.s.liquidMass[i] > 0 ? fin(affinity) && fabs(affinity) <= m.mutol * 2
                                                                      : !(affinity < -m.mutol));
                        }
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) rhs[i] = i < size ? -f[i] : 0.0;
                    if (!solveDense(jac, rhs, size, answer)) finished = true;
                    else {
                        double limiter = fmax(1., fmax(fabs(answer[0]) / .7, fabs(answer[1]) / .18));
                        for (int i = 2; i < size; ++i) limiter = fmax(limiter, fabs(answer[i]) / (c.adaptive ? 2. : .3));
#pragma unroll
                        for (int i = 0; i < 4; ++i) step[i] = i < size ? answer[i] / limiter : 0.0;
                        previous = maxAbs(f, size);
                        // the fractions a coordinate rejects form a prefix (each moves back
                        // toward the valid x as the fraction halves): its end by bisection
                        // on the trial's own expression, kTrials standing for none
                        auto rejects = [&](int trial) {
                            const double fm = ldexp(1.0, -trial);
                            bool bad = false;
                            for (int i = 0; i < t.n; ++i) bad |= rejectedCoordinate(c.adaptive, x[i + 2] + fm * step[i + 2]);
                            return bad;
                        };
                        k = 0;
                        if (rejects(0)) {
                            int lower = 0, upper = kTrials;
                            while (upper - lower > 1) {
                                const int mid = (lower + upper) / 2;
                                if (rejects(mid)) lower = mid; else upper = mid;
                            }
                            k = upper;
                        }
                        st = TRIALS;
                        finished = k >= kTrials;
                    }
                }
            }
        } else if (st == START || st == TRIALS) {
            if (st == TRIALS) ok = ok && maxAbs(fe, size) < previous * (1 - 1e-4 * fraction);
            const unsigned accepted = __ballot_sync(group, ok);
            if (accepted) {
                owner = __ffs(accepted) - 1;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    x[i] = __shfl_sync(group, xe[i], owner);
                    f[i] = __shfl_sync(group, fe[i], owner);
                }
                it = st == START ? 0 : it + 1;
                evaluated = true;
                finished = it >= 90;
                auto within = [&] {
                    return fabs(f[0]) <= m.vtol && fabs(f[1]) <= m.etol && maxAbs(f + 2, t.n) <= m.mutol;
                };
                converged = within();
                if (converged && !finished) {
                    bool whole = true;
                    if (int(lane) == owner) {
                        const Tally keep = c.n;
                        whole = activeResidual(c, t.active, t.n, x, scale, fe, v);
                        c.n = keep;
                    }
                    finished = __ballot_sync(group, !whole) != 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) f[i] = __shfl_sync(group, fe[i], owner);
                    converged = within();
                }
            } else {
                k += width;
                finished = st == START || k >= kTrials;
            }
        }
        if (evaluated && !finished) {
            st = SIDES;
            settled = false;
            attempt = 0;
            if (r == 0) ++c.n.fd;
        }
        if (finished) st = IDLE;
        // stable candidates enter the selection (a candidate's owner holds its state)
        unsigned offers = __ballot_sync(0xffffffffu, stable);
        if (stable) ++c.n.stable;
        while (offers) {
            const int from = __ffs(offers) - 1;
            offers &= offers - 1;
            const double e = __shfl_sync(0xffffffffu, v.entropyD, from);
            const int o = __shfl_sync(0xffffffffu, task, from);
            if (best.takes(e, o)) {
                best = MixBest{true, e, o};
                if (int(lane) == from) storeRecord(*bestRecord, v, kStable);
            }
            __syncwarp();
        }
    }
}

// One search (the candidate list, then the restart temperatures when it found no
// stable candidate) into *bestRecord (shared by the warp): the fixed-partition
// candidates' records, then the tasks.
__device__ __noinline__ bool searchWarp(MixCell& c, const MixTerms& terms, const MixRecord& gas,
                                        const MixRecord& liquid, MixRecord* bestRecord) {
    const ReactiveB200HemModel& m = c.m;
    const unsigned lane = threadIdx.x & 31u;
    MixBest best{false, 0.0, 0};
    auto offer = [&](const MixRecord& record, int order) {
        if (record.status != kStable || !best.takes(record.entropyD, order)) return;
        best = MixBest{true, record.entropyD, order};
        if (lane == 0) *bestRecord = record;
    };
    offer(gas, -2);
    offer(liquid, -1);
    __syncwarp();
    const bool prune = m.stableGasPrune && prunable(m) && gas.status == kStable && gas.s.gasMass > 0 && !c.adaptive;
    if (!prune && m.nl) runTasks(c, terms, false, bestRecord, best);
    if (!best.have && m.nl) runTasks(c, terms, true, bestRecord, best);
    return best.have;
}

// The recovery of one item per warp, items from an on-device counter: the
// candidate search; with the boundary recovery (or in a capillary batch, whose
// transported trace inventories can defeat the reference seeds) a second search
// in log vapour fractions when the first found nothing or left a condensable
// almost entirely liquid beside a gas phase, the larger entropy (the first search
// on a tie) kept. A frozen partition's result is its record. Results go to
// out/success, or to outputs[cell] for the resident form; a failed cell gets its
// seed.
//
// Bound by instruction fetch (see mixture_residual.cuh), whose waits more warps hide:
// 20,011 cells of the four-species gas take 51.9 ms at four blocks a multiprocessor
// (128 registers), 42.3 at eight and 36.4 at sixteen (32, 100 bytes spilled).
__global__ void __launch_bounds__(kSearchBlock, 16) mixtureSearch(MixBatch b) {
    const ReactiveB200HemModel& m = *b.model;
    __shared__ MixRecord found[kSearchBlock / 32][2];
    __shared__ MixTerms terms;
    static_assert(sizeof(MixTerms) % sizeof(double) == 0, "copied by doubles");
    for (unsigned i = threadIdx.x; i < sizeof(MixTerms) / sizeof(double); i += blockDim.x)
        reinterpret_cast<double*>(&terms)[i] = reinterpret_cast<const double*>(b.terms)[i];
    __syncthreads();
    MixRecord* best = found[threadIdx.x >> 5];
    const unsigned lane = threadIdx.x & 31u;
    Tally n;
    unsigned long long succeeded = 0;
    MixCell c{m, {0, 0, 0, 0}, 0.0, ReactiveThermoState{}, false, n};
    for (;;) {
        unsigned i = 0;
        if (lane == 0) i = atomicAdd(b.counters + C_SEARCH, 1u);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= b.count) break;
        loadCell(b, i, c);
        const MixRecord& gas = b.record[kGasRecord][i];
        const ReactiveThermoState* result = nullptr;
        if (gas.status == kInvalid) {
        } else if (frozenItem(b, i)) {
            if (gas.status == kStable) result = &gas.s;
        } else {
            const MixRecord& liquid = b.record[kLiquidRecord][i];
            const bool have = searchWarp(c, terms, gas, liquid, best);
            if (have) result = &best[0].s;
            if (m.boundaryRecovery || b.capillary) {
                bool again = !have;
                if (have)
                    for (int l = 0; l < m.nl; ++l) {
                        const double q = c.q[m.condensable[l]];
                        if (q > 0 && best[0].s.gasMass > 0) again |= best[0].s.liquidMass[l] / q > 1 - 1e-4;
                    }
                if (again) {
                    c.adaptive = true;
                    const bool other = searchWarp(c, terms, b.record[kFullGasRecord] ? b.record[kFullGasRecord][i] : gas,
                                                  liquid, best + 1);
                    if (other && !(have && best[0].entropyD >= best[1].entropyD)) result = &best[1].s;
                }
            }
        }
        const size_t cell = b.order ? size_t(b.order[i]) : size_t(i);
        const double* from = reinterpret_cast<const double*>(result ? result : b.seed + cell);
        double* to = reinterpret_cast<double*>(b.outputs ? &b.outputs[cell].state : b.out + cell);
        constexpr unsigned words = sizeof(ReactiveThermoState) / sizeof(double);
        if (lane < words) to[lane] = from[lane];
        if (lane == 0) {
            if (b.success) b.success[cell] = result ? 1 : 0;
            if (b.outputs) b.outputs[cell].success = result ? 1 : 0;
            succeeded += result ? 1 : 0;
        }
        __syncwarp();  // the shared records are rewritten by the next item
    }
    flushTally(n, b.totals);
    if (lane == 0 && succeeded) atomicAdd(b.totals + M_SUCCEEDED, succeeded);
}

// The capillary primitive initialisation (initializeCapillaryTP,
// src/reactiveThermo/reactiveDeviceFlash.h:589-613), one thread per cell: at the
// seed's (p, T) and liquid mass, with the gas at p - color*jump and the liquid
// at p + (1 - color)*jump, scale the densities so the phase volumes fill the
// cell; q and energy become the normalised densities and their energy where a
// cell succeeds.
__global__ void __launch_bounds__(kBlock) mixtureInitializeKernel(const ReactiveB200HemModel* __restrict__ model,
                                                                 double* q, double* energy, size_t count,
                                                                 const ReactiveThermoState* __restrict__ seed,
                                                                 const ReactiveGpuHemCapillaryInputV2* capillary,
                                                                 ReactiveThermoState* out, int* success,
                                                                 unsigned long long* totals) {
    const ReactiveB200HemModel& m = *model;
    Tally n;
    unsigned long long succeeded = 0;
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < count; i += size_t(blockDim.x) * gridDim.x) {
        MixCell c{m, {0, 0, 0, 0}, energy[i], seed[i], false, n};
        for (int k = 0; k < m.ns && k < kNs; ++k) c.q[k] = q[i * size_t(m.ns) + k];
        c.color = capillary[i].color;
        c.jump = capillary[i].pressureJump;
        bool ok = m.nl == 1 && m.condensedKind[0] == 0 && fin(c.color) && c.color >= 0 && c.color <= 1 && fin(c.jump);
        double liquid[kLiq] = {c.guess.liquidMass[0], 0};
        MixEval unit, value;
        if (ok) ok = evaluate(c, liquid, c.guess.p, c.guess.T, unit, false, nullptr) && fin(unit.volume)
                     && unit.volume > 0;
        if (ok) {
            for (int k = 0; k < m.ns; ++k) c.q[k] /= unit.volume;
            liquid[0] /= unit.volume;
            ok = evaluate(c, liquid, c.guess.p, c.guess.T, value, false, nullptr) && fin(value.energy)
                 && fabs(value.volume - 1) <= m.vtol;
        }
        if (ok) {
            value.s.volumeResidual = fabs(value.volume - 1);
            for (int k = 0; k < m.ns; ++k) q[i * size_t(m.ns) + k] = c.q[k];
            energy[i] = value.energy;
            out[i] = value.s;
        } else out[i] = c.guess;
        success[i] = ok ? 1 : 0;
        succeeded += ok ? 1 : 0;
    }
    atomicAdd(totals + M_PHASES, n.phases);
    atomicAdd(totals + M_SUCCEEDED, succeeded);
}

bool finiteHost(double x) { return x == x && std::fabs(x) <= 1.79769313486231570815e308; }

// The scope this build's mixture flash covers, on top of the reference's model
// validation (src/reactiveThermo/reactiveDeviceFlash.h:80-108).
std::string mixtureScope(const ReactiveB200HemModel& m) {
    if (m.ns < 1 || m.ns > kNs || m.nl < 0 || m.nl > kLiq)
        return "HEM model outside the mixture flash's scope: 1 to 4 gas species and 0 to 2 pure liquids";
    if (m.condensedKind[0] != 0 || m.condensedKind[1] != 0) return "Solid condensed phases are not part of this build";
    if ((m.boundaryRecovery != 0 && m.boundaryRecovery != 1) || (m.scalarRecovery != 0 && m.scalarRecovery != 1)
        || (m.stableGasPrune != 0 && m.stableGasPrune != 1)
        || (m.stableGasPrune && m.nl != 1)
        || (m.enforceSpeciesTemperatureBounds != 0 && m.enforceSpeciesTemperatureBounds != 1))
        return "Invalid CUDA HEM model flags";
    if (!finiteHost(m.Tmin) || !finiteHost(m.Tmax) || !(m.Tmin > 0 && m.Tmax > m.Tmin) || !finiteHost(m.pmin)
        || !finiteHost(m.pmax) || !(m.pmin > 0 && m.pmax > m.pmin) || !finiteHost(m.vtol) || !finiteHost(m.etol)
        || !finiteHost(m.mutol) || !(m.vtol > 0 && m.etol > 0 && m.mutol > 0))
        return "Invalid CUDA HEM model tables or domain";
    if (m.phase[0].ns != m.ns) return "Invalid CUDA HEM gas table";
    for (int k = 0; k < m.ns; ++k) {
        const ReactiveB200Species& sp = m.phase[0].species[k];
        if (!finiteHost(m.weights[k]) || m.weights[k] != sp.molecularWeight || !(sp.a > 0) || !(sp.b > 0)
            || sp.regionCount < 1 || sp.regionCount > REACTIVE_B200_MAX_REGIONS)
            return "Invalid CUDA HEM gas table";
    }
    for (int i = 0; i < m.nl; ++i) {
        const ReactiveB200Table& t = m.phase[i + 1];
        if (m.condensable[i] < 0 || m.condensable[i] >= m.ns || t.ns != 1
            || t.species[0].molecularWeight != m.weights[m.condensable[i]] || !(t.species[0].a > 0)
            || !(t.species[0].b > 0) || t.species[0].regionCount < 1
            || t.species[0].regionCount > REACTIVE_B200_MAX_REGIONS || !finiteHost(m.liquidTmin[i])
            || !finiteHost(m.liquidTc[i]) || !(m.liquidTmin[i] > 0 && m.liquidTc[i] > m.liquidTmin[i]))
            return "Invalid CUDA HEM liquid table or range";
        for (int j = 0; j < i; ++j)
            if (m.condensable[j] == m.condensable[i]) return "Invalid CUDA HEM liquid table or range";
    }
    return "";
}

}  // namespace

struct MixtureFlash {
    int device = 0;
    size_t capacity = 0;
    size_t bytes = 0;
    int ns = 0;
    cudaStream_t stream = nullptr;
    std::vector<void*> blocks;
    ReactiveB200HemModel* model = nullptr;
    MixTerms* terms = nullptr;
    double* q = nullptr;
    double* energy = nullptr;
    ReactiveThermoState* seed = nullptr;
    ReactiveThermoState* out = nullptr;
    int* success = nullptr;
    ReactiveGpuHemCapillaryInputV2* capillary = nullptr;  // allocated by the first capillary batch
    unsigned long long* totals = nullptr;
    MixRecord* record[kRecordKinds] = {};
    unsigned* list = nullptr;
    unsigned* counters = nullptr;
    unsigned newtonBlocks = 1, searchBlocks = 1;  // whole waves of resident blocks
    template <class T> T* alloc(size_t n) {
        void* p = nullptr;
        check(cudaMalloc(&p, n * sizeof(T)), "cudaMalloc");
        blocks.push_back(p);
        bytes += n * sizeof(T);
        return static_cast<T*>(p);
    }
    ~MixtureFlash() {
        if (stream) cudaStreamSynchronize(stream);
        for (void* p : blocks) cudaFree(p);
        if (stream) cudaStreamDestroy(stream);
    }
};

MixtureFlash* mixtureCreate(const ReactiveB200HemModel& m, size_t capacity, int device, std::string& why) {
    why = mixtureScope(m);
    if (!why.empty()) return nullptr;
    std::unique_ptr<MixtureFlash> f(new MixtureFlash);
    f->device = device;
    f->capacity = capacity;
    f->ns = m.ns;
    check(cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking), "cudaStreamCreate");
    // one device allocation for all arrays: a handle is often made for one batch, and
    // each allocation costs it two driver calls (20,011 cells of the production gas,
    // create and destroy: 3.4 ms with an allocation an array, 0.7 to 0.9 ms so)
    auto place = [&](char* base) {
        size_t at = 0;
        auto take = [&](auto*& array, size_t n) {
            if (base) array = reinterpret_cast<std::remove_reference_t<decltype(array)>>(base + at);
            at += (n * sizeof(*array) + 255) / 256 * 256;
        };
        take(f->model, 1);
        take(f->terms, 1);
        take(f->q, capacity * size_t(m.ns));
        take(f->energy, capacity);
        take(f->seed, capacity);
        take(f->out, capacity);
        take(f->success, capacity);
        take(f->totals, M_COUNT);
        take(f->record[kGasRecord], capacity);
        take(f->record[kLiquidRecord], capacity);
        if (m.stableGasPrune) take(f->record[kFullGasRecord], capacity);
        take(f->list, capacity * kRecordKinds);
        take(f->counters, C_COUNT);
        return at;
    };
    place(f->alloc<char>(place(nullptr)));
    int sms = 0, perSm = 0;
    check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "attribute");
    check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, mixtureNewton, kSearchBlock, 0), "occupancy");
    f->newtonBlocks = unsigned(std::max(1, perSm) * std::max(1, sms));
    check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, mixtureSearch, kSearchBlock, 0), "occupancy");
    f->searchBlocks = unsigned(std::max(1, perSm) * std::max(1, sms));
    MixTerms terms;
    mixTerms(m, terms);
    check(cudaMemcpyAsync(f->model, &m, sizeof(m), cudaMemcpyHostToDevice, f->stream), "H2D model");
    check(cudaMemcpyAsync(f->terms, &terms, sizeof(terms), cudaMemcpyHostToDevice, f->stream), "H2D terms");
    check(cudaStreamSynchronize(f->stream), "sync");
    return f.release();
}

void mixtureDestroy(MixtureFlash* f) { delete f; }
size_t mixtureDeviceBytes(const MixtureFlash* f) { return f ? f->bytes : 0; }

// The batch's launches on the handle's stream: the scalar all-gas solves, the
// fixed-partition Newtons they leave, then the searches. The handle's entry lock
// keeps batches (which share the records) one after another.
static void launchRecovery(MixtureFlash* f, MixBatch b) {
    for (int i = 0; i < kRecordKinds; ++i) b.record[i] = f->record[i];
    b.model = f->model;
    b.terms = f->terms;
    b.list = f->list;
    b.counters = f->counters;
    b.totals = f->totals;
    check(cudaMemsetAsync(f->counters, 0, C_COUNT * sizeof(unsigned), f->stream), "memset");
    mixtureScalar<<<gridFor(b.count, kBlock), kBlock, 0, f->stream>>>(b);
    check(cudaGetLastError(), "mixture scalar solves");
    const size_t newtonGroups = kSearchBlock / kNewtonLanes, searchWarps = kSearchBlock / 32;
    const size_t newtonNeed = (kRecordKinds * b.count + newtonGroups - 1) / newtonGroups;
    const size_t searchNeed = (b.count + searchWarps - 1) / searchWarps;
    mixtureNewton<<<unsigned(std::min<size_t>(f->newtonBlocks, newtonNeed)), kSearchBlock, 0, f->stream>>>(b);
    check(cudaGetLastError(), "mixture Newton");
    mixtureSearch<<<unsigned(std::min<size_t>(f->searchBlocks, searchNeed)), kSearchBlock, 0, f->stream>>>(b);
    check(cudaGetLastError(), "mixture search");
}

void mixtureRun(MixtureFlash* f, const double* q, const double* energy, size_t count,
                const ReactiveGpuHemCapillaryInputV2* capillary, ReactiveThermoState* states, int* success,
                ReactiveGpuHemProfileV1& p) {
    require(count && count <= f->capacity, "CUDA HEM batch exceeds capacity");
    check(cudaSetDevice(f->device), "cudaSetDevice");
    const auto begin = std::chrono::steady_clock::now();
    cudaStream_t s = f->stream;
    if (capillary && !f->capillary) f->capillary = f->alloc<ReactiveGpuHemCapillaryInputV2>(f->capacity);
    cudaEvent_t a, b;
    check(cudaEventCreate(&a), "event");
    check(cudaEventCreate(&b), "event");
    check(cudaMemcpyAsync(f->q, q, count * size_t(f->ns) * sizeof(double), cudaMemcpyHostToDevice, s), "H2D q");
    check(cudaMemcpyAsync(f->energy, energy, count * sizeof(double), cudaMemcpyHostToDevice, s), "H2D e");
    check(cudaMemcpyAsync(f->seed, states, count * sizeof(ReactiveThermoState), cudaMemcpyHostToDevice, s), "H2D seed");
    if (capillary)
        check(cudaMemcpyAsync(f->capillary, capillary, count * sizeof(ReactiveGpuHemCapillaryInputV2),
                              cudaMemcpyHostToDevice, s),
              "H2D capillary");
    check(cudaMemsetAsync(f->totals, 0, M_COUNT * sizeof(unsigned long long), s), "memset");
    check(cudaEventRecord(a, s), "event");
    MixBatch batch{};
    batch.q = f->q;
    batch.energy = f->energy;
    batch.count = count;
    batch.seed = f->seed;
    batch.capillary = capillary ? f->capillary : nullptr;
    batch.out = f->out;
    batch.success = f->success;
    launchRecovery(f, batch);
    check(cudaEventRecord(b, s), "event");
    check(cudaMemcpyAsync(states, f->out, count * sizeof(ReactiveThermoState), cudaMemcpyDeviceToHost, s), "D2H");
    check(cudaMemcpyAsync(success, f->success, count * sizeof(int), cudaMemcpyDeviceToHost, s), "D2H success");
    unsigned long long t[M_COUNT] = {};
    check(cudaMemcpyAsync(t, f->totals, sizeof(t), cudaMemcpyDeviceToHost, s), "D2H totals");
    check(cudaStreamSynchronize(s), "sync");
    float kernel = 0;
    cudaEventElapsedTime(&kernel, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    p.batches = 1;
    p.submitted = count;
    p.succeeded = t[M_SUCCEEDED];
    p.deviceFailures = count - p.succeeded;
    p.phaseEvaluations = t[M_PHASES];
    p.residualEvaluations = t[M_RESIDUALS];
    p.flashCandidates = t[M_CANDIDATES];
    p.stableCandidates = t[M_STABLE];
    p.finiteDifferenceJacobians = t[M_FD];
    p.transferBytes = count * ((f->ns + 1) * sizeof(double) + 2 * sizeof(ReactiveThermoState) + sizeof(int)
                               + (capillary ? sizeof(ReactiveGpuHemCapillaryInputV2) : 0));
    p.deviceBytes = f->bytes;
    p.hostBytes = count * sizeof(ReactiveThermoState);
    p.kernelSeconds = kernel / 1000.;
    p.wallSeconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - begin).count();
    p.copySeconds = std::max(0.0, p.wallSeconds - p.kernelSeconds);
}

void mixtureInitialize(MixtureFlash* f, double* q, double* energy, size_t count,
                       const ReactiveGpuHemCapillaryInputV2* capillary, ReactiveThermoState* states, int* success,
                       ReactiveGpuHemProfileV1& p) {
    require(count && count <= f->capacity, "CUDA HEM batch exceeds capacity");
    check(cudaSetDevice(f->device), "cudaSetDevice");
    const auto begin = std::chrono::steady_clock::now();
    cudaStream_t s = f->stream;
    if (!f->capillary) f->capillary = f->alloc<ReactiveGpuHemCapillaryInputV2>(f->capacity);
    const size_t qBytes = count * size_t(f->ns) * sizeof(double);
    check(cudaMemcpyAsync(f->q, q, qBytes, cudaMemcpyHostToDevice, s), "H2D q");
    check(cudaMemcpyAsync(f->energy, energy, count * sizeof(double), cudaMemcpyHostToDevice, s), "H2D e");
    check(cudaMemcpyAsync(f->seed, states, count * sizeof(ReactiveThermoState), cudaMemcpyHostToDevice, s), "H2D seed");
    check(cudaMemcpyAsync(f->capillary, capillary, count * sizeof(ReactiveGpuHemCapillaryInputV2),
                          cudaMemcpyHostToDevice, s),
          "H2D capillary");
    check(cudaMemsetAsync(f->totals, 0, M_COUNT * sizeof(unsigned long long), s), "memset");
    mixtureInitializeKernel<<<gridFor(count, kBlock), kBlock, 0, s>>>(f->model, f->q, f->energy, count, f->seed,
                                                                       f->capillary, f->out, f->success, f->totals);
    check(cudaGetLastError(), "capillary initialisation");
    std::vector<double> nq(count * size_t(f->ns)), ne(count);
    std::vector<ReactiveThermoState> out(count);
    check(cudaMemcpyAsync(nq.data(), f->q, qBytes, cudaMemcpyDeviceToHost, s), "D2H q");
    check(cudaMemcpyAsync(ne.data(), f->energy, count * sizeof(double), cudaMemcpyDeviceToHost, s), "D2H e");
    check(cudaMemcpyAsync(out.data(), f->out, count * sizeof(ReactiveThermoState), cudaMemcpyDeviceToHost, s), "D2H");
    check(cudaMemcpyAsync(success, f->success, count * sizeof(int), cudaMemcpyDeviceToHost, s), "D2H success");
    unsigned long long t[M_COUNT] = {};
    check(cudaMemcpyAsync(t, f->totals, sizeof(t), cudaMemcpyDeviceToHost, s), "D2H totals");
    check(cudaStreamSynchronize(s), "sync");
    p.batches = 1;
    p.submitted = count;
    p.succeeded = t[M_SUCCEEDED];
    p.deviceFailures = count - p.succeeded;
    p.phaseEvaluations = t[M_PHASES];
    // the caller's arrays change only when every cell succeeded
    if (!p.deviceFailures) {
        std::memcpy(q, nq.data(), qBytes);
        std::memcpy(energy, ne.data(), count * sizeof(double));
        std::memcpy(states, out.data(), count * sizeof(ReactiveThermoState));
    }
    p.transferBytes = 2 * (qBytes + count * sizeof(double)) + count * (2 * sizeof(ReactiveThermoState) + sizeof(int)
                                                                      + sizeof(ReactiveGpuHemCapillaryInputV2));
    p.deviceBytes = f->bytes;
    p.hostBytes = qBytes + count * (sizeof(double) + sizeof(ReactiveThermoState));
    p.wallSeconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - begin).count();
}

void mixtureRunResident(MixtureFlash* f, const double* q, const double* energy, const ReactiveThermoState* seed,
                        const ReactiveGpuHemCapillaryInputV2* capillary, const uint32_t* order, size_t count,
                        ReactiveGpuHemOutputV1* output, ReactiveGpuHemProfileV1& p) {
    require(count && count <= f->capacity, "Resident CUDA HEM batch exceeds capacity");
    check(cudaSetDevice(f->device), "cudaSetDevice");
    const auto begin = std::chrono::steady_clock::now();
    cudaStream_t s = f->stream;
    cudaEvent_t a, b;
    check(cudaEventCreate(&a), "event");
    check(cudaEventCreate(&b), "event");
    check(cudaMemsetAsync(f->totals, 0, M_COUNT * sizeof(unsigned long long), s), "memset");
    check(cudaEventRecord(a, s), "event");
    MixBatch batch{};
    batch.q = q;
    batch.energy = energy;
    batch.count = count;
    batch.seed = seed;
    batch.capillary = capillary;
    batch.order = order;
    batch.outputs = output;
    launchRecovery(f, batch);
    check(cudaEventRecord(b, s), "event");
    unsigned long long t[M_COUNT] = {};
    check(cudaMemcpyAsync(t, f->totals, sizeof(t), cudaMemcpyDeviceToHost, s), "D2H totals");
    check(cudaStreamSynchronize(s), "sync");
    float kernel = 0;
    cudaEventElapsedTime(&kernel, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    p.batches = 1;
    p.submitted = count;
    p.succeeded = t[M_SUCCEEDED];
    p.deviceFailures = count - p.succeeded;
    p.phaseEvaluations = t[M_PHASES];
    p.residualEvaluations = t[M_RESIDUALS];
    p.flashCandidates = t[M_CANDIDATES];
    p.stableCandidates = t[M_STABLE];
    p.finiteDifferenceJacobians = t[M_FD];
    p.transferBytes = sizeof(t);
    p.deviceBytes = f->bytes;
    p.kernelSeconds = kernel / 1000.;
    p.wallSeconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - begin).count();
    p.copySeconds = std::max(0.0, p.wallSeconds - p.kernelSeconds);
}

}  // namespace rb200
