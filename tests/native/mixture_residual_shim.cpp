// Test infrastructure only: the two-phase residual formed alone
// (spuma-multiphysics_b200/csrc/mixture_residual.cuh, host and device code from one
// source) compiled for the host beside the residual of the general evaluation,
// built here from the mixture evaluator's phase properties.
#include "mixture_residual.cuh"

using namespace rb200;

namespace {
int generalResidual(const ReactiveB200HemModel& m, const double* q, double energy, bool adaptive, double gasOffset,
                    double liquidOffset, const int* active, int n, const double* x, double scale, double* f) {
    double gas[mix::kMaxNs] = {}, mass[2] = {}, mg = 0, muG[2] = {}, muL[2] = {};
    for (int k = 0; k < m.ns; ++k) gas[k] = q[k];
    for (int j = 0; j < n; ++j) {
        const int i = active[j], k = m.condensable[i];
        if (adaptive) {
            if (!mix::finiteD(x[j + 2]) || x[j + 2] > 0) return 0;
            gas[k] = exp(x[j + 2]) * q[k];
            if (!(gas[k] > 0)) return 0;
            mass[i] = -expm1(x[j + 2]) * q[k];
        } else {
            if (!(x[j + 2] >= 0 && x[j + 2] < 1)) return 0;
            mass[i] = x[j + 2] * q[k];
            gas[k] -= mass[i];
        }
    }
    const double p = exp(x[0]), T = exp(x[1]), pg = p - gasOffset, pl = p + liquidOffset;
    auto inside = [&](double v) { return v >= m.pmin && v <= m.pmax && T >= m.Tmin && T <= m.Tmax; };
    for (int k = 0; k < m.ns; ++k) mg += gas[k];
    if (!inside(p) || !(mg > 0) || !inside(pg)) return 0;
    double Y[mix::kMaxNs] = {};
    for (int k = 0; k < m.ns; ++k) {
        Y[k] = gas[k] / mg;
        const ReactiveB200Species& s = m.phase[0].species[k];
        if (m.enforceSpeciesTemperatureBounds && Y[k] > 0
            && (T < s.regions[0].minimumTemperature || T > s.regions[s.regionCount - 1].maximumTemperature))
            return 0;
    }
    mix::Props prop;
    if (mix::tp(m.phase[0], T, pg, Y, mix::GAS, true, prop) != mix::OK) return 0;
    double volume = mg / prop.rho, content = mg * prop.e;
    for (int i = 0; i < m.nl; ++i) muG[i] = prop.mu[m.condensable[i]] / (mix::kR * T);
    for (int i = 0; i < m.nl; ++i) {
        if (!(q[m.condensable[i]] > 0)) continue;
        int st = mix::OK;
        const double one[mix::kMaxNs] = {1, 0, 0, 0};
        if (!inside(pl) || T < m.liquidTmin[i]) st = mix::BAD_INPUT;
        else if (T >= m.liquidTc[i] * (1 - 1e-10)) st = mix::UNAVAILABLE;
        else st = mix::tp(m.phase[i + 1], T, pl, one, mix::LIQUID, true, prop);
        if (st != mix::OK) {
            if (mass[i] > 0 || (st != mix::UNAVAILABLE && st != mix::NO_ROOT)) return 0;
            muL[i] = HUGE_VAL;
            continue;
        }
        muL[i] = prop.mu[0] / (mix::kR * T);
        if (mass[i] > 0) {
            volume += mass[i] / prop.rho;
            content += mass[i] * prop.e;
        }
    }
    f[0] = volume - 1;
    f[1] = (content - energy) / scale;
    f[2] = f[3] = 0;
    for (int j = 0; j < n; ++j) {
        f[2 + j] = muL[active[j]] - muG[active[j]];
        if (!mix::finiteD(f[2 + j])) return 0;
    }
    return 1;
}
}  // namespace

// codes[i]: the residual's answer; general[i]: the general evaluation's (1 or 0);
// f, g: their residuals (4 a point).
extern "C" int mix_residuals(const ReactiveB200HemModel* m, long count, const double* q, const double* energy,
                             const int* mask, int adaptive, double gasOffset, double liquidOffset, const double* x,
                             const double* scale, int* codes, int* general, double* f, double* g) {
    MixTerms* t = new MixTerms;
    mixTerms(*m, *t);
    const int valid = t->valid;
    for (long i = 0; i < count && valid; ++i) {
        int active[2] = {0, 0}, n = 0;
        for (int l = 0; l < m->nl; ++l)
            if (mask[i] & (1 << l)) active[n++] = l;
        unsigned long long phases = 0;
        codes[i] = mixtureResidual(*t, q + 4 * i, energy[i], adaptive != 0, gasOffset, liquidOffset, m->pmin, m->pmax,
                                   m->Tmin, m->Tmax, active, n, x + 4 * i, scale[i], f + 4 * i, phases);
        general[i] = generalResidual(*m, q + 4 * i, energy[i], adaptive != 0, gasOffset, liquidOffset, active, n,
                                     x + 4 * i, scale[i], g + 4 * i);
    }
    delete t;
    return valid;
}
