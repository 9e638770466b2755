// The residual of a two-phase Newton of the multi-species flash, formed alone.
//
// The search of hem_mixture.cu evaluates a partition hundreds of times a cell and
// keeps the state of one evaluation per candidate. An iteration reads the volume,
// the energy and the differences of the condensables' chemical potentials, in
// which most of an evaluation cancels: with V, iv = 1/(V - b), id = 1/(V^2 + 2bV - b^2)
// and L the attraction logarithm over 2 sqrt2 b of each phase,
//   (mu_l - mu_g)/RT = ln(iv_l / (iv_g x_k)) + b_k (iv_l - iv_g)
//                      - (a_l/RT) (L_l + V_l id_l)
//                      + (L_g (2 s_k - a_g b_k / b) + a_g b_k V_g id_g / b) / RT
// (s_k = sqrt(alpha_k) sum_i x_i a_ki sqrt(alpha_i)): no ideal-gas term, no entropy
// and one logarithm where the separate potentials take nine. The gas and the liquids
// share the species' temperature terms, each cubic polishes the one root it is
// asked for, and the reported-phase line of the gas, which takes a cubic solve of
// its own, is needed only near it (mixtureResidual). What is rejected here is what
// the general evaluation (evaluate) rejects; where a decision comes closer to its
// threshold than rounding can carry, the answer is "undecided" and the general
// evaluation is asked.
//
// The loops over species and liquids stay rolled and the root and its phase's terms are
// calls: a warp's tasks are seldom at the same instruction, so the search is bound by
// instruction fetch once an evaluation's code outgrows the instruction cache
// (unrolled and inlined, 35 of 43 cycles between two instructions of a warp were
// waits for one). 20,011 cells of the four-species gas: 103.5 ms with the general
// evaluation, 62.6 unrolled, 57.3 rolled, 51.9 with the general routines as calls too
// (all at four blocks a multiprocessor).
#pragma once
#include "pr_mixture.cuh"

#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define RB200_HD_INLINE __host__ __device__ __forceinline__
#define RB200_HD_CALL __host__ __device__ __noinline__
#define RB200_ROLLED _Pragma("unroll 1")
#else
#define RB200_HD_INLINE inline
#define RB200_HD_CALL inline
#define RB200_ROLLED
#endif

namespace rb200 {

// What the residual reads of a model, in a form small enough for shared memory.
struct MixRegion {
    double m2, m1, c0, c1, c2, c3, c4, h1, h2, h3, h4, hc;  // cp/R and h/RT in powers of T
};
struct MixSpecies {
    double invW, b, kappa, kappaPlus1, invTc, Tlo, Thi;
    int regions;
    double from[REACTIVE_B200_MAX_REGIONS];  // a region holds T >= from
    MixRegion region[REACTIVE_B200_MAX_REGIONS];
};
struct MixLiquid {
    int species;
    double Tmin, Tend;               // its range; Tend = Tc (1 - 1e-10)
    double tcLine, rhoC, lineSlope;  // its reported-phase line
};
struct MixTerms {
    int valid, ns, nl, bounds;
    double a[mix::kMaxNs][mix::kMaxNs];
    MixSpecies sp[mix::kMaxNs];
    MixLiquid liquid[2];
};

// The terms of a model; valid only where the liquids' tables are the gas species'
// own, the interaction matrix is symmetric and the liquids' lines exist.
inline void mixTerms(const ReactiveB200HemModel& m, MixTerms& t) {
    std::memset(&t, 0, sizeof(t));
    const ReactiveB200Table& g = m.phase[0];
    t.ns = m.ns;
    t.nl = m.nl;
    t.bounds = m.enforceSpeciesTemperatureBounds;
    bool valid = m.nl >= 1 && m.ns >= 1 && m.ns <= mix::kMaxNs;
    for (int k = 0; k < mix::kMaxNs; ++k) {
        MixSpecies& o = t.sp[k];
        o.kappaPlus1 = 1;  // species the model lacks: no amount and neutral terms
        o.invW = 1;
        if (k >= m.ns) continue;
        const ReactiveB200Species& s = g.species[k];
        o.invW = 1 / s.molecularWeight;
        o.b = s.b;
        o.kappa = s.kappa;
        o.kappaPlus1 = 1 + s.kappa;
        const double Tc = s.a * mix::kOmB / (s.b * mix::kOmA * mix::kR);
        valid = valid && Tc > 0 && std::isfinite(Tc);
        o.invTc = 1 / Tc;
        o.regions = s.regionCount;
        o.Tlo = s.regions[0].minimumTemperature;
        o.Thi = s.regions[s.regionCount - 1].maximumTemperature;
        for (int r = 0; r < s.regionCount; ++r) {
            const double edge = s.regions[r].minimumTemperature, *a = s.regions[r].coefficient;
            const bool nine = s.regions[r].polynomial == 9;
            o.from[r] = nine ? edge : std::nextafter(edge, HUGE_VAL);
            const double* c = a + (nine ? 2 : 0);
            o.region[r] = MixRegion{nine ? a[0] : 0.0, nine ? a[1] : 0.0, c[0], c[1], c[2], c[3], c[4],
                                    c[1] / 2, c[2] / 3, c[3] / 4, c[4] / 5, nine ? a[7] : a[5]};
        }
        for (int j = 0; j < m.ns; ++j) {
            t.a[k][j] = g.aBinary[k][j];
            valid = valid && g.aBinary[k][j] == g.aBinary[j][k];
        }
    }
    for (int i = 0; i < m.nl && valid; ++i) {
        const ReactiveB200Table& l = m.phase[i + 1];
        const int k = m.condensable[i];
        const ReactiveB200Species &x = l.species[0], &y = g.species[k];
        valid = l.refPressure == g.refPressure && l.aBinary[0][0] == g.aBinary[k][k]
                && x.molecularWeight == y.molecularWeight && x.a == y.a && x.b == y.b && x.kappa == y.kappa
                && x.regionCount == y.regionCount;
        for (int r = 0; valid && r < y.regionCount; ++r)
            valid = x.regions[r].minimumTemperature == y.regions[r].minimumTemperature
                    && x.regions[r].polynomial == y.regions[r].polynomial
                    && !std::memcmp(x.regions[r].coefficient, y.regions[r].coefficient, sizeof(x.regions[r].coefficient));
        if (!valid) break;
        const double one[mix::kMaxNs] = {1, 0, 0, 0}, tc = l.aBinary[0][0] * mix::kOmB / (x.b * mix::kOmA * mix::kR),
                     pc = mix::kOmB * mix::kR * tc / x.b, W = x.molecularWeight;
        mix::PhaseLine line{};
        valid = mix::phaseLine(l, one, W, tc, pc, line) == mix::OK;
        const double rhoC = W * mix::kOmB / (mix::kOmVc * x.b);
        t.liquid[i] = MixLiquid{k, m.liquidTmin[i], m.liquidTc[i] * (1 - 1e-10), tc, rhoC,
                                (rhoC - line.midT) / (tc - line.tmid)};
    }
    t.valid = valid;
}

enum : int { RESIDUAL_UNDECIDED = -1, RESIDUAL_REJECTED = 0, RESIDUAL_OK = 1 };

RB200_HD_INLINE double polished(double x, double bn, double cn, double dn) {
    for (int it = 0; it < 12; ++it) {
        const double d = fma(fma(3.0, x, 2.0 * bn), x, cn);
        if (fabs(d) <= 1e-300) break;
        const double step = fma(fma(x + bn, x, cn), x, dn) / d;
        x -= step;
        if (fabs(step) <= 4e-15 * fmax(1.0, fabs(x))) break;
    }
    return x;
}

// The gas (largest) or liquid (smallest) root of the cubic at (T, p) by mix::roots'
// rules: rejected where that branch does not exist, undecided within a margin of
// the discriminant's bands, of the covolume, and of the side test of a lone root: its
// volume, or kNoBranch or kUndecidedBranch.
constexpr double kNoBranch = 0, kUndecidedBranch = -1;
static RB200_HD_CALL double branchRoot(double aa, double b, double T, double RT, double p, double tc, bool gas) {
    const double ip = 1.0 / p, RTp = RT * ip, aap = aa * ip, bn = b - RTp, b2 = b * b;
    const double cn = aap - 2.0 * RTp * b - 3.0 * b2, dn = b2 * (RTp + b) - aap * b;
    const double center = -bn * (1.0 / 3.0), delta2 = (bn * bn - 3.0 * cn) * (1.0 / 9.0);
    const double q = 2.0 / 27.0 * (bn * bn * bn) - bn * cn * (1.0 / 3.0) + dn;
    const double delta = delta2 > 0 ? sqrt(delta2) : 0.0, h = 2.0 * delta * delta2, disc = q * q - h * h;
    if (!(fabs(h - fabs(q)) >= fmax(4e-10, 1e-12 * fabs(q))) || !(fabs(disc) >= fmax(4e-14, 1e-12 * (q * q))))
        return kUndecidedBranch;
    bool lone = true;
    double V;
    if (disc > 0) {
        const double sd = .5 * sqrt(disc);
        V = center + cbrt(-.5 * q + sd) + cbrt(-.5 * q - sd);
    } else {
        double sn, cs;
        sincos(acos(fmin(1.0, fmax(-1.0, -.5 * q / (delta * delta2)))) * (1.0 / 3.0), &sn, &cs);
        const double dc = delta * cs, ds = 1.7320508075688772 * delta * sn, margin = 1e-9 * delta;
        const double low = center - dc - ds;
        V = center + 2.0 * dc;
        if (fabs(low - b) <= margin) return kUndecidedBranch;
        lone = low < b;  // the pressure rises without bound toward b: one or three roots above it
        if (lone && !(center - dc + ds < b - margin)) return kUndecidedBranch;
        if (!lone && !gas) V = low;
    }
    V = polished(V, bn, cn, dn);
    if (!(V > b)) return kUndecidedBranch;
    if (!lone || (gas && T > tc)) return V;
    const double side = T > tc ? b * (mix::kOmVc / mix::kOmB) : center;
    if (fabs(V - side) <= 1e-9 * V || fabs(T - tc) <= 1e-9 * tc) return kUndecidedBranch;
    return (V < side) != gas ? V : kNoBranch;
}

// One phase's terms at its root, false where the general evaluation rejects it.
struct MixPhase {
    double iv, id, L, e;  // e: molar energy
};
static RB200_HD_CALL bool phaseAt(double aa, double da, double d2a, double b, double T, double RT, double cpR,
                                        double hRT, double p, double V, MixPhase& o) {
    const double vmb = V - b, den = V * V + 2.0 * V * b - b * b;
    if (!(vmb > 0) || !(den > 0)) return false;
    o.iv = 1.0 / vmb;
    o.id = 1.0 / den;
    const double pe = RT * o.iv - aa * o.id, dpdV = 2.0 * aa * (V + b) * (o.id * o.id) - RT * (o.iv * o.iv);
    if (!(pe > 0) || !(dpdV < 0) || fabs(pe - p) > 1e-7 * fmax(1.0, p)) return false;
    o.L = log((V + (1.0 + mix::kRt2) * b) / (V + (1.0 - mix::kRt2) * b)) * (1.0 / (2.0 * mix::kRt2)) / b;
    o.e = RT * (hRT - 1.0) + o.L * (T * da - aa);
    const double cv = mix::kR * (cpR - 1.0) + o.L * T * d2a;  // cp > cv > 0 where dp/dV < 0
    return cv > 0 && fabs(o.e) <= DBL_MAX;
}

// The residual f of the active set at xe = (ln p, ln T, fractions) for a cell of
// partial densities q (finite, not negative, zero past the model's species) and
// energy density `energy`: as activeResidual.
//
// The gas's label: its density must lie below the line from the critical density
// (T = tc) through midT (T = tmid), midT = half the sum of the liquid and the ideal-gas
// density at tmid and some pressure > 0. The liquid root there is below the zero-pressure
// one, b v0 with v0 the smaller root of v^2 + (2 - A) v + A - 1, A = a(tmid)/(b R tmid)
// (real from A = 4 + 2 sqrt2; A >= 7.2 keeps clear of it), so midT >= W / (2 b v0): a
// density below the line through that bound is gas-like. Above it the liquid root is
// solved for, at the first pressure tried: from A = 4 + 2 sqrt2 the isotherm's liquid
// branch reaches down to p = 0, so the cubic there has three roots or a lone liquid one.
// A smaller A is undecided.
RB200_HD_INLINE int mixtureResidual(const MixTerms& t, const double* q, double energy, bool adaptive,
                                               double gasOffset, double liquidOffset, double pmin, double pmax,
                                               double Tmin, double Tmax, const int* active, int n, const double* xe,
                                               double scale, double* f, unsigned long long& phases) {
    constexpr int K = mix::kMaxNs;
    double gas[K], mass[2] = {0, 0};
#pragma unroll
    for (int k = 0; k < K; ++k) gas[k] = q[k];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        if (j >= n) continue;
        const int s = t.liquid[active[j]].species;
        const double y = xe[2 + j];
        double whole = 0, vapor, liquid;
#pragma unroll
        for (int k = 0; k < K; ++k) whole = k == s ? q[k] : whole;
        if (adaptive) {
            if (!(y <= 0) || !(y >= -DBL_MAX)) return RESIDUAL_REJECTED;
            vapor = exp(y) * whole;
            if (!(vapor > 0)) return RESIDUAL_REJECTED;
            liquid = -expm1(y) * whole;
        } else {
            if (!(y >= 0 && y < 1)) return RESIDUAL_REJECTED;
            liquid = y * whole;
            vapor = whole - liquid;
        }
#pragma unroll
        for (int k = 0; k < K; ++k) gas[k] = k == s ? vapor : gas[k];
        if (active[j] == 0) mass[0] = liquid; else mass[1] = liquid;
    }
    const double p = exp(xe[0]), T = exp(xe[1]), pg = p - gasOffset, pl = p + liquidOffset;
    auto inside = [&](double pressure) { return pressure >= pmin && pressure <= pmax && T >= Tmin && T <= Tmax; };
    if (!inside(p)) return RESIDUAL_REJECTED;
    double mg = 0, moles = 0, x[K];
#pragma unroll
    for (int k = 0; k < K; ++k) mg += gas[k];
    if (!(mg > 0)) return RESIDUAL_REJECTED;
    ++phases;
    if (!inside(pg)) return RESIDUAL_REJECTED;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (t.bounds && gas[k] > 0 && (T < t.sp[k].Tlo || T > t.sp[k].Thi)) return RESIDUAL_REJECTED;
        x[k] = gas[k] * t.sp[k].invW;
        moles += x[k];
    }
    const double iN = 1.0 / moles, W = mg * iN, iT = 1.0 / T, RT = mix::kR * T;
    double alpha[K], dAlpha[K], cpR[K], hRT[K], b = 0, gasCp = 0, gasH = 0;
    RB200_ROLLED
    for (int k = 0; k < K; ++k) {
        const MixSpecies& s = t.sp[k];
        x[k] *= iN;
        const double root = sqrt(T * s.invTc), g = s.kappaPlus1 - s.kappa * root;
        if (fabs(g) <= 1e-14) return RESIDUAL_REJECTED;
        const double half = .5 * s.kappa * root * iT;
        alpha[k] = fabs(g);
        dAlpha[k] = g > 0 ? -half : half;
        int r = 0;
        for (int j = 1; j < s.regions && T >= s.from[j]; ++j) r = j;
        const MixRegion& c = s.region[r];
        cpR[k] = fma(T, fma(T, fma(T, fma(T, c.c4, c.c3), c.c2), c.c1), fma(fma(c.m2, iT, c.m1), iT, c.c0));
        hRT[k] = fma(T, fma(T, fma(T, fma(T, c.h4, c.h3), c.h2), c.h1), fma(c.hc + c.m1 * xe[1] - c.m2 * iT, iT, c.c0));
        b = fma(x[k], s.b, b);
        gasCp = fma(x[k], cpR[k], gasCp);
        gasH = fma(x[k], hRT[k], gasH);
    }
    double aa = 0, da = 0, d2a = 0, a = 0, row[K];
    RB200_ROLLED
    for (int k = 0; k < K; ++k) {
        double plain = 0, sum = 0, slope = 0;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const double w = t.a[k][j] * x[j];
            plain += w;
            sum = fma(w, alpha[j], sum);
            slope = fma(w, dAlpha[j], slope);
        }
        row[k] = sum;
        a = fma(x[k], plain, a);
        aa = fma(x[k], alpha[k] * sum, aa);
        da = fma(x[k], dAlpha[k] * sum, da);
        d2a = fma(x[k], dAlpha[k] * slope, d2a);
    }
    da *= 2.0;
    d2a = 2.0 * d2a - .5 * iT * da;  // alpha'' = -alpha' / 2T
    if (!(a > 0) || !(b > 0) || !(aa > 0)) return RESIDUAL_REJECTED;
    const double ib = 1.0 / b, tc = a * ib * (mix::kOmB / (mix::kOmA * mix::kR));
    MixPhase g;
    const double V = branchRoot(aa, b, T, RT, pg, tc, true);
    if (!(V > 0)) return V == kNoBranch ? RESIDUAL_REJECTED : RESIDUAL_UNDECIDED;
    if (!phaseAt(aa, da, d2a, b, T, RT, gasCp, gasH, pg, V, g)) return RESIDUAL_REJECTED;
    if (!(T >= tc)) {
        const double tmid = tc - 100.0 < 0 ? .5 * tc : tc - 100.0;
        double middle = 0, am[K];
        RB200_ROLLED
        for (int k = 0; k < K; ++k)
            am[k] = x[k] * fabs(t.sp[k].kappaPlus1 - t.sp[k].kappa * sqrt(tmid * t.sp[k].invTc));
        RB200_ROLLED
        for (int k = 0; k < K; ++k) {
            double sum = 0;
#pragma unroll
            for (int j = 0; j < K; ++j) sum = fma(t.a[k][j], am[j], sum);
            middle = fma(am[k], sum, middle);
        }
        const double A = middle * ib / (mix::kR * tmid);
        if (!(A >= 7.2)) return RESIDUAL_UNDECIDED;
        const double v0 = .5 * ((A - 2.0) - sqrt((A - 8.0) * A + 8.0));
        const double rhoC = mix::kOmB / mix::kOmVc, low = rhoC + (tc - T) / (tc - tmid) * (.5 / v0 - rhoC);
        if (!(b < low * (1 - 1e-9) * V)) {  // densities over W / b
            const double ratio = tc / tmid, pc = mix::kOmB * mix::kR * tc * ib;
            const double pp = pc * exp(-.8734 * ratio * ratio - 3.4522 * ratio + 4.2918);
            const double Vm = branchRoot(middle, b, tmid, mix::kR * tmid, pp, tc, false);
            if (!(Vm > 0)) return RESIDUAL_UNDECIDED;
            const double mid = .5 * b * (1.0 / Vm + pp / (mix::kR * tmid));
            const double line = (rhoC + (tc - T) / (tc - tmid) * (mid - rhoC)) * V;
            if (fabs(line - b) <= 1e-9 * b) return RESIDUAL_UNDECIDED;
            if (!(b < line)) return RESIDUAL_REJECTED;
        }
    }
    double volume = moles * V, content = moles * g.e;
    f[0] = f[1] = f[2] = f[3] = 0;
    RB200_ROLLED
    for (int i = 0; i < t.nl; ++i) {
        const MixLiquid& l = t.liquid[i];
        const int k = l.species;
        const double whole = q[k], al = alpha[k], dl = dAlpha[k], cl = cpR[k], hl = hRT[k], xk = x[k], sk = al * row[k],
                     bk = t.sp[k].b, akk = t.a[k][k], invW = t.sp[k].invW;
        const bool is = (n > 0 && active[0] == i) || (n > 1 && active[1] == i);
        if (!(whole > 0)) {
            if (is) return RESIDUAL_UNDECIDED;
            continue;
        }
        ++phases;
        if (!inside(pl) || T < l.Tmin) return RESIDUAL_REJECTED;
        if (T >= l.Tend) {
            if (is) return RESIDUAL_REJECTED;
            continue;
        }
        const double laa = akk * (al * al), lda = 2.0 * akk * (al * dl), ld2a = 2.0 * akk * (dl * dl) - .5 * iT * lda;
        MixPhase liquid;
        const double Vl = branchRoot(laa, bk, T, RT, pl, l.tcLine, false);
        if (Vl == kUndecidedBranch) return RESIDUAL_UNDECIDED;
        bool there = Vl != kNoBranch;
        if (there) {
            if (!phaseAt(laa, lda, ld2a, bk, T, RT, cl, hl, pl, Vl, liquid)) return RESIDUAL_REJECTED;
            const double line = (l.rhoC + (T - l.tcLine) * l.lineSlope) * invW * Vl;  // the line's density over the liquid's
            if (fabs(line - 1.0) <= 1e-9 || fabs(T - l.tcLine) <= 1e-9 * T) return RESIDUAL_UNDECIDED;
            there = T < l.tcLine && line < 1.0;
        }
        if (!is) continue;
        if (!there) return RESIDUAL_REJECTED;
        const double affinity = log(liquid.iv / (g.iv * fmax(1e-300, xk))) + bk * (liquid.iv - g.iv)
                              + ((g.L * (2.0 * sk - aa * bk * ib) + aa * bk * V * g.id * ib)
                                 - laa * (liquid.L + Vl * liquid.id)) / RT;
        if (!(fabs(affinity) <= DBL_MAX)) return RESIDUAL_REJECTED;
        if (n > 1 && active[1] == i) f[3] = affinity; else f[2] = affinity;
        const double m = mass[i];
        if (m > 0) {
            volume += m * invW * Vl;
            content += m * invW * liquid.e;
        }
    }
    f[0] = volume - 1;
    f[1] = (content - energy) / scale;
    return fabs(f[0]) <= DBL_MAX && fabs(f[1]) <= DBL_MAX ? RESIDUAL_OK : RESIDUAL_REJECTED;
}

}  // namespace rb200
