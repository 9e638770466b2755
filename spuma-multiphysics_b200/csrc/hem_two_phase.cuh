// The two-phase Newton of a pure fluid (one species' tables for both phases) in
// registers: the candidates of hem_flash.cuh's twoPhaseSolve, the same unknowns
// (ln p, ln T, beta), residuals, Jacobian, limiter, line search and tests, with
// each evaluation reduced to what an iteration reads.
//
// An iteration needs both roots' volumes, energies, enthalpies and pressure and
// temperature derivatives, and the difference of their chemical potentials:
//   (mu_l - mu_g)/RT = ln(iv_l/iv_g) + b (iv_l - iv_g)
//                      - (a alpha/RT) ((L_l + V_l id_l) - (L_g + V_g id_g))
// (iv = 1/(V - b), id = 1/(V^2 + 2bV - b^2), L the attraction logarithm over
// 2 sqrt2 b), in which the ideal-gas terms cancel: no entropy, no ln T and one
// logarithm for two. cv and the sound speed, which the general evaluation checks
// every time, are positive sums of positive phase terms here (each phase has
// cv > 0 and dp/dV < 0) and are formed once, for the converged state. The middle
// root of the cubic is not polished. That leaves 15 divisions and 3 logarithms of
// 37 and 5, and the iteration's state in registers instead of the work queue's
// lane record on the stack: 1,000,000 cells, 60% saturated, take 3.3 ms for their
// two-phase candidates (the 40^3 step went from 1.49 to 1.11 ms, 1.09 with both roots'
// chains interleaved).
#pragma once
#include "hem_flash.cuh"

namespace rb200 {

struct PhaseTerms {
    double V, iv, id, L, eM, hM, cpM, vp, vt;  // molar; vp, vt = dV/dp, dV/dT
};
struct TwoPhasePoint {
    double p, T, RT, da;
    PhaseTerms gas, liq;
    double f0, f1, f2, lnIv;  // residuals; ln(iv_l / iv_g)
    double gasMass, liqMass, Vp, VT, Ep, ET, energy, cpD, volume;
};

// polishRoot of two roots at once: their steps are independent chains, which one
// thread's instructions then interleave. Each stops moving at its own last step.
__device__ __forceinline__ void polishPair(double& x, double& y, double bn, double cn, double dn) {
    bool moveX = true, moveY = true;
    for (int n = 0; n < 12 && (moveX || moveY); ++n) {
        const double fx = cubicAt(x, bn, cn, dn), dx = (3.0 * x + 2.0 * bn) * x + cn;
        const double fy = cubicAt(y, bn, cn, dn), dy = (3.0 * y + 2.0 * bn) * y + cn;
        const double sx = fx / dx, sy = fy / dy;
        moveX = moveX && fabs(dx) > 1e-300;
        moveY = moveY && fabs(dy) > 1e-300;
        x -= moveX ? sx : 0.0;
        y -= moveY ? sy : 0.0;
        moveX = moveX && !(fabs(sx) <= 4e-15 * fmax(1.0, fabs(x)));
        moveY = moveY && !(fabs(sy) <= 4e-15 * fmax(1.0, fabs(y)));
    }
}

// One root's terms at (T, p), false where the general evaluation rejects it (the
// terms of a rejected root are not read; no branch, so two roots' chains interleave).
__device__ __forceinline__ bool phaseTerms(const PureSpecies& sp, double T, double RT, double aa, double da, double d2a,
                                           double cpR, double hRT, double p, double V, bool gas, PhaseTerms& o) {
    const double b = sp.b, vmb = V - b, den = V * V + sp.twoB * V - sp.bb;
    o.V = V;
    o.iv = 1.0 / vmb;
    o.id = 1.0 / den;
    const double pe = RT * o.iv - aa * o.id;
    const double dpdV = 2.0 * aa * (V + b) * (o.id * o.id) - RT * (o.iv * o.iv), dpdT = kGas * o.iv - da * o.id;
    o.L = log((V + sp.covolumeHi) / (V + sp.covolumeLo)) * sp.invL;
    o.eM = RT * (hRT - 1.0) + o.L * (T * da - aa);
    o.hM = o.eM + pe * V;
    const double cvM = kGas * (cpR - 1.0) + o.L * T * d2a, idp = 1.0 / dpdV;
    o.vp = idp;
    o.vt = -dpdT * idp;
    o.cpM = cvM + T * dpdT * o.vt;
    const bool side = T >= sp.tcLine ? gas : (sp.W < (sp.rhoC + (T - sp.tcLine) * sp.lineSlope) * V) == gas;
    return vmb > 0 && den > 0 && pe > 0 && dpdV < 0 && !(fabs(pe - p) > 1e-7 * fmax(1.0, p)) && side && cvM > 0
           && fin(o.cpM) && fin(o.eM);
}

// Evaluation of the residuals (and their ingredients) at x = (ln p, ln T, beta).
__device__ __forceinline__ bool twoPhasePoint(const HemConst& C, const PureSpecies& sp, double q, double e, double scale,
                                              double lp, double lT, double beta, TwoPhasePoint& o) {
    if (!(beta >= 0 && beta < 1)) return false;
    const double p = exp(lp), T = exp(lT), mass = beta * q, gasMass = q - mass;
    if (!inBounds(C, p, T) || !(q > 0) || !fin(q) || !(gasMass > 0)) return false;
    if (C.enforceBounds && (T < C.gasTmin || T > C.gasTmax)) return false;
    if (T < C.liquidTmin || T >= C.liquidTc * (1 - 1e-10)) return false;
    const double iT = 1.0 / T, root = sqrt(T * sp.invTc), f = sp.kappaPlus1 - sp.kappa * root;
    if (fabs(f) <= 1e-14) return false;
    const double a = fabs(f), half = .5 * sp.kappa * (root * iT), df = f > 0 ? -half : half;
    const double aa = sp.a * (a * a), da = sp.twoA * (a * df), d2a = sp.twoA * (df * df - .5 * df * iT * a);
    const double RT = kGas * T;
    const NasaPowers& n = sp.powers[nasaRegion(sp, T)];
    double cpR = n.c0 + T * (n.c1 + T * (n.c2 + T * (n.c3 + T * n.c4)));
    double hRT = n.c0 + n.hc * iT + T * (n.h1 + T * (n.h2 + T * (n.h3 + T * n.h4)));
    if (n.m1 != 0 || n.m2 != 0) {
        cpR += (n.m2 * iT + n.m1) * iT;
        hRT += (n.m1 * lT - n.m2 * iT) * iT;
    }
    // the cubic: two phases need two physical roots, so three real ones
    const double ip = 1.0 / p, b = sp.b, RTp = RT * ip, aap = aa * ip, bn = b - RTp;
    const double cn = -(2.0 * RTp * b - aap + 3.0 * sp.bb), dn = sp.bb * RTp + sp.bb * b - aap * b;
    const double center = -bn * kThird, delta2 = (bn * bn - 3.0 * cn) * (1.0 / 9.0);
    const double qc = 2.0 * bn * bn * bn * (1.0 / 27.0) - bn * cn * kThird + dn;
    if (!(delta2 > 0)) return false;
    const double delta = sqrt(delta2), h = 2.0 * delta * delta2;
    if (fabs(fabs(h) - fabs(qc)) < 1e-10 || !(qc * qc - h * h < -1e-14)) return false;
    double sn, cs;
    sincos(acos(fmin(1.0, fmax(-1.0, -.5 * qc / (delta * delta2)))) * kThird, &sn, &cs);
    const double dc = delta * cs, ds = 1.7320508075688772 * delta * sn;
    double hi = center + 2.0 * dc, lo = center - dc - ds;
    polishPair(hi, lo, bn, cn, dn);
    if (!(lo > b)) lo = polishRoot(center - dc + ds, bn, cn, dn);  // the liquid-like root of two
    if (!(lo > b) || !(hi > lo) || !fin(hi)) return false;
    const bool gasOk = phaseTerms(sp, T, RT, aa, da, d2a, cpR, hRT, p, hi, true, o.gas);
    const bool liqOk = phaseTerms(sp, T, RT, aa, da, d2a, cpR, hRT, p, lo, false, o.liq);
    if (!gasOk || !liqOk) return false;
    o.p = p;
    o.T = T;
    o.RT = RT;
    o.da = da;
    o.gasMass = gasMass;
    o.liqMass = mass;
    const double ng = gasMass * sp.invW, nl = mass * sp.invW;
    o.volume = ng * o.gas.V + nl * o.liq.V;
    o.energy = ng * o.gas.eM + nl * o.liq.eM;
    o.Vp = ng * o.gas.vp + nl * o.liq.vp;
    o.VT = ng * o.gas.vt + nl * o.liq.vt;
    o.cpD = ng * o.gas.cpM + nl * o.liq.cpM;
    o.Ep = -T * o.VT - p * o.Vp;
    o.ET = o.cpD - p * o.VT;
    o.lnIv = log(o.liq.iv / o.gas.iv);
    o.f0 = o.volume - 1;
    o.f1 = (o.energy - e) / scale;
    o.f2 = o.lnIv + b * (o.liq.iv - o.gas.iv)
         - aa / RT * ((o.liq.L + o.liq.V * o.liq.id) - (o.gas.L + o.gas.V * o.gas.id));
    return fin(o.f0) && fin(o.f1) && fin(o.f2);
}

// A two-phase solve: its iterate, its step and the trial in hand.
struct TwoPhaseSolve {
    double q, e, scale, x0, x1, x2, s0, s1, s2, previous, fraction;
    int it, k;
    bool first;
};
enum : int { TP_RUNNING, TP_FAILED, TP_CONVERGED };

// The start from a beta seed (seed < 0: the previous state's liquid fraction);
// restartT >= 0 replaces the seed T.
__device__ __forceinline__ void twoPhaseStart(const HemConst& C, const CellInput& in, double seed, double restartT,
                                              TwoPhaseSolve& s) {
    const double gT = restartT >= 0 ? restartT : in.gT;
    s.q = in.q;
    s.e = in.e;
    s.scale = fmax(1e5 * in.q, fmax(fabs(in.e), in.q * 2000 * fmax(gT, C.Tmin)));
    s.x0 = log(clampd(in.gp, C.pmin, C.pmax));
    s.x1 = log(clampd(gT, C.Tmin, C.Tmax));
    s.x2 = seed < 0 ? clampd(in.gml / in.q, 1e-8, 1 - 1e-8) : seed;
    s.s0 = s.s1 = s.s2 = 0;
    s.previous = 0;
    s.fraction = 1;
    s.it = s.k = 0;
    s.first = true;
}

// d(f0, f1, f2)/d(ln p, ln T, beta) at an evaluated point.
__device__ __forceinline__ bool twoPhaseJacobian(const PureSpecies& sp, const TwoPhaseSolve& s, const TwoPhasePoint& o,
                                                 double J[3][3], Counts& n) {
    ++n.analytic;
    const double is = 1.0 / s.scale, iRT = 1.0 / o.RT, dV = o.liq.V - o.gas.V, molar = s.q * sp.invW;
    J[0][0] = o.Vp * o.p;
    J[0][1] = o.VT * o.T;
    J[0][2] = molar * dV;
    J[1][0] = o.Ep * o.p * is;
    J[1][1] = o.ET * o.T * is;
    J[1][2] = molar * (o.liq.eM - o.gas.eM) * is;
    J[2][0] = o.p * dV * iRT;
    J[2][1] = -(o.liq.hM - o.gas.hM) * iRT;
    J[2][2] = 0;
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) ok = ok && fin(J[i][j]);
    return ok;
}

// Takes the evaluation `o` (ok) of the solve's current trial and sets the next one,
// or ends the solve.
__device__ __forceinline__ int twoPhaseAdvance(const HemConst& C, const PureSpecies& sp, TwoPhaseSolve& s, bool ok,
                                               const TwoPhasePoint& o, Counts& n) {
    if (s.first) {
        if (!ok) return TP_FAILED;
        s.first = false;
    } else {
        const double largest = fmax(fabs(o.f0), fmax(fabs(o.f1), fabs(o.f2)));
        if (!(ok && largest < s.previous * (1 - 1e-4 * s.fraction))) {
            ++s.k;
            s.fraction *= .5;
            while (s.k < 30 && !(s.x2 + s.fraction * s.s2 >= 0 && s.x2 + s.fraction * s.s2 < 1)) {
                ++n.residuals;
                ++s.k;
                s.fraction *= .5;
            }
            return s.k < 30 ? TP_RUNNING : TP_FAILED;
        }
        s.x0 += s.fraction * s.s0;
        s.x1 += s.fraction * s.s1;
        s.x2 += s.fraction * s.s2;
        if (++s.it >= 90) return TP_FAILED;
    }
    if (fabs(o.f0) <= C.vtol && fabs(o.f1) <= C.etol && fabs(o.f2) <= C.mutol) return TP_CONVERGED;
    double J[3][3], rhs[3] = {-o.f0, -o.f1, -o.f2}, step[3] = {0, 0, 0};
    if (!twoPhaseJacobian(sp, s, o, J, n) || !solveSmallBody(J, rhs, 3, step)) return TP_FAILED;
    const double limiter = fmax(fmax(1., fmax(fabs(step[0]) / .7, fabs(step[1]) / .18)), fabs(step[2]) / .3);
    const double shorten = 1.0 / limiter;
    s.s0 = step[0] * shorten;
    s.s1 = step[1] * shorten;
    s.s2 = step[2] * shorten;
    s.previous = fmax(fabs(o.f0), fmax(fabs(o.f1), fabs(o.f2)));
    s.k = 0;
    s.fraction = 1;
    while (s.k < 30 && !(s.x2 + s.fraction * s.s2 >= 0 && s.x2 + s.fraction * s.s2 < 1)) {
        ++n.residuals;
        ++s.k;
        s.fraction *= .5;
    }
    return s.k < 30 ? TP_RUNNING : TP_FAILED;
}

// A converged solve's state, entropy density and stability; false where the
// equilibrium sound speed rejects it. stable: the affinity of the converged point
// (the point the stability test evaluates).
__device__ __forceinline__ bool twoPhaseState(const HemConst& C, const PureSpecies& sp, const TwoPhaseSolve& s,
                                              const TwoPhasePoint& o, ReactiveThermoState& st, double& entropyD,
                                              bool& stable, Counts& n) {
    double J[3][3], rhs[3] = {-1 / s.q, o.p / (s.q * s.scale), 0}, response[3] = {0, 0, 0};
    if (!twoPhaseJacobian(sp, s, o, J, n) || !solveSmallBody(J, rhs, 3, response)) return false;
    const double squared = o.p * response[0];
    if (!fin(squared) || squared <= 0) return false;
    const double T = o.T, q = s.q, ng = o.gasMass * sp.invW, nl = o.liqMass * sp.invW;
    GasProbe probe;  // for the ideal gas' entropy
    probe.T = T;
    probe.iT = 1.0 / T;
    probe.lnT = log(T);
    const double sR = probeEntropy(sp, probe), lg = log(o.RT * o.gas.iv * sp.invRefP);
    entropyD = ng * (kGas * (sR - lg) + o.gas.L * o.da) + nl * (kGas * (sR - (lg + o.lnIv)) + o.liq.L * o.da);
    Eval v{};
    v.p = o.p;
    v.T = T;
    v.gasMass = o.gasMass;
    v.liqMass = o.liqMass;
    v.volume = o.volume;
    v.energy = o.energy;
    v.entropyD = entropyD;
    v.cpD = o.cpD;
    v.gRho = sp.W / o.gas.V;
    v.lRho = sp.W / o.liq.V;
    const double cp = o.cpD / q, specific = o.volume / q, vp = o.Vp / q, vt = o.VT / q;
    v.cv = (o.cpD + T * o.VT * o.VT / o.Vp) / q;
    const double adiabatic = vp + T * vt * vt / cp;
    if (!fin(v.cv) || v.cv <= 0 || !(adiabatic < 0)) return false;
    v.soundFrozen = sqrt(-specific * specific / adiabatic);
    CandidateOut out{fabs(o.f0), fabs(o.f1), fabs(o.f2), sqrt(squared), s.it};
    if (!fin(v.soundFrozen) || !(v.soundFrozen > 0) || !fin(entropyD) || !(out.soundEq <= v.soundFrozen * (1 + 2e-3)))
        return false;
    stateFromEval(v, q, out, st);
    stable = o.liqMass > 0 ? fabs(o.f2) <= C.mutol * 2 : !(o.f2 < -C.mutol);
    return true;
}

}  // namespace rb200
