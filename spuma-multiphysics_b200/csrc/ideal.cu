// Ideal-gas mixture closure on the device and its vector-Jacobian product.
//
// Recovery per cell follows the reference's scalar closure for pr = 0
// (src/reactiveTransport/reactiveClosureScalar.cuh:9-57): e(T) = h(T) - r T,
// cv(T) = cp(T) - r and p = rho r T from NASA polynomials; starting at the seed
// temperature, a bracket widened by doubling radii (at most 24) around the
// seed, then at most 70 Newton steps T - F/cv kept inside the bracket (else
// bisection), stopping when |F| <= .25 tol max(1e5, cp T). Here the mixture's
// h, cp and r are sums over the species' own NASA regions weighted by the mass
// fractions of the cell (the reference premixes the coefficients of one NASA
// interval on the host), and the frozen sound speed is c^2 = (cp/cv) r T.
#include "pr_eos.cuh"
#include "dual.cuh"
#include "common.cuh"
#include "../../include/reactive_b200_ideal.h"

#include <cmath>
#include <cstring>
#include <memory>
#include <string>

namespace rb200 {
namespace {

constexpr int kIdealMaxSpecies = 4;

struct IdealConst {
    int ns, logs;  // logs: some species' polynomials have the 1/T terms, which read ln T
    double r[kIdealMaxSpecies];  // R / W_k, J/(kg K)
    PureSpecies sp[kIdealMaxSpecies];
    double Tmin, Tmax, tol;
};

// cp/R and h/RT of species k at T (iT = 1/T).
__device__ __forceinline__ void speciesTerms(const PureSpecies& sp, double T, double iT, double& cpR, double& hRT) {
    const NasaPowers& n = sp.powers[nasaRegion(sp, T)];
    cpR = n.c0 + T * (n.c1 + T * (n.c2 + T * (n.c3 + T * n.c4)));
    hRT = n.c0 + n.hc * iT + T * (n.h1 + T * (n.h2 + T * (n.h3 + T * n.h4)));
    if (n.m1 != 0 || n.m2 != 0) {  // only these terms read ln T
        cpR += (n.m2 * iT + n.m1) * iT;
        hRT += (n.m1 * log(T) - n.m2 * iT) * iT;
    }
}

// Energy residual F = rho e(T) - energy and rho cv(T) of the partial densities q
// (qr: each times its gas constant), per volume. The formation energies are as large as
// a hundred times rho cv dT of interest, so they meet the energy they cancel against
// first, in fused multiply-adds of the unrounded partial densities.
template <int NS>
__device__ __forceinline__ void mixture(const IdealConst& G, const double* q, const double* qr, double energy, double T,
                                        double& F, double& cv) {
    double thermal = 0, iT = 0, lT = 0;
    if (G.logs) {
        iT = 1 / T;
        lT = log(T);
    }
    F = -energy;
    cv = 0;
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const NasaPowers& n = G.sp[k].powers[nasaRegion(G.sp[k], T)];
        F = fma(q[k], G.r[k] * n.hc, F);
        thermal += qr[k] * (T * (n.c0 - 1 + T * (n.h1 + T * (n.h2 + T * (n.h3 + T * n.h4)))) + (n.m1 * lT - n.m2 * iT));
        cv += qr[k] * (n.c0 - 1 + T * (n.c1 + T * (n.c2 + T * (n.c3 + T * n.c4))) + (n.m2 * iT + n.m1) * iT);
    }
    F += thermal;
}

__device__ inline bool inRange(const IdealConst& G, double T) { return T >= G.Tmin && T <= G.Tmax && T > 0; }

// The reference's recovery of T from e(T) = e: bracket, then safeguarded Newton.
template <int NS>
__device__ bool bracketedT(const IdealConst& G, const double* q, const double* qr, double energy, double T0, double F0,
                           double tolerance, double& T, double& cv, double& F) {
    T = T0;
    F = F0;
    double lo = T, hi = T, fl = F0, fh = F0, radius = fmax(1., .01 * T);
    for (int j = 0; j < 24 && fabs(F) > tolerance && (fl > 0 || fh < 0); ++j, radius *= 2) {
        double slope;
        if (fl > 0) { lo = fmax(G.Tmin, T0 - radius); mixture<NS>(G, q, qr, energy, lo, fl, slope); }
        if (fh < 0) { hi = fmin(G.Tmax, T0 + radius); mixture<NS>(G, q, qr, energy, hi, fh, slope); }
    }
    bool ok = fabs(F) <= tolerance || (fl <= 0 && fh >= 0 && hi > lo);
    for (int it = 0; ok && it < 70 && fabs(F) > tolerance; ++it) {
        if (F > 0) hi = T; else lo = T;
        const double next = T - F / cv;
        T = isfinite(next) && next > lo && next < hi ? next : .5 * (lo + hi);
        mixture<NS>(G, q, qr, energy, T, F, cv);
    }
    return ok && fabs(F) <= tolerance;
}

// Bound by the latency of the Newton's dependent FP64 chain (each e(T) needs the one
// before it) and by issue. The bracket's probes only confine the Newton steps, and e
// rises with T (cv > 0): whatever the steps, the solution is the same. So the Newton
// runs without them, kept between the iterates that lie on either side of the solution:
// a step past the range's end goes to that end, which ends the search where the solution
// lies beyond it, and one past an iterate to the middle. Only an iterate with cv <= 0, or
// 70 of them, go back to the bracketed form. At the usual few per cent off the seed that
// leaves four evaluations of seven to ten (64^3 two-species box: 24 us a call). Seeds
// far off, 300 K for solutions between 160 and 2,900 K, 262,144 cells of two species:
// 154 us with the bracket first, 191 with it after a Newton that had left it, 45 so.
//
// The accepted iterate takes the Newton step of the residual it was accepted with, at
// no further evaluation. Acceptance is |F| <= .25 tol max(1e5 rho, rho cp T), so that step
// is at most .25 tol max(1e5, cp T) / cv (at IdealGasBox's tol of 1e-13: 4e-14 of T where
// cp T is above 1e5), and by the Newton's quadratic convergence it leaves an error of the
// order of its own relative size squared: T is the solution to round-off, and a smooth
// function of q, for tol below 1e-8, and better than tol for any.
template <int NS>
__global__ void __launch_bounds__(128) idealClosure(const IdealConst* __restrict__ Gp, const double* __restrict__ q,
                                                    size_t stride, size_t count, const double* Tseed, double* Tout,
                                                    ReactiveTransportState* transport, int* success) {
    const IdealConst& G = *Gp;
    for (size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x; c < count; c += size_t(blockDim.x) * gridDim.x) {
        double rho = 0, y[NS], yr[NS], gas = 0;  // partial densities, times the gas constants, their sum
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            rho += y[k] = q[size_t(k) * stride + c];
            gas += yr[k] = y[k] * G.r[k];
        }
        const double mx = q[size_t(NS) * stride + c], my = q[size_t(NS + 1) * stride + c],
                     mz = q[size_t(NS + 2) * stride + c], E = q[size_t(NS + 3) * stride + c];
        const double energy = E - .5 * (mx * mx + my * my + mz * mz) / rho;
        const double T0 = Tseed[c];
        bool ok = isfinite(rho) && rho > 0 && isfinite(energy) && inRange(G, T0);
        double T = T0, cv = 0;
        if (ok) {
            double F;
            mixture<NS>(G, y, yr, energy, T, F, cv);
            const double tolerance = .25 * G.tol * fmax(1e5 * rho, (cv + gas) * T), F0 = F, cv0 = cv;
            double lo = G.Tmin, hi = G.Tmax;
            bool below = false, above = false;  // lo, hi are iterates
            for (int it = 0; cv > 0 && it < 70 && fabs(F) > tolerance; ++it) {
                if (F > 0) { hi = T; above = true; } else { lo = T; below = true; }
                double next = T - F / cv;
                if (!(next < hi)) next = above ? .5 * (lo + hi) : G.Tmax;
                else if (!(next > lo)) next = below ? .5 * (lo + hi) : G.Tmin;
                if (next == T) break;
                T = next;
                mixture<NS>(G, y, yr, energy, T, F, cv);
            }
            ok = cv > 0 && fabs(F) <= tolerance;
            const bool beyond = cv > 0 && ((T == G.Tmax && F < 0) || (T == G.Tmin && F > 0));
            if (!ok && !beyond) {
                cv = cv0;
                ok = bracketedT<NS>(G, y, yr, energy, T0, F0, tolerance, T, cv, F);
            }
            ok = ok && cv > 0;
            if (ok) T = fmin(fmax(T - F / cv, G.Tmin), G.Tmax);
        }
        if (success) success[c] = ok ? 1 : 0;
        if (!ok) continue;
        const double p = gas * T, iRho = 1 / rho;
        const double sound = sqrt((cv + gas) / cv * (p * iRho));
        Tout[c] = T;
        transport[c] = ReactiveTransportState{p, T, rho, cv * iRho, sound, rho, 0.0};
    }
}

// d(state fields)/dq by forward-mode duals seeded on the cell's conserved
// variables; T's derivative by the implicit function theorem on
// f(T, q) = e(T, Y(q)) - e(q) = 0: dT/dq = -(df/dq) / cv.
template <int NS>
__global__ void idealClosureVjp(const IdealConst* __restrict__ Gp, const double* __restrict__ q, size_t stride,
                                size_t count, const double* __restrict__ Tconv,
                                const ReactiveTransportState* __restrict__ bar, double* qBar, size_t barStride) {
    constexpr int N = NS + 4;
    using D = Dual<N>;
    const IdealConst& G = *Gp;
    for (size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x; c < count; c += size_t(blockDim.x) * gridDim.x) {
        D qd[N];
#pragma unroll
        for (int k = 0; k < N; ++k) qd[k] = D::seed(q[size_t(k) * stride + c], k);
        D rho(0.0);
#pragma unroll
        for (int k = 0; k < NS; ++k) rho += qd[k];
        D Y[NS];
#pragma unroll
        for (int k = 0; k < NS; ++k) Y[k] = qd[k] / rho;
        const D m2 = qd[NS] * qd[NS] + qd[NS + 1] * qd[NS + 1] + qd[NS + 2] * qd[NS + 2];
        const D eIn = (qd[NS + 3] - D(.5) * m2 / rho) / rho;
        const double T = Tconv[c];
        // species terms at the converged T (constants), mixed with dual Y
        D e(0.0), cv(0.0), r(0.0);
        double cvSlope = 0, cvv = 0;
        const double iT = 1 / T;
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            double cpR, hRT;
            speciesTerms(G.sp[k], T, iT, cpR, hRT);
            const NasaPowers& n = G.sp[k].powers[nasaRegion(G.sp[k], T)];
            cvv += Y[k].v * G.r[k] * (cpR - 1);
            cvSlope += Y[k].v * G.r[k] * (n.c1 + T * (2 * n.c2 + T * (3 * n.c3 + T * 4 * n.c4))
                                          - (2 * n.m2 * iT + n.m1) * iT * iT);
            e += Y[k] * D(G.r[k] * T * (hRT - 1));
            cv += Y[k] * D(G.r[k] * (cpR - 1));
            r += Y[k] * D(G.r[k]);
        }
        const D f = e - eIn;
        D Td(T);
#pragma unroll
        for (int i = 0; i < N; ++i) Td.d[i] = -f.d[i] / cvv;
        // cv also moves with T
#pragma unroll
        for (int i = 0; i < N; ++i) cv.d[i] += cvSlope * Td.d[i];
        const D p = rho * r * Td;
        const D sound = sqrt((cv + r) / cv * r * Td);
        const ReactiveTransportState b = bar[c];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const double g = b.p * p.d[k] + b.T * Td.d[k] + b.rho * rho.d[k] + b.cv * cv.d[k] + b.sound * sound.d[k]
                + b.gasMass * rho.d[k];
            qBar[size_t(k) * barStride + c] += g;
        }
    }
}

struct IdealDevice {
    int device = 0;
    IdealConst host{};
    IdealConst* dev = nullptr;
    ~IdealDevice() { if (dev) cudaFree(dev); }
};

std::string speciesFromTable(const ReactiveB200Species& s, PureSpecies& sp) {
    if (!(std::isfinite(s.molecularWeight) && s.molecularWeight > 0) || s.regionCount < 1
        || s.regionCount > kMaxRegions)
        return "Invalid ideal-gas species data";
    std::memset(&sp, 0, sizeof(sp));
    sp.W = s.molecularWeight;
    sp.regionCount = s.regionCount;
    for (int r = 0; r < s.regionCount; ++r) {
        const auto& g = s.regions[r];
        if ((g.polynomial != 7 && g.polynomial != 9) || !std::isfinite(g.minimumTemperature)
            || !std::isfinite(g.maximumTemperature) || g.minimumTemperature <= 0
            || g.maximumTemperature <= g.minimumTemperature
            || (r && g.minimumTemperature < s.regions[r - 1].minimumTemperature))
            return "Invalid ideal-gas NASA region";
        for (int j = 0; j < g.polynomial; ++j)
            if (!std::isfinite(g.coefficient[j])) return "Invalid ideal-gas NASA coefficient";
        sp.polynomial[r] = g.polynomial;
        sp.regionMin[r] = g.minimumTemperature;
        for (int j = 0; j < 9; ++j) sp.coeff[r][j] = g.coefficient[j];
        sp.powers[r] = nasaPowers(g.polynomial, g.coefficient);
    }
    sp.regionMaxLast = s.regions[s.regionCount - 1].maximumTemperature;
    return "";
}

void fail(char* error, size_t size, const char* what) {
    if (error && size) std::snprintf(error, size, "%s", what);
}

}  // namespace
}  // namespace rb200

extern "C" {

void* reactive_ideal_gas_create_v3(const void* table, size_t bytes, double Tmin, double Tmax, double tolerance,
                                   char* error, size_t size) {
    using namespace rb200;
    try {
        require(table && bytes == sizeof(ReactiveB200Table), "Invalid ideal-gas table image");
        ReactiveB200Table t;
        std::memcpy(&t, table, sizeof(t));
        require(t.ns >= 1 && t.ns <= kIdealMaxSpecies, "Ideal-gas closure supports 1 to 4 species");
        require(std::isfinite(Tmin) && std::isfinite(Tmax) && Tmin > 0 && Tmax > Tmin, "Invalid temperature range");
        require(std::isfinite(tolerance) && tolerance > 0 && tolerance < 1, "Invalid closure tolerance");
        std::unique_ptr<IdealDevice> d(new IdealDevice);
        d->host.ns = t.ns;
        d->host.logs = 0;
        d->host.Tmin = Tmin;
        d->host.Tmax = Tmax;
        d->host.tol = tolerance;
        for (int k = 0; k < t.ns; ++k) {
            const std::string why = speciesFromTable(t.species[k], d->host.sp[k]);
            require(why.empty(), why.c_str());
            require(Tmin >= t.species[k].regions[0].minimumTemperature
                        && Tmax <= d->host.sp[k].regionMaxLast,
                    "Temperature range outside a species' NASA regions");
            d->host.r[k] = kGas / t.species[k].molecularWeight;
            for (int r = 0; r < t.species[k].regionCount; ++r)
                d->host.logs |= d->host.sp[k].powers[r].m1 != 0 || d->host.sp[k].powers[r].m2 != 0;
        }
        check(cudaGetDevice(&d->device), "cudaGetDevice");
        check(cudaMalloc(&d->dev, sizeof(IdealConst)), "cudaMalloc");
        check(cudaMemcpy(d->dev, &d->host, sizeof(IdealConst), cudaMemcpyHostToDevice), "H2D");
        return d.release();
    } catch (const std::exception& e) {
        fail(error, size, e.what());
        return nullptr;
    }
}

void reactive_ideal_gas_destroy_v3(void* gas) { delete static_cast<rb200::IdealDevice*>(gas); }

int reactive_ideal_gas_run_device_v3(void* gas, const double* q, size_t stride, size_t count, size_t variables,
                                     const double* Tseed, double* T, ReactiveTransportState* transport, int* success,
                                     void* stream, char* error, size_t size) {
    using namespace rb200;
    try {
        require(gas && q && Tseed && T && transport && count && stride >= count, "Invalid ideal-gas arguments");
        auto& d = *static_cast<IdealDevice*>(gas);
        require(variables == size_t(d.host.ns) + 4, "Ideal-gas closure needs variables = species + 4");
        auto s = static_cast<cudaStream_t>(stream);
        const unsigned grid = gridFor(count, 128);
        switch (d.host.ns) {
        case 1: idealClosure<1><<<grid, 128, 0, s>>>(d.dev, q, stride, count, Tseed, T, transport, success); break;
        case 2: idealClosure<2><<<grid, 128, 0, s>>>(d.dev, q, stride, count, Tseed, T, transport, success); break;
        case 3: idealClosure<3><<<grid, 128, 0, s>>>(d.dev, q, stride, count, Tseed, T, transport, success); break;
        default: idealClosure<4><<<grid, 128, 0, s>>>(d.dev, q, stride, count, Tseed, T, transport, success); break;
        }
        check(cudaGetLastError(), "idealClosure");
        return 0;
    } catch (const std::exception& e) {
        fail(error, size, e.what());
        return 1;
    }
}

int reactive_ideal_gas_vjp_device_v3(void* gas, const double* q, size_t stride, size_t count, size_t variables,
                                     const double* T, const ReactiveTransportState* bar, double* qBar,
                                     size_t barStride, void* stream, char* error, size_t size) {
    using namespace rb200;
    try {
        require(gas && q && T && bar && qBar && count && stride >= count && barStride >= count,
                "Invalid ideal-gas VJP arguments");
        auto& d = *static_cast<IdealDevice*>(gas);
        require(variables == size_t(d.host.ns) + 4, "Ideal-gas closure needs variables = species + 4");
        auto s = static_cast<cudaStream_t>(stream);
        const unsigned grid = gridFor(count, 128);
        switch (d.host.ns) {
        case 1: idealClosureVjp<1><<<grid, 128, 0, s>>>(d.dev, q, stride, count, T, bar, qBar, barStride); break;
        case 2: idealClosureVjp<2><<<grid, 128, 0, s>>>(d.dev, q, stride, count, T, bar, qBar, barStride); break;
        case 3: idealClosureVjp<3><<<grid, 128, 0, s>>>(d.dev, q, stride, count, T, bar, qBar, barStride); break;
        default: idealClosureVjp<4><<<grid, 128, 0, s>>>(d.dev, q, stride, count, T, bar, qBar, barStride); break;
        }
        check(cudaGetLastError(), "idealClosureVjp");
        return 0;
    } catch (const std::exception& e) {
        fail(error, size, e.what());
        return 1;
    }
}

}  // extern "C"
