// Differentiation of the matched filter with respect to the template parameters (the north star's adjoint form; the
// reference has no gradients: its template placement maximises the match numerically, ecc_bank_place.py:79-89).
//
// Parameters per trigger, theta = (Mc [M_sun], q = m2/m1 <= 1, chi1z, chi2z, e0 at f_ecc, t_c [s], phi_c). The
// template is the library's TaylorF2 (the phase of taylorf2_kernel: 3.5PN non-spinning, 1.5PN spin-orbit, 2PN
// spin-spin, leading eccentric term), h_k = f^-7/6 exp(-i Phi_k) on kmin <= k < kmax (kmax = the ISCO bin, as the
// bank's templates), Phi = Psi(f) - pi/4 + 2 pi f t_c - phi_c.
//   z = 4 df sum_k conj(h_k) D_k,  sigma^2 = 4 df sum_k |h_k|^2 IP_k,  snr = |z| / sigma
//   chisq = (nb sum_j |z_j|^2 - |z|^2) / sigma^2 over nb equal-power bins (z_j the bin's part of z, edges from the
//   cumulative |h|^2 IP as the pipeline's, held fixed), dof = 2 nb - 2, newsnr (coinc_rank.py:39-46).
// |h_k| does not depend on theta (inside [kmin, kmax)), so d sigma = 0 and dz/dtheta_i = 4 df sum_k i dPhi_k/dtheta_i
// conj(h_k) D_k. dPsi/d(Mc, q, chi1, chi2, e0) comes from forward-mode dual numbers through the phase formula (the
// metric) or its coefficients in f (the gradient) in float64; dPhi/dt_c = 2 pi f, dPhi/dphi_c = -1. The edges are
// found in the kernel (block scan of |h|^2 IP).
//
// The phase metric (the quadratic form of the phase-maximised match, 1 - m ~ dtheta^T g dtheta / 2): with |h|
// independent of theta, g_ij = Cov_w(dPhi/dtheta_i, dPhi/dtheta_j), w_k = |h_k|^2 IP_k; the phi_c row is zero.
#include <cmath>
#include "common.cuh"

namespace gwb {
namespace {

constexpr int kNP = 7;          // parameters
constexpr int kNI = 5;          // intrinsic ones (through the phase formula)
constexpr int kThreads = 256;
constexpr int kMaxBins = 32;
constexpr double kPi = 3.141592653589793;
constexpr double kMsun = 4.925490947641267e-06;    // G M_sun / c^3 in seconds
constexpr double kEuler = 0.5772156649015329;

// forward-mode dual number: value and its derivatives with respect to the kNI intrinsic parameters
struct Dual {
    double v, d[kNI];
};
__device__ __forceinline__ Dual dc(double a) {
    Dual r;
    r.v = a;
#pragma unroll
    for (int i = 0; i < kNI; ++i) r.d[i] = 0.0;
    return r;
}
__device__ __forceinline__ Dual operator+(const Dual& a, const Dual& b) {
    Dual r;
    r.v = a.v + b.v;
#pragma unroll
    for (int i = 0; i < kNI; ++i) r.d[i] = a.d[i] + b.d[i];
    return r;
}
__device__ __forceinline__ Dual operator-(const Dual& a, const Dual& b) {
    Dual r;
    r.v = a.v - b.v;
#pragma unroll
    for (int i = 0; i < kNI; ++i) r.d[i] = a.d[i] - b.d[i];
    return r;
}
__device__ __forceinline__ Dual operator*(const Dual& a, const Dual& b) {
    Dual r;
    r.v = a.v * b.v;
#pragma unroll
    for (int i = 0; i < kNI; ++i) r.d[i] = a.d[i] * b.v + a.v * b.d[i];
    return r;
}
__device__ __forceinline__ Dual operator*(double s, const Dual& a) {
    Dual r;
    r.v = s * a.v;
#pragma unroll
    for (int i = 0; i < kNI; ++i) r.d[i] = s * a.d[i];
    return r;
}
__device__ __forceinline__ Dual operator+(double s, const Dual& a) {
    Dual r = a;
    r.v += s;
    return r;
}
__device__ __forceinline__ Dual operator/(const Dual& a, const Dual& b) {
    Dual r;
    r.v = a.v / b.v;
    const double ib = 1.0 / b.v;
#pragma unroll
    for (int i = 0; i < kNI; ++i) r.d[i] = (a.d[i] - r.v * b.d[i]) * ib;
    return r;
}
// a^p for a constant exponent p (a > 0)
__device__ __forceinline__ Dual dpow(const Dual& a, double p) {
    Dual r;
    r.v = pow(a.v, p);
    const double g = p * r.v / a.v;
#pragma unroll
    for (int i = 0; i < kNI; ++i) r.d[i] = g * a.d[i];
    return r;
}
__device__ __forceinline__ Dual dlog(const Dual& a) {
    Dual r;
    r.v = log(a.v);
    const double g = 1.0 / a.v;
#pragma unroll
    for (int i = 0; i < kNI; ++i) r.d[i] = g * a.d[i];
    return r;
}

// per-trigger quantities of the phase, as functions of (Mc, q, chi1, chi2, e0)
struct PhaseCoef {
    Dual lms;        // log(pi Ms) (v = exp((log(pi Ms) + log f) / 3))
    Dual pre, p2, p3, p4, p5c, p6c, p7, ecc;   // ecc = -2355/1462 e0^2 v0^(19/3)
    double Ms;
};

__device__ PhaseCoef phase_coef(const double* th, double f_ecc) {
    Dual Mc = dc(th[0]), q = dc(th[1]), c1 = dc(th[2]), c2 = dc(th[3]), e0 = dc(th[4]);
    Mc.d[0] = 1.0;
    q.d[1] = 1.0;
    c1.d[2] = 1.0;
    c2.d[3] = 1.0;
    e0.d[4] = 1.0;
    const Dual one_q = 1.0 + q;
    const Dual eta = q / (one_q * one_q);
    const Dual M = Mc * dpow(eta, -0.6);
    const Dual d1 = dc(1.0) / one_q, d2 = q / one_q;
    const Dual beta = (113.0 / 12.0) * (d1 * d1 * c1 + d2 * d2 * c2) + 6.25 * (eta * (c1 + c2));
    const Dual sigma = (474.0 / 48.0) * (eta * c1 * c2);
    PhaseCoef P;
    const Dual Ms = kMsun * M;
    P.Ms = Ms.v;
    P.lms = dlog(kPi * Ms);
    P.pre = dc(3.0 / 128.0) / eta;
    P.p2 = (20.0 / 9.0) * (743.0 / 336.0 + (11.0 / 4.0) * eta);
    P.p3 = -16.0 * kPi + 4.0 * beta;
    P.p4 = 10.0 * (3058673.0 / 7257600.0 + ((5429.0 / 1008.0) * eta + (617.0 / 144.0) * (eta * eta))) - 10.0 * sigma;
    P.p5c = kPi * (38645.0 / 756.0 + (-65.0 / 9.0) * eta);
    P.p6c = (11583231236531.0 / 4694215680.0 - 640.0 / 3.0 * kPi * kPi - 6848.0 / 21.0 * kEuler) +
            ((-15737765635.0 / 3048192.0 + 2255.0 / 12.0 * kPi * kPi) * eta + (76055.0 / 1728.0) * (eta * eta) +
             (-127825.0 / 1296.0) * (eta * eta * eta));
    P.p7 = kPi * (77096675.0 / 254016.0 + ((378515.0 / 1512.0) * eta + (-74045.0 / 756.0) * (eta * eta)));
    const Dual v0 = dpow(kPi * f_ecc * Ms, 1.0 / 3.0);
    P.ecc = (-2355.0 / 1462.0) * (e0 * e0 * dpow(v0, 19.0 / 3.0));
    return P;
}

// Psi(f) and its derivatives with respect to the intrinsic parameters
__device__ __forceinline__ Dual psi_at(const PhaseCoef& P, double f) {
    const double lf = log(f);
    Dual lv = (1.0 / 3.0) * (P.lms + dc(lf));
    Dual v;
    v.v = exp(lv.v);
#pragma unroll
    for (int i = 0; i < kNI; ++i) v.d[i] = v.v * lv.d[i];
    const Dual p5 = P.p5c * (1.0 + 3.0 * (lv - dc(log(0.4082482904638631))));
    const Dual p6 = P.p6c - (6848.0 / 21.0) * (lv + dc(log(4.0)));
    // Horner: 1 + v^2 (p2 + v (p3 + v (p4 + v (p5 + v (p6 + v p7)))))
    Dual series = p6 + v * P.p7;
    series = p5 + v * series;
    series = P.p4 + v * series;
    series = P.p3 + v * series;
    series = P.p2 + v * series;
    series = 1.0 + (v * v) * series;
    // eccentric term: ecc v^(-19/3)
    Dual vm193;
    vm193.v = exp((-19.0 / 3.0) * lv.v);
#pragma unroll
    for (int i = 0; i < kNI; ++i) vm193.d[i] = vm193.v * (-19.0 / 3.0) * lv.d[i];
    series = series + P.ecc * vm193;
    Dual vm5;
    vm5.v = exp(-5.0 * lv.v);
#pragma unroll
    for (int i = 0; i < kNI; ++i) vm5.d[i] = vm5.v * (-5.0) * lv.d[i];
    return P.pre * vm5 * series;
}

__device__ __forceinline__ int kmax_of(double Ms, double df, int flen) {
    const double fisco = 1.0 / (14.696938456699067 * kPi * Ms);     // 6^1.5 pi Ms
    return (int)min((long long)floor(fisco / df) + 1, (long long)flen - 1);
}

// ---- SNR and its gradient ----
// In f alone the phase is linear in ten functions of frequency, whose coefficients hold all of theta: with u = f^(1/3),
//   Psi(f) = sum_m C_m(theta) phi_m(f),  phi = u^-5, u^-3, u^-2, u^-1, 1, l, u, u l, u^2, u^(-34/3),  l = log(f / kF0).
// So dPsi/dtheta_p = sum_m dC_m/dtheta_p phi_m, and the sums over bins that the gradient needs are the moments
// M_m = sum_k q_k phi_m(f_k), one per function (and one of f for t_c), contracted with dC_m/dtheta_p once per
// chi-squared bin instead of a dual-number phase per (bin, parameter).
// Errors: every power is within a few roundings of its value, since each one is multiplied by up to 1e4 rad. A power taken
// as exp(x log a) carries the error of x log a, and a product of n equal factors n times the factor's, so the coefficients
// come from pi Ms and its cube root and the float64 form's phi from f, 1 / f and f^(-1/3) (u^-5 = f^-1 f^(-2/3)). Error of
// Psi against 80-bit arithmetic, 4,096 (trigger, bin) pairs from 20 Hz on, largest / rms in rad: Mc = 1.2 1.1e-11 /
// 1.9e-12, 5 1.4e-12 / 1.8e-13, 25 6.6e-14 / 1.8e-14 (an exponential of the logarithm per term, as psi_at: 3.5e-11 /
// 7.5e-12, 3.3e-12 / 6.5e-13, 1.9e-13 / 3.4e-14; products of w = f^(-1/18): 6.4e-11 / 1.2e-11, 5.2e-12 / 9.2e-13, 3.3e-13 /
// 5.3e-14); amplitude 3.3 / 0.8 units of 2^-53 (6.8 / 3.6; 36 / 9.6). The float32 form rounds the reduced phase to 24 bits
// and keeps the products of w, which cost it no root per bin. l is centred so that the constant and the logarithmic terms,
// which cancel, stay small.
constexpr int kNF = 10;                  // phase functions
constexpr int kNM = kNF + 1;             // moments: the phase functions, then f
constexpr int kOne = 4;                  // phi = 1: the moment is the bin's z
constexpr int kGT = 256;                 // threads per trigger of snr_grad_kernel
constexpr int kWarps = kGT / 32;
constexpr int kTab = 6016;               // bins from kmin on whose l and root of f a CTA keeps for all its triggers (94 KB)
constexpr double kF0 = 128.0;            // a power of two: f / kF0 and kF0 pi Ms are exact

// C_m and its derivatives for m = lane: pre times a^x times a polynomial in (eta, chi), a = (pi Ms)^(1/3), so that
// a^-5 = 1 / (pi Ms a^2), and one division gives every lane its power. The eccentric term's a^(-34/3) v0^(19/3) is
// (pi Ms)^(-34/9 + 19/9) f_ecc^(19/9) = a^-5 ecc0. Ms: the trigger's (its pow is shared with the band's end).
__device__ __forceinline__ Dual phase_function_coef(const double* th, double Ms, double ecc0, int m) {
    Dual q = dc(th[1]), c1 = dc(th[2]), c2 = dc(th[3]);
    q.d[1] = 1.0;
    c1.d[2] = 1.0;
    c2.d[3] = 1.0;
    const Dual one_q = 1.0 + q, iq = dc(1.0) / one_q, qi = q * iq;
    const Dual eta = qi * iq;
    const double ieta = 1.0 / eta.v;
    const double X = kPi * Ms, a = cbrt(X), a2 = a * a;
    Dual la = dc((1.0 / 3.0) * log(kF0 * X));                         // log(a kF0^(1/3)), v = a u
    la.d[0] = 1.0 / (3.0 * th[0]);
    la.d[1] = -0.2 * ieta * eta.d[1];
    const double num = m == 9 ? ecc0 : m == 8 ? a2 : m >= 6 ? a : 1.0;
    const double den = m == 0 || m == 9 ? X * a2 : m == 1 ? X : m == 2 ? a2 : m == 3 ? a : 1.0;
    const double ex = m == 0 || m == 9 ? -5.0 : m == 1 ? -3.0 : m == 2 ? -2.0 : m == 3 ? -1.0 : m == 8 ? 2.0 : m >= 6 ? 1.0 : 0.0;
    Dual pw;
    pw.v = num / den;
#pragma unroll
    for (int i = 0; i < kNI; ++i) pw.d[i] = pw.v * ex * la.d[i];
    const Dual e2 = eta * eta;
    Dual c;
    if (m == 1) {
        c = (20.0 / 9.0) * (743.0 / 336.0 + (11.0 / 4.0) * eta);
    } else if (m == 2 || m == 3) {
        const Dual beta = (113.0 / 12.0) * (iq * iq * c1 + qi * qi * c2) + 6.25 * (eta * (c1 + c2));
        const Dual sigma = (474.0 / 48.0) * (eta * c1 * c2);
        c = m == 2 ? -16.0 * kPi + 4.0 * beta
                   : 10.0 * (3058673.0 / 7257600.0 + ((5429.0 / 1008.0) * eta + (617.0 / 144.0) * e2)) - 10.0 * sigma;
    } else if (m == 4 || m == 5) {
        c = kPi * (38645.0 / 756.0 + (-65.0 / 9.0) * eta);
        if (m == 4) c = c * (1.0 + 3.0 * (la - dc(log(0.4082482904638631))));
    } else if (m == 6) {
        c = (11583231236531.0 / 4694215680.0 - 640.0 / 3.0 * kPi * kPi - 6848.0 / 21.0 * kEuler) +
            ((-15737765635.0 / 3048192.0 + 2255.0 / 12.0 * kPi * kPi) * eta + (76055.0 / 1728.0) * e2 +
             (-127825.0 / 1296.0) * (e2 * eta));
        c = c - (6848.0 / 21.0) * (la + dc(log(4.0)));
    } else if (m == 7) {
        c = dc(-6848.0 / 63.0);
    } else if (m == 8) {
        c = kPi * (77096675.0 / 254016.0 + ((378515.0 / 1512.0) * eta + (-74045.0 / 756.0) * e2));
    } else if (m == 9) {
        c = dc(-2355.0 / 1462.0 * th[4] * th[4]);
        c.d[4] = -2355.0 / 731.0 * th[4];
    } else {
        c = dc(1.0);
    }
    Dual pre = dc(3.0 / 128.0 * ieta);
    pre.d[1] = -pre.v * ieta * eta.d[1];
    return pre * pw * c;
}

// What a CTA keeps per bin: l = log(f / kF0) and a root of f, f^(-1/3) for the float64 form, w = f^(-1/18) for the float32
// form.
template <typename T>
__device__ __forceinline__ double2 log_root(double f) {
    const double l = log(f * (1.0 / kF0));
    if constexpr (sizeof(T) == 8) return make_double2(l, rcbrt(f));
    else return make_double2(l, exp((l + 4.852030263919617) * (-1.0 / 18.0)));        // + log kF0
}
template <typename T>
__device__ __forceinline__ double2 log_root(const double2* tab, int kmin, int k, double df) {
    return k - kmin < kTab ? tab[k - kmin] : log_root<T>((double)k * df);
}
// 1 / f from iu = f^(-1/3): the cube's relative error (8 roundings) squared by one Newton step
__device__ __forceinline__ double inverse(double f, double iu) {
    const double r = iu * iu * iu;
    return fma(r, fma(-f, r, 1.0), r);
}
// f^(-1/N) from a float32 estimate y0 (good to 1e-6): with y0^N f = 1 - d, y0 (1 - d)^(-1/N) by its binomial series
template <int N>
__device__ __forceinline__ double minus_root(double f, double y0) {
    const double y2 = y0 * y0, y4 = y2 * y2, yn = N == 6 ? y4 * y2 : N == 9 ? y4 * y4 * y0 : 0.0;
    static_assert(N == 6 || N == 9, "powers written out");
    const double d = fma(-yn, f, 1.0);
    return fma(y0 * d, fma(d, (N + 1) / (2.0 * N * N), 1.0 / N), y0);
}
// f^(-7/3)
template <typename T>
__device__ __forceinline__ double root_to_73(double root, double f) {
    if constexpr (sizeof(T) == 8) {
        const double r = inverse(f, root);
        return root * r * r;
    }
    const double w3 = root * root * root, iu = w3 * w3, iu3 = iu * iu * iu;
    return iu3 * iu3 * iu;
}

// Equal-power edges of w_k = f^-7/3 IP_k over [kmin, k1): edge j = first k whose inclusive cumulative sum exceeds
// (j / nb) total (the pipeline's edges, offset mode 0). Threads take contiguous ranges; float64 sums, warp and block
// scans, and one walk per thread over its range that sets the edges inside it.
template <typename T>
__device__ void block_edges(const float* __restrict__ ip, double df, int kmin, int k1, int nb, int* e, double* tot_out,
                            double* scan, const double2* tab) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int len = k1 - kmin, chunk = (len + kGT - 1) / kGT;
    const int a = min(kmin + tid * chunk, k1), b = min(a + chunk, k1);
    auto weight = [&](int k) {
        return root_to_73<T>(log_root<T>(tab, kmin, k, df).y, (double)k * df) * (double)ip[k];
    };
    double s = 0.0;
#pragma unroll 4
    for (int k = a; k < b; ++k) s += weight(k);
    double inc = s;                                  // inclusive scan of the threads' sums
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += v;
    }
    if (lane == 31) scan[kGT + 1 + warp] = inc;
    for (int j = tid; j <= nb; j += kGT) e[j] = j == 0 ? kmin : k1;
    __syncthreads();
    double base = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps - 1; ++w) base += w < warp ? scan[kGT + 1 + w] : 0.0;
    scan[tid + 1] = base + inc;
    if (tid == 0) scan[0] = 0.0;
    __syncthreads();
    const double tot = scan[kGT], ex = scan[tid], hi = scan[tid + 1];
    if (tot > 0.0) {                                 // (not for a NaN)
        // the edges j with ex <= (j / nb) tot < hi
        auto target = [&](int j) { return (double)j / (double)nb * tot; };
        int j = max(1, (int)(ex / tot * (double)nb) - 1);
        while (j < nb && target(j) < ex) ++j;
        double t = j < nb ? target(j) : hi;
        if (t < hi) {
            double c = ex;
            for (int k = a; k < b; ++k) {
                c += weight(k);
                while (t < hi && c > t) {
                    e[j] = k;
                    t = ++j < nb ? target(j) : hi;
                }
            }
            while (t < hi) {                         // the range's last sum is hi, to rounding
                e[j] = b - 1;
                t = ++j < nb ? target(j) : hi;
            }
        }
    }
    if (tid == 0) *tot_out = tot;
    __syncthreads();
}

// out row layout (doubles): snr, newsnr, chisq, sigma2, z_re, z_im, kmax, dsnr[7], dnewsnr[7], dchisq[7]
constexpr int kOut = 7 + 3 * kNP;

// CTAs of eight warps, two per SM, stay for all their triggers (blockIdx.x, + gridDim.x, ...), so that log_root of the
// first kTab bins is computed once per CTA, as far as the longest band of its triggers. Per trigger, the
// band is cut into one contiguous run per warp; a lane's bins are 32 apart (coalesced D and IP), and at every chi-squared
// edge the warp adds its 22 sums over the lanes (a halving exchange: 31 shuffles of a double, against 110 for 22 trees)
// and stores them with the edge bin they belong to. Bound: the chain of a trigger (coefficients, edges, runs, final sums)
// with two of them per SM, and the float64 pipe. The former kernel took a barrier and a block reduction per chi-squared
// bin, in which 256 threads share the 20 to 200 bins of 16 s of data, and a dual-number phase with three exp and two pow
// per frequency bin: 803 us for 2,048 triggers of 16 s, float32, now 159. (A CTA per trigger without the table 194, four
// warps per trigger and four CTAs per SM 192, a warp per trigger 291: it waits for the longest band.) The float64 form's
// more exact powers cost it 5%: 330 us a call for 2,048 triggers of 16 s, Mc 4 to 34, 316 with products of w and 1,372 with
// the former kernel (float32 form 303, 304 and 1,320); divided and rooted by the library functions it took 385.
template <typename T>
__global__ void __launch_bounds__(kGT, 2) snr_grad_kernel(const double* __restrict__ params, int n,
                                                             const float2* __restrict__ D, long long ldd,
                                                             const float* __restrict__ IP, long long ldip, int flen,
                                                             double df, int kmin, double ecc0, int nb,
                                                             double* __restrict__ out, long long ldout) {
    constexpr int kNS = 2 * kNM;
    constexpr int kSeg = kMaxBins + kWarps;            // (warp, bin) runs: warp + bin never repeats along the band
    __shared__ double scan[kGT + 1 + kWarps];
    __shared__ int e[kMaxBins + 1];
    __shared__ double tot;
    __shared__ double C[kNF][1 + kNI];
    __shared__ int owner[kSeg];
    __shared__ double seg[kSeg][kNS];
    extern __shared__ double2 tab[];                   // kTab
    __shared__ int s_top;                              // the longest band of this CTA's triggers
    __shared__ double acc[kMaxBins][2 + 2 * kNP];      // per bin: z_j (re, im), dz_j (re, im) x 7
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_top = 0;
    __syncthreads();
    for (int i = blockIdx.x + tid * (int)gridDim.x; i < n; i += kGT * (int)gridDim.x) {
        const double* th = params + (long long)i * kNP;
        const double q1 = 1.0 + th[1], eta = th[1] / (q1 * q1);
        atomicMax(&s_top, kmax_of(kMsun * (th[0] * pow(eta, -0.6)), df, flen));
    }
    __syncthreads();
    for (int k = tid; k < min(kTab, s_top - kmin); k += kGT) tab[k] = log_root<T>((double)(kmin + k) * df);
    __syncthreads();
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const double* th = params + (long long)i * kNP;
        // the end bin from the same operations as phase_coef's value of Ms
        const double q1 = 1.0 + th[1], eta = th[1] / (q1 * q1);
        const double Ms = kMsun * (th[0] * pow(eta, -0.6));
        const int k1 = kmax_of(Ms, df, flen);
        if (k1 <= kmin + 256) {           // no band above kmin (f_ISCO below the low cut): nothing to filter
            if (tid < kOut) out[(long long)i * ldout + tid] = 0.0;
            continue;
        }
        const float* ip = IP + (long long)i * ldip;
        const float2* d = D + (long long)i * ldd;
        if (tid < kSeg) owner[tid] = -1;
        if (warp == kWarps - 1) {
            const Dual c = phase_function_coef(th, Ms, ecc0, min(lane, kNF - 1));
            if (lane < kNF) {
                C[lane][0] = c.v;
#pragma unroll
                for (int p = 0; p < kNI; ++p) C[lane][1 + p] = c.d[p];
            }
        }
        block_edges<T>(ip, df, kmin, k1, nb, e, &tot, scan, tab);   // ends with a barrier
        {
            double cv[kNF];
#pragma unroll
            for (int m = 0; m < kNF; ++m) cv[m] = C[m][0];
            cv[kOne] -= 0.25 * kPi + th[6];
            const double wtc = 2.0 * kPi * th[5];
            const int run = ((k1 - kmin + kGT - 1) / kGT) * 32;    // bins per warp, whole rounds of 32 lanes
            const int A = min(kmin + warp * run, k1), B = min(A + run, k1);
            for (int j = 0; j < nb; ++j) {
                const int lo = max(e[j], A), hi = min(e[j + 1], B);
                if (lo >= hi) continue;                                      // warp-uniform
                double s[kNS];
#pragma unroll
                for (int x = 0; x < kNS; ++x) s[x] = 0.0;
                float2 dn = lo + lane < hi ? d[lo + lane] : make_float2(0.f, 0.f);
                for (int k = lo + lane; k < hi; k += 32) {
                    const float2 dk = dn;
                    if (k + 32 < hi) dn = d[k + 32];
                    const double f = (double)k * df;
                    const double2 t = log_root<T>(tab, kmin, k, df);
                    const double lf = t.x;
                    double iu, iu2, i3, i5, i34, amp64;                      // u^-1, u^-2, u^-3, u^-5, u^(-34/3), f^(-7/6)
                    if constexpr (sizeof(T) == 8) {
                        iu = t.y;
                        iu2 = iu * iu;
                        i3 = inverse(f, iu);
                        i5 = iu2 * i3;
                        const float lg = log2f((float)f);
                        i34 = i5 * (i3 * i3) * minus_root<9>(f, exp2f(lg * (-1.f / 9.f)));
                        amp64 = i3 * minus_root<6>(f, exp2f(lg * (-1.f / 6.f)));
                    } else {
                        const double w = t.y, w2 = w * w, w3 = w2 * w;
                        iu = w3 * w3;
                        iu2 = iu * iu;
                        i3 = iu2 * iu;
                        i5 = i3 * iu2;
                        i34 = i5 * i5 * iu * w2;
                        amp64 = i3 * w3;
                    }
                    const double u = f * iu2;
                    const double phi[kNM] = {i5, i3, iu2, iu, 1.0, lf, u, u * lf, f * iu, i34, f};
                    double ph = cv[kOne], ph2 = wtc * f;                     // two chains
#pragma unroll
                    for (int m = 0; m < kNF; ++m) {
                        if (m < kOne) ph = fma(cv[m], phi[m], ph);
                        if (m > kOne) ph2 = fma(cv[m], phi[m], ph2);
                    }
                    ph += ph2;
                    ph -= 2.0 * kPi * rint(ph * (0.5 / kPi));
                    T sn, cs;
                    if constexpr (sizeof(T) == 8) {
                        sincos(ph, &sn, &cs);
                    } else {
                        sincosf((float)ph, &sn, &cs);
                    }
                    const T amp = (T)amp64;
                    // q = conj(h) D = amp e^{+i ph} D
                    const T hr = amp * cs, hi2 = amp * sn;
                    const double qr = (double)(hr * (T)dk.x - hi2 * (T)dk.y);
                    const double qi = (double)(hr * (T)dk.y + hi2 * (T)dk.x);
#pragma unroll
                    for (int m = 0; m < kNM; ++m) {
                        s[2 * m] = fma(qr, phi[m], s[2 * m]);
                        s[2 * m + 1] = fma(qi, phi[m], s[2 * m + 1]);
                    }
                }
                // lane x ends with the warp's sum of s[x]: each exchange halves the values a lane holds
                double v[16];
                {
                    const bool up = lane & 16;
#pragma unroll
                    for (int x = 0; x < 16; ++x) {
                        const double a = s[x], b = x + 16 < kNS ? s[x + 16 < kNS ? x + 16 : 0] : 0.0;
                        v[x] = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
                    }
                }
#pragma unroll
                for (int h = 8; h >= 1; h >>= 1) {
                    const bool up = lane & h;
#pragma unroll
                    for (int x = 0; x < h; ++x)
                        v[x] = (up ? v[x + h] : v[x]) + __shfl_xor_sync(0xffffffffu, up ? v[x] : v[x + h], h);
                }
                if (lane < kNS) seg[warp + j][lane] = v[0];
                if (lane == 0) owner[warp + j] = j;
            }
        }
        __syncthreads();
        // per (bin, value): the bin's runs in band order, then the contraction with dC / dtheta
        const double c4 = 4.0 * df;
        for (int x = tid; x < nb * (1 + kNP); x += kGT) {
            const int j = x / (1 + kNP), p = x % (1 + kNP) - 1;
            double re = 0.0, im = 0.0;
            for (int w = 0; w < kWarps; ++w) {
                if (owner[j + w] != j) continue;
                const double* M = seg[j + w];
                if (p < 0) {
                    re += M[2 * kOne];
                    im += M[2 * kOne + 1];
                } else if (p < kNI) {
#pragma unroll
                    for (int m = 0; m < kNF; ++m) {
                        re = fma(-C[m][1 + p], M[2 * m + 1], re);
                        im = fma(C[m][1 + p], M[2 * m], im);
                    }
                } else {
                    const int m = p == 5 ? kNF : kOne;
                    const double g = p == 5 ? 2.0 * kPi : -1.0;
                    re -= g * M[2 * m + 1];
                    im += g * M[2 * m];
                }
            }
            acc[j][2 * (p + 1)] = c4 * re;
            acc[j][2 * (p + 1) + 1] = c4 * im;
        }
        __syncthreads();
        if (tid < kNP) {                               // thread p: the outputs of parameter p (thread 0: the values too)
            const int p = tid;
            const double sig2 = c4 * tot;
            double zr = 0.0, zi = 0.0, pw = 0.0, dzr = 0.0, dzi = 0.0, dpw = 0.0;
            for (int j = 0; j < nb; ++j) {
                const double ar = acc[j][0], ai = acc[j][1], br = acc[j][2 + 2 * p], bi = acc[j][3 + 2 * p];
                zr += ar;
                zi += ai;
                pw += ar * ar + ai * ai;
                dzr += br;
                dzi += bi;
                dpw += 2.0 * (ar * br + ai * bi);
            }
            const double az = sqrt(zr * zr + zi * zi), sg = sqrt(sig2);
            const double snr = az / sg;
            const double chisq = ((double)nb * pw - az * az) / sig2;
            const int dof = 2 * nb - 2;
            const double rc = chisq / (double)dof;
            double ns = snr, g = 1.0, gp = 0.0;
            if (rc > 1.0) {
                const double base = (1.0 + rc * rc * rc) / 2.0;
                g = pow(base, -1.0 / 6.0);
                gp = -1.0 / 6.0 * pow(base, -7.0 / 6.0) * 1.5 * rc * rc;   // d g / d rc
                ns = snr * g;
            }
            double* o = out + (long long)i * ldout;
            if (p == 0) {
                o[0] = snr;
                o[1] = ns;
                o[2] = chisq;
                o[3] = sig2;
                o[4] = zr;
                o[5] = zi;
                o[6] = (double)k1;
            }
            const double dabs = az > 0.0 ? (zr * dzr + zi * dzi) / az : 0.0;
            const double dsnr = dabs / sg;
            const double dchi = ((double)nb * dpw - 2.0 * az * dabs) / sig2;
            o[7 + p] = dsnr;
            o[7 + kNP + p] = dsnr * g + snr * gp * dchi / (double)dof;
            o[7 + 2 * kNP + p] = dchi;
        }
        __syncthreads();                               // the next trigger's sums go over this one's
    }
}

// phase metric g (n x 7 x 7): weighted covariance of dPhi/dtheta with weights |h|^2 IP over [kmin, kmax)
__global__ void __launch_bounds__(kThreads) phase_metric_kernel(const double* __restrict__ params, int n,
                                                              const float* __restrict__ IP, long long ldip, int flen,
                                                              double df, int kmin, double f_ecc,
                                                              double* __restrict__ g) {
    const int i = blockIdx.x;
    if (i >= n) return;
    constexpr int NS = 1 + kNP + kNP * (kNP + 1) / 2;
    __shared__ double red[kThreads / 32][NS];
    const double* th = params + (long long)i * kNP;
    const PhaseCoef P = phase_coef(th, f_ecc);
    const int k1 = kmax_of(P.Ms, df, flen);
    if (k1 <= kmin + kThreads) {
        if (threadIdx.x < kNP * kNP) g[(long long)i * kNP * kNP + threadIdx.x] = 0.0;
        return;
    }
    const float* ip = IP + (long long)i * ldip;
    double s[NS];
#pragma unroll
    for (int x = 0; x < NS; ++x) s[x] = 0.0;
    for (int k = kmin + threadIdx.x; k < k1; k += kThreads) {
        const double f = (double)k * df;
        const double w = pow(f, -7.0 / 3.0) * (double)ip[k];
        const Dual ps = psi_at(P, f);
        double dph[kNP];
#pragma unroll
        for (int p = 0; p < kNI; ++p) dph[p] = ps.d[p];
        dph[5] = 2.0 * kPi * f;
        dph[6] = -1.0;
        s[0] += w;
        int c = 1 + kNP;
#pragma unroll
        for (int p = 0; p < kNP; ++p) {
            s[1 + p] += w * dph[p];
#pragma unroll
            for (int q = p; q < kNP; ++q) s[c++] += w * dph[p] * dph[q];
        }
    }
    // fixed-order reduction: warps by shuffles, then warps in order
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int x = 0; x < NS; ++x) {
        double v = s[x];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (lane == 0) red[warp][x] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t[NS];
        for (int x = 0; x < NS; ++x) {
            t[x] = 0.0;
            for (int w = 0; w < kThreads / 32; ++w) t[x] += red[w][x];
        }
        double* gi = g + (long long)i * kNP * kNP;
        int c = 1 + kNP;
        for (int p = 0; p < kNP; ++p)
            for (int q = p; q < kNP; ++q) {
                const double v = t[c++] / t[0] - (t[1 + p] / t[0]) * (t[1 + q] / t[0]);
                gi[p * kNP + q] = v;
                gi[q * kNP + p] = v;
            }
    }
}

// One Levenberg-Marquardt step of the SNR ascent per trigger, in the 6 parameters other than phi_c (|z| does not
// depend on it): near the maximum snr(theta + d) ~ snr(theta) (1 - d^T g d / 2) + grad . d, so the Newton step is
// g^-1 grad / snr; g's eigenvalues span many decades (the Mc - q - chi degeneracy) and the quadratic model fails far
// along the flat directions, so the step is d = (g + lam_i diag g)^-1 grad / snr with the caller adapting lam_i per
// trigger (down after a step that raised the SNR, up after one that did not). Then clamped to the physical ranges
// (Mc > 0, q in [0.05, 1], |chi| <= 0.99, e0 in [0, 0.5]). Cholesky in float64.
__global__ void refine_step_kernel(const double* __restrict__ params, const double* __restrict__ res, long long ldres,
                                   const double* __restrict__ g, const double* __restrict__ lam, int n,
                                   double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    constexpr int m = 6;
    const double* gi = g + (long long)i * kNP * kNP;
    const double* ri = res + (long long)i * ldres;
    double A[m][m], b[m];
    const double snr = ri[0];
    double dmax = 0.0;
    for (int p = 0; p < m; ++p) dmax = fmax(dmax, gi[p * kNP + p]);
    for (int p = 0; p < m; ++p) {
        for (int q = 0; q < m; ++q) A[p][q] = gi[p * kNP + q];
        A[p][p] *= 1.0 + lam[i];
        b[p] = snr > 0.0 ? ri[7 + p] / snr : 0.0;      // dsnr / snr
    }
    // a parameter the phase does not depend on here (e0 at 0: the phase goes with e0^2) has a zero row: it takes no
    // step (its gradient is zero too) and leaves the others' system positive definite
    for (int p = 0; p < m; ++p)
        if (!(gi[p * kNP + p] > 1e-24 * dmax)) {
            for (int q = 0; q < m; ++q) A[p][q] = A[q][p] = 0.0;
            A[p][p] = dmax > 0.0 ? dmax : 1.0;
            b[p] = 0.0;
        }
    bool ok = snr > 0.0;
    for (int p = 0; p < m && ok; ++p) {                 // A = L L^T in place (lower)
        for (int q = 0; q <= p; ++q) {
            double s = A[p][q];
            for (int r = 0; r < q; ++r) s -= A[p][r] * A[q][r];
            if (p == q) {
                if (s <= 0.0) {
                    ok = false;
                    break;
                }
                A[p][p] = sqrt(s);
            } else {
                A[p][q] = s / A[q][q];
            }
        }
    }
    double d[m] = {0, 0, 0, 0, 0, 0};
    if (ok) {
        double y[m];
        for (int p = 0; p < m; ++p) {
            double s = b[p];
            for (int r = 0; r < p; ++r) s -= A[p][r] * y[r];
            y[p] = s / A[p][p];
        }
        for (int p = m - 1; p >= 0; --p) {
            double s = y[p];
            for (int r = p + 1; r < m; ++r) s -= A[r][p] * d[r];
            d[p] = s / A[p][p];
        }
    }
    const double* th = params + (long long)i * kNP;
    double* o = out + (long long)i * kNP;
    for (int p = 0; p < kNP; ++p) o[p] = th[p] + (p < m ? d[p] : 0.0);
    o[0] = fmax(o[0], 0.05 * th[0]);
    o[1] = fmin(fmax(o[1], 0.05), 1.0);
    o[2] = fmin(fmax(o[2], -0.99), 0.99);
    o[3] = fmin(fmax(o[3], -0.99), 0.99);
    o[4] = fmin(fmax(o[4], 0.0), 0.5);
}

}  // namespace
}  // namespace gwb

extern "C" {

int gwb_snr_grad(const double* params, int n, const float* D, long long ldd, const float* IP, long long ldip, int flen,
                 double df, int kmin, double f_ecc, int nbins, int fp64, double* out, long long ldout, void* stream) {
    using namespace gwb;
    GWB_CHECK_ARG(params && D && IP && out, GWB_ERR_ARG, "snr_grad: null pointer");
    GWB_CHECK_ARG(n > 0 && n < (1 << 30) && flen > kmin && kmin > 0 && ldd >= flen && ldip >= 0 && df > 0 &&
                      nbins >= 1 && nbins <= kMaxBins && ldout >= kOut,
                  GWB_ERR_SHAPE, "snr_grad: n=%d flen=%d kmin=%d nbins=%d ldout=%lld", n, flen, kmin, nbins, ldout);
    cudaStream_t s = (cudaStream_t)stream;
    const float2* d = reinterpret_cast<const float2*>(D);
    const int grid = std::min(n, 2 * num_sms());           // two CTAs per SM
    const size_t smem = kTab * sizeof(double2);
    const double ecc0 = f_ecc * f_ecc * std::pow(f_ecc, 1.0 / 9.0);       // f_ecc^(19/9)
    GWB_CUDA(cudaFuncSetAttribute(fp64 ? snr_grad_kernel<double> : snr_grad_kernel<float>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (fp64)
        snr_grad_kernel<double><<<grid, kGT, smem, s>>>(params, n, d, ldd, IP, ldip, flen, df, kmin, ecc0, nbins,
                                                        out, ldout);
    else
        snr_grad_kernel<float><<<grid, kGT, smem, s>>>(params, n, d, ldd, IP, ldip, flen, df, kmin, ecc0, nbins, out,
                                                       ldout);
    GWB_LAUNCH_CHECK("snr_grad_kernel");
    return GWB_OK;
}

int gwb_phase_metric(const double* params, int n, const float* IP, long long ldip, int flen, double df, int kmin,
                     double f_ecc, double* g, void* stream) {
    using namespace gwb;
    GWB_CHECK_ARG(params && IP && g, GWB_ERR_ARG, "phase_metric: null pointer");
    GWB_CHECK_ARG(n > 0 && n < (1 << 30) && flen > kmin && kmin > 0 && ldip >= 0 && df > 0, GWB_ERR_SHAPE,
                  "phase_metric: n=%d flen=%d kmin=%d", n, flen, kmin);
    phase_metric_kernel<<<n, kThreads, 0, (cudaStream_t)stream>>>(params, n, IP, ldip, flen, df, kmin, f_ecc, g);
    GWB_LAUNCH_CHECK("phase_metric_kernel");
    return GWB_OK;
}

int gwb_refine_step(const double* params, const double* res, long long ldres, const double* g, const double* lam,
                    int n, double* out, void* stream) {
    using namespace gwb;
    GWB_CHECK_ARG(params && res && g && lam && out, GWB_ERR_ARG, "refine_step: null pointer");
    GWB_CHECK_ARG(n > 0 && ldres >= kOut, GWB_ERR_SHAPE, "refine_step: n=%d ldres=%lld", n, ldres);
    refine_step_kernel<<<(unsigned)cdiv(n, 128), 128, 0, (cudaStream_t)stream>>>(params, res, ldres, g, lam, n, out);
    GWB_LAUNCH_CHECK("refine_step_kernel");
    return GWB_OK;
}

}  // extern "C"
