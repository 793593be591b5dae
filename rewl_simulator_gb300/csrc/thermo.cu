// Canonical thermodynamics from a density of states, in FP64 on the GPU.
//
// Restates Thermodynamics::calculate_thermodynamics (src/Thermodynamics/thermodynamics.hpp:
// 158-236 with TRAPEZOIDAL_RULE, the reference's default, and 238-297 without): for every
// temperature T_i = Tmin + i (Tmax - Tmin) / nT, a log-sum-exp over the energy bins,
//   x_b = ln g_b - E_b / T,  m = max_b x_b,  w_b = exp(x_b - m) (end bins halved under the
//   trapezoidal rule),  Z = sum_b w_b,
// and the rows [F, U, U2, S, C, observables..., mean count] of its canonical_observables:
// F = -T (m + ln Z) / N, U = sum E w / (N Z), U2 = sum E^2 w / (N^2 Z), S = sum ln g w / (N Z),
// C = N (U2 - U^2) / T^2, O_k = sum O_k w / Z, and the counts column averaged over the bins.
// The reference loops over 50,000 temperatures serially (src/Simulation/main.cpp:13-15,
// 339-351); here one warp (or a few) reduces one temperature, all temperatures in one launch.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cfloat>
#include <limits>
#include <cstdarg>
#include <cstdio>
#include <string>

#include "../../include/rewl.h"

namespace {

thread_local std::string g_thermo_error;

int tfail(int code, const char* fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_thermo_error = buf;
    return code;
}

constexpr int kMaxObs = 20;            // Ashkin-Teller with correlators: 16 averages + the count
constexpr int kWarps = 16;             // per block
constexpr int kExpBits = 11;           // table of 2^(j / 2048)
constexpr int kExpTable = 1 << kExpBits;

struct ThermoArgs {
    const double *E, *lng;             // nb levels
    const float2* x32;                 // {-E, ln g} in single precision
    const long long *Ei, *gi;          // E 2^se and ln g / ln 2 2^sg as integers (62 bits)
    int se, sg;
    const double* obs;                 // K columns of nb values
    const int* not_finite;             // per block of k_levels: an averaged column holds a NaN or an infinity
    int nb, K, counts_col, nT, trapezoid, team;
    double N, Tmin, dT, counts_mean;
    float e_max, g_max;                // largest |E| and |ln g|; e_max < 0: no single-precision pass
    double *temps, *out;
};

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

// 2^(i / 2048) in units of 2^-63, from 2^(1/2), 2^(1/4), ... 2^(1/2048)
__device__ unsigned long long pow2_fraction(int i)
{
    constexpr unsigned long long kRoot[kExpBits] = {
        0xb504f333f9de6484ull, 0x9837f0518db8a96full, 0x8b95c1e3ea8bd6e7ull, 0x85aac367cc487b15ull, 0x82cd8698ac2ba1d7ull,
        0x8164d1f3bc030773ull, 0x80b1ed4fd999ab6cull, 0x8058d7d2d5e5f6b1ull, 0x802c6436d0e04f51ull, 0x8016302f17467628ull,
        0x800b179c82028fd1ull};
    unsigned long long v = 1ull << 63;
#pragma unroll
    for (int k = 0; k < kExpBits; ++k)
        if ((i >> (kExpBits - 1 - k)) & 1) {
            const unsigned long long hi = __umul64hi(v, kRoot[k]), lo = v * kRoot[k];
            v = (hi << 1) + (lo >> 63) + ((lo >> 62) & 1ull);
        }
    return v;
}

// 2^(d 2^-F) as a double, for -1020 <= d 2^-F < 1000, in integer arithmetic: the fraction is split into
// a table index j and a rest g < 2^-11 (P. T. P. Tang, "Table-driven implementation of the exponential
// function in IEEE floating-point arithmetic", ACM TOMS 15, 1989), 2^g = 1 + t + t^2/2 + t^3/6 + t^4/24 with
// t = g ln 2 in units of 2^-75 (the next term is below 2^-64), and the product is rounded to 53 bits once.
__device__ __forceinline__ double pow2_fixed(long long d, int F, const unsigned long long* tab)
{
    const int k = (int)(d >> F);
    const unsigned long long fr = (unsigned long long)d << (64 - F);
    const unsigned long long t = __umul64hi(fr << kExpBits, 0xb17217f7d1cf79acull);      // 2^-75
    const unsigned th = (unsigned)(t >> 32);                                             // 2^-43
    const unsigned long long t2 = __umul64hi(t, t);                                      // 2^-86
    const unsigned t2h = (unsigned)(t2 >> 32);                                           // 2^-54
    const unsigned t3 = __umulhi(__umulhi(t2h, th), 0x2AAAAAABu);                        // t^3 / 6, 2^-65
    const unsigned t4 = __umulhi(__umulhi(t2h, t2h), 0x0AAAAAABu);                       // t^4 / 24, 2^-76
    const unsigned long long p = t + (t2 >> 12) + ((unsigned long long)t3 << 10) + (t4 >> 1);
    const unsigned long long m = tab[(int)(fr >> (64 - kExpBits))];
    const unsigned long long w = m + (__umul64hi(m, p) >> 11);                           // [1, 2) in 2^-63
    return __longlong_as_double(((long long)(k + 1022) << 52) + (long long)((w >> 11) + ((w >> 10) & 1ull)));
}

constexpr double kLog2e = 0x1.71547652b82fep+0, kLog2eLo = 0x1.777d0ffda0d24p-56;

// The caller's levels as k_thermo reads them, a thread each: single precision, integers (ln g / ln 2 formed to
// 106 bits), observables by column.  (On the host this was 90 us of a call with 4,095 levels.)
constexpr int kLevelThreads = 128;
__global__ void __launch_bounds__(kLevelThreads) k_levels(const ThermoArgs a, const double* rows, float2* x32, long long* Ei, long long* gi, double* cols,
                         int* not_finite)
{
    const int b = blockIdx.x * kLevelThreads + threadIdx.x;
    bool finite = true;
    if (b < a.nb) {
        const double e = a.E[b], l = a.lng[b];
        x32[b] = make_float2((float)-e, (float)l);
        const double g = __dmul_rn(l, kLog2e), rest = __dadd_rn(__fma_rn(l, kLog2e, -g), __dmul_rn(l, kLog2eLo));
        Ei[b] = __double2ll_rn(ldexp(e, a.se));
        gi[b] = __double2ll_rn(ldexp(g, a.sg)) + __double2ll_rn(ldexp(rest, a.sg));
        for (int k = 0; k < a.K; ++k) {
            const double v = rows[(size_t)b * a.K + k];
            cols[(size_t)k * a.nb + b] = v;
            finite = finite && (k == a.counts_col || isfinite(v));
        }
    }
    const int any = __syncthreads_or(!finite);
    if (threadIdx.x == 0) not_finite[blockIdx.x] = any;
}

// One warp per temperature; a team of warps where there are few (TEAM).  Bound: the FP64 pipe -- an FP64 warp instruction occupies it for 32
// cycles of the SM, as long as some sixty integer ones -- so what the sums do not need stays off it:
//   * a level whose weight is zero in FP64 (more than 746 below the maximum) is found in single
//     precision, with its rounding error bounded and added to the margin, and skipped: half of the
//     levels of an L = 64 spectrum over the default ladder;
//   * the exponents of the others, relative to the largest, are differences of 62-bit integers, and
//     their exponentials are formed by integer arithmetic to the last bit of a double (above).
// What is left is one addition and three products for the sums and one per observable: 4,095 levels x
// 50,000 temperatures x 5 columns 23.4 -> 2.9 ms (with the copies) from two divisions and a library
// exponential for every level; the same sums with a table exponential in FP64 took 7.9 ms.
// Where the integers could be coarser than FP64 -- energies whose largest values dwarf those that
// count -- a temperature takes the FP64 form of the same sums.
// STAGED: levels in shared memory.  KO: room for observable columns.  TEAM: a.team warps per temperature.
template <bool STAGED, int KO, bool TEAM>
__global__ void __launch_bounds__(32 * kWarps, 1) k_thermo(const ThermoArgs a)
{
    extern __shared__ __align__(16) double sm[];
    __shared__ double part[TEAM ? kWarps : 1][4 + KO];
    __shared__ int at[kWarps];
    unsigned long long* tab = reinterpret_cast<unsigned long long*>(sm);
    double *sE = sm + kExpTable, *sG = sE + a.nb, *sE2 = sG + a.nb;
    float2* sX = reinterpret_cast<float2*>(sE2 + a.nb);
    long long *sEi = reinterpret_cast<long long*>(sX + a.nb), *sgi = sEi + a.nb;
    for (int j = threadIdx.x; j < kExpTable; j += blockDim.x) tab[j] = pow2_fraction(j);
    if (STAGED)
        for (int b = threadIdx.x; b < a.nb; b += blockDim.x) {
            const double e = a.E[b];
            sE[b] = e;
            sE2[b] = e * e;
            sG[b] = a.lng[b];
            sX[b] = a.x32[b];
            sEi[b] = a.Ei[b];
            sgi[b] = a.gi[b];
        }
    int special = 0;
    for (int i = threadIdx.x; i < (a.nb + kLevelThreads - 1) / kLevelThreads; i += blockDim.x) special |= a.not_finite[i];
    // (a level of zero weight counts too where an average is not finite there: NaN or infinity times zero is NaN)
    const bool single = !__syncthreads_or(special) && a.e_max >= 0.f;
    const double* E = STAGED ? sE : a.E;
    const double* G = STAGED ? sG : a.lng;
    const float2* X = STAGED ? sX : a.x32;
    const long long* Ei = STAGED ? sEi : a.Ei;
    const long long* gi = STAGED ? sgi : a.gi;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nb = a.nb;
    // the warps of a temperature share its levels: this one's are first, first + stride ...
    const int team = TEAM ? a.team : 1, teams = kWarps / team, lead = TEAM ? warp / team * team : warp;
    const int first = TEAM ? 32 * (warp - lead) : 0, stride = 32 * team;
    // a barrier of the team's own (teams at different temperatures take different branches)
    auto team_sync = [&] { asm volatile("bar.sync %0, %1;" :: "r"(1 + warp / team), "r"(stride) : "memory"); };
    // combine(v, w) of the values of a team's warps, w one of them, in every lane of all of them
    auto team_all = [&](double v, auto combine) {
        if (!TEAM) return v;
        team_sync();
        if (lane == 0) part[TEAM ? warp : 0][0] = v;
        team_sync();
        v = part[TEAM ? lead : 0][0];
        for (int w = 1; w < team; ++w) v = combine(v, part[TEAM ? lead + w : 0][0]);
        return v;
    };
    for (int t0 = blockIdx.x * teams + (TEAM ? 0 : warp); t0 < a.nT; t0 += gridDim.x * teams) {
        const bool here = !TEAM || t0 + warp / team < a.nT;                // (all warps keep the barriers of a team)
        const int t = !TEAM ? t0 : here ? t0 + warp / team : a.nT - 1;
        const double T = __dadd_rn(a.Tmin, __dmul_rn(a.dT, (double)t));    // rounded as the reference's Tmin + dT * i
        const double rT = 1.0 / T;
        auto exponent = [&](int b) { return G[b] - E[b] / T; };
        // the largest exponent, to the single-precision error `err` of every x32 (three times what its
        // roundings add up to): the exponent of the level found is the reference point, which need not be
        // the largest one to the last bit
        const float r32 = (float)rT;
        const float err = 5e-7f * (a.e_max * r32 + a.g_max) + 1e-3f;
        const bool filter = single && err < 50.f;
        double m;
        float floor32 = -INFINITY;
        int F = 0, top = 0;
        long long c = 0;
        if (filter) {
            float best = -INFINITY;
            for (int b = first + lane; b < nb; b += stride) {
                const float2 v = X[b];
                const float x = fmaf(v.x, r32, v.y);
                if (x > best) { best = x; top = b; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float x = __shfl_xor_sync(0xFFFFFFFFu, best, o);
                const int i = __shfl_xor_sync(0xFFFFFFFFu, top, o);
                if (x > best || (x == best && i < top)) { best = x; top = i; }
            }
            if (TEAM) {
                // the first of the team's largest
                team_sync();
                if (lane == 0) { part[TEAM ? warp : 0][0] = best; at[warp] = top; }
                team_sync();
                for (int w = lead; w < lead + team; ++w) {
                    const float x = (float)part[TEAM ? w : 0][0];
                    if (x > best || (x == best && at[w] < top)) { best = x; top = at[w]; }
                }
            }
            m = exponent(top);
            floor32 = best - 746.f - 2.f * err;
            // fixed point for the levels that count: their energies lie within `span` of the reference's
            float span = 0.f;
            const float2 ref = X[top];
            for (int b = first + lane; b < nb; b += stride) {
                const float2 v = X[b];
                if (!(fmaf(v.x, r32, v.y) < floor32)) span = fmaxf(span, fabsf(v.x - ref.x));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) span = fmaxf(span, __shfl_xor_sync(0xFFFFFFFFu, span, o));
            span = (float)team_all(span, [](double x, double y) { return fmax(x, y); });
            span = 1.0001f * span + 2e-7f * a.e_max;
            const double ch = kLog2e * rT, cl = fma(kLog2e, rT, -ch) + (kLog2e * (fma(-rT, T, 1.0) * rT) + kLog2eLo * rT);
            const float bits = 1.45f * (2.f * span * r32 + 750.f + 2.f * err);     // bound of every exponent difference
            F = min(min(60 - ilogbf(bits), a.se - 3 - ilogb(ch)), min(a.sg, 52));
            // the roundings of the integers against those of x = ln g - E / T and of a weight in FP64
            const double coarse = ldexp(ch, -a.se) + ldexp(1.0, -a.sg) + ldexp(1.0, -F);
            if (F >= 24 && coarse <= 0x1p-53 * (1.0 + (fabs(E[top]) * rT + fabs(m)))) {
                const int up = F + 64 - a.se;
                c = __double2ll_rn(ldexp(ch, up)) + __double2ll_rn(ldexp(cl, up));
            } else {
                F = 0;
            }
        } else {
            m = -INFINITY;
            for (int b = first + lane; b < nb; b += stride) m = fmax(m, exponent(b));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
            m = team_all(m, [](double x, double y) { return fmax(x, y); });
        }

        double z = 0.0, u = 0.0, u2 = 0.0, s = 0.0, o[KO + 1];
#pragma unroll
        for (int k = 0; k < KO; ++k) o[k] = 0.0;
        const long long etop = Ei[top], gtop = gi[top];
        for (int b0 = first; b0 < nb; b0 += stride) {
            const int b = b0 + lane;
            bool counts = b < nb;
            if (filter && counts) {
                const float2 v = X[b];
                counts = !(fmaf(v.x, r32, v.y) < floor32);
            }
            if (!__any_sync(0xFFFFFFFFu, counts)) continue;
            if (counts) {
                double w;
                if (F) {
                    const long long d = ((gi[b] - gtop) >> (a.sg - F)) - __mul64hi(Ei[b] - etop, c);
                    w = (d >> F) >= -1020 ? pow2_fixed(d, F, tab) : 0.0;
                } else {
                    w = exp(exponent(b) - m);
                }
                if (a.trapezoid && (b == 0 || b == nb - 1)) w *= 0.5;
                const double e = E[b];
                z += w;
                u = fma(e, w, u);
                u2 = fma(STAGED ? sE2[b] : e * e, w, u2);
                s = fma(G[b], w, s);
#pragma unroll
                for (int k = 0; k < KO; ++k)
                    if (k < a.K && k != a.counts_col) o[k] = fma(a.obs[(size_t)k * nb + b], w, o[k]);
            }
        }
        z = warp_sum(z);
        u = warp_sum(u);
        u2 = warp_sum(u2);
        s = warp_sum(s);
        if (TEAM) {
#pragma unroll
            for (int k = 0; k < KO; ++k)
                if (k < a.K && k != a.counts_col) o[k] = warp_sum(o[k]);
            double* p = part[TEAM ? warp : 0];
            team_sync();
            if (lane == 0) {
                p[0] = z; p[1] = u; p[2] = u2; p[3] = s;
#pragma unroll
                for (int k = 0; k < KO; ++k) p[4 + k] = o[k];
            }
            team_sync();
            if (warp != lead || !here) continue;
            for (int w = 1; w < team; ++w) {
                const double* v = part[TEAM ? lead + w : 0];
                z += v[0]; u += v[1]; u2 += v[2]; s += v[3];
#pragma unroll
                for (int k = 0; k < KO; ++k) o[k] += v[4 + k];
            }
        }
        double* row = a.out + (size_t)t * (5 + a.K);
#pragma unroll
        for (int k = 0; k < KO; ++k)
            if (k < a.K) {
                if (k == a.counts_col) o[k] = a.counts_mean;
                else o[k] = (TEAM ? o[k] : warp_sum(o[k])) / z;
                if (lane == 0) row[5 + k] = o[k];
            }
        if (lane == 0) {
            const double U = u / (a.N * z), U2 = u2 / (a.N * a.N * z);
            row[0] = -T * (m + log(z)) / a.N;
            row[1] = U;
            row[2] = U2;
            row[3] = s / (a.N * z);
            row[4] = a.N * (U2 - U * U) / (T * T);
            a.temps[t] = T;
        }
    }
}

} // namespace

extern "C" {

const char* rewl_thermo_last_error_string(void) { return g_thermo_error.c_str(); }

int rewl_thermodynamics(const double* E, const double* lng, const double* obs, int32_t nbins, int32_t num_obs,
                        int32_t counts_col, double system_size, double Tmin, double Tmax, int32_t num_T,
                        int32_t trapezoid, int32_t device, double* temperatures, double* out)
{
    if (!E || !lng || !out || !temperatures || nbins < 2 || num_T < 1 || !(system_size > 0) || !(Tmin > 0) ||
        !(Tmax > Tmin) || num_obs < 0 || num_obs > kMaxObs || (num_obs > 0 && !obs) || counts_col >= num_obs)
        return tfail(REWL_EINVAL, "bad arguments (nbins >= 2, 0 < Tmin < Tmax, num_T >= 1, num_obs <= %d)", kMaxObs);
    for (int b = 0; b < nbins; ++b)
        if (!std::isfinite(E[b]) || !std::isfinite(lng[b])) return tfail(REWL_EINVAL, "non-finite energy or ln g at bin %d", b);
    if (cudaSetDevice(device) != cudaSuccess) return tfail(REWL_EDEVICE, "cannot use device %d", device);
    const size_t nrow = 5 + (size_t)num_obs, nb = (size_t)nbins;
    double e_max = 0, g_max = 0, counts = 0;
    for (size_t b = 0; b < nb; ++b) {
        e_max = std::max(e_max, std::fabs(E[b]));
        g_max = std::max(g_max, std::fabs(lng[b]));
        if (counts_col >= 0) counts += obs[b * num_obs + counts_col];
    }
    // the integers: 2^62 above the largest energy, 2^60 above the largest ln g / ln 2
    int xe = 0, xg = 0;
    std::frexp(e_max, &xe);
    std::frexp(g_max * 1.45, &xg);
    // (sg: a shift by sg - F >= sg - 52 bits has to stay below 64 where F is at least 24)
    const int se = std::min(std::max(62 - xe, -900), 900), sg = std::min(std::max(60 - xg, -900), 86);
    ThermoArgs a{};
    a.se = se; a.sg = sg;
    a.nb = nbins; a.K = num_obs; a.counts_col = counts_col; a.nT = num_T; a.trapezoid = trapezoid ? 1 : 0;
    a.N = system_size; a.Tmin = Tmin; a.dT = (Tmax - Tmin) / (double)num_T; a.counts_mean = counts / (double)nbins;
    // single precision locates the levels that count while it can hold them
    const bool filter = e_max < 1e18 && e_max < 1e30 * Tmin && g_max < 1e30 && Tmin > 1e-30;
    a.e_max = filter ? std::nextafter((float)e_max, INFINITY) : -1.f;
    a.g_max = filter ? std::nextafter((float)g_max, INFINITY) : 0.f;
    cudaStream_t st;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return tfail(REWL_EDEVICE, "stream creation failed");
    // one buffer: E, ln g and the observables as the caller has them; what k_levels makes of them (columns, single
    // precision, two integers a level); temperatures and rows;
    // k_levels' flags
    const size_t in = nb * (2 + num_obs), made = nb * (3 + num_obs);
    const size_t blocks = (nb + kLevelThreads - 1) / kLevelThreads, all = in + made + (size_t)num_T * (1 + nrow) + (blocks + 1) / 2;
    double* d = nullptr;
    cudaError_t e = cudaMalloc(&d, all * sizeof(double));
    // (small inputs and results in one copy each: a copy is 5 to 10 us of a call of 200)
    constexpr size_t kSmall = 4096;
    double small[kSmall];
    if (in <= kSmall) {
        std::copy(E, E + nb, small);
        std::copy(lng, lng + nb, small + nb);
        std::copy(obs, obs + (num_obs ? nb * num_obs : 0), small + 2 * nb);
        if (e == cudaSuccess) e = cudaMemcpyAsync(d, small, in * 8, cudaMemcpyHostToDevice, st);
    } else {
        if (e == cudaSuccess) e = cudaMemcpyAsync(d, E, nb * 8, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(d + nb, lng, nb * 8, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess && num_obs) e = cudaMemcpyAsync(d + 2 * nb, obs, nb * num_obs * 8, cudaMemcpyHostToDevice, st);
    }
    if (e == cudaSuccess) {
        double* cols = d + in;
        float2* x32 = reinterpret_cast<float2*>(cols + nb * num_obs);
        long long* Ei = reinterpret_cast<long long*>(x32 + nb);
        int* flags = reinterpret_cast<int*>(d + in + made + (size_t)num_T * (1 + nrow));
        a.E = d; a.lng = d + nb; a.obs = cols; a.x32 = x32; a.Ei = Ei; a.gi = Ei + nb; a.not_finite = flags;
        a.temps = d + in + made; a.out = a.temps + num_T;
        k_levels<<<(unsigned)blocks, kLevelThreads, 0, st>>>(a, d + 2 * nb, x32, Ei, Ei + nb, cols, flags);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        int nsm = 0;
        if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || nsm < 1) nsm = 152;
        const size_t table = kExpTable * sizeof(double), staged = table + nb * 48;
        const bool fits = staged <= 220 * 1024;        // levels up to 4,352 in shared memory
        // Warps per temperature: one where the temperatures fill the device, else as many as keep all blocks
        // in one wave (4,095 levels, 17 columns: 152 temperatures, teams of 1 / 4 / 8 / 16 warps 499 / 331 / 297 /
        // 293 us; 500: 528 / 333 / 386 / 494; 1000, teams of 1 / 2 / 4: 527 / 397 / 421; 2432: 537 / 544 / 604)
        a.team = 1;
        while (a.team < kWarps && 32 * a.team < nbins && 2ll * a.team * num_T <= (long long)kWarps * nsm) a.team *= 2;
        using Kernel = void (*)(const ThermoArgs);
        const Kernel kernels[2][2][3] = {{{k_thermo<false, 0, false>, k_thermo<false, 6, false>, k_thermo<false, kMaxObs, false>},
                                          {k_thermo<true, 0, false>, k_thermo<true, 6, false>, k_thermo<true, kMaxObs, false>}},
                                         {{k_thermo<false, 0, true>, k_thermo<false, 6, true>, k_thermo<false, kMaxObs, true>},
                                          {k_thermo<true, 0, true>, k_thermo<true, 6, true>, k_thermo<true, kMaxObs, true>}}};
        const Kernel fn = kernels[a.team > 1 ? 1 : 0][fits ? 1 : 0][num_obs == 0 ? 0 : num_obs <= 6 ? 1 : 2];
        e = cudaFuncSetAttribute(reinterpret_cast<const void*>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
        if (e == cudaSuccess) {
            const int teams = kWarps / a.team, grid = std::min((num_T + teams - 1) / teams, nsm);
            fn<<<grid, 32 * kWarps, fits ? staged : table, st>>>(a);
            e = cudaGetLastError();
        }
    }
    const size_t rows = (size_t)num_T * nrow, results = num_T + rows;
    if (results <= kSmall) {
        if (e == cudaSuccess) e = cudaMemcpyAsync(small, a.temps, results * 8, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e == cudaSuccess) {
            std::copy(small, small + num_T, temperatures);
            std::copy(small + num_T, small + results, out);
        }
    } else {
        if (e == cudaSuccess) e = cudaMemcpyAsync(out, a.out, rows * 8, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(temperatures, a.temps, (size_t)num_T * 8, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    cudaStreamDestroy(st);
    cudaFree(d);
    if (e != cudaSuccess) return tfail(REWL_EDEVICE, "thermodynamics: %s", cudaGetErrorString(e));
    return REWL_OK;
}

// Susceptibilities and Binder cumulants from the rows of rewl_thermodynamics
// (order_parameter_cumulants.hpp:17-48; calculate_nonlinear_observables,
// ising2d_observables.hpp:166-198 and ashkin_teller2d_observables.hpp:243-282).
int rewl_nonlinear_observables(int32_t model, int32_t correlators, const double* rows, int32_t num_T,
                               int32_t row_len, const double* temperatures, double system_size, double* out)
{
    const bool corr = correlators != 0;
    const int need = 5 + (model == REWL_MODEL_ISING2D ? (corr ? 4 : 3) : (corr ? 16 : 12));
    if (!rows || !temperatures || !out || num_T < 1 || row_len < need || (correlators != 0 && correlators != 1) ||
        (model != REWL_MODEL_ISING2D && model != REWL_MODEL_ASHKIN_TELLER2D))
        return tfail(REWL_EINVAL, "bad arguments (rows of at least %d columns)", need);
    auto susc = [&](double m2, double m, double T) { return system_size * (m2 - m * m) / T; };
    auto binder = [](double m4, double m2) { return 1.0 - (m4 / (m2 * m2)) / 3.0; };
    // calculate_correlation_length(G0, Gq, L) / L with L = (size_t) sqrt(N)
    const size_t Ls = static_cast<size_t>(std::sqrt(system_size));
    auto xi = [&](double G0, double Gq) {
        const double x = Gq == 0. ? DBL_MAX : (static_cast<double>(Ls) / (2. * std::acos(-1.))) * std::sqrt((G0 - Gq) / Gq);
        return x / static_cast<double>(Ls);
    };
    for (int t = 0; t < num_T; ++t) {
        const double* o = rows + (size_t)t * row_len + 5;
        const double T = temperatures[t];
        if (model == REWL_MODEL_ISING2D) {
            double* r = out + (size_t)t * (corr ? 3 : 2);
            r[0] = susc(o[1], o[0], T);
            r[1] = binder(o[2], o[1]);
            if (corr) r[2] = xi(o[1], o[3]);
        } else if (!corr) {
            double* r = out + 8 * (size_t)t;
            const int bases[3] = {0, 3, 9};            // sigma, tau, Baxter
            for (int k = 0; k < 3; ++k) {
                r[2 * k] = susc(o[bases[k] + 1], o[bases[k]], T);
                r[2 * k + 1] = binder(o[bases[k] + 2], o[bases[k] + 1]);
            }
            r[6] = susc(o[7], o[6], T);                 // phi: two-component order parameter
            r[7] = 2.0 * (1.0 - 0.5 * (o[8] / (o[7] * o[7])));
        } else {
            // groups of (|x|, x^2, x^4, G): sigma 0, tau 4, phi 8, Baxter 12; output order
            // sigma, tau, Baxter, phi with (susceptibility, cumulant, correlation length)
            double* r = out + 12 * (size_t)t;
            const int bases[3] = {0, 4, 12};
            for (int k = 0; k < 3; ++k) {
                const double* g = o + bases[k];
                r[3 * k] = susc(g[1], g[0], T);
                r[3 * k + 1] = binder(g[2], g[1]);
                r[3 * k + 2] = xi(g[1], g[3]);
            }
            const double* g = o + 8;
            r[9] = susc(g[1], g[0], T);
            r[10] = 2.0 * (1.0 - 0.5 * (g[2] / (g[1] * g[1])));
            r[11] = xi(g[1], g[3]);
        }
    }
    return REWL_OK;
}

} // extern "C"
