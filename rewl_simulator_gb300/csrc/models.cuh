// The model plugin surface: the reference's Hamiltonian/observables plugins
// (Hamiltonian_t<T>, State_t<T>, Observables_t<T> chosen at compile time,
// src/Hamiltonians/model_hamiltonians.hpp:6-40) as device-side model types.  A
// model type provides, for a configuration held as int8 +-1 planes (Ising: one
// plane; Ashkin-Teller: sigma then tau) on the L x L periodic square lattice with
// site = y L + x:
//   delta_at          energy change of flipping plane a's spin at a site (b the other plane), given its
//                     neighbours; delta_energy works them out
//   flipped_at        the change of that where the neighbour j in plane a has flipped (left_flipped,
//                     right_flipped: the same for a site's left and right neighbour)
//   recalculate       energy and magnetisations from scratch
//   flip              apply a flip and update the magnetisations
//   add_observables   the per-bin moments of update_observables for the current magnetisations
//   add_correlators   the per-bin G(q_min) transforms of the whole configuration
// and, for the sweep kernels' per-chunk bookkeeping,
//   flip_signs        for each magnetisation, the sign of the site's term before a flip of
//                     plane a (the flip changes it by -2 sign; 0: unchanged)
//   corr_site         a site's value in each correlator plane
//   mag_terms         a site's term in each magnetisation
//   add_transforms    the G(q_min) of each correlator plane into the observable columns
// kPlanes spin planes, kMags magnetisations, kCorrPlanes correlator planes, corr_mag[p]
// the magnetisation whose terms are correlator plane p's values.
// Energies are integers in the model's units (Ising: J; Ashkin-Teller: 2^-20, with the
// Baxter fields quantised to that grid), so every sum is exact.  The sweep kernels and the
// initial walk are written against these functions; the engine dispatches on the
// per-instance model id (no runtime multi-backend).
#pragma once

#include <cstdint>

__host__ __device__ inline int nb_up(int i, int L) { int x = i % L, y = i / L; return (y == 0 ? L - 1 : y - 1) * L + x; }
__host__ __device__ inline int nb_left(int i, int L) { int x = i % L, y = i / L; return y * L + (x == 0 ? L - 1 : x - 1); }
__host__ __device__ inline int nb_right(int i, int L) { int x = i % L, y = i / L; return y * L + (x == L - 1 ? 0 : x + 1); }
__host__ __device__ inline int nb_down(int i, int L) { int x = i % L, y = i / L; return (y == L - 1 ? 0 : y + 1) * L + x; }

// a site's neighbours (site indices)
struct Neighbours {
    int up, left, right, down;
};
__host__ __device__ inline Neighbours neighbours(int i, int L) { return {nb_up(i, L), nb_left(i, L), nb_right(i, L), nb_down(i, L)}; }

// adds v to *p in global memory (atomicAdd on a pointer whose address space the compiler does not know
// asks for it at every use, and takes a compare-and-swap loop for shared memory along)
__device__ __forceinline__ void red_global_add(double* p, double v)
{
    asm volatile("red.global.add.f64 [%0], %1;" :: "l"(__cvta_generic_to_global(p)), "d"(v) : "memory");
}

// Conversions to FP64 without the conversion instructions (95 cycles each, and FP64's pipe): a
// whole number |v| < 2^51 as the low bits of 1.5 x 2^52 + v, less 1.5 x 2^52; a positive normal float by its
// exponent and fraction fields (zero stays zero).
__device__ __forceinline__ double whole_double(long long v)
{
    return __longlong_as_double(0x4338000000000000ll + v) - 6755399441055744.0;
}
__device__ __forceinline__ double float_double(float f)
{
    const unsigned u = __float_as_uint(f);
    return __hiloint2double(u == 0 ? 0 : (int)((u >> 3) + (896u << 20)), (int)(u << 29));
}

// Square root of a whole number below 2^31 to FP64's last place: Newton's iteration on x^2 = k with the residual
// in one fused operation, twice, from the single-precision root (22 -> 43 -> more than 53 places)
__device__ inline double whole_root(unsigned k)
{
    const float y = k == 0 ? 0.f : rsqrtf((float)k);
    const double kd = whole_double(k), half = float_double(0.5f * y);
    double x = float_double((float)k * y);
    x = fma(fma(-x, x, kd), half, x);
    return fma(fma(-x, x, kd), half, x);
}

// nearest-neighbour and four-spin couplings in energy units (T: 64 bits, or 32 where the caller knows
// that four times their sum fits)
template <class T>
struct CouplingsOf {
    T J, K;
};
using Couplings = CouplingsOf<int64_t>;

// Fourier_Correlator::compute_correlator (src/Hamiltonians/Correlations/fourier_correlator.hpp:
// 65-118) of plane a, or of the product plane a * b, in the reference's order (one thread):
// half the squared magnitude of the transform of the row sums over y plus that of every site
// over its column x, both at q_min = 2 pi / L (q: L cosines then L sines).
__device__ inline double full_corr(const int8_t* a, const int8_t* b, const double* q, int L)
{
    double rx = 0.0, ix = 0.0, ry = 0.0, iy = 0.0;
    for (int y = 0; y < L; ++y) {
        int rsum = 0;
        for (int x = 0; x < L; ++x) {
            const int v = b ? a[y * L + x] * b[y * L + x] : a[y * L + x];
            rsum += v;
            ry += (double)v * q[x];
            iy += (double)v * q[L + x];
        }
        rx += (double)rsum * q[y];
        ix += (double)rsum * q[L + y];
    }
    return 0.5 * ((rx * rx + ix * ix) + (ry * ry + iy * iy));
}

// 2D Ising, H = -J sum_<ij> s_i s_j (src/Hamiltonians/Ising2d/ising2d_hamiltonian.hpp:162-256).
// One magnetisation M; observables |m|, m^2, m^4 with m = M / N, and G(q_min) of the spins.
struct Ising2dModel {
    static constexpr int kPlanes = 1;
    static constexpr int kMoments = 3;
    static constexpr int kGroups = 1;
    static constexpr int kMags = 1;
    static constexpr int kCorrPlanes = 1;
    __host__ __device__ static constexpr int corr_mag(int) { return 0; }

    __host__ __device__ static void flip_signs(int a, int, int, int* sg) { sg[0] = a; }
    __host__ __device__ static int corr_site(const int8_t* sp, int, int i, int) { return sp[i]; }
    __host__ __device__ static void mag_terms(const int8_t* sp, int, int i, int* t) { t[0] = sp[i]; }
    __device__ static void add_transforms(double* o, const double* G, double in2) { red_global_add(o + 3, in2 * G[0]); }

    template <class T>
    __host__ __device__ static T delta_at(const int8_t* a, const int8_t*, int i, Neighbours n, CouplingsOf<T> c, T)
    {
        const int sum = a[n.up] + a[n.left] + a[n.right] + a[n.down];
        return 2 * (T)a[i] * c.J * sum;
    }
    template <class T>
    __host__ __device__ static T flipped_at(const int8_t* a, const int8_t*, int i, int j, CouplingsOf<T> c)
    {
        return -4 * (T)a[i] * a[j] * c.J;
    }
    __host__ __device__ static int64_t delta_energy(const int8_t* a, const int8_t* b, int i, int L, Couplings c, int64_t h)
    {
        return delta_at(a, b, i, neighbours(i, L), c, h);
    }
    __host__ __device__ static int64_t left_flipped(const int8_t* a, const int8_t* b, int i, int L, Couplings c, int64_t d0)
    {
        return d0 + flipped_at(a, b, i, nb_left(i, L), c);
    }
    __host__ __device__ static int64_t right_flipped(const int8_t* a, const int8_t* b, int i, int L, Couplings c)
    {
        return flipped_at(a, b, i, nb_right(i, L), c);
    }
    // E recomputed as sum_i -1/2 s_i J sum_nb s_nb (ising2d_hamiltonian.hpp:191-210)
    __host__ __device__ static void recalculate(const int8_t* sp, int L, Couplings c, const int64_t*, int64_t& E, int32_t* M)
    {
        const int N = L * L;
        int64_t twiceE = 0;
        int32_t m = 0;
        for (int i = 0; i < N; ++i) {
            const int sum = sp[nb_up(i, L)] + sp[nb_left(i, L)] + sp[nb_right(i, L)] + sp[nb_down(i, L)];
            twiceE -= (int64_t)sp[i] * c.J * sum;
            m += sp[i];
        }
        E = twiceE / 2;
        M[0] = m;
    }
    __host__ __device__ static void flip(int8_t* sp, int, int i, int, int32_t* M)
    {
        M[0] -= 2 * sp[i];
        sp[i] = (int8_t)-sp[i];
    }
    // Ising2d::update_observables (ising2d_hamiltonian.hpp:234-256)
    __device__ static void add_observables(double* o, const int32_t* M, double invN, int)
    {
        const double m = invN * fabs((double)M[0]);
        red_global_add(o, m);
        red_global_add(o + 1, m * m);
        red_global_add(o + 2, m * m * m * m);
    }
    // the same from whole numbers, one group of moments (kGroups) at a time
    __device__ static void add_group(double* o, int, const int32_t* M, double invN, double, int)
    {
        const double m = invN * (double)(unsigned)abs(M[0]), m2 = m * m;
        red_global_add(o, m);
        red_global_add(o + 1, m2);
        red_global_add(o + 2, m2 * m2);
    }
    // CORRELATION_LENGTHS (ising2d_hamiltonian.hpp:246-252): G after the three moments
    __device__ static void add_correlators(double* o, const int8_t* sp, int, int L, const double* q, double in2)
    {
        red_global_add(o + 3, in2 * full_corr(sp, nullptr, q, L));
    }
};

// 2D Ashkin-Teller with Baxter fields, H = -sum_<ij>[J(s s' + t t') + K s t s' t'] - sum_i h_i s_i t_i
// (src/Hamiltonians/Ashkin_Teller2d/ashkin_teller2d_hamiltonian.hpp:53-62,169-318).  Planes sigma
// and tau; magnetisations sigma, tau and Baxter (sigma tau); the 12 moments of |sigma|, |tau|, phi =
// sqrt(sigma^2 + tau^2) and |Baxter|, and their G(q_min) (tau's from sigma, as the reference does).
struct AshkinTeller2dModel {
    static constexpr int kPlanes = 2;
    static constexpr int kMoments = 12;
    static constexpr int kGroups = 2;
    static constexpr int kMags = 3;          // sigma, tau, Baxter
    static constexpr int kCorrPlanes = 2;    // sigma, sigma * tau
    __host__ __device__ static constexpr int corr_mag(int p) { return p == 0 ? 0 : 2; }

    // a: the flipped plane's spin, b: the other plane's
    __host__ __device__ static void flip_signs(int a, int b, int plane, int* sg)
    {
        sg[0] = plane == 0 ? a : 0;
        sg[1] = plane == 0 ? 0 : a;
        sg[2] = a * b;
    }
    __host__ __device__ static int corr_site(const int8_t* sp, int N, int i, int p)
    {
        return p == 0 ? sp[i] : sp[i] * sp[N + i];
    }
    __host__ __device__ static void mag_terms(const int8_t* sp, int N, int i, int* t)
    {
        t[0] = sp[i];
        t[1] = sp[N + i];
        t[2] = sp[i] * sp[N + i];
    }
    // the tau correlator is computed from sigma, as the reference does (ashkin_teller2d_hamiltonian.hpp:
    // 298-299); phi's is the sum of the two
    __device__ static void add_transforms(double* o, const double* G, double in2)
    {
        const double gs = in2 * G[0], gb = in2 * G[1];
        red_global_add(o + 3, gs); red_global_add(o + 7, gs); red_global_add(o + 11, gs + gs); red_global_add(o + 15, gb);
    }

    template <class T>
    __host__ __device__ static T delta_at(const int8_t* a, const int8_t* b, int i, Neighbours n, CouplingsOf<T> c, T h)
    {
        const int u = n.up, l = n.left, r = n.right, d = n.down;
        const int sa = a[u] + a[l] + a[r] + a[d];
        const int sab = a[u] * b[u] + a[l] * b[l] + a[r] * b[r] + a[d] * b[d];
        return 2 * (T)a[i] * (h * b[i] + c.J * sa + c.K * (T)b[i] * sab);
    }
    template <class T>
    __host__ __device__ static T flipped_at(const int8_t* a, const int8_t* b, int i, int j, CouplingsOf<T> c)
    {
        return -4 * (T)a[i] * a[j] * (c.J + c.K * (T)b[i] * b[j]);
    }
    __host__ __device__ static int64_t delta_energy(const int8_t* a, const int8_t* b, int i, int L, Couplings c, int64_t h)
    {
        return delta_at(a, b, i, neighbours(i, L), c, h);
    }
    __host__ __device__ static void recalculate(const int8_t* sp, int L, Couplings c, const int64_t* h, int64_t& E, int32_t* M)
    {
        const int N = L * L;
        const int8_t* s = sp;
        const int8_t* t = sp + N;
        int64_t twiceE = 0;
        int32_t sm = 0, tm = 0, bx = 0;
        for (int i = 0; i < N; ++i) {
            const int u = nb_up(i, L), l = nb_left(i, L), r = nb_right(i, L), d = nb_down(i, L);
            const int ss = s[u] + s[l] + s[r] + s[d];
            const int tt = t[u] + t[l] + t[r] + t[d];
            const int st = s[u] * t[u] + s[l] * t[l] + s[r] * t[r] + s[d] * t[d];
            twiceE -= (int64_t)s[i] * c.J * ss + (int64_t)t[i] * c.J * tt + (int64_t)s[i] * t[i] * c.K * st;
            if (h) twiceE -= 2 * h[i] * s[i] * t[i];
            sm += s[i]; tm += t[i]; bx += s[i] * t[i];
        }
        E = twiceE / 2;
        M[0] = sm; M[1] = tm; M[2] = bx;
    }
    __host__ __device__ static void flip(int8_t* sp, int N, int i, int plane, int32_t* M)
    {
        int8_t* s = sp;
        int8_t* t = sp + N;
        M[2] -= 2 * s[i] * t[i];
        if (plane == 0) { M[0] -= 2 * s[i]; s[i] = (int8_t)-s[i]; }
        else { M[1] -= 2 * t[i]; t[i] = (int8_t)-t[i]; }
    }
    // Ashkin_Teller2d::update_observables (ashkin_teller2d_hamiltonian.hpp:267-318); with
    // correlators each group of three moments is followed by its G(q_min) column
    // (ashkin_teller2d_observables.hpp:36-41)
    __device__ static void add_observables(double* o, const int32_t* M, double invN, int corr)
    {
        const double a = invN * fabs((double)M[0]), t = invN * fabs((double)M[1]), b = invN * fabs((double)M[2]);
        const double p2 = a * a + t * t;
        const int g = corr ? 1 : 0;
        red_global_add(o + 0, a); red_global_add(o + 1, a * a); red_global_add(o + 2, a * a * a * a);
        o += g;
        red_global_add(o + 3, t); red_global_add(o + 4, t * t); red_global_add(o + 5, t * t * t * t);
        o += g;
        red_global_add(o + 6, sqrt(p2)); red_global_add(o + 7, p2); red_global_add(o + 8, p2 * p2);
        o += g;
        red_global_add(o + 9, b); red_global_add(o + 10, b * b); red_global_add(o + 11, b * b * b * b);
    }
    // The same from whole numbers, in two groups: sigma and tau, Baxter and phi.  FP64 bounds it (an
    // instruction takes 32 cycles of an SM, its result 65), and CUDA's sqrt most of all (670 cycles):
    // twelve instructions a group, the root included, which leave room for one another.
    // Magnetisations are at most 128 x 128.
    __device__ static void add_group(double* o, int group, const int32_t* M, double invN, double in2, int corr)
    {
        const int c = 3 + (corr ? 1 : 0);
        const unsigned m = (unsigned)abs(group == 0 ? M[0] : M[2]);
        const unsigned k = (unsigned)(M[1] * M[1]) + (group == 0 ? 0u : (unsigned)(M[0] * M[0]));
        // (m is exact in single precision)
        const double a = invN * float_double((float)m), b = invN * whole_root(k), a2 = a * a, b2 = in2 * whole_double(k);
        double* const oa = o + (group == 0 ? 0 : 3 * c);
        double* const ob = o + (group == 0 ? c : 2 * c);
        red_global_add(oa, a); red_global_add(oa + 1, a2); red_global_add(oa + 2, a2 * a2);
        red_global_add(ob, b); red_global_add(ob + 1, b2); red_global_add(ob + 2, b2 * b2);
    }
    // CORRELATION_LENGTHS (ashkin_teller2d_hamiltonian.hpp:295-315): the tau correlator is
    // computed from sigma as in the reference (:298-299); phi's is the sum of the two
    __device__ static void add_correlators(double* o, const int8_t* sp, int N, int L, const double* q, double in2)
    {
        const double gs = in2 * full_corr(sp, nullptr, q, L);
        const double gb = in2 * full_corr(sp, sp + N, q, L);
        red_global_add(o + 3, gs); red_global_add(o + 7, gs); red_global_add(o + 11, gs + gs); red_global_add(o + 15, gb);
    }
};
