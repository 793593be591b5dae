// GB300 replica-exchange Wang-Landau engine: host driver, device kernels and
// the C ABI declared in include/rewl.h.
//
// Device layout (HBM), structure of arrays:
//   walker slots  s = first_slot(instance) + window * R + replica
//       slot_cfg[s]      configuration currently held by the slot (an exchange
//                        swaps two entries instead of moving lattices)
//       slot_tab[s]      offset of the slot's tables: g (int64, 2^-36 units),
//                        H (uint32 per-stage counts), visits (uint64 cumulative)
//       slot_sweeps[s]   sweeps done (Philox attempt counter base)
//       slot_flavour[s]  Ashkin-Teller which_to_update
//   configurations c: spins (int8; Ising N, Ashkin-Teller sigma plane then tau
//       plane), energy (int64 units of 2^-escale), magnetisations (int32 x3)
//   windows: ln f (int64 2^-36 units), done / 1/t flags, counters, valid-bin mask
//
// Kernels
//   k_init          one thread per walker: initial spins from Philox, then the
//                   deterministic walk into the window (rewl_walker.hpp:79-115)
//   k_sweep_ising_bins  one, two or four walkers per warp; lattice, window table and
//                   thresholds in shared memory; several sites decided at a time on
//                   a binary tree of outcomes (the default Ising kernel)
//   k_sweep_ising_rows  the same one decision after another: short rows in crowded launches
//   k_sweep_ising   one warp per walker; lattice, g and H staged in shared
//                   memory; lanes precompute a row-aligned chunk of <= 32 sites
//                   (energy change with and without the left neighbour flipped,
//                   integer acceptance threshold), lane 0 resolves the serial
//                   Wang-Landau chain in integer arithmetic only (replay, bin
//                   widths that do not divide 4J)
//   k_sweep_tables  any model type of models.cuh with the tables in global memory
//                   (Ashkin-Teller: one plane per pass; Ising windows too large for
//                   shared memory): the tree, with the bins around the walker in
//                   shared memory, or the serial chain
//   k_export_*, k_report  results and counters into pinned host memory
//   k_exchange      one thread per window pair (rewl_simulation.hpp:228-346)
//   k_flat          one block per window: flatness vote, FP64 count-weighted
//                   averaging, histogram reset, REDUCE_LOGDOS, ln f schedule
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cfloat>
#include <cstdarg>
#include <cstddef>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <filesystem>
#include <fstream>
#include <iomanip>
#include <limits>
#include <mutex>
#include <new>
#include <random>
#include <sstream>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/rewl.h"
#include "rng.cuh"
#include "models.cuh"

using namespace rewl;

namespace {

thread_local std::string g_last_error;

int fail(int code, const char* fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_last_error = buf;
    return code;
}

#define CUDA_TRY(expr)                                                                 \
    do {                                                                               \
        cudaError_t _e = (expr);                                                       \
        if (_e != cudaSuccess)                                                         \
            return fail(REWL_EDEVICE, "%s: %s (%s:%d)", #expr, cudaGetErrorString(_e), \
                        __FILE__, __LINE__);                                           \
    } while (0)

constexpr int kMaxReplicas = 64;
constexpr uint32_t kFull = 0xFFFFFFFFu;

enum : int { ERR_BOUNDS = 1, ERR_ADJUST = 2, ERR_REPLAY_EXHAUSTED = 4, ERR_RANGE = 8, ERR_COUNT = 16 };
// |logDoS| at which a window is reported (REWL_ESTATE) instead of risking int64 overflow: 2^62
// units (6.7e7 nats).  Every kernel that adds to g checks the values it wrote against it, and
// every kernel returns without work once the error word is set, so at most one launch's growth
// lies beyond the limit.  The host splits sweep launches so that one launch adds at most
// kLaunchGrowth to any bin (ln f bound x sweeps x degrees of freedom, plus one exchange visit):
// 2^62 + 2^62 - 2^58 stays below 2^63 with room for the acceptance thresholds (< 2^45).
constexpr long long kLogdosLimit = 1LL << 62;
constexpr double kSetLogdosMax = 16777216.0;                // 2^60 units: the largest |g| rewl_set_logdos takes
constexpr long long kLaunchGrowth = (1LL << 62) - (1LL << 58);

// Any device error stops further work: a kernel that finds the error word set returns at once.
// Another block may set the word while this one reads it, so a warp acts on lane 0's reading
// (all 32 lanes must be active) and a block on thread 0's.
__device__ __forceinline__ bool engine_failed(const int32_t* counters)
{
    return *reinterpret_cast<const volatile int32_t*>(counters) != 0;
}
__device__ __forceinline__ bool engine_failed_warp(const int32_t* counters)
{
    return __shfl_sync(0xFFFFFFFFu, (int)engine_failed(counters), 0) != 0;
}

// A launch's derived visits to bin k (its logDoS change over ln f) into the per-stage count
// (uint32, the reference keeps uint64: a count that would pass 2^32 - 1 saturates and is
// reported) and the cumulative visits; also checks the new logDoS against the range limit.
__device__ __forceinline__ int commit_visits(uint32_t* gH, uint64_t* gv, int k, uint32_t h, uint64_t v, long long dv,
                                             long long gnew)           // (h, v: what gH[k], gv[k] hold)
{
    int err = 0;
    const unsigned long long sum = (unsigned long long)h + (unsigned long long)dv;
    if (sum > 0xFFFFFFFFull) err |= ERR_COUNT;
    gH[k] = sum > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)sum;
    gv[k] = v + (uint64_t)dv;
    if (gnew >= kLogdosLimit) err |= ERR_RANGE;
    return err;
}
__device__ __forceinline__ int commit_visits(uint32_t* gH, uint64_t* gv, int k, long long dv, long long gnew)
{
    return commit_visits(gH, gv, k, gH[k], gv[k], dv, gnew);
}

struct InstDev {
    int32_t model, L, N, ndof;
    int32_t nwin, R, first_win, first_slot;
    int32_t bin_shift, escale, chunk, init_mode;
    int64_t J_u, K_u;        // couplings in energy units
    int64_t eglo_u;          // global range start in energy units
    int64_t bin_mul;         // global bin = ((E - eglo_u) * bin_mul) >> bin_shift
    int64_t field_off;       // offset into fields (int64 units per site) or -1
    int64_t qtab_off;        // offset into qtab (cos then sin of q_min x, x < L) or -1 without correlators
    uint64_t seed;           // Philox key: instance_key(descriptor seed)
};

struct WinDev {
    int32_t inst, local, nb, pad;
    int64_t gblo;            // first global bin
    int64_t mask_off;        // offset into the mask array
    int64_t elo_u;           // lower energy edge in units (exact when bin_mul == 1)
};

struct DevPtrs {
    InstDev* inst;
    WinDev* win;
    int32_t* slot_inst;
    int32_t* slot_win;
    int32_t* slot_cfg;
    int64_t* slot_tab;
    int32_t* slot_nb;
    int32_t* slot_flavour;
    uint64_t* slot_sweeps;
    int64_t* slot_draws;
    int64_t* slot_thr_off;
    int64_t* slot_thr_n;
    int64_t* thr;            // replay thresholds
    int64_t* cfg_off;
    int8_t* spins;
    int64_t* cfg_E;
    int32_t* cfg_M;          // 3 per configuration
    int64_t* fields;         // Baxter field per site (units)
    int64_t* g;
    int64_t* gsnap;          // global-table serial chain: logDoS at the start of a sweep launch
    uint32_t* H;
    uint64_t* visits;
    uint8_t* mask;
    int64_t* win_lnf;
    int32_t* win_done;
    int32_t* win_oot;
    uint64_t* win_iter;
    uint64_t* win_sweepctr;
    int32_t* pairs;          // exchange pair lists: (instance, lower window) for dir 0 then dir 1
    int32_t* counters;       // [0] error word, [1] flat events (this call)
    unsigned long long* xround;  // [0] exchange round (its parity is the pairing direction), [1] blocks done
    unsigned long long* stats;  // [0] exch attempted, [1] exch accepted
    double* obs;             // per-bin observable sums (obs_stride per bin), or null when off
    int obs_stride;          // 3 (Ising) or 12 (a batch with Ashkin-Teller instances); 4 or 16 with correlators
    int corr;                // observables carry the G(q_min) correlators
    const double* qtab;      // per instance: cos(q_min x) then sin(q_min x), x < L
    const int2* qfix;        // the same in units of 2^-30 (x) and 2^-60 (y)
};

// --------------------------------------------------------------------------
// Energies in integer units: the model types of models.cuh
// --------------------------------------------------------------------------
__host__ __device__ inline int64_t global_bin(const InstDev& I, int64_t E)
{
    return ((E - I.eglo_u) * I.bin_mul) >> I.bin_shift;
}

// --------------------------------------------------------------------------
// k_init: initial configuration and the deterministic walk into the window
// --------------------------------------------------------------------------
// REWL_Walker::adjust_state_to_range (src/REWL/rewl_walker.hpp:79-115): visit the sites in
// typewriter order from `start`, flipping a spin whenever that moves the energy towards the
// window, until the energy is inside it.  Ashkin-Teller alternates the flipped plane at the
// end of every pass (change_state toggles at the last site).
template <class Model>
__device__ bool adjust_walk(const InstDev& I, const WinDev& W, int8_t* sp, int64_t& E, int32_t* M, int32_t& flavour,
                            const int64_t* h, uint32_t start, int64_t max_steps)
{
    const int L = I.L, N = I.N;
    const Couplings cp{I.J_u, I.K_u};
    auto in_range = [&](int64_t e) { const int64_t b = global_bin(I, e) - W.gblo; return b >= 0 && b < W.nb; };
    bool in = in_range(E);
    int site = (int)start;
    int64_t steps = 0, idle = 0;
    while (!in) {
        // without a flip the decisions repeat within 2N steps: the walk is stuck for good
        if (++steps > max_steps || ++idle > 2 * (int64_t)N) return false;
        ++site;
        if (site == N) { site = 0; flavour ^= 1; }
        const int plane = Model::kPlanes == 1 ? 0 : flavour;
        const int8_t* a = sp + plane * N;
        const int8_t* b = sp + (plane ^ 1) * N;
        const int64_t dE = Model::delta_energy(a, b, site, L, cp, h ? h[site] : 0);
        if (Model::kPlanes == 2 && site == N - 1) flavour ^= 1;     // change_state toggles at the last site
        const int64_t gb = global_bin(I, E) - W.gblo;
        const bool too_low = gb < 0, too_high = gb >= W.nb;
        const int64_t En = E + dE;
        if ((too_low && En > E) || (too_high && En <= E)) {
            E = En;
            idle = 0;
            Model::flip(sp, N, site, plane, M);      // the plane chosen before a toggle
        }
        in = in_range(E);
    }
    return true;
}

template <class Model>
__device__ void init_walker(const InstDev& I, const WinDev& W, int8_t* sp, const int64_t* h, uint32_t uid,
                            int64_t& E, int32_t* M, int32_t& flavour, bool& ok)
{
    const Couplings cp{I.J_u, I.K_u};
    const int init_random = (int)(I.init_mode == 0);
    for (int i = 0; i < I.ndof; ++i)
        sp[i] = init_random ? ((philox_word(I.seed, uid, (uint64_t)i, kStreamInit) >> 31) ? -1 : 1) : 1;
    Model::recalculate(sp, I.L, cp, h, E, M);
    flavour = 0;
    const uint32_t start = mulhi32(philox_word(I.seed, uid, 0, kStreamAdjust), (uint32_t)I.N);
    const int64_t cap = 4000LL * I.ndof;
    ok = adjust_walk<Model>(I, W, sp, E, M, flavour, h, start, cap);
    // a greedy walk can stick in a local extremum: retry from all +1 (walks up
    // from the ground state) and then from the checkerboard (walks down from the top)
    for (int attempt = 1; attempt <= 2 && !ok; ++attempt) {
        for (int i = 0; i < I.ndof; ++i) {
            const int site = i % I.N, x = site % I.L, y = site / I.L;
            sp[i] = (attempt == 1 || ((x + y) & 1) == 0) ? 1 : -1;
        }
        Model::recalculate(sp, I.L, cp, h, E, M);
        flavour = 0;
        ok = adjust_walk<Model>(I, W, sp, E, M, flavour, h, start, cap);
    }
}

__global__ void k_init(DevPtrs P, int nslots, int init_mode_mask_unused)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nslots) return;
    const int ii = P.slot_inst[s];
    const InstDev I = P.inst[ii];
    const WinDev W = P.win[P.slot_win[s]];
    const int c = P.slot_cfg[s];
    int8_t* sp = P.spins + P.cfg_off[c];
    const uint32_t uid = (uint32_t)(s - I.first_slot);
    const int64_t* h = I.field_off >= 0 ? P.fields + I.field_off : nullptr;
    int64_t E = 0; int32_t M[3] = {0, 0, 0}; int32_t flavour = 0;
    bool ok = false;
    if (I.model == REWL_MODEL_ISING2D) init_walker<Ising2dModel>(I, W, sp, h, uid, E, M, flavour, ok);
    else init_walker<AshkinTeller2dModel>(I, W, sp, h, uid, E, M, flavour, ok);
    if (!ok) atomicOr(&P.counters[0], ERR_ADJUST);
    P.cfg_E[c] = E;
    P.cfg_M[3 * c] = M[0]; P.cfg_M[3 * c + 1] = M[1]; P.cfg_M[3 * c + 2] = M[2];
    P.slot_flavour[s] = flavour;
}

// Recompute energies and magnetisations of given configurations (after imports).
__global__ void k_recalc(DevPtrs P, const int32_t* cfgs, const int32_t* insts, int n)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int c = cfgs[k];
    const InstDev I = P.inst[insts[k]];
    const int8_t* sp = P.spins + P.cfg_off[c];
    const int64_t* h = I.field_off >= 0 ? P.fields + I.field_off : nullptr;
    int64_t E; int32_t M[3] = {0, 0, 0};
    const Couplings cp{I.J_u, I.K_u};
    if (I.model == REWL_MODEL_ISING2D) Ising2dModel::recalculate(sp, I.L, cp, h, E, M);
    else AshkinTeller2dModel::recalculate(sp, I.L, cp, h, E, M);
    P.cfg_E[c] = E;
    P.cfg_M[3 * c] = M[0]; P.cfg_M[3 * c + 1] = M[1]; P.cfg_M[3 * c + 2] = M[2];
}

// --------------------------------------------------------------------------
// Sweep kernels
// --------------------------------------------------------------------------
// Per-bin observable sums (observables on): for every attempted flip and every
// exchange touch, the walker's observables after it are added at its bin.  Ising:
// |m|, m^2, m^4 with m = M / N (Ising2d::update_observables,
// src/Hamiltonians/Ising2d/ising2d_hamiltonian.hpp:234-256); Ashkin-Teller: the 12
// moments of Ashkin_Teller2d::update_observables (ashkin_teller2d_hamiltonian.hpp:267-318).
// The reference keeps running means (v + c avg) / (c + 1) (ising2d_observables.hpp:134-145);
// the export divides these sums by the visits instead, equal up to FP64 rounding.
// G(q_min) correlators (CORRELATION_LENGTHS, on in the reference's default build).  At
// every visit of a bin whose count before the visit is a multiple of counts_per_transform
// = 1000 (src/Hamiltonians/Correlations/fourier_correlator.hpp:11), the walker's G is added
// at the bin (Ising2d::update_observables, ising2d_hamiltonian.hpp:246-252;
// Ashkin_Teller2d::update_observables, ashkin_teller2d_hamiltonian.hpp:295-315).  The
// reference keeps the running mean over those transforms (ising2d_observables.hpp:148-159);
// the export divides the sum by their number, ceil(visits / 1000).
constexpr unsigned long long kCountsPerTransform = 1000;

// Fourier_Correlator::compute_correlator (fourier_correlator.hpp:65-118) of one plane of
// +-1 values v(y, x): half the squared magnitude of the transform of the row sums over y
// plus that of the column sums over x, both at q_min = 2 pi / L (q: L cosines then L sines).
// rs and cs are the plane's row and column sums before the chunk; the chunk (row y,
// columns x0 ..) has flipped the sites of its steps 0..j whose acceptance bit is set: row
// y changes by dr and column x0 + k by -2 val(k), val(k) the site's value before the
// chunk.  The reference adds the same products site by site in row-major order; the two
// agree to FP64 rounding.
template <class V>
__device__ double plane_corr(const int* rs, const int* cs, const double* q, int L, int y, int dr, int x0, int j,
                             unsigned acc, V val)
{
    double rx = 0.0, ix = 0.0, ry = 0.0, iy = 0.0;
    for (int t = 0; t < L; ++t) {
        const double c = q[t], sn = q[L + t];
        const double r = (double)(rs[t] + (t == y ? dr : 0));
        const int k = t - x0;
        const int cl = cs[t] - ((k >= 0 && k <= j && ((acc >> k) & 1u)) ? 2 * val(k) : 0);
        rx += r * c;
        ix += r * sn;
        ry += (double)cl * c;
        iy += (double)cl * sn;
    }
    return 0.5 * ((rx * rx + ix * ix) + (ry * ry + iy * iy));
}

// The same by P lanes together, for the step that all of them name: lane l takes the quantity
// l % (4 NC) -- of its plane l / 4 % NC: the cosine and sine sums over rows, then over columns --
// and of its terms every P / (4 NC)-th.  rs, cs, flips (accepted flips of the chunk that change
// the lane's plane, up to the step), up (the steps whose term was +1 before) are the lane's
// plane's; the plane's four lanes return 2 G.  The sums are whole numbers (sums times table
// entries of 60 binary places), so a term costs two integer multiplications instead of five FP64
// instructions at 32 cycles of an SM each, and the only rounding is of the table and of the
// final squares.
template <int P, int NC>
__device__ double plane_power(const int* rs, const int* cs, const int2* q, int L, int y, int x0, unsigned flips,
                              unsigned up, int lane)
{
    constexpr int NQ = 4 * NC;
    const bool col = (lane & 2) != 0;
    const int* v = col ? cs : rs;
    if (lane & 1) q += L;
    const int dr = -2 * ((int)__popc(flips & up) - (int)__popc(flips & ~up));
    long long hi = 0, lo = 0;                              // below 2^14 sites x 2^30
#pragma unroll 4
    for (int t = lane / NQ; t < L; t += P / NQ) {
        const int2 c = q[t];
        const int k = t - x0;
        const bool in = (unsigned)k < 32u && ((flips >> k) & 1u) != 0;
        int r = v[t];
        if (col) r -= !in ? 0 : (up >> k) & 1u ? 2 : -2;
        else r += t == y ? dr : 0;
        hi += (long long)r * c.x;
        lo += (long long)r * c.y;
    }
#pragma unroll
    for (int m = NQ; m < P; m *= 2) {
        hi += __shfl_xor_sync(kFull, hi, m);
        lo += __shfl_xor_sync(kFull, lo, m);
    }
    const double x = fma(whole_double(hi), 1.0 / 1073741824.0, whole_double(lo) * (1.0 / 1152921504606846976.0));
    double g = x * x;
    g += __shfl_xor_sync(kFull, g, 1);
    g += __shfl_xor_sync(kFull, g, 2);
    return g;
}

__device__ __forceinline__ int mod_transform(unsigned long long x)     // x % kCountsPerTransform
{
    static_assert(kCountsPerTransform == 1000, "2^32 = 296 modulo 1000");
    return (int)(((unsigned)(x >> 32) % 1000u * 296u + (unsigned)x % 1000u) % 1000u);
}

// Row and column sums of a plane (value(i) for site i) into rs, cs, by `stride` lanes.
template <class V>
__device__ void plane_sums(int* rs, int* cs, int L, int lane, V value, int stride = 32)
{
    for (int t = lane; t < L; t += stride) {
        int r = 0, c = 0;
        for (int u = 0; u < L; ++u) { r += value(t * L + u); c += value(u * L + t); }
        rs[t] = r;
        cs[t] = c;
    }
}

// flips of a chunk's steps 0..j that turned a +1 into -1 minus those that turned -1 into +1
__device__ __forceinline__ int chunk_dm(unsigned acc, unsigned plus, int j)
{
    const unsigned le = j >= 31 ? 0xFFFFFFFFu : ((2u << j) - 1u);
    return -2 * ((int)__popc(acc & plus & le) - (int)__popc(acc & ~plus & le));
}

struct SweepParams;
using SweepKernel = void (*)(const SweepParams);

struct SweepParams {
    DevPtrs P;
    const int32_t* slots;    // walkers of this launch
    int nslots;
    int nsweeps;
    int smem_per_warp;       // bytes
    int nbcap;               // table capacity per warp (Ising, shared memory)
    int counts;              // bin-tracking kernel: visit counts beside g in shared memory
    int moments;             // bin-tracking kernel with observables: moment sums in shared memory
    int cache;               // global-table kernel: bins of each walker's table in shared memory
};

// Per-warp staging of one chunk for the lane-0 resolver: energy change without /
// with the left neighbour flipped, wrap correction (x = L-1 sees the row start),
// acceptance threshold.
struct Stage {
    long long T[32];
    int d0[32];
    int d1[32];
    int wc[32];
    int seq[32];             // bin after each step (observables)
};

// Accept chain of one chunk of C sites, executed identically by all 32 lanes
// (every lane holds the same E, b, gc, acc).  Lane j owns site j's precomputed
// values; they reach every lane by shuffles that depend on nothing in the chain,
// so the unrolled loop issues them early.  The proposal of step j+1 depends on
// step j's outcome only through (E, left-neighbour flip, wrap flip): both
// candidates are formed and their logDoS entries loaded before step j resolves,
// which takes the shared-memory latency off the chain.  The only store that can
// land between such a prefetch and its use is step j's own, to the bin step j
// ends in: that case takes the freshly stored value.
template <int C>
__device__ __forceinline__ void resolve_chunk_all_lanes(int& E, int& b, long long& gc, unsigned& acc,
                                                        long long* gs, const int Ewlo, const int sh, const int nb,
                                                        const long long lnf, const int my_d0, const int my_d1,
                                                        const int my_wc, const long long my_T)
{
    int En = E + __shfl_sync(kFull, my_d0, 0);
    int bn = (En - Ewlo) >> sh;
    bool inr = (unsigned)bn < (unsigned)nb;
    long long gn = gs[inr ? bn : b];
#pragma unroll
    for (int j = 0; j < C; ++j) {
        const long long Tj = __shfl_sync(kFull, my_T, j);
        int E0 = 0, E1 = 0, b0 = 0, b1 = 0;
        bool i0 = false, i1 = false;
        long long g0 = 0, g1 = 0;
        if (j + 1 < C) {
            const int d0n = __shfl_sync(kFull, my_d0, j + 1);
            const int d1n = __shfl_sync(kFull, my_d1, j + 1);
            const int wcn = __shfl_sync(kFull, my_wc, j + 1);
            const int w0 = (acc & 1u) ? wcn : 0;
            const int w1 = (j == 0 || (acc & 1u)) ? wcn : 0;
            E0 = E + d0n + w0;
            E1 = En + d1n + w1;
            b0 = (E0 - Ewlo) >> sh;
            b1 = (E1 - Ewlo) >> sh;
            i0 = (unsigned)b0 < (unsigned)nb;
            i1 = (unsigned)b1 < (unsigned)nb;
            g0 = gs[i0 ? b0 : 0];
            g1 = gs[i1 ? b1 : 0];
        }
        const bool a = inr && (gn - gc < Tj);
        if (a) { E = En; b = bn; gc = gn; acc |= 1u << j; }
        gc += lnf;
        gs[b] = gc;
        if (j + 1 < C) {
            En = a ? E1 : E0;
            bn = a ? b1 : b0;
            inr = a ? i1 : i0;
            gn = a ? g1 : g0;
            if (bn == b) gn = gc;
        }
    }
}

// Ising sweeps.  One warp per walker; lattice and logDoS staged in shared memory
// for the whole launch.  Per-stage counts are not kept in the loop: within a
// launch every visit adds the same ln f, so the counts added to bin k are
// (g_end[k] - g_start[k]) / ln f exactly (ln f >= one 2^-36 unit always).
template <bool REPLAY, int VARIANT>
__global__ void __launch_bounds__(256) k_sweep_ising(const SweepParams p)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int li = blockIdx.x * (blockDim.x >> 5) + wib;
    if (li >= p.nslots || engine_failed_warp(p.P.counters)) return;
    const DevPtrs& P = p.P;
    const int s = p.slots[li];
    const InstDev I = P.inst[P.slot_inst[s]];
    const int w = P.slot_win[s];
    const WinDev W = P.win[w];
    const int L = I.L, N = I.N, C = I.chunk, nb = W.nb;
    unsigned char* base = smem + (size_t)wib * p.smem_per_warp;
    long long* gs = reinterpret_cast<long long*>(base);
    Stage* st = reinterpret_cast<Stage*>(gs + p.nbcap);
    int8_t* lat = reinterpret_cast<int8_t*>(st + 1);
    int* rsum = reinterpret_cast<int*>(lat + ((N + 15) & ~15));   // correlators: row and column sums
    int* csum = rsum + L;

    const int cfg = P.slot_cfg[s];
    int8_t* gl = P.spins + P.cfg_off[cfg];
    for (int i = lane; i < N; i += 32) lat[i] = gl[i];
    long long* gg = reinterpret_cast<long long*>(P.g + P.slot_tab[s]);
    for (int k = lane; k < nb; k += 32) gs[k] = gg[k];
    __syncwarp();
    const bool corr = P.obs != nullptr && P.corr;
    if (corr) {
        plane_sums(rsum, csum, L, lane, [&](int i) { return (int)lat[i]; });
        __syncwarp();
    }

    const int J = (int)I.J_u;
    const int sh = I.bin_shift;
    const int Ewlo = (int)W.elo_u;
    const long long lnf = P.win_lnf[w];
    const uint64_t sweeps0 = P.slot_sweeps[s];
    const uint32_t uid = (uint32_t)(s - I.first_slot);
    const uint64_t seed = I.seed;
    const bool obs_on = P.obs != nullptr;   // observables: the lane-0 resolver records each step's bin
    const bool all_lanes = (!REPLAY) && VARIANT == 3 && !obs_on && (C == 32 || C == 16 || C == 24 || C == 8 || C == 4);
    const double invN = 1.0 / (double)N;

    int E = (int)P.cfg_E[cfg];
    int M = P.cfg_M[3 * cfg];
    int b = (E - Ewlo) >> sh;
    if (b < 0 || b >= nb) {
        if (lane == 0) atomicOr(&P.counters[0], ERR_BOUNDS);
        return;
    }
    long long gc = gs[b];
    long long draws = 0, thr_off = 0, thr_n = 0;
    int err = 0;
    if (REPLAY) { draws = P.slot_draws[s]; thr_off = P.slot_thr_off[s]; thr_n = P.slot_thr_n[s]; }

    for (int sw = 0; sw < p.nsweeps; ++sw) {
        const uint64_t A0 = (sweeps0 + (uint64_t)sw) * (uint64_t)N;
        for (int c0 = 0; c0 < N; c0 += C) {
            // chunk = sites c0 .. c0+C-1 of one row (C divides L)
            const int y = c0 / L, x0 = c0 - y * L, x = x0 + lane;
            const int row = y * L;
            int si = 0, d0 = 0, d1 = 0, wc = 0;
            long long T = 0;
            if (lane < C) {
                si = lat[row + x];
                const Couplings cp{J, 0};
                const int i = row + x;
                d0 = (int)Ising2dModel::delta_energy(lat, nullptr, i, L, cp, 0);
                d1 = lane > 0 ? (int)Ising2dModel::left_flipped(lat, nullptr, i, L, cp, d0) : d0;
                wc = (C == L && lane == L - 1) ? (int)Ising2dModel::right_flipped(lat, nullptr, i, L, cp) : 0;
                if (!REPLAY) {
                    const uint32_t word = philox_word(seed, uid, A0 + (uint64_t)(c0 + lane), kStreamWL);
                    T = accept_threshold(neglog_u32(word));
                }
            }
            unsigned acc = 0;
            if (all_lanes) {
                switch (C) {
                case 32: resolve_chunk_all_lanes<32>(E, b, gc, acc, gs, Ewlo, sh, nb, lnf, d0, d1, wc, T); break;
                case 24: resolve_chunk_all_lanes<24>(E, b, gc, acc, gs, Ewlo, sh, nb, lnf, d0, d1, wc, T); break;
                case 16: resolve_chunk_all_lanes<16>(E, b, gc, acc, gs, Ewlo, sh, nb, lnf, d0, d1, wc, T); break;
                case 8: resolve_chunk_all_lanes<8>(E, b, gc, acc, gs, Ewlo, sh, nb, lnf, d0, d1, wc, T); break;
                default: resolve_chunk_all_lanes<4>(E, b, gc, acc, gs, Ewlo, sh, nb, lnf, d0, d1, wc, T); break;
                }
            } else {
                if (lane < C) { st->d0[lane] = d0; st->d1[lane] = d1; st->wc[lane] = wc; st->T[lane] = T; }
                __syncwarp();
                if (lane == 0) {
                    int En = E + st->d0[0];
                    int bn = (En - Ewlo) >> sh;
                    bool inr = (unsigned)bn < (unsigned)nb;
                    long long gn = gs[inr ? bn : b];
                    for (int j = 0; j < C; ++j) {
                        int E0 = 0, E1 = 0, b0 = 0, b1 = 0;
                        bool i0 = false, i1 = false;
                        long long g0 = 0, g1 = 0;
                        if (j + 1 < C) {
                            const int w0 = (acc & 1u) ? st->wc[j + 1] : 0;
                            const int w1 = (j == 0 || (acc & 1u)) ? st->wc[j + 1] : 0;
                            E0 = E + st->d0[j + 1] + w0;
                            E1 = En + st->d1[j + 1] + w1;
                            b0 = (E0 - Ewlo) >> sh;
                            b1 = (E1 - Ewlo) >> sh;
                            i0 = (unsigned)b0 < (unsigned)nb;
                            i1 = (unsigned)b1 < (unsigned)nb;
                            g0 = gs[i0 ? b0 : 0];
                            g1 = gs[i1 ? b1 : 0];
                        }
                        const long long d = gn - gc;
                        bool a;
                        if (!REPLAY) {
                            a = inr && (d < st->T[j]);
                        } else if (inr && d > 0) {
                            if (draws >= thr_n) { err = ERR_REPLAY_EXHAUSTED; a = false; }
                            else { a = d < P.thr[thr_off + draws]; ++draws; }
                        } else {
                            a = inr;
                        }
                        if (a) { E = En; b = bn; gc = gn; acc |= 1u << j; }
                        gc += lnf;
                        gs[b] = gc;
                        if (obs_on) st->seq[j] = b;
                        En = a ? E1 : E0;
                        bn = a ? b1 : b0;
                        inr = a ? i1 : i0;
                        gn = a ? g1 : g0;
                        if (bn == b) gn = gc;
                    }
                }
                // lane 0 holds the chain state; every lane needs it
                acc = __shfl_sync(kFull, acc, 0);
                E = __shfl_sync(kFull, E, 0);
                b = __shfl_sync(kFull, b, 0);
                gc = __shfl_sync(kFull, gc, 0);
                if (REPLAY) { draws = __shfl_sync(kFull, draws, 0); err = __shfl_sync(kFull, err, 0); }
            }
            const unsigned plus = __ballot_sync(kFull, lane < C && si > 0);
            if (obs_on) {
                __syncwarp();
                if (lane < C)
                {
                    const int32_t Mv[1] = {M + chunk_dm(acc, plus, lane)};
                    Ising2dModel::add_observables(P.obs + (size_t)(P.slot_tab[s] + st->seq[lane]) * P.obs_stride, Mv,
                                                  invN, P.corr);
                }
                if (corr) {
                    const int bin = lane < C ? st->seq[lane] : -1 - lane;
                    const unsigned grp = __match_any_sync(kFull, bin);
                    if (lane < C) {
                        // the bin's count before step `lane`: its visits after the chunk (the
                        // launch's start value plus the change of g over ln f) minus the chunk's
                        // visits to it from step `lane` on
                        const unsigned long long after =
                            P.visits[P.slot_tab[s] + bin] + (unsigned long long)((gs[bin] - gg[bin]) / lnf);
                        const unsigned long long seen = after - (unsigned long long)__popc(grp >> lane);
                        if (seen % kCountsPerTransform == 0) {
                            const double G = plane_corr(rsum, csum, P.qtab + I.qtab_off, L, y, chunk_dm(acc, plus, lane),
                                                        x0, lane, acc, [&](int k) { return (int)lat[row + x0 + k]; });
                            atomicAdd(P.obs + (size_t)(P.slot_tab[s] + bin) * P.obs_stride + 3, invN * invN * G);
                        }
                    }
                    __syncwarp();
                    // the chunk's flips into the row and column sums
                    if (lane < C && ((acc >> lane) & 1u)) csum[x] -= 2 * si;
                    if (lane == 0) rsum[y] += -2 * ((int)__popc(acc & plus) - (int)__popc(acc & ~plus));
                }
            }
            if (lane < C && ((acc >> lane) & 1u)) lat[row + x] = (int8_t)(-si);
            M += -2 * ((int)__popc(acc & plus) - (int)__popc(acc & ~plus));
            __syncwarp();
        }
    }
    // write back: lattice, logDoS, counts and visits derived from the logDoS change
    for (int i = lane; i < N; i += 32) gl[i] = lat[i];
    uint32_t* gH = P.H + P.slot_tab[s];
    uint64_t* gv = P.visits + P.slot_tab[s];
    for (int k = lane; k < nb; k += 32) {
        const long long gnew = gs[k];
        const long long dv = (gnew - gg[k]) / lnf;
        const int e = commit_visits(gH, gv, k, dv, gnew);
        if (e) atomicOr(&P.counters[0], e);
        gg[k] = gnew;
    }
    if (lane == 0) {
        P.cfg_E[cfg] = E;
        P.cfg_M[3 * cfg] = M;
        P.slot_sweeps[s] = sweeps0 + (uint64_t)p.nsweeps;
        if (REPLAY) P.slot_draws[s] = draws;
        if (err) atomicOr(&P.counters[0], err);
    }
}

// ---------------------------------------------------------------------------
// Bin-tracking Ising sweeps (used when every energy change is a whole number of
// bins: 4|J| divisible by the bin width, as for J = 1 and width 4).
//
// The chain of accept decisions of one walker is serial, but a few decisions
// ahead there are few outcomes: G walkers share a warp, P = 32 / G lanes each,
// and a walker's lanes are the nodes of the binary tree of its next D = log2(P)
// decisions (lane 1 the first decision, lanes 2k and 2k + 1 the decision after
// lane k's rejection / acceptance; lane 0 idles).  A block of D sites is then:
//   * every node forms its own position relative to the block's start (the sum
//     of the bin changes its ancestors accepted), its proposal, and how often
//     the path to it visits either bin within the block -- all independent of
//     where the block starts, so this is done while the block before it is
//     being decided;
//   * once the start is known, every node loads g at its two bins (two shared
//     loads for D decisions instead of D dependent ones), decides, and one vote
//     hands all decisions to all lanes;
//   * a node is on the path if its ancestors decided its way (one masked
//     compare); the D nodes on the path commit g + visits x ln f, in order of
//     their sites, and the last of them publishes the new position.
// Energy changes are multiples of 4|J|: with a = the number of neighbours that
// agree, a flip moves the walker by (a - 2) x q bins (q = 4 J / width), and a
// left neighbour flipped just before changes a by one.  Positions inside a block
// are sums of at most five such steps and live in the four bytes of a register:
// a byte-wise prefix sum is one multiplication by 0x01010101.
//
// The lattice is one bit per spin (1: spin -1), a row being nch chunks of at most
// 32 sites, one word each; chunks are cut into blocks of D sites (the last one
// shorter).  The agreement counts of a chunk come from its words by bit-sliced
// addition and are handed to the nodes through shared memory (`slots`).
//
// The table carries kGuard sentinel bins on each side holding INT64_MAX: a
// proposal outside the window fails the compare by itself, and nodes below an
// out-of-window proposal (never on the path) still read inside the table.
// ---------------------------------------------------------------------------
constexpr int kGuard = 20;                                // 2 x 5 decisions x |q| <= 2 bins
constexpr long long kGuardValue = 0x7FFFFFFFFFFFFFFFLL;   // never below g + threshold

__device__ __forceinline__ long long lds64(const char* base, int off)
{
    return *reinterpret_cast<const long long*>(base + off);
}
__device__ __forceinline__ void sts64(char* base, int off, long long v) { *reinterpret_cast<long long*>(base + off) = v; }

// acc + n f for an int64 f = f_hi 2^32 + f_lo (f_lo signed): two multiply-adds
__device__ __forceinline__ long long mad_units(long long acc, int n, int f_lo, int f_hi)
{
    long long r;
    asm("{\n\t.reg .b32 lo, hi;\n\tmad.wide.s32 %0, %1, %2, %4;\n\tmov.b64 {lo, hi}, %0;\n\tmad.lo.s32 hi, %1, %3, hi;\n\t"
        "mov.b64 %0, {lo, hi};\n\t}"
        : "=&l"(r) : "r"(n), "r"(f_lo), "r"(f_hi), "l"(acc));
    return r;
}

// a b + c on the multiply-add pipe, whatever a and b are: the integer ALU is the busier one
__device__ __forceinline__ unsigned mad32(unsigned a, unsigned b, unsigned c)
{
    unsigned r;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}

// adds 1 (v) to the 32-bit word at shared address `addr` (+ OFFSET)
template <int OFFSET = 0>
__device__ __forceinline__ void red_shared_inc(unsigned addr)
{
    asm volatile("red.shared.add.u32 [%0 + %1], 1;" :: "r"(addr), "n"(OFFSET) : "memory");
}
__device__ __forceinline__ void red_shared_add(unsigned addr, int v)
{
    asm volatile("red.shared.add.s32 [%0], %1;" :: "r"(addr), "r"(v) : "memory");
}

// chunk layout of a row of L sites: `n` words, the first `rem` of `base` + 1 sites, the others of `base`
struct RowChunks {
    int n, base, rem;
    __host__ __device__ explicit RowChunks(int L) : n((L + 31) / 32), base(L / n), rem(L % n) {}
    __host__ __device__ int len(int c) const { return base + (c < rem ? 1 : 0); }
    __host__ __device__ int start(int c) const { return c * base + (c < rem ? c : rem); }
    __host__ __device__ int of(int x) const { return x < rem * (base + 1) ? x / (base + 1) : rem + (x - rem * (base + 1)) / base; }
};

template <int G>
struct BinsTree {
    static constexpr int kLanes = 32 / G;
    static constexpr int kDepth = G == 1 ? 5 : G == 2 ? 4 : 3;
    static constexpr int kBlocks = (32 + kDepth - 1) / kDepth;      // blocks of the longest chunk
    static constexpr int kSlot = kDepth == 5 ? 16 : 8;              // bytes per block: agreement counts, then left terms
    static constexpr int kRing = G == 4 ? 128 : 256;                // thresholds kept per walker
    static_assert(kLanes == 1 << kDepth, "one lane per node");
};

// Ising moments of a bin as whole numbers, in words that reductions add to without looking: |M|,
// M^2 in two parts, M^4 in four, `bits` binary digits each (the last ones what is left).  `visits`
// visits cannot overflow a word; after as many the words are added to the observable sums in
// global memory and start at zero again.
constexpr int kObsWords = 7;
struct MomentParts {
    int bits;
    unsigned visits;
    __host__ __device__ explicit MomentParts(int N) : bits(N <= 8192 ? 18 : 16), visits(1u << (32 - bits)) {}
};

// shared memory of one walker (of G a warp): table with guards, lattice words, thresholds, two chunks' slots;
// with observables the bins of a chunk's steps and (acc) the
// moments' integer sums, with correlators row and column sums and counts
template <int G>
__host__ __device__ inline int bins_smem(int nbcap, int L, bool obs, bool corr, bool cnt, bool acc)
{
    const RowChunks rc(L);
    return (nbcap + 2 * kGuard) * (cnt ? 16 : 8) + ((rc.n * L * 4 + 15) & ~15) + BinsTree<G>::kRing * 8 +
           2 * BinsTree<G>::kBlocks * BinsTree<G>::kSlot + 16 + (obs ? 32 * 4 : 0) + (corr ? 8 * L + 4 * nbcap : 0) + (acc ? 4 * kObsWords * nbcap : 0);
}

// Bound: a warp alone on its scheduler by the latency of a block (about 265 cycles per five decisions:
// shared loads, vote, warp maximum and the integer instructions between them; 23 instructions per
// flip), several by instruction issue (16 per flip with two walkers each, the ALU 77 % busy on the
// busiest scheduler).  Measured against one decision after another: L = 64, 512 walkers 70 -> 58
// cycles per flip, 3072 walkers 4.62 -> 4.70e10 flips/s; L = 20, 32 walkers, whose rows had no chunk of
// eight, 376 -> 71.
//
__host__ inline int bins_smem(int G, int nbcap, int L, bool obs, bool corr, bool cnt, bool acc)
{
    const int raw = G == 1 ? bins_smem<1>(nbcap, L, obs, corr, cnt, acc) : G == 2 ? bins_smem<2>(nbcap, L, obs, corr, cnt, acc)
                                                                               : bins_smem<4>(nbcap, L, obs, corr, cnt, acc);
    return ((raw + 127) & ~127) + 16;                          // + 16 skews the walkers' banks
}

// The sweeps of one warp's G walkers (launch position warp_index; its shared memory starts at
// warp_base, one region of p.smem_per_warp bytes per walker).
template <int G, bool OBS, bool CNT>
__device__ __forceinline__ void sweep_bins_warp(const SweepParams& p, const int warp_index, unsigned char* warp_base)
{
    using T = BinsTree<G>;
    constexpr int RS = CNT ? 16 : 8, RW = RS / 8;            // table record: g, with CNT followed by the launch's visits
    constexpr int P = T::kLanes, D = T::kDepth, SPL = 32 / P, RING = T::kRing;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int grp = lane / P, q = lane - grp * P, gbase = grp * P;
    const int li = warp_index * G + grp;
    const bool valid = li < p.nslots;
    if (__ballot_sync(kFull, valid) == 0 || engine_failed_warp(p.P.counters)) return;   // no walkers, or stopped
    const DevPtrs& P_ = p.P;
    const int s = p.slots[valid ? li : 0];                     // idle groups shadow a walker, never write
    const InstDev I = P_.inst[P_.slot_inst[s]];
    const int w = P_.slot_win[s];
    const WinDev W = P_.win[w];
    const int L = I.L, N = I.N, nb = W.nb;
    const RowChunks rc(L);
    unsigned char* base = warp_base + (size_t)grp * p.smem_per_warp;
    long long* gs = reinterpret_cast<long long*>(base) + RW * kGuard;            // records -kGuard .. nb+kGuard-1
    uint32_t* lat = reinterpret_cast<uint32_t*>(base + (p.nbcap + 2 * kGuard) * RS);   // [L][rc.n] words
    long long* Tb = reinterpret_cast<long long*>(reinterpret_cast<unsigned char*>(lat) + ((rc.n * L * 4 + 15) & ~15));
    unsigned char* slots = reinterpret_cast<unsigned char*>(Tb + RING);          // 2 chunks of T::kBlocks slots
    int* seqb = reinterpret_cast<int*>(slots + 2 * T::kBlocks * T::kSlot) + 4;   // a chunk's bins (observables)
    int* rsum = seqb + (OBS ? 32 : 0);                                           // correlators: row sums,
    int* csum = rsum + L;                                                        // column sums,
    int* bcnt = csum + L;                                                        // visits before a bin's next transform
    const bool corr = OBS && P_.corr, moments = OBS && p.moments;
    unsigned* mom = reinterpret_cast<unsigned*>(corr ? bcnt + p.nbcap : rsum);   // moment sums (observables)
    // table positions are byte offsets from the start of shared memory, so that the
    // accesses need no address arithmetic
    char* const sm = reinterpret_cast<char*>(smem);
    const int gsoff = (int)(reinterpret_cast<char*>(gs) - sm);
    const unsigned smbase = (unsigned)__cvta_generic_to_shared(sm);
    const int sink = (int)(reinterpret_cast<char*>(seqb - 4) - sm);

    const int cfg = P_.slot_cfg[s];
    int8_t* gl = P_.spins + P_.cfg_off[cfg];
    long long* gg = reinterpret_cast<long long*>(P_.g + P_.slot_tab[s]);
    for (int k = q - kGuard; k < nb + kGuard; k += P) {
        gs[RW * k] = k >= 0 && k < nb ? gg[k] : kGuardValue;
        if (CNT) gs[RW * k + 1] = 0;
    }
    // every slot starts as "no change" (count 2, left term 1), so that a short block's missing
    // sites keep positions inside the table; bytes past a slot's D sites stay zero
    for (int k = q; k < 2 * T::kBlocks * T::kSlot; k += P) {
        const int half = k % T::kSlot / (T::kSlot / 2), j = k % (T::kSlot / 2);
        slots[k] = j < D ? (unsigned char)(half ? 1 : 2) : (unsigned char)0;
    }
    int minus = 0;                                             // spins -1 seen by this walker (all its lanes agree)
    for (int c = 0, i = 0; c < rc.n * L; ++c) {
        const int len = rc.len(c % rc.n);
        uint32_t bits = 0;
#pragma unroll
        for (int k = 0; k < SPL; ++k) {
            const int jj = q + k * P;
            const unsigned bal = __ballot_sync(kFull, jj < len && gl[i + jj] < 0);
            bits |= (P == 32 ? bal : ((bal >> gbase) & (0xFFFFFFFFu >> (32 - P)))) << (k * P % 32);
        }
        if (q == 0) lat[c] = bits;
        minus += __popc(bits);
        i += len;
    }
    __syncwarp();
    auto spin = [&](int i) {
        const int y = i / L, x = i - y * L, c = rc.of(x);
        return (lat[y * rc.n + c] >> (x - rc.start(c))) & 1u ? -1 : 1;
    };
    const double invN = 1.0 / (double)N;
    double* ob = OBS ? P_.obs + (size_t)P_.slot_tab[s] * P_.obs_stride : nullptr;
    const MomentParts parts(N);
    unsigned booked = 0;                                       // visits in the moments' words
    const int reach2 = (int)(((unsigned long long)N * N) >> parts.bits) != 0 ? 2 : 1;      // parts of M^2, M^4
    int reach4 = 1;
    for (unsigned long long x = (unsigned long long)N * N * N * N; (x >>= parts.bits) != 0;) ++reach4;
    if (moments)
        for (int k = q; k < nb * kObsWords; k += P) mom[k] = 0;
    // the words into the sums of m = |M| / N
    auto book_moments = [&] {
        const double in2 = invN * invN, unit = (double)(1u << parts.bits);
        __syncwarp();
        if (valid)
            for (int k = q; k < nb; k += P) {
                unsigned* t = mom + kObsWords * k;
                double* o = ob + (size_t)k * P_.obs_stride;
                if ((t[0] | t[1] | t[2]) != 0) {               // (M = 0 adds nothing)
                    o[0] += invN * (double)t[0];
                    o[1] += in2 * (unit * (double)t[2] + (double)t[1]);
                    o[2] += in2 * in2 * (((unit * (double)t[6] + (double)t[5]) * unit + (double)t[4]) * unit + (double)t[3]);
                    for (int j = 0; j < kObsWords; ++j) t[j] = 0;
                }
            }
        __syncwarp();
    };
    if (corr) {
        plane_sums(rsum, csum, L, q, spin, P);
        const uint64_t* gv0 = P_.visits + P_.slot_tab[s];
        for (int k = q; k < nb; k += P) {
            const int r = mod_transform(gv0[k]);
            bcnt[k] = r == 0 ? 0 : (int)kCountsPerTransform - r;
        }
        __syncwarp();
    }

    const int sh = I.bin_shift;
    const int q8 = (int)((4 * I.J_u) >> sh) * RS;              // table bytes per agreeing neighbour
    const int Ewlo = (int)W.elo_u;
    const long long lnf = P_.win_lnf[w];
    const int lnf_lo = (int)(uint32_t)lnf;                     // ln f = lnf_hi 2^32 + lnf_lo, lnf_lo signed
    const int lnf_hi = (int)((lnf - (long long)lnf_lo) >> 32);
    const uint64_t sweeps0 = P_.slot_sweeps[s];
    const uint32_t uid = (uint32_t)(s - I.first_slot);
    const uint32_t k0 = (uint32_t)I.seed ^ uid, k1 = (uint32_t)(I.seed >> 32);

    const int E0 = (int)P_.cfg_E[cfg];
    const int b0 = (E0 - Ewlo) >> sh;
    const bool bad = ((E0 - Ewlo) & ((1 << sh) - 1)) != 0 || b0 < 0 || b0 >= nb;
    if (__ballot_sync(kFull, valid && bad)) {
        if (lane == 0) atomicOr(&P_.counters[0], ERR_BOUNDS);
        return;
    }
    int M = N - 2 * minus;

    // this lane's node: level (decisions before it), the ancestors' decisions that lead to it
    const int lvl = q == 0 ? 0 : 31 - __clz(q);
    const int lvla = q == 0 ? 32 : lvl;                        // the idle lane is beyond every block
    unsigned want = 0, anc = 0;                                // ancestors' vote bits: needed value, mask
    unsigned mA = 0, mB = 0, K = 0, L80 = 0;                   // byte masks of accepted / twice accepted steps, biases
    bool first = false, last = false;                          // first decision accepted; the one before this node's
    {
        int bias = 0;
        bool prev = false;
        for (int i = 0; i < lvl; ++i) {
            const int node = q >> (lvl - i);
            const bool a = (q >> (lvl - 1 - i)) & 1;
            anc |= 1u << node;
            if (a) want |= 1u << node;
            if (a) { mA |= 0xFFu << (8 * i); bias += 2; }
            if (a && prev) { mB |= 0xFFu << (8 * i); bias += 1; }
            K |= (unsigned)(16 - bias) << (8 * i);
            L80 |= 0x80u << (8 * i);
            if (i == 0) first = a;
            prev = a;
        }
        last = prev;
        if (q == 0) { anc = 1u; want = 1u; }                   // its vote is always 0: never on the path
    }
    const unsigned selC = lvl == 0 ? 0x5554u : 0x5550u | (unsigned)(lvl - 1);
    const unsigned selE = 0x7770u | (unsigned)lvl, selX = last ? 0x7770u | (unsigned)lvl : 0x7777u;
    const int pbias = 2 + (last ? 1 : 0);
    const unsigned KP = 0u - (unsigned)pbias * 0x01010101u;
    const int kC = -16 * q8, kP = -(16 + pbias) * q8;
    const int shiftC = first ? -1 : 0, shiftP = (first || lvl == 0) ? -1 : 0;    // left neighbour of the block's first site
    const bool leaf = lvl == D - 1 && q != 0;
    // what a leaf publishes with its position: the decisions of its path in bits 20.. (its own: bit 20 + D - 1)
    int pathc = 0;
    for (int i = 0; i < lvl; ++i)
        if ((q >> (lvl - 1 - i)) & 1) pathc |= 1 << (20 + i);
    const unsigned pathP = (unsigned)pathc + (0x80000000u | 1u << (20 + D - 1));
    // Sums on the multiply-add pipe and fewer of them where one walker has the warp: its instructions
    // wait for the integer ALU (L = 64, 59.4 -> 58.1 cycles per flip).  Several walkers' warps take turns
    // and do better with the plain sums (135 against 138), as do observables (126.1, 126.8).
    constexpr bool kMad = G == 1 && !OBS;
    unsigned one = 1;                                          // (not to be folded)
    if (kMad) asm volatile("" : "+r"(one));
    auto mad = [&](unsigned a, unsigned b, unsigned c) { return kMad ? mad32(a, b, c) : a * b + c; };
    auto sum = [&](unsigned a, unsigned b) { return kMad ? mad32(a, one, b) : a + b; };
    const unsigned tboff = (unsigned)(reinterpret_cast<char*>(Tb) - sm);

    // thresholds of P Philox blocks (four attempts each) from block `blk` on into the ring
    auto draw = [&](uint64_t blk) {
        const uint64_t a = blk + (uint64_t)q;
        const Philox4 r = philox4x32_10(Philox4{(uint32_t)a, (uint32_t)(a >> 32), kStreamWL, 0u}, k0, k1);
        longlong2* dst = reinterpret_cast<longlong2*>(Tb + (((uint32_t)a * 4u) & (RING - 1)));
        longlong2 t01, t23;
        t01.x = word_threshold(r.x);
        t01.y = word_threshold(r.y);
        t23.x = word_threshold(r.z);
        t23.y = word_threshold(r.w);
        dst[0] = t01;
        dst[1] = t23;
    };

    // Agreement counts and left terms of the chunk (y, c), into slots `buf`.  The words are read as
    // they stand, before the flips of the chunk being processed (word index cprev) except for its
    // decisions `acc` known by now -- the left neighbour of the chunk's first site excepted, whose
    // flip the nodes add themselves.
    constexpr int kBuf = T::kBlocks * T::kSlot;
    int myslot[SPL];
#pragma unroll
    for (int k = 0; k < SPL; ++k) {
        const int jj = q + k * P;
        myslot[k] = (jj / D) * T::kSlot + jj % D;
    }
    struct Planes {
        unsigned sw, su, al, t1, c1;                           // the chunk's word; up disagreements; partial sums
    };
    auto write_slots = [&](const Planes& f, unsigned up_flips, int c, int len, int from, int buf) {
        const unsigned au = ~(f.su ^ up_flips);
        const unsigned t0 = au ^ f.al, c0 = au & f.al;
        const unsigned a0 = t0 ^ f.t1, a1 = c0 ^ f.c1 ^ (t0 & f.t1), a2 = c0 & f.c1;
        unsigned char* dst = slots + buf * kBuf;
#pragma unroll
        for (int k = 0; k < SPL; ++k) {
            const int jj = q + k * P;
            const unsigned e = ((a0 >> jj) & 1u) + 2u * ((a1 >> jj) & 1u) + 4u * ((a2 >> jj) & 1u);
            const unsigned x = jj == 0 && c == 0 ? 1u : 2u - 2u * ((f.al >> jj) & 1u);
            if (jj < len && jj >= from) {
                dst[myslot[k]] = (unsigned char)e;
                dst[myslot[k] + T::kSlot / 2] = (unsigned char)x;
            }
        }
    };
    auto publish = [&](int y, int c, int buf, int cprev, unsigned acc) {
        const int up = y == 0 ? L - 1 : y - 1, dn = y == L - 1 ? 0 : y + 1;
        const int cl = c == 0 ? rc.n - 1 : c - 1, cr = c == rc.n - 1 ? 0 : c + 1;
        const int len = rc.len(c), row = y * rc.n;
        const unsigned sw = lat[row + c], uw = lat[up * rc.n + c], dw = lat[dn * rc.n + c], lw = lat[row + cl];
        const unsigned rw = lat[row + cr] ^ (row + cr == cprev ? acc : 0u);
        const unsigned lb = (sw << 1) | ((lw >> (rc.len(cl) - 1)) & 1u);
        const unsigned rb = (sw >> 1) | ((rw & 1u) << (len - 1));
        const unsigned ar = ~(sw ^ rb), ad = ~(sw ^ dw);
        Planes f;
        f.sw = sw;
        f.su = sw ^ uw;
        f.al = ~(sw ^ lb);
        f.t1 = ar ^ ad;
        f.c1 = ar & ad;
        write_slots(f, up * rc.n + c == cprev ? acc : 0u, c, len, 0, buf);
        return f;
    };

    // A node's part of a block that does not depend on where the block starts: the slots and the
    // threshold it reads, then its positions, then the visits of its path to either bin.
    struct Slot {
        unsigned e0, e1, x0, x1;
        long long t;
    };
    struct Node {
        int rC, rP, nC, nP, x0;
        long long t;
    };
    auto fetch = [&](const unsigned char* slot, uint32_t attempt) {
        Slot f;
        if (D == 5) {
            const uint4 v = *reinterpret_cast<const uint4*>(slot);
            f.e0 = v.x; f.e1 = v.y; f.x0 = v.z; f.x1 = v.w;
        } else {
            const uint2 v = *reinterpret_cast<const uint2*>(slot);
            f.e0 = v.x; f.e1 = 0u; f.x0 = v.y; f.x1 = 0u;
        }
        if (kMad) f.t = lds64(sm, (int)sum(mad(attempt, 8u, (unsigned)(8 * lvl)) & (8 * RING - 1), tboff));
        else f.t = Tb[(attempt + (uint32_t)lvl) & (RING - 1)];
        return f;
    };
    auto node = [&](const Slot& f) {
        const unsigned S = kMad ? mad32(f.e0 & mA, 0x01010101u, mad32(f.x0 & mB, 0x01010101u, K))   // positions after each step, + 16
                                : ((f.e0 & mA) + (f.x0 & mB)) * 0x01010101u + K;
        const unsigned cb = __byte_perm(S, 0x10u, selC);
        const unsigned pb = cb + __byte_perm(f.e0, f.e1, selE) + __byte_perm(f.x0, f.x1, selX);
        Node n;
        n.rC = (int)cb * q8 + kC;
        n.rP = (int)pb * q8 + kP;
        n.x0 = ((int)(f.x0 & 0xFFu) - 1) * q8;
        n.nC = __popc(~sum(S ^ (cb * 0x01010101u), 0x7F7F7F7Fu) & L80);         // steps of the path that ended here
        n.nP = __popc(~sum(S ^ (pb * 0x01010101u + KP), 0x7F7F7F7Fu) & L80);
        n.t = f.t;
        return n;
    };

    // what the last block left: the position (byte offset, bits 0-19), its decisions (from bit 20 on),
    // and in the sign whether its last site flipped
    unsigned state = (unsigned)(gsoff + b0 * RS);
    unsigned acc = 0;                                          // the current chunk's decisions so far
    // one block of nlev sites (at the chunk's site j0): its nodes `n`; the next block's slots are
    // read (ahead()) between the loads and the decision, its node work is done behind the vote
    auto block = [&](const Node n, const int nlev, int j0, auto ahead) {
        const int root = (int)(state & 0xFFFFFu);
        const int shift = ((int)state >> 31) & n.x0;
        const int aC = root + n.rC + (shift & shiftC), aP = root + n.rP + (shift & shiftP);
        long long gC, gP;
        int dn = n.nC - n.nP;
        if (CNT) {
            const longlong2 c = *reinterpret_cast<const longlong2*>(sm + aC), d = *reinterpret_cast<const longlong2*>(sm + aP);
            gC = c.x; gP = d.x;
            dn += (int)c.y - (int)d.y;
        } else {
            gC = lds64(sm, aC);
            gP = lds64(sm, aP);
        }
        const Slot f = ahead();
        const bool live = lvla < nlev;
        const bool a = gP < mad_units(gC + n.t, dn, lnf_lo, lnf_hi) && live;
        const unsigned B = __ballot_sync(kFull, a) >> gbase;
        const bool on = ((B ^ want) & anc) == 0;
        const int fin = a ? aP : aC;
        constexpr unsigned kFlip = 0x80000000u | 1u << (20 + D - 1);       // the node's own decision
        unsigned v = kMad ? (unsigned)fin + (a ? pathP : (unsigned)pathc)
                          : a ? (unsigned)(aP + pathc) + kFlip : (unsigned)(aC + pathc);
        if (G <= 2) {
            v = on && leaf ? v : 0u;
            if (G == 1) v = __reduce_max_sync(kFull, v);
            else {
                const unsigned v0 = __reduce_max_sync(kFull, grp == 0 ? v : 0u), v1 = __reduce_max_sync(kFull, grp == 0 ? 0u : v);
                v = grp == 0 ? v0 : v1;
            }
        } else {
            const unsigned O = __ballot_sync(kFull, on && leaf) & ((0xFFFFFFFFu >> (32 - P)) << gbase);
            v = __shfl_sync(kFull, v, 31 - __clz(O));
        }
        if (OBS && on && live) seqb[j0 + lvl] = fin;
        if (CNT) {
            // lanes off the path count in a word nobody reads (a predicated reduction costs a branch)
            if (kMad) red_shared_inc<8>(smbase + (unsigned)(on && live ? fin : sink - 8));
            else red_shared_inc(smbase + (unsigned)(on && live ? fin + 8 : sink));
        } else {
            const int vis = (a ? n.nP : n.nC) + 1;
            const long long gn = mad_units(a ? gP : gC, vis, lnf_lo, lnf_hi);
            const int sl = on && live ? lvl : -1;
#pragma unroll
            for (int i = 0; i < D; ++i) {
                if (sl == i) sts64(sm, fin, gn);
                __syncwarp();                                  // a later visit's value replaces an earlier one's
            }
        }
        const Node next = node(f);
        __syncwarp();
        const unsigned path = (v >> 20) & ((1u << D) - 1u);
        acc |= path << j0;
        state = nlev == D ? v : (v & 0x7FFFFFFFu) | (path << (32 - nlev) & 0x80000000u);
        return next;
    };

    const uint64_t A0 = sweeps0 * (uint64_t)N;                 // first attempt
    uint64_t drawn = A0 >> 2;                                  // first Philox block not drawn
    int ready = -(int)(A0 & 3);                                // thresholds in the ring from the current chunk on
    for (; ready < 64; ready += 4 * P, drawn += P) draw(drawn);
    Planes next_planes = publish(0, 0, 0, -1, 0u);
    unsigned up_flips = 0;                                     // the flips of the chunk above (whole-row chunks)
    __syncwarp();
    const bool wraps = rc.n == 1;                              // a row is one chunk: its last site sees its first
    int y = 0, ci = 0, buf = 0;
    uint32_t at = (uint32_t)A0;                                // the current chunk's first attempt (ring index)
    uint64_t left = (uint64_t)p.nsweeps * (uint64_t)N;
    // the change of a whole-row chunk's last count when the row's first site has flipped
    auto wrap_term = [&](int yy) {
        const unsigned sw = lat[yy * rc.n];
        return (((sw >> (L - 1)) ^ sw) & 1u) ? 1 : -1;         // first and last disagree: a flip makes them agree
    };
    const int blocks_min = (rc.base + D - 1) / D;
    // rows of one block: the last site's wrap term depends on the block's own first decision
    auto node_row = [&](const unsigned char* slot, uint32_t attempt, int len, int yy) {
        unsigned w0 = 0, w1 = 0;
        if (first) (len < 5 ? w0 : w1) = (unsigned)wrap_term(yy) << (len < 5 ? 8 * (len - 1) : 0);
        Slot f = fetch(slot, attempt);
        f.e0 += w0;
        f.e1 += w1;
        return node(f);
    };
    Node n = blocks_min == 1 ? node_row(slots, at, L, 0) : node(fetch(slots, at));
    while (left > 0) {
        const int len = rc.len(ci), nblk = (len + D - 1) / D;
        const int cw = y * rc.n + ci;
        int yn = y, cn = ci + 1;
        if (cn == rc.n) { cn = 0; yn = y + 1 == L ? 0 : y + 1; }
        if (ready < 64) {
            draw(drawn);
            drawn += P;
            ready += 4 * P;
            __syncwarp();
        }
        acc = 0;
        const unsigned char* cur = slots + buf * kBuf;
        const unsigned char* nxt = slots + (buf ^ 1) * kBuf;
        const Planes planes = next_planes;
        const unsigned old = planes.sw;
        auto none = [&] { return Slot{}; };
        // the change of the last site's count where the row's first site has flipped (its right neighbour)
        auto wrap_byte = [&] {
            const unsigned t = ((old >> (len - 1)) ^ old) & 1u ? 1u : 0xFFFFFFFFu;
            return wraps && (acc & 1u) ? t << (8 * (((len - 1) % D) & 3)) : 0u;
        };
        const bool fifth = D == 5 && (len - 1) % D == 4;
        if (blocks_min >= 3) {
            // three blocks or more: every block's node work runs while the block before it decides.
            // The next chunk's slots are published during the last block but one; where the chunk
            // above it is this one, the counts of its last two blocks are written again during its
            // first block, with this chunk's last decisions.
            uint32_t k = at + D;
            const unsigned char* slot = cur + T::kSlot;
            const int late = (nblk - 2) * D;
            n = block(n, D, 0, [&] {
                if (nblk == 3) {
                    if (wraps) write_slots(planes, up_flips, ci, len, late, buf);
                    __syncwarp();
                    return fetch(slot, k);
                }
                const Slot m = fetch(slot, k);
                if (wraps) write_slots(planes, up_flips, ci, len, late, buf);
                return m;
            });
            k += D;
            slot += T::kSlot;
            int j0 = D;
#pragma unroll 2
            for (; j0 < late; j0 += D, k += D, slot += T::kSlot)
                n = block(n, D, j0, [&] { return fetch(slot, k); });
            n = block(n, D, j0, [&] {
                const unsigned wr = wrap_byte();
                Slot m = fetch(slot, k);
                m.e0 += fifth ? 0u : wr;
                m.e1 += fifth ? wr : 0u;
                next_planes = publish(yn, cn, buf ^ 1, cw, acc);
                return m;
            });
            j0 += D;
            n = block(n, len - j0, j0, [&] { return fetch(nxt, at + (uint32_t)len); });
        } else if (nblk == 2) {
            n = block(n, D, 0, none);
            const unsigned wr = wrap_byte();
            Slot f = fetch(cur + T::kSlot, at + D);
            f.e0 += fifth ? 0u : wr;
            f.e1 += fifth ? wr : 0u;
            n = node(f);
            publish(yn, cn, buf ^ 1, cw, acc);
            __syncwarp();
            n = block(n, len - D, D, [&] { return fetch(nxt, at + (uint32_t)len); });
        } else {
            n = block(n, len, 0, none);
        }
        // the chunk's flips
        if (q == 0) lat[cw] = old ^ acc;
        __syncwarp();
        up_flips = acc;
        if (blocks_min < 3) {
            // short rows: the next row's counts with all of this one's decisions
            next_planes = publish(yn, cn, buf ^ 1, -1, 0u);
            __syncwarp();
            if (nblk == 1) n = node_row(nxt, at + (uint32_t)len, L, yn);
        }
        if (OBS) {
            // the chunk's moments and correlators, one step per lane, by reductions that return nothing and
            // with no look at the chunk's own repeats of a bin unless a transform may be due (16 steps
            // of L = 16: 1370 -> 650 cycles beside the 1500 of their decisions)
            const unsigned plus = ~old & (0xFFFFFFFFu >> (32 - len));
            const int x0 = rc.start(ci);
            if (moments && (booked += (unsigned)len) > parts.visits) {
                book_moments();
                booked = (unsigned)len;
            }
#pragma unroll
            for (int i = 0; i < SPL; ++i) {
                const int jj = q + i * P;
                const bool mine = valid && jj < len;
                const int off = mine ? seqb[jj] : -1 - lane;
                const int b = mine ? (off - gsoff) / RS : 0;
                const int Mj = M + chunk_dm(acc, plus, jj);
                // visits of the bin before its next transform (correlators), ahead of the chunk
                const int before = corr && mine ? bcnt[b] : 32;
                if (moments) {
                    const unsigned m = (unsigned)abs(Mj), m2 = m * m, low = (1u << parts.bits) - 1u;
                    const unsigned long long m4 = (unsigned long long)m2 * m2;
                    const unsigned t = mine ? (unsigned)__cvta_generic_to_shared(mom + kObsWords * b) : 0u;
                    auto add = [&](int k, unsigned v) { red_shared_add(mine ? t + 4 * k : smbase + (unsigned)sink, (int)v); };
                    add(0, m);
                    add(1, m2 & low);
                    if (reach2 > 1) add(2, m2 >> parts.bits);
                    add(3, (unsigned)m4 & low);
                    if (reach4 > 1) add(4, (unsigned)(m4 >> parts.bits) & low);
                    if (reach4 > 2) add(5, (unsigned)(m4 >> (2 * parts.bits)) & low);
                    if (reach4 > 3) add(6, (unsigned)(m4 >> (3 * parts.bits)));
                } else if (mine) {
                    const int32_t Mv[1] = {Mj};
                    Ising2dModel::add_observables(ob + (size_t)b * P_.obs_stride, Mv, invN, P_.corr);
                }
                if (corr) {
                    // G(q_min) at the steps whose bin count before the visit is a multiple of 1000
                    bool due = false;
                    if (__any_sync(kFull, before < len)) {
                        const unsigned same = __match_any_sync(kFull, off), earlier = same & ((1u << lane) - 1u);
                        due = mine && before == __popc(earlier);
                        bool todo = due;
                        for (unsigned all; (all = __ballot_sync(kFull, todo)) != 0;) {
                            // one step of each walker of the warp
                            const unsigned own = (all >> gbase) & (0xFFFFFFFFu >> (32 - P));
                            const int e = own ? __ffs((int)own) - 1 : 0, je = e + i * P;
                            const unsigned le = je >= 31 ? 0xFFFFFFFFu : ((2u << je) - 1u);
                            const double Gq = plane_power<P, 1>(rsum, csum, P_.qfix + I.qtab_off, L, y, x0, acc & le, plus, q);
                            if (own != 0 && q == e) {
                                red_global_add(ob + (size_t)b * P_.obs_stride + 3, 0.5 * invN * invN * Gq);
                                todo = false;
                            }
                        }
                    }
                    __syncwarp();                              // every lane has read its bin's count
                    red_shared_add(mine ? (unsigned)__cvta_generic_to_shared(bcnt + b) : smbase + (unsigned)sink,
                                   due ? (int)kCountsPerTransform - 1 : -1);
                    __syncwarp();
                }
            }
            if (corr) {
                // the chunk's flips into the row and column sums
#pragma unroll
                for (int i = 0; i < SPL; ++i) {
                    const int jj = q + i * P;
                    const bool flipped = valid && jj < len && ((acc >> jj) & 1u);
                    red_shared_add(flipped ? (unsigned)__cvta_generic_to_shared(csum + x0 + jj) : smbase + (unsigned)sink,
                                   (old >> jj) & 1u ? 2 : -2);
                }
                const int dr = chunk_dm(acc, plus, 31);
                if (valid && q == 0) red_shared_add((unsigned)__cvta_generic_to_shared(rsum + y), dr);
            }
            M += chunk_dm(acc, plus, 31);
            __syncwarp();
        }
        left -= (uint64_t)len;
        at += (uint32_t)len;
        ready -= len;
        y = yn; ci = cn; buf ^= 1;
    }
    __syncwarp();
    int down = 0;                                              // spins -1 at the end
    for (int c = 0, i = 0; c < rc.n * L; ++c) {
        const int len = rc.len(c % rc.n);
        const unsigned bits = lat[c];
        down += __popc(bits);
        if (valid)
            for (int jj = q; jj < len; jj += P) gl[i + jj] = (bits >> jj) & 1u ? -1 : 1;
        i += len;
    }
    if (valid) {
        uint32_t* gH = P_.H + P_.slot_tab[s];
        uint64_t* gv = P_.visits + P_.slot_tab[s];
        for (int k = q; k < nb; k += P) {
            const long long dv = CNT ? gs[RW * k + 1] : (gs[k] - gg[k]) / lnf;
            const long long gnew = CNT ? gs[RW * k] + dv * lnf : gs[k];
            const int e = commit_visits(gH, gv, k, dv, gnew);
            if (e) atomicOr(&P_.counters[0], e);
            gg[k] = gnew;
        }
        if (moments) book_moments();
        if (q == 0) {
            const int root = (int)(state & 0xFFFFFu);
            if ((unsigned)(root - gsoff) >= (unsigned)(nb * RS)) atomicOr(&P_.counters[0], ERR_BOUNDS);
            P_.cfg_E[cfg] = (long long)Ewlo + ((long long)((root - gsoff) / RS) << sh);
            P_.cfg_M[3 * cfg] = N - 2 * down;
            P_.slot_sweeps[s] = sweeps0 + (uint64_t)p.nsweeps;
        }
    }
}

// BLOCKS: of 128 threads on an SM that the registers leave room for.  The observables take 190 to 212 registers,
// which 8 to 10 warps of an SM have; with 168 it holds 12, the better form where there are as many (L = 64, moments,
// 2944 walkers, two a warp: 26.2 -> 33.0e9 flips/s; 2048: 31.2 -> 30.6).
template <int G, bool OBS, bool CNT, int BLOCKS>
__global__ void __launch_bounds__(128, BLOCKS) k_sweep_ising_bins(const SweepParams p)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int wib = threadIdx.x >> 5;
    sweep_bins_warp<G, OBS, CNT>(p, blockIdx.x * (blockDim.x >> 5) + wib, smem + (size_t)wib * G * p.smem_per_warp);
}

template <int G>
SweepKernel bins_kernel_t(bool obs, bool cnt, bool crowded)
{
    if (!obs) return cnt ? k_sweep_ising_bins<G, false, true, 1> : k_sweep_ising_bins<G, false, false, 1>;
    if (crowded) return cnt ? k_sweep_ising_bins<G, true, true, 3> : k_sweep_ising_bins<G, true, false, 3>;
    return cnt ? k_sweep_ising_bins<G, true, true, 1> : k_sweep_ising_bins<G, true, false, 1>;
}

SweepKernel bins_kernel(int G, bool obs, bool cnt, bool crowded)
{
    return G == 1 ? bins_kernel_t<1>(obs, cnt, crowded) : G == 2 ? bins_kernel_t<2>(obs, cnt, crowded) : bins_kernel_t<4>(obs, cnt, crowded);
}

// ---------------------------------------------------------------------------
// The same sweeps one decision after another, for lattices whose rows are one chunk of C = 4, 8 or 16 sites, in crowded
// launches.  A block of the tree costs the same however few sites the row leaves it, and the counts of a row are
// formed anew for every few blocks; the chain's step is 16 instructions and a dependent shared load, which several
// walkers a warp and several warps hide.  Per row the walker's lanes form each site's table offsets (without / with its left neighbour flipped; the last
// site's wrap term) from the lattice before the row above is decided, and correct them for that row's flips; all lanes
// then go through the row in lockstep, the two proposals a step may lead to formed while its predecessor is decided.
// Measured against the tree, four walkers a warp, cycles per flip of a walker: 5952 walkers, L = 4 531 -> 266, L = 8
// 315 -> 168 (with moments 500 -> 243), L = 16 249 -> 148 (364 -> 242); 1200 walkers 203 -> 157, 152 -> 96, 105 -> 79 (two
// a warp); with correlators L = 16 202 -> 200 and 250 -> 313, which stays with the tree.
// ---------------------------------------------------------------------------
__host__ __device__ inline int rows_smem(int nbcap, int C, bool obs, bool corr)
{
    return (nbcap + 2 * kGuard) * 8 + C * C + 8 * C * 8 + 2 * C * 8 + (obs ? 4 * C : 0) + (corr ? 8 * C + 4 * nbcap : 0);
}

template <int G, int C, bool OBS>
__global__ void __launch_bounds__(128, OBS ? 3 : 1) k_sweep_ising_rows(const SweepParams p)
{
    constexpr int P = 32 / G, N = C * C;
    constexpr int SPL = (C + P - 1) / P;                       // sites per lane in a row
    static_assert(C % 4 == 0 && C >= 4 && C <= 16 && G > 1, "rows");
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int grp = lane / P, q = lane - grp * P, gbase = grp * P;
    const int li = (blockIdx.x * (blockDim.x >> 5) + wib) * G + grp;
    const bool valid = li < p.nslots;
    if (__ballot_sync(kFull, valid) == 0 || engine_failed_warp(p.P.counters)) return;   // no walkers, or stopped
    const DevPtrs& P_ = p.P;
    const int s = p.slots[valid ? li : 0];                     // idle groups shadow a walker, never write
    const InstDev I = P_.inst[P_.slot_inst[s]];
    const int w = P_.slot_win[s];
    const WinDev W = P_.win[w];
    const int nb = W.nb;
    unsigned char* base = smem + (size_t)(wib * G + grp) * p.smem_per_warp;
    long long* gs = reinterpret_cast<long long*>(base) + kGuard;                // gs[-kGuard .. nb + kGuard)
    int8_t* lat = reinterpret_cast<int8_t*>(base + (p.nbcap + 2 * kGuard) * 8);
    long long* Tb = reinterpret_cast<long long*>(lat + N);                      // 2 x 4C thresholds (+ ln f)
    int2* Db = reinterpret_cast<int2*>(Tb + 8 * C);                             // 2 x C offset pairs
    int* seqb = reinterpret_cast<int*>(Db + 2 * C);                             // a row's bins (observables)
    int* rsum = seqb + C;                                                       // correlators: row sums,
    int* csum = rsum + C;                                                       // column sums,
    int* bcnt = csum + C;                                                       // bin counts modulo 1000
    char* const sm = reinterpret_cast<char*>(smem);                             // table positions: bytes from here
    const int gsoff = (int)(reinterpret_cast<char*>(gs) - sm);

    const int cfg = P_.slot_cfg[s];
    int8_t* gl = P_.spins + P_.cfg_off[cfg];
    long long* gg = reinterpret_cast<long long*>(P_.g + P_.slot_tab[s]);
    for (int i = q; i < N; i += P) lat[i] = gl[i];
    for (int k = q - kGuard; k < nb + kGuard; k += P) gs[k] = k >= 0 && k < nb ? gg[k] : kGuardValue;
    __syncwarp();
    const bool corr = OBS && P_.corr;
    if (corr) {
        plane_sums(rsum, csum, C, q, [&](int i) { return (int)lat[i]; }, P);
        const uint64_t* gv0 = P_.visits + P_.slot_tab[s];
        for (int k = q; k < nb; k += P) bcnt[k] = mod_transform(gv0[k]);
        __syncwarp();
    }

    const int J = (int)I.J_u, sh = I.bin_shift;
    const int Ewlo = (int)W.elo_u;
    const long long lnf = P_.win_lnf[w];
    const uint64_t sweeps0 = P_.slot_sweeps[s];
    const uint32_t uid = (uint32_t)(s - I.first_slot);
    const uint32_t k0 = (uint32_t)I.seed ^ uid, k1 = (uint32_t)(I.seed >> 32);
    const int E0 = (int)P_.cfg_E[cfg];
    const int b0 = (E0 - Ewlo) >> sh;
    const bool bad = ((E0 - Ewlo) & ((1 << sh) - 1)) != 0 || b0 < 0 || b0 >= nb;
    if (__ballot_sync(kFull, valid && bad)) {
        if (lane == 0) atomicOr(&P_.counters[0], ERR_BOUNDS);
        return;
    }
    int M = P_.cfg_M[3 * cfg];
    const double invN = 1.0 / (double)N;
    double* ob = OBS ? P_.obs + (size_t)P_.slot_tab[s] * P_.obs_stride : nullptr;

    // thresholds of the 4C attempts from `a0` on (a multiple of 4) into batch `buf`
    auto draw = [&](uint64_t a0, int buf) {
        longlong2* dst = reinterpret_cast<longlong2*>(Tb + buf * 4 * C);
#pragma unroll
        for (int k = 0; k < SPL; ++k) {
            const int bi = q + k * P;
            if (bi < C) {
                const uint64_t blk = (a0 >> 2) + (uint64_t)bi;
                const Philox4 r = philox4x32_10(Philox4{(uint32_t)blk, (uint32_t)(blk >> 32), kStreamWL, 0u}, k0, k1);
                dst[2 * bi] = make_longlong2(word_threshold(r.x) + lnf, word_threshold(r.y) + lnf);
                dst[2 * bi + 1] = make_longlong2(word_threshold(r.z) + lnf, word_threshold(r.w) + lnf);
            }
        }
    };

    // A row's sites as the lattice stands, before the flips of the row above: spin, energy change without / with the
    // left neighbour flipped, the correction if the site above flips; the last site's if the first flips.
    int ns[SPL], nd0[SPL], nd1[SPL], nup[SPL], nwrap = 0;
    auto prepare = [&](int y) {
        const int8_t *row = lat + y * C, *up = lat + (y == 0 ? C - 1 : y - 1) * C, *down = lat + (y == C - 1 ? 0 : y + 1) * C;
#pragma unroll
        for (int k = 0; k < SPL; ++k) {
            const int x = q + k * P;
            ns[k] = nd0[k] = nd1[k] = nup[k] = 0;
            if (x < C) {
                const int si = row[x], su = up[x], sl = row[x == 0 ? C - 1 : x - 1], sr = row[x == C - 1 ? 0 : x + 1];
                ns[k] = si;
                nd0[k] = 2 * J * si * (su + sl + sr + down[x]);
                nd1[k] = x > 0 ? nd0[k] - 4 * J * si * sl : nd0[k];
                nup[k] = 4 * J * si * su;
                if (x == C - 1) nwrap = -4 * J * si * sr;
            }
        }
    };
    auto finish = [&](int k, unsigned flips) {                 // table offsets, the row above having flipped `flips`
        const int c = (flips >> (q + k * P)) & 1u ? nup[k] : 0;
        return make_int2(((nd0[k] - c) >> sh) * 8, ((nd1[k] - c) >> sh) * 8);
    };
    auto wrap_offset = [&] { return __shfl_sync(kFull, (nwrap >> sh) * 8, gbase + (C - 1) % P); };

    const uint64_t A0 = sweeps0 * (uint64_t)N;
    draw(A0, 0);
    prepare(0);
    int cs[SPL];                                               // spins of the current row
#pragma unroll
    for (int k = 0; k < SPL; ++k) {
        cs[k] = ns[k];
        if (q + k * P < C) Db[q + k * P] = finish(k, 0u);
    }
    int cwrap = wrap_offset();
    __syncwarp();
    int2 E4[4];                                                // offsets and thresholds of the row's first four sites
    long long T4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { E4[i] = Db[i]; T4[i] = Tb[i]; }

    int bc = gsoff + b0 * 8;                                   // current bin, g there, proposal, g there
    long long gcv = gs[b0];
    int bp = bc + E4[0].x;
    long long gp = lds64(sm, bp);
    int q0 = bc + E4[1].x, q1 = bp + E4[1].y;                  // the next proposal: this one rejected / accepted
    long long bound = gcv - lnf + T4[0];

    const int64_t total = (int64_t)p.nsweeps * C;
    int y = 0;
    for (int64_t t = 0; t < total; ++t) {
        const int64_t tn = t + 1;
        const int yn = y + 1 == C ? 0 : y + 1;
        const long long* Tc = Tb + ((t >> 2) & 1) * 4 * C + (t & 3) * C;
        const long long* Tn = Tb + ((tn >> 2) & 1) * 4 * C + (tn & 3) * C;
        const int2* Dc = Db + (t & 1) * C;
        int2* Dn = Db + (tn & 1) * C;
        if ((tn & 3) == 0 && tn < total) {                     // the next row opens a batch: its buffer is not in use
            draw(A0 + (uint64_t)tn * C, (tn >> 2) & 1);
            __syncwarp();
        }
        prepare(yn);
        long long Tr[C + 1];
        int2 Er[C];
#pragma unroll
        for (int i = 0; i < 4; ++i) { Tr[i] = T4[i]; Er[i] = E4[i]; }
        Tr[C] = Tn[0];
        unsigned acc = 0;
#pragma unroll
        for (int j = 0; j < C; ++j) {
            if ((j & 1) == 0 && j + 6 <= C) {                  // inputs are read four sites ahead
                const longlong2 tv = reinterpret_cast<const longlong2*>(Tc)[(j + 4) >> 1];
                const int4 d = reinterpret_cast<const int4*>(Dc)[(j + 4) >> 1];
                Tr[j + 4] = tv.x; Tr[j + 5] = tv.y;
                Er[j + 4] = make_int2(d.x, d.y); Er[j + 5] = make_int2(d.z, d.w);
            }
            const bool a = gp < bound;
            const long long sel = a ? gp : gcv;
            const int bnew = a ? bp : bc;
            gcv = sel + lnf;
            sts64(sm, bnew, gcv);
            if (OBS) seqb[j] = bnew;
            if (a) acc |= 1u << j;
            if (j == 1 || j == 3) {                            // the next row's first sites: those above them are decided
#pragma unroll
                for (int i = j - 1; i <= j; ++i) {
                    const int2 v = finish(i / P, acc);
                    E4[i] = make_int2(__shfl_sync(kFull, v.x, gbase + i % P), __shfl_sync(kFull, v.y, gbase + i % P));
                }
            }
            bound = sel + Tr[j + 1];
            bp = a ? q1 : q0;
            gp = lds64(sm, bp);                                // after this step's store
            const int2 ev = j + 2 < C ? Er[j + 2] : E4[j + 2 - C];
            const int wv = j + 2 == C - 1 && (acc & 1u) ? cwrap : 0;           // a row's last site sees its first
            q0 = bnew + ev.x + wv;
            q1 = bp + ev.y + wv;
            bc = bnew;
        }
        unsigned plus = 0;
#pragma unroll
        for (int k = 0; k < SPL; ++k) {
            const int x = q + k * P;
            const unsigned bal = __ballot_sync(kFull, x < C && cs[k] > 0);
            plus |= ((bal >> gbase) & ((1u << P) - 1u)) << (k * P);
            if (x < C && ((acc >> x) & 1u)) lat[y * C + x] = (int8_t)(-cs[k]);
        }
        if (OBS) {
            __syncwarp();
            int first[SPL], visits[SPL];                       // is the step its bin's first of the row; the row's visits to it
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                const int x = q + k * P;
                first[k] = visits[k] = 0;
                if (!valid || x >= C) continue;
                const int b = (seqb[x] - gsoff) >> 3;
                const int32_t Mv[1] = {M + chunk_dm(acc, plus, x)};
                Ising2dModel::add_observables(ob + (size_t)b * P_.obs_stride, Mv, invN, P_.corr);
                if (corr) {
                    // G(q_min) at the steps whose bin count before the visit is a multiple of 1000: bcnt before the row
                    // and the row's earlier visits.  (The lattice already holds the row's flips.)
                    int earlier = 0;
#pragma unroll
                    for (int j = 0; j < C; ++j) {
                        const int eq = seqb[j] == seqb[x] ? 1 : 0;
                        earlier += j < x ? eq : 0;
                        visits[k] += eq;
                    }
                    first[k] = earlier == 0;
                    if ((bcnt[b] + earlier) % (int)kCountsPerTransform == 0) {
                        const double Gq = plane_corr(rsum, csum, P_.qtab + I.qtab_off, C, y, chunk_dm(acc, plus, x), 0, x, acc,
                                                     [&](int i) { return -(int)lat[y * C + i]; });
                        red_global_add(ob + (size_t)b * P_.obs_stride + 3, invN * invN * Gq);
                    }
                }
            }
            if (corr) {
                __syncwarp();
#pragma unroll
                for (int k = 0; k < SPL; ++k) {
                    const int x = q + k * P;
                    if (valid && x < C && ((acc >> x) & 1u)) csum[x] += 2 * (int)lat[y * C + x];
                    if (first[k]) bcnt[(seqb[x] - gsoff) >> 3] += visits[k];
                }
                if (valid && q == 0) rsum[y] += chunk_dm(acc, plus, 31);
            }
        }
        M += chunk_dm(acc, plus, 31);
        // the next row
#pragma unroll
        for (int k = 0; k < SPL; ++k) {
            cs[k] = ns[k];
            if (q + k * P < C) Dn[q + k * P] = finish(k, acc);
        }
        cwrap = wrap_offset();
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) T4[i] = Tn[i];
        y = yn;
    }
    __syncwarp();
    if (valid) {
        for (int i = q; i < N; i += P) gl[i] = lat[i];
        uint32_t* gH = P_.H + P_.slot_tab[s];
        uint64_t* gv = P_.visits + P_.slot_tab[s];
        for (int k = q; k < nb; k += P) {
            const long long gnew = gs[k];
            const int e = commit_visits(gH, gv, k, (gnew - gg[k]) / lnf, gnew);
            if (e) atomicOr(&P_.counters[0], e);
            gg[k] = gnew;
        }
        if (q == 0) {
            if ((unsigned)(bc - gsoff) >= (unsigned)(nb * 8)) atomicOr(&P_.counters[0], ERR_BOUNDS);
            P_.cfg_E[cfg] = (long long)Ewlo + ((long long)((bc - gsoff) >> 3) << sh);
            P_.cfg_M[3 * cfg] = M;
            P_.slot_sweeps[s] = sweeps0 + (uint64_t)p.nsweeps;
        }
    }
}

template <int G>
SweepKernel rows_kernel_t(int C, bool obs)
{
    if (C == 4) return obs ? k_sweep_ising_rows<G, 4, true> : k_sweep_ising_rows<G, 4, false>;
    if (C == 8) return obs ? k_sweep_ising_rows<G, 8, true> : k_sweep_ising_rows<G, 8, false>;
    return obs ? k_sweep_ising_rows<G, 16, true> : k_sweep_ising_rows<G, 16, false>;
}

SweepKernel rows_kernel(int G, int C, bool obs) { return G == 2 ? rows_kernel_t<2>(C, obs) : rows_kernel_t<4>(C, obs); }

// Ashkin-Teller: sweep = sigma pass then tau pass (wang_landau.hpp:109-119); the flavour toggles
// after each pass.  A window holds tens of thousands of bins, so its logDoS stays in global memory;
// the part around the walker is held in shared memory (TableCache below).
constexpr int kMinCache = 2048;
constexpr int kTableReach = 512;           // serial chain: bins on either side prefetched per chunk

// a Philox block gives four attempts' words, so that a warp draws 128 thresholds at a time (32 at a
// time, one word a lane, was 700 cycles a chunk)
constexpr int kTableRing = 256;
struct TableStage {
    longlong2 du[32 + 8];    // per site: {proposal, proposal after its left neighbour flipped in this chunk};
                             // tree: 32-bit, {proposal, change of it when the left neighbour flips}
    long long wcu;           // row-wrap correction of the last site when the chunk is a whole row
    int seq[32];             // bin after each step (observables)
    unsigned sink;           // counts the lanes off the path, read by nobody
    unsigned pad[5];
    long long T[kTableRing]; // acceptance thresholds, by attempt modulo kTableRing (serial chain: the chunk's 32)
};
constexpr int kSerialStage = offsetof(TableStage, T) + 32 * 8;         // what the serial chain has of it
static_assert(kSerialStage % 16 == 0 && offsetof(TableStage, T) % 16 == 0 && sizeof(TableStage) % 16 == 0, "what follows is 16-byte aligned");

// Chain state of one Ashkin-Teller walker (lane 0).  The energy is carried as its
// position v = (E - E_lo) * bin_mul - gblo << bin_shift, in units of the bin
// numerator within the window, so that a proposal's bin is (v + dv) >> bin_shift:
// one add and one shift instead of a multiply per candidate.
struct TableChain {
    long long v, vn, gc, draws;
    long long G0, G1;        // logDoS loaded for step j's proposal if step j-1 was rejected / accepted
    long long T;             // step j's threshold
    longlong2 q;             // step j+1's proposals
    int b, bn, err;
    bool inr, ap;            // step j's proposal in the window; step j-1 accepted
    unsigned acc;
};

// One step j of a chunk decided serially by lane 0, software-pipelined two deep: replayed runs
// (REPLAY), whose recorded uniforms are consumed on demand, energy changes too large for the tree's
// positions, and crowded launches with observables.  Unrolled by four, the next step's threshold read a
// step ahead, the replayed form compiled apart: Ashkin-Teller L = 32, 2048 walkers 8.6 -> 9.2e9 flips/s, with moments
// 6.6 -> 7.1e9.  On entry (vn, bn, inr) is step j's proposal, and its logDoS is G1 or G0
// (as step j-1 was accepted or not), loaded during step j-1.  With PREFETCH the two proposals of step
// j+1 (step j rejected: from v; accepted: from vn) are loaded first.  A value loaded before step j-1's
// write to bin b is stale exactly when the proposal is b: gc replaces it.  LOADQ: step j+2 exists and
// its proposals are read from shared memory now.  WRAPFIX: step j+1 is the last site of a whole-row
// chunk, whose right neighbour is the row's first site, flipped in this chunk iff bit 0 of acc.
template <bool REPLAY, bool OBS, bool PREFETCH, bool LOADQ, bool WRAPFIX>
__device__ __forceinline__ void serial_step(TableChain& c, const int j, TableStage* st, long long* gg, const int nb,
                                        const int sh, const long long lnf, const DevPtrs& P,
                                        const long long thr_off, const long long thr_n)
{
    long long t0 = 0, t1 = 0, G0 = 0, G1 = 0, Tn = 0;
    longlong2 qn = make_longlong2(0, 0);
    int b0 = 0, b1 = 0;
    bool i0 = false, i1 = false;
    if (LOADQ) qn = st->du[j + 2];
    if (PREFETCH) {
        if (!REPLAY) Tn = st->T[j + 1];
        t0 = c.v + c.q.x;
        t1 = c.vn + c.q.y;
        if (WRAPFIX) {
            const long long wcu = st->wcu;
            if (c.acc & 1u) t0 += wcu;
            if (j == 0 || (c.acc & 1u)) t1 += wcu;
        }
        b0 = (int)(t0 >> sh);
        b1 = (int)(t1 >> sh);
        i0 = (unsigned)b0 < (unsigned)nb;
        i1 = (unsigned)b1 < (unsigned)nb;
        G0 = gg[min((unsigned)b0, (unsigned)(nb - 1))];
        G1 = gg[min((unsigned)b1, (unsigned)(nb - 1))];
    }
    const long long gn = c.bn == c.b ? c.gc : (c.ap ? c.G1 : c.G0);
    const long long d = gn - c.gc;
    bool a;
    if (!REPLAY) {
        a = c.inr && (d < c.T);
    } else if (c.inr && d > 0) {
        if (c.draws >= thr_n) { c.err = ERR_REPLAY_EXHAUSTED; a = false; }
        else { a = d < P.thr[thr_off + c.draws]; ++c.draws; }
    } else {
        a = c.inr;
    }
    if (a) { c.v = c.vn; c.b = c.bn; c.gc = gn; c.acc |= 1u << j; }
    c.gc += lnf;
    gg[c.b] = c.gc;
    if (OBS) st->seq[j] = c.b;
    if (PREFETCH) {
        c.vn = a ? t1 : t0;
        c.bn = a ? b1 : b0;
        c.inr = a ? i1 : i0;
        c.G0 = G0; c.G1 = G1; c.ap = a;
        c.T = Tn;
        c.q = qn;
    }
}

// The same chunk decided five sites at a time on the binary tree of outcomes, as the bin-tracking
// kernel does it (above), one walker per warp: lane q >= 1 is the node at level log2(q), lane 0 stands
// for the walker's present bin.  Positions are 32-bit bin numerators relative to the bin the block
// starts in, without the trailing binary zeros that all energy changes share (the bin multiplier's);
// a node's is a sum of its path's changes, each times a lane constant 0 or 1 (integer multiply-adds,
// which leave the ALU to the rest).  The path's bins come from the ancestor lanes by shuffle.
struct TableTree {
    static constexpr int D = 5;
    int lvl, lvla;                         // level, level for the length check
    unsigned want, anc, path;              // ancestors' votes: needed value, mask; the decisions that lead here
    int up[D - 1];                         // the ancestor at each level (beyond the node's own: itself)
    int took[D - 1], both[D - 1];          // 0/1: the decision at a level was to flip; so was the one before it
    int own, ownx;                         // 0/1: there is a proposal (not in lane 0); its left neighbour flipped
    int firstP;                            // 0/1: the proposal sees the flip of the block's left neighbour
    int dwell[D];                          // steps of the way here that end at the block's first bin, and at the
                                           // proposal accepted at each level
    bool first, last, leaf;                // first decision on the way here; the one before this node
    __device__ explicit TableTree(int q)
    {
        lvl = q == 0 ? 0 : 31 - __clz(q);
        lvla = q == 0 ? 32 : lvl;
        want = anc = path = 0;
#pragma unroll
        for (int i = 0; i < D - 1; ++i) {
            const bool above = i < lvl, a = above && ((q >> (lvl - 1 - i)) & 1);
            up[i] = above ? q >> (lvl - i) : q;
            if (above) anc |= 1u << up[i];
            if (a) { want |= 1u << up[i]; path |= 1u << i; }
        }
#pragma unroll
        for (int k = 0; k < D; ++k) {
            bool here = k == 0;            // k: the first bin, then the proposals of levels 0 ..
            dwell[k] = 0;
#pragma unroll
            for (int i = 0; i < D - 1; ++i) {
                if (accepts(i)) here = k == i + 1;
                dwell[k] += here && i < lvl ? 1 : 0;
            }
        }
        first = accepts(0);
        last = lvl > 0 && accepts(lvl - 1);
        if (q == 0) { anc = 1u; want = 1u; }                   // its vote is always 0: never on the path
        leaf = lvl == D - 1;
#pragma unroll
        for (int i = 0; i < D - 1; ++i) {
            took[i] = accepts(i) ? 1 : 0;
            both[i] = i > 0 && accepts(i) && accepts(i - 1) ? 1 : 0;
            keep(took[i]);
            keep(both[i]);
        }
        own = q == 0 ? 0 : 1;
        ownx = own && last ? 1 : 0;
        firstP = first || q == 1 ? 1 : 0;
        keep(own); keep(ownx); keep(firstP);
        // lane constants: kept in registers, not worked out again in every block
        keep(want); keep(anc); keep(path); keep(lvl); keep(lvla);
#pragma unroll
        for (int i = 0; i < D - 1; ++i) keep(up[i]);
#pragma unroll
        for (int k = 0; k < D; ++k) keep(dwell[k]);
    }
    template <class T>
    __device__ static void keep(T& x) { asm volatile("" : "+r"(x)); }
    __device__ bool accepts(int i) const { return (path >> i) & 1u; }
};

// The part of a walker's table around its present bin, in shared memory: bins [lo, lo + size) at slot
// bin mod size, g when the bin came in and the visits since (g now = g + visits x ln f).  A bin's
// visits are booked (g, per-stage count, cumulative visits) when it leaves; bins outside are always
// up to date in global memory.
struct TableCache {
    long long* g;
    unsigned* n;
    int size, lo, nb;                      // size: a power of two
    long long* gg;
    uint32_t* gH;
    uint64_t* gv;
    long long lnf;
    int err;
    __device__ __forceinline__ bool holds(int b) const { return (unsigned)(b - lo) < (unsigned)size; }
    // the window's bins up to `margin` from b are all cached
    __device__ __forceinline__ bool within(int b, int margin) const
    {
        return (lo == 0 || b - margin >= lo) && (lo + size >= nb || b + margin < lo + size);
    }
    // (kBatch bins of a lane at a time, their loads before their stores: a walker at high energies recentres
    // once per 1700 flips: 51,000 cycles with one bin's loads and stores after another's, 15,000 so)
    static constexpr int kBatch = 4;
    __device__ void fill(int first, int last, int lane)
    {
        for (int b = first + lane; b < last; b += 32 * kBatch) {
            long long x[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int k = b + 32 * i;
                x[i] = k < min(last, nb) ? gg[k] : 0;
            }
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int k = b + 32 * i;
                if (k < last) {
                    g[k & (size - 1)] = x[i];
                    n[k & (size - 1)] = 0;
                }
            }
        }
    }
    __device__ void book(int first, int last, int lane)
    {
        for (int b = first + lane; b < last; b += 32 * kBatch) {
            unsigned v[kBatch];
            uint32_t h[kBatch];
            uint64_t c[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int k = b + 32 * i;
                v[i] = k < last ? n[k & (size - 1)] : 0u;
                h[i] = v[i] ? gH[k] : 0u;
                c[i] = v[i] ? gv[k] : 0u;
            }
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int k = b + 32 * i;
                if (v[i]) {
                    const long long gnew = g[k & (size - 1)] + (long long)v[i] * lnf;
                    gg[k] = gnew;
                    err |= commit_visits(gH, gv, k, h[i], c[i], v[i], gnew);
                }
            }
        }
    }
    // around bin b (all lanes)
    __device__ void centre(int b, int lane)
    {
        const int to = max(0, min(b - size / 2, nb - size));
        if (to == lo) return;
        __syncwarp();
        const int out0 = to > lo ? lo : max(to + size, lo), out1 = to > lo ? min(to, lo + size) : lo + size;
        const int in0 = to > lo ? max(lo + size, to) : to, in1 = to > lo ? to + size : min(lo, to + size);
        book(out0, out1, lane);
        lo = to;
        __syncwarp();
        fill(in0, in1, lane);
        __syncwarp();
    }
};

// Sweeps of any model type of models.cuh with the window tables in global memory (the
// Ashkin-Teller instances, whose windows hold tens of thousands of bins, and Ising windows too
// large for shared memory).  One warp per walker; the planes sweep in turn (sigma then tau for
// Ashkin-Teller, wang_landau.hpp:109-119), the flipped plane toggling after each pass.
// The sweeps of one walker (launch position li; the warp's shared memory starts at warp_base).
//
// Bound: the latency of one block of five decisions (about 400 cycles at one warp per scheduler:
// shared loads and shuffles of the bins, vote and reductions, half of it instruction issue), once per five
// flips, and about 900 cycles a chunk of energy changes, thresholds and loop; with many walkers per SM the
// instructions and the cached bins that fit.  Ashkin-Teller L = 32, bins of 0.05, 8 windows x 4 walkers,
// cycles per flip from flat tables: 32 walkers 192 as a chain of dependent global loads and stores, 169 as a
// tree of 64-bit positions with 32 thresholds a draw, 122 now; 512 walkers 411, 210, 149; 2048 walkers 832,
// 557, 411 (with the tables of a longer run 432, the chain 439: two waves of seven warps per SM, each with
// its cached bins).
enum TableMode : int { kTableSerial = 0, kTableTree = 1, kTableReplay = 2 };

template <class Model, int MODE, bool OBS>
__device__ __forceinline__ void sweep_tables_warp(const SweepParams& p, const int li, unsigned char* warp_base)
{
    constexpr int NP = Model::kPlanes, NM = Model::kMags, NC = Model::kCorrPlanes;
    const int lane = threadIdx.x & 31;
    if (li >= p.nslots || engine_failed_warp(p.P.counters)) return;
    const DevPtrs& P = p.P;
    const int s = p.slots[li];
    const InstDev I = P.inst[P.slot_inst[s]];
    const int w = P.slot_win[s];
    const WinDev W = P.win[w];
    const int L = I.L, N = I.N, nb = W.nb;
    const RowChunks rc(L);
    // from the start of shared memory, so that the accesses below are shared-memory accesses
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned char* base = smem + (int)(warp_base - smem);
    constexpr bool TREE = MODE == kTableTree, REPLAY = MODE == kTableReplay;
    TableStage* st = reinterpret_cast<TableStage*>(base);
    int8_t* sp = reinterpret_cast<int8_t*>(base) + (TREE ? (int)sizeof(TableStage) : kSerialStage);     // NP planes of N spins
    const int64_t* hf = I.field_off >= 0 ? P.fields + I.field_off : nullptr;

    const int cfg = P.slot_cfg[s];
    int8_t* gl = P.spins + P.cfg_off[cfg];
    for (int i = lane; i < NP * N; i += 32) sp[i] = gl[i];
    long long* gg = reinterpret_cast<long long*>(P.g + P.slot_tab[s]);
    // the serial chain works on the table in global memory and derives the visits from a copy of it
    long long* g0 = !TREE ? reinterpret_cast<long long*>(P.gsnap + P.slot_tab[s]) : nullptr;
    if (!TREE)
        for (int k = lane; k < nb; k += 32) g0[k] = gg[k];
    __syncwarp();
    // correlators: row sums rs[p] and column sums cs[p] of every correlator plane
    int* sums = reinterpret_cast<int*>(sp + ((NP * N + 15) & ~15));
    TableCache tab;
    tab.size = p.cache;
    tab.g = reinterpret_cast<long long*>(reinterpret_cast<unsigned char*>(sums) + (P.corr ? (8 * NP * L + 15) & ~15 : 0));
    tab.n = reinterpret_cast<unsigned*>(tab.g + tab.size);
    tab.nb = nb;
    tab.gg = gg;
    tab.gH = P.H + P.slot_tab[s];
    tab.gv = P.visits + P.slot_tab[s];
    tab.err = 0;
    const bool corr = OBS && P.corr;
    const double invN = 1.0 / (double)N;
    double* const ob = OBS ? P.obs + (size_t)P.slot_tab[s] * P.obs_stride : nullptr;
    if (corr) {
        for (int cp = 0; cp < NC; ++cp)
            plane_sums(sums + 2 * L * cp, sums + 2 * L * cp + L, L, lane,
                       [&](int i) { return Model::corr_site(sp, N, i, cp); });
        __syncwarp();
    }

    const long long lnf = P.win_lnf[w];
    const uint64_t sweeps0 = P.slot_sweeps[s];
    const uint32_t uid = (uint32_t)(s - I.first_slot);
    const uint64_t seed = I.seed;
    const long long eglo = I.eglo_u, mul = I.bin_mul;
    const int sh = I.bin_shift;
    const long long vlo = (long long)W.gblo << sh;     // window start in bin-numerator units
    // couplings and fields in position units, for the tree without their common trailing zeros
    using Pos = std::conditional_t<TREE, int, long long>;
    // (the multiplier's, and one more: a flip changes the energy by an even number)
    const int zm = TREE ? min(__ffsll(mul) - 1, sh) : 0, even = TREE && zm < sh ? 1 : 0;
    const int zeros = zm + even, shz = sh - zeros;
    const long long mulz = mul >> zm;
    const CouplingsOf<Pos> cpl{(Pos)(I.J_u * mulz), (Pos)(I.K_u * mulz)};
    auto field = [&](int i) { return hf ? (Pos)(hf[i] * mulz) : Pos(0); };
    int2* const dx = reinterpret_cast<int2*>(st->du);
    const bool wraps = rc.n == 1;                      // a row is one chunk: its last site sees its first
    int flavour = NP == 1 ? 0 : P.slot_flavour[s];

    TableChain c{};                                    // serial chain, lane 0
    int32_t M[3] = {0, 0, 0};                          // the magnetisations
    long long thr_off = 0, thr_n = 0;
    long long vr = ((long long)P.cfg_E[cfg] - eglo) * mul - vlo;       // the walker's position
    for (int m = 0; m < NM; ++m) M[m] = P.cfg_M[3 * cfg + m];
    if ((vr >> sh) < 0 || (vr >> sh) >= nb) {
        if (lane == 0) atomicOr(&P.counters[0], ERR_BOUNDS);
        return;
    }
    if (!TREE && lane == 0) {
        c.v = vr;
        c.b = (int)(vr >> sh);
        c.gc = gg[c.b];
        if (REPLAY) { c.draws = P.slot_draws[s]; thr_off = P.slot_thr_off[s]; thr_n = P.slot_thr_n[s]; }
    }
    // the tree's position: bin, numerator within it in units of 2^zeros, and what is below them for good
    int b0 = (int)(vr >> sh), fr = (int)((vr >> zeros) & ((1ll << shz) - 1));
    const long long below = vr & ((1ll << zeros) - 1);
    if (TREE) {
        tab.lnf = lnf;
        tab.lo = max(0, min(b0 - tab.size / 2, nb - tab.size));
        tab.fill(tab.lo, tab.lo + tab.size, lane);
    }
    const unsigned sink = (unsigned)__cvta_generic_to_shared(&st->sink);
    const TableTree tree(lane);
    constexpr int D = TableTree::D;
    const int lnf_lo = (int)(uint32_t)lnf, lnf_hi = (int)((lnf - (long long)(int)(uint32_t)lnf) >> 32);
    const uint64_t attempts0 = sweeps0 * (uint64_t)NP * (uint64_t)N;   // the launch's first attempt
    uint64_t attempt = attempts0;                      // of the current chunk
    Pos hnext = TREE ? field(min(lane, N - 1)) : Pos(0);      // field of the chunk's site
    uint64_t drawn = attempts0 >> 2;                   // next Philox block
    int ready = -(int)(attempts0 & 3);                 // thresholds in the ring from the current chunk on
    auto draw = [&] {
        const uint64_t blk = drawn + (uint64_t)lane;
        const Philox4 r = philox4x32_10(Philox4{(uint32_t)blk, (uint32_t)(blk >> 32), kStreamWL, 0u}, (uint32_t)seed ^ uid,
                                        (uint32_t)(seed >> 32));
        longlong2* t = reinterpret_cast<longlong2*>(st->T + (((uint32_t)blk * 4u) & (kTableRing - 1)));
        t[0] = make_longlong2(word_threshold(r.x), word_threshold(r.y));
        t[1] = make_longlong2(word_threshold(r.z), word_threshold(r.w));
        drawn += 32;
        ready += 128;
    };
    if (TREE) draw();

    struct Node { int rC, rP, x0; long long T; };      // position and proposal relative to the block's start
    auto node = [&](int j0) {
        const int2* d = dx + j0;
        Node n;
        const int2 d0 = d[0];
        n.x0 = d0.y;
        n.rC = tree.took[0] * d0.x;
#pragma unroll
        for (int i = 1; i < D - 1; ++i) {
            const int2 v = d[i];
            n.rC += tree.took[i] * v.x + tree.both[i] * v.y;
        }
        const int2 v = d[tree.lvl];
        n.rP = n.rC + tree.own * v.x + tree.ownx * v.y;
        n.T = st->T[((uint32_t)attempt + (uint32_t)(j0 + tree.lvl)) & (kTableRing - 1)];
        return n;
    };

    for (int sw = 0; sw < p.nsweeps; ++sw) {
        for (int pass = 0; pass < NP; ++pass) {
            const int plane = NP == 1 ? 0 : flavour;
            int8_t* A = sp + plane * N;
            const int8_t* B = NP == 1 ? A : sp + (plane ^ 1) * N;
            for (int ch = 0, cc = 0, y = 0, c0 = 0, C = rc.len(0); ch < L * rc.n; ++ch) {
                const int x0 = c0 - y * L;
                if (TREE) {
                    if (!tab.within(b0, tab.size / 8)) tab.centre(b0, lane);
                } else {
                    // the lines of g within kTableReach bins of the walker's bin into L1 (the chunk's proposals
                    // mostly fall there), one line per lane per 512 bins
                    const int bcur = __shfl_sync(kFull, c.b, 0);
                    for (int k = lane * 16 - kTableReach; k <= kTableReach; k += 32 * 16) {
                        const int bb = bcur + k;
                        if ((unsigned)bb < (unsigned)nb) asm volatile("prefetch.global.L1 [%0];" ::"l"(gg + bb));
                    }
                }
                int ai = 0, sg[NM], far = 0;
                for (int m = 0; m < NM; ++m) sg[m] = 0;
                const Pos h = hnext;                   // (read while the chunk before it was decided)
                if (lane < C) {
                    const int i = c0 + lane, x = x0 + lane;
                    const Neighbours nbr{y == 0 ? i + (L - 1) * L : i - L, x == 0 ? i + L - 1 : i - 1,
                                         x == L - 1 ? i - (L - 1) : i + 1, y == L - 1 ? i - (L - 1) * L : i + L};
                    ai = A[i];
                    Model::flip_signs(ai, B[i], plane, sg);
                    const Pos d0 = Model::delta_at(A, B, i, nbr, cpl, TREE ? h : field(i));
                    const Pos dl = lane > 0 ? Model::flipped_at(A, B, i, nbr.left, cpl) : Pos(0);
                    // where the chunk is a row: the change of its last site's once the first has flipped
                    const Pos wrap = wraps && lane == C - 1 ? Model::flipped_at(A, B, i, nbr.right, cpl) >> even : Pos(0);
                    if constexpr (TREE) {
                        const int2 d = make_int2(d0 >> even, dl >> even);
                        const int last = abs(wrap);
                        dx[lane] = d;
                        far = (max(abs(d.x), abs(d.x + d.y)) + last >> shz) + 1;
                    } else {
                        st->du[lane] = make_longlong2(d0, d0 + dl);
                    }
                    if (wraps && lane == C - 1) st->wcu = wrap;
                    if (!TREE && !REPLAY) st->T[lane] = word_threshold(philox_word(seed, uid, attempt + (uint64_t)lane, kStreamWL));
                }
                // bins a block's nodes can lie away from its start: five steps, the last site's with its wrap term
                // (fields and the other bonds can cancel what it would be part of)
                const int reach = TREE ? D * (int)__reduce_max_sync(kFull, (unsigned)far) : 0;
                __syncwarp();
                // the next chunk: position, first site, length
                int cn = cc + 1, yn = y;
                if (cn == rc.n) { cn = 0; ++yn; }
                const int Cn = rc.len(cn);
                unsigned acc = 0;
                if (!TREE) {
                    if (lane == 0) {
                        c.acc = 0;
                        c.vn = c.v + st->du[0].x;
                        c.bn = (int)(c.vn >> sh);
                        c.inr = (unsigned)c.bn < (unsigned)nb;
                        c.G0 = c.G1 = gg[min((unsigned)c.bn, (unsigned)(nb - 1))];
                        c.ap = false;
                        if (!REPLAY) c.T = st->T[0];
                        if (C == 1) {
                            serial_step<REPLAY, OBS, false, false, false>(c, 0, st, gg, nb, sh, lnf, P, thr_off, thr_n);
                        } else {
                            c.q = st->du[1];
#pragma unroll 4
                            for (int j = 0; j < C - 2; ++j)
                                serial_step<REPLAY, OBS, true, true, false>(c, j, st, gg, nb, sh, lnf, P, thr_off, thr_n);
                            if (wraps) serial_step<REPLAY, OBS, true, false, true>(c, C - 2, st, gg, nb, sh, lnf, P, thr_off, thr_n);
                            else serial_step<REPLAY, OBS, true, false, false>(c, C - 2, st, gg, nb, sh, lnf, P, thr_off, thr_n);
                            serial_step<REPLAY, OBS, false, false, false>(c, C - 1, st, gg, nb, sh, lnf, P, thr_off, thr_n);
                        }
                    }
                    acc = __shfl_sync(kFull, c.acc, 0);
                } else {
                    // first bins from which a block stays among the cached ones (none: a span of 0 far away)
                    int near0 = tab.lo == 0 ? 0 : tab.lo + reach;
                    const int near1 = tab.lo + tab.size >= nb ? nb - 1 : tab.lo + tab.size - 1 - reach;
                    const unsigned nears = near1 >= near0 ? (unsigned)(near1 - near0) : 0u;
                    if (near1 < near0) near0 = nb;
                    int flipped = 0;                   // all ones: the block's left neighbour flipped just before it
                    // one block of nlev sites from the chunk's site j0, `ahead` the work that does not wait for
                    // it.  NEAR: every bin its lanes can name is cached.
                    auto block = [&](auto near, const Node& n, int nlev, int j0, int wC, int wP, auto ahead) {
                        constexpr bool NEAR = decltype(near)::value;
                        const int x0 = flipped & n.x0;
                        const int vC = tree.took[0] * x0 + (fr + n.rC + wC), vP = tree.firstP * x0 + (fr + n.rP + wP);
                        const int oC = vC >> shz, oP = vP >> shz;          // bins from the block's first one
                        const int bC = b0 + oC, bP = b0 + oP;
                        const int kP = bP & (tab.size - 1), kC = bC & (tab.size - 1);
                        long long gP = tab.g[kP], gC = tab.g[kC];
                        int cP = (int)tab.n[kP], cC = (int)tab.n[kC];
                        // (a node below an out-of-window proposal is never on the path: what it reads does not matter)
                        const bool inr = (unsigned)bP < (unsigned)nb;
                        if (!NEAR) {
                            if (inr && !tab.holds(bP)) { gP = gg[bP]; cP = 0; }
                            if ((unsigned)bC < (unsigned)nb && !tab.holds(bC)) { gC = gg[bC]; cC = 0; }
                        }
                        // visits to this node's two bins on the way here: its path stays `dwell` steps at the
                        // block's first bin and at every accepted proposal
                        int nC = oC == 0 ? tree.dwell[0] : 0, nP = oP == 0 ? tree.dwell[0] : 0;
#pragma unroll
                        for (int i = 0; i < D - 1; ++i) {
                            const int o = __shfl_sync(kFull, oP, tree.up[i]);
                            nC += o == oC ? tree.dwell[i + 1] : 0;
                            nP += o == oP ? tree.dwell[i + 1] : 0;
                        }
                        const bool live = tree.lvla < nlev;
                        const long long bound = mad_units(gC + n.T, (cC + nC) - (cP + nP), lnf_lo, lnf_hi);
                        const bool a = (gP < bound) & live & inr;
                        const unsigned vote = __ballot_sync(kFull, a);
                        const bool on = ((vote ^ tree.want) & tree.anc) == 0;
                        const unsigned v = (unsigned)(a ? vP : vC) ^ 0x80000000u;      // (in order as unsigned)
                        const bool mine = on && live, end = on && tree.leaf;
                        const int bin = a ? bP : bC;
                        // the last node of the path has the walker's position and the block's decisions
                        const int to = (int)(__reduce_max_sync(kFull, end ? v : 0u) ^ 0x80000000u);
                        const unsigned path = __reduce_max_sync(kFull, end ? tree.path | (a ? 1u << (D - 1) : 0u) : 0u);
                        if (OBS && mine) st->seq[j0 + tree.lvl] = bin;
                        if (!NEAR && __any_sync(kFull, mine && !tab.holds(bin))) {
                            // a step outside the cached bins: booked at once, in order
                            const int sl = mine ? tree.lvl : -1;
                            for (int i = 0; i < D; ++i) {
                                if (sl == i) {
                                    if (tab.holds(bin)) tab.n[bin & (tab.size - 1)] += 1u;
                                    else {
                                        const long long gnew = gg[bin] + lnf;
                                        gg[bin] = gnew;
                                        tab.err |= commit_visits(tab.gH, tab.gv, bin, 1, gnew);
                                    }
                                }
                                __syncwarp();
                            }
                        } else {
                            red_shared_inc(mine ? (unsigned)__cvta_generic_to_shared(tab.n + (bin & (tab.size - 1))) : sink);
                        }
                        ahead();
                        __syncwarp();
                        b0 += to >> shz;
                        fr = to & ((1 << shz) - 1);
                        acc |= path << j0;
                        flipped = -((int)(path >> (nlev - 1)) & 1);
                    };
                    auto decide = [&](const Node& n, int nlev, int j0, int wC, int wP, auto ahead) {
                        if ((unsigned)(b0 - near0) <= nears) block(std::true_type{}, n, nlev, j0, wC, wP, ahead);
                        else block(std::false_type{}, n, nlev, j0, wC, wP, ahead);
                    };
                    Node n = node(0);
                    int j0 = 0;
                    for (; j0 + D < C; j0 += D) {
                        Node next;
                        decide(n, D, j0, 0, 0, [&] { next = node(j0 + D); });
                        n = next;
                    }
                    // the chunk's last block; where the chunk is a row, its last site sees the first one's flip
                    int wC = 0, wP = 0;
                    if (wraps) {
                        const int li = C - 1 - j0;
                        const int t = (j0 > 0 ? (acc & 1u) != 0 : tree.first) ? (int)st->wcu : 0;
                        if (tree.lvla == li) wP = t;           // (not the idle lane)
                        else if (tree.accepts(li)) wC = wP = t;
                    }
                    decide(n, C - j0, j0, wC, wP, [&] {
                        if (ready < C + Cn) draw();
                        ready -= C;
                        hnext = field(min((ch + 1 == L * rc.n ? 0 : c0 + C) + lane, N - 1));
                    });
                }
                // per magnetisation that the plane's flips change: the steps whose accepted flip lowers it
                // (its term was +1; the others raise it); the change after step j is -2 (lowered - raised)
                // up to j
                unsigned plus[NM] = {};
                int total[NM] = {};                    // by the whole chunk
                auto changes = [&](int m) { return m == NM - 1 || m == plane; };
                auto dm = [&](int m, int j) {
                    const unsigned le = acc & (0xFFFFFFFFu >> (31 - j));
                    return changes(m) ? 2 * (int)__popc(le) - 4 * (int)__popc(le & plus[m]) : 0;
                };
                if (OBS)
                    for (int m = 0; m < NM; ++m) {
                        plus[m] = __ballot_sync(kFull, lane < C && sg[m] > 0);
                        total[m] = dm(m, 31);
                    }
                if (OBS) {
                    __syncwarp();
                    const int bin = lane < C ? st->seq[lane] : -1 - lane;
                    // correlators: the bin's visits booked so far and those not booked yet (this chunk's
                    // are among them), read ahead of the moments
                    unsigned long long after = 1;
                    if (corr && lane < C)
                        after = tab.gv[bin] +
                                (!TREE ? (unsigned long long)((gg[bin] - g0[bin]) / lnf)
                                       : tab.holds(bin) ? (unsigned long long)tab.n[bin & (tab.size - 1)] : 0ull);
                    // Moments: short chunks leave lanes for two groups of them at once.  Moments and
                    // correlators are FP64's latency: 12 steps of L = 12, 4300 -> 2200 cycles beside the 3400
                    // of their decisions, with a transform in one chunk of six (1100 cycles; a lane alone 2500).
                    const int per = Model::kGroups > 1 && C <= 16 ? 16 : 32;
                    const int step = lane & (per - 1);
                    if (step < C) {
                        int32_t Mv[3] = {0, 0, 0};
                        for (int m = 0; m < NM; ++m) Mv[m] = M[m] + dm(m, step);
                        double* o = ob + (size_t)((unsigned)st->seq[step] * (unsigned)P.obs_stride);
                        for (int g = lane / per; g < Model::kGroups; g += 32 / per)
                            Model::add_group(o, g, Mv, invN, invN * invN, P.corr);
                    }
                    if (corr) {
                        // steps whose bin count before the visit is a multiple of 1000: the count after
                        // the chunk less the chunk's visits from the step on
                        const int last = mod_transform(after - 1);
                        if (__any_sync(kFull, lane < C && last < C)) {
                            const unsigned grp = __match_any_sync(kFull, bin);
                            unsigned todo = __ballot_sync(kFull, lane < C && last == __popc(grp >> lane) - 1);
                            const int cp = lane / 4 % NC, m = Model::corr_mag(cp);
                            unsigned up = 0;
                            for (int k = 0; k < NM; ++k)
                                if (k == m) up = plus[k];
                            for (; todo != 0; todo &= todo - 1) {
                                const int j = __ffs((int)todo) - 1;
                                // a correlator plane changes where its magnetisation's terms do
                                const unsigned flips = changes(m) ? acc & (0xFFFFFFFFu >> (31 - j)) : 0u;
                                const double g = plane_power<32, NC>(sums + 2 * L * cp, sums + 2 * L * cp + L,
                                                                     P.qfix + I.qtab_off, L, y, x0, flips, up, lane);
                                double G[NC];
                                for (int k = 0; k < NC; ++k) G[k] = __shfl_sync(kFull, g, 4 * k);
                                if (lane == j)
                                    Model::add_transforms(ob + (size_t)bin * P.obs_stride, G, 0.5 * invN * invN);
                            }
                        }
                        __syncwarp();
                        // the chunk's flips into the sums
                        for (int cp = 0; cp < NC; ++cp) {
                            const int m = Model::corr_mag(cp);
                            if (!changes(m)) continue;
                            if (lane < C && ((acc >> lane) & 1u))
                                red_shared_add((unsigned)__cvta_generic_to_shared(sums + 2 * L * cp + L + x0 + lane), -2 * sg[m]);
                            if (lane == 0) red_shared_add((unsigned)__cvta_generic_to_shared(sums + 2 * L * cp + y), total[m]);
                        }
                    }
                }
                if (lane < C && ((acc >> lane) & 1u)) A[c0 + lane] = (int8_t)(-ai);
                if (OBS)
                    for (int m = 0; m < NM; ++m) M[m] += total[m];
                __syncwarp();
                attempt += (uint64_t)C;
                c0 += C;
                cc = cn; y = yn; C = Cn;
            }
            if (NP == 2) flavour ^= 1;
        }
    }
    for (int i = lane; i < NP * N; i += 32) gl[i] = sp[i];
    int sum[NM];
    for (int m = 0; m < NM; ++m) sum[m] = 0;
    for (int i = lane; i < N; i += 32) {
        int t[NM];
        Model::mag_terms(sp, N, i, t);
        for (int m = 0; m < NM; ++m) sum[m] += t[m];
    }
    for (int m = 0; m < NM; ++m) M[m] = __reduce_add_sync(kFull, sum[m]);
    __syncwarp();
    if (!TREE) {
        for (int k = lane; k < nb; k += 32) {
            const long long gnew = gg[k], dg = gnew - g0[k];
            if (dg != 0) tab.err |= commit_visits(tab.gH, tab.gv, k, dg / lnf, gnew);
        }
    } else {
        tab.book(tab.lo, min(tab.lo + tab.size, nb), lane);
    }
    if (tab.err) atomicOr(&P.counters[0], tab.err);
    if (lane == 0) {
        vr = TREE ? ((long long)b0 << sh) + ((long long)fr << zeros) + below : c.v;
        P.cfg_E[cfg] = eglo + (vr + vlo) / mul;
        for (int m = 0; m < NM; ++m) P.cfg_M[3 * cfg + m] = M[m];
        P.slot_sweeps[s] = sweeps0 + (uint64_t)p.nsweeps;
        if (NP == 2) P.slot_flavour[s] = flavour;
        if (REPLAY) P.slot_draws[s] = c.draws;
        if (c.err) atomicOr(&P.counters[0], c.err);
    }
}

template <class Model, int MODE, bool OBS>
__global__ void __launch_bounds__(256, 2) k_sweep_tables(const SweepParams p)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int wib = threadIdx.x >> 5;
    sweep_tables_warp<Model, MODE, OBS>(p, blockIdx.x * (blockDim.x >> 5) + wib, smem + (size_t)wib * p.smem_per_warp);
}

// --------------------------------------------------------------------------
// One persistent, work-stealing launch for every launch group of a batch
// (rewl_batch_desc.persistent): a grid sized to the resident capacity, each warp
// taking the next walker from a device counter until all walkers of the sweep phase
// are done.  A task is one walker (one walker per warp); tasks are ordered by
// expected cost, the Ashkin-Teller walkers and the largest lattices first.  Each
// kind of group runs its own kernel's per-warp function, not inlined here, so the
// fused kernel's registers are those of its dispatch loop plus the largest callee.
// --------------------------------------------------------------------------
enum FusedKind : int {
    kFusedBins = 0, kFusedTablesIsing = 1, kFusedTablesAT = 2
};
constexpr int kMaxFusedGroups = 16;

struct FusedGroup {
    const int32_t* slots;
    int nslots, smem_per_warp, nbcap, kind, first_task, counts, moments, cache;
};

struct FusedParams {
    DevPtrs P;
    int nsweeps, ngroups, ntasks, slot_bytes;
    unsigned int* counter;
    FusedGroup g[kMaxFusedGroups];
};

template <bool OBS>
__device__ __noinline__ void fused_bins(const SweepParams& p, int unit, unsigned char* base)
{
    if (p.counts) sweep_bins_warp<1, OBS, true>(p, unit, base);
    else sweep_bins_warp<1, OBS, false>(p, unit, base);
}

template <class Model, bool OBS>
__device__ __noinline__ void fused_tables(const SweepParams& p, int unit, unsigned char* base)
{
    if (p.cache) sweep_tables_warp<Model, kTableTree, OBS>(p, unit, base);
    else sweep_tables_warp<Model, kTableSerial, OBS>(p, unit, base);
}

// (three blocks an SM: without saying so the compiler settles at 128 registers and spills, 5 % slower on Ising L = 32)
template <bool OBS>
__global__ void __launch_bounds__(128, 3) k_sweep_fused(const FusedParams fp)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    unsigned char* base = smem + (size_t)wib * fp.slot_bytes;
    for (;;) {
        int t = 0;
        if (lane == 0) t = (int)atomicAdd(fp.counter, 1u);
        t = __shfl_sync(kFull, t, 0);
        if (t >= fp.ntasks) break;
        int gi = 0;
        while (gi + 1 < fp.ngroups && t >= fp.g[gi + 1].first_task) ++gi;
        const FusedGroup& G = fp.g[gi];
        SweepParams sp;
        sp.P = fp.P; sp.slots = G.slots; sp.nslots = G.nslots; sp.nsweeps = fp.nsweeps;
        sp.smem_per_warp = G.smem_per_warp; sp.nbcap = G.nbcap; sp.counts = G.counts; sp.moments = G.moments; sp.cache = G.cache;
        const int unit = t - G.first_task;
        switch (G.kind) {
        case kFusedBins: fused_bins<OBS>(sp, unit, base); break;
        case kFusedTablesIsing: fused_tables<Ising2dModel, OBS>(sp, unit, base); break;
        default: fused_tables<AshkinTeller2dModel, OBS>(sp, unit, base); break;
        }
        __syncwarp();
    }
}

// --------------------------------------------------------------------------
// Replica exchange: one thread per (instance, lower window) pair of the round
// --------------------------------------------------------------------------
__device__ inline int64_t slot_local_bin(const DevPtrs& P, const InstDev& I, int slot, int64_t E)
{
    const WinDev& W = P.win[P.slot_win[slot]];
    return global_bin(I, E) - W.gblo;
}

__device__ inline void touch(const DevPtrs& P, const InstDev& I, int slot)
{
    const int c = P.slot_cfg[slot];
    const int64_t b = slot_local_bin(P, I, slot, P.cfg_E[c]);
    const int w = P.slot_win[slot];
    if (b < 0 || b >= P.slot_nb[slot]) { atomicOr(&P.counters[0], ERR_BOUNDS); return; }
    const int64_t o = P.slot_tab[slot] + b;
    const long long gnew = P.g[o] + P.win_lnf[w];
    P.g[o] = gnew;
    if (P.H[o] == 0xFFFFFFFFu) atomicOr(&P.counters[0], ERR_COUNT);   // saturated, as in commit_visits
    else P.H[o] += 1u;
    if (gnew >= kLogdosLimit) atomicOr(&P.counters[0], ERR_RANGE);
    const uint64_t seen = P.visits[o];         // the bin's count before this visit
    P.visits[o] = seen + 1u;
    if (P.obs) {
        double* ob = P.obs + (size_t)o * P.obs_stride;
        const double invN = 1.0 / (double)I.N;
        const int32_t* Mc = P.cfg_M + 3 * c;
        const bool due = P.corr && seen % kCountsPerTransform == 0;
        const double* q = P.qtab + I.qtab_off;
        const int8_t* sp = P.spins + P.cfg_off[c];
        if (I.model == REWL_MODEL_ISING2D) {
            Ising2dModel::add_observables(ob, Mc, invN, P.corr);
            if (due) Ising2dModel::add_correlators(ob, sp, I.N, I.L, q, invN * invN);
        } else {
            AshkinTeller2dModel::add_observables(ob, Mc, invN, P.corr);
            if (due) AshkinTeller2dModel::add_correlators(ob, sp, I.N, I.L, q, invN * invN);
        }
    }
}

__device__ void exchange_pair(const DevPtrs& P, const int32_t* pairs, int k, uint64_t round)
{
    const int ii = pairs[2 * k], lw = pairs[2 * k + 1];
    const InstDev I = P.inst[ii];
    const int R = I.R;
    int perm[kMaxReplicas];
    for (int r = 0; r < R; ++r) perm[r] = r;
    // keyed by the instance's own seed only, like its sweeps: an instance's trajectory does not
    // depend on the other instances of the batch or on its position among them
    const uint32_t xuid = 0x80000000u;
    const uint32_t w3 = (uint32_t)((round << 8) ^ (uint64_t)lw);
    for (int i = R - 1; i >= 1; --i) {
        const uint32_t word = philox_word(I.seed, xuid, (uint64_t)(R - 1 - i), kStreamExchange, w3);
        const int j = (int)mulhi32(word, (uint32_t)(i + 1));
        const int t = perm[i]; perm[i] = perm[j]; perm[j] = t;
    }
    unsigned long long att = 0, accn = 0;
    for (int r = 0; r < R; ++r) {
        const int lo = I.first_slot + lw * R + r;
        const int hi = I.first_slot + (lw + 1) * R + perm[r];
        const int cl = P.slot_cfg[lo], ch = P.slot_cfg[hi];
        const int64_t El = P.cfg_E[cl], Eh = P.cfg_E[ch];
        const int64_t bl_l = slot_local_bin(P, I, lo, El), bl_h = slot_local_bin(P, I, lo, Eh);
        const int64_t bh_l = slot_local_bin(P, I, hi, El), bh_h = slot_local_bin(P, I, hi, Eh);
        ++att;
        bool accept = false;
        if (bl_l < 0 || bl_l >= P.slot_nb[lo] || bh_h < 0 || bh_h >= P.slot_nb[hi]) {
            atomicOr(&P.counters[0], ERR_BOUNDS);    // a walker outside its own window: skip the pair
            continue;
        }
        if (bl_h >= 0 && bl_h < P.slot_nb[lo] && bh_l >= 0 && bh_l < P.slot_nb[hi]) {
            const int64_t* gl = P.g + P.slot_tab[lo];
            const int64_t* gh = P.g + P.slot_tab[hi];
            const int64_t a = gl[bl_h] - gl[bl_l];
            const int64_t c = gh[bh_l] - gh[bh_h];
            const int64_t d = (a > 0 ? a : 0) + (c > 0 ? c : 0);
            // acceptance words follow the R - 1 pairing words: counter 32 + r while R <= 32, 64 + r above
            const uint32_t word = philox_word(I.seed, xuid, (uint64_t)((R <= 32 ? 32 : 64) + r), kStreamExchange, w3);
            accept = d < accept_threshold(neglog_u32(word));
        }
        if (accept) { P.slot_cfg[lo] = ch; P.slot_cfg[hi] = cl; ++accn; }
        touch(P, I, lo);
        touch(P, I, hi);
    }
    atomicAdd(&P.stats[0], att);
    atomicAdd(&P.stats[1], accn);
}

// One exchange round: one thread per (instance, lower window) pair of the round's direction.
// The round counter lives on the device (so that a captured cycle replays correctly): every
// thread reads it first, and the last block to finish advances it.
__global__ void k_exchange(DevPtrs P, const int32_t* pairs0, int n0, const int32_t* pairs1, int n1)
{
    __shared__ bool last;
    const uint64_t round = *(volatile unsigned long long*)P.xround;
    const int dir = (int)(round & 1u);
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    // after a device error no pair moves; the round still advances with the host's mirror
    if (k < (dir ? n1 : n0) && !engine_failed(P.counters)) exchange_pair(P, dir ? pairs1 : pairs0, k, round);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(&P.xround[1], 1ull) == (unsigned long long)(gridDim.x - 1);
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        P.xround[1] = 0;
        P.xround[0] = round + 1;
    }
}

// --------------------------------------------------------------------------
// Flatness, averaging, reset, ln f: one block per window
// --------------------------------------------------------------------------
struct FlatParams {
    DevPtrs P;
    int nwin_total;
    int flat_mode;
    int mask_mode;
    int one_over_t;
    int reduce;
    uint64_t flat_num, flat_den;   // min * n * den >= num * sum
    float flat_param_f;
    double lnf_final;
    uint64_t sweeps_since_check;
};

struct OpMin { __device__ unsigned long long operator()(unsigned long long a, unsigned long long b) const { return a < b ? a : b; } };
struct OpMax { __device__ unsigned long long operator()(unsigned long long a, unsigned long long b) const { return a > b ? a : b; } };
struct OpAdd { __device__ unsigned long long operator()(unsigned long long a, unsigned long long b) const { return a + b; } };

template <typename T, typename Op>
__device__ T block_reduce(T v, Op op, T* sh, T identity)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_down_sync(kFull, v, o));
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    if (wid == 0) {
        v = lane < nw ? sh[lane] : identity;
        for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_down_sync(kFull, v, o));
        if (lane == 0) sh[0] = v;
    }
    __syncthreads();
    const T r = sh[0];
    __syncthreads();
    return r;
}

__device__ inline bool bin_valid(const DevPtrs& P, const WinDev& W, int first_slot_of_win, int R, int b, int mask_mode)
{
    if (!P.mask[W.mask_off + b]) return false;
    if (mask_mode == REWL_MASK_VISITED) {
        for (int r = 0; r < R; ++r)
            if (P.visits[P.slot_tab[first_slot_of_win + r] + b]) return true;
        return false;
    }
    return true;
}

__global__ void __launch_bounds__(256) k_flat(const FlatParams fp)
{
    __shared__ unsigned long long red_u[32];
    __shared__ int flat_sh, stop_sh;
    __shared__ long long g0_sh[kMaxReplicas];
    const DevPtrs& P = fp.P;
    const int w = blockIdx.x;
    const WinDev W = P.win[w];
    const InstDev I = P.inst[W.inst];
    const int R = I.R;
    const int first = I.first_slot + W.local * R;
    const int nb = W.nb;

    if (threadIdx.x == 0) {
        stop_sh = engine_failed(P.counters);
        if (!stop_sh) P.win_sweepctr[w] += fp.sweeps_since_check;
        flat_sh = 1;
    }
    __syncthreads();
    if (stop_sh) return;

    for (int r = 0; r < R; ++r) {
        const uint32_t* H = P.H + P.slot_tab[first + r];
        const int64_t* g = P.g + P.slot_tab[first + r];
        unsigned long long mn = ~0ull, mx = 0, sum = 0, n = 0, zero = 0, big = 0;
        for (int b = threadIdx.x; b < nb; b += blockDim.x) {
            // a window that never goes flat (a replica trapped away from part of its
            // range) lets ln g grow without bound: report it before int64 overflows
            big |= (unsigned long long)(g[b] >= kLogdosLimit || g[b] <= -kLogdosLimit);
            if (!bin_valid(P, W, first, R, b, fp.mask_mode)) continue;
            const unsigned long long h = H[b];
            mn = h < mn ? h : mn; mx = h > mx ? h : mx; sum += h; ++n; zero += (h == 0);
        }
        mn = block_reduce(mn, OpMin(), red_u, ~0ull);
        mx = block_reduce(mx, OpMax(), red_u, 0ull);
        sum = block_reduce(sum, OpAdd(), red_u, 0ull);
        n = block_reduce(n, OpAdd(), red_u, 0ull);
        zero = block_reduce(zero, OpAdd(), red_u, 0ull);
        big = block_reduce(big, OpMax(), red_u, 0ull);
        if (threadIdx.x == 0) {
            if (big) { atomicOr(&P.counters[0], ERR_RANGE); flat_sh = 0; }   // no averaging or reset
            bool f;
            if (fp.flat_mode == REWL_FLAT_ALL_VISITED) f = P.win_oot[w] ? true : (zero == 0);
            else if (n == 0 || mn == 0) f = false;
            else if (fp.flat_mode == REWL_FLAT_MAX_MIN_RATIO)
                f = __fdiv_rn(__ull2float_rn(mx - mn), __ull2float_rn(mn)) <= fp.flat_param_f;
            else
                f = (unsigned __int128)mn * n * fp.flat_den >= (unsigned __int128)fp.flat_num * sum;
            if (!f) flat_sh = 0;
        }
        __syncthreads();
    }
    if (!flat_sh) return;

    // count-weighted average of the replicas' logDoS (rewl_simulation.hpp:361-454)
    if (R > 1) {
        const double inv = 1.0 / kLogdosScale;
        for (int b = threadIdx.x; b < nb; b += blockDim.x) {
            unsigned long long tot = 0;
            for (int r = 0; r < R; ++r) tot += P.H[P.slot_tab[first + r] + b];
            long long avg;
            if (tot == 0) avg = P.g[P.slot_tab[first] + b];
            else {
                double acc = 0.0;
                const double dtot = __ull2double_rn(tot);
                for (int r = 0; r < R; ++r) {
                    const int64_t o = P.slot_tab[first + r] + b;
                    const double wt = __ddiv_rn(__uint2double_rn(P.H[o]), dtot);
                    const double gr = __dmul_rn(__ll2double_rn(P.g[o]), inv);
                    acc = __dadd_rn(acc, __dmul_rn(wt, gr));
                }
                avg = __double2ll_rn(__dmul_rn(acc, kLogdosScale));
            }
            for (int r = 0; r < R; ++r) P.g[P.slot_tab[first + r] + b] = avg;
        }
        __syncthreads();
    }
    if (threadIdx.x < R) g0_sh[threadIdx.x] = P.g[P.slot_tab[first + threadIdx.x]];
    __syncthreads();
    for (int r = 0; r < R; ++r) {
        const int64_t o = P.slot_tab[first + r];
        const long long red = fp.reduce ? g0_sh[r] : 0;
        for (int b = threadIdx.x; b < nb; b += blockDim.x) { P.H[o + b] = 0; P.g[o + b] -= red; }
    }
    if (threadIdx.x == 0) {
        const uint64_t t = P.win_sweepctr[w] * P.win_iter[w];
        long long lnf = P.win_lnf[w];
        int oot = P.win_oot[w];
        if (fp.one_over_t && !oot && t > 0 && __ll2double_rn(lnf) <= __ddiv_rn(kLogdosScale, __ull2double_rn(t))) oot = 1;
        if (oot && t > 0) lnf = (long long)((((unsigned long long)1 << kLogdosBits) + t / 2) / t);
        else lnf = lnf >> 1;
        if (lnf < 1) lnf = 1;                  // the 2^-36 grid's smallest increment
        P.win_lnf[w] = lnf;
        P.win_oot[w] = oot;
        P.win_done[w] = (__ll2double_rn(lnf) / kLogdosScale) < fp.lnf_final ? 1 : 0;
        P.win_iter[w] += 1;
        P.win_sweepctr[w] = 0;
        atomicAdd(&P.counters[1], 1);
    }
}

// What the host reads after a check interval, in one go.
struct Report {
    unsigned long long stats[2];   // exchanges attempted, accepted
    int32_t counters[2];           // error word, flat events of the last check
    int32_t windows_done;
};

// (one block) into host memory
__global__ void k_report(DevPtrs P, int nwin, Report* out)
{
    __shared__ int done;
    if (threadIdx.x == 0) done = 0;
    __syncthreads();
    int n = 0;
    for (int w = threadIdx.x; w < nwin; w += blockDim.x) n += P.win_done[w];
    if (n) atomicAdd(&done, n);
    __syncthreads();
    if (threadIdx.x == 0) *out = Report{{P.stats[0], P.stats[1]}, {P.counters[0], P.counters[1]}, done};
}

// Observable columns of a model, before the count column: Ising |m|, m^2, m^4 (+ G(q_min));
// Ashkin-Teller 12 moments (+ a G(q_min) after each group of three).
__host__ __device__ inline int obs_columns(int model, bool corr) { return model == REWL_MODEL_ISING2D ? (corr ? 4 : 3) : (corr ? 16 : 12); }
__host__ __device__ inline bool is_corr_column(int model, bool corr, int k) { return corr && (model == REWL_MODEL_ISING2D ? k == 3 : (k & 3) == 3); }

// Rows b0 .. b0 + rows - 1 of [nb][K + 1]: K averages and the update count, from the sums of slots
// first .. first + count - 1, into host memory (a thread per entry).  Moments: sum over the slots /
// total count (the count-weighted mean of the replicas' running means).  G(q_min): each slot's sum
// over its transforms, ceil(count / 1000) of them, weighted by the slot's count in the same way.
__global__ void k_export_observables(DevPtrs P, int model, int first, int count, int b0, int rows, double* out)
{
    const int K = obs_columns(model, P.corr != 0);
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)rows * (K + 1)) return;
    const int b = b0 + (int)(i / (K + 1)), k = (int)(i % (K + 1));
    const bool transform = is_corr_column(model, P.corr != 0, k);
    double sum = 0.0;
    unsigned long long cnt = 0;
    for (int s = first; s < first + count; ++s) {
        const int64_t o = P.slot_tab[s] + b;
        const unsigned long long v = P.visits[o];
        cnt += v;
        if (k == K || (transform && !v)) continue;
        const double x = P.obs[(size_t)o * P.obs_stride + k];
        if (!transform) { sum = __dadd_rn(sum, x); continue; }
        const double mean = x / (double)((v + kCountsPerTransform - 1) / kCountsPerTransform);
        sum = __dadd_rn(sum, count == 1 ? mean : __dmul_rn((double)v, mean));
    }
    out[i] = k == K ? (double)cnt : !cnt ? 0.0 : (count == 1 && transform) ? sum : sum / (double)cnt;
}

// A window's logDoS, the replicas weighted by their visits, into host memory.
__global__ void k_export_logdos(DevPtrs P, int first, int count, int b0, int rows, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows) return;
    const int b = b0 + i;
    double total = 0.0, acc = 0.0;
    for (int s = first; s < first + count; ++s) total = __dadd_rn(total, (double)P.visits[P.slot_tab[s] + b]);
    if (total == 0.0 || count == 1) acc = (double)P.g[P.slot_tab[first] + b] / kLogdosScale;
    else
        for (int s = first; s < first + count; ++s) {
            const int64_t o = P.slot_tab[s] + b;
            acc = __dadd_rn(acc, __dmul_rn((double)P.visits[o] / total, (double)P.g[o] / kLogdosScale));
        }
    out[i] = acc;
}

__global__ void k_reset_window(DevPtrs P, int w, int reduce)
{
    const WinDev W = P.win[w];
    const InstDev I = P.inst[W.inst];
    const int first = I.first_slot + W.local * I.R;
    for (int r = 0; r < I.R; ++r) {
        const int64_t o = P.slot_tab[first + r];
        const long long g0 = P.g[o];
        __syncthreads();
        for (int b = threadIdx.x; b < W.nb; b += blockDim.x) { P.H[o + b] = 0; if (reduce) P.g[o + b] -= g0; }
        __syncthreads();
    }
}

// --------------------------------------------------------------------------
// Host side
// --------------------------------------------------------------------------
template <typename T>
struct DBuf {
    T* p = nullptr;
    size_t n = 0;
    int alloc(size_t count)
    {
        n = count;
        if (count == 0) return REWL_OK;
        if (cudaMalloc(&p, count * sizeof(T)) != cudaSuccess) return fail(REWL_ENOMEM, "cudaMalloc of %zu bytes failed", count * sizeof(T));
        return REWL_OK;
    }
    void free_()
    {
        if (p) cudaFree(p);
        p = nullptr; n = 0;
    }
};

struct HostInst {
    rewl_instance_desc d;
    InstDev dev;
    std::vector<double> fields;     // quantised
    double bw;
    std::vector<WinDev> wins;
    std::vector<double> wmin, wmax;
};

struct Launch {
    int model;
    std::vector<int32_t> slots;
    int smem_per_warp = 0;  // per walker for the bin-tracking kernel, per warp otherwise
    int nbcap = 0;
    int wpb = 1;            // warps per block
    int bins = 0;           // Ising bin-tracking kernel with `walkers_per_warp` walkers per warp
    int walkers_per_warp = 1;
    int counts = 0;         // bin-tracking kernel: visit counts beside g in shared memory (16 bytes per bin)
    int moments = 0;        // bin-tracking kernel with observables: moment sums in shared memory
    int crowded = 0;        // bin-tracking kernel with observables: the form of 168 registers
    int rows = 0;           // k_sweep_ising_rows in its place: sites of a row
    int maxL = 0;
    int tree = 0;           // the global-table kernel may decide on the tree of outcomes
    int tables = 0;         // the global-table kernel (k_sweep_tables)
    int cache = 0;          // its bins of each walker's table in shared memory (a power of two); 0: the serial chain
    int carveout = -1;      // global-table kernel: shared-memory carveout (percent) that leaves the rest to L1
    DBuf<int32_t> d_slots;
};

template <class Model>
SweepKernel table_kernel_t(int mode, bool obs)
{
    if (mode == kTableTree) return obs ? k_sweep_tables<Model, kTableTree, true> : k_sweep_tables<Model, kTableTree, false>;
    if (mode == kTableReplay) return obs ? k_sweep_tables<Model, kTableReplay, true> : k_sweep_tables<Model, kTableReplay, false>;
    return obs ? k_sweep_tables<Model, kTableSerial, true> : k_sweep_tables<Model, kTableSerial, false>;
}

SweepKernel table_kernel(int model, int mode, bool obs)
{
    return model == REWL_MODEL_ISING2D ? table_kernel_t<Ising2dModel>(mode, obs)
                                       : table_kernel_t<AshkinTeller2dModel>(mode, obs);
}

} // namespace

struct rewl_engine {
    rewl_batch_desc desc;
    std::vector<HostInst> inst;
    int nslots = 0, nwin_total = 0;
    std::vector<int32_t> h_slot_inst, h_slot_win, h_slot_nb;
    std::vector<int64_t> h_slot_tab;
    std::vector<int64_t> h_cfg_off;
    std::vector<WinDev> h_wins;
    int64_t table_total = 0, spin_total = 0, mask_total = 0;
    std::vector<int32_t> pairs_dir[2];
    int direction = 0;
    uint64_t exch_round = 0;
    uint64_t sweeps_since_check = 0;
    int64_t sweeps_total = 0, cycles = 0, flat_events = 0, flips_total = 0;
    int64_t flips_per_sweep = 0;
    // sweep launches are split so that one launch adds at most kLaunchGrowth to a bin: an upper
    // bound of every window's ln f (2^-36 units; k_flat only lowers it, except the 1/t rule,
    // which never exceeds 1) and the largest number of degrees of freedom of a walker
    int64_t lnf_bound_u = 0, ndof_max = 0;
    // rewl_batch_desc.persistent: every launch group in one work-stealing launch (k_sweep_fused)
    bool fused = false;
    FusedParams fused_p{};
    int fused_grid = 0, fused_block = 128;
    size_t fused_smem = 0;
    DBuf<unsigned int> fused_counter;
    cudaStream_t stream = nullptr;
    std::vector<Launch> launches;
    std::vector<cudaEvent_t> ev_pool;
    size_t ev_used = 0;
    // one check interval captured as a CUDA graph (rewl_batch_desc.graphs): the host counters it
    // advances per replay, and the timing events recorded inside it
    cudaGraphExec_t cycle_exec = nullptr;
    bool capturing = false;
    int64_t g_sweeps = 0, g_flips = 0, g_launches = 0, g_kernel_launches = 0, g_rounds = 0;
    std::vector<cudaEvent_t> g_events;
    double graph_sweep_ms = 0;          // sweep-phase time of replayed graphs since the last timing read
    bool tuned = false;
    int64_t kernel_launches = 0;        // sweep-kernel launches since the last timing read
    int64_t launches_total = 0;         // every engine kernel since creation
    int sweep_variant = 3;              // REWL_SWEEP_VARIANT: 3 all-lane Ising resolver (default), 2 lane-0, 4 global tables

    DBuf<InstDev> d_inst;
    DBuf<WinDev> d_win;
    DBuf<int32_t> slot_inst, slot_win, slot_cfg, slot_nb, slot_flavour, pairs[2];
    DBuf<int64_t> slot_tab, slot_draws, slot_thr_off, slot_thr_n, cfg_off, cfg_E, fields, g, win_lnf;
    DBuf<uint64_t> slot_sweeps, visits, win_iter, win_sweepctr;
    DBuf<int8_t> spins;
    DBuf<int32_t> cfg_M, win_done, win_oot, counters;
    DBuf<uint32_t> H;
    DBuf<uint8_t> mask;
    DBuf<unsigned long long> stats;
    DBuf<int64_t> thr;
    DBuf<double> obs;           // per-bin observable sums (observables on)
    DBuf<int64_t> gsnap;        // global-table serial chain: logDoS copy taken by each sweep launch
    DBuf<double> qtab;          // correlator kernels (observables == 2)
    DBuf<int2> qfix;
    DBuf<unsigned long long> xround;   // exchange round and the exchange kernel's done-block count
    std::vector<cudaStream_t> gstreams; // one per launch group when there are several (they run concurrently)
    cudaEvent_t fork_ev = nullptr;
    std::vector<cudaEvent_t> join_ev;
    int obs_stride = 0;
    std::vector<int64_t> h_thr_off, h_thr_n;
    std::vector<int64_t> h_fields;
    std::vector<uint8_t> h_mask;
    std::vector<double> h_qtab;
    std::vector<int2> h_qfix;

    DevPtrs ptrs() const
    {
        DevPtrs P;
        P.inst = d_inst.p; P.win = d_win.p;
        P.slot_inst = slot_inst.p; P.slot_win = slot_win.p; P.slot_cfg = slot_cfg.p; P.slot_tab = slot_tab.p;
        P.slot_nb = slot_nb.p; P.slot_flavour = slot_flavour.p; P.slot_sweeps = slot_sweeps.p;
        P.slot_draws = slot_draws.p; P.slot_thr_off = slot_thr_off.p; P.slot_thr_n = slot_thr_n.p; P.thr = thr.p;
        P.cfg_off = cfg_off.p; P.spins = spins.p; P.cfg_E = cfg_E.p; P.cfg_M = cfg_M.p; P.fields = fields.p;
        P.g = g.p; P.gsnap = gsnap.p; P.H = H.p; P.visits = visits.p; P.mask = mask.p;
        P.win_lnf = win_lnf.p; P.win_done = win_done.p; P.win_oot = win_oot.p; P.win_iter = win_iter.p;
        P.win_sweepctr = win_sweepctr.p; P.pairs = nullptr; P.counters = counters.p; P.stats = stats.p;
        P.xround = xround.p;
        P.obs = obs.p; P.obs_stride = obs_stride;
        P.corr = desc.observables == 2 ? 1 : 0; P.qtab = qtab.p; P.qfix = qfix.p;
        return P;
    }

    void drop_graph()
    {
        if (cycle_exec) cudaGraphExecDestroy(cycle_exec);
        cycle_exec = nullptr;
        for (auto ev : g_events) cudaEventDestroy(ev);
        g_events.clear();
    }

    // pinned host memory that kernels write results to: a Report, then rows of an export
    static constexpr size_t kReportBytes = 256, kExportBytes = 4u << 20;
    char* pinned = nullptr;
    size_t export_doubles = 0;
    std::mutex export_mu;

    void release()
    {
        if (pinned) cudaFreeHost(pinned);
        pinned = nullptr;
        d_inst.free_(); d_win.free_();
        slot_inst.free_(); slot_win.free_(); slot_cfg.free_(); slot_nb.free_(); slot_flavour.free_();
        pairs[0].free_(); pairs[1].free_();
        obs.free_(); gsnap.free_(); qtab.free_(); qfix.free_(); xround.free_(); fused_counter.free_();
        for (cudaStream_t st : gstreams) cudaStreamDestroy(st);
        gstreams.clear();
        for (cudaEvent_t ev : join_ev) cudaEventDestroy(ev);
        join_ev.clear();
        if (fork_ev) { cudaEventDestroy(fork_ev); fork_ev = nullptr; }
        slot_tab.free_(); slot_draws.free_(); slot_thr_off.free_(); slot_thr_n.free_(); cfg_off.free_();
        cfg_E.free_(); fields.free_(); g.free_(); win_lnf.free_(); slot_sweeps.free_(); visits.free_();
        win_iter.free_(); win_sweepctr.free_(); spins.free_(); cfg_M.free_(); win_done.free_(); win_oot.free_();
        counters.free_(); H.free_(); mask.free_(); stats.free_(); thr.free_();
        for (auto& l : launches) l.d_slots.free_();
        for (auto e : ev_pool) cudaEventDestroy(e);
        ev_pool.clear();
        drop_graph();
        if (stream) cudaStreamDestroy(stream);
        stream = nullptr;
    }
};

namespace {

bool is_pow2_multiple(double v, int escale, int& shift)
{
    const double u = std::ldexp(v, escale);
    if (u < 1.0 || u != std::floor(u)) return false;
    const long long x = (long long)u;
    if (x & (x - 1)) return false;
    shift = 0;
    while ((1LL << shift) < x) ++shift;
    return true;
}

int largest_chunk(int L)
{
    for (int c = std::min(L, 32); c >= 1; --c)
        if (L % c == 0) return c;
    return 1;
}

// glazier::construct_windows, EQUAL_WINDOWS branch (src/REWL/glazier.hpp:305-351),
// carried out in units of bins: window k starts at the previous window's start
// plus the whole bins up to its nominal start, and spans the whole bins that
// cover its nominal width, clipped to the global range.  For integer widths
// this is the reference's arithmetic exactly; for fractional widths it avoids
// the bin the reference's double ceil/clip can lose.
int make_windows(const rewl_instance_desc& d, std::vector<double>& mins, std::vector<double>& maxs,
                 std::vector<int64_t>& gblo, std::vector<int>& nbins)
{
    const int nw = d.num_windows;
    const double gmin = d.energy_min, gmax = d.energy_max, bw = d.bin_width, ov = d.window_overlap;
    mins.assign(nw, 0); maxs.assign(nw, 0); gblo.assign(nw, 0); nbins.assign(nw, 0);
    const double span = (gmax - gmin) / bw;
    const int64_t G = (int64_t)std::llround(span);
    if (std::fabs(span - (double)G) > 1e-6 * std::max(1.0, span) || G < 1) return -1;
    const double denom = 1 + (nw - 1) * (1 - ov);
    const double size = (gmax - gmin) / denom;
    const double eps = 1e-9;
    for (int k = 0; k < nw; ++k) {
        const double raw_min = gmin + (double)k * (1 - ov) * size;
        const double raw_max = raw_min + size;
        int64_t lo = 0;
        if (k != 0) lo = gblo[k - 1] + (int64_t)std::floor((raw_min - mins[k - 1]) / bw + eps);
        const double wmin = gmin + bw * (double)lo;
        int64_t hi = lo + (int64_t)std::ceil((raw_max - wmin) / bw - eps);
        if (hi > G) hi = G;
        gblo[k] = lo;
        nbins[k] = (int)(hi - lo);
        mins[k] = wmin;
        maxs[k] = gmin + bw * (double)hi;
    }
    return 0;
}

void static_mask(const rewl_instance_desc& d, double wmin, int nb, uint8_t* m)
{
    for (int b = 0; b < nb; ++b) m[b] = 1;
    if (d.model != REWL_MODEL_ISING2D) return;
    // Ising on an L x L torus: E = -2N + 4 and E = 2N - 4 never occur; all
    // energies are -2N + 4k (with J = 1; scaled by |J| in general).
    const double N = (double)d.L * d.L, J = std::fabs(d.J);
    for (int b = 0; b < nb; ++b) {
        const double lo = wmin + d.bin_width * b, hi = lo + d.bin_width;
        bool any = false;
        for (double e = std::ceil((lo + 2 * N * J) / (4 * J)) * 4 * J - 2 * N * J; e < hi; e += 4 * J) {
            if (e < -2 * N * J || e > 2 * N * J) continue;
            if (e == -2 * N * J + 4 * J || e == 2 * N * J - 4 * J) continue;
            any = true;
        }
        m[b] = any ? 1 : 0;
    }
}

template <typename T>
int upload(DBuf<T>& b, const std::vector<T>& v, cudaStream_t s)
{
    int rc = b.alloc(v.size());
    if (rc) return rc;
    if (!v.empty()) CUDA_TRY(cudaMemcpyAsync(b.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
    return REWL_OK;
}

int build_host(rewl_engine* e)
{
    const rewl_batch_desc& D = e->desc;
    if (D.num_instances < 1 || !D.instances) return fail(REWL_EINVAL, "no instances");
    if (D.sweeps_per_exchange < 1 || D.sweeps_per_check < D.sweeps_per_exchange || D.sweeps_per_check % D.sweeps_per_exchange)
        return fail(REWL_EINVAL, "sweeps_per_check must be a positive multiple of sweeps_per_exchange");
    if (!(D.lnf_initial > 0) || !(D.lnf_final > 0) || D.lnf_initial > 64)
        return fail(REWL_EINVAL, "ln f must be positive and the initial ln f at most 64");
    if (D.flatness_mode < 0 || D.flatness_mode > 2) return fail(REWL_EINVAL, "bad flatness mode");
    if (D.mask_mode < 0 || D.mask_mode > 1) return fail(REWL_EINVAL, "bad mask mode");
    if (D.rng_mode != REWL_RNG_PHILOX && D.rng_mode != REWL_RNG_REPLAY) return fail(REWL_EINVAL, "bad rng mode");
    if (D.warps_per_block != 0 && D.warps_per_block != 1 && D.warps_per_block != 2 && D.warps_per_block != 4 && D.warps_per_block != 8)
        return fail(REWL_EINVAL, "warps_per_block must be 0, 1, 2, 4 or 8");
    if (D.observables < 0 || D.observables > 2)
        return fail(REWL_EINVAL, "observables must be 0 (off), 1 (moments) or 2 (moments and G(q_min) correlators)");
    if (D.walkers_per_warp != 0 && D.walkers_per_warp != 1 && D.walkers_per_warp != 2 && D.walkers_per_warp != 4)
        return fail(REWL_EINVAL, "walkers_per_warp must be 0, 1, 2 or 4");
    if (D.persistent != 0 && D.persistent != 1) return fail(REWL_EINVAL, "persistent must be 0 or 1");
    if (D.persistent && D.rng_mode == REWL_RNG_REPLAY)
        return fail(REWL_EINVAL, "the persistent launch runs Philox streams only (rng_mode REWL_RNG_PHILOX)");
    if (D.persistent && D.walkers_per_warp > 1)
        return fail(REWL_EINVAL, "the persistent launch runs one walker per warp");
    int slot = 0, win = 0;
    int64_t tab = 0, spin = 0, maskoff = 0, fieldoff = 0;
    std::vector<int64_t> h_fields;
    std::vector<uint8_t> h_mask;
    std::vector<double> h_qtab;
    e->inst.resize(D.num_instances);
    for (int ii = 0; ii < D.num_instances; ++ii) {
        const rewl_instance_desc& d = D.instances[ii];
        HostInst& H = e->inst[ii];
        H.d = d;
        if (d.model != REWL_MODEL_ISING2D && d.model != REWL_MODEL_ASHKIN_TELLER2D) return fail(REWL_EINVAL, "instance %d: bad model", ii);
        if (d.L < 2 || d.L > 128) return fail(REWL_EINVAL, "instance %d: L must be in [2, 128]", ii);
        if (d.num_windows < 1 || d.replicas_per_window < 1 || d.replicas_per_window > kMaxReplicas)
            return fail(REWL_EINVAL, "instance %d: need >= 1 window and 1..%d replicas", ii, kMaxReplicas);
        if (!(d.window_overlap >= 0 && d.window_overlap < 1)) return fail(REWL_EINVAL, "instance %d: overlap must be in [0,1)", ii);
        if (!(d.energy_max > d.energy_min) || !(d.bin_width > 0)) return fail(REWL_EINVAL, "instance %d: bad energy range", ii);
        if (d.init_mode != 0 && d.init_mode != 1) return fail(REWL_EINVAL, "instance %d: bad init mode", ii);
        InstDev I{};
        I.model = d.model; I.L = d.L; I.N = d.L * d.L; I.ndof = d.model == REWL_MODEL_ISING2D ? I.N : 2 * I.N;
        I.nwin = d.num_windows; I.R = d.replicas_per_window; I.first_win = win; I.first_slot = slot;
        I.seed = instance_key(d.seed); I.chunk = largest_chunk(d.L); I.init_mode = d.init_mode;
        int shift = 0;
        if (d.model == REWL_MODEL_ISING2D) {
            if (d.J != std::floor(d.J) || d.J == 0 || std::fabs(d.J) > 1024) return fail(REWL_EINVAL, "instance %d: Ising J must be a non-zero integer", ii);
            if (d.fields) return fail(REWL_EINVAL, "instance %d: random fields are supported for the Ashkin-Teller model only", ii);
            I.escale = 0; I.J_u = (int64_t)d.J; I.K_u = 0;
            if (!is_pow2_multiple(d.bin_width, 0, shift)) return fail(REWL_EINVAL, "instance %d: Ising bin width must be a power of two >= 1", ii);
            I.bin_mul = 1; I.bin_shift = shift;
            if (d.energy_min != std::floor(d.energy_min)) return fail(REWL_EINVAL, "instance %d: energy_min must be an integer", ii);
            if (std::fabs(d.energy_min) + std::fabs(d.energy_max) > 1e8) return fail(REWL_EINVAL, "instance %d: energy range too large", ii);
        } else {
            I.escale = 20;
            const double Ju = std::ldexp(d.J, 20), Ku = std::ldexp(d.K, 20);
            if (Ju != std::floor(Ju) || Ku != std::floor(Ku)) return fail(REWL_EINVAL, "instance %d: J and K must be multiples of 2^-20", ii);
            I.J_u = (int64_t)Ju; I.K_u = (int64_t)Ku;
            const double inv = 1.0 / d.bin_width;
            if (is_pow2_multiple(d.bin_width, 20, shift)) { I.bin_mul = 1; I.bin_shift = shift; }
            else if (std::fabs(inv - std::nearbyint(inv)) < 1e-9 * inv && inv <= 4096) { I.bin_mul = (int64_t)std::llround(inv); I.bin_shift = 20; }
            else return fail(REWL_EINVAL, "instance %d: Ashkin-Teller bin width must be 1/n or a power of two", ii);
            const double emu = std::ldexp(d.energy_min, 20);
            if (emu != std::floor(emu)) return fail(REWL_EINVAL, "instance %d: energy_min must be a multiple of 2^-20", ii);
        }
        I.eglo_u = (int64_t)std::llround(std::ldexp(d.energy_min, I.escale));
        if (d.fields) {
            I.field_off = fieldoff;
            H.fields.resize(I.N);
            for (int i = 0; i < I.N; ++i) {
                const double q = std::nearbyint(std::ldexp(d.fields[i], 20));
                if (!std::isfinite(q) || std::fabs(q) > 1e15) return fail(REWL_EINVAL, "instance %d: bad field value", ii);
                H.fields[i] = std::ldexp(q, -20);
                h_fields.push_back((int64_t)q);
            }
            fieldoff += I.N;
        } else I.field_off = -1;
        if (D.observables == 2) {
            // Transform_Kernel (src/Hamiltonians/Correlations/fourier_correlator.hpp:14-42), from the
            // host's libm like the reference's own table
            I.qtab_off = (int64_t)h_qtab.size();
            const double qmin = 2. * std::acos(-1.) / static_cast<double>(d.L);
            for (int x = 0; x < d.L; ++x) h_qtab.push_back(std::cos(qmin * static_cast<double>(x)));
            for (int x = 0; x < d.L; ++x) h_qtab.push_back(std::sin(qmin * static_cast<double>(x)));
        } else I.qtab_off = -1;
        std::vector<double> mins, maxs; std::vector<int64_t> gblo; std::vector<int> nbins;
        if (make_windows(d, mins, maxs, gblo, nbins))
            return fail(REWL_EINVAL, "instance %d: the energy range is not a whole number of bins", ii);
        for (int k = 0; k < d.num_windows; ++k) {
            if (nbins[k] < 1) return fail(REWL_EINVAL, "instance %d: window %d is empty", ii, k);
            if (k > 0 && gblo[k] >= gblo[k - 1] + nbins[k - 1]) return fail(REWL_EINVAL, "instance %d: windows %d and %d do not overlap", ii, k - 1, k);
        }
        H.bw = d.bin_width;
        H.wmin = mins; H.wmax = maxs;
        for (int k = 0; k < d.num_windows; ++k) {
            WinDev W{};
            W.inst = ii; W.local = k; W.nb = nbins[k]; W.gblo = gblo[k]; W.mask_off = maskoff;
            W.elo_u = I.eglo_u + (I.bin_mul == 1 ? (gblo[k] << I.bin_shift) : 0);
            std::vector<uint8_t> m(nbins[k]);
            static_mask(d, mins[k], nbins[k], m.data());
            h_mask.insert(h_mask.end(), m.begin(), m.end());
            maskoff += nbins[k];
            H.wins.push_back(W);
            e->h_wins.push_back(W);
            for (int r = 0; r < d.replicas_per_window; ++r) {
                e->h_slot_inst.push_back(ii);
                e->h_slot_win.push_back(win + k);
                e->h_slot_nb.push_back(nbins[k]);
                e->h_slot_tab.push_back(tab);
                tab += nbins[k];
                e->h_cfg_off.push_back(spin);
                spin += I.ndof;
            }
        }
        if (d.model == REWL_MODEL_ISING2D) {
            // integer arithmetic in int32 inside the kernel
            const double emax_abs = 2.0 * I.N * std::fabs(d.J);
            if (emax_abs > 1e9 || std::fabs(d.energy_min) > 1e9 || std::fabs(d.energy_max) > 1e9)
                return fail(REWL_EINVAL, "instance %d: energies exceed int32", ii);
        }
        H.dev = I;
        slot += d.num_windows * d.replicas_per_window;
        win += d.num_windows;
        e->flips_per_sweep += (int64_t)d.num_windows * d.replicas_per_window * I.ndof;
        e->ndof_max = std::max<int64_t>(e->ndof_max, I.ndof);
    }
    e->lnf_bound_u = std::max<int64_t>(std::max<int64_t>(1, (int64_t)std::llround(D.lnf_initial * kLogdosScale)),
                                       D.one_over_t ? (int64_t)kLogdosScale : 0);
    e->nslots = slot; e->nwin_total = win;
    e->table_total = tab; e->spin_total = spin; e->mask_total = maskoff;
    // exchange pair lists
    for (int dir = 0; dir < 2; ++dir) {
        e->pairs_dir[dir].clear();
        for (int ii = 0; ii < D.num_instances; ++ii)
            for (int lw = dir; lw + 1 < D.instances[ii].num_windows; lw += 2) { e->pairs_dir[dir].push_back(ii); e->pairs_dir[dir].push_back(lw); }
    }
    e->h_fields = std::move(h_fields);
    for (const double c : h_qtab) {
        const double units = std::ldexp(c, 30), whole = std::nearbyint(units);
        e->h_qfix.push_back(make_int2((int)whole, (int)std::nearbyint(std::ldexp(units - whole, 30))));
    }
    e->h_qtab = std::move(h_qtab);
    e->h_mask = std::move(h_mask);
    return REWL_OK;
}

int upload_all(rewl_engine* e)
{
    const rewl_batch_desc& D = e->desc;
    const int slot = e->nslots, win = e->nwin_total;
    const int64_t tab = e->table_total, spin = e->spin_total;
    cudaStream_t s = e->stream;
    std::vector<InstDev> hinst;
    for (auto& H : e->inst) hinst.push_back(H.dev);
    int rc;
    if ((rc = upload(e->d_inst, hinst, s)) || (rc = upload(e->d_win, e->h_wins, s)) ||
        (rc = upload(e->slot_inst, e->h_slot_inst, s)) || (rc = upload(e->slot_win, e->h_slot_win, s)) ||
        (rc = upload(e->slot_nb, e->h_slot_nb, s)) || (rc = upload(e->slot_tab, e->h_slot_tab, s)) ||
        (rc = upload(e->cfg_off, e->h_cfg_off, s)) || (rc = upload(e->fields, e->h_fields, s)) ||
        (rc = upload(e->qtab, e->h_qtab, s)) || (rc = upload(e->qfix, e->h_qfix, s)) ||
        (rc = upload(e->mask, e->h_mask, s)) || (rc = upload(e->pairs[0], e->pairs_dir[0], s)) ||
        (rc = upload(e->pairs[1], e->pairs_dir[1], s)))
        return rc;
    std::vector<int32_t> cfg(slot);
    for (int i = 0; i < slot; ++i) cfg[i] = i;
    if ((rc = upload(e->slot_cfg, cfg, s))) return rc;
    if ((rc = e->slot_flavour.alloc(slot)) || (rc = e->slot_sweeps.alloc(slot)) || (rc = e->slot_draws.alloc(slot)) ||
        (rc = e->slot_thr_off.alloc(slot)) || (rc = e->slot_thr_n.alloc(slot)) || (rc = e->cfg_E.alloc(slot)) ||
        (rc = e->cfg_M.alloc(3 * (size_t)slot)) || (rc = e->spins.alloc(spin)) || (rc = e->g.alloc(tab)) ||
        (rc = e->H.alloc(tab)) || (rc = e->visits.alloc(tab)) || (rc = e->win_lnf.alloc(win)) ||
        (rc = e->win_done.alloc(win)) || (rc = e->win_oot.alloc(win)) || (rc = e->win_iter.alloc(win)) ||
        (rc = e->win_sweepctr.alloc(win)) || (rc = e->counters.alloc(4)) || (rc = e->stats.alloc(2)) ||
        (rc = e->xround.alloc(2)))
        return rc;
    CUDA_TRY(cudaMemsetAsync(e->slot_sweeps.p, 0, slot * sizeof(uint64_t), s));
    CUDA_TRY(cudaMemsetAsync(e->slot_draws.p, 0, slot * sizeof(int64_t), s));
    CUDA_TRY(cudaMemsetAsync(e->slot_thr_off.p, 0, slot * sizeof(int64_t), s));
    CUDA_TRY(cudaMemsetAsync(e->slot_thr_n.p, 0, slot * sizeof(int64_t), s));
    if (tab) {
        CUDA_TRY(cudaMemsetAsync(e->g.p, 0, tab * sizeof(int64_t), s));
        CUDA_TRY(cudaMemsetAsync(e->H.p, 0, tab * sizeof(uint32_t), s));
        CUDA_TRY(cudaMemsetAsync(e->visits.p, 0, tab * sizeof(uint64_t), s));
    }
    bool any_at = false;
    for (const auto& hi : e->inst) any_at = any_at || hi.d.model == REWL_MODEL_ASHKIN_TELLER2D;
    if (D.observables && tab) {
        e->obs_stride = any_at ? (D.observables == 2 ? 16 : 12) : (D.observables == 2 ? 4 : 3);
        if ((rc = e->obs.alloc((size_t)tab * e->obs_stride))) return rc;
        CUDA_TRY(cudaMemsetAsync(e->obs.p, 0, (size_t)tab * e->obs_stride * sizeof(double), s));
    }
    std::vector<int64_t> lnf(win, std::max<int64_t>(1, (int64_t)std::llround(D.lnf_initial * kLogdosScale)));
    CUDA_TRY(cudaMemcpyAsync(e->win_lnf.p, lnf.data(), win * sizeof(int64_t), cudaMemcpyHostToDevice, s));
    CUDA_TRY(cudaMemsetAsync(e->win_done.p, 0, win * sizeof(int32_t), s));
    CUDA_TRY(cudaMemsetAsync(e->win_oot.p, 0, win * sizeof(int32_t), s));
    std::vector<uint64_t> ones(win, 1);
    CUDA_TRY(cudaMemcpyAsync(e->win_iter.p, ones.data(), win * sizeof(uint64_t), cudaMemcpyHostToDevice, s));
    CUDA_TRY(cudaMemsetAsync(e->win_sweepctr.p, 0, win * sizeof(uint64_t), s));
    CUDA_TRY(cudaMemsetAsync(e->counters.p, 0, 4 * sizeof(int32_t), s));
    CUDA_TRY(cudaMemsetAsync(e->stats.p, 0, 2 * sizeof(unsigned long long), s));
    CUDA_TRY(cudaMemsetAsync(e->xround.p, 0, 2 * sizeof(unsigned long long), s));
    return REWL_OK;
}

bool bins_eligible(const InstDev& I, const rewl_batch_desc& D, int max_window_bins)
{
    if (I.model != REWL_MODEL_ISING2D || D.rng_mode != REWL_RNG_PHILOX || I.L < 3) return false;
    // the window table, with its guard bins, and the lattice live in shared memory (with the
    // correlators also the bin counts and the row and column sums)
    const size_t need = (size_t)bins_smem<1>((max_window_bins + 3) & ~1, I.L, D.observables != 0, D.observables == 2, false, false) + 256;
    if (need > 200 * 1024) return false;
    const long long step = 4 * std::llabs(I.J_u);            // every energy change is a multiple of 4|J|
    if (step % (1LL << I.bin_shift) != 0) return false;
    // a proposal lands at most 2 x 4|J| / width bins away; the guard bins cover five of them
    const long long maxbins = (8 * std::llabs(I.J_u)) >> I.bin_shift;
    if (5 * maxbins > kGuard) return false;
    // energies are -2 N J plus multiples of 4|J|: the bins' lower edges have to be energies
    return ((-2 * (long long)I.N * I.J_u - I.eglo_u) & ((1LL << I.bin_shift) - 1)) == 0;
}

// The global-table kernel's tree adds up to five energy changes to a position within a bin in 32 bits,
// in numerator units without the zeros that all changes end in (three changes more leave room for the
// terms on the way): bins of 0.05 take single flips of up to 100 energy units, bins of 1 of up to 500.
// Beyond that, the serial chain.
double largest_move(const HostInst& H)                 // of a flip, in energy units
{
    double h = 0;
    for (double f : H.fields) h = std::max(h, std::fabs(f));
    return 2.0 * (4.0 * std::fabs((double)H.dev.J_u) + 4.0 * std::fabs((double)H.dev.K_u) + std::ldexp(h, H.dev.escale));
}

int tree_eligible(const HostInst& H, const rewl_batch_desc& D)
{
    if (D.rng_mode != REWL_RNG_PHILOX) return 0;
    int zeros = 0;
    while (zeros < H.dev.bin_shift && (H.dev.bin_mul >> zeros & 1) == 0) ++zeros;
    const double move = largest_move(H);
    const int even = zeros < H.dev.bin_shift ? 1 : 0;
    return 8.0 * std::ldexp(move, -even) * (double)(H.dev.bin_mul >> zeros) + std::ldexp(1.0, H.dev.bin_shift - zeros - even) < 2147483648.0 ? 1 : 0;
}

int table_mode(const rewl_engine* e, const Launch& l)
{
    return l.cache ? kTableTree : e->desc.rng_mode == REWL_RNG_REPLAY ? kTableReplay : kTableSerial;
}

// Streaming multiprocessors of the engine's device (152 on a GB300).
int sm_count(const rewl_engine* e)
{
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, e->desc.device) != cudaSuccess || n < 1) n = 152;
    return n;
}

// The serial chain reads the tables in global memory through L1, so its shared-memory carveout is
// the smallest that still holds the blocks resident on an SM (the CUDA runtime's default split leaves
// L1 far less); the tree keeps the walkers' surroundings in shared memory and takes all of it (with a
// carveout just large enough, 512 walkers at L = 24 ran in two waves: 418 against 221 cycles per flip).
int at_carveout(rewl_engine* e, Launch& l)
{
    if (!l.tables) return REWL_OK;
    const int nsm = sm_count(e);
    const SweepKernel fn = table_kernel(l.model, table_mode(e, l), e->desc.observables != 0);
    const int threads = 32 * l.wpb;
    const size_t smem = (size_t)l.wpb * l.smem_per_warp;
    int occ = 0;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, threads, smem));
    const int blocks = ((int)l.slots.size() + l.wpb - 1) / l.wpb;
    const int per_sm = std::max(1, std::min(occ, (blocks + nsm - 1) / nsm));
    int smem_sm = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, e->desc.device));
    const size_t need = (size_t)per_sm * (smem + 1024);
    l.carveout = l.cache ? 100 : (int)std::min<size_t>(100, (need * 100 + smem_sm - 1) / (size_t)smem_sm);
    return REWL_OK;
}

// Blocks of `smem` bytes that an SM's shared memory holds (228 KB, 1 KB of it per block reserved, in units of 128 bytes)
int blocks_per_sm(int smem) { return std::max(1, 228 * 1024 / ((smem + 1024 + 127) & ~127)); }

// The time of a launch of n walkers of the bin-tracking kernel, G a warp, in cycles per flip of a walker: as many
// warps as registers (12 warps) and shared memory hold on an SM run at once, in full waves and a last one, and take what
// the busiest of its four schedulers does.  Measured at L = 48, windows of 114 bins, 1 to 3 warps a scheduler; equals
// go to more walkers a warp, which shorter rows prefer (L = 16, 768 walkers, one a warp 2.67, two 2.58 ms).
// What it decides (L = 64, e9 flips/s): visits beside g cost a bin 16 bytes instead of 8 and save the ordered stores of a
// block's g (2048 walkers of 245 bins 39.5 against 32.3, of 865 bins 25.5 against 34.0, of 4097 bins 9.6 against 17.4);
// moments in shared memory take 28 bytes a bin and save reductions to global memory (2048 walkers of 245 bins 31.2
// against 29.0, 2944 walkers 26.2 against 33.0); two walkers a warp up to 24 walkers an SM, four beyond (4096 walkers of
// 245 bins 41.1 against 55.2).
// rows: k_sweep_ising_rows with rows of so many sites.
double bins_cycles(int n, int nsm, int G, bool obs, bool cnt, bool mom, int rows, int smem)
{
    static const double kCycles[6][3][3] = {
        {{72, 97, 132}, {98, 131, 177}, {120, 165, 219}},              // g alone
        {{65, 88, 116}, {88, 114, 153}, {123, 159, 202}},              // visits beside g (one a warp: 84, 113 at L = 48)
        {{108, 128, 161}, {153, 179, 221}, {226, 264, 320}},           // observables: g alone
        {{95, 119, 159}, {128, 162, 216}, {196, 239, 285}},            //   moments in shared memory
        {{101, 118, 147}, {142, 168, 208}, {230, 266, 303}},           //   visits beside g
        {{88, 110, 145}, {119, 151, 200}, {199, 245, 290}}};           //   both
    static const double kRows[2][2][2][3] = {{{{117, 144, 185}, {97, 125, 168}}, {{200, 222, 258}, {178, 208, 245}}},      // 8
                                             {{{79, 93, 120}, {88, 112, 149}}, {{124, 139, 170}, {179, 203, 245}}}};       // 16
    const double* t = rows ? kRows[rows == 16][obs][G == 4] : kCycles[obs ? 2 + 2 * cnt + mom : cnt][G == 1 ? 0 : G == 2 ? 1 : 2];
    const int warps = ((n + G - 1) / G + nsm - 1) / nsm;
    const int room = std::min(12, blocks_per_sm(G * smem));
    const int waves = (warps - 1) / room, rest = warps - waves * room;
    return waves * t[(room - 1) / 4] + t[(rest - 1) / 4];
}

// The shape of a launch group of the bin-tracking kernel: walkers per warp (G; 0: any), visits beside g and moments in
// shared memory, the cheapest that fits; fewer walkers a warp where G's do not fit a block.  Rows of 4, 8 and 16 sites go
// one decision after another (k_sweep_ising_rows) once there are more walkers than schedulers, but for L = 16 with
// correlators.
void shape_bins(const rewl_engine* e, Launch& l, int nsm, int G)
{
    const bool obs = e->desc.observables != 0, corr = e->desc.observables == 2;
    const int n = e->desc.persistent ? e->nslots : (int)l.slots.size();
    double best = 0;
    l.rows = 0;
    if ((l.maxL == 4 || l.maxL == 8 || (l.maxL == 16 && !corr)) && !e->desc.persistent && n > 4 * nsm && G != 1) {
        const int smem = ((rows_smem(l.nbcap, l.maxL, obs, corr) + 127) & ~127) + 16;
        for (int g : {4, 2}) {
            if ((G && g > G) || g * smem > 200 * 1024) continue;
            const double t = bins_cycles(n, nsm, g, obs, false, false, l.maxL, smem);
            if (best != 0 && (G || t >= best)) continue;
            best = t;
            l.walkers_per_warp = g; l.counts = l.moments = l.crowded = 0; l.smem_per_warp = smem; l.rows = l.maxL;
        }
        if (l.rows) return;
    }
    for (int g : {4, 2, 1}) {
        if (G ? g > G : g > 1 && g > n) continue;
        for (int c = 3; c >= 0; --c) {
            const bool cnt = c & 1, mom = c & 2;
            if (mom && !obs) continue;
            const int smem = bins_smem(g, l.nbcap, l.maxL, obs, corr, cnt, mom);
            if (g * smem > 200 * 1024 && (g > 1 || c > 0)) continue;
            const double t = bins_cycles(n, nsm, g, obs, cnt, mom, 0, smem);
            if (best != 0 && t >= best) continue;
            best = t;
            l.walkers_per_warp = g; l.counts = cnt; l.moments = mom; l.smem_per_warp = smem;
        }
        if (G && best != 0) break;
    }
    l.crowded = obs && (n + l.walkers_per_warp - 1) / l.walkers_per_warp > 8 * nsm &&
                blocks_per_sm(l.walkers_per_warp * l.smem_per_warp) > 8;
}

// A launch group's shape: walkers per warp (bin-tracking kernel) and warps per block, if the
// block's shared memory fits.
bool shape_fits(const Launch& l, int G, int wpb)
{
    return (size_t)wpb * (l.bins ? G : 1) * l.smem_per_warp <= 200 * 1024;
}

// Bins of each walker's table that the global-table kernel's tree keeps in shared memory (a power of two; 0: the serial
// chain is the better form, which only launches with observables take: the others are within 2 % in long launches, and
// the chain's copy of the tables makes short ones 1.3 times as long), for n walkers of nb bins whose flips move them up
// to `move` bins; `fixed` bytes a walker beside them, 12 a bin.  Time in cycles per flip of a walker: as many warps as registers (16) and shared memory hold run at
// once, in full waves and a last one; the fewer moves the cached bins span, the more often the walker leaves them.
// Measured on Ashkin-Teller L = 12 to 32, bins of 0.05, 0.25 and 1.0 (moves of 300, 60 and 15 bins), e9 flips/s:
//   1024 walkers, 512 / 1024 / 2048 bins: bins of 0.05 4.0 / 6.3 / 8.9, of 0.25 11.6 / 12.9 / 13.4
//   2048 walkers, 512 / 1024 / 2048 bins / chain: 0.05 7.0 / 7.5 / 9.5 / 9.2, 0.25 16.6 / 13.5 / 13.5 / 11.5; with moments
//   5.2 / 4.9 / 5.8 / 7.1 and 9.6 / 7.1 / 7.3 / 8.4 (the moments' FP64 latency wants warps)
// More than kMinCache bins only where all of the engine's walkers could have them (an uneven batch of 352 walkers, 256 of
// them Ashkin-Teller: 4096 bins 10.4 ms, 8192 11.2).
int table_cache(int n, int all, int nsm, int observables, int nb, double move, int fixed_tree, int fixed_chain)
{
    static const double kTree[4] = {150, 215, 265, 300}, kChain[4] = {310, 370, 440, 480};       // warps a scheduler
    static const double kObs[2][3] = {{1.0, 1.7, 1.85}, {1.0, 1.3, 1.6}};
    auto cycles = [&](const double* t, int smem) {
        const int warps = (n + nsm - 1) / nsm, room = std::min(16, blocks_per_sm(smem));
        const int waves = (warps - 1) / room, rest = warps - waves * room;
        return waves * t[(room - 1) / 4] + t[(rest - 1) / 4];
    };
    int cache = 0;
    double best = observables ? cycles(kChain, fixed_chain) * kObs[1][observables] : DBL_MAX;
    for (int c = 256; fixed_tree + 12 * c <= 200 * 1024; c *= 2) {
        if (c > kMinCache && blocks_per_sm(fixed_tree + 12 * c) < (all + nsm - 1) / nsm) break;
        const double moves = c / move;
        const double reach = c >= nb || moves >= 24 ? 1.0 : moves >= 12 ? 0.95 : moves >= 6 ? 0.9 : moves >= 3 ? 0.71 : moves >= 1.5 ? 0.5 : 0.35;
        const double t = cycles(kTree, fixed_tree + 12 * c) * kObs[0][observables] / reach;
        if (t <= best) { best = t; cache = c; }                // (equals go to more bins)
        if (c >= nb) break;
    }
    return cache;
}

// The persistent launch: every group's walkers as tasks of one work-stealing kernel.  Groups are
// ordered by the expected cost of one walker's sweep (degrees of freedom x cycles per flip of
// its kernel, measured: table kernel ~130 on the tree and ~440 in the serial chain, bin-tracking
// ~60), the dearest first, so that the last tasks taken are short.  Every warp gets the largest
// shared-memory region any group needs.
int plan_fused(rewl_engine* e, int nsm)
{
    if (e->launches.size() > (size_t)kMaxFusedGroups)
        return fail(REWL_EINVAL, "the persistent launch takes at most %d launch groups (%zu here)", kMaxFusedGroups,
                    e->launches.size());
    std::vector<std::pair<double, size_t>> order;
    for (size_t gi = 0; gi < e->launches.size(); ++gi) {
        const Launch& l = e->launches[gi];
        int ndof = 0;
        for (int s : l.slots) ndof = std::max(ndof, e->inst[e->h_slot_inst[s]].dev.ndof);
        order.push_back({-(double)ndof * (l.bins ? 60.0 : l.cache ? 130.0 : 440.0), gi});
    }
    std::stable_sort(order.begin(), order.end());
    FusedParams& F = e->fused_p;
    F = FusedParams{};
    int task = 0, slot = 16;
    for (size_t k = 0; k < order.size(); ++k) {
        const Launch& l = e->launches[order[k].second];
        FusedGroup& G = F.g[k];
        G.slots = l.d_slots.p; G.nslots = (int)l.slots.size(); G.smem_per_warp = l.smem_per_warp; G.nbcap = l.nbcap; G.counts = l.counts; G.moments = l.moments; G.cache = l.cache;
        if (l.bins)
            G.kind = kFusedBins;
        else if (l.tables)
            G.kind = l.model == REWL_MODEL_ISING2D ? kFusedTablesIsing : kFusedTablesAT;
        else
            return fail(REWL_EINVAL, "internal: a launch group without a persistent form");
        G.first_task = task;
        task += G.nslots;
        slot = std::max(slot, l.smem_per_warp);
    }
    F.ngroups = (int)order.size();
    F.ntasks = task;
    F.slot_bytes = (slot + 15) & ~15;
    int warps = 4;
    while (warps > 1 && (size_t)warps * F.slot_bytes > 200 * 1024) warps >>= 1;
    if ((size_t)F.slot_bytes > 220 * 1024) return fail(REWL_EINVAL, "a walker needs %d bytes of shared memory", F.slot_bytes);
    e->fused_block = 32 * warps;
    e->fused_smem = (size_t)warps * F.slot_bytes;
    CUDA_TRY(cudaFuncSetAttribute(k_sweep_fused<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    CUDA_TRY(cudaFuncSetAttribute(k_sweep_fused<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    int per_sm = 0;
    if (e->desc.observables)
        CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sweep_fused<true>, e->fused_block, e->fused_smem));
    else
        CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sweep_fused<false>, e->fused_block, e->fused_smem));
    const int need = (task + warps - 1) / warps;
    e->fused_grid = std::max(1, std::min(need, std::max(1, per_sm) * nsm));
    if (int rc = e->fused_counter.alloc(1)) return rc;
    e->fused = true;
    return REWL_OK;
}

int plan_launches(rewl_engine* e)
{
    const int nsm = sm_count(e);
    // group walkers by (model, bin-tracking kernel, sites, tree) so each launch has one
    // kernel shape and the walkers sharing a warp run the same number of chunks
    struct Key { int model, bins, sites, tree; };
    std::vector<Key> keys;
    std::vector<Launch> plans;
    for (int s = 0; s < e->nslots; ++s) {
        const HostInst& H = e->inst[e->h_slot_inst[s]];
        int max_nb = 0;
        for (const auto& wd : H.wins) max_nb = std::max(max_nb, wd.nb);
        const int bins = bins_eligible(H.dev, e->desc, max_nb) && getenv("REWL_SWEEP_VARIANT") == nullptr ? 1 : 0;
        Key k{H.d.model, bins, bins ? H.dev.N : 0, tree_eligible(H, e->desc)};
        size_t idx = 0;
        for (; idx < keys.size(); ++idx)
            if (keys[idx].model == k.model && keys[idx].bins == k.bins && keys[idx].sites == k.sites &&
                keys[idx].tree == k.tree)
                break;
        if (idx == keys.size()) {
            keys.push_back(k);
            Launch l;
            l.model = k.model; l.bins = k.bins; l.tree = k.tree;
            plans.push_back(std::move(l));
        }
        plans[idx].slots.push_back(s);
    }
    int table_walkers = 0;                                     // of all groups that may have their tables in global memory
    for (const auto& l : plans) table_walkers += l.bins ? 0 : (int)l.slots.size();
    for (auto& l : plans) {
        int maxN = 0, maxnb = 0, maxL = 0;
        const bool corr = e->desc.observables == 2;
        for (int s : l.slots) {
            maxN = std::max(maxN, e->inst[e->h_slot_inst[s]].dev.N);
            maxL = std::max(maxL, e->inst[e->h_slot_inst[s]].dev.L);
            maxnb = std::max(maxnb, e->h_slot_nb[s]);
        }
        const int n = (int)l.slots.size();
        if (l.bins) {
            const int G = e->desc.persistent ? 1 : e->desc.walkers_per_warp;
            l.nbcap = (maxnb + 1) & ~1;
            l.maxL = maxL;
            const int least = bins_smem(std::max(G, 1), l.nbcap, maxL, e->desc.observables != 0, corr, false, false);
            if ((size_t)least * std::max(G, 1) > 220 * 1024) return fail(REWL_EINVAL, "a walker needs %d bytes of shared memory", least);
            shape_bins(e, l, nsm, G);
            // one warp a block: the schedulers fill evenly (L = 24, 5952 walkers, four a warp: blocks of four warps 44.5,
            // of one 59.0e9 flips/s)
            int wpb = e->desc.warps_per_block ? e->desc.warps_per_block : 1;
            wpb = std::min(wpb, 4);                                // the kernel's launch bounds: 128 threads
            while (wpb > 1 && (size_t)wpb * l.walkers_per_warp * l.smem_per_warp > 200 * 1024) wpb >>= 1;
            l.wpb = wpb;
        } else {
            const size_t ising_smem = (size_t)(((maxnb + 1) & ~1) * 8 + sizeof(Stage) + ((maxN + 15) & ~15) + (corr ? 8 * maxL : 0));
            // Ising windows live in shared memory unless they do not fit there (or the
            // global-table kernel is asked for)
            l.tables = l.model != REWL_MODEL_ISING2D || e->sweep_variant == 4 || ising_smem > 200 * 1024 ||
                       e->desc.persistent;             // the persistent launch has the global-table form only
            if (!l.tables) {
                l.nbcap = (maxnb + 1) & ~1;
                l.smem_per_warp = (int)ising_smem;
            } else {
                const int planes = l.model == REWL_MODEL_ISING2D ? 1 : 2;
                l.nbcap = 0;
                auto fixed = [&](size_t stage) {
                    return (int)(stage + ((planes * maxN + 15) & ~15) + (corr ? (8 * planes * maxL + 15) & ~15 : 0));
                };
                if (l.tree && e->desc.persistent) {
                    // eight walkers an SM, but no less than 2048 bins
                    l.cache = 256;
                    const int f = fixed(sizeof(TableStage));
                    while (l.cache < maxnb && f + 24 * l.cache <= 200 * 1024 &&
                           (l.cache < kMinCache || f + 24 * l.cache + 1040 <= 225 * 1024 / 8))
                        l.cache *= 2;
                } else if (l.tree) {
                    double move = 1.0;
                    for (int s : l.slots) {
                        const HostInst& H = e->inst[e->h_slot_inst[s]];
                        move = std::max(move, std::ldexp(largest_move(H) * (double)H.dev.bin_mul, -H.dev.bin_shift));
                    }
                    l.cache = table_cache(table_walkers, e->nslots, nsm, e->desc.observables, maxnb, move, fixed(sizeof(TableStage)), fixed(kSerialStage));
                }
                l.smem_per_warp = fixed(l.cache ? sizeof(TableStage) : kSerialStage) + 12 * l.cache;
            }
        }
        if (!l.bins) {
            l.smem_per_warp = (l.smem_per_warp + 15) & ~15;
            int wpb = e->desc.warps_per_block;
            if (wpb == 0) wpb = (l.tables && l.cache) || n <= nsm * 2 ? 1 : n <= nsm * 8 ? 2 : 4;
            while (wpb > 1 && (size_t)wpb * l.smem_per_warp > 200 * 1024) wpb >>= 1;
            if ((size_t)l.smem_per_warp > 220 * 1024) return fail(REWL_EINVAL, "a walker needs %d bytes of shared memory (limit 220 KiB)", l.smem_per_warp);
            l.wpb = wpb;
        }
        int rc = upload(l.d_slots, l.slots, e->stream);
        if (rc) return rc;
        e->launches.push_back(std::move(l));
    }
    CUDA_TRY(cudaFuncSetAttribute(k_sweep_ising<false, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    CUDA_TRY(cudaFuncSetAttribute(k_sweep_ising<false, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    CUDA_TRY(cudaFuncSetAttribute(k_sweep_ising<true, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    for (int r = 0; r < 3; ++r)
        for (int o = 0; o < 2; ++o)
            for (int m : {REWL_MODEL_ISING2D, REWL_MODEL_ASHKIN_TELLER2D})
                CUDA_TRY(cudaFuncSetAttribute(table_kernel(m, r, o), cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    for (auto& l : e->launches) {
        if (int rc = at_carveout(e, l)) return rc;
        // the serial chain copies each walker's logDoS at the start of a launch
        if (l.tables && !l.cache && !e->gsnap.p && e->table_total > 0)
            if (int rc = e->gsnap.alloc(e->table_total)) return rc;
    }
    for (int G : {2, 4})
        for (int C : {4, 8, 16})
            for (int o = 0; o < 2; ++o)
                CUDA_TRY(cudaFuncSetAttribute(rows_kernel(G, C, o), cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    for (int G : {1, 2, 4})
        for (int o = 0; o < 8; ++o)
            CUDA_TRY(cudaFuncSetAttribute(bins_kernel(G, o & 1, o & 2, o & 4), cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    if (e->desc.persistent) return plan_fused(e, nsm);
    if (e->launches.size() > 1) {
        CUDA_TRY(cudaEventCreateWithFlags(&e->fork_ev, cudaEventDisableTiming));
        for (size_t gi = 0; gi < e->launches.size(); ++gi) {
            cudaStream_t st;
            cudaEvent_t ev;
            CUDA_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
            e->gstreams.push_back(st);
            CUDA_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
            e->join_ev.push_back(ev);
        }
    }
    return REWL_OK;
}

// New fields whose energy changes the tree of the global-table kernel cannot hold: the instance's
// launch group goes over to the serial chain.
int leave_tree(rewl_engine* e, int ii)
{
    if (tree_eligible(e->inst[ii], e->desc)) return REWL_OK;
    for (auto& l : e->launches) {
        if (!l.cache) continue;
        bool here = false;
        for (int s : l.slots) here = here || e->h_slot_inst[s] == ii;
        if (!here) continue;
        if (!e->gsnap.p)
            if (int rc = e->gsnap.alloc(e->table_total)) return rc;
        l.cache = 0;
        for (int g = 0; g < e->fused_p.ngroups; ++g)
            if (e->fused_p.g[g].slots == l.d_slots.p) e->fused_p.g[g].cache = 0;
        if (int rc = at_carveout(e, l)) return rc;
        e->drop_graph();
    }
    return REWL_OK;
}

int device_error(int word)
{
    if (word & ERR_BOUNDS) return fail(REWL_EBOUNDS, "a walker's energy left its window (device error word %d)", word);
    if (word & ERR_ADJUST) return fail(REWL_EINVAL, "a walker could not reach its window");
    if (word & ERR_REPLAY_EXHAUSTED) return fail(REWL_EINVAL, "replay uniform stream exhausted");
    if (word & ERR_RANGE)
        return fail(REWL_ESTATE, "a window's logDoS passed 2^62 units (6.7e7 nats) without a flat event: "
                                 "a replica is trapped away from part of its window");
    if (word & ERR_COUNT)
        return fail(REWL_ESTATE, "a per-stage histogram count passed 2^32 - 1 without a flat event");
    return REWL_OK;
}

// Waits for the stream and reads the device's counters.  One kernel that writes to pinned memory and
// one wait; a copy to pageable memory is a wait of its own (a check interval ended with eight of them
// and four waits: L = 8, 3 windows x 2 walkers, 2 x 20 sweeps, 285 -> 214 us an interval).
int read_report(rewl_engine* e, Report* r)
{
    std::lock_guard<std::mutex> lock(e->export_mu);
    k_report<<<1, 128, 0, e->stream>>>(e->ptrs(), e->nwin_total, reinterpret_cast<Report*>(e->pinned));
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    std::memcpy(r, e->pinned, sizeof *r);
    return REWL_OK;
}

int check_device_error(rewl_engine* e)
{
    Report r;
    if (int rc = read_report(e, &r)) return rc;
    return device_error(r.counters[0]);
}

int alloc_pinned(rewl_engine* e)
{
    size_t most = 1;
    for (int s = 0; s < e->nslots; ++s) {
        const int width = e->desc.observables ? obs_columns(e->inst[e->h_slot_inst[s]].d.model, e->desc.observables == 2) + 1 : 1;
        most = std::max(most, (size_t)e->h_slot_nb[s] * width);
    }
    e->export_doubles = std::max<size_t>(64, std::min(most, rewl_engine::kExportBytes / 8));
    if (cudaHostAlloc(reinterpret_cast<void**>(&e->pinned), rewl_engine::kReportBytes + e->export_doubles * 8, cudaHostAllocDefault) != cudaSuccess) {
        e->pinned = nullptr;
        return fail(REWL_ENOMEM, "pinned host memory for exports");
    }
    return REWL_OK;
}

// [nb][width] doubles from a kernel that launch(first row, rows, destination) starts, through pinned memory
template <class F>
int export_rows(rewl_engine* e, int nb, int width, double* out, F launch)
{
    std::lock_guard<std::mutex> lock(e->export_mu);
    double* staged = reinterpret_cast<double*>(e->pinned + rewl_engine::kReportBytes);
    const int most = (int)(e->export_doubles / (size_t)width);
    for (int b0 = 0; b0 < nb; b0 += most) {
        const int rows = std::min(most, nb - b0);
        launch(b0, rows, staged);
        CUDA_TRY(cudaGetLastError());
        CUDA_TRY(cudaStreamSynchronize(e->stream));
        std::memcpy(out + (size_t)b0 * width, staged, (size_t)rows * width * 8);
    }
    return REWL_OK;
}

cudaEvent_t next_event(rewl_engine* e)
{
    if (e->capturing) {                // a timing event owned by the captured graph
        cudaEvent_t ev;
        cudaEventCreate(&ev);
        e->g_events.push_back(ev);
        return ev;
    }
    if (e->ev_used == e->ev_pool.size()) {
        cudaEvent_t ev;
        cudaEventCreate(&ev);
        e->ev_pool.push_back(ev);
    }
    return e->ev_pool[e->ev_used++];
}

// One launch group's sweeps on a stream (its kernel and shape fixed by plan_launches or the
// autotuner).
int launch_group(rewl_engine* e, Launch& l, cudaStream_t stream, int nsweeps, const DevPtrs& P)
{
    const bool replay = e->desc.rng_mode == REWL_RNG_REPLAY;
    SweepParams sp;
    sp.P = P; sp.slots = l.d_slots.p; sp.nslots = (int)l.slots.size(); sp.nsweeps = nsweeps;
    sp.smem_per_warp = l.smem_per_warp; sp.nbcap = l.nbcap; sp.counts = l.counts; sp.moments = l.moments; sp.cache = l.cache;
    if (l.bins) {
        const int G = l.walkers_per_warp;
        const int warps = (sp.nslots + G - 1) / G;
        const int blocks = (warps + l.wpb - 1) / l.wpb;
        const size_t smem = (size_t)l.wpb * G * l.smem_per_warp;
        const SweepKernel fn = l.rows ? rows_kernel(G, l.rows, P.obs != nullptr) : bins_kernel(G, P.obs != nullptr, l.counts, l.crowded);
        fn<<<blocks, 32 * l.wpb, smem, stream>>>(sp);
    } else {
        const int blocks = (sp.nslots + l.wpb - 1) / l.wpb;
        const size_t smem = (size_t)l.wpb * l.smem_per_warp;
        if (l.tables) {
            const SweepKernel fn = table_kernel(l.model, table_mode(e, l), e->desc.observables != 0);
            if (l.carveout >= 0) CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, l.carveout));
            fn<<<blocks, 32 * l.wpb, smem, stream>>>(sp);
        } else {
            if (replay) k_sweep_ising<true, 2><<<blocks, 32 * l.wpb, smem, stream>>>(sp);
            else if (e->sweep_variant == 2) k_sweep_ising<false, 2><<<blocks, 32 * l.wpb, smem, stream>>>(sp);
            else k_sweep_ising<false, 3><<<blocks, 32 * l.wpb, smem, stream>>>(sp);
        }
    }
    CUDA_TRY(cudaGetLastError());
    e->kernel_launches++;
    e->launches_total++;
    return REWL_OK;
}

// A timing event on the engine stream; inside a stream capture it must become an event node of
// the graph (a plain record there only marks a dependency).
cudaError_t record_timing(rewl_engine* e)
{
    cudaEvent_t ev = next_event(e);
    return e->capturing ? cudaEventRecordWithFlags(ev, e->stream, cudaEventRecordExternal) : cudaEventRecord(ev, e->stream);
}

// Sweeps per launch such that one launch plus one exchange visit add at most kLaunchGrowth to
// any bin: lnf_bound x (sweeps x ndof_max + 1) <= kLaunchGrowth.
int max_launch_sweeps(const rewl_engine* e)
{
    const int64_t visits = kLaunchGrowth / std::max<int64_t>(1, e->lnf_bound_u) - 1;
    // the bin-tracking kernel counts a launch's visits in 31 bits
    return (int)std::max<int64_t>(1, std::min<int64_t>(1 << 20, std::min<int64_t>(visits, INT32_MAX) / std::max<int64_t>(1, e->ndof_max)));
}

// Raise the ln f bound (rewl_set_lnf, rewl_restore); a captured check interval split its sweeps
// for the old bound, so it is captured again.
void raise_lnf_bound(rewl_engine* e, int64_t lnf_u)
{
    if (lnf_u <= e->lnf_bound_u) return;
    const int before = max_launch_sweeps(e);
    e->lnf_bound_u = lnf_u;
    if (max_launch_sweeps(e) != before) e->drop_graph();
}

int launch_sweeps_once(rewl_engine* e, int nsweeps);

int launch_sweeps(rewl_engine* e, int nsweeps)
{
    const int most = max_launch_sweeps(e);
    while (nsweeps > 0) {
        const int n = std::min(nsweeps, most);
        if (int rc = launch_sweeps_once(e, n)) return rc;
        nsweeps -= n;
    }
    return REWL_OK;
}

int launch_sweeps_once(rewl_engine* e, int nsweeps)
{
    const DevPtrs P = e->ptrs();
    CUDA_TRY(record_timing(e));
    if (e->fused) {
        FusedParams F = e->fused_p;
        F.P = P;
        F.nsweeps = nsweeps;
        F.counter = e->fused_counter.p;
        CUDA_TRY(cudaMemsetAsync(e->fused_counter.p, 0, sizeof(unsigned int), e->stream));
        if (e->desc.observables) k_sweep_fused<true><<<e->fused_grid, e->fused_block, e->fused_smem, e->stream>>>(F);
        else k_sweep_fused<false><<<e->fused_grid, e->fused_block, e->fused_smem, e->stream>>>(F);
        CUDA_TRY(cudaGetLastError());
        e->kernel_launches++;
        e->launches_total++;
        CUDA_TRY(record_timing(e));
        e->sweeps_total += nsweeps;
        e->sweeps_since_check += nsweeps;
        e->flips_total += (int64_t)nsweeps * e->flips_per_sweep;
        return REWL_OK;
    }
    // several launch groups (models, lattice sizes, kernel shapes) run concurrently, each on
    // its own stream forked from and joined back into the engine stream; they touch disjoint
    // walkers
    const bool fork = e->gstreams.size() == e->launches.size() && e->launches.size() > 1;
    if (fork) CUDA_TRY(cudaEventRecord(e->fork_ev, e->stream));
    for (size_t gi = 0; gi < e->launches.size(); ++gi) {
        const cudaStream_t stream = fork ? e->gstreams[gi] : e->stream;
        if (fork) CUDA_TRY(cudaStreamWaitEvent(stream, e->fork_ev, 0));
        if (int rc = launch_group(e, e->launches[gi], stream, nsweeps, P)) return rc;
        if (fork) {
            CUDA_TRY(cudaEventRecord(e->join_ev[gi], stream));
            CUDA_TRY(cudaStreamWaitEvent(e->stream, e->join_ev[gi], 0));
        }
    }
    CUDA_TRY(record_timing(e));
    e->sweeps_total += nsweeps;
    e->sweeps_since_check += nsweeps;
    e->flips_total += (int64_t)nsweeps * e->flips_per_sweep;
    return REWL_OK;
}

int launch_exchange(rewl_engine* e)
{
    // the kernel reads the round (and from its parity the direction) on the device and
    // advances it; the host keeps a mirror for snapshots
    const int n0 = (int)e->pairs_dir[0].size() / 2, n1 = (int)e->pairs_dir[1].size() / 2;
    const int blocks = std::max(1, (std::max(n0, n1) + 127) / 128);
    k_exchange<<<blocks, 128, 0, e->stream>>>(e->ptrs(), e->pairs[0].p, n0, e->pairs[1].p, n1);
    CUDA_TRY(cudaGetLastError());
    e->launches_total++;
    e->direction ^= 1;
    e->exch_round++;
    return REWL_OK;
}

int launch_flat(rewl_engine* e)
{
    FlatParams fp;
    fp.P = e->ptrs();
    fp.nwin_total = e->nwin_total;
    fp.flat_mode = e->desc.flatness_mode;
    fp.mask_mode = e->desc.mask_mode;
    fp.one_over_t = e->desc.one_over_t;
    fp.reduce = e->desc.reduce_logdos;
    fp.flat_den = 1000000;
    fp.flat_num = (uint64_t)std::llround(e->desc.flatness_param * 1e6);
    fp.flat_param_f = (float)e->desc.flatness_param;
    fp.lnf_final = e->desc.lnf_final;
    fp.sweeps_since_check = e->sweeps_since_check;
    e->sweeps_since_check = 0;
    k_flat<<<e->nwin_total, 256, 0, e->stream>>>(fp);
    CUDA_TRY(cudaGetLastError());
    e->launches_total++;
    return REWL_OK;
}

bool valid_walker(const rewl_engine* e, int w) { return e && w >= 0 && w < e->nslots; }

int window_index(const rewl_engine* e, int ii, int w)
{
    if (!e || ii < 0 || ii >= (int)e->inst.size()) return -1;
    if (w < 0 || w >= e->inst[ii].d.num_windows) return -1;
    return e->inst[ii].dev.first_win + w;
}

// ------------------------------------------------------------------------
// Host restatement of concatenate_tables (multiple overlap) for the logDoS
// (src/util/concatenate_rewl_tables.hpp:167-305) with derivative_of_vector
// (src/util/numerical_derivatives.hpp:47-70) and the concatenation-point
// search (src/util/vector_matching.hpp:38-88).
// ------------------------------------------------------------------------
double derivative(size_t i, const std::vector<double>& f, const std::vector<double>& a)
{
    const size_t n = f.size();
    if (i == 0) return (f[1] - f[0]) / (a[1] - a[0]);
    if (i == n - 1) return (f[i] - f[i - 1]) / (a[i] - a[i - 1]);
    if (i == 1 || i == n - 2) return (f[i + 1] - f[i - 1]) / (2. * (a[i] - a[i - 1]));
    return (-f[i + 2] + 8. * f[i + 1] - 8. * f[i - 1] + f[i - 2]) / (12. * (a[i] - a[i - 1]));
}

// reference_abs: compare derivative differences as the reference's compiled code does.  Its
// find_left_concatenation_indices calls an unqualified abs() on a double in a translation unit
// that includes only <cmath> and <vector>, which resolves to the C library's int abs(int): every
// |difference| is truncated to an integer, so the splice lands on the first overlapping bin unless
// some derivative difference reaches 1.  Without it the true |difference| is minimised.
inline double beta_gap(double d, bool reference_abs)
{
    if (!reference_abs) return std::fabs(d);
    const double t = std::trunc(d);                       // double -> int conversion truncates
    return std::fabs(std::max(-2147483647.0, std::min(2147483647.0, t)));
}

// O (optional): per window, rows of nobs observables; they are averaged in each overlap as the
// reference does (average_two_windows, src/util/concatenate_rewl_tables.hpp:42-49, weighted by
// the number of windows already averaged at the bin) into fo.
int concatenate(const std::vector<std::vector<double>>& E, const std::vector<std::vector<double>>& G,
                std::vector<double>& fe, std::vector<double>& fg, bool reference_abs = false,
                const std::vector<std::vector<double>>* O = nullptr, int nobs = 0, std::vector<double>* fo = nullptr)
{
    fe = E[0]; fg = G[0];
    std::vector<size_t> overlap(fe.size(), 1);
    if (O) *fo = (*O)[0];
    for (size_t w = 1; w < E.size(); ++w) {
        const auto& er = E[w]; const auto& gr = G[w];
        if (er.size() < 2 || fe.size() < 2) return fail(REWL_EINVAL, "window %zu has fewer than 2 valid bins", w);
        long left_start = -1;
        for (long k = (long)fe.size() - 1; k >= 0; --k) if (fe[k] == er[0]) { left_start = k; break; }
        if (left_start < 0) return fail(REWL_EINVAL, "windows %zu and %zu do not overlap", w - 1, w);
        const size_t nleft = fe.size();
        if (nleft - (size_t)left_start > er.size()) return fail(REWL_EINVAL, "window %zu lies inside window %zu", w, w - 1);
        double beta_diff = beta_gap(derivative((size_t)left_start, fg, fe) - derivative(0, gr, er), reference_abs);
        size_t cl = (size_t)left_start;
        for (size_t idx = 1; idx != nleft - (size_t)left_start; ++idx) {
            const double lb = derivative((size_t)left_start + idx, fg, fe), rb = derivative(idx, gr, er);
            const double gap = beta_gap(lb - rb, reference_abs);
            if ((gap + 0.5) < (beta_diff + 0.5)) { beta_diff = gap; cl = (size_t)left_start + idx; }
        }
        double shifter = 0;
        size_t right_idx = 0;
        for (size_t idx = (size_t)left_start; idx != fe.size(); ++idx) {
            right_idx = idx - (size_t)left_start;
            if (O) {
                const double c = (double)overlap[idx];
                for (int k = 0; k < nobs; ++k) {
                    double& v = (*fo)[idx * nobs + k];
                    v = (c * v + 1.0 * (*O)[w][right_idx * nobs + k]) / (double)(overlap[idx] + 1);
                }
            }
            ++overlap[idx];
            if (idx == cl) shifter = fg[idx] - gr[right_idx];
            else if (idx > cl) fg[idx] = gr[right_idx] + shifter;
        }
        for (size_t idx = right_idx + 1; idx < er.size(); ++idx) {
            fe.push_back(er[idx]);
            fg.push_back(gr[idx] + shifter);
            overlap.push_back(1);
            if (O)
                for (int k = 0; k < nobs; ++k) fo->push_back((*O)[w][idx * nobs + k]);
        }
    }
    return REWL_OK;
}

// normalize_logDoS (src/util/array_shift.hpp:15-43) step for step: the shift that makes
// sum_E g(E) = states_per_site^N (halved for a half spectrum).  Its running maximum starts at 0.
double normalisation_shift(const std::vector<double>& g, double states_per_site, double system_size, bool half)
{
    double mx = 0.0;
    for (double v : g) mx = mx > v ? mx : v;
    double sum = 0.0;
    for (double v : g) sum += std::exp(-(mx - v));
    sum = std::log(sum);
    sum += mx;
    return system_size * std::log(states_per_site) - sum - std::log(2.) * (half ? 1.0 : 0.0);
}

} // namespace

// ============================================================================
// C ABI
// ============================================================================
extern "C" {

const char* rewl_last_error_string(void) { return g_last_error.c_str(); }

int rewl_create(const rewl_batch_desc* desc, rewl_engine** out)
{
    if (!desc || !out) return fail(REWL_EINVAL, "null argument");
    *out = nullptr;
    rewl_engine* e = new rewl_engine();
    e->desc = *desc;
    // REWL_SWEEP_VARIANT: 2 the general Ising kernel's lane-0 resolver, 3 its all-lane resolver,
    // 4 the global-table kernel for Ising too (any of them turns the bin-tracking kernel off)
    if (const char* v = std::getenv("REWL_SWEEP_VARIANT")) {
        const int k = std::atoi(v);
        e->sweep_variant = (k == 2 || k == 4) ? k : 3;
    }
    int rc = build_host(e);               // descriptor validation and layout: host only
    if (rc) { delete e; return rc; }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { delete e; return fail(REWL_EDEVICE, "no CUDA device"); }
    if (desc->device < 0 || desc->device >= ndev) { delete e; return fail(REWL_EINVAL, "device %d out of range", desc->device); }
    if (cudaSetDevice(desc->device) != cudaSuccess || cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete e; return fail(REWL_EDEVICE, "cannot open device %d", desc->device);
    }
    rc = upload_all(e);
    if (!rc) rc = alloc_pinned(e);
    if (!rc) rc = plan_launches(e);
    if (!rc) {
        k_init<<<(e->nslots + 63) / 64, 64, 0, e->stream>>>(e->ptrs(), e->nslots, 0);
        cudaError_t ce = cudaGetLastError();
        if (ce != cudaSuccess) rc = fail(REWL_EDEVICE, "k_init launch: %s", cudaGetErrorString(ce));
    }
    if (!rc) rc = check_device_error(e);
    if (rc) { e->release(); delete e; return rc; }
    *out = e;
    return REWL_OK;
}

int rewl_destroy(rewl_engine* e)
{
    if (!e) return REWL_OK;
    cudaSetDevice(e->desc.device);
    if (e->stream) cudaStreamSynchronize(e->stream);
    e->release();
    delete e;
    return REWL_OK;
}

int rewl_num_walkers(const rewl_engine* e, int32_t* n)
{
    if (!e || !n) return fail(REWL_EINVAL, "null argument");
    *n = e->nslots;
    return REWL_OK;
}

int rewl_walker_info(const rewl_engine* e, int32_t w, int32_t* inst, int32_t* win, int32_t* rep)
{
    if (!valid_walker(e, w)) return fail(REWL_EINVAL, "walker %d out of range", w);
    const int ii = e->h_slot_inst[w];
    const WinDev& W = e->h_wins[e->h_slot_win[w]];
    if (inst) *inst = ii;
    if (win) *win = W.local;
    if (rep) *rep = (w - e->inst[ii].dev.first_slot) % e->inst[ii].dev.R;
    return REWL_OK;
}

int rewl_window_info(const rewl_engine* e, int32_t ii, int32_t w, double* emin, double* emax, int32_t* nb)
{
    const int wi = window_index(e, ii, w);
    if (wi < 0) return fail(REWL_EINVAL, "window (%d, %d) out of range", ii, w);
    if (emin) *emin = e->inst[ii].wmin[w];
    if (emax) *emax = e->inst[ii].wmax[w];
    if (nb) *nb = e->h_wins[wi].nb;
    return REWL_OK;
}

int rewl_import_dofs(rewl_engine* e, int32_t w, const int8_t* dofs, int32_t flavour)
{
    if (!valid_walker(e, w) || !dofs) return fail(REWL_EINVAL, "bad walker or null dofs");
    if (flavour != 0 && flavour != 1) return fail(REWL_EINVAL, "flavour must be 0 or 1");
    const int ii = e->h_slot_inst[w];
    const InstDev& I = e->inst[ii].dev;
    for (int i = 0; i < I.ndof; ++i)
        if (dofs[i] != 1 && dofs[i] != -1) return fail(REWL_EINVAL, "spins must be +1 or -1");
    cudaSetDevice(e->desc.device);
    int32_t cfg;
    CUDA_TRY(cudaMemcpyAsync(&cfg, e->slot_cfg.p + w, sizeof cfg, cudaMemcpyDeviceToHost, e->stream));
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    CUDA_TRY(cudaMemcpyAsync(e->spins.p + e->h_cfg_off[cfg], dofs, I.ndof, cudaMemcpyHostToDevice, e->stream));
    CUDA_TRY(cudaMemcpyAsync(e->slot_flavour.p + w, &flavour, sizeof flavour, cudaMemcpyHostToDevice, e->stream));
    int32_t* tmp = nullptr;
    CUDA_TRY(cudaMalloc(&tmp, 2 * sizeof(int32_t)));
    int32_t hv[2] = {cfg, ii};
    CUDA_TRY(cudaMemcpyAsync(tmp, hv, sizeof hv, cudaMemcpyHostToDevice, e->stream));
    k_recalc<<<1, 32, 0, e->stream>>>(e->ptrs(), tmp, tmp + 1, 1);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    cudaFree(tmp);
    // the energy must be inside the walker's window
    int64_t E;
    CUDA_TRY(cudaMemcpy(&E, e->cfg_E.p + cfg, sizeof E, cudaMemcpyDeviceToHost));
    const WinDev& W = e->h_wins[e->h_slot_win[w]];
    const int64_t gb = (((E - I.eglo_u) * I.bin_mul) >> I.bin_shift) - W.gblo;
    if (gb < 0 || gb >= W.nb) return fail(REWL_EINVAL, "imported configuration has energy outside the walker's window");
    return REWL_OK;
}

// Random fields drawn as the reference's Disorder::generate_random_field does
// (src/Hamiltonians/Disorder/random_fields.hpp:41-75), from the given seed instead of the
// clock.  One std::mt19937_64 stream read through std::uniform_real_distribution<double>(0, 1)
// (random_number_generator, src/util/random_number_generators.hpp:14-31); for every site 20
// values are drawn and discarded, then one is kept.  Uniform: 2 h (2u - 1).  Gaussian
// (get_gaussian, :33-57): Box-Muller on (u, v), both redrawn while u <= DBL_EPSILON; a third
// uniform keeps the cosine value when below 1/2, else the sine value, combined as the
// reference combines them (z0 * c + z1 * !c) so that the doubles agree bit for bit.
int rewl_generate_fields(uint64_t seed, double strength, int32_t distribution, int64_t num_sites, double* out)
{
    if (num_sites < 0 || (num_sites > 0 && !out)) return fail(REWL_EINVAL, "num_sites must be >= 0 and out non-null");
    if (distribution != REWL_DISORDER_UNIFORM && distribution != REWL_DISORDER_GAUSSIAN)
        return fail(REWL_EINVAL, "distribution must be REWL_DISORDER_UNIFORM or REWL_DISORDER_GAUSSIAN");
    std::mt19937_64 gen(seed);
    std::uniform_real_distribution<double> unit(0.0, 1.0);
    const double two_pi = 2.0 * std::acos(-1.0);
    auto draw = [&]() -> double {
        if (distribution == REWL_DISORDER_UNIFORM) return 2.0 * strength * (-1.0 + 2.0 * unit(gen));
        double u = unit(gen), v = unit(gen);
        while (u <= std::numeric_limits<double>::epsilon()) {
            u = unit(gen);
            v = unit(gen);
        }
        const double r = strength * std::sqrt(-2.0 * std::log(u));
        const double z0 = r * std::cos(two_pi * v) + 0.0;
        const double z1 = r * std::sin(two_pi * v) + 0.0;
        const bool c = unit(gen) < 0.5;
        return z0 * c + z1 * !c;
    };
    constexpr int kDiscarded = 20;
    for (int64_t i = 0; i < num_sites; ++i) {
        for (int k = 0; k < kDiscarded; ++k) (void)draw();
        out[i] = draw();
    }
    return REWL_OK;
}

int rewl_import_disorder(rewl_engine* e, int32_t ii, const double* fields)
{
    if (!e || ii < 0 || ii >= (int)e->inst.size() || !fields) return fail(REWL_EINVAL, "bad instance or null fields");
    HostInst& H = e->inst[ii];
    if (H.dev.model != REWL_MODEL_ASHKIN_TELLER2D || H.dev.field_off < 0)
        return fail(REWL_EINVAL, "instance %d was created without fields", ii);
    std::vector<int64_t> q(H.dev.N);
    for (int i = 0; i < H.dev.N; ++i) {
        const double v = std::nearbyint(std::ldexp(fields[i], 20));
        if (!std::isfinite(v)) return fail(REWL_EINVAL, "bad field value");
        q[i] = (int64_t)v; H.fields[i] = std::ldexp(v, -20);
    }
    cudaSetDevice(e->desc.device);
    if (int rc = leave_tree(e, ii)) return rc;
    CUDA_TRY(cudaMemcpyAsync(e->fields.p + H.dev.field_off, q.data(), q.size() * 8, cudaMemcpyHostToDevice, e->stream));
    const int n = H.dev.nwin * H.dev.R;
    std::vector<int32_t> cfgs(n), insts(n, ii);
    CUDA_TRY(cudaMemcpyAsync(cfgs.data(), e->slot_cfg.p + H.dev.first_slot, n * 4, cudaMemcpyDeviceToHost, e->stream));
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    int32_t* tmp = nullptr;
    CUDA_TRY(cudaMalloc(&tmp, 2 * n * sizeof(int32_t)));
    CUDA_TRY(cudaMemcpyAsync(tmp, cfgs.data(), n * 4, cudaMemcpyHostToDevice, e->stream));
    CUDA_TRY(cudaMemcpyAsync(tmp + n, insts.data(), n * 4, cudaMemcpyHostToDevice, e->stream));
    k_recalc<<<(n + 63) / 64, 64, 0, e->stream>>>(e->ptrs(), tmp, tmp + n, n);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    cudaFree(tmp);
    return REWL_OK;
}

int rewl_set_logdos(rewl_engine* e, int32_t ii, int32_t w, const double* logdos)
{
    const int wi = window_index(e, ii, w);
    if (wi < 0 || !logdos) return fail(REWL_EINVAL, "bad window or null logdos");
    const int nb = e->h_wins[wi].nb;
    std::vector<int64_t> q(nb);
    for (int b = 0; b < nb; ++b) {
        // a quarter of the 2^62-unit ceiling (1.68e7 nats): room for a first stage to follow
        if (!std::isfinite(logdos[b]) || std::fabs(logdos[b]) > kSetLogdosMax) return fail(REWL_EINVAL, "logdos values must be finite and |g| <= 2^60 units (1.68e7 nats)");
        q[b] = (int64_t)std::nearbyint(logdos[b] * kLogdosScale);
    }
    cudaSetDevice(e->desc.device);
    const InstDev& I = e->inst[ii].dev;
    for (int r = 0; r < I.R; ++r) {
        const int s = I.first_slot + w * I.R + r;
        CUDA_TRY(cudaMemcpyAsync(e->g.p + e->h_slot_tab[s], q.data(), nb * 8, cudaMemcpyHostToDevice, e->stream));
    }
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    return REWL_OK;
}

int rewl_set_lnf(rewl_engine* e, int32_t ii, int32_t w, double lnf)
{
    const int wi = window_index(e, ii, w);
    if (wi < 0 || !(lnf > 0) || lnf > 64) return fail(REWL_EINVAL, "bad window or ln f");
    const int64_t q = std::max<int64_t>(1, (int64_t)std::llround(lnf * kLogdosScale));
    cudaSetDevice(e->desc.device);
    raise_lnf_bound(e, q);
    CUDA_TRY(cudaMemcpyAsync(e->win_lnf.p + wi, &q, 8, cudaMemcpyHostToDevice, e->stream));
    const int32_t done = (lnf < e->desc.lnf_final) ? 1 : 0;
    CUDA_TRY(cudaMemcpyAsync(e->win_done.p + wi, &done, 4, cudaMemcpyHostToDevice, e->stream));
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    return REWL_OK;
}

int rewl_set_uniform_stream(rewl_engine* e, int32_t w, const double* u, size_t n)
{
    if (!valid_walker(e, w) || (!u && n)) return fail(REWL_EINVAL, "bad walker or null stream");
    if (e->desc.rng_mode != REWL_RNG_REPLAY) return fail(REWL_ESTATE, "engine was not created in replay mode");
    // accept <=> u < exp(-dg) for the float dg; since exp(-f) falls with f, the
    // accepted floats are those below tau = the smallest float with exp(-tau) <= u
    std::vector<int64_t> T(n);
    for (size_t k = 0; k < n; ++k) {
        const double x = u[k];
        if (!(x >= 0.0 && x < 1.0)) return fail(REWL_EINVAL, "uniform %zu not in [0,1)", k);
        if (x == 0.0) { T[k] = INT64_MAX; continue; }
        float f = (float)(-std::log(x));
        if (!(f > 0)) f = 1e-30f;
        while (f > 0 && !(std::exp(-(double)f) > x)) f = std::nextafter(f, 0.0f);
        while (std::exp(-(double)std::nextafter(f, INFINITY)) > x) f = std::nextafter(f, INFINITY);
        const float tau = std::nextafter(f, INFINITY);
        T[k] = (tau < 1e-30f) ? 1 : accept_threshold(tau);
    }
    cudaSetDevice(e->desc.device);
    // append to the walker-private table (reallocate the pool)
    const size_t old = e->thr.n;
    std::vector<int64_t> all(old + n);
    if (old) CUDA_TRY(cudaMemcpy(all.data(), e->thr.p, old * 8, cudaMemcpyDeviceToHost));
    std::copy(T.begin(), T.end(), all.begin() + old);
    e->thr.free_();
    int rc = e->thr.alloc(all.size());
    if (rc) return rc;
    CUDA_TRY(cudaMemcpy(e->thr.p, all.data(), all.size() * 8, cudaMemcpyHostToDevice));
    const int64_t off = (int64_t)old, cnt = (int64_t)n, zero = 0;
    CUDA_TRY(cudaMemcpy(e->slot_thr_off.p + w, &off, 8, cudaMemcpyHostToDevice));
    CUDA_TRY(cudaMemcpy(e->slot_thr_n.p + w, &cnt, 8, cudaMemcpyHostToDevice));
    CUDA_TRY(cudaMemcpy(e->slot_draws.p + w, &zero, 8, cudaMemcpyHostToDevice));
    return REWL_OK;
}

int rewl_run_sweeps(rewl_engine* e, int64_t n)
{
    if (!e || n < 0) return fail(REWL_EINVAL, "bad arguments");
    cudaSetDevice(e->desc.device);
    while (n > 0) {
        const int chunk = (int)std::min<int64_t>(n, 1 << 20);
        int rc = launch_sweeps(e, chunk);
        if (rc) return rc;
        n -= chunk;
    }
    return check_device_error(e);
}

int rewl_exchange(rewl_engine* e)
{
    if (!e) return fail(REWL_EINVAL, "null engine");
    cudaSetDevice(e->desc.device);
    int rc = launch_exchange(e);
    if (rc) return rc;
    return check_device_error(e);
}

namespace {
// After k_flat: the number of windows that went flat, and the device error word.
int finish_check(rewl_engine* e, Report* r)
{
    if (int rc = read_report(e, r)) return rc;
    e->flat_events += r->counters[1];
    e->cycles++;
    return device_error(r->counters[0]);
}

void fill_status(const rewl_engine* e, const Report& r, rewl_status* st)
{
    std::memset(st, 0, sizeof *st);
    st->sweeps = e->sweeps_total;
    st->cycles = e->cycles;
    st->flat_events = e->flat_events;
    st->windows_total = e->nwin_total;
    st->windows_done = r.windows_done;
    st->all_done = st->windows_done == st->windows_total;
    st->exchanges_attempted = (int64_t)r.stats[0];
    st->exchanges_accepted = (int64_t)r.stats[1];
    st->attempted_flips = e->flips_total;
    st->device_error = r.counters[0];
    st->kernel_launches = e->launches_total;
}

int check_flat(rewl_engine* e, Report* r)
{
    CUDA_TRY(cudaMemsetAsync(e->counters.p + 1, 0, 4, e->stream));
    if (int rc = launch_flat(e)) return rc;
    return finish_check(e, r);
}

// Capture one check interval (rounds x (sweeps + exchange), then the flatness step) as a CUDA
// graph.  Nothing runs during capture, so the host counters the launches advance are put back
// and applied per replay instead.
int capture_cycle(rewl_engine* e)
{
    const int se = e->desc.sweeps_per_exchange, rounds = e->desc.sweeps_per_check / se;
    const int64_t s0 = e->sweeps_total, f0 = e->flips_total, l0 = e->launches_total, k0 = e->kernel_launches;
    const uint64_t r0 = e->exch_round;
    const int d0 = e->direction;
    const size_t ev0 = e->ev_used;
    e->drop_graph();
    CUDA_TRY(cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeRelaxed));
    e->capturing = true;
    int rc = REWL_OK;
    for (int r = 0; r < rounds && rc == REWL_OK; ++r) {
        rc = launch_sweeps(e, se);
        if (rc == REWL_OK) rc = launch_exchange(e);
    }
    if (rc == REWL_OK && cudaMemsetAsync(e->counters.p + 1, 0, 4, e->stream) != cudaSuccess)
        rc = fail(REWL_EDEVICE, "memset during capture failed");
    if (rc == REWL_OK) rc = launch_flat(e);
    e->capturing = false;
    cudaGraph_t graph = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(e->stream, &graph);
    if (rc == REWL_OK && ce != cudaSuccess) rc = fail(REWL_EDEVICE, "stream capture: %s", cudaGetErrorString(ce));
    if (rc == REWL_OK && cudaGraphInstantiate(&e->cycle_exec, graph, 0) != cudaSuccess) {
        e->cycle_exec = nullptr;
        rc = fail(REWL_EDEVICE, "graph instantiation failed");
    }
    if (graph) cudaGraphDestroy(graph);
    e->g_sweeps = e->sweeps_total - s0; e->g_flips = e->flips_total - f0;
    e->g_launches = e->launches_total - l0; e->g_kernel_launches = e->kernel_launches - k0; e->g_rounds = rounds;
    e->sweeps_total = s0; e->flips_total = f0; e->launches_total = l0; e->kernel_launches = k0;
    e->exch_round = r0; e->direction = d0; e->sweeps_since_check = 0; e->ev_used = ev0;
    if (rc) e->drop_graph();
    return rc;
}

// One check interval by replaying the captured graph.
int replay_cycle(rewl_engine* e, Report* r)
{
    if (!e->cycle_exec)
        if (int rc = capture_cycle(e)) return rc;
    CUDA_TRY(cudaGraphLaunch(e->cycle_exec, e->stream));
    e->sweeps_total += e->g_sweeps; e->flips_total += e->g_flips;
    e->launches_total += e->g_launches; e->kernel_launches += e->g_kernel_launches;
    e->exch_round += (uint64_t)e->g_rounds;
    e->direction ^= (int)(e->g_rounds & 1);
    int rc = finish_check(e, r);            // synchronises the stream
    for (size_t k = 0; k + 1 < e->g_events.size(); k += 2) {
        float t = 0;                        // timing only: a failed read leaves it out
        if (cudaEventElapsedTime(&t, e->g_events[k], e->g_events[k + 1]) == cudaSuccess) e->graph_sweep_ms += t;
        else (void)cudaGetLastError();
    }
    return rc;
}
} // namespace

int rewl_check_flat(rewl_engine* e, int32_t* num_flat)
{
    if (!e) return fail(REWL_EINVAL, "null engine");
    cudaSetDevice(e->desc.device);
    Report r{};
    const int rc = check_flat(e, &r);
    if (num_flat) *num_flat = r.counters[1];
    return rc;
}

int rewl_reset_histograms(rewl_engine* e, int32_t ii, int32_t w, int32_t reduce)
{
    const int wi = window_index(e, ii, w);
    if (wi < 0) return fail(REWL_EINVAL, "bad window");
    cudaSetDevice(e->desc.device);
    k_reset_window<<<1, 256, 0, e->stream>>>(e->ptrs(), wi, reduce);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    return REWL_OK;
}

int rewl_get_status(rewl_engine* e, rewl_status* st)
{
    if (!e || !st) return fail(REWL_EINVAL, "null argument");
    cudaSetDevice(e->desc.device);
    Report r;
    if (int rc = read_report(e, &r)) return rc;
    fill_status(e, r, st);
    return REWL_OK;
}

int rewl_run_cycles(rewl_engine* e, int64_t ncycles, int64_t timeout_ms, rewl_status* st)
{
    if (!e || ncycles < 0) return fail(REWL_EINVAL, "bad arguments");
    cudaSetDevice(e->desc.device);
    const auto t0 = std::chrono::steady_clock::now();
    const int se = e->desc.sweeps_per_exchange, rounds = e->desc.sweeps_per_check / se;
    int rc = REWL_OK;
    if (e->desc.autotune && !e->tuned && (rc = rewl_autotune(e, 0))) return rc;
    for (int64_t c = 0; c < ncycles; ++c) {
        Report report;
        // a whole check interval replays as one graph unless sweeps were run by hand since the
        // last check (the captured flatness step assumes exactly one interval of sweeps)
        const bool graph = e->desc.graphs && e->desc.rng_mode != REWL_RNG_REPLAY && e->sweeps_since_check == 0;
        if (graph) {
            if ((rc = replay_cycle(e, &report))) return rc;
        } else {
            for (int r = 0; r < rounds; ++r) {
                if ((rc = launch_sweeps(e, se))) return rc;
                if ((rc = launch_exchange(e))) return rc;
            }
            if ((rc = check_flat(e, &report))) return rc;
        }
        rewl_status s;
        fill_status(e, report, &s);
        if (st) *st = s;
        if (s.all_done) break;
        if (timeout_ms > 0) {
            const auto ms = std::chrono::duration_cast<std::chrono::milliseconds>(std::chrono::steady_clock::now() - t0).count();
            if (ms > timeout_ms) return fail(REWL_ETIMEDOUT, "run_cycles deadline of %lld ms passed", (long long)timeout_ms);
        }
    }
    if (st && ncycles == 0) return rewl_get_status(e, st);
    return REWL_OK;
}

namespace {
// Observables of slots first .. first + count - 1 (k_export_observables): the sums stay on the device, only
// the averages cross (L = 12, K + 1 = 17 columns of 8228 bins, 4 replicas: 4.3 MB and four waits, 660 us;
// 1.1 MB and one, 146 us).
int export_obs(rewl_engine* e, int ii, int first, int count, double* out)
{
    if (!e->obs.p) return fail(REWL_ESTATE, "the engine was created without observables (rewl_batch_desc.observables)");
    const int model = e->inst[ii].d.model, width = obs_columns(model, e->desc.observables == 2) + 1;
    return export_rows(e, e->h_slot_nb[first], width, out, [&](int b0, int rows, double* to) {
        k_export_observables<<<(unsigned)(((long long)rows * width + 127) / 128), 128, 0, e->stream>>>(e->ptrs(), model, first, count, b0, rows, to);
    });
}
} // namespace

int rewl_export_observables(rewl_engine* e, int32_t w, double* out)
{
    if (!valid_walker(e, w) || !out) return fail(REWL_EINVAL, "walker %d out of range or null output", w);
    cudaSetDevice(e->desc.device);
    return export_obs(e, e->h_slot_inst[w], w, 1, out);
}

int rewl_export_window_observables(rewl_engine* e, int32_t ii, int32_t w, double* out)
{
    if (window_index(e, ii, w) < 0 || !out) return fail(REWL_EINVAL, "bad window or null output");
    cudaSetDevice(e->desc.device);
    const InstDev& I = e->inst[ii].dev;
    return export_obs(e, ii, I.first_slot + w * I.R, I.R, out);
}

int rewl_export_walker(rewl_engine* e, int32_t w, int8_t* dofs, double* state, uint64_t* counts, double* logdos, uint64_t* visits)
{
    if (!valid_walker(e, w)) return fail(REWL_EINVAL, "walker %d out of range", w);
    cudaSetDevice(e->desc.device);
    const int ii = e->h_slot_inst[w];
    const InstDev& I = e->inst[ii].dev;
    int32_t cfg, flav;
    CUDA_TRY(cudaMemcpyAsync(&cfg, e->slot_cfg.p + w, 4, cudaMemcpyDeviceToHost, e->stream));
    CUDA_TRY(cudaMemcpyAsync(&flav, e->slot_flavour.p + w, 4, cudaMemcpyDeviceToHost, e->stream));
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    if (dofs) CUDA_TRY(cudaMemcpyAsync(dofs, e->spins.p + e->h_cfg_off[cfg], I.ndof, cudaMemcpyDeviceToHost, e->stream));
    int64_t E; int32_t M[3];
    CUDA_TRY(cudaMemcpyAsync(&E, e->cfg_E.p + cfg, 8, cudaMemcpyDeviceToHost, e->stream));
    CUDA_TRY(cudaMemcpyAsync(M, e->cfg_M.p + 3 * cfg, 12, cudaMemcpyDeviceToHost, e->stream));
    const int nb = e->h_slot_nb[w];
    const int64_t off = e->h_slot_tab[w];
    std::vector<int64_t> g(nb); std::vector<uint32_t> h(nb);
    CUDA_TRY(cudaMemcpyAsync(g.data(), e->g.p + off, nb * 8, cudaMemcpyDeviceToHost, e->stream));
    CUDA_TRY(cudaMemcpyAsync(h.data(), e->H.p + off, nb * 4, cudaMemcpyDeviceToHost, e->stream));
    if (visits) CUDA_TRY(cudaMemcpyAsync(visits, e->visits.p + off, nb * 8, cudaMemcpyDeviceToHost, e->stream));
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    if (state) {
        const double Ed = std::ldexp((double)E, -I.escale);
        if (I.model == REWL_MODEL_ISING2D) { state[0] = Ed; state[1] = M[0]; }
        else { state[0] = Ed; state[1] = M[0]; state[2] = M[1]; state[3] = M[2]; state[4] = flav; }
    }
    if (counts) for (int b = 0; b < nb; ++b) counts[b] = h[b];
    if (logdos) for (int b = 0; b < nb; ++b) logdos[b] = (double)g[b] / kLogdosScale;
    return REWL_OK;
}

int rewl_export_window_logdos(rewl_engine* e, int32_t ii, int32_t w, double* out)
{
    const int wi = window_index(e, ii, w);
    if (wi < 0 || !out) return fail(REWL_EINVAL, "bad window or null output");
    cudaSetDevice(e->desc.device);
    const InstDev& I = e->inst[ii].dev;
    return export_rows(e, e->h_wins[wi].nb, 1, out, [&](int b0, int rows, double* to) {
        k_export_logdos<<<(rows + 127) / 128, 128, 0, e->stream>>>(e->ptrs(), I.first_slot + w * I.R, I.R, b0, rows, to);
    });
}

int rewl_export_window_mask(rewl_engine* e, int32_t ii, int32_t w, uint8_t* out)
{
    const int wi = window_index(e, ii, w);
    if (wi < 0 || !out) return fail(REWL_EINVAL, "bad window or null output");
    cudaSetDevice(e->desc.device);
    const WinDev& W = e->h_wins[wi];
    const InstDev& I = e->inst[ii].dev;
    CUDA_TRY(cudaMemcpyAsync(out, e->mask.p + W.mask_off, W.nb, cudaMemcpyDeviceToHost, e->stream));
    std::vector<uint64_t> v((size_t)I.R * W.nb);
    for (int r = 0; r < I.R; ++r)
        CUDA_TRY(cudaMemcpyAsync(v.data() + (size_t)r * W.nb, e->visits.p + e->h_slot_tab[I.first_slot + w * I.R + r], W.nb * 8, cudaMemcpyDeviceToHost, e->stream));
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    if (e->desc.mask_mode == REWL_MASK_VISITED)
        for (int b = 0; b < W.nb; ++b) {
            bool any = false;
            for (int r = 0; r < I.R; ++r) any |= v[(size_t)r * W.nb + b] != 0;
            if (!any) out[b] = 0;
        }
    return REWL_OK;
}

int rewl_window_state(rewl_engine* e, int32_t ii, int32_t w, double* lnf, int32_t* done)
{
    const int wi = window_index(e, ii, w);
    if (wi < 0) return fail(REWL_EINVAL, "bad window");
    cudaSetDevice(e->desc.device);
    int64_t q; int32_t d;
    CUDA_TRY(cudaMemcpyAsync(&q, e->win_lnf.p + wi, 8, cudaMemcpyDeviceToHost, e->stream));
    CUDA_TRY(cudaMemcpyAsync(&d, e->win_done.p + wi, 4, cudaMemcpyDeviceToHost, e->stream));
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    if (lnf) *lnf = (double)q / kLogdosScale;
    if (done) *done = d;
    return REWL_OK;
}

int rewl_global_logdos(rewl_engine* e, int32_t ii, int32_t half_spectrum, double* energies, double* logdos, int32_t* count)
{
    if (!e || ii < 0 || ii >= (int)e->inst.size() || !count) return fail(REWL_EINVAL, "bad arguments");
    const HostInst& H = e->inst[ii];
    std::vector<std::vector<double>> Es, Gs;
    for (int w = 0; w < H.d.num_windows; ++w) {
        const int nb = H.wins[w].nb;
        std::vector<double> g(nb); std::vector<uint8_t> m(nb);
        int rc = rewl_export_window_logdos(e, ii, w, g.data());
        if (!rc) rc = rewl_export_window_mask(e, ii, w, m.data());
        if (rc) return rc;
        std::vector<double> ee, gg;
        for (int b = 0; b < nb; ++b)
            if (m[b]) { ee.push_back(H.wmin[w] + H.bw * b); gg.push_back(g[b]); }
        Es.push_back(ee); Gs.push_back(gg);
    }
    std::vector<double> fe, fg;
    int rc = concatenate(Es, Gs, fe, fg);
    if (rc) return rc;
    const double states = H.dev.model == REWL_MODEL_ISING2D ? 2.0 : 4.0;
    const double shift = normalisation_shift(fg, states, (double)H.dev.N, half_spectrum != 0);
    if ((int)fe.size() > *count) { *count = (int)fe.size(); return fail(REWL_EINVAL, "output capacity too small (%zu needed)", fe.size()); }
    for (size_t k = 0; k < fe.size(); ++k) { if (energies) energies[k] = fe[k]; if (logdos) logdos[k] = fg[k] + shift; }
    *count = (int)fe.size();
    return REWL_OK;
}

// Observables on the concatenated energy axis (the energies of rewl_global_logdos): every
// window's count-weighted replica average (rewl_export_window_observables) is combined across
// the windows that hold an energy by the reference's running mean
// average_two_windows(final, window, overlapping_windows, 1)
// (src/util/concatenate_rewl_tables.hpp:43-49, 241-256), in window order.
int rewl_concatenate_windows(int32_t num_windows, const int32_t* sizes, const double* energies, const double* logdos,
                             int32_t num_obs, const double* obs, double states_per_site, int64_t system_size,
                             int32_t half_spectrum, int32_t match, double* out_energies, double* out_logdos,
                             double* out_obs, int32_t* count)
{
    if (num_windows < 1 || !sizes || !energies || !logdos || !count || system_size < 1 || !(states_per_site > 0) ||
        num_obs < 0 || (num_obs > 0 && !obs))
        return fail(REWL_EINVAL, "bad arguments");
    if (match != REWL_MATCH_DERIVATIVE && match != REWL_MATCH_REFERENCE) return fail(REWL_EINVAL, "bad match rule");
    std::vector<std::vector<double>> Es(num_windows), Gs(num_windows), Os(num_obs > 0 ? num_windows : 0);
    size_t off = 0;
    for (int w = 0; w < num_windows; ++w) {
        if (sizes[w] < 2) return fail(REWL_EINVAL, "window %d has fewer than 2 rows", w);
        Es[w].assign(energies + off, energies + off + sizes[w]);
        Gs[w].assign(logdos + off, logdos + off + sizes[w]);
        if (num_obs > 0) Os[w].assign(obs + off * num_obs, obs + (off + sizes[w]) * num_obs);
        off += (size_t)sizes[w];
    }
    std::vector<double> fe, fg, fo;
    int rc = concatenate(Es, Gs, fe, fg, match == REWL_MATCH_REFERENCE, num_obs > 0 ? &Os : nullptr, num_obs, &fo);
    if (rc) return rc;
    if ((int64_t)fe.size() > *count) { *count = (int32_t)fe.size(); return fail(REWL_EINVAL, "output capacity too small (%zu needed)", fe.size()); }
    const double shift = normalisation_shift(fg, states_per_site, (double)system_size, half_spectrum != 0);
    for (size_t k = 0; k < fe.size(); ++k) {
        if (out_energies) out_energies[k] = fe[k];
        if (out_logdos) out_logdos[k] = fg[k] + shift;
    }
    if (out_obs && num_obs > 0) std::copy(fo.begin(), fo.end(), out_obs);
    *count = (int32_t)fe.size();
    return REWL_OK;
}

int rewl_global_observables(rewl_engine* e, int32_t ii, double* obs, int32_t* count)
{
    if (!e || ii < 0 || ii >= (int)e->inst.size() || !count) return fail(REWL_EINVAL, "bad arguments");
    if (!e->obs.p) return fail(REWL_ESTATE, "the engine was created without observables (rewl_batch_desc.observables)");
    const HostInst& H = e->inst[ii];
    const int cols = obs_columns(H.d.model, e->desc.observables == 2) + 1;
    const bool half = H.d.model != REWL_MODEL_ISING2D && H.d.energy_max <= 0.0;
    int n = 0;
    int rc = rewl_global_logdos(e, ii, half ? 1 : 0, nullptr, nullptr, &n);
    if (rc && n == 0) return rc;
    std::vector<double> E(n);
    if ((rc = rewl_global_logdos(e, ii, half ? 1 : 0, E.data(), nullptr, &n))) return rc;
    if (n > *count) { *count = n; return fail(REWL_EINVAL, "output capacity too small (%d rows needed)", n); }
    // running means keyed by the global bin index
    std::vector<double> mean;
    std::vector<int64_t> key0;
    std::vector<int> nwin;
    int64_t kmin = INT64_MAX, kmax = INT64_MIN;
    for (int w = 0; w < H.d.num_windows; ++w) {
        kmin = std::min<int64_t>(kmin, H.wins[w].gblo);
        kmax = std::max<int64_t>(kmax, H.wins[w].gblo + H.wins[w].nb);
    }
    mean.assign((size_t)(kmax - kmin) * cols, 0.0);
    nwin.assign((size_t)(kmax - kmin), 0);
    for (int w = 0; w < H.d.num_windows; ++w) {
        const int nb = H.wins[w].nb;
        std::vector<double> o((size_t)nb * cols);
        std::vector<uint8_t> m(nb);
        if ((rc = rewl_export_window_observables(e, ii, w, o.data())) || (rc = rewl_export_window_mask(e, ii, w, m.data())))
            return rc;
        for (int b = 0; b < nb; ++b) {
            if (!m[b]) continue;
            const size_t k = (size_t)(H.wins[w].gblo + b - kmin);
            const int c = nwin[k];
            for (int j = 0; j < cols; ++j) {
                double& v = mean[k * cols + j];
                v = c == 0 ? o[(size_t)b * cols + j] : ((double)c * v + o[(size_t)b * cols + j]) / (double)(c + 1);
            }
            ++nwin[k];
        }
    }
    for (int r = 0; r < n; ++r) {
        const int64_t k = (int64_t)std::llround((E[r] - H.d.energy_min) / H.bw) - kmin;
        if (k < 0 || k >= kmax - kmin || nwin[k] == 0) return fail(REWL_ESTATE, "energy %g has no window observables", E[r]);
        for (int j = 0; j < cols; ++j) obs[(size_t)r * cols + j] = mean[(size_t)k * cols + j];
    }
    *count = n;
    return REWL_OK;
}

namespace {
std::vector<std::string> split_names(const char* names)
{
    std::vector<std::string> v;
    if (!names) return v;
    std::stringstream ss(names);
    std::string line;
    while (std::getline(ss, line, '\n'))
        if (!line.empty()) v.push_back(line);
    return v;
}

// '#' header lines naming the columns (first_cols, then names), as the reference's writers do
void column_header(std::ofstream& f, const char* title, const std::vector<std::string>& first_cols,
                   const std::vector<std::string>& names)
{
    f << "# " << title;
    int col = 0;
    for (const auto& c : first_cols) f << "\n#    " << ++col << ": " << c;
    for (const auto& c : names) f << "\n#    " << ++col << ": " << c;
    f << "\n#\n";
}

int write_table(const char* dir, const char* stem, const char* file_string, const char* header, const char* title,
                const std::vector<std::string>& first_cols, const char* names, int32_t rows, int32_t cols,
                const double* a, const double* b, double scale, const double* values)
{
    if (!dir || !file_string || rows < 1 || cols < 0 || !a || (cols > 0 && !values))
        return fail(REWL_EINVAL, "bad arguments");
    const std::filesystem::path path = std::filesystem::path(dir) / (std::string(stem) + "-" + file_string + ".txt");
    std::ofstream f(path);
    if (!f) return fail(REWL_EINVAL, "cannot open %s for writing", path.string().c_str());
    if (header) f << header;
    column_header(f, title, first_cols, split_names(names));
    f << std::setprecision(std::numeric_limits<double>::digits10) << std::scientific;
    for (int32_t r = 0; r < rows; ++r) {
        f << a[r] / scale << ",";
        if (b) f << b[r] / scale << (cols > 0 ? "," : "");
        for (int32_t c = 0; c < cols; ++c) f << values[(size_t)r * cols + c] << (c + 1 < cols ? "," : "");
        if (r + 1 < rows) f << "\n";
    }
    return f.good() ? REWL_OK : fail(REWL_EINVAL, "write to %s failed", path.string().c_str());
}
} // namespace

// Text formats of the reference's writers (comma-delimited rows, src/Simulation/main_headers.hpp:18;
// '#' header lines; std::scientific with 15 digits): write_microcanonical_observables
// (src/util/write_microcanonical_observables.hpp:16-65), write_observables_to_file
// (src/Thermodynamics/write_self_averaged_observables.hpp:15-59), write_nonlinear_obs_to_file
// (src/Thermodynamics/write_nonlinear_observables.hpp:13-57).
int rewl_write_microcanonical(const char* dir, const char* file_string, const char* header, const char* names,
                              int32_t num_bins, int32_t num_obs, double system_size, const double* energies,
                              const double* logdos, const double* obs)
{
    if (!logdos || !(system_size > 0)) return fail(REWL_EINVAL, "bad arguments");
    return write_table(dir, "microcanonical_observables", file_string, header, "Intensive Observable Names by Column",
                       {"Energy", "logDoS"}, names, num_bins, num_obs, energies, logdos, system_size, obs);
}

int rewl_write_self_averaged(const char* dir, const char* file_string, const char* header, const char* names,
                             int32_t num_T, int32_t num_cols, const double* temperatures, const double* rows)
{
    return write_table(dir, "self_averaged_observables", file_string, header, "Intensive Observable Names by Column",
                       {"Temperature"}, names, num_T, num_cols, temperatures, nullptr, 1.0, rows);
}

int rewl_write_nonlinear(const char* dir, const char* file_string, const char* header, const char* names,
                         int32_t num_T, int32_t num_cols, const double* temperatures, const double* rows)
{
    return write_table(dir, "nonlinear_observables", file_string, header,
                       "Intensive Nonlinear Observable Names by Column", {"Temperature"}, names, num_T, num_cols,
                       temperatures, nullptr, 1.0, rows);
}

// The reference's post-processing of one instance (src/Simulation/main.cpp:241-365): concatenated,
// normalised ln g and observables -> microcanonical file; canonical thermodynamics over the
// temperature ladder (GPU, FP64) -> self-averaged file; susceptibilities and cumulants ->
// nonlinear file.  Without observables the files carry the energy columns only.
int rewl_write_outputs(rewl_engine* e, int32_t ii, const char* dir, const char* file_string, const char* header,
                       double Tmin, double Tmax, int32_t num_T)
{
    if (!e || ii < 0 || ii >= (int)e->inst.size() || !dir || !file_string || num_T < 1) return fail(REWL_EINVAL, "bad arguments");
    const HostInst& H = e->inst[ii];
    const bool ising = H.d.model == REWL_MODEL_ISING2D;
    const bool half = !ising && H.d.energy_max <= 0.0;
    int n = 0;
    rewl_global_logdos(e, ii, half ? 1 : 0, nullptr, nullptr, &n);
    std::vector<double> E(n), G(n);
    int rc = rewl_global_logdos(e, ii, half ? 1 : 0, E.data(), G.data(), &n);
    if (rc) return rc;
    const bool corr = e->desc.observables == 2;
    const int cols = e->obs.p ? obs_columns(H.d.model, corr) + 1 : 0;
    std::vector<double> O((size_t)n * std::max(cols, 1));
    if (cols && (rc = rewl_global_observables(e, ii, O.data(), &n))) return rc;
    // Obs::string_names (ising2d_observables.hpp:40-46, ashkin_teller2d_observables.hpp:64-82)
    const char* sys_names = !cols ? "" : ising
        ? (corr ? "Magnetization\nMagnetization2\nMagnetization4\nG(qmin)\nCounts per Bin"
                : "Magnetization\nMagnetization2\nMagnetization4\nCounts per Bin")
        : (corr ? "Sigma Mag\nSigma Mag2\nSigma Mag4\nSigma G(qmin)\nTau Mag\nTau Mag2\nTau Mag4\nTau G(qmin)\n"
                  "Phi\nPhi2\nPhi4\nPhi G(qmin)\nBaxter\nBaxter2\nBaxter4\nBaxter G(qmin)\nCounts per Bin"
                : "Sigma Mag\nSigma Mag2\nSigma Mag4\nTau Mag\nTau Mag2\nTau Mag4\nPhi\nPhi2\nPhi4\nBaxter\nBaxter2\nBaxter4\nCounts per Bin");
    const double N = (double)H.dev.N;
    if ((rc = rewl_write_microcanonical(dir, file_string, header, sys_names, n, cols, N, E.data(), G.data(), O.data())))
        return rc;
    std::vector<double> T(num_T), rows((size_t)num_T * (5 + cols));
    rc = rewl_thermodynamics(E.data(), G.data(), cols ? O.data() : nullptr, n, cols, cols - 1, N, Tmin, Tmax, num_T, 1,
                             e->desc.device, T.data(), rows.data());
    if (rc) return fail(rc, "thermodynamics: %s", rewl_thermo_last_error_string());
    const std::string thermal = std::string("Free Energy\nEnergy\nEnergy2\nEntropy\nSpecific Heat") + (cols ? "\n" : "") + sys_names;
    if ((rc = rewl_write_self_averaged(dir, file_string, header, thermal.c_str(), num_T, 5 + cols, T.data(), rows.data())))
        return rc;
    if (!cols) return REWL_OK;
    const int nl = ising ? (corr ? 3 : 2) : (corr ? 12 : 8);
    std::vector<double> nonlin((size_t)num_T * nl);
    if ((rc = rewl_nonlinear_observables(H.d.model, corr ? 1 : 0, rows.data(), num_T, 5 + cols, T.data(), N, nonlin.data())))
        return fail(rc, "nonlinear observables: %s", rewl_thermo_last_error_string());
    // Obs::nonlinear_obs_strings (ising2d_observables.hpp:40-46, ashkin_teller2d_observables.hpp:64-82)
    const char* nl_names = ising
        ? (corr ? "Susceptibility\nBinder Cumulant\nCorrelation Length over L" : "Susceptibility\nBinder Cumulant")
        : (corr ? "Sigma Susceptibility\nSigma Binder Cumulant\nSigma Correlation Length over L\n"
                  "Tau Susceptibility\nTau Binder Cumulant\nTau Correlation Length over L\n"
                  "Baxter Susceptibility\nBaxter Binder Cumulant\nBaxter Correlation Length over L\n"
                  "Phi Susceptibility\nPhi Binder Cumulant\nPhi Correlation Length over L"
                : "Sigma Susceptibility\nSigma Binder Cumulant\nTau Susceptibility\nTau Binder Cumulant\n"
                  "Baxter Susceptibility\nBaxter Binder Cumulant\nPhi Susceptibility\nPhi Binder Cumulant");
    return rewl_write_nonlinear(dir, file_string, header, nl_names, num_T, nl, T.data(), nonlin.data());
}

int rewl_sweep_kernel_time(rewl_engine* e, double* ms, int64_t* launches)
{
    if (!e) return fail(REWL_EINVAL, "null engine");
    cudaSetDevice(e->desc.device);
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    double total = 0;
    for (size_t k = 0; k + 1 < e->ev_used; k += 2) {
        float t = 0;
        CUDA_TRY(cudaEventElapsedTime(&t, e->ev_pool[k], e->ev_pool[k + 1]));
        total += t;
    }
    if (ms) *ms = total + e->graph_sweep_ms;
    if (launches) *launches = e->kernel_launches;
    e->ev_used = 0;
    e->kernel_launches = 0;
    e->graph_sweep_ms = 0;
    return REWL_OK;
}

namespace {
struct SnapPart { void* dev; size_t bytes; };

std::vector<SnapPart> snapshot_parts(rewl_engine* e)
{
    auto P = [](auto& b) { return SnapPart{(void*)b.p, b.n * sizeof(*b.p)}; };
    return {P(e->slot_cfg), P(e->slot_flavour), P(e->slot_sweeps), P(e->slot_draws), P(e->cfg_E), P(e->cfg_M),
            P(e->spins), P(e->g), P(e->H), P(e->visits), P(e->win_lnf), P(e->win_done), P(e->win_oot),
            P(e->win_iter), P(e->win_sweepctr), P(e->stats), P(e->obs)};
}

struct SnapHeader {
    uint64_t magic, bytes, exch_round, sweeps_since_check;
    int64_t sweeps_total, cycles, flat_events, flips_total;
    int32_t direction, nslots, nwin, pad;
};
constexpr uint64_t kSnapMagic = 0x5245574C534E4150ull;   // "REWLSNAP"
} // namespace

int rewl_snapshot_size(const rewl_engine* e, size_t* bytes)
{
    if (!e || !bytes) return fail(REWL_EINVAL, "null argument");
    size_t n = sizeof(SnapHeader);
    for (auto& p : snapshot_parts(const_cast<rewl_engine*>(e))) n += (p.bytes + 15) & ~size_t(15);
    *bytes = n;
    return REWL_OK;
}

int rewl_snapshot(rewl_engine* e, void* buffer, size_t bytes)
{
    size_t need = 0;
    if (int rc = rewl_snapshot_size(e, &need)) return rc;
    if (!buffer || bytes < need) return fail(REWL_EINVAL, "snapshot buffer too small (%zu bytes needed)", need);
    cudaSetDevice(e->desc.device);
    SnapHeader h{kSnapMagic, need, e->exch_round, e->sweeps_since_check, e->sweeps_total, e->cycles, e->flat_events,
                 e->flips_total, e->direction, e->nslots, e->nwin_total, 0};
    std::memcpy(buffer, &h, sizeof h);
    char* dst = static_cast<char*>(buffer) + sizeof h;
    for (auto& p : snapshot_parts(e)) {
        if (p.bytes) CUDA_TRY(cudaMemcpyAsync(dst, p.dev, p.bytes, cudaMemcpyDeviceToHost, e->stream));
        dst += (p.bytes + 15) & ~size_t(15);
    }
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    return REWL_OK;
}

int rewl_restore(rewl_engine* e, const void* buffer, size_t bytes)
{
    size_t need = 0;
    if (int rc = rewl_snapshot_size(e, &need)) return rc;
    if (!buffer || bytes < need) return fail(REWL_EINVAL, "snapshot buffer too small (%zu bytes needed)", need);
    SnapHeader h;
    std::memcpy(&h, buffer, sizeof h);
    if (h.magic != kSnapMagic || h.bytes != need || h.nslots != e->nslots || h.nwin != e->nwin_total)
        return fail(REWL_EINVAL, "snapshot does not match this engine's layout");
    cudaSetDevice(e->desc.device);
    const char* src = static_cast<const char*>(buffer) + sizeof h;
    for (auto& p : snapshot_parts(e)) {
        if (p.bytes) CUDA_TRY(cudaMemcpyAsync(p.dev, src, p.bytes, cudaMemcpyHostToDevice, e->stream));
        if (p.dev == (void*)e->win_lnf.p)          // the restored ln f values bound the launch size
            for (size_t k = 0; k < p.bytes / 8; ++k) {
                int64_t v;
                std::memcpy(&v, src + 8 * k, 8);
                raise_lnf_bound(e, v);
            }
        src += (p.bytes + 15) & ~size_t(15);
    }
    const unsigned long long xr[2] = {h.exch_round, 0};
    CUDA_TRY(cudaMemcpyAsync(e->xround.p, xr, sizeof xr, cudaMemcpyHostToDevice, e->stream));
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    e->exch_round = h.exch_round; e->sweeps_since_check = h.sweeps_since_check; e->sweeps_total = h.sweeps_total;
    e->cycles = h.cycles; e->flat_events = h.flat_events; e->flips_total = h.flips_total; e->direction = h.direction;
    return REWL_OK;
}

// Autotuner: for every launch group with more than one admissible shape (walkers per warp 1, 2
// or 4 for the bin-tracking kernel, warps per block 1, 2, 4 or 8, within what the descriptor
// fixes), time sweeps of that group alone in each shape and keep the fastest.  The trials run
// on the live state, which is saved before and restored after, so tuning leaves the simulation
// exactly where it was; a walker's trajectory does not depend on the shape.
int rewl_autotune(rewl_engine* e, int32_t sweeps)
{
    if (!e || sweeps < 0) return fail(REWL_EINVAL, "bad arguments");
    if (e->fused) { e->tuned = true; return REWL_OK; }     // one walker per warp, grid sized to residency
    cudaSetDevice(e->desc.device);
    size_t bytes = 0;
    if (int rc = rewl_snapshot_size(e, &bytes)) return rc;
    std::vector<char> snap;
    try {
        snap.resize(bytes);
    } catch (const std::bad_alloc&) {
        return fail(REWL_ENOMEM, "autotune: no host memory for the %zu-byte state copy", bytes);
    }
    if (int rc = rewl_snapshot(e, snap.data(), bytes)) return rc;
    const int64_t l0 = e->launches_total, k0 = e->kernel_launches;
    cudaEvent_t a = nullptr, b = nullptr;
    int rc = REWL_OK;
    auto ck = [&](cudaError_t ce) {
        if (ce != cudaSuccess && rc == REWL_OK) rc = fail(REWL_EDEVICE, "autotune: %s", cudaGetErrorString(ce));
        return rc == REWL_OK;
    };
    ck(cudaEventCreate(&a));
    ck(cudaEventCreate(&b));
    const DevPtrs P = e->ptrs();
    for (auto& l : e->launches) {
        if (rc) break;
        int64_t dof = 0;
        for (int s : l.slots) dof += e->inst[e->h_slot_inst[s]].dev.ndof;
        // about 2e7 attempted flips of the group per trial, at least one sweep
        const int ts = std::min(max_launch_sweeps(e),
                                sweeps > 0 ? sweeps
                                           : (int)std::max<int64_t>(1, std::min<int64_t>(e->desc.sweeps_per_exchange,
                                                                                          20000000 / std::max<int64_t>(1, dof))));
        std::vector<std::pair<int, int>> cand;
        const int planned = l.walkers_per_warp, nsm = sm_count(e);
        auto shape = [&](int G, int W) {
            if (l.bins) shape_bins(e, l, nsm, G);
            l.wpb = W;
            return !l.bins || l.walkers_per_warp == G;
        };
        std::pair<int, int> pick{planned, l.wpb};
        // the bin-tracking kernel takes at most 4 warps per block (its launch bounds); 4 walkers
        // per warp is left to the planner's rule for very large batches
        for (int G : {1, 2, 4}) {
            if (l.bins ? G > (int)l.slots.size() || (G == 4 && planned < 4) : G > 1) continue;
            if (e->desc.walkers_per_warp && l.bins && G != e->desc.walkers_per_warp) continue;
            if (!shape(G, pick.second)) continue;
            for (int W : {1, 2, 4, 8}) {
                if (l.bins && W > 4) continue;
                if (e->desc.warps_per_block && W != std::min(e->desc.warps_per_block, l.bins ? 4 : 8)) continue;
                if (shape_fits(l, G, W)) cand.push_back({G, W});
            }
        }
        shape(pick.first, pick.second);
        if (cand.size() < 2) continue;
        float best = FLT_MAX;
        for (const auto& c : cand) {
            shape(c.first, c.second);
            if ((rc = at_carveout(e, l))) break;
            if ((rc = launch_group(e, l, e->stream, ts, P))) break;         // warm-up
            if (!ck(cudaEventRecord(a, e->stream))) break;
            if ((rc = launch_group(e, l, e->stream, ts, P))) break;
            if (!ck(cudaEventRecord(b, e->stream)) || !ck(cudaEventSynchronize(b))) break;
            float ms = 0;
            if (!ck(cudaEventElapsedTime(&ms, a, b))) break;
            if (ms < best) { best = ms; pick = c; }
        }
        shape(pick.first, pick.second);
        if (int r2 = at_carveout(e, l)) if (rc == REWL_OK) rc = r2;
    }
    if (a) cudaEventDestroy(a);
    if (b) cudaEventDestroy(b);
    if (rc == REWL_OK) rc = check_device_error(e);
    const int rr = rewl_restore(e, snap.data(), bytes);
    e->launches_total = l0;
    e->kernel_launches = k0;
    e->drop_graph();
    e->tuned = true;
    return rc ? rc : rr;
}

int rewl_launch_shapes(rewl_engine* e, int32_t* shapes, int32_t* count)
{
    if (!e || !count) return fail(REWL_EINVAL, "bad arguments");
    const int n = (int)e->launches.size();
    if (shapes && *count >= n)
        for (int i = 0; i < n; ++i) {
            const Launch& l = e->launches[i];
            shapes[4 * i] = l.model; shapes[4 * i + 1] = l.bins ? 1 : 0;
            shapes[4 * i + 2] = l.bins ? l.walkers_per_warp : 1; shapes[4 * i + 3] = l.wpb;
        }
    *count = n;
    return REWL_OK;
}

int rewl_get_stream(rewl_engine* e, void** stream)
{
    if (!e || !stream) return fail(REWL_EINVAL, "null argument");
    *stream = (void*)e->stream;
    return REWL_OK;
}

} // extern "C"
