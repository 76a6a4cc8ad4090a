// Kernels and launch templates of the explicit step, shared by the two
// translation units that compile them: nicr_step.cu (the drop-in form,
// nvcc -fmad=false, bit-identical to the reference) and nicr_step_fast.cu
// (the reciprocal form, compiled with FMA contraction). Everything here has
// internal linkage, so each unit holds its own instances of what it uses.
#pragma once
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <set>
#include <utility>
#include <vector>
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include "nicr_kernels.h"
#include "nicr_physics.h"

namespace nicr {

// Dynamic shared memory above 48 KB is opted into per kernel and per device,
// once (setting it again is harmless, skipping it on a second device is not).
static void ensure_smem_attr(const void* kernel, int bytes) {
    static std::mutex mu;
    static std::set<std::pair<const void*, int>> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if (done.insert({kernel, dev}).second)
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

namespace {

__device__ __forceinline__ int wrapi(int v, int n) {
    v %= n;
    return v < 0 ? v + n : v;
}

// Warp + block reduction of double-double values (fixed order => deterministic).
__device__ __forceinline__ DD shfl_dd(DD v, int off) {
    DD r;
    r.hi = __shfl_down_sync(0xffffffffu, v.hi, off);
    r.lo = __shfl_down_sync(0xffffffffu, v.lo, off);
    return r;
}
template <int N>
__device__ void block_reduce_dd(DD (&v)[N], long long& cnt, DD* sdd, long long* scnt) {
    const int lane = threadIdx.x & 31;
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int nthreads = blockDim.x * blockDim.y * blockDim.z;
    const int w = tid >> 5, nw = (nthreads + 31) >> 5;
    // Most CTAs of a step book nothing, and few warps of the others do: warps
    // without a nonzero value skip their shuffles, CTAs without one everything
    // (a double-double sum with zeros is exact, so the result is the same).
    bool nz = cnt != 0;
    for (int q = 0; q < N; ++q) nz = nz || v[q].hi != 0. || v[q].lo != 0.;
    if (!__syncthreads_or(nz)) return;
    // lanes of a warp are consecutive linear thread ids because blockDim.x is a multiple of 32
    const bool any = __any_sync(0xffffffffu, nz);
    if (any)
        for (int off = 16; off > 0; off >>= 1) {
            for (int q = 0; q < N; ++q) v[q] = dd_add(v[q], shfl_dd(v[q], off));
            cnt += __shfl_down_sync(0xffffffffu, cnt, off);
        }
    if (lane == 0) {
        for (int q = 0; q < N; ++q) sdd[w * N + q] = v[q];
        scnt[w] = any ? cnt : -1;   // -1: nothing from this warp
    }
    __syncthreads();
    if (w == 0) {   // the warps' values by one warp: 3 dependent additions for 8 warps instead of 8
        const bool has = lane < nw && scnt[lane] >= 0;
        for (int q = 0; q < N; ++q) v[q] = has ? sdd[lane * N + q] : DD{0., 0.};
        cnt = has ? scnt[lane] : 0;
        int off = 16;
        while (off >= nw) off >>= 1;
        for (; off > 0; off >>= 1) {
            for (int q = 0; q < N; ++q) v[q] = dd_add(v[q], shfl_dd(v[q], off));
            cnt += __shfl_down_sync(0xffffffffu, cnt, off);
        }
    }
}

// Whether this step must not run: a step of this batch was rejected, or the
// previous one just was (its commit has not run yet, or runs beside this step).
// The words are read where a Blocked is made and waited for where it is tested,
// so a kernel can stage its first planes meanwhile.
struct Blocked {
    int failed;
    unsigned long long key;
    __device__ __forceinline__ Blocked(const StepParams& P, const Status* st)
        : failed(*(const volatile int*)&st->failed),
          key(!P.slab && P.err_slot >= 0 ? *(const volatile unsigned long long*)&st->slot_err[P.err_slot ^ 1] : ERR_NONE) {}
    __device__ __forceinline__ explicit operator bool() const { return failed != 0 || key != ERR_NONE; }
};
__device__ __forceinline__ bool step_blocked(const StepParams& P, const Status* st) { return (bool)Blocked(P, st); }
// What a march pass leaves.
enum MarchEnd { kMarched, kMarchAgain, kMarchBlocked };

// Commits the pending step of parity q, if any, by one CTA: partial sums
// (thread t: partials t, t + nthreads, ...; deterministic), then the budget is
// advanced only when no trial failed (fields swap only on acceptance, 3S:821).
// sdd, scnt: block_reduce_dd's scratch.
__device__ __forceinline__ void commit_pending(const StepPartial* __restrict__ partials, int q_par, DevBudget* budget,
                                               Status* st, DD* sdd, long long* scnt) {
    const int tid = threadIdx.x + blockDim.x * threadIdx.y, nthreads = blockDim.x * blockDim.y;
    const int nblocks = st->pending[q_par];
    if (nblocks == 0) return;
    const unsigned long long key = st->slot_err[q_par];
    __syncthreads();
    if (key != ERR_NONE) {
        if (tid == 0) {
            st->err_key = key;
            st->failed = 1;
            st->failed_step = st->steps_done;
            st->pending[q_par] = 0;
        }
        return;
    }
    DD acc[5] = {{0., 0.}, {0., 0.}, {0., 0.}, {0., 0.}, {0., 0.}};
    long long clipped = 0;
    for (int b = tid; b < nblocks; b += nthreads) {
        for (int q = 0; q < 5; ++q) {
            const DD v{partials[b].s[q][0], partials[b].s[q][1]};
            if (v.hi != 0. || v.lo != 0.) acc[q] = dd_add(acc[q], v);
        }
        clipped += partials[b].clipped;
    }
    block_reduce_dd<5>(acc, clipped, sdd, scnt);
    if (tid == 0) {
        // slots: ckO ckCr clipO clipCr bcO -> budget indices 2 3 4 5 6
        for (int q = 0; q < 5; ++q) {
            DD b{budget->v[2 + q][0], budget->v[2 + q][1]};
            b = dd_add(b, acc[q]);
            budget->v[2 + q][0] = b.hi;
            budget->v[2 + q][1] = b.lo;
        }
        budget->clipped += clipped;
        st->steps_done += 1;
        st->pending[q_par] = 0;
    }
}

// Tile geometry of the fused step kernel.
template <int DIM, int TA, int TB>
struct Tile {
    static constexpr int HA2 = DIM == 3 ? 2 : 0;   // row halo of the o/cr tiles
    static constexpr int HA1 = DIM == 3 ? 1 : 0;   // row halo of the phi/mu/M tiles
    static constexpr int RA2 = TA + 2 * HA2, RB2 = TB + 4;
    static constexpr int RA1 = TA + 2 * HA1, RB1 = TB + 2;
    static constexpr int S2 = RA2 * RB2, S1 = RA1 * RB1;
    // shared memory: o[4], cr[4] (halo 2); p[3] (halo 1); muO, muCr, mo, mc [2] (halo 1)
    static constexpr int SMEM_DOUBLES = 8 * S2 + 3 * S1 + 8 * S1;
    static constexpr int NT = TA * TB;
    static constexpr int SCRATCH_DOUBLES = 32 * (5 * 2 + 1);   // the block reduction's (32 warps x 5 DD + counts)
    static constexpr size_t SMEM_BYTES = (SMEM_DOUBLES + SCRATCH_DOUBLES + 12 * NT) * sizeof(double);   // and the books
    // every thread stages at most two points of each halo tile
    static_assert(2 * NT >= S2 && 2 * NT >= S1, "tile halo larger than two points per thread");
    __device__ static int i2(int a, int b) { return (a + HA2) * RB2 + (b + 2); }
    __device__ static int i1(int a, int b) { return (a + HA1) * RB1 + (b + 1); }
};

// Divisions of the cell arithmetic, as policies the shared arithmetic (lead
// points, cell updates) is written against. Reciprocal (kFast): no divisions;
// that form's expressions use the folded constants of FastC. The exact
// policies return quotients in a carried scale 1/S: up() from an unscaled
// numerator, same() from one in the carried scale, plain() unscaled from
// unscaled; the caller folds S into the constant that multiplies a sum.
//
// DivRun: quotients carried times 2^128 (xdiv_scaled), so a Laplacian's three
// quotients and the faces of a divergence are never scaled back: 4 FP64
// operations per division, 5 from an unscaled numerator, or 2 (TWO below),
// instead of 6. It keeps in `low` the smallest
// 2 * (high word) - 1 of the quotients (zero wraps to the largest), from which
// one comparison at the end of the march tells whether any nonzero quotient
// was subnormal (two integer operations per division instead of five).
// Infinite and NaN quotients reach a trial value and fail its test. A CTA (or
// thread) that saw either marches again with DivExact before it publishes
// anything, so every result is still the IEEE quotient.
constexpr unsigned kLowQuotient = 0x101FFFFDu;   // 2 * 0x080FFFFF - 1: scaled quotients below 2^-894
struct Reciprocal {
    static constexpr bool kFast = true;
    const StepParams& P;
    unsigned& low;   // unused
};
// TWO: every divisor takes two operations (division_in_two; dx, dx^2 and dt of
// the default configurations, 93% of random divisors), instead of four or, from
// an unscaled numerator, five: 256^3 with 8 fields 2720 -> 2356 us per two
// steps, 151 x 101 x 101 static 1204 -> 1090 us per ten.
template <bool TWO>
struct DivRun {
    static constexpr bool kFast = false;
    static constexpr double S = 0x1p-128;
    const StepParams& P;
    unsigned& low;
    __device__ double note(double qs) const {
        low = min(low, 2u * (unsigned)__double2hiint(qs) - 1u);
        return qs;
    }
    __device__ double same(double as, const DivF& d) const { return note(TWO ? xdiv_scaled2(as, d) : xdiv_scaled(as, d)); }
    __device__ double up(double a, const DivC& d) const { return note(TWO ? xdiv_up2(a, d) : xdiv_up(a, d)); }
    __device__ double plain(double a, const DivC& d) const { return __dmul_rn(up(a, d), 0x1p-128); }
    // a quotient that no trial value depends on: infinite and NaN are noted here
    __device__ double plain_checked(double a, const DivC& d) const {
        const double q = plain(a, d);
        if (!isfinite(q)) low = 0;
        return q;
    }
    __device__ double dt() const { return P.dt_s; }
    __device__ double etaK() const { return P.etaK_s; }
};
// exact for every numerator: xdiv, with the IEEE division (an out-of-line
// call) for numerators outside the guarded range; nothing is scaled
struct DivExact {
    static constexpr bool kFast = false;
    static constexpr double S = 1.;
    const StepParams& P;
    unsigned& low;   // unused: every result is exact
    __device__ double same(double a, const DivC& d) const { return xdiv(a, d); }
    __device__ double up(double a, const DivC& d) const { return xdiv(a, d); }
    __device__ double plain(double a, const DivC& d) const { return xdiv(a, d); }
    __device__ double plain_checked(double a, const DivC& d) const { return xdiv(a, d); }
    __device__ double dt() const { return P.dt; }
    __device__ double etaK() const { return P.eta_K; }
};
// The policy of a march pass: 0 the reciprocal form; 1 the drop-in form's
// first pass (exact quotients, out-of-range numerators flagged), 3 the same
// where two operations divide by every run constant; 2 the drop-in form's
// recomputation of a CTA whose first pass raised the flag.
template <int DM> struct DivOf;
template <> struct DivOf<0> { using T = Reciprocal; };
template <> struct DivOf<1> { using T = DivRun<false>; };
template <> struct DivOf<2> { using T = DivExact; };
template <> struct DivOf<3> { using T = DivRun<true>; };
template <int DM> constexpr bool kFirstPass = (DM & 1) != 0;
// The error word a launch with parameters P reports its first failing trial to.
__device__ __forceinline__ unsigned long long* err_word(const StepParams& P, Status* st) {
    return P.err_slot < 0 ? &st->err_key : &st->slot_err[P.err_slot];
}

// eta_trial's range test (3S:514-526); NaN fails it.
__device__ __forceinline__ bool eta_in_range(double v) { return v >= -1.e-12 && v <= 1. + 1.e-12; }

// eta_trial of one field at one cell: v = eta - (dt L_eta)(deta - K lap eta),
// from the centre c, its X neighbours (m: lower, p: upper) and its row (a) and
// column (b) neighbours. cell() gives what all fields of a cell share.
// Reciprocal form: the increment is c (T - 2 W' c^2) - K' lap c with dt L_eta
// folded into T, W' and the weights K' of the neighbour sums, 11 operations
// instead of 21; the sum c + ... is rounded once, as before.
template <int DIM, class Dv>
struct EtaTrial {
    const Dv& dv;
    const StepParams& P;
    double S, phi, T;
    __device__ EtaTrial(const Dv& d, const StepParams& p, double s, double ph) : dv(d), P(p), S(s), phi(ph), T(0.) {
        if constexpr (Dv::kFast) T = fma(p.f.tS, s, fma(p.f.tH, h_fast(ph), -p.f.t1));
    }
    __device__ double operator()(double c, double xm, double xp, double am, double ap, double bm, double bp) const {
        if constexpr (Dv::kFast) {
            const FastC& f = P.f;
            double l = fma(f.e0, c, f.eb * (bp + bm));
            if (DIM == 3) l = fma(f.ea, ap + am, l);
            l = fma(f.ex, xp + xm, l);
            return c - fma(c, fma(-f.e2, c * c, T), -l);
        } else {
            double lap;
            const DivSet& d = P.div;
            if (DIM == 3)
                lap = dv.up(xp - 2. * c + xm, d.dxdx) + dv.up(ap - 2. * c + am, d.dada) + dv.up(bp - 2. * c + bm, d.dbdb);
            else
                lap = dv.up(xp - 2. * c + xm, d.dxdx) + dv.up(bp - 2. * c + bm, d.dbdb);
            const double force = grain_deta(c, S, phi, P.eta_W, P.eta_A) - dv.etaK() * lap;
            return c - P.dt_etaL * force;
        }
    }
};
// The key of the first of n fields (in reference order) whose trial at idx, already stored, fails the range test.
__device__ __forceinline__ unsigned long long eta_fail_key(const double* eta_next, int n, long long nstore,
                                                           long long key_ncells, long long cell) {
    for (int q = 0; q < n; ++q)
        if (!eta_in_range(eta_next[(long long)q * nstore]))
            return ERR_ETA_BASE + (unsigned long long)q * (unsigned long long)key_ncells + (unsigned long long)cell;
    return ERR_NONE;
}

// A thread's budget sums (ckO ckCr clipO clipCr bcO, hi and lo), clipped cells
// and first failing trial, kept out of the registers: few cells touch them,
// and 24 registers across the march made the exact forms spill. Slot q of the
// 12 words lies NT words after slot q - 1, so the threads' slots of one kind
// are neighbours. SharedBook: in shared memory (the step kernel). LocalBook:
// in local memory (the one-pass kernel, whose tile fills shared memory and
// whose chunks are long enough to hide it; in the step kernel its traffic cost
// 8% on the 151 x 101 x 101 grid).
template <int NT>
struct SharedBook {
    double* w;
    __device__ explicit SharedBook(double* base) : w(base) {
        for (int q = 0; q < 11; ++q) w[q * NT] = 0.;   // the clipped count's zero bits too
        key() = ERR_NONE;
    }
    __device__ double& v(int q) { return w[q * NT]; }
    __device__ long long& clipped() { return *reinterpret_cast<long long*>(w + 10 * NT); }
    __device__ unsigned long long& key() { return *reinterpret_cast<unsigned long long*>(w + 11 * NT); }
    __device__ void add(int q, double b) {
        const DD r = dd_add(DD{v(2 * q), v(2 * q + 1)}, b);
        v(2 * q) = r.hi;
        v(2 * q + 1) = r.lo;
    }
    __device__ void clip() { clipped() += 1; }
    __device__ void fail(unsigned long long k) { key() = min(key(), k); }
};
struct LocalBook {
    volatile double w[10];
    volatile long long n;
    volatile unsigned long long k0;
    __device__ LocalBook() {
        for (int q = 0; q < 10; ++q) w[q] = 0.;
        n = 0;
        k0 = ERR_NONE;
    }
    __device__ double v(int q) { return w[q]; }
    __device__ long long clipped() { return n; }
    __device__ unsigned long long key() { return k0; }
    __device__ void add(int q, double b) {
        const DD r = dd_add(DD{w[2 * q], w[2 * q + 1]}, b);
        w[2 * q] = r.hi;
        w[2 * q + 1] = r.lo;
    }
    __device__ void clip() { n = n + 1; }
    __device__ void fail(unsigned long long k) { k0 = min((unsigned long long)k0, k); }
};

struct CenterVals {
    double o, cr, p, hh, muO, muCr, mo, mc;   // hh = h(p), reused by Ck
};

// SLAB instances update the plane range [P.x_lo, P.x_hi) of a slab's stored
// planes and report keys with P's offsets to P's error word; the whole-domain
// instances keep range and keys compile-time.
template <int DIM, int TA, int TB, bool FAST, bool SLAB = false>
struct StepKernel {
    using T = Tile<DIM, TA, TB>;

    // Per-thread in-plane offsets (row*pitch + col, periodic wrap applied once
    // per CTA) of the staging slots this thread fills: slot q = tid + k*NT.
    struct Offs {
        int o2[2];   // radius-2 tile points (o, cr)
        int o1[2];   // radius-1 tile points (phi)
        int gl[2];   // lead points: own cell, then the halo ring point tid (gb)
    };
    __device__ static Offs make_offs(const Grid& g, int a0, int b0) {
        Offs f;
        const int tid = threadIdx.x + TB * threadIdx.y;
        for (int k = 0; k < 2; ++k) {
            int q = tid + k * T::NT;
            f.o2[k] = -1;
            if (q < T::S2) {
                const int a = q / T::RB2 - T::HA2, b = q % T::RB2 - 2;
                f.o2[k] = (DIM == 3 ? wrapi(a0 + a, g.na) : 0) * g.pb + wrapi(b0 + b, g.nb);
            }
            f.o1[k] = -1;
            if (q < T::S1) {
                const int a = q / T::RB1 - T::HA1, b = q % T::RB1 - 1;
                f.o1[k] = (DIM == 3 ? wrapi(a0 + a, g.na) : 0) * g.pb + wrapi(b0 + b, g.nb);
            }
        }
        const int ta = DIM == 3 ? threadIdx.y : 0, tb = threadIdx.x;
        f.gl[0] = (DIM == 3 ? wrapi(a0 + ta, g.na) : 0) * g.pb + wrapi(b0 + tb, g.nb);
        f.gl[1] = -1;
        if (tid < T::S1 - T::NT) {
            int a, b;
            ring_point(tid, a, b);
            f.gl[1] = (DIM == 3 ? wrapi(a0 + a, g.na) : 0) * g.pb + wrapi(b0 + b, g.nb);
        }
        return f;
    }
    // halo ring enumeration: columns -1 and TB over all halo rows, then rows -1 and TA
    __device__ static void ring_point(int hq, int& a, int& b) {
        if (hq < 2 * T::RA1) {
            a = hq / 2 - T::HA1;
            b = (hq & 1) ? TB : -1;
        } else {
            const int r = hq - 2 * T::RA1;
            a = (r / TB) ? TA : -1;
            b = r % TB;
        }
    }

    // Loads plane xg (clamped to [0,nx-1]) of o and cr with a radius-2 halo
    // into a ring slot. The concentration inlet replaces o in plane 0 by
    // layerO before the step (enforce_legacy_layer, 3S:593-596).
    __device__ static void load_oc(const StepParams& P, const double* __restrict__ o,
                                   const double* __restrict__ cr, int xg, double* so, double* scr, const Offs& f) {
        const Grid& g = P.g;
        xg = xg < 0 ? 0 : (xg > g.nx - 1 ? g.nx - 1 : xg);
        const bool inlet = P.inlet && xg == 0;
        const long long base = (long long)xg * g.plane;
        const int tid = threadIdx.x + TB * threadIdx.y;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (f.o2[k] < 0) continue;
            const int q = tid + k * T::NT;
            const long long idx = base + f.o2[k];
            so[q] = inlet ? P.layer_o : __ldg(o + idx);
            scr[q] = __ldg(cr + idx);
        }
    }
    __device__ static void load_p(const StepParams& P, const double* __restrict__ p, int xg, double* sp,
                                  const Offs& f) {
        const Grid& g = P.g;
        xg = xg < 0 ? 0 : (xg > g.nx - 1 ? g.nx - 1 : xg);
        const long long base = (long long)xg * g.plane;
        const int tid = threadIdx.x + TB * threadIdx.y;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (f.o1[k] < 0) continue;
            sp[tid + k * T::NT] = __ldg(p + base + f.o1[k]);
        }
    }

    // Software pipelining of the staging: the loads of a later plane are issued
    // into registers before the arithmetic of the current plane and stored to
    // shared memory after it, so their latency overlaps the computation.
    struct Prefetch {
        double o[2], cr[2], p[2];
        double gbl[2];   // gb at the lead points (own cell, ring point) of the next lead plane
        double s2;       // eta_s2 at the own cell of the next update plane
    };
    // gb at the lead points of plane x (0 when grains are off)
    __device__ static void fetch_gb(const StepParams& P, const double* __restrict__ gb, int x, const Offs& f,
                                    double (&r)[2]) {
        const long long base = (long long)x * P.g.plane;
        r[0] = P.grains ? __ldg(gb + base + f.gl[0]) : 0.;
        r[1] = (P.grains && f.gl[1] >= 0) ? __ldg(gb + base + f.gl[1]) : 0.;
    }
    __device__ static void fetch(const StepParams& P, const double* __restrict__ o, const double* __restrict__ cr,
                                 const double* __restrict__ p, const double* __restrict__ gb,
                                 const double* __restrict__ s2, int xoc, int xp, int xs, bool own, const Offs& f,
                                 Prefetch& r) {
        fetch_gb(P, gb, xp, f, r.gbl);
        r.s2 = (P.phi_eta && own) ? __ldg(s2 + (long long)xs * P.g.plane + f.gl[0]) : 0.;
        const Grid& g = P.g;
        const int xo = xoc < 0 ? 0 : (xoc > g.nx - 1 ? g.nx - 1 : xoc);
        const int xq = xp < 0 ? 0 : (xp > g.nx - 1 ? g.nx - 1 : xp);
        const bool inlet = P.inlet && xo == 0;
        const long long bo = (long long)xo * g.plane, bq = (long long)xq * g.plane;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (f.o2[k] >= 0) {
                r.o[k] = inlet ? P.layer_o : __ldg(o + bo + f.o2[k]);
                r.cr[k] = __ldg(cr + bo + f.o2[k]);
            }
            if (f.o1[k] >= 0) r.p[k] = __ldg(p + bq + f.o1[k]);
        }
    }
    __device__ static void store(const Prefetch& r, double* so, double* scr, double* sp, const Offs& f) {
        const int tid = threadIdx.x + TB * threadIdx.y;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (f.o2[k] >= 0) { so[tid + k * T::NT] = r.o[k]; scr[tid + k * T::NT] = r.cr[k]; }
            if (f.o1[k] >= 0) sp[tid + k * T::NT] = r.p[k];
        }
    }

    // mu and M at tile point (a,b) of real plane x; writes the mu/M slot.
    template <class Dv>
    __device__ static CenterVals lead_core(const Dv& dv, const StepParams& k, bool o_on, const double* som,
                                           const double* so0, const double* sop, const double* scm, const double* sc0,
                                           const double* scp, const double* sp, double* smuO, double* smuCr,
                                           double* smo, double* smc, int a, int b, double gbv) {
        const int c2 = T::i2(a, b), c1 = T::i1(a, b);
        const double oc = so0[c2], cc = sc0[c2];
        const double pc = sp[c1];
        CenterVals v;
        v.o = oc; v.cr = cc; v.p = pc;
        if constexpr (Dv::kFast) {
            // mu = (1-h) A + h B - 2 k lap with the inner sums as chained
            // multiply-adds (no further from 80-bit values than the separate
            // operations), the mobility's bulk factor folded with the GB
            // enhancement; second differences, not weighted neighbour sums, so
            // that mu of a uniform composition carries no rounding of 2 k / dx^2
            const FastC& f = k.f;
            const double hh = h_fast(pc);
            v.hh = hh;
            auto second = [](double m, double c, double p) { return fma(-2., c, p + m); };
            double lapO = f.wb * second(so0[T::i2(a, b - 1)], oc, so0[T::i2(a, b + 1)]);
            double lapC = f.wb * second(sc0[T::i2(a, b - 1)], cc, sc0[T::i2(a, b + 1)]);
            if (DIM == 3) {
                lapO = fma(f.wa, second(so0[T::i2(a - 1, b)], oc, so0[T::i2(a + 1, b)]), lapO);
                lapC = fma(f.wa, second(sc0[T::i2(a - 1, b)], cc, sc0[T::i2(a + 1, b)]), lapC);
            }
            lapO = fma(f.wx, second(som[c2], oc, sop[c2]), lapO);
            lapC = fma(f.wx, second(scm[c2], cc, scp[c2]), lapC);
            const double ao = fma(12000000., oc, fma(3200000., cc, -298432.));
            const double ac = fma(1166528.60789006, cc, fma(3200000., oc, -97045.64));
            const double bo = fma(24000000., oc, fma(-13800000., cc, -8880000.));
            const double bc = fma(14000000., cc, fma(-13800000., oc, 2680000.));
            v.muO = fma(-2. * Phys::ko, lapO, fma(hh, bo, (1. - hh) * ao));
            v.muCr = fma(-2. * Phys::kc, lapC, fma(hh, bc, (1. - hh) * ac));
            const double mbo = fma(f.gbo, gbv, Phys::bmo), mbc = fma(f.gbc, gbv, Phys::bmc);
            // not mbo + h (boo - mbo): in oxide (h = 1) that would leave boo with
            // the rounding of the GB-enhanced mbo, up to 1e4 times larger
            v.mo = o_on ? oc * fma(hh, Phys::boo, (1. - hh) * mbo) : 0.;
            v.mc = cc * fma(hh, Phys::boc, (1. - hh) * mbc);
        } else {
            double lapO, lapC;
            const DivSet& d = k.div;
            if (DIM == 3) {
                lapO = dv.up(sop[c2] - 2. * oc + som[c2], d.dxdx)
                     + dv.up(so0[T::i2(a + 1, b)] - 2. * oc + so0[T::i2(a - 1, b)], d.dada)
                     + dv.up(so0[T::i2(a, b + 1)] - 2. * oc + so0[T::i2(a, b - 1)], d.dbdb);
                lapC = dv.up(scp[c2] - 2. * cc + scm[c2], d.dxdx)
                     + dv.up(sc0[T::i2(a + 1, b)] - 2. * cc + sc0[T::i2(a - 1, b)], d.dada)
                     + dv.up(sc0[T::i2(a, b + 1)] - 2. * cc + sc0[T::i2(a, b - 1)], d.dbdb);
            } else {
                lapO = dv.up(sop[c2] - 2. * oc + som[c2], d.dxdx)
                     + dv.up(so0[T::i2(a, b + 1)] - 2. * oc + so0[T::i2(a, b - 1)], d.dbdb);
                lapC = dv.up(scp[c2] - 2. * cc + scm[c2], d.dxdx)
                     + dv.up(sc0[T::i2(a, b + 1)] - 2. * cc + sc0[T::i2(a, b - 1)], d.dbdb);
            }
            const double hh = h(pc);
            v.hh = hh;
            v.muO = mu_o_local(oc, cc, hh) - 2. * Phys::ko * Dv::S * lapO;
            v.muCr = mu_cr_local(oc, cc, hh) - 2. * Phys::kc * Dv::S * lapC;
            v.mo = o_on ? mobility(oc, hh, gbv, Phys::bmo, Phys::boo, k.gbm1_o) : 0.;
            v.mc = mobility(cc, hh, gbv, Phys::bmc, Phys::boc, k.gbm1_cr);
        }
        smuO[c1] = v.muO; smuCr[c1] = v.muCr; smo[c1] = v.mo; smc[c1] = v.mc;
        return v;
    }
    // The flux divergence, phi force and Ck of the cell at (ta, tb) of plane u
    // (C: plane u, L: plane u+1, pP: phi of plane u-1, leftO/leftCr: its -X
    // face fluxes), before the trial test and the clamps.
    struct CoreOut {
        double onv, crv, pnv, rightO, rightCr, dO, dCr;
    };
    template <class Dv>
    __device__ static CoreOut cell_core(const Dv& dv, const StepParams& k, bool o_on, bool ck_legacy, bool phi_eta,
                                        const CenterVals& C, const CenterVals& L, double pP, double leftO,
                                        double leftCr, double s2u, const double* mO, const double* mC,
                                        const double* mo_, const double* mc_, const double* spu, int c1, int bp,
                                        int bm, int ap, int am) {
        CoreOut r;
        if constexpr (Dv::kFast) {
            // faces without their factor -1/(2 dx): the carried X face too (face_x)
            const FastC& f = k.f;
            r.rightO = (C.mo + L.mo) * (L.muO - C.muO);
            r.rightCr = (C.mc + L.mc) * (L.muCr - C.muCr);
            const double oo = C.o, cc = C.cr, pp = C.p, hh = C.hh;
            double onv = oo, crv;
            {
                const double m0 = mc_[c1], mu0 = mC[c1];
                double t = f.fb * fma(m0 + mc_[bp], mC[bp] - mu0, (mc_[bm] + m0) * (mC[bm] - mu0));
                if (DIM == 3) t = fma(f.fa, fma(m0 + mc_[ap], mC[ap] - mu0, (mc_[am] + m0) * (mC[am] - mu0)), t);
                crv = cc + fma(f.fx, r.rightCr - leftCr, t);
            }
            if (o_on) {
                const double m0 = mo_[c1], mu0 = mO[c1];
                double t = f.fb * fma(m0 + mo_[bp], mO[bp] - mu0, (mo_[bm] + m0) * (mO[bm] - mu0));
                if (DIM == 3) t = fma(f.fa, fma(m0 + mo_[ap], mO[ap] - mu0, (mo_[am] + m0) * (mO[am] - mu0)), t);
                onv = oo + fma(f.fx, r.rightO - leftO, t);
            }
            // phi force: p (p-1) [2W (2p-1) + 30 p (p-1) X], X = foxide - fmetal plus half the eta energy's slope
            const double pq = pp * (pp - 1.);
            double X = fma(oo, fma(6000000., oo, fma(-17000000., cc, -8581568.)),
                           fma(cc, fma(6416735.696054969, cc, 2777045.64), f.x0));
            if (phi_eta) X = fma(s2u, f.hS, fma(f.hH, hh, X));
            const double G = fma(30. * pq, X, fma(4. * Phys::W, pp, -2. * Phys::W));
            double l = fma(f.p0, pp, f.pb * (spu[bp] + spu[bm]));
            if (DIM == 3) l = fma(f.pa, spu[ap] + spu[am], l);
            l = fma(f.px, L.p + pP, l);
            r.pnv = pp + fma(-k.dtL * pq, G, l);
            r.dO = 0.;
            r.dCr = 0.;
            if (ck_legacy) {
                const double hn = h_fast(r.pnv);
                r.dO = f.ckO * fma(Phys::oxideO - onv, hn, -((Phys::oxideO - oo) * hh));
                r.dCr = f.ckCr * fma(Phys::oxideCr - crv, hn, -((Phys::oxideCr - cc) * hh));
                onv += r.dO;
                crv += r.dCr;
            }
            r.onv = onv;
            r.crv = crv;
            return r;
        } else {
        // x faces: the right face of u is the left face of u+1 (same expression);
        // the faces stay in the carried scale, the divergence's numerators too
        const DivSet& d = k.div;
        r.rightO = dv.up(-.5 * (C.mo + L.mo) * (L.muO - C.muO), d.dx);
        r.rightCr = dv.up(-.5 * (C.mc + L.mc) * (L.muCr - C.muCr), d.dx);
        double divO = 0., divCr;
        {
            const double mc0 = mc_[c1], mu0 = mC[c1];
            const double front = dv.up(-.5 * (mc0 + mc_[bp]) * (mC[bp] - mu0), d.db);
            const double back = dv.up(-.5 * (mc_[bm] + mc0) * (mu0 - mC[bm]), d.db);
            if (DIM == 3) {
                const double top = dv.up(-.5 * (mc0 + mc_[ap]) * (mC[ap] - mu0), d.da);
                const double bottom = dv.up(-.5 * (mc_[am] + mc0) * (mu0 - mC[am]), d.da);
                divCr = dv.same(leftCr - r.rightCr, d.dx) + dv.same(bottom - top, d.da) + dv.same(back - front, d.db);
            } else {
                divCr = dv.same(leftCr - r.rightCr, d.dx) + dv.same(back - front, d.db);
            }
        }
        if (o_on) {
            const double m0 = mo_[c1], mu0 = mO[c1];
            const double front = dv.up(-.5 * (m0 + mo_[bp]) * (mO[bp] - mu0), d.db);
            const double back = dv.up(-.5 * (mo_[bm] + m0) * (mu0 - mO[bm]), d.db);
            if (DIM == 3) {
                const double top = dv.up(-.5 * (m0 + mo_[ap]) * (mO[ap] - mu0), d.da);
                const double bottom = dv.up(-.5 * (mo_[am] + m0) * (mu0 - mO[am]), d.da);
                divO = dv.same(leftO - r.rightO, d.dx) + dv.same(bottom - top, d.da) + dv.same(back - front, d.db);
            } else {
                divO = dv.same(leftO - r.rightO, d.dx) + dv.same(back - front, d.db);
            }
        }
        const double oo = C.o, cc = C.cr, pp = C.p;
        double onv = o_on ? oo + dv.dt() * divO : oo;
        double crv = cc + dv.dt() * divCr;
        double lapP;
        if (DIM == 3)
            lapP = dv.up(L.p - 2. * pp + pP, d.dxdx) + dv.up(spu[ap] - 2. * pp + spu[am], d.dada)
                 + dv.up(spu[bp] - 2. * pp + spu[bm], d.dbdb);
        else
            lapP = dv.up(L.p - 2. * pp + pP, d.dxdx) + dv.up(spu[bp] - 2. * pp + spu[bm], d.dbdb);
        const double hpv = 30. * pp * pp * (pp - 1.) * (pp - 1.);
        double fp = Phys::W * (4. * pp * pp * pp - 6. * pp * pp + 2. * pp)
                  + hpv * (foxide(oo, cc) - fmetal(oo, cc)) - 2. * Phys::kp * Dv::S * lapP;
        if (phi_eta) fp += grain_dphi(s2u, pp, k.eta_W, k.eta_A);
        r.pnv = pp - k.dtL * fp;
        r.dO = 0.;
        r.dCr = 0.;
        if (ck_legacy) {
            const double hn = h(r.pnv);
            r.dO = dv.plain(-Phys::ckO * ((Phys::oxideO - onv) * hn - (Phys::oxideO - oo) * C.hh), d.dt);
            r.dCr = dv.plain(-Phys::ckCr * ((Phys::oxideCr - crv) * hn - (Phys::oxideCr - cc) * C.hh), d.dt);
            onv += r.dO;
            crv += r.dCr;
        }
        r.onv = onv;
        r.crv = crv;
        return r;
        }
    }
    // The trial test and the legacy clamps of one cell (3S:790-811), its stores
    // (on, crn, pn: the cell's places) and bookkeeping. Cells whose new o and cr
    // have a high word below 1.0's (in [0, 1), no sign) and a finite phi need
    // none of the tests: one unsigned comparison instead of ten FP64 ones. All
    // others, and cells with Ck increments, take the branch after the stores,
    // which stores again what the clamps change. cell(): the cell's index in
    // reference loop order.
    template <class Book, class CellFn>
    __device__ static void finish_cell(const CoreOut& R, bool bounds_legacy, double* on, double* crn, double* pn,
                                       Book& book, CellFn cell) {
        const unsigned ho = (unsigned)__double2hiint(R.onv), hc = (unsigned)__double2hiint(R.crv),
                       hp = (unsigned)__double2hiint(R.pnv);
        double pnv = R.pnv;
        bool plain;
        if (bounds_legacy) {
            plain = max(ho, hc) < 0x3FF00000u && (hp & 0x7FFFFFFFu) < 0x7FF00000u;
            pnv = pnv > .99999 ? 1. : pnv;
            pnv = pnv < 1.e-5 ? 0. : pnv;
        } else {
            plain = max(ho, hc) < 0x3FE00000u && hp < 0x3FF00000u;   // o, cr < 1/2, phi in [0, 1)
        }
        *on = R.onv;
        *crn = R.crv;
        *pn = pnv;
        if (!plain || R.dO != 0. || R.dCr != 0.) {
            const bool nonfinite = !isfinite(R.onv) || !isfinite(R.crv) || !isfinite(R.pnv);
            bool outside = false;
            if (nonfinite) {
                *pn = R.pnv;
            } else if (bounds_legacy) {
                const double oc = sclamp(R.onv, 0., 1.), ccr = sclamp(R.crv, 0., 1.);
                const double clO = oc - R.onv, clCr = ccr - R.crv;
                if (oc != R.onv || ccr != R.crv) {
                    book.clip();
                    *on = oc;
                    *crn = ccr;
                }
                // adding +-0 to a normalised double-double leaves it unchanged,
                // so zero increments are skipped
                if (clO != 0.) book.add(2, clO);
                if (clCr != 0.) book.add(3, clCr);
            } else {
                outside = R.onv < -1.e-12 || R.crv < -1.e-12 || R.onv + R.crv > 1. + 1.e-12 || R.pnv < -1.e-12 ||
                          R.pnv > 1. + 1.e-12;
            }
            if (nonfinite || outside)
                book.fail((unsigned long long)cell() * 4ull + (nonfinite ? 0ull : 1ull));
            if (R.dO != 0.) book.add(0, R.dO);
            if (R.dCr != 0.) book.add(1, R.dCr);
        }
    }
    // The X face between two cells as the march carries it: the flux in the
    // carried scale (exact forms) or times -2 dx (reciprocal form).
    template <class Dv>
    __device__ static double face_x(const Dv& dv, double m0, double m1, double mu0, double mu1) {
        if constexpr (Dv::kFast) return (m0 + m1) * (mu1 - mu0);
        else return dv.up(-.5 * (m0 + m1) * (mu1 - mu0), dv.P.div.dx);
    }
    // The surface-mobility closure of the O face at X = 0 with bc=mu
    // (left_flux, 3S:621-628): the carried face, and the budget's increment.
    template <class Dv, class Book>
    __device__ static double surface_face(const Dv& dv, const StepParams& P, bool o_on, const CenterVals& C, double gb0,
                                          Book& book) {
        double lf = 0., carry = 0., inc;
        if (o_on) {
            const double mf = mobility(P.surface_c_ref, h(C.p), gb0, Phys::bmo, Phys::boo, P.gbm1_o);
            if constexpr (Dv::kFast) {
                carry = -4. * mf * (P.mu_res - C.muO);
                lf = (2. * mf * (P.mu_res - C.muO)) * P.f.rdx;
            } else {
                carry = dv.up(2. * mf * (P.mu_res - C.muO), P.div.dx);
                lf = carry * Dv::S;
            }
        }
        if constexpr (Dv::kFast) inc = (P.dt * lf) * P.f.rdx;
        else inc = dv.plain_checked(P.dt * lf, P.div.dx);
        book.add(4, inc);
        return carry;
    }
    // One march over the CTA's chunk with the division policy of DM (DivOf).
    // A first pass returns kMarchAgain, without publishing its failure keys or
    // budget partials, when a numerator of the chunk left the guarded range;
    // kMarchBlocked when the step must not run (nothing written).
    template <int DM>
    __device__ static MarchEnd run_body(const StepParams& P, const double* __restrict__ o, const double* __restrict__ cr,
                                    const double* __restrict__ p, const double* __restrict__ gb,
                                    const double* __restrict__ s2, double* __restrict__ on,
                                    double* __restrict__ crn, double* __restrict__ pn,
                                    StepPartial* __restrict__ partials, Status* st, int bx, int by, int bz, int blin) {
        extern __shared__ __align__(16) double smem[];
        double* so = smem;                 // 4 slots x S2
        double* scr = so + 4 * T::S2;      // 4 slots x S2
        double* sp = scr + 4 * T::S2;      // 3 slots x S1
        double* smuO = sp + 3 * T::S1;     // 2 slots x S1
        double* smuCr = smuO + 2 * T::S1;
        double* smo = smuCr + 2 * T::S1;
        double* smc = smo + 2 * T::S1;
        DD* sdd = reinterpret_cast<DD*>(smc + 2 * T::S1);
        long long* scnt = reinterpret_cast<long long*>(sdd + 32 * 5);

        const Grid& g = P.g;
        const int ta = DIM == 3 ? threadIdx.y : 0, tb = threadIdx.x;
        const int a0 = DIM == 3 ? by * TA : 0, b0 = bx * TB;
        const int i0 = (SLAB ? P.x_lo : 0) + bz * P.xchunk;
        const int i1 = min(SLAB ? P.x_hi : g.nx, i0 + P.xchunk);
        const int row = a0 + ta, col = b0 + tb;
        const bool active = (DIM == 3 ? row < g.na : true) && col < g.nb;
        const Blocked blocked(P, st);
        const Offs offs = make_offs(g, a0, b0);

        SharedBook<T::NT> book(smem + T::SMEM_DOUBLES + T::SCRATCH_DOUBLES + ta * TB + tb);

        unsigned low = kFirstPass<DM> && P.div_gate == 1 ? 0u : ~0u;
        const typename DivOf<DM>::T dv{P, low};

        auto slot3 = [](int w) { return ((w % 3) + 3) % 3; };
        // o/cr ring of 4 planes: the plane staged at the top of an iteration
        // (x+2) never overlaps the window x-1..x+1 that slower warps may still
        // be reading in lead(x), so one barrier per plane suffices
        auto oslot = [&](int w) { return so + (w & 3) * T::S2; };
        auto cslot = [&](int w) { return scr + (w & 3) * T::S2; };
        auto pslot = [&](int x) { return sp + slot3(x) * T::S1; };

        // Computes the lead plane x (real plane) over the tile + radius-1 halo.
        auto lead = [&](int x, const double (&gbl)[2]) -> CenterVals {
            const double *som = oslot(x - 1), *so0 = oslot(x), *sop = oslot(x + 1);
            const double *scm = cslot(x - 1), *sc0 = cslot(x), *scp = cslot(x + 1);
            const double* spx = pslot(x);
            double* mO = smuO + (x & 1) * T::S1;
            double* mC = smuCr + (x & 1) * T::S1;
            double* mo_ = smo + (x & 1) * T::S1;
            double* mc_ = smc + (x & 1) * T::S1;
            CenterVals own = lead_core(dv, P, P.o_on != 0, som, so0, sop, scm, sc0, scp, spx, mO, mC, mo_, mc_, ta,
                                       tb, gbl[0]);
            // halo ring points: one per thread for the first S1-NT threads
            static_assert(T::S1 - T::NT <= T::NT, "ring larger than the CTA");
            const int tid = threadIdx.x + TB * threadIdx.y;
            if (offs.gl[1] >= 0) {
                int a, b;
                ring_point(tid, a, b);
                lead_core(dv, P, P.o_on != 0, som, so0, sop, scm, sc0, scp, spx, mO, mC, mo_, mc_, a, b, gbl[1]);
            }
            return own;
        };

        CenterVals C, L;
        double pP, FxO, FxCr;
        // ---- prologue: centre values of the first update plane and its left
        // x-face flux. All planes it reads are requested at once, the march's
        // first prefetch and the words of an earlier rejection with them: a round
        // trip each was waited for before (64^3, 4 planes per chunk: 511 -> 491 us
        // per twenty steps; a 20-domain sweep 2562 -> 2433 us per ten)
        double gb0[2];
        load_oc(P, o, cr, i0 - 1, oslot(i0 - 1), cslot(i0 - 1), offs);
        load_oc(P, o, cr, i0, oslot(i0), cslot(i0), offs);
        load_oc(P, o, cr, i0 + 1, oslot(i0 + 1), cslot(i0 + 1), offs);
        load_p(P, p, i0, pslot(i0), offs);
        fetch_gb(P, gb, i0, offs, gb0);
        double s2u = (P.phi_eta && active) ? __ldg(s2 + (long long)i0 * g.plane + offs.gl[0]) : 0.;
        Prefetch pf;
        if (i0 == 0) {
            if (i0 + 1 <= g.nx - 1) fetch(P, o, cr, p, gb, s2, i0 + 2, i0 + 1, i0 + 1, active, offs, pf);
            __syncthreads();
            if (blocked) return kMarchBlocked;
            C = lead(0, gb0);
            __syncthreads();
            // ghost plane -1: copies of plane 0 (3S:187, 3S:613-615, 3S:616-619)
            const double muOg = (P.bc == 1 && P.o_on) ? 2. * P.mu_res - C.muO : C.muO;
            FxO = face_x(dv, C.mo, C.mo, muOg, C.muO);
            FxCr = face_x(dv, C.mc, C.mc, C.muCr, C.muCr);
            pP = C.p;
        } else {
            load_oc(P, o, cr, i0 - 2, oslot(i0 - 2), cslot(i0 - 2), offs);
            load_p(P, p, i0 - 1, pslot(i0 - 1), offs);
            double gbm[2];
            fetch_gb(P, gb, i0 - 1, offs, gbm);
            if (i0 + 1 <= g.nx - 1) fetch(P, o, cr, p, gb, s2, i0 + 2, i0 + 1, i0 + 1, active, offs, pf);
            __syncthreads();
            if (blocked) return kMarchBlocked;
            const CenterVals Pv = lead(i0 - 1, gbm);
            C = lead(i0, gb0);
            __syncthreads();
            FxO = face_x(dv, Pv.mo, C.mo, Pv.muO, C.muO);
            FxCr = face_x(dv, Pv.mc, C.mc, Pv.muCr, C.muCr);
            pP = Pv.p;
        }

        for (int u = i0; u < i1; ++u) {
            const int x = u + 1;
            double s2n = 0.;
            if (x <= g.nx - 1) {
                // one barrier per plane: it orders this plane's staging before
                // lead(x), and the previous update(u-1) (which read the mu/M
                // slot lead(x) now overwrites) before lead(x)
                store(pf, oslot(x + 1), cslot(x + 1), pslot(x), offs);
                const double gbl[2] = {pf.gbl[0], pf.gbl[1]};
                s2n = pf.s2;
                __syncthreads();
                if (x + 1 <= g.nx - 1 && u + 1 < i1)
                    fetch(P, o, cr, p, gb, s2, x + 2, x + 1, x + 1, active, offs, pf);
                L = lead(x, gbl);
            } else {
                L = C;  // ghost plane nx: Neumann copy of plane nx-1 (mu and M copied too)
                // no staging in this iteration, but update(nx-1) reads the mu/M
                // that lead(nx-1) of other warps wrote in the previous one
                __syncthreads();
            }
            if (active) {
                const double* mO = smuO + (u & 1) * T::S1;
                const double* mC = smuCr + (u & 1) * T::S1;
                const double* mo_ = smo + (u & 1) * T::S1;
                const double* mc_ = smc + (u & 1) * T::S1;
                const double* spu = pslot(u);
                const int c1 = T::i1(ta, tb);
                const int bp = T::i1(ta, tb + 1), bm = T::i1(ta, tb - 1);
                const int ap = T::i1(ta + 1, tb), am = T::i1(ta - 1, tb);
                const long long gidx = (long long)u * g.plane + (long long)row * g.pb + col;
                double leftO = FxO;
                if (u == 0 && P.bc == 1) {
                    leftO = surface_face(dv, P, P.o_on != 0, C, P.grains ? __ldg(gb + gidx) : 0., book);
                }
                if (u == 0 && P.inlet) book.add(4, P.layer_o - __ldg(o + gidx));

                // fluxes, phi force and Ck (3S:761-811)
                const CoreOut R = cell_core(dv, P, P.o_on != 0, P.ck == 0, P.phi_eta != 0, C, L, pP, leftO, FxCr,
                                            s2u, mO, mC, mo_, mc_, spu, c1, bp, bm, ap, am);
                FxO = R.rightO; FxCr = R.rightCr;
                finish_cell(R, P.bounds == 1, on + gidx, crn + gidx, pn + gidx, book, [&]() {
                    return ((long long)u * g.na + row) * g.nb + col + (SLAB ? P.cell_off : 0);
                });
            }
            pP = C.p;
            C = L;
            s2u = s2n;
        }
        const unsigned long long errkey = book.key();
        if (kFirstPass<DM> && __syncthreads_or(low <= kLowQuotient || errkey != ERR_NONE)) return kMarchAgain;
        if (errkey != ERR_NONE) atomicMin(err_word(P, st), errkey);
        DD acc[5];
        long long clipped = book.clipped();
        for (int q = 0; q < 5; ++q) acc[q] = DD{book.v(2 * q), book.v(2 * q + 1)};
        block_reduce_dd<5>(acc, clipped, sdd, scnt);
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            StepPartial& out = partials[blin];
            for (int q = 0; q < 5; ++q) { out.s[q][0] = acc[q].hi; out.s[q][1] = acc[q].lo; }
            out.clipped = clipped;
        }
        return kMarched;
    }

    // One CTA's chunk of a step of nblocks CTAs (this one at blin); with a
    // budget, CTA nblocks commits the previous step instead: a commit in its
    // own launch, or by the step's last CTA, cost 5 us per step between steps
    // of 8 (2D 128^2) to 30 us (64^3). In the drop-in form a chunk whose quotients
    // could not all be certified is marched again with every quotient exact
    // (IEEE division for those), rewriting its trial values, before keys and
    // partials are published.
    __device__ static void run(const StepParams& P, const double* __restrict__ o, const double* __restrict__ cr,
                               const double* __restrict__ p, const double* __restrict__ gb,
                               const double* __restrict__ s2, double* __restrict__ on,
                               double* __restrict__ crn, double* __restrict__ pn,
                               StepPartial* __restrict__ partials, const StepPartial* __restrict__ prev,
                               DevBudget* budget, Status* st, int bx, int by, int bz, int blin, int nblocks) {
        if (!SLAB && budget) {
            if (blin == nblocks) {
                extern __shared__ __align__(16) double smem[];
                DD* sdd = reinterpret_cast<DD*>(smem + T::SMEM_DOUBLES);
                commit_pending(prev, P.err_slot ^ 1, budget, st, sdd, reinterpret_cast<long long*>(sdd + 32 * 5));
                return;
            }
        }
        MarchEnd end;
        if (FAST) {
            end = run_body<0>(P, o, cr, p, gb, s2, on, crn, pn, partials, st, bx, by, bz, blin);
        } else {
            end = P.div_gate == 2 ? run_body<3>(P, o, cr, p, gb, s2, on, crn, pn, partials, st, bx, by, bz, blin)
                                  : run_body<1>(P, o, cr, p, gb, s2, on, crn, pn, partials, st, bx, by, bz, blin);
            if (end == kMarchAgain) {
                __syncthreads();
                run_body<2>(P, o, cr, p, gb, s2, on, crn, pn, partials, st, bx, by, bz, blin);
            }
        }
        if (!SLAB && budget && end != kMarchBlocked && blin == 0 && threadIdx.x == 0 && threadIdx.y == 0)
            st->pending[P.err_slot] = nblocks;
    }
};

template <int DIM, int TA, int TB, int MINB, bool FAST, bool SLAB = false>
__global__ void __launch_bounds__(TA * TB, MINB)
k_step_main(const StepParams P, const double* __restrict__ o, const double* __restrict__ cr,
            const double* __restrict__ p, const double* __restrict__ gb, const double* __restrict__ s2,
            double* __restrict__ on, double* __restrict__ crn, double* __restrict__ pn,
            StepPartial* __restrict__ partials, const StepPartial* __restrict__ prev, DevBudget* budget, Status* st,
            int gx, int gy, int nblocks) {
    const int t = blockIdx.x;
    StepKernel<DIM, TA, TB, FAST, SLAB>::run(P, o, cr, p, gb, s2, on, crn, pn, partials, prev, budget, st, t % gx,
                                             (t / gx) % gy, t / (gx * gy), t, nblocks);
}

constexpr int TA3 = 8, TB3 = 32;    // 3D tile: 8 rows x 32 columns, 256 threads
constexpr int TA2 = 1, TB2 = 128;   // 2D tile: 128 columns

template <int DIM, int TA, int TB>
dim3 step_grid(const StepParams& P) {
    const Grid& g = P.g;
    return dim3((g.nb + TB - 1) / TB, DIM == 3 ? (g.na + TA - 1) / TA : 1, (P.x_hi - P.x_lo + P.xchunk - 1) / P.xchunk);
}

// eta_trial (3S:514-526): v = eta - (dt*L_eta)*(deta - K*lap(eta)); must lie in
// [-1e-12, 1+1e-12]. Writes the trial and the mask of the trial values (the
// next step's gb and eta_s2, identical to rebuild_eta_mask on them).
template <int DIM, int DM>
__device__ __forceinline__ unsigned eta_cell_pass(const StepParams& P, int neta, const double* __restrict__ eta,
                                         const double* __restrict__ s2, const double* __restrict__ p,
                                         double* __restrict__ eta_next, double* __restrict__ gb_next,
                                         double* __restrict__ s2_next, int x, int row, int col,
                                         unsigned long long& errkey) {
    const Grid& g = P.g;
    unsigned low = kFirstPass<DM> && P.div_gate == 1 ? 0u : ~0u;
    const typename DivOf<DM>::T dv{P, low};
    const long long idx = (long long)x * g.plane + (long long)row * g.pb + col;
    const long long cell = ((long long)x * g.na + row) * g.nb + col + P.cell_off;
    const long long ixm = x > 0 ? idx - g.plane : idx, ixp = x < g.nx - 1 ? idx + g.plane : idx;
    const long long rbase = (long long)x * g.plane;
    const long long ibm = rbase + (long long)row * g.pb + (col == 0 ? g.nb - 1 : col - 1);
    const long long ibp = rbase + (long long)row * g.pb + (col == g.nb - 1 ? 0 : col + 1);
    long long iam = idx, iap = idx;
    if (DIM == 3) {
        iam = rbase + (long long)(row == 0 ? g.na - 1 : row - 1) * g.pb + col;
        iap = rbase + (long long)(row == g.na - 1 ? 0 : row + 1) * g.pb + col;
    }
    const EtaTrial<DIM, typename DivOf<DM>::T> trial(dv, P, __ldg(s2 + idx), __ldg(p + idx));
    double Sn = 0., pairs = 0.;
    bool in_range = true;
    for (int q = 0; q < neta; ++q) {
        const double* e = eta + (long long)q * g.nstore;
        const double v = trial(__ldg(e + idx), __ldg(e + ixm), __ldg(e + ixp), __ldg(e + iam), __ldg(e + iap),
                               __ldg(e + ibm), __ldg(e + ibp));
        in_range = in_range && eta_in_range(v);
        eta_next[(long long)q * g.nstore + idx] = v;
        const double sq = v * v;
        pairs += Sn * sq;
        Sn += sq;
    }
    if (!in_range) errkey = min(errkey, eta_fail_key(eta_next + idx, neta, g.nstore, P.key_ncells, cell));
    s2_next[idx] = Sn;
    gb_next[idx] = P.eta_scale * smin(1., 16. * pairs);
    return kFirstPass<DM> && (low <= kLowQuotient || errkey != ERR_NONE);
}
// The cell's eta update with the division policy of the form; in the drop-in
// form a cell whose numerators left the exact-division range is recomputed
// with every quotient exact (its values rewritten, its key taken from the
// recomputation).
template <int DIM, bool FAST>
__device__ __forceinline__ void eta_cell(const StepParams& P, int neta, const double* __restrict__ eta,
                                         const double* __restrict__ s2, const double* __restrict__ p,
                                         double* __restrict__ eta_next, double* __restrict__ gb_next,
                                         double* __restrict__ s2_next, int x, int row, int col,
                                         unsigned long long& errkey) {
    if (FAST) {
        eta_cell_pass<DIM, 0>(P, neta, eta, s2, p, eta_next, gb_next, s2_next, x, row, col, errkey);
        return;
    }
    unsigned long long k = ERR_NONE;
    if (P.div_gate == 2 ? eta_cell_pass<DIM, 3>(P, neta, eta, s2, p, eta_next, gb_next, s2_next, x, row, col, k)
                        : eta_cell_pass<DIM, 1>(P, neta, eta, s2, p, eta_next, gb_next, s2_next, x, row, col, k)) {
        k = ERR_NONE;
        eta_cell_pass<DIM, 2>(P, neta, eta, s2, p, eta_next, gb_next, s2_next, x, row, col, k);
    }
    errkey = min(errkey, k);
}

// Bounds for 5 CTAs/SM: the load-latency-bound per-cell kernel measured 1.13 ms
// vs 1.29 ms unbounded (62 registers, 4/SM) at 256^3 with 8 fields and the
// division of that build, 1.27 ms at 6/SM. At the 48 registers of 5/SM the exact
// form's three passes (div_gate is known at launch only) spill 84 bytes in 3D
// and 192 in 2D, the reciprocal form 48 bytes in 3D.
template <int DIM, bool FAST>
__global__ void __launch_bounds__(256, 5) k_eta_update(const StepParams P, int neta, const double* __restrict__ eta,
                             const double* __restrict__ s2, const double* __restrict__ p,
                             double* __restrict__ eta_next, double* __restrict__ gb_next,
                             double* __restrict__ s2_next, Status* st) {
    if (step_blocked(P, st)) return;
    const Grid& g = P.g;
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = DIM == 3 ? blockIdx.y * blockDim.y + threadIdx.y : 0;
    if (col >= g.nb || row >= g.na) return;
    unsigned long long errkey = ERR_NONE;
    eta_cell<DIM, FAST>(P, neta, eta, s2, p, eta_next, gb_next, s2_next, P.x_lo + blockIdx.z, row, col, errkey);
    if (errkey != ERR_NONE) atomicMin(err_word(P, st), errkey);
}

// X-marching form of the eta update for a compile-time number of fields N:
// each thread owns one (row, col) column of a chunk of planes and keeps
// eta(x-1), eta(x), eta(x+1) of its column in registers, so each field value
// is read from HBM once; the four in-plane neighbours come from L1 (they are
// the neighbouring threads' own loads). All N loads of the next plane are
// issued before the arithmetic of the current plane.
// NCAP is the register capacity; the first n <= NCAP fields are updated (the
// stand-alone kernel instantiates NCAP = n, so the guards fold away). SLAB
// instances take the plane range and key offsets from P; the whole-domain
// instances keep them compile-time (the runtime range cost this kernel's
// schedule 85% at 128 registers).
// One march of a thread's column with the division policy of DM (DivOf);
// returns the flag of numerators outside the exact-division range (first pass).
template <int DIM, int DM, int NCAP, bool SLAB>
__device__ __forceinline__ unsigned eta_march_pass(const StepParams& P, int n, const double* __restrict__ eta,
                                                   const double* __restrict__ p, double* __restrict__ eta_next,
                                                   double* __restrict__ gb_next, double* __restrict__ s2_next,
                                                   int row, int col, int i0, int i1, unsigned long long& errkey) {
    const Grid& g = P.g;
    unsigned low = kFirstPass<DM> && P.div_gate == 1 ? 0u : ~0u;
    const typename DivOf<DM>::T dv{P, low};
    const long long rc = (long long)row * g.pb + col;
    const long long cbm = (long long)row * g.pb + (col == 0 ? g.nb - 1 : col - 1);
    const long long cbp = (long long)row * g.pb + (col == g.nb - 1 ? 0 : col + 1);
    long long cam = rc, cap = rc;
    if (DIM == 3) {
        cam = (long long)(row == 0 ? g.na - 1 : row - 1) * g.pb + col;
        cap = (long long)(row == g.na - 1 ? 0 : row + 1) * g.pb + col;
    }
    double ep[NCAP], ec[NCAP], en[NCAP];
    {
        const long long bm = (long long)(i0 > 0 ? i0 - 1 : 0) * g.plane, b0 = (long long)i0 * g.plane;
#pragma unroll
        for (int q = 0; q < NCAP; ++q) {
            if (q < n) {
                ep[q] = __ldg(eta + (long long)q * g.nstore + bm + rc);
                ec[q] = __ldg(eta + (long long)q * g.nstore + b0 + rc);
            }
        }
    }
    for (int x = i0; x < i1; ++x) {
        const long long base = (long long)x * g.plane;
        const long long bnext = (long long)(x < g.nx - 1 ? x + 1 : x) * g.plane;
#pragma unroll
        for (int q = 0; q < NCAP; ++q)
            if (q < n) en[q] = __ldg(eta + (long long)q * g.nstore + bnext + rc);
        const double phi = __ldg(p + base + rc);
        double S = 0.;
#pragma unroll
        for (int q = 0; q < NCAP; ++q)
            if (q < n) S += ec[q] * ec[q];
        const long long cell = ((long long)x * g.na + row) * g.nb + col + (SLAB ? P.cell_off : 0);
        const EtaTrial<DIM, typename DivOf<DM>::T> trial(dv, P, S, phi);
        double Sn = 0., pairs = 0.;
        bool in_range = true;
#pragma unroll
        for (int q = 0; q < NCAP; ++q) {
            if (q >= n) break;
            const double* e = eta + (long long)q * g.nstore + base;
            double am = 0., ap = 0.;
            if (DIM == 3) { am = __ldg(e + cam); ap = __ldg(e + cap); }
            const double v = trial(ec[q], ep[q], en[q], am, ap, __ldg(e + cbm), __ldg(e + cbp));
            in_range = in_range && eta_in_range(v);
            eta_next[(long long)q * g.nstore + base + rc] = v;
            const double sq = v * v;
            pairs += Sn * sq;
            Sn += sq;
        }
        if (!in_range)
            errkey = min(errkey, eta_fail_key(eta_next + base + rc, n, g.nstore, SLAB ? P.key_ncells : g.ncells, cell));
        s2_next[base + rc] = Sn;
        gb_next[base + rc] = P.eta_scale * smin(1., 16. * pairs);
#pragma unroll
        for (int q = 0; q < NCAP; ++q)
            if (q < n) { ep[q] = ec[q]; ec[q] = en[q]; }
    }
    return kFirstPass<DM> && (low <= kLowQuotient || errkey != ERR_NONE);
}

// X-marching form of the eta update for a compile-time number of fields N:
// each thread owns one (row, col) column of a chunk of planes and keeps
// eta(x-1), eta(x), eta(x+1) of its column in registers, so each field value
// is read from HBM once; the four in-plane neighbours come from L1 (they are
// the neighbouring threads' own loads). All N loads of the next plane are
// issued before the arithmetic of the current plane.
// NCAP is the register capacity; the first n <= NCAP fields are updated (the
// stand-alone kernel instantiates NCAP = n, so the guards fold away). SLAB
// instances take the plane range and key offsets from P; the whole-domain
// instances keep them compile-time (the runtime range cost this kernel's
// schedule 85% at 128 registers). In the drop-in form a column whose
// numerators left the exact-division range is marched again with every
// quotient exact before its key is merged (its trial values rewritten).
template <int DIM, bool FAST, int NCAP, bool SLAB = false>
__device__ __forceinline__ void eta_march_body(const StepParams& P, int n, const double* __restrict__ eta,
                                               const double* __restrict__ p, double* __restrict__ eta_next,
                                               double* __restrict__ gb_next, double* __restrict__ s2_next,
                                               Status* st, int bx, int by, int bz) {
    if (step_blocked(P, st)) return;
    const Grid& g = P.g;
    const int col = bx * blockDim.x + threadIdx.x;
    const int row = DIM == 3 ? by * blockDim.y + threadIdx.y : 0;
    if (col >= g.nb || row >= g.na) return;
    const int i0 = (SLAB ? P.x_lo : 0) + bz * P.xchunk, i1 = min(SLAB ? P.x_hi : g.nx, i0 + P.xchunk);
    unsigned long long errkey = ERR_NONE;
    if (FAST) {
        eta_march_pass<DIM, 0, NCAP, SLAB>(P, n, eta, p, eta_next, gb_next, s2_next, row, col, i0, i1, errkey);
    } else if (P.div_gate == 2 ? eta_march_pass<DIM, 3, NCAP, SLAB>(P, n, eta, p, eta_next, gb_next, s2_next, row, col,
                                                                    i0, i1, errkey)
                               : eta_march_pass<DIM, 1, NCAP, SLAB>(P, n, eta, p, eta_next, gb_next, s2_next, row, col,
                                                                    i0, i1, errkey)) {
        errkey = ERR_NONE;
        eta_march_pass<DIM, 2, NCAP, SLAB>(P, n, eta, p, eta_next, gb_next, s2_next, row, col, i0, i1, errkey);
    }
    if (errkey != ERR_NONE) atomicMin(err_word(P, st), errkey);
}

// 2 CTAs/SM stated in the bounds: the register count stays <= 128 either way,
// but the schedule compiled for it measured 15% faster on B200 (0.58 vs 0.69
// ms at 256^3 with 8 fields, same box); bounds for 3 CTAs/SM spill and lose.
template <int DIM, bool FAST, int N, bool SLAB = false>
__global__ void __launch_bounds__(256, 2)
k_eta_march(const StepParams P, const double* __restrict__ eta, const double* __restrict__ p,
            double* __restrict__ eta_next, double* __restrict__ gb_next, double* __restrict__ s2_next, Status* st) {
    eta_march_body<DIM, FAST, N, SLAB>(P, N, eta, p, eta_next, gb_next, s2_next, st, blockIdx.x, blockIdx.y, blockIdx.z);
}

template <int DIM, bool FAST, int N>
static void launch_eta_march(const StepParams& P, const double* eta, const double* p, double* eta_next,
                             double* gb_next, double* s2_next, Status* st, cudaStream_t stream) {
    const Grid& g = P.g;
    if (DIM == 3) {
        const dim3 grid((g.nb + 31) / 32, (g.na + 7) / 8, (P.x_hi - P.x_lo + P.xchunk - 1) / P.xchunk);
        if (P.slab)   // 3D only
            k_eta_march<3, FAST, N, true><<<grid, dim3(32, 8), 0, stream>>>(P, eta, p, eta_next, gb_next, s2_next, st);
        else
            k_eta_march<3, FAST, N><<<grid, dim3(32, 8), 0, stream>>>(P, eta, p, eta_next, gb_next, s2_next, st);
    } else {
        const dim3 grid((g.nb + 127) / 128, 1, (g.nx + P.xchunk - 1) / P.xchunk);
        k_eta_march<2, FAST, N><<<grid, dim3(128, 1), 0, stream>>>(P, eta, p, eta_next, gb_next, s2_next, st);
    }
}

// Horizontal fusion of the step kernel and the eta march (3D): within a step
// the two are independent (the step kernel reads o, cr, phi, gb, eta_s2 and
// writes the trial o, cr, phi; the eta update reads eta and the current phi
// and writes the next eta, gb, eta_s2), and the step kernel is bound by FP64
// issue while the march waits on HBM. Each CTA draws a ticket and takes the
// step tile or the eta column block the ticket names; the tickets alternate
// between the two kinds while both last, so the SMs run both kinds at once
// and their pipes overlap. The CTAs compute what the separate kernels compute
// (the same bodies; step partial sums at the step kernel's block index).
// Opt-in (NICR_FUSED=1): at 256^3 with 8 fields it measured 1.122 ms per step
// against 1.129 ms for the two launches. Both kernels hold 2 CTAs/SM at 128
// registers and each is bound by the latency its own warps hide; an SM that
// runs one CTA of each gives each kind half the warps, which costs about what
// the overlap gains.
struct FusedStep {
    int n_step, n_eta;     // CTAs of each kind
    int gx_s, gy_s;        // step grid (x, y; z = X chunks)
    int gx_e, gy_e;        // eta march grid (x, y; z = X chunks)
    unsigned* ticket;      // zero at launch
};
template <bool FAST, int N>
__global__ void __launch_bounds__(TA3 * TB3, 2)
k_step_eta(const StepParams P, const FusedStep F, const double* __restrict__ o, const double* __restrict__ cr,
           const double* __restrict__ p, const double* __restrict__ gb, const double* __restrict__ s2,
           double* __restrict__ on, double* __restrict__ crn, double* __restrict__ pn,
           StepPartial* __restrict__ partials, const double* __restrict__ eta, double* __restrict__ eta_next,
           double* __restrict__ gb_next, double* __restrict__ s2_next, Status* st) {
    __shared__ int s_ticket;
    if (threadIdx.x == 0 && threadIdx.y == 0) s_ticket = (int)atomicAdd(F.ticket, 1u);
    __syncthreads();
    const int t = s_ticket, pairs = min(F.n_step, F.n_eta);
    int role, idx;
    if (t < 2 * pairs) {
        role = t & 1;
        idx = t >> 1;
    } else {
        role = F.n_step > F.n_eta ? 0 : 1;
        idx = pairs + (t - 2 * pairs);
    }
    if (role == 0) {
        const int bx = idx % F.gx_s, r = idx / F.gx_s;
        // this launch commits nothing: it leaves its step pending (the one before was flushed)
        if (idx == 0 && threadIdx.x == 0 && threadIdx.y == 0 && !st->failed) st->pending[P.err_slot] = F.n_step;
        StepKernel<3, TA3, TB3, FAST>::run(P, o, cr, p, gb, s2, on, crn, pn, partials, nullptr, nullptr, st, bx,
                                           r % F.gy_s, r / F.gy_s, idx, F.n_step);
    } else {
        const int bx = idx % F.gx_e, r = idx / F.gx_e;
        eta_march_body<3, FAST, N>(P, N, eta, p, eta_next, gb_next, s2_next, st, bx, r % F.gy_e, r / F.gy_e);
    }
}

template <bool FAST, int N>
static void launch_step_eta_n(const StepParams& P, const double* o, const double* cr, const double* p,
                              const double* gb, const double* s2, double* on, double* crn, double* pn,
                              StepPartial* partials, const double* eta, double* eta_next, double* gb_next,
                              double* s2_next, unsigned* ticket, Status* st, cudaStream_t stream, int* nblocks_out) {
    using T = Tile<3, TA3, TB3>;
    const Grid& g = P.g;
    const dim3 gs = step_grid<3, TA3, TB3>(P);
    const dim3 ge((g.nb + 31) / 32, (g.na + 7) / 8, (P.x_hi - P.x_lo + P.xchunk - 1) / P.xchunk);
    FusedStep F;
    F.gx_s = (int)gs.x; F.gy_s = (int)gs.y; F.n_step = (int)(gs.x * gs.y * gs.z);
    F.gx_e = (int)ge.x; F.gy_e = (int)ge.y; F.n_eta = (int)(ge.x * ge.y * ge.z);
    F.ticket = ticket;
    ensure_smem_attr((const void*)k_step_eta<FAST, N>, (int)T::SMEM_BYTES);
    cudaMemsetAsync(ticket, 0, sizeof(unsigned), stream);
    k_step_eta<FAST, N><<<F.n_step + F.n_eta, dim3(TB3, TA3), T::SMEM_BYTES, stream>>>(
        P, F, o, cr, p, gb, s2, on, crn, pn, partials, eta, eta_next, gb_next, s2_next, st);
    if (nblocks_out) *nblocks_out = F.n_step;
}

template <bool FAST>
static void step_eta_prepare(int neta) {
    using T = Tile<3, TA3, TB3>;
    switch (neta) {
#define NICR_FUSED_PREP(n) \
    case n: ensure_smem_attr((const void*)k_step_eta<FAST, n>, (int)T::SMEM_BYTES); break;
        NICR_FUSED_PREP(1) NICR_FUSED_PREP(2) NICR_FUSED_PREP(3) NICR_FUSED_PREP(4) NICR_FUSED_PREP(5)
        NICR_FUSED_PREP(6) NICR_FUSED_PREP(7) NICR_FUSED_PREP(8) NICR_FUSED_PREP(9) NICR_FUSED_PREP(10)
        NICR_FUSED_PREP(11) NICR_FUSED_PREP(12) NICR_FUSED_PREP(13) NICR_FUSED_PREP(14) NICR_FUSED_PREP(15)
        NICR_FUSED_PREP(16)
#undef NICR_FUSED_PREP
        default: break;
    }
}

template <bool FAST>
static bool launch_step_eta_form(const StepParams& P, int neta, const double* o, const double* cr, const double* p,
                                 const double* gb, const double* s2, double* on, double* crn, double* pn,
                                 StepPartial* partials, const double* eta, double* eta_next, double* gb_next,
                                 double* s2_next, unsigned* ticket, Status* st, cudaStream_t stream,
                                 int* nblocks_out) {
    if (P.g.dim != 3 || P.slab) return false;
    switch (neta) {
#define NICR_FUSED_CASE(n)                                                                                   \
    case n:                                                                                                  \
        launch_step_eta_n<FAST, n>(P, o, cr, p, gb, s2, on, crn, pn, partials, eta, eta_next, gb_next, s2_next, \
                                   ticket, st, stream, nblocks_out);                                         \
        return true;
        NICR_FUSED_CASE(1) NICR_FUSED_CASE(2) NICR_FUSED_CASE(3) NICR_FUSED_CASE(4) NICR_FUSED_CASE(5)
        NICR_FUSED_CASE(6) NICR_FUSED_CASE(7) NICR_FUSED_CASE(8) NICR_FUSED_CASE(9) NICR_FUSED_CASE(10)
        NICR_FUSED_CASE(11) NICR_FUSED_CASE(12) NICR_FUSED_CASE(13) NICR_FUSED_CASE(14) NICR_FUSED_CASE(15)
        NICR_FUSED_CASE(16)
#undef NICR_FUSED_CASE
        default: return false;
    }
}

// Dispatch to the compile-time field counts 1..16; false when N is larger.
template <int DIM, bool FAST>
static bool eta_march_dispatch(int neta, const StepParams& P, const double* eta, const double* p, double* eta_next,
                               double* gb_next, double* s2_next, Status* st, cudaStream_t stream) {
    switch (neta) {
#define NICR_ETA_CASE(n) \
    case n: launch_eta_march<DIM, FAST, n>(P, eta, p, eta_next, gb_next, s2_next, st, stream); return true;
        NICR_ETA_CASE(1) NICR_ETA_CASE(2) NICR_ETA_CASE(3) NICR_ETA_CASE(4) NICR_ETA_CASE(5) NICR_ETA_CASE(6)
        NICR_ETA_CASE(7) NICR_ETA_CASE(8) NICR_ETA_CASE(9) NICR_ETA_CASE(10) NICR_ETA_CASE(11) NICR_ETA_CASE(12)
        NICR_ETA_CASE(13) NICR_ETA_CASE(14) NICR_ETA_CASE(15) NICR_ETA_CASE(16)
#undef NICR_ETA_CASE
        default: return false;
    }
}

// TMA-staged form of the eta update (3D, row count a multiple of 8, column
// count a multiple of 32, N <= 16 fields), selected by NICR_ETA_KERNEL=tma.
// Measured at 256^3 with 8 fields it is slower than the register march
// (0.72 vs 0.58 ms reciprocal, 1.31 vs 1.15 ms drop-in): the per-plane
// barrier and the seven shared-memory reads per field leave 16 warps per SM
// latency-bound, where the march runs barrier-free from registers and L1. Each CTA owns an 8 x 32 tile and
// marches along its X chunk; one thread stages every plane of all N fields
// with five tensor copies (cp.async.bulk.tensor, the fields as the fourth
// dimension): the tile, the two halo rows (periodic wrap by coordinate) and
// the two 2-column halo strips, into a four-plane shared-memory ring whose
// slots complete on mbarriers. The copy of plane x+2 is issued while plane x
// is updated, and the threads read the stencil from shared memory, so the
// loads hold no registers and cost one instruction per box. Every x
// coordinate is b0, b0 +- 2, b0 + 32, nb - 2 or 0: a multiple of 2 doubles
// (16 bytes) because nb is a multiple of 32. Waits are bounded: a wait that
// runs out sets st->timeout, and the CTA returns after a bounded wait for its
// copies in flight. The arithmetic is the other forms' (same operand order).
__device__ __forceinline__ unsigned smem_u32(const void* ptr) { return (unsigned)__cvta_generic_to_shared(ptr); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int x, int y, int z, int w,
                                            unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];\n" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
        : "memory");
}

constexpr int kTmaRing = 4;
constexpr long long kTmaWaitLimit = 1LL << 22;   // try_wait rounds before a wait is declared lost

template <int N>
struct TmaStage {
    static constexpr int TA = 8, TB = 32;
    static constexpr int INT = N * TA * TB, ROW = N * TB, COL = N * TA * 2;
    static constexpr int DOUBLES = INT + 2 * ROW + 2 * COL;   // 128-byte multiple for every N
    static constexpr unsigned BYTES = DOUBLES * 8;
    static constexpr size_t SMEM = (size_t)kTmaRing * BYTES + 128;   // + alignment slack
};

template <bool FAST, int N>
__global__ void __launch_bounds__(256, 2)
k_eta_tma(const StepParams P, const __grid_constant__ CUtensorMap m_int, const __grid_constant__ CUtensorMap m_row,
          const __grid_constant__ CUtensorMap m_col, const double* __restrict__ p, double* __restrict__ eta_next,
          double* __restrict__ gb_next, double* __restrict__ s2_next, Status* st) {
    using S = TmaStage<N>;
    constexpr int TA = S::TA, TB = S::TB;
    extern __shared__ unsigned char tma_smem_raw[];
    __shared__ unsigned long long bars[kTmaRing];
    if (step_blocked(P, st)) return;
    const Grid& g = P.g;
    double* ring = reinterpret_cast<double*>(((unsigned long long)tma_smem_raw + 127ull) & ~127ull);
    const int ta = threadIdx.y, tb = threadIdx.x, tid = tb + TB * ta;
    const int a0 = blockIdx.y * TA, b0 = blockIdx.x * TB;
    const int i0 = blockIdx.z * P.xchunk, i1 = min(g.nx, i0 + P.xchunk);
    const int row = a0 + ta, col = b0 + tb;
    const int ytop = a0 == 0 ? g.na - 1 : a0 - 1, ybot = a0 + TA == g.na ? 0 : a0 + TA;
    const int xl = b0 == 0 ? g.nb - 2 : b0 - 2, xr = b0 + TB == g.nb ? 0 : b0 + TB;
    // plane q >= i0 - 1 lives in ring slot (q - i0 + 1) % kTmaRing
    auto slot_of = [&](int q) { return (q - i0 + 1) % kTmaRing; };
    auto stage_of = [&](int q) { return ring + (size_t)slot_of(q) * S::DOUBLES; };
    auto issue = [&](int q) {   // thread 0
        const int xg = q < 0 ? 0 : (q > g.nx - 1 ? g.nx - 1 : q);
        double* s = stage_of(q);
        unsigned long long* bar = &bars[slot_of(q)];
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        mbar_expect_tx(bar, S::BYTES);
        tma_load_4d(s, &m_int, b0, a0, xg, 0, bar);
        tma_load_4d(s + S::INT, &m_row, b0, ytop, xg, 0, bar);
        tma_load_4d(s + S::INT + S::ROW, &m_row, b0, ybot, xg, 0, bar);
        tma_load_4d(s + S::INT + 2 * S::ROW, &m_col, xl, a0, xg, 0, bar);
        tma_load_4d(s + S::INT + 2 * S::ROW + S::COL, &m_col, xr, a0, xg, 0, bar);
    };
    bool ok = true;
    auto wait = [&](int q) {
        const int k = q - i0 + 1;
        const unsigned parity = (unsigned)((k / kTmaRing) & 1);
        unsigned long long* bar = &bars[k % kTmaRing];
        for (long long it = 0; ok && !mbar_try_wait(bar, parity); ++it)
            if (it > kTmaWaitLimit) ok = false;
    };
    if (tid == 0) {
        for (int r = 0; r < kTmaRing; ++r) mbar_init(&bars[r], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    int issued = i0 - 2;   // last plane whose copy was issued
    if (tid == 0) {
        for (int q = i0 - 1; q <= i0 + 1 && q <= i1; ++q) issue(q);
    }
    issued = min(i0 + 1, i1);
    wait(i0 - 1);
    wait(i0);
    const long long own = (long long)row * g.pb + col;
    const int c = ta * TB + tb;   // own point in the tile
    unsigned long long errkey = ERR_NONE;
    int x = i0;
    for (; x < i1; ++x) {
        // all threads finished plane x-1 (the slot of plane x+2 held plane x-2)
        if (__syncthreads_or(!ok)) break;
        if (x + 2 <= i1) {
            if (tid == 0) issue(x + 2);
            issued = x + 2;
        }
        wait(x + 1);
        if (!ok) continue;   // reported at the next barrier
        const double* sm = stage_of(x - 1);
        const double* s0 = stage_of(x);
        const double* sp = stage_of(x + 1);
        const double* top = s0 + S::INT;
        const double* bot = top + S::ROW;
        const double* lft = bot + S::ROW;
        const double* rgt = lft + S::COL;
        const long long base = (long long)x * g.plane;
        const double phi = __ldg(p + base + own);
        double S2 = 0.;
#pragma unroll
        for (int q = 0; q < N; ++q) {
            const double v = s0[q * TA * TB + c];
            S2 += v * v;
        }
        const long long cell = ((long long)x * g.na + row) * g.nb + col;
        unsigned low = ~0u;   // the exact policy divides every quotient exactly
        using Dv = typename DivOf<FAST ? 0 : 2>::T;
        const Dv dv{P, low};
        const EtaTrial<3, Dv> trial(dv, P, S2, phi);
        double Sn = 0., pairs = 0.;
#pragma unroll
        for (int q = 0; q < N; ++q) {
            const int o = q * TA * TB;
            const double c0 = s0[o + c];
            const double am = ta == 0 ? top[q * TB + tb] : s0[o + c - TB];
            const double ap = ta == TA - 1 ? bot[q * TB + tb] : s0[o + c + TB];
            const double bm = tb == 0 ? lft[(q * TA + ta) * 2 + 1] : s0[o + c - 1];
            const double bp = tb == TB - 1 ? rgt[(q * TA + ta) * 2] : s0[o + c + 1];
            const double v = trial(c0, sm[o + c], sp[o + c], am, ap, bm, bp);
            if (!eta_in_range(v))
                errkey = min(errkey, ERR_ETA_BASE + (unsigned long long)q * (unsigned long long)g.ncells + (unsigned long long)cell);
            eta_next[(long long)q * g.nstore + base + own] = v;
            const double sq = v * v;
            pairs += Sn * sq;
            Sn += sq;
        }
        s2_next[base + own] = Sn;
        gb_next[base + own] = P.eta_scale * smin(1., 16. * pairs);
    }
    if (__syncthreads_or(!ok)) {
        // a wait ran out: flag it, give the copies in flight a bounded time to land, leave
        if (tid == 0) {
            atomicOr(&st->timeout, 1);
            for (int q = i0 - 1; q <= issued; ++q) {
                const int k = q - i0 + 1;
                unsigned long long* bar = &bars[k % kTmaRing];
                for (long long it = 0; it <= kTmaWaitLimit && !mbar_try_wait(bar, (unsigned)((k / kTmaRing) & 1)); ++it) {
                }
            }
        }
        __syncthreads();
        return;
    }
    if (errkey != ERR_NONE) atomicMin(err_word(P, st), errkey);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (the
// library links the CUDA runtime statically and not libcuda).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    }
    return fn;
}

// The N eta fields of one buffer as a 4D tensor (columns, rows, planes,
// fields), boxes of bx x by x 1 x bw (bw = N: every field at once).
static bool encode_eta_map(CUtensorMap* m, const Grid& g, int n, const double* eta, unsigned bx, unsigned by,
                           unsigned bw) {
    const auto enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)g.nb, (cuuint64_t)g.na, (cuuint64_t)g.nx, (cuuint64_t)n};
    const cuuint64_t strides[3] = {(cuuint64_t)g.pb * 8, (cuuint64_t)g.plane * 8, (cuuint64_t)g.nstore * 8};
    const cuuint32_t box[4] = {bx, by, 1, bw};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<double*>(eta), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Launches the TMA-staged eta update when the grid allows it; false otherwise.
template <bool FAST, int N>
static bool launch_eta_tma_n(const StepParams& P, const double* eta, const double* p, double* eta_next,
                             double* gb_next, double* s2_next, Status* st, cudaStream_t stream) {
    const Grid& g = P.g;
    CUtensorMap mi, mr, mc;
    if (!encode_eta_map(&mi, g, N, eta, 32, 8, N) || !encode_eta_map(&mr, g, N, eta, 32, 1, N) ||
        !encode_eta_map(&mc, g, N, eta, 2, 8, N))
        return false;
    const size_t smem = TmaStage<N>::SMEM;
    ensure_smem_attr((const void*)k_eta_tma<FAST, N>, (int)smem);
    const dim3 grid(g.nb / 32, g.na / 8, (g.nx + P.xchunk - 1) / P.xchunk);
    k_eta_tma<FAST, N><<<grid, dim3(32, 8), smem, stream>>>(P, mi, mr, mc, p, eta_next, gb_next, s2_next, st);
    return true;
}

template <bool FAST>
static bool launch_eta_tma(int neta, const StepParams& P, const double* eta, const double* p, double* eta_next,
                           double* gb_next, double* s2_next, Status* st, cudaStream_t stream) {
    const Grid& g = P.g;
    if (g.dim != 3 || g.nb % 32 != 0 || g.na % 8 != 0 || g.nb < 32 || neta < 1 || neta > 16) return false;
    if ((reinterpret_cast<unsigned long long>(eta) & 15ull) != 0) return false;
    switch (neta) {
#define NICR_TMA_CASE(n) \
    case n: return launch_eta_tma_n<FAST, n>(P, eta, p, eta_next, gb_next, s2_next, st, stream);
        NICR_TMA_CASE(1) NICR_TMA_CASE(2) NICR_TMA_CASE(3) NICR_TMA_CASE(4) NICR_TMA_CASE(5) NICR_TMA_CASE(6)
        NICR_TMA_CASE(7) NICR_TMA_CASE(8) NICR_TMA_CASE(9) NICR_TMA_CASE(10) NICR_TMA_CASE(11) NICR_TMA_CASE(12)
        NICR_TMA_CASE(13) NICR_TMA_CASE(14) NICR_TMA_CASE(15) NICR_TMA_CASE(16)
#undef NICR_TMA_CASE
        default: return false;
    }
}

// Streaming form of the eta update: each CTA owns a rows x columns tile,
// marches along X and stages every eta plane once (radius-1 halo) in a
// three-plane shared-memory ring, so every field is read from HBM about once.
// S = sum eta_g^2 is rebuilt from the staged centres in g order, which is the
// same arithmetic as rebuild_eta_mask and therefore the same value as eta_s2.
template <int DIM, int TA, int TB, bool FAST>
__global__ void __launch_bounds__(TA * TB)
k_eta_stream(const StepParams P, int neta, const double* __restrict__ eta, const double* __restrict__ p,
             double* __restrict__ eta_next, double* __restrict__ gb_next, double* __restrict__ s2_next,
             Status* st) {
    constexpr int HA = DIM == 3 ? 1 : 0;
    constexpr int RA = TA + 2 * HA, RB = TB + 2, S1 = RA * RB, NT = TA * TB;
    extern __shared__ __align__(16) double ring[];   // [3][neta][S1], then S1 int offsets
    if (step_blocked(P, st)) return;
    const Grid& g = P.g;
    const int ta = DIM == 3 ? threadIdx.y : 0, tb = threadIdx.x;
    const int a0 = DIM == 3 ? blockIdx.y * TA : 0, b0 = blockIdx.x * TB;
    const int i0 = blockIdx.z * P.xchunk, i1 = min(g.nx, i0 + P.xchunk);
    const int row = a0 + ta, col = b0 + tb;
    const bool active = (DIM == 3 ? row < g.na : true) && col < g.nb;
    const int tid = threadIdx.x + TB * threadIdx.y;
    int* toff = reinterpret_cast<int*>(ring + (size_t)3 * neta * S1);
    for (int r = tid; r < S1; r += NT) {
        const int a = r / RB - HA, b = r % RB - 1;
        toff[r] = (DIM == 3 ? wrapi(a0 + a, g.na) : 0) * g.pb + wrapi(b0 + b, g.nb);
    }
    __syncthreads();
    auto slot = [&](int x) { return ring + (size_t)(((x % 3) + 3) % 3) * neta * S1; };
    auto load = [&](int x) {
        const int xg = x < 0 ? 0 : (x > g.nx - 1 ? g.nx - 1 : x);
        double* dst = slot(x);
        const double* src = eta + (long long)xg * g.plane;
        for (int e = 0; e < neta; ++e) {
            const double* se = src + (long long)e * g.nstore;
            double* de = dst + e * S1;
            for (int r = tid; r < S1; r += NT) de[r] = __ldg(se + toff[r]);
        }
    };
    const int c1 = (ta + HA) * RB + (tb + 1);
    const int bp = c1 + 1, bm = c1 - 1, ap = c1 + RB, am = c1 - RB;
    unsigned long long errkey = ERR_NONE;
    load(i0 - 1);
    load(i0);
    for (int u = i0; u < i1; ++u) {
        load(u + 1);
        __syncthreads();
        if (active) {
            const double* sm = slot(u - 1);
            const double* s0 = slot(u);
            const double* sp = slot(u + 1);
            const long long idx = (long long)u * g.plane + (long long)row * g.pb + col;
            const long long cell = ((long long)u * g.na + row) * g.nb + col;
            double S = 0.;
            for (int e = 0; e < neta; ++e) {
                const double v = s0[e * S1 + c1];
                S += v * v;
            }
            unsigned low = ~0u;   // the exact policy divides every quotient exactly
            using Dv = typename DivOf<FAST ? 0 : 2>::T;
            const Dv dv{P, low};
            const EtaTrial<DIM, Dv> trial(dv, P, S, __ldg(p + idx));
            double Sn = 0., pairs = 0.;
            for (int e = 0; e < neta; ++e) {
                const int o = e * S1;
                const double v = trial(s0[o + c1], sm[o + c1], sp[o + c1], s0[o + am], s0[o + ap], s0[o + bm], s0[o + bp]);
                if (!eta_in_range(v))
                    errkey = min(errkey, ERR_ETA_BASE + (unsigned long long)e * (unsigned long long)g.ncells + (unsigned long long)cell);
                eta_next[(long long)e * g.nstore + idx] = v;
                const double sq = v * v;
                pairs += Sn * sq;
                Sn += sq;
            }
            s2_next[idx] = Sn;
            gb_next[idx] = P.eta_scale * smin(1., 16. * pairs);
        }
        __syncthreads();   // slot(u-1) is refilled with plane u+2 next
    }
    if (errkey != ERR_NONE) atomicMin(err_word(P, st), errkey);
}

// Batched step: one launch advances up to kBatchMax domains of one
// dimensionality and arithmetic form. The per-domain parameters and buffers
// sit in the kernel's parameter space (read through the constant cache with a
// block-uniform index); block b belongs to the last domain whose first block
// is <= b and runs exactly the CTA (bx, by, bz) the single-domain launch would
// run, with the same partial-sum slot, so every domain's result is identical
// to its own nicr_step.
// The compact batch: the block's domain's parameters are the shared ones with
// the domain's grid, inlet value and ranges.
template <int DIM, int TA, int TB, int MINB, bool FAST>
__global__ void __launch_bounds__(TA * TB, MINB) k_step_batch_slim(const __grid_constant__ StepBatchSlim B) {
    int lo = 0, hi = B.n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (B.d[mid].block0 <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const BatchSlim& D = B.d[lo];
    StepParams P = B.base;
    P.g = D.g;
    P.layer_o = D.layer_o;
    P.inlet = D.inlet;
    P.x_hi = D.x_hi;
    P.key_ncells = D.key_ncells;
    P.err_slot = D.err_slot;
    const int t = (int)blockIdx.x - D.block0;
    const int bx = t % D.gx, r = t / D.gx, by = r % D.gy, bz = r / D.gy;
    StepKernel<DIM, TA, TB, FAST>::run(P, D.o, D.cr, D.p, D.gb, D.s2, D.on, D.crn, D.pn, D.partials, D.prev,
                                       D.budget, D.st, bx, by, bz, t, D.nblocks);
}

template <int DIM, int TA, int TB, int MINB, bool FAST>
__global__ void __launch_bounds__(TA * TB, MINB) k_step_batch(const __grid_constant__ StepBatch B) {
    int lo = 0, hi = B.n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (B.d[mid].block0 <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const BatchDomain& D = B.d[lo];
    const int t = (int)blockIdx.x - D.block0;
    const int bx = t % D.gx, r = t / D.gx, by = r % D.gy, bz = r / D.gy;
    StepKernel<DIM, TA, TB, FAST>::run(D.sp, D.o, D.cr, D.p, D.gb, D.s2, D.on, D.crn, D.pn, D.partials,
                                       D.prev, D.budget, D.st, bx, by, bz, t, D.nblocks);
}

}  // namespace

// The 3D step kernel holds 2 CTAs per SM: its staging loads are
// software-pipelined, its budget books fill shared memory (85 KB per CTA), and
// a third CTA's 80 registers spill.
template <int DIM, int TA, int TB, int MINB, bool FAST, bool SLAB>
static void launch_step_n(const StepParams& P, const double* o, const double* cr, const double* p, const double* gb,
                          const double* s2, double* on, double* crn, double* pn, StepPartial* partials,
                          const StepPartial* prev, DevBudget* budget, Status* st, cudaStream_t stream,
                          int* nblocks_out) {
    using T = Tile<DIM, TA, TB>;
    const dim3 grid = step_grid<DIM, TA, TB>(P);
    const int nblocks = (int)(grid.x * grid.y * grid.z);
    // the CTAs of the launch bounds fit the SM's 228 KB (1 KB of it taken per CTA)
    static_assert(MINB * (T::SMEM_BYTES + 1024) <= 228 * 1024, "shared memory holds fewer CTAs than the launch bounds state");
    ensure_smem_attr((const void*)k_step_main<DIM, TA, TB, MINB, FAST, SLAB>, (int)T::SMEM_BYTES);
    k_step_main<DIM, TA, TB, MINB, FAST, SLAB><<<nblocks + (budget ? 1 : 0), dim3(TB, TA), T::SMEM_BYTES, stream>>>(
        P, o, cr, p, gb, s2, on, crn, pn, partials, prev, budget, st, (int)grid.x, (int)grid.y, nblocks);
    if (nblocks_out) *nblocks_out = nblocks;
}

template <bool FAST>
static void launch_step_form(const StepParams& P, const double* o, const double* cr, const double* p,
                             const double* gb, const double* s2, double* on, double* crn, double* pn,
                             StepPartial* partials, const StepPartial* prev, DevBudget* budget, Status* st,
                             cudaStream_t stream, int* nblocks_out) {
#define NICR_STEP_FORM_ARGS P, o, cr, p, gb, s2, on, crn, pn, partials, prev, budget, st, stream, nblocks_out
    if (P.g.dim == 3) {
        if (P.slab) launch_step_n<3, TA3, TB3, 2, FAST, true>(NICR_STEP_FORM_ARGS);
        else launch_step_n<3, TA3, TB3, 2, FAST, false>(NICR_STEP_FORM_ARGS);
    } else {
        launch_step_n<2, TA2, TB2, 4, FAST, false>(NICR_STEP_FORM_ARGS);
    }
#undef NICR_STEP_FORM_ARGS
}

template <bool FAST>
static void launch_eta_form(const StepParams& P, int neta, const double* eta, const double* s2, const double* p,
                            double* eta_next, double* gb_next, double* s2_next, Status* st, cudaStream_t stream) {
    const Grid& g = P.g;
    // The streaming kernel stalls on its per-plane barriers until the next
    // plane has arrived; it is kept only as a tuning option.
    // Kernel choice (measured on B200 at 256^3 with 8 fields): the X-marching
    // kernel for the reciprocal form (0.63 ms vs 0.94 ms per step), the
    // per-cell kernel for the drop-in form, where the unrolled verified
    // divisions of the marching kernel cost more than its saved loads (1.84 ms
    // vs 1.29 ms). NICR_ETA_KERNEL=march|simple|stream overrides for tuning.
    static int simple = -1, march = -1, tma = -1;
    if (simple < 0) {
        const char* e = getenv("NICR_ETA_KERNEL");
        simple = (e && e[0] == 's' && e[1] == 't') ? 0 : 1;
        march = e ? (e[0] == 'm' ? 1 : 0) : -2;
        tma = (e && e[0] == 't') ? 1 : 0;
    }
    const bool slab = P.slab != 0;   // X slabs use the march or the per-cell kernel
    if (tma && !slab && launch_eta_tma<FAST>(neta, P, eta, p, eta_next, gb_next, s2_next, st, stream)) return;
    if (march == 1 || (march == -2 && FAST)) {
        const bool done = g.dim == 3 ? eta_march_dispatch<3, FAST>(neta, P, eta, p, eta_next, gb_next, s2_next, st, stream)
                                     : eta_march_dispatch<2, FAST>(neta, P, eta, p, eta_next, gb_next, s2_next, st, stream);
        if (done) return;
    }
    if (g.dim == 3) {
        constexpr int TA = 8, TB = 32, S1 = (TA + 2) * (TB + 2);
        const size_t smem = (size_t)3 * neta * S1 * sizeof(double) + S1 * sizeof(int);
        if (!simple && !slab && smem <= 200 * 1024) {
            ensure_smem_attr((const void*)k_eta_stream<3, TA, TB, FAST>, 200 * 1024);
            const dim3 grid((g.nb + TB - 1) / TB, (g.na + TA - 1) / TA, (g.nx + P.xchunk - 1) / P.xchunk);
            k_eta_stream<3, TA, TB, FAST><<<grid, dim3(TB, TA), smem, stream>>>(P, neta, eta, p, eta_next, gb_next, s2_next, st);
            return;
        }
        const dim3 block(32, 8);
        const dim3 grid((g.nb + 31) / 32, (g.na + 7) / 8, P.x_hi - P.x_lo);
        k_eta_update<3, FAST><<<grid, block, 0, stream>>>(P, neta, eta, s2, p, eta_next, gb_next, s2_next, st);
    } else {
        constexpr int TB = 128, S1 = TB + 2;
        const size_t smem = (size_t)3 * neta * S1 * sizeof(double) + S1 * sizeof(int);
        if (!simple && smem <= 200 * 1024) {
            ensure_smem_attr((const void*)k_eta_stream<2, 1, TB, FAST>, 200 * 1024);
            const dim3 grid((g.nb + TB - 1) / TB, 1, (g.nx + P.xchunk - 1) / P.xchunk);
            k_eta_stream<2, 1, TB, FAST><<<grid, dim3(TB, 1), smem, stream>>>(P, neta, eta, p, eta_next, gb_next, s2_next, st);
            return;
        }
        const dim3 block(128, 1);
        const dim3 grid((g.nb + 127) / 128, 1, g.nx);
        k_eta_update<2, FAST><<<grid, block, 0, stream>>>(P, neta, eta, s2, p, eta_next, gb_next, s2_next, st);
    }
}

template <int DIM, int TA, int TB, int MINB, bool FAST>
static void launch_batch_slim(const StepBatchSlim& B, int nblocks, cudaStream_t stream) {
    using T = Tile<DIM, TA, TB>;
    ensure_smem_attr((const void*)k_step_batch_slim<DIM, TA, TB, MINB, FAST>, (int)T::SMEM_BYTES);
    k_step_batch_slim<DIM, TA, TB, MINB, FAST><<<nblocks, dim3(TB, TA), T::SMEM_BYTES, stream>>>(B);
}

template <int DIM, int TA, int TB, int MINB, bool FAST>
static void launch_batch_group(StepBatch& B, int nblocks, cudaStream_t stream) {
    using T = Tile<DIM, TA, TB>;
    ensure_smem_attr((const void*)k_step_batch<DIM, TA, TB, MINB, FAST>, (int)T::SMEM_BYTES);
    k_step_batch<DIM, TA, TB, MINB, FAST><<<nblocks, dim3(TB, TA), T::SMEM_BYTES, stream>>>(B);
}

}  // namespace nicr
