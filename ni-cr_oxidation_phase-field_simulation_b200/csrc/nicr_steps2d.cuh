// Many steps of a small 2D domain in one launch. A 2D step of 128^2 cells is a
// few hundred nanoseconds of arithmetic; as one launch per step it took 8.3 us,
// launch, prologue and a serial march along X included. Here the domain's tiles
// stay resident, one CTA of TX x 32 cells per SM (cooperative launch), and a
// grid barrier separates the steps: per step every CTA reads its tile and halo
// from L2, computes mu and M on the tile and its ring (one thread per point, so
// the ring costs no second pass), updates its cells (the step and the eta
// trials) into the other buffers and arrives. 3.8 us per step at 128^2
// (a run of 4000 steps).
//
// Everything other CTAs wrote is read with ld.cg (L2): L1 may hold older lines.
// A step's failing trials go to the error word of its parity; after the barrier
// every CTA reads the same word, so all stop at the same step. A CTA is at most
// one step ahead of another, so the other parity's word is never the one being
// read. Budget increments of a step (at most one of each kind per cell) are
// held until the step is accepted, then added to the thread's double-double
// sums, which are reduced once per launch (k_steps2d_commit). The barrier's
// wait is bounded: a CTA that gives up sets st->timeout and leaves, and the
// others run out of their own waits.
// Included by the two units that compile the step kernels.
#pragma once

namespace nicr {
namespace {

constexpr int kBarrierSpins = 1 << 23;   // polls of the grid barrier before it is declared lost

// A cell's budget increments of one step, kept until the step is accepted.
struct CellBook {
    double inc[5];
    int clipped;
    unsigned long long k;
    __device__ void clear() {
#pragma unroll
        for (int q = 0; q < 5; ++q) inc[q] = 0.;
        clipped = 0;
        k = ERR_NONE;
    }
    __device__ void add(int q, double b) { inc[q] = b; }   // each kind occurs once per cell and step
    __device__ void clip() { clipped = 1; }
    __device__ void fail(unsigned long long key) { k = min(k, key); }
};

template <bool FAST, int TX>
struct Steps2D {
    using SK = StepKernel<2, 1, 32, FAST>;
    static constexpr int TB = 32, W2 = TB + 4, W1 = TB + 2;
    static constexpr int N2 = (TX + 4) * W2, N1 = (TX + 2) * W1;   // points of the radius-2 and radius-1 tiles
    static constexpr int NT = (N1 + 31) / 32 * 32;
    static_assert(2 * NT >= N2, "two staged points per thread");

    struct Smem {
        double o[N2], cr[N2];
        double p[N1], muO[N1], muCr[N1], mo[N1], mc[N1];
        double book[12 * NT];
        DD sdd[32 * 5];
        long long scnt[32];
    };

    // Lead points and cells of one step with the division policy of DM (DivOf);
    // true (first pass): the tile must be computed again with exact divisions.
    template <int DM>
    __device__ static bool step_tile(const StepParams& P, const Steps2DArgs& A, Smem& s, int par, int gpar, int epar,
                                     double gbv, double o_raw, double s2u, int x0, int col, CellBook& book) {
        unsigned low = kFirstPass<DM> && P.div_gate == 1 ? 0u : ~0u;
        const typename DivOf<DM>::T dv{P, low};
        const Grid& g = P.g;
        const int tid = threadIdx.x;
        const bool o_on = P.o_on != 0;
        book.clear();
        {
            const int a = tid / W1, b = tid - a * W1 - 1;   // tile rows -1 .. TX as a = 0 .. TX + 1
            const int x = x0 + a - 1;
            if (tid < N1 && x >= 0 && x < g.nx) {
                const double *so0 = s.o + (a + 1) * W2, *sc0 = s.cr + (a + 1) * W2;
                const int r = a * W1;
                SK::lead_core(dv, P, o_on, so0 - W2, so0, so0 + W2, sc0 - W2, sc0, sc0 + W2, s.p + r, s.muO + r, s.muCr + r,
                              s.mo + r, s.mc + r, 0, b, gbv);
            }
        }
        __syncthreads();
        const int ta = tid >> 5, tb = tid & 31, x = x0 + ta;
        if (ta < TX && x < g.nx && col < g.nb) {
            const int r = (ta + 1) * W1, c1 = tb + 1;
            const double *mO = s.muO + r, *mC = s.muCr + r, *mo_ = s.mo + r, *mc_ = s.mc + r, *spu = s.p + r;
            CenterVals C, L, B;   // this plane, the one above, the one below (Neumann copies at the ends)
            C.o = s.o[(ta + 2) * W2 + tb + 2];
            C.cr = s.cr[(ta + 2) * W2 + tb + 2];
            C.p = spu[c1];
            C.hh = FAST ? h_fast(C.p) : h(C.p);
            C.muO = mO[c1]; C.muCr = mC[c1]; C.mo = mo_[c1]; C.mc = mc_[c1];
            L = C;
            B = C;
            if (x < g.nx - 1) {
                L.p = spu[c1 + W1];
                L.muO = mO[c1 + W1]; L.muCr = mC[c1 + W1]; L.mo = mo_[c1 + W1]; L.mc = mc_[c1 + W1];
            }
            double FxO, FxCr;
            if (x > 0) {
                B.p = spu[c1 - W1];
                B.muO = mO[c1 - W1]; B.muCr = mC[c1 - W1]; B.mo = mo_[c1 - W1]; B.mc = mc_[c1 - W1];
                FxO = SK::face_x(dv, B.mo, C.mo, B.muO, C.muO);
            } else {
                // ghost plane -1: copies of plane 0 (2D:163-169, 2D:428-430)
                FxO = SK::face_x(dv, C.mo, C.mo, (P.bc == 1 && o_on) ? 2. * P.mu_res - C.muO : C.muO, C.muO);
            }
            FxCr = SK::face_x(dv, B.mc, C.mc, B.muCr, C.muCr);
            const long long idx = (long long)x * g.plane + col;
            auto cell = [&]() { return (long long)x * g.nb + col; };
            if (x == 0 && P.bc == 1) FxO = SK::surface_face(dv, P, o_on, C, P.grains ? gb_own(A, gpar, idx) : 0., book);
            if (x == 0 && P.inlet) book.add(4, P.layer_o - o_raw);
            const typename SK::CoreOut R = SK::cell_core(dv, P, o_on, P.ck == 0, P.phi_eta != 0, C, L, B.p, FxO, FxCr, s2u,
                                                         mO, mC, mo_, mc_, spu, c1, c1 + 1, c1 - 1, 0, 0);
            const int nx = par ^ 1;
            SK::finish_cell(R, P.bounds == 1, A.o[nx] + idx, A.cr[nx] + idx, A.p[nx] + idx, book, cell);
            if (A.neta > 0) {   // eta_trial (2D:347-359) and the mask of the trial values
                const double* e = A.eta[epar];
                double* en = A.eta[epar ^ 1];
                const long long ixm = x > 0 ? idx - g.plane : idx, ixp = x < g.nx - 1 ? idx + g.plane : idx;
                const long long ibm = idx + (col == 0 ? g.nb - 1 : -1), ibp = idx + (col == g.nb - 1 ? 1 - g.nb : 1);
                const EtaTrial<2, typename DivOf<DM>::T> trial(dv, P, s2u, C.p);
                double Sn = 0., pairs = 0.;
                bool in_range = true;
                for (int q = 0; q < A.neta; ++q, e += g.nstore, en += g.nstore) {
                    const double v = trial(__ldcg(e + idx), __ldcg(e + ixm), __ldcg(e + ixp), 0., 0., __ldcg(e + ibm),
                                           __ldcg(e + ibp));
                    in_range = in_range && eta_in_range(v);
                    en[idx] = v;
                    const double sq = v * v;
                    pairs += Sn * sq;
                    Sn += sq;
                }
                if (!in_range) book.fail(eta_fail_key(A.eta[epar ^ 1] + idx, A.neta, g.nstore, g.ncells, cell()));
                A.s2[gpar ^ 1][idx] = Sn;
                A.gb[gpar ^ 1][idx] = P.eta_scale * smin(1., 16. * pairs);
            }
        }
        return kFirstPass<DM> && __syncthreads_or(low <= kLowQuotient || book.k != ERR_NONE);
    }
    __device__ static double gb_own(const Steps2DArgs& A, int gpar, long long idx) { return __ldcg(A.gb[gpar] + idx); }

    // Arrives at the grid barrier and waits for round n of it; false when the wait ran out.
    __device__ static bool grid_barrier(Status* st, unsigned long long n) {
        __syncthreads();
        bool ok = true;
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(&st->barrier, 1ull);
            const unsigned long long want = n * gridDim.x;
            int spin = 0;
            while (*(volatile unsigned long long*)&st->barrier < want)
                if (++spin > kBarrierSpins) { ok = false; break; }
            __threadfence();
        }
        return !__syncthreads_or(!ok);
    }

    __device__ static void run(const StepParams& P, const Steps2DArgs& A, Status* st) {
        extern __shared__ __align__(16) unsigned char steps2d_smem[];
        Smem& s = *reinterpret_cast<Smem*>(steps2d_smem);
        if (st->failed) return;   // an earlier step of this batch was rejected (every CTA reads the same)
        const Grid& g = P.g;
        const int tid = threadIdx.x;
        const int ntx = (g.nx + TX - 1) / TX;
        const int x0 = (int)(blockIdx.x % ntx) * TX, b0 = (int)(blockIdx.x / ntx) * TB;
        // this thread's staging points, lead point and cell, as offsets in a field
        int o2[2];
        bool in2[2];   // the inlet replaces o there
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int q = tid + k * NT;
            const int x = min(max(x0 + q / W2 - 2, 0), g.nx - 1);
            o2[k] = q < N2 ? (int)(x * g.plane) + wrapi(b0 + q % W2 - 2, g.nb) : -1;
            in2[k] = P.inlet && x == 0;
        }
        int o1 = -1;
        if (tid < N1) o1 = (int)(min(max(x0 + tid / W1 - 1, 0), g.nx - 1) * g.plane) + wrapi(b0 + tid % W1 - 1, g.nb);
        const int cx = x0 + (tid >> 5), col = b0 + (tid & 31);
        const bool owner = (tid >> 5) < TX && cx < g.nx && col < g.nb;
        const int oc = owner ? (int)(cx * g.plane) + col : -1;
        SharedBook<NT> total(s.book + tid);
        CellBook book;
        int par = A.par, gpar = A.gpar, epar = A.epar, done = 0;
        unsigned long long key = ERR_NONE;
        for (int n = 0; n < A.nsteps; ++n) {
            const double *o = A.o[par], *cr = A.cr[par];
#pragma unroll
            for (int k = 0; k < 2; ++k)
                if (o2[k] >= 0) {
                    const double v = __ldcg(o + o2[k]);
                    s.o[tid + k * NT] = in2[k] ? P.layer_o : v;
                    s.cr[tid + k * NT] = __ldcg(cr + o2[k]);
                }
            double gbv = 0., o_raw = 0., s2u = 0.;
            if (o1 >= 0) {
                s.p[tid] = __ldcg(A.p[par] + o1);
                if (P.grains) gbv = __ldcg(A.gb[gpar] + o1);
            }
            if (oc >= 0) {
                if (P.inlet && cx == 0) o_raw = __ldcg(o + oc);
                if (P.phi_eta) s2u = __ldcg(A.s2[gpar] + oc);
            }
            __syncthreads();
            if (FAST) {
                step_tile<0>(P, A, s, par, gpar, epar, gbv, o_raw, s2u, x0, col, book);
            } else if (P.div_gate == 2 ? step_tile<3>(P, A, s, par, gpar, epar, gbv, o_raw, s2u, x0, col, book)
                                       : step_tile<1>(P, A, s, par, gpar, epar, gbv, o_raw, s2u, x0, col, book)) {
                step_tile<2>(P, A, s, par, gpar, epar, gbv, o_raw, s2u, x0, col, book);
            }
            if (book.k != ERR_NONE) atomicMin(&st->slot_err[n & 1], book.k);
            if (!grid_barrier(st, (unsigned long long)n + 1)) {
                if (tid == 0) atomicOr(&st->timeout, 1);
                return;
            }
            key = *(volatile unsigned long long*)&st->slot_err[n & 1];
            if (key != ERR_NONE) break;   // the same word for every CTA
#pragma unroll
            for (int q = 0; q < 5; ++q)
                if (book.inc[q] != 0.) total.add(q, book.inc[q]);
            if (book.clipped) total.clip();
            par ^= 1;
            if (A.neta > 0) { gpar ^= 1; epar ^= 1; }
            ++done;
        }
        DD acc[5];
        long long clipped = total.clipped();
        for (int q = 0; q < 5; ++q) acc[q] = DD{total.v(2 * q), total.v(2 * q + 1)};
        block_reduce_dd<5>(acc, clipped, s.sdd, s.scnt);
        if (tid == 0) {
            StepPartial& out = A.partials[blockIdx.x];
            for (int q = 0; q < 5; ++q) { out.s[q][0] = acc[q].hi; out.s[q][1] = acc[q].lo; }
            out.clipped = clipped;
            if (blockIdx.x == 0) {
                st->multi_steps = done;
                st->multi_key = key;
            }
        }
    }
};

template <bool FAST, int TX>
__global__ void __launch_bounds__(Steps2D<FAST, TX>::NT, 1)
k_steps2d(const __grid_constant__ StepParams P, const __grid_constant__ Steps2DArgs A, Status* st) {
    Steps2D<FAST, TX>::run(P, A, st);
}

template <bool FAST, int TX>
static bool launch_steps2d_n(const StepParams& P, const Steps2DArgs& A, int ctas, Status* st, cudaStream_t stream) {
    using K = Steps2D<FAST, TX>;
    const void* kernel = (const void*)k_steps2d<FAST, TX>;
    ensure_smem_attr(kernel, (int)sizeof(typename K::Smem));
    void* args[] = {const_cast<StepParams*>(&P), const_cast<Steps2DArgs*>(&A), &st};
    return cudaLaunchCooperativeKernel(kernel, dim3(ctas), dim3(K::NT), args, sizeof(typename K::Smem), stream) == cudaSuccess;
}

template <bool FAST>
static bool launch_steps2d_form(const StepParams& P, const Steps2DArgs& A, int tx, int ctas, Status* st,
                                cudaStream_t stream) {
    switch (tx) {
        case 2: return launch_steps2d_n<FAST, 2>(P, A, ctas, st, stream);
        case 4: return launch_steps2d_n<FAST, 4>(P, A, ctas, st, stream);
        case 8: return launch_steps2d_n<FAST, 8>(P, A, ctas, st, stream);
        default: return false;
    }
}

}  // namespace
}  // namespace nicr
