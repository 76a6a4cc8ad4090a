// Launch interface between the host model (g++) and the CUDA kernels (nvcc).
// Plain C++: parameter blocks passed by value to the kernels, and launchers.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include <vector>

#include "nicr_physics.h"

namespace nicr {

// Device layout of one field. X (planes) is slowest like the reference
// (3S:165-167); inside a plane, rows (3D: Y) then columns (3D: Z, 2D: Y), the
// column pitch padded to a multiple of 8 doubles so that every row starts on a
// 64-byte boundary. No ghost cells are stored: the kernels apply Neumann X and
// periodic row/column boundaries while staging tiles.
struct Grid {
    int dim;          // 2 or 3
    int nx;           // planes (reference X)
    int na;           // rows: 3D ny, 2D 1
    int nb;           // columns: 3D nz, 2D ny
    int pb;           // padded column pitch (elements)
    long long plane;  // na * pb
    long long ncells; // nx * na * nb
    long long nstore; // nx * plane
};

// Device status word of one domain: sticky failure flag, first failing trial
// (minimum key in reference loop order), step counters.
struct Status {
    unsigned long long err_key;   // ERR_NONE when no trial failed this step
    int failed;                   // a step of this batch was rejected
    int timeout;                  // a kernel's bounded wait for its own copies ran out
    long long failed_step;        // index (steps_done) of the rejected step
    long long steps_done;         // accepted steps since creation
    // First failing trial of the step that reads buffer parity q, in slot q.
    // Slab form: the slabs of a domain agree on a step's outcome by reading
    // every slab's slot of that step (launch_step_finalize_slab). Whole
    // domains: the next step's launch reads it (see launch_step_main).
    unsigned long long slot_err[2];
    int pending[2];               // partials of the step of parity q that await their commit (0: none)
    // a launch of many steps (launch_steps2d): grid barrier arrivals, accepted
    // steps and the key that ended it, for its commit
    unsigned long long barrier, multi_key;
    int multi_steps, pad_;
};
constexpr unsigned long long ERR_NONE = ~0ull;
constexpr unsigned long long ERR_ETA_BASE = 1ull << 62;

// Budget in double-double (Budget, 3S:217); order nucO nucCr ckO ckCr clipO clipCr bcO bcCr
struct DevBudget {
    double v[8][2];
    long long nuclei, clipped;
    double initialO[2], initialCr[2];
};

// Per-CTA partial sums of one step (ckO ckCr clipO clipCr bcO as hi/lo) + clipped count
struct StepPartial {
    double s[5][2];
    long long clipped;
};

// Exact divisions by the run constants (drop-in form): dx*dx etc. are the
// Laplacian denominators (3S:193-195); X, rows (a), columns (b).
struct DivSet {
    DivC dxdx, dada, dbdb, dt;
    DivF dx, da, db;
};
// The reciprocal form's run constants, folded on the host so that the kernels
// spend one multiply-add per neighbour pair and no separate scaling.
struct FastC {
    double rdx;                // 1 / dx
    double wx, wa, wb, w0;     // 1/dx^2, 1/da^2, 1/db^2 and minus twice their sum: the Laplacian's weights
    double fx, fa, fb;         // dt / (2 dx^2) ...: the flux divergence's weights
    double gbo, gbc;           // bulk mobility times (gb_factor - 1)
    double px, pa, pb, p0;     // dt L 2 kp times the Laplacian's weights
    double ex, ea, eb, e0;     // dt eta_L K times the Laplacian's weights
    double tS, tH, t1, e2;     // dt eta_L times 3W, W + A, W, 2W
    double x0, hS, hH;         // phi force: constant term, (W + A)/2, W/2
    double ckO, ckCr;          // -Ck / dt
};

struct StepParams {
    Grid g;
    double dx, dt;               // spacing along X
    double dt_s, etaK_s;         // 2^-128 dt and 2^-128 eta_K (after scaled quotients)
    union {                      // by form: the other form's constants are not needed
        DivSet div;              // fast == 0
        FastC f;                 // fast == 1
    };
    double dtL;                  // dt * Physics::L
    double layer_o;
    double gbm1_o, gbm1_cr;      // gb_factor_o - 1, gb_factor_cr - 1
    double mu_res, surface_c_ref;
    double eta_W, eta_A, eta_K, dt_etaL, eta_scale;
    int bc, ck, bounds;
    int o_on;                    // oxygen_diffusion
    int grains;                  // GB mask active in mobility
    int phi_eta;                 // eta coupling in the phi force (has_eta)
    int inlet;                   // bc == concentration && oxygen_diffusion
    int xchunk;                  // planes per CTA along X
    int fast;                    // arithmetic form: 0 drop-in (bit-identical), 1 reciprocal divisions
    // Planes updated: [x_lo, x_hi) of the g.nx stored planes. A whole domain
    // updates all of them; an X slab of a larger domain stores halo planes
    // below and above its own, which the kernels read but do not write.
    int x_lo, x_hi;
    // Failing-trial keys in whole-domain reference order: the cell index is
    // offset by cell_off and eta keys count key_ncells cells per field.
    long long cell_off, key_ncells;
    // Error word of this step: -1 st->err_key, 0/1 st->slot_err[err_slot]
    int err_slot;
    int slab, pad_;              // an X slab (its plane range and key offsets apply)
    // drop-in form: 1 when a divisor or a constant after a scaled quotient
    // lies outside the certified range, so every chunk is divided by IEEE
    // division; 2 when two operations divide by each of them (division_in_two)
    unsigned div_gate;
};
// The run constants of the configured form (spacings along X, rows, columns);
// the other scalar members of sp are set already. Returns the exact divisions,
// which the refresh of either form uses.
inline DivSet fill_form_constants(StepParams& sp, int dim, double dx, double da, double db) {
    DivSet d;
    d.dxdx = make_divc(dx * dx);
    d.dada = make_divc(da * da);
    d.dbdb = make_divc(db * db);
    d.dx = make_divc(dx);
    d.da = make_divc(da);
    d.db = make_divc(db);
    d.dt = make_divc(sp.dt);
    if (!sp.fast) {
        sp.div = d;
        sp.dt_s = std::ldexp(sp.dt, -128);
        sp.etaK_s = std::ldexp(sp.eta_K, -128);
        const bool k_ok = sp.eta_K == 0. || (std::fabs(sp.eta_K) >= std::ldexp(1., -500) && std::fabs(sp.eta_K) <= std::ldexp(1., 500));
        bool in_range = k_ok, in_two = true;
        for (double b : {d.dxdx.b, d.dada.b, d.dbdb.b, d.dt.b, d.dx.b, d.da.b, d.db.b}) {
            in_range = in_range && div_in_range(b);
            in_two = in_two && division_in_two(b);
        }
        sp.div_gate = !in_range ? 1u : in_two ? 2u : 0u;
        return d;
    }
    FastC f{};
    f.rdx = d.dx.rb;
    f.wx = d.dxdx.rb;
    f.wa = dim == 3 ? d.dada.rb : 0.;
    f.wb = d.dbdb.rb;
    f.w0 = -2. * (f.wx + f.wa + f.wb);
    f.fx = 0.5 * sp.dt * (d.dx.rb * d.dx.rb);
    f.fa = 0.5 * sp.dt * (d.da.rb * d.da.rb);
    f.fb = 0.5 * sp.dt * (d.db.rb * d.db.rb);
    f.gbo = Phys::bmo * sp.gbm1_o;
    f.gbc = Phys::bmc * sp.gbm1_cr;
    const double kp = sp.dtL * 2. * Phys::kp, ke = sp.dt_etaL * sp.eta_K;
    f.px = kp * f.wx; f.pa = kp * f.wa; f.pb = kp * f.wb; f.p0 = -2. * (f.px + f.pa + f.pb);
    f.ex = ke * f.wx; f.ea = ke * f.wa; f.eb = ke * f.wb; f.e0 = -2. * (f.ex + f.ea + f.eb);
    f.tS = sp.dt_etaL * 3. * sp.eta_W;
    f.tH = sp.dt_etaL * (sp.eta_W + sp.eta_A);
    f.t1 = sp.dt_etaL * sp.eta_W;
    f.e2 = 2. * f.t1;
    f.hS = 0.5 * (sp.eta_W + sp.eta_A);
    f.hH = 0.5 * sp.eta_W;
    f.x0 = 1922722.2974223055 - (sp.phi_eta ? f.hH : 0.);   // foxide - fmetal at o = cr = 0, and -W/2
    f.ckO = -Phys::ckO / sp.dt;
    f.ckCr = -Phys::ckCr / sp.dt;
    sp.f = f;
    return d;
}
// The whole-domain values of the range fields (every plane, no offset).
inline void whole_domain_range(StepParams& sp) {
    sp.x_lo = 0;
    sp.x_hi = sp.g.nx;
    sp.cell_off = 0;
    sp.key_ncells = sp.g.ncells;
    sp.err_slot = -1;
}

// ---- step --------------------------------------------------------------------
// Main fused step: mu, M, six-face fluxes, phi, Ck, bounds -> trial buffers.
// With a budget (P.err_slot = the buffer parity) the commit is deferred: the
// launch leaves its partials in `partials` as pending, and one extra CTA of it
// commits the previous step from `prev` (the other parity's partials) beside
// the step's own CTAs; launch_step_flush commits the last one. Whatever else
// can fail the step (the eta update) is launched before the step kernel.
// Without a budget nothing is committed and the caller reads the partials.
void launch_step_main(const StepParams& P, const double* o, const double* cr, const double* p,
                      const double* gb, const double* s2, double* on, double* crn, double* pn,
                      StepPartial* partials, const StepPartial* prev, DevBudget* budget, Status* st,
                      cudaStream_t stream, int* nblocks_out);
int step_main_blocks(const StepParams& P);
// Planes per CTA along X for grid g (step and eta kernels), and one chunk for
// the n domains of a batch. NICR_XCHUNK forces a chunk for tuning runs.
int choose_xchunk(const Grid& g);
// The same choice for the one-pass step (16 x 32 tiles, one CTA per SM).
int choose_xchunk_fused(const Grid& g);
int choose_xchunk_batch(const Grid* grids, int n);
// The chunks a measured choice tries for a largest X extent nxmax: nxmax halved
// repeatedly, the powers of two below it and the chunk in use, longest first.
std::vector<int> xchunk_candidates(int nxmax, int in_use);
// Per-device kernel attributes of the step kernel P selects, set outside any
// stream capture (launch_step_main sets them on first use otherwise).
void step_kernels_prepare(const StepParams& P);
// The reciprocal form's launchers (nicr_step_fast.cu, compiled with FMA
// contraction); the generic launchers dispatch to them when P.fast is set.
void launch_step_main_fast(const StepParams& P, const double* o, const double* cr, const double* p, const double* gb,
                           const double* s2, double* on, double* crn, double* pn, StepPartial* partials,
                           const StepPartial* prev, DevBudget* budget, Status* st, cudaStream_t stream,
                           int* nblocks_out);
void launch_eta_update_fast(const StepParams& P, int neta, const double* eta, const double* s2, const double* p,
                            double* eta_next, double* gb_next, double* s2_next, Status* st, cudaStream_t stream);
void step_kernels_prepare_fast(const StepParams& P);
// Eta mask: S = sum eta^2, pairs, gb = scale*min(1,16*pairs) (3S:495-507)
void launch_eta_mask(const StepParams& P, int neta, const double* eta, double* gb, double* s2,
                     double* pairs, Status* st, cudaStream_t stream);
// Eta trial update (3S:514-526) + next-step mask from the trial values
void launch_eta_update(const StepParams& P, int neta, const double* eta, const double* s2,
                       const double* p, double* eta_next, double* gb_next, double* s2_next,
                       Status* st, cudaStream_t stream);
// Batched step of many domains in one launch per group of <= kBatchMax domains
// of one dimensionality and arithmetic form (consecutive entries). Each entry
// carries the domain's parameters and buffers; gx, gy, block0 are filled by the
// launcher, nblocks (the domain's partial-sum count) is written back.
struct BatchDomain {
    StepParams sp;
    const double *o, *cr, *p, *gb, *s2;
    double *on, *crn, *pn;
    StepPartial* partials;
    const StepPartial* prev;
    DevBudget* budget;
    Status* st;
    int gx, gy, block0, nblocks;
};
constexpr int kBatchMax = 48;   // 48 entries: ~32,000 bytes of kernel parameters (limit 32,764)
struct StepBatch {
    int n, pad;
    BatchDomain d[kBatchMax];
};
// Compact form of a batch whose domains share every step parameter except
// the grid, the inlet value and the plane/key ranges that follow from the
// grid (a parameter sweep over sizes, O supply, Cr and Ksp, which the step
// kernel does not read): the shared parameters once, ~170 bytes per domain,
// so one launch serves up to kBatchSlimMax domains.
struct BatchSlim {
    Grid g;
    double layer_o;
    long long key_ncells;
    int x_hi, inlet, gx, gy, block0, nblocks, err_slot, pad;
    const double *o, *cr, *p, *gb, *s2;
    double *on, *crn, *pn;
    StepPartial* partials;
    const StepPartial* prev;
    DevBudget* budget;
    Status* st;
};
constexpr int kBatchSlimMax = 160;   // 160 x 192 bytes + the shared parameters: < 31.5 KB of kernel parameters
struct StepBatchSlim {
    StepParams base;
    int n, pad;
    BatchSlim d[kBatchSlimMax];
};
// returns the number of launches: one for the whole batch in the compact
// form when it applies, else one per group of kBatchMax domains
int launch_step_batch(BatchDomain* doms, int n, cudaStream_t stream);
void launch_batch_slim_fast(const StepBatchSlim& B, int nblocks, int dim, cudaStream_t stream);
void launch_batch_group_fast(StepBatch& B, int nblocks, int dim, cudaStream_t stream);

// One launch for the step kernel and the eta update of one step (reciprocal
// form, 3D, 1..16 eta fields): the two are independent within a step, and
// their CTAs share the SMs (see k_step_eta). ticket: one word of device
// memory, zeroed by the launcher before each launch. Returns false (nothing
// launched) when the form does not apply; nblocks_out receives the step
// kernel's partial-sum count.
bool launch_step_eta_fast(const StepParams& P, int neta, const double* o, const double* cr, const double* p,
                          const double* gb, const double* s2, double* on, double* crn, double* pn,
                          StepPartial* partials, const double* eta, double* eta_next, double* gb_next,
                          double* s2_next, unsigned* ticket, Status* st, cudaStream_t stream, int* nblocks_out);
void step_eta_prepare_fast(const StepParams& P, int neta);

// One HBM pass per step (3D, evolving eta): the step kernel and the eta
// update fused into one X march with the eta planes staged by TMA and S / gb
// rebuilt on chip (k_step_fused, nicr_step_fused.cuh). It reads o, cr, p and
// the n eta fields and writes the trial o, cr, p and eta; gb and eta_s2 are
// neither read nor written. Applies to 1 <= n <= 8 fields, rows a multiple of
// 16 and columns a multiple of 32 (step_fused_applies); the launchers return
// false and launch nothing otherwise. The drop-in form is bit-identical to
// the two-kernel form.
bool step_fused_applies(const Grid& g, int neta);
bool launch_step_fused(const StepParams& P, int neta, const double* o, const double* cr, const double* p,
                       const double* eta, double* on, double* crn, double* pn, double* eta_next,
                       StepPartial* partials, const StepPartial* prev, DevBudget* budget, Status* st,
                       cudaStream_t stream, int* nblocks_out);
bool launch_step_fused_fast(const StepParams& P, int neta, const double* o, const double* cr, const double* p,
                            const double* eta, double* on, double* crn, double* pn, double* eta_next,
                            StepPartial* partials, const StepPartial* prev, DevBudget* budget, Status* st,
                            cudaStream_t stream, int* nblocks_out);
// kernel attributes of the fused step, set outside any stream capture
void step_fused_prepare(const StepParams& P, int neta);
void step_fused_prepare_fast(const StepParams& P, int neta);

// The seven arrays of a 3D VTI frame in file order (X fastest) and type, for
// the output path (nicr_vti.cu). range gets bit a set when array a holds a
// finite value outside the Float32 range.
struct VtiArgs {
    Grid g;
    int has_eta, neta;
    const double *p, *o, *cr, *muO, *muCr, *gb, *grain, *eta;
};
void launch_vti_arrays(const VtiArgs& a, void* out, bool f64, unsigned* range, cudaStream_t stream);

// Many steps of a small 2D domain in one cooperative launch and its commit
// (nicr_steps2d.cuh): steps2d_tile gives the tile's planes TX for which the
// domain's CTAs of TX x 32 cells are resident one per SM (0: too large, or no
// cooperative launches on the device). The buffers are read at parities par,
// gpar, epar and written at the others, toggling with each accepted step (gpar
// and epar only with evolving eta, neta > 0).
struct Steps2DArgs {
    double *o[2], *cr[2], *p[2], *gb[2], *s2[2], *eta[2];
    StepPartial* partials;
    int neta, nsteps, par, gpar, epar, pad;
};
constexpr int kSteps2DMost = 4096;   // steps per launch (tens of milliseconds)
int steps2d_tile(const Grid& g, int* ctas);
bool launch_steps2d(const StepParams& P, const Steps2DArgs& A, int tx, int ctas, DevBudget* budget, Status* st,
                    Status* host, cudaStream_t stream);
bool launch_steps2d_fast(const StepParams& P, const Steps2DArgs& A, int tx, int ctas, Status* st, cudaStream_t stream);
// Commits each domain's pending step, if any: its partials (of parity q at
// partials + q * cap) reduced, then budget and counters unless a trial failed;
// the status word is written to the host either way.
struct FlushDomain {
    const StepPartial* partials;
    DevBudget* budget;
    Status* st;
    Status* host;   // pinned host memory that receives the status
    int cap, pad;
};
constexpr int kFlushMax = 512;   // 512 x 40 bytes of kernel parameters
struct FlushList {
    FlushDomain d[kFlushMax];
};
void launch_step_flush(const FlushDomain* doms, int n, cudaStream_t stream);
// Slab form of the commit: the step is rejected when any slab's error word
// of this step (peers[j]->slot_err[slot], read after every slab's step
// kernels completed) holds a failing trial; the minimum key is recorded in
// st->err_key. peers may live on other GPUs (peer access enabled).
constexpr int kMaxSlabs = 16;
struct SlabPeers {
    const Status* st[kMaxSlabs];
    int n, slot;
};
void launch_step_finalize_slab(const StepPartial* partials, int nblocks, DevBudget* budget, Status* st,
                               const SlabPeers& peers, cudaStream_t stream);
// One process per slab: the slab's error word of the step (slot) as a signed
// agreement word (kAgreeNone when every trial passed, else the key), which
// the ranks reduce with a MIN collective; the commit then reads the result.
constexpr long long kAgreeNone = 0x7fffffffffffffffLL;
void launch_agree_word(const Status* st, int slot, long long* agree, cudaStream_t stream);
void launch_step_finalize_agreed(const StepPartial* partials, int nblocks, DevBudget* budget, Status* st,
                                 const long long* agreed, cudaStream_t stream);
// Copies up to kCopySegs strided runs of doubles (rows x n, 16-byte aligned
// addresses and counts of whole double pairs) in one launch; destinations may
// be another GPU's memory (peer access enabled): the halo exchange of the
// slab form. Skipped when st->failed is set (st may be null).
constexpr int kCopySegs = 24;
struct CopySeg {
    const double* src;
    double* dst;
    long long n, rows, src_pitch, dst_pitch;   // doubles
};
struct CopyList {
    CopySeg s[kCopySegs];
    int count, pad;
};
void launch_copy_segments(const CopyList& L, const Status* st, cudaStream_t stream);
// Refresh for output: mu_O, mu_Cr, M_O, M_Cr at every cell (3S:597-620)
void launch_refresh(const StepParams& P, const double* o, const double* cr, const double* p,
                    const double* gb, double* muO, double* muCr, double* mo, double* mc,
                    cudaStream_t stream);

// Device self-check of the exact division: mismatches against IEEE a/b
long long check_division(double b, long long n, unsigned long long seed, long long* tested);

// ---- init --------------------------------------------------------------------
struct InitParams {
    Grid g;
    int ng;
    double nxd, nyd, nzd;        // grid extents as doubles (periods)
    double bulk_cr, layer_o;
    int inlet_layer;             // bc == concentration
    // X slab: stored plane 0 is domain plane x_off; sums and counts cover the
    // own planes [x_lo, x_hi) only. A whole domain: 0, 0, g.nx.
    int x_off, x_lo, x_hi;
};
void launch_init_fields(const InitParams& I, double* o, double* cr, double* p, cudaStream_t stream);
// 3D Voronoi labels (first nearest seed under minimum image) and the distance
// to the nearest bisector (3S:450-466). seeds: x,y,z per seed. competitor
// (may be null) receives the 0-based seed of the nearest bisector (-1: none).
void launch_voronoi3(const InitParams& I, const double* seeds, double* grain, double* db,
                     int* volumes, int* competitor, cudaStream_t stream);
// Face adjacency of the grains (ng x ng bytes, set to 1 for adjacent pairs)
void launch_grain_adjacency(const InitParams& I, const double* grain, unsigned char* adj, cudaStream_t stream);
// 3D eta initial weights: per competitor g, the bisector distance (3S:469-494);
// the owner's slot receives -1. Output layout eta[g*nstore + idx].
void launch_eta_dist3(const InitParams& I, const double* seeds, const double* grain, double* eta,
                      cudaStream_t stream);
// Centre seed (3S:725-751): stamps the ball and accumulates nucO, nucCr, cells
void launch_center_seed(const InitParams& I, double cx, double cy, double cz, double r, int neta,
                        double* o, double* cr, double* p, double* eta, StepPartial* partials,
                        cudaStream_t stream, int* nblocks_out);
// Generic dd sum over the partial array (first nsum slots + count) into out
void launch_reduce_partials(const StepPartial* partials, int nblocks, StepPartial* out,
                            cudaStream_t stream);

// ---- diagnostics ---------------------------------------------------------------
// sums o, cr, p, h(p) (dd) and min/max of O, Cr, Ni, phi (3S:963-977)
struct DiagOut {
    double sum[4][2];
    double mn[4], mx[4];   // O, Cr, Ni(=1-o-cr, min only), phi
    long long mni[4], mxi[4];  // first cell (reference order) attaining each extremum
};
// grain_log statistics (3S:566-590): scalars, per-grain dominant cells and
// weighted amounts, and the discrete grain energy (3S:546-565)
struct GrainParams {
    Grid g;
    int dim, neta;
    double dx, da, db, K, W, A;
    DivC v_dx, v_da, v_db;       // exact divisions by dx, da, db
    const double* pairs;   // 2D: eta_pairs of the last mask (2D:337); unused in 3D
    int x_above;           // the plane after g's last one is stored and in the domain (an X slab
                           // below another): the last plane keeps its +X gradient term
};
struct GrainOut {
    double lo, hi, slo, shi, gbmax;
    double sum[3][2];      // S, (1-h) gb, energy
    long long unassigned;
};
struct GrainWork {
    unsigned long long* cells;  // neta
    void* parts;                // grain_blocks() * grain_part_bytes()
    double* amount_parts;       // grain_blocks() * neta * 2
};
size_t grain_part_bytes();
int grain_blocks(long long ncells);
void launch_grain_stats(const GrainParams& G, const double* eta, const double* s2, const double* p, const double* gb,
                        GrainWork& W, GrainOut* out, double* amount_out, long long* cells_out, cudaStream_t stream);

void launch_diagnostics(const Grid& g, const double* o, const double* cr, const double* p,
                        DiagOut* partials, int* nblocks, DiagOut* out, cudaStream_t stream);

}  // namespace nicr
