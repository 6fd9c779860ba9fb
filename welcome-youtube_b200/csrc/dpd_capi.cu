// dpd_capi.cu -- the C ABI of libdpd.so (include/dpd.h): handles, device
// memory, CUDA graphs of the step, state in/out, error reporting.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <string>
#include <numeric>
#include <type_traits>
#include <vector>

#include <cuda.h>

#include "../../include/dpd.h"
#include "dpd_internal.h"

static_assert(sizeof(dpd_event) == sizeof(EventDev), "event layout");

static thread_local std::string g_err;

static int fail(int code, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

// the error message of a call made outside this file (dpd_cells.cu)
int lib_error(int code, const char *msg) {
    g_err = msg;
    return code;
}

#define CK(call)                                                                                        \
    do {                                                                                                \
        cudaError_t e_ = (call);                                                                        \
        if (e_ != cudaSuccess) {                                                                        \
            cudaGetLastError(); /* a refused call's error is this call's, not the next one's */         \
            return fail(DPD_E_CUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
        }                                                                                               \
    } while (0)

// reverse-mode storage (defined here: the handle keeps it between windows)
namespace {
struct FullCk {  // a full configuration of the engine's current buffer
    float2 *pos, *vh, *vt, *f;
    uint32_t *tg;
    int2 *link;
    int32_t *cstart;
};
struct SegState {  // what a force VJP needs of one configuration, and the sort that made it
    float2 *pos, *vt;
    uint32_t *tg;
    int2 *link;
    int32_t *cstart, *src;
};
struct AdjBufs {
    std::vector<FullCk> ck;     // the start of each segment
    std::vector<SegState> seg;  // the configurations of one segment after its start
    float2 *vh[2], *f[2];       // the half-step velocities and forces of a segment's steps, in turn
    float2 *X[2], *V[2], *F[2]; // the adjoint state of one configuration and of the one before, in turn
    float2 *xb, *vb;
    float2 *G;                  // the loss's own x_bar of ng configurations
    int ng = 0;
    double *hist, *wgt, *grad;
    double *gsum;            // per replica: the sum of the x cotangents (stirring)
    long long *stir;         // per replica: the stirring sums of a segment's steps
};
}  // namespace

struct dpd_handle {
    int nrep = 0;
    std::vector<dpd_params> params;
    std::vector<RepDev> rh;
    int64_t N = 0, C = 0;
    int nmax = 0;
    cudaStream_t s = nullptr;
    RepDev *d_rep = nullptr;
    Chunk *d_bch = nullptr, *d_cch = nullptr;
    int nbch = 0, ncch = 0;
    Bufs b{};
    int cur = 0;
    // force kernel: 0 = cell tiles in shared memory (half shell), 1 = one thread per bead (full shell)
    int force_kernel = 0;      // 0 cell tiles, 1 thread per bead, 2 cell tiles staged by bulk copies
    int sort_mode = 2;          // see sort_form
    uint32_t *count2[2] = {nullptr, nullptr};  // counts of next positions, one array per buffer parity
    int32_t *bins = nullptr;    // the cells' rows of beads (see k_binfix), null where the boxes have none
    int tile_threads = 256;     // threads per CTA of the tile kernel (256 or 512: tiles of up to that many local cells)
    int tile_w = 8, tile_h = 16;
    TileDesc *d_tiles = nullptr;
    int ntiles = 0;
    std::vector<int32_t> tile0; // first tile of each replica, and the end
    bool any_chem = false;
    bool any_stir = false;      // some replica stirs: its term sums are cleared before each permute
    bool keys_valid = false;
    int64_t step = 0;
    // CUDA graphs of gsteps consecutive steps, one per starting buffer parity
    cudaGraphExec_t gexec[2] = {nullptr, nullptr};
    // the stats ring: every step writes replica ring_rep's row into ring[step % ring_slots]
    unsigned long long *ring = nullptr;
    int32_t ring_rep = 0, ring_slots = 0;
    int gflip[2] = {0, 0};      // buffer parity change of one replay (steps + the extra sorts of catalyst checks)
    int gsteps = 0;
    // the reference's catalyst chemistry: replicas with chem_kind 1, the period of their checks
    bool any_cat = false, any_lipid = false;
    bool any_mol = false;       // some replica has branched lipids (k_mol_forces)
    int stream_grid = 1;        // blocks per replica of the catalyst stream kernel
    int64_t cat_period = 0;
    // reverse-mode storage (adj_layout)
    char *adj_mem = nullptr;    // one allocation, laid out anew by each call that uses it
    size_t adj_bytes = 0;
    int64_t window_mem = -1;    // dpd_set_window_memory (-1: the default rule)
    // staging for state in/out
    char *stage = nullptr;
    int dev = 0;                // the device the handle was made on
    // where copies of the device's status and of a stats row arrive (pageable: pinned memory saves a call 1-2 us and
    // costs the handle 2.5 ms to make)
    struct HostSide {
        DevStatus st;
        unsigned long long row[OBS_N];
    } *host = nullptr;
    // cluster analysis scratch (allocated on first use): union-find parents, sizes, sums
    int *ana_parent = nullptr, *ana_size = nullptr, *ana_min = nullptr;
    int32_t *ana_label = nullptr;
    unsigned long long *ana_acc = nullptr;
    std::vector<void *> allocs;
};

extern "C" const char *dpd_last_error(void) { return g_err.c_str(); }
extern "C" const char *dpd_version(void) { return "libdpd 0.1 (sm_100a)"; }

extern "C" int dpd_params_default(dpd_params *p) {
    if (!p) return fail(DPD_E_ARG, "null params");
    memset(p, 0, sizeof *p);
    p->L = 64.0;   // reference defaults: cel/engine/oercel.c:237-299
    p->dt = 0.03;
    p->lambda = 0.65;
    p->gamma = 4.5;
    p->kT = 1.0;
    for (int i = 0; i < DPD_MAXT * DPD_MAXT; i++) p->a[i] = 25.0;
    p->k_bond = 100.0;
    p->r0 = 0.5;
    p->k_angle = 10.0;
    p->stir_n = 1;
    p->kT_period = 1000.0;
    p->chem_kind = 0;
    p->syn_tries = 8;   // catalyst chemistry: the reference's defaults, oercel.c:262-290
    p->syn_relax = 20;
    p->lip_nH = 1;
    p->lip_nT = 3;
    p->feed_mode = 1;
    p->r_cat = 1.2;
    p->p_syn_a = 0.02;
    p->p_syn_b = 0.06;
    p->p_rep_a = 0.001;
    p->p_rep_b = 0.001;
    p->mu = 0.02;
    p->p_ld = 2e-4;
    p->p_kd = 5e-4;
    p->p_nd = 1e-4;
    p->p_feed = 1e-3;
    p->feed_cap = 0.12;
    p->vent_x = -1.0;
    p->vent_y = -1.0;
    p->vent_r = 5.0;
    p->r0_head = 0.5;
    p->vent_w = 4.0;
    p->seed = 1;
    p->noise = 0;
    p->chem = 0;
    p->n_chem = 1;
    p->n_t_min = 2;
    p->max_chain = 12;  // reference MAXMLEN, oercel.c:50
    p->p_break = 1e-5;
    p->p_grow = 1e-3;
    p->p_bond = 1e-2;
    p->r_grow = 1.0;
    p->r_bond = 0.6;
    return DPD_OK;
}

static uint32_t threshold(double p) {
    const double t = std::floor(p * 4294967296.0);
    if (!(t > 0.0)) return 0u;
    if (t >= 4294967295.0) return 0xFFFFFFFFu;
    return (uint32_t)t;
}

static int make_rep(const dpd_params &p, int b0, int n, int c0, RepDev &R) {
    memset(&R, 0, sizeof R);
    if (!(p.L >= 3.0) || !std::isfinite(p.L)) return fail(DPD_E_ARG, "L must be >= 3 (got %g)", p.L);
    if (!(p.dt > 0.0)) return fail(DPD_E_ARG, "dt must be > 0");
    if (!(p.kT > 0.0)) return fail(DPD_E_ARG, "kT must be > 0");
    if (p.gamma < 0.0) return fail(DPD_E_ARG, "gamma must be >= 0");
    if (p.noise != 0 && p.noise != 1) return fail(DPD_E_ARG, "noise must be 0 (philox) or 1 (mix13)");
    if (p.chem && p.n_chem < 1) return fail(DPD_E_ARG, "n_chem must be >= 1");
    if (p.chem && (p.max_chain < 2 || p.max_chain > 1000)) return fail(DPD_E_ARG, "max_chain must be 2..1000");
    if (p.chem && !(p.r_grow > 0.0 && p.r_grow <= 1.0 && p.r_bond > 0.0 && p.r_bond <= 1.0))
        return fail(DPD_E_ARG, "reaction radii must lie in (0, 1]");
    for (int i = 0; i < DPD_MAXT; i++)
        for (int j = 0; j < DPD_MAXT; j++)
            if (p.a[i * DPD_MAXT + j] != p.a[j * DPD_MAXT + i]) return fail(DPD_E_ARG, "a_ij must be symmetric");
    R.L = (float)p.L;
    R.halfL = 0.5f * R.L;
    R.ncx = R.ncy = (int)std::floor((double)R.L);
    R.icsx = R.ncx / (double)R.L;
    R.icsy = R.ncy / (double)R.L;
    R.b0 = b0;
    R.n = n;
    R.c0 = c0;
    R.ncell = R.ncx * R.ncy;
    R.dt = (float)p.dt;
    R.dt2 = (float)(p.dt * p.dt);
    R.cvt = (float)((0.5 + p.lambda) * p.dt);
    R.hdt = (float)(0.5 * p.dt);
    R.gamma = (float)p.gamma;
    R.sdt = (float)(std::sqrt(2.0 * p.gamma * p.kT) / std::sqrt(p.dt));
    R.kb = (float)p.k_bond;
    R.r0 = (float)p.r0;
    for (int i = 0; i < DPD_MAXT * DPD_MAXT; i++) R.a[i] = (float)p.a[i];
    R.seed = p.seed;
    R.noise = p.noise;
    R.chem = p.chem;
    R.n_chem = p.n_chem;
    R.thr_break = threshold(p.p_break);
    R.thr_grow = threshold(p.p_grow);
    R.thr_bond = threshold(p.p_bond);
    R.r2_grow = (float)(p.r_grow * p.r_grow);
    R.r2_bond = (float)(p.r_bond * p.r_bond);
    R.n_t_min = p.n_t_min;
    R.max_chain = p.max_chain;
    if (p.warmup < 0) return fail(DPD_E_ARG, "warmup must be >= 0");
    R.warm_end = (long long)p.warm_end;
    R.warm_inv = p.warmup > 0 ? 1.0 / (double)p.warmup : 0.0;
    if (p.k_angle < 0.0 || !std::isfinite(p.k_angle)) return fail(DPD_E_ARG, "k_angle must be >= 0");
    R.ka = (float)p.k_angle;
    if (p.stir_A != 0.0 && p.stir_n < 1) return fail(DPD_E_ARG, "stir_n must be >= 1");
    if (!std::isfinite(p.stir_A)) return fail(DPD_E_ARG, "stir_A must be finite");
    R.stir_A = (float)p.stir_A;
    R.stir_k = p.stir_A != 0.0 ? (double)p.stir_n / p.L : 0.0;
    if (p.kT_amp != 0.0) {
        if (!(p.kT_period > 0.0)) return fail(DPD_E_ARG, "kT_period must be > 0");
        if (!(p.kT - std::fabs(p.kT_amp) > 0.0)) return fail(DPD_E_ARG, "kT - |kT_amp| must be > 0");
    }
    R.kT = p.kT;
    R.kT_amp = p.kT_amp;
    R.kT_w = p.kT_amp != 0.0 ? 2.0 * M_PI / p.kT_period : 0.0;
    R.gamma_d = p.gamma;
    R.dt_d = p.dt;
    R.t_anchor = p.t_anchor;
    R.step_anchor = (long long)p.step_anchor;
    R.kb_d = p.k_bond;
    R.r0_d = p.r0;
    R.ka_d = p.k_angle;
    R.chem_kind = p.chem_kind;
    if (p.chem_kind != 0 && p.chem_kind != 1) return fail(DPD_E_ARG, "chem_kind must be 0 (lipid) or 1 (catalyst)");
    // the lipid template: branched shapes need it for their bonds, the catalyst chemistry for new lipids
    dpd_template M;
    const bool need_mol = p.lip_arch != 0 || (p.chem && p.chem_kind == 1);
    if (dpd_lipid_template(&p, &M) != DPD_OK) {
        if (need_mol) return fail(DPD_E_ARG, "lipid shape: lip_arch 0..3 with 2..%d beads (lip_nH >= 1, lip_nT >= 1 "
                                             "for branched shapes)", DPD_MAXML);
        M.mlen = p.lip_nH + p.lip_nT;
        M.nH = p.lip_nH;
    }
    R.arch = p.lip_arch;
    if (p.chem && p.chem_kind == 1) {
        const int ml = M.mlen;
        double ext = 0.0;  // the template's reach from its centroid
        for (int b = 0; b < ml; b++) ext = std::max(ext, std::sqrt(M.px[b] * M.px[b] + M.py[b] * M.py[b]));
        if (!(p.r_cat > 0.0) || p.syn_tries < 1 || p.syn_tries > DPD_CAT_MAXTR || p.syn_relax < 0 || p.syn_nN < 0 ||
            p.syn_nN > ml)
            return fail(DPD_E_ARG, "need r_cat > 0, 1 <= syn_tries <= %d, syn_relax >= 0, 0 <= syn_nN <= mlen",
                        DPD_CAT_MAXTR);
        if (p.feed_mode < 0 || p.feed_mode > 2 || p.vent_kind < 0 || p.vent_kind > 2)
            return fail(DPD_E_ARG, "feed_mode 0..2, vent_kind 0..2");
        if (p.p_feed < 0.0 || p.p_feed > 1.0 || p.feed_cap < 0.0 || p.feed_cap >= 1.0)
            return fail(DPD_E_ARG, "p_feed in [0, 1], feed_cap in [0, 1)");
        // the cells a catalyst's visit can reach: the N window, the new chain's
        // extent around the centroid, and the energy and relaxation windows
        const double reach = 1.0 + 0.05 * p.syn_relax, ics = R.ncx / (double)R.L;
        const int wmax = std::max({(int)std::ceil((p.r_cat + 0.5) * ics), (int)std::ceil(1.5 * ics),
                                   (int)std::ceil((reach + 0.5) * ics)});
        R.cat_E = (int)std::ceil((p.r_cat + ext) * ics) + 2 + wmax;
        if (2 * (int)std::ceil((reach + 0.5) * ics) + 1 > R.ncx)
            return fail(DPD_E_ARG, "box too small for the catalyst windows (L must exceed 2 (r_cat, reach) + 1)");
    }
    R.syn_tries = p.syn_tries;
    R.syn_relax = p.syn_relax;
    R.syn_nN = p.syn_nN;
    R.lip_nH = M.nH;  // heads first, mlen beads (the template's, for every shape)
    R.lip_nT = M.mlen - M.nH;
    R.feed_mode = p.feed_mode;
    R.vent_kind = p.vent_kind;
    R.r_cat = p.r_cat;
    R.p_syn_a = p.p_syn_a;
    R.p_syn_b = p.p_syn_b;
    R.p_rep_a = p.p_rep_a;
    R.p_rep_b = p.p_rep_b;
    R.mu = p.mu;
    R.p_ld = p.p_ld;
    R.p_kd = p.p_kd;
    R.p_nd = p.p_nd;
    R.p_feed = p.p_feed;
    R.feed_cap = p.feed_cap;
    R.vent_x = p.vent_x < 0.0 ? 0.5 * p.L : p.vent_x;  // the reference centres an unset vent (oercel.c:607-608)
    R.vent_y = p.vent_y < 0.0 ? 0.5 * p.L : p.vent_y;
    R.vent_r = p.vent_r;
    R.vent_w = p.vent_w;
    return DPD_OK;
}

template <typename T>
static int dalloc(dpd_handle *h, T **p, size_t count) {
    void *q = nullptr;
    const size_t bytes = count * sizeof(T) + 64;
    cudaError_t e = cudaMalloc(&q, bytes);
    if (e != cudaSuccess) return fail(DPD_E_NOMEM, "cudaMalloc(%zu): %s", bytes, cudaGetErrorString(e));
    h->allocs.push_back(q);
    *p = (T *)q;
    return DPD_OK;
}

#define TRY(x)                       \
    do {                             \
        int r_ = (x);                \
        if (r_ != DPD_OK) return r_; \
    } while (0)

// graph length: with catalyst chemistry a multiple of its period (so that a
// replay starting on a multiple of the period holds the checks in place)
static int graph_len(const dpd_handle *h, int g) {
    g = std::max(1, g);
    const int64_t P = h->cat_period;
    if (P > 0 && P <= 1024) g = (int)(((g + P - 1) / P) * P);
    return g;
}

static void drop_graphs(dpd_handle *h) {
    for (int k = 0; k < 2; k++)
        if (h->gexec[k]) {
            cudaGraphExecDestroy(h->gexec[k]);
            h->gexec[k] = nullptr;
        }
}

static void free_adj(dpd_handle *h) {
    if (h->adj_mem) cudaFree(h->adj_mem);
    h->adj_mem = nullptr;
    h->adj_bytes = 0;
}

static void free_all(dpd_handle *h) {
    drop_graphs(h);
    free_adj(h);
    for (void *p : h->allocs) cudaFree(p);
    h->allocs.clear();
    delete h->host;
    h->host = nullptr;
    if (h->s) cudaStreamDestroy(h->s);
}

// cell tiles of every replica: w x h cells (narrower boxes get narrower tiles,
// so that a tile and its halo never hold the same column or row twice)
static int build_tiles(dpd_handle *h) {
    const int maxc = h->force_kernel == 0 ? h->tile_threads : 256;
    if (h->tile_w < 1 || h->tile_h < 1 || (h->tile_w + 2) * (h->tile_h + 2) > maxc)
        return fail(DPD_E_ARG, "tile shape %dx%d: need (w+2)(h+2) <= %d", h->tile_w, h->tile_h, maxc);
    std::vector<TileDesc> t;
    h->tile0.clear();
    for (int r = 0; r < h->nrep; r++) {
        h->tile0.push_back((int32_t)t.size());
        const RepDev &R = h->rh[r];
        const int w = std::min(h->tile_w, R.ncx - 2), hh = std::min(h->tile_h, R.ncy - 2);
        for (int cx = 0; cx < R.ncx; cx += w)
            for (int cy = 0; cy < R.ncy; cy += hh)
                t.push_back({r, cx, cy, std::min(w, R.ncx - cx), std::min(hh, R.ncy - cy), (int32_t)R.c0, R.ncx, R.ncy});
    }
    h->tile0.push_back((int32_t)t.size());
    for (void *old : {(void *)h->d_tiles, (void *)h->b.rowpart}) {
        if (!old) continue;
        cudaFree(old);
        for (auto &p : h->allocs)
            if (p == old) p = nullptr;
    }
    h->d_tiles = nullptr;
    h->b.rowpart = nullptr;
    TRY(dalloc(h, &h->d_tiles, t.size()));
    TRY(dalloc(h, &h->b.rowpart, t.size() * ROW_WORDS));
    CK(cudaMemcpy(h->d_tiles, t.data(), t.size() * sizeof(TileDesc), cudaMemcpyHostToDevice));
    h->ntiles = (int)t.size();
    return DPD_OK;
}

// The default tile shape: of all shapes up to 256 local cells, the one with the
// least (10 + (w + 1)(h + 2)) x waves.  (w + 1)(h + 2) are the cells whose beads
// a CTA walks (its own and the halo's, less the last column), 10 stands for its
// fixed phases, and the grid runs in waves of 4 CTAs on 148 SMs, at least one,
// in quarters.  Against the best of 32 shapes on seventeen handles from 4,096
// beads to 4.4 M in 256 boxes this picks within 1.5 % of the step's time on
// average (7 % at worst); 8 x 16 halved until there were four tiles an SM was
// within 14 % on average: 25.9 against 20.6 us a step at 65,536 beads, 640
// against 599 on the 256 boxes.  Shapes whose halo would hold more beads than
// the shared memory at the handle's densest replica are left out.
static void choose_tile(dpd_handle *h) {
    double dense = 0.0;
    for (const RepDev &R : h->rh) dense = std::max(dense, (double)R.n / R.ncell);
    double best = 1e300;
    for (int w = 2; w <= 14; w++)
        for (int t = w; t <= 2 * w + 2; t++) {
            const double local = (w + 2.0) * (t + 2.0), beads = local * dense;
            if (local > 256.0 || (beads + 5.0 * std::sqrt(beads) > 1408.0 && best < 1e300)) continue;
            int64_t tiles = 0;
            for (const RepDev &R : h->rh) {
                const int rw = std::min(w, R.ncx - 2), rt = std::min(t, R.ncy - 2);
                tiles += (int64_t)((R.ncx + rw - 1) / rw) * ((R.ncy + rt - 1) / rt);
            }
            const double waves = std::max(1.0, std::ceil(4.0 * tiles / (4 * 148)) / 4.0);
            const double cost = (10.0 + (w + 1.0) * (t + 2.0)) * waves;
            if (cost < best) {
                best = cost;
                h->tile_w = w;
                h->tile_h = t;
            }
        }
}

// The kernels of the cell sort, from the handle's sort_mode and what its boxes
// allow: scan of the counts in two passes or in one, placement and fix-up; a
// block-local scan whose prefixes placement and fix-up add; or the bins.
enum class SortForm { TWO_PASS, LOOK_BACK, PREFIXES, BINS };

static SortForm sort_form(const dpd_handle *h) {
    if (h->sort_mode == 1) return SortForm::LOOK_BACK;
    if (h->sort_mode == 0) return SortForm::TWO_PASS;
    if (h->bins) return SortForm::BINS;
    return sort_pfx_fits(h->C) ? SortForm::PREFIXES : SortForm::TWO_PASS;
}

// b with the counts of buffer parity cur and, for the sort from bins, the bins
static Bufs at_parity(const dpd_handle *h, Bufs b, int cur) {
    b.count = h->count2[cur];
    b.bins = sort_form(h) == SortForm::BINS ? h->bins : nullptr;
    return b;
}

// the row the tile force kernel assembles for the stats ring, if one is registered
static RowOut ring_row(const dpd_handle *h) {
    RowOut row;
    if (!h->ring || h->force_kernel != 0) return row;
    row.rep = h->ring_rep;
    row.slots = h->ring_slots;
    row.host = h->ring;
    row.tile0 = h->tile0[row.rep];
    row.ntile = h->tile0[row.rep + 1] - row.tile0;
    return row;
}

// the stirring sums are accumulated by the permute kernel and read by the forces
static void clear_stir(dpd_handle *h, const Bufs &b) {
    if (h->any_stir) cudaMemsetAsync(b.stir, 0, (size_t)h->nrep * sizeof(long long), h->s);
}

// The sort of buffer cur's counted keys into cell order (cell starts, src,
// dest), with the stirring sums cleared for the permute that follows and row,
// the stats row of the step before, collected.
static void enqueue_cell_sort(dpd_handle *h, const Bufs &b0, int cur, bool step_inc, RowOut row = RowOut()) {
    const Bufs b = at_parity(h, b0, cur);
    StepHead head;
    head.row = row;
    if (h->any_stir) {
        head.stir = b.stir;
        head.nstir = h->nrep;
    }
    const SortForm form = sort_form(h);
    if (form == SortForm::BINS) {
        launch_sort_bins(b, h->count2[cur ^ 1], h->C, step_inc, h->d_cch, h->ncch, -1, head, h->s);
        return;
    }
    if (form == SortForm::PREFIXES) {
        launch_sort_pfx(b, h->C, step_inc, h->d_bch, h->nbch, h->d_cch, h->ncch, -1, head, h->s);
        return;
    }
    if (row.rep >= 0) launch_row_collect(b, row, h->s);
    clear_stir(h, b);
    if (form == SortForm::LOOK_BACK) launch_scan_lb(b, h->C, step_inc, h->s);
    else launch_scan(b, h->C, step_inc, h->s);
    launch_place(b, h->d_bch, h->nbch, h->s);
    launch_cellfix(b, h->d_cch, h->ncch, h->s);
}

// the handle's buffers for a sort by the placement kernels (no bins)
static Bufs plain_counts(const dpd_handle *h) {
    Bufs b = h->b;
    b.count = h->count2[h->cur];
    b.bins = nullptr;
    return b;
}

// clear the counts (both parities, and the crowded cells' lists) and count the
// current (or the next) positions of buffer cur of b
static void enqueue_keys(dpd_handle *h, const Bufs &b0, int cur, bool next) {
    cudaMemsetAsync(h->count2[0], 0, (h->bins ? 3 : 2) * (size_t)CELL_WORDS(h->C) * sizeof(uint32_t), h->s);
    launch_keys(at_parity(h, b0, cur), cur, h->d_rep, h->d_bch, h->nbch, next, h->s);
}

// forces of buffer cur of b.  row: a stats row the tile kernel assembles on the
// way (the other kernels leave it to the caller)
static void enqueue_forces(dpd_handle *h, const Bufs &b0, int cur, bool next_keys,
                           RowOut row = RowOut()) {
    const Bufs b = at_parity(h, b0, cur);
    if (h->any_mol) launch_mol_forces(b, cur, h->d_rep, h->d_bch, h->nbch, h->s);
    if (h->force_kernel == 0)
        launch_forces_tile(b, cur, h->d_rep, h->d_tiles, h->ntiles, h->tile_threads, next_keys, h->s, row);
    else if (h->force_kernel == 2) launch_forces_bulk(b, cur, h->d_rep, h->d_tiles, h->ntiles, next_keys, h->s);
    else launch_forces(b, cur, h->d_rep, h->d_bch, h->nbch, true, true, next_keys, h->s);
}

static int create_impl(dpd_handle *h, const dpd_params *params, int32_t nrep, const int32_t *n_beads) {
    h->nrep = nrep;
    h->params.assign(params, params + nrep);
    h->rh.resize(nrep);
    int64_t b0 = 0, c0 = 0;
    for (int r = 0; r < nrep; r++) {
        if (n_beads[r] < 2) return fail(DPD_E_ARG, "replica %d: need at least 2 beads", r);
        TRY(make_rep(params[r], (int)b0, n_beads[r], (int)c0, h->rh[r]));
        h->any_chem = h->any_chem || params[r].chem;
        h->any_lipid = h->any_lipid || (params[r].chem && params[r].chem_kind == 0);
        if (params[r].chem && params[r].chem_kind == 1) {
            h->any_cat = true;
            const int64_t a = h->cat_period ? h->cat_period : 1, c = params[r].n_chem;
            h->cat_period = a / std::gcd(a, c) * c;
        }
        h->any_stir = h->any_stir || params[r].stir_A != 0.0;
        h->any_mol = h->any_mol || params[r].lip_arch != 0;
        b0 += n_beads[r];
        c0 += h->rh[r].ncell;
        h->nmax = std::max(h->nmax, (int)n_beads[r]);
        if (b0 > (int64_t)GID_MASK || c0 > (int64_t)0x7fffffff - 8)
            return fail(DPD_E_ARG, "too many beads or cells (beads < 2^29 in total)");
    }
    h->N = b0;
    h->C = c0;
    // work chunks: CTAs never straddle replicas
    std::vector<Chunk> bch, cch;
    for (int r = 0; r < nrep; r++) {
        const RepDev &R = h->rh[r];
        h->rh[r].ch0 = (int32_t)bch.size();
        for (int k = 0; k < R.n; k += BEAD_TPB) bch.push_back({r, R.b0 + k, R.b0 + std::min(R.n, k + BEAD_TPB), 0});
        h->rh[r].nch = (int32_t)bch.size() - h->rh[r].ch0;
        for (int k = 0; k < R.ncell; k += CELL_TPB)
            cch.push_back({r, R.c0 + k, R.c0 + std::min(R.ncell, k + CELL_TPB), 0});
    }
    h->nbch = (int)bch.size();
    h->ncch = (int)cch.size();
    CK(cudaStreamCreateWithFlags(&h->s, cudaStreamNonBlocking));
    if (tile_setup() != 0) return fail(DPD_E_CUDA, "cannot reserve %zu bytes of shared memory per CTA", tile_smem_bytes());
    if (const char *e = getenv("DPD_FORCES"))
        h->force_kernel = strcmp(e, "bead") == 0 ? 1 : (strcmp(e, "bulk") == 0 ? 2 : 0);

    choose_tile(h);
    CK(cudaGetDevice(&h->dev));
    h->host = new dpd_handle::HostSide();
    // the handle's arrays, carved from one allocation that is cleared as a whole
    std::vector<std::pair<void **, size_t>> plan;
    auto want = [&](auto **q, size_t count) { plan.push_back({(void **)q, count * sizeof(**q)}); };
    Bufs &b = h->b;
    const size_t N = (size_t)h->N, C = (size_t)h->C;
    want(&h->d_rep, nrep);
    want(&h->d_bch, bch.size());
    want(&h->d_cch, cch.size());
    for (int k = 0; k < 2; k++) {
        want(&b.pos[k], N);
        want(&b.vh[k], N);
        want(&b.vt[k], N);
        want(&b.f[k], N);
        want(&b.tg[k], N);
        want(&b.link[k], N);
    }
    want(&b.key, N);
    want(&b.fill, C + 4);
    want(&b.src, N);
    want(&b.dest, N);
    // Bins up to ten beads a cell: a row of 32 is then too short for about one cell in 10^8 of a random soup (denser
    // boxes keep the placement kernel); and up to 196,608 cells, where the kernel saved is worth more than the force
    // kernel's wait for the counts: 13.3 against 18.3 us a step at 1,024 cells, 21.4 (26.1) at 16,384, 44.0 (47.0) at
    // 65,536, 88.9 (91.0) at 176,400, but 126.2 (120.7) at 262,144.
    double dense = 0.0;
    for (int r = 0; r < nrep; r++) dense = std::max(dense, (double)h->rh[r].n / h->rh[r].ncell);
    const bool bins = dense <= 10.0 && C <= 196608;
    // the counts of both parities and, with bins, the crowded cells' lists (these are cleared together), the rows and
    // the lists' links: one array, each part on a 16-byte boundary
    want(&h->count2[0], bins ? 3 * CELL_WORDS(C) + C * BIN_CAP + N : 2 * CELL_WORDS(C));
    want(&b.cstart, C + 4);
    want(&b.bsum, C / SCAN_PER_BLOCK + 2);
    want(&b.scan_state, C / SCAN_PER_BLOCK + 2);
    want(&b.scan_ticket, 1);
    want(&b.claim, N);
    want(&b.req, N);
    want(&b.grow_list, N);
    want(&b.bond_list, N);
    b.evcap = 1 << 20;
    want(&b.events, (size_t)b.evcap);
    want(&b.status, 1);
    want(&b.step, 1);
    want(&b.obs, (size_t)nrep * OBS_N);
    want(&b.obs_out, (size_t)nrep * OBS_N);
    want(&b.obs_done, (size_t)nrep);
    want(&b.row_pending, 1);
    want(&b.hist, 4096);
    want(&b.stir, (size_t)nrep);
    want(&b.rng, (size_t)4 * nrep);
    want(&b.cat_list, N);
    want(&b.cat_cnt, (size_t)h->nbch + 1);
    want(&b.cat_ncnt, (size_t)h->nbch + 1);
    want(&b.resort, (size_t)nrep + 1);
    want(&b.cat_nk, (size_t)nrep);
    want(&b.cat_near, N);
    want(&b.cat_cell, N);
    want(&b.cat_mark, C);
    want(&b.fmol, N);
    uint64_t *dj = nullptr;
    std::vector<uint64_t> jt;
    if (h->any_cat) {
        // the catalyst checks' draw streams: 3 n + 4096 draws per replica, 64-draw blocks
        long long so = 0;
        int nblk = 1;
        for (int r = 0; r < nrep; r++) {
            const int dcap = (int)((3ll * h->rh[r].n + 4096 + 63) / 64 * 64);
            h->rh[r].so = so;
            h->rh[r].dcap = dcap;
            so += dcap;
            nblk = std::max(nblk, dcap / 64);
        }
        if (jump_table(nblk, jt) != 0) return fail(DPD_E_STATE, "xoshiro256** polynomial not found");
        want(&dj, jt.size());
        want(&b.stream, (size_t)so);
        want(&b.sblock, (size_t)so / 16);
        want(&b.cat_dn, (size_t)nrep);
        want(&b.shuf, 8 * N);
        b.shuf_n = (long long)N;
        h->stream_grid = (nblk + 255) / 256;
    }
    dpd_template *dm = nullptr;
    want(&dm, (size_t)nrep);
    // staging for set/get state: 8 float + 3 int32 + 1 byte arrays of nmax
    want(&h->stage, (size_t)h->nmax * (8 * 4 + 3 * 4 + 1) + 16 * 256);
    size_t total = 0;
    for (auto &q : plan) total += (q.second + 64 + 255) & ~(size_t)255;
    char *base = nullptr;
    TRY(dalloc(h, &base, total));
    CK(cudaMemset(base, 0, total));
    for (auto &q : plan) {
        *q.first = base;
        base += (q.second + 64 + 255) & ~(size_t)255;
    }
    h->count2[1] = h->count2[0] + CELL_WORDS(C);
    if (bins) h->bins = (int32_t *)(h->count2[1] + 2 * CELL_WORDS(C));
    b.cells = (int32_t)C;
    b.jump = dj;
    b.mol = dm;
    CK(cudaMemcpy(h->d_rep, h->rh.data(), nrep * sizeof(RepDev), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(h->d_bch, bch.data(), bch.size() * sizeof(Chunk), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(h->d_cch, cch.data(), cch.size() * sizeof(Chunk), cudaMemcpyHostToDevice));
    if (dj) CK(cudaMemcpy(dj, jt.data(), jt.size() * sizeof(uint64_t), cudaMemcpyHostToDevice));
    std::vector<dpd_template> mols(nrep);
    for (int r = 0; r < nrep; r++)
        if (dpd_lipid_template(&h->params[r], &mols[r]) != DPD_OK) std::memset(&mols[r], 0, sizeof(dpd_template));
    CK(cudaMemcpy(dm, mols.data(), (size_t)nrep * sizeof(dpd_template), cudaMemcpyHostToDevice));
    if (h->any_cat && catalyst_setup() != 0)
        return fail(DPD_E_CUDA, "cannot reserve shared memory for the catalyst kernel");
    CK(cudaMemset(b.claim, 0xFF, N * sizeof(uint32_t)));
    CK(cudaMemset(b.req, 0xFF, N * sizeof(int32_t)));
    for (int k = 0; k < 2; k++) CK(cudaMemset(b.link[k], 0xFF, N * sizeof(int2)));
    // graph length: even (the buffers alternate every step), ~4M bead-steps per replay
    int g = (int)std::max<int64_t>(1, std::min<int64_t>(64, (4 << 20) / std::max<int64_t>(1, h->N)));
    if (const char *e = getenv("DPD_GRAPH_STEPS")) g = atoi(e);
    h->gsteps = graph_len(h, g);
    TRY(build_tiles(h));
    return DPD_OK;
}

extern "C" int dpd_create(const dpd_params *params, int32_t n_replicas, const int32_t *n_beads, dpd_handle **out) {
    if (!params || !n_beads || !out || n_replicas < 1) return fail(DPD_E_ARG, "bad arguments to dpd_create");
    *out = nullptr;
    dpd_handle *h = new dpd_handle();
    const int r = create_impl(h, params, n_replicas, n_beads);
    if (r != DPD_OK) {
        free_all(h);
        delete h;
        return r;
    }
    *out = h;
    return DPD_OK;
}

extern "C" int dpd_destroy(dpd_handle *h) {
    if (!h) return DPD_OK;
    cudaStreamSynchronize(h->s);
    free_all(h);
    delete h;
    return DPD_OK;
}

extern "C" int dpd_sizes(const dpd_handle *h, int32_t r, int64_t *n_total, int32_t *n_beads, int32_t *n_cells) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    if (n_total) *n_total = h->N;
    if (r >= 0 && r < h->nrep) {
        if (n_beads) *n_beads = h->rh[r].n;
        if (n_cells) *n_cells = h->rh[r].ncell;
    } else if (n_beads || n_cells) {
        return fail(DPD_E_ARG, "replica %d out of range", r);
    }
    return DPD_OK;
}

// ---------------------------------------------------------------- status

static int check_status(dpd_handle *h) {
    CK(cudaMemcpyAsync(&h->host->st, h->b.status, sizeof(DevStatus), cudaMemcpyDeviceToHost, h->s));
    CK(cudaStreamSynchronize(h->s));
    const DevStatus st = h->host->st;
    if (st.flags) {
        CK(cudaMemsetAsync(&h->b.status->flags, 0, sizeof(unsigned), h->s));
        CK(cudaStreamSynchronize(h->s));
        if (st.flags & DPD_F_WAIT)
            return fail(DPD_E_TIMEOUT, "a bounded device wait gave up (bulk copies of the force kernel, or the scan)");
        if (st.flags & DPD_F_ANALYSIS) return fail(DPD_E_STATE, "cluster analysis did not converge");
        if (st.flags & DPD_F_CATALYST)
            return fail(DPD_E_STATE, "a catalyst's neighbourhood did not fit the staging area, or a search found "
                                     "more than 256 candidates or 512 relaxation neighbours (too crowded)");
        if (st.flags & DPD_F_TILE)
            return fail(DPD_E_SORT_OVERFLOW, "a cell tile and its halo held more beads than fit in shared memory");
        if (st.flags & DPD_F_FORCE) return fail(DPD_E_STATE, "a pair or bond force above 2048 (fixed-point range)");
        if (st.flags & DPD_F_NONFINITE) return fail(DPD_E_STATE, "non-finite force (flags 0x%x)", st.flags);
        if (st.flags & DPD_F_OUTSIDE)
            return fail(DPD_E_STATE, "a bead moved more than one box length in one step (flags 0x%x)", st.flags);
        if (st.flags & DPD_F_EVENTS)
            return fail(DPD_E_EVENT_OVERFLOW, "event buffer full (%u events since the last read)", st.nevents);
        if (st.flags & DPD_F_CHAIN) return fail(DPD_E_CHAIN, "broken lipid chain");
    }
    return DPD_OK;
}

static int ensure_replica(const dpd_handle *h, int r) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    if (r < 0 || r >= h->nrep) return fail(DPD_E_ARG, "replica %d out of range (0..%d)", r, h->nrep - 1);
    return DPD_OK;
}

// ---------------------------------------------------------------- state in/out

struct ArrayArg {
    const void *p;
    size_t bytes, align;
};

// Are all of these (null ones aside) arrays in one allocation each on the
// handle's device, aligned for its kernels?  They can then be read or written
// in place; anything else goes through the staging arrays and copies that take
// any pointer, and that refuse an array which is shorter than the replica.
// An array in the allocation of the one before needs no lookup (0.3 us).
static bool on_device(const dpd_handle *h, std::initializer_list<ArrayArg> args) {
    static const auto attributes = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuPointerGetAttributes", &f, cudaEnableDefault, &found) != cudaSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return (decltype(&cuPointerGetAttributes))f;
    }();
    if (!attributes) return false;
    CUdeviceptr start = 0;
    size_t size = 0;
    for (const ArrayArg &a : args) {
        if (!a.p) continue;
        if ((uintptr_t)a.p % a.align != 0) return false;
        auto inside = [&] {
            const size_t at = (size_t)((CUdeviceptr)a.p - start);  // (wraps before the start)
            return at <= size && size - at >= a.bytes;
        };
        if (size && inside()) continue;
        unsigned type = 0, managed = 0;
        int dev = -1;
        CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                      CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                      CU_POINTER_ATTRIBUTE_RANGE_SIZE};
        void *got[] = {&type, &managed, &dev, &start, &size};
        if (attributes(sizeof(what) / sizeof(what[0]), what, got, (CUdeviceptr)a.p) != CUDA_SUCCESS ||
            type != CU_MEMORYTYPE_DEVICE || managed || dev != h->dev || !inside())
            return false;
    }
    return true;
}

extern "C" int dpd_set_state(dpd_handle *h, int32_t r, const float *x, const float *y, const float *vx,
                             const float *vy, const uint8_t *type, const uint32_t *gid, const int32_t *prev,
                             const int32_t *next) {
    TRY(ensure_replica(h, r));
    if (!x || !y || !vx || !vy || !type) return fail(DPD_E_ARG, "x, y, vx, vy and type are required");
    const RepDev &R = h->rh[r];
    const size_t n = (size_t)R.n, a = ((n * 4 + 255) / 256) * 256;
    char *p = h->stage;
    float *sx = (float *)p, *sy = (float *)(p + a), *svx = (float *)(p + 2 * a), *svy = (float *)(p + 3 * a);
    uint32_t *sg = (uint32_t *)(p + 4 * a);
    int32_t *sp = (int32_t *)(p + 5 * a), *sn = (int32_t *)(p + 6 * a);
    uint8_t *st = (uint8_t *)(p + 7 * a);
    const size_t w = n * 4;
    if (on_device(h, {{x, w, 4}, {y, w, 4}, {vx, w, 4}, {vy, w, 4}, {type, n, 1}, {gid, w, 4}, {prev, w, 4},
                      {next, w, 4}})) {
        launch_pack(h->b, h->cur, R.b0, (int)n, R.L, x, y, vx, vy, type, gid, prev, next, h->s);
    } else {
        CK(cudaMemcpyAsync(sx, x, n * 4, cudaMemcpyDefault, h->s));
        CK(cudaMemcpyAsync(sy, y, n * 4, cudaMemcpyDefault, h->s));
        CK(cudaMemcpyAsync(svx, vx, n * 4, cudaMemcpyDefault, h->s));
        CK(cudaMemcpyAsync(svy, vy, n * 4, cudaMemcpyDefault, h->s));
        CK(cudaMemcpyAsync(st, type, n, cudaMemcpyDefault, h->s));
        if (gid) CK(cudaMemcpyAsync(sg, gid, n * 4, cudaMemcpyDefault, h->s));
        if (prev) CK(cudaMemcpyAsync(sp, prev, n * 4, cudaMemcpyDefault, h->s));
        if (next) CK(cudaMemcpyAsync(sn, next, n * 4, cudaMemcpyDefault, h->s));
        launch_pack(h->b, h->cur, R.b0, (int)n, R.L, sx, sy, svx, svy, st, gid ? sg : nullptr, prev ? sp : nullptr,
                    next ? sn : nullptr, h->s);
    }
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(&h->host->st, h->b.status, sizeof(DevStatus), cudaMemcpyDeviceToHost, h->s));
    CK(cudaStreamSynchronize(h->s));
    h->keys_valid = false;
    unsigned flags = h->host->st.flags;
    if (flags & DPD_F_INPUT) {
        flags &= ~DPD_F_INPUT;
        CK(cudaMemcpy(&h->b.status->flags, &flags, sizeof flags, cudaMemcpyHostToDevice));
        return fail(DPD_E_ARG, "set_state: a non-finite position, a type >= %d, a gid >= n or a link outside "
                               "[-1, n) (replica %d)", DPD_MAXT, r);
    }
    return DPD_OK;
}

extern "C" int dpd_get_state(dpd_handle *h, int32_t r, float *x, float *y, float *vhx, float *vhy, float *vtx,
                             float *vty, float *fx, float *fy, uint8_t *type, uint32_t *gid, int32_t *prev,
                             int32_t *next) {
    TRY(ensure_replica(h, r));
    const RepDev &R = h->rh[r];
    const size_t n = (size_t)R.n, a = ((n * 4 + 255) / 256) * 256;
    const size_t w = n * 4;
    if (on_device(h, {{x, w, 4}, {y, w, 4}, {vhx, w, 4}, {vhy, w, 4}, {vtx, w, 4}, {vty, w, 4}, {fx, w, 4}, {fy, w, 4},
                      {type, n, 1}, {gid, w, 4}, {prev, w, 4}, {next, w, 4}})) {
        launch_unpack(h->b, h->cur, R.b0, (int)n, x, y, vhx, vhy, vtx, vty, fx, fy, type, gid, prev, next, h->s);
        CK(cudaGetLastError());
        CK(cudaStreamSynchronize(h->s));
        return DPD_OK;
    }
    char *p = h->stage;
    float *f8[8];
    for (int k = 0; k < 8; k++) f8[k] = (float *)(p + k * a);
    uint32_t *sg = (uint32_t *)(p + 8 * a);
    int32_t *sp = (int32_t *)(p + 9 * a), *sn = (int32_t *)(p + 10 * a);
    uint8_t *st = (uint8_t *)(p + 11 * a);
    launch_unpack(h->b, h->cur, R.b0, (int)n, f8[0], f8[1], f8[2], f8[3], f8[4], f8[5], f8[6], f8[7], st, sg, sp,
                  sn, h->s);
    CK(cudaGetLastError());
    float *outs[8] = {x, y, vhx, vhy, vtx, vty, fx, fy};
    for (int k = 0; k < 8; k++)
        if (outs[k]) CK(cudaMemcpyAsync(outs[k], f8[k], n * 4, cudaMemcpyDefault, h->s));
    if (type) CK(cudaMemcpyAsync(type, st, n, cudaMemcpyDefault, h->s));
    if (gid) CK(cudaMemcpyAsync(gid, sg, n * 4, cudaMemcpyDefault, h->s));
    if (prev) CK(cudaMemcpyAsync(prev, sp, n * 4, cudaMemcpyDefault, h->s));
    if (next) CK(cudaMemcpyAsync(next, sn, n * 4, cudaMemcpyDefault, h->s));
    CK(cudaStreamSynchronize(h->s));
    return DPD_OK;
}

extern "C" int dpd_set_dynamics(dpd_handle *h, int32_t r, const float *vhx, const float *vhy, const float *fx,
                                const float *fy, const float *vtx, const float *vty) {
    TRY(ensure_replica(h, r));
    const RepDev &R = h->rh[r];
    const size_t n = (size_t)R.n, a = ((n * 4 + 255) / 256) * 256;
    const float *in[6] = {vhx, vhy, fx, fy, vtx, vty};
    float *sg[6];
    for (int k = 0; k < 6; k++) {
        sg[k] = (float *)(h->stage + k * a);
        if (in[k]) CK(cudaMemcpyAsync(sg[k], in[k], n * 4, cudaMemcpyDefault, h->s));
    }
    launch_set_dynamics(h->b, h->cur, R.b0, (int)n, vhx ? sg[0] : nullptr, vhy ? sg[1] : nullptr,
                        fx ? sg[2] : nullptr, fy ? sg[3] : nullptr, vtx ? sg[4] : nullptr, vty ? sg[5] : nullptr,
                        h->s);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(h->s));
    h->keys_valid = false;
    return DPD_OK;
}

// ---------------------------------------------------------------- phases

static void enqueue_sort(dpd_handle *h, PermuteMode mode) {
    // counts of the CURRENT positions
    enqueue_keys(h, h->b, h->cur, false);
    enqueue_cell_sort(h, h->b, h->cur, false);
    launch_permute(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, mode, h->s);
    h->cur ^= 1;
}

static int set_device_step(dpd_handle *h, int64_t step) {
    launch_set_step(h->b.step, (long long)step, h->s);
    CK(cudaGetLastError());
    h->step = step;
    return DPD_OK;
}

static void enqueue_next_keys(dpd_handle *h) {
    enqueue_keys(h, h->b, h->cur, true);
    h->keys_valid = true;
}

extern "C" int dpd_prime(dpd_handle *h) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    enqueue_sort(h, PERM_PRIME);
    enqueue_forces(h, h->b, h->cur, false);
    launch_halfkick(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, h->s);
    enqueue_next_keys(h);
    CK(cudaGetLastError());
    return check_status(h);
}

extern "C" int dpd_resume(dpd_handle *h) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    enqueue_sort(h, PERM_SORT);
    enqueue_next_keys(h);
    CK(cudaGetLastError());
    return check_status(h);
}

extern "C" int dpd_get_step(const dpd_handle *h, int64_t *step) {
    if (!h || !step) return fail(DPD_E_ARG, "null argument");
    *step = h->step;
    return DPD_OK;
}

extern "C" int dpd_set_step(dpd_handle *h, int64_t step) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    return set_device_step(h, step);
}

extern "C" int dpd_build_cells(dpd_handle *h) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    enqueue_sort(h, PERM_SORT);
    h->keys_valid = false;
    CK(cudaGetLastError());
    return check_status(h);
}

extern "C" int dpd_get_cells(dpd_handle *h, int32_t r, int32_t *cstart) {
    TRY(ensure_replica(h, r));
    if (!cstart) return fail(DPD_E_ARG, "null cstart");
    const RepDev &R = h->rh[r];
    std::vector<int32_t> tmp(R.ncell + 1);
    CK(cudaMemcpyAsync(tmp.data(), h->b.cstart + R.c0, (R.ncell + 1) * sizeof(int32_t), cudaMemcpyDeviceToHost,
                       h->s));
    CK(cudaStreamSynchronize(h->s));
    for (auto &v : tmp) v -= R.b0;
    CK(cudaMemcpy(cstart, tmp.data(), tmp.size() * sizeof(int32_t), cudaMemcpyDefault));
    return DPD_OK;
}

extern "C" int dpd_forces(dpd_handle *h, int64_t step) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    TRY(set_device_step(h, step));
    enqueue_forces(h, h->b, h->cur, false);
    h->keys_valid = false;
    CK(cudaGetLastError());
    return check_status(h);
}

static int partial_forces(dpd_handle *h, int32_t r, bool pair, bool bond, float *fx, float *fy) {
    // computed into the spare force buffer so the stored forces stay untouched
    Bufs b = h->b;
    b.f[h->cur] = h->b.f[h->cur ^ 1];
    if (bond && h->any_mol) launch_mol_forces(b, h->cur, h->d_rep, h->d_bch, h->nbch, h->s);
    launch_forces(b, h->cur, h->d_rep, h->d_bch, h->nbch, pair, bond, false, h->s);
    CK(cudaGetLastError());
    const RepDev &R = h->rh[r];
    const size_t n = (size_t)R.n, a = ((n * 4 + 255) / 256) * 256;
    float *sx = (float *)h->stage, *sy = (float *)(h->stage + a);
    Bufs u = h->b;
    u.f[h->cur] = b.f[h->cur];
    launch_unpack(u, h->cur, R.b0, (int)n, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, sx, sy, nullptr,
                  nullptr, nullptr, nullptr, h->s);
    CK(cudaGetLastError());
    if (fx) CK(cudaMemcpyAsync(fx, sx, n * 4, cudaMemcpyDefault, h->s));
    if (fy) CK(cudaMemcpyAsync(fy, sy, n * 4, cudaMemcpyDefault, h->s));
    CK(cudaStreamSynchronize(h->s));
    return check_status(h);
}

extern "C" int dpd_pair_forces(dpd_handle *h, int32_t r, int64_t step, float *fx, float *fy) {
    TRY(ensure_replica(h, r));
    TRY(set_device_step(h, step));
    return partial_forces(h, r, true, false, fx, fy);
}

extern "C" int dpd_bond_forces(dpd_handle *h, int32_t r, float *fx, float *fy, float *maxbond) {
    TRY(ensure_replica(h, r));
    unsigned long long *slot = h->b.obs + (size_t)r * OBS_N + 4;
    CK(cudaMemsetAsync(slot, 0, sizeof(unsigned long long), h->s));
    TRY(partial_forces(h, r, false, true, fx, fy));
    if (maxbond) {
        unsigned long long v = 0;
        CK(cudaMemcpy(&v, slot, sizeof v, cudaMemcpyDeviceToHost));
        uint32_t bits = (uint32_t)v;
        memcpy(maxbond, &bits, 4);
    }
    return DPD_OK;
}

extern "C" int dpd_integrate(dpd_handle *h) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    launch_integrate(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, h->s);
    h->keys_valid = false;
    CK(cudaGetLastError());
    return check_status(h);
}

extern "C" int dpd_chemistry(dpd_handle *h, int64_t step) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    TRY(set_device_step(h, step));
    CK(cudaMemsetAsync(&h->b.status->n_grow, 0, 2 * sizeof(unsigned), h->s));
    launch_chem_scan(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, h->s);
    launch_chem_lists(h->b, h->cur, h->d_rep, h->s);
    // the catalyst chemistry as the reference's chemistry(): no sort afterwards
    if (h->any_cat) launch_catalyst(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, h->nrep, h->C, h->nmax, h->stream_grid, h->s);
    CK(cudaGetLastError());
    return check_status(h);
}

// ---------------------------------------------------------------- the step

// does a catalyst check of some replica fall on step s
static bool cat_at(const dpd_handle *h, int64_t s) {
    if (!h->any_cat) return false;
    for (const auto &p : h->params)
        if (p.chem && p.chem_kind == 1 && p.n_chem > 0 && s % p.n_chem == 0) return true;
    return false;
}

// one step producing step number s.  A step with a catalyst check follows the
// reference's order (oercel.c:2337-2349): the update with every bead kept in
// the slot of the last sort, the check on that order and cell index (the
// catalysts and the food candidates are taken in slot order), then the sort of
// the new configuration.  A replica in which a bead moved 0.5 or more is
// sorted before its check too (launch_resort, no-ops otherwise).  Other steps
// fuse the update into the sort whose counts the previous force kernel made.
static void enqueue_step(dpd_handle *h, int64_t s) {
    const bool cat = cat_at(h, s);
    const RowOut row = ring_row(h);
    if (!cat) {
        enqueue_cell_sort(h, h->b, h->cur, true, row);
    } else {
        if (row.rep >= 0) launch_row_collect(h->b, row, h->s);
        launch_step_begin(h->b, h->nrep, h->s);
        clear_stir(h, h->b);
    }
    launch_permute(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, cat ? PERM_KEEP : PERM_STEP, h->s);
    h->cur ^= 1;
    if (h->any_lipid) launch_chem_lists(h->b, h->cur, h->d_rep, h->s);
    if (cat) {
        launch_resort(plain_counts(h), h->cur, h->d_rep, h->d_bch, h->nbch, h->d_cch, h->ncch, h->C, h->s);
        launch_catalyst(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, h->nrep, h->C, h->nmax, h->stream_grid, h->s);
        enqueue_sort(h, PERM_SORT);
    }
    // the step's stats row into the ring: assembled by the tile force kernel's
    // epilogue from the beads it holds anyway, else by a pass of its own
    if (row.rep >= 0) {
        enqueue_forces(h, h->b, h->cur, true, row);
    } else {
        enqueue_forces(h, h->b, h->cur, true);
        if (h->ring)
            launch_observables(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, h->ring_rep, false, h->ring, h->ring_slots,
                               h->s);
    }
}

// capture gsteps steps starting from the current buffer parity and step s0
// (with catalyst chemistry s0 is a multiple of its period: the graph then
// holds the checks at the same places on every replay)
static int build_graph(dpd_handle *h, int64_t s0) {
    const int cur0 = h->cur;
    if (h->gexec[cur0]) {
        CK(cudaGraphExecDestroy(h->gexec[cur0]));
        h->gexec[cur0] = nullptr;
    }
    cudaGraph_t g = nullptr;
    CK(cudaStreamBeginCapture(h->s, cudaStreamCaptureModeThreadLocal));
    for (int k = 0; k < h->gsteps; k++) enqueue_step(h, s0 + 1 + k);
    const cudaError_t e = cudaStreamEndCapture(h->s, &g);
    h->gflip[cur0] = h->cur ^ cur0;
    h->cur = cur0;  // capture only recorded the launches
    if (e != cudaSuccess) return fail(DPD_E_CUDA, "graph capture: %s", cudaGetErrorString(e));
    const cudaError_t e2 = cudaGraphInstantiate(&h->gexec[cur0], g, 0);
    cudaGraphDestroy(g);
    if (e2 != cudaSuccess) return fail(DPD_E_CUDA, "graph instantiate: %s", cudaGetErrorString(e2));
    return DPD_OK;
}

// enqueue nsteps steps: whole graphs while they fit, eager launches for the rest
static int enqueue_steps(dpd_handle *h, int64_t nsteps) {
    if (nsteps < 0) return fail(DPD_E_ARG, "nsteps must be >= 0");
    if (nsteps == 0) return DPD_OK;
    if (!h->keys_valid) enqueue_next_keys(h);
    int64_t left = nsteps, s = h->step;
    const int64_t P = h->cat_period;
    const bool graphs = getenv("DPD_NO_GRAPH") == nullptr && (P == 0 || h->gsteps % P == 0);
    while (left > 0) {
        if (graphs && left >= h->gsteps && (P == 0 || s % P == 0)) {
            if (!h->gexec[h->cur]) TRY(build_graph(h, s));
            CK(cudaGraphLaunch(h->gexec[h->cur], h->s));
            h->cur ^= h->gflip[h->cur];
            left -= h->gsteps;
            s += h->gsteps;
        } else {
            enqueue_step(h, s + 1);
            left--;
            s++;
        }
    }
    const RowOut row = ring_row(h);
    if (row.rep >= 0) launch_row_collect(h->b, row, h->s);  // the last step's row
    CK(cudaGetLastError());
    h->step += nsteps;
    return DPD_OK;
}

extern "C" int dpd_step(dpd_handle *h, int64_t nsteps) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    TRY(enqueue_steps(h, nsteps));
    return check_status(h);
}

extern "C" int dpd_step_async(dpd_handle *h, int64_t nsteps) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    return enqueue_steps(h, nsteps);
}

extern "C" int dpd_sync(dpd_handle *h) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    return check_status(h);
}

extern "C" int dpd_set_tuning(dpd_handle *h, const dpd_tuning *t) {
    if (!h || !t) return fail(DPD_E_ARG, "null argument");
    if (t->force_kernel < 0 || t->force_kernel > 2) return fail(DPD_E_ARG, "force_kernel must be 0, 1 or 2");
    if (t->force_kernel == 2 && t->tile_w + 2 > 32)
        return fail(DPD_E_ARG, "the bulk-staged force kernel takes tiles of at most 30 columns");
    if (t->graph_steps < 1) return fail(DPD_E_ARG, "graph_steps must be >= 1");
    if (t->sort_mode < 0 || t->sort_mode > 2) return fail(DPD_E_ARG, "sort_mode must be 0, 1 or 2");
    if (t->tile_threads != 256 && t->tile_threads != 512) return fail(DPD_E_ARG, "tile_threads must be 256 or 512");
    CK(cudaStreamSynchronize(h->s));
    const int ow = h->tile_w, oh = h->tile_h, ofk = h->force_kernel, ott = h->tile_threads;
    h->tile_w = t->tile_w;
    h->tile_h = t->tile_h;
    h->force_kernel = t->force_kernel;
    h->tile_threads = t->tile_threads;
    const int r = build_tiles(h);
    if (r != DPD_OK) {
        h->tile_w = ow;
        h->tile_h = oh;
        h->force_kernel = ofk;
        h->tile_threads = ott;
        build_tiles(h);
        return r;
    }
    if (t->sort_mode != h->sort_mode) h->keys_valid = false;  // the modes keep the next keys differently
    h->sort_mode = t->sort_mode;
    h->gsteps = graph_len(h, t->graph_steps);
    drop_graphs(h);
    return DPD_OK;
}

extern "C" int dpd_get_tuning(const dpd_handle *h, dpd_tuning *t) {
    if (!h || !t) return fail(DPD_E_ARG, "null argument");
    t->force_kernel = h->force_kernel;
    t->tile_w = h->tile_w;
    t->tile_h = h->tile_h;
    t->graph_steps = h->gsteps;
    t->sort_mode = h->sort_mode;
    t->tile_threads = h->tile_threads;
    return DPD_OK;
}

extern "C" int dpd_set_graph_steps(dpd_handle *h, int32_t steps) {
    if (!h || steps < 1) return fail(DPD_E_ARG, "graph length must be >= 1");
    CK(cudaStreamSynchronize(h->s));
    drop_graphs(h);
    h->gsteps = graph_len(h, steps);
    return DPD_OK;
}

// One step launched kernel by kernel with CUDA events between the launches on
// the handle's stream; ms[k] = device time of kernel k (scan1 (the whole scan
// in one pass, or the block-local one; 0 ms where the sort is one kernel),
// scan2 (0 ms but for the scan in two passes), place (0 ms with bins), cellfix,
// permute, [2 chemistry], [catalyst check + its sort], forces).  The step is a
// real step; on a step with a catalyst check the first entry is the
// step counter's kernel, the next three are not launched (0 ms) and the
// permute keeps the slot order.
extern "C" int dpd_profile_step(dpd_handle *h, float *ms, int32_t cap, int32_t *n_out) {
    if (!h || !ms || !n_out) return fail(DPD_E_ARG, "null argument");
    if (!h->keys_valid) enqueue_next_keys(h);
    const bool cat = cat_at(h, h->step + 1);
    const int nk = 6 + (h->any_lipid ? 2 : 0) + (cat ? 1 : 0);
    if (cap < nk) return fail(DPD_E_ARG, "need room for %d kernel times", nk);
    std::vector<cudaEvent_t> ev(nk + 1);
    for (auto &e : ev) CK(cudaEventCreate(&e));
    int k = 0;
    CK(cudaEventRecord(ev[k++], h->s));
    const Bufs sb = at_parity(h, h->b, h->cur);
    uint32_t *other = h->count2[h->cur ^ 1];
    const SortForm form = sort_form(h);
    const bool bins = form == SortForm::BINS, pfx = form == SortForm::PREFIXES;
    if (!cat) {
        if (bins) launch_sort_bins(sb, other, h->C, true, h->d_cch, h->ncch, 0, StepHead(), h->s);
        else if (pfx) launch_sort_pfx(sb, h->C, true, h->d_bch, h->nbch, h->d_cch, h->ncch, 0, StepHead(), h->s);
        else if (form == SortForm::LOOK_BACK) launch_scan_lb(sb, h->C, true, h->s);
        else launch_scan_part(sb, h->C, true, 1, h->s);
    } else {
        launch_step_begin(h->b, h->nrep, h->s);
    }
    CK(cudaEventRecord(ev[k++], h->s));
    if (!cat && form == SortForm::TWO_PASS) launch_scan_part(sb, h->C, true, 2, h->s);
    CK(cudaEventRecord(ev[k++], h->s));
    if (!cat && !bins) {
        if (pfx) launch_sort_pfx(sb, h->C, true, h->d_bch, h->nbch, h->d_cch, h->ncch, 1, StepHead(), h->s);
        else launch_place(sb, h->d_bch, h->nbch, h->s);
    }
    CK(cudaEventRecord(ev[k++], h->s));
    if (!cat) {
        if (bins) launch_sort_bins(sb, other, h->C, true, h->d_cch, h->ncch, 1, StepHead(), h->s);
        else if (pfx) launch_sort_pfx(sb, h->C, true, h->d_bch, h->nbch, h->d_cch, h->ncch, 2, StepHead(), h->s);
        else launch_cellfix(sb, h->d_cch, h->ncch, h->s);
    }
    CK(cudaEventRecord(ev[k++], h->s));
    clear_stir(h, h->b);
    launch_permute(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, cat ? PERM_KEEP : PERM_STEP, h->s);
    CK(cudaEventRecord(ev[k++], h->s));
    h->cur ^= 1;
    if (h->any_lipid) {  // one kernel; the second chemistry entry is 0
        launch_chem_lists(h->b, h->cur, h->d_rep, h->s);
        for (int c = 0; c < 2; c++) CK(cudaEventRecord(ev[k++], h->s));
    }
    if (cat) {
        launch_resort(plain_counts(h), h->cur, h->d_rep, h->d_bch, h->nbch, h->d_cch, h->ncch, h->C, h->s);
        launch_catalyst(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, h->nrep, h->C, h->nmax, h->stream_grid, h->s);
        enqueue_sort(h, PERM_SORT);
        CK(cudaEventRecord(ev[k++], h->s));
    }
    enqueue_forces(h, h->b, h->cur, true);
    CK(cudaEventRecord(ev[k++], h->s));
    CK(cudaGetLastError());
    CK(cudaEventSynchronize(ev[nk]));
    for (int q = 0; q < nk; q++) CK(cudaEventElapsedTime(&ms[q], ev[q], ev[q + 1]));
    for (auto &e : ev) cudaEventDestroy(e);
    h->step += 1;
    *n_out = nk;
    return check_status(h);
}

extern "C" int dpd_type_clusters(dpd_handle *h, int32_t r, int32_t type, double rcut, int64_t *out) {
    TRY(ensure_replica(h, r));
    if (!out) return fail(DPD_E_ARG, "null output");
    if (type < 0 || type >= DPD_MAXT) return fail(DPD_E_ARG, "type must be 0..%d", DPD_MAXT - 1);
    if (!(rcut > 0.0 && rcut <= 1.0)) return fail(DPD_E_ARG, "rcut must be in (0, 1]");
    if (!h->ana_parent) {
        TRY(dalloc(h, &h->ana_parent, (size_t)h->N));
        TRY(dalloc(h, &h->ana_size, (size_t)h->N));
        TRY(dalloc(h, &h->ana_acc, 8));
    }
    launch_type_clusters(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, r, type, rcut, h->ana_parent, h->ana_size,
                         h->ana_acc, h->s);
    CK(cudaGetLastError());
    unsigned long long acc[8];
    CK(cudaMemcpyAsync(acc, h->ana_acc, sizeof acc, cudaMemcpyDeviceToHost, h->s));
    TRY(check_status(h));
    out[0] = (int64_t)acc[4];  // beads of the type (the sum of the cluster sizes)
    out[1] = (int64_t)acc[2];  // clusters
    out[2] = (int64_t)acc[5];  // largest cluster
    out[3] = (int64_t)acc[3];  // sum of squared cluster sizes
    out[4] = (int64_t)acc[0];  // neighbours within 1 of the type's beads, all types
    out[5] = (int64_t)acc[1];  // the same, of the type
    return DPD_OK;
}

extern "C" int dpd_aggregates(dpd_handle *h, int32_t r, double r_tail, int32_t min_lipids, int64_t *out,
                              int32_t *agg_of_gid) {
    TRY(ensure_replica(h, r));
    if (!out) return fail(DPD_E_ARG, "null output");
    if (!(r_tail > 0.0 && r_tail <= 1.0)) return fail(DPD_E_ARG, "r_tail must be in (0, 1]");
    if (!h->ana_parent) {
        TRY(dalloc(h, &h->ana_parent, (size_t)h->N));
        TRY(dalloc(h, &h->ana_size, (size_t)h->N));
        TRY(dalloc(h, &h->ana_acc, 8));
    }
    if (!h->ana_min) {
        TRY(dalloc(h, &h->ana_min, (size_t)h->N));
        TRY(dalloc(h, &h->ana_label, (size_t)h->nmax));
    }
    const RepDev &R = h->rh[r];
    launch_aggregates(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, r, R.n, r_tail, min_lipids, h->ana_parent,
                      h->ana_size, h->ana_min, h->ana_acc, agg_of_gid ? h->ana_label : nullptr, h->s);
    CK(cudaGetLastError());
    unsigned long long acc[8];
    CK(cudaMemcpyAsync(acc, h->ana_acc, sizeof acc, cudaMemcpyDeviceToHost, h->s));
    if (agg_of_gid) CK(cudaMemcpyAsync(agg_of_gid, h->ana_label, (size_t)R.n * sizeof(int32_t), cudaMemcpyDefault, h->s));
    TRY(check_status(h));
    out[0] = (int64_t)acc[4];  // molecules
    out[1] = (int64_t)acc[2];  // aggregates
    out[2] = (int64_t)acc[3];  // membranes (aggregates of >= min_lipids molecules)
    out[3] = (int64_t)acc[6];  // molecules in smaller aggregates
    out[4] = (int64_t)acc[5];  // the largest aggregate (molecules)
    return DPD_OK;
}

extern "C" int dpd_get_events(dpd_handle *h, dpd_event *out, int32_t cap, int32_t *n_out) {
    if (!h || !n_out) return fail(DPD_E_ARG, "null argument");
    DevStatus st;
    CK(cudaMemcpyAsync(&st, h->b.status, sizeof st, cudaMemcpyDeviceToHost, h->s));
    CK(cudaStreamSynchronize(h->s));
    const int have = (int)std::min<unsigned>(st.nevents, (unsigned)h->b.evcap);
    if (!out) {  // count only, nothing is cleared
        *n_out = have;
        return DPD_OK;
    }
    const int n = std::min(have, cap < 0 ? 0 : cap);
    if (n > 0) CK(cudaMemcpy(out, h->b.events, (size_t)n * sizeof(dpd_event), cudaMemcpyDefault));
    *n_out = n;
    CK(cudaMemset(&h->b.status->nevents, 0, sizeof(unsigned)));
    if (st.nevents > (unsigned)h->b.evcap)
        return fail(DPD_E_EVENT_OVERFLOW, "%u events were recorded, %d kept", st.nevents, h->b.evcap);
    if (have > n) return fail(DPD_E_EVENT_OVERFLOW, "%d events pending, %d copied: the rest were dropped", have, n);
    return DPD_OK;
}

// host memory the device can write through the same address (pinned, mapped)
static bool device_writable_host(const void *p) {
    cudaPointerAttributes pa;
    const bool ok = cudaPointerGetAttributes(&pa, p) == cudaSuccess && pa.type == cudaMemoryTypeHost &&
                    pa.devicePointer == p;
    cudaGetLastError();
    return ok;
}

extern "C" int dpd_events_async(dpd_handle *h, dpd_event *out, int32_t cap, int32_t *n_out) {
    if (!h || !out || !n_out) return fail(DPD_E_ARG, "null argument");
    if (cap < 1) return fail(DPD_E_ARG, "the event buffer needs room for at least one event");
    static_assert(sizeof(dpd_event) == sizeof(EventDev), "dpd_event and the device log agree");
    if (!device_writable_host(out) || !device_writable_host(n_out))
        return fail(DPD_E_ARG, "the event buffer and its count must be pinned host memory the device can write "
                               "(cudaHostAlloc, cudaHostRegister)");
    launch_events_out(h->b, (EventDev *)out, cap, (int *)n_out, h->s);
    CK(cudaGetLastError());
    return DPD_OK;
}

// the sums of a stats row on the stream, copied into v (OBS_N words) when the
// stream gets there: one kernel, whose last block hands the row over to obs_out
// and clears the running sums (the max bond restarts per stats row), and one copy
static int enqueue_observables(dpd_handle *h, int32_t r, bool virial, unsigned long long *v) {
    // pinned host memory the device can reach: the kernel writes the row there itself
    unsigned long long *direct = nullptr;
    cudaPointerAttributes pa;
    if (cudaPointerGetAttributes(&pa, v) == cudaSuccess && pa.type == cudaMemoryTypeHost &&
        pa.devicePointer == (void *)v)
        direct = v;
    cudaGetLastError();
    launch_observables(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, r, virial, direct, 0, h->s);
    CK(cudaGetLastError());
    if (!direct)
        CK(cudaMemcpyAsync(v, h->b.obs_out + (size_t)r * OBS_N, OBS_N * sizeof(unsigned long long),
                           cudaMemcpyDeviceToHost, h->s));
    return DPD_OK;
}

static void decode_observables(const RepDev &R, const unsigned long long *v, double *out) {
    for (int k = 0; k < 16; k++) out[k] = 0.0;
    out[0] = (double)(long long)v[2] / OBS_FIX / (2.0 * R.n - 2.0);
    out[1] = (double)(long long)v[0] / OBS_FIX;
    out[2] = (double)(long long)v[1] / OBS_FIX;
    out[3] = (double)(long long)v[3] / OBS_FIX / ((double)R.L * (double)R.L);
    uint32_t bits = (uint32_t)v[4];
    float mb;
    memcpy(&mb, &bits, 4);
    out[4] = mb;
    out[5] = (double)v[5];
    for (int t = 0; t < 8; t++) out[8 + t] = (double)v[8 + t];
}

static int observables_impl(dpd_handle *h, int32_t r, bool virial, double *out) {
    TRY(ensure_replica(h, r));
    if (!out) return fail(DPD_E_ARG, "null out");
    TRY(enqueue_observables(h, r, virial, h->host->row));
    CK(cudaStreamSynchronize(h->s));
    decode_observables(h->rh[r], h->host->row, out);
    return DPD_OK;
}

extern "C" int dpd_stats_async(dpd_handle *h, int32_t r, uint64_t *raw) {
    TRY(ensure_replica(h, r));
    if (!raw) return fail(DPD_E_ARG, "null raw buffer");
    return enqueue_observables(h, r, false, (unsigned long long *)raw);
}

extern "C" int dpd_stats_ring(dpd_handle *h, int32_t r, uint64_t *ring, int32_t nslots) {
    TRY(ensure_replica(h, r));
    if (ring) {
        if (nslots < 1) return fail(DPD_E_ARG, "the ring needs at least one slot");
        cudaPointerAttributes pa;
        const bool ok = cudaPointerGetAttributes(&pa, ring) == cudaSuccess && pa.type == cudaMemoryTypeHost &&
                        pa.devicePointer == (void *)ring;
        cudaGetLastError();
        if (!ok) return fail(DPD_E_ARG, "the stats ring must be pinned host memory the device can write "
                                        "(cudaHostAlloc, cudaHostRegister)");
    }
    CK(cudaStreamSynchronize(h->s));
    h->ring = (unsigned long long *)ring;
    h->ring_rep = ring ? r : 0;
    h->ring_slots = ring ? nslots : 0;
    drop_graphs(h);  // the step graphs are captured again with (or without) the row
    return DPD_OK;
}

extern "C" int dpd_stats_decode(const dpd_handle *h, int32_t r, const uint64_t *raw, double *out) {
    if (!h || !raw || !out) return fail(DPD_E_ARG, "null argument");
    if (r < 0 || r >= h->nrep) return fail(DPD_E_ARG, "replica %d out of range", r);
    decode_observables(h->rh[r], (const unsigned long long *)raw, out);
    return DPD_OK;
}

extern "C" int dpd_observables(dpd_handle *h, int32_t r, double *out) { return observables_impl(h, r, true, out); }

extern "C" int dpd_stats(dpd_handle *h, int32_t r, double *out) { return observables_impl(h, r, false, out); }

extern "C" int dpd_pair_hist(dpd_handle *h, int32_t r, int32_t ta, int32_t tb, double rmax, int32_t nbin,
                             double *hist) {
    TRY(ensure_replica(h, r));
    if (!hist || nbin < 1 || nbin > 4096 || !(rmax > 0.0 && rmax <= 3.0))
        return fail(DPD_E_ARG, "need 1 <= nbin <= 4096 and 0 < rmax <= 3");
    CK(cudaMemsetAsync(h->b.hist, 0, nbin * sizeof(unsigned long long), h->s));
    launch_pair_hist(h->b, h->cur, h->d_rep, h->d_bch, h->rh[r].nch, r, ta, tb, rmax, nbin, h->s);
    CK(cudaGetLastError());
    std::vector<unsigned long long> v(nbin);
    CK(cudaMemcpyAsync(v.data(), h->b.hist, nbin * sizeof(unsigned long long), cudaMemcpyDeviceToHost, h->s));
    CK(cudaStreamSynchronize(h->s));
    for (int k = 0; k < nbin; k++) hist[k] = (double)v[k];
    return DPD_OK;
}

extern "C" int dpd_get_stream(const dpd_handle *h, void **stream) {
    if (!h || !stream) return fail(DPD_E_ARG, "null argument");
    *stream = (void *)h->s;
    return DPD_OK;
}

extern "C" int dpd_set_rng(dpd_handle *h, int32_t r, const uint64_t *state) {
    TRY(ensure_replica(h, r));
    if (!state) return fail(DPD_E_ARG, "null state");
    CK(cudaMemcpyAsync(h->b.rng + 4 * r, state, 4 * sizeof(uint64_t), cudaMemcpyDefault, h->s));
    CK(cudaStreamSynchronize(h->s));
    return DPD_OK;
}

extern "C" int dpd_get_rng(dpd_handle *h, int32_t r, uint64_t *state) {
    TRY(ensure_replica(h, r));
    if (!state) return fail(DPD_E_ARG, "null state");
    CK(cudaMemcpyAsync(state, h->b.rng + 4 * r, 4 * sizeof(uint64_t), cudaMemcpyDefault, h->s));
    CK(cudaStreamSynchronize(h->s));
    return DPD_OK;
}

extern "C" int dpd_kernels_per_step(const dpd_handle *h, int32_t *n_plain, int32_t *n_chem) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    // the scan, placement and fix-up of the sort, permute, forces (+ the chemistry kernels)
    const SortForm form = sort_form(h);
    const int sort = form == SortForm::TWO_PASS ? 4 : form == SortForm::BINS ? (sort_bins_one(h->C) ? 1 : 2) : 3;
    if (n_plain) *n_plain = sort + 2 + (h->any_lipid ? chem_kernel_count() : 0);
    if (n_chem) *n_chem = chem_kernel_count();
    return DPD_OK;
}

// ---------------------------------------------------------------- parameters in place

extern "C" int dpd_set_params(dpd_handle *h, int32_t r, const dpd_params *p) {
    TRY(ensure_replica(h, r));
    if (!p) return fail(DPD_E_ARG, "null params");
    RepDev R;
    const RepDev &old = h->rh[r];
    TRY(make_rep(*p, old.b0, old.n, old.c0, R));
    if (R.ncx != old.ncx || R.L != old.L) return fail(DPD_E_ARG, "dpd_set_params cannot change the box size");
    R.ch0 = old.ch0;
    R.nch = old.nch;
    R.so = old.so;
    R.dcap = old.dcap;
    if ((p->chem && p->chem_kind == 1) != (h->params[r].chem && h->params[r].chem_kind == 1) && !h->any_cat)
        return fail(DPD_E_ARG, "dpd_set_params cannot switch the catalyst chemistry on: create the handle with it");
    if (p->lip_arch != 0 && !h->any_mol)
        return fail(DPD_E_ARG, "dpd_set_params cannot switch to branched lipids: create the handle with them");
    CK(cudaStreamSynchronize(h->s));
    h->rh[r] = R;
    h->params[r] = *p;
    CK(cudaMemcpy(h->d_rep + r, &R, sizeof R, cudaMemcpyHostToDevice));
    {
        dpd_template M;
        if (dpd_lipid_template(p, &M) != DPD_OK) std::memset(&M, 0, sizeof M);
        CK(cudaMemcpy((dpd_template *)h->b.mol + r, &M, sizeof M, cudaMemcpyHostToDevice));
    }
    bool any = false;
    h->any_lipid = false;
    h->cat_period = 0;
    for (auto &q : h->params) {
        any = any || q.chem;
        h->any_lipid = h->any_lipid || (q.chem && q.chem_kind == 0);
        if (q.chem && q.chem_kind == 1) {
            const int64_t a = h->cat_period ? h->cat_period : 1, c = q.n_chem;
            h->cat_period = a / std::gcd(a, c) * c;
        }
    }
    h->gsteps = graph_len(h, h->gsteps);
    drop_graphs(h);
    bool stir = false;
    for (auto &q : h->params) stir = stir || q.stir_A != 0.0;
    if (stir && !h->any_stir) {
        // the current sums were not kept: rebuild them with a sort in place
        h->any_stir = true;
        drop_graphs(h);
        enqueue_sort(h, PERM_SORT);
        h->keys_valid = false;
    }
    h->any_stir = stir;
    if (any != h->any_chem) {
        h->any_chem = any;
        drop_graphs(h);
    }
    return DPD_OK;
}

// ---------------------------------------------------------------- reverse mode

// an array's place in the storage of the reverse mode
static size_t adj_place(size_t bytes) { return (bytes + 64 + 255) & ~(size_t)255; }

// the arrays of a reverse pass over nseg stored configurations after nck
// checkpoints, with the loss's x_bar of ng configurations, laid out from base
// on (or, base null, only measured); returns the bytes they take
static size_t adj_layout(const dpd_handle *h, char *base, int nck, int nseg, int ng, int nbin, AdjBufs &A) {
    const size_t N = (size_t)h->N, C = (size_t)h->C;
    size_t at = 0;
    auto want = [&](auto **p, size_t count) {
        *p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(base ? base + at : nullptr);
        at += adj_place(count * sizeof(**p));
    };
    A = AdjBufs();
    A.ck.resize(nck);
    for (auto &c : A.ck) {
        want(&c.pos, N);
        want(&c.vh, N);
        want(&c.vt, N);
        want(&c.f, N);
        want(&c.tg, N);
        want(&c.link, N);
        want(&c.cstart, C + 1);
    }
    A.seg.resize(nseg);
    for (auto &c : A.seg) {
        want(&c.pos, N);
        want(&c.vt, N);
        want(&c.tg, N);
        want(&c.link, N);
        want(&c.cstart, C + 1);
        want(&c.src, N);
    }
    for (int k = 0; k < 2; k++) {
        want(&A.vh[k], N);
        want(&A.f[k], N);
        want(&A.X[k], N);
        want(&A.V[k], N);
        want(&A.F[k], N);
    }
    A.ng = ng;
    want(&A.G, N * ng);
    want(&A.xb, N);
    want(&A.vb, N);
    want(&A.hist, (size_t)h->nrep * nbin);
    want(&A.wgt, (size_t)h->nrep * nbin);
    want(&A.grad, (size_t)h->nrep * DPD_NGRAD);
    want(&A.gsum, (size_t)h->nrep);
    want(&A.stir, (size_t)h->nrep);
    return at;
}

// The storage stays with the handle: one allocation of the most that a call
// needed, laid out anew by each call (an allocation per call would cost a
// device synchronisation, and each call's arrays beside the last one's more
// than either asked for).
static int adj_setup(dpd_handle *h, int nck, int nseg, int ng, int nbin, AdjBufs &A) {
    const size_t bytes = adj_layout(h, nullptr, nck, nseg, ng, nbin, A);
    if (bytes > h->adj_bytes) {
        free_adj(h);
        const cudaError_t e = cudaMalloc(&h->adj_mem, bytes);
        if (e != cudaSuccess) {
            h->adj_mem = nullptr;
            return fail(DPD_E_NOMEM, "cudaMalloc for the adjoint: %s", cudaGetErrorString(e));
        }
        h->adj_bytes = bytes;
    }
    adj_layout(h, h->adj_mem, nck, nseg, ng, nbin, A);
    return DPD_OK;
}

static void ck_save(dpd_handle *h, const FullCk &c) {
    const size_t N = (size_t)h->N, C = (size_t)h->C;
    const int k = h->cur;
    cudaMemcpyAsync(c.pos, h->b.pos[k], N * sizeof(float2), cudaMemcpyDeviceToDevice, h->s);
    cudaMemcpyAsync(c.vh, h->b.vh[k], N * sizeof(float2), cudaMemcpyDeviceToDevice, h->s);
    cudaMemcpyAsync(c.vt, h->b.vt[k], N * sizeof(float2), cudaMemcpyDeviceToDevice, h->s);
    cudaMemcpyAsync(c.f, h->b.f[k], N * sizeof(float2), cudaMemcpyDeviceToDevice, h->s);
    cudaMemcpyAsync(c.tg, h->b.tg[k], N * sizeof(uint32_t), cudaMemcpyDeviceToDevice, h->s);
    cudaMemcpyAsync(c.link, h->b.link[k], N * sizeof(int2), cudaMemcpyDeviceToDevice, h->s);
    cudaMemcpyAsync(c.cstart, h->b.cstart, (C + 1) * sizeof(int32_t), cudaMemcpyDeviceToDevice, h->s);
}

// the configuration at step s of segment sg (0: its checkpoint)
static StateView seg_view(const AdjBufs &A, int sg, int s) {
    if (s == 0) {
        const FullCk &c = A.ck[sg];
        return StateView{c.pos, c.vt, c.tg, c.link, c.cstart};
    }
    const SegState &c = A.seg[s - 1];
    return StateView{c.pos, c.vt, c.tg, c.link, c.cstart};
}

static StateView view_cur(dpd_handle *h) {
    const int k = h->cur;
    return StateView{h->b.pos[k], h->b.vt[k], h->b.tg[k], h->b.link[k], h->b.cstart};
}

static void enqueue_plain_step(dpd_handle *h) {  // one step without chemistry (windows require chem off)
    enqueue_cell_sort(h, h->b, h->cur, true);
    launch_permute(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, PERM_STEP, h->s);
    h->cur ^= 1;
    enqueue_forces(h, h->b, h->cur, true);
}

// The handle's buffers with the configurations at steps s - 1 and s of segment
// sg in their place (buffer parities par0 + s - 1 and par0 + s): a step of a
// segment reads one stored configuration and writes the next, and nothing is
// copied.  Keys, counts and the sort's scratch are the handle's own.
static Bufs seg_bufs(dpd_handle *h, AdjBufs &A, int sg, int s, int par0) {
    Bufs b = h->b;
    const FullCk &c = A.ck[sg];
    const int from = (par0 + s - 1) & 1, to = (par0 + s) & 1;
    b.pos[from] = s == 1 ? c.pos : A.seg[s - 2].pos;
    b.vt[from] = s == 1 ? c.vt : A.seg[s - 2].vt;
    b.tg[from] = s == 1 ? c.tg : A.seg[s - 2].tg;
    b.link[from] = s == 1 ? c.link : A.seg[s - 2].link;
    b.vh[from] = s == 1 ? c.vh : A.vh[from];
    b.f[from] = s == 1 ? c.f : A.f[from];
    const SegState &t = A.seg[s - 1];
    b.pos[to] = t.pos;
    b.vt[to] = t.vt;
    b.tg[to] = t.tg;
    b.link[to] = t.link;
    b.vh[to] = A.vh[to];
    b.f[to] = A.f[to];
    b.cstart = t.cstart;
    b.src = t.src;
    b.stir = A.stir;
    return b;
}

static void enqueue_seg_step(dpd_handle *h, AdjBufs &A, int sg, int s, int par0) {
    const Bufs b = seg_bufs(h, A, sg, s, par0);
    const int from = (par0 + s - 1) & 1;
    enqueue_cell_sort(h, b, from, true);
    launch_permute(b, from, h->d_rep, h->d_bch, h->nbch, PERM_STEP, h->s);
    enqueue_forces(h, b, from ^ 1, true);
}

// A differentiated window, enqueued: its steps with the loss's histogram, then
// (after the loss's weights are on the device) its reverse pass over the steps
// after `stop`, in nseg segments of `len` steps (the first may be shorter).
struct Window {
    int64_t nsteps;
    int len, nseg;     // nseg 0: no reverse pass
    const dpd_rdf_spec *spec;
    int64_t step0;     // the step the window starts from, or
    const FitDev *fd;  // where the device keeps it (a captured iteration), else null
    int64_t first_loss() const { return nsteps - spec->last_steps + 1; }  // window steps whose state enters the loss
    // the step the horizon leaves: nothing before it is differentiated
    int64_t stop() const { return spec->horizon > 0 ? std::max<int64_t>(0, first_loss() - 1 - spec->horizon) : 0; }
    int64_t start(int sg) const { return std::max(stop(), nsteps - (int64_t)(nseg - sg) * len); }
};

// The segments of the reverse pass and the storage for them.  The forward pass
// keeps the configurations of the last segment; the others are stepped again
// from their checkpoints.  So the longest segments that fit are taken, all
// steps in one where that fits, in the larger of
//   what the caller's interval asks for: a checkpoint every ckpt steps of the
//   window and the configurations of ckpt steps;
//   a thirty-second of the device's memory, while four times that is free or
//   held already (a failed allocation: the caller's interval), or what
//   dpd_set_window_memory says.
// The loss's x_bar of the configurations that its kernels take together counts
// too; where it does not fit they take fewer, at least one (that one is scratch,
// as the arrays of one configuration are).
// A step made again costs a forward step: at 16,384 beads, a window of 200
// steps with 70 differentiated, 60 of 260 steps were (the window and its gradient 8.2 ms,
// 6.8 without); 24 boxes of 65,536, 70 of 250 differentiated, 50 of 300
// (114.7 ms, 106.0 without, 3.8 GB of configurations).
static int window_setup(dpd_handle *h, int ckpt, Window &w, AdjBufs &A) {
    const size_t N = (size_t)h->N, cells = adj_place((size_t)(h->C + 1) * sizeof(int32_t));
    const size_t vec = adj_place(N * sizeof(float2)), word = adj_place(N * sizeof(uint32_t));
    const size_t ck_bytes = 5 * vec + word + cells, seg_bytes = 3 * vec + 2 * word + cells;
    auto g_bytes = [&](int64_t ng) { return adj_place((size_t)ng * N * sizeof(float2)); };
    const int64_t steps = w.nsteps - w.stop(), batch = std::min(rdf_batch(h->nbch), w.spec->last_steps);
    const size_t asked = (size_t)((w.nsteps + ckpt - 1) / ckpt) * ck_bytes + (size_t)ckpt * seg_bytes;
    auto takes = [&](int nseg, int64_t len) {
        return (size_t)nseg * ck_bytes + (size_t)len * seg_bytes + g_bytes(std::min(len, batch));
    };
    size_t may = asked, free_now = 0, total = 0;
    if (h->window_mem >= 0) {
        may = std::max(may, (size_t)h->window_mem);
    } else {
        const size_t scratch = adj_layout(h, nullptr, 0, 0, 0, w.spec->nbin, A) - g_bytes(0);
        const size_t held = h->adj_bytes > scratch ? h->adj_bytes - scratch : 0;
        may = std::max(may, held);
        if (takes(1, steps) > may) {
            if (cudaMemGetInfo(&free_now, &total) != cudaSuccess) cudaGetLastError();
            may = std::max(may, std::min(total / 32, (free_now + held) / 4));
        }
    }
    for (;;) {
        for (w.nseg = 1;; w.nseg++) {  // ends: segments of at most ckpt steps fit
            const int64_t len = (steps + w.nseg - 1) / w.nseg;
            w.len = (int)len;
            if (len <= ckpt || (len <= INT_MAX && takes(w.nseg, len) <= may)) break;
        }
        const size_t states = (size_t)w.nseg * ck_bytes + (size_t)w.len * seg_bytes;
        int ng = (int)std::min<int64_t>(w.len, batch);
        while (ng > 1 && states + g_bytes(ng) > may) ng--;
        const int rc = adj_setup(h, w.nseg, w.len, ng, w.spec->nbin, A);
        if (rc != DPD_E_NOMEM || may == asked) return rc;
        cudaGetLastError();  // the failed allocation's
        may = asked;
    }
}

static void window_forward(dpd_handle *h, AdjBufs &A, const Window &w) {
    const float rmax = (float)w.spec->rmax, sig = (float)w.spec->sigma;
    const int cur0 = h->cur, nb = w.spec->nbin;
    cudaMemsetAsync(A.hist, 0, (size_t)h->nrep * nb * sizeof(double), h->s);
    int par0 = 0, last = 0;  // steps of the last segment, whose configurations stay stored for the reverse pass
    int sg = -1;  // the segment of the step
    const int batch = rdf_batch(h->nbch);
    RdfViews views;
    int nv = 0;
    for (int64_t k = 1; k <= w.nsteps; k++) {
        if (sg + 1 < w.nseg && k - 1 == w.start(sg + 1)) ck_save(h, A.ck[++sg]);
        if (w.nseg > 0 && sg == w.nseg - 1) enqueue_seg_step(h, A, sg, ++last, par0 = h->cur);
        else enqueue_plain_step(h);
        if (k < w.first_loss()) continue;
        views.v[nv++] = last ? seg_view(A, sg, last) : view_cur(h);
        if (!last || nv == batch || k == w.nsteps) {  // kept configurations wait for a launch's worth of them
            launch_rdf(views, nv, h->d_rep, h->d_bch, h->nbch, w.spec->ta, w.spec->tb, nb, rmax, sig, A.hist, h->s);
            nv = 0;
        }
    }
    if (!last) return;
    // the end of the window into the handle's buffers, those it started from (a captured iteration is replayed there)
    const SegState &e = A.seg[last - 1];
    const size_t N = (size_t)h->N, C = (size_t)h->C;
    h->cur = cur0;
    cudaMemcpyAsync(h->b.pos[cur0], e.pos, N * sizeof(float2), cudaMemcpyDeviceToDevice, h->s);
    cudaMemcpyAsync(h->b.vh[cur0], A.vh[(par0 + last) & 1], N * sizeof(float2), cudaMemcpyDeviceToDevice, h->s);
    cudaMemcpyAsync(h->b.vt[cur0], e.vt, N * sizeof(float2), cudaMemcpyDeviceToDevice, h->s);
    cudaMemcpyAsync(h->b.f[cur0], A.f[(par0 + last) & 1], N * sizeof(float2), cudaMemcpyDeviceToDevice, h->s);
    cudaMemcpyAsync(h->b.tg[cur0], e.tg, N * sizeof(uint32_t), cudaMemcpyDeviceToDevice, h->s);
    cudaMemcpyAsync(h->b.link[cur0], e.link, N * sizeof(int2), cudaMemcpyDeviceToDevice, h->s);
    cudaMemcpyAsync(h->b.cstart, e.cstart, (C + 1) * sizeof(int32_t), cudaMemcpyDeviceToDevice, h->s);
    if (h->any_stir)
        cudaMemcpyAsync(h->b.stir, A.stir, (size_t)h->nrep * sizeof(long long), cudaMemcpyDeviceToDevice, h->s);
    h->keys_valid = false;  // the reverse pass uses the handle's keys and counts
}

// the device's step number to the window's step k
static void window_set_step(dpd_handle *h, const Window &w, int64_t k) {
    if (w.fd) launch_set_step_rel(h->b.step, w.fd, k, h->s);
    else launch_set_step(h->b.step, (long long)(w.step0 + k), h->s);
}

// The reverse pass: segment by segment, the states of each (but the last,
// stored by the forward pass) recomputed from its checkpoint.  state[0..2] (may be null) receive the device
// arrays of the start state's cotangents in gid order.
static void window_reverse(dpd_handle *h, AdjBufs &A, const Window &w, const float2 **state) {
    const float rmax = (float)w.spec->rmax, sig = (float)w.spec->sigma;
    const size_t N = (size_t)h->N;
    const dpd_template *mol = h->any_mol ? h->b.mol : nullptr;
    const long long *base = w.fd ? &w.fd->base : nullptr;
    int p = 0;  // which of X, V, F hold the adjoint state
    cudaMemsetAsync(A.X[0], 0, N * sizeof(float2), h->s);
    cudaMemsetAsync(A.V[0], 0, N * sizeof(float2), h->s);
    cudaMemsetAsync(A.F[0], 0, N * sizeof(float2), h->s);
    cudaMemsetAsync(A.grad, 0, (size_t)h->nrep * DPD_NGRAD * sizeof(double), h->s);
    const int64_t first_loss = w.first_loss();
    for (int sg = w.nseg - 1; sg >= 0; sg--) {
        const int64_t k0 = w.start(sg);
        const int len = (int)(w.start(sg + 1) - k0);
        if (sg < w.nseg - 1) {
            window_set_step(h, w, k0);
            enqueue_keys(h, seg_bufs(h, A, sg, 1, 0), 0, true);
            for (int s = 1; s <= len; s++) enqueue_seg_step(h, A, sg, s, 0);
        }
        int g0 = 0, ng = 0;  // A.G holds the loss's x_bar of the segment's steps g0, g0 - 1, ... (ng of them)
        for (int s = len; s > 0; s--) {
            const int64_t k = k0 + s;
            const bool in_loss = k >= first_loss;
            if (in_loss && (g0 < s || g0 - s >= ng)) {
                g0 = s;
                ng = (int)std::min<int64_t>(std::min(s, A.ng), k - first_loss + 1);
                RdfViews views;
                for (int u = 0; u < ng; u++) views.v[u] = seg_view(A, sg, s - u);
                launch_rdf_vjp(views, ng, h->d_rep, h->d_bch, h->nbch, w.spec->ta, w.spec->tb, w.spec->nbin, rmax, sig,
                               A.wgt, A.G, N, h->s);
            }
            const AdjUpdate up{A.X[p], A.V[p], A.X[p ^ 1], A.V[p ^ 1], A.F[p ^ 1], A.seg[s - 1].src,
                               in_loss ? A.G + (size_t)(g0 - s) * N : nullptr, w.spec->ta, w.spec->tb};
            launch_force_vjp(seg_view(A, sg, s), w.step0 + k, h->d_rep, h->d_bch, h->nbch, A.F[p], A.xb, A.vb, A.grad,
                             A.gsum, h->nrep, h->any_stir, mol, h->s, base, &up);
            p ^= 1;
        }
    }
    // the forces stored at the first differentiated step (the window start without a horizon) depend on the parameters too
    const StateView v0 = seg_view(A, 0, 0);
    launch_force_vjp(v0, w.step0 + w.stop(), h->d_rep, h->d_bch, h->nbch, A.F[p], A.xb, A.vb, A.grad, A.gsum, h->nrep,
                     h->any_stir, mol, h->s, base);
    if (state) {
        launch_adj_state(v0.tg, h->d_rep, h->d_bch, h->nbch, A.X[p], A.V[p], A.xb, A.vb, A.X[p ^ 1], A.V[p ^ 1],
                         A.F[p ^ 1], h->s);
        state[0] = A.X[p ^ 1];
        state[1] = A.V[p ^ 1];
        state[2] = A.F[p ^ 1];
    }
    window_set_step(h, w, w.nsteps);
}

static int check_window(dpd_handle *h, int64_t nsteps, const dpd_rdf_spec *spec, const double *target) {
    if (nsteps < 1) return fail(DPD_E_ARG, "window of at least one step");
    if (!spec || !target) return fail(DPD_E_ARG, "null loss specification");
    if (spec->nbin < 1 || spec->nbin > 4096 || !(spec->rmax > 0.0) || !(spec->sigma > 0.0) || spec->last_steps < 1 ||
        spec->last_steps > nsteps || spec->horizon < 0)
        return fail(DPD_E_ARG, "bad loss specification");
    for (auto &p : h->params) {
        if (p.chem) return fail(DPD_E_ARG, "chemistry must be off inside a differentiated window");
        if (p.warmup > 0 && h->step < p.warm_end)
            return fail(DPD_E_ARG, "the repulsion warm-up must be over before a differentiated window");
    }
    return DPD_OK;
}

// host side of the loss: mean histogram -> rdf, loss and the weights dL/dh of every bin
static void rdf_loss(dpd_handle *h, const dpd_rdf_spec *spec, const std::vector<double> &hist,
                     const std::vector<long long> &npairs, const double *target, double *loss, double *rdf_out,
                     std::vector<double> *wgt) {
    const int nb = spec->nbin;
    const double dr = spec->rmax / nb;
    for (int r = 0; r < h->nrep; r++) {
        const double L = (double)h->rh[r].L, area = L * L;
        double sum = 0.0;
        for (int b = 0; b < nb; b++) {
            const double rb = (b + 0.5) * dr;
            const double norm = (npairs[r] > 0) ? area / ((double)npairs[r] * 2.0 * M_PI * rb * dr) : 0.0;
            const double g = hist[(size_t)r * nb + b] / spec->last_steps * norm;
            if (rdf_out) rdf_out[(size_t)r * nb + b] = g;
            const double e = g - target[(size_t)r * nb + b];
            sum += e * e;
            if (wgt) (*wgt)[(size_t)r * nb + b] = 2.0 * e / nb * norm / spec->last_steps;
        }
        if (loss) loss[r] = sum / nb;
    }
}

// unordered pairs of the loss types per replica (the types do not change in a window)
static int count_pairs(dpd_handle *h, const dpd_rdf_spec *spec, std::vector<long long> &npairs) {
    npairs.assign(h->nrep, 0);
    // every replica's row into obs_out, then one copy
    for (int r = 0; r < h->nrep; r++)
        launch_observables(h->b, h->cur, h->d_rep, h->d_bch, h->nbch, r, false, nullptr, 0, h->s);
    CK(cudaGetLastError());
    std::vector<unsigned long long> rows((size_t)h->nrep * OBS_N);
    CK(cudaMemcpyAsync(rows.data(), h->b.obs_out, rows.size() * sizeof(rows[0]), cudaMemcpyDeviceToHost, h->s));
    CK(cudaStreamSynchronize(h->s));
    for (int r = 0; r < h->nrep; r++) {
        double o[16];
        decode_observables(h->rh[r], rows.data() + (size_t)r * OBS_N, o);
        const long long na = (long long)o[8 + spec->ta], nb = (long long)o[8 + spec->tb];
        npairs[r] = spec->ta == spec->tb ? na * (na - 1) / 2 : na * nb;
    }
    return DPD_OK;
}

// state_out (optional): the cotangents of the start state, gid order packed by
// replica, x/y interleaved: [0] positions, [1] stored half-step velocities,
// [2] predicted velocities (2 N floats each; host or device memory)
static int window_impl(dpd_handle *h, int64_t nsteps, int32_t ckpt, const dpd_rdf_spec *spec, const double *target,
                       double *loss, double *grad, double *rdf_out, bool backward, float *const *state_out = nullptr) {
    TRY(check_window(h, nsteps, spec, target));
    if (state_out && spec->horizon > 0)
        return fail(DPD_E_ARG, "start-state cotangents need the full reverse pass (horizon 0)");
    if (ckpt < 1 || ckpt > nsteps) ckpt = (int32_t)nsteps;
    const int nb = spec->nbin;
    std::vector<long long> npairs;
    TRY(count_pairs(h, spec, npairs));
    AdjBufs A;
    Window w{nsteps, 0, 0, spec, h->step, nullptr};
    TRY(backward ? window_setup(h, ckpt, w, A) : adj_setup(h, 0, 0, 0, nb, A));
    if (!h->keys_valid) enqueue_next_keys(h);
    window_forward(h, A, w);
    CK(cudaGetLastError());
    h->step = w.step0 + nsteps;
    std::vector<double> hist((size_t)h->nrep * nb), wgt((size_t)h->nrep * nb);
    CK(cudaMemcpyAsync(hist.data(), A.hist, hist.size() * sizeof(double), cudaMemcpyDeviceToHost, h->s));
    CK(cudaStreamSynchronize(h->s));
    TRY(check_status(h));
    rdf_loss(h, spec, hist, npairs, target, loss, rdf_out, &wgt);
    if (!backward) return DPD_OK;
    CK(cudaMemcpyAsync(A.wgt, wgt.data(), wgt.size() * sizeof(double), cudaMemcpyHostToDevice, h->s));
    const float2 *state[3] = {nullptr, nullptr, nullptr};
    window_reverse(h, A, w, state_out ? state : nullptr);
    CK(cudaGetLastError());
    if (state_out)
        for (int k = 0; k < 3; k++)
            if (state_out[k])
                CK(cudaMemcpyAsync(state_out[k], state[k], (size_t)h->N * sizeof(float2), cudaMemcpyDefault, h->s));
    if (grad) {
        CK(cudaMemcpyAsync(grad, A.grad, (size_t)h->nrep * DPD_NGRAD * sizeof(double), cudaMemcpyDefault, h->s));
    }
    CK(cudaStreamSynchronize(h->s));
    return check_status(h);
}

extern "C" int dpd_set_window_memory(dpd_handle *h, int64_t bytes) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    CK(cudaStreamSynchronize(h->s));
    free_adj(h);  // what an earlier limit allowed
    h->window_mem = bytes < 0 ? -1 : bytes;
    return DPD_OK;
}

extern "C" int dpd_window_loss(dpd_handle *h, int64_t nsteps, const dpd_rdf_spec *spec, const double *target,
                               double *loss, double *rdf_out) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    return window_impl(h, nsteps, (int32_t)nsteps, spec, target, loss, nullptr, rdf_out, false);
}

extern "C" int dpd_window_adjoint(dpd_handle *h, int64_t nsteps, int32_t ckpt_every, const dpd_rdf_spec *spec,
                                  const double *target, double *loss, double *grad, double *rdf_out) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    return window_impl(h, nsteps, ckpt_every, spec, target, loss, grad, rdf_out, true);
}

extern "C" int dpd_window_adjoint_state(dpd_handle *h, int64_t nsteps, int32_t ckpt_every, const dpd_rdf_spec *spec,
                                        const double *target, double *loss, double *grad, double *rdf_out,
                                        float *xbar, float *vhbar, float *vtbar) {
    if (!h) return fail(DPD_E_ARG, "null handle");
    float *const out[3] = {xbar, vhbar, vtbar};
    return window_impl(h, nsteps, ckpt_every, spec, target, loss, grad, rdf_out, true, out);
}

// ---------------------------------------------------------------- a fit as one captured graph
//
// One optimizer iteration of a shared-a_ij fit, enqueued without any host
// step: the window (full checkpoints every ckpt steps), the loss and its bin
// weights (k_rdf_loss), the reverse pass (the steps relative to the window's
// first, kept on the device), and the update (k_fit_update).  The iteration
// ends with the window's last state in the buffers of the parity it started
// from, so the captured graph can be replayed for the next iteration.
struct FitArgs {
    Window w;
    FitDev *fd;
    const long long *npairs;
    const double *target;
    double *loss, *grad, *value;  // iters x nrep, iters x nfit, iters x nfit
};

static void enqueue_fit_iteration(dpd_handle *h, AdjBufs &A, const FitArgs &a) {
    const dpd_rdf_spec *spec = a.w.spec;
    launch_fit_begin(h->b.step, a.fd, h->s);
    enqueue_next_keys(h);
    window_forward(h, A, a.w);
    launch_rdf_loss(h->d_rep, h->nrep, A.hist, a.npairs, a.target, spec->nbin, spec->rmax, spec->last_steps, a.loss,
                    A.wgt, a.fd, h->s);
    window_reverse(h, A, a.w, nullptr);
    launch_fit_update(h->d_rep, h->nrep, A.grad, a.fd, a.grad, a.value, h->s);
}

extern "C" int dpd_fit_graph(dpd_handle *h, int64_t nsteps, int32_t ckpt, const dpd_rdf_spec *spec,
                             const double *target, const dpd_fit_spec *fit, int32_t iters, double *loss, double *grad,
                             double *values) {
    TRY(check_window(h, nsteps, spec, target));
    if (!fit || fit->n < 1 || fit->n > DPD_MAXT * DPD_MAXT) return fail(DPD_E_ARG, "fit: 1 to 64 slots");
    if (iters < 1) return fail(DPD_E_ARG, "fit: at least one iteration");
    if (!(fit->lr > 0.0) || !(fit->beta1 >= 0.0 && fit->beta1 < 1.0) || !(fit->beta2 >= 0.0 && fit->beta2 < 1.0) ||
        !(fit->eps > 0.0))
        return fail(DPD_E_ARG, "fit: lr > 0, 0 <= beta < 1, eps > 0");
    FitDev F;
    std::memset(&F, 0, sizeof F);
    F.nfit = fit->n;
    F.lr = fit->lr;
    F.beta1 = fit->beta1;
    F.beta2 = fit->beta2;
    F.eps = fit->eps;
    for (int k = 0; k < fit->n; k++) {
        const int s = fit->slot[k], i = s / DPD_MAXT, j = s % DPD_MAXT;
        if (s < 0 || s >= DPD_MAXT * DPD_MAXT || i > j)
            return fail(DPD_E_ARG, "fit: slot %d is not i * 8 + j with i <= j", s);
        for (int q = 0; q < k; q++)
            if (fit->slot[q] == s) return fail(DPD_E_ARG, "fit: slot %d twice", s);
        F.slot[k] = s;
        F.value[k] = h->params[0].a[s];
        for (int r = 1; r < h->nrep; r++)
            if (h->params[r].a[s] != F.value[k])
                return fail(DPD_E_ARG, "fit: a shared slot (%d) must start equal in every replica", s);
    }
    if (ckpt < 1 || ckpt > nsteps) ckpt = (int32_t)nsteps;
    const int nb = spec->nbin, nrep = h->nrep;
    std::vector<long long> npairs;
    TRY(count_pairs(h, spec, npairs));
    AdjBufs A;
    Window w{nsteps, 0, 0, spec, 0, nullptr};
    TRY(window_setup(h, ckpt, w, A));
    // the fit's own device memory, freed before returning
    char *mem = nullptr;
    const size_t o_np = ((sizeof(FitDev) + 255) / 256) * 256, o_tg = o_np + (((size_t)nrep * 8 + 255) / 256) * 256;
    const size_t o_loss = o_tg + (((size_t)nrep * nb * 8 + 255) / 256) * 256;
    const size_t o_grad = o_loss + (((size_t)iters * nrep * 8 + 255) / 256) * 256;
    const size_t o_val = o_grad + (((size_t)iters * fit->n * 8 + 255) / 256) * 256;
    const size_t total = o_val + (((size_t)iters * fit->n * 8 + 255) / 256) * 256;
    if (cudaMalloc(&mem, total) != cudaSuccess) return fail(DPD_E_NOMEM, "cudaMalloc(%zu) for the fit", total);
    FitArgs a;
    a.w = w;
    a.w.fd = a.fd = (FitDev *)mem;
    a.npairs = (const long long *)(mem + o_np);
    a.target = (const double *)(mem + o_tg);
    a.loss = (double *)(mem + o_loss);
    a.grad = (double *)(mem + o_grad);
    a.value = (double *)(mem + o_val);
    int rc = DPD_OK;
    cudaGraph_t g = nullptr;
    cudaGraphExec_t ge = nullptr;
    const int cur0 = h->cur;
    do {
        if (cudaMemcpy(mem, &F, sizeof F, cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaMemcpy(mem + o_np, npairs.data(), nrep * sizeof(long long), cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaMemcpy(mem + o_tg, target, (size_t)nrep * nb * sizeof(double), cudaMemcpyDefault) != cudaSuccess) {
            rc = fail(DPD_E_CUDA, "fit: copies to the device: %s", cudaGetErrorString(cudaGetLastError()));
            break;
        }
        if (cudaStreamSynchronize(h->s) != cudaSuccess ||
            cudaStreamBeginCapture(h->s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            rc = fail(DPD_E_CUDA, "fit: capture: %s", cudaGetErrorString(cudaGetLastError()));
            break;
        }
        enqueue_fit_iteration(h, A, a);
        const cudaError_t e = cudaStreamEndCapture(h->s, &g);
        h->cur = cur0;
        if (e != cudaSuccess || cudaGraphInstantiate(&ge, g, 0) != cudaSuccess) {
            rc = fail(DPD_E_CUDA, "fit: graph: %s", cudaGetErrorString(e != cudaSuccess ? e : cudaGetLastError()));
            break;
        }
        for (int it = 0; it < iters && rc == DPD_OK; it++)
            if (cudaGraphLaunch(ge, h->s) != cudaSuccess) rc = fail(DPD_E_CUDA, "fit: launch");
        if (rc != DPD_OK) break;
        if (cudaStreamSynchronize(h->s) != cudaSuccess) {
            rc = fail(DPD_E_CUDA, "fit: %s", cudaGetErrorString(cudaGetLastError()));
            break;
        }
        if ((rc = check_status(h)) != DPD_OK) break;
        FitDev out;
        if (cudaMemcpy(&out, mem, sizeof out, cudaMemcpyDeviceToHost) != cudaSuccess ||
            (loss && cudaMemcpy(loss, a.loss, (size_t)iters * nrep * 8, cudaMemcpyDefault) != cudaSuccess) ||
            (grad && cudaMemcpy(grad, a.grad, (size_t)iters * fit->n * 8, cudaMemcpyDefault) != cudaSuccess) ||
            (values && cudaMemcpy(values, a.value, (size_t)iters * fit->n * 8, cudaMemcpyDefault) != cudaSuccess)) {
            rc = fail(DPD_E_CUDA, "fit: copies from the device");
            break;
        }
        if (values)
            for (int k = 0; k < fit->n; k++) values[(size_t)iters * fit->n + k] = out.value[k];
        // the host's view of the handle: the steps taken, the fitted values in every replica
        h->step += (int64_t)iters * nsteps;
        h->keys_valid = false;
        for (int r = 0; r < nrep && rc == DPD_OK; r++) {
            dpd_params p = h->params[r];
            for (int k = 0; k < fit->n; k++) {
                const int s = fit->slot[k], i = s / DPD_MAXT, j = s % DPD_MAXT;
                p.a[i * DPD_MAXT + j] = p.a[j * DPD_MAXT + i] = out.value[k];
            }
            rc = dpd_set_params(h, r, &p);
        }
    } while (false);
    if (ge) cudaGraphExecDestroy(ge);
    if (g) cudaGraphDestroy(g);
    cudaFree(mem);
    return rc;
}

extern "C" int dpd_force_vjp(dpd_handle *h, int32_t r, int64_t step, const float *gx, const float *gy, float *xbar_x,
                             float *xbar_y, float *vbar_x, float *vbar_y, double *grad) {
    TRY(ensure_replica(h, r));
    if (!gx || !gy) return fail(DPD_E_ARG, "null cotangent");
    const RepDev &R = h->rh[r];
    const size_t n = (size_t)R.n, N = (size_t)h->N, a = ((n * 4 + 255) / 256) * 256;
    AdjBufs A;
    TRY(adj_setup(h, 0, 0, 0, 1, A));
    CK(cudaMemsetAsync(A.grad, 0, (size_t)h->nrep * DPD_NGRAD * sizeof(double), h->s));
    if (h->nrep > 1) CK(cudaMemsetAsync(A.F[0], 0, N * sizeof(float2), h->s));  // the other replicas' cotangents
    const float *sx = gx, *sy = gy;
    if (!on_device(h, {{gx, n * 4, 4}, {gy, n * 4, 4}})) {
        sx = (float *)h->stage;
        sy = (float *)(h->stage + a);
        CK(cudaMemcpyAsync(h->stage, gx, n * 4, cudaMemcpyDefault, h->s));
        CK(cudaMemcpyAsync(h->stage + a, gy, n * 4, cudaMemcpyDefault, h->s));
    }
    // pack the cotangent into the replica's slots via the state packer's force field
    Bufs u = h->b;
    u.f[h->cur] = A.F[0];
    launch_set_dynamics(u, h->cur, R.b0, (int)n, nullptr, nullptr, sx, sy, nullptr, nullptr, h->s);
    launch_force_vjp(view_cur(h), step, h->d_rep, h->d_bch, h->nbch, A.F[0], A.xb, A.vb, A.grad, A.gsum, h->nrep,
                     h->any_stir, h->any_mol ? h->b.mol : nullptr, h->s);
    CK(cudaGetLastError());
    float *outs[4] = {xbar_x, xbar_y, vbar_x, vbar_y};
    float *st[4];
    const bool direct =
        on_device(h, {{outs[0], n * 4, 4}, {outs[1], n * 4, 4}, {outs[2], n * 4, 4}, {outs[3], n * 4, 4}});
    for (int k = 0; k < 4; k++) st[k] = direct ? outs[k] : (float *)(h->stage + k * a);
    Bufs w = h->b;
    w.f[h->cur] = A.xb;
    w.vh[h->cur] = A.vb;
    launch_unpack(w, h->cur, R.b0, (int)n, nullptr, nullptr, st[2], st[3], nullptr, nullptr, st[0], st[1], nullptr,
                  nullptr, nullptr, nullptr, h->s);
    CK(cudaGetLastError());
    for (int k = 0; k < 4; k++)
        if (outs[k] && !direct) CK(cudaMemcpyAsync(outs[k], st[k], n * 4, cudaMemcpyDefault, h->s));
    if (grad) CK(cudaMemcpyAsync(grad, A.grad + (size_t)r * DPD_NGRAD, DPD_NGRAD * sizeof(double), cudaMemcpyDefault, h->s));
    CK(cudaStreamSynchronize(h->s));
    return DPD_OK;
}
