// fdtd_solver.cu -- device-resident FDTD instance: runs on chip, or CUDA-graph replay of the fused step.
//
// A solver owns, in HBM: two buffers of each of the six fields (ping-pong), the four coefficient
// arrays, the source waveform and a one-entry work list (InstDesc + tile prefix).  A run of T steps is
// one launch where the grid fits on chip (run_resident).  Otherwise it replays a captured graph of
// launches, of two steps each or of one, followed by one "advance" launch that moves the
// instance's step counter, so the only host work per graph is one cudaGraphLaunch.  This is the
// scheduler's execution of an iterated FDTD cycle: the per-task dispatch of the reference
// (ptask/task.cpp:3822-3900 -> ptask/cutask.cpp:634-705, six launches per step with host-side
// readiness checks) becomes one replayed graph.
#include "ptk_internal.h"

#include <algorithm>
#include <climits>
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

namespace ptk {

__global__ void k_store_desc(InstDesc *dst, InstDesc v) { *dst = v; }

__global__ void k_store_tile0(int *dst, int a, int b)
{
    dst[0] = a;
    dst[1] = b;
}

static int store_desc(InstDesc *d_dst, const InstDesc &v, cudaStream_t s)
{
    k_store_desc<<<1, 1, 0, s>>>(d_dst, v);
    PTK_CUDA_TRY(cudaGetLastError());
    count_launches(1);
    return PTK_OK;
}

// x cells per thread for a row of nx cells: the widest tile that keeps most lanes busy.
int default_vec(int nx)
{
    if (nx >= 96) return 4;
    if (nx >= 40) return 2;
    return 1;
}

// Default tile shape: rows of 8, z depth chosen so the grid holds several waves of CTAs.
static void default_tiles(int nx, int ny, int nz, int *by, int *kc, int *vec)
{
    *by = 8;
    *vec = default_vec(nx);
    const int tx = 32 * *vec;
    const long long cols = (long long)((nx + tx - 1) / tx) * ((ny + 7) / 8);
    const long long want = 4LL * std::max(1, sm_count()) * 2;   // ~4 waves at 2 CTAs per SM
    long long zc = (want + cols - 1) / std::max(1LL, cols);
    int k = (int)((nz + zc - 1) / std::max(1LL, zc));
    if (k < 16) k = 16;
    if (k >= nz) k = 0;
    *kc = k;
}

// Grids of more than this many cells start with the staged kernel's shape, whose runs are resident launches or
// take two steps per pass (24^3: 1.6 us per step against 12.8; 32^3: 1.6 against 5.5; 256^3: 87 against 215).  Smaller
// ones keep the register kernel and a launch per step not for speed (16^3, 70 steps: 894 us, on chip 112; 6^3: 494 and
// 102) but because the launches of their default runs are a published figure (ptk_solver_last_launches: the steps, and
// one per 32).  A caller who wants the speed sets the staged or the tuned shape.
static constexpr long long kStagedCells = 1 << 12;

// Where the default solver of a larger grid keeps the register kernel for what is not fused: on rows so short that
// the staged tiles, 128 cells wide, are mostly empty, while one register tile of 32 cells covers them (us per step,
// register and staged: 8x500x400 161 and 206, 18x330x210 62 and 72, 32x200x190 40 and 41, 33x200x190, two tiles, 66 and 43).
// And for single steps where little else is in them than the staged graph's start, 5 us longer, and its walls'
// launch: up to 48 cells (40x160x200 48 and 52, 48x150x150 41 and 43, 64x150x150 46 and 44), and on thin grids (1200x1200x1
// 52 and 62, 3000x3000x2 342 and 350, 800x800x3 47 and 50; 1000x300x4 29 and 34, 60x3000x6 35 and 39, but 2000x2000x4 253 and 213).
static constexpr int kNarrow = 32, kNarrowSingle = 48, kThin = 3, kThinSmall = 7;
static constexpr long long kSmallCells = 2 << 20;

// Uniform coefficients v = (Ca, Cb, Da, Db), and the one-entry table that goes with them.
__global__ void k_uniform_coefs(float *Ca, float *Cb, float *Da, float *Db, long long n, float4 v, float4 *tab)
{
    const long long q0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q0 == 0) *tab = v;
    for (long long q = q0; q < n; q += (long long)gridDim.x * blockDim.x) {
        Ca[q] = v.x;
        Cb[q] = v.y;
        Da[q] = v.z;
        Db[q] = v.w;
    }
}

struct GraphKey {
    int len, by, kc, vec, stages, pair;
    bool operator<(const GraphKey &o) const
    {
        return std::tie(len, by, kc, vec, stages, pair) < std::tie(o.len, o.by, o.kc, o.vec, o.stages, o.pair);
    }
};

}  // namespace ptk

using namespace ptk;

// Fused steps per replayed graph, and of those that go two per launch: a graph's faces, its advance and the gap to
// the next one cost 11 us, 4 % of 16 launches at 128x96x80 (8.76 us per step; with 64 steps 8.60, with 128 8.55).
static constexpr int kChunk = 32, kPairChunk = 64;

struct ptk_solver {
    ptk_fdtd_params p;
    Layout L;
    std::vector<void *> parts; // the device allocations, one as a rule, that hold the arrays below but wave and d_xch
    size_t held_bytes = 0, wave_bytes = 0;
    float *buf[2][6] = {};
    float *coef[4] = {};
    float *wave = nullptr;
    int nwave = 0;
    long long src = -1;
    int step = 0;              // host mirror of the device step counter
    int par = 0;               // buffer that holds the fields
    int by = 0, kc = 0, vec = 4, stages = 0;
    bool ours = true;          // that shape is the default or the autotuner's: short runs may take another form
    ptk_tile_config alt{};     // runs of up to alt_steps steps in such a form, where no fused one is taken
    int alt_steps = 0;
    int *d_err = nullptr;      // raised by the staged kernel if a bounded wait expires
    void *d_tma = nullptr;     // tensor maps of the staged kernel (encoded for tma_by rows)
    int tma_by = 0;
    unsigned char *mat = nullptr;   // material index of the coefficients (one byte per node)
    float *mat_tab = nullptr;       // its table, kMaxMaterials x (Ca, Cb, Da, Db)
    MaterialInfo minfo{};           // materials in the table; nmat 0 = per-cell arrays only
    bool mat_enabled = true;
    long long *d_face0 = nullptr;   // {0, face nodes}: the staged path advances faces per chunk
    long long faces = 0;
    int *d_work = nullptr;          // staged path: tile counters, one per step of a chunk
    int total_tiles = 0;
    bool resident = false;          // the grid fits on chip: staged shapes run whole runs in one launch
    bool refused = false;           // such a launch could not be placed: not tried again
    ResidentPlan rplan{};
    ulonglong2 *d_xch = nullptr;    // its ghost rows in flight
    unsigned seq = 0;               // and the sequence number of the last step
    bool pair = false;              // staged shapes take long runs two steps at a time (fdtd_step_pair.cu)
    PairPlan pplan{};
    bool pair_maps = false;         // its tensor maps are encoded
    void *d_tma_pair = nullptr;
    bool fused_ready = false;       // prepare_fused has run
    bool plain = false;             // the autotuner compares tile shapes by their own kernels
    InstDesc *d_desc = nullptr;
    int *d_tile0 = nullptr;
    cudaStream_t cap = nullptr;   // capture stream
    std::map<GraphKey, cudaGraphExec_t> graphs;
    long long last_launches = 0, last_graphs = 0;
    std::mutex mu;
};

namespace ptk {

// The staged kernel reads the material index when the coefficients have one and an instantiation
// of the shape exists; otherwise the per-cell arrays, with the shape clamped to a dense one (10- and
// 11-row tiles have only a 3-plane ring with the per-cell arrays; 5 and 6 planes exist only with
// the index).
static bool use_mat(const ptk_solver *s)
{
    return s->stages > 0 && s->mat_enabled && s->minfo.nmat > 0 && yee_bulk_smem_bytes(s->by, s->stages, true) > 0;
}

struct RunShape {
    int by, stages;
    bool mat;
};

// How the two-step kernel would get the coefficients, or -1: four arrays that all vary are not for it.
static int pair_mode(const ptk_solver *s)
{
    if (!s->mat_enabled || s->stages <= 0) return -1;
    if (use_mat(s)) return s->minfo.simple ? PAIR_SIMPLE : PAIR_TABLE;
    return s->minfo.simple ? PAIR_CELLS : -1;
}

static RunShape run_shape(const ptk_solver *s)
{
    if (s->stages <= 0) return {s->by, 0, false};
    if (use_mat(s)) return {s->by, s->stages, true};
    if (yee_bulk_smem_bytes(s->by, s->stages, false) > 0) return {s->by, s->stages, false};
    // same rows with the 3-plane ring the per-cell arrays leave room for (10 and 11 rows), else 4
    if (yee_bulk_smem_bytes(s->by, 3, false) > 0) return {s->by, 3, false};
    return {s->by >= 8 ? 8 : 4, 4, false};
}

// What the resident and the two-step kernel need, made when a staged shape is first set: the plan, the
// exchange buffer (zeroed once) or where the tensor maps go.
static int prepare_fused(ptk_solver *s)
{
    if (s->fused_ready) return PTK_OK;
    s->fused_ready = true;
    cudaStream_t st = default_stream();
    if (plan_resident(s->L.nx, s->L.ny, s->L.nz, sm_count(), &s->rplan)) {
        if (pool_alloc(s->rplan.xch_bytes, st, (void **)&s->d_xch) == PTK_OK) {
            PTK_CUDA_TRY(cudaMemsetAsync(s->d_xch, 0, s->rplan.xch_bytes, st));
            PTK_CUDA_TRY(cudaStreamSynchronize(st));   // runs may come on any stream
            s->resident = true;
        } else {
            clear_error();   // no room for it: the tile shape's own kernel runs
        }
    } else if (plan_pair(s->L.nx, s->L.ny, s->L.nz, &s->pplan)) {
        s->pplan.args.tma = s->d_tma_pair;
        for (int b = 0; b < 2; ++b)
            for (int f = 0; f < 6; ++f) s->pplan.args.buf[b][f] = s->buf[b][f];
        s->pair = true;
    }
    return PTK_OK;
}

// Vacuum coefficients as the material index has them: one entry, every id 0.
static int uniform_vacuum(ptk_solver *s, cudaStream_t st, bool clear_index)
{
    // Scalar coefficients of the reference: (params.Dt/params.eps0), (params.Dt/params.mu0) in FP32.
    const float4 v = make_float4(1.0f, s->p.Dt / s->p.eps0, 1.0f, s->p.Dt / s->p.mu0);
    if (clear_index) PTK_CUDA_TRY(cudaMemsetAsync(s->mat, 0, (size_t)s->L.total, st));
    const int blocks = (int)std::min<long long>((s->L.total + 255) / 256, 16LL * std::max(1, sm_count()));
    k_uniform_coefs<<<blocks, 256, 0, st>>>(s->coef[0], s->coef[1], s->coef[2], s->coef[3], s->L.total, v,
                                            reinterpret_cast<float4 *>(s->mat_tab));
    PTK_CUDA_TRY(cudaGetLastError());
    count_launches(1);
    s->minfo = MaterialInfo{};
    if (s->mat_enabled) s->minfo = MaterialInfo{1, 1, v.w};
    return PTK_OK;
}

// What the default shape's short runs take instead (kNarrow).
static void default_alt(ptk_solver *s)
{
    const int nx = s->L.nx, nz = s->L.nz;
    const bool narrow = nx <= kNarrowSingle && nx <= 32 * default_vec(nx);   // one register tile in x
    const bool thin = nz <= kThin || (nz <= kThinSmall && (long long)nx * s->L.ny * nz < kSmallCells);
    if (!narrow && !thin) return;
    s->alt = ptk_tile_config{};
    default_tiles(nx, s->L.ny, nz, &s->alt.by, &s->alt.kc, &s->alt.vec);
    s->alt_steps = nx <= kNarrow ? INT_MAX : 1;
}

// No run is fused after all: with the library's shape all take the best step kernel known.
static void short_runs_off_chip(ptk_solver *s)
{
    if (!s->ours) return;
    if (s->alt.by > 0) s->alt_steps = INT_MAX;   // the autotuner's
    else default_alt(s);
}

// The staged kernel's shape without timing: 11 rows, a 4-plane ring and the depth that fills whole waves
// of resident CTAs best.
static int staged_default(int nx, int ny, int nz, ptk_tile_config *cfg)
{
    const int by = 11, stages = 4, vec = yee_bulk_tile_vec(by);
    int kc = 0;
    balanced_depths(nx, ny, nz, by, vec, yee_bulk_resident_ctas(by, stages, true), &kc, 1);
    *cfg = {by, kc >= nz ? 0 : kc, vec, stages};
    return PTK_OK;
}

static int rebuild_material(ptk_solver *s, cudaStream_t st)
{
    s->minfo = MaterialInfo{};
    if (!s->mat_enabled) return PTK_OK;
    const float *const c[4] = {s->coef[0], s->coef[1], s->coef[2], s->coef[3]};
    return build_material_index(c, s->L, s->mat, s->mat_tab, &s->minfo, st);
}

static InstDesc host_desc(const ptk_solver *s, int steps_left)
{
    InstDesc d{};
    for (int b = 0; b < 2; ++b)
        for (int f = 0; f < 6; ++f) d.buf[b][f] = s->buf[b][f];
    for (int c = 0; c < 4; ++c) d.coef[c] = s->coef[c];
    d.wave = s->wave;
    d.plane = s->L.plane;
    d.nx = s->L.nx; d.ny = s->L.ny; d.nz = s->L.nz; d.pitch = s->L.pitch;
    d.cx = s->p.Cx; d.cy = s->p.Cy; d.cz = s->p.Cz;
    d.src = s->nwave > 0 ? s->src : -1;
    d.nwave = s->nwave;
    d.step = s->step;
    d.par = s->par;
    d.steps_left = steps_left;
    const RunShape rs = run_shape(s);
    if (rs.mat) {
        d.mat = s->mat;
        d.mat_tab = s->mat_tab;
        d.nmat = s->minfo.nmat;
    }
    plan_tiles(d, rs.by, s->kc, rs.stages > 0 ? yee_bulk_tile_vec(rs.by) : s->vec);
    if (rs.stages > 0) d.face_tiles = 0;   // faces: launch_yee_faces_steps, once per chunk
    return d;
}


static int solver_sync_desc(ptk_solver *s, int steps_left, cudaStream_t st)
{
    InstDesc d = host_desc(s, steps_left);
    s->total_tiles = d.tiles_x * d.tiles_y * d.tiles_z + d.face_tiles;
    const RunShape rs = run_shape(s);
    if (rs.stages > 0) {
        if (s->tma_by != rs.by) {
            // The arrays never move, so the maps change only with the tile rows.
            alignas(64) unsigned char maps[kTmaSetBytes];
            InstDesc e = d;
            e.mat = s->mat;   // the index map is always encoded; the kernel variant decides its use
            int rc = encode_tma_set(e, rs.by, maps);
            if (rc) return rc;
            PTK_CUDA_TRY(cudaStreamSynchronize(st));
            PTK_CUDA_TRY(cudaMemcpy(s->d_tma, maps, kTmaSetBytes, cudaMemcpyHostToDevice));
            s->tma_by = rs.by;
        }
        d.tma = s->d_tma;
    }
    int rc = store_desc(s->d_desc, d, st);
    if (rc) return rc;
    k_store_tile0<<<1, 1, 0, st>>>(s->d_tile0, 0, s->total_tiles);
    PTK_CUDA_TRY(cudaGetLastError());
    count_launches(1);
    return PTK_OK;
}

// The autotuner's choices: a shape, and what its short runs take instead (ptk_solver::alt).
struct Tuned {
    ptk_tile_config best;
    float ms;
    ptk_tile_config alt;
    int alt_steps;
};
static std::mutex g_tune_mu;
static std::map<std::tuple<int, int, int>, Tuned> g_tune_cache;

static bool same_tiles(const ptk_tile_config &a, const ptk_tile_config &b)
{
    return a.by == b.by && a.kc == b.kc && a.vec == b.vec && a.stages == b.stages;
}

static void drop_graphs(ptk_solver *s)
{
    for (auto &kv : s->graphs) cudaGraphExecDestroy(kv.second);
    s->graphs.clear();
}

// Graph of `len` fused steps + one advance for this solver's current tile shape.
static int solver_graph(ptk_solver *s, int len, bool pair, cudaGraphExec_t *out)
{
    const RunShape rs = run_shape(s);
    const int mode = pair_mode(s);
    GraphKey key{len, rs.by, s->kc, s->vec, rs.stages * 2 + (rs.mat ? 1 : 0), pair ? 1 + mode : 0};
    auto it = s->graphs.find(key);
    if (it != s->graphs.end()) {
        *out = it->second;
        return PTK_OK;
    }
    if (!s->cap) PTK_CUDA_TRY(cudaStreamCreateWithFlags(&s->cap, cudaStreamNonBlocking));
    // The staged kernel runs as a persistent grid of resident CTAs taking tiles from a counter, so
    // a CTA streams several tiles through one ring and the last wave is balanced.
    const int grid = rs.stages > 0 ? yee_bulk_resident_ctas(rs.by, rs.stages, rs.mat) : 0;
    PTK_CUDA_TRY(cudaStreamBeginCapture(s->cap, cudaStreamCaptureModeThreadLocal));
    set_capturing(true);
    int rc = PTK_OK;
    if (rs.stages > 0) {
        if (cudaMemsetAsync(s->d_work, 0, sizeof(int) * len, s->cap) != cudaSuccess)
            rc = set_error(PTK_ERR_CUDA, "tile counter reset failed");
        else
            count_launches(1);
    }
    const int pairs = pair ? len / 2 : 0, flips = len - pairs;
    for (int q = 0; q < pairs && rc == PTK_OK; ++q) rc = launch_yee_pair(s->d_desc, s->pplan, mode, q, s->d_err, s->cap);
    for (int q = 2 * pairs; q < len && rc == PTK_OK; ++q)
        rc = rs.stages > 0
                 ? launch_yee_step_bulk(s->d_desc, s->d_tile0, 1, s->total_tiles, q, rs.by, rs.stages, grid, s->d_err,
                                        s->cap, s->d_work, rs.mat, /*lazy=*/true, q - pairs)
                 : launch_yee_step_v(s->d_desc, s->d_tile0, 1, s->total_tiles, q, s->by, s->vec, 0, s->cap);
    if (rc == PTK_OK && rs.stages > 0)
        rc = launch_yee_faces_steps(s->d_desc, s->d_face0, 1, s->faces, 0, len, s->cap, flips);
    if (rc == PTK_OK) rc = launch_advance(s->d_desc, 1, len, s->cap, flips);
    set_capturing(false);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(s->cap, &g);
    if (rc) {
        if (g) cudaGraphDestroy(g);
        return rc;
    }
    if (e != cudaSuccess) return set_error(PTK_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(e));
    cudaGraphExec_t ex = nullptr;
    e = cudaGraphInstantiate(&ex, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return set_error(PTK_ERR_CUDA, "graph instantiate failed: %s", cudaGetErrorString(e));
    s->graphs[key] = ex;
    *out = ex;
    return PTK_OK;
}

// Larger grids with a material index, or with a Cb per cell and nothing else that varies (160^3: 25.4 us per
// step against 83 by the one-step kernel with four arrays), take runs of this many steps or more two steps per
// launch (fdtd_step_pair.cu); shorter ones run the tile shape that was set.
static constexpr int kPairSteps = 16;

static int run_resident(ptk_solver *s, int steps, cudaStream_t st)
{
    // As the replayed graphs of the other runs: not part of a capture.
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    PTK_CUDA_TRY(cudaStreamIsCapturing(st, &capturing));
    if (capturing != cudaStreamCaptureStatusNone) return set_error(PTK_ERR_CUDA, "a run is not permitted when the stream is capturing");
    ResidentArgs a{};
    // In place, but for a single step: no exchange then tells that a neighbour has read the rows it needs.
    const int to = steps == 1 ? s->par ^ 1 : s->par;
    for (int f = 0; f < 6; ++f) {
        a.in[f] = s->buf[s->par][f];
        a.out[f] = s->buf[to][f];
    }
    for (int c = 0; c < 4; ++c) a.coef[c] = s->coef[c];
    const int coef = s->mat_enabled && s->minfo.simple ? COEF_SIMPLE : COEF_DENSE;
    a.db = s->minfo.db;
    a.wave = s->wave;
    a.src = s->nwave > 0 ? s->src : -1;
    a.nwave = s->nwave;
    a.step = s->step;
    a.steps = steps;
    a.nx = s->L.nx; a.ny = s->L.ny; a.nz = s->L.nz; a.pitch = s->L.pitch;
    a.plane = s->L.plane;
    a.cx = s->p.Cx; a.cy = s->p.Cy; a.cz = s->p.Cz;
    a.xch = s->d_xch;
    a.seq = s->seq;
    a.err = s->d_err;
    int rc = launch_yee_resident(s->rplan, coef, a, st);
    if (rc) return rc;
    s->seq += (unsigned)steps;
    s->last_launches = 1;
    s->par = to;
    s->step += steps;
    return PTK_OK;
}

// The solver's tiles for as long as the object lives.
class TilesAs {
    ptk_solver *s;
    ptk_tile_config own;

  public:
    TilesAs(ptk_solver *s, const ptk_tile_config &c) : s(s), own{s->by, s->kc, s->vec, s->stages} { set(c); }
    ~TilesAs() { set(own); }
    void set(const ptk_tile_config &c) { s->by = c.by; s->kc = c.kc; s->vec = c.vec; s->stages = c.stages; }
};

static int run_steps(ptk_solver *s, int steps, bool pair, cudaStream_t st);

int solver_run(ptk_solver *s, int steps, cudaStream_t st)
{
    if (steps < 0) return set_error(PTK_ERR_INVALID, "negative step count");
    s->last_launches = s->last_graphs = 0;
    if (steps == 0) return PTK_OK;
    const bool alt = s->ours && steps <= s->alt_steps;
    if (s->resident && s->stages > 0 && !s->plain && (s->ours ? !alt : steps >= kResidentSteps)) {
        const int rc = run_resident(s, steps, st);
        if (rc != kNotPlaced) return rc;
        s->resident = false;
        s->refused = true;
        short_runs_off_chip(s);
        return solver_run(s, steps, st);
    }
    const bool pair = s->pair && pair_mode(s) >= 0 && steps >= kPairSteps && !s->plain;
    if (alt && !pair) {
        TilesAs other(s, s->alt);
        return run_steps(s, steps, false, st);
    }
    return run_steps(s, steps, pair, st);
}

// A run by replayed graphs.
static int run_steps(ptk_solver *s, int steps, bool pair, cudaStream_t st)
{
    int rc = solver_sync_desc(s, steps, st);
    if (rc) return rc;
    if (pair && !s->pair_maps) {   // the arrays never move: encoded once
        alignas(64) unsigned char maps[kTmaSetBytes];
        InstDesc e = host_desc(s, steps);
        e.mat = s->mat;
        rc = encode_pair_maps(e, s->pplan, maps);
        if (rc) return rc;
        PTK_CUDA_TRY(cudaStreamSynchronize(st));
        PTK_CUDA_TRY(cudaMemcpy(s->d_tma_pair, maps, kTmaSetBytes, cudaMemcpyHostToDevice));
        s->pair_maps = true;
    }
    int left = steps;
    while (left > 0) {
        const int len = std::min(left, pair ? kPairChunk : kChunk), flips = pair ? len - len / 2 : len;
        cudaGraphExec_t ex;
        rc = solver_graph(s, len, pair, &ex);
        if (rc) return rc;
        PTK_CUDA_TRY(cudaGraphLaunch(ex, st));
        count_graph_launch(flips + 1 + (run_shape(s).stages > 0 && s->faces > 0 ? 1 : 0));   // with the staged kernels' walls
        s->last_launches += flips + 1;
        ++s->last_graphs;
        s->par = (s->par + flips) & 1;
        left -= len;
    }
    s->step += steps;
    return PTK_OK;
}

static size_t field_bytes(int f, const ptk_fdtd_params &p)
{
    int ex, ey, ez;
    field_extents(f, p.Nx, p.Ny, p.Nz, &ex, &ey, &ez);
    return (size_t)ex * ey * ez * sizeof(float);
}

// Device staging of host arrays: a field's slot, and how much is staged in one go.
static size_t stage_bytes(int f, const ptk_fdtd_params &p) { return (field_bytes(f, p) + 255) / 256 * 256; }
static constexpr size_t kStageTogether = (size_t)256 << 20;

// Staging of `n` arrays from `first` on, bytes(first, n) in all; of the first alone (n becomes 1) where the device
// has no room for them together.
template <class Bytes>
static int stage_alloc(int first, int &n, const Bytes &bytes, cudaStream_t st, char **stage)
{
    int rc = pool_alloc(bytes(first, n), st, (void **)stage);
    if (rc == PTK_ERR_NOMEM && n > 1) {
        clear_error();
        n = 1;
        rc = pool_alloc(bytes(first, n), st, (void **)stage);
    }
    return rc;
}

}  // namespace ptk

static inline cudaStream_t S(void *s) { return s ? (cudaStream_t)s : default_stream(); }

static int validate_params(const ptk_fdtd_params *p)
{
    PTK_CHECK_ARG(p, "params is NULL");
    PTK_CHECK_ARG(p->Nx >= 1 && p->Ny >= 1 && p->Nz >= 1, "grid %dx%dx%d must be at least 1x1x1",
                  p->Nx, p->Ny, p->Nz);
    PTK_CHECK_ARG((long long)p->Nx * p->Ny * p->Nz <= (1LL << 33), "grid too large");
    return PTK_OK;
}

extern "C" {

int ptk_solver_create(const ptk_fdtd_params *p, ptk_solver **out)
try {
    clear_error();
    int rc = validate_params(p);
    if (rc) return rc;
    PTK_CHECK_ARG(out, "out is NULL");
    rc = ensure_init();
    if (rc) return rc;
    ptk_solver *s = new ptk_solver();
    s->p = *p;
    s->L = make_layout(p->Nx, p->Ny, p->Nz);
    default_tiles(p->Nx, p->Ny, p->Nz, &s->by, &s->kc, &s->vec);
    cudaStream_t st = default_stream();
    const size_t bytes = (size_t)s->L.total * sizeof(float);
    // Everything but the waveform and the exchange buffer: places of one block, 256-byte aligned, those that start at
    // zero first; allocations of their own where the device has room for each but no block that holds them all.
    struct Place {
        void **to;
        size_t bytes;
        bool zero;
    };
    std::vector<Place> places;
    for (int b = 0; b < 2; ++b)
        for (int f = 0; f < 6; ++f) places.push_back({(void **)&s->buf[b][f], bytes, true});
    places.push_back({(void **)&s->mat, (size_t)s->L.total, true});
    places.push_back({(void **)&s->d_err, sizeof(int), true});
    for (int c = 0; c < 4; ++c) places.push_back({(void **)&s->coef[c], bytes, false});
    places.push_back({(void **)&s->mat_tab, sizeof(float) * 4 * kMaxMaterials, false});
    places.push_back({(void **)&s->d_desc, sizeof(InstDesc), false});
    places.push_back({(void **)&s->d_tile0, 2 * sizeof(int), false});
    places.push_back({&s->d_tma, kTmaSetBytes, false});
    places.push_back({&s->d_tma_pair, kTmaSetBytes, false});
    places.push_back({(void **)&s->d_face0, 2 * sizeof(long long), false});
    places.push_back({(void **)&s->d_work, sizeof(int) * kPairChunk, false});
    size_t cleared = 0;
    for (Place &q : places) {
        q.bytes = (q.bytes + 255) / 256 * 256;
        s->held_bytes += q.bytes;
        if (q.zero) cleared += q.bytes;
    }
    s->parts.reserve(places.size());
    void *base = nullptr;
    rc = pool_alloc(s->held_bytes, st, &base);
    if (rc == PTK_OK) {
        s->parts.push_back(base);
        char *at = static_cast<char *>(base);
        for (const Place &q : places) {
            *q.to = at;
            at += q.bytes;
        }
        if (cudaMemsetAsync(base, 0, cleared, st) != cudaSuccess) rc = set_error(PTK_ERR_CUDA, "solver initialisation failed");
    } else if (rc == PTK_ERR_NOMEM) {
        clear_error();
        rc = PTK_OK;
        for (const Place &q : places) {
            rc = pool_alloc(q.bytes, st, q.to);
            if (rc) break;
            s->parts.push_back(*q.to);
            if (q.zero && cudaMemsetAsync(*q.to, 0, q.bytes, st) != cudaSuccess) rc = set_error(PTK_ERR_CUDA, "solver initialisation failed");
            if (rc) break;
        }
    }
    if (rc) {
        ptk_solver_destroy(s);
        return rc;
    }
    s->faces = face_nodes(p->Nx, p->Ny, p->Nz);
    const long long f0[2] = {0, s->faces};   // pageable: staged before the call returns
    if (((uintptr_t)s->d_tma | (uintptr_t)s->d_tma_pair) & 63) rc = set_error(PTK_ERR_CUDA, "tensor-map buffer is not 64-byte aligned");
    if (rc == PTK_OK && cudaMemcpyAsync(s->d_face0, f0, sizeof f0, cudaMemcpyHostToDevice, st) != cudaSuccess)
        rc = set_error(PTK_ERR_CUDA, "solver initialisation failed");
    if (rc == PTK_OK) rc = uniform_vacuum(s, st, /*clear_index=*/false);
    if (rc == PTK_OK && (long long)p->Nx * p->Ny * p->Nz > kStagedCells) {
        ptk_tile_config c;
        rc = staged_default(p->Nx, p->Ny, p->Nz, &c);
        s->by = c.by; s->kc = c.kc; s->vec = c.vec; s->stages = c.stages;
        if (rc == PTK_OK) rc = prepare_fused(s);
        if (rc == PTK_OK && !s->resident) default_alt(s);
    }
    if (rc == PTK_OK && cudaStreamSynchronize(st) != cudaSuccess) rc = set_error(PTK_ERR_CUDA, "solver initialisation failed");
    if (rc) {
        ptk_solver_destroy(s);
        return rc;
    }
    *out = s;
    return PTK_OK;
} PTK_CATCH_ALL

int ptk_solver_destroy(ptk_solver *s)
{
    if (!s) return PTK_OK;
    cudaStream_t st = default_stream();
    {
        std::lock_guard<std::mutex> lk(s->mu);
        drop_graphs(s);
        for (void *q : s->parts) pool_free(q, st);
        pool_free(s->wave, st);
        pool_free(s->d_xch, st);
        if (s->cap) cudaStreamDestroy(s->cap);
    }
    cudaStreamSynchronize(st);
    delete s;
    return PTK_OK;
}

int ptk_solver_set_fields(ptk_solver *s, const float *const f[6], int where, void *stream)
{
    clear_error();
    PTK_CHECK_ARG(s && f, "NULL argument");
    std::lock_guard<std::mutex> lk(s->mu);
    cudaStream_t st = S(stream);
    for (int q = 0; q < 6; ++q) PTK_CHECK_ARG(f[q], "field %d is NULL", q);
    float *const *dst = s->buf[s->par], *const *wall = s->buf[s->par ^ 1];
    // New fields end the state that an expired wait left behind.
    if (where != PTK_HOST) return launch_pack_fields(f, s->L, dst, wall, 0, 6, st, s->d_err);
    // Host fields pass through device staging, all six at once where that is small, else one by one.
    auto bytes = [s](int first, int n) {
        size_t b = 0;
        for (int q = first; q < first + n; ++q) b += stage_bytes(q, s->p);
        return b;
    };
    int per = bytes(0, 6) <= kStageTogether ? 6 : 1;
    for (int q0 = 0; q0 < 6; q0 += per) {
        char *stage = nullptr;
        int rc = stage_alloc(q0, per, bytes, st, &stage);
        if (rc) return rc;
        const float *src[6] = {};
        char *at = stage;
        for (int q = q0; q < q0 + per; ++q) {
            src[q] = (const float *)at;
            PTK_CUDA_TRY(cudaMemcpyAsync(at, f[q], field_bytes(q, s->p), cudaMemcpyHostToDevice, st));
            at += stage_bytes(q, s->p);
        }
        rc = launch_pack_fields(src, s->L, dst, wall, q0, per, st, s->d_err);
        pool_free(stage, st);
        if (rc) return rc;
    }
    return PTK_OK;
}

int ptk_solver_get_fields(ptk_solver *s, float *const f[6], int where, void *stream)
{
    clear_error();
    PTK_CHECK_ARG(s && f, "NULL argument");
    std::lock_guard<std::mutex> lk(s->mu);
    cudaStream_t st = S(stream);
    for (int q = 0; q < 6; ++q) PTK_CHECK_ARG(f[q], "field %d is NULL", q);
    const float *const *src = s->buf[s->par];
    if (where != PTK_HOST) return launch_unpack_fields(src, s->L, f, 0, 6, st, s->d_err);
    auto bytes = [s](int first, int n) {
        size_t b = 0;
        for (int q = first; q < first + n; ++q) b += stage_bytes(q, s->p);
        return b;
    };
    int per = bytes(0, 6) <= kStageTogether ? 6 : 1;
    for (int q0 = 0; q0 < 6; q0 += per) {
        char *stage = nullptr;
        int rc = stage_alloc(q0, per, bytes, st, &stage);
        if (rc) return rc;
        float *dst[6] = {};
        char *at = stage;
        for (int q = q0; q < q0 + per; ++q) {
            dst[q] = (float *)at;
            at += stage_bytes(q, s->p);
        }
        rc = launch_unpack_fields(src, s->L, dst, q0, per, st);
        for (int q = q0; q < q0 + per && !rc; ++q)
            if (cudaMemcpyAsync(f[q], dst[q], field_bytes(q, s->p), cudaMemcpyDeviceToHost, st) != cudaSuccess)
                rc = set_error(PTK_ERR_CUDA, "download failed: %s", cudaGetErrorString(cudaGetLastError()));
        pool_free(stage, st);
        if (rc) return rc;
    }
    if (where == PTK_HOST) {
        int err = 0;
        PTK_CUDA_TRY(cudaMemcpyAsync(&err, s->d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
        PTK_CUDA_TRY(cudaStreamSynchronize(st));
        if (err)
            return set_error(PTK_ERR_TIMEOUT, "a bounded wait of the staged step kernel expired; the fields are invalid");
    }
    return PTK_OK;
}

int ptk_solver_set_coefficients(ptk_solver *s, const float *Ca, const float *Cb, const float *Da,
                                const float *Db, int where, void *stream)
{
    clear_error();
    PTK_CHECK_ARG(s && Ca && Cb && Da && Db, "NULL argument");
    std::lock_guard<std::mutex> lk(s->mu);
    cudaStream_t st = S(stream);
    const float *src[4] = {Ca, Cb, Da, Db};
    const size_t bytes = (size_t)s->p.Nx * s->p.Ny * s->p.Nz * sizeof(float), slot = (bytes + 255) / 256 * 256;
    int per = where != PTK_HOST || 4 * slot <= kStageTogether ? 4 : 1;
    for (int c0 = 0; c0 < 4; c0 += per) {
        const float *from[4] = {};
        char *stage = nullptr;
        int rc = where == PTK_HOST ? stage_alloc(c0, per, [slot](int, int n) { return n * slot; }, st, &stage) : PTK_OK;
        if (rc) return rc;
        for (int c = c0; c < c0 + per; ++c) {
            from[c] = where == PTK_HOST ? (const float *)(stage + (c - c0) * slot) : src[c];
            if (where == PTK_HOST)
                PTK_CUDA_TRY(cudaMemcpyAsync(stage + (c - c0) * slot, src[c], bytes, cudaMemcpyHostToDevice, st));
        }
        rc = launch_pack_coefs(from, s->L, s->coef, c0, per, st);
        if (stage) pool_free(stage, st);
        if (rc) return rc;
    }
    return rebuild_material(s, st);
}

int ptk_solver_set_vacuum(ptk_solver *s, void *stream)
{
    PTK_CHECK_ARG(s, "NULL solver");
    cudaStream_t st = S(stream);
    const int rc = uniform_vacuum(s, st, /*clear_index=*/true);
    if (rc) return rc;
    PTK_CUDA_TRY(cudaStreamSynchronize(st));
    return PTK_OK;
}

int ptk_solver_set_source(ptk_solver *s, int i, int j, int k, const float *wave, int nwave, int where,
                          void *stream)
{
    clear_error();
    PTK_CHECK_ARG(s, "NULL solver");
    std::lock_guard<std::mutex> lk(s->mu);
    cudaStream_t st = S(stream);
    if (nwave <= 0 || !wave) {
        s->nwave = 0;
        s->src = -1;
        return PTK_OK;
    }
    PTK_CHECK_ARG(i >= 1 && i < s->p.Nx && j >= 1 && j < s->p.Ny && k >= 0 && k < s->p.Nz,
                  "source node (%d,%d,%d) must be an interior Ez node of a %dx%dx%d grid", i, j, k,
                  s->p.Nx, s->p.Ny, s->p.Nz);
    if (s->wave) pool_free(s->wave, st);
    s->wave = nullptr;
    s->wave_bytes = 0;
    int rc = pool_alloc((size_t)nwave * sizeof(float), st, (void **)&s->wave);
    if (rc) return rc;
    s->wave_bytes = (size_t)nwave * sizeof(float);
    PTK_CUDA_TRY(cudaMemcpyAsync(s->wave, wave, (size_t)nwave * sizeof(float),
                                 where == PTK_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, st));
    s->nwave = nwave;
    s->src = (long long)i + (long long)s->L.pitch * j + s->L.plane * k;
    return PTK_OK;
}

int ptk_solver_reset_clock(ptk_solver *s, void *stream)
{
    PTK_CHECK_ARG(s, "NULL solver");
    (void)stream;
    std::lock_guard<std::mutex> lk(s->mu);
    s->step = 0;
    return PTK_OK;
}

int ptk_solver_set_tiles(ptk_solver *s, const ptk_tile_config *cfg)
{
    PTK_CHECK_ARG(s && cfg, "NULL argument");
    std::lock_guard<std::mutex> lk(s->mu);
    int by = cfg->by, kc = cfg->kc, vec = cfg->vec;
    if (by == 0 && kc == 0) {
        int dv = 4;
        default_tiles(s->p.Nx, s->p.Ny, s->p.Nz, &by, &kc, &dv);
        if (vec == 0) vec = dv;
    }
    const int stages = cfg->stages;
    if (stages > 0) vec = yee_bulk_tile_vec(by);
    if (vec == 0) vec = default_vec(s->p.Nx);
    PTK_CHECK_ARG(by == 4 || by == 8 || by == 16 || (stages > 0 && (by == 7 || by == 10 || by == 11 || by == 23)),
                  "tile rows must be 4, 8 or 16, or 7, 10, 11 or 23 with a staged ring (got %d)", by);
    PTK_CHECK_ARG(vec == 1 || vec == 2 || vec == 4, "cells per thread must be 1, 2 or 4 (got %d)", vec);
    PTK_CHECK_ARG(stages == 0 || yee_bulk_smem_bytes(by, stages, false) > 0 || yee_bulk_smem_bytes(by, stages, true) > 0,
                  "no staged kernel for %d rows with %d stages", by, stages);
    PTK_CHECK_ARG(kc >= 0, "tile depth must be >= 0");
    if (kc >= s->p.Nz) kc = 0;
    s->by = by;
    s->kc = kc;
    s->vec = vec;
    s->stages = stages;
    s->ours = false;
    s->alt = ptk_tile_config{};
    s->alt_steps = 0;
    {   // the autotuner's shape for this grid leaves the form of short runs to the solver, any other is taken at its word
        std::lock_guard<std::mutex> tk(g_tune_mu);
        auto it = g_tune_cache.find({s->p.Nx, s->p.Ny, s->p.Nz});
        if (it != g_tune_cache.end() && same_tiles(it->second.best, {by, kc, vec, stages})) {
            s->ours = true;
            s->alt = it->second.alt;
            s->alt_steps = it->second.alt_steps;
            if (s->refused) short_runs_off_chip(s);
        }
    }
    return stages > 0 ? prepare_fused(s) : PTK_OK;
}

int ptk_solver_use_material_index(ptk_solver *s, int enable, void *stream)
{
    clear_error();
    PTK_CHECK_ARG(s, "NULL solver");
    std::lock_guard<std::mutex> lk(s->mu);
    s->mat_enabled = enable != 0;
    return rebuild_material(s, S(stream));
}

int ptk_solver_material_count(const ptk_solver *s, int *nmat)
{
    PTK_CHECK_ARG(s && nmat, "NULL argument");
    *nmat = s->mat_enabled ? s->minfo.nmat : 0;
    return PTK_OK;
}

int ptk_solver_kernel(const ptk_solver *s, int *stages, int *material_index)
{
    PTK_CHECK_ARG(s && stages && material_index, "NULL argument");
    RunShape rs = run_shape(s);
    if (s->ours && s->alt_steps == INT_MAX) rs = {s->alt.by, s->alt.stages, false};   // a register shape
    *stages = rs.stages;
    *material_index = rs.mat ? 1 : 0;
    return PTK_OK;
}

int ptk_solver_get_tiles(const ptk_solver *s, ptk_tile_config *cfg)
{
    PTK_CHECK_ARG(s && cfg, "NULL argument");
    cfg->by = s->by;
    cfg->kc = s->kc;
    cfg->vec = s->vec;
    cfg->stages = s->stages;
    return PTK_OK;
}

int ptk_solver_run(ptk_solver *s, int steps, void *stream)
try {
    clear_error();
    PTK_CHECK_ARG(s, "NULL solver");
    std::lock_guard<std::mutex> lk(s->mu);
    return solver_run(s, steps, S(stream));
} PTK_CATCH_ALL

int ptk_selftest_solver_expiry(ptk_solver *s, void *stream)
{
    clear_error();
    PTK_CHECK_ARG(s, "NULL solver");
    std::lock_guard<std::mutex> lk(s->mu);
    PTK_CUDA_TRY(cudaMemsetAsync(s->d_err, 1, 1, S(stream)));
    return PTK_OK;
}

int ptk_solver_bytes(const ptk_solver *s, size_t *bytes)
{
    PTK_CHECK_ARG(s && bytes, "NULL argument");
    *bytes = s->held_bytes + s->wave_bytes + (s->d_xch ? s->rplan.xch_bytes : 0);
    return PTK_OK;
}

int ptk_solver_last_launches(const ptk_solver *s, long long *launches)
{
    PTK_CHECK_ARG(s && launches, "NULL argument");
    *launches = s->last_launches;
    return PTK_OK;
}

int ptk_solver_last_graphs(const ptk_solver *s, long long *graphs)
{
    PTK_CHECK_ARG(s && graphs, "NULL argument");
    *graphs = s->last_graphs;
    return PTK_OK;
}

int ptk_fdtd_solve(const ptk_fdtd_params *p, float *const fields[6], const float *Ca, const float *Cb,
                   const float *Da, const float *Db, int si, int sj, int sk, const float *wave,
                   int nwave, int steps, float *ms)
try {
    clear_error();
    ptk_solver *s = nullptr;
    int rc = ptk_solver_create(p, &s);
    if (rc) return rc;
    cudaStream_t st = default_stream();
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, st);
    rc = ptk_solver_set_fields(s, fields, PTK_HOST, st);
    if (!rc && Ca) rc = ptk_solver_set_coefficients(s, Ca, Cb, Da, Db, PTK_HOST, st);
    if (!rc && wave && nwave > 0) rc = ptk_solver_set_source(s, si, sj, sk, wave, nwave, PTK_HOST, st);
    if (!rc) rc = ptk_solver_run(s, steps, st);
    if (!rc) rc = ptk_solver_get_fields(s, fields, PTK_HOST, st);
    cudaEventRecord(e1, st);
    cudaEventSynchronize(e1);
    if (ms) cudaEventElapsedTime(ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    ptk_solver_destroy(s);
    return rc;
} PTK_CATCH_ALL

int ptk_launch_field_update(int field, const float *in0, const float *in1, const float *in2,
                            const ptk_fdtd_params *p, float *out, void *stream)
{
    clear_error();
    int rc = validate_params(p);
    if (rc) return rc;
    PTK_CHECK_ARG(field >= 0 && field < 6, "field id %d out of range", field);
    PTK_CHECK_ARG(in0 && in1 && in2 && out, "NULL buffer");
    rc = ensure_init();
    if (rc) return rc;
    return launch_field_ref(field, in0, in1, in2, *p, out, S(stream));
}

int ptk_launch_h_half_step(const float *const in[6], float *const out_h[3], const ptk_fdtd_params *p,
                           void *stream)
{
    clear_error();
    int rc = validate_params(p);
    if (rc) return rc;
    PTK_CHECK_ARG(in && out_h, "NULL buffer");
    rc = ensure_init();
    if (rc) return rc;
    return launch_h_half(in, out_h, *p, S(stream));
}

int ptk_launch_e_half_step(const float *const e_in[3], const float *const h_new[3],
                           float *const out_e[3], const ptk_fdtd_params *p, void *stream)
{
    clear_error();
    int rc = validate_params(p);
    if (rc) return rc;
    PTK_CHECK_ARG(e_in && h_new && out_e, "NULL buffer");
    rc = ensure_init();
    if (rc) return rc;
    return launch_e_half(e_in, h_new, out_e, *p, S(stream));
}

// --------------------------------------------------------------------------------------------
// Autotuner: time candidate (rows, depth) shapes on a scratch solver of the requested size.
// --------------------------------------------------------------------------------------------
int ptk_autotune_tiles(int Nx, int Ny, int Nz, ptk_tile_config *best, float *best_ms)
try {
    clear_error();
    PTK_CHECK_ARG(best, "NULL argument");
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tune_cache.find({Nx, Ny, Nz});
        if (it != g_tune_cache.end()) {
            *best = it->second.best;
            if (best_ms) *best_ms = it->second.ms;
            return PTK_OK;
        }
    }
    ptk_fdtd_params p{};
    int rc = ptk_reference_params(Nx, Ny, Nz, &p);
    if (rc) return rc;
    ptk_solver *s = nullptr;
    rc = ptk_solver_create(&p, &s);
    if (rc) return rc;
    cudaStream_t st = default_stream();
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int rows[3] = {4, 8, 16};
    const int depths[6] = {8, 16, 32, 64, 128, 0};
    const long long cells = (long long)Nx * Ny * Nz;
    const int steps = (int)std::max(4LL, std::min(64LL, 400000000LL / std::max(1LL, cells)));
    float best_t = 1e30f;
    ptk_tile_config bc{8, 0, default_vec(Nx), 0}, single = bc;   // the shape, and what its short runs take
    int alt_steps = 0;
    std::vector<ptk_tile_config> cands;
    // Fixed depths plus the two that fill whole waves of resident CTAs best for each kernel.
    auto add = [&](int by, int vec, int stages, int resident) {
        std::vector<int> ks;
        for (int kc : depths)
            if (!(stages > 0 && kc == 8)) ks.push_back(kc);
        int bal[4];
        int nb = balanced_depths(Nx, Ny, Nz, by, vec, resident, bal, 2);
        if (stages > 0) nb += leftover_depths(Nx, Ny, Nz, by, vec, resident, bal + nb, 2);
        for (int q = 0; q < nb; ++q)
            if (std::find(ks.begin(), ks.end(), bal[q]) == ks.end()) ks.push_back(bal[q]);
        for (int kc : ks)
            if (kc == 0 || kc < Nz) cands.push_back({by, kc, vec, stages});
    };
    for (int vec : {1, 2, 4})
        for (int by : rows) {
            if (32 * vec > 2 * std::max(Nx, 32)) continue;   // tiles far wider than the grid
            add(by, vec, 0, yee_resident_ctas(by, vec));
        }
    rc = prepare_fused(s);
    // Staged shapes: timed on vacuum coefficients, i.e. with the material index where the shape has it.
    const int staged[17][2] = {{4, 2}, {4, 3}, {4, 4}, {4, 5}, {4, 6}, {8, 2}, {8, 3}, {8, 4}, {8, 5}, {8, 6},
                               {10, 4}, {10, 5}, {11, 4}, {23, 3}, {23, 4}, {7, 3}, {7, 4}};
    for (const auto &bs : staged) {
        // grids that fit on chip: a staged shape's runs are resident launches, whatever its tiles
        if (s->resident && !(bs[0] == 11 && bs[1] == 4)) continue;
        const bool m = yee_bulk_smem_bytes(bs[0], bs[1], true) > 0;
        add(bs[0], yee_bulk_tile_vec(bs[0]), bs[1], yee_bulk_resident_ctas(bs[0], bs[1], m));
    }
    // ms per step of one shape over n steps after a 2-step warm-up (< 0: the shape does not run)
    auto time_shape = [&](const ptk_tile_config &c, int n) -> float {
        if (ptk_solver_set_tiles(s, &c)) return -1.f;
        if (ptk_solver_run(s, 2, st)) return -2.f;
        cudaEventRecord(e0, st);
        if (ptk_solver_run(s, n, st)) return -2.f;
        cudaEventRecord(e1, st);
        cudaEventSynchronize(e1);
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        return ms / n;
    };
    // ms per call of runs of a single step, by the shape's own kernel or as a fused run
    auto time_single = [&](const ptk_tile_config &c, bool plain) -> float {
        if (ptk_solver_set_tiles(s, &c)) return -1.f;
        s->plain = plain;
        s->ours = !plain;
        s->alt_steps = 0;
        const int n = 64;
        float ms = 0;
        for (int pass = 0; pass < 2; ++pass) {   // the first warms up
            cudaEventRecord(e0, st);
            for (int q = 0; q < n; ++q)
                if (ptk_solver_run(s, 1, st)) return -1.f;
            cudaEventRecord(e1, st);
            cudaEventSynchronize(e1);
            cudaEventElapsedTime(&ms, e0, e1);
        }
        return ms / n;
    };
    s->plain = true;   // shapes are compared by their own kernels
    // First pass: every candidate, briefly.  Second pass: the closest few again over longer runs,
    // twice in alternating order, since shapes within a few per cent of each other trade places
    // in short timings.
    std::vector<std::pair<float, ptk_tile_config>> timed;
    for (const ptk_tile_config &c : cands) {
        const float ms = time_shape(c, steps);
        if (ms == -2.f) { rc = PTK_ERR_CUDA; break; }
        if (ms > 0) timed.push_back({ms, c});
    }
    if (!rc && !timed.empty()) {
        std::stable_sort(timed.begin(), timed.end(),
                         [](const std::pair<float, ptk_tile_config> &a, const std::pair<float, ptk_tile_config> &b) {
                             return a.first < b.first;
                         });
        std::vector<std::pair<float, ptk_tile_config>> top;
        for (const auto &e : timed)
            if (top.size() < 4 && e.first <= timed[0].first * 1.05f) top.push_back({0.f, e.second});
        for (int pass = 0; pass < 2 && !rc && top.size() > 1; ++pass)
            for (size_t q = 0; q < top.size() && !rc; ++q) {
                auto &e = top[pass ? top.size() - 1 - q : q];
                const float ms = time_shape(e.second, std::max(8 * steps, 128));
                if (ms < 0) rc = PTK_ERR_CUDA; else e.first += ms;
            }
        if (top.size() == 1) top[0].first = 2 * timed[0].first;
        for (const auto &e : top)
            if (e.first / 2 < best_t) {
                best_t = e.first / 2;
                bc = e.second;
            }
        // Staged shapes take long runs through the resident or the two-step kernel: the best of them is
        // compared by such a run.  The best shape by its own kernel stays for the runs that are not fused.
        s->plain = false;
        single = bc;
        if ((s->resident || s->pair) && !rc)
            for (const auto &e : timed)
                if (e.second.stages > 0) {
                    const float ms = time_shape(bc.stages > 0 ? bc : e.second, std::max(8 * steps, 128));
                    if (ms < 0) {
                        rc = PTK_ERR_CUDA;
                    } else if (ms < best_t || bc.stages > 0) {
                        best_t = ms;
                        if (bc.stages == 0) bc = e.second;
                    }
                    break;
                }
        if (!rc && s->resident && bc.stages > 0) {
            // On chip every run is fused but, where that is faster, the single step (96^3: 25 us, fused 30; 64^3: 18,
            // fused 15; two steps 38 and 35).
            const float own = time_single(single, true), fused = time_single(bc, false);
            if (own < 0 || fused < 0) rc = PTK_ERR_CUDA;
            else if (own < fused) alt_steps = 1;
        } else if (!rc && !same_tiles(single, bc)) {
            alt_steps = INT_MAX;   // narrow grids: the staged tiles are mostly empty
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    ptk_solver_destroy(s);
    if (rc) return rc;
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_tune_cache[{Nx, Ny, Nz}] = {bc, best_t, single, alt_steps};
    }
    *best = bc;
    if (best_ms) *best_ms = best_t;
    return PTK_OK;
} PTK_CATCH_ALL

int ptk_default_tiles(int Nx, int Ny, int Nz, ptk_tile_config *cfg)
try {
    clear_error();
    PTK_CHECK_ARG(cfg, "NULL argument");
    PTK_CHECK_ARG(Nx >= 1 && Ny >= 1 && Nz >= 1, "grid %dx%dx%d must be at least 1x1x1", Nx, Ny, Nz);
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tune_cache.find({Nx, Ny, Nz});
        if (it != g_tune_cache.end()) {
            *cfg = it->second.best;
            return PTK_OK;
        }
    }
    int rc = ensure_init();
    if (rc) return rc;
    return staged_default(Nx, Ny, Nz, cfg);
} PTK_CATCH_ALL

}  // extern "C"
