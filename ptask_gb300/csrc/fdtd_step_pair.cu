// fdtd_step_pair.cu -- two time steps of the Yee update in one pass over memory.
//
// The one-step kernels move 49 bytes per cell update and run within 5-12 % of the copy bandwidth on
// large grids: more speed needs fewer bytes per update.  Here a CTA streams the z planes of a tile
// once and advances them by two steps: 24.5 bytes per update plus the tile's halo.
//
// A tile is a frame of RF rows of lw units (four x cells), one thread per unit, whole rows next to
// one another in thread order.  Two steps reach two nodes down and one up in every direction, so a
// frame yields its rows 2 .. RF-2 and its columns 2 .. 4lw-3 (all of them at the grid's walls); the
// rest is recomputed by neighbouring tiles.  Per plane k:
//
//   H1(k)      from E0(k), E0(k+1) in the TMA ring             arrive at barrier 1
//   E2(k-2)    from H2(k-2) (after barrier 2 of plane k-1); H2, E2 stored
//   E1(k)      from H1(k), H1(k-1)                             after barrier 1
//   H2(k-1)    from E1(k-1), E1(k)                             arrive at barrier 2
//
// A thread keeps its own H1, E1, H2 of the planes involved in registers; its y neighbours' values go
// through shared memory rows (one slot per thread, so every access is conflict free), its x
// neighbours' through shuffles and, between warps, one pair of floats per warp.  The barriers are
// mbarriers with a quarter of a plane's work between a warp's arrival and its wait, so warps rarely
// stand still; the rows are double buffered to allow that.
//
// What bounds it: the time a warp takes for a plane, some 3300 cycles for 570 instructions, a fifth of them in
// the three waits; 48 % of the issue slots and 4.7 of 6.8 TB/s are used at 256^3.  Warps that wait for their
// neighbours only (counters polled in shared memory, 107 us per step against 93 at the time), a fourth ring
// stage with fewer warps (100) and two CTAs of half the frame per SM (95) were all slower.  A launch starts while
// the one before it ends (programmatic dependent launch) and waits only before its first copy: 1.1 us a step.
//
// A batch of instances (MANY) is a CTA per tile, scheduled by the hardware, deepest first: the start of a CTA
// (3 us) is paid per tile, but a list of uneven tiles balances itself.  94 % of the persistent
// form's rate on one 256^3, 160 G updates/s on mixes of 32..192 (the one-step kernel: 82).
//
// The ring, its bounded waits and the continuous issue across a CTA's tiles are those of the
// one-step kernel (fdtd_step_bulk.cu).  Arithmetic is the same, operation for operation; with
// Ca = Da = 1 (PAIR_SIMPLE) the products with them are left out, which changes no bit.  PAIR_CELLS takes Cb
// from its array, 26 bytes per update: the ring has no room for a seventh field, but a thread needs only its
// own unit, loaded into registers a plane ahead.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "fdtd_chain.cuh"
#include "fdtd_device.cuh"
#include "fdtd_tma.cuh"

#include <type_traits>

namespace ptk {

namespace {

using namespace tma;

// Threads of a CTA at most, with 168 registers each: the code that the compiler makes for 11 warps takes 3-6 %
// less time per plane than for 12 (256^3: 87 us per step against 90-93), and 8 warps with more registers lose
// more to the smaller frame's halo (103) than they gain.
constexpr int kPairThreads = 352;
constexpr int kPairWarps = kPairThreads / 32;
constexpr int kPairStages = 3;
constexpr size_t kPairSmem = 232448;
// rows exchanged through shared memory, twice: Hx1, Hz1, Ex1, Ez1, Hx2, Hz2
constexpr int kRowArrays = 6;
enum { R_HX1 = 0, R_HZ1 = 1, R_EX1 = 2, R_EZ1 = 3, R_HX2 = 4, R_HZ2 = 5 };
// pairs exchanged between warps, twice: (Hy1, Hz1).w of lane 31, (Ey1, Ez1).x of lane 0, (Hy2, Hz2).w of lane 31
constexpr int kEdgeArrays = 3;
enum { X_H1 = 0, X_E1 = 1, X_H2 = 2 };

// Shared memory, at compile-time places so that an access is one offset register and an immediate:
// ring stages of six fields (frames of up to kPairThreads units and a row of up to kMaxLw more) and
// the material ids, then the exchanged rows, pairs, coefficient table and barriers.
constexpr int kMaxLw = 60;            // a TMA box is at most 256 elements wide, the ids 15 more than the row
constexpr int kField = (16 * (kPairThreads + kMaxLw + 1) + 127) / 128 * 128;
constexpr int kIds = 3072;
constexpr int kFull = 6 * kField + kIds, kStage = kFull + 128;   // its barrier behind them
constexpr int kRowsAt = kPairStages * kStage, kRowBuf = kRowArrays * kField;
constexpr int kEdge = 8 * (kPairWarps + 2), kEdgeBuf = kEdgeArrays * kEdge, kEdgesAt = kRowsAt + 2 * kRowBuf;
constexpr int kTabAt = (kEdgesAt + 2 * kEdgeBuf + 15) / 16 * 16, kBar1 = kTabAt + 16 * kMaxMaterials, kBar2 = kBar1 + 8;
constexpr int kBaseAt = kBar2 + 8, kArgsAt = kBaseAt + 16;
constexpr int kPairBytes = kArgsAt + (int)sizeof(PairArgs);
static_assert(kPairBytes <= (int)kPairSmem, "the frame, its rows and the ring fit one CTA");

__device__ __forceinline__ float4 lds4(const char *sm, int o) { return *reinterpret_cast<const float4 *>(sm + o); }
__device__ __forceinline__ void sts4(char *sm, int o, float4 v) { *reinterpret_cast<float4 *>(sm + o) = v; }

__device__ __forceinline__ float2 lds2(const char *sm, int o) { return *reinterpret_cast<const float2 *>(sm + o); }
__device__ __forceinline__ float lds1(const char *sm, int o) { return *reinterpret_cast<const float *>(sm + o); }

__device__ __forceinline__ uint64_t *bar_at(char *sm, int o) { return reinterpret_cast<uint64_t *>(sm + o); }

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_done(uint32_t bar, uint32_t parity)
{
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return done != 0;
}

struct F3 {
    float4 x, y, z;
};

// Packed pairs of FP32 (sm_100 and up): two cells in one instruction, each rounded as its scalar form.
// ptxas fuses a packed product and the packed sum that takes it, .rn or not, which would change the bits;
// a sum is therefore a packed multiply-add by one (or minus one), exact in its product, whose ones come from the
// launch arguments so that the compiler cannot see them.
struct P2 {
    float a, b;
};
__device__ __forceinline__ P2 sub2(float a0, float a1, float b0, float b1)
{
    P2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tsub.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.a), "=f"(r.b)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
    return r;
}
__device__ __forceinline__ P2 mul2(float a0, float a1, float b0, float b1)
{
    P2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.a), "=f"(r.b)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
    return r;
}

// a one + b: the sum a + b, or with one = -1 the difference b - a
__device__ __forceinline__ P2 sum2(float a0, float a1, float one, P2 b)
{
    P2 r;
    asm("{\n\t.reg .b64 x, y, z, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %4};\n\tmov.b64 z, {%5, %6};\n\t"
        "fma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}"
        : "=f"(r.a), "=f"(r.b)
        : "f"(a0), "f"(a1), "f"(one), "f"(b.a), "f"(b.b));
    return r;
}

// What every update takes: Cx, Cy, Cz, and 1 and -1.
struct Scalars {
    float cx, cy, cz, one, minus;
};

// Two cells: h <- d h + c (da s1 - db s2) from the differences da, db.
template <bool D1>
__device__ __forceinline__ void upd2(float &h0, float &h1, float d0, float d1, float c0, float c1, P2 da, float s1, P2 db, float s2,
                                     const Scalars &S)
{
    const P2 p = mul2(da.a, da.b, s1, s1), m = mul2(db.a, db.b, s2, s2), curl = sum2(m.a, m.b, S.minus, p);
    const P2 t = mul2(c0, c1, curl.a, curl.b);
    P2 g{h0, h1};
    if constexpr (!D1) g = mul2(d0, d1, h0, h1);
    g = sum2(g.a, g.b, S.one, t);
    h0 = g.a;
    h1 = g.b;
}

// All four cells of a unit; differences of whole units, or (x) along the unit with its neighbour n.
struct D4 {
    P2 lo, hi;
};
__device__ __forceinline__ D4 diff(const float4 &a, const float4 &b)
{
    return {sub2(a.x, a.y, b.x, b.y), sub2(a.z, a.w, b.z, b.w)};
}
__device__ __forceinline__ D4 diff_up(const float4 &a, float n)     // a[i + 1] - a[i]
{
    return {{__fsub_rn(a.y, a.x), __fsub_rn(a.z, a.y)}, {__fsub_rn(a.w, a.z), __fsub_rn(n, a.w)}};
}
__device__ __forceinline__ D4 diff_down(const float4 &a, float n)   // a[i] - a[i - 1]
{
    return {{__fsub_rn(a.x, n), __fsub_rn(a.y, a.x)}, {__fsub_rn(a.z, a.y), __fsub_rn(a.w, a.z)}};
}
template <bool D1>
__device__ __forceinline__ void upd4(float4 &h, const float4 &d, const float4 &c, const D4 &da, float s1, const D4 &db, float s2,
                                     const Scalars &S)
{
    upd2<D1>(h.x, h.y, d.x, d.y, c.x, c.y, da.lo, s1, db.lo, s2, S);
    upd2<D1>(h.z, h.w, d.z, d.w, c.z, c.w, da.hi, s1, db.hi, s2, S);
}

// H <- D H + C curl(E): E at the node, Ex, Ey one plane up, Ex, Ez one row up, Ey, Ez one cell on.
template <bool D1>
__device__ __forceinline__ void h_update(F3 &h, const float4 &D, const float4 &C, const F3 &e, const float4 &exk, const float4 &eyk,
                                         const float4 &exj, const float4 &ezj, float eyn, float ezn, const Scalars &S)
{
    upd4<D1>(h.x, D, C, diff(eyk, e.y), S.cz, diff(ezj, e.z), S.cy, S);
    upd4<D1>(h.y, D, C, diff_up(e.z, ezn), S.cx, diff(exk, e.x), S.cz, S);
    upd4<D1>(h.z, D, C, diff(exj, e.x), S.cy, diff_up(e.y, eyn), S.cx, S);
}

// Where a node's E is updated (not on a wall): by row, by plane, by cell of the unit.
struct Inside {
    bool j, x0, x1, x2, x3;
};

// E <- D E + C curl(H) off the walls: H at the node, Hx, Hy one plane down, Hx, Hz one row down, Hy, Hz one cell back.
template <bool D1>
__device__ __forceinline__ void e_update(F3 &e, const float4 &D, const float4 &C, const F3 &h, const float4 &hxk, const float4 &hyk,
                                         const float4 &hxj, const float4 &hzj, float hyp, float hzp, const Inside &in, bool k,
                                         const Scalars &S)
{
    float4 n = e.x;
    upd4<D1>(n, D, C, diff(h.z, hzj), S.cy, diff(h.y, hyk), S.cz, S);
    if (in.j && k) e.x = n;
    n = e.y;
    upd4<D1>(n, D, C, diff(h.x, hxk), S.cz, diff_down(h.z, hzp), S.cx, S);
    if (k && in.x0) e.y.x = n.x;
    if (k && in.x1) e.y.y = n.y;
    if (k && in.x2) e.y.z = n.z;
    if (k && in.x3) e.y.w = n.w;
    n = e.z;
    upd4<D1>(n, D, C, diff_down(h.y, hyp), S.cx, diff(h.x, hxj), S.cy, S);
    if (in.j && in.x0) e.z.x = n.x;
    if (in.j && in.x1) e.z.y = n.y;
    if (in.j && in.x2) e.z.z = n.z;
    if (in.j && in.x3) e.z.w = n.w;
}

__device__ __forceinline__ void add_source(float4 &ez, int cell, float v)
{
    if (cell == 0) ez.x = __fadd_rn(ez.x, v);
    else if (cell == 1) ez.y = __fadd_rn(ez.y, v);
    else if (cell == 2) ez.z = __fadd_rn(ez.z, v);
    else ez.w = __fadd_rn(ez.w, v);
}

// Da, Db (or Ca, Cb) of four material ids; PAIR_SIMPLE: Cb only, D unused.
template <int MODE>
__device__ __forceinline__ void lookup(const float *tab, unsigned ids, int half, float4 &D, float4 &C)
{
    if constexpr (MODE == PAIR_SIMPLE) {
        D = make_float4(1.f, 1.f, 1.f, 1.f);
        C = make_float4(tab[ids & 255u], tab[(ids >> 8) & 255u], tab[(ids >> 16) & 255u], tab[ids >> 24]);
    } else {
        const float2 *t = reinterpret_cast<const float2 *>(tab) + half;
        const float2 a = t[2 * (ids & 255u)], b = t[2 * ((ids >> 8) & 255u)], c = t[2 * ((ids >> 16) & 255u)], d = t[2 * (ids >> 24)];
        D = make_float4(a.x, b.x, c.x, d.x);
        C = make_float4(a.y, b.y, c.y, d.y);
    }
}

}  // namespace

// MANY: a CTA per tile of the batch's instances, in list order; a warp finds its block's instance among the
// tile counts' prefix sums, and the instance's arguments move to shared memory.  Otherwise: one instance, whose
// tiles a CTA takes with the grid's stride.
template <int MODE, bool MANY>
__global__ void __launch_bounds__(kPairThreads, 1)
    k_yee_pair(const InstDesc *__restrict__ D, const PairArgs P1, const PairArgs *__restrict__ PN, const int *__restrict__ tile0, int ninst,
               int q, int *err)
{
    constexpr bool D1 = MODE != PAIR_TABLE, CELLS = MODE == PAIR_CELLS;
    constexpr int S = kPairStages;
    extern __shared__ __align__(128) char sm[];
    const PairArgs &P = MANY ? *reinterpret_cast<const PairArgs *>(sm + kArgsAt) : P1;
    int t = blockIdx.x;
    if constexpr (MANY) {
        // 32 probes a round: the last instance whose first tile is not after this block's
        int lo = 0, n = ninst;
        while (n > 1) {
            const int lane = threadIdx.x & 31, step = (n + 31) / 32;
            const int c = __popc(__ballot_sync(0xffffffffu, lane * step < n && __ldg(tile0 + lo + min(lane * step, n - 1)) <= t)) - 1;
            lo += c * step;
            n = min(step, n - c * step);
        }
        t -= __ldg(tile0 + lo);
        D += lo;
        const int *from = reinterpret_cast<const int *>(PN + lo);
        for (int w = threadIdx.x; w < (int)(sizeof(PairArgs) / 4); w += blockDim.x) reinterpret_cast<int *>(sm + kArgsAt)[w] = __ldg(from + w);
    }
    float *tab = reinterpret_cast<float *>(sm + kTabAt);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (smem_u32(sm) & 127u) {   // TMA destinations need 128-byte alignment: refuse, do not fault
        if (tid == 0) atomicOr(err, 2);
        return;
    }
    if (tid == 0) {
        for (int s = 0; s < S; ++s) mbar_init(bar_at(sm, s * kStage + kFull), 1);
        mbar_init(bar_at(sm, kBar1), blockDim.x / 32);
        mbar_init(bar_at(sm, kBar2), blockDim.x / 32);
        *reinterpret_cast<uint32_t *>(sm + kBaseAt) = smem_u32(sm);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const float4 *gtab = reinterpret_cast<const float4 *>(D->mat_tab);
    for (int m = tid; m < D->nmat; m += blockDim.x) {
        const float4 v = __ldg(gtab + m);
        if (MODE == PAIR_SIMPLE) tab[m] = v.y;
        else reinterpret_cast<float4 *>(tab)[m] = v;
    }
    const float dbu = MODE == PAIR_SIMPLE ? __ldg(gtab).w : CELLS ? __ldg(D->coef[3]) : 0.f;
    __syncthreads();

    // The window's base for the barriers' addresses, read back so that it stays in a register: the compiler
    // would rather work it out again at every barrier.
    const uint32_t base = *reinterpret_cast<volatile uint32_t *>(sm + kBaseAt);
    const int lw = P.lw, RF = P.rf;
    const int par = (D->par + q) & 1, step = D->step + 2 * q;
    const CUtensorMap *maps = static_cast<const CUtensorMap *>(P.tma);
    const int nx = D->nx, ny = D->ny, nz = D->nz;
    const Scalars sc{D->cx, D->cy, D->cz, P.one, -P.one};
    const long long src = D->src;
    const float w1 = src >= 0 && step < D->nwave ? __ldg(D->wave + step) : 0.f;
    const float w2 = src >= 0 && step + 1 < D->nwave ? __ldg(D->wave + step + 1) : 0.f;
    // One instance: the six pointers are launch constants.  MANY: one, and the distance of the fields.
    float *const o0 = P.buf[par ^ 1][0];
    const long long apart = MANY ? P.buf[par ^ 1][1] - o0 : 0;
    float *const oHx = o0, *const oHy = MANY ? o0 + apart : P.buf[par ^ 1][1], *const oHz = MANY ? o0 + 2 * apart : P.buf[par ^ 1][2];
    float *const oEx = MANY ? o0 + 3 * apart : P.buf[par ^ 1][3], *const oEy = MANY ? o0 + 4 * apart : P.buf[par ^ 1][4];
    float *const oEz = MANY ? o0 + 5 * apart : P.buf[par ^ 1][5];
    const unsigned pitch = D->pitch, plane = (unsigned)D->plane;

    // A tile's frame and planes: the planes kstart .. k1 + 1 are loaded, the last one as "next" only.
    auto tile_at = [&](int t, int &xt, int &yt, int &k0, int &k1, int &kstart) {
        const int zt = t / (P.nxt * P.nyt), r = t - zt * P.nxt * P.nyt;
        xt = r % P.nxt;
        yt = r / P.nxt;
        k0 = zt * P.kc;
        k1 = min(k0 + P.kc, nz);
        kstart = max(k0 - 2, 0);
    };
    // Copies of plane k of the frame at (px, py) into the ring slot at byte c, by one warp.
    auto issue = [&](int px, int py, int k, int c) {
        if (lane == 0) mbar_expect_tx(bar_at(sm, c + kFull), (uint32_t)(CELLS ? P.tx_bytes - P.mw * P.rf : P.tx_bytes));
        __syncwarp();
        if (lane < (CELLS ? 6 : 7))
            tma_load_3d(sm + c + lane * kField, lane < 6 ? maps + par * 6 + lane : maps + 12,
                        lane < 6 ? px : px & ~15, py, k, bar_at(sm, c + kFull));
    };
    if (lane < (CELLS ? 6 : 7)) tma_acquire(lane < 6 ? maps + par * 6 + lane : maps + 12);
    // Everything above is constant over a chunk; the fields are the launch's before this one.
    chain_wait();
    if (t < P.tiles) {
        int xt, yt, k0, k1, kstart;
        tile_at(t, xt, yt, k0, k1, kstart);
        if (warp == 0)   // a tile has more planes than the ring
            for (int s = 0; s < S; ++s) issue(xt * (4 * lw - 4), yt * (RF - 3), kstart + s, s * kStage);
    }

    // this thread's unit of the frame; threads beyond it repeat the last one without storing
    const int r = min(tid / lw, RF - 1), sl = min(tid, lw * RF - 1), lx = sl - r * lw;
    const int o = 16 * sl, rs = 16 * lw, ot = 16 * tid, od = max(ot - rs, 0);
    const bool edge_hi = lane == 31, edge_lo = lane == 0 && tid > 0;
    // Pairs from the next warp and the one before; lanes that need none read a pair nobody uses.
    const int e_own = 8 * warp + 8, e_hi = edge_hi ? e_own + 8 : 0, e_lo = edge_lo ? e_own - 8 : 0;
    const int o_hi = edge_hi ? o + 16 : 0;   // in a ring stage: the float beyond the unit
    // The ring: byte of the current plane's slot, and the parity of its barrier's next phase; a plane computed
    // per phase of the barriers 1 and 2.  The warps take turns at refilling the ring.
    int cs = 0, turn = 0;
    unsigned cph = 0, n = 0;
    const int nwarps = blockDim.x / 32;
    bool failed = false;
    auto wait = [&](int bar, unsigned phase) {
        if (!mbar_done(base + bar, phase & 1) && !failed && !mbar_wait(bar_at(sm, bar), phase & 1)) {
            failed = true;
            atomicOr(err, 1);
        }
    };

    for (; t < P.tiles; t += gridDim.x) {
        int xt, yt, k0, k1, kstart;
        tile_at(t, xt, yt, k0, k1, kstart);
        const int xs = xt * (4 * lw - 4), js = yt * (RF - 3);
        const int i = xs + 4 * lx, j = js + r;
        const Inside in{j >= 1 && j < ny, i >= 1 && i < nx, i + 1 < nx, i + 2 < nx, i + 3 < nx};
        // cells of the unit that this tile yields: all four, its upper or lower two, or (at the grid's end) the first few
        const bool row_out = tid < lw * RF && j < ny && r <= RF - 2 && (yt == 0 || r >= 2);
        const int left = nx - i;
        const bool upper = xt > 0 && lx == 0, lower = xt + 1 < P.nxt && lx == lw - 1;
        const bool full = row_out && !upper && !lower && left >= 4, part = row_out && left > 0 && !full;
        unsigned off = (unsigned)i + pitch * (unsigned)j + plane * (unsigned)kstart;   // of plane k
        // the source's plane and cell in this unit
        int src_k = -1, src_c = 0;
        if (src >= 0) {
            const int sk = (int)(src / plane), rem = (int)(src - (long long)sk * plane), sj = rem / (int)pitch, si = rem - sj * (int)pitch;
            if (sj == j && si >= i && si < i + 4) { src_k = sk; src_c = si - i; }
        }
        const int mo = 6 * kField + r * P.mw + (xs & 15) + 4 * lx;

        // PAIR_CELLS: Cb of the node, loaded a plane ahead; units beyond the rows repeat one within
        const float *const cbp = CELLS ? D->coef[1] + (min((unsigned)i, pitch - 4) + pitch * (unsigned)min(j, ny)) : nullptr;
        auto cb_at = [&](int k) {   // volatile: stays where it is written, a plane before its use
            float4 v;
            asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                         : "l"(cbp + plane * (unsigned)min(k, nz)));
            return v;
        };
        float4 cb_n{};
        if constexpr (CELLS) cb_n = cb_at(kstart);

        F3 H1a{}, H1b{}, E1a{}, E1b{}, H2a{}, H2b{};
        float4 cba{}, cbb{};               // Ca = Da = 1: Cb of two planes
        unsigned ida = 0, idb = 0;         // otherwise their material ids

        // E2(kk) from H2(kk) (own, and the rows of buffer B), H2(kk-1); H2 and E2 stored.
        auto seg_c = [&](auto buffer, int kk, unsigned offc, unsigned ph, F3 &E1, const F3 &H2, const F3 &H2m, const float4 &cb, unsigned ids) {
            constexpr int B = decltype(buffer)::value, rows = kRowsAt + B * kRowBuf;
            const char *rd = sm + od;
            float hyp = __shfl_up_sync(0xffffffffu, H2.y.w, 1), hzp = __shfl_up_sync(0xffffffffu, H2.z.w, 1);
            wait(kBar2, ph);
            const float2 e = lds2(sm + e_lo, kEdgesAt + B * kEdgeBuf + X_H2 * kEdge);
            if (edge_lo) { hyp = e.x; hzp = e.y; }
            const float4 hxj = lds4(rd, rows + R_HX2 * kField), hzj = lds4(rd, rows + R_HZ2 * kField);
            float4 Dc = make_float4(1.f, 1.f, 1.f, 1.f), Cc = cb;
            if constexpr (MODE == PAIR_TABLE) lookup<MODE>(tab, ids, 0, Dc, Cc);
            e_update<D1>(E1, Dc, Cc, H2, H2m.x, H2m.y, hxj, hzj, hyp, hzp, in, kk >= 1, sc);
            if (kk == src_k) add_source(E1.z, src_c, w2);
            if (full) {
                *reinterpret_cast<float4 *>(oHx + offc) = H2.x;
                *reinterpret_cast<float4 *>(oHy + offc) = H2.y;
                *reinterpret_cast<float4 *>(oHz + offc) = H2.z;
                *reinterpret_cast<float4 *>(oEx + offc) = E1.x;
                *reinterpret_cast<float4 *>(oEy + offc) = E1.y;
                *reinterpret_cast<float4 *>(oEz + offc) = E1.z;
            } else if (part) {
                if (left >= 4) {
                    auto put = [&](float *p, const float4 &v) {
                        *reinterpret_cast<float2 *>(p + offc + (upper ? 2 : 0)) = upper ? make_float2(v.z, v.w) : make_float2(v.x, v.y);
                    };
                    put(oHx, H2.x); put(oHy, H2.y); put(oHz, H2.z);
                    put(oEx, E1.x); put(oEy, E1.y); put(oEz, E1.z);
                } else {
                    auto put = [&](float *p, const float4 &v) {
                        if (!upper) p[offc] = v.x;
                        if (!upper && left > 1) p[offc + 1] = v.y;
                        if (!lower && left > 2) p[offc + 2] = v.z;
                    };
                    put(oHx, H2.x); put(oHy, H2.y); put(oHz, H2.z);
                    put(oEx, E1.x); put(oEy, E1.y); put(oEz, E1.z);
                }
            }
        };

        // One plane, in buffer B of the rows and pairs (alternating within a tile: what the last plane of a
        // tile leaves in its buffer has been read when the next tile's first plane writes there).  On entry E1
        // holds E1(k-2), E1m E1(k-1), H1m H1(k-1), H2p H2(k-2), H2 H2(k-3), cb and id plane k-2's; on exit H1,
        // E1, H2 hold H1(k), E1(k), H2(k-1), cb and id plane k's.  The caller swaps the names.
        auto plane_step = [&](auto buffer, int k, F3 &H1, const F3 &H1m, F3 &E1, const F3 &E1m, F3 &H2, const F3 &H2p, float4 &cb,
                              unsigned &id, unsigned id_m) {
            constexpr int B = decltype(buffer)::value, rows = kRowsAt + B * kRowBuf, rows_m = kRowsAt + (B ^ 1) * kRowBuf;
            constexpr int pairs = kEdgesAt + B * kEdgeBuf, pairs_m = kEdgesAt + (B ^ 1) * kEdgeBuf;
            const int ns = cs == (S - 1) * kStage ? 0 : cs + kStage;
            const unsigned nph = cs == (S - 1) * kStage ? cph ^ 1 : cph;
            char *const rw = sm + ot;   // own slot of the rows
            if (k == kstart) wait(cs + kFull, cph);
            const char *cur = sm + cs, *co = cur + o, *no = sm + ns + o;
            // ---- H1(k) ----
            F3 e0;
            e0.x = lds4(co, 3 * kField);
            e0.y = lds4(co, 4 * kField);
            e0.z = lds4(co, 5 * kField);
            unsigned ids = 0;
            [[maybe_unused]] const float4 cb_k = cb_n;
            if constexpr (CELLS) cb_n = cb_at(k + 1);
            if constexpr (!CELLS) ids = *reinterpret_cast<const unsigned *>(cur + mo);
            float4 Dh = make_float4(1.f, 1.f, 1.f, 1.f), Ch = make_float4(dbu, dbu, dbu, dbu);
            {
                const char *cj = co + rs, *ch = cur + o_hi;
                const float4 exj = lds4(cj, 3 * kField), ezj = lds4(cj, 5 * kField);
                H1.x = lds4(co, 0);
                H1.y = lds4(co, kField);
                H1.z = lds4(co, 2 * kField);
                const float eyl = lds1(ch, 4 * kField), ezl = lds1(ch, 5 * kField);
                wait(ns + kFull, nph);
                const float4 exk = lds4(no, 3 * kField), eyk = lds4(no, 4 * kField);
                float ezn = __shfl_down_sync(0xffffffffu, e0.z.x, 1), eyn = __shfl_down_sync(0xffffffffu, e0.y.x, 1);
                if (edge_hi) { eyn = eyl; ezn = ezl; }
                if constexpr (MODE == PAIR_TABLE) lookup<MODE>(tab, ids, 1, Dh, Ch);
                h_update<D1>(H1, Dh, Ch, e0, exk, eyk, exj, ezj, eyn, ezn, sc);
            }
            sts4(rw, rows + R_HX1 * kField, H1.x);
            sts4(rw, rows + R_HZ1 * kField, H1.z);
            if (edge_hi) *reinterpret_cast<float2 *>(sm + e_own + pairs + X_H1 * kEdge) = make_float2(H1.y.w, H1.z.w);
            __syncwarp();
            if (lane == 0) mbar_arrive(base + kBar1);
            // ---- E2(k-2) ----
            if (k - 2 >= k0) seg_c(std::integral_constant<int, (B ^ 1)>(), k - 2, off - 2 * plane, n - 1, E1, H2p, H2, cb, id);
            // ---- E1(k) ----
            float4 Dc = make_float4(1.f, 1.f, 1.f, 1.f);
            id = ids;
            if constexpr (CELLS) cb = cb_k;
            else lookup<MODE>(tab, ids, 0, Dc, cb);
            float hyp = __shfl_up_sync(0xffffffffu, H1.y.w, 1), hzp = __shfl_up_sync(0xffffffffu, H1.z.w, 1);
            float ezn = __shfl_down_sync(0xffffffffu, E1m.z.x, 1), eyn = __shfl_down_sync(0xffffffffu, E1m.y.x, 1);
            wait(kBar1, n);
            // Every warp has read plane k's slot (and, on the tile's last plane, k + 1's): refill it with the
            // plane S on, of this tile or the next.
            if (warp == turn) {
                if (k + S <= k1 + 1) {
                    issue(xs, js, k + S, cs);
                } else if (t + (int)gridDim.x < P.tiles) {
                    int xt2, yt2, a, b2, ks2;
                    tile_at(t + gridDim.x, xt2, yt2, a, b2, ks2);
                    issue(xt2 * (4 * lw - 4), yt2 * (RF - 3), ks2 + k + S - k1 - 2, cs);
                    if (k == k1) issue(xt2 * (4 * lw - 4), yt2 * (RF - 3), ks2 + S - 1, ns);
                }
            }
            turn = turn + 1 == nwarps ? 0 : turn + 1;
            const char *rd = sm + od, *rj = sm + ot + rs;
            const float2 eh = lds2(sm + e_lo, pairs + X_H1 * kEdge), ee = lds2(sm + e_hi, pairs_m + X_E1 * kEdge);
            const float4 hxj = lds4(rd, rows + R_HX1 * kField), hzj = lds4(rd, rows + R_HZ1 * kField);
            const float4 exj = lds4(rj, rows_m + R_EX1 * kField), ezj = lds4(rj, rows_m + R_EZ1 * kField);   // for H2 below
            if (edge_lo) { hyp = eh.x; hzp = eh.y; }
            if (edge_hi) { eyn = ee.x; ezn = ee.y; }
            E1 = e0;
            e_update<D1>(E1, Dc, cb, H1, H1m.x, H1m.y, hxj, hzj, hyp, hzp, in, k >= 1 && k < nz, sc);
            if (k == src_k) add_source(E1.z, src_c, w1);
            sts4(rw, rows + R_EX1 * kField, E1.x);
            sts4(rw, rows + R_EZ1 * kField, E1.z);
            if (lane == 0) *reinterpret_cast<float2 *>(sm + e_own + pairs + X_E1 * kEdge) = make_float2(E1.y.x, E1.z.x);
            // ---- H2(k-1) ----
            if (k > kstart) {
                if constexpr (MODE == PAIR_TABLE) lookup<MODE>(tab, id_m, 1, Dh, Ch);
                H2 = H1m;
                h_update<D1>(H2, Dh, Ch, E1m, E1.x, E1.y, exj, ezj, eyn, ezn, sc);
                sts4(rw, rows + R_HX2 * kField, H2.x);
                sts4(rw, rows + R_HZ2 * kField, H2.z);
                if (edge_hi) *reinterpret_cast<float2 *>(sm + e_own + pairs + X_H2 * kEdge) = make_float2(H2.y.w, H2.z.w);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(base + kBar2);
            off += plane;
            ++n;
            cs = ns;
            cph = nph;
        };

        constexpr std::integral_constant<int, 0> even{};
        constexpr std::integral_constant<int, 1> uneven{};
        int k = kstart;
        for (; k + 1 <= k1; k += 2) {
            plane_step(even, k, H1a, H1b, E1a, E1b, H2a, H2b, cba, ida, idb);
            plane_step(uneven, k + 1, H1b, H1a, E1b, E1a, H2b, H2a, cbb, idb, ida);
        }
        if (k == k1) {
            plane_step(even, k, H1a, H1b, E1a, E1b, H2a, H2b, cba, ida, idb);
            seg_c(even, k1 - 1, off - 2 * plane, n - 1, E1b, H2a, H2b, cbb, idb);
        } else {
            seg_c(uneven, k1 - 1, off - 2 * plane, n - 1, E1a, H2b, H2a, cba, ida);
        }
        // past the tile's last plane, which was read as "next" only
        cs += kStage;
        if (cs == S * kStage) { cs = 0; cph ^= 1; }
    }
    // Every issued plane has normally been waited for.  If a wait expired, let the copies still in
    // flight land (bounded) before this CTA's shared memory is released.
    if (tid == 0)
        for (int s = 0; s < S; ++s) mbar_wait(bar_at(sm, s * kStage + kFull), s * kStage < cs ? cph : cph ^ 1);
}

namespace {

// Bytes of a stage's copies.
void lay_out(PairPlan &p)
{
    PairArgs &a = p.args;
    a.tx_bytes = 16 * a.lw * (6 * a.rf + 2) + a.mw * a.rf;   // Ex, Ez: one row more
    p.smem = kPairBytes;
    a.one = 1.0f;
}

}  // namespace

// The frame of nxt tiles in x and at least `nyt` in y, with no more rows than that needs.  False when no such
// frame exists; a->nyt may come out larger, where the threads or the room for the ids do not allow the rows.  Every
// grid of 4 rows or more has a frame for some nxt.
static bool pair_frame(int nx, int ny, int nxt, int nyt, int threads, PairArgs *a)
{
    a->nxt = nxt;
    a->lw = (nx + 1 + 4 * (nxt - 1) + 4 * nxt - 1) / (4 * nxt);
    if (a->lw > kMaxLw || (a->lw < 8 && nxt > 1)) return false;
    a->mw = (4 * a->lw + 12 + 15) / 16 * 16;
    const int most = std::min(std::min(threads / a->lw, 255), std::min(ny + 1, kIds / a->mw));
    if (most < 5) return false;
    const int least = ny <= most - 1 ? 1 : 1 + (ny - (most - 1) + most - 4) / (most - 3);   // tiles with all those rows
    a->nyt = std::max(nyt, least);
    a->rf = std::min(most, std::max(5, (ny + 1 + 3 * (a->nyt - 1) + a->nyt - 1) / a->nyt));
    return a->nyt == 1 || (a->nyt - 1) * (a->rf - 3) < ny - 2;   // the last tile has rows of its own
}

static bool pair_fits(int nx, int ny, int nz) { return make_layout(nx, ny, nz).total * 4 < 1LL << 32 && nz >= 8; }

// The tile shape with the least estimated time for two steps: rounds of resident CTAs times the planes each
// streams (its depth, the planes recomputed at its start, the ring's turn at its end) times a plane's time, which
// grows with the frame's warps (320 threads of 352: taken as 0.94 of the time)
// and is 7-14 % longer with rows of 9 to 11 units than of 13 and more.
bool plan_pair(int nx, int ny, int nz, PairPlan *out)
{
    const int sms = sm_count();
    double best = 1e30;
    bool found = false;
    if (sms <= 0 || !pair_fits(nx, ny, nz)) return false;
    for (int nxt = 1; nxt <= 64; ++nxt)
        for (int more = 0, nyt = 1; more < 6; ++more, ++nyt) {   // the fewest rows of tiles, and a few more of lower ones
            PairPlan p{};
            if (!pair_frame(nx, ny, nxt, nyt, kPairThreads, &p.args)) break;
            nyt = p.args.nyt;
            p.threads = (p.args.lw * p.args.rf + 31) / 32 * 32;
            const double plane = (0.35 + 0.65 * p.threads / kPairThreads) * (1 + 8.0 / (p.args.lw * p.args.lw));
            for (int nzt = 1; nzt <= nz / 8; ++nzt) {
                const int kc = (nz + nzt - 1) / nzt;
                if ((nz + kc - 1) / kc != nzt) continue;
                const long long tiles = (long long)nxt * nyt * nzt, waves = (tiles + sms - 1) / sms;
                p.args.nzt = nzt; p.args.kc = kc; p.args.tiles = (int)tiles;
                p.grid = (int)std::min<long long>(tiles, sms);
                const double c = (double)waves * (kc + 3.5) * plane;
                if (c < best) {
                    lay_out(p);
                    best = c;
                    *out = p;
                    found = true;
                }
            }
        }
    return found;
}

constexpr int kBatchThreads = kPairThreads;

// In a batch every CTA has all its threads, so the frame is the one with the fewest tiles per plane.  It does
// not depend on the rest of the batch; the depth does (plan_pair_depths).
bool plan_pair_member(int nx, int ny, int nz, PairPlan *out)
{
    bool found = false;
    if (!pair_fits(nx, ny, nz)) return false;
    for (int nxt = 1; nxt <= 64; ++nxt) {
        PairPlan p{};
        if (!pair_frame(nx, ny, nxt, 1, kBatchThreads, &p.args)) continue;
        if (!found || nxt * p.args.nyt < out->args.nxt * out->args.nyt) {
            lay_out(p);
            *out = p;
            found = true;
        }
    }
    return found;
}

static int pair_depth(int nz, int cap)   // near-equal tiles of at most cap planes, if that leaves 8 in each
{
    const int parts = std::max(1, std::min((nz + cap - 1) / cap, nz / 8));
    return (nz + parts - 1) / parts;
}

// The depths of a batch's tiles: the cap whose list has the least bound on its time, which is the smaller of
// whole rounds of the deepest tile and (a free SM takes the next tile, deepest first) the mean load plus one
// tile.  A tile costs its planes, those recomputed, and its CTA's start (about five planes' time).
void plan_pair_depths(PairPlan *const plans[], const int nz[], int n)
{
    constexpr double kStart = 8.5;
    const int sms = std::max(1, sm_count());
    int deepest = 8, cap = 8;
    for (int q = 0; q < n; ++q) deepest = std::max(deepest, nz[q]);
    double best = 1e30;
    for (int c = 8; c <= deepest; c += 1 + c / 16) {
        double tiles = 0, load = 0;
        int top = 0;
        for (int q = 0; q < n; ++q) {
            const int kc = pair_depth(nz[q], c), t = plans[q]->args.nxt * plans[q]->args.nyt * ((nz[q] + kc - 1) / kc);
            tiles += t;
            load += t * (kc + kStart);
            top = std::max(top, kc);
        }
        const double rounds = std::ceil(tiles / sms) * (top + kStart), mean = load / sms + top + kStart;
        if (std::min(rounds, mean) < best) {
            best = std::min(rounds, mean);
            cap = c;
        }
    }
    for (int q = 0; q < n; ++q) {
        PairArgs &a = plans[q]->args;
        a.kc = pair_depth(nz[q], cap);
        a.nzt = (nz[q] + a.kc - 1) / a.kc;
        a.tiles = a.nxt * a.nyt * a.nzt;
    }
}

int encode_pair_maps(const InstDesc &d, const PairPlan &p, void *host_out)
{
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc) return set_error(PTK_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    CUtensorMap *out = static_cast<CUtensorMap *>(host_out);
    const cuuint64_t dims[3] = {(cuuint64_t)d.pitch, (cuuint64_t)d.ny + 1, (cuuint64_t)d.nz + 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    for (int m = 0; m < 13; ++m) {
        const bool u8 = m == 12;
        const int f = m % 6;
        void *base = u8 ? (void *)d.mat : (void *)d.buf[m / 6][f];
        const cuuint64_t e = u8 ? 1 : 4, strides[2] = {(cuuint64_t)d.pitch * e, (cuuint64_t)d.plane * e};
        const cuuint32_t box[3] = {(cuuint32_t)(u8 ? p.args.mw : 4 * p.args.lw),
                                   (cuuint32_t)(p.args.rf + (!u8 && (f == 3 || f == 5) ? 1 : 0)), 1};
        CUresult r = enc(&out[m], u8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box,
                         estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return set_error(PTK_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) for map %d", (int)r, m);
    }
    return PTK_OK;
}

template <int MODE, bool MANY>
static int launch_pair(const InstDesc *d_inst, const PairArgs &one, const PairArgs *many, const int *tile0, int ninst, int grid, int threads,
                       int pair, int *err, cudaStream_t s)
{
    PTK_CUDA_TRY(cudaFuncSetAttribute(k_yee_pair<MODE, MANY>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairBytes));
    PTK_CUDA_TRY(launch_chained(k_yee_pair<MODE, MANY>, dim3(grid), dim3(threads), kPairBytes, s, pair > 0, d_inst, one, many, tile0, ninst,
                                pair, err));
    count_launches(1);
    return PTK_OK;
}

int launch_yee_pair(const InstDesc *d_inst, const PairPlan &p, int mode, int pair, int *err, cudaStream_t s)
{
    return mode == PAIR_SIMPLE ? launch_pair<PAIR_SIMPLE, false>(d_inst, p.args, nullptr, nullptr, 1, p.grid, p.threads, pair, err, s)
           : mode == PAIR_CELLS  ? launch_pair<PAIR_CELLS, false>(d_inst, p.args, nullptr, nullptr, 1, p.grid, p.threads, pair, err, s)
                                 : launch_pair<PAIR_TABLE, false>(d_inst, p.args, nullptr, nullptr, 1, p.grid, p.threads, pair, err, s);
}

int launch_yee_pair_batch(const InstDesc *d_insts, const PairArgs *d_args, const int *d_tile0, int ninst, int tiles, int pair, int *err,
                          cudaStream_t s)
{
    return launch_pair<PAIR_SIMPLE, true>(d_insts, PairArgs{}, d_args, d_tile0, ninst, tiles, kBatchThreads, pair, err, s);
}

}  // namespace ptk
