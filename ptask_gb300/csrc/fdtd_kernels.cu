// fdtd_kernels.cu -- sm_103a kernels for the Yee-grid FDTD task graph.
//
// The update equations are those of the reference's six field tasks
// (ptaskUnitTest/graphfdtd.cpp:185-312, HLSL twins ptaskUnitTest/fdtdKernels/{Hx..Ez}Comp.hlsl),
// generalised to per-cell coefficients:
//   H' = Da*H + Db*curl(E)            (reference: Da = 1, Db = Dt/mu0)
//   E' = Ca*E + Cb*curl(H')           (reference: Ca = 1, Cb = Dt/eps0), PEC faces copied through.
// Every floating-point operation is issued with an explicit round-to-nearest intrinsic so that no
// multiply-add is contracted; with Ca = Da = 1 the results are bit-identical to the reference's
// FP32 host code.
//
// Kernels here:
//   k_yee_step<BY>   fused H+E step over a work list of tiles of one or many instances (padded
//                    layout), operands in registers.  Bandwidth bound: 64 algorithmic bytes per cell.
//   k_field_ref      the reference's per-field task kernels (dense layout), one field per launch.
//   k_rows           reference layout <-> padded layout.
#include "fdtd_chain.cuh"
#include "fdtd_device.cuh"

#include <cstdio>

namespace ptk {

#define FULL_MASK 0xffffffffu

// h + c*((a1-a0)*s1 - (b1-b0)*s2): the reference's scalar form (graphfdtd.cpp:198 and siblings).
__device__ __forceinline__ float yee_ref(float h, float c, float a1, float a0, float s1, float b1,
                                         float b0, float s2)
{
    const float curl = __fsub_rn(__fmul_rn(__fsub_rn(a1, a0), s1), __fmul_rn(__fsub_rn(b1, b0), s2));
    return __fadd_rn(h, __fmul_rn(c, curl));
}

// V consecutive x cells held by one thread (V = 1, 2, 4: 32-, 64- or 128-bit accesses).
template <int V>
struct __align__(4 * V) Vec {
    float v[V];
};

template <int V>
__device__ __forceinline__ Vec<V> ldv(const float *__restrict__ p)
{
    Vec<V> r;
    if constexpr (V == 4) {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
        r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w;
    } else if constexpr (V == 2) {
        const float2 t = __ldg(reinterpret_cast<const float2 *>(p));
        r.v[0] = t.x; r.v[1] = t.y;
    } else {
        r.v[0] = __ldg(p);
    }
    return r;
}

template <int V>
__device__ __forceinline__ Vec<V> zerov()
{
    Vec<V> r;
#pragma unroll
    for (int e = 0; e < V; ++e) r.v[e] = 0.f;
    return r;
}

// Store the first `n` (1..V) elements of v at p; one aligned vector store when n == V.
template <int V>
__device__ __forceinline__ void stv(float *p, const Vec<V> &v, int n)
{
    if (n >= V) {
        if constexpr (V == 4) *reinterpret_cast<float4 *>(p) = make_float4(v.v[0], v.v[1], v.v[2], v.v[3]);
        else if constexpr (V == 2) *reinterpret_cast<float2 *>(p) = make_float2(v.v[0], v.v[1]);
        else p[0] = v.v[0];
    } else {
#pragma unroll
        for (int e = 0; e < V; ++e)
            if (e < n) p[e] = v.v[e];
    }
}

// ---------------------------------------------------------------------------------------------
// Fused Yee step.  One CTA owns a main tile of 32*V (x) by BY (y) cells and a range of z planes
// [k0, k1); it streams the planes in order, keeping the previous plane's new Hx, Hy and the next
// plane's Ex, Ey in registers (sliding window), so every array element is read from HBM once per
// step.  Thread (lane, ty): ty = 1..BY own row y0+ty-1, V consecutive x cells per lane (V*32-bit
// loads and stores); ty = 0 is a halo row y0-1 that only recomputes new Hx, Hz for the E update of
// row y0.  In-plane neighbours: x+1 / x-1 through warp shuffles (lane 31 / lane 0 fetch the one
// cell beyond the tile), y+1 / y-1 through shared memory.  A tile that starts at k0 > 0 first
// recomputes new Hx, Hy on plane k0-1 ("warm" plane, no stores).
// Work list: blockIdx.x indexes the concatenated tiles of all instances (tile0 = prefix sums);
// each instance's main tiles are followed by its face tiles.  Every instance of a launch must have
// been planned with vec == V.
// ---------------------------------------------------------------------------------------------
template <int BY, int V>
__global__ void __launch_bounds__(32 * (BY + 1), BY <= 4 ? 4 : (BY <= 8 ? 2 : 1))
k_yee_step(const InstDesc *__restrict__ insts, const int *__restrict__ tile0, int ninst, int s_off,
           int total_tiles)
{
    constexpr int TX = 32 * V;
    __shared__ Vec<V> sEx[BY + 1][32];
    __shared__ Vec<V> sEz[BY + 1][32];
    __shared__ Vec<V> sHx[BY + 1][32];
    __shared__ Vec<V> sHz[BY + 1][32];

    // Persistent form: a CTA takes tiles blockIdx.x, blockIdx.x + gridDim.x, ...  Shared memory is
    // safe to reuse across tiles: every plane ends with a barrier after the last read of sEx/sEz,
    // and sHx/sHz are first written after the next tile's first barrier.
    for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) {
    int lo = 0, hi = ninst;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(tile0 + mid) <= t) lo = mid; else hi = mid;
    }
    const InstDesc *__restrict__ D = insts + lo;
    if (s_off >= D->steps_left) continue;
    const int lt = t - __ldg(tile0 + lo);
    const int step = D->step + s_off;
    const int par = (D->par + s_off) & 1;
    const int nmain = D->tiles_x * D->tiles_y * D->tiles_z;
    if (lt >= nmain) {
        yee_faces(D, par, lt - nmain, 32 * (BY + 1) * kFaceCellsPerThread);
        continue;
    }

    const int nx = D->nx, ny = D->ny, nz = D->nz, pitch = D->pitch, kc = D->kc;
    const long long plane = D->plane;
    const float cx = D->cx, cy = D->cy, cz = D->cz;
    const float *__restrict__ Hx = D->buf[par][0];
    const float *__restrict__ Hy = D->buf[par][1];
    const float *__restrict__ Hz = D->buf[par][2];
    const float *__restrict__ Ex = D->buf[par][3];
    const float *__restrict__ Ey = D->buf[par][4];
    const float *__restrict__ Ez = D->buf[par][5];
    float *__restrict__ oHx = D->buf[par ^ 1][0];
    float *__restrict__ oHy = D->buf[par ^ 1][1];
    float *__restrict__ oHz = D->buf[par ^ 1][2];
    float *__restrict__ oEx = D->buf[par ^ 1][3];
    float *__restrict__ oEy = D->buf[par ^ 1][4];
    float *__restrict__ oEz = D->buf[par ^ 1][5];
    const float *__restrict__ Ca = D->coef[0];
    const float *__restrict__ Cb = D->coef[1];
    const float *__restrict__ Da = D->coef[2];
    const float *__restrict__ Db = D->coef[3];
    const long long src = D->src;
    const float srcv = (src >= 0 && step < D->nwave) ? __ldg(D->wave + step) : 0.f;

    int r = lt;
    const int xt = r % D->tiles_x; r /= D->tiles_x;
    const int yt = r % D->tiles_y;
    const int zt = r / D->tiles_y;
    const int x0 = xt * TX, y0 = yt * BY;
    const int k0 = zt * kc, k1 = min(k0 + kc, nz);
    const int kstart = k0 > 0 ? k0 - 1 : k0;

    const int lane = threadIdx.x, ty = threadIdx.y;
    const int i = x0 + V * lane;
    const int j = y0 + ty - 1;
    const bool halo = (ty == 0);
    const bool xin = (i <= nx);               // vector holds at least one node of the row
    const bool jrow = (j >= 0 && j < ny);     // a row of cells (or a valid halo row)
    const bool jshare = (!halo && j == ny);   // the wall row: only lends Ex, Ez to row Ny-1
    const int nout = min(V, nx - i);          // cells of this vector inside [0, Nx)
    const bool xl = (lane == 31) && (x0 + TX <= nx);   // one node beyond the tile exists
    const bool hcol = (!halo) && (lane == 0) && (x0 > 0) && jrow;   // lane 0 recomputes x0-1

    // Offsets are formed only for rows that exist (j >= 0).
    long long off = (long long)i + (long long)pitch * (j < 0 ? 0 : j) + plane * kstart;

    Vec<V> ex0 = zerov<V>(), ey0 = zerov<V>();   // Ex(k), Ey(k)
    Vec<V> hxp = zerov<V>(), hyp = zerov<V>();   // new Hx, Hy on plane k-1
    if (!halo && xin) {
        if (jrow || jshare) ex0 = ldv<V>(Ex + off);
        if (jrow) ey0 = ldv<V>(Ey + off);
    }

    for (int k = kstart; k < k1; ++k, off += plane) {
        const bool warm = (k < k0);
        Vec<V> hx = zerov<V>(), hy = zerov<V>(), hz = zerov<V>(), ez = zerov<V>(), ex1 = zerov<V>(), ey1 = zerov<V>();
        Vec<V> da = zerov<V>(), db = zerov<V>(), ca = zerov<V>(), cb = zerov<V>();
        Vec<V> exj1 = zerov<V>(), ezj1 = zerov<V>();
        float ez_l = 0.f, ey_l = 0.f;                                  // lane 31: x0+TX
        float hy_h = 0.f, hz_h = 0.f, ez_h = 0.f, ex_h0 = 0.f, ex_h1 = 0.f, ex_hj = 0.f,
              ey_h = 0.f, da_h = 0.f, db_h = 0.f;                        // lane 0: x0-1

        // ---- loads ----------------------------------------------------------------------
        if (halo) {
            if (!warm && jrow && xin) {
                hx = ldv<V>(Hx + off); hz = ldv<V>(Hz + off); ez = ldv<V>(Ez + off);
                ex0 = ldv<V>(Ex + off); ey0 = ldv<V>(Ey + off); ey1 = ldv<V>(Ey + off + plane);
                da = ldv<V>(Da + off); db = ldv<V>(Db + off);
                if (xl) ey_l = __ldg(Ey + off + V);
            }
        } else if (jrow && xin) {
            hx = ldv<V>(Hx + off); hy = ldv<V>(Hy + off); ez = ldv<V>(Ez + off);
            ex1 = ldv<V>(Ex + off + plane); ey1 = ldv<V>(Ey + off + plane);
            da = ldv<V>(Da + off); db = ldv<V>(Db + off);
            if (!warm) { hz = ldv<V>(Hz + off); ca = ldv<V>(Ca + off); cb = ldv<V>(Cb + off); }
            if (ty == BY) { exj1 = ldv<V>(Ex + off + pitch); ezj1 = ldv<V>(Ez + off + pitch); }
            if (xl) { ez_l = __ldg(Ez + off + V); ey_l = __ldg(Ey + off + V); }
            if (hcol && !warm) {
                const long long oh = off - 1;
                hy_h = __ldg(Hy + oh); hz_h = __ldg(Hz + oh); ez_h = __ldg(Ez + oh);
                ex_h0 = __ldg(Ex + oh); ex_h1 = __ldg(Ex + oh + plane); ex_hj = __ldg(Ex + oh + pitch);
                ey_h = __ldg(Ey + oh); da_h = __ldg(Da + oh); db_h = __ldg(Db + oh);
            }
        } else if (jshare && xin) {
            ex0 = ldv<V>(Ex + off); ez = ldv<V>(Ez + off);
        }

        // ---- share Ex, Ez of each row with the row above (its y+1 neighbour) -----------------
        sEx[ty][lane] = ex0;
        sEz[ty][lane] = ez;
        __syncthreads();
        if (ty < BY) {
            exj1 = sEx[ty + 1][lane];
            ezj1 = sEz[ty + 1][lane];
        }

        // ---- x+1 neighbours through shuffles ----------------------------------------------
        float ez_n = __shfl_down_sync(FULL_MASK, ez.v[0], 1);
        float ey_n = __shfl_down_sync(FULL_MASK, ey0.v[0], 1);
        if (lane == 31) { ez_n = ez_l; ey_n = ey_l; }

        // ---- new H on plane k ---------------------------------------------------------------
        Vec<V> hxn, hyn, hzn;
#pragma unroll
        for (int e = 0; e < V; ++e) {
            const float ez_ip = e < V - 1 ? ez.v[e + 1] : ez_n;
            const float ey_ip = e < V - 1 ? ey0.v[e + 1] : ey_n;
            hxn.v[e] = yee(da.v[e], hx.v[e], db.v[e], ey1.v[e], ey0.v[e], cz, ezj1.v[e], ez.v[e], cy);
            hyn.v[e] = yee(da.v[e], hy.v[e], db.v[e], ez_ip, ez.v[e], cx, ex1.v[e], ex0.v[e], cz);
            hzn.v[e] = yee(da.v[e], hz.v[e], db.v[e], exj1.v[e], ex0.v[e], cy, ey_ip, ey0.v[e], cx);
        }
        // halo column x0-1 (lane 0 of the cell rows): new Hy, Hz
        float hyh = 0.f, hzh = 0.f;
        if (hcol && !warm) {
            hyh = yee(da_h, hy_h, db_h, ez.v[0], ez_h, cx, ex_h1, ex_h0, cz);
            hzh = yee(da_h, hz_h, db_h, ex_hj, ex_h0, cy, ey0.v[0], ey_h, cx);
        }

        if (!warm) {
            sHx[ty][lane] = hxn;
            sHz[ty][lane] = hzn;
        }
        __syncthreads();

        // ---- x-1 neighbours of new Hy, Hz ---------------------------------------------------
        float hy_p = __shfl_up_sync(FULL_MASK, hyn.v[V - 1], 1);
        float hz_p = __shfl_up_sync(FULL_MASK, hzn.v[V - 1], 1);
        if (lane == 0) { hy_p = hyh; hz_p = hzh; }

        if (!halo && jrow && xin) {
            if (!warm) {
                const Vec<V> hxj = sHx[ty - 1][lane];   // new Hx at j-1
                const Vec<V> hzj = sHz[ty - 1][lane];   // new Hz at j-1
                Vec<V> exn, eyn, ezn;
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const int x = i + e;
                    const float hy_im = e > 0 ? hyn.v[e - 1] : hy_p;
                    const float hz_im = e > 0 ? hzn.v[e - 1] : hz_p;
                    exn.v[e] = (j >= 1 && k >= 1)
                        ? yee(ca.v[e], ex0.v[e], cb.v[e], hzn.v[e], hzj.v[e], cy, hyn.v[e], hyp.v[e], cz)
                        : ex0.v[e];
                    eyn.v[e] = (x >= 1 && k >= 1)
                        ? yee(ca.v[e], ey0.v[e], cb.v[e], hxn.v[e], hxp.v[e], cz, hzn.v[e], hz_im, cx)
                        : ey0.v[e];
                    ezn.v[e] = (x >= 1 && j >= 1)
                        ? yee(ca.v[e], ez.v[e], cb.v[e], hyn.v[e], hy_im, cx, hxn.v[e], hxj.v[e], cy)
                        : ez.v[e];
                }
                if (src >= 0) {
                    const long long dsrc = src - off;
                    if (dsrc >= 0 && dsrc < V) {
#pragma unroll
                        for (int e = 0; e < V; ++e)
                            if (e == (int)dsrc) ezn.v[e] = __fadd_rn(ezn.v[e], srcv);
                    }
                }
                if (nout > 0) {
                    stv<V>(oHx + off, hxn, nout); stv<V>(oHy + off, hyn, nout); stv<V>(oHz + off, hzn, nout);
                    stv<V>(oEx + off, exn, nout); stv<V>(oEy + off, eyn, nout); stv<V>(oEz + off, ezn, nout);
                }
            }
            hxp = hxn;
            hyp = hyn;
            ex0 = ex1;
            ey0 = ey1;
        }
    }
    }   // tile loop
}

__global__ void k_advance(InstDesc *insts, int ninst, int nsteps, int flips)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= ninst) return;
    InstDesc &d = insts[q];
    const int n = min(nsteps, d.steps_left);
    if (n > 0) {
        d.step += n;
        d.steps_left -= n;
        d.par = (d.par + (flips < 0 ? n : flips)) & 1;
    }
}

int face_tile_cells(int by) { return 32 * (by + 1) * kFaceCellsPerThread; }

void plan_tiles(InstDesc &d, int by, int kc, int vec)
{
    const int kcc = (kc <= 0 || kc > d.nz) ? d.nz : kc;
    const int tx = 32 * vec;
    d.vec = vec;
    d.kc = kcc;
    d.tiles_x = (d.nx + tx - 1) / tx;
    d.tiles_y = (d.ny + by - 1) / by;
    d.tiles_z = (d.nz + kcc - 1) / kcc;
    const long long fc = (long long)d.ny * d.nz + (long long)d.nx * d.nz + (long long)d.nx * d.ny;
    const int per = face_tile_cells(by);
    d.face_tiles = (int)((fc + per - 1) / per);
}

void plan_tiles(InstDesc &d, int by, int kc) { plan_tiles(d, by, kc, 4); }

int balanced_depths(int nx, int ny, int nz, int by, int vec, int resident, int *out, int n)
{
    if (resident <= 0 || n <= 0 || by <= 0 || vec <= 0) return 0;
    const long long cols = (long long)((nx + 32 * vec - 1) / (32 * vec)) * ((ny + by - 1) / by);
    std::vector<std::pair<long long, int>> c;
    for (int tz = 1; tz <= nz; ++tz) {
        const int kc = (nz + tz - 1) / tz;
        if ((nz + kc - 1) / kc != tz) continue;   // same depth as a smaller tz
        if (kc < 4) break;
        const long long waves = (cols * tz + resident - 1) / resident;
        c.push_back({waves * (kc + (tz > 1 ? 1 : 0) + 2), kc >= nz ? 0 : kc});
    }
    std::stable_sort(c.begin(), c.end(),
                     [](const std::pair<long long, int> &a, const std::pair<long long, int> &b) { return a.first < b.first; });
    int k = 0;
    for (const auto &e : c) {
        if (k == n) break;
        out[k++] = e.second;
    }
    return k;
}

int leftover_depths(int nx, int ny, int nz, int by, int vec, int resident, int *out, int n)
{
    if (resident <= 0 || n <= 0 || by <= 0 || vec <= 0) return 0;
    const long long cols = (long long)((nx + 32 * vec - 1) / (32 * vec)) * ((ny + by - 1) / by);
    const long long layers = resident / cols, extra = resident - layers * cols;
    if (layers < 1 || extra < 1) return 0;
    const long long rounds = (cols + extra - 1) / extra;   // leftover tiles per extra CTA
    int k = 0;
    for (int kc = 4; kc < nz && k < n; ++kc) {
        const long long rest = nz - layers * kc;
        if (rest <= 0) break;
        if (rest >= kc) continue;   // a full further layer, not a leftover
        if (rounds * (rest + 2) <= kc + 1) out[k++] = kc;
    }
    return k;
}

template <int BY, int V>
static void launch_by_v(const InstDesc *d_insts, const int *d_tile0, int ninst, int total_tiles, int s_offset,
                        int g, cudaStream_t s)
{
    k_yee_step<BY, V><<<g, dim3(32, BY + 1), 0, s>>>(d_insts, d_tile0, ninst, s_offset, total_tiles);
}

int launch_yee_step_v(const InstDesc *d_insts, const int *d_tile0, int ninst, int total_tiles, int s_offset,
                      int by, int vec, int grid, cudaStream_t s)
{
    if (total_tiles <= 0) return PTK_OK;
    const int g = (grid <= 0 || grid > total_tiles) ? total_tiles : grid;
#define PTK_CASE(B, W)                                                                       \
    if (by == B && vec == W) {                                                               \
        launch_by_v<B, W>(d_insts, d_tile0, ninst, total_tiles, s_offset, g, s);             \
        PTK_CUDA_TRY(cudaGetLastError());                                                    \
        count_launches(1);                                                                   \
        return PTK_OK;                                                                       \
    }
    PTK_CASE(4, 1) PTK_CASE(4, 2) PTK_CASE(4, 4)
    PTK_CASE(8, 1) PTK_CASE(8, 2) PTK_CASE(8, 4)
    PTK_CASE(16, 1) PTK_CASE(16, 2) PTK_CASE(16, 4)
#undef PTK_CASE
    return set_error(PTK_ERR_INVALID, "tile rows must be 4, 8 or 16 and cells per thread 1, 2 or 4 (got %d, %d)",
                     by, vec);
}

int launch_yee_step_grid(const InstDesc *d_insts, const int *d_tile0, int ninst, int total_tiles,
                         int s_offset, int by, int grid, cudaStream_t s)
{
    return launch_yee_step_v(d_insts, d_tile0, ninst, total_tiles, s_offset, by, 4, grid, s);
}

int launch_yee_step(const InstDesc *d_insts, const int *d_tile0, int ninst, int total_tiles,
                    int s_offset, int by, cudaStream_t s)
{
    return launch_yee_step_v(d_insts, d_tile0, ninst, total_tiles, s_offset, by, 4, 0, s);
}

int yee_resident_ctas(int by, int vec)
{
    int per_sm = 0;
    cudaError_t e = cudaErrorInvalidValue;
#define PTK_OCC(B, W)                                                                               \
    if (by == B && vec == W)                                                                        \
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_yee_step<B, W>, 32 * (B + 1), 0);
    PTK_OCC(4, 1) PTK_OCC(4, 2) PTK_OCC(4, 4)
    PTK_OCC(8, 1) PTK_OCC(8, 2) PTK_OCC(8, 4)
    PTK_OCC(16, 1) PTK_OCC(16, 2) PTK_OCC(16, 4)
#undef PTK_OCC
    if (e != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return per_sm * sm_count();
}

int yee_resident_ctas(int by) { return yee_resident_ctas(by, 4); }

int launch_advance(InstDesc *d_insts, int ninst, int nsteps, cudaStream_t s, int flips)
{
    if (ninst <= 0) return PTK_OK;
    k_advance<<<(ninst + 127) / 128, 128, 0, s>>>(d_insts, ninst, nsteps, flips);
    PTK_CUDA_TRY(cudaGetLastError());
    count_launches(1);
    return PTK_OK;
}

// ---------------------------------------------------------------------------------------------
// Layout conversion.
// ---------------------------------------------------------------------------------------------
// Bound by memory: a warp moves four rows at a time, two loads a row in flight per lane.  Rows of a
// dense field start anywhere, so accesses are 32 lanes of one float.  One launch moves all the arrays
// (blockIdx.y).  256^3, six fields: packed in 132 us, 6.1 TB/s (a block per row, one load in flight and
// both buffers written in full took 512), unpacked in 121 us, 6.6 TB/s (514).
constexpr int kRowBatch = 4, kRowThreads = 256;

struct RowMove {
    const float *src[6];
    int *err;                  // UNPACK: where set, the fields become NaN; PACK: cleared (may be null)
    float *dst[6], *wall[6];   // wall: where nodes of the walls i = Nx, j = Ny, k = Nz go as well, or null
    int ex[6], ey[6], rows[6]; // dense extents
    int nx, ny, nz, pitch;
    long long plane;
};

enum { ROWS_PACK = 0, ROWS_UNPACK = 1, ROWS_COEF = 2 };

// PACK: dense field to padded nodes; UNPACK: back; COEF: per-cell array (Nx,Ny,Nz) to padded nodes
// (Nx+1,Ny+1,Nz+1), wall nodes take the nearest cell.
template <int MODE>
__global__ void __launch_bounds__(kRowThreads) k_rows(const RowMove A)
{
    const int f = blockIdx.y, lane = threadIdx.x & 31;
    const int ex = A.ex[f], ey = A.ey[f], rows = A.rows[f];
    const float *__restrict__ src = A.src[f];
    float *__restrict__ dst = A.dst[f];
    float *__restrict__ wall = A.wall[f];
    const bool bad = MODE == ROWS_UNPACK && A.err && *A.err;
    if (MODE == ROWS_PACK && A.err && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *A.err = 0;
    const int step = gridDim.x * (kRowThreads / 32) * kRowBatch;
    for (int r0 = (blockIdx.x * (kRowThreads / 32) + (threadIdx.x >> 5)) * kRowBatch; r0 < rows; r0 += step) {
        long long so[kRowBatch], to[kRowBatch];
        bool on[kRowBatch], edge[kRowBatch];
#pragma unroll
        for (int q = 0; q < kRowBatch; ++q) {
            const int r = r0 + q, k = r / ey, j = r - k * ey;
            on[q] = r < rows;
            edge[q] = j == A.ny || k == A.nz;
            const long long pad = (long long)A.pitch * j + A.plane * k, dense = (long long)r * ex;
            so[q] = MODE == ROWS_PACK ? dense
                    : MODE == ROWS_UNPACK ? pad : (long long)A.nx * (min(j, A.ny - 1) + (long long)A.ny * min(k, A.nz - 1));
            to[q] = MODE == ROWS_UNPACK ? dense : pad;
        }
        for (int i = lane; i < ex; i += 64) {
            const int i0 = MODE == ROWS_COEF ? min(i, A.nx - 1) : i, i1 = MODE == ROWS_COEF ? min(i + 32, A.nx - 1) : i + 32;
            float v[kRowBatch][2];
#pragma unroll
            for (int q = 0; q < kRowBatch; ++q) {
                if (on[q]) v[q][0] = src[so[q] + i0];
                if (on[q] && i + 32 < ex) v[q][1] = src[so[q] + i1];
            }
#pragma unroll
            for (int q = 0; q < kRowBatch; ++q)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int x = i + 32 * h;
                    if (!on[q] || x >= ex) continue;
                    dst[to[q] + x] = MODE == ROWS_UNPACK && bad ? __int_as_float(0x7fffffff) : v[q][h];
                    if (MODE == ROWS_PACK && wall && (edge[q] || x == A.nx)) wall[to[q] + x] = v[q][h];
                }
        }
    }
}

__global__ void k_fill(float *__restrict__ dst, long long n, float v)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x)
        dst[q] = v;
}

static dim3 rows_grid(int rows, int n)
{
    const int per = kRowThreads / 32 * kRowBatch;
    return dim3(std::max(1, std::min((rows + per - 1) / per, 8 * std::max(1, sm_count()))), n);
}

static RowMove row_move(const Layout &L)
{
    RowMove a{};
    a.nx = L.nx; a.ny = L.ny; a.nz = L.nz; a.pitch = L.pitch; a.plane = L.plane;
    return a;
}

int launch_pack_fields(const float *const src[], const Layout &L, float *const dst[], float *const wall[], int first, int n,
                       cudaStream_t s, int *clear)
{
    RowMove a = row_move(L);
    a.err = clear;
    int most = 1;
    for (int q = 0; q < n; ++q) {
        int ez;
        a.src[q] = src[first + q]; a.dst[q] = dst[first + q]; a.wall[q] = wall ? wall[first + q] : nullptr;
        field_extents(first + q, L.nx, L.ny, L.nz, &a.ex[q], &a.ey[q], &ez);
        a.rows[q] = a.ey[q] * ez;
        most = std::max(most, a.rows[q]);
    }
    k_rows<ROWS_PACK><<<rows_grid(most, n), kRowThreads, 0, s>>>(a);
    PTK_CUDA_TRY(cudaGetLastError());
    count_launches(1);
    return PTK_OK;
}

int launch_unpack_fields(const float *const src[], const Layout &L, float *const dst[], int first, int n, cudaStream_t s,
                         const int *err)
{
    RowMove a = row_move(L);
    a.err = const_cast<int *>(err);   // read only
    int most = 1;
    for (int q = 0; q < n; ++q) {
        int ez;
        a.src[q] = src[first + q]; a.dst[q] = dst[first + q];
        field_extents(first + q, L.nx, L.ny, L.nz, &a.ex[q], &a.ey[q], &ez);
        a.rows[q] = a.ey[q] * ez;
        most = std::max(most, a.rows[q]);
    }
    k_rows<ROWS_UNPACK><<<rows_grid(most, n), kRowThreads, 0, s>>>(a);
    PTK_CUDA_TRY(cudaGetLastError());
    count_launches(1);
    return PTK_OK;
}

int launch_pack_coefs(const float *const src[], const Layout &L, float *const dst[], int first, int n, cudaStream_t s)
{
    RowMove a = row_move(L);
    for (int q = 0; q < n; ++q) {
        a.src[q] = src[first + q]; a.dst[q] = dst[first + q];
        a.ex[q] = L.nx + 1; a.ey[q] = L.ny + 1; a.rows[q] = (L.ny + 1) * (L.nz + 1);
    }
    k_rows<ROWS_COEF><<<rows_grid((L.ny + 1) * (L.nz + 1), n), kRowThreads, 0, s>>>(a);
    PTK_CUDA_TRY(cudaGetLastError());
    count_launches(1);
    return PTK_OK;
}

int launch_fill(float *dst, long long n, float v, cudaStream_t s)
{
    if (n <= 0) return PTK_OK;
    long long blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    k_fill<<<(int)blocks, 256, 0, s>>>(dst, n, v);
    PTK_CUDA_TRY(cudaGetLastError());
    count_launches(1);
    return PTK_OK;
}

// ---------------------------------------------------------------------------------------------
// The reference's task kernels over dense arrays.  Bound by memory (L2 where the fields fit it): a warp
// takes 32 nodes of a row through kTaskPlanes planes with all their loads in flight, and a z neighbour
// is the next plane's own value.  Fields that would give fewer than two blocks per SM that way take a
// plane per warp.  Rows start anywhere, so accesses are single floats.  Per launch, against a thread
// per node in blocks of 128 along x, in a captured chain: 64x64x4 0.92 us (1.44), 45x64x50 1.35 (2.70),
// 200x150x100 8.3 (17.0), 256^3 47 (85); called one by one at 200x150x100 8.6 (19.6).
// ---------------------------------------------------------------------------------------------
constexpr int kTaskRows = 8, kTaskPlanes = 4;

static dim3 task_grid(int ex, int ey, int ez, int planes)
{
    return dim3((ex + 31) / 32, (ey + kTaskRows - 1) / kTaskRows, (ez + planes - 1) / planes);
}

// One field: out = a + c * ((p' - p) s1 - (q' - q) s2), where the differences of p and q run along
// directions DP and DQ (0 x, 1 y, 2 z): upwards for H (E false), downwards for E, whose wall nodes are
// copied.
struct FieldTask {
    const float *a, *p, *q;
    float *out;
    int ex, ey, ez;                  // extents of a and out
    int prow, qrow;                  // row lengths of p and q
    long long aplane, pplane, qplane;
    int nx, ny, nz;
    float c, s1, s2;
};

template <bool E, int DP, int DQ, int PL>
__global__ void __launch_bounds__(32 * kTaskRows) k_field_ref(const FieldTask T)
{
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * kTaskRows + threadIdx.y, k0 = blockIdx.z * PL;
    if (i >= T.ex || j >= T.ey) return;
    const int n = min(PL, T.ez - k0);
    const float *a = T.a + i + (long long)T.ex * j + T.aplane * k0;
    const float *p = T.p + i + (long long)T.prow * j + T.pplane * k0;
    const float *q = T.q + i + (long long)T.qrow * j + T.qplane * k0;
    float *out = T.out + i + (long long)T.ex * j + T.aplane * k0;
    constexpr int way = E ? -1 : 1;
    const long long dp = way * (DP == 0 ? 1LL : DP == 1 ? (long long)T.prow : T.pplane);
    const long long dq = way * (DQ == 0 ? 1LL : DQ == 1 ? (long long)T.qrow : T.qplane);
    // E: inside the walls in the two directions across the field's own
    const bool in = !E || (((DP != 0 && DQ != 0) || (i >= 1 && i <= T.nx - 1)) && ((DP != 1 && DQ != 1) || (j >= 1 && j <= T.ny - 1)));
    float av[PL], pn[PL], pf[PL], qn[PL], qf[PL];
    bool on[PL];
    chain_wait();
#pragma unroll
    for (int u = 0; u < PL; ++u) {
        const bool z = !E || (DP != 2 && DQ != 2) || (k0 + u >= 1 && k0 + u <= T.nz - 1);
        on[u] = u < n && in && z;
        if (u < n) av[u] = a[u * T.aplane];
        // the z neighbour of one plane is the node of another: loaded once
        const bool mine = u < n && in;
        if (on[u] || (mine && DP == 2 && !E && u > 0)) pn[u] = p[u * T.pplane];
        if (on[u] || (mine && DQ == 2 && !E && u > 0)) qn[u] = q[u * T.qplane];
        if (on[u] && (DP != 2 || (E && u == 0) || (E && !on[u > 0 ? u - 1 : 0]) || (!E && u + 1 >= n))) pf[u] = p[u * T.pplane + dp];
        if (on[u] && (DQ != 2 || (E && u == 0) || (E && !on[u > 0 ? u - 1 : 0]) || (!E && u + 1 >= n))) qf[u] = q[u * T.qplane + dq];
    }
#pragma unroll
    for (int u = 0; u < PL; ++u) {
        if (u >= n) break;
        float v = av[u];
        if (on[u]) {
            const int w = E ? (u > 0 ? u - 1 : 0) : (u + 1 < PL ? u + 1 : u);
            const bool other = E ? (u > 0 && on[w]) : u + 1 < n;
            const float pp = DP == 2 && other ? pn[w] : pf[u], qq = DQ == 2 && other ? qn[w] : qf[u];
            v = E ? yee_ref(v, T.c, pn[u], pp, T.s1, qn[u], qq, T.s2) : yee_ref(v, T.c, pp, pn[u], T.s1, qq, qn[u], T.s2);
        }
        out[u * T.aplane] = v;
    }
}

void field_extents(int f, int nx, int ny, int nz, int *ex, int *ey, int *ez)
{
    *ex = nx + ((f == PTK_HX || f == PTK_EY || f == PTK_EZ) ? 1 : 0);
    *ey = ny + ((f == PTK_HY || f == PTK_EX || f == PTK_EZ) ? 1 : 0);
    *ez = nz + ((f == PTK_HZ || f == PTK_EX || f == PTK_EY) ? 1 : 0);
}

template <int PL>
static cudaError_t field_task(int field, const FieldTask &t, cudaStream_t s)
{
    void (*const k[6])(const FieldTask) = {k_field_ref<false, 2, 1, PL>, k_field_ref<false, 0, 2, PL>, k_field_ref<false, 1, 0, PL>,
                                           k_field_ref<true, 1, 2, PL>,  k_field_ref<true, 2, 0, PL>,  k_field_ref<true, 0, 1, PL>};
    return launch_chained(k[field], task_grid(t.ex, t.ey, t.ez, PL), dim3(32, kTaskRows), 0, s, true, t);
}

int launch_field_ref(int field, const float *in0, const float *in1, const float *in2,
                     const ptk_fdtd_params &p, float *out, cudaStream_t s)
{
    // p and q of each field: which input, and which field's extents it has
    static const int pin[6] = {1, 2, 1, 2, 1, 2}, pf[6] = {PTK_EY, PTK_EZ, PTK_EX, PTK_HZ, PTK_HX, PTK_HY};
    static const int qf[6] = {PTK_EZ, PTK_EX, PTK_EY, PTK_HY, PTK_HZ, PTK_HX};
    const float sc[3] = {p.Cx, p.Cy, p.Cz};
    static const int dp[6] = {2, 0, 1, 1, 2, 0}, dq[6] = {1, 2, 0, 2, 0, 1};
    const float *in[3] = {in0, in1, in2};
    FieldTask t{};
    t.a = in0; t.p = in[pin[field]]; t.q = in[3 - pin[field]]; t.out = out;
    int ey, ez;
    field_extents(field, p.Nx, p.Ny, p.Nz, &t.ex, &t.ey, &t.ez);
    t.aplane = (long long)t.ex * t.ey;
    field_extents(pf[field], p.Nx, p.Ny, p.Nz, &t.prow, &ey, &ez);
    t.pplane = (long long)t.prow * ey;
    field_extents(qf[field], p.Nx, p.Ny, p.Nz, &t.qrow, &ey, &ez);
    t.qplane = (long long)t.qrow * ey;
    t.nx = p.Nx; t.ny = p.Ny; t.nz = p.Nz;
    t.c = field < 3 ? p.Dt / p.mu0 : p.Dt / p.eps0;
    t.s1 = sc[dp[field]]; t.s2 = sc[dq[field]];
    const dim3 grid = task_grid(t.ex, t.ey, t.ez, kTaskPlanes);
    const bool large = (long long)grid.x * grid.y * grid.z >= 2 * std::max(1, sm_count());
    PTK_CUDA_TRY(large ? field_task<kTaskPlanes>(field, t, s) : field_task<1>(field, t, s));
    count_launches(1);
    return PTK_OK;
}

}  // namespace ptk
