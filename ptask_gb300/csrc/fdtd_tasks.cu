// fdtd_tasks.cu -- the half-step task kernels over dense reference-layout blocks (those of the cyclic
// FDTD graph with per-cell coefficients, in place, and the scalar ones into new blocks), plus CUDA-graph
// capture entry points used by the PTask scheduler.
//
// Both half steps are safe in place: a new H value depends only on the old H value of the same
// node and on E; a new E value only on the old E value of the same node and on H.  The cyclic graph
// therefore circulates one datablock per field through in-out ports, with no allocation per step
// (the reference allocates a new output block per task dispatch, OutputPort.cpp:536).
#include "fdtd_chain.cuh"
#include "ptk_internal.h"

namespace ptk {

__device__ __forceinline__ float yee_c(float d, float h, float c, float a1, float a0, float s1, float b1,
                                       float b0, float s2)
{
    const float curl = __fsub_rn(__fmul_rn(__fsub_rn(a1, a0), s1), __fmul_rn(__fsub_rn(b1, b0), s2));
    return __fadd_rn(__fmul_rn(d, h), __fmul_rn(c, curl));
}

// Bound by memory: a warp takes 32 nodes of a row through kPlanes planes with all their loads in
// flight; Ex, Ey (H step) and Hx, Hy (E step) of one plane serve the next as its z neighbours.
constexpr int kRows = 8, kPlanes = 2;

// H' = Da*H + Db*curl(E) with per-cell Da, Db (COEF), or H + c*curl(E); out may be the input.
struct HalfStep {
    const float *h[3], *e[3];
    float *out[3];
    const float *d, *c;           // COEF: Da, Db (or Ca, Cb)
    int nx, ny, nz;
    float cs, cx, cy, cz;         // !COEF: the scalar coefficient
    long long src;                // COEF, E: dense Ez index of the source (-1 none), its waveform and step counter
    const float *wave;
    int nwave;
    int *counter;
};

template <bool COEF>
__device__ __forceinline__ float upd(float d, float h, float c, float a1, float a0, float s1, float b1, float b0, float s2)
{
    if constexpr (COEF) return yee_c(d, h, c, a1, a0, s1, b1, b0, s2);
    const float curl = __fsub_rn(__fmul_rn(__fsub_rn(a1, a0), s1), __fmul_rn(__fsub_rn(b1, b0), s2));
    return __fadd_rn(h, __fmul_rn(c, curl));
}

template <bool COEF>
__global__ void __launch_bounds__(32 * kRows) k_h_step(const HalfStep T)
{
    const int nx = T.nx, ny = T.ny, nz = T.nz;
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * kRows + threadIdx.y, k0 = blockIdx.z * kPlanes;
    if (i > nx || j > ny) return;
    const bool xi = i < nx, yi = j < ny;
    // offsets of node (i, j, k0) in each array's own extents, and their planes
    const long long pHx = (long long)(nx + 1) * ny, pHy = (long long)nx * (ny + 1), pHz = (long long)nx * ny;
    const long long pEx = pHy, pEy = pHx, pEz = (long long)(nx + 1) * (ny + 1);
    const long long oHx = i + (long long)(nx + 1) * j + pHx * k0, oHy = i + (long long)nx * j + pHy * k0, oHz = i + (long long)nx * j + pHz * k0;
    const long long oEx = oHy, oEy = oHx, oEz = i + (long long)(nx + 1) * j + pEz * k0;
    const float *Hx = T.h[0], *Hy = T.h[1], *Hz = T.h[2], *Ex = T.e[0], *Ey = T.e[1], *Ez = T.e[2];
    chain_wait();
    float hx[kPlanes], hy[kPlanes], hz[kPlanes], ex[kPlanes + 1], ey[kPlanes + 1], ez[kPlanes];
    float exj[kPlanes], ezj[kPlanes], eyi[kPlanes], ezi[kPlanes], d[kPlanes], c[kPlanes];
#pragma unroll
    for (int u = 0; u <= kPlanes; ++u) {
        if (k0 + u > nz) continue;
        if (xi) ex[u] = Ex[oEx + pEx * u];
        if (yi) ey[u] = Ey[oEy + pEy * u];
    }
#pragma unroll
    for (int u = 0; u < kPlanes; ++u) {
        const int k = k0 + u;
        if (k > nz) continue;
        const bool zi = k < nz;
        if (yi && zi) { hx[u] = Hx[oHx + pHx * u]; ezj[u] = Ez[oEz + pEz * u + nx + 1]; }
        if (xi && zi) { hy[u] = Hy[oHy + pHy * u]; ezi[u] = Ez[oEz + pEz * u + 1]; }
        if (zi) ez[u] = Ez[oEz + pEz * u];
        if (xi && yi) {
            hz[u] = Hz[oHz + pHz * u];
            exj[u] = Ex[oEx + pEx * u + nx];
            eyi[u] = Ey[oEy + pEy * u + 1];
        }
        d[u] = 1.f;
        c[u] = T.cs;
        if constexpr (COEF) {   // wall nodes take the nearest cell
            const long long cell = min(i, nx - 1) + (long long)nx * min(j, ny - 1) + (long long)nx * ny * min(k, nz - 1);
            d[u] = T.d[cell];
            c[u] = T.c[cell];
        }
    }
#pragma unroll
    for (int u = 0; u < kPlanes; ++u) {
        const int k = k0 + u;
        if (k > nz) continue;
        const bool zi = k < nz;
        if (yi && zi) T.out[0][oHx + pHx * u] = upd<COEF>(d[u], hx[u], c[u], ey[u + 1], ey[u], T.cz, ezj[u], ez[u], T.cy);
        if (xi && zi) T.out[1][oHy + pHy * u] = upd<COEF>(d[u], hy[u], c[u], ezi[u], ez[u], T.cx, ex[u + 1], ex[u], T.cz);
        if (xi && yi) T.out[2][oHz + pHz * u] = upd<COEF>(d[u], hz[u], c[u], exj[u], ex[u], T.cy, eyi[u], ey[u], T.cx);
    }
}

// E' = Ca*E + Cb*curl(H') (COEF, in place: wall nodes stay) or E + c*curl(H') (wall nodes copied).
template <bool COEF>
__global__ void __launch_bounds__(32 * kRows) k_e_step(const HalfStep T)
{
    const int nx = T.nx, ny = T.ny, nz = T.nz;
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * kRows + threadIdx.y, k0 = blockIdx.z * kPlanes;
    if (i > nx || j > ny) return;
    const bool xi = i < nx, yi = j < ny;                             // nodes of Ex, Ez and of Ey, Ez in x and y
    const bool xin = i >= 1 && i <= nx - 1, yin = j >= 1 && j <= ny - 1;   // off the walls
    const long long pHx = (long long)(nx + 1) * ny, pHy = (long long)nx * (ny + 1), pHz = (long long)nx * ny;
    const long long pEx = pHy, pEy = pHx, pEz = (long long)(nx + 1) * (ny + 1);
    const long long oHx = i + (long long)(nx + 1) * j + pHx * k0, oHy = i + (long long)nx * j + pHy * k0, oHz = i + (long long)nx * j + pHz * k0;
    const long long oEx = oHy, oEy = oHx, oEz = i + (long long)(nx + 1) * j + pEz * k0;
    const float *Hx = T.h[0], *Hy = T.h[1], *Hz = T.h[2], *Ex = T.e[0], *Ey = T.e[1], *Ez = T.e[2];
    chain_wait();
    float ex[kPlanes], ey[kPlanes], ez[kPlanes], hx[kPlanes + 1], hy[kPlanes + 1], hz[kPlanes];   // hx[u]: plane k0 + u - 1
    float hxj[kPlanes], hzj[kPlanes], hyi[kPlanes], hzi[kPlanes], d[kPlanes], c[kPlanes];
#pragma unroll
    for (int u = 0; u <= kPlanes; ++u) {
        const int k = k0 + u - 1;
        if (k < 0 || k >= nz) continue;
        if (yi && (xin || yin)) hx[u] = Hx[oHx + pHx * (u - 1)];
        if (xi && (xin || yin)) hy[u] = Hy[oHy + pHy * (u - 1)];
    }
#pragma unroll
    for (int u = 0; u < kPlanes; ++u) {
        const int k = k0 + u;
        if (k > nz) continue;
        const bool zi = k < nz, zin = k >= 1 && zi;
        if (xi && (!COEF || (yin && zin))) ex[u] = Ex[oEx + pEx * u];
        if (yi && (!COEF || (xin && zin))) ey[u] = Ey[oEy + pEy * u];
        if (zi && (!COEF || (xin && yin))) ez[u] = Ez[oEz + pEz * u];
        if (xi && yi && zin) hz[u] = Hz[oHz + pHz * u];
        if (xi && yin && zin) hzj[u] = Hz[oHz + pHz * u - nx];
        if (xin && yi && zin) hzi[u] = Hz[oHz + pHz * u - 1];
        if (xin && yin && zi) {
            hxj[u] = Hx[oHx + pHx * u - (nx + 1)];
            hyi[u] = Hy[oHy + pHy * u - 1];
        }
        d[u] = 1.f;
        c[u] = T.cs;
        if constexpr (COEF)
            if (xi && yi && zi) {
                const long long cell = oHz + pHz * u;
                d[u] = T.d[cell];
                c[u] = T.c[cell];
            }
    }
#pragma unroll
    for (int u = 0; u < kPlanes; ++u) {
        const int k = k0 + u;
        if (k > nz) continue;
        const bool zi = k < nz, zin = k >= 1 && zi;
        if (xi && yin && zin) T.out[0][oEx + pEx * u] = upd<COEF>(d[u], ex[u], c[u], hz[u], hzj[u], T.cy, hy[u + 1], hy[u], T.cz);
        else if (!COEF && xi) T.out[0][oEx + pEx * u] = ex[u];
        if (xin && yi && zin) T.out[1][oEy + pEy * u] = upd<COEF>(d[u], ey[u], c[u], hx[u + 1], hx[u], T.cz, hz[u], hzi[u], T.cx);
        else if (!COEF && yi) T.out[1][oEy + pEy * u] = ey[u];
        if (xin && yin && zi) {
            float v = upd<COEF>(d[u], ez[u], c[u], hy[u + 1], hyi[u], T.cx, hx[u + 1], hxj[u], T.cy);
            if (COEF && oEz + pEz * u == T.src && T.counter) {
                // Only this thread touches the counter, so the read-modify-write needs no atomics.
                const int n = *T.counter;
                if (n < T.nwave) v = __fadd_rn(v, T.wave[n]);
                *T.counter = n + 1;
            }
            T.out[2][oEz + pEz * u] = v;
        } else if (!COEF && zi) {
            T.out[2][oEz + pEz * u] = ez[u];
        }
    }
}

static HalfStep half_step(const float *const h[3], const float *const e[3], float *const out[3], const ptk_fdtd_params &p)
{
    HalfStep t{};
    for (int q = 0; q < 3; ++q) {
        t.h[q] = h[q];
        t.e[q] = e[q];
        t.out[q] = out[q];
    }
    t.nx = p.Nx; t.ny = p.Ny; t.nz = p.Nz;
    t.cx = p.Cx; t.cy = p.Cy; t.cz = p.Cz;
    t.src = -1;
    return t;
}

static dim3 half_grid(const HalfStep &t)
{
    return dim3(t.nx / 32 + 1, t.ny / kRows + 1, t.nz / kPlanes + 1);
}

int launch_h_half(const float *const in[6], float *const out[3], const ptk_fdtd_params &p, cudaStream_t s)
{
    HalfStep t = half_step(in, in + 3, out, p);
    t.cs = p.Dt / p.mu0;
    PTK_CUDA_TRY(launch_chained(k_h_step<false>, half_grid(t), dim3(32, kRows), 0, s, true, t));
    count_launches(1);
    return PTK_OK;
}

int launch_e_half(const float *const e_in[3], const float *const h_new[3], float *const out[3], const ptk_fdtd_params &p,
                  cudaStream_t s)
{
    HalfStep t = half_step(h_new, e_in, out, p);
    t.cs = p.Dt / p.eps0;
    PTK_CUDA_TRY(launch_chained(k_e_step<false>, half_grid(t), dim3(32, kRows), 0, s, true, t));
    count_launches(1);
    return PTK_OK;
}

}  // namespace ptk

using namespace ptk;

static inline cudaStream_t S(void *s) { return s ? (cudaStream_t)s : default_stream(); }

extern "C" {

int ptk_launch_h_step_coef(float *const h[3], const float *const e[3], const float *Da, const float *Db,
                           const ptk_fdtd_params *p, void *stream)
{
    PTK_CHECK_ARG(h && e && Da && Db && p, "NULL argument");
    PTK_CHECK_ARG(p->Nx >= 1 && p->Ny >= 1 && p->Nz >= 1, "bad grid");
    int rc = ensure_init();
    if (rc) return rc;
    HalfStep t = half_step(h, e, h, *p);
    t.d = Da;
    t.c = Db;
    PTK_CUDA_TRY(launch_chained(k_h_step<true>, half_grid(t), dim3(32, kRows), 0, S(stream), true, t));
    count_launches(1);
    return PTK_OK;
}

int ptk_launch_e_step_coef(float *const e[3], const float *const h[3], const float *Ca, const float *Cb,
                           const ptk_fdtd_params *p, int si, int sj, int sk, const float *wave, int nwave,
                           int *step_counter, void *stream)
{
    PTK_CHECK_ARG(e && h && Ca && Cb && p, "NULL argument");
    PTK_CHECK_ARG(p->Nx >= 1 && p->Ny >= 1 && p->Nz >= 1, "bad grid");
    int rc = ensure_init();
    if (rc) return rc;
    long long src = -1;
    if (wave && nwave > 0 && step_counter) {
        PTK_CHECK_ARG(si >= 1 && si < p->Nx && sj >= 1 && sj < p->Ny && sk >= 0 && sk < p->Nz,
                      "source node (%d,%d,%d) must be an interior Ez node", si, sj, sk);
        src = (long long)si + (long long)(p->Nx + 1) * sj + (long long)(p->Nx + 1) * (p->Ny + 1) * sk;
    }
    HalfStep t = half_step(h, e, e, *p);
    t.d = Ca;
    t.c = Cb;
    t.src = src;
    t.wave = wave;
    t.nwave = nwave;
    t.counter = src >= 0 ? step_counter : nullptr;
    PTK_CUDA_TRY(launch_chained(k_e_step<true>, half_grid(t), dim3(32, kRows), 0, S(stream), true, t));
    count_launches(1);
    return PTK_OK;
}

int ptk_capture_begin(void *stream)
{
    PTK_CHECK_ARG(stream, "capture needs an explicit stream");
    PTK_CUDA_TRY(cudaStreamBeginCapture((cudaStream_t)stream, cudaStreamCaptureModeThreadLocal));
    set_capturing(true);
    return PTK_OK;
}

int ptk_capture_end(void *stream, void **graph_exec)
{
    PTK_CHECK_ARG(stream && graph_exec, "NULL argument");
    set_capturing(false);
    cudaGraph_t g = nullptr;
    PTK_CUDA_TRY(cudaStreamEndCapture((cudaStream_t)stream, &g));
    cudaGraphExec_t ex = nullptr;
    cudaError_t e = cudaGraphInstantiate(&ex, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return set_error(PTK_ERR_CUDA, "graph instantiate: %s", cudaGetErrorString(e));
    *graph_exec = ex;
    return PTK_OK;
}

int ptk_graph_exec_launch(void *graph_exec, void *stream, long long kernel_nodes)
{
    PTK_CHECK_ARG(graph_exec, "NULL graph");
    PTK_CUDA_TRY(cudaGraphLaunch((cudaGraphExec_t)graph_exec, S(stream)));
    count_graph_launch(kernel_nodes);
    return PTK_OK;
}

int ptk_graph_exec_destroy(void *graph_exec)
{
    if (!graph_exec) return PTK_OK;
    PTK_CUDA_TRY(cudaGraphExecDestroy((cudaGraphExec_t)graph_exec));
    return PTK_OK;
}

}  // extern "C"
