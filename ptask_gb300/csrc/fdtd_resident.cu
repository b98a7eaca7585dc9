// fdtd_resident.cu -- a whole run of time steps in one launch, for grids whose fields fit on chip.
//
// The step kernels read and write every field from global memory once per step and meet at a kernel
// boundary.  On grids of up to about 0.9 million cells that boundary (launch, pipeline fill, drain)
// costs more than the step.  Here the grid is cut into bricks, one per SM: Nx x by x bz cells, whole
// rows in x, whose six fields stay in shared memory for the whole run.  Per step: H pass, barrier, E
// pass, barrier, ghost exchange, barrier.  A thread takes four x cells of a row through consecutive
// planes, keeping the values that the next plane shares; x neighbours come from warp shuffles.
//
// One exchange per step: a brick computes the H rows just below it (j = y0-1 and k = z0-1) itself,
// from ghost rows of E on both sides, so only E rows travel (to the four face neighbours and two
// diagonal ones).  A ghost value travels with a sequence number in the same 64-bit word, so a reader
// polls the data itself: no fence, no separate flag, one trip through L2.  Two slots by step parity:
// a brick writes a slot again two steps later, after its neighbour's rows of the step between have
// arrived, i.e. after that neighbour has consumed the slot.  Sequence numbers continue from launch
// to launch, counted by the host, so the buffer is cleared only when it is made, and what a launch that gave
// up has left in it is never taken for a later one's.
//
// The bricks wait on one another, so the launch is cooperative (all bricks resident at once) and
// every wait is bounded: on expiry the error word is raised and the launch ends with invalid fields,
// which the host reports as PTK_ERR_TIMEOUT.  Where they cannot all be resident (a stream or context with fewer
// SMs than the device) the launch is refused and its callers take a launch per step.
//
// Arithmetic is that of the step kernels, operation for operation.  With Ca = Da = 1 the products
// Ca*E and Da*H are the factors themselves, bit for bit, and are left out (COEF_SIMPLE).
#include "ptk_internal.h"

namespace ptk {

namespace {

constexpr unsigned long long kWaitNs = 1000000000ull;   // a wait gives up after 1 s of global time
constexpr int kWaitPolls = 1 << 22;                     // and after this many polls in any case

__device__ __forceinline__ unsigned long long clock_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned long long with_seq(float v, unsigned seq)
{
    return (unsigned long long)__float_as_uint(v) | ((unsigned long long)seq << 32);
}

// A ghost unit is four floats, each in the low half of a 64-bit word whose high half is the sequence
// number of the step it belongs to; 64-bit words are written and read whole.  The two 16-byte halves
// of a unit lie `half` apart, so that a warp's access to either covers whole sectors.
__device__ __forceinline__ void send_unit(ulonglong2 *dst, int half, float4 v, unsigned seq)
{
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(dst), "l"(with_seq(v.x, seq)), "l"(with_seq(v.y, seq))
                 : "memory");
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(dst + half), "l"(with_seq(v.z, seq)),
                 "l"(with_seq(v.w, seq))
                 : "memory");
}

__device__ __forceinline__ ulonglong2 load_pair(const ulonglong2 *src)
{
    ulonglong2 r;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(r.x), "=l"(r.y) : "l"(src) : "memory");
    return r;
}

__device__ __forceinline__ bool arrived(ulonglong2 a, ulonglong2 b, unsigned seq)
{
    return (unsigned)(a.x >> 32) == seq && (unsigned)(a.y >> 32) == seq && (unsigned)(b.x >> 32) == seq &&
           (unsigned)(b.y >> 32) == seq;
}

__device__ __forceinline__ float4 values(ulonglong2 a, ulonglong2 b)
{
    return make_float4(__uint_as_float((unsigned)a.x), __uint_as_float((unsigned)a.y), __uint_as_float((unsigned)b.x),
                       __uint_as_float((unsigned)b.y));
}

// d*h + c*((a1-a0)*s1 - (b1-b0)*s2), every operation rounded separately; D1: d is 1, d*h is h.
template <bool D1>
__device__ __forceinline__ float upd(float d, float h, float c, float a1, float a0, float s1, float b1, float b0, float s2)
{
    const float curl = __fsub_rn(__fmul_rn(__fsub_rn(a1, a0), s1), __fmul_rn(__fsub_rn(b1, b0), s2));
    return __fadd_rn(D1 ? h : __fmul_rn(d, h), __fmul_rn(c, curl));
}

__device__ __forceinline__ float4 ldg4(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }

// Shared memory by byte offset: a thread's accesses are one offset register, a uniform array base and
// an immediate.
__device__ __forceinline__ float4 lds4(const char *sm, int o) { return *reinterpret_cast<const float4 *>(sm + o); }
__device__ __forceinline__ void sts4(char *sm, int o, float4 v) { *reinterpret_cast<float4 *>(sm + o) = v; }

// v = the float at byte offset o where `take` is set (predicated: no branch).
__device__ __forceinline__ void lds_if(float &v, uint32_t sm_addr, int o, bool take)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t@p ld.shared.f32 %0, [%1];\n\t}"
                 : "+f"(v)
                 : "r"(sm_addr + o), "r"((int)take)
                 : "memory");
}

// Rows of the six fields in shared memory, in float4 slots, lwp slots a row (the last one holds the
// wall node i = Nx).  Row (y, z) is relative to the brick: E rows run from -1 to by, H rows from -1 to
// by - 1 (the rows at -1 are ghosts of E and the H rows that the brick computes below itself), so
// that the three E (and the three H) arrays have the same strides.
struct Rows {
    int base[6];   // first slot
    int total;
};

__host__ __device__ inline int rows_y(int by, int f) { return f < 3 ? by + 1 : by + 2; }
__host__ __device__ inline int below_z(int f) { return f == 2 ? 0 : 1; }   // Hz has no plane at z = -1

__host__ __device__ inline Rows rows_of(int by, int bz, int lwp)
{
    Rows r;
    int o = 0;
    for (int f = 0; f < 6; ++f) {
        r.base[f] = o;
        o += rows_y(by, f) * (bz + below_z(f) + (f == 3 || f == 4 ? 1 : 0)) * lwp;   // Ex, Ey(bz)
    }
    r.total = o;
    return r;
}

__host__ __device__ inline int row_slot(const Rows &R, int by, int lwp, int f, int y, int z)
{
    return R.base[f] + ((z + below_z(f)) * rows_y(by, f) + y + 1) * lwp;
}

// Ghost row g of a brick, in the order of its exchange slots: below in y Ex, Ey, Ez(-1, z); above
// Ex, Ez(byv, z); below in z Ex, Ey, Ez(y, -1); above Ex, Ey(y, bzv); then Ey(-1, bzv) and Ez(byv, -1).
// It is row (y, z) of field f (f < 0: the brick has no such row); sent: a neighbour sends it every
// step (otherwise it is a wall).  The same row of the neighbour on the other side, brick (ty, tz) on,
// is what this brick sends there: its own row (sy, sz) of that field (sf < 0: no such neighbour).
struct GhostRow {
    int f = -1, y = 0, z = 0, sf = -1, sy = 0, sz = 0, ty = 0, tz = 0;
    bool sent = false;
};

__host__ __device__ inline int ghost_rows(int by, int bz) { return 5 * bz + 5 * by + 2; }

__host__ __device__ inline GhostRow ghost_row(int g, int by, int bz, int byv, int bzv, bool ylo, bool yhi, bool zlo,
                                              bool zhi)
{
    GhostRow r;
    if (g < 5 * bz) {                        // rows across y
        const bool lo = g < 3 * bz;
        const int q = lo ? g : g - 3 * bz, z = q % bz, comp = q / bz, f = lo ? 3 + comp : 3 + 2 * comp;
        if (z >= bzv) return r;
        r.y = lo ? -1 : byv; r.z = z; r.sz = z;
        if (lo ? ylo : true) { r.f = f; r.sent = lo ? true : yhi; }
        if (lo ? yhi : ylo) { r.sf = f; r.sy = lo ? byv - 1 : 0; r.ty = lo ? 1 : -1; }
    } else if (g < 5 * bz + 5 * by) {        // rows across z
        const bool lo = g < 5 * bz + 3 * by;
        const int q = lo ? g - 5 * bz : g - 5 * bz - 3 * by, y = q % by, f = 3 + q / by;
        if (y >= byv) return r;
        r.y = y; r.z = lo ? -1 : bzv; r.sy = y;
        if (lo ? zlo : true) { r.f = f; r.sent = lo ? true : zhi; }
        if (lo ? zhi : zlo) { r.sf = f; r.sz = lo ? bzv - 1 : 0; r.tz = lo ? 1 : -1; }
    } else if (g == 5 * bz + 5 * by) {       // Ey(-1, bzv)
        r.y = -1; r.z = bzv;
        if (ylo) { r.f = 4; r.sent = zhi; }
        if (yhi && zlo) { r.sf = 4; r.sy = byv - 1; r.ty = 1; r.tz = -1; }
    } else {                                 // Ez(byv, -1)
        r.y = byv; r.z = -1;
        if (zlo) { r.f = 5; r.sent = yhi; }
        if (ylo && zhi) { r.sf = 5; r.sz = bzv - 1; r.ty = -1; r.tz = 1; }
    }
    return r;
}

// A unit of the H rows that a brick computes below itself: its slots (below in y: Hx, Hz from Ex,
// Ez, Ey and Ex at j+1; below in z: Hx, Hy and Ex at k+1).
struct __align__(16) BelowUnit {
    unsigned short hx, h2, ex, ez, ey, eyk, exn, iny;
};

// CTAs have up to 384 threads (168 registers each) with four or six ghost units a thread, or up to 512
// (128 registers) with five.  More threads spill: 768 ran 96^3 at 6.9 us per step against 5.6.
constexpr int kThreads = 512, kThreadsLow = 384, kMinThreads = 64;
constexpr int kMaxItems = 6;
constexpr size_t kSmem = 232448;    // shared memory of a CTA

// An exchange slot holds the first halves of its units, then the second ones.
__host__ __device__ inline int slot_half(int units) { return (units + 1) & ~1; }

size_t shared_bytes(const ResidentPlan &p)
{
    return sizeof(float4) * (size_t)rows_of(p.by, p.bz, p.lwp).total + sizeof(BelowUnit) * (size_t)(p.by + p.bz) * p.lw + 16;
}

}  // namespace

// What bounds it: on small grids the exchange (one trip through L2 per step) and the latency of the
// passes; at 96^3 shared-memory bandwidth, 22 accesses of 16 bytes per unit and step.
template <int COEF, int kMaxT, int kItems>
__global__ void __launch_bounds__(kMaxT, 1) k_yee_resident(const ResidentArgs A)
{
    extern __shared__ __align__(16) char sm[];
    constexpr bool D1 = COEF == COEF_SIMPLE;
    const int lw = A.lw, lwp = A.lwp, by = A.by, bz = A.bz, half = A.half, T = A.threads;
    BelowUnit *below = reinterpret_cast<BelowUnit *>(sm + A.below);
    volatile int *sfail = reinterpret_cast<int *>(sm + A.fail);
    const uint32_t sma = (uint32_t)__cvta_generic_to_shared(sm);

    const int tid = threadIdx.x, lane = tid & 31;
    const int cta = blockIdx.x, yb = cta % A.nby, zb = cta / A.nby;
    const int y0 = yb * by, z0 = zb * bz;
    const int byv = min(by, A.ny - y0), bzv = min(bz, A.nz - z0);
    const bool ylo = yb > 0, yhi = yb + 1 < A.nby, zlo = zb > 0, zhi = zb + 1 < A.nbz;
    const int nx = A.nx, pitch = A.pitch;
    const long long plane = A.plane;
    const float cx = A.cx, cy = A.cy, cz = A.cz;

    // ---- setup: every row's values, the units below the brick, this thread's share of the exchange -----
    const Rows R = rows_of(by, bz, lwp);
    const int NR = ghost_rows(by, bz);
    if (tid == 0) *sfail = 0;
#pragma unroll 1
    for (int f = 0; f < 6; ++f) {
        const int ry = rows_y(by, f), n = (f < 5 ? R.base[f + 1] : R.total) - R.base[f];
#pragma unroll 2
        for (int q = tid; q < n; q += T) {
            const int row = q / lwp, x = q - row * lwp;
            const int j = y0 + row % ry - 1, k = z0 + row / ry - below_z(f);
            sts4(sm, 16 * (R.base[f] + q), j >= 0 && k >= 0 && j <= A.ny && k <= A.nz
                                               ? ldg4(A.in[f] + 4 * x + (long long)pitch * j + plane * k)
                                               : make_float4(0.f, 0.f, 0.f, 0.f));
        }
    }
    const int nhy = ylo ? bzv : 0, nhz = zlo ? byv : 0, nbelow = (nhy + nhz) * lw;
#pragma unroll 1
    for (int q = tid; q < nbelow; q += T) {
        const int h = q / lw, x = q - h * lw, iny = h < nhy;
        const int y = iny ? -1 : h - nhy, z = iny ? h : -1;
        BelowUnit w;
        w.hx = row_slot(R, by, lwp, 0, y, z) + x;
        w.h2 = row_slot(R, by, lwp, iny ? 2 : 1, y, z) + x;
        w.ex = row_slot(R, by, lwp, 3, y, z) + x;
        w.ey = row_slot(R, by, lwp, 4, y, z) + x;
        w.ez = row_slot(R, by, lwp, 5, y, z) + x;
        w.eyk = row_slot(R, by, lwp, 4, y, z + 1) + x;
        w.exn = row_slot(R, by, lwp, 3, iny ? y + 1 : y, iny ? z : z + 1) + x;
        w.iny = iny;
        below[q] = w;
    }
    // ghost unit tid + b * T of the brick's list: what is sent from which offset to which unit of the
    // buffer, and where the received one goes (-1: nothing)
    int xsrc[kItems], xto[kItems], xdst[kItems];
#pragma unroll
    for (int b = 0; b < kItems; ++b) {
        const int q = tid + b * T, g = q / lw, x = q - g * lw;
        xto[b] = xdst[b] = -1;
        xsrc[b] = 0;
        if (g < NR) {
            const GhostRow r = ghost_row(g, by, bz, byv, bzv, ylo, yhi, zlo, zhi);
            if (r.sent) xdst[b] = 16 * (row_slot(R, by, lwp, r.f, r.y, r.z) + x);
            if (r.sf >= 0) {
                xsrc[b] = 16 * (row_slot(R, by, lwp, r.sf, r.sy, r.sz) + x);
                xto[b] = 4 * (cta + r.ty + r.tz * A.nby) * half + g * lw + x;
            }
        }
    }

    // ---- this thread's column: x unit lx, row y, planes zc .. zc + nu - 1 of the brick ----------------
    const int lx = tid % lw, c = tid / (lw * by), y = tid / lw - c * by, zc = c * A.kz, i = 4 * lx;
    const int nu = y < byv ? max(0, min(A.kz, bzv - zc)) : 0;
    const int nmax = __reduce_max_sync(0xffffffffu, nu);    // planes of the warp: shuffles need every lane
    const long long off0 = i + (long long)pitch * (y0 + y) + plane * (z0 + zc);
    // byte offsets: bases of the arrays, strides, and the column's first unit in an E and in an H array
    const int bHx = A.base[0], bHy = A.base[1], bHz = A.base[2], bEx = A.base[3], bEy = A.base[4], bEz = A.base[5];
    const int rs = A.row, pE = A.plane_e, pH = A.plane_h;   // one row, one plane on
    const int ys = nu > 0 ? y : 0, zs = nu > 0 ? zc : 0;   // threads without cells read a row of the brick
    const int oE0 = (zs + 1) * pE + (ys + 1) * rs + 16 * lx, oH0 = (zs + 1) * pH + (ys + 1) * rs + 16 * lx;
    const bool last = lane == 31 || lx == lw - 1;       // x+1 is not the next lane's
    const bool first = lane == 0 && lx > 0;             // x-1 is not the lane before's
    const bool in0 = lx > 0 && i < nx, in1 = i + 1 < nx, in2 = i + 2 < nx, in3 = i + 3 < nx;   // 0 < x < Nx
    const bool j1 = y0 + ys >= 1;
    int src_z = -1, src_e = 0;                          // the source's plane of the column and cell of the unit
    if (A.src >= 0) {
        const long long d = A.src - off0, dz = d >= 0 ? d / plane : -1, e = d - dz * plane;
        if (d >= 0 && dz < nu && e < 4) { src_z = (int)dz; src_e = (int)e; }
    }
    const float dbu = A.db;   // COEF_SIMPLE: the one Db
    const int qb = min(T - 1 - tid, (by + bz) * lw - 1);

    unsigned seq = A.seq;
    __syncthreads();

    for (int step = 0; step < A.steps; ++step) {
        ++seq;
        // ================= H pass =================
        BelowUnit w = below[qb];   // qb < room of the list for every thread
        {
            int oE = oE0, oH = oH0;
            float4 X = lds4(sm, bEx + oE), Y = lds4(sm, bEy + oE);
#pragma unroll 2
            for (int u = 0; u < nmax; ++u) {
                float4 D = make_float4(1.f, 1.f, 1.f, 1.f), C = make_float4(dbu, dbu, dbu, dbu);
                if (COEF == COEF_DENSE && u < nu) {
                    D = ldg4(A.coef[2] + off0 + plane * u);
                    C = ldg4(A.coef[3] + off0 + plane * u);
                }
                const float4 Z = lds4(sm, bEz + oE);
                const float4 exj = lds4(sm, bEx + oE + rs), ezj = lds4(sm, bEz + oE + rs);
                const float4 exk = lds4(sm, bEx + oE + pE), eyk = lds4(sm, bEy + oE + pE);
                float4 hx = lds4(sm, bHx + oH), hy = lds4(sm, bHy + oH), hz = lds4(sm, bHz + oH);
                float ezn = __shfl_down_sync(0xffffffffu, Z.x, 1), eyn = __shfl_down_sync(0xffffffffu, Y.x, 1);
                lds_if(ezn, sma, bEz + oE + 16, last);
                lds_if(eyn, sma, bEy + oE + 16, last);
                hx.x = upd<D1>(D.x, hx.x, C.x, eyk.x, Y.x, cz, ezj.x, Z.x, cy);
                hx.y = upd<D1>(D.y, hx.y, C.y, eyk.y, Y.y, cz, ezj.y, Z.y, cy);
                hx.z = upd<D1>(D.z, hx.z, C.z, eyk.z, Y.z, cz, ezj.z, Z.z, cy);
                hx.w = upd<D1>(D.w, hx.w, C.w, eyk.w, Y.w, cz, ezj.w, Z.w, cy);
                hy.x = upd<D1>(D.x, hy.x, C.x, Z.y, Z.x, cx, exk.x, X.x, cz);
                hy.y = upd<D1>(D.y, hy.y, C.y, Z.z, Z.y, cx, exk.y, X.y, cz);
                hy.z = upd<D1>(D.z, hy.z, C.z, Z.w, Z.z, cx, exk.z, X.z, cz);
                hy.w = upd<D1>(D.w, hy.w, C.w, ezn, Z.w, cx, exk.w, X.w, cz);
                hz.x = upd<D1>(D.x, hz.x, C.x, exj.x, X.x, cy, Y.y, Y.x, cx);
                hz.y = upd<D1>(D.y, hz.y, C.y, exj.y, X.y, cy, Y.z, Y.y, cx);
                hz.z = upd<D1>(D.z, hz.z, C.z, exj.z, X.z, cy, Y.w, Y.z, cx);
                hz.w = upd<D1>(D.w, hz.w, C.w, exj.w, X.w, cy, eyn, Y.w, cx);
                if (u < nu) {
                    sts4(sm, bHx + oH, hx);
                    sts4(sm, bHy + oH, hy);
                    sts4(sm, bHz + oH, hz);
                    if (u + 1 < nu) {   // a lane whose column has ended stays at its last plane
                        oE += pE;
                        oH += pH;
                    }
                    X = exk;
                    Y = eyk;
                }
            }
        }
        // the H rows below the brick, from the last thread on: those have fewest cells
#pragma unroll 1
        for (int q = T - 1 - tid; q < nbelow; q += T) {
            if (q >= T) w = below[q];
            float4 D = make_float4(1.f, 1.f, 1.f, 1.f), C = make_float4(dbu, dbu, dbu, dbu);
            if (COEF == COEF_DENSE) {
                const int h = q / lw, x = q - h * lw;
                const long long o = 4 * x + (long long)pitch * (w.iny ? y0 - 1 : y0 + h - nhy) + plane * (w.iny ? z0 + h : z0 - 1);
                D = ldg4(A.coef[2] + o);
                C = ldg4(A.coef[3] + o);
            }
            const float4 Y = lds4(sm, 16 * w.ey), Z = lds4(sm, 16 * w.ez);
            {
                const float4 Yk = lds4(sm, 16 * w.eyk), Zj = lds4(sm, 16 * w.ez + rs);
                float4 a = lds4(sm, 16 * w.hx);
                a.x = upd<D1>(D.x, a.x, C.x, Yk.x, Y.x, cz, Zj.x, Z.x, cy);
                a.y = upd<D1>(D.y, a.y, C.y, Yk.y, Y.y, cz, Zj.y, Z.y, cy);
                a.z = upd<D1>(D.z, a.z, C.z, Yk.z, Y.z, cz, Zj.z, Z.z, cy);
                a.w = upd<D1>(D.w, a.w, C.w, Yk.w, Y.w, cz, Zj.w, Z.w, cy);
                sts4(sm, 16 * w.hx, a);
            }
            // Hz (below in y): (Ex(j+1) - Ex) Cy - (Ey(i+1) - Ey) Cx; Hy (below in z): (Ez(i+1) - Ez) Cx -
            // (Ex(k+1) - Ex) Cz.  W is the operand differenced in x.
            const float4 X = lds4(sm, 16 * w.ex), Xn = lds4(sm, 16 * w.exn), W = w.iny ? Y : Z;
            const float n = *reinterpret_cast<const float *>(sm + 16 * (w.iny ? w.ey : w.ez) + 16);
            float4 b = lds4(sm, 16 * w.h2);
            if (w.iny) {
                b.x = upd<D1>(D.x, b.x, C.x, Xn.x, X.x, cy, W.y, W.x, cx);
                b.y = upd<D1>(D.y, b.y, C.y, Xn.y, X.y, cy, W.z, W.y, cx);
                b.z = upd<D1>(D.z, b.z, C.z, Xn.z, X.z, cy, W.w, W.z, cx);
                b.w = upd<D1>(D.w, b.w, C.w, Xn.w, X.w, cy, n, W.w, cx);
            } else {
                b.x = upd<D1>(D.x, b.x, C.x, W.y, W.x, cx, Xn.x, X.x, cz);
                b.y = upd<D1>(D.y, b.y, C.y, W.z, W.y, cx, Xn.y, X.y, cz);
                b.z = upd<D1>(D.z, b.z, C.z, W.w, W.z, cx, Xn.z, X.z, cz);
                b.w = upd<D1>(D.w, b.w, C.w, n, W.w, cx, Xn.w, X.w, cz);
            }
            sts4(sm, 16 * w.h2, b);
        }
        __syncthreads();
        // ================= E pass =================
        {
            int oE = oE0, oH = oH0;
            float4 xk = lds4(sm, bHx + oH - pH), yk = lds4(sm, bHy + oH - pH);   // Hx, Hy of the plane below
            bool k1 = z0 + zs >= 1;
#pragma unroll 2
            for (int u = 0; u < nmax; ++u) {
                float4 D = make_float4(1.f, 1.f, 1.f, 1.f), C = D;
                if (u < nu) {
                    C = ldg4(A.coef[1] + off0 + plane * u);
                    if (COEF == COEF_DENSE) D = ldg4(A.coef[0] + off0 + plane * u);
                }
                const float4 X = lds4(sm, bHx + oH), Y = lds4(sm, bHy + oH), Z = lds4(sm, bHz + oH);
                const float4 xj = lds4(sm, bHx + oH - rs), zj = lds4(sm, bHz + oH - rs);
                float4 ex = lds4(sm, bEx + oE), ey = lds4(sm, bEy + oE), ez = lds4(sm, bEz + oE), n;
                float hyp = __shfl_up_sync(0xffffffffu, Y.w, 1), hzp = __shfl_up_sync(0xffffffffu, Z.w, 1);
                lds_if(hyp, sma, bHy + oH - 4, first);
                lds_if(hzp, sma, bHz + oH - 4, first);
                n.x = upd<D1>(D.x, ex.x, C.x, Z.x, zj.x, cy, Y.x, yk.x, cz);
                n.y = upd<D1>(D.y, ex.y, C.y, Z.y, zj.y, cy, Y.y, yk.y, cz);
                n.z = upd<D1>(D.z, ex.z, C.z, Z.z, zj.z, cy, Y.z, yk.z, cz);
                n.w = upd<D1>(D.w, ex.w, C.w, Z.w, zj.w, cy, Y.w, yk.w, cz);
                if (j1 && k1) ex = n;
                n.x = upd<D1>(D.x, ey.x, C.x, X.x, xk.x, cz, Z.x, hzp, cx);
                n.y = upd<D1>(D.y, ey.y, C.y, X.y, xk.y, cz, Z.y, Z.x, cx);
                n.z = upd<D1>(D.z, ey.z, C.z, X.z, xk.z, cz, Z.z, Z.y, cx);
                n.w = upd<D1>(D.w, ey.w, C.w, X.w, xk.w, cz, Z.w, Z.z, cx);
                if (k1 && in0) ey.x = n.x;
                if (k1 && in1) ey.y = n.y;
                if (k1 && in2) ey.z = n.z;
                if (k1 && in3) ey.w = n.w;
                n.x = upd<D1>(D.x, ez.x, C.x, Y.x, hyp, cx, X.x, xj.x, cy);
                n.y = upd<D1>(D.y, ez.y, C.y, Y.y, Y.x, cx, X.y, xj.y, cy);
                n.z = upd<D1>(D.z, ez.z, C.z, Y.z, Y.y, cx, X.z, xj.z, cy);
                n.w = upd<D1>(D.w, ez.w, C.w, Y.w, Y.z, cx, X.w, xj.w, cy);
                if (j1 && in0) ez.x = n.x;
                if (j1 && in1) ez.y = n.y;
                if (j1 && in2) ez.z = n.z;
                if (j1 && in3) ez.w = n.w;
                if (u == src_z) {
                    const float wv = A.step + step < A.nwave ? __ldg(A.wave + A.step + step) : 0.f;
                    if (src_e == 0) ez.x = __fadd_rn(ez.x, wv);
                    else if (src_e == 1) ez.y = __fadd_rn(ez.y, wv);
                    else if (src_e == 2) ez.z = __fadd_rn(ez.z, wv);
                    else ez.w = __fadd_rn(ez.w, wv);
                }
                if (u < nu) {
                    sts4(sm, bEx + oE, ex);
                    sts4(sm, bEy + oE, ey);
                    sts4(sm, bEz + oE, ez);
                    if (u + 1 < nu) {
                        oE += pE;
                        oH += pH;
                    }
                    xk = X;
                    yk = Y;
                    k1 = true;
                }
            }
        }
        __syncthreads();
        if (step + 1 == A.steps) break;
        // ================= exchange: boundary rows out, ghost rows of the next step in ==================
        {
            ulonglong2 *const xo = A.xch + ((seq & 1) ? 2 * half : 0);
#pragma unroll
            for (int b = 0; b < kItems; ++b)
                if (xto[b] >= 0) send_unit(xo + xto[b], half, lds4(sm, xsrc[b]), seq);
            const ulonglong2 *const p = xo + 4 * cta * half + tid;
            unsigned long long t0 = 0;
            int pending = 0;
#pragma unroll
            for (int b = 0; b < kItems; ++b) pending |= xdst[b] >= 0 ? 1 << b : 0;
#pragma unroll 1
            for (int it = 0; pending; ++it) {
                ulonglong2 v[kItems][2];
#pragma unroll
                for (int b = 0; b < kItems; ++b)
                    if (pending >> b & 1) {
                        v[b][0] = load_pair(p + b * T);
                        v[b][1] = load_pair(p + b * T + half);
                    }
#pragma unroll
                for (int b = 0; b < kItems; ++b)
                    if ((pending >> b & 1) && arrived(v[b][0], v[b][1], seq)) {
                        sts4(sm, xdst[b], values(v[b][0], v[b][1]));
                        pending &= ~(1 << b);
                    }
                if (it == 0) {
                    t0 = clock_ns();
                } else if (it >= kWaitPolls || ((it & 63) == 0 && (clock_ns() - t0 > kWaitNs || *(volatile int *)A.err))) {
                    *sfail = 1;
                    atomicOr(A.err, 1);
                    break;
                }
            }
        }
        __syncthreads();
        if (*sfail) break;   // written before this barrier only; all threads leave together
    }

    // ---- results: the cells of the brick --------------------------------------------------------------
#pragma unroll 1
    for (int f = 0; f < 6; ++f)
#pragma unroll 2
        for (int u = 0; u < nu; ++u) {
            const float4 v = lds4(sm, A.base[f] + (f < 3 ? oH0 + u * pH : oE0 + u * pE));
            float *dst = A.out[f] + off0 + plane * u;
            if (in3) {
                *reinterpret_cast<float4 *>(dst) = v;
            } else {
                dst[0] = v.x;
                if (in1) dst[1] = v.y;
                if (in2) dst[2] = v.z;
            }
        }

    // The H nodes beyond the last cell (Hx at i = Nx, Hy at j = Ny, Hz at k = Nz): their curl is that
    // of wall E, which never changes, and nothing reads them, so each advances alone.
    const int ny = A.ny, nz = A.nz;
    const long long fa = (long long)ny * nz, fb = (long long)nx * nz, fc = (long long)nx * ny;
    for (long long q = (long long)cta * T + tid; q < fa + fb + fc; q += (long long)gridDim.x * T) {
        long long o;
        int f;
        float a1, a0, s1, b1, b0, s2;
        if (q < fa) {
            o = nx + (long long)pitch * (q % ny) + plane * (q / ny);
            f = 0;
            a1 = A.in[4][o + plane]; a0 = A.in[4][o]; s1 = cz; b1 = A.in[5][o + pitch]; b0 = A.in[5][o]; s2 = cy;
        } else if (q < fa + fb) {
            const long long r = q - fa;
            o = r % nx + (long long)pitch * ny + plane * (r / nx);
            f = 1;
            a1 = A.in[5][o + 1]; a0 = A.in[5][o]; s1 = cx; b1 = A.in[3][o + plane]; b0 = A.in[3][o]; s2 = cz;
        } else {
            const long long r = q - fa - fb;
            o = r % nx + (long long)pitch * (r / nx) + plane * nz;
            f = 2;
            a1 = A.in[3][o + pitch]; a0 = A.in[3][o]; s1 = cy; b1 = A.in[4][o + 1]; b0 = A.in[4][o]; s2 = cx;
        }
        const float d = A.coef[2] ? A.coef[2][o] : 1.f, cc = A.coef[3] ? A.coef[3][o] : A.db;
        float h = A.in[f][o];
        for (int s = 0; s < A.steps; ++s) h = upd<false>(d, h, cc, a1, a0, s1, b1, b0, s2);
        A.out[f][o] = h;
    }
}

namespace {

using Kernel = void (*)(const ResidentArgs);

template <int COEF>
Kernel kernel_of(const ResidentPlan &p)
{
    return p.threads > kThreadsLow ? k_yee_resident<COEF, kThreads, 5>
                                   : p.items <= 4 ? k_yee_resident<COEF, kThreadsLow, 4> : k_yee_resident<COEF, kThreadsLow, kMaxItems>;
}

// CTA shape of a brick: columns of kz planes, as many threads as fit, and enough for the exchange.
bool shape_cta(ResidentPlan &p)
{
    const int per = p.lw * p.by;   // threads of one plane
    if (per > kThreads) return false;
    p.kz = 1;
    while ((long long)per * ((p.bz + p.kz - 1) / p.kz) > kThreads) ++p.kz;
    p.nzc = (p.bz + p.kz - 1) / p.kz;
    p.kz = (p.bz + p.nzc - 1) / p.nzc;
    const int ghosts = ghost_rows(p.by, p.bz) * p.lw;
    p.threads = std::max(per * p.nzc, kMinThreads);
    // a thread per ghost unit if it can be: fewer sends one after another (32^3 1.58 us per step, with four each 1.83)
    p.threads = (std::max(p.threads, std::min(kThreadsLow, ghosts)) + 31) / 32 * 32;
    p.items = (ghosts + p.threads - 1) / p.threads;
    auto room = [&] { return p.threads > kThreadsLow ? 5 : kMaxItems; };
    if (p.items > room()) {
        p.threads = kThreads;
        p.items = (ghosts + kThreads - 1) / kThreads;
        if (p.items > room()) return false;
    }
    p.smem = shared_bytes(p);
    p.xch_bytes = sizeof(ulonglong2) * 4 * (size_t)slot_half(ghosts) * p.nby * p.nbz;
    return p.xch_bytes <= (size_t)1 << 30 && p.smem <= kSmem && rows_of(p.by, p.bz, p.lwp).total < 65536;
}

}  // namespace

// The brick shape with the least estimated time per step among those that fit: shared-memory cycles
// of the passes plus the ghost rows (sent, polled, stored), plus a part that does not shrink with the brick
// (latency of a pass, longer with more planes per thread).
bool plan_resident(int nx, int ny, int nz, int sms, ResidentPlan *out)
{
    double best = 1e30;
    bool found = false;
    for (int bz = 1; bz <= std::min(nz, 64); ++bz) {
        const int nbz = (nz + bz - 1) / bz, cols = sms / nbz;
        if (cols < 1) continue;
        // the narrowest brick that leaves no more of them than SMs: a wider one only costs more
        ResidentPlan p{};
        p.bz = bz; p.nbz = nbz;
        p.by = (ny + cols - 1) / cols;
        p.nby = (ny + p.by - 1) / p.by;
        p.lw = (nx + 3) / 4; p.lwp = nx / 4 + 1;
        if (!shape_cta(p)) continue;
        const double units = (double)p.lw * p.by * bz, ghosts = (double)p.lw * ghost_rows(p.by, bz);
        const double cost = units * 3.0 + ghosts * 1.0 + 250.0 * p.kz + 600.0;
        if (cost < best) {
            best = cost;
            *out = p;
            found = true;
        }
    }
    return found;
}

int launch_yee_resident(const ResidentPlan &p, int coef, ResidentArgs a, cudaStream_t s)
{
    const void *k = (const void *)(coef == COEF_SIMPLE ? kernel_of<COEF_SIMPLE>(p) : kernel_of<COEF_DENSE>(p));
    // set on every call: cheap, and right for whatever device is current
    PTK_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem));
    a.lw = p.lw; a.lwp = p.lwp; a.by = p.by; a.bz = p.bz; a.nby = p.nby; a.nbz = p.nbz; a.kz = p.kz;
    const Rows R = rows_of(p.by, p.bz, p.lwp);
    for (int f = 0; f < 6; ++f) a.base[f] = 16 * (R.base[f] - (f == 2 ? (p.by + 1) * p.lwp : 0));   // Hz starts at z = 0
    a.row = 16 * p.lwp; a.plane_e = (p.by + 2) * a.row; a.plane_h = (p.by + 1) * a.row;
    a.below = 16 * R.total; a.fail = a.below + (int)sizeof(BelowUnit) * (p.by + p.bz) * p.lw;
    a.half = slot_half(ghost_rows(p.by, p.bz) * p.lw);
    a.threads = p.threads;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p.nby * p.nbz);
    cfg.blockDim = dim3(p.threads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    void *args[] = {&a};
    const cudaError_t e = cudaLaunchKernelExC(&cfg, k, args);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return kNotPlaced;
    }
    PTK_CUDA_TRY(e);
    count_launches(1);
    return PTK_OK;
}

}  // namespace ptk
