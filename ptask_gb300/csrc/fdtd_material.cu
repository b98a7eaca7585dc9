// fdtd_material.cu -- per-node material index of an instance's coefficient arrays.
//
// FDTD problems are built from a few materials, so the four per-cell coefficient arrays (Ca, Cb,
// Da, Db: 16 bytes per node) hold few distinct tuples.  The staged step kernel can read a one-byte
// material id per node and the tuple from a table instead (49 bytes of traffic per cell update
// instead of 64).  This file finds the distinct tuples on the device:
//
//   1. k_mat_insert: every node's tuple (compared bit for bit) goes into an open-addressing hash
//      table of kSlots slots; lanes of a warp holding the same tuple insert it once.  A slot is
//      claimed with atomicCAS, filled, then published; readers of a claimed slot wait for the
//      publication with a bounded poll (on expiry an error word is raised and the index is not
//      used).
//   2. k_mat_compact: one block numbers the occupied slots in slot order and writes the table.
//   3. k_mat_index: every node looks its tuple up and stores the id.
//
// More than kMaxMaterials distinct tuples (or a raised error word) leaves the index unused: the
// caller keeps the per-cell arrays.  The values in the table are the arrays' own bits, so results
// are identical either way.
#include "ptk_internal.h"

namespace ptk {

namespace {

constexpr int kSlots = 1024;
constexpr int kPollLimit = 1 << 20;

struct MatScratch {
    unsigned state[kSlots];   // 0 empty, 1 being filled, 2 published
    uint4 key[kSlots];
    int id[kSlots];
    int count;                // distinct tuples inserted
    int err;                  // 1: a poll expired, 2: the table filled up
    int varied;               // a node with Ca or Da other than 1, or another Db than the first node's
    MaterialInfo info;        // result
};

__device__ __forceinline__ unsigned mix(uint4 k)
{
    unsigned h = k.x * 0x9E3779B1u;
    h = (h ^ k.y) * 0x85EBCA77u;
    h = (h ^ k.z) * 0xC2B2AE3Du;
    h = (h ^ k.w) * 0x27D4EB2Fu;
    return h ^ (h >> 15);
}

__device__ __forceinline__ uint4 tuple_at(const float *const *c, long long o)
{
    return make_uint4(__float_as_uint(__ldg(c[0] + o)), __float_as_uint(__ldg(c[1] + o)),
                      __float_as_uint(__ldg(c[2] + o)), __float_as_uint(__ldg(c[3] + o)));
}

__device__ __forceinline__ bool same(uint4 a, uint4 b) { return a.x == b.x && a.y == b.y && a.z == b.z && a.w == b.w; }

__device__ uint4 read_key(const MatScratch *S, int h)
{
    const volatile unsigned *k = reinterpret_cast<const volatile unsigned *>(&S->key[h]);
    return make_uint4(k[0], k[1], k[2], k[3]);
}

__device__ void insert(MatScratch *S, uint4 key)
{
    // Too many materials already: the index will not be used, and a full table would cost every node
    // a walk through all of it (160^3 cells with a permittivity each: 357 ms).
    if (*reinterpret_cast<volatile int *>(&S->count) > kMaxMaterials) return;
    unsigned h = mix(key) & (kSlots - 1);
    for (int probe = 0; probe < kSlots; ++probe, h = (h + 1) & (kSlots - 1)) {
        // Most nodes repeat a tuple that is already published: check with a plain read first, so
        // that only new tuples contend for a slot with an atomic.
        if (reinterpret_cast<volatile unsigned *>(S->state)[h] == 2u) {
            __threadfence();
            if (same(read_key(S, h), key)) return;
            continue;
        }
        const unsigned st = atomicCAS(&S->state[h], 0u, 1u);
        if (st == 0u) {
            S->key[h] = key;
            __threadfence();
            atomicExch(&S->state[h], 2u);
            atomicAdd(&S->count, 1);
            return;
        }
        int it = 0;
        while (reinterpret_cast<volatile unsigned *>(S->state)[h] != 2u && ++it < kPollLimit) {
        }
        if (it >= kPollLimit) {
            atomicOr(&S->err, 1);
            return;
        }
        __threadfence();
        if (same(read_key(S, h), key)) return;
    }
    atomicOr(&S->err, 2);
}

// The (nx+1) x (ny+1) x (nz+1) node grid by rows (row padding is not part of the problem): a warp takes
// a row at a time.
struct Nodes {
    int nx, ny, pitch, rows;
    long long plane;
    __device__ long long row(int r) const { return (long long)pitch * (r % (ny + 1)) + plane * (r / (ny + 1)); }
};

__global__ void __launch_bounds__(256) k_mat_insert(const float *Ca, const float *Cb, const float *Da, const float *Db, Nodes N,
                                                    MatScratch *S)
{
    const float *c[4] = {Ca, Cb, Da, Db};
    const int lane = threadIdx.x & 31;
    const unsigned db = __float_as_uint(__ldg(Db));
    uint4 last = make_uint4(0, 0, 0, 0);   // the tuple this lane saw last (in the table already)
    bool have_last = false, varied = false;
    for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < N.rows; r += gridDim.x * 8) {
        const long long o = N.row(r);
        const bool full = *reinterpret_cast<volatile int *>(&S->count) > kMaxMaterials;   // no index: only `varied` is left to see
        for (int i = lane; i <= N.nx; i += 32) {
            const uint4 key = tuple_at(c, o + i);
            varied |= key.x != 0x3f800000u || key.z != 0x3f800000u || key.w != db;
            if (full) continue;
            const bool fresh = !(have_last && same(key, last));
            const unsigned act = __activemask();
            if (!__any_sync(act, fresh)) continue;
            // lanes with the same tuple (all four words equal) let their lowest lane insert it
            const unsigned m = __match_any_sync(act, key.x) & __match_any_sync(act, key.y) &
                               __match_any_sync(act, key.z) & __match_any_sync(act, key.w);
            if (lane == __ffs(m) - 1 && fresh) insert(S, key);
            last = key;   // inserted by this lane or by that one
            have_last = true;
        }
    }
    if (varied) S->varied = 1;
}

// Numbers the occupied slots in slot order, a thread per slot (one thread for all of them: 56 us).
__global__ void __launch_bounds__(kSlots) k_mat_compact(MatScratch *S, float4 *tab, const float *Db)
{
    __shared__ int before[kSlots / 32];
    const int h = threadIdx.x, lane = h & 31, warp = h >> 5;
    const bool on = S->state[h] == 2u;
    const unsigned mask = __ballot_sync(0xffffffffu, on);
    if (lane == 0) before[warp] = __popc(mask);
    __syncthreads();
    int id = __popc(mask & ((1u << lane) - 1)), n = 0;
    for (int w = 0; w < kSlots / 32; ++w) {
        if (w == warp) id += n;
        n += before[w];
    }
    if (on) {
        const uint4 k = S->key[h];
        if (id < kMaxMaterials)
            tab[id] = make_float4(__uint_as_float(k.x), __uint_as_float(k.y), __uint_as_float(k.z), __uint_as_float(k.w));
        S->id[h] = id;
    }
    if (h == 0) {
        S->info.nmat = (S->err || n > kMaxMaterials || n != S->count) ? 0 : n;
        S->info.simple = !S->varied;
        S->info.db = *Db;
    }
}

__global__ void __launch_bounds__(256) k_mat_index(const float *Ca, const float *Cb, const float *Da, const float *Db, Nodes N,
                                                   const MatScratch *S, unsigned char *mat)
{
    if (S->info.nmat == 0) return;
    const float *c[4] = {Ca, Cb, Da, Db};
    uint4 last = make_uint4(0, 0, 0, 0);   // the tuple looked up last
    int id = -1;
    for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < N.rows; r += gridDim.x * 8) {
        const long long o = N.row(r);
        for (int i = threadIdx.x & 31; i <= N.nx; i += 32) {
            const uint4 key = tuple_at(c, o + i);
            if (id < 0 || !same(key, last)) {
                unsigned h = mix(key) & (kSlots - 1);
                for (int probe = 0; probe < kSlots; ++probe, h = (h + 1) & (kSlots - 1))
                    if (S->state[h] == 2u && same(S->key[h], key)) {
                        id = S->id[h];
                        break;
                    }
                last = key;
            }
            mat[o + i] = (unsigned char)id;
        }
    }
}

}  // namespace

int build_material_index(const float *const coef[4], const Layout &L, unsigned char *mat, float *tab, MaterialInfo *info,
                         cudaStream_t s)
{
    PTK_CHECK_ARG(coef && mat && tab && info, "NULL argument");
    *info = MaterialInfo{};
    MatScratch *S = nullptr;
    int rc = pool_alloc(sizeof(MatScratch), s, (void **)&S);
    if (rc) return rc;
    PTK_CUDA_TRY(cudaMemsetAsync(S, 0, sizeof(MatScratch), s));
    Nodes N{L.nx, L.ny, L.pitch, (L.ny + 1) * (L.nz + 1), L.plane};
    const int grid = std::min((N.rows + 7) / 8, 8 * std::max(1, sm_count()));
    k_mat_insert<<<grid, 256, 0, s>>>(coef[0], coef[1], coef[2], coef[3], N, S);
    k_mat_compact<<<1, kSlots, 0, s>>>(S, reinterpret_cast<float4 *>(tab), coef[3]);
    k_mat_index<<<grid, 256, 0, s>>>(coef[0], coef[1], coef[2], coef[3], N, S, mat);
    PTK_CUDA_TRY(cudaGetLastError());
    count_launches(3);
    MaterialInfo h;
    PTK_CUDA_TRY(cudaMemcpyAsync(&h, &S->info, sizeof h, cudaMemcpyDeviceToHost, s));
    PTK_CUDA_TRY(cudaStreamSynchronize(s));
    pool_free(S, s);
    *info = h;
    return PTK_OK;
}

}  // namespace ptk
