// Batched solves of many independent systems of uneven size in one device-driven loop.
//
// The reference solves one system per RMatrixSolver::solve call
// (src/rmatrixsolver.cpp:158-201); callers such as a transient or multi-load-case
// run, or many small meshes, then pay one solve's launch and synchronisation
// costs per system.  Here the systems are packed block-diagonally into one
// matrix, each padded to a multiple of 32 rows with identity rows, so that
// every 32-row SELL slice belongs to exactly one system.  Each system keeps its
// own CG state (the same CgState and transitions as the single-system solver:
// stop on FP64 true relative residual, FP64 or mixed precision with reliable
// updates).  Per iteration two kernels (direction + SpMV, update) run over the
// active systems' slices in chunks of one per warp, counted from a system's first
// slice: every block takes a contiguous range of the list's chunks, so most blocks
// work for one system, and adds up each chunk; the last block to finish with a
// system (a ticket per system) adds the chunks' sums in their order and advances
// that system's state.  So a system's sums do not depend on the grid, nor on the
// systems beside it.
// A system whose update asks for a residual check waits (the next directions and
// updates skip it) until the check that ends each body of kBatchIterations
// iterations, an FP64 SpMV over the systems that asked.  The loop is one CUDA
// graph `while` node; the tail kernel rebuilds the active list and keeps the loop
// running while any system is active.
#include "krylov.cuh"

#include <algorithm>
#include <chrono>
#include <cstring>
#include <vector>

struct rsg_batch {
    uint32_t n_sys = 0;
    uint32_t user_rows = 0, pad_rows = 0;
    rsg_csr *A = nullptr;                  // padded block-diagonal matrix
    std::vector<uint32_t> user_begin, pad_begin;
    uint32_t *d_slice_sys = nullptr;       // system of each slice
    uint32_t *d_sys_slice = nullptr;       // first slice of each system (n_sys + 1)
    uint32_t *d_user2pad = nullptr;        // padded row of each user row
    // grid of the slice kernels picked by rsg_batch_autotune (0 = the built-in default)
    int32_t g64 = 0, g32 = 0;
    double it64 = 0, it32 = 0, it64_default = 0, it32_default = 0;
    uint32_t tune_candidates = 0;
    bool tuned = false;
};

namespace rsg {
namespace {

struct BatchCtl {
    uint32_t body_count;
    uint32_t body_limit;
    int32_t timeout;
    int32_t keep;
    uint32_t cut;  // bodies in a row in which no system made more than one iteration
};

constexpr int kBatchIterations = 4;
constexpr uint32_t kChunk = kWarpsPerBlock;  // slices of a chunk
constexpr uint32_t kHold = 32;               // chunks that a block holds the warps' sums of

struct BView {
    const uint32_t *slice_sys;
    const uint32_t *sys_slice;
    uint32_t n_slices, n_sys;
};

// Systems a kernel visits.  One entry holds all that a block needs to start on a system, so that finding
// its place takes two round trips to memory (the head beside the entries' first words, then the entry)
// instead of a binary search through a chain of them.
struct ListHead {
    uint32_t n_sys;     // number of listed systems
    uint32_t n_chunks;  // their chunks in total
};
struct Active {
    ListHead *head;
    uint4 *entry;  // per listed system, list_entry
};
// {system | (slices of its last chunk - 1) << 29, first and last + 1 of its chunks in the list, its first slice}
__host__ __device__ __forceinline__ uint4 list_entry(uint32_t sys, uint32_t at, uint32_t first, uint32_t slices)
{
    return make_uint4(sys | (slices - 1) % kChunk << 29, at, at + (slices + kChunk - 1) / kChunk, first);
}
constexpr uint32_t kSysMask = (1u << 29) - 1;

// Block-wide (blockDim.x == kBlock): lists in order the systems of `in` (0..n_in when it has no entries)
// that keep(system) accepts.  Every thread calls it; keep must give the same answer on both of its calls.
template <class KEEP>
__device__ __forceinline__ void build_list(uint32_t n_in, const uint4 *in, const uint32_t *sys_slice, const Active &out,
                                           KEEP keep)
{
    __shared__ uint32_t cnt_sys[kBlock], cnt_sl[kBlock];
    const uint32_t t = threadIdx.x, per = (n_in + blockDim.x - 1) / blockDim.x;
    const uint32_t i0 = min(n_in, t * per), i1 = min(n_in, i0 + per);
    uint32_t ns = 0, nsl = 0;
    for (uint32_t i = i0; i < i1; i++) {
        const uint32_t sys = in ? in[i].x & kSysMask : i;
        if (keep(sys)) {
            ns++;
            nsl += (sys_slice[sys + 1] - sys_slice[sys] + kChunk - 1) / kChunk;
        }
    }
    // exclusive scans over the block
    uint32_t a = ns, b = nsl;
    const uint32_t lane = t & 31u, warp = t >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, b, o);
        if (lane >= uint32_t(o)) {
            a += x;
            b += y;
        }
    }
    if (lane == 31) {
        cnt_sys[warp] = a;
        cnt_sl[warp] = b;
    }
    __syncthreads();
    for (uint32_t w = 0; w < warp; w++) {
        a += cnt_sys[w];
        b += cnt_sl[w];
    }
    if (t == blockDim.x - 1) *out.head = ListHead{a, b};
    uint32_t o = a - ns, pre = b - nsl;
    for (uint32_t i = i0; i < i1; i++) {
        const uint32_t sys = in ? in[i].x & kSysMask : i;
        if (keep(sys)) {
            const uint32_t first = sys_slice[sys];
            const uint4 e = list_entry(sys, pre, first, sys_slice[sys + 1] - first);
            out.entry[o++] = e;
            pre = e.z;
        }
    }
    __syncthreads();
}

// SELL row product of this lane's row in slice s.
template <typename V, class GX>
__device__ __forceinline__ V sell_row(const Sell<V> &M, uint32_t s, int lane, GX &gx)
{
    const uint32_t row0 = s * 32u, row = row0 + lane;
    const uint32_t len = row < M.n ? __ldg(&M.rp[row + 1]) - __ldg(&M.rp[row]) : 0u;
    const uint32_t g4 = __ldg(&M.slice_len4[s]);
    const size_t base = size_t(__ldg(&M.slice_ptr[s])) + 4u * lane;
    V acc = V(0);
#pragma unroll 4
    for (uint32_t g = 0; g < g4; g++) {
        const size_t e = base + size_t(g) * 128u;
        V v[4];
        ld4(M.val + e, v);
        uint32_t c[4];
        if (M.off) {
            const short4 o = __ldcs(reinterpret_cast<const short4 *>(M.off + e));
            c[0] = uint32_t(int(row0) + o.x);
            c[1] = uint32_t(int(row0) + o.y);
            c[2] = uint32_t(int(row0) + o.z);
            c[3] = uint32_t(int(row0) + o.w);
        } else {
            const uint4 o = __ldcs(reinterpret_cast<const uint4 *>(M.col + e));
            c[0] = o.x;
            c[1] = o.y;
            c[2] = o.z;
            c[3] = o.w;
        }
#pragma unroll
        for (int t = 0; t < 4; t++)
            if (4u * g + t < len) acc = row_acc(acc, v[t], V(gx(c[t])));
    }
    return acc;
}

// The state transition that a phase's per-system sums lead to (the same transitions as the single-system
// solver).
enum RedKind { RED_INIT_RES = 0, RED_INIT_Z, RED_DIR64, RED_DIR32, RED_UPD64, RED_UPD32, RED_CHK64, RED_CHK32, RED_TRUE };

template <int NV, int KIND>
__device__ __forceinline__ void finalize(CgState *st, const double (&acc)[NV], double *relres, uint32_t sys)
{
    if constexpr (KIND == RED_INIT_RES) {
        st->rn = sqrt(acc[0]);
        st->bn = sqrt(acc[1]);
        st->max_r = st->rn;
        st->sigma = st->bn > 0.0 ? 1.0 / st->bn : 1.0;
        if (!(st->rn > st->rtol * st->bn)) {
            st->done = 1;
            st->converged = 1;
            st->status = isfinite(st->rn) ? RSG_OK : RSG_BREAKDOWN;
        }
    } else if constexpr (KIND == RED_INIT_Z) {
        st->rho = st->rho_new = acc[0];
        st->beta = 0.0;
    } else if constexpr (KIND == RED_DIR64 || KIND == RED_DIR32) {
        double pq = acc[0];
        if constexpr (KIND == RED_DIR32) {
            if (pq == 0.0) pq = 1e-300;
        } else {
            pq = clamp_pq(pq, st->eps);
        }
        st->pq = pq;
        st->rho = st->rho_new;
        st->alpha = st->rho / pq;
        st->fold = 0;
        st->pcur ^= 1u;
    } else if constexpr (KIND == RED_UPD64) {
        finalize_update64(st, acc[0], acc[1], acc[2]);
    } else if constexpr (KIND == RED_UPD32) {
        finalize_update_mixed(st, acc[0], acc[1]);
    } else if constexpr (KIND == RED_CHK64) {
        finalize_check64(st, acc[0], sqrt(acc[1]));
    } else if constexpr (KIND == RED_CHK32) {
        finalize_check_mixed(st, acc[0], sqrt(acc[1]));
    } else {
        relres[sys] = acc[1] > 0.0 ? sqrt(acc[0] / acc[1]) : sqrt(acc[0]);
    }
}


// The blocks' loop over the listed systems' chunks.  Block j takes chunks [j per, (j + 1) per) of the list; systems
// that `skip(st)` rejects are jumped over as a whole.  For every visited slice one warp runs `body(s, st, v)`, which
// returns the lane's contributions; a chunk's sum is its warps' sums in order.  A system that lies in one block is
// finished there; otherwise the block stores its chunks' sums, and the last block to take the system's ticket adds
// them.  24 uneven cubes (0.39M rows), ms a solve, mixed / FP64: sums and transition as kernels of their own after
// every phase, with the check in every iteration, 14.2 / 13.4; a warp's slices of a block added up by the lanes,
// which made a system's bits depend on the grid and on its companions, 11.0 / 10.5; chunks 9.9 / 9.6.  64 cubes of 8 to
// 60 hexes a side, mixed: 75.5, 57.4 and 59.4 (a warp sum per slice).  16, 64 and 128 chunks held: within 2%.
struct Sums {
    double *part;          // [batch_parts][3]: a system's chunks from its first slice / kChunk + its number on
    unsigned int *ticket;  // per system, zero between uses
    double *relres;        // RED_TRUE only
};
inline size_t batch_parts(uint32_t n_slices, uint32_t n_sys) { return size_t(n_slices) / kChunk + n_sys; }

template <int NV, int KIND, class SKIP, class BODY>
__device__ __forceinline__ void batch_run(const BView &B, const Active L, CgState *S, const Sums &T, SKIP skip, BODY body)
{
    __shared__ double sh[NV * 32];
    __shared__ __align__(16) double hold[NV][kHold][kChunk];
    __shared__ CgState s;
    __shared__ int last_sh;
    const uint32_t warp = threadIdx.x >> 5;
    // the entries that start at or before this block's first chunk are the first of the list: count them
    uint32_t begin = threadIdx.x < B.n_sys ? L.entry[threadIdx.x].y : 0u;
    const uint32_t total = L.head->n_chunks, n_list = L.head->n_sys;
    const uint32_t per = (total + gridDim.x - 1) / gridDim.x;
    uint32_t a = min(uint64_t(total), uint64_t(blockIdx.x) * per);
    const uint32_t a_end = min(total, a + per);
    if (a >= a_end) return;
    uint32_t k = 0;
    for (uint32_t i = 0; i < n_list; i += blockDim.x) {
        if (i) begin = i + threadIdx.x < n_list ? L.entry[i + threadIdx.x].y : 0u;
        k += __syncthreads_count(i + threadIdx.x < n_list && begin <= a);
    }
    k--;
    for (; a < a_end; k++) {
        const uint4 e = L.entry[k];
        const uint32_t sys = e.x & kSysMask, k_begin = e.y, k_end = e.z, stop = min(a_end, k_end);
        CgState *st = &S[sys];
        if (!skip(st)) {
            const uint32_t chunks = k_end - k_begin;
            double *part = T.part + (size_t(e.w / kChunk) + sys) * NV;
            const bool here = chunks <= kHold && a == k_begin && stop == k_end;  // all of it, in one go
            double v[NV];
            for (; a < stop; a += kHold) {
                const uint32_t m = min(kHold, stop - a);
                for (uint32_t j = 0; j < m; j++) {
                    const uint32_t c = a + j - k_begin;
                    double t[NV];
#pragma unroll
                    for (int q = 0; q < NV; q++) t[q] = 0.0;
                    if (c + 1 < chunks || warp <= e.x >> 29) body(e.w + c * kChunk + warp, st, t);
#pragma unroll
                    for (int q = 0; q < NV; q++) t[q] = warp_sum(t[q]);
                    if ((threadIdx.x & 31) == 0)
#pragma unroll
                        for (int q = 0; q < NV; q++) hold[q][j][warp] = t[q];
                }
                __syncthreads();
#pragma unroll
                for (int q = 0; q < NV; q++) {
                    v[q] = 0.0;
                    if (threadIdx.x < m) {
                        const double2 *w = reinterpret_cast<const double2 *>(hold[q][threadIdx.x]);
                        const double2 w0 = w[0], w2 = w[1], w4 = w[2], w6 = w[3];
                        v[q] = ((w0.x + w0.y) + (w2.x + w2.y)) + ((w4.x + w4.y) + (w6.x + w6.y));
                        if (!here) part[size_t(a + threadIdx.x - k_begin) * NV + q] = v[q];
                    }
                }
                __syncthreads();
            }
            const uint32_t n_blocks = (k_end - 1) / per - k_begin / per + 1;
            if (threadIdx.x == 0) {
                last_sh = 1;
                if (n_blocks > 1) {
                    unsigned int t;
                    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(t) : "l"(T.ticket + sys) : "memory");
                    last_sh = t == n_blocks - 1;
                }
            }
            __syncthreads();
            if (last_sh) {
                for (uint32_t w = threadIdx.x; w < kStateWords; w += blockDim.x)
                    reinterpret_cast<uint32_t *>(&s)[w] = __ldcg(reinterpret_cast<const uint32_t *>(st) + w);
                if (!here) {
#pragma unroll
                    for (int q = 0; q < NV; q++) v[q] = 0.0;
#pragma unroll 4
                    for (uint32_t i = threadIdx.x; i < chunks; i += blockDim.x)
#pragma unroll
                        for (int q = 0; q < NV; q++) v[q] += __ldcg(&part[size_t(i) * NV + q]);
                    if (threadIdx.x == 0) T.ticket[sys] = 0u;
                }
                block_sum<NV>(v, sh);
                if (threadIdx.x == 0) finalize<NV, KIND>(&s, v, T.relres, sys);
                __syncthreads();
                if (KIND != RED_TRUE)
                    for (uint32_t w = threadIdx.x; w < kStateWords; w += blockDim.x)
                        reinterpret_cast<uint32_t *>(st)[w] = reinterpret_cast<const uint32_t *>(&s)[w];
                __syncthreads();
            }
        }
        a = stop;
    }
}

#define BATCH_ROWS_LOOP                                                                                      \
    const int lane = threadIdx.x & 31;                                                                      \
    const uint32_t warps_total = gridDim.x * (blockDim.x >> 5);                                             \
    for (uint32_t s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); s < B.n_slices; s += warps_total)

__global__ void __launch_bounds__(kBlock) bk_init_res(Sell<double> M, BView B, const Active L, const double *__restrict__ b,
                                                      const double *__restrict__ x, double *__restrict__ r,
                                                      Sums T, CgState *S)
{
    const int lane = threadIdx.x & 31;
    auto gx = [&](uint32_t c) { return x[c]; };
    batch_run<2, RED_INIT_RES>(
        B, L, S, T, [](const CgState *) { return false; },
        [&](uint32_t s, CgState *, double(&v)[2]) {
            const double ax = sell_row<double>(M, s, lane, gx);
            const uint32_t row = s * 32u + lane;
            v[0] = v[1] = 0.0;
            if (row < M.n) {
                const double ri = b[row] - ax;
                r[row] = ri;
                v[0] = ri * ri;
                v[1] = b[row] * b[row];
            }
        });
}

template <bool MIXED>
__global__ void __launch_bounds__(kBlock) bk_init_z(BView B, const Active L, uint32_t n, const double *__restrict__ d,
                                                    const float *__restrict__ d32, const double *__restrict__ r,
                                                    double *__restrict__ z, float *__restrict__ r32,
                                                    float *__restrict__ z32, Sums T, CgState *S)
{
    const int lane = threadIdx.x & 31;
    batch_run<1, RED_INIT_Z>(
        B, L, S, T, [](const CgState *st) { return st->done != 0; },
        [&](uint32_t s, CgState *st, double(&v)[1]) {
            const uint32_t row = s * 32u + lane;
            v[0] = 0.0;
            if (row < n) {
                if (MIXED) {
                    const float rf = float(r[row] * st->sigma);
                    const float zf = d32 ? d32[row] * rf : rf;
                    r32[row] = rf;
                    z32[row] = zf;
                    v[0] = double(rf) * double(zf);
                } else {
                    const double zi = d ? d[row] * r[row] : r[row];
                    z[row] = zi;
                    v[0] = r[row] * zi;
                }
            }
        });
}

// Six blocks an SM: 40 registers and 84 to 88 bytes spilled, all the same the fastest but for single sizes; ms a solve
// with six, five and four, 24 cubes mixed 9.9, 9.9, 10.0, FP64 9.6, 10.0, 9.3; 64 cubes mixed 59.4, 58.8, 64.6, FP64 74.9,
// 77.4, 75.8.
template <typename V, bool MIXED>
__global__ void __launch_bounds__(kBlock, 6) bk_dir(Sell<V> M, BView B, const Active L, const V *__restrict__ z, V *p0,
                                                 V *p1, V *__restrict__ q, double *__restrict__ x,
                                                 float *__restrict__ y, Sums T, CgState *S)
{
    pdl_wait();
    pdl_release();
    const int lane = threadIdx.x & 31;
    batch_run<1, MIXED ? RED_DIR32 : RED_DIR64>(
        B, L, S, T, [](const CgState *st) { return st->done != 0 || st->need_check != 0; },
        [&](uint32_t s, CgState *st, double(&v)[1]) {
            const V beta = V(st->beta);
            const V *__restrict__ p_old = st->pcur ? p1 : p0;
            V *__restrict__ p_new = st->pcur ? p0 : p1;
            auto gx = [&](uint32_t c) { return MIXED ? V(fmaf(float(beta), float(p_old[c]), float(z[c])))
                                                     : V(fma(double(beta), double(p_old[c]), double(z[c]))); };
            const V ax = sell_row<V>(M, s, lane, gx);
            const uint32_t row = s * 32u + lane;
            v[0] = 0.0;
            if (row < M.n) {
                const V p = gx(row);
                p_new[row] = p;
                q[row] = ax;
                v[0] = double(p) * double(ax);
                if (MIXED && st->fold) {
                    x[row] = fma(double(y[row]), 1.0 / st->sigma, x[row]);
                    y[row] = 0.f;
                }
            }
        });
}

template <typename V, bool MIXED>
__global__ void __launch_bounds__(kBlock, 6) bk_update(BView B, const Active L, uint32_t n, const V *__restrict__ d,
                                                    const V *p0, const V *p1, const V *__restrict__ q,
                                                    V *__restrict__ xy, V *__restrict__ r, V *__restrict__ z,
                                                    Sums T, CgState *S)
{
    pdl_wait();
    pdl_release();
    const int lane = threadIdx.x & 31;
    batch_run<3, MIXED ? RED_UPD32 : RED_UPD64>(
        B, L, S, T, [](const CgState *st) { return st->done != 0 || st->need_check != 0; },
        [&](uint32_t s, CgState *st, double(&v)[3]) {
            const V alpha = V(st->alpha);
            const V *__restrict__ p = st->pcur ? p1 : p0;
            const uint32_t row = s * 32u + lane;
            v[0] = v[1] = v[2] = 0.0;
            if (row < n) {
                const V xi = MIXED ? V(fmaf(float(alpha), float(p[row]), float(xy[row])))
                                   : V(fma(double(alpha), double(p[row]), double(xy[row])));
                const V ri = MIXED ? V(fmaf(-float(alpha), float(q[row]), float(r[row])))
                                   : V(fma(-double(alpha), double(q[row]), double(r[row])));
                const V zi = d ? d[row] * ri : ri;
                xy[row] = xi;
                r[row] = ri;
                z[row] = zi;
                v[0] = double(ri) * double(zi);
                v[1] = double(ri) * double(ri);
                v[2] = double(xi) * double(xi);
            }
        });
}

template <bool MIXED>
__global__ void __launch_bounds__(kBlock) bk_check(Sell<double> M, BView B, const Active L, const double *__restrict__ d,
                                                   const float *__restrict__ d32, const double *__restrict__ b,
                                                   const double *__restrict__ x, const float *__restrict__ y,
                                                   double *__restrict__ r, double *__restrict__ z,
                                                   float *__restrict__ r32, float *__restrict__ z32, Sums T,
                                                   CgState *S)
{
    pdl_wait();
    pdl_release();
    const int lane = threadIdx.x & 31;
    batch_run<2, MIXED ? RED_CHK32 : RED_CHK64>(
        B, L, S, T, [](const CgState *st) { return st->done != 0 || st->need_check == 0; },
        [&](uint32_t s, CgState *st, double(&v)[2]) {
            const double sigma = st->sigma, inv_sigma = 1.0 / sigma;
            auto gx = [&](uint32_t c) { return MIXED ? fma(double(y[c]), inv_sigma, x[c]) : x[c]; };
            const double ax = sell_row<double>(M, s, lane, gx);
            const uint32_t row = s * 32u + lane;
            v[0] = v[1] = 0.0;
            if (row < M.n) {
                const double ri = b[row] - ax;
                v[1] = ri * ri;
                if (MIXED) {
                    const float rf = float(ri * sigma);
                    const float zf = d32 ? d32[row] * rf : rf;
                    r32[row] = rf;
                    z32[row] = zf;
                    v[0] = double(rf) * double(zf);
                } else {
                    const double zi = d ? d[row] * ri : ri;
                    r[row] = ri;
                    z[row] = zi;
                    v[0] = ri * zi;
                }
            }
        });
}

__global__ void bk_fold(BView B, uint32_t n, double *__restrict__ x, float *__restrict__ y, const CgState *S)
{
    BATCH_ROWS_LOOP
    {
        const uint32_t row = s * 32u + lane;
        if (row < n) {
            x[row] = fma(double(y[row]), 1.0 / S[B.slice_sys[s]].sigma, x[row]);
            y[row] = 0.f;
        }
    }
}

__global__ void bk_true_res(Sell<double> M, BView B, const Active L, const double *__restrict__ b, const double *__restrict__ x,
                            Sums T, CgState *S)
{
    const int lane = threadIdx.x & 31;
    auto gx = [&](uint32_t c) { return x[c]; };
    batch_run<2, RED_TRUE>(
        B, L, S, T, [](const CgState *) { return false; },
        [&](uint32_t s, CgState *, double(&v)[2]) {
            const double ax = sell_row<double>(M, s, lane, gx);
            const uint32_t row = s * 32u + lane;
            v[0] = v[1] = 0.0;
            if (row < M.n) {
                const double ri = b[row] - ax;
                v[0] = ri * ri;
                v[1] = b[row] * b[row];
            }
        });
}

// The systems of L that asked for a residual check.
__global__ void __launch_bounds__(kBlock) bk_list(const CgState *S, const uint32_t *sys_slice, const Active L, const Active L_chk)
{
    pdl_wait();
    pdl_release();
    build_list(L.head->n_sys, L.entry, sys_slice, L_chk, [&](uint32_t i) { return S[i].done == 0 && S[i].need_check != 0; });
}

// Loop control: rebuilds the list of active systems, keeps the graph's while node
// running while any system is active, enforces the hard limit.
__global__ void __launch_bounds__(kBlock) bk_tail(CgState *S, const uint32_t *sys_slice, uint32_t n_sys,
                                                  const Active L, BatchCtl *ctl, cudaGraphConditionalHandle h,
                                                  int use_cond, int iterations)
{
    pdl_wait();
    pdl_release();
    bool far = iterations < 4;  // some system made more than one iteration (kCutBodies)
    for (uint32_t i = threadIdx.x; i < n_sys; i += blockDim.x) {
        const uint32_t it = S[i].it;
        far = far || it - S[i].last_it > 1;
        S[i].last_it = it;
    }
    const int any_far = __syncthreads_or(far);
    build_list(n_sys, nullptr, sys_slice, L, [&](uint32_t i) { return S[i].done == 0; });
    if (threadIdx.x == 0) {
        const uint32_t bc = ++ctl->body_count;
        int keep = L.head->n_sys > 0;
        if (keep && bc >= ctl->body_limit) {
            ctl->timeout = 1;
            keep = 0;
        }
        const uint32_t cut = any_far ? 0u : ctl->cut + 1;
        ctl->cut = cut;
        if (use_cond) cudaGraphSetConditional(h, keep && cut < kCutBodies ? 1u : 0u);
        ctl->keep = keep;
    }
}

__global__ void bk_to_f32(uint32_t n, const double *__restrict__ src, float *__restrict__ dst)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        dst[i] = float(src[i]);
}

__global__ void bk_scatter(uint32_t n_user, const uint32_t *__restrict__ map, const double *__restrict__ src,
                           double *__restrict__ dst)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_user; i += gridDim.x * blockDim.x)
        dst[map[i]] = src[i];
}
__global__ void bk_gather(uint32_t n_user, const uint32_t *__restrict__ map, const double *__restrict__ src,
                          double *__restrict__ dst)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_user; i += gridDim.x * blockDim.x)
        dst[i] = src[map[i]];
}

}  // namespace
}  // namespace rsg

using namespace rsg;

extern "C" {

rsg_status rsg_batch_create(rsg_context *ctx, uint32_t n_sys, const uint32_t *sys_row_begin, const uint32_t *row_ptr,
                            const uint32_t *col_idx, const double *values, rsg_batch **out)
{
    if (!ctx || !out || !sys_row_begin || !row_ptr || n_sys == 0)
        return set_error(ctx, RSG_ERR_INVALID_ARG, "batch_create: bad arguments");
    *out = nullptr;
    RSG_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    if (sys_row_begin[0] != 0) return set_error(ctx, RSG_ERR_INVALID_ARG, "batch_create: systems must start at row 0");
    auto *B = new rsg_batch;
    B->n_sys = n_sys;
    B->user_begin.assign(sys_row_begin, sys_row_begin + n_sys + 1);
    B->pad_begin.assign(size_t(n_sys) + 1, 0);
    uint64_t pad_total = 0;
    for (uint32_t s = 0; s < n_sys; s++) {
        if (B->user_begin[s + 1] < B->user_begin[s] || B->user_begin[s + 1] == B->user_begin[s]) {
            delete B;
            return set_error(ctx, RSG_ERR_INVALID_ARG, "batch_create: empty or decreasing system %u", s);
        }
        B->pad_begin[s] = uint32_t(pad_total);
        pad_total += (uint64_t(B->user_begin[s + 1] - B->user_begin[s]) + 31u) & ~uint64_t(31);
        if (pad_total > 0xffffff00ull) {
            delete B;
            return set_error(ctx, RSG_ERR_INVALID_ARG, "batch_create: more than 2^32 rows after padding");
        }
    }
    B->pad_begin[n_sys] = uint32_t(pad_total);
    B->user_rows = B->user_begin[n_sys];
    B->pad_rows = uint32_t(pad_total);
    if (row_ptr[0] != 0) {
        delete B;
        return set_error(ctx, RSG_ERR_INVALID_ARG, "batch_create: row_ptr[0] != 0");
    }
    // padded block-diagonal CSR; identity rows fill each system to a multiple of 32
    std::vector<uint32_t> rp(size_t(pad_total) + 1, 0), ci, map(B->user_rows);
    std::vector<double> val;
    ci.reserve(row_ptr[B->user_rows] + (pad_total - B->user_rows));
    val.reserve(ci.capacity());
    std::vector<uint32_t> slice_sys(pad_total / 32), sys_slice(size_t(n_sys) + 1);
    uint32_t prow = 0;
    for (uint32_t s = 0; s < n_sys; s++) {
        const uint32_t u0 = B->user_begin[s], u1 = B->user_begin[s + 1], p0 = B->pad_begin[s], p1 = B->pad_begin[s + 1];
        sys_slice[s] = p0 / 32;
        for (uint32_t q = p0 / 32; q < p1 / 32; q++) slice_sys[q] = s;
        for (uint32_t i = u0; i < u1; i++) {
            map[i] = p0 + (i - u0);
            for (uint32_t j = row_ptr[i]; j < row_ptr[i + 1]; j++) {
                const uint32_t c = col_idx[j];
                if (c < u0 || c >= u1) {
                    delete B;
                    return set_error(ctx, RSG_ERR_INVALID_ARG,
                                     "batch_create: row %u has column %u outside its system %u", i, c, s);
                }
                ci.push_back(p0 + (c - u0));
                val.push_back(values[j]);
            }
            rp[++prow] = uint32_t(ci.size());
        }
        for (uint32_t i = p0 + (u1 - u0); i < p1; i++) {
            ci.push_back(i);
            val.push_back(1.0);
            rp[++prow] = uint32_t(ci.size());
        }
    }
    sys_slice[n_sys] = uint32_t(pad_total / 32);
    rsg_status st = csr_create_ex(ctx, B->pad_rows, rp.data(), ci.data(), val.data(), RSG_MEM_HOST, 1, &B->A);
    if (st != RSG_OK) {
        delete B;
        return st;
    }
    if (!B->A->use_sell) {
        rsg_csr_destroy(ctx, B->A);
        delete B;
        return set_error(ctx, RSG_ERR_UNSUPPORTED, "batch_create: rows too uneven for the SELL-32 layout");
    }
    auto up = [&](uint32_t **d, const std::vector<uint32_t> &h) -> bool {
        return cudaMalloc(d, std::max<size_t>(h.size(), 1) * sizeof(uint32_t)) == cudaSuccess &&
               cudaMemcpy(*d, h.data(), h.size() * sizeof(uint32_t), cudaMemcpyHostToDevice) == cudaSuccess;
    };
    if (!up(&B->d_slice_sys, slice_sys) || !up(&B->d_sys_slice, sys_slice) || !up(&B->d_user2pad, map)) {
        rsg_batch_destroy(ctx, B);
        return set_error(ctx, RSG_ERR_OUT_OF_MEMORY, "batch_create: maps");
    }
    *out = B;
    return RSG_OK;
}

void rsg_batch_destroy(rsg_context *ctx, rsg_batch *B)
{
    if (!B) return;
    if (ctx) {
        cudaSetDevice(ctx->device);
        cudaStreamSynchronize(ctx->stream);
    }
    if (B->A) rsg_csr_destroy(ctx, B->A);
    cudaFree(B->d_slice_sys);
    cudaFree(B->d_sys_slice);
    cudaFree(B->d_user2pad);
    delete B;
}

rsg_status rsg_batch_info(const rsg_batch *B, uint32_t *n_sys, uint32_t *rows, uint32_t *padded_rows, uint64_t *nnz)
{
    if (!B) return RSG_ERR_INVALID_ARG;
    if (n_sys) *n_sys = B->n_sys;
    if (rows) *rows = B->user_rows;
    if (padded_rows) *padded_rows = B->pad_rows;
    if (nnz) *nnz = B->A->nnz;
    return RSG_OK;
}

rsg_status rsg_batch_solve(rsg_context *ctx, rsg_batch *B, const rsg_solver_conf *conf, int32_t prec_type,
                           const double *b, double *x, int32_t memory, rsg_stats *per_system, rsg_stats *summary)
{
    if (!ctx || !B || !conf || !b || !x) return set_error(ctx, RSG_ERR_INVALID_ARG, "batch_solve: null argument");
    if (conf->solver_type != RSG_SOLVER_CG)
        return set_error(ctx, RSG_ERR_UNSUPPORTED, "batch_solve: CG only");
    if (conf->stop_rule != RSG_STOP_TRUE_RELRES)
        return set_error(ctx, RSG_ERR_INVALID_ARG, "batch_solve: stop_rule must be TRUE_RELRES");
    if (prec_type != RSG_PREC_NONE && prec_type != RSG_PREC_JACOBI)
        return set_error(ctx, RSG_ERR_UNSUPPORTED, "batch_solve: preconditioner must be NONE or JACOBI");
    RSG_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    const bool mixed = conf->precision == RSG_PRECISION_MIXED;
    const uint32_t n = B->pad_rows, ns = B->n_sys, nsl = n / 32;
    const uint32_t max_it = std::max<uint32_t>(conf->n_outer, 1);
    const size_t vn = arena_bytes(n, sizeof(double)), vf = arena_bytes(n, sizeof(float));
    size_t bytes = 8 * vn + arena_bytes(batch_parts(nsl, ns) * 3, sizeof(double)) + arena_bytes(ns, sizeof(CgState)) +
                   arena_bytes(ns, sizeof(unsigned int)) +
                   3 * arena_bytes(1, sizeof(ListHead)) + 3 * arena_bytes(ns, sizeof(uint4)) +
                   arena_bytes(ns, sizeof(double)) + arena_bytes(1, sizeof(BatchCtl)) + 2 * arena_bytes(B->user_rows, 8);
    if (mixed) bytes += 7 * vf;
    RSG_TRY(arena_reserve(ctx, bytes));
    double *bp = arena_take<double>(ctx, n), *xp = arena_take<double>(ctx, n), *r = arena_take<double>(ctx, n),
           *z = arena_take<double>(ctx, n), *p0 = arena_take<double>(ctx, n), *p1 = arena_take<double>(ctx, n),
           *q = arena_take<double>(ctx, n), *d = arena_take<double>(ctx, n);
    Sums T = {};
    T.part = arena_take<double>(ctx, batch_parts(nsl, ns) * 3);
    T.ticket = arena_take<unsigned int>(ctx, ns);
    CgState *S = arena_take<CgState>(ctx, ns);
    double *relres = T.relres = arena_take<double>(ctx, ns);
    BatchCtl *ctl = arena_take<BatchCtl>(ctx, 1);
    Active L_all, L_act, L_chk;  // every system; the active ones; those that asked for a check (bk_list)
    for (Active *l : {&L_all, &L_act, &L_chk}) {
        l->head = arena_take<ListHead>(ctx, 1);
        l->entry = arena_take<uint4>(ctx, ns);
    }
    double *bu = memory == RSG_MEM_HOST ? arena_take<double>(ctx, B->user_rows) : const_cast<double *>(b);
    double *xu = memory == RSG_MEM_HOST ? arena_take<double>(ctx, B->user_rows) : x;
    float *r32 = nullptr, *z32 = nullptr, *pa = nullptr, *pb = nullptr, *q32 = nullptr, *y32 = nullptr, *d32 = nullptr;
    if (mixed) {
        r32 = arena_take<float>(ctx, n);
        z32 = arena_take<float>(ctx, n);
        pa = arena_take<float>(ctx, n);
        pb = arena_take<float>(ctx, n);
        q32 = arena_take<float>(ctx, n);
        y32 = arena_take<float>(ctx, n);
        d32 = arena_take<float>(ctx, n);
    }
    cudaStream_t sm = ctx->stream;
    const auto t0 = std::chrono::steady_clock::now();
    if (memory == RSG_MEM_HOST) {
        RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(bu, b, size_t(B->user_rows) * 8, cudaMemcpyHostToDevice, sm));
        RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(xu, x, size_t(B->user_rows) * 8, cudaMemcpyHostToDevice, sm));
    }
    RSG_CHECK_CUDA(ctx, cudaMemsetAsync(bp, 0, size_t(n) * 8, sm));
    RSG_CHECK_CUDA(ctx, cudaMemsetAsync(xp, 0, size_t(n) * 8, sm));
    RSG_CHECK_CUDA(ctx, cudaMemsetAsync(p0, 0, size_t(n) * 8, sm));
    RSG_CHECK_CUDA(ctx, cudaMemsetAsync(p1, 0, size_t(n) * 8, sm));
    if (mixed) {
        RSG_CHECK_CUDA(ctx, cudaMemsetAsync(pa, 0, size_t(n) * 4, sm));
        RSG_CHECK_CUDA(ctx, cudaMemsetAsync(pb, 0, size_t(n) * 4, sm));
        RSG_CHECK_CUDA(ctx, cudaMemsetAsync(y32, 0, size_t(n) * 4, sm));
    }
    const int gu = std::min(grid_for(ctx, (const void *)bk_scatter, kBlock, 0, B->user_rows), kMaxGrid);
    bk_scatter<<<gu, kBlock, 0, sm>>>(B->user_rows, B->d_user2pad, bu, bp);
    bk_scatter<<<gu, kBlock, 0, sm>>>(B->user_rows, B->d_user2pad, xu, xp);
    const bool jac = prec_type == RSG_PREC_JACOBI;
    if (jac) {
        RSG_TRY(jacobi_build(ctx, B->A, d));
        if (mixed) {
            const int gv = std::min(grid_for(ctx, (const void *)bk_to_f32, kBlock, 0, n), kMaxGrid);
            bk_to_f32<<<gv, kBlock, 0, sm>>>(n, d, d32);
        }
    }
    // per-system state
    {
        CgState h;
        std::memset(&h, 0, sizeof(h));
        // no equation scaling here (each system keeps its own magnitude), so the
        // reference's p^T A p clamp, calibrated for scaled equations, is off
        h.eps = 0.0;
        h.cvg = conf->cvg;
        h.rtol = conf->rtol;
        h.delta = conf->reliable_delta > 0.0 && conf->reliable_delta < 1.0 ? conf->reliable_delta : kReliableDelta;
        h.sigma = 1.0;
        h.max_it = max_it;
        h.stop_rule = RSG_STOP_TRUE_RELRES;
        std::vector<CgState> hs(ns, h);
        RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(S, hs.data(), ns * sizeof(CgState), cudaMemcpyHostToDevice, sm));
        BatchCtl c = {0, body_limit_for(max_it), 0, 1, 0};
        RSG_CHECK_CUDA(ctx, cudaMemsetAsync(T.ticket, 0, ns * sizeof(unsigned int), sm));
        RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(ctl, &c, sizeof(c), cudaMemcpyHostToDevice, sm));
        // the lists start with every system
        std::vector<uint4> entry(ns);
        uint32_t chunks = 0;
        for (uint32_t i = 0; i < ns; i++) {
            const uint32_t first = B->pad_begin[i] / 32;
            entry[i] = list_entry(i, chunks, first, B->pad_begin[i + 1] / 32 - first);
            chunks = entry[i].z;
        }
        const ListHead head = {ns, chunks};
        for (const Active *l : {&L_all, &L_act, &L_chk}) {
            RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(l->head, &head, sizeof(head), cudaMemcpyHostToDevice, sm));
            RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(l->entry, entry.data(), ns * sizeof(uint4), cudaMemcpyHostToDevice, sm));
        }
        RSG_CHECK_CUDA(ctx, cudaStreamSynchronize(sm));
    }
    const BView V{B->d_slice_sys, B->d_sys_slice, nsl, ns};
    const Sell<double> M64 = sell_view<double>(B->A);
    const Sell<float> M32 = sell_view<float>(B->A);
    const int g_tuned = B->tuned ? (mixed ? B->g32 : B->g64) : 0;
    const int g = g_tuned > 0
                      ? g_tuned
                      : std::min(grid_for(ctx,
                                          mixed ? (const void *)bk_dir<float, true> : (const void *)bk_dir<double, false>,
                                          kBlock, 0, (long long)nsl * 32),
                                 kMaxGrid);
    cudaEventRecord(ctx->ev[0], sm);
    bk_init_res<<<g, kBlock, 0, sm>>>(M64, V, L_all, bp, xp, r, T, S);
    if (mixed)
        bk_init_z<true><<<g, kBlock, 0, sm>>>(V, L_all, n, jac ? d : nullptr, jac ? d32 : nullptr, r, z, r32, z32, T, S);
    else
        bk_init_z<false><<<g, kBlock, 0, sm>>>(V, L_all, n, jac ? d : nullptr, nullptr, r, z, r32, z32, T, S);
    RSG_CHECK_CUDA(ctx, cudaGetLastError());

    auto body = [&](cudaGraphConditionalHandle h, int use_cond, bool pdl, int iterations) {
        for (int it = 0; it < iterations; it++) {
            if (!mixed) {
                launch_k(sm, pdl, bk_dir<double, false>, g, kBlock, 0, M64, V, L_act, z, p0, p1, q, xp,
                         (float *)nullptr, T, S);
                launch_k(sm, pdl, bk_update<double, false>, g, kBlock, 0, V, L_act, n, jac ? d : (double *)nullptr, p0,
                         p1, q, xp, r, z, T, S);
            } else {
                launch_k(sm, pdl, bk_dir<float, true>, g, kBlock, 0, M32, V, L_act, z32, pa, pb, q32, xp, y32, T, S);
                launch_k(sm, pdl, bk_update<float, true>, g, kBlock, 0, V, L_act, n, jac ? d32 : (float *)nullptr, pa, pb,
                         q32, y32, r32, z32, T, S);
            }
        }
        launch_k(sm, pdl, bk_list, 1, kBlock, 0, S, B->d_sys_slice, L_act, L_chk);
        if (!mixed)
            launch_k(sm, pdl, bk_check<false>, g, kBlock, 0, M64, V, L_chk, jac ? d : (double *)nullptr, (float *)nullptr,
                     bp, xp, (float *)nullptr, r, z, (float *)nullptr, (float *)nullptr, T, S);
        else
            launch_k(sm, pdl, bk_check<true>, g, kBlock, 0, M64, V, L_chk, (double *)nullptr, jac ? d32 : (float *)nullptr,
                     bp, xp, y32, r, z, r32, z32, T, S);
        launch_k(sm, pdl, bk_tail, 1, kBlock, 0, S, B->d_sys_slice, ns, L_act, ctl, h, use_cond, iterations);
    };
    const bool pdl = pdl_for(B->A, mixed);

    if (conf->use_graph) {
        int iterations = kBatchIterations;  // of a body, or one (kCutBodies)
        int32_t *keep = reinterpret_cast<int32_t *>(ctx->pinned);
        do {
            cudaGraph_t graph = nullptr;
            cudaGraphExec_t exec = nullptr;
            RSG_TRY(while_graph(ctx, pdl, [&](cudaGraphConditionalHandle h, bool with_pdl) {
                body(h, 1, with_pdl, iterations);
            }, &graph, &exec));
            cudaError_t e = cudaGraphLaunch(exec, sm);
            if (e == cudaSuccess) e = cudaMemcpyAsync(keep, &ctl->keep, sizeof(int32_t), cudaMemcpyDeviceToHost, sm);
            const cudaError_t sync = cudaStreamSynchronize(sm);
            cudaGraphExecDestroy(exec);
            cudaGraphDestroy(graph);
            if (e == cudaSuccess) e = sync;
            if (e != cudaSuccess) return set_error(ctx, RSG_ERR_CUDA, "batch solve: %s", cudaGetErrorString(e));
            iterations = 1;
        } while (*keep);
    } else {
        const uint32_t polls = std::max<uint32_t>(1, conf->check_interval / kBatchIterations);
        int32_t *keep = reinterpret_cast<int32_t *>(ctx->pinned);
        for (;;) {
            for (uint32_t k = 0; k < polls; k++) body(0, 0, pdl, kBatchIterations);
            RSG_CHECK_CUDA(ctx, cudaGetLastError());
            RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(keep, &ctl->keep, sizeof(int32_t), cudaMemcpyDeviceToHost, sm));
            RSG_CHECK_CUDA(ctx, cudaStreamSynchronize(sm));
            if (!*keep) break;
        }
    }
    if (mixed) bk_fold<<<g, kBlock, 0, sm>>>(V, n, xp, y32, S);
    bk_true_res<<<g, kBlock, 0, sm>>>(M64, V, L_all, bp, xp, T, S);
    cudaEventRecord(ctx->ev[1], sm);
    bk_gather<<<gu, kBlock, 0, sm>>>(B->user_rows, B->d_user2pad, xp, xu);
    if (memory == RSG_MEM_HOST)
        RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(x, xu, size_t(B->user_rows) * 8, cudaMemcpyDeviceToHost, sm));
    std::vector<CgState> hs(ns);
    std::vector<double> rr(ns);
    BatchCtl hc;
    RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(hs.data(), S, ns * sizeof(CgState), cudaMemcpyDeviceToHost, sm));
    RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(rr.data(), relres, ns * sizeof(double), cudaMemcpyDeviceToHost, sm));
    RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(&hc, ctl, sizeof(hc), cudaMemcpyDeviceToHost, sm));
    RSG_CHECK_CUDA(ctx, cudaStreamSynchronize(sm));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
    rsg_stats sum;
    std::memset(&sum, 0, sizeof(sum));
    sum.converged = 1;
    rsg_status worst = RSG_OK;
    for (uint32_t s = 0; s < ns; s++) {
        rsg_stats st;
        std::memset(&st, 0, sizeof(st));
        st.iterations = hs[s].it;
        st.outer = hs[s].n_updates;
        st.error = hs[s].error;
        st.true_relres = rr[s];
        st.norm_b = hs[s].bn;
        st.converged = hs[s].converged;
        st.status = hs[s].ticket[7] ? RSG_ERR_TIMEOUT : hs[s].status;
        if (hs[s].done == 0) st.status = RSG_NOT_CONVERGED;
        if (per_system) per_system[s] = st;
        sum.iterations = std::max(sum.iterations, st.iterations);
        sum.outer += st.outer;
        sum.true_relres = std::max(sum.true_relres, st.true_relres);
        sum.converged &= st.converged;
        if (st.status != RSG_OK && (worst == RSG_OK || st.status < 0)) worst = rsg_status(st.status);
    }
    if (hc.timeout) worst = RSG_ERR_TIMEOUT;
    sum.status = worst;
    sum.seconds_solve = ms * 1e-3;
    sum.seconds_setup =
        std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() - sum.seconds_solve;
    if (summary) *summary = sum;
    if (worst == RSG_ERR_TIMEOUT) return set_error(ctx, RSG_ERR_TIMEOUT, "batch solve hit its hard limit");
    return worst;
}


// Batch autotuner (no reference counterpart): the grid of the slice kernels (direction,
// update, check) is chosen per precision by timing short fixed-length batch solves
// (every system runs kTuneIters iterations: rtol 0 is never met) for the built-in
// default and multiples of the SM count; three solves per candidate, median.
rsg_status rsg_batch_autotune(rsg_context *ctx, rsg_batch *B, rsg_tune_info *out)
{
    if (!ctx || !B) return set_error(ctx, RSG_ERR_INVALID_ARG, "batch_autotune: bad arguments");
    RSG_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    constexpr uint32_t kTuneIters = 32;
    constexpr int kReps = 3;
    const size_t nu = B->user_rows;
    double *b = nullptr, *x = nullptr;
    if (cudaMalloc(&b, nu * sizeof(double)) != cudaSuccess || cudaMalloc(&x, nu * sizeof(double)) != cudaSuccess) {
        cudaFree(b);
        return set_error(ctx, RSG_ERR_OUT_OF_MEMORY, "batch_autotune: vectors");
    }
    std::vector<double> ones(nu, 1.0);
    rsg_status s = RSG_OK;
    if (cudaMemcpy(b, ones.data(), nu * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
        s = set_error(ctx, RSG_ERR_CUDA, "batch_autotune: upload");
    rsg_solver_conf c;
    rsg_conf_default(&c);
    c.n_outer = kTuneIters;
    c.stop_rule = RSG_STOP_TRUE_RELRES;
    c.rtol = 0.0;
    const uint32_t nsl = B->A->n_slices;
    std::vector<int> cand = {0};
    for (int k : {1, 2, 3, 4, 6, 8}) cand.push_back(k * ctx->num_sms);
    cand.push_back(int(std::min<long long>(((long long)nsl * 32 + kBlock - 1) / kBlock, (long long)kMaxGrid)));
    B->tuned = true;
    uint32_t count = 0;
    for (int32_t prec : {RSG_PRECISION_FP64, RSG_PRECISION_MIXED}) {
        if (s != RSG_OK) break;
        c.precision = prec;
        int32_t &gsel = prec == RSG_PRECISION_FP64 ? B->g64 : B->g32;
        double best = 1e300, def = 0;
        int bestg = 0;
        for (int gc : cand) {
            gsel = gc;
            double t[kReps];
            for (int r = 0; r < kReps && s == RSG_OK; r++) {
                if (cudaMemsetAsync(x, 0, nu * sizeof(double), ctx->stream) != cudaSuccess) {
                    s = set_error(ctx, RSG_ERR_CUDA, "batch_autotune: memset");
                    break;
                }
                rsg_stats sum;
                const rsg_status rs = rsg_batch_solve(ctx, B, &c, RSG_PREC_JACOBI, b, x, RSG_MEM_DEVICE, nullptr, &sum);
                if (rs < 0) {
                    s = rs;
                    break;
                }
                t[r] = sum.seconds_solve / double(std::max<uint32_t>(sum.iterations, 1));
                count++;
            }
            if (s != RSG_OK) break;
            std::sort(t, t + kReps);
            const double tm = t[kReps / 2];
            if (gc == 0) def = tm;
            if (tm < best) {
                best = tm;
                bestg = gc;
            }
        }
        gsel = bestg;
        (prec == RSG_PRECISION_FP64 ? B->it64 : B->it32) = best;
        (prec == RSG_PRECISION_FP64 ? B->it64_default : B->it32_default) = def;
    }
    cudaStreamSynchronize(ctx->stream);
    cudaFree(b);
    cudaFree(x);
    if (s != RSG_OK) {
        B->tuned = false;
        B->g64 = B->g32 = 0;
        return s;
    }
    B->tune_candidates = count;
    if (out) {
        std::memset(out, 0, sizeof(*out));
        out->tuned = 1;
        out->format = 1;
        out->rows_per_warp = 32;
        out->grid_dir_fp64 = out->grid_update_fp64 = uint32_t(B->g64);
        out->grid_dir_fp32 = out->grid_update_fp32 = uint32_t(B->g32);
        out->seconds_iter_fp64 = B->it64;
        out->seconds_iter_fp32 = B->it32;
        out->seconds_iter_fp64_default = B->it64_default;
        out->seconds_iter_fp32_default = B->it32_default;
        out->candidates = count;
    }
    return RSG_OK;
}

}  // extern "C"
