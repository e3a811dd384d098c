// The CG loop of a small system with its matrix resident in shared memory.
//
// A CG iteration on a few thousand rows is latency: in the persistent loop of cg_persist.cu every
// phase walks slice pointers, matrix, gathers, partials and a grid barrier through L2 -- 12.8 us per
// FP64 iteration at 8k rows, for 2 MB of traffic.  Here each CTA keeps its rows of the matrix, its
// window of p and its part of x and r on the SM for the whole loop:
//
//   rows      CTA c owns a contiguous range of rows (whole update units, see below) and, as columns reach
//             at most `band` rows away, reads p only in a window around it;
//   p         p = z + beta p is formed once per iteration for the whole window, in shared memory (the
//             other loops form it for every gathered column);
//   A p       one thread per row over the SELL-32 values in shared memory;
//   update    x, r and d of a row pair (FP64) or quadruple (FP32) stay in one thread's registers;
//   exchange  per iteration only z (to the CTAs whose window holds it) and one partial sum per warp.
//
// Two transports.  CLUSTER: up to 16 CTAs of one thread-block cluster; z and the sums are written into
// the other CTAs' shared memory, the phases are separated by the hardware cluster barrier.  Otherwise
// one CTA per SM (cooperative launch), z and the sums through L2 and the grid barrier of grid_sync.cuh.
//
// Same results bit for bit as the graph loop (cg.cu): a warp's row products, pairs and quadruples are
// those of a warp of the kernel it replaces, each warp sum is exchanged, and every CTA adds them in the
// order of the graph kernels' block and grid reductions -- which needs grids with one slice and at most
// one pair (quadruple) per thread, checked by the launcher.  Every CTA applies the same state
// transitions (krylov.cuh) to its own copy of the state, so all take the same decisions.
//
// Bound by dependent latencies (cycles of one FP64 iteration at 8k rows, 15 CTAs, about 10,400 = 5.3 us:
// window 600, products 3000, reductions' trees 950 + 1400 of 40-cycle additions, update with its division
// 1700, two cluster barriers 2600).  Per iteration, Jacobi, heat cubes, us: persistent loop -> this one
//   cluster     567 rows FP64 17.6 (graph; ragged slices) -> 3.4; 1.9k FP64 -> 3.5, mixed -> 3.7;
//               8.4k FP64 12.8 -> 5.6; 16k mixed -> 6.4
//   CTA per SM  16k FP64 -> 7.0; 37k FP64 -> 8.4, mixed -> 7.3; 64k mixed 13.8 -> 10; 113k FP64 -> 12.1,
//               mixed -> 9.7
// Rows per CTA of a cluster: 192 gives 3.4 / 3.5 us at 567 / 1.9k rows, 384 3.7 / 3.9, 576 4.4 / 4.3.
// Storing warp sums to the other CTAs one by one or gathered into runs first made no difference.
#include "grid_sync.cuh"
#include "krylov.cuh"

#include <algorithm>

namespace rsg {
namespace {

constexpr uint32_t kMaxCluster = 16;
constexpr uint32_t kResidentThreads = 640;   // most threads of a CTA (96 registers each)
constexpr size_t kResidentSmem = 224 * 1024;

struct ResArgs {
    Sell<double> S64;
    Sell<float> S32;
    uint32_t n, band, ctas, win_max;
    const double *b, *d;
    const float *d32;
    double *x, *r, *z;
    float *r32, *z32, *y32;
    double *ws;           // grid transport: warp sums (dir, update, check)
    double *left;         // grid transport: the leftover rows' p and q
    CgState *st;
    unsigned int *bar, *err;
    // byte offsets in shared memory
    uint32_t o_off, o_p, o_z, o_q, o_len, o_base, o_ws, o_left;
};

// Rows of an update warp: 32 pairs (FP64) or 32 quadruples (FP32).
template <bool MIXED>
__host__ __device__ constexpr uint32_t unit_rows() { return MIXED ? 128u : 64u; }

__host__ __device__ inline uint32_t first_row(uint32_t n, uint32_t unit, uint32_t ctas, uint32_t c)
{
    const uint32_t units = (n + unit - 1) / unit;
    return uint32_t(uint64_t(units) * c / ctas) * unit;
}
// Window of the rows [rb, re): whole groups of four rows.
__host__ __device__ inline uint32_t win_lo(uint32_t rb, uint32_t band) { return (rb > band ? rb - band : 0u) & ~3u; }
__host__ __device__ inline uint32_t win_hi(uint32_t n, uint32_t re, uint32_t band)
{
    return ((re + band < n ? re + band : n) + 3u) & ~3u;
}

__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster(uint32_t a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster_vec(uint32_t a, const double (&v)[2])
{
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v[0]), "d"(v[1]) : "memory");
}
__device__ __forceinline__ void st_cluster_vec(uint32_t a, const float (&v)[4])
{
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3])
                 : "memory");
}
__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Four consecutive elements of a row: FP64 values as two 16-byte halves in separate 512-byte runs (the
// global layout's 32 bytes per lane would put lanes four apart on the same banks).
__device__ __forceinline__ void lds4(const double *v, uint32_t e, uint32_t lane, double (&o)[4])
{
    const double2 a = *reinterpret_cast<const double2 *>(v + e + lane * 2);
    const double2 b = *reinterpret_cast<const double2 *>(v + e + 64 + lane * 2);
    o[0] = a.x;
    o[1] = a.y;
    o[2] = b.x;
    o[3] = b.y;
}
__device__ __forceinline__ void lds4(const float *v, uint32_t e, uint32_t lane, float (&o)[4])
{
    const float4 a = *reinterpret_cast<const float4 *>(v + e + lane * 4);
    o[0] = a.x;
    o[1] = a.y;
    o[2] = a.z;
    o[3] = a.w;
}
__device__ __forceinline__ uint32_t smem_slot(const double *, uint32_t e)
{
    return (e & ~127u) | ((e & 2u) << 5) | ((e & 124u) >> 1) | (e & 1u);
}
__device__ __forceinline__ uint32_t smem_slot(const float *, uint32_t e) { return e; }

__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }

// The graph kernels' grid reduction over warp sums ws[k * pitch + w] (pitch: a multiple of 8, zeros past
// the last warp): blocks of eight warps (block_sum's tree), then thread b of a 256-thread block adds blocks
// b, b + 256, ... and block_sum adds the threads.  Levels that would only add zeros are skipped (x + 0 = x):
// a dependent FP64 addition costs about 40 cycles.  COH: the sums come from other CTAs through L2 -- every
// CTA reads the same few lines at the same moment, so they are read once each, coalesced, and the blocks'
// tree runs on shuffles into `blk`.  Valid in every thread; `shw` (NV * 8) may be reused after the next
// __syncthreads.
template <int NV, bool COH>
__device__ __forceinline__ void tree_sum(const double *ws, uint32_t pitch, double *blk, double *shw,
                                         double (&total)[NV])
{
    const uint32_t blocks = pitch / 8, warp = threadIdx.x >> 5;
    if constexpr (COH) {
        constexpr int M = NV == 1 ? 8 : 4;  // loads per thread in flight
        for (uint32_t t0 = warp * 32; t0 < pitch; t0 += M * blockDim.x) {
            double v[M][NV];
#pragma unroll
            for (int i = 0; i < M; i++) {
                const uint32_t t = t0 + i * blockDim.x + (threadIdx.x & 31);
#pragma unroll
                for (int k = 0; k < NV; k++) v[i][k] = t < pitch ? __ldcg(ws + size_t(k) * pitch + t) : 0.0;
            }
#pragma unroll
            for (int i = 0; i < M; i++) {
                if (t0 + i * blockDim.x >= pitch) break;
#pragma unroll
                for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                    for (int k = 0; k < NV; k++) v[i][k] += __shfl_xor_sync(0xffffffffu, v[i][k], o);
                const uint32_t t = t0 + i * blockDim.x + (threadIdx.x & 31);
                if ((t & 7) == 0 && t < pitch)
#pragma unroll
                    for (int k = 0; k < NV; k++) blk[k * blocks + t / 8] = v[i][k];
            }
        }
        __syncthreads();
    }
    if (warp < kWarpsPerBlock && warp * 32 < blocks) {
        double acc[NV];
#pragma unroll
        for (int k = 0; k < NV; k++) acc[k] = 0.0;
        for (uint32_t b = threadIdx.x; b < blocks; b += kBlock) {
            if constexpr (COH) {
#pragma unroll
                for (int k = 0; k < NV; k++) acc[k] += blk[k * blocks + b];
            } else {
#pragma unroll
                for (int k = 0; k < NV; k++) {
                    const double2 *p = reinterpret_cast<const double2 *>(ws + size_t(k) * pitch + 8 * b);
                    const double2 w0 = p[0], w2 = p[1], w4 = p[2], w6 = p[3];
                    acc[k] += ((w0.x + w4.x) + (w2.x + w6.x)) + ((w0.y + w4.y) + (w2.y + w6.y));
                }
            }
        }
#pragma unroll
        for (uint32_t o = 16; o > 0; o >>= 1)
            if (o < blocks)
#pragma unroll
                for (int k = 0; k < NV; k++) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], int(o));
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int k = 0; k < NV; k++) shw[k * 8 + warp] = acc[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) {
        const double *w = shw + k * 8;  // warps past the last block left theirs at zero
        if (blocks <= 32) total[k] = w[0];
        else if (blocks <= 64) total[k] = w[0] + w[1];
        else total[k] = ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
    }
}

template <bool MIXED, int PK, bool CLUSTER>
__global__ void __launch_bounds__(kResidentThreads) k_cg_resident(ResArgs a)
{
    using T = typename std::conditional<MIXED, float, double>::type;
    constexpr uint32_t U = unit_rows<MIXED>();
    constexpr int N = MIXED ? 4 : 2;     // rows per update thread
    constexpr int NU = MIXED ? 2 : 3;    // sums of the update
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ CgState s;
    __shared__ double shw[2][24];
    __shared__ uint32_t win0[kMaxCluster];

    T *val = reinterpret_cast<T *>(smem);
    int16_t *off = reinterpret_cast<int16_t *>(smem + a.o_off);
    T *pbuf = reinterpret_cast<T *>(smem + a.o_p), *zw = reinterpret_cast<T *>(smem + a.o_z);
    T *q = reinterpret_cast<T *>(smem + a.o_q);
    uint16_t *rlen = reinterpret_cast<uint16_t *>(smem + a.o_len);
    uint32_t *sbase = reinterpret_cast<uint32_t *>(smem + a.o_base);  // first element of each slice (and the end)
    const uint32_t n = a.n, tid = threadIdx.x, lane = tid & 31u, cta = blockIdx.x;
    const uint32_t n_slices = (n + 31) / 32, n_units = (n + U - 1) / U;
    const uint32_t pitch_s = (n_slices + 7) & ~7u, pitch_u = (n_units + 7) & ~7u;
    double *wsA = CLUSTER ? reinterpret_cast<double *>(smem + a.o_ws) : a.ws;
    double *wsB = wsA + pitch_s, *wsC = wsB + size_t(NU) * pitch_u;
    double *blk = reinterpret_cast<double *>(smem + a.o_ws);  // the other transport's block sums
    T *left = CLUSTER ? reinterpret_cast<T *>(smem + a.o_left) : reinterpret_cast<T *>(a.left);
    const uint32_t rb = first_row(n, U, a.ctas, cta), re = min(n, first_row(n, U, a.ctas, cta + 1));
    const uint32_t lo = win_lo(rb, a.band), hi = win_hi(n, re, a.band);
    const T *zg = MIXED ? reinterpret_cast<const T *>(a.z32) : reinterpret_cast<const T *>(a.z);
    const uint32_t s0 = rb / 32, s1 = (re + 31) / 32, win = hi - lo;
    // The last warp advances the state; the others (`workers` threads) hold rows, pairs and the window.
    const uint32_t workers = blockDim.x - 32;
    const bool chief = tid == workers;

    // ---- load: matrix, window ----
    {
        const uint32_t e0 = a.S64.slice_ptr[s0], e1 = a.S64.slice_ptr[s1];
        const T *gv = MIXED ? reinterpret_cast<const T *>(a.S32.val) : reinterpret_cast<const T *>(a.S64.val);
        for (uint32_t e = tid; e < e1 - e0; e += blockDim.x) {
            val[smem_slot(val, e)] = gv[e0 + e];
            off[e] = a.S64.off[e0 + e];
        }
        for (uint32_t i = tid; i <= s1 - s0; i += blockDim.x) sbase[i] = a.S64.slice_ptr[s0 + i] - e0;
        for (uint32_t i = tid; i < re - rb; i += blockDim.x) rlen[i] = uint16_t(a.S64.rp[rb + i + 1] - a.S64.rp[rb + i]);
        for (uint32_t i = tid; i < win; i += blockDim.x) {
            pbuf[i] = T(0);
            if (CLUSTER) zw[i] = zg[lo + i];
        }
        if (CLUSTER || cta == 0) {  // the sums' padding (a.ws is shared by all CTAs)
            const uint32_t words = pitch_s + NU * pitch_u + 2 * pitch_s;
            for (uint32_t i = tid; i < words; i += blockDim.x) {
                const bool pad = i < pitch_s ? i >= n_slices
                                 : i < pitch_s + NU * pitch_u ? (i - pitch_s) % pitch_u >= n_units
                                                              : (i - pitch_s - NU * pitch_u) % pitch_s >= n_slices;
                if (pad) wsA[i] = 0.0;
            }
        }
        if (tid < 48) shw[tid / 24][tid % 24] = 0.0;
        if (tid < a.ctas && tid < kMaxCluster) win0[tid] = win_lo(first_row(n, U, a.ctas, tid), a.band);
        if (chief) {
            s = *a.st;
            if (cta != 0) {  // CTA 0 alone records the convergence history
                s.history = nullptr;
                s.trend_hist = nullptr;
            }
        }
    }
    // this thread's pair / quadruple of rows, and the CTAs whose windows hold it
    const uint32_t n_main = n / N * N;
    const bool has_vec = tid < workers && rb + (tid + 1) * N <= min(re, n_main);
    const uint32_t cta_units = (first_row(n, U, a.ctas, cta + 1) - rb) / U;  // update warps of this CTA
    // the n % N leftover rows belong to the first threads of CTA 0, as in k_cg_update / k_mx_update
    const bool has_left = cta == 0 && n_main + tid < n;
    const uint32_t vrow = rb + tid * N, lrow = n_main + tid;
    auto targets = [&](uint32_t row, uint32_t &c0, uint32_t &c1) {
        c0 = a.ctas;
        c1 = 0;
        for (uint32_t c = 0; c < a.ctas; c++) {
            const uint32_t cb = first_row(n, U, a.ctas, c), ce = min(n, first_row(n, U, a.ctas, c + 1));
            if (row >= win_lo(cb, a.band) && row < win_hi(n, ce, a.band)) {
                c0 = min(c0, c);
                c1 = c + 1;
            }
        }
    };
    uint32_t vc0 = 0, vc1 = 0, lc0 = 0, lc1 = 0;
    if (CLUSTER) {
        if (has_vec) targets(vrow, vc0, vc1);
        if (has_left) targets(lrow, lc0, lc1);
    }
    T rv[N], xv[N], dv[N], rl = T(0), xl = T(0), dl = T(1);  // xv: x (FP64) or y (FP32)
    const T *gr = MIXED ? reinterpret_cast<const T *>(a.r32) : reinterpret_cast<const T *>(a.r);
    T *gx = MIXED ? reinterpret_cast<T *>(a.y32) : reinterpret_cast<T *>(a.x);
    const T *gd = MIXED ? reinterpret_cast<const T *>(a.d32) : reinterpret_cast<const T *>(a.d);
#pragma unroll
    for (int e = 0; e < N; e++) {
        rv[e] = has_vec ? gr[vrow + e] : T(0);
        xv[e] = has_vec ? gx[vrow + e] : T(0);
        dv[e] = has_vec && PK == 1 ? gd[vrow + e] : T(1);
    }
    if (has_left) {
        rl = gr[lrow];
        xl = gx[lrow];
        if (PK == 1) dl = gd[lrow];
    }
    __syncthreads();
    if (CLUSTER) cluster_barrier();  // every CTA of the cluster runs before its shared memory is written

    unsigned int passed = 0;
    const uint32_t z_addr = uint32_t(__cvta_generic_to_shared(zw));
    auto put_sum = [&](double *ws, uint32_t slot, double v) {  // a warp sum (the same in every lane)
        if (CLUSTER) {
            if (lane < a.ctas) st_cluster(cluster_addr(uint32_t(__cvta_generic_to_shared(ws + slot)), lane), v);
        } else if (lane == 0) {
            ws[slot] = v;
        }
    };
    auto put_left = [&](uint32_t i, T v) {  // into CTA 0
        if (CLUSTER) st_cluster(cluster_addr(uint32_t(__cvta_generic_to_shared(left + i)), 0), v);
        else left[i] = v;
    };
    auto get_left = [&](uint32_t i) { return CLUSTER ? left[i] : __ldcg(left + i); };
    auto put_z = [&](uint32_t row, T v, uint32_t c0, uint32_t c1) {
        if (CLUSTER)
            for (uint32_t c = c0; c < c1; c++)
                st_cluster(cluster_addr(z_addr + (row - win0[c]) * uint32_t(sizeof(T)), c), v);
        else const_cast<T *>(zg)[row] = v;
    };
    auto barrier = [&]() -> bool {
        if (CLUSTER) {
            cluster_barrier();
            return true;
        }
        return grid_barrier_count(a.bar, a.err, passed);
    };
    // The loop runs ahead of its own stopping rule: the direction and the product of the next iteration
    // start as soon as beta is known, while the chief (one thread: two divisions, two square roots, about
    // 1000 cycles) decides whether there is a next iteration.  Nothing they write outlives a "no": p is
    // double-buffered, q and the sums are rewritten.
    int half = 0;  // the chief's: iterations so far, modulo the graph body's two
    auto end_of_iteration = [&]() {  // the graph's tail after each body of two iterations
        half ^= 1;
        if (half == 0) {
            const uint32_t bc = ++s.body_count;
            if (!s.done && bc >= s.body_limit) {
                s.done = 1;
                s.status = RSG_ERR_TIMEOUT;
            }
        }
    };
    // four consecutive z of the window; through L2, the first ZI groups of a thread are loaded as soon as
    // they are complete, before the sums that give beta
    auto z_group = [&](uint32_t i, T (&zz)[4]) {
        if constexpr (MIXED) {
            const float4 t = CLUSTER ? *reinterpret_cast<const float4 *>(zw + i)
                                     : __ldcg(reinterpret_cast<const float4 *>(zg + lo + i));
            zz[0] = t.x;
            zz[1] = t.y;
            zz[2] = t.z;
            zz[3] = t.w;
        } else {
            const double2 *src = reinterpret_cast<const double2 *>(CLUSTER ? zw + i : zg + lo + i);
            const double2 t = CLUSTER ? src[0] : __ldcg(src), u = CLUSTER ? src[1] : __ldcg(src + 1);
            zz[0] = t.x;
            zz[1] = t.y;
            zz[2] = u.x;
            zz[3] = u.y;
        }
    };
    constexpr int ZI = 3;
    T zr[ZI][4];
    auto load_z = [&]() {
        if (CLUSTER || tid >= workers) return;
#pragma unroll
        for (int j = 0; j < ZI; j++) {
            const uint32_t i = (tid + j * workers) * 4;
            if (i < win) z_group(i, zr[j]);
        }
    };
    load_z();
    bool ok = true, fold = false;
    double beta_d = s.beta;
    T *po = pbuf, *p = pbuf + a.win_max;
    for (;;) {
        // ---- p = z + beta p over the window; q = A p; p^T q (k_cg_dir / k_mx_dir) ----
        if (tid < workers) {
            if (MIXED && fold) {  // after a refresh the FP32 correction joins x
                const double inv_sigma = 1.0 / s.sigma;
                if (has_vec)
#pragma unroll
                    for (int e = 0; e < N; e++) {
                        a.x[vrow + e] = fma(double(xv[e]), inv_sigma, a.x[vrow + e]);
                        xv[e] = T(0);
                    }
                if (has_left) {
                    a.x[lrow] = fma(double(xl), inv_sigma, a.x[lrow]);
                    xl = T(0);
                }
            }
            const T beta = T(beta_d);
            uint32_t i = tid * 4;
            if constexpr (!CLUSTER) {
#pragma unroll
                for (int j = 0; j < ZI; j++, i += workers * 4)
                    if (i < win)
#pragma unroll
                        for (int e = 0; e < 4; e++) p[i + e] = fma_t(beta, po[i + e], zr[j][e]);
            }
            for (; i < win; i += workers * 4) {
                T zz[4];
                z_group(i, zz);
#pragma unroll
                for (int e = 0; e < 4; e++) p[i + e] = fma_t(beta, po[i + e], zz[e]);
            }
            asm volatile("bar.sync 1, %0;" ::"r"(workers) : "memory");  // the workers only
            for (uint32_t i0 = tid & ~31u; i0 < re - rb; i0 += workers) {
                const uint32_t i = i0 + lane, row = rb + i;
                const bool valid = row < re;
                const uint32_t len = valid ? rlen[i] : 0u;
                const uint32_t b0 = sbase[i >> 5], g4 = (sbase[(i >> 5) + 1] - b0) >> 7;
                const T *pw = p + (row & ~31u) - lo;
                T v = T(0);
#pragma unroll 4
                for (uint32_t g = 0; g < g4; g++) {
                    T m[4];
                    lds4(val, b0 + g * 128, lane, m);
                    const short4 o = *reinterpret_cast<const short4 *>(off + b0 + g * 128 + lane * 4);
                    const int c[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                    for (int t = 0; t < 4; t++)
                        if (4u * g + t < len) v = row_acc(v, m[t], pw[c[t]]);
                }
                const T pr = valid ? p[row - lo] : T(0);
                double w = 0.0;
                if constexpr (MIXED) {
                    Dot2 pq;
                    if (valid) pq.add_prod(pr, v);
                    w = pq.value();
                } else {
                    if (valid) w += pr * v;
                }
                put_sum(wsA, s0 + (i >> 5), warp_sum(w));
                if (valid) {
                    q[i] = v;
                    if (row >= n_main) {
                        put_left(row - n_main, v);
                        put_left(4 + row - n_main, pr);
                    }
                }
            }
        }
        __syncthreads();
        if (s.done) break;

        // ---- true residual when the recurrence asked for it (k_cg_check / k_mx_check): rare, FP64 matrix
        //      and x from global memory; then the direction again ----
        if (s.need_check) {
            if (has_vec)
#pragma unroll
                for (int e = 0; e < N; e++) gx[vrow + e] = xv[e];
            if (has_left) gx[lrow] = xl;
            if (!(ok = barrier())) break;
            const double sigma = s.sigma, inv_sigma = 1.0 / sigma;
            for (uint32_t sl = s0 + (tid >> 5); sl < s1; sl += blockDim.x >> 5) {
                const uint32_t row = sl * 32 + lane;
                const bool valid = row < re;
                double ax = 0.0, acc[2] = {0.0, 0.0};
                const uint32_t len = valid ? rlen[row - rb] : 0u, g4 = a.S64.slice_len4[sl];
                for (uint32_t g = 0; g < g4; g++) {
                    const size_t e = size_t(a.S64.slice_ptr[sl]) + size_t(g) * 128u + 4u * lane;
                    double v[4];
                    ld4(a.S64.val + e, v);
                    const short4 o = *reinterpret_cast<const short4 *>(a.S64.off + e);
                    const int c[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                    for (int t = 0; t < 4; t++)
                        if (4u * g + t < len) {
                            const uint32_t col = uint32_t(int(sl * 32) + c[t]);
                            const double xc = MIXED ? fma(double(__ldcg(gx + col)), inv_sigma, __ldcg(a.x + col))
                                                    : double(__ldcg(gx + col));
                            ax = row_acc(ax, v[t], xc);
                        }
                }
                if (valid) {
                    const double ri = a.b[row] - ax;
                    const T rt = MIXED ? T(ri * sigma) : T(ri);
                    const T zt = PK == 1 ? gd[row] * rt : rt;
                    acc[1] += ri * ri;
                    if constexpr (MIXED) {
                        Dot2 rz;
                        rz.add_prod(rt, zt);
                        acc[0] = rz.value();
                    } else {
                        acc[0] += rt * zt;
                    }
                    q[row - rb] = rt;
                    if (row >= n_main) put_left(8 + row - n_main, rt);
                    uint32_t c0 = 0, c1 = 0;
                    if (CLUSTER) targets(row, c0, c1);
                    put_z(row, zt, c0, c1);
                }
                put_sum(wsC, sl, warp_sum(acc[0]));
                put_sum(wsC, pitch_s + sl, warp_sum(acc[1]));
            }
            if (!(ok = barrier())) break;
            if (has_vec)
#pragma unroll
                for (int e = 0; e < N; e++) rv[e] = q[vrow - rb + e];
            if (has_left) rl = get_left(8 + tid);
            load_z();
            double tot[2];
            tree_sum<2, !CLUSTER>(wsC, pitch_s, blk, shw[0], tot);
            if (chief) {
                if constexpr (MIXED) finalize_check_mixed(&s, tot[0], sqrt(tot[1]));
                else finalize_check64(&s, tot[0], sqrt(tot[1]));
                end_of_iteration();
            }
            __syncthreads();
            if (s.done) break;
            beta_d = s.beta;
            fold = MIXED && s.fold;
            continue;
        }
        fold = false;
        if (!(ok = barrier())) break;

        // ---- alpha; x += alpha p, r -= alpha q, z = P r; r^T z, ||r||^2, ||x||^2 (k_cg_update / k_mx_update) ----
        {
            double tot[1];
            tree_sum<1, !CLUSTER>(wsA, pitch_s, blk, shw[0], tot);
            double pq = tot[0];
            if (MIXED) {
                if (pq == 0.0 || !isfinite(pq)) pq = (pq == 0.0) ? 1e-300 : pq;
            } else {
                pq = clamp_pq(pq, s.eps);
            }
            const double alpha_d = s.rho_new / pq;
            if (chief) {  // none of these is read before the next barrier
                s.pq = pq;
                s.rho = s.rho_new;
                s.alpha = alpha_d;
                s.fold = 0;
            }
            const T alpha = T(alpha_d);
            if ((tid >> 5) < cta_units) {  // whole warps
                double acc[3] = {0.0, 0.0, 0.0};
                Dot2 rz, rr;
                if (has_vec) {
                    T zv[N];
                    const uint32_t i = vrow - rb, w = vrow - lo;
#pragma unroll
                    for (int e = 0; e < N; e++) {
                        xv[e] = fma_t(alpha, p[w + e], xv[e]);
                        rv[e] = fma_t(-alpha, q[i + e], rv[e]);
                        zv[e] = PK == 1 ? dv[e] * rv[e] : rv[e];
                    }
                    if constexpr (CLUSTER) {
                        for (uint32_t c = vc0; c < vc1; c++)
                            st_cluster_vec(cluster_addr(z_addr + (vrow - win0[c]) * uint32_t(sizeof(T)), c), zv);
                    } else if constexpr (MIXED) {
                        *reinterpret_cast<float4 *>(a.z32 + vrow) = make_float4(zv[0], zv[1], zv[2], zv[3]);
                    } else {
                        *reinterpret_cast<double2 *>(a.z + vrow) = make_double2(zv[0], zv[1]);
                    }
                    if constexpr (MIXED) {
#pragma unroll
                        for (int e = 0; e < N; e++) rz.add_prod(rv[e], zv[e]);
#pragma unroll
                        for (int e = 0; e < N; e++) rr.add_prod(rv[e], rv[e]);
                    } else {
                        acc[0] += rv[0] * zv[0] + rv[1] * zv[1];
                        acc[1] += rv[0] * rv[0] + rv[1] * rv[1];
                        acc[2] += xv[0] * xv[0] + xv[1] * xv[1];
                    }
                }
                if (has_left) {
                    xl = fma_t(alpha, get_left(4 + tid), xl);
                    rl = fma_t(-alpha, get_left(tid), rl);
                    const T zl = PK == 1 ? dl * rl : rl;
                    put_z(lrow, zl, lc0, lc1);
                    if constexpr (MIXED) {
                        rz.add_prod(rl, zl);
                        rr.add_prod(rl, rl);
                    } else {
                        acc[0] += rl * zl;
                        acc[1] += rl * rl;
                        acc[2] += xl * xl;
                    }
                }
                if constexpr (MIXED) {
                    acc[0] = rz.value();
                    acc[1] = rr.value();
                }
                const uint32_t unit = rb / U + (tid >> 5);
#pragma unroll
                for (int k = 0; k < NU; k++) put_sum(wsB, k * pitch_u + unit, warp_sum(acc[k]));
            }
        }
        if (!(ok = barrier())) break;
        {
            load_z();
            double tot[NU];
            tree_sum<NU, !CLUSTER>(wsB, pitch_u, blk, shw[1], tot);
            beta_d = tot[0] / s.rho;  // as finalize_update64 / finalize_update_mixed, which leave rho alone
            if (chief) {
                if constexpr (MIXED) finalize_update_mixed(&s, tot[0], tot[1]);
                else finalize_update64(&s, tot[0], tot[1], tot[2]);
                if (s.done || !s.need_check) end_of_iteration();
            }
        }
        T *t = po;
        po = p;
        p = t;
    }
    if (has_vec)
#pragma unroll
        for (int e = 0; e < N; e++) gx[vrow + e] = xv[e];
    if (has_left) gx[lrow] = xl;
    if (chief) {
        if (!ok) {
            s.done = 1;
            s.status = RSG_ERR_TIMEOUT;
        } else if (half == 1) {
            ++s.body_count;  // the graph's tail of the body in which the loop ended
        }
        if (cta == 0) *a.st = s;
    }
    if (CLUSTER) cluster_barrier();  // no CTA leaves while another may still write to it
}

struct ResPlan {
    uint32_t ctas = 0, threads = 0;
    size_t smem = 0;
};

// Lays the CTAs' shared memory out for `ctas` CTAs; false when it does not fit.
template <bool MIXED>
bool plan_smem(const rsg_csr *A, uint32_t ctas, bool cluster, ResArgs &a, ResPlan &pl)
{
    constexpr uint32_t U = unit_rows<MIXED>();
    constexpr size_t sz = MIXED ? sizeof(float) : sizeof(double);
    const uint32_t n = A->n;
    uint32_t rows = 0, win = 0;
    for (uint32_t c = 0; c < ctas; c++) {
        const uint32_t rb = first_row(n, U, ctas, c), re = first_row(n, U, ctas, c + 1);
        rows = std::max(rows, re - rb);
        win = std::max(win, win_hi(n, std::min(n, re), A->band) - win_lo(rb, A->band));
    }
    const uint32_t per_thread = MIXED ? 4u : 2u;
    if (rows > (kResidentThreads - 32) * per_thread) return false;
    const size_t elems = size_t(rows / 32) * ((A->max_row + 3) / 4) * 128;
    const uint32_t n_slices = (n + 31) / 32, n_units = (n + U - 1) / U;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o += (bytes + 15) & ~size_t(15);
        return uint32_t(std::min<size_t>(at, 0xffffffffu));
    };
    take(elems * sz);
    a.o_off = take(elems * sizeof(int16_t));
    a.o_p = take(2 * size_t(win) * sz);
    a.win_max = win;
    a.o_z = take(cluster ? size_t(win) * sz : 0);
    a.o_q = take(size_t(rows) * sz);
    a.o_len = take(size_t(rows) * sizeof(uint16_t));
    a.o_base = take((size_t(rows) / 32 + 1) * sizeof(uint32_t));
    const size_t ps = (size_t(n_slices) + 7) & ~size_t(7), pu = (size_t(n_units) + 7) & ~size_t(7);
    a.o_ws = take((cluster ? 3 * (ps + pu) : std::max(2 * ps, 3 * pu) / 8) * sizeof(double));
    a.o_left = take(cluster ? 12 * sz : 0);
    pl.smem = o;
    pl.ctas = ctas;
    pl.threads = std::min(kResidentThreads, std::max<uint32_t>(kBlock, (rows + 31u) & ~31u) + 32u);
    a.ctas = ctas;
    return o <= kResidentSmem;
}

template <bool MIXED, int PK>
rsg_status run_resident(rsg_context *ctx, const CgArgs &cg, ResArgs &a, bool *ran)
{
    constexpr uint32_t U = unit_rows<MIXED>();
    const rsg_csr *A = cg.A;
    const uint32_t n = A->n, n_units = (n + U - 1) / U;
    ResPlan pl;
    // one cluster: CTAs of about kClusterRows rows, more where shared memory does not hold their rows
    constexpr uint32_t kClusterRows = 192;
    const uint32_t most = std::min(kMaxCluster, n_units);
    for (uint32_t c = std::min(most, (n + kClusterRows - 1) / kClusterRows); c <= most; c++) {
        if (!plan_smem<MIXED>(A, c, true, a, pl)) continue;
        auto k = k_cg_resident<MIXED, PK, true>;
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kResidentSmem));
        cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = c;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c);
        cfg.blockDim = dim3(pl.threads);
        cfg.dynamicSmemBytes = pl.smem;
        cfg.stream = ctx->stream;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) != cudaSuccess || clusters < 1) {
            (void)cudaGetLastError();
            continue;
        }
        if (cudaLaunchKernelEx(&cfg, k, a) != cudaSuccess) {
            (void)cudaGetLastError();
            return RSG_OK;
        }
        *ran = true;
        return RSG_OK;
    }
    // one CTA per SM
    if (!plan_smem<MIXED>(A, std::min(uint32_t(ctx->num_sms), n_units), false, a, pl)) return RSG_OK;
    const void *k = (const void *)k_cg_resident<MIXED, PK, false>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kResidentSmem));
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, int(pl.threads), pl.smem) != cudaSuccess ||
        per_sm < 1) {
        (void)cudaGetLastError();
        return RSG_OK;
    }
    void *args[] = {&a};
    if (cudaLaunchCooperativeKernel(k, dim3(pl.ctas), dim3(pl.threads), args, pl.smem, ctx->stream) != cudaSuccess) {
        (void)cudaGetLastError();
        return RSG_OK;
    }
    *ran = true;
    return RSG_OK;
}

}  // namespace

// Runs the loop of cg.cu's run_typed with the matrix resident in shared memory; *ran = false (and nothing
// launched) when the system or the grids do not allow it, and the caller takes another loop.
rsg_status cg_resident_run(rsg_context *ctx, const CgArgs &cg, int g_dir, int g_upd, int g_chk, bool *ran)
{
    *ran = false;
    const rsg_csr *A = cg.A;
    const int pk = cg.P.kind;
    const uint64_t n = A->n, n_slices = (n + 31) / 32;
    if ((pk != 0 && pk != 1) || !A->use_sell || !A->soff || A->max_row > 0xffffu) return RSG_OK;
    // the warp sums stand for the graph kernels' partials only with one slice, and at most one pair or
    // quadruple of rows, per thread of their grids
    if (uint64_t(g_dir) * kWarpsPerBlock < n_slices || uint64_t(g_chk) * kWarpsPerBlock < n_slices ||
        uint64_t(g_upd) * kBlock < (cg.mixed ? n / 4 : n / 2) || uint64_t(g_upd) * kBlock < 4)
        return RSG_OK;
    if (std::max(g_dir, std::max(g_upd, g_chk)) > kMaxGrid) return RSG_OK;
    double *ws = nullptr;
    unsigned int *bar = nullptr;
    RSG_TRY(persist_workspace(ctx, &ws, &bar));
    if (!ws || 6 * n_slices + 64 > size_t(6) * kMaxGrid) return RSG_OK;
    ResArgs a = {};
    a.S64 = sell_view<double>(A);
    a.S32 = sell_view<float>(A);
    a.n = A->n;
    a.band = A->band;
    a.b = cg.b;
    a.d = cg.P.d;
    a.d32 = cg.P.d32;
    a.x = cg.x;
    a.r = cg.r;
    a.z = cg.z;
    a.r32 = cg.r32;
    a.z32 = cg.z32;
    a.y32 = cg.y32;
    a.left = ws;
    a.ws = ws + 16;
    a.st = cg.st;
    a.bar = bar;
    a.err = ctx->errw;
    if (cg.mixed) return pk ? run_resident<true, 1>(ctx, cg, a, ran) : run_resident<true, 0>(ctx, cg, a, ran);
    return pk ? run_resident<false, 1>(ctx, cg, a, ran) : run_resident<false, 0>(ctx, cg, a, ran);
}

}  // namespace rsg
