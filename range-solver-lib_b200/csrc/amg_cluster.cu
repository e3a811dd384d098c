// The small coarse levels of the multilevel cycle in one thread-block cluster.
//
// From level 2 on (the second K-cycle level; 3.3k rows at 60^3) the cycle is a chain of a dozen kernels per
// visit, two visits per cycle, each kernel a handful of dependent round trips to L2 and the launch of the
// next: more than half of the preconditioner's time.  Here one
// cluster of 16 CTAs runs a whole visit (two flexible-CG steps preconditioned by the V-cycle over the
// levels below, the dense coarsest solve included) with those levels resident in its shared memory:
//
//   ownership  CTA c owns a contiguous range of every level's aggregates, and the rows of those aggregates;
//              its rows' entries (FP32 values, 16-bit columns) are packed per CTA when the hierarchy is
//              built and copied to shared memory while the preceding kernel still runs;
//   vectors    a CTA holds the gathered vectors over the window of columns that its rows reach; whoever
//              computes a value stores it into the windows of all CTAs that hold it (distributed shared
//              memory); the coarse correction goes to the aggregate's owner only;
//   phases     separated by the hardware cluster barrier (about 0.7 us for 16 CTAs).
//
// Every row, aggregate and dense product is added in the launched kernels' order (4 lanes per row, eight
// row slots per aggregate, ...), so the same bits.  The K-cycle's dot products are not: each CTA adds its
// rows' products (compensated, one row group of four lanes after another), then its warps, then the 16 CTAs
// in order.  The persistent kernel of amg.cu does the same where this one replaces launched kernels
// (CP_KC_DOTS2/3), so both give one result.  One smoothing sweep per side; other settings stay launched.
//
// What bounds it: at 60^3 a visit is about 60k cycles: 17 cluster barriers of 1 to 1.5k, the six passes over
// the first level's rows (3 to 5k each, bank conflicts of the gathers), the spreads.  The whole CG loop
// (mixed, tolerance 1e-10), launched -> this kernel: 20^3 2.66 -> 2.55 ms, 30^3 3.35 -> 2.85, 45^3 4.39 ->
// 3.90, 60^3 5.12 -> 4.45, 70^3 6.35 -> 5.64, 75^3 6.96 -> 6.13.
//
// Where the line lies (kAmgClusterRows): the launched kernels spread a level over all SMs, this one over 16,
// and a larger first level also leaves three smoothed levels before the dense one (80^3, 7.8k rows: 7.70
// against 7.73 ms; 85^3, 9.3k: 8.30 against 8.64; 100^3, 15k: 11.0 against 12.3).  So up to 7168 rows.
#include "amg.cuh"

#include <algorithm>
#include <cstring>
#include <vector>

namespace rsg {
namespace {

constexpr uint32_t C = kAmgClusterCtas;
constexpr int kClThreads = kAmgClusterThreads;
constexpr int kClChunk = 8;  // entries per lane in flight, as csr_row_dot of amg.cu
constexpr size_t kClSmem = 232448 - 1024;  // the largest CTA's shared memory less the kernel's own

// What one CTA owns of one level; offsets in bytes from the CTA's packed data.
struct ClDesc {
    uint32_t lo, hi;                // window of the level's rows that the CTA holds
    uint32_t nr, nI, I0;            // owned rows; owned aggregates (next-level rows I0 .. I0 + nI)
    uint32_t o_row, o_rptr, o_val, o_col, o_arow, o_la, o_dw, o_dwc, o_perm;
};
struct ClHead {
    ClDesc lv[kAmgMaxLevels];
    uint32_t o_inv, bytes;          // owned rows of the dense inverse; packed bytes in all
    uint32_t pad[2];
};

// The packed data's layout for CTA c from the extents of its rows (lo, hi, rows, entries per level).
__host__ __device__ inline void cl_layout(const AmgClusterMap &m, uint32_t c, const uint32_t *ext, ClHead &h)
{
    uint32_t o = uint32_t(sizeof(ClHead));
    auto take = [&](uint32_t bytes) {
        const uint32_t at = o;
        o += (bytes + 15u) & ~15u;
        return at;
    };
    for (uint32_t j = 0; j < m.nl; j++) {
        ClDesc &d = h.lv[j];
        const uint32_t *e = ext + (j * C + c) * 4;
        const uint32_t nc = m.n[j + 1];
        d.lo = e[0];
        d.hi = e[1];
        d.nr = e[2];
        d.I0 = uint32_t(uint64_t(nc) * c / C);
        d.nI = uint32_t(uint64_t(nc) * (c + 1) / C) - d.I0;
        d.o_row = take(d.nr * 2);  // less lo
        d.o_rptr = take((d.nr + 1) * 2);
        d.o_val = take(e[3] * 4);
        d.o_col = take(e[3] * 2);
        d.o_arow = take((d.nI + 1) * 4);
        d.o_la = take(d.nr * 2);
        d.o_dw = take(d.nr * 4);
        d.o_dwc = take(d.nI * 4);
        d.o_perm = take(d.nr * 2);
        if (j + 1 == m.nl) h.o_inv = take(d.nI * nc * 4);
    }
    h.bytes = o;
}

struct ClSrc {  // a level as the launched kernels see it
    uint32_t n, nc;
    const uint32_t *rp, *ci, *ptr, *rows;
    const float *val, *dw, *dwc;
};
struct ClSrcs {
    ClSrc lv[kAmgMaxLevels];
    const float *inv;
    uint16_t *place;  // scratch: `window` places per CTA and level
    uint32_t window;
};

// Extents of CTA blockIdx.x's rows of level blockIdx.y: {lo, hi, rows, entries}.
__global__ void __launch_bounds__(256) k_cl_extent(ClSrcs s, uint32_t *ext)
{
    __shared__ uint32_t sh[4];
    const ClSrc &L = s.lv[blockIdx.y];
    const uint32_t I0 = uint32_t(uint64_t(L.nc) * blockIdx.x / C), I1 = uint32_t(uint64_t(L.nc) * (blockIdx.x + 1) / C);
    const uint32_t k0 = L.ptr[I0], k1 = L.ptr[I1];
    if (threadIdx.x < 4) sh[threadIdx.x] = threadIdx.x == 0 ? 0xffffffffu : 0u;
    __syncthreads();
    uint32_t lo = 0xffffffffu, hi = 0, nnz = 0;
    for (uint32_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const uint32_t row = L.rows[k], b = L.rp[row], e = L.rp[row + 1];
        lo = min(lo, row);
        hi = max(hi, row + 1);
        nnz += e - b;
        for (uint32_t j = b; j < e; j++) {
            const uint32_t c = L.ci[j];
            lo = min(lo, c);
            hi = max(hi, c + 1);
        }
    }
    atomicMin(&sh[0], lo);
    atomicMax(&sh[1], hi);
    atomicAdd(&sh[3], nnz);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t *o = ext + (blockIdx.y * C + blockIdx.x) * 4;
        o[0] = k1 > k0 ? sh[0] : 0u;
        o[1] = k1 > k0 ? sh[1] : 0u;
        o[2] = k1 - k0;
        o[3] = sh[3];
    }
}

// Running exclusive scan over tiles of one value per thread of a block of 512 (sc: 512 words).  `carry`, the sum of
// the tiles before this one, is each thread's own: nothing but sc is shared, and it may be written again on return.
__device__ __forceinline__ uint32_t scan_tile(uint32_t v, uint32_t *sc, uint32_t &carry)
{
    sc[threadIdx.x] = v;
    __syncthreads();
    for (uint32_t o = 1; o < 512; o <<= 1) {
        const uint32_t x = threadIdx.x >= o ? sc[threadIdx.x - o] : 0u;
        __syncthreads();
        sc[threadIdx.x] += x;
        __syncthreads();
    }
    const uint32_t at = carry + sc[threadIdx.x] - v;
    carry += sc[511];
    __syncthreads();
    return at;
}

__global__ void __launch_bounds__(512) k_cl_pack(ClSrcs s, AmgClusterMap m, const uint32_t *ext, uint8_t *blob)
{
    __shared__ ClHead h;
    __shared__ uint32_t sc[512];
    uint8_t *out = blob + size_t(blockIdx.x) * m.stride;
    if (threadIdx.x == 0) {
        cl_layout(m, blockIdx.x, ext, h);
        *reinterpret_cast<ClHead *>(out) = h;
    }
    __syncthreads();
    for (uint32_t j = 0; j < m.nl; j++) {
        const ClSrc &L = s.lv[j];
        const ClDesc &d = h.lv[j];
        const uint32_t k0 = L.ptr[d.I0];
        uint16_t *row = reinterpret_cast<uint16_t *>(out + d.o_row), *rptr = reinterpret_cast<uint16_t *>(out + d.o_rptr);
        uint32_t *arow = reinterpret_cast<uint32_t *>(out + d.o_arow);
        uint16_t *la = reinterpret_cast<uint16_t *>(out + d.o_la), *col = reinterpret_cast<uint16_t *>(out + d.o_col);
        float *val = reinterpret_cast<float *>(out + d.o_val), *dw = reinterpret_cast<float *>(out + d.o_dw);
        float *dwc = reinterpret_cast<float *>(out + d.o_dwc);
        for (uint32_t i = threadIdx.x; i <= d.nI; i += blockDim.x) {
            arow[i] = L.ptr[d.I0 + i] - k0;
            if (i < d.nI) {
                dwc[i] = L.dwc[d.I0 + i];
                for (uint32_t k = L.ptr[d.I0 + i]; k < L.ptr[d.I0 + i + 1]; k++) la[k - k0] = uint16_t(i);
            }
        }
        // the owned rows in ascending order: their places, counted over the window
        uint16_t *perm = reinterpret_cast<uint16_t *>(out + d.o_perm);
        uint16_t *place = s.place + (size_t(blockIdx.x) * m.nl + j) * s.window;
        for (uint32_t i = threadIdx.x; i < d.hi - d.lo; i += blockDim.x) place[i] = 0xffffu;
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < d.nr; k += blockDim.x) place[L.rows[k0 + k] - d.lo] = uint16_t(k);
        __syncthreads();
        uint32_t carry = 0;
        for (uint32_t t0 = 0; t0 < d.hi - d.lo; t0 += blockDim.x) {
            const uint32_t i = t0 + threadIdx.x;
            const uint16_t k = i < d.hi - d.lo ? place[i] : uint16_t(0xffffu);
            const uint32_t mine = k != 0xffffu;
            const uint32_t at = scan_tile(mine, sc, carry);
            if (mine) perm[at] = k;
        }
        // row pointers: a running scan over tiles of 512 rows
        carry = 0;
        for (uint32_t t0 = 0; t0 < d.nr; t0 += blockDim.x) {
            const uint32_t k = t0 + threadIdx.x;
            uint32_t len = 0, r = 0;
            if (k < d.nr) {
                r = L.rows[k0 + k];
                len = L.rp[r + 1] - L.rp[r];
                row[k] = uint16_t(r - d.lo);
                dw[k] = L.dw[r];
            }
            const uint32_t at = scan_tile(len, sc, carry);
            if (k < d.nr) {
                rptr[k] = uint16_t(at);
                for (uint32_t i = 0; i < len; i++) {
                    val[at + i] = L.val[L.rp[r] + i];
                    col[at + i] = uint16_t(L.ci[L.rp[r] + i] - d.lo);
                }
            }
        }
        if (threadIdx.x == 0) rptr[d.nr] = uint16_t(carry);
        if (j + 1 == m.nl) {
            float *inv = reinterpret_cast<float *>(out + h.o_inv);
            for (uint32_t i = threadIdx.x; i < d.nI * L.nc; i += blockDim.x) inv[i] = s.inv[size_t(d.I0) * L.nc + i];
        }
    }
}

__device__ __forceinline__ uint32_t map_cta(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void put(uint32_t a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v));  // ordered by the barrier, which clobbers memory
}
__device__ __forceinline__ void put(uint32_t a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v));
}
__device__ __forceinline__ void cl_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct ClIo {
    const uint8_t *blob;
    const float *b, *x1;  // level l0: right-hand side and first smoothing step
    float *c1, *c2;       // out: the two directions
    double *sc;           // out: the level's K-cycle scalars
    const CgState *st;
};

__global__ void __launch_bounds__(kClThreads) k_amg_cluster(AmgClusterMap m, ClIo io)
{
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ double sh[3 * 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, cta = blockIdx.x;
    constexpr uint32_t kWarps = kClThreads / 32;

    // ---- the packed levels, and every CTA's windows, before waiting on the preceding kernel ----
    {
        const uint8_t *src = io.blob + size_t(cta) * m.stride;
        const uint32_t bytes = reinterpret_cast<const ClHead *>(src)->bytes;
        const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
        uint4 *d4 = reinterpret_cast<uint4 *>(smem + m.o_blob);
        for (uint32_t i = tid; i < bytes / 16; i += kClThreads) d4[i] = s4[i];
        uint32_t *win = reinterpret_cast<uint32_t *>(smem + m.o_win);
        for (uint32_t i = tid; i < m.nl * C; i += kClThreads) {
            const ClDesc &d = reinterpret_cast<const ClHead *>(io.blob + size_t(i % C) * m.stride)->lv[i / C];
            win[2 * i] = d.lo;
            win[2 * i + 1] = d.hi;
        }
    }
    pdl_wait();
    pdl_release();
    if (io.st && io.st->done) return;  // the same answer in every CTA
    __syncthreads();
    const uint8_t *blob = smem + m.o_blob;
    const ClHead &h = *reinterpret_cast<const ClHead *>(blob);
    const uint32_t *win = reinterpret_cast<const uint32_t *>(smem + m.o_win);
    const uint32_t base = uint32_t(__cvta_generic_to_shared(smem));
    auto f32 = [&](uint32_t o) { return reinterpret_cast<float *>(smem + o); };
    float *bown = f32(m.o_bown), *v1 = f32(m.o_v1), *r2 = f32(m.o_r2);
    float *bd = f32(m.o_bd), *part_s = f32(m.o_part), *xo = f32(m.o_xo);
    double *ws = reinterpret_cast<double *>(smem + m.o_ws);

    // Values of `count` rows of level j in ascending row order, at(i, row) giving the i-th and its row, into the
    // array at offset o of every CTA whose window holds the row.  A warp takes 32 of them, or, when there are
    // few, some of their targets.  Consecutive lanes store (nearly) consecutive words: values stored by whoever
    // computed them, in aggregate order, took one packet each (5k to 20k cycles a phase for 950 rows).
    auto spread = [&](uint32_t j, uint32_t count, uint32_t o, auto at) {
        const uint32_t lo = lane < C ? win[2 * (j * C + lane)] : 0u, hi = lane < C ? win[2 * (j * C + lane) + 1] : 0u;
        const uint32_t chunks = (count + 31) / 32;
        uint32_t parts = 1;
        while (parts < C && chunks * parts * 2 <= kWarps) parts *= 2;
        for (uint32_t t = warp; t < chunks * parts; t += kWarps) {
            const uint32_t i = t / parts * 32, last = min(31u, count - 1 - i);
            uint32_t row = 0;
            const bool valid = lane <= last;
            const float v = valid ? at(i + lane, row) : 0.f;
            const uint32_t r0 = __shfl_sync(0xffffffffu, row, 0), r1 = __shfl_sync(0xffffffffu, row, int(last));
            uint32_t to = __ballot_sync(0xffffffffu, lane < C && lane % parts == t % parts && lo <= r1 && hi > r0);
            while (to) {
                const int c = __ffs(int(to)) - 1;
                to &= to - 1;
                const uint32_t clo = __shfl_sync(0xffffffffu, lo, c), chi = __shfl_sync(0xffffffffu, hi, c);
                if (valid && row >= clo && row < chi) put(map_cta(base + o + (row - clo) * 4, uint32_t(c)), v);
            }
        }
    };
    // the owned rows of level j: f(place among them, place in the window)
    auto spread_owned = [&](uint32_t j, uint32_t o, auto f) {
        const ClDesc &d = h.lv[j];
        const uint16_t *perm = reinterpret_cast<const uint16_t *>(blob + d.o_perm);
        const uint16_t *rows = reinterpret_cast<const uint16_t *>(blob + d.o_row);
        spread(j, d.nr, o, [&](uint32_t i, uint32_t &row) {
            const uint32_t k = perm[i];
            row = d.lo + rows[k];
            return f(k, rows[k]);
        });
    };
    {
        const ClDesc &d = h.lv[0];
        const uint16_t *row = reinterpret_cast<const uint16_t *>(blob + d.o_row);
        for (uint32_t k = tid; k < d.nr; k += kClThreads) bown[k] = io.b[d.lo + row[k]];
        float *ga = f32(m.o_ga[0]);
        for (uint32_t i = tid; i < d.hi - d.lo; i += kClThreads) ga[i] = io.x1[d.lo + i];
    }
    cl_barrier();  // every CTA runs, and its own part is loaded, before others write to it

    // sum over row k of level j of value * g(column), by the row's four lanes (csr_row_dot's order)
    auto row_dot = [&](const ClDesc &d, const float *g, uint32_t k, bool valid) {
        const uint16_t *rptr = reinterpret_cast<const uint16_t *>(blob + d.o_rptr);
        const float *val = reinterpret_cast<const float *>(blob + d.o_val);
        const uint16_t *col = reinterpret_cast<const uint16_t *>(blob + d.o_col);
        const uint32_t beg = valid ? rptr[k] : 0u, end = valid ? rptr[k + 1] : 0u;
        float acc = 0.f;
        for (uint32_t j0 = beg + (lane & 3u); j0 < end; j0 += 4 * kClChunk) {
            float v[kClChunk], x[kClChunk];
#pragma unroll
            for (int t = 0; t < kClChunk; t++) {
                const bool ok = j0 + 4 * t < end;
                const uint32_t at = ok ? j0 + 4 * t : j0;
                const float w = val[at], y = g[col[at]];
                v[t] = ok ? w : 0.f;
                x[t] = ok ? y : 0.f;
            }
#pragma unroll
            for (int t = 0; t < kClChunk; t++) acc = fmaf(v[t], x[t], acc);
        }
        return acc;
    };

    // residual of level j from ga (right-hand side: own array rb when given, else the window's), restricted
    auto restrict_level = [&](uint32_t j, const float *rb) {
        const ClDesc &d = h.lv[j];
        const float *ga = f32(m.o_ga[j]), *bw = f32(m.o_bw[j]);
        const uint16_t *row = reinterpret_cast<const uint16_t *>(blob + d.o_row);
        const uint32_t *arow = reinterpret_cast<const uint32_t *>(blob + d.o_arow);
        const float *dwc = reinterpret_cast<const float *>(blob + d.o_dwc);
        for (uint32_t i = warp; i < d.nI; i += kWarps) {
            float part = 0.f;
            for (uint32_t k = arow[i] + (lane >> 2); k < arow[i + 1]; k += 8) {
                const float acc = row_dot(d, ga, k, true);
                part += ((lane & 3u) == 0 ? (rb ? rb[k] : bw[row[k]]) : 0.f) - acc;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
            if (lane == 0) part_s[i] = part;
        }
        __syncthreads();
        if (j + 1 == m.nl) {  // the dense level's right-hand side: to every CTA
            for (uint32_t t = tid; t < d.nI * C; t += kClThreads)
                put(map_cta(base + m.o_bd + (d.I0 + t % d.nI) * 4, t / d.nI), part_s[t % d.nI]);
        } else {
            spread(j + 1, d.nI, m.o_bw[j + 1], [&](uint32_t i, uint32_t &row) {
                row = d.I0 + i;
                return part_s[i];
            });
            spread(j + 1, d.nI, m.o_ga[j + 1], [&](uint32_t i, uint32_t &row) {
                row = d.I0 + i;
                return dwc[i] * part_s[i];
            });
        }
    };
    // gb = ga + s P e over the windows, from each row's owner
    auto correct = [&](uint32_t j) {
        const ClDesc &d = h.lv[j];
        const float *ga = f32(m.o_ga[j]), *e = f32(m.o_e[j]);
        const uint16_t *la = reinterpret_cast<const uint16_t *>(blob + d.o_la);
        spread_owned(j, m.o_gb[j], [&](uint32_t k, uint32_t w) { return fmaf(m.scale, e[la[k]], ga[w]); });
    };
    // the corrected smoothing sweep: the level's result to the aggregate's owner above (j > 0), or, on the
    // first level, into ga of every window and to `out`
    auto sweep = [&](uint32_t j, const float *rb, float *out) {
        const ClDesc &d = h.lv[j];
        const float *gb = f32(m.o_gb[j]), *bw = f32(m.o_bw[j]);
        const uint16_t *row = reinterpret_cast<const uint16_t *>(blob + d.o_row);
        const float *dw = reinterpret_cast<const float *>(blob + d.o_dw);
        for (uint32_t k0 = warp * 8; k0 < d.nr; k0 += kWarps * 8) {
            const uint32_t k = k0 + (lane >> 2);
            const bool valid = k < d.nr;
            float acc = row_dot(d, gb, k, valid);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            if (!valid) continue;
            const uint32_t w = row[k], r = d.lo + w, q = lane & 3u;
            const float res = (j == 0 ? rb[k] : bw[w]) - acc;
            const float x = fmaf(dw[k], res, gb[w]);
            if (j == 0) {
                if (q == 0) xo[k] = x;
            } else if (q == 0) {
                // row r is aggregate r of the level above: its owner, and its place there
                const uint32_t n = m.n[j], c = uint32_t((uint64_t(r + 1) * C - 1) / n);
                put(map_cta(base + m.o_e[j - 1] + (r - uint32_t(uint64_t(n) * c / C)) * 4, c), x);
            }
        }
        if (j == 0) {
            __syncthreads();
            spread_owned(0, m.o_ga[0], [&](uint32_t k, uint32_t) { return xo[k]; });
            for (uint32_t k = tid; k < d.nr; k += kClThreads) out[d.lo + row[k]] = xo[k];
        }
    };
    // e = inv b on the owned rows of the coarsest level (the owned aggregates of the last smoothed one)
    auto dense = [&]() {
        const ClDesc &d = h.lv[m.nl - 1];
        const uint32_t n = m.n[m.nl];
        const float *inv = reinterpret_cast<const float *>(blob + h.o_inv);
        float *e = f32(m.o_e[m.nl - 1]);
        for (uint32_t i = warp; i < d.nI; i += kWarps) {
            float s = 0.f;
#pragma unroll
            for (int t = 0; t < int(kAmgCoarsest / 32); t++) {
                const uint32_t j = lane + 32u * uint32_t(t);
                if (j < n) s = fmaf(inv[size_t(i) * n + j], bd[j], s);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) e[i] = s;
        }
        __syncthreads();
    };
    auto cycle = [&](const float *rb, float *out) {
        for (uint32_t j = 0; j < m.nl; j++) {
            restrict_level(j, j == 0 ? rb : nullptr);
            cl_barrier();
        }
        dense();
        for (uint32_t j = m.nl; j-- > 0;) {
            correct(j);
            cl_barrier();
            sweep(j, rb, out);
            cl_barrier();
        }
    };
    // v = A c (c in ga): dot products c.v, c.y1, c.y2 over all CTAs; v is kept when asked for
    auto products = [&](const float *y1, const float *y2, float *keep) {
        const ClDesc &d = h.lv[0];
        const float *ga = f32(m.o_ga[0]);
        const uint16_t *row = reinterpret_cast<const uint16_t *>(blob + d.o_row);
        Dot2 s0, s1, s2;
        for (uint32_t k0 = warp * 8; k0 < d.nr; k0 += kWarps * 8) {
            const uint32_t k = k0 + (lane >> 2);
            const bool valid = k < d.nr;
            float acc = row_dot(d, ga, k, valid);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            if (valid && (lane & 3u) == 0) {
                const float c = ga[row[k]];
                s0.add_prod(c, acc);
                s1.add_prod(c, y1[k]);
                if (y2) s2.add_prod(c, y2[k]);
                if (keep) keep[k] = acc;
            }
        }
        double v[3] = {s0.value(), s1.value(), s2.value()};
        block_sum<3>(v, sh);
        if (tid < C) {  // thread 0 has the sums: pass them along the first warp
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const double x = __shfl_sync((1u << C) - 1u, v[q], 0);
                put(map_cta(base + m.o_ws + (q * C + cta) * 8, tid), x);
            }
        }
        cl_barrier();
        if (tid < 3) {
            double t = 0.0;
            for (uint32_t c = 0; c < C; c++) t += ws[tid * C + c];
            sh[tid] = t;
        }
        __syncthreads();
    };

    __shared__ float a1_sh;
    cycle(bown, io.c1);
    products(bown, nullptr, v1);
    if (tid == 0) {
        a1_sh = sh[0] > 0.0 ? float(sh[1] / sh[0]) : 0.f;
        if (cta == 0) {
            io.sc[0] = sh[0];
            io.sc[1] = sh[1];
        }
    }
    __syncthreads();
    {  // r2 = b - a1 v1, x1 = dw r2 (k_amg_kc_r2)
        const float a1 = a1_sh;
        const ClDesc &d = h.lv[0];
        const float *dw = reinterpret_cast<const float *>(blob + d.o_dw);
        for (uint32_t k = tid; k < d.nr; k += kClThreads) {
            const float r = fmaf(-a1, v1[k], bown[k]);
            r2[k] = r;
        }
        __syncthreads();
        spread_owned(0, m.o_ga[0], [&](uint32_t k, uint32_t) { return dw[k] * r2[k]; });
    }
    cl_barrier();
    cycle(r2, io.c2);
    products(v1, r2, nullptr);
    if (cta == 0 && tid == 0) {
        io.sc[2] = sh[0];
        io.sc[3] = sh[1];
        io.sc[4] = sh[2];
    }
    cl_barrier();  // no CTA leaves while another may still write to it
}

}  // namespace

// Queues the extents of the levels from kAmgClusterLevel on (read back by the caller's next
// synchronisation); H->cluster.level stays 0 when the hierarchy has no such levels.
rsg_status amg_cluster_extents(rsg_context *ctx, AmgHierarchy *H)
{
    AmgCluster &K = H->cluster;
    K.level = 0;
    K.map = AmgClusterMap{};
    const int l0 = kAmgClusterLevel;
    if (!H->dense_coarsest || l0 > kAmgKLevels || l0 >= H->levels - 1 || H->L[l0].n > kAmgClusterRows) return RSG_OK;
    ClSrcs s = {};
    AmgClusterMap &m = K.map;
    m.nl = uint32_t(H->levels - 1 - l0);
    for (uint32_t j = 0; j <= m.nl; j++) {
        const AmgLevel &F = H->L[l0 + int(j)];
        m.n[j] = F.n;
        if (j < m.nl) {
            const AmgLevel &N = H->L[l0 + int(j) + 1];
            s.lv[j] = ClSrc{F.n, N.n, F.rp, F.ci, F.agg_ptr.p, F.agg_rows.p, F.val32, F.dw.p, N.dw.p};
        }
    }
    s.inv = H->coarse_inv.p;
    if (!K.ext.ensure(size_t(kAmgMaxLevels) * C * 4) ||
        (!K.ext_h && cudaMallocHost(&K.ext_h, size_t(kAmgMaxLevels) * C * 4 * sizeof(uint32_t)) != cudaSuccess)) {
        (void)cudaGetLastError();  // no memory for it: the launched kernels
        return RSG_OK;
    }
    k_cl_extent<<<dim3(C, m.nl), 256, 0, ctx->stream>>>(s, K.ext.p);
    RSG_CHECK_CUDA(ctx, cudaGetLastError());
    RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(K.ext_h, K.ext.p, size_t(m.nl) * C * 4 * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                                        ctx->stream));
    K.level = l0;
    return RSG_OK;
}

// After that synchronisation: lays the shared memory out and packs the levels; level = 0 when they do not fit.
rsg_status amg_cluster_pack(rsg_context *ctx, AmgHierarchy *H)
{
    AmgCluster &K = H->cluster;
    if (!K.level) return RSG_OK;
    const int l0 = K.level;
    K.level = 0;
    AmgClusterMap &m = K.map;
    m.scale = kAmgScale1;
    uint32_t o = 0;
    auto take = [&](uint64_t bytes) {
        const uint32_t at = o;
        o = uint32_t(std::min<uint64_t>(o + ((bytes + 15) & ~uint64_t(15)), 1u << 30));
        return at;
    };
    uint32_t nr0 = 0, nI0 = 0, window = 0;
    for (uint32_t j = 0; j < m.nl; j++) {
        uint32_t w = 0, nr = 0, nI = 0;
        for (uint32_t c = 0; c < C; c++) {
            const uint32_t *e = K.ext_h + (j * C + c) * 4;
            w = std::max(w, e[1] - e[0]);
            nr = std::max(nr, e[2]);
            nI = std::max(nI, uint32_t(uint64_t(m.n[j + 1]) * (c + 1) / C) - uint32_t(uint64_t(m.n[j + 1]) * c / C));
        }
        window = std::max(window, w);
        m.o_ga[j] = take(uint64_t(w) * 4);
        m.o_gb[j] = take(uint64_t(w) * 4);
        m.o_bw[j] = take(j ? uint64_t(w) * 4 : 0);
        m.o_e[j] = take(uint64_t(nI) * 4);
        if (j == 0) nr0 = nr;
        nI0 = std::max(nI0, nI);
    }
    m.o_bown = take(uint64_t(nr0) * 4);
    m.o_v1 = take(uint64_t(nr0) * 4);
    m.o_r2 = take(uint64_t(nr0) * 4);
    m.o_xo = take(uint64_t(nr0) * 4);
    m.o_part = take(uint64_t(nI0) * 4);
    m.o_bd = take(kAmgCoarsest * 4);
    m.o_ws = take(3 * C * sizeof(double));
    m.o_win = take(uint64_t(m.nl) * C * 2 * 4);
    m.o_blob = o;
    m.stride = 0;
    for (uint32_t c = 0; c < C; c++) {
        ClHead h;
        cl_layout(m, c, K.ext_h, h);
        m.stride = std::max(m.stride, h.bytes);
    }
    const size_t smem = size_t(o) + m.stride;
    if (smem > kClSmem) return RSG_OK;  // (so windows, rows and entries of a CTA also fit 16 bits)
    cudaFuncSetAttribute(k_amg_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kClSmem));
    cudaFuncSetAttribute(k_amg_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (K.supported < 0) {  // the device can place such a cluster (asked once, for the largest shared memory)
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = C;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(C);
        cfg.blockDim = dim3(kClThreads);
        cfg.dynamicSmemBytes = kClSmem;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int clusters = 0;
        K.supported = cudaOccupancyMaxActiveClusters(&clusters, k_amg_cluster, &cfg) == cudaSuccess && clusters > 0;
        (void)cudaGetLastError();
    }
    if (!K.supported) return RSG_OK;
    if (!K.blob.ensure(size_t(m.stride) * C) || !K.place.ensure(size_t(C) * m.nl * window)) {
        (void)cudaGetLastError();
        return RSG_OK;
    }
    ClSrcs s = {};
    for (uint32_t j = 0; j < m.nl; j++) {
        const AmgLevel &F = H->L[l0 + int(j)], &N = H->L[l0 + int(j) + 1];
        s.lv[j] = ClSrc{F.n, N.n, F.rp, F.ci, F.agg_ptr.p, F.agg_rows.p, F.val32, F.dw.p, N.dw.p};
    }
    s.inv = H->coarse_inv.p;
    s.place = K.place.p;
    s.window = window;
    k_cl_pack<<<C, 512, 0, ctx->stream>>>(s, m, K.ext.p, K.blob.p);
    RSG_CHECK_CUDA(ctx, cudaGetLastError());
    K.smem = uint32_t(smem);
    K.level = l0;
    return RSG_OK;
}

void amg_cluster_launch(rsg_context *ctx, const AmgHierarchy *H, const CgState *st, bool pdl)
{
    const AmgCluster &K = H->cluster;
    const AmgLevel &F = H->L[K.level];
    const ClIo io{K.blob.p, F.b.p, F.x1.p, F.c1.p, F.c2.p, H->kc_sc.p + 8 * K.level, st};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = K.smem;
    cfg.stream = ctx->stream;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 2 : 1;
    cudaLaunchKernelEx(&cfg, k_amg_cluster, K.map, io);
}

}  // namespace rsg
