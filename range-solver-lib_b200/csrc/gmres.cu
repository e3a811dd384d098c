// Restarted GMRES(m) on the GPU, restating RMatrixSolver::solveGMRES
// (src/rmatrixsolver.cpp:357-581):
//   cycle start  true residual ro = b - A x, ||x||, beta = ||ro||, error and
//                stopping rule (:401-427)
//   inner step k v_k = w / h_{k,k-1} (v_0 = ro / beta), z_k = P v_k (:430-446)
//                w = A z_k (:451-455) and h_{i,k} = v_i^T w for i <= k (:457-484)
//                in one kernel (k_gm_step)
//                w -= sum_i h_{i,k} v_i, ||w||, P w (:486-510), and in its last
//                block the Givens rotations on column k, the g update and the
//                inner exit when |g_{k+1}| < 1e-4 beta (:519-550) (k_gm_correct)
// The basis is stored unnormalised: slot k + 1 of V holds w and slot k + 1 of Z
// holds P w as k_gm_correct leaves them, and inv[k + 1] = 1 / ||w|| multiplies
// whatever is read from those slots, so an inner step is two launches and V is
// never rewritten.  (The learned preconditioner needs v_k itself: there k_gm_vz
// normalises the slot in place and inv stays 1.)  In FP32 without a preconditioner
// a slot of Z is also scaled by a power of two, next to 1 / the norm of the slot
// before: the product's row sums, taken before inv is applied, would be ~ ||A||^2,
// past FP32's range from entries of 1e19 on and with lost bits below 1e-17.
//   cycle end    back substitution (:554-567), x += sum_j z_j y_j (:570-578)
// Z is stored, so a variable preconditioner (flexible GMRES) needs no change.
// Each cycle is one captured CUDA graph; the host polls the device state once
// per cycle.
// Mixed precision: the Arnoldi vectors V, Z, w and the matrix of the inner
// steps are FP32 (dot products accumulated in FP64), while the true residual at
// every restart (FP64 matrix), the Hessenberg matrix, the Givens rotations, the
// least-squares solve and the solution update x += Z y stay FP64 -- restarted
// GMRES as iterative refinement with an FP32 inner cycle.
#include "gmres.cuh"
#include "gnn.cuh"

#include <cmath>

namespace rsg {

template <int RPW>
__global__ void __launch_bounds__(kBlock) k_gm_residual(Csr<double> M, Sell<double> S, int use_sell, const double *__restrict__ b,
                                                        const double *__restrict__ x, double *__restrict__ ro,
                                                        double *__restrict__ H, double *__restrict__ g,
                                                        double *partials, GmresState *st)
{
    pdl_wait();
    pdl_release();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double sh[96];
    if (st->done) return;
    double acc[3] = {0.0, 0.0, 0.0};
    auto gx = [&](uint32_t c) { return x[c]; };
    auto epi = [&](uint32_t row, double ax) {
        const double r = b[row] - ax;
        ro[row] = r;
        acc[0] += x[row] * x[row];
        acc[1] += r * r;
        acc[2] += b[row] * b[row];
    };
    for_rows_any<double, RPW>(M, S, use_sell != 0, gx, epi, smem_raw, &st->ticket[7], true);
    double tot[3];
    if (grid_sum<3>(acc, partials, &st->ticket[0], sh, tot)) {
        const uint32_t m = st->m;
        for (uint32_t i = threadIdx.x; i < (m + 1) * m; i += blockDim.x) H[i] = 0.0;
        for (uint32_t i = threadIdx.x; i <= m; i += blockDim.x) g[i] = 0.0;
        __syncthreads();
        if (threadIdx.x == 0) {
            const double xn = sqrt(tot[0]), beta = sqrt(tot[1]);
            if (st->outer == 0) st->bn = sqrt(tot[2]);
            double norm = st->an * xn + st->bn;
            if (fabs(norm) < st->eps) norm = st->eps;
            const double err = beta / norm;
            st->trend = err - st->error;
            st->error = err;
            st->xn = xn;
            st->beta = beta;
            if (st->history) {
                st->history[st->outer_logged] = err;
                st->trend_hist[st->outer_logged] = st->trend;
            }
            st->outer_logged++;
            bool stop;
            if (st->stop_rule == RSG_STOP_REFERENCE) {
                stop = !dev_isnormal(err) || !dev_isnormal(st->trend) || err < st->cvg || fabs(st->trend) < st->eps * st->eps;
                if (stop) {
                    st->converged = 1;
                    st->status = isfinite(err) ? RSG_OK : RSG_BREAKDOWN;
                }
            } else {
                stop = !(beta > st->rtol * st->bn);
                if (stop) {
                    st->converged = isfinite(beta) ? 1 : 0;
                    st->status = isfinite(beta) ? RSG_OK : RSG_BREAKDOWN;
                }
            }
            if (stop) {
                st->done = 1;
            } else {
                g[0] = beta;
                st->k = 0;
                st->inner_done = 0;
                st->cycle_len = 0;
            }
        }
    }
}

// 16-byte packs of the basis type.
template <typename T>
struct Pack;
template <>
struct Pack<double> {
    static constexpr int N = 2;
    __device__ __forceinline__ static void ld(const double *p, double (&v)[2])
    {
        const double2 t = *reinterpret_cast<const double2 *>(p);
        v[0] = t.x;
        v[1] = t.y;
    }
    __device__ __forceinline__ static void st(double *p, const double (&v)[2])
    {
        *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
    }
};
template <>
struct Pack<float> {
    static constexpr int N = 4;
    __device__ __forceinline__ static void ld(const float *p, float (&v)[4])
    {
        const float4 t = *reinterpret_cast<const float4 *>(p);
        v[0] = t.x;
        v[1] = t.y;
        v[2] = t.z;
        v[3] = t.w;
    }
    __device__ __forceinline__ static void st(float *p, const float (&v)[4])
    {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};

// v_k = src / s (0 if s == 0), z_k = P v_k.  src = ro for k = 0, else slot k of V, in place.  T: vector
// type of the Arnoldi vectors (double, or float in mixed precision); D: preconditioner values.
template <int PK, typename T, typename D>
__global__ void __launch_bounds__(kBlock) k_gm_vz(uint32_t n, size_t ld, uint32_t w_, const D *__restrict__ d,
                                                  const double *__restrict__ ro, const double *__restrict__ wnorm,
                                                  T *V, T *Z, double *inv, const GmresState *st, uint32_t k)
{
    pdl_wait();
    pdl_release();
    if (st->done || st->inner_done) return;
    const double s = (k == 0) ? st->beta : wnorm[k];
    T *v = V + size_t(k) * ld, *z = Z + size_t(k) * ld;
    if (blockIdx.x == 0 && threadIdx.x == 0) inv[k] = inv[kVInv + k] = 1.0;
    const uint32_t G = PK == 2 ? w_ : 1, ng = n / G;
    for (uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x; gi < ng; gi += gridDim.x * blockDim.x) {
        T vl[kMaxBlock];
        for (uint32_t j = 0; j < G; j++) {
            const size_t i = size_t(gi) * G + j;
            const double src = (k == 0) ? ro[i] : double(v[i]);
            vl[j] = T((s == 0.0) ? 0.0 : src / s);
            v[i] = vl[j];
        }
        if (PK == 0) z[gi] = vl[0];
        else if (PK == 1) z[gi] = T(d[gi]) * vl[0];
        else
            for (uint32_t j = 0; j < G; j++) {
                const D *row = d + (size_t(gi) * G + j) * G;
                T acc = T(0);
                for (uint32_t l = 0; l < G; l++) acc += T(row[l]) * vl[l];
                z[size_t(gi) * G + j] = acc;
            }
    }
}

// w = A z_k, for matrices without the SELL-32 copy (k_gm_step then starts from the stored w).
template <int RPW, typename T>
__global__ void __launch_bounds__(kBlock) k_gm_spmv(Csr<T> M, const T *__restrict__ z, T *__restrict__ wv,
                                                    const double *inv, GmresState *st, uint32_t k)
{
    pdl_wait();
    pdl_release();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (st->done || st->inner_done) return;
    const double s = inv[k];
    auto gx = [&](uint32_t c) { return z[c]; };
    auto epi = [&](uint32_t row, T v) { wv[row] = T(double(v) * s); };
    for_rows_tma<T, RPW>(M, gx, epi, smem_raw, &st->ticket[7], true);
}

// One Arnoldi product: w = A z_k (FUSE; otherwise w is read) and h_i = v_i^T w for i <= k.
//
// A block takes tiles of 256 rows: its eight warps form w of their 32-row slices, leave it in shared
// memory, and then split the vectors (warp j takes v_j, v_{j+8}, ...: JM of them at most), each reading
// its vectors' tile with 16-byte loads and keeping one accumulator per vector and thread.  So w is
// read once instead of once per vector, and a vector costs one warp reduction per block instead of a
// block reduction.  Bound by the chain of a launch (state, slices, gathers, vectors, ticket, partials)
// up to about ten vectors and by reading V above.  61^3 convection-diffusion (226,981 rows, 1.6M
// entries, FP64, GMRES(30)), an inner step on average: w, normalisation, product, dots and correction as
// four launches with w re-read per vector 59.4 us; this kernel and k_gm_correct 27.8 us (20.0 -> 9.7 ms a
// solve).  A separate product kernel in front of the dots: 32.3 us.
template <typename T, bool FUSE, int JM>
__global__ void __launch_bounds__(kBlock) k_gm_step(Sell<T> S, uint32_t n, size_t ld, const T *V, const T *__restrict__ z,
                                                    T *wv, double *__restrict__ H, double *__restrict__ hv,
                                                    const double *inv, double *partials, GmresState *st, uint32_t k)
{
    pdl_wait();
    pdl_release();
    using P = Pack<T>;
    __shared__ __align__(16) T ws[kBlock];
    __shared__ bool is_last;
    if (st->done || st->inner_done) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double s = FUSE ? inv[k] : 1.0;
    double acc[JM];
#pragma unroll
    for (int j = 0; j < JM; j++) acc[j] = 0.0;
    const uint32_t tiles = (n + kBlock - 1) / kBlock;
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint32_t row0 = t * kBlock;
        if (FUSE) {
            T mine = T(0);
            auto gx = [&](uint32_t c) { return z[c]; };
            auto epi = [&](uint32_t row, T v) {
                mine = T(double(v) * s);
                wv[row] = mine;
            };
            for_rows_sell_v<T>(S, gx, epi, t, tiles);  // exactly this tile: one slice per warp
            ws[threadIdx.x] = mine;
        } else {
            const uint32_t row = row0 + threadIdx.x;
            ws[threadIdx.x] = row < n ? wv[row] : T(0);
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < JM; j++) {
            const uint32_t i = uint32_t(warp + 8 * j);
            if (i <= k) {
                const T *v = V + size_t(i) * ld + row0;
                if (row0 + kBlock <= n) {
                    constexpr int L = kBlock / (32 * P::N);
                    T a[L][P::N];
#pragma unroll
                    for (int u = 0; u < L; u++) P::ld(v + (u * 32 + lane) * P::N, a[u]);
#pragma unroll
                    for (int u = 0; u < L; u++) {
                        T b[P::N];
                        P::ld(ws + (u * 32 + lane) * P::N, b);
#pragma unroll
                        for (int e = 0; e < P::N; e++) acc[j] += double(b[e]) * double(a[u][e]);
                    }
                } else {
                    for (uint32_t e = lane; row0 + e < n; e += 32) acc[j] += double(ws[e]) * double(v[e]);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < JM; j++) {
        const uint32_t i = uint32_t(warp + 8 * j);
        if (i <= k) {
            const double v = warp_sum(acc[j]);
            if (lane == 0) partials[size_t(i) * gridDim.x + blockIdx.x] = v;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        is_last = (atomicAdd(&st->ticket[1], 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    // the last block adds the partials: a warp sums its vectors side by side, so that all their loads
    // are in flight together
    const uint32_t m = st->m;
#pragma unroll
    for (int j = 0; j < JM; j++) acc[j] = 0.0;
#pragma unroll 4
    for (uint32_t bx = lane; bx < gridDim.x; bx += 32)
#pragma unroll
        for (int j = 0; j < JM; j++) {
            const uint32_t i = uint32_t(warp + 8 * j);
            if (i <= k) acc[j] += __ldcg(&partials[size_t(i) * gridDim.x + bx]);
        }
#pragma unroll
    for (int j = 0; j < JM; j++) {
        const uint32_t i = uint32_t(warp + 8 * j);
        if (i <= k) {
            const double sum = warp_sum(acc[j]);
            if (lane == 0) {
                const double h = sum * inv[kVInv + i];  // v_i = inv_i (slot i)
                H[size_t(i) * m + k] = h;
                hv[i] = h * inv[kVInv + i];             // the factor of slot i in w -= h_i v_i
            }
        }
    }
    if (threadIdx.x == 0) st->ticket[1] = 0u;
}

// w -= sum_i h_i v_i (hv holds h_i inv_i, the factor of slot i), P w and ||w||; the last block applies
// the Givens rotations to column k.  16-byte loads of V, eight vectors in flight; the rotations, a
// serial chain, run on shared-memory copies of the column (from L2 each of its 2k loads cost a round
// trip: about 10 us of a step at k = 30).
template <int PK, typename T, typename D>
__global__ void __launch_bounds__(kBlock) k_gm_correct(uint32_t n, size_t ld, uint32_t w_, const D *__restrict__ d,
                                                       const T *V, T *wv, T *__restrict__ zn,
                                                       const double *__restrict__ hv_g, double *__restrict__ H,
                                                       double *__restrict__ cs, double *__restrict__ sn,
                                                       double *__restrict__ g, double *__restrict__ wnorm,
                                                       double *inv, double *partials, GmresState *st, uint32_t k)
{
    pdl_wait();
    pdl_release();
    using P = Pack<T>;
    __shared__ double sh[32];
    __shared__ double hv[kMaxRestart + 1];
    __shared__ double hc[kMaxRestart + 1], cc[kMaxRestart], ss[kMaxRestart];
    if (st->done || st->inner_done) return;
    constexpr bool kScaleZ = PK == 0 && sizeof(T) == 4;
    const T zs = kScaleZ ? T(st->zscale) : T(1);
    for (uint32_t i = threadIdx.x; i <= k; i += blockDim.x) hv[i] = hv_g[i];
    __syncthreads();
    double acc[1] = {0.0};
    auto row_value = [&](uint32_t j) {
        double value = double(wv[j]);
        for (uint32_t i = 0; i <= k; i++) value -= hv[i] * double(V[size_t(i) * ld + j]);
        return T(value);
    };
    constexpr int N = P::N;
    // val -= sum_i hv_i v_i for the N rows at vp of slot 0
    auto project = [&](const T *vp, double (&val)[N]) {
        uint32_t i = 0;
        for (; i + 8 <= k + 1; i += 8) {
            T a[8][N];
#pragma unroll
            for (int u = 0; u < 8; u++) P::ld(vp + size_t(i + u) * ld, a[u]);
#pragma unroll
            for (int u = 0; u < 8; u++)
#pragma unroll
                for (int e = 0; e < N; e++) val[e] -= hv[i + u] * double(a[u][e]);
        }
        if (i <= k) {  // the last one to seven vectors, loaded together
            T a[7][N];
#pragma unroll
            for (int u = 0; u < 7; u++)
                if (i + u <= k) P::ld(vp + size_t(i + u) * ld, a[u]);
#pragma unroll
            for (int u = 0; u < 7; u++)
                if (i + u <= k)
#pragma unroll
                    for (int e = 0; e < N; e++) val[e] -= hv[i + u] * double(a[u][e]);
        }
    };
    if (PK < 2) {
        const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
        const uint32_t np = n / N;
        for (uint32_t p = tid; p < np; p += stride) {
            T w[N];
            P::ld(wv + size_t(p) * N, w);
            double val[N];
#pragma unroll
            for (int e = 0; e < N; e++) val[e] = double(w[e]);
            project(V + size_t(p) * N, val);
            T z[N];
#pragma unroll
            for (int e = 0; e < N; e++) {
                w[e] = T(val[e]);
                acc[0] += double(w[e]) * double(w[e]);
                z[e] = PK == 1 ? T(d[size_t(p) * N + e]) * w[e] : kScaleZ ? zs * w[e] : w[e];
            }
            P::st(wv + size_t(p) * N, w);
            if (zn) P::st(zn + size_t(p) * N, z);
        }
        const uint32_t j = np * N + tid;
        if (j < n) {
            const T w = row_value(j);
            wv[j] = w;
            acc[0] += double(w) * double(w);
            if (zn) zn[j] = PK == 1 ? T(d[j]) * w : kScaleZ ? zs * w : w;
        }
    } else {
        // Blocks of G rows: tiles of whole blocks and whole packs, w as above and through shared memory, then a row of
        // its block's inverse per thread.  A thread per block of rows, strided and one vector at a time, left 209k
        // rows at 60.5 us a step with G = 3 and 110.5 with G = 8, FP64, m = 30: now 50.3 and 54.2 (mixed 46.6 and
        // 83.0: 42.6 and 45.4); with m = 100 and G = 8 it was slower than a launch per operation had been.
        __shared__ __align__(16) T ws[PK == 2 ? kBlock * N : 1];
        const uint32_t G = w_, rows = kBlock / G * G * N;
        for (uint64_t t0 = uint64_t(blockIdx.x) * rows; t0 < n; t0 += uint64_t(gridDim.x) * rows) {
            const uint32_t cnt = uint32_t(min(uint64_t(rows), n - t0)), own = threadIdx.x * N;
            if (own + N <= cnt) {
                T w[N];
                P::ld(wv + t0 + own, w);
                double val[N];
#pragma unroll
                for (int e = 0; e < N; e++) val[e] = double(w[e]);
                project(V + t0 + own, val);
#pragma unroll
                for (int e = 0; e < N; e++) {
                    w[e] = T(val[e]);
                    acc[0] += double(w[e]) * double(w[e]);
                }
                P::st(wv + t0 + own, w);
                P::st(ws + own, w);
            } else if (own < cnt) {
                for (uint32_t j = own; j < cnt; j++) {
                    const T w = row_value(uint32_t(t0) + j);
                    wv[t0 + j] = ws[j] = w;
                    acc[0] += double(w) * double(w);
                }
            }
            __syncthreads();
            if (zn)
                for (uint32_t j = threadIdx.x; j < cnt; j += kBlock) {
                    const D *row = d + (size_t(t0) + j) * G;
                    const T *wl = ws + j / G * G;
                    T z = T(0);
                    for (uint32_t l = 0; l < G; l++) z += T(row[l]) * wl[l];
                    zn[t0 + j] = z;
                }
            __syncthreads();
        }
    }
    double tot[1];
    if (!grid_sum<1>(acc, partials, &st->ticket[2], sh, tot)) return;
    const uint32_t m = st->m;
    for (uint32_t i = threadIdx.x; i <= k; i += blockDim.x) {
        hc[i] = __ldcg(&H[size_t(i) * m + k]);
        if (i < k) {
            cc[i] = __ldcg(&cs[i]);
            ss[i] = __ldcg(&sn[i]);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // v_{k+1} = w / h_{k+1,k}: its scale is kept in inv, h_{k+1,k} itself is rotated away
        const double hn = sqrt(tot[0]);
        wnorm[k + 1] = hn;
        const double s = hn == 0.0 ? 0.0 : 1.0 / hn;
        inv[kVInv + k + 1] = s;
        inv[k + 1] = kScaleZ ? s / double(zs) : s;
        if (kScaleZ) st->zscale = zscale_for(hn);
        for (uint32_t i = 1; i <= k; i++) {
            const double hsave = hc[i - 1], hi = hc[i];
            hc[i - 1] = cc[i - 1] * hsave + ss[i - 1] * hi;
            hc[i] = -ss[i - 1] * hsave + cc[i - 1] * hi;
        }
        const double hk = hc[k];
        const double gg = sqrt(hk * hk + hn * hn);
        double ck = 0.0, sk = 0.0;
        if (gg != 0.0) {
            ck = hk / gg;
            sk = hn / gg;
        }
        cs[k] = ck;
        sn[k] = sk;
        hc[k] = gg;
        const double gk = g[k], gn = -sk * gk;
        g[k + 1] = gn;
        g[k] = ck * gk;
        H[size_t(k + 1) * m + k] = 0.0;
        st->total_inner++;
        st->cycle_len = k + 1;
        if (fabs(gn) < st->beta * 1.0e-4) st->inner_done = 1;
        st->k = k + 1;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i <= k; i += blockDim.x) H[size_t(i) * m + k] = hc[i];
}

// Back substitution (:554-567) by one block, column by column: as soon as y_j is known every thread
// subtracts y_j h_ij from its own g_i, the order in which the reference's row loop subtracts them.
// y is returned with the slots' scale: y_j inv_j multiplies slot j of Z.
__global__ void __launch_bounds__(kMaxRestart) k_gm_backsub(const double *__restrict__ H, const double *__restrict__ g,
                                                            const double *__restrict__ inv, double *__restrict__ y,
                                                            const GmresState *st)
{
    pdl_wait();
    pdl_release();
    __shared__ double yj;
    if (st->done) return;
    const uint32_t m = st->m, it = st->cycle_len, i = threadIdx.x;
    double gi = i < it ? g[i] : 0.0;
    const double hii = i < it ? H[size_t(i) * m + i] : 0.0;
    double next = it > 0 && i < it - 1 ? H[size_t(i) * m + it - 1] : 0.0;
    for (int j = int(it) - 1; j >= 0; j--) {
        const double hij = next;
        next = j > 0 && int(i) < j - 1 ? H[size_t(i) * m + j - 1] : 0.0;  // the next column, loaded ahead
        if (int(i) == j) {
            yj = hii == 0.0 ? 0.0 : gi / hii;
            y[j] = yj * inv[j];
        }
        __syncthreads();
        if (int(i) < j) gi -= yj * hij;
        __syncthreads();
    }
}

// x += sum_j y_j z_j (:570-578), 16-byte loads, eight vectors in flight.
template <typename T>
__global__ void __launch_bounds__(kBlock) k_gm_update(uint32_t n, size_t ld, const T *__restrict__ Z,
                                                      const double *__restrict__ y_g, double *__restrict__ x,
                                                      GmresState *st)
{
    pdl_wait();
    pdl_release();
    using P = Pack<T>;
    constexpr int N = P::N;
    __shared__ double y[kMaxRestart];
    if (st->done) return;
    const uint32_t len = st->cycle_len;
    for (uint32_t j = threadIdx.x; j < len; j += blockDim.x) y[j] = y_g[j];
    __syncthreads();
    const uint32_t np = n / N, tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (uint32_t p = tid; p < np; p += stride) {
        double xv[N];
#pragma unroll
        for (int e = 0; e < N; e++) xv[e] = x[size_t(p) * N + e];
        const T *zp = Z + size_t(p) * N;
        for (uint32_t j = 0; j < len; j += 8) {
            T a[8][N];
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (j + u < len) P::ld(zp + size_t(j + u) * ld, a[u]);
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (j + u < len)
#pragma unroll
                    for (int e = 0; e < N; e++) xv[e] += double(a[u][e]) * y[j + u];
        }
#pragma unroll
        for (int e = 0; e < N; e++) x[size_t(p) * N + e] = xv[e];
    }
    const uint32_t i = np * N + tid;
    if (i < n) {
        double xi = x[i];
        for (uint32_t j = 0; j < len; j++) xi += double(Z[size_t(j) * ld + i]) * y[j];
        x[i] = xi;
    }
}

__global__ void k_gm_cycle_end(GmresState *st)
{
    pdl_wait();
    pdl_release();
    if (threadIdx.x != 0) return;
    if (st->done) return;
    st->outer++;
    if (st->outer >= st->max_outer) {
        st->done = 1;
        st->status = RSG_NOT_CONVERGED;
    }
}

size_t gmres_workspace_bytes(uint32_t n, uint32_t m, bool mixed, uint32_t w)
{
    const size_t vn = arena_bytes(n, sizeof(double));
    const size_t vt = arena_bytes(size_t(m + 1) * gmres_ld(n), mixed ? sizeof(float) : sizeof(double));
    return 2 * vt + vn + arena_bytes(size_t(m + 1) * m, sizeof(double)) + 6 * arena_bytes(m + 2, sizeof(double)) +
           arena_bytes(kVInv + m + 2, sizeof(double)) +
           (mixed ? arena_bytes(size_t(n) * w, sizeof(float)) : 0);
}

rsg_status gmres_carve(rsg_context *ctx, GmresArgs &a, uint32_t n, uint32_t m)
{
    if (m > kMaxRestart) return set_error(ctx, RSG_ERR_UNSUPPORTED, "GMRES restart length %u > %u", m, kMaxRestart);
    if (a.mixed) {
        a.V32 = arena_take<float>(ctx, size_t(m + 1) * gmres_ld(n));
        a.Z32 = arena_take<float>(ctx, size_t(m + 1) * gmres_ld(n));
    } else {
        a.V = arena_take<double>(ctx, size_t(m + 1) * gmres_ld(n));
        a.Z = arena_take<double>(ctx, size_t(m + 1) * gmres_ld(n));
    }
    a.ro = arena_take<double>(ctx, n);
    a.H = arena_take<double>(ctx, size_t(m + 1) * m);
    a.cs = arena_take<double>(ctx, m + 2);
    a.sn = arena_take<double>(ctx, m + 2);
    a.g = arena_take<double>(ctx, m + 2);
    a.y = arena_take<double>(ctx, m + 2);
    a.hv = arena_take<double>(ctx, m + 2);
    a.wnorm = arena_take<double>(ctx, m + 2);
    a.inv = arena_take<double>(ctx, kVInv + m + 2);
    if (!a.inv) return set_error(ctx, RSG_ERR_OUT_OF_MEMORY, "GMRES workspace");
    return RSG_OK;
}

namespace {

constexpr double kLearnedMinDrop = 0.1;

// k_gm_step with the accumulator count of step k (vectors per warp: (k + 1) / 8 rounded up, to a power of two).
template <typename T, bool FUSE>
void launch_step(cudaStream_t st, bool pdl, int grid, const GmresArgs &a, const Sell<T> &S, uint32_t n, size_t ld,
                 const T *V, const T *z, T *w, uint32_t k)
{
    const uint32_t jm = (k + 8) / 8;
    auto go = [&](auto kernel) {
        launch_k(st, pdl, kernel, grid, kBlock, 0, S, n, ld, V, z, w, a.H, a.hv, (const double *)a.inv, a.partials,
                 a.st, k);
    };
    if (jm <= 1) go(k_gm_step<T, FUSE, 1>);
    else if (jm <= 2) go(k_gm_step<T, FUSE, 2>);
    else if (jm <= 4) go(k_gm_step<T, FUSE, 4>);
    else if (jm <= 8) go(k_gm_step<T, FUSE, 8>);
    else go(k_gm_step<T, FUSE, 16>);
}

template <int RPW, int PK>
rsg_status run_typed(rsg_context *ctx, const GmresArgs &a, double *seconds)
{
    const uint32_t n = a.A->n, m = a.m;
    const size_t ld = gmres_ld(n);
    const Csr<double> M = view<double>(a.A, true);
    const size_t s64 = a.A->use_sell ? 0 : tma_smem<double>();
    cudaFuncSetAttribute(k_gm_residual<RPW>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(tma_smem<double>()));
    cudaFuncSetAttribute(k_gm_spmv<RPW, double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         int(tma_smem<double>()));
    cudaFuncSetAttribute(k_gm_spmv<RPW, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(tma_smem<float>()));
    const Sell<double> S = sell_view<double>(a.A);
    const Csr<float> M32 = view<float>(a.A, true);
    const Sell<float> S32 = sell_view<float>(a.A);
    const size_t s32 = a.A->use_sell ? 0 : tma_smem<float>();
    const int us = a.A->use_sell;
    const long long ct = (long long)n * 32 / RPW;
    (void)ct;
    const int g_sp = spmv_grid(ctx, a.A, (const void *)k_gm_spmv<RPW, double>, s64, RPW);
    const int g_sp32 = spmv_grid(ctx, a.A, (const void *)k_gm_spmv<RPW, float>, s32, RPW);
    const int g_res = spmv_grid(ctx, a.A, (const void *)k_gm_residual<RPW>, s64, RPW);
    const int g_vec = std::min(grid_for(ctx, (const void *)k_gm_update<double>, kBlock, 0, n), kMaxGrid);
    const int g_cor = std::min(grid_for(ctx, (const void *)k_gm_correct<PK, double, double>, kBlock, 0,
                                        (long long)n / (a.mixed ? 4 : 2)),
                               kMaxGrid);
    // k_gm_step: every block takes the same number of tiles (the fewest that one wave of blocks allows),
    // since each block adds a ticket and (k + 1) partials.  226,981 rows = 887 tiles, 740 resident
    // blocks: 444 blocks of two tiles 9.65 ms a solve; all 740 (some with two) 10.1 ms; one tile per block
    // (888 blocks at 40 registers) 11.4 ms; 296 blocks of three 10.5 ms.
    const int tiles = int((n + kBlock - 1) / kBlock);
    const int full = std::min(grid_for(ctx, (const void *)k_gm_step<double, true, 4>, kBlock, 0, 1ll << 40), 1024);
    const int g_dot = (tiles + (tiles + full - 1) / full - 1) / ((tiles + full - 1) / full);

    // One captured graph per cycle; with the learned preconditioner a second graph
    // (Jacobi z_k) is captured as the fallback.
    auto capture = [&](rsg_learned *G, bool pdl, bool gnn_pdl, cudaGraph_t *graph, cudaGraphExec_t *exec) -> rsg_status {
        if (G) RSG_TRY(gnn_prepare(ctx, G, a.A, false));  // no allocation inside the capture
        RSG_CHECK_CUDA(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        cudaStream_t st = ctx->stream;
        launch_k(st, pdl, k_gm_residual<RPW>, g_res, kBlock, s64, M, S, us, a.b, a.x, a.ro, a.H, a.g, a.partials,
                 a.st);
        for (uint32_t k = 0; k < m; k++) {
            if (a.mixed) {  // FP32 Arnoldi step
                float *z = a.Z32 + size_t(k) * ld, *w = a.V32 + size_t(k + 1) * ld;
                if (k == 0)
                    launch_k(st, pdl, k_gm_vz<PK, float, float>, g_vec, kBlock, 0, n, ld, a.P.w, a.P.d32, a.ro,
                             a.wnorm, a.V32, a.Z32, a.inv, a.st, k);
                if (us) {
                    launch_step<float, true>(st, pdl, g_dot, a, S32, n, ld, a.V32, z, w, k);
                } else {
                    launch_k(st, pdl, k_gm_spmv<RPW, float>, g_sp32, kBlock, s32, M32, z, w, (const double *)a.inv,
                             a.st, k);
                    launch_step<float, false>(st, pdl, g_dot, a, S32, n, ld, a.V32, z, w, k);
                }
                launch_k(st, pdl, k_gm_correct<PK, float, float>, g_cor, kBlock, 0, n, ld, a.P.w, a.P.d32, a.V32, w,
                         a.Z32 + size_t(k + 1) * ld, a.hv, a.H, a.cs, a.sn, a.g, a.wnorm, a.inv, a.partials, a.st, k);
                continue;
            }
            double *z = a.Z + size_t(k) * ld, *w = a.V + size_t(k + 1) * ld;
            if (k == 0 || G)
                launch_k(st, pdl, k_gm_vz<PK, double, double>, g_vec, kBlock, 0, n, ld, a.P.w, a.P.d, a.ro, a.wnorm,
                         a.V, a.Z, a.inv, a.st, k);
            if (G) {  // flexible GMRES: z_k = M(v_k) from the network (Z is stored, src/rmatrixsolver.cpp:446)
                const rsg_status gs = gnn_forward(ctx, G, a.A, a.V + size_t(k) * ld, z, nullptr, false, true, gnn_pdl);
                if (gs != RSG_OK) {
                    cudaGraph_t dummy = nullptr;
                    cudaStreamEndCapture(ctx->stream, &dummy);
                    if (dummy) cudaGraphDestroy(dummy);
                    return gs;
                }
            }
            if (us) {
                launch_step<double, true>(st, pdl, g_dot, a, S, n, ld, a.V, z, w, k);
            } else {
                launch_k(st, pdl, k_gm_spmv<RPW, double>, g_sp, kBlock, s64, M, z, w, (const double *)a.inv, a.st, k);
                launch_step<double, false>(st, pdl, g_dot, a, S, n, ld, a.V, z, w, k);
            }
            launch_k(st, pdl, k_gm_correct<PK, double, double>, g_cor, kBlock, 0, n, ld, a.P.w, a.P.d, a.V, w,
                     G ? nullptr : a.Z + size_t(k + 1) * ld, a.hv, a.H, a.cs, a.sn, a.g, a.wnorm, a.inv, a.partials,
                     a.st, k);
        }
        launch_k(st, pdl, k_gm_backsub, 1, int(kMaxRestart), 0, a.H, a.g, a.inv, a.y, a.st);
        if (a.mixed) launch_k(st, pdl, k_gm_update<float>, g_vec, kBlock, 0, n, ld, a.Z32, a.y, a.x, a.st);
        else launch_k(st, pdl, k_gm_update<double>, g_vec, kBlock, 0, n, ld, a.Z, a.y, a.x, a.st);
        launch_k(st, pdl, k_gm_cycle_end, 1, 32, 0, a.st);
        cudaError_t e = cudaStreamEndCapture(ctx->stream, graph);
        if (e != cudaSuccess) return set_error(ctx, RSG_ERR_CUDA, "GMRES capture: %s", cudaGetErrorString(e));
        e = cudaGraphInstantiate(exec, *graph, 0);
        if (e != cudaSuccess) {
            cudaGraphDestroy(*graph);
            *graph = nullptr;
            return set_error(ctx, RSG_ERR_CUDA, "GMRES instantiate: %s", cudaGetErrorString(e));
        }
        return RSG_OK;
    };
    // with programmatic dependent launch when the CG policy picks it for A, else (or if the
    // driver refuses the programmatic edges) plain launches
    auto capture_any = [&](rsg_learned *G, cudaGraph_t *graph, cudaGraphExec_t *exec) -> rsg_status {
        const bool pdl = pdl_for(a.A, a.mixed);
        rsg_status r = capture(G, pdl, true, graph, exec);
        if (r != RSG_OK && r != RSG_ERR_OUT_OF_MEMORY && (pdl || (G && pdl_allowed()))) {
            (void)cudaGetLastError();
            r = capture(G, false, false, graph, exec);
        }
        return r;
    };
    cudaGraph_t graph = nullptr, graph_j = nullptr;
    cudaGraphExec_t exec = nullptr, exec_j = nullptr;
    rsg_status s = capture_any(a.G, &graph, &exec);
    if (s == RSG_OK && a.G) s = capture_any(nullptr, &graph_j, &exec_j);
    if (s != RSG_OK) {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        return s;
    }
    cudaError_t e = cudaSuccess;
    cudaEventRecord(ctx->ev[0], ctx->stream);
    int32_t *done_h = reinterpret_cast<int32_t *>(ctx->pinned);
    double *beta_h = ctx->pinned + 1;
    bool learned = a.G != nullptr;
    double beta_prev = 0.0;
    if (a.fallbacks) *a.fallbacks = 0;
    // k_gm_cycle_end marks the state done after max_outer cycles; the host bound is a backstop
    const uint64_t max_cycles = uint64_t(a.st_max_outer) + 2;
    for (uint64_t cycle = 0; cycle < max_cycles; cycle++) {
        e = cudaGraphLaunch(learned ? exec : (exec_j ? exec_j : exec), ctx->stream);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(done_h, &a.st->done, sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess && a.G)
            e = cudaMemcpyAsync(beta_h, &a.st->beta, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) {
            s = set_error(ctx, RSG_ERR_CUDA, "GMRES cycle: %s", cudaGetErrorString(e));
            break;
        }
        if (*done_h) break;
        // beta of this cycle is the residual left by the previous one: a learned cycle
        // that removed less than kLearnedMinDrop of it hands over to Jacobi for good
        if (learned && cycle > 0 && !(*beta_h < (1.0 - kLearnedMinDrop) * beta_prev)) {
            learned = false;
            if (a.fallbacks) (*a.fallbacks)++;
        }
        beta_prev = *beta_h;
    }
    cudaEventRecord(ctx->ev[1], ctx->stream);
    cudaStreamSynchronize(ctx->stream);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
    *seconds = ms * 1e-3;
    if (exec_j) cudaGraphExecDestroy(exec_j);
    if (graph_j) cudaGraphDestroy(graph_j);
    cudaGraphExecDestroy(exec);
    cudaGraphDestroy(graph);
    return s;
}

}  // namespace

rsg_status gmres_run(rsg_context *ctx, const GmresArgs &a, double *seconds)
{
    const int rpw = pick_rpw(a.A);
    switch (a.P.kind) {
    case 0: RSG_RPW_DISPATCH(rpw, return (run_typed<RPW, 0>(ctx, a, seconds)));
    case 1: RSG_RPW_DISPATCH(rpw, return (run_typed<RPW, 1>(ctx, a, seconds)));
    default: RSG_RPW_DISPATCH(rpw, return (run_typed<RPW, 2>(ctx, a, seconds)));
    }
    return RSG_ERR_UNSUPPORTED;
}

}  // namespace rsg
