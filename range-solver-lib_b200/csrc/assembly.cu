// GPU stiffness assembly for linear tetrahedra (heat: 1 DOF/node, elasticity:
// 3 DOFs/node), deterministic and atomic-free.
//
// One thread owns one free row.  It walks its node's adjacent tets in
// ascending tet order (traction triangles first for elasticity, as the
// reference assembles surfaces before volumes), recomputes the tet's element
// row it needs (constant-gradient P1 element: B = grad N, V = |det J| / 6),
// applies the theta scheme and the Dirichlet lifting of
// RSolverHeat/RSolverStress::assemblyMatrix, and adds the row into its own CSR
// entries through the plan's scatter offsets.  Every entry therefore sums its
// element contributions in the same order as the reference's sequential
// element loop, and repeated assemblies are bitwise identical.
//
// Reference lines restated: heat element src/rsolverheat.cpp:397-435, heat
// assembly :755-820; elasticity element src/rsolverstress.cpp:613-693,
// traction :498-507, assembly :1654-1772.
#include "assembly_plan.h"
#include "csr.cuh"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>

struct rsg_assembly {
    uint64_t id = 0;           // its own among all plans ever made; a matrix made from it carries it (rsg_csr::plan)
    uint32_t n_nodes = 0, n_tets = 0, n_tris = 0, dofs = 1, n_free = 0;
    uint64_t nnz = 0;
    double *xyz = nullptr;
    uint32_t *tets = nullptr, *tris = nullptr, *book = nullptr;
    uint32_t *row_node = nullptr;
    uint8_t *row_comp = nullptr;
    uint32_t *rp = nullptr, *ci = nullptr;
    uint32_t *adj_ptr = nullptr, *adj_elem = nullptr;
    uint8_t *adj_loc = nullptr;
    uint16_t *adj_off = nullptr;
    // heat plans, instead of xyz and adj_*: the (row, adjacent tet) pairs (AsmPair) and the coordinates by fours
    uint4 *pair = nullptr;
    uint32_t *pair_ptr = nullptr;
    double4 *xyz4 = nullptr;
    bool near = false;
    uint32_t *tadj_ptr = nullptr, *tadj_tri = nullptr;
    uint8_t *node_mask = nullptr;
    double *stage = nullptr;   // host inputs staged on the device
    size_t stage_cap = 0;
    uint32_t max_row = 0;      // longest row of the pattern (the thread-local kernels take short rows)
    int kind = 0;              // rsg::kPlanHeat / kPlanStress / kPlanMagnetostatics
};

namespace rsg {

enum { kPlanHeat = 1, kPlanStress = 2, kPlanMagnetostatics = 3 };

namespace {

__device__ __forceinline__ double tet_geometry(const double *__restrict__ xyz, const uint4 t, double G[4][3])
{
    double X0[3], a[3], b[3], c[3];
    for (int k = 0; k < 3; k++) X0[k] = xyz[3 * size_t(t.x) + k];
    for (int k = 0; k < 3; k++) {
        a[k] = xyz[3 * size_t(t.y) + k] - X0[k];
        b[k] = xyz[3 * size_t(t.z) + k] - X0[k];
        c[k] = xyz[3 * size_t(t.w) + k] - X0[k];
    }
    const double bc[3] = {b[1] * c[2] - b[2] * c[1], b[2] * c[0] - b[0] * c[2], b[0] * c[1] - b[1] * c[0]};
    const double ca[3] = {c[1] * a[2] - c[2] * a[1], c[2] * a[0] - c[0] * a[2], c[0] * a[1] - c[1] * a[0]};
    const double ab[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
    const double det = a[0] * bc[0] + a[1] * bc[1] + a[2] * bc[2];
    for (int k = 0; k < 3; k++) {
        G[1][k] = bc[k] / det;
        G[2][k] = ca[k] / det;
        G[3][k] = ab[k] / det;
        G[0][k] = -(G[1][k] + G[2][k] + G[3][k]);
    }
    return fabs(det) / 6.0;
}

// Row m of the gradient matrix selected without indexing G by a run-time m (which would put G
// in local memory).
__device__ __forceinline__ void grad_row(const double G[4][3], int m, double gm[3])
{
    for (int c = 0; c < 3; c++) gm[c] = m == 0 ? G[0][c] : m == 1 ? G[1][c] : m == 2 ? G[2][c] : G[3][c];
}

__device__ __forceinline__ uint32_t node_of(const uint4 t, int k)
{
    return k == 0 ? t.x : k == 1 ? t.y : k == 2 ? t.z : t.w;
}

// ---- heat ----
// A thread reads its (row, adjacent tet) pairs as AsmPair (assembly_plan.h), a warp's as one contiguous 512 bytes.
// The host packs them while it builds the plan: packed on the device out of the unpacked arrays, a plan of 10^3 /
// 40^3 / 100^3 hexes took 1.2 / 16.6 / 344 ms to make (1.0 / 14.9 / 332 before there were pairs) and held both, 0.7 GB
// at 100^3; packed by the host 0.7 / 14.3 / 321.

__device__ __forceinline__ double4 ld_node(const double4 *p)
{
    double4 v;  // one 32-byte load (sm_100)
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}

struct HeatIn {
    const uint4 *pair;
    const uint32_t *pair_ptr;
    const double4 *xyz;
    const uint4 *tets;
    const double *k_e, *q_e, *rhoc_e, *node_t;
    int transient;
    double alpha, dt;
    const uint32_t *row_node;
};

constexpr uint32_t kNoEntry = 0xffffu;

template <bool NEAR>
__device__ __forceinline__ void unpack_pair(const HeatIn &h, const uint4 pr, uint32_t row_node, uint32_t &m,
                                            uint32_t (&node)[4], uint32_t (&off)[4])
{
    if constexpr (NEAR) {
        m = pr.y & 3u;
        for (int n = 0; n < 4; n++) {
            const uint32_t o = (pr.y >> (2 + 6 * n)) & 63u;
            off[n] = o == 63u ? kNoEntry : o;
        }
        node[0] = row_node + uint32_t(int(int16_t(pr.z & 0xffffu)));
        node[1] = row_node + uint32_t(int(int16_t(pr.z >> 16)));
        node[2] = row_node + uint32_t(int(int16_t(pr.w & 0xffffu)));
        node[3] = row_node + uint32_t(int(int16_t(pr.w >> 16)));
    } else {
        m = pr.y;
        off[0] = pr.z & 0xffffu;
        off[1] = pr.z >> 16;
        off[2] = pr.w & 0xffffu;
        off[3] = pr.w >> 16;
        const uint4 tv = __ldg(h.tets + pr.x);
        node[0] = tv.x;
        node[1] = tv.y;
        node[2] = tv.z;
        node[3] = tv.w;
    }
}

// Contribution of one pair: Ar[n] for the tet's 4 nodes (theta scheme applied when transient) and the
// right-hand side part be (source, transient history, Dirichlet lifting).  The gradients are kept as
// cofactors c_n = det grad N_n, so that grad N_m . grad N_n |det| / 6 = c_m . c_n / (6 |det|) takes one
// division where dividing every gradient took nine.
template <bool NEAR>
__device__ __forceinline__ void heat_pair(const HeatIn &h, const uint4 pr, uint32_t row_node, double (&Ar)[4],
                                          double &be, uint32_t (&off)[4])
{
    const uint32_t e = pr.x;
    uint32_t m, node[4];
    unpack_pair<NEAR>(h, pr, row_node, m, node, off);
    const double4 p0 = ld_node(h.xyz + node[0]), p1 = ld_node(h.xyz + node[1]), p2 = ld_node(h.xyz + node[2]),
                  p3 = ld_node(h.xyz + node[3]);
    const double k = __ldg(h.k_e + e), q = __ldg(h.q_e + e);
    const double a[3] = {p1.x - p0.x, p1.y - p0.y, p1.z - p0.z};
    const double b[3] = {p2.x - p0.x, p2.y - p0.y, p2.z - p0.z};
    const double c[3] = {p3.x - p0.x, p3.y - p0.y, p3.z - p0.z};
    double C[4][3] = {{0.0, 0.0, 0.0},
                      {b[1] * c[2] - b[2] * c[1], b[2] * c[0] - b[0] * c[2], b[0] * c[1] - b[1] * c[0]},
                      {c[1] * a[2] - c[2] * a[1], c[2] * a[0] - c[0] * a[2], c[0] * a[1] - c[1] * a[0]},
                      {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]}};
    const double det = fabs(a[0] * C[1][0] + a[1] * C[1][1] + a[2] * C[1][2]);
    for (int i = 0; i < 3; i++) C[0][i] = -(C[1][i] + C[2][i] + C[3][i]);
    double cm[3];
    for (int i = 0; i < 3; i++) cm[i] = m == 0 ? C[0][i] : m == 1 ? C[1][i] : m == 2 ? C[2][i] : C[3][i];
    const double s = k / (6.0 * det), V = det / 6.0;
    for (int n = 0; n < 4; n++) Ar[n] = (cm[0] * C[n][0] + cm[1] * C[n][1] + cm[2] * C[n][2]) * s;
    const double fe = q * V / 4.0;
    if (h.transient) {
        const double rc = __ldg(h.rhoc_e + e);
        be = h.dt * fe;
        for (int n = 0; n < 4; n++) {
            const double Me = rc * V * (int(m) == n ? 2.0 : 1.0) / 20.0;
            const double Ke = Ar[n];
            Ar[n] = Me + h.alpha * h.dt * Ke;
            be += (Me - (1.0 - h.alpha) * h.dt * Ke) * __ldg(h.node_t + node[n]);
        }
    } else {
        be = fe;
    }
    for (int n = 0; n < 4; n++)
        if (off[n] == kNoEntry) be -= Ar[n] * __ldg(h.node_t + node[n]);  // a fixed node
}

// Where the assembled row goes: the CSR values and, once the matrix exists, every copy a refresh would
// otherwise make in passes of its own (FP32, SELL-32 in both precisions) and ||A||_F^2.
struct HeatOut {
    double *val;
    double *b;
    float *val32 = nullptr;  // null: only val and b
    double *sval = nullptr;  // null: no SELL-32 copy
    float *sval32 = nullptr;
    const uint32_t *slice_ptr = nullptr;
    double *partials = nullptr;
    unsigned int *ticket = nullptr;
    double *norm = nullptr;
};

// Rows accumulated in global memory (any row length); val and b only.
template <bool NEAR>
__global__ void __launch_bounds__(kBlock) k_asm_heat(uint32_t n_free, const uint32_t *__restrict__ rp, HeatIn h,
                                                     HeatOut o)
{
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n_free; r += gridDim.x * blockDim.x) {
        const uint32_t start = rp[r], end = rp[r + 1], s = r >> 5, a = h.row_node[r];
        for (uint32_t j = start; j < end; j++) o.val[j] = 0.0;
        double bs = 0.0;
        for (uint32_t t = h.pair_ptr[s]; t < h.pair_ptr[s + 1]; t++) {
            const uint4 pr = h.pair[size_t(t) * 32 + (r & 31u)];
            if (pr.x == RSG_EOD) break;
            double Ar[4], be;
            uint32_t off[4];
            heat_pair<NEAR>(h, pr, a, Ar, be, off);
            bs += be;
            for (int n = 0; n < 4; n++)
                if (off[n] != kNoEntry) o.val[start + off[n]] += Ar[n];
        }
        o.b[r] = bs;
    }
}

// One thread per row with the row accumulated in shared memory (rows of up to kLocalRowMax entries; the
// launch sizes it for the plan's longest row): the same per-entry order as k_asm_heat without
// read-modify-write round trips through global memory.  Entry j of a thread is at acc[j * (kBlock + 1) +
// thread], conflict-free both for a thread's own row and for half-warps that copy whole rows.
//
// Bound by the L1 traffic of the pairs' scattered 8-byte conductivities and sources and of the node
// coordinates (24 pairs a row; L1 at 63% and FP64 at 21% of peak in the wide form).  Whole numeric assembly
// of 100^3 hexes (6M tets, 1M rows): 945 us with separate index, offset and node arrays, nine divisions a
// pair, one thread's scattered stores and three refresh passes (703 + 94 + 136 us); 500 us with the wide
// form, 464 us with the near form.  Three blocks an SM (80 registers and 20 to 28 bytes spilled): two 524, four (64
// registers, more spills) 521 us.
// Loading the next pairs' conductivities a step ahead was slower (503-564 us), as was keeping the row's
// own node out of the loads.
constexpr uint32_t kLocalRowMax = 32;
constexpr size_t heat_local_smem(uint32_t max_row) { return size_t(max_row) * (kBlock + 1) * sizeof(double); }

template <bool NEAR>
__global__ void __launch_bounds__(kBlock, 3) k_asm_heat_local(uint32_t n_free, uint32_t max_row,
                                                           const uint32_t *__restrict__ rp, HeatIn h, HeatOut o)
{
    extern __shared__ double acc_s[];
    __shared__ double sh[32];
    constexpr uint32_t kStride = kBlock + 1;
    const uint32_t lane = threadIdx.x & 31u, wbase = threadIdx.x & ~31u;
    double *acc = acc_s + threadIdx.x;
    double nrm[1] = {0.0};
    for (uint32_t r0 = blockIdx.x * blockDim.x + wbase; r0 < n_free; r0 += gridDim.x * blockDim.x) {
        const uint32_t r = r0 + lane, s = r0 >> 5;
        const bool valid = r < n_free;
        const uint32_t start = valid ? rp[r] : 0u, len = valid ? min(rp[r + 1] - start, max_row) : 0u;
        const uint32_t a = valid ? h.row_node[r] : 0u;
        for (uint32_t j = 0; j < len; j++) acc[j * kStride] = 0.0;
        double bs = 0.0;
        const uint32_t t1 = h.pair_ptr[s + 1];
        uint32_t t = h.pair_ptr[s];
        uint4 next = t < t1 ? __ldcs(h.pair + size_t(t) * 32 + lane) : make_uint4(RSG_EOD, 0, 0, 0);
        for (; t < t1; t++) {
            const uint4 pr = next;
            if (t + 1 < t1) next = __ldcs(h.pair + size_t(t + 1) * 32 + lane);
            if (pr.x == RSG_EOD) continue;
            double Ar[4], be;
            uint32_t off[4];
            heat_pair<NEAR>(h, pr, a, Ar, be, off);
            bs += be;
            for (int n = 0; n < 4; n++)
                if (off[n] < len) acc[off[n] * kStride] += Ar[n];
        }
        if (valid) o.b[r] = bs;
        if (o.val32) {
            for (uint32_t j = 0; j < len; j++) {
                const double v = acc[j * kStride];
                nrm[0] += v * v;
            }
            if (o.sval) {
                const size_t base = size_t(o.slice_ptr[s]) + 4u * lane;
                for (uint32_t j = 0; j < len; j += 4) {
                    double v[4];
                    for (uint32_t u = 0; u < 4; u++) v[u] = j + u < len ? acc[(j + u) * kStride] : 0.0;
                    const size_t e = base + size_t(j >> 2) * 128u;
                    *reinterpret_cast<double2 *>(o.sval + e) = make_double2(v[0], v[1]);
                    *reinterpret_cast<double2 *>(o.sval + e + 2) = make_double2(v[2], v[3]);
                    *reinterpret_cast<float4 *>(o.sval32 + e) =
                        make_float4(__double2float_rn(v[0]), __double2float_rn(v[1]), __double2float_rn(v[2]),
                                    __double2float_rn(v[3]));
                }
            }
        }
        __syncwarp();
        // the CSR rows of the warp, half a warp per row: consecutive lanes store consecutive entries
        const uint32_t sub = lane & 15u;
        for (uint32_t i = 0; i < 32; i += 2) {
            const uint32_t row = i + (lane >> 4);
            const uint32_t rs = __shfl_sync(0xffffffffu, start, row), rl = __shfl_sync(0xffffffffu, len, row);
            for (uint32_t j = sub; j < rl; j += 16) {
                const double v = acc_s[j * kStride + wbase + row];
                o.val[rs + j] = v;
                if (o.val32) o.val32[rs + j] = __double2float_rn(v);
            }
        }
        __syncwarp();
    }
    if (!o.val32) return;
    double tot[1];
    if (grid_sum<1>(nrm, o.partials, o.ticket, sh, tot) && threadIdx.x == 0) *o.norm = sqrt(tot[0]);
}

// Row (3n+j) of the 12x6 strain-displacement matrix Be (strain order xx yy zz yz xz xy).
__device__ __forceinline__ void be_row(const double g[3], int j, double out[6])
{
    for (int k = 0; k < 6; k++) out[k] = 0.0;
    if (j == 0) {
        out[0] = g[0];
        out[4] = g[2];
        out[5] = g[1];
    } else if (j == 1) {
        out[1] = g[1];
        out[3] = g[2];
        out[5] = g[0];
    } else {
        out[2] = g[2];
        out[3] = g[1];
        out[4] = g[0];
    }
}

// Right-hand side of one traction triangle for component i (thickness 0: no stiffness).
__device__ __forceinline__ double traction_fe(uint32_t f, int i, const double *__restrict__ xyz,
                                              const uint32_t *__restrict__ tris, const double *__restrict__ traction,
                                              int transient, double dt)
{
    const uint32_t v0 = tris[3 * size_t(f)], v1 = tris[3 * size_t(f) + 1], v2 = tris[3 * size_t(f) + 2];
    double p[3], q[3];
    for (int k = 0; k < 3; k++) {
        p[k] = xyz[3 * size_t(v1) + k] - xyz[3 * size_t(v0) + k];
        q[k] = xyz[3 * size_t(v2) + k] - xyz[3 * size_t(v0) + k];
    }
    const double cr[3] = {p[1] * q[2] - p[2] * q[1], p[2] * q[0] - p[0] * q[2], p[0] * q[1] - p[1] * q[0]};
    const double area = 0.5 * sqrt(cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]);
    const double fe = traction[3 * size_t(f) + i] * area / 3.0;
    return transient ? dt * fe : fe;
}

// Contribution of one (row node a, component i, adjacent tet) triple: Ar[3n+j] for the
// tet's 4 nodes x 3 components (theta scheme applied when transient) and its be.
__device__ __forceinline__ void stress_adj(uint32_t t, int i, const uint32_t *__restrict__ adj_elem,
                                           const uint8_t *__restrict__ adj_loc, const double *__restrict__ xyz,
                                           const uint4 *__restrict__ tets, const uint32_t *__restrict__ book,
                                           const double *__restrict__ e_mod, const double *__restrict__ nu,
                                           const double *__restrict__ rho_e, const double *__restrict__ gravity,
                                           const double *__restrict__ texp_e, const double *__restrict__ dtemp_e,
                                           const double *__restrict__ node_u, int transient, double alpha, double dt,
                                           double (&Ar)[12], double &be, uint4 &tv)
{
    const uint32_t e = adj_elem[t];
    const int m = adj_loc[t];
    tv = tets[e];
    double G[4][3];
    const double V = tet_geometry(xyz, tv, G);
    const double E = e_mod[e], v = nu[e];
    const double f = E / ((1.0 + v) * (1.0 - 2.0 * v));
    double De[6][6];
    for (int p = 0; p < 6; p++)
        for (int q = 0; q < 6; q++) De[p][q] = 0.0;
    De[0][0] = 1.0 - v; De[0][1] = v;       De[0][2] = v;
    De[1][0] = v;       De[1][1] = 1.0 - v; De[1][2] = v;
    De[2][0] = v;       De[2][1] = v;       De[2][2] = 1.0 - v;
    De[3][3] = De[4][4] = De[5][5] = (1.0 - 2.0 * v) / 2.0;
    for (int p = 0; p < 6; p++)
        for (int q = 0; q < 6; q++) De[p][q] *= f;
    double Bm[6], BD[6];
    double gm[3];
    grad_row(G, m, gm);
    be_row(gm, i, Bm);
    for (int q = 0; q < 6; q++) {
        double s = 0.0;
        for (int k = 0; k < 6; k++) s += Bm[k] * De[k][q];
        BD[q] = s;
    }
    for (int n = 0; n < 4; n++)
        for (int j = 0; j < 3; j++) {
            double Bn[6];
            be_row(G[n], j, Bn);
            double s = 0.0;
            for (int k = 0; k < 6; k++) s += BD[k] * Bn[k];
            Ar[3 * n + j] = s * V;
        }
    double fe = gravity[i] * rho_e[e] * V / 4.0;
    for (int k = 0; k < 3; k++) fe += texp_e[e] * dtemp_e[e] * BD[k] * V;
    if (transient) {
        be = dt * fe;
        const double mv = rho_e[e] * V;
        for (int n = 0; n < 4; n++)
            for (int j = 0; j < 3; j++) {
                const double Me = (j == i) ? mv * (m == n ? 2.0 : 1.0) / 20.0 : 0.0;
                const double Ke = Ar[3 * n + j];
                Ar[3 * n + j] = Me + alpha * dt * Ke;
                be += (Me - (1.0 - alpha) * dt * Ke) * node_u[3 * size_t(node_of(tv, n)) + j];
            }
    } else {
        be = fe;
    }
    for (int n = 0; n < 4; n++) {
        const uint32_t nd = node_of(tv, n);
        for (int j = 0; j < 3; j++)
            if (book[3 * size_t(nd) + j] == RSG_EOD) be -= Ar[3 * n + j] * node_u[3 * size_t(nd) + j];
    }
}

// Rows accumulated in global memory (any row length).
__global__ void __launch_bounds__(128) k_asm_stress(
    uint32_t n_free, const uint32_t *__restrict__ row_node, const uint8_t *__restrict__ row_comp,
    const uint32_t *__restrict__ rp, const uint32_t *__restrict__ adj_ptr, const uint32_t *__restrict__ adj_elem,
    const uint8_t *__restrict__ adj_loc, const ushort4 *__restrict__ adj_off, const uint32_t *__restrict__ tadj_ptr,
    const uint32_t *__restrict__ tadj_tri, const uint8_t *__restrict__ node_mask, const double *__restrict__ xyz,
    const uint4 *__restrict__ tets, const uint32_t *__restrict__ tris, const uint32_t *__restrict__ book,
    const double *__restrict__ e_mod, const double *__restrict__ nu, const double *__restrict__ rho_e,
    const double *__restrict__ gravity, const double *__restrict__ texp_e, const double *__restrict__ dtemp_e,
    const double *__restrict__ traction, const double *__restrict__ node_u, int transient, double alpha, double dt,
    double *__restrict__ val, double *__restrict__ b)
{
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n_free; r += gridDim.x * blockDim.x) {
        const uint32_t a = row_node[r], start = rp[r], end = rp[r + 1];
        const int i = row_comp[r];
        for (uint32_t j = start; j < end; j++) val[j] = 0.0;
        double bs = 0.0;
        for (uint32_t t = tadj_ptr[a]; t < tadj_ptr[a + 1]; t++)
            bs += traction_fe(tadj_tri[t], i, xyz, tris, traction, transient, dt);
        for (uint32_t t = adj_ptr[a]; t < adj_ptr[a + 1]; t++) {
            double Ar[12], be;
            uint4 tv;
            stress_adj(t, i, adj_elem, adj_loc, xyz, tets, book, e_mod, nu, rho_e, gravity, texp_e, dtemp_e, node_u,
                       transient, alpha, dt, Ar, be, tv);
            bs += be;
            const ushort4 off4 = adj_off[t];
            const uint16_t off[4] = {off4.x, off4.y, off4.z, off4.w};
            for (int n = 0; n < 4; n++) {
                if (off[n] == 0xffffu) continue;
                const uint8_t mask = node_mask[node_of(tv, n)];
                uint32_t rank = 0;
                for (int j = 0; j < 3; j++)
                    if (mask & (1u << j)) val[start + off[n] + rank++] += Ar[3 * n + j];
            }
        }
        b[r] = bs;
    }
}

// One thread per row with the row accumulated in shared memory (rows of up to
// kLocalStressRowMax entries, the launch sizes it for the plan's longest row), as k_asm_heat_local.
constexpr uint32_t kLocalStressRowMax = 96;
constexpr int kStressBlock = 128;
constexpr size_t kStressLocalSmemMax = size_t(kLocalStressRowMax) * kStressBlock * sizeof(double);

__global__ void __launch_bounds__(128) k_asm_stress_local(
    uint32_t n_free, const uint32_t *__restrict__ row_node, const uint8_t *__restrict__ row_comp,
    const uint32_t *__restrict__ rp, const uint32_t *__restrict__ adj_ptr, const uint32_t *__restrict__ adj_elem,
    const uint8_t *__restrict__ adj_loc, const ushort4 *__restrict__ adj_off, const uint32_t *__restrict__ tadj_ptr,
    const uint32_t *__restrict__ tadj_tri, const uint8_t *__restrict__ node_mask, const double *__restrict__ xyz,
    const uint4 *__restrict__ tets, const uint32_t *__restrict__ tris, const uint32_t *__restrict__ book,
    const double *__restrict__ e_mod, const double *__restrict__ nu, const double *__restrict__ rho_e,
    const double *__restrict__ gravity, const double *__restrict__ texp_e, const double *__restrict__ dtemp_e,
    const double *__restrict__ traction, const double *__restrict__ node_u, int transient, double alpha, double dt,
    double *__restrict__ val, double *__restrict__ b)
{
    extern __shared__ double acc_s[];
    double *acc = acc_s + threadIdx.x;
    const uint32_t stride = blockDim.x;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n_free; r += gridDim.x * blockDim.x) {
        const uint32_t a = row_node[r], start = rp[r], len = min(rp[r + 1] - start, kLocalStressRowMax);
        const int i = row_comp[r];
        for (uint32_t j = 0; j < len; j++) acc[j * stride] = 0.0;
        double bs = 0.0;
        for (uint32_t t = tadj_ptr[a]; t < tadj_ptr[a + 1]; t++)
            bs += traction_fe(tadj_tri[t], i, xyz, tris, traction, transient, dt);
        for (uint32_t t = adj_ptr[a]; t < adj_ptr[a + 1]; t++) {
            double Ar[12], be;
            uint4 tv;
            stress_adj(t, i, adj_elem, adj_loc, xyz, tets, book, e_mod, nu, rho_e, gravity, texp_e, dtemp_e, node_u,
                       transient, alpha, dt, Ar, be, tv);
            bs += be;
            const ushort4 off4 = adj_off[t];
            const uint16_t off[4] = {off4.x, off4.y, off4.z, off4.w};
            for (int n = 0; n < 4; n++) {
                if (off[n] == 0xffffu) continue;
                const uint8_t mask = node_mask[node_of(tv, n)];
                uint32_t rank = 0;
                for (int j = 0; j < 3; j++)
                    if (mask & (1u << j)) {
                        const uint32_t pos = off[n] + rank++;
                        if (pos < len) acc[pos * stride] += Ar[3 * n + j];
                    }
            }
        }
        for (uint32_t j = 0; j < len; j++) val[start + j] = acc[j * stride];
        b[r] = bs;
    }
}

// vacuum permittivity, RSolverGeneric::e0 (src/rsolvergeneric.cpp:13)
constexpr double kE0 = 8.854187817e-12;

// Contribution of one (row node, component i, adjacent tet) triple to a magnetostatic row
// (src/rsolvermagnetostatics.cpp:94-119, lifting :240-254): Ar[3n+j] = -(grad N_m . grad N_n) V
// on the component diagonal (j == i) and an explicit 0 elsewhere, be = e0 V/4 (grad N_m x J)_i
// with J the row node's current density, minus the lifting by disabled nodes' potentials.
__device__ __forceinline__ void magneto_adj(uint32_t t, int i, const uint32_t *__restrict__ adj_elem,
                                            const uint8_t *__restrict__ adj_loc, const double *__restrict__ xyz,
                                            const uint4 *__restrict__ tets, const uint32_t *__restrict__ book,
                                            const double *__restrict__ J, const double *__restrict__ node_a,
                                            double (&Ar)[12], double &be, uint4 &tv)
{
    const uint32_t e = adj_elem[t];
    const int m = adj_loc[t];
    tv = tets[e];
    double G[4][3];
    const double V = tet_geometry(xyz, tv, G);
    double gm[3];
    grad_row(G, m, gm);
    for (int n = 0; n < 4; n++) {
        const double v = (gm[0] * G[n][0] + gm[1] * G[n][1] + gm[2] * G[n][2]) * V;
        for (int j = 0; j < 3; j++) Ar[3 * n + j] = j == i ? 0.0 - v : 0.0;
    }
    const double js = i == 0 ? -gm[2] * J[1] + gm[1] * J[2]
                    : i == 1 ? gm[2] * J[0] - gm[0] * J[2]
                             : -gm[1] * J[0] + gm[0] * J[1];
    be = V / 4.0 * kE0 * js;
    for (int n = 0; n < 4; n++) {
        const uint32_t nd = node_of(tv, n);
        if (book[3 * size_t(nd)] == RSG_EOD)
            for (int j = 0; j < 3; j++) be -= Ar[3 * n + j] * node_a[3 * size_t(nd) + j];
    }
}

// One thread per row, the row accumulated in global memory (any row length).
__global__ void __launch_bounds__(128) k_asm_magneto(
    uint32_t n_free, const uint32_t *__restrict__ row_node, const uint8_t *__restrict__ row_comp,
    const uint32_t *__restrict__ rp, const uint32_t *__restrict__ adj_ptr, const uint32_t *__restrict__ adj_elem,
    const uint8_t *__restrict__ adj_loc, const ushort4 *__restrict__ adj_off, const uint8_t *__restrict__ node_mask,
    const double *__restrict__ xyz, const uint4 *__restrict__ tets, const uint32_t *__restrict__ book,
    const double *__restrict__ node_j, const double *__restrict__ node_a, double *__restrict__ val,
    double *__restrict__ b)
{
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n_free; r += gridDim.x * blockDim.x) {
        const uint32_t a = row_node[r], start = rp[r], len = rp[r + 1] - start;
        const int i = row_comp[r];
        for (uint32_t j = 0; j < len; j++) val[start + j] = 0.0;
        const double J[3] = {node_j[3 * size_t(a)], node_j[3 * size_t(a) + 1], node_j[3 * size_t(a) + 2]};
        double bs = 0.0;
        for (uint32_t t = adj_ptr[a]; t < adj_ptr[a + 1]; t++) {
            double Ar[12], be;
            uint4 tv;
            magneto_adj(t, i, adj_elem, adj_loc, xyz, tets, book, J, node_a, Ar, be, tv);
            bs += be;
            const ushort4 off4 = adj_off[t];
            const uint16_t off[4] = {off4.x, off4.y, off4.z, off4.w};
            for (int n = 0; n < 4; n++) {
                if (off[n] == 0xffffu) continue;
                const uint8_t mask = node_mask[node_of(tv, n)];
                uint32_t rank = 0;
                for (int j = 0; j < 3; j++)
                    if (mask & (1u << j)) val[start + off[n] + rank++] += Ar[3 * n + j];
            }
        }
        b[r] = bs;
    }
}

// One thread per free node.  Its three component rows (3p, 3p+1, 3p+2: a node's components are
// enabled or disabled together, checked when the plan is made) share the column pattern, the
// element geometry and the -(grad N_m . grad N_n) V values of the diagonal blocks, so each
// adjacent tet's geometry is computed once for the three rows, and one shared-memory slot per
// neighbour node accumulates the diagonal-block value.  Entry (n, j) of row i is that sum when
// j == i and an exact +0.0 otherwise; the right-hand side of each row follows magneto_adj's
// sequence.  The bits equal the row kernel's (tests compare them).
__global__ void __launch_bounds__(128) k_asm_magneto_node(
    uint32_t n_free_nodes, const uint32_t *__restrict__ row_node, const uint32_t *__restrict__ rp,
    const uint32_t *__restrict__ adj_ptr, const uint32_t *__restrict__ adj_elem, const uint8_t *__restrict__ adj_loc,
    const ushort4 *__restrict__ adj_off, const double *__restrict__ xyz, const uint4 *__restrict__ tets,
    const uint32_t *__restrict__ book, const double *__restrict__ node_j, const double *__restrict__ node_a,
    double *__restrict__ val, double *__restrict__ b)
{
    extern __shared__ double acc_s[];
    double *acc = acc_s + threadIdx.x;
    const uint32_t stride = blockDim.x;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n_free_nodes; q += gridDim.x * blockDim.x) {
        const uint32_t r0 = 3 * q, a = row_node[r0], len = rp[r0 + 1] - rp[r0];
        const uint32_t slots = min(len / 3, kLocalStressRowMax / 3);
        for (uint32_t s = 0; s < slots; s++) acc[s * stride] = 0.0;
        const double J[3] = {node_j[3 * size_t(a)], node_j[3 * size_t(a) + 1], node_j[3 * size_t(a) + 2]};
        double bs[3] = {0.0, 0.0, 0.0};
        for (uint32_t t = adj_ptr[a]; t < adj_ptr[a + 1]; t++) {
            const uint32_t e = adj_elem[t];
            const int m = adj_loc[t];
            const uint4 tv = tets[e];
            double G[4][3];
            const double V = tet_geometry(xyz, tv, G);
            double gm[3];
            grad_row(G, m, gm);
            double dv[4];  // diagonal-block value of the pair (m, n)
            for (int n = 0; n < 4; n++) dv[n] = 0.0 - (gm[0] * G[n][0] + gm[1] * G[n][1] + gm[2] * G[n][2]) * V;
            const double js[3] = {-gm[2] * J[1] + gm[1] * J[2], gm[2] * J[0] - gm[0] * J[2],
                                  -gm[1] * J[0] + gm[0] * J[1]};
            double be[3];
            for (int i = 0; i < 3; i++) be[i] = V / 4.0 * kE0 * js[i];
            for (int n = 0; n < 4; n++) {
                const uint32_t nd = node_of(tv, n);
                if (book[3 * size_t(nd)] == RSG_EOD)
                    for (int i = 0; i < 3; i++)
                        for (int j = 0; j < 3; j++) be[i] -= (j == i ? dv[n] : 0.0) * node_a[3 * size_t(nd) + j];
            }
            for (int i = 0; i < 3; i++) bs[i] += be[i];
            const ushort4 off4 = adj_off[t];
            const uint16_t off[4] = {off4.x, off4.y, off4.z, off4.w};
            for (int n = 0; n < 4; n++)
                if (off[n] != 0xffffu && off[n] / 3u < slots) acc[(off[n] / 3u) * stride] += dv[n];
        }
        for (int i = 0; i < 3; i++) {
            const uint32_t start = rp[r0 + i];
            for (uint32_t s = 0; s < slots; s++) {
                const double d = acc[s * stride];
                for (int j = 0; j < 3; j++) val[start + 3 * s + j] = j == i ? d : 0.0;
            }
            b[r0 + i] = bs[i];
        }
    }
}

// node_values[node * dofs + c] = x[book[node * dofs + c]] for every free DOF (the
// Dirichlet values stay): the solution back into the nodal field, e.g. the
// previous-step temperatures of the next transient assembly.
__global__ void k_asm_scatter(uint32_t n_entries, const uint32_t *__restrict__ book, const double *__restrict__ x,
                              double *__restrict__ node_values)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_entries; i += gridDim.x * blockDim.x) {
        const uint32_t pos = book[i];
        if (pos != RSG_EOD) node_values[i] = x[pos];
    }
}

// RSG_ASM_ROW_THREADS=1 selects the kernels that accumulate in global memory (tests compare the two)
bool row_threads_forced()
{
    const char *v = std::getenv("RSG_ASM_ROW_THREADS");
    return v && v[0] == '1';
}

template <typename T>
rsg_status upload(rsg_context *ctx, T **dst, const T *src, size_t count)
{
    if (count == 0) count = 1;
    RSG_CHECK_CUDA(ctx, cudaMalloc(dst, count * sizeof(T)));
    if (src) RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(*dst, src, count * sizeof(T), cudaMemcpyHostToDevice, ctx->stream));
    return RSG_OK;
}

void free_plan(rsg_assembly *p)
{
    if (!p) return;
    void *ptrs[] = {p->xyz, p->tets, p->tris, p->book, p->row_node, p->row_comp, p->rp, p->ci, p->adj_ptr,
                    p->adj_elem, p->adj_loc, p->adj_off, p->pair,     p->pair_ptr, p->xyz4, p->tadj_ptr,
                    p->tadj_tri, p->node_mask, p->stage};
    for (void *q : ptrs)
        if (q) cudaFree(q);
    delete p;
}

rsg_status create_plan(rsg_context *ctx, uint32_t n_nodes, const double *xyz, uint32_t n_tets, const uint32_t *tets,
                       uint32_t n_tris, const uint32_t *tris, const uint32_t *book, uint32_t dofs, uint32_t n_free,
                       int kind, rsg_assembly **out)
{
    if (!ctx || !out || !xyz || !tets || !book || n_nodes == 0 || n_tets == 0 || n_free == 0 ||
        (n_tris && !tris))
        return set_error(ctx, RSG_ERR_INVALID_ARG, "assembly_create: bad arguments");
    *out = nullptr;
    RSG_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    AsmPlanHost H;
    std::string err;
    const bool heat = kind == kPlanHeat;
    if (!build_assembly_plan(n_nodes, n_tets, tets, n_tris, tris, book, dofs, n_free, heat, H, err))
        return set_error(ctx, RSG_ERR_INVALID_ARG, "assembly_create: %s", err.c_str());
    static std::atomic<uint64_t> plans{0};
    auto *p = new rsg_assembly;
    p->id = ++plans;
    p->kind = kind;
    p->n_nodes = n_nodes;
    p->n_tets = n_tets;
    p->n_tris = n_tris;
    p->dofs = dofs;
    p->n_free = n_free;
    p->nnz = H.ci.size();
    for (size_t r = 0; r + 1 < H.rp.size(); r++) p->max_row = std::max(p->max_row, H.rp[r + 1] - H.rp[r]);
    rsg_status s = RSG_OK;
    auto chk = [&](rsg_status r) {
        if (s == RSG_OK) s = r;
    };
    std::vector<double> xyz4;
    if (heat) {
        xyz4.resize(size_t(n_nodes) * 4);
        for (size_t i = 0; i < n_nodes; i++)
            for (int k = 0; k < 3; k++) xyz4[4 * i + k] = xyz[3 * i + k];
        p->near = H.near;
        chk(upload(ctx, &p->xyz4, reinterpret_cast<const double4 *>(xyz4.data()), n_nodes));
        chk(upload(ctx, &p->pair, reinterpret_cast<const uint4 *>(H.pair.get()), size_t(H.pair_ptr.back()) * 32));
        chk(upload(ctx, &p->pair_ptr, H.pair_ptr.data(), H.pair_ptr.size()));
    } else {
        chk(upload(ctx, &p->xyz, xyz, size_t(n_nodes) * 3));
        chk(upload(ctx, &p->adj_ptr, H.adj_ptr.data(), H.adj_ptr.size()));
        chk(upload(ctx, &p->adj_elem, H.adj_elem.data(), H.adj_elem.size()));
        chk(upload(ctx, &p->adj_loc, H.adj_loc.data(), H.adj_loc.size()));
        chk(upload(ctx, &p->adj_off, H.adj_off.data(), H.adj_off.size()));
    }
    chk(upload(ctx, &p->tets, tets, size_t(n_tets) * 4));
    chk(upload(ctx, &p->tris, n_tris ? tris : nullptr, size_t(n_tris) * 3));
    chk(upload(ctx, &p->book, book, size_t(n_nodes) * dofs));
    chk(upload(ctx, &p->row_node, H.row_node.data(), H.row_node.size()));
    chk(upload(ctx, &p->row_comp, H.row_comp.data(), H.row_comp.size()));
    chk(upload(ctx, &p->rp, H.rp.data(), H.rp.size()));
    chk(upload(ctx, &p->ci, H.ci.data(), H.ci.size()));
    chk(upload(ctx, &p->tadj_ptr, H.tadj_ptr.data(), H.tadj_ptr.size()));
    chk(upload(ctx, &p->tadj_tri, H.tadj_tri.empty() ? nullptr : H.tadj_tri.data(), H.tadj_tri.size()));
    chk(upload(ctx, &p->node_mask, H.node_mask.data(), H.node_mask.size()));
    if (s == RSG_OK) {
        cudaError_t e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) s = set_error(ctx, RSG_ERR_CUDA, "assembly upload: %s", cudaGetErrorString(e));
    }
    if (s != RSG_OK) {
        free_plan(p);
        return s;
    }
    *out = p;
    return RSG_OK;
}

// Stage host arrays on the device; returns device pointers in the same order.
rsg_status stage_inputs(rsg_context *ctx, rsg_assembly *p, int32_t memory, std::initializer_list<size_t> counts,
                        std::initializer_list<const double *> srcs, const double **dst)
{
    if (memory == RSG_MEM_DEVICE) {
        size_t k = 0;
        for (const double *s : srcs) dst[k++] = s;
        return RSG_OK;
    }
    size_t total = 0;
    for (size_t c : counts) total += (c + 31) & ~size_t(31);
    if (total > p->stage_cap) {
        if (p->stage) {
            RSG_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            cudaFree(p->stage);
        }
        p->stage = nullptr;
        RSG_CHECK_CUDA(ctx, cudaMalloc(&p->stage, total * sizeof(double)));
        p->stage_cap = total;
    }
    size_t o = 0, k = 0;
    auto ci = counts.begin();
    for (const double *s : srcs) {
        const size_t c = *ci++;
        if (s) {
            RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(p->stage + o, s, c * sizeof(double), cudaMemcpyHostToDevice,
                                                ctx->stream));
            dst[k] = p->stage + o;
        } else {
            dst[k] = nullptr;
        }
        k++;
        o += (c + 31) & ~size_t(31);
    }
    return RSG_OK;
}

// Create *A from the plan pattern on the first call; afterwards write into its values.
template <class Launch>
rsg_status assemble_into(rsg_context *ctx, rsg_assembly *p, rsg_csr **A, Launch launch)
{
    if (*A) {
        if ((*A)->n != p->n_free || (*A)->nnz != p->nnz)
            return set_error(ctx, RSG_ERR_INVALID_ARG, "assemble: matrix does not match the plan's pattern");
        launch((*A)->val);
        RSG_CHECK_CUDA(ctx, cudaGetLastError());
        return csr_refresh(ctx, *A);
    }
    double *tmp = nullptr;
    RSG_CHECK_CUDA(ctx, cudaMalloc(&tmp, std::max<size_t>(p->nnz, 1) * sizeof(double)));
    launch(tmp);
    cudaError_t e = cudaGetLastError();
    rsg_status s = e == cudaSuccess ? RSG_OK : set_error(ctx, RSG_ERR_CUDA, "assemble: %s", cudaGetErrorString(e));
    if (s == RSG_OK) s = rsg_csr_create(ctx, p->n_free, p->rp, p->ci, tmp, RSG_MEM_DEVICE, A);
    if (s == RSG_OK) (*A)->plan = p->id;
    cudaStreamSynchronize(ctx->stream);
    cudaFree(tmp);
    return s;
}

}  // namespace
}  // namespace rsg

using namespace rsg;

extern "C" {

rsg_status rsg_assembly_create_heat(rsg_context *ctx, uint32_t n_nodes, const double *xyz, uint32_t n_tets,
                                    const uint32_t *tets, const uint32_t *book, uint32_t n_free, rsg_assembly **out)
{
    return create_plan(ctx, n_nodes, xyz, n_tets, tets, 0, nullptr, book, 1, n_free, kPlanHeat, out);
}

rsg_status rsg_assembly_create_stress(rsg_context *ctx, uint32_t n_nodes, const double *xyz, uint32_t n_tets,
                                      const uint32_t *tets, uint32_t n_tris, const uint32_t *tris,
                                      const uint32_t *book, uint32_t n_free, rsg_assembly **out)
{
    return create_plan(ctx, n_nodes, xyz, n_tets, tets, n_tris, tris, book, 3, n_free, kPlanStress, out);
}

rsg_status rsg_assembly_create_magnetostatics(rsg_context *ctx, uint32_t n_nodes, const double *xyz,
                                              uint32_t n_tets, const uint32_t *tets, const uint32_t *book,
                                              uint32_t n_free, rsg_assembly **out)
{
    if (!ctx || !book || !out) return set_error(ctx, RSG_ERR_INVALID_ARG, "assembly_create_magnetostatics: bad arguments");
    // one node book position per node (src/rsolvermagnetostatics.cpp:245, :261): the three
    // potential components of a node are enabled or disabled together, at 3 * position + c
    for (uint32_t nd = 0; nd < n_nodes; nd++) {
        const int eod = int(book[3 * size_t(nd)] == RSG_EOD) + int(book[3 * size_t(nd) + 1] == RSG_EOD) +
                        int(book[3 * size_t(nd) + 2] == RSG_EOD);
        if (eod != 0 && eod != 3)
            return set_error(ctx, RSG_ERR_INVALID_ARG,
                             "assembly_create_magnetostatics: node %u has some but not all components disabled", nd);
        const uint32_t p0 = book[3 * size_t(nd)];
        if (eod == 0 && (p0 % 3 != 0 || book[3 * size_t(nd) + 1] != p0 + 1 || book[3 * size_t(nd) + 2] != p0 + 2))
            return set_error(ctx, RSG_ERR_INVALID_ARG,
                             "assembly_create_magnetostatics: node %u: components must sit at 3*position + c", nd);
    }
    return create_plan(ctx, n_nodes, xyz, n_tets, tets, 0, nullptr, book, 3, n_free, kPlanMagnetostatics, out);
}

void rsg_assembly_destroy(rsg_context *ctx, rsg_assembly *plan)
{
    if (ctx) {
        cudaSetDevice(ctx->device);
        cudaStreamSynchronize(ctx->stream);
    }
    free_plan(plan);
}

rsg_status rsg_assembly_info(const rsg_assembly *plan, uint32_t *n_free, uint64_t *nnz)
{
    if (!plan) return RSG_ERR_INVALID_ARG;
    if (n_free) *n_free = plan->n_free;
    if (nnz) *nnz = plan->nnz;
    return RSG_OK;
}

rsg_status rsg_assemble_heat(rsg_context *ctx, rsg_assembly *p, const double *k_e, const double *q_e,
                             const double *rhoc_e, const double *node_t, const rsg_time *time, int32_t memory,
                             rsg_csr **A, double *b_device)
{
    if (!ctx || !p || !k_e || !q_e || !node_t || !A || !b_device || p->kind != kPlanHeat)
        return set_error(ctx, RSG_ERR_INVALID_ARG, "assemble_heat: bad arguments");
    const bool transient = time && time->transient;
    if (transient && !rhoc_e) return set_error(ctx, RSG_ERR_INVALID_ARG, "assemble_heat: transient needs rhoc_e");
    RSG_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    const double *d[4];
    RSG_TRY(stage_inputs(ctx, p, memory, {p->n_tets, p->n_tets, p->n_tets, p->n_nodes},
                         {k_e, q_e, transient ? rhoc_e : nullptr, node_t}, d));
    const double alpha = time ? time->alpha : 1.0, dt = time ? time->dt : 0.0;
    const HeatIn h{p->pair, p->pair_ptr, p->xyz4, reinterpret_cast<const uint4 *>(p->tets), d[0], d[1], d[2], d[3],
                   transient ? 1 : 0, alpha, dt, p->row_node};
    auto rows_kernel = p->near ? k_asm_heat<true> : k_asm_heat<false>;
    auto local_kernel = p->near ? k_asm_heat_local<true> : k_asm_heat_local<false>;
    if (p->max_row > kLocalRowMax || row_threads_forced()) {
        const int grid = std::min(grid_for(ctx, (const void *)rows_kernel, kBlock, 0, p->n_free), kMaxGrid * 4);
        return assemble_into(ctx, p, A, [&](double *val) {
            rows_kernel<<<grid, kBlock, 0, ctx->stream>>>(p->n_free, p->rp, h, HeatOut{val, b_device});
        });
    }
    // shared memory for the plan's longest row only (15 entries on tet meshes of structured hexes)
    const uint32_t rows = std::max<uint32_t>(p->max_row, 1);
    const size_t smem = heat_local_smem(rows);
    RSG_CHECK_CUDA(ctx, cudaFuncSetAttribute(local_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             int(heat_local_smem(kLocalRowMax))));
    const int grid = std::min(grid_for(ctx, (const void *)local_kernel, kBlock, smem, p->n_free), kMaxGrid);
    // The kernel lays the copies out by the plan's rows, so it writes them only into a matrix that was made from
    // this plan; one of another pattern with the same counts (a renumbered mesh) has other slices.
    if (!*A || (*A)->plan != p->id)
        return assemble_into(ctx, p, A, [&](double *val) {
            local_kernel<<<grid, kBlock, smem, ctx->stream>>>(p->n_free, rows, p->rp, h, HeatOut{val, b_device});
        });
    rsg_csr *M = *A;
    RSG_TRY(arena_reserve(ctx, arena_bytes(32, sizeof(double)) + arena_bytes(size_t(grid), sizeof(double))));
    double *scal = arena_take<double>(ctx, 32);
    HeatOut o{M->val, b_device};
    o.val32 = M->val32;
    o.sval = M->sval;
    o.sval32 = M->sval32;
    o.slice_ptr = M->slice_ptr;
    o.partials = arena_take<double>(ctx, grid);
    o.ticket = reinterpret_cast<unsigned int *>(scal + 16);
    o.norm = scal;
    RSG_CHECK_CUDA(ctx, cudaMemsetAsync(scal, 0, 32 * sizeof(double), ctx->stream));
    local_kernel<<<grid, kBlock, smem, ctx->stream>>>(p->n_free, rows, p->rp, h, o);
    RSG_CHECK_CUDA(ctx, cudaGetLastError());
    RSG_CHECK_CUDA(ctx, cudaMemcpyAsync(ctx->pinned, scal, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    RSG_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    M->norm = ctx->pinned[0];
    return RSG_OK;
}

rsg_status rsg_assemble_stress(rsg_context *ctx, rsg_assembly *p, const double *e_mod, const double *nu,
                               const double *rho_e, const double *gravity, const double *texp_e,
                               const double *dtemp_e, const double *traction, const double *node_u,
                               const rsg_time *time, int32_t memory, rsg_csr **A, double *b_device)
{
    if (!ctx || !p || !e_mod || !nu || !rho_e || !gravity || !texp_e || !dtemp_e || !node_u || !A || !b_device ||
        p->kind != kPlanStress || (p->n_tris && !traction))
        return set_error(ctx, RSG_ERR_INVALID_ARG, "assemble_stress: bad arguments");
    RSG_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    const bool transient = time && time->transient;
    const double *d[8];
    RSG_TRY(stage_inputs(ctx, p, memory,
                         {p->n_tets, p->n_tets, p->n_tets, 3, p->n_tets, p->n_tets, size_t(p->n_tris) * 3,
                          size_t(p->n_nodes) * 3},
                         {e_mod, nu, rho_e, gravity, texp_e, dtemp_e, p->n_tris ? traction : nullptr, node_u}, d));
    const double alpha = time ? time->alpha : 1.0, dt = time ? time->dt : 0.0;
    const bool local = p->max_row <= kLocalStressRowMax && !row_threads_forced();
    auto kern = local ? k_asm_stress_local : k_asm_stress;
    const int block = kStressBlock;
    const size_t smem = local ? size_t(std::max<uint32_t>(p->max_row, 1)) * block * sizeof(double) : 0;
    if (local)
        RSG_CHECK_CUDA(ctx, cudaFuncSetAttribute(k_asm_stress_local, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 int(kStressLocalSmemMax)));
    const int grid = std::min(grid_for(ctx, (const void *)kern, block, smem, p->n_free), kMaxGrid * 4);
    return assemble_into(ctx, p, A, [&](double *val) {
        kern<<<grid, block, smem, ctx->stream>>>(
            p->n_free, p->row_node, p->row_comp, p->rp, p->adj_ptr, p->adj_elem, p->adj_loc,
            reinterpret_cast<const ushort4 *>(p->adj_off), p->tadj_ptr, p->tadj_tri, p->node_mask, p->xyz,
            reinterpret_cast<const uint4 *>(p->tets), p->tris, p->book, d[0], d[1], d[2], d[3], d[4], d[5], d[6],
            d[7], transient ? 1 : 0, alpha, dt, val, b_device);
    });
}

rsg_status rsg_assemble_magnetostatics(rsg_context *ctx, rsg_assembly *p, const double *node_j,
                                       const double *node_a, int32_t memory, rsg_csr **A, double *b_device)
{
    if (!ctx || !p || !node_j || !node_a || !A || !b_device || p->kind != kPlanMagnetostatics)
        return set_error(ctx, RSG_ERR_INVALID_ARG, "assemble_magnetostatics: bad arguments");
    RSG_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    const double *d[2];
    RSG_TRY(stage_inputs(ctx, p, memory, {size_t(p->n_nodes) * 3, size_t(p->n_nodes) * 3}, {node_j, node_a}, d));
    const int block = kStressBlock;
    if (p->max_row <= kLocalStressRowMax && !row_threads_forced()) {
        const uint32_t nodes = p->n_free / 3;
        const size_t smem = size_t(std::max<uint32_t>(p->max_row / 3, 1)) * block * sizeof(double);
        const int grid = std::min(grid_for(ctx, (const void *)k_asm_magneto_node, block, smem, nodes), kMaxGrid * 4);
        return assemble_into(ctx, p, A, [&](double *val) {
            k_asm_magneto_node<<<grid, block, smem, ctx->stream>>>(
                nodes, p->row_node, p->rp, p->adj_ptr, p->adj_elem, p->adj_loc,
                reinterpret_cast<const ushort4 *>(p->adj_off), p->xyz, reinterpret_cast<const uint4 *>(p->tets),
                p->book, d[0], d[1], val, b_device);
        });
    }
    const int grid = std::min(grid_for(ctx, (const void *)k_asm_magneto, block, 0, p->n_free), kMaxGrid * 4);
    return assemble_into(ctx, p, A, [&](double *val) {
        k_asm_magneto<<<grid, block, 0, ctx->stream>>>(p->n_free, p->row_node, p->row_comp, p->rp, p->adj_ptr,
                                                       p->adj_elem, p->adj_loc,
                                                       reinterpret_cast<const ushort4 *>(p->adj_off), p->node_mask,
                                                       p->xyz, reinterpret_cast<const uint4 *>(p->tets), p->book,
                                                       d[0], d[1], val, b_device);
    });
}

rsg_status rsg_assembly_scatter(rsg_context *ctx, const rsg_assembly *p, const double *x_device,
                                double *node_values_device)
{
    if (!ctx || !p || !x_device || !node_values_device)
        return set_error(ctx, RSG_ERR_INVALID_ARG, "assembly_scatter: bad arguments");
    RSG_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    const uint32_t ne = p->n_nodes * p->dofs;
    const int grid = std::min(grid_for(ctx, (const void *)k_asm_scatter, kBlock, 0, ne), kMaxGrid);
    k_asm_scatter<<<grid, kBlock, 0, ctx->stream>>>(ne, p->book, x_device, node_values_device);
    RSG_CHECK_CUDA(ctx, cudaGetLastError());
    return RSG_OK;
}

}  // extern "C"
