// Internal interface of restarted (flexible) GMRES.
#pragma once

#include "krylov.cuh"

#include <cmath>

namespace rsg {

constexpr uint32_t kMaxRestart = 128;
constexpr uint32_t kVInv = kMaxRestart + 2;

struct GmresState {
    double beta;          // ||r|| at the start of the current cycle
    double bn, an, xn;
    double error, trend, cvg, eps, rtol;
    uint32_t m, max_outer;
    uint32_t outer;       // cycles started
    uint32_t outer_logged;
    uint32_t total_inner;
    uint32_t k;           // current inner step
    uint32_t cycle_len;   // Krylov vectors used by the current cycle
    int32_t inner_done;
    float zscale;         // FP32 without a preconditioner: factor of the next slot of Z (zscale_for)
    int32_t done, status, converged, stop_rule;
    unsigned int ticket[8];
    double *history;
    double *trend_hist;
};

struct GmresArgs {
    const rsg_csr *A;
    Precond P;
    const double *b;
    double *x;
    double *partials;     // >= (m+1) * kMaxGrid doubles
    GmresState *st;
    uint32_t m;
    bool flexible;
    // carved buffers (V, Z in FP64, or V32, Z32 in mixed precision; slot stride gmres_ld(n)); inv[k] is
    // the factor that turns slot k of Z into z_k, inv[kVInv + k] that of slot k of V into v_k
    double *V, *Z, *ro, *H, *cs, *sn, *g, *y, *hv, *wnorm, *inv;
    bool mixed = false;
    float *V32 = nullptr, *Z32 = nullptr;
    uint32_t st_max_outer;
    rsg_learned *G = nullptr;   // learned (variable) preconditioner: z_k = M(v_k)
    uint32_t *fallbacks = nullptr;  // out: cycles handed over to Jacobi
};

// The power of two next to 1 / size, as far as FP32 holds it and its inverse (1 for a size of 0, inf or NaN).
__host__ __device__ inline float zscale_for(double size)
{
    if (!(size > 0.0) || size > 1.7976931348623157e308) return 1.f;
    int e;
    (void)frexp(size, &e);
    return ldexpf(1.f, e > 120 ? -120 : e < -120 ? 120 : -e);
}

// Elements between two basis vectors: slots start on 16 bytes in either precision.
inline size_t gmres_ld(uint32_t n) { return (size_t(n) + 3) & ~size_t(3); }
size_t gmres_workspace_bytes(uint32_t n, uint32_t m, bool mixed, uint32_t w);
rsg_status gmres_carve(rsg_context *ctx, GmresArgs &a, uint32_t n, uint32_t m);
rsg_status gmres_run(rsg_context *ctx, const GmresArgs &a, double *seconds);

}  // namespace rsg
