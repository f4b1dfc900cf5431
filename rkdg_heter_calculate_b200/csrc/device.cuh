// Device code shared by the CUDA translation units: basis tables, state packs,
// physics helpers, the stage kernels' functions and the limiter's arithmetic.
// Each unit has its own copy of the tables in constant memory
// (upload_module_tables).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <string>
#include <type_traits>

#include "per_device.hpp"
#include "rkdg_internal.hpp"
#include "roots.cuh"

namespace rkdg {

// -------------------------------------------------------------- tables --
template <typename Real>
struct Tab {
    Real vphi[kMaxNQ][kMaxNB];
    Real vdxi[kMaxNQ][kMaxNB];  // weight * d psi / d xi
    Real veta[kMaxNQ][kMaxNB];  // weight * d psi / d eta
    Real ephi[3][kMaxNG][kMaxNB];
    Real ephiw[3][kMaxNG][kMaxNB];  // 2 w_g psi_i at point g of edge k (surface projection)
    Real ew[kMaxNG];
    Real mphi[3][2];
    Real minv[2][3];
};

// rule configurations: index = 2 * (nq == 7 ? 0 : nq == 6 ? 1 : 2) + (ng == 3 ? 0 : 1)
constexpr int kNumCfg = 6;
static __constant__ Tab<double> c_tab_d[kNumCfg];
static __constant__ Tab<float> c_tab_f[kNumCfg];

// FP32 tables with every value in both lanes of a pair, for the packed
// two-lane FP32 arithmetic (f32x2) of the tile kernel; nephiw = -(2 w_g psi_i).
struct Tab2 {
    float2 vphi[kMaxNQ][kMaxNB];
    float2 vdxi[kMaxNQ][kMaxNB];
    float2 veta[kMaxNQ][kMaxNB];
    float2 ephi[3][kMaxNG][kMaxNB];
    float2 nephiw[3][kMaxNG][kMaxNB];
};
static __constant__ Tab2 c_tab_f2[kNumCfg];
// The edge tables in global memory, [3][NG][NB] packed per configuration: a
// CTA copies its configuration's into shared memory with coalesced loads
// (through the constant bank each lane's own address is a replay, which with
// the FP64 reference state per thread cost the FP32 P2 stage 5 %).
static __device__ float2 g_ephi_f2[kNumCfg][3 * kMaxNG * kMaxNB];
static __device__ double g_ephi_d[kNumCfg][3 * kMaxNG * kMaxNB];

// Two-lane FP32 arithmetic (PTX fma/mul/add/sub .f32x2, sm_100a): each lane is
// one IEEE single-precision operation (a fused multiply-add rounds once).
// The pairing fixes the order of operations; a scalar build may contract a
// sum of products differently and so differ in the last bit.
__device__ __forceinline__ float2 f2fma(float2 a, float2 b, float2 c) {
    float2 r;
    asm("{\n .reg .b64 a, b, c, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n mov.b64 c, {%6, %7};\n"
        " fma.rn.f32x2 d, a, b, c;\n mov.b64 {%0, %1}, d;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
__device__ __forceinline__ float2 f2mul(float2 a, float2 b) {
    float2 r;
    asm("{\n .reg .b64 a, b, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n"
        " mul.rn.f32x2 d, a, b;\n mov.b64 {%0, %1}, d;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 f2add(float2 a, float2 b) {
    float2 r;
    asm("{\n .reg .b64 a, b, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n"
        " add.rn.f32x2 d, a, b;\n mov.b64 {%0, %1}, d;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 f2sub(float2 a, float2 b) {
    float2 r;
    asm("{\n .reg .b64 a, b, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n"
        " sub.rn.f32x2 d, a, b;\n mov.b64 {%0, %1}, d;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

__host__ __device__ constexpr int cfg_index(int nq, int ng) {
    return 2 * (nq == 7 ? 0 : (nq == 6 ? 1 : 2)) + (ng == 3 ? 0 : 1);
}

template <typename Real>
__device__ __forceinline__ const Tab<Real>& tab(int c);
template <>
__device__ __forceinline__ const Tab<double>& tab<double>(int c) { return c_tab_d[c]; }
template <>
__device__ __forceinline__ const Tab<float>& tab<float>(int c) { return c_tab_f[c]; }

static void upload_module_tables(int nq, int ng) {
    RuleTables t = make_tables(nq, ng);
    // the stage kernels take psi_0 as one at every volume and edge point and
    // skip the eta-derivative of psi_1 (a function of xi alone): both hold
    // exactly for the native basis
    for (int q = 0; q < nq; ++q)
        if (t.vphi[q][0] != 1.0 || t.veta_w[q][1] != 0.0)
            throw Error{RKDG_ERR_INVALID, "basis tables: psi_0 not one or psi_1 not a function of xi"};
    for (int k = 0; k < 3; ++k)
        for (int g = 0; g < ng; ++g)
            if (t.ephi[k][g][0] != 1.0)
                throw Error{RKDG_ERR_INVALID, "basis tables: psi_0 not one on the edges"};
    Tab<double> d{};
    Tab<float> f{};
    for (int q = 0; q < kMaxNQ; ++q)
        for (int i = 0; i < kMaxNB; ++i) {
            d.vphi[q][i] = t.vphi[q][i];
            d.vdxi[q][i] = t.vdxi_w[q][i];
            d.veta[q][i] = t.veta_w[q][i];
            f.vphi[q][i] = (float)t.vphi[q][i];
            f.vdxi[q][i] = (float)t.vdxi_w[q][i];
            f.veta[q][i] = (float)t.veta_w[q][i];
        }
    for (int k = 0; k < 3; ++k)
        for (int g = 0; g < kMaxNG; ++g)
            for (int i = 0; i < kMaxNB; ++i) {
                d.ephi[k][g][i] = t.ephi[k][g][i];
                f.ephi[k][g][i] = (float)t.ephi[k][g][i];
                d.ephiw[k][g][i] = 2.0 * t.ew[g] * t.ephi[k][g][i];
                f.ephiw[k][g][i] = (float)(2.0 * t.ew[g] * t.ephi[k][g][i]);
            }
    for (int g = 0; g < kMaxNG; ++g) {
        d.ew[g] = t.ew[g];
        f.ew[g] = (float)t.ew[g];
    }
    for (int k = 0; k < 3; ++k)
        for (int j = 0; j < 2; ++j) {
            d.mphi[k][j] = t.mphi[k][j];
            f.mphi[k][j] = (float)t.mphi[k][j];
            d.minv[j][k] = t.minv[j][k];
            f.minv[j][k] = (float)t.minv[j][k];
        }
    Tab2 f2{};
    auto dup = [](double x) { return make_float2((float)x, (float)x); };
    for (int q = 0; q < kMaxNQ; ++q)
        for (int i = 0; i < kMaxNB; ++i) {
            f2.vphi[q][i] = dup(t.vphi[q][i]);
            f2.vdxi[q][i] = dup(t.vdxi_w[q][i]);
            f2.veta[q][i] = dup(t.veta_w[q][i]);
        }
    for (int k = 0; k < 3; ++k)
        for (int g = 0; g < kMaxNG; ++g)
            for (int i = 0; i < kMaxNB; ++i) {
                f2.ephi[k][g][i] = dup(t.ephi[k][g][i]);
                f2.nephiw[k][g][i] = make_float2(-f.ephiw[k][g][i], -f.ephiw[k][g][i]);
            }
    const int c = cfg_index(nq, ng);
    RKDG_CUDA_TRY(cudaMemcpyToSymbol(c_tab_d, &d, sizeof(d), sizeof(d) * c));
    RKDG_CUDA_TRY(cudaMemcpyToSymbol(c_tab_f, &f, sizeof(f), sizeof(f) * c));
    RKDG_CUDA_TRY(cudaMemcpyToSymbol(c_tab_f2, &f2, sizeof(f2), sizeof(f2) * c));
    const int nb = ng == 2 ? 3 : 6;  // P1 and P2 edge rules
    float2 ef[3 * kMaxNG * kMaxNB] = {};
    double ed[3 * kMaxNG * kMaxNB] = {};
    for (int k = 0; k < 3; ++k)
        for (int g = 0; g < ng; ++g)
            for (int i = 0; i < nb; ++i) {
                ef[(k * ng + g) * nb + i] = dup(t.ephi[k][g][i]);
                ed[(k * ng + g) * nb + i] = t.ephi[k][g][i];
            }
    RKDG_CUDA_TRY(cudaMemcpyToSymbol(g_ephi_f2, ef, sizeof(ef), sizeof(ef) * c));
    RKDG_CUDA_TRY(cudaMemcpyToSymbol(g_ephi_d, ed, sizeof(ed), sizeof(ed) * c));
}

// --------------------------------------------------------- state packs --
// States are read with ordinary loads: a kernel launched early
// (launch_dependent) is alive while the one ahead writes them, and the
// read-only path (__ldg, or a const __restrict__ kernel parameter) is for
// memory that nothing writes in a kernel's lifetime.
template <typename Real, int NB>
__device__ __forceinline__ void load_state(const Real* U, int ld, int e, Real u[NB][4]) {
    if constexpr (sizeof(Real) == 8) {
        const double2* p = reinterpret_cast<const double2*>(U);
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            double2 a = p[(size_t)(2 * i) * ld + e];
            double2 b = p[(size_t)(2 * i + 1) * ld + e];
            u[i][0] = a.x;
            u[i][1] = a.y;
            u[i][2] = b.x;
            u[i][3] = b.y;
        }
    } else {
        const float4* p = reinterpret_cast<const float4*>(U);
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            float4 a = p[(size_t)i * ld + e];
            u[i][0] = a.x;
            u[i][1] = a.y;
            u[i][2] = a.z;
            u[i][3] = a.w;
        }
    }
}

template <typename Real, int NB>
__device__ __forceinline__ void load_mean(const Real* U, int ld, int e, Real m[4]) {
    Real u[1][4];
    load_state<Real, 1>(U, ld, e, u);
    m[0] = u[0][0], m[1] = u[0][1], m[2] = u[0][2], m[3] = u[0][3];
}

// FP32 states store every cell mean as its deviation from the solve's
// reference (far-field) state, so that rounding scales with the flow's
// deviation instead of with the state (the SSP-RK combination coefficients
// sum to one, so stage updates apply to deviations unchanged); FP64 states
// store the mean itself.  ref_of returns the offset to add to a stored mean.
template <typename Real>
__device__ __forceinline__ Real ref_of(const double* ref, int v) {
    if constexpr (sizeof(Real) == 4) return (Real)ref[v];
    else return Real(0);
}
template <typename Real>
__host__ __device__ constexpr bool stores_deviation() { return sizeof(Real) == 4; }

struct Ref4 {
    double v[4];
};

// the modes I0..NB-1 of a state
template <typename Real, int I0, int NB>
__device__ __forceinline__ void store_rows(Real* U, int ld, int e, const Real u[NB][4]) {
#pragma unroll
    for (int i = I0; i < NB; ++i) {
        if constexpr (sizeof(Real) == 8) {
            double2* p = reinterpret_cast<double2*>(U);
            p[(size_t)(2 * i) * ld + e] = make_double2(u[i][0], u[i][1]);
            p[(size_t)(2 * i + 1) * ld + e] = make_double2(u[i][2], u[i][3]);
        } else {
            reinterpret_cast<float4*>(U)[(size_t)i * ld + e] = make_float4(u[i][0], u[i][1], u[i][2], u[i][3]);
        }
    }
}
template <typename Real, int NB>
__device__ __forceinline__ void store_state(Real* U, int ld, int e, const Real u[NB][4]) {
    store_rows<Real, 0, NB>(U, ld, e, u);
}

// ------------------------------------------------------------- physics --
// Reciprocal and square root: within one unit in the last place in FP64
// (roots.cuh); in FP32 the PTX approximations (rcp.approx, rsqrt.approx:
// about 1 ulp), which the FP32 precision form's tolerance absorbs, with
// subnormal inputs and results flushed to zero (.ftz: one instruction each,
// no subnormal range handling; the arguments are densities, pressures, edge
// lengths and wave-speed differences, all far above the subnormal range).
__device__ __forceinline__ float rcp_ftz(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ double rcp_(double x) { return rcp_f64(x); }
__device__ __forceinline__ float rcp_(float x) { return rcp_ftz(x); }
__device__ __forceinline__ double sqrt_(double x) { return sqrt_f64(x); }
__device__ __forceinline__ float sqrt_(float x) { return __fmul_rn(x, rsqrt_ftz(x)); }
// Operations that the compiler may not contract with their neighbours: a sum
// of products written with them and fma rounds alike in every kernel.
__device__ __forceinline__ double add_(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
// length and reciprocal length from the squared length: one root for both
__device__ __forceinline__ void lengths_(double x, double& len, double& inv) { roots_f64(x, len, inv); }
__device__ __forceinline__ void lengths_(float x, float& len, float& inv) {
    inv = rsqrt_ftz(x);
    len = __fmul_rn(x, inv);
}

// Ghost state of a boundary edge (the reference's boundaryCondition kernel,
// src/kernelfunctions.cu:184-268, applied inline): 1 far field, 2 outflow
// copy, 3 slip wall mirroring the momentum about the unit normal.
template <typename Real>
__device__ __forceinline__ void ghost(int tag, const Real u[4], const Real far[4], Real nx, Real ny,
                                      Real g[4]) {
    if (tag == RKDG_BC_FARFIELD) {
        g[0] = far[0], g[1] = far[1], g[2] = far[2], g[3] = far[3];
    } else if (tag == RKDG_BC_OUTFLOW) {
        g[0] = u[0], g[1] = u[1], g[2] = u[2], g[3] = u[3];
    } else {
        const Real c = fma(ny, ny, -mul_(nx, nx)), d = mul_(Real(2), mul_(nx, ny));
        g[0] = u[0];
        g[3] = u[3];
        g[1] = fma(u[1], c, -mul_(d, u[2]));
        g[2] = fma(-u[2], c, -mul_(d, u[1]));
    }
}

// LLF coefficient from the average of the two cell means
// (src/kernelfunctions.cu:370-387), scaled by the edge length.
template <typename Real>
__device__ __forceinline__ Real llf_alpha(const Real mL[4], const Real mR[4], Real Nx, Real Ny, Real len, Real gamma,
                                          Real gm1) {
    Real m[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) m[v] = mul_(Real(0.5), add_(mL[v], mR[v]));
    const Real ir = rcp_(m[0]), vx = mul_(m[1], ir), vy = mul_(m[2], ir);
    const Real p = mul_(gm1, fma(Real(-0.5), fma(m[1], vx, mul_(m[2], vy)), m[3]));
    return fma(sqrt_(mul_(mul_(gamma, p), ir)), len, fabs(fma(vx, Nx, mul_(vy, Ny))));
}

// ------------------------------------------- deviation form (FP32 path) --
// FP32 states hold each cell mean as its deviation d = U - U_r from the
// solve's reference state U_r (the far field).  The flux terms of a stage
// are formed from d directly: the reference flux F(U_r) integrates to zero
// over every element (its volume and surface integrals cancel exactly for a
// constant flux), so only F(U_r + d) - F(U_r) enters the residual, and its
// rounding scales with the deviation instead of the state.  Primitive
// deviations: du = (dm - u_r drho) / rho, dp = (gamma - 1)(dE - 1/2 (m_r.du
// + dm.u)), with rho = rho_r + drho and u = u_r + du.
template <typename Real>
struct RefState {
    Real rho, mx, my, E, u, v, p, Ep;  // Ep = E + p
};
// of solve sid, from the table formed on the host (ref_state32)
__device__ __forceinline__ RefState<float> ref_state(const float* tab, int sid) {
    const float4* t = reinterpret_cast<const float4*>(tab) + 2 * sid;
    const float4 a = __ldg(t), b = __ldg(t + 1);
    return RefState<float>{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
}
template <typename Real>
struct DevPrims {
    Real rho, ir, du, dv, u, v, dp;
};
template <typename Real>
__device__ __forceinline__ DevPrims<Real> dev_prims(const Real d[4], const RefState<Real>& r, Real gm1) {
    DevPrims<Real> w;
    w.rho = add_(r.rho, d[0]);
    w.ir = rcp_(w.rho);
    w.du = mul_(fma(-r.u, d[0], d[1]), w.ir);
    w.dv = mul_(fma(-r.v, d[0], d[2]), w.ir);
    w.u = add_(r.u, w.du);
    w.v = add_(r.v, w.dv);
    w.dp = mul_(gm1, fma(Real(-0.5), fma(r.mx, w.du, fma(r.my, w.dv, fma(d[1], w.u, mul_(d[2], w.v)))), d[3]));
    return w;
}
// F(U_r + d).N - F(U_r).N for a (scaled or unit) normal N.
template <typename Real>
__device__ __forceinline__ void dev_flux(const Real d[4], const DevPrims<Real>& w, const RefState<Real>& r,
                                         Real Nx, Real Ny, Real f[4]) {
    const Real q = fma(w.u, Nx, mul_(w.v, Ny)), dq = fma(w.du, Nx, mul_(w.dv, Ny));
    f[0] = fma(d[1], Nx, mul_(d[2], Ny));
    f[1] = fma(r.mx, dq, fma(d[1], q, mul_(w.dp, Nx)));
    f[2] = fma(r.my, dq, fma(d[2], q, mul_(w.dp, Ny)));
    f[3] = fma(r.Ep, dq, mul_(add_(d[3], w.dp), q));
}
// Ghost deviation across a boundary edge (the far field is the reference
// state, so its deviation is zero; walls mirror the momentum).
template <typename Real>
__device__ __forceinline__ void ghost_dev(int tag, const Real d[4], const RefState<Real>& r, Real nx, Real ny,
                                          Real g[4]) {
    if (tag == RKDG_BC_FARFIELD) {
        g[0] = g[1] = g[2] = g[3] = Real(0);
    } else if (tag == RKDG_BC_OUTFLOW) {
        g[0] = d[0], g[1] = d[1], g[2] = d[2], g[3] = d[3];
    } else {
        const Real mn = mul_(Real(-2), fma(add_(r.mx, d[1]), nx, mul_(add_(r.my, d[2]), ny)));
        g[0] = d[0];
        g[1] = fma(mn, nx, d[1]);
        g[2] = fma(mn, ny, d[2]);
        g[3] = d[3];
    }
}
// HLLC (as hllc_flux, stage_fp64.cuh) in deviation form: returns
// F^ - F(U_r).n.  With d_K = rho_K (S_K - q_K), the contact offsets
// D_K = S_M - q_K come from pressure and velocity differences only,
//   D_L = (p_R - p_L + d_R (q_L - q_R)) / (d_L - d_R),
//   D_R = (p_R - p_L + d_L (q_L - q_R)) / (d_L - d_R),
// and the star flux is F*_K = F_K + S_K (U*_K - U_K) with
//   U*_K - U_K = D_K / (S_K - S_M) (U_K + (0, d_K n, d_K S_M + p_K)).
// One selection: the result is F_K + c (U_K + ex) with K = L when S_L >= 0,
// R when S_R <= 0 (both with c = 0) and else the side of S_M (S_M stays
// finite while either side has a positive sound speed).
__device__ __forceinline__ void hllc_dev(const float dL[4], const float dR[4], float nx, float ny, float gamma,
                                         const RefState<float>& r, float f[4]) {
    const float gm1 = add_(gamma, -1.0f);
    const DevPrims<float> L = dev_prims(dL, r, gm1), R = dev_prims(dR, r, gm1);
    const float pL = add_(r.p, L.dp), pR = add_(r.p, R.dp);
    const float qL = fma(L.u, nx, mul_(L.v, ny)), qR = fma(R.u, nx, mul_(R.v, ny));
    const float dqLR = fma(add_(L.du, -R.du), nx, mul_(add_(L.dv, -R.dv), ny));  // q_L - q_R
    const float cL = sqrt_(mul_(mul_(gamma, pL), L.ir)), cR = sqrt_(mul_(mul_(gamma, pR), R.ir));
    const float SL = fmin(add_(qL, -cL), add_(qR, -cR)), SR = fmax(add_(qL, cL), add_(qR, cR));
    float FL[4], FR[4];
    dev_flux(dL, L, r, nx, ny, FL);
    dev_flux(dR, R, r, nx, ny, FR);
    const float kL = mul_(L.rho, add_(SL, -qL)), kR = mul_(R.rho, add_(SR, -qR));
    const float idk = rcp_(add_(kL, -kR));
    const float dpRL = add_(R.dp, -L.dp);
    const float DL = mul_(fma(kR, dqLR, dpRL), idk), DR = mul_(fma(kL, dqLR, dpRL), idk);
    const float SM = add_(qL, DL);
    const bool sl = SL >= 0.0f, sr = SR <= 0.0f;
    const bool left = sl || (!sr && SM >= 0.0f);
    const float S = left ? SL : SR, D = left ? DL : DR, k = left ? kL : kR, p = left ? pL : pR;
    const float c = (sl || sr) ? 0.0f : mul_(mul_(S, D), rcp_(add_(S, -SM)));
    const float UK[4] = {add_(r.rho, left ? dL[0] : dR[0]), add_(r.mx, left ? dL[1] : dR[1]),
                         add_(r.my, left ? dL[2] : dR[2]), add_(r.E, left ? dL[3] : dR[3])};
    const float ex[4] = {0.0f, mul_(k, nx), mul_(k, ny), fma(k, SM, p)};
    const float2 cc = make_float2(c, c);  // by component pairs
    const float2 e01 = f2add(make_float2(UK[0], UK[1]), make_float2(ex[0], ex[1]));
    const float2 e23 = f2add(make_float2(UK[2], UK[3]), make_float2(ex[2], ex[3]));
    const float2 r01 = f2fma(cc, e01, make_float2(left ? FL[0] : FR[0], left ? FL[1] : FR[1]));
    const float2 r23 = f2fma(cc, e23, make_float2(left ? FL[2] : FR[2], left ? FL[3] : FR[3]));
    f[0] = r01.x, f[1] = r01.y, f[2] = r23.x, f[3] = r23.y;
}

// ---------------------------------------------------------- reductions --
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Block-wide max of up to three non-negative doubles, then one atomicMax
// each on their bit patterns (ordered like the values for x >= 0; a NaN
// compares above +inf and so propagates).
__device__ __forceinline__ void block_max3_atomic(double a, double b, double c,
                                                  unsigned long long* da,
                                                  unsigned long long* db,
                                                  unsigned long long* dc) {
    __shared__ double sm[3][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    a = warp_max(a);
    b = warp_max(b);
    c = warp_max(c);
    if (lane == 0) {
        sm[0][wid] = a;
        sm[1][wid] = b;
        sm[2][wid] = c;
    }
    __syncthreads();
    if (wid == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        a = lane < nw ? sm[0][lane] : 0.0;
        b = lane < nw ? sm[1][lane] : 0.0;
        c = lane < nw ? sm[2][lane] : 0.0;
        a = warp_max(a);
        b = warp_max(b);
        c = warp_max(c);
        if (lane == 0) {
            if (da) atomicMax(da, (unsigned long long)__double_as_longlong(a));
            if (db) atomicMax(db, (unsigned long long)__double_as_longlong(b));
            if (dc) atomicMax(dc, (unsigned long long)__double_as_longlong(c));
        }
    }
}

// sqrt that returns 0 at 0 (the FP32 form uses the reciprocal square root).
__device__ __forceinline__ double sqrt0_(double x) { return sqrt(x); }
__device__ __forceinline__ float sqrt0_(float x) { return x > 0.0f ? __fmul_rn(x, rsqrt_ftz(x)) : 0.0f; }

// Edge lengths |N_k| and 1 / area of an element from its FP64 J^-1 rows:
// N_k = 2 area (r0 + r1, -r0, -r1) formed in the working precision from
// the rounded rows, its length there; 1 / area = 2 det J^-1.  The tile kernel forms the same
// values in phase A.
template <typename Real>
__device__ __forceinline__ void elem_lengths(double2 r0, double2 r1, Real len[3], Real& inv_area) {
    const double det = r0.x * r1.y - r0.y * r1.x;
    inv_area = (Real)(2.0 * det);
    const Real area2 = rcp_((Real)det);
    const Real ax = (Real)r0.x, ay = (Real)r0.y, bx = (Real)r1.x, by = (Real)r1.y;
    const Real cx[3] = {ax + bx, -ax, -bx}, cy[3] = {ay + by, -ay, -by};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const Real Nx = cx[k] * area2, Ny = cy[k] * area2;
        len[k] = sqrt_(Nx * Nx + Ny * Ny);
    }
}

// (|u| + c) * perimeter / area of a cell mean (src/kernelfunctions.cu:19-25)
// in the working precision; the max over cells and dt = CFL / max are FP64.
// A non-physical mean (rho <= 0, p <= 0, NaN) sets bad and returns NaN.
template <typename Real>
__device__ __forceinline__ double wave_of(const Real m[4], Real gamma, const Real len[3], Real inv_area,
                                          bool& bad) {
    const Real ri = rcp_(m[0]);
    const Real u = mul_(m[1], ri), v = mul_(m[2], ri);
    const Real p = mul_(add_(gamma, Real(-1)), fma(Real(-0.5), fma(m[1], u, mul_(m[2], v)), m[3]));
    bad = !(m[0] > Real(0)) || !(p > Real(0));
    const Real c = sqrt0_(mul_(mul_(gamma, p), ri));
    const Real w = mul_(add_(sqrt0_(fma(u, u, mul_(v, v))), c), mul_(add_(add_(len[0], len[1]), len[2]), inv_area));
    return bad ? __longlong_as_double(0x7ff8000000000000LL) : (double)w;
}

// ------------------------------------------------------------ the stage --
// MODE_STAGE_COMP: the FP32 stage of RKDG_FP32C (cell means updated in FP64
// from their high and low parts); MODE_LIMITED (added to a stage mode): the
// stage is followed by the TVB limiter and writes its per-tile test
// (tvb_keeps) for it.  Kernels without MODE_LIMITED carry none of that code.
enum { MODE_STAGE = 0, MODE_RESIDUAL = 1, MODE_STAGE_COMP = 2, MODE_LIMITED = 4 };

// The limiter's reciprocals and roots.  FP32: IEEE, since a limited element is
// a discontinuous function of them (only the elements that tvb_keeps does not
// pass pay: 806,400 limited triangles take 20.5 ms per 100 steps either way);
// FP64: those of the fluxes.
__device__ __forceinline__ double lim_rcp(double x) { return rcp_f64(x); }
__device__ __forceinline__ float lim_rcp(float x) { return __frcp_rn(x); }
__device__ __forceinline__ void lim_lengths(double x, double& len, double& inv) { roots_f64(x, len, inv); }
__device__ __forceinline__ void lim_lengths(float x, float& len, float& inv) {
    len = __fsqrt_rn(x);
    inv = __frcp_rn(len);
}

// Exact test that the TVB limiter (limit_element) leaves an element unchanged: every
// row of its left eigenvector matrix has 1-norm at most B (|q|, |q_t| <=
// |vx| + |vy|, |nx| + |ny| <= 1.5; 1.001 covers rounding), so when B times
// the largest |P1 midpoint increment| (tilde) is within the smallest TVB
// threshold, every characteristic increment is kept.  A non-physical mean
// (NaN bound) fails the test.  The stage kernel applies it to each stage's
// output per tile, so the limiter can skip whole tiles.  Its FP32 reciprocal
// and root are the approximate ones: their error, some 2^-22, is far inside
// the 1.001, and the IEEE ones in every element of every stage made the limited
// step 2.5 % slower.
template <typename Real>
__device__ __forceinline__ bool tvb_keeps(const Real mean[4], Real gamma, Real tmax, Real thr_min) {
    const Real ir = rcp_(mean[0]), vx = mean[1] * ir, vy = mean[2] * ir;
    const Real k2 = Real(0.5) * (vx * vx + vy * vy);
    const Real p = (gamma - Real(1)) * (mean[3] - mean[0] * k2);
    Real c, ic;
    lengths_(gamma * p * ir, c, ic);
    const Real b1 = (gamma - Real(1)) * (ic * ic), b2 = b1 * k2;
    const Real av = fabs(vx) + fabs(vy);
    const Real B0 = Real(0.5) * (b2 + av * ic + b1 * av + Real(1.5) * ic + b1);
    const Real B1 = fabs(Real(1) - b2) + b1 * av + b1;
    const Real B2 = av + Real(1.5);
    const Real B = fmax(fmax(B0, B1), B2) * Real(1.001);
    return B * tmax <= thr_min;
}
// The TVB thresholds M (2 |m_k - b0|)^2 of an element's three edges (m_k
// the edge midpoint, b0 the centroid): m_k - b0 = J d_k with the
// reference-element offsets d_0 = (1/6, 1/6), d_1 = (-1/3, 1/6),
// d_2 = (1/6, -1/3) and the columns of J, x_1 - x_0 = (c0x, c0y) and
// x_2 - x_0 = (c1x, c1y); also the unit directions (m_k - b0)/|m_k - b0|.
template <typename Real>
__device__ __forceinline__ void tvb_geometry(Real c0x, Real c0y, Real c1x, Real c1y, Real tvb_m, Real dirx[3],
                                             Real diry[3], Real thr[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const Real dxi = k == 1 ? Real(-1.0 / 3.0) : Real(1.0 / 6.0), deta = k == 2 ? Real(-1.0 / 3.0) : Real(1.0 / 6.0);
        const Real dx = fma(c0x, dxi, mul_(c1x, deta)), dy = fma(c0y, dxi, mul_(c1y, deta));
        const Real r2 = fma(dx, dx, mul_(dy, dy));
        Real rl, irl;
        lim_lengths(r2, rl, irl);
        dirx[k] = mul_(dx, irl);
        diry[k] = mul_(dy, irl);
        thr[k] = mul_(tvb_m, mul_(Real(4), r2));
    }
}
#include "stage_tiled.cuh"
#include "stage_fp64.cuh"

// ------------------------------------------------------------ limiter --
// TVB minmod on characteristic variables for the P1 part (Cockburn & Shu,
// J. Comput. Phys. 141 (1998) 199-224, sec. 2.4/3.3).  In place: only
// modes >= 1 change, and neighbours read only cell means.  Per edge k the
// table holds (alpha, beta) of m_k - b0 = alpha (b_k - b0) + beta (b_j - b0)
// in the working precision (rows k of [3][ld]); the pairing edge j is bit
// 12 + k of the packed connectivity word, and the direction m_k - b0 (edge
// midpoint minus centroid) with its length, the TVB threshold's scale, are
// formed here from J^-1: m_k - b0 = J d_k with the reference-element offsets
// d_0 = (1/6, 1/6), d_1 = (-1/3, 1/6), d_2 = (1/6, -1/3), and J = (J^-1)^-1.
template <typename Real>
using LimitPair = typename std::conditional<sizeof(Real) == 8, double2, float2>::type;
// lo / hi for 0 <= lo <= hi, also of subnormals: a component that is zero in
// the far field decays to them ahead of a front, and the reciprocals of
// subnormals are infinite or NaN.  FP32: the IEEE quotient; FP64: scaled into
// the normal range by a power of two (the IEEE quotient there made the limited
// Mach-3 case of 32,256 triangles 3.7 % slower, 3.13 -> 3.24 ms per 100 steps).
__device__ __forceinline__ float ratio(float lo, float hi) { return lo / hi; }
__device__ __forceinline__ double ratio(double lo, double hi) {
    const double s = hi < 1e-290 ? 0x1p200 : 1.0;
    return mul_(mul_(lo, s), rcp_f64(mul_(hi, s)));
}
// The new P1 modes m1, m2 of an element from its mean, its modes and the
// neighbours' means near (filled in here across boundary edges); false when
// every characteristic increment is kept.  Sums of products are spelled out
// (add_, mul_, fma), so every kernel that limits gives the same bits.
template <typename Real>
__device__ __forceinline__ bool limit_modes(double2 r0, double2 r1, int4 cn, const LimitPair<Real> ab[3],
                                         const Real mean[4], Real near[3][4], Real m1[4], Real m2[4], Real gamma,
                                         Real tvb_m, const double* farp, const Tab<Real>* tbp) {
    const Tab<Real>& tb = *tbp;
    Real tilde[3][4];
    const unsigned pair_bits = ((unsigned)cn.w >> 12) & 7u;
    // the directions and threshold scales in the working precision: FP64
    // for the parity path, FP32 (from the FP64 J^-1 rows) for the FP32 forms
    const Real idet = lim_rcp((Real)fma(r0.x, r1.y, -mul_(r0.y, r1.x)));  // det J
    // columns of J: x_1 - x_0 and x_2 - x_0
    Real dirx[3], diry[3], thrk[3];
    tvb_geometry<Real>(mul_((Real)r1.y, idet), -mul_((Real)r1.x, idet), -mul_((Real)r0.y, idet), mul_((Real)r0.x, idet),
                       tvb_m, dirx, diry, thrk);
    Real tmax = Real(0);
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            tilde[k][v] = fma(tb.mphi[k][0], m1[v], mul_(tb.mphi[k][1], m2[v]));
            tmax = fmax(tmax, fabs(tilde[k][v]));
        }
    // exact early exit (tvb_keeps): uniform and near-uniform regions skip
    // the decompositions
    if (tvb_keeps<Real>(mean, gamma, tmax, fmin(fmin(thrk[0], thrk[1]), thrk[2]))) return false;
    // the mean's velocity, sound speed and enthalpy (the eigenvectors below)
    const Real gm1 = add_(gamma, Real(-1)), ir = lim_rcp(mean[0]), vx = mul_(mean[1], ir), vy = mul_(mean[2], ir);
    const Real k2 = mul_(Real(0.5), fma(vx, vx, mul_(vy, vy)));
    const Real p = mul_(gm1, fma(-mean[0], k2, mean[3])), H = mul_(add_(mean[3], p), ir);
    Real c, ic;
    lim_lengths(mul_(mul_(gamma, p), ir), c, ic);
    const Real b1 = mul_(gm1, mul_(ic, ic)), b2 = mul_(b1, k2);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if ((k == 0 ? cn.x : (k == 1 ? cn.y : cn.z)) >= 0) continue;
        // ghost mean across a boundary edge, mirrored about the unit normal
        // of edge k (N_k / area = 2(r0+r1), -2 r0, -2 r1)
        const int tag = ((unsigned)cn.w >> (6 + 2 * k)) & 3u;
        const double Nx = k == 0 ? add_(r0.x, r1.x) : (k == 1 ? -r0.x : -r1.x);
        const double Ny = k == 0 ? add_(r0.y, r1.y) : (k == 1 ? -r0.y : -r1.y);
        double len, il;
        roots_f64(fma(Nx, Nx, mul_(Ny, Ny)), len, il);
        const Real far[4] = {(Real)farp[0], (Real)farp[1], (Real)farp[2], (Real)farp[3]};
        ghost<Real>(tag, mean, far, (Real)mul_(Nx, il), (Real)mul_(Ny, il), near[k]);
    }
    bool limited = false;
    Real delta[3][4];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const Real al = (Real)ab[k].x, be = (Real)ab[k].y;
        const bool third = (pair_bits >> k) & 1u;  // pairs with edge k + 2, else k + 1
        const Real nx = dirx[k], ny = diry[k], thr = thrk[k];
        Real dbar[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const Real nj = third ? near[(k + 2) % 3][v] : near[(k + 1) % 3][v];
            dbar[v] = mul_(Real(1.5), fma(al, add_(near[k][v], -mean[v]), mul_(be, add_(nj, -mean[v]))));
        }
        // characteristic components in direction n at the mean: with
        // s = b2 a0 - b1 (v.m - aE) and d = (q a0 - m.n) / c they are
        // (s + d) / 2, a0 - s, -q_t a0 - n_y m_x + n_x m_y and (s - d) / 2
        const Real q = fma(vx, nx, mul_(vy, ny)), qt = fma(vy, nx, -mul_(vx, ny));
        Real wl[4], w[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const Real* a = i ? dbar : tilde[k];
            const Real s = fma(b2, a[0], -mul_(b1, fma(vx, a[1], fma(vy, a[2], -a[3]))));
            const Real d = mul_(fma(q, a[0], -fma(a[1], nx, mul_(a[2], ny))), ic);
            w[i][0] = mul_(Real(0.5), add_(s, d)), w[i][1] = add_(a[0], -s);
            w[i][2] = fma(nx, a[2], -fma(ny, a[1], mul_(qt, a[0]))), w[i][3] = mul_(Real(0.5), add_(s, -d));
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const Real wt = w[0][r], wd = w[1][r];
            const Real mm = (wt > Real(0) && wd > Real(0)) ? fmin(wt, wd)
                            : (wt < Real(0) && wd < Real(0)) ? fmax(wt, wd)
                                                             : Real(0);
            wl[r] = fabs(wt) <= thr ? wt : mm;
            limited = limited || wl[r] != wt;
        }
        // back through the right eigenvectors
        const Real sum = add_(add_(wl[0], wl[1]), wl[3]), dif = mul_(add_(wl[3], -wl[0]), c);
        delta[k][0] = sum;
        delta[k][1] = fma(vx, sum, fma(nx, dif, -mul_(ny, wl[2])));
        delta[k][2] = fma(vy, sum, fma(ny, dif, mul_(nx, wl[2])));
        delta[k][3] = fma(H, add_(wl[0], wl[3]), fma(q, dif, fma(k2, wl[1], mul_(qt, wl[2]))));
    }
    if (!limited) return false;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const Real s = add_(add_(delta[0][v], delta[1][v]), delta[2][v]);
        if (s != Real(0)) {
            Real pos = Real(0), neg = Real(0);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                pos = add_(pos, fmax(Real(0), delta[k][v]));
                neg = add_(neg, fmax(Real(0), -delta[k][v]));
            }
            // theta+ = min(1, neg / pos), theta- = min(1, pos / neg): one of them is 1
            const Real lo = fmin(pos, neg), hi = fmax(pos, neg), th = ratio(lo, hi);
            const Real tp = pos > neg ? th : Real(1), tn = neg > pos ? th : Real(1);
#pragma unroll
            for (int k = 0; k < 3; ++k)
                delta[k][v] = fma(tp, fmax(Real(0), delta[k][v]), -mul_(tn, fmax(Real(0), -delta[k][v])));
        }
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        m1[v] = fma(tb.minv[0][0], delta[0][v], fma(tb.minv[0][1], delta[1][v], mul_(tb.minv[0][2], delta[2][v])));
        m2[v] = fma(tb.minv[1][0], delta[0][v], fma(tb.minv[1][1], delta[1][v], mul_(tb.minv[1][2], delta[2][v])));
    }
    return true;
}

}  // namespace rkdg
