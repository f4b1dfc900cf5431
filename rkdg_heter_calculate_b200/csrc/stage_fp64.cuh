// FP64 form of the tile-staged stage kernel (included by device.cuh after
// stage_tiled.cuh, whose staging pipeline, tile tables and shared-memory
// areas it shares): one thread per element.
//
// An element's modes and residual are held as the rows they are stored in,
// pairs (rho, rho u) and (rho v, rho E), and traces and fluxes lie in shared
// memory as two arrays of 16-byte halves, each contiguous over the elements:
// 16-byte accesses at a 32-byte stride would meet in the banks.
//
// What bounds it: latency at 12 warps per SM (168 registers): the FP64 pipe
// is busy 40 % and issue 34 % of the time.  980,000 P2 HLLC triangles:
// 0.723 ms per step with IEEE divides and roots, two-sided fluxes and
// 32-byte traces, 0.585 as it is (7-point LLF 0.683 -> 0.549).
//
// Every sum of products is spelled as fused multiply-adds and roundings that
// the compiler may not contract (add_, mul_), so each kernel built from these
// functions gives a tile the same bits.
//
// Measured and dropped: two lanes per element, each with one pair of
// components (24 warps per SM at 80 registers instead of 12 at 168): 45 %
// more instructions -- every basis-table value then feeds two multiply-adds
// instead of four, and the point states are exchanged -- made the
// 980,000-triangle P2 step 14 % slower.

// sum_i tab[i] u_i (psi_0 is one at every point; upload_tables checks it)
template <int NB>
__device__ __forceinline__ void point_value(const double* tab, const double2 u[NB][2], double2 s[2]) {
    s[0] = u[0][0], s[1] = u[0][1];
#pragma unroll
    for (int i = 1; i < NB; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            s[h].x = fma(tab[i], u[i][h].x, s[h].x);
            s[h].y = fma(tab[i], u[i][h].y, s[h].y);
        }
}

// Edge normals N_k = 2 area (r0 + r1, -r0, -r1) from the rows r of J^-1.
struct ElemGeom {
    double j00, j01, j10, j11;  // rows of 2 area J^-1 = (-N_1; -N_2)
    double det;                 // det J^-1 = 1 / (2 area)
};
__device__ __forceinline__ ElemGeom elem_geom(double2 r0, double2 r1, double Nx[3], double Ny[3]) {
    ElemGeom g;
    g.det = fma(r0.x, r1.y, -mul_(r0.y, r1.x));
    const double s = rcp_f64(g.det);
    Nx[0] = mul_(add_(r0.x, r1.x), s), Ny[0] = mul_(add_(r0.y, r1.y), s);
    g.j00 = mul_(r0.x, s), g.j01 = mul_(r0.y, s), g.j10 = mul_(r1.x, s), g.j11 = mul_(r1.y, s);
    Nx[1] = -g.j00, Ny[1] = -g.j01, Nx[2] = -g.j10, Ny[2] = -g.j11;
    return g;
}

// Volume term of rows 1.. (psi_1 is a function of xi alone).
template <int NB, int NQ>
__device__ __forceinline__ void volume_term(const Tab<double>& tb, const double2 u[NB][2], const ElemGeom& g,
                                            double gm1, double2 R[NB][2]) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        double2 w[2];
        point_value<NB>(tb.vphi[q], u, w);
        const double ri = rcp_f64(w[0].x), vx = mul_(w[0].y, ri), vy = mul_(w[1].x, ri);
        const double p = mul_(gm1, fma(-0.5, fma(w[0].y, vx, mul_(w[1].x, vy)), w[1].y));
        const double ep = add_(w[1].y, p);
        // through row r of 2 area J^-1, by its contravariant speed q_r
        const double q0 = fma(g.j00, vx, mul_(g.j01, vy)), q1 = fma(g.j10, vx, mul_(g.j11, vy));
        const double2 fx[2] = {make_double2(mul_(w[0].x, q0), fma(w[0].y, q0, mul_(g.j00, p))),
                               make_double2(fma(w[1].x, q0, mul_(g.j01, p)), mul_(ep, q0))};
        const double2 fy[2] = {make_double2(mul_(w[0].x, q1), fma(w[0].y, q1, mul_(g.j10, p))),
                               make_double2(fma(w[1].x, q1, mul_(g.j11, p)), mul_(ep, q1))};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int i = 1; i < NB; ++i) {
                R[i][h].x = fma(fx[h].x, tb.vdxi[q][i], R[i][h].x);
                R[i][h].y = fma(fx[h].y, tb.vdxi[q][i], R[i][h].y);
            }
#pragma unroll
            for (int i = 2; i < NB; ++i) {
                R[i][h].x = fma(fy[h].x, tb.veta[q][i], R[i][h].x);
                R[i][h].y = fma(fy[h].y, tb.veta[q][i], R[i][h].y);
            }
        }
    }
}

// The numerical flux through the scaled normal N = len n at one point: LLF
// with the edge's coefficient alpha (scaled by len), or HLLC (hllc_flux).
__device__ __forceinline__ void llf_flux(const double uL[4], const double uR[4], double Nx, double Ny, double alpha,
                                         double gm1, double f[4]) {
    double s[4];
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        const double* u = side ? uR : uL;
        const double ri = rcp_f64(u[0]);
        const double vx = mul_(u[1], ri), vy = mul_(u[2], ri);
        const double p = mul_(gm1, fma(-0.5, fma(u[1], vx, mul_(u[2], vy)), u[3]));
        const double q = fma(vx, Nx, mul_(vy, Ny));
        if (side == 0) {
            s[0] = mul_(u[0], q), s[1] = fma(u[1], q, mul_(p, Nx)), s[2] = fma(u[2], q, mul_(p, Ny)),
            s[3] = mul_(add_(u[3], p), q);
        } else {
            s[0] = fma(u[0], q, s[0]), s[1] = fma(u[1], q, fma(p, Nx, s[1])), s[2] = fma(u[2], q, fma(p, Ny, s[2])),
            s[3] = fma(add_(u[3], p), q, s[3]);
        }
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) f[v] = mul_(0.5, fma(-alpha, add_(uR[v], -uL[v]), s[v]));
}
// HLLC through the unit normal (Toro, Riemann Solvers and Numerical Methods
// for Fluid Dynamics, 3rd ed., sec. 10.4): Davis wave-speed bounds (eq.
// 10.48), contact speed S_M (eq. 10.37).  Branch-free with one selection:
// the result is F_K + c (U_K + ex) with K = L when S_L >= 0, R when S_R <= 0
// (both with c = 0) and else the side of S_M, where
//   c (U_K + ex) = S_K (U*_K - U_K),  ex = (0, d_K n, d_K S_M + p_K),
//   d_K = rho_K (S_K - q_K),  c = S_K (S_M - q_K) / (S_K - S_M),
// so a warp whose points fall in different wave regions runs one path and
// only the selected side's physical flux is formed.  (One reciprocal of the
// product of the densities costs as much as two, 0.587 ms per step against
// 0.585 on 980,000 triangles, and is out of range where each density alone is
// not.)
__device__ __forceinline__ void hllc_flux(const double uL[4], const double uR[4], double nx, double ny, double gamma,
                                          double f[4]) {
    const double gm1 = add_(gamma, -1.0);
    const double iL = rcp_f64(uL[0]), iR = rcp_f64(uR[0]);
    const double vxL = mul_(uL[1], iL), vyL = mul_(uL[2], iL), vxR = mul_(uR[1], iR), vyR = mul_(uR[2], iR);
    const double pL = mul_(gm1, fma(-0.5, fma(uL[1], vxL, mul_(uL[2], vyL)), uL[3]));
    const double pR = mul_(gm1, fma(-0.5, fma(uR[1], vxR, mul_(uR[2], vyR)), uR[3]));
    const double qL = fma(vxL, nx, mul_(vyL, ny)), qR = fma(vxR, nx, mul_(vyR, ny));
    const double cL = sqrt_f64(mul_(mul_(gamma, pL), iL)), cR = sqrt_f64(mul_(mul_(gamma, pR), iR));
    const double SL = fmin(add_(qL, -cL), add_(qR, -cR)), SR = fmax(add_(qL, cL), add_(qR, cR));
    const double dL = mul_(uL[0], add_(SL, -qL)), dR = mul_(uR[0], add_(SR, -qR));
    const bool sl = SL >= 0.0, sr = SR <= 0.0, star = !sl && !sr;
    // (without a star region S_M is not part of the result, and may be NaN:
    // two states of zero pressure and the same speed have dL = dR = 0)
    const double SM = star ? mul_(fma(dL, qL, fma(-dR, qR, add_(pR, -pL))), rcp_f64(add_(dL, -dR))) : 0.0;
    const bool left = sl || (star && SM >= 0.0);
    const double d = left ? dL : dR, p = left ? pL : pR, q = left ? qL : qR, S = left ? SL : SR;
    const double u0 = left ? uL[0] : uR[0], u1 = left ? uL[1] : uR[1], u2 = left ? uL[2] : uR[2],
                 ep = add_(left ? uL[3] : uR[3], p);
    const double c = star ? mul_(mul_(S, add_(SM, -q)), rcp_f64(add_(S, -SM))) : 0.0;
    f[0] = fma(c, u0, mul_(u0, q));
    f[1] = fma(c, fma(d, nx, u1), fma(u1, q, mul_(p, nx)));
    f[2] = fma(c, fma(d, ny, u2), fma(u2, q, mul_(p, ny)));
    f[3] = fma(c, fma(d, SM, ep), mul_(ep, q));
}
// Runge-Kutta combination U^n + b ((U - U^n) + dt R) of one value; without
// U^n, b (U + dt R).
__device__ __forceinline__ double rk_combine(double u, double u0, double r, double dt, double b) {
    return fma(b, fma(dt, r, add_(u, -u0)), u0);
}

// The flux tasks of a tile: own traces s_tr [3 NG][2][BT], halo traces s_htr
// [NG][2][HM] followed by the halo means (LLF), the tile's means s_mean
// [2][BT] (LLF); NT threads.
template <int NG, int FLUX, int BT, int NT>
__device__ __forceinline__ void flux_tasks64(int nt, const uint16_t* s_task, const int4* s_code, const double* s_nrm,
                                             double2* s_tr, const double2* s_mean, double2* s_htr, int HM,
                                             const double* s_far, double gamma) {
    constexpr int NC = TiledLayout<double, BT>::NC;
    const double gm1 = add_(gamma, -1.0);
    for (int j = threadIdx.x; j < nt; j += NT) {
        const int tkj = s_task[j];
        const int le = tkj >> 2, k = tkj & 3;
        const int c = reinterpret_cast<const int*>(s_code + le)[k];
        const int kind = c & 3, se = (c >> 2) & 3, idx = c >> 4;
        // physical normal N (|N| = edge length) and unit normal of edge k
        const double Nx = s_nrm[(NC * k + 0) * BT + le], Ny = s_nrm[(NC * k + 1) * BT + le];
        double len, il;
        roots_f64(fma(Nx, Nx, mul_(Ny, Ny)), len, il);
        const double nx = mul_(Nx, il), ny = mul_(Ny, il);
        // the other side's values: in-tile slots, or the halo rows
        const bool bnd = kind == EDGE_BOUNDARY;
        double2* nb = kind == EDGE_HALO ? s_htr + idx : s_tr + 2 * se * NG * BT + idx;
        const int nld = kind == EDGE_HALO ? HM : BT;
        double alpha = 0.0;
        if constexpr (FLUX == RKDG_FLUX_LLF) {
            double2 x = s_mean[le], y = s_mean[BT + le];
            const double mL[4] = {x.x, x.y, y.x, y.y};
            double mR[4];
            if (kind == EDGE_BOUNDARY) {
                ghost<double>(se, mL, s_far, nx, ny, mR);
            } else {
                const double2* mb = kind == EDGE_HALO ? nb + 2 * NG * HM : s_mean + idx;
                x = mb[0], y = mb[nld];
                mR[0] = x.x, mR[1] = x.y, mR[2] = y.x, mR[3] = y.y;
            }
            alpha = llf_alpha<double>(mL, mR, Nx, Ny, len, gamma, gm1);
        }
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            double2* slot = s_tr + 2 * (k * NG + g) * BT + le;
            double2 x = slot[0], y = slot[BT];
            const double uL[4] = {x.x, x.y, y.x, y.y};
            double uR[4], f[4];
            // the neighbour's point NG-1-g on its edge se pairs with ours
            // (src/kernelfunctions.cu:545-549)
            // of a boundary edge the other slot is the own one
            double2* np = bnd ? slot : nb + 2 * (NG - 1 - g) * nld;
            x = np[0], y = np[nld];
            uR[0] = x.x, uR[1] = x.y, uR[2] = y.x, uR[3] = y.y;
            if (bnd) ghost<double>(se, uL, s_far, nx, ny, uR);
            if constexpr (FLUX == RKDG_FLUX_LLF) {
                llf_flux(uL, uR, Nx, Ny, alpha, gm1, f);
            } else {
                hllc_flux(uL, uR, nx, ny, gamma, f);
#pragma unroll
                for (int v = 0; v < 4; ++v) f[v] = mul_(f[v], len);
            }
            // each slot of an edge is read by this task alone: the other
            // side's slot takes the negated flux (an in-tile neighbour's; a
            // halo's is read no more; a boundary's is overwritten at once),
            // the computing side's the flux
            np[0] = make_double2(-f[0], -f[1]);
            np[nld] = make_double2(-f[2], -f[3]);
            slot[0] = make_double2(f[0], f[1]);
            slot[BT] = make_double2(f[2], f[3]);
        }
    }
}

// Surface term: the outward fluxes in an element's own slots.
template <int NB, int NG, int BT>
__device__ __forceinline__ void project64(const Tab<double>& tb, const double2* s_tr, double2 R[NB][2]) {
#pragma unroll
    for (int s = 0; s < 3 * NG; ++s) {
        const double* w = tb.ephiw[s / NG][s % NG];
        const double2 f[2] = {s_tr[2 * s * BT + threadIdx.x], s_tr[(2 * s + 1) * BT + threadIdx.x]};
#pragma unroll
        for (int i = 0; i < NB; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                R[i][h].x = fma(-f[h].x, w[i], R[i][h].x);
                R[i][h].y = fma(-f[h].y, w[i], R[i][h].y);
            }
    }
}

// One tile, as tile_stage (stage_tiled.cuh).  Own trace slot s = k NG + g,
// half h of element x lies at s_tr[(2 s + h) BT + x]; a halo neighbour's
// traces (and mean) overwrite its own staged rows, slot s half h in row
// 2 s + h.
template <int NB, int NQ, int NG, int FLUX, int MODE, int BT>
__device__ __forceinline__ bool tile_stage_fp64(const StageArgs& a, const TileArgs& ta, const int4 d0, const int4 d1,
                                           unsigned char* smem_raw, unsigned char* stg, const int nxt,
                                           const int ntiles, uint64_t* bar, const ElemGeom& geo,
                                           const double* s_far, const double* s_ephi, double (*s_red)[3],
                                                const double* s_dt) {
    constexpr int NT = BT;
    constexpr int CFG = cfg_index(NQ, NG);
    const Tab<double>& tb = c_tab_d[CFG];
    const int HM = ta.max_halo;
    constexpr int NC = TiledLayout<double, BT>::NC;
    double* s_nrm = reinterpret_cast<double*>(smem_raw);                                      // [3][NC][BT] Nx, Ny
    int4* s_code = reinterpret_cast<int4*>(smem_raw + TiledLayout<double, BT>::code_off);     // [BT]
    uint16_t* s_task = reinterpret_cast<uint16_t*>(s_code + BT);                              // [3 BT] flux tasks
    double2* s_tr = reinterpret_cast<double2*>(s_task + 3 * BT);                              // [3 NG][2][BT]
    constexpr int MEANS = FLUX == RKDG_FLUX_LLF ? 1 : 0;                                      // LLF needs cell means
    double2* s_mean = s_tr + 2 * 3 * NG * BT;                                                 // [2][BT] (LLF)
    double2* s_stg = reinterpret_cast<double2*>(stg);
    const int tid = threadIdx.x;
    const int sid = d0.z;
    StepCtl* ctl = a.ctl + sid;
    const int e0 = d0.x;
    const bool active = tid < d0.y;
    const int sx = active ? tid : 0, ee = e0 + sx;
    const double gamma = a.gamma, gm1 = add_(gamma, -1.0);
    const int nh = d1.y, nt = d1.w;

    // ------------------------------------------------------------ phase A
    double2 R[NB][2], u[NB][2];
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) u[i][h] = s_stg[(2 * i + h) * BT + sx], R[i][h] = make_double2(0.0, 0.0);
    __syncthreads();  // staged rows consumed: the area takes the halo states
    {
        const char* Ub = static_cast<const char*>(a.U);
        for (int h = tid; h < nh; h += NT) {
            const int n = __ldg(&ta.halo[d1.x + h].x);
#pragma unroll
            for (int r = 0; r < 2 * NB; ++r)
                cp_async16(stg + ((size_t)r * HM + h) * 16, Ub + ((size_t)r * a.ld + n) * 16);
        }
    }
    if constexpr (MEANS) s_mean[tid] = u[0][0], s_mean[BT + tid] = u[0][1];
    volume_term<NB, NQ>(tb, u, geo, gm1, R);
#pragma unroll
    for (int s = 0; s < 3 * NG; ++s) {
        double2 t[2];
        point_value<NB>(tb.ephi[s / NG][s % NG], u, t);
        s_tr[2 * s * BT + tid] = t[0], s_tr[(2 * s + 1) * BT + tid] = t[1];
    }
    cp_async_wait_all();
    __syncthreads();  // s_ephi visible below; own traces complete; halo states landed
    for (int h = tid; h < nh; h += NT) {
        const int he = __ldg(&ta.halo[d1.x + h].y);
#pragma unroll
        for (int i = 0; i < NB; ++i) u[i][0] = s_stg[2 * i * HM + h], u[i][1] = s_stg[(2 * i + 1) * HM + h];
        if constexpr (MEANS) s_stg[2 * NG * HM + h] = u[0][0], s_stg[(2 * NG + 1) * HM + h] = u[0][1];
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            double2 t[2];
            point_value<NB>(s_ephi + (he * NG + g) * NB, u, t);
            s_stg[2 * g * HM + h] = t[0], s_stg[(2 * g + 1) * HM + h] = t[1];
        }
    }
    __syncthreads();  // halo traces complete
    int4 nd0 = make_int4(0, 0, 0, 0);
    if (tid == 0 && nxt < ntiles) {  // the CTA's next tile (only this thread reads its descriptor)
        nd0 = __ldg(ta.desc + 2 * nxt);
        stage_prefetch<double, true>(a, ta, nd0, __ldg(ta.desc + 2 * nxt + 1));
    }

    // ------------------------------------------------------------ phase B
    flux_tasks64<NG, FLUX, BT, BT>(nt, s_task, s_code, s_nrm, s_tr, s_mean, s_stg, HM, s_far, gamma);
    __syncthreads();  // fluxes complete, halo traces read: the staging area takes the next tile's rows
    if (tid == 0 && nxt < ntiles) {
        fence_proxy_async();
        stage_copy<double, BT>(a, nd0, stg, bar);
    }

    // ------------------------------------------------------------ phase C
    // every own slot now holds the outward flux of its edge point
    project64<NB, NG, BT>(tb, s_tr, R);

    double2* Uout = static_cast<double2*>(a.Unew) + ee;
    if (MODE == MODE_RESIDUAL) {
        if (active)
#pragma unroll
            for (int r = 0; r < 2 * NB; ++r)
                Uout[(size_t)r * a.ld] = make_double2(R[r / 2][r % 2].x * geo.det, R[r / 2][r % 2].y * geo.det);
        return false;
    }
    const double dt = mul_(*s_dt, geo.det), cb = a.b;
    const double2* Uin = static_cast<const double2*>(a.U) + ee;
    double u0m[2] = {0.0, 0.0};  // U^n's means of rho and rho E
    if (a.U0 != nullptr) {
        const double2* U0 = static_cast<const double2*>(a.U0) + ee;
#pragma unroll
        for (int r = 0; r < 2 * NB; ++r) {
            const double2 x = Uin[(size_t)r * a.ld];  // stored values (L2 hits)
            const double2 y = U0[(size_t)r * a.ld];
            if (r == 0) u0m[0] = y.x;
            if (r == 1) u0m[1] = y.y;
            double2& v = R[r / 2][r % 2];
            v = make_double2(rk_combine(x.x, y.x, v.x, dt, cb), rk_combine(x.y, y.y, v.y, dt, cb));
        }
    } else {
#pragma unroll
        for (int r = 0; r < 2 * NB; ++r) {
            const double2 x = Uin[(size_t)r * a.ld];
            double2& v = R[r / 2][r % 2];
            v = make_double2(mul_(cb, fma(dt, v.x, x.x)), mul_(cb, fma(dt, v.y, x.y)));
        }
    }
    if (active)
#pragma unroll
        for (int r = 0; r < 2 * NB; ++r) Uout[(size_t)r * a.ld] = R[r / 2][r % 2];
    if (!a.last_stage && !(MODE & MODE_LIMITED)) return false;

    const double m[4] = {R[0][0].x, R[0][0].y, R[0][1].x, R[0][1].y};
    if (a.last_stage) {
        // CFL wave maximum (and the residual monitor when asked) of the new
        // state: a max over each warp; after the tile's closing barrier one
        // atomic per tile on the solve's control block
        double wv = 0.0, m0 = 0.0, m1 = 0.0;
        if (active) {
            bool bad;
            double len[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double Nx = s_nrm[(NC * k + 0) * BT + tid], Ny = s_nrm[(NC * k + 1) * BT + tid];
                len[k] = sqrt_f64(fma(Nx, Nx, mul_(Ny, Ny)));
            }
            wv = wave_of<double>(m, gamma, len, 2.0 * geo.det, bad);
            if (bad) atomicOr(&ctl->error, 1);
            if (a.monitor) {
                m0 = fabs(add_(m[0], -u0m[0]));
                m1 = fabs(add_(m[3], -u0m[1]));
            }
        }
        wv = warp_max(wv);
        if (a.monitor) {
            m0 = warp_max(m0);
            m1 = warp_max(m1);
        }
        if ((tid & 31) == 0) {
            s_red[tid >> 5][0] = wv;
            s_red[tid >> 5][1] = m0;
            s_red[tid >> 5][2] = m1;
        }
    }
    bool need = false;
    if constexpr (MODE & MODE_LIMITED) {
        // the limiter's exact test on the new state (see tile_stage)
        double tmax = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                tmax = fmax(tmax, fabs(fma(tb.mphi[k][0], R[1][h].x, tb.mphi[k][1] * R[2][h].x)));
                tmax = fmax(tmax, fabs(fma(tb.mphi[k][0], R[1][h].y, tb.mphi[k][1] * R[2][h].y)));
            }
        if (active && (a.limiter_on == nullptr || a.limiter_on[sid])) {
            double dirx[3], diry[3], thr[3];
            tvb_geometry<double>(geo.j11, -geo.j10, -geo.j01, geo.j00, a.tvb_m, dirx, diry, thr);
            need = !tvb_keeps<double>(m, gamma, tmax, fmin(fmin(thr[0], thr[1]), thr[2]));
        }
    }
    return need;
}

// Resident CTAs per SM: 12 warps (P2: 168 registers, 70 KB of shared memory
// per 128-element CTA) and 16 (P1: 128 registers).  LAT: 8 and 12 warps
// without spills, for launches whose tiles all fit on the device at once,
// where a tile's latency rather than the throughput of many sets the time.
template <int ORD, int BT, int LAT>
struct Fp64Occupancy {
    static constexpr int warps = LAT ? (ORD == 1 ? 12 : 8) : (ORD == 1 ? 16 : 12);
    static constexpr int value = warps * 32 / BT > 0 ? warps * 32 / BT : 1;
};

// As tiled_stage_kernel (stage_tiled.cuh).
template <int NQ2, int FLUX, int MODE, int ORD, int BT, int LAT>
__global__ void __launch_bounds__(BT, Fp64Occupancy<ORD, BT, LAT>::value)
    stage_fp64_kernel(const StageArgs a, const TileArgs ta) {
    using SM = TiledSmem<double, ORD, FLUX, BT>;
    constexpr int NT = BT, NC = TiledLayout<double, BT>::NC;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ double s_red[NT / 32][3];  // per-warp maxima of a last stage
    __shared__ double s_dt;               // the tile's solve's dt (read before the staging wait)
    __shared__ double s_far[4];           // its far-field state
    unsigned char* stg = smem_raw + SM::stage_offset(ta.max_halo);
    const int ntiles = ta.ntiles_dev ? *ta.ntiles_dev : ta.ntiles;
    int tile = blockIdx.x;
    if (tile >= ntiles) {  // a launch without a tile also completes only after the ones ahead of it
        grid_dependency_wait();
        return;
    }
    const int tid = threadIdx.x;
    int4 d0 = __ldg(ta.desc + 2 * tile), d1 = __ldg(ta.desc + 2 * tile + 1);
    grid_dependents_launch();
    if (tid == 0) mbar_init(&s_bar, 1);
    __syncthreads();
    if (tid == 0) {
        grid_dependency_wait();
        stage_copy<double, BT>(a, d0, stg, &s_bar);
        stage_prefetch<double, false>(a, ta, d0, d1);
    }
    __shared__ double s_ephi[ORD == 3 ? 2 : 1][3 * kMaxNG * kMaxNB];
    load_edge_table<ORD, NQ2, BT>(g_ephi_d, s_ephi);  // (read after later barriers)
    const double2* jinv2 = reinterpret_cast<const double2*>(a.jinv);
    double* s_nrm = reinterpret_cast<double*>(smem_raw);
    int4* s_code = reinterpret_cast<int4*>(smem_raw + TiledLayout<double, BT>::code_off);
    uint16_t* s_task = reinterpret_cast<uint16_t*>(s_code + BT);
    uint32_t parity = 0;
    for (;; tile += gridDim.x, d0 = __ldg(ta.desc + 2 * tile), d1 = __ldg(ta.desc + 2 * tile + 1)) {
        const int nxt = tile + gridDim.x;
        // the work that needs only the geometry and the lists, while the state rows arrive
        const int ex = d0.x + (tid < d0.y ? tid : 0);
        const double2 r0 = __ldg(jinv2 + ex), r1 = __ldg(jinv2 + a.ld + ex);
        grid_dependency_wait();
        const int done = MODE != MODE_RESIDUAL ? a.ctl[d0.z].done : 0;
        if (MODE != MODE_RESIDUAL && tid == 0) s_dt = a.ctl[d0.z].dt;
        if (tid < 4)
            s_far[tid] = a.far_sid ? a.far_sid[4 * d0.z + tid]
                                   : (tid < 2 ? (tid == 0 ? a.far[0] : a.far[1]) : (tid == 2 ? a.far[2] : a.far[3]));
        for (int h = tid; h < d1.w; h += NT) s_task[h] = __ldg(ta.task + d1.z + h);
        s_code[tid] = __ldg(ta.code + ex);
        double Nx[3], Ny[3];
        const ElemGeom geo = elem_geom(r0, r1, Nx, Ny);
#pragma unroll
        for (int k = 0; k < 3; ++k) s_nrm[(NC * k + 0) * BT + tid] = Nx[k], s_nrm[(NC * k + 1) * BT + tid] = Ny[k];
        const bool ok = mbar_wait(&s_bar, parity);
        if (__syncthreads_or(!ok)) {  // also: every thread has seen this phase complete
            if (tid == 0) atomicOr(&a.ctl[d0.z].error, 2);
            return;
        }
        parity ^= 1u;
        if (done) {  // finished solve: pass the tile on
            if (nxt >= ntiles) return;
            if (tid == 0) stage_copy<double, BT>(a, __ldg(ta.desc + 2 * nxt), stg, &s_bar);
            continue;
        }
        bool need;
        if (ORD == 2 || (ORD == 3 && d0.w == 2))
            need = tile_stage_fp64<6, NQ2, 3, FLUX, MODE, BT>(a, ta, d0, d1, smem_raw, stg, nxt, ntiles, &s_bar, geo, s_far,
                                                             s_ephi[0], s_red, &s_dt);
        else
            need = tile_stage_fp64<3, 3, 2, FLUX, MODE, BT>(a, ta, d0, d1, smem_raw, stg, nxt, ntiles, &s_bar, geo, s_far,
                                                           s_ephi[ORD == 3 ? 1 : 0], s_red, &s_dt);
        // shared memory is reused by the next tile (with the limiter the
        // barrier also ORs its test over the tile)
        if constexpr (MODE & MODE_LIMITED) {
            const int any = __syncthreads_or(need);
            if (tid == 0 && any && atomicExch(a.tile_flags + tile, 1) == 0) {
                const int slot = atomicAdd(a.tile_list, 1);
                if (slot < a.tile_cap) a.tile_list[kListHead + slot] = tile;
            }
        } else {
            __syncthreads();
        }
        if (MODE != MODE_RESIDUAL && a.last_stage && tid == 0) tile_maxima_atomic<double, NT>(a, a.ctl + d0.z, s_red);
        if (nxt >= ntiles) return;
    }
}
