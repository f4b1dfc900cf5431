// Resident solve kernel (included by resident_fp*.cu): whole time steps of one
// solve whose tiles all fit on the device at once, in one cooperative launch.
//
// A CTA owns one tile of 128 elements for the launch and keeps its state, U^n
// and geometry in shared memory.  Per RK stage it forms its elements' traces,
// publishes those on edges to other tiles (and the cell means LLF needs) in an
// exchange buffer, forms its volume integral while the neighbours' arrive,
// and then runs the flux tasks, projection and update of the stage kernels on
// the same shared-memory layout with the same functions, so a solve gets the
// same bits as through them (stage_tiled.cuh, stage_fp64.cuh).  With the TVB
// limiter the new cell means are exchanged the same way and each tile limits
// its own elements (limit_modes).
//
// Synchronisation is between neighbouring tiles only, by the data itself: each
// 8-byte word of the exchange buffer holds 4 bytes of a value and the number
// of the stage it belongs to, and a reader loads an edge's words until all
// carry the stage it is in.  That is one trip through L2 where a value, a
// fence, a flag and its poll are four (4,600 of 11,700 cycles of a stage on
// 3,200 P1 triangles).  The buffer is doubled by the parity of the stage: a
// tile can be at most one stage ahead of a neighbour.  A step's time step
// needs the maximum wave speed of all tiles: each adds its own to the step's
// slot and counts itself in, and the sum is awaited only beside the flux tasks
// of the next step's first stage.  Every wait is bounded (kStageWaitNs) and
// reports through the control block, as the staging waits do, and ends the
// solve there.
//
// The edges other tiles read are formed and published first (from the table
// in shared memory, by a runtime edge), the tile's own traces after them.  With
// 256 threads (NT), warps 4-7 do that and collect the neighbours' while warps
// 0-3 form the volume integral and the third edge's traces, and the flux tasks
// (about 217 per tile) take one round.
//
// Why: on meshes of this size a step through the stage kernels is four to
// seven launches, each a launch gap, a chain of dependent loads and one tile's
// latency, on a device that is mostly idle.
struct ResidentArgs {
    void* U;             // [rows][ld] the state, in and out
    const double* jinv;
    const int4* conn;    // with the limiter
    const void* lim;     // with the limiter
    StepCtl* ctl;
    double gamma, tvb_m;
    const double* far;   // [4]
    const float* ref32;  // [8]
    int ld, rk, nsteps, monitor;
    const int* slot;     // [3][ld] the slot each element edge is published in (-1: none)
    int slots;           // one per halo entry, in the order of the tiles' halo lists
    ulonglong2* trace;   // [2][rows][2][slots] the exchanged traces and means (LLF)
    ulonglong2* mean;    // [2][mean rows][2][slots] the exchanged means of a limited stage
    unsigned epoch;      // stages numbered before this launch
    unsigned long long* wave;  // [nsteps] zero before and after: per-step wave-speed maxima, as bits
    unsigned* count;           // [nsteps] likewise: tiles that have added theirs
    unsigned long long* mon;   // [2] likewise: the monitor of a one-step launch
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void add_release(unsigned* p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Waits until *p, a count that only grows, reaches want; false after the limit.
__device__ __forceinline__ bool wait_count(const unsigned* p, unsigned want) {
    if ((int)(ld_acquire(p) - want) >= 0) return true;
    const uint64_t t0 = global_ns();
    for (uint32_t it = 1; it < (1u << 26); ++it) {
        if ((int)(ld_acquire(p) - want) >= 0) return true;
        if ((it & 255u) == 0 && global_ns() - t0 > kStageWaitNs) return false;
    }
    return false;
}

// A 16-byte row v to or from the exchange buffer, as two 16-byte halves of two
// words (4 bytes of the row, stage number) each; halves lie ns slots apart.
__device__ __forceinline__ void publish_row(ulonglong2* p, size_t ns, uint4 v, unsigned ep) {
    const unsigned long long tag = (unsigned long long)ep << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(tag | v.x), "l"(tag | v.y) : "memory");
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p + ns), "l"(tag | v.z), "l"(tag | v.w) : "memory");
}
__device__ __forceinline__ ulonglong2 load_half(const ulonglong2* p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
// N rows of one slot, rows 2 ns apart, once all their words carry stage ep;
// false after the limit.  (Loads started earlier, under the last traces, come
// back without the neighbours' words and cost a second trip: 5.3 -> 6.0 us a
// stage on 9,240 triangles.)
template <int N>
__device__ __forceinline__ bool collect_rows(const ulonglong2* p, size_t ns, unsigned ep, uint4 out[N]) {
    uint64_t t0 = 0;
    for (uint32_t it = 0; it < (1u << 26); ++it) {
        ulonglong2 h[2 * N];
#pragma unroll
        for (int r = 0; r < 2 * N; ++r) h[r] = load_half(p + (size_t)r * ns);
        unsigned miss = 0;
#pragma unroll
        for (int r = 0; r < 2 * N; ++r) miss |= ((unsigned)(h[r].x >> 32) ^ ep) | ((unsigned)(h[r].y >> 32) ^ ep);
        if (miss == 0) {
#pragma unroll
            for (int r = 0; r < N; ++r)
                out[r] = make_uint4((unsigned)h[2 * r].x, (unsigned)h[2 * r].y, (unsigned)h[2 * r + 1].x, (unsigned)h[2 * r + 1].y);
            return true;
        }
        if (it == 0) t0 = global_ns();
        else if ((it & 255u) == 0 && global_ns() - t0 > kStageWaitNs) return false;
    }
    return false;
}
__device__ __forceinline__ uint4 row_bits(float4 v) {
    return make_uint4(__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w));
}
__device__ __forceinline__ uint4 row_bits(double2 v) {
    const unsigned long long x = __double_as_longlong(v.x), y = __double_as_longlong(v.y);
    return make_uint4((unsigned)x, (unsigned)(x >> 32), (unsigned)y, (unsigned)(y >> 32));
}
__device__ __forceinline__ void bits_row(uint4 b, float4& v) {
    v = make_float4(__uint_as_float(b.x), __uint_as_float(b.y), __uint_as_float(b.z), __uint_as_float(b.w));
}
__device__ __forceinline__ void bits_row(uint4 b, double2& v) {
    v = make_double2(__longlong_as_double((long long)(b.x | ((unsigned long long)b.y << 32))),
                     __longlong_as_double((long long)(b.z | ((unsigned long long)b.w << 32))));
}

// Shared memory of a resident CTA: as TiledSmem's work area, then the halo
// traces, the state rows and U^n's rows.
template <typename Real, int NB, int NG, int FLUX, int LIM, int COMP>
struct ResidentSmem {
    static constexpr int BT = kTile, W = (int)sizeof(Real) / 4;  // 16-byte rows of a 4-vector
    static constexpr int SR = NB * W + COMP;                     // state rows
    static constexpr int M = FLUX == RKDG_FLUX_LLF ? 1 : 0;      // LLF exchanges means
    static constexpr int TR = (NG + M) * W;                      // exchanged rows per slot
    static constexpr size_t tr_off = TiledLayout<Real, BT>::code_off + sizeof(int4) * BT + sizeof(uint16_t) * 3 * BT;
    static constexpr size_t mean_off = tr_off + sizeof(Vec4<Real>) * 3 * NG * BT;
    static constexpr size_t htr_off = mean_off + (M || LIM ? sizeof(Vec4<Real>) * BT : 0);
    __host__ __device__ static constexpr size_t u_off(int hm) { return htr_off + (size_t)16 * (NG + M) * W * hm; }
    __host__ __device__ static constexpr size_t bytes(int hm) { return u_off(hm) + (size_t)2 * 16 * SR * BT; }
};

// CTAs per SM the registers are held to: 255 per thread in FP64 (one CTA of 256
// threads or two of 128), 128 in FP32 (two or four).
template <typename Real, int NB, int NQ, int NG, int FLUX, int LIM, int COMP, int NT>
__global__ void __launch_bounds__(NT, (sizeof(Real) == 8 ? 256 : 512) / NT) resident_kernel(const ResidentArgs a, const TileArgs ta) {
    using SM = ResidentSmem<Real, NB, NG, FLUX, LIM, COMP>;
    using Row = typename std::conditional<sizeof(Real) == 8, double2, float4>::type;
    constexpr bool D = sizeof(Real) == 8;
    constexpr int BT = kTile, W = SM::W, SR = SM::SR, NC = TiledLayout<Real, BT>::NC, CFG = cfg_index(NQ, NG);
    constexpr int MEANS = SM::M;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Real* s_nrm = reinterpret_cast<Real*>(smem_raw);
    int4* s_code = reinterpret_cast<int4*>(smem_raw + TiledLayout<Real, BT>::code_off);
    uint16_t* s_task = reinterpret_cast<uint16_t*>(s_code + BT);
    Row* s_tr = reinterpret_cast<Row*>(smem_raw + SM::tr_off);
    Row* s_mean = reinterpret_cast<Row*>(smem_raw + SM::mean_off);  // [W][BT] (LLF, limiter)
    Row* s_htr = reinterpret_cast<Row*>(smem_raw + SM::htr_off);
    const int HM = ta.max_halo;
    Row* s_u = reinterpret_cast<Row*>(smem_raw + SM::u_off(HM));  // [SR][BT]
    Row* s_u0 = s_u + SR * BT;                                    // [SR][BT]
    __shared__ Real s_red[BT / 32][3];
    __shared__ double s_dt, s_far[4];
    using Tab1 = typename std::conditional<D, double, float2>::type;
    __shared__ Tab1 s_ephi[3 * NG * NB];  // edge table for a runtime edge
    if constexpr (D)
        for (int x = threadIdx.x; x < 3 * NG * NB; x += NT) s_ephi[x] = __ldg(&g_ephi_d[CFG][x]);
    else
        for (int x = threadIdx.x; x < 3 * NG * NB; x += NT) s_ephi[x] = __ldg(&g_ephi_f2[CFG][x]);
    __shared__ int s_stop, s_end;  // leave at this step's dt; begin no further step
    // element threads (all, or the first 128) and, with 256 threads, those
    // that form and exchange the traces of element el
    const int tid = threadIdx.x, el = tid % BT;
    const bool elem = NT == BT || tid < BT, trace = NT == BT || tid >= BT;
    const int4 d0 = __ldg(ta.desc + 2 * blockIdx.x), d1 = __ldg(ta.desc + 2 * blockIdx.x + 1);
    const bool active = el < d0.y;
    const int e = d0.x + (active ? el : 0), nh = d1.y, nt = d1.w;
    const size_t ld = a.ld;
    Row* U = static_cast<Row*>(a.U) + e;
    if (elem)
        for (int r = 0; r < SR; ++r) s_u[r * BT + el] = U[r * ld];
    const int4 code = __ldg(ta.code + e);
    if (elem) s_code[el] = code;
    for (int h = tid; h < nt; h += NT) s_task[h] = __ldg(ta.task + d1.z + h);
    const bool reads = trace && el < nh;  // collects halo entry el
    if (tid < 4) s_far[tid] = a.far[tid];
    // geometry and reference state, as the stage kernels form them
    const double2* j2 = reinterpret_cast<const double2*>(a.jinv);
    double det;
    [[maybe_unused]] ElemGeom geo;
    [[maybe_unused]] TilePre<float> pre;
    if constexpr (D) {
        double Nx[3], Ny[3];
        geo = elem_geom(__ldg(j2 + e), __ldg(j2 + ld + e), Nx, Ny);
        det = geo.det;
        if (elem)
#pragma unroll
            for (int k = 0; k < 3; ++k) s_nrm[(NC * k + 0) * BT + el] = Nx[k], s_nrm[(NC * k + 1) * BT + el] = Ny[k];
    } else {
        pre.rs = ref_state(a.ref32, 0);
        tile_geom<BT>(__ldg(j2 + e), __ldg(j2 + ld + e), elem ? s_nrm + el : nullptr, pre);
        det = pre.det;
    }
    const Real gamma = (Real)a.gamma, gm1 = add_(gamma, Real(-1));
    // the slots of this element's edges that other tiles read, and of the
    // halo entry this thread collects (coalesced: halo lists are contiguous)
    int out[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) out[k] = active ? __ldg(a.slot + (size_t)k * ld + e) : -1;
    const int out_mask = (out[0] >= 0 ? 1 : 0) | (out[1] >= 0 ? 2 : 0) | (out[2] >= 0 ? 4 : 0);
    const size_t ns = a.slots, in = d1.x + el;
    // the cell mean of the current state, in full
    auto put_mean = [&]() {
        if constexpr (D) {
            s_mean[el] = s_u[el], s_mean[BT + el] = s_u[BT + el];
        } else {
            const float4 m = s_u[el];
            s_mean[el] = make_float4(add_(m.x, pre.rs.rho), add_(m.y, pre.rs.mx), add_(m.z, pre.rs.my), add_(m.w, pre.rs.E));
        }
    };
    if (LIM && elem) put_mean();
    // the control block, in the last thread (its warp has the fewest flux tasks)
    double t = 0, t_final = 0, dt_fixed = 0, cfl = 0, dt_used = 0;
    unsigned long long wave0 = 0;
    int done = 0, steps = 0, bad_dt = 0;
    constexpr int CT = NT - 1;
    if (tid == CT) {
        const volatile StepCtl* c = a.ctl;
        t = c->t, t_final = c->t_final, dt_fixed = c->dt_fixed, cfl = c->cfl, wave0 = c->wave_bits, done = c->done;
    }
    if (tid == CT) {
        if (t_final > 0 && !(t_final - t > 0)) done = 1;
        s_end = done;
        s_stop = 0;
    }
    unsigned ep = a.epoch;
    bool ok = true;
    __syncthreads();
    for (int step = 0; step < a.nsteps && !s_end; ++step) {
        for (int s = 0; s < a.rk; ++s) {
            ++ep;
            const size_t par = ep & 1u;
            ulonglong2* xt = a.trace + par * SM::TR * 2 * ns;
            // --------------------------------------------------- phase A
            [[maybe_unused]] double2 R2[D ? NB : 1][2];
            [[maybe_unused]] float R1[D ? 1 : NB][4];
            if constexpr (D) {
                double2 u[NB][2];
#pragma unroll
                for (int i = 0; i < NB; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) u[i][h] = s_u[(2 * i + h) * BT + el];
                const Tab<double>& tb = c_tab_d[CFG];
                auto own_traces = [&](int k) {  // into shared memory
#pragma unroll
                    for (int g = 0; g < NG; ++g) {
                        const int x = k * NG + g;
                        double2 v[2];
                        point_value<NB>(tb.ephi[k][g], u, v);
                        s_tr[2 * x * BT + el] = v[0], s_tr[(2 * x + 1) * BT + el] = v[1];
                    }
                };
                if (trace) {
                    for (int m = out_mask; m; m &= m - 1) {  // the edges other tiles read, before the others
                        const int k = __ffs(m) - 1;
                        ulonglong2* xs = xt + (k == 0 ? out[0] : (k == 1 ? out[1] : out[2]));
#pragma unroll
                        for (int g = 0; g < NG; ++g) {
                            double2 v[2];
                            point_value<NB>(s_ephi + (k * NG + g) * NB, u, v);
                            publish_row(xs + 4 * g * ns, ns, row_bits(v[0]), ep);
                            publish_row(xs + (4 * g + 2) * ns, ns, row_bits(v[1]), ep);
                        }
                        if constexpr (MEANS) {
                            publish_row(xs + 4 * NG * ns, ns, row_bits(u[0][0]), ep);
                            publish_row(xs + (4 * NG + 2) * ns, ns, row_bits(u[0][1]), ep);
                        }
                    }
                    if constexpr (MEANS && !LIM) put_mean();
                    own_traces(0);
                    own_traces(1);
                    if (NT == BT) own_traces(2);
                }
                if (elem) {
#pragma unroll
                    for (int i = 0; i < NB; ++i)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            if (s == 0) s_u0[(2 * i + h) * BT + el] = u[i][h];
                            R2[i][h] = make_double2(0.0, 0.0);
                        }
                    volume_term<NB, NQ>(tb, u, geo, gm1, R2);
                    if (NT > BT) own_traces(2);
                }
            } else {
                float u[NB][4];
                load_staged<NB, BT>(reinterpret_cast<const unsigned char*>(s_u), el, u);
                const Tab2& t2 = c_tab_f2[CFG];
                auto own_traces = [&](int k) {  // into shared memory
#pragma unroll
                    for (int g = 0; g < NG; ++g) {
                        float v[4];
                        comb_rows<NB>(t2.ephi[k][g], u, lo2(u[0]), hi2(u[0]), v);
                        s_tr[(k * NG + g) * BT + el] = make_float4(v[0], v[1], v[2], v[3]);
                    }
                };
                if (trace) {
                    if constexpr (MEANS && !LIM) put_mean();
                    for (int m = out_mask; m; m &= m - 1) {  // the edges other tiles read, before the others
                        const int k = __ffs(m) - 1;
                        ulonglong2* xs = xt + (k == 0 ? out[0] : (k == 1 ? out[1] : out[2]));
#pragma unroll
                        for (int g = 0; g < NG; ++g) {
                            float v[4];
                            comb_rows<NB>(s_ephi + (k * NG + g) * NB, u, lo2(u[0]), hi2(u[0]), v);
                            publish_row(xs + 2 * g * ns, ns, row_bits(make_float4(v[0], v[1], v[2], v[3])), ep);
                        }
                        if constexpr (MEANS) publish_row(xs + 2 * NG * ns, ns, row_bits(s_mean[el]), ep);
                    }
                    own_traces(0);
                    own_traces(1);
                    if (NT == BT) own_traces(2);
                }
                if (elem) {
                    if (s == 0)
#pragma unroll
                        for (int r = 0; r < SR; ++r) s_u0[r * BT + el] = s_u[r * BT + el];
#pragma unroll
                    for (int i = 0; i < NB; ++i)
#pragma unroll
                        for (int v = 0; v < 4; ++v) R1[i][v] = 0.0f;
                    volume32<NB, NQ>(t2, u, pre.rs, pre.j00, pre.j01, pre.j10, pre.j11, gm1, R1);
                    if (NT > BT) own_traces(2);
                }
            }
            if (reads) {  // the neighbour's traces on the shared edge, and its mean
                uint4 v[SM::TR];
                ok = collect_rows<SM::TR>(xt + in, ns, ep, v) && ok;  // (a lost mean of the stage before counts too)
#pragma unroll
                for (int r = 0; r < SM::TR; ++r) bits_row(v[r], s_htr[r * HM + el]);
            }
            if (__syncthreads_or(!ok)) goto lost;
            // --------------------------------------------------- phase B
            if constexpr (D)
                flux_tasks64<NG, FLUX, BT, NT>(nt, s_task, s_code, s_nrm, s_tr, s_mean, s_htr, HM, s_far, gamma);
            else
                flux_tasks32<NG, FLUX, BT, NT>(nt, s_task, s_code, s_nrm, reinterpret_cast<Vec4<float>*>(s_tr),
                                           reinterpret_cast<const Vec4<float>*>(s_mean),
                                           reinterpret_cast<Vec4<float>*>(s_htr), HM, pre.rs, gamma);
            if (s == 0 && tid == CT) {  // dt of the step, as step_begin_kernel
                unsigned long long wb = wave0;
                int stop = 0;
                if (step > 0) {
                    if (!wait_count(a.count + step - 1, gridDim.x)) stop = 2;
                    wb = __ldcg(a.wave + step - 1);
                }
                double dt = dt_fixed > 0 ? dt_fixed : cfl / __longlong_as_double((long long)wb);
                bool last = false;
                if (t_final > 0 && dt >= t_final - t) {
                    dt = t_final - t;
                    last = true;
                }
                if (stop == 0 && (!(dt > 0) || !isfinite(dt))) {  // non-physical state: stop, report
                    stop = 1;
                    bad_dt = 1;
                    done = 1;
                    add_release(a.count + step, 1u);  // (it has read the control block and the sums)
                }
                if (stop == 0) {
                    t = last ? t_final : t + dt;
                    dt_used = dt;
                    ++steps;
                    if (t_final > 0 && !(t_final - t > 0) && step + 1 < a.nsteps) {
                        done = 1;
                        s_end = 1;
                    }
                }
                s_dt = dt;
                s_stop = stop;
            }
            __syncthreads();
            if (s == 0 && s_stop) {
                if (s_stop == 2) goto lost;
                goto finished;  // s_u still holds the state the step started from
            }
            // --------------------------------------------------- phase C
            if (elem) {
            const bool last_stage = s == a.rk - 1;
            const double dtd = s_dt, b = s == 0 ? 1.0 : (a.rk == 2 ? 0.5 : (s == 1 ? 0.25 : 2.0 / 3.0));
            Real m[4], q[3][4], u0m[2];  // the new mean and P1 modes; U^n's means of rho and rho E
            if constexpr (D) {
                project64<NB, NG, BT>(c_tab_d[CFG], s_tr, R2);
                const double dt = mul_(dtd, det);
#pragma unroll
                for (int r = 0; r < SR; ++r) {
                    const double2 x = s_u[r * BT + el], y = s_u0[r * BT + el];
                    double2& v = R2[r / 2][r % 2];
                    if (s > 0) v = make_double2(rk_combine(x.x, y.x, v.x, dt, b), rk_combine(x.y, y.y, v.y, dt, b));
                    else v = make_double2(mul_(b, fma(dt, v.x, x.x)), mul_(b, fma(dt, v.y, x.y)));
                    s_u[r * BT + el] = v;
                }
                u0m[0] = s_u0[el].x, u0m[1] = s_u0[BT + el].y;
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    q[i][0] = R2[i][0].x, q[i][1] = R2[i][0].y, q[i][2] = R2[i][1].x, q[i][3] = R2[i][1].y;
#pragma unroll
                for (int v = 0; v < 4; ++v) m[v] = q[0][v];
            } else {
                project32<NB, NG, BT>(c_tab_f2[CFG], reinterpret_cast<const Vec4<float>*>(s_tr), R1);
                const float dt = (float)mul_(dtd, det), cb = (float)b;
#pragma unroll
                for (int i = COMP; i < NB; ++i) {
                    float u[4], u0[4];
                    get4(reinterpret_cast<const Vec4<float>*>(s_u) + i * BT + el, u);
                    get4(reinterpret_cast<const Vec4<float>*>(s_u0) + i * BT + el, u0);
                    if (s > 0) update_row32(u, u0, dt, cb, R1[i]);
                    else update_row32(u, dt, cb, R1[i]);
                    put4(reinterpret_cast<Vec4<float>*>(s_u) + i * BT + el, R1[i]);
                }
                if constexpr (COMP) {
                    float h[4], l[4], h0[4] = {}, l0[4] = {}, low[4];
                    get4(reinterpret_cast<const Vec4<float>*>(s_u) + el, h);
                    get4(reinterpret_cast<const Vec4<float>*>(s_u) + NB * BT + el, l);
                    if (s > 0) {
                        get4(reinterpret_cast<const Vec4<float>*>(s_u0) + el, h0);
                        get4(reinterpret_cast<const Vec4<float>*>(s_u0) + NB * BT + el, l0);
                    }
                    update_mean32c(h, l, h0, l0, mul_(dtd, det), b, R1[0], low);
                    put4(reinterpret_cast<Vec4<float>*>(s_u) + el, R1[0]);
                    put4(reinterpret_cast<Vec4<float>*>(s_u) + NB * BT + el, low);
                }
                u0m[0] = s_u0[el].x, u0m[1] = s_u0[el].w;
                const float far[4] = {pre.rs.rho, pre.rs.mx, pre.rs.my, pre.rs.E};
#pragma unroll
                for (int v = 0; v < 4; ++v) {
#pragma unroll
                    for (int i = 0; i < 3; ++i) q[i][v] = R1[i][v];
                    m[v] = add_(q[0][v], far[v]);
                }
            }
            if (last_stage) {  // CFL wave maximum and monitor, as the stage kernels'
                Real wv = Real(0), m0 = Real(0), m1 = Real(0);
                if (active) {
                    bool bad;
                    Real len[3];
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const Real Nx = s_nrm[(NC * k + 0) * BT + el], Ny = s_nrm[(NC * k + 1) * BT + el];
                        len[k] = sqrt_(fma(Nx, Nx, mul_(Ny, Ny)));
                    }
                    wv = (Real)wave_of<Real>(m, gamma, len, (Real)(2.0 * det), bad);
                    if (bad) atomicOr(&a.ctl->error, 1);
                    if (a.monitor) m0 = fabs(add_(q[0][0], -u0m[0])), m1 = fabs(add_(q[0][3], -u0m[1]));
                }
                wv = warp_max(wv);
                if (a.monitor) m0 = warp_max(m0), m1 = warp_max(m1);
                if ((tid & 31) == 0) s_red[tid >> 5][0] = wv, s_red[tid >> 5][1] = m0, s_red[tid >> 5][2] = m1;
            }
            if constexpr (LIM) {
                // the new means, then each tile limits its own elements
                ulonglong2* xm = a.mean + par * W * 2 * ns;
                put_mean();
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    if (out[k] >= 0)
#pragma unroll
                        for (int r = 0; r < W; ++r) publish_row(xm + 2 * r * ns + out[k], ns, row_bits(s_mean[r * BT + el]), ep);
                bool need = false;
                if (active) {
                    const Tab<Real>& tb = tab<Real>(CFG);
                    Real tmax = Real(0), dirx[3], diry[3], thr[3];
#pragma unroll
                    for (int k = 0; k < 3; ++k)
#pragma unroll
                        for (int v = 0; v < 4; ++v)
                            tmax = fmax(tmax, fabs(fma(tb.mphi[k][0], q[1][v], mul_(tb.mphi[k][1], q[2][v]))));
                    if constexpr (D) tvb_geometry<Real>(geo.j11, -geo.j10, -geo.j01, geo.j00, a.tvb_m, dirx, diry, thr);
                    else tvb_geometry<Real>(pre.j11, -pre.j10, -pre.j01, pre.j00, (Real)a.tvb_m, dirx, diry, thr);
                    need = !tvb_keeps<Real>(m, gamma, tmax, fmin(fmin(thr[0], thr[1]), thr[2]));
                }
                // the tile's means are in shared memory
                asm volatile("bar.sync 1, %0;" ::"n"(BT) : "memory");
                if (need) {
                    const int4 cn = __ldg(a.conn + e);
                    const LimitPair<Real>* lim = static_cast<const LimitPair<Real>*>(a.lim) + e;
                    const LimitPair<Real> ab[3] = {__ldg(lim), __ldg(lim + ld), __ldg(lim + 2 * ld)};
                    Real near[3][4] = {};
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const int ne = k == 0 ? cn.x : (k == 1 ? cn.y : cn.z);
                        if (ne < 0) continue;
                        const int x = ne - d0.x;
                        const bool inside = x >= 0 && x < d0.y;
                        Row v[W];
                        if (inside) {
#pragma unroll
                            for (int r = 0; r < W; ++r) v[r] = s_mean[r * BT + x];
                        } else {
                            uint4 w[W];
                            const int c = k == 0 ? code.x : (k == 1 ? code.y : code.z);
                            ok = collect_rows<W>(xm + d1.x + (c >> 4), ns, ep, w) && ok;
#pragma unroll
                            for (int r = 0; r < W; ++r) bits_row(w[r], v[r]);
                        }
                        if constexpr (D) near[k][0] = v[0].x, near[k][1] = v[0].y, near[k][2] = v[1].x, near[k][3] = v[1].y;
                        else near[k][0] = v[0].x, near[k][1] = v[0].y, near[k][2] = v[0].z, near[k][3] = v[0].w;
                    }
                    Real m1[4] = {q[1][0], q[1][1], q[1][2], q[1][3]}, m2[4] = {q[2][0], q[2][1], q[2][2], q[2][3]};
                    if (ok && limit_modes<Real>(__ldg(j2 + e), __ldg(j2 + ld + e), cn, ab, m, near, m1, m2, gamma,
                                                (Real)a.tvb_m, s_far, &tab<Real>(CFG))) {
                        Real* su = reinterpret_cast<Real*>(s_u);
                        constexpr int V = 4 / W;  // values per row
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            su[((1 * W + v / V) * BT + el) * V + v % V] = m1[v];
                            su[((2 * W + v / V) * BT + el) * V + v % V] = m2[v];
#pragma unroll
                            for (int i = 3; i < NB; ++i) su[((i * W + v / V) * BT + el) * V + v % V] = Real(0);
                        }
                    }
                }
                // s_mean's readers are behind the next stage's barriers before it is written again
            }
            }  // element threads
            if (NT > BT || s == a.rk - 1) __syncthreads();  // the new state, and the last stage's maxima
            if (s == a.rk - 1 && tid == 0) {
                Real w = s_red[0][0], x = s_red[0][1], y = s_red[0][2];
#pragma unroll
                for (int k = 1; k < BT / 32; ++k)
                    w = fmax(w, s_red[k][0]), x = fmax(x, s_red[k][1]), y = fmax(y, s_red[k][2]);
                atomicMax(a.wave + step, (unsigned long long)__double_as_longlong((double)w));
                if (a.monitor) {
                    atomicMax(a.mon + 0, (unsigned long long)__double_as_longlong((double)x));
                    atomicMax(a.mon + 1, (unsigned long long)__double_as_longlong((double)y));
                }
                add_release(a.count + step, 1u);
            }
        }
    }
finished:
    if (active && elem)
        for (int r = 0; r < SR; ++r) U[r * ld] = s_u[r * BT + el];
    if (blockIdx.x == 0 && tid == CT) {
        StepCtl* c = a.ctl;
        // the block changes only after every tile has read it
        if (steps + bad_dt > 0 && !wait_count(a.count + steps + bad_dt - 1, gridDim.x)) ok = false;
        if (steps > 0) {
            c->wave_bits = __ldcg(a.wave + steps - 1);
            c->mon_bits[0] = a.monitor ? __ldcg(a.mon + 0) : 0ull;
            c->mon_bits[1] = a.monitor ? __ldcg(a.mon + 1) : 0ull;
            c->dt = dt_used;
            c->t = t;
            c->step += steps;
        }
        if (done) c->done = 1;
        if (bad_dt) atomicOr(&c->error, 1);
    }
    if (__syncthreads_or(!ok)) goto lost;
    // every tile has counted itself into the last step, so none will read the
    // sums again: zero for the next launch (after an error the host clears
    // them as well)
    if (blockIdx.x == 0) {
        for (int i = tid; i < a.nsteps; i += NT) a.wave[i] = 0ull, a.count[i] = 0u;
        if (tid < 2) a.mon[tid] = 0ull;
    }
    return;
lost:  // a wait ran out: report and leave (the other tiles' waits run out too);
       // launches queued behind find the solve done and leave at once
    if (tid == 0) {
        atomicOr(&a.ctl->error, 2);
        atomicExch(&a.ctl->done, 1);
    }
}

// ------------------------------------------------------------- host --
namespace {

template <typename Real, int NB, int NQ, int NG, int FLUX, int LIM, int COMP>
struct ResidentForm {
    using SM = ResidentSmem<Real, NB, NG, FLUX, LIM, COMP>;
    template <int NT>
    static constexpr auto kernel() { return &resident_kernel<Real, NB, NQ, NG, FLUX, LIM, COMP, NT>; }
    // tiles the device holds at once with NT threads each
    template <int NT>
    static int fit(int max_halo) {
        if (max_halo > kTile || SM::bytes(max_halo) > smem_limit()) return 0;
        static PerDevice<std::map<int, int>> answers;  // by halo size
        return answers.use(current_device(), [&](std::map<int, int>& known) {
            if (known.empty()) {  // the whole opt-in size, whatever halo lists come later
                RKDG_CUDA_TRY(cudaFuncSetAttribute(kernel<NT>(), cudaFuncAttributePreferredSharedMemoryCarveout,
                                                   (int)cudaSharedmemCarveoutMaxShared));
                RKDG_CUDA_TRY(cudaFuncSetAttribute(kernel<NT>(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)smem_limit()));
            }
            const auto it = known.find(max_halo);
            if (it != known.end()) return it->second;
            int n = 0;
            RKDG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel<NT>(), NT, SM::bytes(max_halo)));
            return known[max_halo] = n * sm_count();
        });
    }
    // no fewer, without a look at the kernels: by shared memory
    static int bound(int max_halo) {
        if (max_halo > kTile || SM::bytes(max_halo) > smem_limit()) return 0;
        return (int)(smem_per_sm() / SM::bytes(max_halo)) * sm_count();
    }
    static int tiles(int max_halo, bool wide) { return wide ? fit<256>(max_halo) : fit<128>(max_halo); }
    // with 256 threads per tile (wide) or 128
    // (false: refused as a whole, as under a limit on the SMs a process may use)
    static bool launch(ResidentArgs a, TileArgs t, bool wide, cudaStream_t s) {
        void* args[] = {&a, &t};
        tiles(t.max_halo, wide);  // (sets the kernel's attributes)
        const void* k = wide ? (const void*)kernel<256>() : (const void*)kernel<128>();
        const cudaError_t e = cudaLaunchCooperativeKernel(k, dim3(t.ntiles), dim3(wide ? 256 : 128), args,
                                                          SM::bytes(t.max_halo), s);
        if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
            cudaGetLastError();
            return false;
        }
        RKDG_CUDA_TRY(e);
        return true;
    }
};

// calls f with the form of a method
template <typename Real, int LIM, typename F>
auto with_resident(int order, int nq, int flux, bool comp, F&& f) {
    auto flx = [&](auto nb, auto q, auto g, auto fl) {
        constexpr int NB = decltype(nb)::value, NQ = decltype(q)::value, NG = decltype(g)::value;
        constexpr int FL = decltype(fl)::value;
        if constexpr (sizeof(Real) == 4)
            if (comp) return f(ResidentForm<Real, NB, NQ, NG, FL, LIM, 1>{});
        return f(ResidentForm<Real, NB, NQ, NG, FL, LIM, 0>{});
    };
    auto rule = [&](auto nb, auto q, auto g) {
        if (flux == RKDG_FLUX_HLLC) return flx(nb, q, g, std::integral_constant<int, RKDG_FLUX_HLLC>{});
        return flx(nb, q, g, std::integral_constant<int, RKDG_FLUX_LLF>{});
    };
    using I = std::integral_constant<int, 3>;
    using S = std::integral_constant<int, 6>;
    if (order == 1) return rule(I{}, I{}, std::integral_constant<int, 2>{});
    if (nq == 7) return rule(S{}, std::integral_constant<int, 7>{}, I{});
    return rule(S{}, S{}, I{});
}

template <typename Real, int LIM>
bool launch_resident(const StageArgs& a, const TileArgs& t, const void* lim, ResidentWork& w, int order, int nq, int flux,
                     int rk, int steps, bool monitor, bool wide, cudaStream_t stream) {
    ResidentArgs r{};
    r.U = a.Unew;
    r.jinv = a.jinv, r.conn = a.conn, r.lim = lim, r.ctl = a.ctl;
    r.gamma = a.gamma, r.tvb_m = a.tvb_m, r.far = a.far_sid, r.ref32 = a.ref32;
    r.ld = a.ld, r.rk = rk, r.nsteps = steps, r.monitor = monitor ? 1 : 0;
    r.slot = w.slot, r.slots = w.slots;
    r.trace = static_cast<ulonglong2*>(w.trace), r.mean = static_cast<ulonglong2*>(w.mean), r.epoch = w.epoch;
    r.wave = reinterpret_cast<unsigned long long*>(w.sums);
    r.mon = r.wave + kResidentSteps;
    r.count = reinterpret_cast<unsigned*>(r.mon + 2);
    w.epoch += (unsigned)(steps * rk);
    if (!w.clean) RKDG_CUDA_TRY(cudaMemsetAsync(w.sums, 0, kResidentSums, stream));
    w.clean = true;  // each launch leaves them so, unless it reports an error
    return with_resident<Real, LIM>(order, nq, flux, a.lo_row >= 0,
                                    [&](auto form) { return form.launch(r, t, wide, stream); });
}

// the unit of a translation unit
template <typename Real, int LIM>
constexpr ResidentUnit resident_unit_of() {
    return ResidentUnit{
        [](int order, int nq, int flux, bool comp, int max_halo, bool wide) {
            return with_resident<Real, LIM>(order, nq, flux, comp, [&](auto form) { return form.tiles(max_halo, wide); });
        },
        [](int order, int flux, bool comp, int max_halo) {
            return with_resident<Real, LIM>(order, 6, flux, comp, [&](auto form) { return form.bound(max_halo); });
        },
        upload_module_tables, launch_resident<Real, LIM>};
}

}  // namespace
