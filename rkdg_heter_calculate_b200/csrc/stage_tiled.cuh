// Tile-staged fused stage kernel (included by device.cuh): the staging
// pipeline and the FP32 kernel (FP64: stage_fp64.cuh).
//
// A tile is up to BT consecutive (locality-ordered) elements of one
// solve; its descriptor names the element range, the solve, the polynomial
// order, and its halo and flux-task ranges.  One CTA processes a tile:
//   phase A  each thread: its element's state, volume integral (registers),
//            traces at the 3*NG edge points and cell mean -> shared memory;
//            the CTA together: traces of the out-of-tile (halo) neighbours
//            on the shared edges -> shared memory.
//   phase B  the tile's flux tasks (each interior in-tile edge once, from
//            its lower-index side; every halo and boundary edge from the
//            in-tile side), spread evenly over the threads; the physical
//            flux (normal scaled by the edge length) overwrites the
//            computing side's trace slot, its negation the other side's.
//   phase C  each thread adds the fluxes in its own nine (P1: six) slots to
//            the residual and applies the stage update.
// The kernel loops over tiles (tile = blockIdx.x + k * gridDim.x), so one
// launch serves a single solve (one CTA per tile) or a persistent pass over
// the packed tiles of many solves of uneven size and mixed order, each with
// its own dt, CFL measure and monitor.  A tile's arithmetic depends only on
// its own solve's data: results are deterministic and identical whether a
// solve runs alone or in a batch.
//
// What bounds it: the instructions of 24 (P1: 32) warps per SM and, at the
// start of a CTA, the chain descriptor -> geometry, codes and lists -> state
// (a quarter of a tile's 20,000 cycles on 500,000 triangles).  So every load
// that needs no other is issued first, nobody waits for the thread that
// issues the copies, the reference state comes from a table, and the edge
// tables are loaded once per CTA: 980,000 P2 triangles 0.288 -> 0.263 ms per
// step in FP32 and 0.310 -> 0.289 in FP32C, P1 with LLF 0.171 -> 0.158; with
// overlapping launches and branch-free flux stores 0.254, 0.276 and 0.148.
//
// Staging pipeline: a tile's own state rows are contiguous 16-byte rows in
// HBM (pack p of element e at (p ld + e) 16), so one thread moves them into
// shared memory with bulk asynchronous copies (cp.async.bulk, completion
// counted in bytes on an mbarrier).  The copies for the CTA's next tile are
// issued once the current tile's halo traces are formed, and run under its
// flux and update work; the next tile's J^-1, edge-code and U^n rows and its
// halo and task lists are prefetched into L2 at the same time.

// ------------------------------------------------------------- staging --
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void bulk_prefetch_l2(const void* src, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
// 16-byte asynchronous gather into shared memory (completion per thread).
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// Orders this thread's earlier generic-proxy shared-memory accesses before
// later asynchronous-proxy (bulk copy) accesses.
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Programmatic dependent launch (kernels launched by launch_dependent): a
// kernel lets the next one of its stream start while its own last CTAs run,
// and the next does what needs only tables (descriptors, geometry, lists) and
// then waits here until everything before it is complete and visible.
__device__ __forceinline__ void grid_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Waits for the barrier phase of the given parity; gives up after limit_ns
// nanoseconds (two seconds for the stage kernel's staging waits) or 2^26
// polls, returning false.
constexpr uint64_t kStageWaitNs = 2000000000ull;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns = kStageWaitNs) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (uint32_t it = 1; it < (1u << 26); ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 255u) == 0 && global_ns() - t0 > limit_ns) return false;
    }
    return false;
}

// Shared memory of one CTA: the work area (edge normals, edge codes, flux
// tasks, own traces and means, as 4-vectors), sized for the largest tile
// layout the kernel dispatches (P1 tiles of a mixed pack use a prefix),
// then the staging area.  The staging area first receives the tile's own
// state rows by bulk copy (SROWS rows of 16 bytes per element); once phase A
// has read them, the halo neighbours' states by 16-byte gathers ([SROWS][hm]
// rows).  Each halo thread then overwrites its own neighbour's first rows
// with that neighbour's traces (and mean), which phase B reads, and
// the next tile's rows are copied in after phase B.  This keeps an FP32 CTA
// within the shared memory of six per SM (P2) and an FP64 one within that of
// three (P2) or four (P1).  J^-1 and the edge codes are read per thread (L2
// hits, prefetched with the rows) while the rows arrive.
template <typename Real>
struct alignas(16) Vec4 {
    Real x, y, z, w;
};
template <typename Real>
__device__ __forceinline__ void put4(Vec4<Real>* p, const Real a[4]) {
    Vec4<Real> t;
    t.x = a[0], t.y = a[1], t.z = a[2], t.w = a[3];
    *p = t;
}
template <typename Real>
__device__ __forceinline__ void get4(const Vec4<Real>* p, Real a[4]) {
    const Vec4<Real> t = *p;
    a[0] = t.x, a[1] = t.y, a[2] = t.z, a[3] = t.w;
}
// Per-element linear algebra on 4-vectors (the conservative components), in
// lane pairs (components 0-1 and 2-3) with the f32x2 helpers and the paired
// tables.  (Pairing the
// two sides of the HLLC flux the same way executed fewer instructions but
// more register moves and ran slower.)
__device__ __forceinline__ float2 lo2(const float a[4]) { return make_float2(a[0], a[1]); }
__device__ __forceinline__ float2 hi2(const float a[4]) { return make_float2(a[2], a[3]); }
__device__ __forceinline__ void set4(float a[4], float2 l, float2 h) { a[0] = l.x, a[1] = l.y, a[2] = h.x, a[3] = h.y; }
// out = c + sum_{i >= 1} tab[i] u_i
template <int NB>
__device__ __forceinline__ void comb_rows(const float2* tab, const float u[NB][4], float2 cl, float2 ch,
                                          float out[4]) {
#pragma unroll
    for (int i = 1; i < NB; ++i) {
        cl = f2fma(tab[i], lo2(u[i]), cl);
        ch = f2fma(tab[i], hi2(u[i]), ch);
    }
    set4(out, cl, ch);
}
// R_i += f tab[i] for i >= I0
template <int I0, int NB>
__device__ __forceinline__ void acc_rows(float R[NB][4], const float f[4], const float2* tab) {
    const float2 fl = lo2(f), fh = hi2(f);
#pragma unroll
    for (int i = I0; i < NB; ++i) set4(R[i], f2fma(fl, tab[i], lo2(R[i])), f2fma(fh, tab[i], hi2(R[i])));
}

template <typename Real, int BT>
struct TiledLayout {
    // edge normals per element: (Nx, Ny) per edge, the length formed where
    // used (as it was formed when stored: the same bits); this keeps an FP64
    // P2 CTA with the LLF means within the shared memory of three per SM
    static constexpr int NC = 2;
    static constexpr size_t code_off = (sizeof(Real) * 3 * NC * BT + 15) / 16 * 16;
};

// Cell means (own and halo) are kept only where the LLF coefficient needs
// them.
template <typename Real, int ORD, int FLUX, int BT>
struct TiledSmem {
    static constexpr int NG = ORD == 1 ? 2 : 3;
    static constexpr int SROWS = (ORD == 1 ? 3 : 6) * (int)(sizeof(Real) / 4);
    static constexpr int MEANS = FLUX == RKDG_FLUX_LLF ? 1 : 0;
    __host__ __device__ static constexpr size_t work(int) {
        return TiledLayout<Real, BT>::code_off + sizeof(int4) * BT + sizeof(uint16_t) * 3 * BT +
               sizeof(Vec4<Real>) * ((size_t)3 * NG * BT + MEANS * BT);
    }
    __host__ __device__ static constexpr size_t stage_offset(int hm) { return (work(hm) + 127) / 128 * 128; }
    __host__ __device__ static constexpr size_t stage_rows(int hm) {
        return (size_t)SROWS * (BT > hm ? BT : hm);
    }
    __host__ __device__ static constexpr size_t bytes(int hm) { return stage_offset(hm) + stage_rows(hm) * 16; }
};

// Resident CTAs per SM the register allocation is held to: 24 warps per SM
// for kernels with P2 tiles (80 registers; 128-element tiles at most 37 KB of
// shared memory per CTA) and 32 for P1-only kernels (64 registers; their
// tiles need about 27 KB, and the extra warps hide more of the tile
// pipeline's latency: 11 % faster on the limited Mach-3 step), whatever the
// tile size.
template <int ORD, int BT>
struct TiledOccupancy {
    static constexpr int warps = ORD == 1 ? 32 : 24;
    static constexpr int value = warps * 32 / BT > 0 ? warps * 32 / BT : 1;
};

// Issues the bulk copies of tile d's state rows into the staging area (one
// thread; completion counted on bar).
template <typename Real, int BT>
__device__ __forceinline__ void stage_copy(const StageArgs& a, const int4 d, unsigned char* stg, uint64_t* bar) {
    const int rows = (d.w == 2 ? 6 : 3) * (int)(sizeof(Real) / 4);
    const uint32_t rb = (uint32_t)d.y * 16u;
    mbar_expect_tx(bar, rb * (uint32_t)rows);
    const char* U = static_cast<const char*>(a.U);
    for (int r = 0; r < rows; ++r)
        bulk_g2s(stg + (size_t)r * BT * 16, U + ((size_t)r * a.ld + d.x) * 16, rb, bar);
}
// L2 prefetches of tile d's J^-1 and edge-code rows, U^n rows, the rows of
// the means' low parts (RKDG_FP32C) and halo and task lists, and with STATE
// its state rows (one thread; the tables are padded so that the 16-byte
// rounding stays inside them).
template <typename Real, bool STATE>
__device__ __forceinline__ void stage_prefetch(const StageArgs& a, const TileArgs& ta, const int4 d,
                                               const int4 dd) {
    const int rows = (d.w == 2 ? 6 : 3) * (int)(sizeof(Real) / 4);
    const uint32_t rb = (uint32_t)d.y * 16u;
    if constexpr (STATE) {
        const char* U = static_cast<const char*>(a.U);
        for (int r = 0; r < rows; ++r) bulk_prefetch_l2(U + ((size_t)r * a.ld + d.x) * 16, rb);
    }
    const char* J = reinterpret_cast<const char*>(a.jinv);
    bulk_prefetch_l2(J + (size_t)d.x * 16, rb);
    bulk_prefetch_l2(J + ((size_t)a.ld + d.x) * 16, rb);
    bulk_prefetch_l2(ta.code + d.x, rb);
    if (a.U0 != nullptr) {
        const char* U0 = static_cast<const char*>(a.U0);
        for (int r = 0; r < rows; ++r) bulk_prefetch_l2(U0 + ((size_t)r * a.ld + d.x) * 16, rb);
    }
    if (a.lo_row >= 0) {  // RKDG_FP32C: the low parts of the means, read by the update
        const size_t lo = ((size_t)a.lo_row * a.ld + d.x) * 16;
        bulk_prefetch_l2(static_cast<const char*>(a.U) + lo, rb);
        if (a.U0 != nullptr) bulk_prefetch_l2(static_cast<const char*>(a.U0) + lo, rb);
    }
    if (dd.y > 0) {
        const uintptr_t b = reinterpret_cast<uintptr_t>(ta.halo + dd.x) & ~uintptr_t(15);
        const uintptr_t e = (reinterpret_cast<uintptr_t>(ta.halo + dd.x + dd.y) + 15) & ~uintptr_t(15);
        bulk_prefetch_l2(reinterpret_cast<const void*>(b), (uint32_t)(e - b));
    }
    if (dd.w > 0) {
        const uintptr_t b = reinterpret_cast<uintptr_t>(ta.task + dd.z) & ~uintptr_t(15);
        const uintptr_t e = (reinterpret_cast<uintptr_t>(ta.task + dd.z + dd.w) + 15) & ~uintptr_t(15);
        bulk_prefetch_l2(reinterpret_cast<const void*>(b), (uint32_t)(e - b));
    }
}

// Element x's state from the staging rows.
template <int NB, int BT>
__device__ __forceinline__ void load_staged(const unsigned char* stg, int x, float u[NB][4]) {
    const float4* p = reinterpret_cast<const float4*>(stg);
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const float4 a = p[i * BT + x];
        u[i][0] = a.x;
        u[i][1] = a.y;
        u[i][2] = a.z;
        u[i][3] = a.w;
    }
}

// One CTA per tile (no next tile of its own): the last warp prefetches the
// tile a full device of CTAs further on, which a CTA yet to start will run,
// so that its loads find L2 instead of HBM (980,000 triangles, FP32C P2:
// 0.296 -> 0.289 ms per step; the FP64 kernel loses 2 % by it, its tiles
// being longer than HBM's latency matters).
template <typename Real, int BT>
__device__ __forceinline__ void prefetch_ahead(const StageArgs& a, const TileArgs& ta, int nxt, int ntiles) {
    if (threadIdx.x != BT - 32 || nxt < ntiles) return;
    const int t = (int)blockIdx.x + ta.ahead;
    if (ta.ahead > 0 && t < ntiles) stage_prefetch<Real, true>(a, ta, __ldg(ta.desc + 2 * t), __ldg(ta.desc + 2 * t + 1));
}

// The part of a tile's work that needs only its descriptors, J^-1 rows and
// edge codes: edge normals and codes into shared memory, the solve's
// reference state, the halo and task list entries.  Formed while the tile's
// state rows are still in flight.
template <typename Real>
struct TilePre {
    RefState<Real> rs;
    Real inv_area, j00, j01, j10, j11;  // 1 / area; rows of 2 area J^-1
    double det;                         // det J^-1 = 1 / (2 area)
    int2 hh[3];
};
// The geometry of TilePre, and the edge normals into s_nrm, the element's
// entry of [3][NC][BT] (or null).
template <int BT>
__device__ __forceinline__ void tile_geom(const double2 r0, const double2 r1, float* s_nrm, TilePre<float>& t) {
    using Real = float;
    constexpr int NC = TiledLayout<Real, BT>::NC;
    // edge normals N_k (length = edge length; N_k / area = 2(r0 + r1), -2 r0,
    // -2 r1) from the FP64 J^-1 rows, kept in the working precision.  The
    // residual is accumulated scaled by 2 area (= 1 / det J^-1): the volume
    // term through 2 area J^-1 = (-N_1; -N_2), the surface term through the
    // table 2 w_g psi_i, and the factor det J^-1 applied once in the update.
    t.det = fma(r0.x, r1.y, -mul_(r0.y, r1.x));
    t.inv_area = (Real)(2.0 * t.det);
    // from the rounded J^-1 rows (a few ulp, without an FP64 reciprocal)
    const Real area2 = rcp_((Real)t.det);
    const Real ax = (Real)r0.x, ay = (Real)r0.y, bx = (Real)r1.x, by = (Real)r1.y;
    const Real cx[3] = {add_(ax, bx), -ax, -bx}, cy[3] = {add_(ay, by), -ay, -by};
    Real Nx[3], Ny[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        Nx[k] = mul_(cx[k], area2), Ny[k] = mul_(cy[k], area2);
        if (s_nrm) s_nrm[(NC * k + 0) * BT] = Nx[k], s_nrm[(NC * k + 1) * BT] = Ny[k];
    }
    t.j00 = -Nx[1], t.j01 = -Ny[1], t.j10 = -Nx[2], t.j11 = -Ny[2];
}
template <typename Real, int BT>
__device__ __forceinline__ TilePre<Real> tile_pre(const StageArgs& a, const TileArgs& ta, const int4 d0,
                                                  const int4 d1, const double2 r0, const double2 r1,
                                                  const int4 code, unsigned char* smem_raw) {
    const int tid = threadIdx.x;
    TilePre<Real> t;
    t.rs = ref_state(a.ref32, d0.z);
    // the halo and task lists (L2 hits: prefetched with the tile's rows)
    const int h0 = d1.x, nh = d1.y, t0 = d1.z, nt = d1.w;
    int4* s_code = reinterpret_cast<int4*>(smem_raw + TiledLayout<Real, BT>::code_off);  // [BT]
    uint16_t* s_task = reinterpret_cast<uint16_t*>(s_code + BT);                         // [3 BT]
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const int h = tid + r * BT;
        t.hh[r] = h < nh ? __ldg(ta.halo + h0 + h) : make_int2(0, 0);
        // the flux tasks straight into the work area (not the staging area)
        if (h < nt) s_task[h] = __ldg(ta.task + t0 + h);
    }
    s_code[tid] = code;
    tile_geom<BT>(r0, r1, reinterpret_cast<Real*>(smem_raw) + tid, t);
    return t;
}

// The neighbour-side edge tables (runtime edge index) of the orders a kernel
// runs, from global memory into shared memory: [0] the P2 (or only) order's,
// [1] P1's in a mixed kernel.
template <int ORD, int NQ2, int BT, typename T>
__device__ __forceinline__ void load_edge_table(const T (*g)[3 * kMaxNG * kMaxNB], T (*s)[3 * kMaxNG * kMaxNB]) {
    constexpr int P1 = cfg_index(3, 2);
    constexpr int n = ORD == 1 ? 3 * 2 * 3 : 3 * 3 * 6;
    for (int x = threadIdx.x; x < n; x += BT) s[0][x] = __ldg(&g[ORD == 1 ? P1 : cfg_index(NQ2, 3)][x]);
    if constexpr (ORD == 3)
        for (int x = threadIdx.x; x < 3 * 2 * 3; x += BT) s[1][x] = __ldg(&g[P1][x]);
}

// Volume term of rows 1.. from an element's modes u: flux deviations through
// the rows of 2 area J^-1.  The quadrature loop is unrolled by two only (a
// smaller body keeps the instruction cache warm across the CTAs on an SM;
// full unrolling is 2 % slower, none 1 %).  psi_0 is one at every point and
// psi_1 (a function of xi alone) has no eta-derivative term.
template <int NB, int NQ>
__device__ __forceinline__ void volume32(const Tab2& t2, const float u[NB][4], const RefState<float>& rs, float j00,
                                         float j01, float j10, float j11, float gm1, float R[NB][4]) {
#pragma unroll 2
    for (int q = 0; q < NQ; ++q) {
        float w[4], fx[4], fy[4];
        comb_rows<NB>(t2.vphi[q], u, lo2(u[0]), hi2(u[0]), w);
        const DevPrims<float> pw = dev_prims(w, rs, gm1);
        dev_flux(w, pw, rs, j00, j01, fx);
        dev_flux(w, pw, rs, j10, j11, fy);
        acc_rows<1, NB>(R, fx, t2.vdxi[q]);
        acc_rows<2, NB>(R, fy, t2.veta[q]);
    }
}

// The flux tasks of a tile: own traces s_tr [3][NG][BT], halo traces s_htr
// [NG][HM] followed by the halo means (LLF), the tile's means s_mean (LLF).
template <int NG, int FLUX, int BT, int NT>
__device__ __forceinline__ void flux_tasks32(int nt, const uint16_t* s_task, const int4* s_code, const float* s_nrm,
                                             Vec4<float>* s_tr, const Vec4<float>* s_mean, Vec4<float>* s_htr, int HM,
                                             const RefState<float>& rs, float gamma) {
    using Real = float;
    using V4 = Vec4<float>;
    constexpr int NC = TiledLayout<Real, BT>::NC;
    constexpr bool MEANS = FLUX == RKDG_FLUX_LLF;
    const Real gm1 = add_(gamma, -1.0f);
    const Real far[4] = {rs.rho, rs.mx, rs.my, rs.E};
    for (int j = threadIdx.x; j < nt; j += NT) {
        const int tkj = s_task[j];
        const int le = tkj >> 2, k = tkj & 3;
        const int c = reinterpret_cast<const int*>(s_code + le)[k];
        const int kind = c & 3, se = (c >> 2) & 3, idx = c >> 4;
        // physical normal N (|N| = edge length) and unit normal of edge k
        const Real Nx = s_nrm[(NC * k + 0) * BT + le], Ny = s_nrm[(NC * k + 1) * BT + le];
        Real len, il;
        lengths_(fma(Nx, Nx, mul_(Ny, Ny)), len, il);
        const Real nx = mul_(Nx, il), ny = mul_(Ny, il);
        const bool bnd = kind == EDGE_BOUNDARY;
        // the other side's slots: halo rows or in-tile slots
        V4* other = kind == EDGE_HALO ? s_htr + idx : s_tr + se * NG * BT + idx;
        const int stride = kind == EDGE_HALO ? HM : BT;
        Real alpha = Real(0);
        if constexpr (MEANS) {
            Real mL[4], mR[4];
            get4(s_mean + le, mL);
            if (kind == EDGE_BOUNDARY) ghost<Real>(se, mL, far, nx, ny, mR);
            else get4(kind == EDGE_HALO ? s_htr + NG * HM + idx : s_mean + idx, mR);
            alpha = llf_alpha<Real>(mL, mR, Nx, Ny, len, gamma, gm1);
        }
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            Real uL[4], uR[4];
            V4* slot = s_tr + (k * NG + g) * BT + le;
            get4(slot, uL);
            // the neighbour's point NG-1-g on its edge se pairs with ours
            // (src/kernelfunctions.cu:545-549); of a boundary edge the other
            // slot is the own one
            V4* nslot = bnd ? slot : other + (NG - 1 - g) * stride;
            get4(nslot, uR);
            if (bnd) ghost_dev<Real>(se, uL, rs, nx, ny, uR);
            Real fh[4], fn[4];  // the flux out of this side and into the neighbour
            if (FLUX == RKDG_FLUX_LLF) {
                Real fL[4], fR[4];
                dev_flux(uL, dev_prims(uL, rs, gm1), rs, Nx, Ny, fL);
                dev_flux(uR, dev_prims(uR, rs, gm1), rs, Nx, Ny, fR);
                const float2 na = make_float2(-alpha, -alpha);
                const float2 tl = f2fma(na, f2sub(lo2(uR), lo2(uL)), f2add(lo2(fL), lo2(fR)));
                const float2 th = f2fma(na, f2sub(hi2(uR), hi2(uL)), f2add(hi2(fL), hi2(fR)));
                const float2 hp = make_float2(0.5f, 0.5f), hn = make_float2(-0.5f, -0.5f);
                set4(fh, f2mul(hp, tl), f2mul(hp, th));
                set4(fn, f2mul(hn, tl), f2mul(hn, th));
            } else {
                Real f[4];
                hllc_dev(uL, uR, nx, ny, gamma, rs, f);
                const float2 l = make_float2(len, len), nl = make_float2(-len, -len);
                set4(fh, f2mul(lo2(f), l), f2mul(hi2(f), l));
                set4(fn, f2mul(lo2(f), nl), f2mul(hi2(f), nl));
            }
            // each slot of an edge is read by this task alone: the other
            // side's slot takes the negated flux (an in-tile neighbour's; a
            // halo's is read no more; a boundary's is overwritten at once),
            // the computing side's the flux
            put4(nslot, fn);
            put4(slot, fh);
        }
    }
}

// Surface term: the outward fluxes in an element's own slots.
template <int NB, int NG, int BT>
__device__ __forceinline__ void project32(const Tab2& t2, const Vec4<float>* s_tr, float R[NB][4]) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            float f[4];
            get4(s_tr + (k * NG + g) * BT + threadIdx.x, f);
            acc_rows<0, NB>(R, f, t2.nephiw[k][g]);
        }
}

// Runge-Kutta update of one row: U^n + b ((U - U^n) + dt R) (a U^n + b (U +
// dt L) with a + b = 1 exactly: 1/3 and 2/3 both round up in FP32, and a
// scale of 1 + 3e-8 per step would accumulate), or b (U + dt R) in a first
// stage.
__device__ __forceinline__ void update_row32(const float u[4], const float u0[4], float dt, float b, float r[4]) {
    const float2 dt2 = make_float2(dt, dt), b2 = make_float2(b, b);
    set4(r, f2fma(b2, f2fma(dt2, lo2(r), f2sub(lo2(u), lo2(u0))), lo2(u0)),
         f2fma(b2, f2fma(dt2, hi2(r), f2sub(hi2(u), hi2(u0))), hi2(u0)));
}
__device__ __forceinline__ void update_row32(const float u[4], float dt, float b, float r[4]) {
    const float2 dt2 = make_float2(dt, dt), b2 = make_float2(b, b);
    set4(r, f2mul(b2, f2fma(dt2, lo2(r), lo2(u))), f2mul(b2, f2fma(dt2, hi2(r), hi2(u))));
}
// RKDG_FP32C: the mean's update in FP64 from its high and low parts (h, l;
// U^n's h0, l0, zero in a first stage), split again, so that the mean's
// storage rounding does not accumulate over the stages.
__device__ __forceinline__ void update_mean32c(const float h[4], const float l[4], const float h0[4], const float l0[4],
                                               double dt, double b, float r[4], float low[4]) {
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const double m = add_((double)h[v], (double)l[v]), m0 = add_((double)h0[v], (double)l0[v]);
        const double y = fma(b, fma(dt, (double)r[v], add_(m, -m0)), m0);
        r[v] = (float)y;
        low[v] = (float)add_(y, -(double)r[v]);
    }
}

// Returns, when the stage is followed by the TVB limiter (a.tile_flags set),
// whether the limiter may change this thread's element (tvb_keeps fails).
template <typename Real, int NB, int NQ, int NG, int FLUX, int MODE, int BT>
__device__ __forceinline__ bool tile_stage(const StageArgs& a, const TileArgs& ta, const int4 d0,
                                           const int4 d1, unsigned char* smem_raw, unsigned char* stg,
                                           const int nxt, const int ntiles, uint64_t* bar,
                                           const TilePre<Real>& pre, const float2* s_ephi, Real (*s_red)[3],
                                           const double* s_dt) {
    constexpr int CFG = cfg_index(NQ, NG);
    using V4 = Vec4<Real>;
    const Tab<Real>& tb = tab<Real>(CFG);
    const int HM = ta.max_halo;
    constexpr int NC = TiledLayout<Real, BT>::NC;
    Real* s_nrm = reinterpret_cast<Real*>(smem_raw);                       // [3][NC][BT] Nx, Ny
    int4* s_code = reinterpret_cast<int4*>(smem_raw + TiledLayout<Real, BT>::code_off);  // [BT]
    uint16_t* s_task = reinterpret_cast<uint16_t*>(s_code + BT);           // [3 BT] flux tasks
    V4* s_tr = reinterpret_cast<V4*>(s_task + 3 * BT);                     // [3][NG][BT] own traces
    constexpr int MEANS = FLUX == RKDG_FLUX_LLF ? 1 : 0;                   // LLF needs cell means
    V4* s_mean = s_tr + 3 * NG * BT;                                       // [BT] (LLF)
    // halo traces and means: in the staging rows, over each neighbour's own
    // staged state (trace g of halo h in row g, entry h; its mean in row NG).
    // Each halo thread writes only its own entry, after it has read the rows
    // there.
    V4* s_htr = reinterpret_cast<V4*>(stg);
    V4* s_hmean = s_htr + NG * HM;  // (LLF)
    const Tab2& t2 = c_tab_f2[CFG];   // paired tables of the lane-pair arithmetic
    const int sid = d0.z;
    StepCtl* ctl = a.ctl + sid;

    const int tid = threadIdx.x;
    const int e0 = d0.x;
    const int e = e0 + tid;
    const bool active = tid < d0.y;
    const int ee = active ? e : e0;
    const int sx = active ? tid : 0;  // staging row index
    const Real* U = static_cast<const Real*>(a.U);
    const Real gamma = (Real)a.gamma, gm1 = gamma - Real(1);
    // traces and fluxes in deviation form about the reference state; a
    // stored mean is the deviation from it
    const RefState<Real> rs = pre.rs;
    const Real far[4] = {rs.rho, rs.mx, rs.my, rs.E};

    // ------------------------------------------------------------ phase A
    constexpr int SR = NB;  // 16-byte rows of a state
    const int nh = d1.y, nt = d1.w;
    const int2* hh = pre.hh;
    Real R[NB][4];
    Real u[NB][4];
    const double det = pre.det;
    const Real inv_area = pre.inv_area;
    const Real j00 = pre.j00, j01 = pre.j01, j10 = pre.j10, j11 = pre.j11;  // rows of 2 area J^-1
    {
        load_staged<NB, BT>(stg, sx, u);
        __syncthreads();  // staged rows consumed: the area takes the halo states
        {
            const char* Ub = static_cast<const char*>(a.U);
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const int h = tid + r * BT;
                if (h < nh) {
#pragma unroll
                    for (int q = 0; q < SR; ++q)
                        cp_async16(stg + ((size_t)q * HM + h) * 16, Ub + ((size_t)q * a.ld + hh[r].x) * 16);
                }
            }
        }
        {
            Real mfull[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) mfull[v] = add_(u[0][v], far[v]);  // the cell mean itself
            if constexpr (MEANS) put4(s_mean + tid, mfull);
        }
#pragma unroll
        for (int i = 0; i < NB; ++i)
#pragma unroll
            for (int v = 0; v < 4; ++v) R[i][v] = Real(0);
        volume32<NB, NQ>(t2, u, rs, j00, j01, j10, j11, gm1, R);
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                Real t[4];
                comb_rows<NB>(t2.ephi[k][g], u, lo2(u[0]), hi2(u[0]), t);
                put4(s_tr + (k * NG + g) * BT + tid, t);
            }
    }
    cp_async_wait_all();
    __syncthreads();  // s_ephi visible below; own traces complete; halo states landed
    {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int h = tid + r * BT;
            if (h < nh) {
                Real un[NB][4];
                const float4* p = reinterpret_cast<const float4*>(stg);
#pragma unroll
                for (int i = 0; i < NB; ++i) {
                    const float4 x = p[i * HM + h];
                    un[i][0] = x.x, un[i][1] = x.y, un[i][2] = x.z, un[i][3] = x.w;
                }
                if constexpr (MEANS) {
                    Real mfull[4];
#pragma unroll
                    for (int v = 0; v < 4; ++v) mfull[v] = add_(un[0][v], far[v]);
                    put4(s_hmean + h, mfull);
                }
                const int he = hh[r].y;
#pragma unroll
                for (int g = 0; g < NG; ++g) {
                    Real t[4];
                    comb_rows<NB>(s_ephi + (he * NG + g) * NB, un, lo2(un[0]), hi2(un[0]), t);
                    put4(s_htr + g * HM + h, t);
                }
            }
        }
    }
    __syncthreads();  // halo traces complete
    int4 nd0 = make_int4(0, 0, 0, 0);
    if (tid == 0 && nxt < ntiles) {  // the CTA's next tile (only this thread reads its descriptor)
        nd0 = __ldg(ta.desc + 2 * nxt);
        stage_prefetch<Real, true>(a, ta, nd0, __ldg(ta.desc + 2 * nxt + 1));
    }
    prefetch_ahead<Real, BT>(a, ta, nxt, ntiles);

    // ------------------------------------------------------------ phase B
    flux_tasks32<NG, FLUX, BT, BT>(nt, s_task, s_code, s_nrm, s_tr, s_mean, s_htr, HM, rs, gamma);
    __syncthreads();  // fluxes complete, halo traces read: the staging area takes the next tile's rows
    if (tid == 0 && nxt < ntiles) {
        fence_proxy_async();
        stage_copy<Real, BT>(a, nd0, stg, bar);
    }

    // ------------------------------------------------------------ phase C
    // every own slot now holds the outward flux of its edge point
    project32<NB, NG, BT>(t2, s_tr, R);

    Real* Uout = static_cast<Real*>(a.Unew);
    if (MODE == MODE_RESIDUAL) {
        const Real sc = (Real)det;
#pragma unroll
        for (int i = 0; i < NB; ++i)
#pragma unroll
            for (int v = 0; v < 4; ++v) R[i][v] *= sc;
        if (active) store_state<Real, NB>(Uout, a.ld, e, R);
        return false;
    }
    const double dtd = *s_dt;
    const Real dt = (Real)mul_(dtd, det), cb = (Real)a.b;
    Real u0m[4] = {Real(0), Real(0), Real(0), Real(0)};
    // RKDG_FP32C (comp): row 0 is updated in FP64 below, not here
    constexpr bool comp = (MODE & MODE_STAGE_COMP) != 0;
    load_state<Real, NB>(U, a.ld, ee, u);  // stored values (L2 hit)
    const size_t lr = comp ? (size_t)a.lo_row * a.ld : 0;
    float4 l = make_float4(0.f, 0.f, 0.f, 0.f), l0 = l;
    if constexpr (comp) l = reinterpret_cast<const float4*>(a.U)[lr + ee];
    if (a.U0 != nullptr) {
        Real u0[NB][4];
        load_state<Real, NB>(static_cast<const Real*>(a.U0), a.ld, ee, u0);
        if constexpr (comp) l0 = reinterpret_cast<const float4*>(a.U0)[lr + ee];
#pragma unroll
        for (int i = comp ? 1 : 0; i < NB; ++i) update_row32(u[i], u0[i], dt, cb, R[i]);
#pragma unroll
        for (int v = 0; v < 4; ++v) u0m[v] = u0[0][v];
    } else {
#pragma unroll
        for (int i = comp ? 1 : 0; i < NB; ++i) update_row32(u[i], dt, cb, R[i]);
    }
    if constexpr (comp) {
        // RKDG_FP32C: the cell mean is the unevaluated sum of its stored high
        // part (row 0) and low part (row lo_row).  Rows 1.. are stored as
        // updated above; R[0] still holds the mean's residual, and the
        // mean's update runs in FP64 from both parts, split again into a
        // high and a low float, so the mean's storage rounding does not
        // accumulate over the stages.
        if (active) store_rows<Real, 1, NB>(Uout, a.ld, e, R);
        const float lv[4] = {l.x, l.y, l.z, l.w}, l0v[4] = {l0.x, l0.y, l0.z, l0.w};
        float nl[4];
        update_mean32c(u[0], lv, u0m, l0v, mul_(dtd, det), a.b, R[0], nl);
        if (active) {
            reinterpret_cast<float4*>(a.Unew)[e] = make_float4(R[0][0], R[0][1], R[0][2], R[0][3]);
            reinterpret_cast<float4*>(a.Unew)[lr + e] = make_float4(nl[0], nl[1], nl[2], nl[3]);
        }
    } else {
        if (active) store_state<Real, NB>(Uout, a.ld, e, R);
    }
    if (a.last_stage) {
        // CFL wave maximum (and the residual monitor when asked) of the new
        // state: a max over each warp in the working precision into s_red;
        // after the tile's closing barrier one thread takes the max over the
        // warps and makes one atomic per tile on the solve's control block
        // (a solve's atomics meet at one address, so their number is kept
        // small)
        Real wv = Real(0), m0 = Real(0), m1 = Real(0);
        if (active) {
            bool bad;
            Real m[4], len[3];
#pragma unroll
            for (int v = 0; v < 4; ++v) m[v] = add_(R[0][v], far[v]);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const Real Nx = s_nrm[(NC * k + 0) * BT + tid], Ny = s_nrm[(NC * k + 1) * BT + tid];
                len[k] = sqrt_(fma(Nx, Nx, mul_(Ny, Ny)));
            }
            wv = (Real)wave_of<Real>(m, gamma, len, inv_area, bad);
            if (bad) atomicOr(&ctl->error, 1);
            if (a.monitor) {
                m0 = fabs(add_(R[0][0], -u0m[0]));
                m1 = fabs(add_(R[0][3], -u0m[3]));
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
      if (active && (a.limiter_on == nullptr || a.limiter_on[sid])) {
        // the limiter's exact test on the new state (its P1 part at the edge
        // midpoints, the mean, the TVB thresholds from the rows of 2 area
        // J^-1: the columns of J are (j11, -j10) and (-j01, j00))
        Real mean[4], tmax = Real(0);
#pragma unroll
        for (int v = 0; v < 4; ++v) mean[v] = add_(R[0][v], far[v]);
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int v = 0; v < 4; ++v) tmax = fmax(tmax, fabs(tb.mphi[k][0] * R[1][v] + tb.mphi[k][1] * R[2][v]));
        Real dirx[3], diry[3], thr[3];
        tvb_geometry<Real>(j11, -j10, -j01, j00, (Real)a.tvb_m, dirx, diry, thr);
        need = !tvb_keeps<Real>(mean, gamma, tmax, fmin(fmin(thr[0], thr[1]), thr[2]));
      }
    }
    return need;
}

// The tile's maxima from s_red into its solve's control block (one thread,
// after the barrier that closes the tile; bits of a non-negative double
// order like the values).
template <typename Real, int NT>
__device__ __forceinline__ void tile_maxima_atomic(const StageArgs& a, StepCtl* ctl, const Real (*s_red)[3]) {
    Real w = s_red[0][0], m0 = s_red[0][1], m1 = s_red[0][2];
#pragma unroll
    for (int k = 1; k < NT / 32; ++k) {
        w = fmax(w, s_red[k][0]);
        m0 = fmax(m0, s_red[k][1]);
        m1 = fmax(m1, s_red[k][2]);
    }
    atomicMax(&ctl->wave_bits, (unsigned long long)__double_as_longlong((double)w));
    if (a.monitor) {
        atomicMax(&ctl->mon_bits[0], (unsigned long long)__double_as_longlong((double)m0));
        atomicMax(&ctl->mon_bits[1], (unsigned long long)__double_as_longlong((double)m1));
    }
}

// ORD: 1 = P1 tiles only, 2 = P2 tiles only, 3 = both (dispatch per tile;
// P2 tiles use the NQ2-point volume rule, P1 tiles the 3/2-point rules).
// BT: elements per tile = threads per CTA.
// A barrier wait that times out sets bit 1 of the solve's error word and
// ends the CTA (all threads together).
template <int NQ2, int FLUX, int MODE, int ORD, int BT>
__global__ void __launch_bounds__(BT, TiledOccupancy<ORD, BT>::value)
    tiled_stage_kernel(const StageArgs a, const TileArgs ta) {
    using Real = float;
    using SM = TiledSmem<Real, ORD, FLUX, BT>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ Real s_red[BT / 32][3];  // per-warp maxima of a last stage
    __shared__ double s_dt;             // the tile's solve's dt (read before the staging wait)
    unsigned char* stg = smem_raw + SM::stage_offset(ta.max_halo);
    const int ntiles = ta.ntiles_dev ? *ta.ntiles_dev : ta.ntiles;
    int tile = blockIdx.x;
    if (tile >= ntiles) {  // a launch without a tile also completes only after the ones ahead of it
        grid_dependency_wait();
        return;
    }
    // every thread's descriptor load is in flight while the barrier is set
    // up; nobody waits for the thread that issues the copies
    int4 d0 = __ldg(ta.desc + 2 * tile), d1 = __ldg(ta.desc + 2 * tile + 1);
    grid_dependents_launch();
    if (threadIdx.x == 0) mbar_init(&s_bar, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        grid_dependency_wait();
        stage_copy<Real, BT>(a, d0, stg, &s_bar);
    }
    __shared__ float2 s_ephi[ORD == 3 ? 2 : 1][3 * kMaxNG * kMaxNB];
    load_edge_table<ORD, NQ2, BT>(g_ephi_f2, s_ephi);  // (read after later barriers)
    const double2* jinv2 = reinterpret_cast<const double2*>(a.jinv);
    uint32_t parity = 0;
    for (;; tile += gridDim.x, d0 = __ldg(ta.desc + 2 * tile), d1 = __ldg(ta.desc + 2 * tile + 1)) {
        const int nxt = tile + gridDim.x;
        // this thread's J^-1 rows and edge codes, and the work that needs
        // only them, while the state rows arrive
        const int ex = d0.x + ((int)threadIdx.x < d0.y ? (int)threadIdx.x : 0);
        const double2 r0 = __ldg(jinv2 + ex), r1 = __ldg(jinv2 + a.ld + ex);
        const int4 code = __ldg(ta.code + ex);
        grid_dependency_wait();
        const int done = MODE != MODE_RESIDUAL ? a.ctl[d0.z].done : 0;
        if (MODE != MODE_RESIDUAL && threadIdx.x == 0) s_dt = a.ctl[d0.z].dt;
        const TilePre<Real> pre = tile_pre<Real, BT>(a, ta, d0, d1, r0, r1, code, smem_raw);
        const bool ok = mbar_wait(&s_bar, parity);
        if (__syncthreads_or(!ok)) {  // also: every thread has seen this phase complete
            if (threadIdx.x == 0) atomicOr(&a.ctl[d0.z].error, 2);
            return;
        }
        parity ^= 1u;
        if (done) {  // finished solve: pass the tile on
            if (nxt >= ntiles) return;
            if (threadIdx.x == 0) stage_copy<Real, BT>(a, __ldg(ta.desc + 2 * nxt), stg, &s_bar);
            continue;
        }
        bool need;
        if (ORD == 2 || (ORD == 3 && d0.w == 2))
            need = tile_stage<Real, 6, NQ2, 3, FLUX, MODE, BT>(a, ta, d0, d1, smem_raw, stg, nxt, ntiles, &s_bar, pre,
                                                              s_ephi[0], s_red, &s_dt);
        else
            need = tile_stage<Real, 3, 3, 2, FLUX, MODE, BT>(a, ta, d0, d1, smem_raw, stg, nxt, ntiles, &s_bar, pre,
                                                            s_ephi[ORD == 3 ? 1 : 0], s_red, &s_dt);
        // shared memory is reused by the next tile (with the limiter the
        // barrier also ORs its test over the tile)
        if constexpr (MODE & MODE_LIMITED) {
            const int any = __syncthreads_or(need);
            if (threadIdx.x == 0 && any && atomicExch(a.tile_flags + tile, 1) == 0) {
                const int slot = atomicAdd(a.tile_list, 1);
                if (slot < a.tile_cap) a.tile_list[kListHead + slot] = tile;
            }
        } else {
            __syncthreads();
        }
        if (MODE != MODE_RESIDUAL && a.last_stage && threadIdx.x == 0)
            tile_maxima_atomic<Real, BT>(a, a.ctl + d0.z, s_red);
        if (nxt >= ntiles) return;
    }
}
