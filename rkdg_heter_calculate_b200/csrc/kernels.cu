// sm_100a kernels of the RKDG residual and time-step path.
//
// One fused kernel per Runge-Kutta stage replaces the reference's chain of
// nine launches per stage (src/kernelfunctions.cu:84-748): the tile-staged
// stage kernel (stage_tiled.cuh) evaluates each element's state at the
// volume points, projects the contravariant Euler fluxes onto the basis
// gradients, forms the edge traces and the Riemann flux at the Gauss points
// of every edge once per tile, and applies the SSP-RK stage update in its
// epilogue.  Nothing but the state is written to HBM: traces, fluxes and
// residuals live in registers and shared memory.  Device functions common to
// the CUDA sources are in device.cuh; solves that fit on the device run whole
// steps in one launch (resident.cuh).  This file also holds the limiter's
// kernel, the CFL/step kernels and the boundary conversions.
//
// HBM layout (element-interleaved packs for 128-bit accesses):
//   state  : row r = 4*i + v (basis i, variable v), packs of W = 16/sizeof(Real)
//            rows; pack p of element e at ((p*ld + e) * W)  -> one 16-byte
//            load per pack, a warp reads 512 contiguous bytes; RKDG_FP32C
//            adds one pack row holding the low parts of the cell means;
//   jinv   : FP64 rows of J^-1, [2][ld] double2 = (r0x, r0y), (r1x, r1y);
//   conn   : [ld] int4 = (neighbour 0, 1, 2, packed shared-edge/boundary tags).
// The basis is orthonormal under the area average on the reference
// triangle, so M = area * I and every geometric factor of the stage comes
// from J^-1: the scaled normals N_k/area are 2(r0+r1), -2 r0, -2 r1.
#include "device.cuh"

namespace rkdg {

// Self-test of the bounded wait: one thread arms an mbarrier for 16 bytes
// that no copy ever delivers and waits on it with the given limit; out[0] =
// 1 if the wait gave up, out[1] = nanoseconds waited.  Nothing is in flight
// when it returns.
__global__ void wait_selftest_kernel(uint64_t limit_ns, unsigned long long* out) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x != 0) return;
    mbar_init(&bar, 1);
    mbar_expect_tx(&bar, 16);
    const uint64_t t0 = global_ns();
    const bool ok = mbar_wait(&bar, 0, limit_ns);
    out[0] = ok ? 0ull : 1ull;
    out[1] = global_ns() - t0;
}

// CFL measure of the current state per solve (first step, rkdg_compute_dt):
// one CTA per tile (its threads loop over the tile's elements), a block max
// per tile, one atomicMax into its solve.
constexpr int kAuxBlock = 128;
template <typename Real>
__global__ void __launch_bounds__(kAuxBlock) wave_kernel(const TileArgs ta, int ld,
                                                         const Real* __restrict__ U,
                                                         const double* __restrict__ jinv, double gamma,
                                                         StepCtl* ctl, const double* __restrict__ refs) {
    const int ntiles = ta.ntiles_dev ? *ta.ntiles_dev : ta.ntiles;
    if ((int)blockIdx.x >= ntiles) return;
    const int4 d0 = __ldg(ta.desc + 2 * blockIdx.x);
    StepCtl* c = ctl + d0.z;
    const double* ref = refs + 4 * d0.z;
    double w = 0.0;
    for (int x = threadIdx.x; x < d0.y; x += blockDim.x) {
        const int e = d0.x + x;
        Real m[4];
        load_mean<Real, 1>(U, ld, e, m);
        const double2* j2 = reinterpret_cast<const double2*>(jinv);
        bool bad;
        Real mm[4], len[3], ia;
#pragma unroll
        for (int v = 0; v < 4; ++v) mm[v] = m[v] + ref_of<Real>(ref, v);
        elem_lengths<Real>(j2[e], j2[ld + e], len, ia);
        w = fmax(w, wave_of<Real>(mm, (Real)gamma, len, ia, bad));
        if (bad) atomicOr(&c->error, 1);
    }
    block_max3_atomic(w, 0.0, 0.0, &c->wave_bits, nullptr, nullptr);
}

__global__ void reset_wave_kernel(StepCtl* ctl, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) ctl[i].wave_bits = 0ull;
}

// dt of the step: CFL (or fixed), clipped to land on t_final; advances t.
__global__ void step_begin_kernel(StepCtl* ctls, int n, int chain) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    grid_dependents_launch();
    grid_dependency_wait();
    if (i >= n) return;
    StepCtl* ctl = ctls + i;
    if (ctl->done || (chain >= 0 && ctl->chain != chain)) return;
    double dt = ctl->dt_fixed > 0 ? ctl->dt_fixed : ctl->cfl / __longlong_as_double((long long)ctl->wave_bits);
    bool last = false;
    if (ctl->t_final > 0) {
        double rem = ctl->t_final - ctl->t;
        if (!(rem > 0)) {
            ctl->done = 1;
            return;
        }
        if (dt >= rem) {
            dt = rem;
            last = true;
        }
    }
    if (!(dt > 0) || !isfinite(dt)) {  // non-physical state: stop, report
        ctl->error |= 1;
        ctl->done = 1;
        return;
    }
    ctl->dt = dt;
    ctl->t = last ? ctl->t_final : ctl->t + dt;
    ctl->step += 1;
    ctl->wave_bits = 0ull;
    ctl->mon_bits[0] = 0ull;
    ctl->mon_bits[1] = 0ull;
}

template <typename Real, int NB>
__device__ __forceinline__ void limit_element(int e, int ld, Real* U,
                                              const int4* __restrict__ conn,
                                              const void* __restrict__ limv,
                                              const double* __restrict__ jinv, double gamma,
                                              const double* f, double tvb_m, const Tab<Real>& tb) {
    using Pair = LimitPair<Real>;
    const Pair* lim = static_cast<const Pair*>(limv);
    const double2* j2 = reinterpret_cast<const double2*>(jinv);
    const double2 r0 = __ldg(j2 + e), r1 = __ldg(j2 + ld + e);
    const int4 cn = __ldg(conn + e);
    const Pair ab[3] = {__ldg(lim + e), __ldg(lim + (size_t)ld + e), __ldg(lim + (size_t)2 * ld + e)};
    Real u[3][4], mean[4], near[3][4] = {};
    load_state<Real, 3>(U, ld, e, u);
    // The neighbours' means are loaded beside the element's own rows (they
    // depend on its connectivity alone), one round trip instead of two.
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int ne = k == 0 ? cn.x : (k == 1 ? cn.y : cn.z);
        if (ne >= 0) load_mean<Real, 1>(U, ld, ne, near[k]);
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        mean[v] = u[0][v] + ref_of<Real>(f, v);
#pragma unroll
        for (int k = 0; k < 3; ++k) near[k][v] += ref_of<Real>(f, v);
    }
    Real m1[4] = {u[1][0], u[1][1], u[1][2], u[1][3]}, m2[4] = {u[2][0], u[2][1], u[2][2], u[2][3]};
    if (!limit_modes<Real>(r0, r1, cn, ab, mean, near, m1, m2, (Real)gamma, (Real)tvb_m, f, &tb)) return;
    Real out[NB][4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        out[1][v] = m1[v];
        out[2][v] = m2[v];
#pragma unroll
        for (int i = 3; i < NB; ++i) out[i][v] = Real(0);
    }
    store_rows<Real, 1, NB>(U, ld, e, out);  // the mean stays: other blocks read it
}

// One tile of the limiter (all threads of the CTA): tiles of solves whose
// flag is 0 (when flags is set) or whose control block says done are
// skipped; P1 and P2 tiles limit their P1 part (P2 tiles drop their
// quadratic modes where limited).
template <typename Real>
__device__ __forceinline__ void limit_tile(const TileArgs& ta, int tile, int ld, Real* U,
                                           const int4* __restrict__ conn, const void* __restrict__ lim,
                                           const double* __restrict__ jinv, const int* __restrict__ flags,
                                           const double* __restrict__ refs, double gamma, double tvb_m, int cfg1,
                                           int cfg2, const StepCtl* ctl) {
    const int4 d0 = __ldg(ta.desc + 2 * tile);
    if ((flags && !flags[d0.z]) || (ctl && ctl[d0.z].done)) return;
    const double* f = refs + 4 * d0.z;
    for (int x = threadIdx.x; x < d0.y; x += blockDim.x) {
        const int e = d0.x + x;
        if (d0.w == 2)
            limit_element<Real, 6>(e, ld, U, conn, lim, jinv, gamma, f, tvb_m, tab<Real>(cfg2));
        else
            limit_element<Real, 3>(e, ld, U, conn, lim, jinv, gamma, f, tvb_m, tab<Real>(cfg1));
    }
}

// The limiter over tiles (one solve, a pack of solves or the serving pool).
// Every path runs this one kernel, so a solve limits to the same bits
// wherever it runs.  Without a tile list every tile is visited; with one
// (the stage kernel's LimitList), only the listed tiles, spread over the
// CTAs of a persistent grid: most of a flow's tiles cannot change (no
// element fails tvb_keeps) and cost nothing.
template <typename Real>
__global__ void __launch_bounds__(kAuxBlock) tiled_limiter_kernel(const TileArgs ta, int ld,
                                                              Real* U,
                                                              const int4* __restrict__ conn,
                                                              const void* __restrict__ lim,
                                                              const double* __restrict__ jinv,
                                                              const int* __restrict__ flags,
                                                              const double* __restrict__ refs,
                                                              double gamma, double tvb_m,
                                                              int cfg1, int cfg2,
                                                              const StepCtl* ctl,
                                                              int* __restrict__ tile_flags,
                                                              int* __restrict__ tile_list, int tile_cap) {
    grid_dependents_launch();
    grid_dependency_wait();
    if (tile_list == nullptr) {
        const int ntiles = ta.ntiles_dev ? *ta.ntiles_dev : ta.ntiles;
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
            limit_tile<Real>(ta, tile, ld, U, conn, lim, jinv, flags, refs, gamma, tvb_m, cfg1, cfg2, ctl);
        return;
    }
    // every CTA reads the count before the last one resets it (the reset
    // follows every CTA's arrival below)
    const int n = min(*(volatile int*)tile_list, tile_cap);
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const int tile = tile_list[kListHead + i];
        limit_tile<Real>(ta, tile, ld, U, conn, lim, jinv, flags, refs, gamma, tvb_m, cfg1, cfg2, ctl);
        if (threadIdx.x == 0) tile_flags[tile] = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(tile_list + 1, 1) == (int)gridDim.x - 1) {  // the last CTA: empty list for the next stage
            tile_list[0] = 0;
            tile_list[1] = 0;
        }
    }
}

// ------------------------------------------------- halo row exchange --
// Rows 0..nrows-1 (16-byte packs) of the listed elements of a state, to or
// from a contiguous buffer [n][nrows]: the pack and unpack of a partition's
// halo exchange.  An index outside [0, T) is skipped and sets bit 2 of the
// error word.
__global__ void gather_rows_kernel(const int4* __restrict__ U, int ld, int T, const int* __restrict__ idx, int n,
                                   int nrows, int4* __restrict__ out, int* err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * nrows) return;
    const int j = i / nrows, r = i - j * nrows;
    const int e = idx[j];
    if (e < 0 || e >= T) {
        atomicOr(err, 4);
        return;
    }
    out[i] = U[(size_t)r * ld + e];
}

__global__ void scatter_rows_kernel(int4* __restrict__ U, int ld, int T, const int* __restrict__ idx, int n,
                                    int nrows, const int4* __restrict__ in, int* err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * nrows) return;
    const int j = i / nrows, r = i - j * nrows;
    const int e = idx[j];
    if (e < 0 || e >= T) {
        atomicOr(err, 4);
        return;
    }
    U[(size_t)r * ld + e] = in[i];
}

// ---------------------------------------------------- basis conversion --
// Caller layout [4][NB][ldh] FP64 (caller element order) <-> HBM packs
// (internal order), with an optional per-element basis change.
template <typename Real, int NB>
__global__ void import_kernel(int T, int ld, const double* __restrict__ st, int ldh,
                              const double* __restrict__ conv, const int32_t* __restrict__ perm,
                              Real* __restrict__ U, Ref4 ref, int lo_row) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= T) return;
    const int c = perm ? perm[e] : e;
    double a[NB][4];
#pragma unroll
    for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int i = 0; i < NB; ++i) a[i][v] = st[((size_t)v * NB + i) * ldh + c];
    Real b[NB][4];
    if (conv) {
        const double* C = conv + (size_t)36 * e;
#pragma unroll
        for (int j = 0; j < NB; ++j)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                double s = 0;
#pragma unroll
                for (int i = 0; i < NB; ++i) s += a[i][v] * C[6 * i + j];
                b[j][v] = (Real)s;
            }
    } else {
#pragma unroll
        for (int i = 0; i < NB; ++i)
#pragma unroll
            for (int v = 0; v < 4; ++v) b[i][v] = (Real)a[i][v];
    }
    float lo[4] = {0.f, 0.f, 0.f, 0.f};
    if (stores_deviation<Real>()) {  // mean row = basis 0 (basis-invariant)
        const double* Cm = conv ? conv + (size_t)36 * e : nullptr;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            double m = 0;
            if (Cm) {
#pragma unroll
                for (int i = 0; i < NB; ++i) m += a[i][v] * Cm[6 * i];
            } else {
                m = a[0][v];
            }
            b[0][v] = (Real)(m - ref.v[v]);
            lo[v] = (float)((m - ref.v[v]) - (double)b[0][v]);
        }
    }
    store_state<Real, NB>(U, ld, e, b);
    if (sizeof(Real) == 4 && lo_row >= 0)  // FP32C: the low parts of the cell means
        reinterpret_cast<float4*>(U)[(size_t)lo_row * ld + e] = make_float4(lo[0], lo[1], lo[2], lo[3]);
}

template <typename Real, int NB>
__global__ void export_kernel(int T, int ld, const Real* __restrict__ U,
                              const double* __restrict__ conv, const int32_t* __restrict__ perm,
                              double* __restrict__ st, int ldh, int residual_scale,
                              const double* __restrict__ jinv, Ref4 ref, int lo_row) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= T) return;
    const int c = perm ? perm[e] : e;
    Real bl[NB][4];
    load_state<Real, NB>(U, ld, e, bl);
    double b[NB][4];
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
        for (int v = 0; v < 4; ++v) b[i][v] = (double)bl[i][v];
    if (sizeof(Real) == 4 && lo_row >= 0 && !residual_scale) {  // FP32C: add the low parts
        const float4 l = reinterpret_cast<const float4*>(U)[(size_t)lo_row * ld + e];
        b[0][0] += (double)l.x, b[0][1] += (double)l.y, b[0][2] += (double)l.z, b[0][3] += (double)l.w;
    }
    if (stores_deviation<Real>() && !residual_scale)
#pragma unroll
        for (int v = 0; v < 4; ++v) b[0][v] += ref.v[v];
    double scale = 1.0;
    if (residual_scale) {  // area = 1 / (2 det J^-1)
        const double2* j2 = reinterpret_cast<const double2*>(jinv);
        double2 r0 = j2[e], r1 = j2[ld + e];
        scale = 0.5 / (r0.x * r1.y - r0.y * r1.x);
    }
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            double s;
            if (conv) {
                const double* M = conv + (size_t)36 * e + 6 * i;
                s = 0;
#pragma unroll
                for (int j = 0; j < NB; ++j) s += M[j] * b[j][v];
            } else {
                s = b[i][v];
            }
            st[((size_t)v * NB + i) * ldh + c] = scale * s;
        }
}

// --------------------------------------------------- conservation totals --
constexpr int kTotBlock = 256;
int totals_partial_count(int T) { return (T + kTotBlock - 1) / kTotBlock; }

template <typename Real>
__global__ void __launch_bounds__(kTotBlock) totals_partial_kernel(int T, int ld,
                                                                   const Real* __restrict__ U,
                                                                   const double* __restrict__ jinv,
                                                                   double* __restrict__ partial,
                                                                   Ref4 ref, int lo_row) {
    __shared__ double s[4][kTotBlock];
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    double v4[4] = {0, 0, 0, 0};
    if (e < T) {
        Real m[4];
        load_mean<Real, 1>(U, ld, e, m);
        const double2* j2 = reinterpret_cast<const double2*>(jinv);
        double2 r0 = j2[e], r1 = j2[ld + e];
        double area = 0.5 / (r0.x * r1.y - r0.y * r1.x);
        double lo[4] = {0.0, 0.0, 0.0, 0.0};
        if (sizeof(Real) == 4 && lo_row >= 0) {  // FP32C: the low parts of the means
            const float4 l = reinterpret_cast<const float4*>(U)[(size_t)lo_row * ld + e];
            lo[0] = l.x, lo[1] = l.y, lo[2] = l.z, lo[3] = l.w;
        }
        for (int v = 0; v < 4; ++v)
            v4[v] = area * (((double)m[v] + lo[v]) + (stores_deviation<Real>() ? ref.v[v] : 0.0));
    }
    for (int v = 0; v < 4; ++v) s[v][threadIdx.x] = v4[v];
    __syncthreads();
    for (int o = kTotBlock / 2; o > 0; o >>= 1) {  // fixed-order tree: deterministic
        if (threadIdx.x < o)
            for (int v = 0; v < 4; ++v) s[v][threadIdx.x] += s[v][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int v = 0; v < 4; ++v) partial[(size_t)4 * blockIdx.x + v] = s[v][0];
}

__global__ void __launch_bounds__(kTotBlock) totals_final_kernel(int n, const double* __restrict__ partial,
                                                                 double* __restrict__ out) {
    __shared__ double s[4][kTotBlock];
    double acc[4] = {0, 0, 0, 0};
    for (int i = threadIdx.x; i < n; i += kTotBlock)
        for (int v = 0; v < 4; ++v) acc[v] += partial[(size_t)4 * i + v];
    for (int v = 0; v < 4; ++v) s[v][threadIdx.x] = acc[v];
    __syncthreads();
    for (int o = kTotBlock / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o)
            for (int v = 0; v < 4; ++v) s[v][threadIdx.x] += s[v][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int v = 0; v < 4; ++v) out[v] = s[v][0];
}

// ----------------------------------------------------------- launchers --
void upload_tables(int nq, int ng) { upload_module_tables(nq, ng); }

int current_device() {
    int dev = 0;
    RKDG_CUDA_TRY(cudaGetDevice(&dev));
    return dev;
}

// An attribute of the current device, asked for once on each (none is zero).
static int device_attribute(PerDevice<int>& kept, cudaDeviceAttr attr) {
    const int dev = current_device();
    return kept.use(dev, [&](int& v) {
        if (v == 0) RKDG_CUDA_TRY(cudaDeviceGetAttribute(&v, attr, dev));
        return v;
    });
}

// The device's largest opt-in dynamic + static shared memory per CTA, less
// the kernels' static shared memory (barrier, maxima, dt, tables).
size_t smem_limit() {
    static PerDevice<int> limit;
    return (size_t)device_attribute(limit, cudaDevAttrMaxSharedMemoryPerBlockOptin) - 1024;
}

int smem_per_sm() {
    static PerDevice<int> n;
    return device_attribute(n, cudaDevAttrMaxSharedMemoryPerMultiprocessor);
}

int sm_count() {
    static PerDevice<int> n;
    return device_attribute(n, cudaDevAttrMultiProcessorCount);
}

namespace {

// Launches a kernel that may start before the one ahead of it in its stream
// has finished (early); the kernel calls grid_dependency_wait before it touches
// anything that one writes.  Only kernels that do so are launched this way.
template <typename... P, typename... A>
void launch_dependent(bool early, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = early ? 1 : 0;
    RKDG_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

// The stage kernel of an arithmetic type.
template <typename Real, int NQ2, int FLUX, int MODE, int ORD, int BT, int LAT = 0>
constexpr auto stage_kernel() {
    if constexpr (sizeof(Real) == 8) return &stage_fp64_kernel<NQ2, FLUX, MODE, ORD, BT, LAT>;
    else return &tiled_stage_kernel<NQ2, FLUX, MODE, ORD, BT>;
}
// Shared-memory attributes of one instantiation for a halo size; returns the
// dynamic shared memory per CTA.
template <typename Real, int NQ2, int FLUX, int MODE, int ORD, int BT, int LAT = 0>
size_t prepare_tiled(int max_halo) {
    const size_t smem = TiledSmem<Real, ORD, FLUX, BT>::bytes(max_halo);
    if (smem > smem_limit())
        throw Error{RKDG_ERR_INVALID, "tiles of " + std::to_string(BT) + " elements with halo lists of " +
                                          std::to_string(max_halo) + " entries need " + std::to_string(smem) +
                                          " bytes of shared memory per CTA, above the device's limit: use "
                                          "128-element tiles or the locality order"};
    constexpr auto kernel = stage_kernel<Real, NQ2, FLUX, MODE, ORD, BT, LAT>();
    // dynamic + static shared memory above 48 KB needs the opt-in.  Per
    // instantiation; raised when a context with a larger halo appears.
    static PerDevice<size_t> opt_in;
    opt_in.use(current_device(), [&](size_t& configured) {
        if (configured == 0)  // give shared memory the whole carveout
            RKDG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                               (int)cudaSharedmemCarveoutMaxShared));
        if (smem > configured) {
            RKDG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            configured = smem;
        }
    });
    return smem;
}

template <typename Real, int NQ2, int FLUX, int MODE, int ORD, int BT>
int occupancy_tiled(int max_halo) {
    const size_t smem = prepare_tiled<Real, NQ2, FLUX, MODE, ORD, BT>(max_halo);
    static PerDevice<std::map<size_t, int>> answers;  // by shared memory
    return answers.use(current_device(), [&](std::map<size_t, int>& known) {
        const auto it = known.find(smem);
        if (it != known.end()) return it->second;
        constexpr auto kernel = stage_kernel<Real, NQ2, FLUX, MODE, ORD, BT>();
        int n = 0;
        RKDG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, BT, smem));
        return known[smem] = n;
    });
}

template <typename Real, int NQ2, int FLUX, int MODE, int ORD, int BT, int LAT = 0>
void launch_tiled(const StageArgs& a, const TileArgs& t, int ctas, cudaStream_t s) {
    const size_t smem = prepare_tiled<Real, NQ2, FLUX, MODE, ORD, BT, LAT>(t.max_halo);
    const int grid = (ctas > 0 && ctas < t.ntiles) ? ctas : t.ntiles;
    constexpr auto kernel = stage_kernel<Real, NQ2, FLUX, MODE, ORD, BT, LAT>();
    TileArgs ta = t;
    // FP32 kernels prefetch a device of CTAs ahead (prefetch_ahead).  Below 7/8
    // of such a device they start only after the launch before: CTAs that start
    // early fill the free places of some SMs, and a stage of less than one wave
    // then runs unevenly spread.  Every form measured crosses over at 0.8 to
    // 0.9 of its device (us per step, early against after):
    //   P2 HLLC, 888 places   703 tiles 37.1, 35.3   784 tiles 36.8, 37.5
    //   P2 LLF FP32C          589 tiles 34.4, 31.8   644 tiles 34.7, 36.2
    //   P2 LLF limited        757 tiles 50.8, 51.0   886 tiles 52.2, 53.8
    //   P1 HLLC, 1184 places  1001 tiles 27.7, 27.3  1041 tiles 27.9, 28.7
    //   P1 LLF limited        1001 tiles 37.2, 35.6  1098 tiles 37.2, 38.5
    // FP64 gains at every size (352 to 3,907 tiles: 1-4 %).
    bool early = true;
    if constexpr (sizeof(Real) == 4) {
        const int device = sm_count() * occupancy_tiled<Real, NQ2, FLUX, MODE, ORD, BT>(t.max_halo);
        if (grid == t.ntiles) ta.ahead = device;
        early = 8 * (int64_t)grid >= 7 * (int64_t)device;
    }
    if (grid > 0) launch_dependent(early, kernel, grid, BT, smem, s, a, ta);
}

// Tile sizes the stage kernel is built for: 128 everywhere, 256 for the
// stage (not the residual) kernels the batch autotuner may pick.  FP64
// launches of one CTA per tile whose tiles all fit on the device at once
// run the latency form (fewer warps per SM, no register spills: 3,200- and
// 28,800-triangle P2 meshes step 3-4 % faster than in the throughput form).
template <typename Real, int NQ2, int FLUX, int MODE, int ORD>
void launch_tiled_bt(const StageArgs& a, const TileArgs& t, int ctas, cudaStream_t s) {
    if (t.tile == 128) {
        if constexpr (sizeof(Real) == 8) {
            const int fit = sm_count() * Fp64Occupancy<ORD, 128, 1>::value;
            if ((ctas <= 0 || ctas >= t.ntiles) && t.ntiles_dev == nullptr && t.ntiles <= fit)
                return launch_tiled<Real, NQ2, FLUX, MODE, ORD, 128, 1>(a, t, ctas, s);
        }
        return launch_tiled<Real, NQ2, FLUX, MODE, ORD, 128>(a, t, ctas, s);
    }
    if constexpr (MODE != MODE_RESIDUAL && !(MODE & MODE_LIMITED))
        if (t.tile == 256) return launch_tiled<Real, NQ2, FLUX, MODE, ORD, 256>(a, t, ctas, s);
    throw Error{RKDG_ERR_INVALID, "no stage kernel for a tile of " + std::to_string(t.tile) + " elements"};
}

template <typename Real, int FLUX, int MODE>
void dispatch_tiled(const StageArgs& a, const TileArgs& t, int order, int nq, int ctas,
                    cudaStream_t s) {
    if (order == 1) return launch_tiled_bt<Real, 6, FLUX, MODE, 1>(a, t, ctas, s);
    if (order == 2 && nq == 7) return launch_tiled_bt<Real, 7, FLUX, MODE, 2>(a, t, ctas, s);
    if (order == 2 && nq == 6) return launch_tiled_bt<Real, 6, FLUX, MODE, 2>(a, t, ctas, s);
    if (order == 3 && nq == 6) return launch_tiled_bt<Real, 6, FLUX, MODE, 3>(a, t, ctas, s);
    throw Error{RKDG_ERR_INVALID, "unsupported order/rule combination for the tiled kernel"};
}

template <int MODE>
void dispatch(const StageArgs& a, const TileArgs& t, int order, int nq, int flux, int prec, int ctas,
              cudaStream_t s) {
    const bool hllc = flux == RKDG_FLUX_HLLC;
    if (prec == RKDG_FP32) {
        if (hllc) dispatch_tiled<float, RKDG_FLUX_HLLC, MODE>(a, t, order, nq, ctas, s);
        else dispatch_tiled<float, RKDG_FLUX_LLF, MODE>(a, t, order, nq, ctas, s);
    } else if constexpr (!(MODE & MODE_STAGE_COMP)) {
        if (hllc) dispatch_tiled<double, RKDG_FLUX_HLLC, MODE>(a, t, order, nq, ctas, s);
        else dispatch_tiled<double, RKDG_FLUX_LLF, MODE>(a, t, order, nq, ctas, s);
    } else {
        throw Error{RKDG_ERR_INVALID, "a low-part row needs the FP32 stage"};
    }
    RKDG_CUDA_TRY(cudaGetLastError());
}

}  // namespace

void launch_stage(const StageArgs& a, const TileArgs& t, int order, int nq, int flux, int prec, int ctas,
                  cudaStream_t stream) {
    if (a.tile_flags != nullptr) {
        if (a.lo_row >= 0) dispatch<MODE_STAGE_COMP | MODE_LIMITED>(a, t, order, nq, flux, prec, ctas, stream);
        else dispatch<MODE_STAGE | MODE_LIMITED>(a, t, order, nq, flux, prec, ctas, stream);
    } else {
        if (a.lo_row >= 0) dispatch<MODE_STAGE_COMP>(a, t, order, nq, flux, prec, ctas, stream);
        else dispatch<MODE_STAGE>(a, t, order, nq, flux, prec, ctas, stream);
    }
}

void launch_residual(const StageArgs& a, const TileArgs& t, int order, int nq, int flux, int prec, int ctas,
                     cudaStream_t stream) {
    dispatch<MODE_RESIDUAL>(a, t, order, nq, flux, prec, ctas, stream);
}

void wait_selftest(double limit_s, int* timed_out, double* waited_s) {
    unsigned long long* d = nullptr;
    RKDG_CUDA_TRY(cudaMalloc(&d, 2 * sizeof(unsigned long long)));
    unsigned long long h[2] = {0, 0};
    wait_selftest_kernel<<<1, 32>>>((uint64_t)(limit_s * 1e9), d);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) throw Error{RKDG_ERR_CUDA, std::string("wait self-test: ") + cudaGetErrorString(e)};
    *timed_out = (int)h[0];
    *waited_s = (double)h[1] * 1e-9;
}

void launch_wave(const TileArgs& t, int ld, const void* U, int prec, const double* jinv,
                 double gamma, StepCtl* ctl, int nsolves, const double* refs, cudaStream_t stream) {
    if (nsolves > 0) reset_wave_kernel<<<(nsolves + 127) / 128, 128, 0, stream>>>(ctl, nsolves);
    if (t.ntiles > 0) {
        if (prec == RKDG_FP32)
            wave_kernel<float><<<t.ntiles, kAuxBlock, 0, stream>>>(t, ld, static_cast<const float*>(U), jinv, gamma, ctl, refs);
        else
            wave_kernel<double><<<t.ntiles, kAuxBlock, 0, stream>>>(t, ld, static_cast<const double*>(U), jinv, gamma, ctl, refs);
    }
    RKDG_CUDA_TRY(cudaGetLastError());
}

void launch_step_begin(StepCtl* ctl, int nsolves, int chain, cudaStream_t stream) {
    launch_dependent(true, step_begin_kernel, (nsolves + 127) / 128, 128, 0, stream, ctl, nsolves, chain);
}

namespace {
template <typename Real, int FLUX>
int occupancy_for(int order, int nq, int tile, int max_halo) {
    auto pick = [&](auto bt) -> int {
        constexpr int BT = decltype(bt)::value;
        if (order == 1) return occupancy_tiled<Real, 6, FLUX, MODE_STAGE, 1, BT>(max_halo);
        if (order == 3) return occupancy_tiled<Real, 6, FLUX, MODE_STAGE, 3, BT>(max_halo);
        if (nq == 7) return occupancy_tiled<Real, 7, FLUX, MODE_STAGE, 2, BT>(max_halo);
        return occupancy_tiled<Real, 6, FLUX, MODE_STAGE, 2, BT>(max_halo);
    };
    if (tile == 256) return pick(std::integral_constant<int, 256>{});
    return pick(std::integral_constant<int, 128>{});
}
}  // namespace

size_t tiled_smem_bytes(int prec, int order, int flux, int max_halo, int tile) {
    auto f = [&](auto r, auto bt) -> size_t {
        using Real = decltype(r);
        constexpr int BT = decltype(bt)::value;
        const bool h = flux == RKDG_FLUX_HLLC;
        if (order == 1)
            return h ? TiledSmem<Real, 1, RKDG_FLUX_HLLC, BT>::bytes(max_halo) : TiledSmem<Real, 1, RKDG_FLUX_LLF, BT>::bytes(max_halo);
        if (order == 2)
            return h ? TiledSmem<Real, 2, RKDG_FLUX_HLLC, BT>::bytes(max_halo) : TiledSmem<Real, 2, RKDG_FLUX_LLF, BT>::bytes(max_halo);
        return h ? TiledSmem<Real, 3, RKDG_FLUX_HLLC, BT>::bytes(max_halo) : TiledSmem<Real, 3, RKDG_FLUX_LLF, BT>::bytes(max_halo);
    };
    if (prec == RKDG_FP32)
        return tile == 256 ? f(0.0f, std::integral_constant<int, 256>{}) : f(0.0f, std::integral_constant<int, 128>{});
    return tile == 256 ? f(0.0, std::integral_constant<int, 256>{}) : f(0.0, std::integral_constant<int, 128>{});
}

bool tiled_fits(int prec, int order, int flux, int max_halo, int tile) {
    return tiled_smem_bytes(prec, order, flux, max_halo, tile) <= smem_limit();
}

int tiled_max_ctas_per_sm(int prec, int order, int nq, int flux, int max_halo, int tile) {
    const bool h = flux == RKDG_FLUX_HLLC;
    if (prec == RKDG_FP32)
        return h ? occupancy_for<float, RKDG_FLUX_HLLC>(order, nq, tile, max_halo)
                 : occupancy_for<float, RKDG_FLUX_LLF>(order, nq, tile, max_halo);
    return h ? occupancy_for<double, RKDG_FLUX_HLLC>(order, nq, tile, max_halo)
             : occupancy_for<double, RKDG_FLUX_LLF>(order, nq, tile, max_halo);
}

void launch_tiled_limiter(const TileArgs& t, int ctas, int ld, void* U, const int4* conn,
                          const void* lim, const double* jinv, const int* flags,
                          const double* refs, int prec, int nq2, double gamma, double tvb_m,
                          const StepCtl* ctl, int* tile_flags, int* tile_list, int tile_cap,
                          cudaStream_t stream) {
    const int cfg1 = cfg_index(3, 2), cfg2 = cfg_index(nq2, 3);
    if (tile_list != nullptr && tile_flags == nullptr)
        throw Error{RKDG_ERR_INVALID, "a limiter tile list needs its tile flags"};
    // one CTA per tile, or a persistent grid (the caller's, else four CTAs
    // per SM) over a tile list
    int grid = ctas > 0 ? ctas : std::max(1, t.ntiles);
    if (tile_list != nullptr && ctas <= 0) grid = std::max(1, std::min(t.ntiles, 4 * sm_count()));
    if (prec == RKDG_FP32)
        launch_dependent(true, tiled_limiter_kernel<float>, grid, kAuxBlock, 0, stream, t, ld, static_cast<float*>(U), conn, lim, jinv, flags, refs, gamma, tvb_m, cfg1, cfg2, ctl, tile_flags, tile_list, tile_cap);
    else
        launch_dependent(true, tiled_limiter_kernel<double>, grid, kAuxBlock, 0, stream, t, ld, static_cast<double*>(U), conn, lim, jinv, flags, refs, gamma, tvb_m, cfg1, cfg2, ctl, tile_flags, tile_list, tile_cap);
}

void launch_rows(bool gather, void* U, int ld, int T, const int* idx, int n, int nrows, void* buf, int* err,
                 cudaStream_t stream) {
    const int total = n * nrows;
    if (total <= 0) return;
    const int grid = (total + 255) / 256;
    if (gather)
        gather_rows_kernel<<<grid, 256, 0, stream>>>(static_cast<const int4*>(U), ld, T, idx, n, nrows,
                                                      static_cast<int4*>(buf), err);
    else
        scatter_rows_kernel<<<grid, 256, 0, stream>>>(static_cast<int4*>(U), ld, T, idx, n, nrows,
                                                       static_cast<const int4*>(buf), err);
    RKDG_CUDA_TRY(cudaGetLastError());
}

void launch_import(int T, int ld, const double* staging, int ldh, const double* conv,
                   const int32_t* perm, void* U, int order, int prec, const double* ref, int lo_row,
                   cudaStream_t stream) {
    Ref4 r{{ref[0], ref[1], ref[2], ref[3]}};
    const int grid = (T + 127) / 128;
    if (prec == RKDG_FP32) {
        if (order == 1) import_kernel<float, 3><<<grid, 128, 0, stream>>>(T, ld, staging, ldh, conv, perm, static_cast<float*>(U), r, lo_row);
        else import_kernel<float, 6><<<grid, 128, 0, stream>>>(T, ld, staging, ldh, conv, perm, static_cast<float*>(U), r, lo_row);
    } else {
        if (order == 1) import_kernel<double, 3><<<grid, 128, 0, stream>>>(T, ld, staging, ldh, conv, perm, static_cast<double*>(U), r, -1);
        else import_kernel<double, 6><<<grid, 128, 0, stream>>>(T, ld, staging, ldh, conv, perm, static_cast<double*>(U), r, -1);
    }
    RKDG_CUDA_TRY(cudaGetLastError());
}

void launch_export(int T, int ld, const void* U, const double* conv, const int32_t* perm,
                   double* staging, int ldh, int order, int prec, int residual_scale,
                   const double* jinv, const double* ref, int lo_row, cudaStream_t stream) {
    Ref4 r{{ref[0], ref[1], ref[2], ref[3]}};
    const int grid = (T + 127) / 128;
    if (prec == RKDG_FP32) {
        if (order == 1) export_kernel<float, 3><<<grid, 128, 0, stream>>>(T, ld, static_cast<const float*>(U), conv, perm, staging, ldh, residual_scale, jinv, r, lo_row);
        else export_kernel<float, 6><<<grid, 128, 0, stream>>>(T, ld, static_cast<const float*>(U), conv, perm, staging, ldh, residual_scale, jinv, r, lo_row);
    } else {
        if (order == 1) export_kernel<double, 3><<<grid, 128, 0, stream>>>(T, ld, static_cast<const double*>(U), conv, perm, staging, ldh, residual_scale, jinv, r, -1);
        else export_kernel<double, 6><<<grid, 128, 0, stream>>>(T, ld, static_cast<const double*>(U), conv, perm, staging, ldh, residual_scale, jinv, r, -1);
    }
    RKDG_CUDA_TRY(cudaGetLastError());
}

void launch_totals(int T, int ld, const void* U, int order, int prec, const double* jinv,
                   double* partial, double* out4, const double* ref, int lo_row, cudaStream_t stream) {
    Ref4 r{{ref[0], ref[1], ref[2], ref[3]}};
    (void)order;
    const int n = totals_partial_count(T);
    if (prec == RKDG_FP32)
        totals_partial_kernel<float><<<n, kTotBlock, 0, stream>>>(T, ld, static_cast<const float*>(U), jinv, partial, r, lo_row);
    else
        totals_partial_kernel<double><<<n, kTotBlock, 0, stream>>>(T, ld, static_cast<const double*>(U), jinv, partial, r, -1);
    totals_final_kernel<<<1, kTotBlock, 0, stream>>>(n, partial, out4);
    RKDG_CUDA_TRY(cudaGetLastError());
}

}  // namespace rkdg
