// fvm_api.cu -- the C ABI (include/fvm_b200.h): solve handle, device buffers,
// TMA descriptors, step orchestration, CUDA-graph replay, readback and
// measurement hooks.  Host C++ only launches kernels; there is no CPU
// compute path for anything the reference runs on the GPU.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/fvm_b200.h"
#include "fvm_kernels.cuh"
#include "fvm_tma.cuh"

using namespace fvm;

#define FVM_STR2(x) #x
#define FVM_STR(x) FVM_STR2(x)

// ------------------------------------------------------------ error text
static thread_local std::string g_last_error = "";

static int set_err(int code, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_last_error = buf;
    return code;
}

extern "C" const char *fvm_last_error(void) { return g_last_error.c_str(); }

#define CK(call)                                                                                       \
    do {                                                                                               \
        cudaError_t _e = (call);                                                                       \
        if (_e != cudaSuccess)                                                                         \
            return set_err(FVM_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(_e)); \
    } while (0)

#define CKA(call)                                                                                      \
    do {                                                                                               \
        cudaError_t _e = (call);                                                                       \
        if (_e != cudaSuccess)                                                                         \
            return set_err(FVM_ERR_ALLOC, "%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(_e)); \
    } while (0)

#define CHECK_HANDLE(h)                                                                 \
    do {                                                                                \
        if (!(h)) return set_err(FVM_ERR_INVALID, "%s: null handle", __func__);         \
    } while (0)

#define CHECK_INIT(h)                                                                   \
    do {                                                                                \
        CHECK_HANDLE(h);                                                                \
        if (!(h)->Un) return set_err(FVM_ERR_STATE, "%s: solver not initialized", __func__); \
    } while (0)

// ------------------------------------------------------ parameter helpers
extern "C" void fvm_params_default(fvm_sim_params *p) {
    if (!p) return;
    memset(p, 0, sizeof(*p));
    p->nx = 512;
    p->ny = 256;
    p->dx = 1.0f;
    p->dy = 1.0f;
    p->domain_width = 10.0f;
    p->domain_height = 5.0f;
    p->mach = 3.0f;
    p->T_inf = 300.0f;
    p->p_inf = 101325.0f;
    p->obstacle_x = 2.5f;
    p->obstacle_y = 2.5f;
    p->obstacle_r = 0.5f;
    p->obstacle_shape = FVM_SHAPE_CIRCLE;
    p->cfl = 0.5f;
    p->dt = 1e-6f;
    p->enable_viscosity = false;
    p->cfl_visc = 0.4f;
    p->adiabatic_wall = true;
    p->T_wall = 300.0f;
    p->paused = true;
}

// SimParams::computeDerived (src/include/common.h:93-101)
extern "C" void fvm_params_compute_derived(fvm_sim_params *p) {
    if (!p) return;
    p->rho_inf = p->p_inf / (R_GAS * p->T_inf);
    p->c_inf = sqrtf(GAMMA * R_GAS * p->T_inf);
    p->u_inf = p->mach * p->c_inf;
    p->dx = p->domain_width / (float)p->nx;
    p->dy = p->domain_height / (float)p->ny;
    p->obstacle_y = p->domain_height / 2.0f;
}

extern "C" void fvm_ext_default(fvm_ext *e) {
    if (!e) return;
    memset(e, 0, sizeof(*e));
    e->flux_scheme = FVM_FLUX_HLLC;
    e->limiter = FVM_LIMITER_MINMOD;
    e->prandtl = PRANDTL_REF;
    e->dt_policy = FVM_DT_FIXED;
    e->cone_half_angle = 0.2617993877991494f;
    e->cone_length = 0.3f;
    e->ref_length = 0.0f;
}

// ------------------------------------------------------------ TMA encode
typedef CUresult (*PFN_encodeTiled_t)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                      const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                      CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                      CUtensorMapFloatOOBfill);

static PFN_encodeTiled_t get_encode() {
    static PFN_encodeTiled_t fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_encodeTiled_t>(p);
    }
    return fn;
}

// 3-D map over (x, y, field) of one 5-plane state; box = (box_w, 1, 5).
static int encode_state_map(CUtensorMap *m, float *base, const GridDesc &g, int box_w) {
    PFN_encodeTiled_t enc = get_encode();
    if (!enc) return set_err(FVM_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled unavailable");
    cuuint64_t dims[3] = {(cuuint64_t)g.nx, (cuuint64_t)g.ny, 5};
    cuuint64_t strides[2] = {(cuuint64_t)g.pitch * 4, (cuuint64_t)g.plane * 4};
    cuuint32_t box[3] = {(cuuint32_t)box_w, 1, 5};
    cuuint32_t es[3] = {1, 1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_err(FVM_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return FVM_OK;
}

#include "fvm_handle.h"

static const char *kKernelNames[] = {"stage1", "stage2", "viscous_pre", "viscous_post", "ghost1", "ghost2",
                                     "set_scalars"};

static cudaEvent_t take_event(fvm_handle *h) {
    if (!h->event_pool.empty()) {
        cudaEvent_t e = h->event_pool.back();
        h->event_pool.pop_back();
        return e;
    }
    cudaEvent_t e;
    cudaEventCreate(&e);
    return e;
}

static void resolve_timing(fvm_handle *h) {
    if (h->pending.empty()) return;
    cudaStreamSynchronize(h->stream);
    for (auto &t : h->pending) {
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, t.a, t.b);
        auto &slot = h->ktimes[kKernelNames[t.kernel]];
        slot.first += 1;
        slot.second += ms;
        h->event_pool.push_back(t.a);
        h->event_pool.push_back(t.b);
    }
    h->pending.clear();
}

// Runs `fn` (one kernel launch) bracketed by events when timing is on.
template <class F>
static cudaError_t timed(fvm_handle *h, int kernel, F fn) {
    if (!h->timing) {
        h->launches++;
        return fn();
    }
    TimedLaunch t{kernel, take_event(h), take_event(h)};
    cudaEventRecord(t.a, h->stream);
    cudaError_t e = fn();
    cudaEventRecord(t.b, h->stream);
    h->pending.push_back(t);
    h->launches++;
    return e;
}

static void drop_graphs(fvm_handle *h) {
    h->plain_steps = 0;
    for (int k = 0; k < 2; k++) {
        if (h->graph[k]) cudaGraphExecDestroy(h->graph[k]);
        h->graph[k] = nullptr;
        if (h->graph1[k]) cudaGraphExecDestroy(h->graph1[k]);
        h->graph1[k] = nullptr;
    }
}

static void free_buffers(fvm_handle *h) {
    drop_graphs(h);
    for (int k = 0; k < NBUF; k++) {
        if (h->buf[k]) cudaFree(h->buf[k]);
        h->buf[k] = nullptr;
    }
    if (h->sdf) cudaFree(h->sdf);
    if (h->ct) cudaFree(h->ct);
    if (h->mask) cudaFree(h->mask);
    if (h->ghosts) cudaFree(h->ghosts);
    if (h->d_diag) cudaFree(h->d_diag);
    h->sdf = nullptr;
    h->ct = nullptr;
    h->mask = nullptr;
    h->ghosts = nullptr;
    h->d_diag = nullptr;
    h->n_ghost = h->ghost_cap = 0;
    h->bytes = 0;
    h->parity_base = nullptr;
}

// Launch tuning of the marching kernels per grid class: threads per CTA,
// input ring depth (rows) and rows per CTA.  The default comes from
// heuristic_tune below; FVM_TUNE="nt,ring,rows" overrides it; fvm_autotune
// measures the candidates and caches the winner per grid class for the
// process.
struct TuneKey {
    int nx, ny, viscous, scheme, limiter;
    bool operator<(const TuneKey &o) const {
        return std::tie(nx, ny, viscous, scheme, limiter) < std::tie(o.nx, o.ny, o.viscous, o.scheme, o.limiter);
    }
};
static std::map<TuneKey, StageTune> g_tune_cache;

// Rows per CTA of a marching kernel that keeps `slots` CTAs resident.  If the
// whole grid fits into one resident wave with tiles of at most 24 rows, the
// shortest such tiles: every CTA starts at once and none is left for a second,
// nearly empty wave.  Else about 96 row bands, or 64 from 2000 rows up: several
// waves, which the block scheduler evens out, of tiles tall enough to keep the
// halo rows cheap (the more waves, the taller).
// Measured on B200, step in us by rows: Euler 2048x1024 (one wave from 20)
// 16: 127, 20: 117, 24: 131; 2400x1200 12: 159, 24: 166; 3000x1500 16: 225, 32:
// 231; NS 3000x1500 16: 334, 32: 341; 4096x2048 20: 578, 32: 573, 64: 632;
// 6000x3000 24: 1150, 40: 1128; 8192x4096 40: 2036, 64: 2020.
static int march_rows(int nx, int ny, int slots) {
    const int strips = (nx + 123) / 124;
    for (int rows = 4; rows <= 24; rows += 4)
        if ((long long)strips * ((ny + rows - 1) / rows) <= slots) return rows;
    const double want = ny / (ny < 2000 ? 96.0 : 64.0);
    int best = 12;
    for (int rows : {16, 20, 24, 32, 40, 48, 64})
        if (std::abs(rows - want) < std::abs(best - want)) best = rows;
    return best;
}

// Default launch shape before (or without) autotuning: marching kernels of 128
// threads with a 4-row input ring, and the flat stage kernel up to 1.5 million
// cells.  There a marching stage leaves the chip mostly idle: a CTA works
// through its row pairs one after another (2 us each, the latency of one
// pair's dependent arithmetic) and taller tiles mean fewer CTAs, while the flat
// kernel has a thread for every face at once; above, the flat kernel's
// two-cell halo (1.45 times the cells of a 32x14 tile, 1.88 of a 32x6 one) costs
// more than that.
// Measured Euler steps, marching (best rows) -> flat, us: 256x128 22.6 -> 16.4,
// 512x256 27.3 -> 20.6, 1024x512 49.2 -> 40.0, 1501x777 77.3 -> 72.7, 1800x900
// 96.6 -> 98.8, 2048x1024 116.9 -> 123.7.  Tiles of 32x14 cells, or of 32x6
// while the taller ones would give fewer than 3 CTAs per SM (512x256 20.6
// against 22.6 us, 640x320 25.7 either way, 1024x512 44.0 against 40.0).
static StageTune heuristic_tune(int nx, int ny) {
    constexpr int kSms = 148;
    // 6 stage CTAs and 5 viscous CTAs of 128 threads per SM
    StageTune t{128, 4, march_rows(nx, ny, 6 * kSms), march_rows(nx, ny, 5 * kSms), 0};
    if ((long long)nx * ny <= 1500000) t.flat_pairs = (long long)((nx + 31) / 32) * ((ny + 13) / 14) < 3 * kSms ? 3 : 7;
    return t;
}

static StageTune pick_tune(const fvm_handle *h, int nx, int ny) {
    const char *env = getenv("FVM_TUNE");
    if (env) {
        int x = 0, y = 0, z = 0;
        if (sscanf(env, "%d,%d,%d", &x, &y, &z) == 3 && (x == 128 || x == 256) && (y == 4 || y == 6) && z >= 4 &&
            (z & 1) == 0)
            return StageTune{x, y, z};
    }
    TuneKey k{nx, ny, h->prm.enable_viscosity ? 1 : 0, h->ext.flux_scheme, h->ext.limiter};
    auto it = g_tune_cache.find(k);
    if (it != g_tune_cache.end()) return it->second;
    return heuristic_tune(nx, ny);
}

static int alloc_buffers(fvm_handle *h, int nx, int ny) {
    free_buffers(h);
    GridDesc g;
    g.nx = nx;
    g.ny = ny;
    g.pitch = (nx + 31) / 32 * 32;
    g.plane = (long long)g.pitch * ny;
    g.dx = h->prm.dx;
    g.dy = h->prm.dy;
    h->g = g;
    const size_t state_bytes = (size_t)g.plane * 5 * sizeof(float);
    for (int k = 0; k < NBUF; k++) {
        CKA(cudaMalloc(&h->buf[k], state_bytes));
        CK(cudaMemsetAsync(h->buf[k], 0, state_bytes, h->stream));
    }
    CKA(cudaMalloc(&h->sdf, (size_t)g.plane * sizeof(float)));
    CKA(cudaMalloc(&h->ct, (size_t)nx * ny));
    CKA(cudaMalloc(&h->mask, (size_t)g.plane));
    CK(cudaMemsetAsync(h->ct, 0, (size_t)nx * ny, h->stream));
    h->diag_parts = diagnostics_parts(g);
    CKA(cudaMalloc(&h->d_diag, (size_t)h->diag_parts * 8 * sizeof(double)));
    h->bytes = state_bytes * NBUF + (size_t)g.plane * 5 + (size_t)nx * ny + (size_t)h->diag_parts * 8 * 8;
    h->tune = pick_tune(h, nx, ny);
    return FVM_OK;
}

static int build_maps(fvm_handle *h) {
    CK(prepare_step_kernels(h->tune));
    for (int k = 0; k < NBUF; k++) {
        int r = encode_state_map(&h->tm_in[k], h->buf[k], h->g, stage_box_in(h->tune));
        if (r) return r;
        r = encode_state_map(&h->tm_ctr[k], h->buf[k], h->g, stage_box_blend(h->tune));
        if (r) return r;
    }
    return FVM_OK;
}

static Freestream freestream(const fvm_sim_params &p) { return Freestream{p.rho_inf, p.u_inf, p.v_inf, p.p_inf}; }
static WallParams wall(const fvm_sim_params &p) {
    return WallParams{p.enable_viscosity, p.adiabatic_wall, p.T_wall};
}

__global__ void k_set_scalars(DevScalars *sc, float dt, float t, int set_t) {
    sc->dt = dt;
    if (set_t) sc->t = t;
}

__global__ void k_zero_scalars(DevScalars *sc) {
    sc->red[0] = sc->red[1] = 0.0f;
    sc->cfl[0] = sc->cfl[1] = 0.0f;
    sc->counter = 0;
    sc->err = 0;
    sc->nonfinite = 0;
}

// Geometry from the current parameters: SDF + classes (optionally with the
// zero-state fix-up of newly exposed cells), masks and the ghost table.
static int build_geometry(fvm_handle *h, bool fixup) {
    const fvm_sim_params &p = h->prm;
    ShapeParamsHost s{p.obstacle_x, p.obstacle_y, p.obstacle_r, p.obstacle_rotation, p.wing_rotation,
                      h->ext.cone_half_angle, h->ext.cone_length, p.obstacle_shape};
    launch_sdf(h->g, s, h->sdf, h->ct, fixup ? h->Un : nullptr, h->stream);
    CK(cudaGetLastError());
    launch_mask(h->g, h->ct, h->mask, h->stream);
    CK(cudaGetLastError());
    // one pass fills the table and counts; only a table that proves too small
    // (the first one) is allocated and filled again
    int *const count = reinterpret_cast<int *>(h->h_res);
    auto fill = [&]() -> int {
        CK(cudaMemsetAsync(h->d_count, 0, sizeof(int), h->stream));
        launch_ghost_table(h->g, h->sdf, h->ct, h->ghosts, h->ghost_cap, h->d_count, h->stream);
        CK(cudaGetLastError());
        return FVM_OK;
    };
    if (int r = fill()) return r;
    CK(cudaMemcpyAsync(count, h->d_count, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    const int n = *count;
    if (n > h->ghost_cap) {
        if (h->ghosts) cudaFree(h->ghosts);
        h->ghosts = nullptr;
        h->ghost_cap = h->n_ghost = 0;
        CKA(cudaMalloc(&h->ghosts, (size_t)std::max(n, 64) * sizeof(GhostInfo)));
        h->ghost_cap = std::max(n, 64);
        if (int r = fill()) return r;
    }
    h->n_ghost = n;
    drop_graphs(h);
    return FVM_OK;
}

// Boundary conditions on the current state (both phases), set-up path.
static int apply_bc_full(fvm_handle *h) {
    CK(launch_bc_phase1(h->g, h->Un, h->mask, freestream(h->prm), h->buf[BUF_S], h->stream));
    if (h->n_ghost > 0) {
        GhostArgs ga{};
        ga.g = h->g;
        ga.list = h->ghosts;
        ga.n = h->n_ghost;
        ga.A = h->Un;
        ga.B1 = h->buf[BUF_S];
        ga.B2 = nullptr;
        ga.sc = h->sc;
        ga.fs = freestream(h->prm);
        ga.wall = wall(h->prm);
        CK(launch_ghost(ga, h->stream));
    }
    return FVM_OK;
}

// ------------------------------------------------------------- lifecycle
extern "C" int fvm_create(fvm_handle **out) {
    if (!out) return set_err(FVM_ERR_INVALID, "fvm_create: null out");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0)
        return set_err(FVM_ERR_CUDA, "fvm_create: no CUDA device");
    fvm_handle *h = new fvm_handle();
    cudaGetDevice(&h->device);
    int major = 0, minor = 0;
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, h->device);
    cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, h->device);
    if (major != 10) {
        delete h;
        return set_err(FVM_ERR_UNSUPPORTED, "fvm_create: device sm_%d%d, this build targets sm_100a", major, minor);
    }
    if (cudaStreamCreateWithFlags(&h->own, cudaStreamNonBlocking) != cudaSuccess) {
        delete h;
        return set_err(FVM_ERR_CUDA, "fvm_create: stream creation failed");
    }
    h->stream = h->own;
    fvm_params_default(&h->prm);
    fvm_ext_default(&h->ext);
    if (cudaMalloc(&h->sc, sizeof(DevScalars)) != cudaSuccess || cudaMalloc(&h->d_count, sizeof(int)) != cudaSuccess ||
        cudaMalloc(&h->d_tmp, 16) != cudaSuccess || cudaMalloc(&h->d_counter, sizeof(int)) != cudaSuccess ||
        cudaMalloc(&h->d_disp, sizeof(DisplayDesc)) != cudaSuccess ||
        cudaMallocHost(&h->h_sc, sizeof(DevScalars) + 8 * sizeof(double) + sizeof(HostScalars)) != cudaSuccess) {
        delete h;
        return set_err(FVM_ERR_ALLOC, "fvm_create: allocation failed");
    }
    static_assert(sizeof(DevScalars) % alignof(double) == 0, "the results follow the mirror");
    h->h_res = reinterpret_cast<double *>(h->h_sc + 1);
    h->h_now = reinterpret_cast<HostScalars *>(h->h_res + 8);
    cudaMemsetAsync(h->sc, 0, sizeof(DevScalars), h->stream);
    cudaMemsetAsync(h->d_disp, 0, sizeof(DisplayDesc), h->stream);
    cudaMemsetAsync(h->d_tmp, 0, 16, h->stream);
    cudaStreamSynchronize(h->stream);
    *out = h;
    return FVM_OK;
}

extern "C" int fvm_destroy(fvm_handle *h) {
    if (!h) return FVM_OK;
    cudaStreamSynchronize(h->stream);
    resolve_timing(h);
    free_buffers(h);
    for (auto e : h->event_pool) cudaEventDestroy(e);
    if (h->sc) cudaFree(h->sc);
    if (h->d_count) cudaFree(h->d_count);
    if (h->d_tmp) cudaFree(h->d_tmp);
    if (h->d_counter) cudaFree(h->d_counter);
    if (h->d_disp) cudaFree(h->d_disp);
    if (h->h_sc) cudaFreeHost(h->h_sc);
    if (h->own) cudaStreamDestroy(h->own);
    delete h;
    return FVM_OK;
}

extern "C" int fvm_set_stream(fvm_handle *h, void *stream) {
    CHECK_HANDLE(h);
    cudaStreamSynchronize(h->stream);
    h->stream = stream ? reinterpret_cast<cudaStream_t>(stream) : h->own;
    drop_graphs(h);
    return FVM_OK;
}

static int validate(const fvm_sim_params *p, const fvm_ext *e) {
    if (!p) return set_err(FVM_ERR_INVALID, "null params");
    if (p->nx <= 0 || p->ny <= 0) return set_err(FVM_ERR_INVALID, "nx, ny must be positive (got %d, %d)", p->nx, p->ny);
    if ((long long)p->nx * p->ny > (1LL << 31) - 1) return set_err(FVM_ERR_INVALID, "grid too large");
    if (!(p->dx > 0.0f) || !(p->dy > 0.0f)) return set_err(FVM_ERR_INVALID, "dx, dy must be positive");
    if (p->obstacle_shape < 0 || p->obstacle_shape > 6) return set_err(FVM_ERR_INVALID, "unknown obstacle shape");
    if (e) {
        if (e->flux_scheme < 0 || e->flux_scheme > 1) return set_err(FVM_ERR_INVALID, "unknown flux scheme");
        if (e->limiter < 0 || e->limiter > 1) return set_err(FVM_ERR_INVALID, "unknown limiter");
        if (e->dt_policy < 0 || e->dt_policy > 1) return set_err(FVM_ERR_INVALID, "unknown dt policy");
        if (!(e->prandtl > 0.0f)) return set_err(FVM_ERR_INVALID, "prandtl must be positive");
    }
    return FVM_OK;
}

extern "C" int fvm_reset(fvm_handle *h, const fvm_sim_params *p) {
    CHECK_INIT(h);
    if (int r = validate(p, nullptr)) return r;
    if (p->nx != h->g.nx || p->ny != h->g.ny)
        return set_err(FVM_ERR_INVALID, "fvm_reset: grid %dx%d differs from the allocated %dx%d (use fvm_initialize)",
                       p->nx, p->ny, h->g.nx, h->g.ny);
    h->disp_fresh = false;
    h->prm = *p;
    h->g.dx = p->dx;
    h->g.dy = p->dy;
    k_zero_scalars<<<1, 1, 0, h->stream>>>(h->sc);
    h->now_valid = false;
    h->launches_at_sc_copy = -1;  // the host copy of the scalars is out of date
    CK(cudaGetLastError());
    launch_init(h->g, h->Un, freestream(h->prm), h->stream);
    CK(cudaGetLastError());
    if (int r = build_geometry(h, false)) return r;
    if (int r = apply_bc_full(h)) return r;
    CK(cudaStreamSynchronize(h->stream));
    h->dt_ready = false;
    h->cfl_valid = false;
    return FVM_OK;
}

extern "C" int fvm_initialize(fvm_handle *h, const fvm_sim_params *p, const fvm_ext *ext) {
    CHECK_HANDLE(h);
    if (int r = validate(p, ext)) return r;
    if (h->disp) {  // a registered display field is sized for the old grid
        CK(launch_set_display(h->d_disp, nullptr, 0, h->stream));
        h->disp = nullptr;
    }
    h->disp_fresh = false;
    h->prm = *p;
    if (ext) h->ext = *ext;
    if (int r = alloc_buffers(h, p->nx, p->ny)) return r;
    if (int r = build_maps(h)) return r;
    return fvm_reset(h, p);
}

extern "C" int fvm_resize(fvm_handle *h, int nx, int ny) {
    CHECK_HANDLE(h);
    if (nx <= 0 || ny <= 0) return set_err(FVM_ERR_INVALID, "fvm_resize: nx, ny must be positive");
    if (h->Un && nx == h->g.nx && ny == h->g.ny) return FVM_OK;
    if (h->disp) {  // a registered display field is sized for the old grid
        CK(launch_set_display(h->d_disp, nullptr, 0, h->stream));
        h->disp = nullptr;
    }
    h->disp_fresh = false;
    h->prm.nx = nx;
    h->prm.ny = ny;
    if (int r = alloc_buffers(h, nx, ny)) return r;
    return build_maps(h);
}

extern "C" int fvm_set_ext(fvm_handle *h, const fvm_ext *ext) {
    CHECK_HANDLE(h);
    if (int r = validate(&h->prm, ext)) return r;
    if (!ext) return set_err(FVM_ERR_INVALID, "null ext");
    h->ext = *ext;
    drop_graphs(h);
    h->dt_ready = false;
    return FVM_OK;
}

extern "C" int fvm_update_obstacle(fvm_handle *h, const fvm_sim_params *p) {
    CHECK_INIT(h);
    if (int r = validate(p, nullptr)) return r;
    h->disp_fresh = false;
    h->prm = *p;
    if (int r = build_geometry(h, true)) return r;
    if (int r = apply_bc_full(h)) return r;
    h->cfl_valid = false;
    h->dt_ready = false;
    return FVM_OK;
}

// --------------------------------------------------------------- stepping
static StepArgs step_args(fvm_handle *h, float *out, int apply_bc, int cfl, float dt_scale) {
    StepArgs a{};
    a.g = h->g;
    a.out = out;
    a.mask = h->mask;
    a.sc = h->sc;
    a.fs = freestream(h->prm);
    a.wall = wall(h->prm);
    a.prandtl = h->ext.prandtl;
    a.ref_prandtl = (h->ext.prandtl == PRANDTL_REF) ? 1 : 0;
    a.rows_per_cta = h->tune.rows;
    a.apply_bc = apply_bc;
    a.cfl = cfl;
    a.dt_scale = dt_scale;
    a.pdl = 1;
    return a;
}

static GhostArgs ghost_args(fvm_handle *h, float *A, const float *B1, const float *B2, int cfl, int finalize) {
    GhostArgs ga{};
    ga.g = h->g;
    ga.list = h->ghosts;
    ga.n = h->n_ghost;
    ga.A = A;
    ga.B1 = B1;
    ga.B2 = B2;
    ga.sc = h->sc;
    ga.fs = freestream(h->prm);
    ga.wall = wall(h->prm);
    ga.cfl = cfl;
    ga.finalize = finalize;
    ga.recompute_dt = h->ext.dt_policy == FVM_DT_RECOMPUTE;
    ga.cfl_num = h->prm.cfl;
    ga.cfl_visc = h->prm.cfl_visc;
    ga.min_dx = fminf(h->prm.dx, h->prm.dy);
    ga.viscous = h->prm.enable_viscosity ? 1 : 0;
    return ga;
}

// A stage launch: the flat kernel on small grids, the marching one on others.
static cudaError_t stage(fvm_handle *h, int which, int in, int blend, const StepArgs &a) {
    const int sch = h->ext.flux_scheme, lim = h->ext.limiter, pairs = h->tune.flat_pairs;
    if (pairs) return launch_stage_flat(which, sch, lim, pairs, h->buf[in], h->buf[blend], a, h->stream);
    return launch_stage(which, sch, lim, h->tune, h->tm_in[in], h->tm_ctr[blend], a, h->stream);
}

// A viscous half step, with its own tile height.
static cudaError_t viscous_pass(fvm_handle *h, int in, StepArgs a) {
    if (h->tune.visc_rows) a.rows_per_cta = h->tune.visc_rows;
    return launch_viscous(h->tune, h->tm_in[in], a, h->stream);
}

// One step's launches; leaves U^{n+1} in buf[BUF_X] (the caller swaps).  to_host:
// its last pass writes the scalars to the host as well.  Only the last step of
// a call does: completing the writes across the bus holds the next step back
// (256x128: 17.4 us a step instead of 16.4 when every step did), but spares
// the host a copy (one step, its time step and back: 43 -> 34 us).
static int enqueue_step(fvm_handle *h, bool to_host) {
    cudaStream_t st = h->stream;
    float *Un = h->buf[BUF_N], *Us = h->buf[BUF_S], *Ux = h->buf[BUF_X], *Ud = h->buf[BUF_D];
    if (!h->prm.enable_viscosity) {
        // a marching pass followed by a ghost pass lets it launch early (its
        // few CTAs then wait on the device); a marching successor is not
        // launched early, its CTAs would spread unevenly over the SMs that
        // free up first
        StepArgs a1 = step_args(h, Us, 1, 0, 1.0f);
        a1.early_launch = 1;
        CK(timed(h, 0, [&] { return stage(h, 1, BUF_N, BUF_N, a1); }));
        GhostArgs g1 = ghost_args(h, Us, Un, nullptr, 0, 0);
        CK(timed(h, 4, [&] { return launch_ghost(g1, st); }));
        StepArgs a2 = step_args(h, Ux, 1, 1, 1.0f);
        a2.disp = h->disp ? h->d_disp : nullptr;
        a2.early_launch = 1;
        CK(timed(h, 1, [&] { return stage(h, 2, BUF_S, BUF_N, a2); }));
        GhostArgs g2 = ghost_args(h, Ux, Un, Us, 1, 1);
        g2.host = to_host ? h->h_now : nullptr;
        g2.disp = h->disp ? h->d_disp : nullptr;
        CK(timed(h, 5, [&] { return launch_ghost(g2, st); }));
    } else {
        StepArgs v1 = step_args(h, Ud, 0, 0, 0.5f);
        CK(timed(h, 2, [&] { return viscous_pass(h, BUF_N, v1); }));
        StepArgs a1 = step_args(h, Us, 1, 0, 1.0f);
        a1.early_launch = 1;
        CK(timed(h, 0, [&] { return stage(h, 1, BUF_D, BUF_D, a1); }));
        GhostArgs g1 = ghost_args(h, Us, Ud, nullptr, 0, 0);
        CK(timed(h, 4, [&] { return launch_ghost(g1, st); }));
        // stage 2 blends with the diffused U^n and overwrites it in place;
        // launched plainly: with programmatic serialization behind the ghost
        // pass this step ran 4 % slower at 1024x512 (the Euler stage 2 gains)
        StepArgs a2 = step_args(h, Ud, 0, 0, 1.0f);
        a2.pdl = 0;
        CK(timed(h, 1, [&] { return stage(h, 2, BUF_S, BUF_D, a2); }));
        StepArgs v2 = step_args(h, Ux, 1, 2, 0.5f);
        v2.disp = h->disp ? h->d_disp : nullptr;
        v2.early_launch = 1;
        CK(timed(h, 3, [&] { return viscous_pass(h, BUF_D, v2); }));
        GhostArgs g2 = ghost_args(h, Ux, Ud, nullptr, 2, 1);
        g2.host = to_host ? h->h_now : nullptr;
        g2.disp = h->disp ? h->d_disp : nullptr;
        CK(timed(h, 5, [&] { return launch_ghost(g2, st); }));
    }
    return FVM_OK;
}

static void swap_state(fvm_handle *h) {
    std::swap(h->buf[BUF_N], h->buf[BUF_X]);
    std::swap(h->tm_in[BUF_N], h->tm_in[BUF_X]);
    std::swap(h->tm_ctr[BUF_N], h->tm_ctr[BUF_X]);
}

// Make sc->dt hold the dt of the next step.
static int prepare_dt(fvm_handle *h, fvm_sim_params *p) {
    if (h->ext.dt_policy == FVM_DT_FIXED) {
        // the step kernels never change sc->dt under this policy: write it
        // only when the caller's dt differs from the one already there
        if (h->dt_ready && h->fixed_dt == p->dt) return FVM_OK;
        k_set_scalars<<<1, 1, 0, h->stream>>>(h->sc, p->dt, p->t_current, 0);
        CK(cudaGetLastError());
        h->launches++;
        h->fixed_dt = p->dt;
        h->dt_ready = true;
        return FVM_OK;
    }
    if (!h->dt_ready) {
        float dt = 0.0f;
        if (int r = fvm_compute_dt(h, p, &dt)) return r;
        k_set_scalars<<<1, 1, 0, h->stream>>>(h->sc, dt, p->t_current, 1);
        CK(cudaGetLastError());
        h->launches++;
        h->dt_ready = true;
    }
    return FVM_OK;
}

// What a captured step holds besides the geometry (which drops the graphs by itself).
static unsigned long long graph_key(fvm_handle *h) {
    unsigned long long k = (unsigned long long)h->prm.enable_viscosity;
    k = k * 31 + h->ext.flux_scheme;
    k = k * 31 + h->ext.limiter;
    k = k * 131 + h->tune.nt;
    k = k * 131 + h->tune.ring;
    k = k * 1031 + h->tune.rows;
    k = k * 1031 + h->tune.visc_rows;
    k = k * 11 + h->tune.flat_pairs;
    k = k * 1000003ULL + (unsigned long long)h->n_ghost;
    k = k * 7 + h->ext.dt_policy;
    k = k * 1000003ULL + (unsigned long long)(uintptr_t)h->stream;
    k = k * 3 + (h->disp != nullptr ? 1 : 0);  // display-field variants of the last passes
    uint32_t c1, c2;
    memcpy(&c1, &h->prm.cfl, 4);
    memcpy(&c2, &h->prm.cfl_visc, 4);
    k = k * 1000003ULL + c1;
    k = k * 1000003ULL + c2;
    return k;
}

// Status of a device error word.
static int error_status(unsigned err) {
    if (err & kErrTimeout) return set_err(FVM_ERR_TIMEOUT, "a bounded device wait expired (error word 0x%x)", err);
    if (err & kErrSmemAlign)
        return set_err(FVM_ERR_CUDA, "shared-memory staging area not 128-byte aligned; step skipped (error word 0x%x)",
                       err);
    return FVM_OK;
}

// The scalars on the host, once the stream is idle: as the last kernel that
// changed them wrote them, or else copied.  Either way the mirror h_sc, which
// fvm_read_dt reads, holds them too.
static int sync_scalars(fvm_handle *h) {
    if (h->now_valid) {
        CK(cudaStreamSynchronize(h->stream));
        const HostScalars &n = *h->h_now;
        DevScalars &m = *h->h_sc;
        m.cfl[0] = n.cfl[0];
        m.cfl[1] = n.cfl[1];
        m.dt_last = n.dt_last;
        m.t = n.t;
        m.err = n.err;
        return FVM_OK;
    }
    CK(cudaMemcpyAsync(h->h_sc, h->sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    const DevScalars &d = *h->h_sc;
    *h->h_now = HostScalars{{d.cfl[0], d.cfl[1]}, d.dt_last, d.t, d.err, 0u};
    return FVM_OK;
}

static int check_device_error(fvm_handle *h) {
    if (int r = sync_scalars(h)) return r;
    return error_status(h->h_now->err);
}

static int finish_steps(fvm_handle *h, fvm_sim_params *p, int n, bool to_host) {
    h->now_valid = to_host;
    if (h->ext.dt_policy == FVM_DT_FIXED) {
        for (int k = 0; k < n; k++) p->t_current += p->dt;
        p->step += n;
    } else {
        if (int r = check_device_error(h)) return r;
        p->dt = h->h_now->dt_last;
        p->t_current = h->h_now->t;
        p->step += n;
    }
    h->cfl_valid = true;
    return FVM_OK;
}

// Which ping-pong buffer holds U^n (0: the one that held it at the first
// captured step); the captured pointers depend on it.
static int state_parity(fvm_handle *h) {
    if (!h->parity_base) h->parity_base = h->buf[BUF_N];
    return (h->buf[BUF_N] == h->parity_base) ? 0 : 1;
}

// Steps after which the step graphs are captured.  Capturing and instantiating
// both parities costs 0.2 ms on the host; a step's four to six plain launches
// cost it 10-15 us, hidden behind the 16 us and more of the kernels, so a graph
// saves at most 4 us a step (NS 1024x512: 59.6 against 63.3 us; Euler steps are
// the same either way).  A solve whose geometry or parameters change every few
// steps therefore never captures; a call long enough to earn the capture back
// does at once.
constexpr int kGraphAfter = 16, kGraphLongCall = 64;

// Whether the next n steps run as graphs: the one they need exists, or enough
// steps have run (or very many are asked for) to capture it.  A stream that is
// itself being captured keeps to the graph path, which the runtime refuses there.
static bool want_graphs(fvm_handle *h, int n) {
    const unsigned long long key = graph_key(h);
    if (key != h->step_key) {
        drop_graphs(h);
        h->step_key = key;
    }
    if (h->plain_steps >= kGraphAfter || n > kGraphLongCall || h->tuning) return true;
    const int par = state_parity(h);
    if (n >= 2 ? h->graph[par] != nullptr : h->graph1[par] != nullptr) return true;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(h->stream, &cap) == cudaSuccess && cap != cudaStreamCaptureStatusNone;
}

// Captured graphs of `nsteps` steps (2 or 1) for both buffer parities, built
// together the first time either is needed, so no later call pays for a capture
// and an instantiation.  The other parity's graph is captured with the state
// pointers swapped and restored afterwards; capture launches nothing.
static int ensure_graphs(fvm_handle *h, int nsteps, cudaGraphExec_t *graphs) {
    const int cur = state_parity(h);
    for (int par = 0; par < 2; par++) {
        if (graphs[par]) continue;
        const bool other = par != cur;
        if (other) swap_state(h);
        cudaGraph_t gr;
        cudaError_t eb = cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal);
        if (eb != cudaSuccess) {
            if (other) swap_state(h);
            CK(eb);
        }
        long long before = h->launches;
        // two steps swap the state twice (also when a step fails to enqueue),
        // one step not at all: the pointers end as they began
        // (the one-step graph is always a call's last step)
        int r = enqueue_step(h, nsteps == 1);
        if (nsteps == 2) {
            swap_state(h);
            if (!r) r = enqueue_step(h, false);
            swap_state(h);
        }
        cudaError_t ec = cudaStreamEndCapture(h->stream, &gr);
        h->launches = before;
        if (other) swap_state(h);
        if (r) {
            if (ec == cudaSuccess) cudaGraphDestroy(gr);
            return r;
        }
        CK(ec);
        cudaError_t ei = cudaGraphInstantiate(&graphs[par], gr, 0);
        cudaGraphDestroy(gr);
        CK(ei);
        h->graphs_captured++;
    }
    return FVM_OK;
}

extern "C" int fvm_step(fvm_handle *h, fvm_sim_params *p) { return fvm_steps(h, p, 1); }

extern "C" int fvm_steps(fvm_handle *h, fvm_sim_params *p, int n) {
    CHECK_INIT(h);
    if (!p) return set_err(FVM_ERR_INVALID, "null params");
    if (n < 0) return set_err(FVM_ERR_INVALID, "negative step count");
    if (n == 0) return FVM_OK;
    h->disp_fresh = false;  // until every step is queued
    h->now_valid = false;
    // per-step knobs the reference reads from params on every call
    h->prm.cfl = p->cfl;
    h->prm.cfl_visc = p->cfl_visc;
    h->prm.dt = p->dt;
    if (p->enable_viscosity != h->prm.enable_viscosity || p->adiabatic_wall != h->prm.adiabatic_wall ||
        p->T_wall != h->prm.T_wall) {
        h->prm.enable_viscosity = p->enable_viscosity;
        h->prm.adiabatic_wall = p->adiabatic_wall;
        h->prm.T_wall = p->T_wall;
        drop_graphs(h);
    }
    if (int r = prepare_dt(h, p)) return r;
    const bool use_graph = !h->timing && h->stream != nullptr && h->stream != cudaStreamLegacy &&
                           h->stream != cudaStreamPerThread && getenv("FVM_NO_GRAPH") == nullptr && want_graphs(h, n);
    int done = 0;
    bool to_host = false;  // whether the last step queued writes the scalars to the host
    if (use_graph && n >= 2) {
        const int par = state_parity(h);
        if (int r = ensure_graphs(h, 2, h->graph)) return r;
        const int per_step = h->prm.enable_viscosity ? 6 : 4;
        for (; done + 2 <= n; done += 2) {
            CK(cudaGraphLaunch(h->graph[par], h->stream));
            h->graphs_launched++;
            h->launches += 2 * per_step;
        }
    }
    if (use_graph && done < n) {
        // one remaining step: a captured single step for this buffer parity
        const int par = state_parity(h);
        if (int r = ensure_graphs(h, 1, h->graph1)) return r;
        CK(cudaGraphLaunch(h->graph1[par], h->stream));
        h->graphs_launched++;
        h->launches += h->prm.enable_viscosity ? 6 : 4;
        swap_state(h);
        to_host = true;
        done++;
    }
    for (; done < n; done++) {
        to_host = done == n - 1;
        if (int r = enqueue_step(h, to_host)) return r;
        swap_state(h);
        h->plain_steps++;
    }
    const int rf = finish_steps(h, p, n, to_host);
    h->disp_fresh = rf == FVM_OK && h->disp != nullptr;
    return rf;
}

extern "C" int fvm_synchronize(fvm_handle *h) {
    CHECK_HANDLE(h);
    CK(cudaStreamSynchronize(h->stream));
    resolve_timing(h);
    // only kernels set the error word: when none was launched since
    // fvm_queue_dt copied the device scalars (the reference's per-frame
    // queue / synchronize / read sequence), that copy, complete now, holds it
    if (h->launches == h->launches_at_sc_copy) return error_status(h->h_sc->err);
    return check_device_error(h);
}

static int queue_cfl(fvm_handle *h) {
    CK(launch_cfl_state(h->g, h->Un, h->mask, h->sc, h->h_now, h->stream));
    h->launches++;
    h->cfl_valid = true;
    h->now_valid = true;
    return FVM_OK;
}

// CFL maxima of the current state: after a step they come from the fused
// reduction (mu of the last viscous half step, as the reference's d_mu_);
// otherwise from a standalone pass over the state.
static int cfl_maxima(fvm_handle *h, float *ms, float *mn) {
    if (!h->cfl_valid) {
        if (int r = queue_cfl(h)) return r;
    }
    if (int r = sync_scalars(h)) return r;
    *ms = h->h_now->cfl[0];
    *mn = h->h_now->cfl[1];
    return FVM_OK;
}

// readTimeStepResult (src/solver.cu:3250-3265)
static float dt_from_maxima(const fvm_sim_params *p, float max_speed, float max_nu) {
    float min_dx = fminf(p->dx, p->dy);
    float dt = p->cfl * min_dx / (max_speed + 1e-10f);
    if (p->enable_viscosity) {
        float dt_visc = p->cfl_visc * min_dx * min_dx / (max_nu + 1e-10f);
        dt = fminf(dt, dt_visc);
    }
    return dt;
}

extern "C" int fvm_compute_dt(fvm_handle *h, const fvm_sim_params *p, float *dt_out) {
    CHECK_INIT(h);
    if (!p || !dt_out) return set_err(FVM_ERR_INVALID, "null argument");
    float ms = 0.0f, mn = 0.0f;
    if (int r = cfl_maxima(h, &ms, &mn)) return r;
    *dt_out = dt_from_maxima(p, ms, mn);
    return FVM_OK;
}

extern "C" int fvm_queue_dt(fvm_handle *h, const fvm_sim_params *p) {
    CHECK_INIT(h);
    if (!p) return set_err(FVM_ERR_INVALID, "null params");
    if (!h->cfl_valid) {
        if (int r = queue_cfl(h)) return r;
    }
    CK(cudaMemcpyAsync(h->h_sc, h->sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, h->stream));
    h->launches_at_sc_copy = h->launches;
    return FVM_OK;
}

extern "C" int fvm_read_dt(fvm_handle *h, const fvm_sim_params *p, float *dt_out) {
    CHECK_INIT(h);
    if (!p || !dt_out) return set_err(FVM_ERR_INVALID, "null argument");
    *dt_out = dt_from_maxima(p, h->h_sc->cfl[0], h->h_sc->cfl[1]);
    return FVM_OK;
}

// --------------------------------------------------------------- readback
extern "C" int fvm_get_cell_types(fvm_handle *h, uint8_t *host_types) {
    CHECK_INIT(h);
    if (!host_types) return set_err(FVM_ERR_INVALID, "null buffer");
    CK(cudaMemcpyAsync(host_types, h->ct, (size_t)h->g.nx * h->g.ny, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return FVM_OK;
}

extern "C" int fvm_get_sdf(fvm_handle *h, float *host_sdf) {
    CHECK_INIT(h);
    if (!host_sdf) return set_err(FVM_ERR_INVALID, "null buffer");
    CK(cudaMemcpy2DAsync(host_sdf, (size_t)h->g.nx * 4, h->sdf, (size_t)h->g.pitch * 4, (size_t)h->g.nx * 4, h->g.ny,
                         cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return FVM_OK;
}

// The five planes of a state (pitched rows, `base` the first) into host arrays
// of nx*ny floats (null: skipped), queued on the stream.  A copy for each, also
// where the arrays happen to follow each other: they may be allocations of
// their own, and the runtime need not accept a copy across page-locked ones.
int fvm_internal_copy_fields(const GridDesc &g, const float *base, float *const dst[5], cudaStream_t st) {
    const size_t row = (size_t)g.nx * 4, pitch = (size_t)g.pitch * 4;
    for (int k = 0; k < 5; k++)
        if (dst[k])
            CK(cudaMemcpy2DAsync(dst[k], row, base + (size_t)k * g.plane, pitch, row, g.ny, cudaMemcpyDeviceToHost,
                                 st));
    return FVM_OK;
}

// The same into one array that holds the planes one after another, as the
// device does: one copy.
int fvm_internal_copy_state(const GridDesc &g, const float *base, float *planes, cudaStream_t st) {
    const size_t row = (size_t)g.nx * 4, pitch = (size_t)g.pitch * 4;
    if (row == pitch)
        CK(cudaMemcpyAsync(planes, base, row * g.ny * 5, cudaMemcpyDeviceToHost, st));
    else
        CK(cudaMemcpy2DAsync(planes, row, base, pitch, row, (size_t)g.ny * 5, cudaMemcpyDeviceToHost, st));
    return FVM_OK;
}

extern "C" int fvm_read_fields(fvm_handle *h, float *rho, float *rho_u, float *rho_v, float *E, float *rho_e) {
    CHECK_INIT(h);
    float *const dst[5] = {rho, rho_u, rho_v, E, rho_e};
    if (int r = fvm_internal_copy_fields(h->g, h->Un, dst, h->stream)) return r;
    CK(cudaStreamSynchronize(h->stream));
    return FVM_OK;
}

extern "C" int fvm_read_state(fvm_handle *h, float *planes) {
    CHECK_INIT(h);
    if (!planes) return set_err(FVM_ERR_INVALID, "null buffer");
    if (int r = fvm_internal_copy_state(h->g, h->Un, planes, h->stream)) return r;
    CK(cudaStreamSynchronize(h->stream));
    return FVM_OK;
}

static int check_region(const fvm_handle *h, int i0, int j0, int w, int hgt) {
    if (i0 < 0 || j0 < 0 || w <= 0 || hgt <= 0 || (long long)i0 + w > h->g.nx || (long long)j0 + hgt > h->g.ny)
        return set_err(FVM_ERR_INVALID, "region [%d, %d) x [%d, %d) outside the %d x %d grid", i0, i0 + w, j0, j0 + hgt,
                       h->g.nx, h->g.ny);
    return FVM_OK;
}

extern "C" int fvm_read_region(fvm_handle *h, int i0, int j0, int w, int hgt, float *rho, float *rho_u,
                               float *rho_v, float *E, float *rho_e) {
    CHECK_INIT(h);
    if (int r = check_region(h, i0, j0, w, hgt)) return r;
    float *dst[5] = {rho, rho_u, rho_v, E, rho_e};
    const size_t off = (size_t)j0 * h->g.pitch + i0;
    for (int k = 0; k < 5; k++) {
        if (!dst[k]) continue;
        CK(cudaMemcpy2DAsync(dst[k], (size_t)w * 4, h->Un + (size_t)k * h->g.plane + off, (size_t)h->g.pitch * 4,
                             (size_t)w * 4, hgt, cudaMemcpyDeviceToHost, h->stream));
    }
    CK(cudaStreamSynchronize(h->stream));
    return FVM_OK;
}

extern "C" int fvm_read_region_geometry(fvm_handle *h, int i0, int j0, int w, int hgt, float *sdf,
                                        uint8_t *cell_types) {
    CHECK_INIT(h);
    if (int r = check_region(h, i0, j0, w, hgt)) return r;
    if (sdf)
        CK(cudaMemcpy2DAsync(sdf, (size_t)w * 4, h->sdf + (size_t)j0 * h->g.pitch + i0, (size_t)h->g.pitch * 4,
                             (size_t)w * 4, hgt, cudaMemcpyDeviceToHost, h->stream));
    if (cell_types)
        CK(cudaMemcpy2DAsync(cell_types, (size_t)w, h->ct + (size_t)j0 * h->g.nx + i0, (size_t)h->g.nx, (size_t)w,
                             hgt, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return FVM_OK;
}

extern "C" int fvm_write_fields(fvm_handle *h, const float *rho, const float *rho_u, const float *rho_v,
                                const float *E, const float *rho_e) {
    CHECK_INIT(h);
    h->disp_fresh = false;
    const float *src[5] = {rho, rho_u, rho_v, E, rho_e};
    for (int k = 0; k < 5; k++) {
        if (!src[k]) continue;
        CK(cudaMemcpy2DAsync(h->Un + (size_t)k * h->g.plane, (size_t)h->g.pitch * 4, src[k], (size_t)h->g.nx * 4,
                             (size_t)h->g.nx * 4, h->g.ny, cudaMemcpyHostToDevice, h->stream));
    }
    CK(cudaStreamSynchronize(h->stream));
    h->cfl_valid = false;
    h->dt_ready = false;
    return FVM_OK;
}

extern "C" int fvm_read_primitives(fvm_handle *h, float *u, float *v, float *p, float *T) {
    CHECK_INIT(h);
    const size_t n = (size_t)h->g.nx * h->g.ny;
    float *d = nullptr;
    CKA(cudaMallocAsync(&d, n * 4 * sizeof(float), h->stream));
    CK(launch_primitives(h->g, h->Un, d, d + n, d + 2 * n, d + 3 * n, h->stream));
    h->launches++;
    float *dst[4] = {u, v, p, T};
    for (int k = 0; k < 4; k++)
        if (dst[k]) CK(cudaMemcpyAsync(dst[k], d + k * n, n * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaFreeAsync(d, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return FVM_OK;
}

extern "C" int fvm_field_to_device(fvm_handle *h, int kind, float *dev_dst) {
    CHECK_INIT(h);
    if (!dev_dst) return set_err(FVM_ERR_INVALID, "null destination");
    if (kind < 0 || kind > 4) return set_err(FVM_ERR_INVALID, "unknown field kind %d", kind);
    const bool into_display = h->disp && dev_dst == h->disp;
    // the registered display field, already written by the last step
    if (into_display && kind == h->disp_kind && h->disp_fresh) return FVM_OK;
    CK(launch_derived(kind, h->g, h->Un, dev_dst, h->stream));
    h->launches++;
    if (into_display) h->disp_fresh = kind == h->disp_kind;
    return FVM_OK;
}

extern "C" int fvm_set_display_field(fvm_handle *h, int kind, float *dev_dst) {
    CHECK_INIT(h);
    if (dev_dst && (kind < 0 || kind > 4)) return set_err(FVM_ERR_INVALID, "unknown field kind %d", kind);
    if (dev_dst == h->disp && (!dev_dst || kind == h->disp_kind)) return FVM_OK;
    // the descriptor is updated in stream order, before the next step reads it
    CK(launch_set_display(h->d_disp, dev_dst, dev_dst ? kind : 0, h->stream));
    h->launches++;
    h->disp = dev_dst;
    h->disp_kind = dev_dst ? kind : 0;
    h->disp_fresh = false;
    return FVM_OK;
}

extern "C" int fvm_cell_types_to_device(fvm_handle *h, float *dev_dst) {
    CHECK_INIT(h);
    if (!dev_dst) return set_err(FVM_ERR_INVALID, "null destination");
    CK(launch_ct_to_float(h->g, h->ct, dev_dst, h->stream));
    h->launches++;
    return FVM_OK;
}

extern "C" int fvm_vector_arrows(fvm_handle *h, float *dev_vertex_data, int max_vertices, int step, float u_inf,
                                 float max_arrow_length, float arrow_head_angle, float arrow_head_length,
                                 int *n_vertices_out) {
    CHECK_INIT(h);
    if (!dev_vertex_data || !n_vertices_out || step <= 0 || max_vertices < 0)
        return set_err(FVM_ERR_INVALID, "fvm_vector_arrows: bad argument");
    CK(cudaMemsetAsync(h->d_counter, 0, sizeof(int), h->stream));
    CK(launch_arrows_cap(h->g, h->Un, dev_vertex_data, max_vertices, h->d_counter, step, u_inf, max_arrow_length,
                         arrow_head_angle, arrow_head_length, h->stream));
    h->launches++;
    int n = 0;
    CK(cudaMemcpyAsync(&n, h->d_counter, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    *n_vertices_out = n;
    return FVM_OK;
}

// ------------------------------------------------------------------ stats
static int max_reduce(fvm_handle *h, int what, float *out) {
    CHECK_INIT(h);
    if (!out) return set_err(FVM_ERR_INVALID, "null output");
    float *res = reinterpret_cast<float *>(h->h_res);
    CK(launch_max_reduce(what, h->g, h->Un, h->d_tmp, res, h->stream));
    h->launches++;
    CK(cudaStreamSynchronize(h->stream));
    *out = *res;
    return FVM_OK;
}
extern "C" int fvm_max_temperature(fvm_handle *h, float *out) { return max_reduce(h, 0, out); }
extern "C" int fvm_max_mach(fvm_handle *h, float *out) { return max_reduce(h, 1, out); }

extern "C" int fvm_memory_usage(fvm_handle *h, size_t *bytes) {
    CHECK_HANDLE(h);
    if (!bytes) return set_err(FVM_ERR_INVALID, "null output");
    *bytes = h->bytes + (size_t)h->ghost_cap * sizeof(GhostInfo) + sizeof(DevScalars);
    return FVM_OK;
}

extern "C" int fvm_gpu_mem_info(size_t *free_bytes, size_t *total_bytes) {
    if (!free_bytes || !total_bytes) return set_err(FVM_ERR_INVALID, "null output");
    CK(cudaMemGetInfo(free_bytes, total_bytes));
    return FVM_OK;
}

extern "C" int fvm_diagnostics(fvm_handle *h, fvm_diag *out) {
    CHECK_INIT(h);
    if (!out) return set_err(FVM_ERR_INVALID, "null output");
    const double *r = h->h_res;
    CK(launch_diagnostics(h->g, h->Un, h->mask, h->prm.enable_viscosity ? 1 : 0, h->ext.prandtl,
                          h->ext.prandtl == PRANDTL_REF, h->d_diag, h->diag_parts,
                          reinterpret_cast<unsigned *>(h->d_tmp + 2), h->h_res, h->stream));
    h->launches++;
    CK(cudaStreamSynchronize(h->stream));
    memset(out, 0, sizeof(*out));
    out->force_x = r[0];
    out->force_y = r[1];
    const double q_inf = 0.5 * (double)h->prm.rho_inf * (double)h->prm.u_inf * (double)h->prm.u_inf;
    const double L = h->ext.ref_length > 0 ? (double)h->ext.ref_length : 2.0 * (double)h->prm.obstacle_r;
    out->cd = (q_inf > 0 && L > 0) ? r[0] / (q_inf * L) : 0.0;
    out->cl = (q_inf > 0 && L > 0) ? r[1] / (q_inf * L) : 0.0;
    out->mass = r[2];
    out->mom_x = r[3];
    out->mom_y = r[4];
    out->energy = r[5];
    out->wall_heat = r[6];
    out->wall_heat_max = r[7];
    return FVM_OK;
}

extern "C" int fvm_shock_standoff(fvm_handle *h, double *standoff_out) {
    CHECK_INIT(h);
    if (!standoff_out) return set_err(FVM_ERR_INVALID, "null output");
    const double g = 1.4, pinf = h->prm.p_inf;
    const double cinf = std::sqrt(g * pinf / (double)h->prm.rho_inf);
    const double M = (double)h->prm.u_inf / cinf;
    if (!(M > 1.0)) {
        *standoff_out = NAN;
        return FVM_OK;
    }
    const double p2 = pinf * (1.0 + 2.0 * g / (g + 1.0) * (M * M - 1.0));
    CK(launch_standoff(h->g, h->Un, h->sdf, pinf + 0.5 * (p2 - pinf), h->h_res, h->stream));
    h->launches++;
    CK(cudaStreamSynchronize(h->stream));
    *standoff_out = h->h_res[0];
    return FVM_OK;
}

// ------------------------------------------------------------ measurement
extern "C" int fvm_set_kernel_timing(fvm_handle *h, int enable) {
    CHECK_HANDLE(h);
    resolve_timing(h);
    h->timing = enable != 0;
    h->ktimes.clear();
    return FVM_OK;
}

extern "C" int fvm_kernel_times(fvm_handle *h, fvm_kernel_time *out, int cap, int *count_out) {
    CHECK_HANDLE(h);
    resolve_timing(h);
    int n = 0;
    for (auto &kv : h->ktimes) {
        if (out && n < cap) {
            memset(&out[n], 0, sizeof(out[n]));
            snprintf(out[n].name, sizeof(out[n].name), "%s", kv.first.c_str());
            out[n].launches = kv.second.first;
            out[n].total_ms = kv.second.second;
        }
        n++;
    }
    if (count_out) *count_out = n;
    return FVM_OK;
}

extern "C" int fvm_launch_count(fvm_handle *h, long long *count_out) {
    CHECK_HANDLE(h);
    if (!count_out) return set_err(FVM_ERR_INVALID, "null output");
    *count_out = h->launches;
    return FVM_OK;
}

// Time each candidate tuning over `steps` steps from a snapshot of the
// current state (restored after every candidate) and keep the fastest.  The
// steps replay graphs, as those of the solve that is tuned will; each
// candidate's are captured by its warm-up.
extern "C" int fvm_autotune(fvm_handle *h, const fvm_sim_params *p, int steps, float *best_ms_out) {
    CHECK_INIT(h);
    if (!p || steps < 2) return set_err(FVM_ERR_INVALID, "fvm_autotune: need params and steps >= 2");
    const size_t bytes = (size_t)h->g.plane * 5 * sizeof(float);
    float *snap = nullptr;
    CKA(cudaMalloc(&snap, bytes));
    CK(cudaMemcpyAsync(snap, h->buf[BUF_N], bytes, cudaMemcpyDeviceToDevice, h->stream));
    const StageTune before = h->tune;
    const bool timing = h->timing;
    h->timing = false;
    h->tuning = true;
    fvm_sim_params q = *p;
    StageTune best = before;
    float best_ms = 1e30f;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int rc = FVM_OK;
    // tile heights between the powers of two let the tuner fill the last
    // wave of CTAs (e.g. 8192x4096: 64-row tiles are 4.83 waves on 148 SMs)
    constexpr int kRows = 13;
    const int nts[2] = {128, 256}, rings[2] = {4, 6},
              rows[kRows] = {4, 8, 16, 24, 32, 40, 48, 56, 64, 80, 96, 128, 256};
    // the default shape (with the flat stage kernel on small grids), then the
    // marching shapes
    std::vector<StageTune> cands{heuristic_tune(h->g.nx, h->g.ny)};
    for (int a1 = 0; a1 < 2; a1++)
        for (int a2 = 0; a2 < 2; a2++)
            for (int a3 = 0; a3 < kRows; a3++)
                if (rows[a3] <= std::max(16, h->g.ny)) cands.push_back(StageTune{nts[a1], rings[a2], rows[a3]});
    for (const StageTune &cand : cands) {
        h->tune = cand;
        drop_graphs(h);
        if ((rc = build_maps(h)) != FVM_OK) break;
        fvm_sim_params w = q;
        if ((rc = fvm_steps(h, &w, 3)) != FVM_OK) break;  // warm: one graph of each kind
        cudaEventRecord(e0, h->stream);
        if ((rc = fvm_steps(h, &w, steps)) != FVM_OK) break;
        cudaEventRecord(e1, h->stream);
        cudaEventSynchronize(e1);
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        ms /= steps;
        if (ms < best_ms) {
            best_ms = ms;
            best = cand;
        }
        // restore the state for the next candidate (buffer roles may have swapped)
        cudaMemcpyAsync(h->buf[BUF_N], snap, bytes, cudaMemcpyDeviceToDevice, h->stream);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    h->tune = (rc == FVM_OK) ? best : before;
    drop_graphs(h);
    int r2 = build_maps(h);
    cudaMemcpyAsync(h->buf[BUF_N], snap, bytes, cudaMemcpyDeviceToDevice, h->stream);
    cudaStreamSynchronize(h->stream);
    cudaFree(snap);
    h->timing = timing;
    h->tuning = false;
    h->cfl_valid = false;
    h->dt_ready = false;
    h->disp_fresh = false;  // the tuning steps wrote it; the state is restored
    if (rc != FVM_OK) return rc;
    if (r2 != FVM_OK) return r2;
    g_tune_cache[TuneKey{h->g.nx, h->g.ny, h->prm.enable_viscosity ? 1 : 0, h->ext.flux_scheme, h->ext.limiter}] =
        best;
    if (best_ms_out) *best_ms_out = best_ms;
    return FVM_OK;
}

extern "C" int fvm_set_tune(fvm_handle *h, int nt, int ring, int rows) {
    CHECK_INIT(h);
    if (!(nt == 128 || nt == 256) || !(ring == 4 || ring == 6) || rows < 4 || rows > 65536 || (rows & 1))
        return set_err(FVM_ERR_INVALID,
                       "fvm_set_tune: threads 128 or 256, ring 4 or 6, even rows 4..65536 (got %d, %d, %d)", nt, ring,
                       rows);
    h->tune = StageTune{nt, ring, rows};
    drop_graphs(h);
    return build_maps(h);
}

extern "C" int fvm_nonfinite_count(fvm_handle *h, unsigned long long *count, int reset) {
    CHECK_INIT(h);
    unsigned v = 0;
    CK(cudaMemcpyAsync(&v, &h->sc->nonfinite, sizeof(unsigned), cudaMemcpyDeviceToHost, h->stream));
    if (reset) CK(cudaMemsetAsync(&h->sc->nonfinite, 0, sizeof(unsigned), h->stream));
    CK(cudaStreamSynchronize(h->stream));
    if (count) *count = v;
    return FVM_OK;
}

extern "C" int fvm_get_tune(fvm_handle *h, int *nt, int *ring, int *rows) {
    CHECK_INIT(h);
    if (nt) *nt = h->tune.nt;
    if (ring) *ring = h->tune.ring;
    if (rows) *rows = h->tune.rows;
    return FVM_OK;
}

extern "C" int fvm_debug_stage1(fvm_handle *h, float dt, int with_ghost, float *rho, float *rho_u, float *rho_v,
                                float *E, float *rho_e) {
    CHECK_INIT(h);
    k_set_scalars<<<1, 1, 0, h->stream>>>(h->sc, dt, 0.0f, 0);
    h->launches_at_sc_copy = -1;
    h->now_valid = false;
    CK(cudaGetLastError());
    float *Un = h->buf[BUF_N], *Us = h->buf[BUF_S];
    StepArgs a1 = step_args(h, Us, 1, 0, 1.0f);
    CK(stage(h, 1, BUF_N, BUF_N, a1));
    if (with_ghost && h->n_ghost > 0) {
        GhostArgs g1 = ghost_args(h, Us, Un, nullptr, 0, 0);
        CK(launch_ghost(g1, h->stream));
    }
    float *dst[5] = {rho, rho_u, rho_v, E, rho_e};
    for (int k = 0; k < 5; k++)
        if (dst[k])
            CK(cudaMemcpy2DAsync(dst[k], (size_t)h->g.nx * 4, Us + (size_t)k * h->g.plane, (size_t)h->g.pitch * 4,
                                 (size_t)h->g.nx * 4, h->g.ny, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->dt_ready = false;
    return check_device_error(h);
}

int fvm_internal_build_maps(fvm_handle *h) { return build_maps(h); }
int fvm_internal_compute_dt(fvm_handle *h, const fvm_sim_params *p, float *dt) { return fvm_compute_dt(h, p, dt); }
int fvm_internal_set_error(int code, const char *msg) { return set_err(code, "%s", msg); }

extern "C" int fvm_debug_wait_timeout(fvm_handle *h, long long limit_cycles) {
    CHECK_INIT(h);
    if (limit_cycles <= 0 || limit_cycles > kWaitCycles)
        return set_err(FVM_ERR_INVALID, "fvm_debug_wait_timeout: limit must be in 1..%lld cycles", kWaitCycles);
    CK(cudaStreamSynchronize(h->stream));
    h->now_valid = false;
    CK(launch_wait_probe(h->sc, limit_cycles, h->stream));
    const int r = check_device_error(h);
    // clear the error word the probe set, so the solve goes on
    unsigned zero = 0;
    CK(cudaMemcpyAsync(&h->sc->err, &zero, sizeof(unsigned), cudaMemcpyHostToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->launches_at_sc_copy = -1;
    return r;
}

extern "C" int fvm_debug_ghost_table(fvm_handle *h, int *out, int cap, int *count_out) {
    CHECK_INIT(h);
    static_assert(sizeof(GhostInfo) == 6 * sizeof(int), "GhostInfo layout");
    if (count_out) *count_out = h->n_ghost;
    int n = std::min(cap, h->n_ghost);
    if (out && n > 0) {
        std::vector<GhostInfo> t((size_t)n);
        CK(cudaMemcpy(t.data(), h->ghosts, (size_t)n * sizeof(GhostInfo), cudaMemcpyDeviceToHost));
        for (int k = 0; k < n; k++) {
            int *o = out + (size_t)k * 7;
            o[0] = (int)((long long)t[k].j * h->g.pitch + t[k].i);
            memcpy(o + 1, &t[k], sizeof(GhostInfo));
        }
    }
    return FVM_OK;
}

extern "C" int fvm_debug_graph_count(fvm_handle *h, long long *captured_out, long long *launched_out) {
    CHECK_HANDLE(h);
    if (captured_out) *captured_out = h->graphs_captured;
    if (launched_out) *launched_out = h->graphs_launched;
    return FVM_OK;
}

extern "C" const char *fvm_build_info(void) {
    return "fvm_b200: sm_100a, nvcc " FVM_STR(__CUDACC_VER_MAJOR__) "." FVM_STR(__CUDACC_VER_MINOR__)
           ", --use_fast_math, marching TMA and flat stage kernels";
}
