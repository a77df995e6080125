// fvm_aux.cu -- off-step kernels behind the reference's readback / statistics
// API: derived fields into device buffers, max-temperature / max-Mach
// reductions, velocity arrows, FP64 diagnostics and the shock standoff scan.
#include <cstdint>

#include "fvm_colortable.h"
#include "fvm_kernels.cuh"
#include "fvm_quads.cuh"
#include "fvm_tma.cuh"

namespace fvm {

__global__ void k_primitives(GridDesc g, const float *U, float *u, float *v, float *p, float *T) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.nx || j >= g.ny) return;
    size_t c = (size_t)j * g.pitch + i, d = (size_t)j * g.nx + i;
    float uu, vv, pp, TT;
    prim_from_cons(U[c], U[g.plane + c], U[2 * g.plane + c], U[3 * g.plane + c], U[4 * g.plane + c], uu, vv, pp, TT);
    if (u) u[d] = uu;
    if (v) v[d] = vv;
    if (p) p[d] = pp;
    if (T) T[d] = TT;
}

// The four cells a thread of a whole-field pass handles.  GROUP: a group of
// four neighbours of a row, for destinations whose groups are 16-byte aligned.
// Otherwise cells 32 apart in the dense order, so that a warp's loads and
// stores are each 32 consecutive cells whatever the row length: four 4-byte
// (16-byte) stores of neighbours per thread would leave each store of the warp
// a quarter (half) of its sectors.
template <bool GROUP>
struct Cells4 {
    size_t c[4], d[4];  // pitched and dense index
    int n;              // cells inside the grid
    __device__ __forceinline__ Cells4(const GridDesc &g, unsigned e) {
        if (GROUP) {
            const Quad q = quad_at(g, e);
            n = q.n;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                c[k] = q.c + k;
                d[k] = q.d + k;
            }
        } else {
            const unsigned total = (unsigned)g.nx * (unsigned)g.ny, first = (e & ~31u) * 4u + (e & 31u);
            unsigned j = first / (unsigned)g.nx, i = first - j * (unsigned)g.nx;
            n = 0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const unsigned at = first + 32u * k;
                n += at < total && at >= first ? 1 : 0;
                c[k] = (size_t)j * g.pitch + i;
                d[k] = at;
                for (i += 32u; i >= (unsigned)g.nx; i -= (unsigned)g.nx) j++;
            }
        }
    }
    // threads that cover a grid
    __host__ __device__ static unsigned threads(const GridDesc &g) {
        return GROUP ? quads(g) : ((unsigned)g.nx * (unsigned)g.ny + 127u) / 128u * 32u;
    }
};

// A derived field's inputs (derived_value): only the planes the kind reads, the
// others zero.
template <int KIND, bool GROUP>
struct DerivedIn {
    float rho[4], ru[4], rv[4], re[4];
    __device__ __forceinline__ static void plane(float *dst, bool used, const float *p, const Cells4<GROUP> &q) {
        if (GROUP) {
            const float4 v = used ? __ldg(reinterpret_cast<const float4 *>(p + q.c[0])) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            dst[0] = v.x;
            dst[1] = v.y;
            dst[2] = v.z;
            dst[3] = v.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++) dst[k] = used && k < q.n ? __ldg(p + q.c[k]) : 0.0f;
        }
    }
    __device__ __forceinline__ DerivedIn(const GridDesc &g, const float *U, const Cells4<GROUP> &q) {
        plane(rho, KIND != 1, U, q);
        plane(ru, KIND >= 3, U + g.plane, q);
        plane(rv, KIND >= 3, U + 2 * g.plane, q);
        plane(re, KIND != 2 && KIND != 3, U + 4 * g.plane, q);
    }
    __device__ __forceinline__ float value(int k) const { return derived_value(KIND, rho[k], ru[k], rv[k], re[k]); }
};

// Derived field into a dense nx*ny destination: 8 (density, pressure) to 20
// (Mach) bytes per cell, DRAM-bound.  One launch per kind, so that only the
// planes the kind needs are read.  Measured at 8192x4096, all four planes read
// a cell at a time -> this: density and pressure 135 -> 39 us, temperature
// 135 -> 53, speed 135 -> 72, Mach 135 -> 92 (7.3 TB/s); at 4999x2501
// density 53 -> 18, Mach 55 -> 41.
template <int KIND, bool GROUP>
__global__ void __launch_bounds__(256) k_derived(GridDesc g, const float *__restrict__ U, float *__restrict__ dst) {
    const unsigned e = blockIdx.x * 256u + threadIdx.x;
    if (e >= Cells4<GROUP>::threads(g)) return;
    const Cells4<GROUP> q(g, e);
    const DerivedIn<KIND, GROUP> in(g, U, q);
    if (GROUP) {
        *reinterpret_cast<float4 *>(dst + q.d[0]) = make_float4(in.value(0), in.value(1), in.value(2), in.value(3));
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (k < q.n) dst[q.d[k]] = in.value(k);
    }
}

// (1 - w) a + w b, rounded the same way in every kernel variant (an image's
// bytes must not depend on it).
__device__ __forceinline__ float lerp_texel(float w, float a, float b) {
    return __fmaf_rn(w, b, __fmul_rn(1.0f - w, a));
}

// the tables in the order of enum fvm_colormap
__device__ const ColormapLUT kColorTables[5] = {colormap_lut(0), colormap_lut(1), colormap_lut(2), colormap_lut(3),
                                                colormap_lut(4)};

// The renderer's field pass (FIELD_FRAGMENT_SHADER, src/renderer.cpp:47-77)
// with one pixel per cell: SOLID and GHOST cells dark grey, others the
// derived value normalised by (v - lo) / (hi - lo + 1e-4), clamped to [0, 1],
// then looked up in the 256-entry colour table the way a linearly filtered,
// edge-clamped 1-D texture samples it.  FMT 0: RGBA float, 1: RGBA8.
// The table sits in shared memory as pairs of neighbouring entries, so a
// lookup is two vector loads; indexed in the kernel's parameters (constant
// memory), lanes with different entries were served one after the other.
// Mach -> RGBA8 at 8192x4096: 214 us indexed in constant memory, 112 us here
// (21 B per cell, 6.3-6.5 TB/s); Mach -> RGBA float at 5000x2500 94 -> 71.
template <int KIND, int FMT, bool GROUP>
__global__ void __launch_bounds__(256) k_colormap(GridDesc g, const float *__restrict__ U,
                                                  const uint8_t *__restrict__ mask, int colormap, float lo,
                                                  float hi, void *__restrict__ out) {
    static_assert(!GROUP || FMT == 1, "groups of four only for 4-byte pixels");
    // entry i: {r_i, g_i, b_i, r_i+1}, {g_i+1, b_i+1, -, -}
    __shared__ float4 ta[256];
    __shared__ float2 tb[256];
    {
        const int i = threadIdx.x, n = min(i + 1, 255);
        const float *rgb = kColorTables[colormap].rgb;
        ta[i] = make_float4(rgb[3 * i], rgb[3 * i + 1], rgb[3 * i + 2], rgb[3 * n]);
        tb[i] = make_float2(rgb[3 * n + 1], rgb[3 * n + 2]);
    }
    __syncthreads();
    const unsigned total = Cells4<GROUP>::threads(g);
    for (unsigned e = blockIdx.x * 256u + threadIdx.x; e < total; e += gridDim.x * 256u) {
        const Cells4<GROUP> q(g, e);
        const DerivedIn<KIND, GROUP> in(g, U, q);
        uint32_t m4 = 0u;  // mask bytes of the four cells
        if (GROUP) {
            m4 = __ldg(reinterpret_cast<const uint32_t *>(mask + q.c[0]));
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (k < q.n) m4 |= (uint32_t)__ldg(mask + q.c[k]) << (8 * k);
        }
        float4 px[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float r, gr, b;
            if ((m4 >> (8 * k)) & MB_WALL) {
                r = gr = b = 0.3f;
            } else {
                // the value rounded before lo comes off: fused with its last
                // product in some variants, bytes depended on the variant
                const float s = fminf(fmaxf(__fsub_rn(in.value(k), lo) / (hi - lo + 0.0001f), 0.0f), 1.0f);
                const float u = s * 256.0f - 0.5f;
                const float fl = floorf(u);
                const float w = u - fl;
                // the texel pair (fl, fl + 1) clamped to the edge: below the
                // first texel both are entry 0
                const int i0 = min(max((int)fl, 0), 255);
                const float4 A = ta[i0];
                const float2 B = tb[i0];
                const bool first = (int)fl < 0;
                r = lerp_texel(w, A.x, first ? A.x : A.w);
                gr = lerp_texel(w, A.y, first ? A.y : B.x);
                b = lerp_texel(w, A.z, first ? A.z : B.y);
            }
            px[k] = make_float4(r, gr, b, 1.0f);
        }
        if (FMT == 0) {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (k < q.n) reinterpret_cast<float4 *>(out)[q.d[k]] = px[k];
        } else {
            auto quant = [](float x) { return (unsigned)__float2int_rn(fminf(fmaxf(x, 0.0f), 1.0f) * 255.0f); };
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; k++)
                w[k] = quant(px[k].x) | (quant(px[k].y) << 8) | (quant(px[k].z) << 16) | (255u << 24);
            uint32_t *const o = reinterpret_cast<uint32_t *>(out);
            if (GROUP) {
                *reinterpret_cast<uint4 *>(o + q.d[0]) = make_uint4(w[0], w[1], w[2], w[3]);
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (k < q.n) o[q.d[k]] = w[k];
            }
        }
    }
}

// cellTypeToFloatKernel (src/solver.cu:3444-3450); both arrays are dense, four
// cells per thread: side by side where the destination is 16-byte aligned
// (VEC), else 256 apart, so that a warp's scalar stores are consecutive.
template <bool VEC>
__global__ void __launch_bounds__(256) k_ct_to_float(long long n, const uint8_t *__restrict__ ct,
                                                     float *__restrict__ dst) {
    if (VEC) {
        const long long e = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
        if (e + 4 <= n) {
            const uchar4 c = *reinterpret_cast<const uchar4 *>(ct + e);
            *reinterpret_cast<float4 *>(dst + e) = make_float4(static_cast<float>(c.x), static_cast<float>(c.y),
                                                               static_cast<float>(c.z), static_cast<float>(c.w));
            return;
        }
        for (long long k = e; k < n; k++) dst[k] = static_cast<float>(ct[k]);
    } else {
        const long long e = (long long)blockIdx.x * 1024 + threadIdx.x;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (e + 256 * k < n) dst[e + 256 * k] = static_cast<float>(ct[e + 256 * k]);
    }
}

// WHAT = 0: max temperature of the primitives (getMaxTemperature,
// src/solver.cu:2835-2867); WHAT = 1: max local Mach (computeMachNumberKernel,
// src/solver.cu:2782-2794).  The last block writes the maximum to `out` in
// pinned host memory and leaves the scratch {maximum, counter} zero for the
// next call: no memset before and no copy after.  2048x1024: 12.4 us one cell
// at a time, 10.0 us here.
template <int WHAT>
__global__ void __launch_bounds__(256, 6) k_max_reduce(GridDesc g, const float *__restrict__ U, float *scratch,
                                                    float *out) {
    float m = 0.0f;
    const unsigned total = quads(g);
    for (unsigned e = blockIdx.x * 256u + threadIdx.x; e < total; e += gridDim.x * 256u) {
        const Quad q = quad_at(g, e);
        const float4 R = load4(U, q), RU = load4(U + g.plane, q), RV = load4(U + 2 * g.plane, q),
                     E = load4(U + 3 * g.plane, q), RE = load4(U + 4 * g.plane, q);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float u, v, p, T;
            const float rho = lane4(R, k);
            prim_from_cons(rho, lane4(RU, k), lane4(RV, k), lane4(E, k), lane4(RE, k), u, v, p, T);
            float x;
            if (WHAT == 0) {
                x = T;
            } else {
                float rho_val = rho + 1e-10f;
                float speed = sqrtf(u * u + v * v);
                float cs = sqrtf(GAMMA * p / rho_val);
                x = speed / (cs + 1e-10f);
            }
            if (k < q.n) m = fmaxf(m, x);
        }
    }
    __shared__ float ws[8];
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float mm = 0.0f;
        for (int k = 0; k < 8; k++) mm = fmaxf(mm, ws[k]);
        atomic_max_nonneg(scratch, mm);
    }
    if (last_block(reinterpret_cast<unsigned *>(scratch + 1)) && threadIdx.x == 0) {
        *out = __uint_as_float(atomicExch(reinterpret_cast<unsigned *>(scratch), 0u));
        __threadfence_system();
    }
}

// generateVectorArrowsKernel (src/solver.cu:3689-3796).  Slots come from an
// atomic counter like the reference; writes past `cap_vertices` are skipped
// (the reference does not check), the counter still reports the total.
__global__ void k_arrows(GridDesc g, const float *U, float *vertexData, int *counter, int cap_vertices, int step,
                         float u_inf, float maxArrowLength, float arrowHeadAngle, float arrowHeadLength) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int j = blockIdx.y * blockDim.y + threadIdx.y;
    i = i * step + step / 2;
    j = j * step + step / 2;
    if (i >= g.nx || j >= g.ny) return;
    size_t c = (size_t)j * g.pitch + i;
    float u_val, v_val, pp, TT;
    prim_from_cons(U[c], U[g.plane + c], U[2 * g.plane + c], U[3 * g.plane + c], U[4 * g.plane + c], u_val, v_val,
                   pp, TT);
    float speed = sqrtf(u_val * u_val + v_val * v_val);
    if (speed < 1e-6f * u_inf) return;
    float normalizedSpeed = fminf(speed / (u_inf * 1.5f), 1.0f);
    float startX = (float)i / g.nx * 2.0f - 1.0f;
    float startY = (float)j / g.ny * 2.0f - 1.0f;
    float dirX = u_val / speed;
    float dirY = v_val / speed;
    float arrowLength = maxArrowLength * normalizedSpeed;
    float endX = startX + dirX * arrowLength;
    float endY = startY + dirY * arrowLength;
    float headLen = arrowLength * arrowHeadLength;
    float cosA = cosf(arrowHeadAngle);
    float sinA = sinf(arrowHeadAngle);
    float head1X = endX - headLen * (dirX * cosA - dirY * sinA);
    float head1Y = endY - headLen * (dirX * sinA + dirY * cosA);
    float head2X = endX - headLen * (dirX * cosA + dirY * sinA);
    float head2Y = endY - headLen * (-dirX * sinA + dirY * cosA);
    int vertexOffset = atomicAdd(counter, 8);
    if (vertexOffset + 8 > cap_vertices) return;
    float *o = vertexData + (size_t)vertexOffset * 5;
    const float xs[6] = {startX, endX, endX, head1X, endX, head2X};
    const float ys[6] = {startY, endY, endY, head1Y, endY, head2Y};
    for (int k = 0; k < 6; k++) {
        o[k * 5 + 0] = xs[k];
        o[k * 5 + 1] = ys[k];
        o[k * 5 + 2] = 0.0f;
        o[k * 5 + 3] = 0.0f;
        o[k * 5 + 4] = 0.0f;
    }
}

// ---------------------------------------------------------------- diagnostics
// FP64 wall forces, heat flux and conserved totals (no reference counterpart).
// Wall faces lie between a wall cell (solid/ghost) and a non-wall cell; the
// force on the obstacle is (-p_face n + tau.n) dA, n the unit normal from the
// wall cell to the fluid cell, p_face the pressure of the left/bottom cell
// (the reference's wall-face flux, src/solver.cu:1594,1679), tau and q at the
// fluid cell.  Deterministic: the sums' order depends on the grid alone.
constexpr int kDiag = 8;  // fx, fy, mass, mx, my, E, heat, heat_max

struct DiagCtx {
    GridDesc g;
    const float *U;
    const uint8_t *mask;
    ViscArgs va;
};

__device__ __forceinline__ void prim_at(const DiagCtx &d, int i, int j, float &u, float &v, float &p, float &T) {
    size_t c = (size_t)j * d.g.pitch + i;
    const long long pl = d.g.plane;
    prim_from_cons(d.U[c], d.U[pl + c], d.U[2 * pl + c], d.U[3 * pl + c], d.U[4 * pl + c], u, v, p, T);
}

__device__ void stress_at(const DiagCtx &d, int i, int j, float out[5]) {
    const int nx = d.g.nx, ny = d.g.ny;
    float uC, vC, pC, TC, uE, vE, pE, TE, uW, vW, pW, TW, uN, vN, pN, TN, uS, vS, pS, TS;
    prim_at(d, i, j, uC, vC, pC, TC);
    prim_at(d, min(i + 1, nx - 1), j, uE, vE, pE, TE);
    prim_at(d, max(i - 1, 0), j, uW, vW, pW, TW);
    prim_at(d, i, min(j + 1, ny - 1), uN, vN, pN, TN);
    prim_at(d, i, max(j - 1, 0), uS, vS, pS, TS);
    stress_heat(uC, vC, TC, uE, uW, uN, uS, vE, vW, vN, vS, TE, TW, TN, TS, i == 0, i == nx - 1, j == 0, j == ny - 1,
                d.va, out);
}

// The wall face between cell (i, j) and its right (dir 0) or upper (dir 1)
// neighbour; wa: (i, j) is the wall.
__device__ __forceinline__ void diag_face(const DiagCtx &d, int i, int j, int dir, bool wa, int viscous,
                                          double acc[kDiag]) {
    const double sgn = wa ? 1.0 : -1.0;
    const int fi = wa ? (dir == 0 ? i + 1 : i) : i;
    const int fj = wa ? (dir == 0 ? j : j + 1) : j;
    const double dA = dir == 0 ? (double)d.g.dy : (double)d.g.dx;
    const double nxn = dir == 0 ? sgn : 0.0, nyn = dir == 1 ? sgn : 0.0;
    float u, v, p, T;
    prim_at(d, i, j, u, v, p, T);
    double fx = -(double)p * nxn * dA, fy = -(double)p * nyn * dA;
    if (viscous) {
        float t5[5];
        stress_at(d, fi, fj, t5);
        fx += ((double)t5[0] * nxn + (double)t5[2] * nyn) * dA;
        fy += ((double)t5[2] * nxn + (double)t5[1] * nyn) * dA;
        const double qw = -((double)t5[3] * nxn + (double)t5[4] * nyn);
        acc[6] += qw * dA;
        acc[7] = fmax(acc[7], qw);
    }
    acc[0] += fx;
    acc[1] += fy;
}

__device__ __forceinline__ double diag_combine(int k, double a, double b) { return k == 7 ? fmax(a, b) : a + b; }

// Per-block partials, then the last block to finish sums them in a fixed
// order (one warp per quantity, lane l the partials l, l+32, ..., then a
// shuffle tree), so the result does not depend on which block that is; it
// goes straight to pinned host memory.  Reads 16 B of state and 1 B of mask
// per cell: the loads of a group of four cells are issued together and the
// walls are found four cells at a time on the mask words.  A wall face costs
// some 30 scattered loads; each warp lists its faces in shared memory (in the
// order of its cells) and works them off 32 at a time, one per lane, instead
// of one lane after another for the faces its own cells have.  2048x1024:
// 18 us; one cell per thread with a second kernel in which one thread summed
// the partials took 36 + 160 us, faces in their cells' lanes 33 us.
constexpr int kFaceList = 32 + 256;  // less than a round left over, plus all faces of 32 groups
__global__ void __launch_bounds__(256, 4) k_diagnostics(DiagCtx d, int viscous, double *partials, unsigned *counter,
                                                     double *out) {
    __shared__ unsigned long long faces[8][kFaceList];  // group index * 8 + face of the group: k (x-faces), 4 + k (y-faces)
    double acc[kDiag];
#pragma unroll
    for (int k = 0; k < kDiag; k++) acc[k] = 0.0;
    const GridDesc g = d.g;
    const unsigned total = quads(g);
    constexpr uint32_t W4 = MB_WALL * 0x01010101u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned long long *list = faces[warp];
    int listed = 0;
    // one listed face per lane
    auto work = [&](int at, bool mine) {
        __syncwarp();
        if (mine) {
            const unsigned long long code = list[at];
            const Quad q = quad_at(g, (unsigned)(code >> 3));
            const int i = q.i + (int)(code & 3u), dir = (int)(code >> 2) & 1;
            diag_face(d, i, q.j, dir, (d.mask[(size_t)q.j * g.pitch + i] & MB_WALL) != 0, viscous, acc);
        }
        __syncwarp();
    };
    for (unsigned e0 = blockIdx.x * 256u + 32u * warp; e0 < total; e0 += gridDim.x * 256u) {
        const unsigned e = e0 + lane;
        uint32_t bits = 0u;
        if (e < total) {
            const Quad q = quad_at(g, e);
            const uint8_t *mrow = d.mask + q.c;
            const float4 R = load4(d.U, q), RU = load4(d.U + g.plane, q), RV = load4(d.U + 2 * g.plane, q),
                         E = load4(d.U + 3 * g.plane, q);
            const bool top = q.j >= g.ny - 1, right = q.i + 4 >= g.nx;
            const uint32_t m = __ldg(reinterpret_cast<const uint32_t *>(mrow)) & W4;
            const uint32_t up = __ldg(reinterpret_cast<const uint32_t *>(top ? mrow : mrow + g.pitch)) & W4;
            const uint32_t next = right ? 0u : (uint32_t)__ldg(mrow + 4) & MB_WALL;
            // cells of the group inside the grid; a last column has no right neighbour
            const uint32_t in = W4 >> (8 * (4 - q.n));
            const uint32_t inx = right ? in >> 8 : in;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if ((in & ~m) >> (8 * k) & MB_WALL) {
                    acc[2] += (double)lane4(R, k);
                    acc[3] += (double)lane4(RU, k);
                    acc[4] += (double)lane4(RV, k);
                    acc[5] += (double)lane4(E, k);
                }
            }
            const uint32_t fx = (m ^ ((m >> 8) | (next << 24))) & inx, fy = (m ^ up) & in;
#pragma unroll
            for (int k = 0; k < 4; k++)
                bits |= ((fx >> (8 * k)) & 1u) << k | ((fy >> (8 * k)) & 1u) << (4 + k);
        }
        if (__any_sync(0xffffffffu, bits != 0u)) {
            int before = __popc(bits);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before += y;
            }
            const int added = __shfl_sync(0xffffffffu, before, 31);
            int at = listed + before - __popc(bits);
            for (uint32_t b = bits; b; b &= b - 1u) list[at++] = (unsigned long long)e * 8u + (unsigned)(__ffs(b) - 1);
            for (listed += added; listed >= 32; listed -= 32) work(listed - 32 + lane, true);
            __syncwarp();
        }
    }
    work(lane, lane < listed);
    const double area = (double)g.dx * (double)g.dy;
#pragma unroll
    for (int k = 2; k < 6; k++) acc[k] *= area;
    __shared__ double s[8][kDiag];
#pragma unroll
    for (int k = 0; k < kDiag; k++) {
        double x = acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x = diag_combine(k, x, __shfl_xor_sync(0xffffffffu, x, o));
        if (lane == 0) s[warp][k] = x;
    }
    __syncthreads();
    if (threadIdx.x < kDiag) {
        double x = s[0][threadIdx.x];
        for (int w = 1; w < 8; w++) x = diag_combine(threadIdx.x, x, s[w][threadIdx.x]);
        partials[(size_t)blockIdx.x * kDiag + threadIdx.x] = x;
    }
    if (!last_block(counter)) return;
    static_assert(kDiag == 8, "one warp per quantity");
    double x = 0.0;
    for (unsigned b = lane; b < gridDim.x; b += 32)
        x = diag_combine(warp, x, __ldcg(&partials[(size_t)b * kDiag + warp]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = diag_combine(warp, x, __shfl_xor_sync(0xffffffffu, x, o));
    if (lane == 0) {
        out[warp] = x;
        __threadfence_system();
    }
}

// Smallest index found by the block's threads (INT_MAX: none).
__device__ __forceinline__ int block_min_index(int x) {
    __shared__ int first;
    if (threadIdx.x == 0) first = 0x7fffffff;
    __syncthreads();
    x = __reduce_min_sync(0xffffffffu, x);
    if ((threadIdx.x & 31) == 0 && x != 0x7fffffff) atomicMin(&first, x);
    __syncthreads();
    const int r = first;
    __syncthreads();
    return r;
}

// Shock standoff along row ny/2 (see fvm_b200.h): the first downward zero of
// the distance field, then the first upward crossing of p_mid before it.  One
// block looks at 1024 cells at a time and stops at the first hit (one thread
// scanning the row paid a load's latency per cell: 80 us at 2048x1024, 5 us
// here).  The result goes to pinned host memory.
__global__ void __launch_bounds__(1024) k_standoff(GridDesc g, const float *U, const float *sdf, double p_mid,
                                                   double *out) {
    const size_t row = (size_t)(g.ny / 2) * g.pitch;
    const double dxd = g.dx;
    int ib = 0x7fffffff;
    for (int i0 = 0; i0 + 1 < g.nx && ib == 0x7fffffff; i0 += 1024) {
        const int i = i0 + (int)threadIdx.x;
        const bool hit = i + 1 < g.nx && sdf[row + i] > 0.0f && sdf[row + i + 1] <= 0.0f;
        ib = block_min_index(hit ? i : 0x7fffffff);
    }
    int is = 0x7fffffff;
    if (ib != 0x7fffffff) {
        auto pressure = [&](int i) {
            const size_t c = row + i;
            float u, v, p, T;
            prim_from_cons(U[c], U[g.plane + c], U[2 * g.plane + c], U[3 * g.plane + c], U[4 * g.plane + c], u, v, p, T);
            return (double)p;
        };
        for (int i0 = 1; i0 <= ib && is == 0x7fffffff; i0 += 1024) {
            const int i = i0 + (int)threadIdx.x;
            const bool hit = i <= ib && pressure(i - 1) < p_mid && pressure(i) >= p_mid;
            is = block_min_index(hit ? i : 0x7fffffff);
        }
        if (threadIdx.x == 0 && is != 0x7fffffff) {
            const double a = sdf[row + ib], b = sdf[row + ib + 1];
            const double xb = (ib + 0.5) * dxd + dxd * a / (a - b);
            const double p0 = pressure(is - 1), p1 = pressure(is);
            const double xs = (is - 1 + 0.5) * dxd + dxd * (p_mid - p0) / (p1 - p0);
            *out = xb - xs;
        }
    }
    if (threadIdx.x == 0) {
        if (is == 0x7fffffff) *out = __longlong_as_double(0x7ff8000000000000ULL);
        __threadfence_system();
    }
}

// ------------------------------------------------------------- launchers
static dim3 grid2d(const GridDesc &g, dim3 b) { return dim3((g.nx + b.x - 1) / b.x, (g.ny + b.y - 1) / b.y); }

cudaError_t launch_primitives(const GridDesc &g, const float *U, float *u, float *v, float *p, float *T,
                              cudaStream_t st) {
    dim3 b(32, 8);
    k_primitives<<<grid2d(g, b), b, 0, st>>>(g, U, u, v, p, T);
    return cudaGetLastError();
}

// whether every group of four cells of a dense nx*ny array of `elem`-byte
// cells starts on a 16-byte boundary when four cells are 16 bytes
static bool dense_aligned(const GridDesc &g, const void *p) {
    return (g.nx & 3) == 0 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
}

template <bool GROUP>
static unsigned cell_blocks(const GridDesc &g) {
    return (Cells4<GROUP>::threads(g) + 255u) / 256u;
}

template <int KIND>
static void colormap_k(const GridDesc &g, const float *U, const uint8_t *mask, int colormap, float lo,
                       float hi, void *out, int fmt, cudaStream_t st) {
    // enough blocks to fill the chip several times over, each filling its table once
    constexpr unsigned kCap = 148 * 32;
    if (fmt == 0)
        k_colormap<KIND, 0, false><<<std::min(kCap, cell_blocks<false>(g)), 256, 0, st>>>(g, U, mask, colormap, lo, hi, out);
    else if (dense_aligned(g, out))
        k_colormap<KIND, 1, true><<<std::min(kCap, cell_blocks<true>(g)), 256, 0, st>>>(g, U, mask, colormap, lo, hi, out);
    else
        k_colormap<KIND, 1, false><<<std::min(kCap, cell_blocks<false>(g)), 256, 0, st>>>(g, U, mask, colormap, lo, hi, out);
}

cudaError_t launch_colormap(int kind, const GridDesc &g, const float *U, const uint8_t *mask, int colormap,
                            float lo, float hi, void *out, int fmt, cudaStream_t st) {
    switch (kind) {
    case 0: colormap_k<0>(g, U, mask, colormap, lo, hi, out, fmt, st); break;
    case 1: colormap_k<1>(g, U, mask, colormap, lo, hi, out, fmt, st); break;
    case 2: colormap_k<2>(g, U, mask, colormap, lo, hi, out, fmt, st); break;
    case 3: colormap_k<3>(g, U, mask, colormap, lo, hi, out, fmt, st); break;
    default: colormap_k<4>(g, U, mask, colormap, lo, hi, out, fmt, st); break;
    }
    return cudaGetLastError();
}

template <int KIND>
static void derived_k(const GridDesc &g, const float *U, float *dst, cudaStream_t st) {
    if (dense_aligned(g, dst))
        k_derived<KIND, true><<<cell_blocks<true>(g), 256, 0, st>>>(g, U, dst);
    else
        k_derived<KIND, false><<<cell_blocks<false>(g), 256, 0, st>>>(g, U, dst);
}

cudaError_t launch_derived(int kind, const GridDesc &g, const float *U, float *dst, cudaStream_t st) {
    switch (kind) {
    case 0: derived_k<0>(g, U, dst, st); break;
    case 1: derived_k<1>(g, U, dst, st); break;
    case 2: derived_k<2>(g, U, dst, st); break;
    case 3: derived_k<3>(g, U, dst, st); break;
    default: derived_k<4>(g, U, dst, st); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_ct_to_float(const GridDesc &g, const uint8_t *ct, float *dst, cudaStream_t st) {
    const long long n = (long long)g.nx * g.ny;
    const unsigned nb = (unsigned)((n + 1023) / 1024);
    if ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0)
        k_ct_to_float<true><<<nb, 256, 0, st>>>(n, ct, dst);
    else
        k_ct_to_float<false><<<nb, 256, 0, st>>>(n, ct, dst);
    return cudaGetLastError();
}

cudaError_t launch_max_reduce(int what, const GridDesc &g, const float *U, float *scratch, float *out_host,
                              cudaStream_t st) {
    const unsigned nb = quad_blocks(g, 148 * 6);  // one resident wave
    if (what == 0)
        k_max_reduce<0><<<nb, 256, 0, st>>>(g, U, scratch, out_host);
    else
        k_max_reduce<1><<<nb, 256, 0, st>>>(g, U, scratch, out_host);
    return cudaGetLastError();
}

cudaError_t launch_arrows_cap(const GridDesc &g, const float *U, float *vertex, int cap, int *counter, int step,
                              float u_inf, float max_len, float head_angle, float head_len, cudaStream_t st) {
    int ax = (g.nx + step - 1) / step, ay = (g.ny + step - 1) / step;
    dim3 b(16, 16), gr((ax + 15) / 16, (ay + 15) / 16);
    k_arrows<<<gr, b, 0, st>>>(g, U, vertex, counter, cap, step, u_inf, max_len, head_angle, head_len);
    return cudaGetLastError();
}

int diagnostics_parts(const GridDesc &g) { return (int)quad_blocks(g, 592); }

cudaError_t launch_diagnostics(const GridDesc &g, const float *U, const uint8_t *mask, int viscous, float prandtl,
                               int ref_prandtl, double *partials, int nparts, unsigned *counter, double *out_host,
                               cudaStream_t st) {
    DiagCtx d;
    d.g = g;
    d.U = U;
    d.mask = mask;
    d.va = viscous_args(g.dx, g.dy, prandtl, ref_prandtl != 0);
    k_diagnostics<<<nparts, 256, 0, st>>>(d, viscous, partials, counter, out_host);
    return cudaGetLastError();
}

cudaError_t launch_standoff(const GridDesc &g, const float *U, const float *sdf, double p_mid, double *out_host,
                            cudaStream_t st) {
    k_standoff<<<1, 1024, 0, st>>>(g, U, sdf, p_mid, out_host);
    return cudaGetLastError();
}

}  // namespace fvm
