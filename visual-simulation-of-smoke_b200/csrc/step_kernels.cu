// Step kernels of the B200 smoke library (everything except the pressure solve, which is in pcg.cu).
//
// Reference behaviour: backend-cuda.cu:840-1609 and the step order of :2000-2057. Design differences:
//  - every face kernel produces the SETTLED face value in one pass: the reference's update kernel, its three
//    enforce_*_boundaries passes and its periodic sync become one read-only-input kernel writing a separate
//    output buffer (no in-place races, no D2D copies). A non-periodic domain face copies the settled value of
//    its interior neighbour for OUTFLOW (backend-cuda.cu:1023-1024), a face touching a solid cell takes the
//    mean solid velocity (:1036-1063), and face n of a periodic axis equals face 0 (:1170-1189);
//  - the three face axes run in one launch (block ranges per axis);
//  - temperature and density share one back-trace per cell;
//  - the density fill of solid cells is a precomputed (cell, nearest fluid cell) list built when occupancy
//    changes, instead of a per-step Chebyshev-shell search (:1243-1290).
#include <cmath>

#include "launch.h"
#include "pdl.cuh"

namespace smoke_b200 {

namespace {

constexpr int kThreads = 256;

inline unsigned blocks_for(uint64_t count, int threads = kThreads) { return static_cast<unsigned>((count + threads - 1) / threads); }
// SMs of the current device (1 where it cannot be read: the launch then reports why).
inline unsigned sm_count() {
    int dev = 0, sms = 1;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 1u;
    return static_cast<unsigned>(sms);
}

// The step's elementwise kernels call f(q, x, y, z), q linear, for one cell per thread, kThreads consecutive ones per block, or
// (COLUMN) for `planes` cells of a column (x, y): block blockIdx.x takes kThreads consecutive cells of a plane, blockIdx.y a run
// of planes (see column_planes). The form is the kernel's template argument: one kernel that chose between them by `planes`
// carried the column's loop into the one-cell form (84^3: face force 14.6 -> 15.4 us, projection 9.6 -> 11.2).
template <bool COLUMN, class F>
__device__ __forceinline__ void for_column(const StepParams& P, int planes, F&& f) {
    uint32_t q = blockIdx.x * kThreads + threadIdx.x;
    if constexpr (COLUMN) {
        const uint32_t slab = static_cast<uint32_t>(P.nx) * P.ny;
        if (q >= slab) return;
        const int y = static_cast<int>(P.div_nx.div(q)), x = static_cast<int>(q - static_cast<uint32_t>(y) * P.nx);
        int z = blockIdx.y * planes;
        const int z1 = imin(z + planes, P.nz);
        q += static_cast<uint32_t>(z) * slab;
#pragma unroll 1
        for (; z < z1; ++z, q += slab) f(q, x, y, z);
    } else {
        if (q >= P.n) return;
        int x, y, z;
        cell_xyz(P, q, x, y, z);
        f(q, x, y, z);
    }
}
// The same over the faces of axis A, with the block's index b along the plane.
template <int A, bool COLUMN, class F>
__device__ __forceinline__ void for_face_column(const StepParams& P, unsigned b, int planes, F&& f) {
    uint32_t q = b * kThreads + threadIdx.x;
    if constexpr (COLUMN) {
        const uint32_t sx = fsx<A>(P), slab = sx * fsy<A>(P);
        if (q >= slab) return;
        const int j = static_cast<int>(P.div_fx[A].div(q)), i = static_cast<int>(q - static_cast<uint32_t>(j) * sx);
        int k = blockIdx.y * planes;
        const int k1 = imin(k + planes, fsz<A>(P));
        q += static_cast<uint32_t>(k) * slab;
#pragma unroll 1
        for (; k < k1; ++k, q += slab) f(q, i, j, k);
    } else {
        if (q >= (A == 0 ? P.nu : (A == 1 ? P.nv : P.nw))) return;
        int i, j, k;
        face_ijk<A>(P, q, i, j, k);
        f(q, i, j, k);
    }
}

// Flow-resolved cell lookup: wraps periodic axes, false when outside a non-periodic domain (:146-151).
__device__ __forceinline__ bool resolve_flow(const StepParams& P, int& x, int& y, int& z) {
    if (P.fper[0]) x = wrapi(x, P.nx);
    if (P.fper[1]) y = wrapi(y, P.ny);
    if (P.fper[2]) z = wrapi(z, P.nz);
    return x >= 0 && x < P.nx && y >= 0 && y < P.ny && z >= 0 && z < P.nz;
}

// Mean solid velocity of the solid cells on either side of face (i,j,k) of axis A, if any (:1036-1063).
template <int A>
__device__ __forceinline__ bool solid_face(const StepParams& P, int i, int j, int k, const uint8_t* __restrict__ occ, const float* __restrict__ solid, float& out) {
    int l[3] = {i, j, k};
    int r[3] = {i, j, k};
    l[A] -= 1;
    const bool hl = resolve_flow(P, l[0], l[1], l[2]);
    const bool hr = resolve_flow(P, r[0], r[1], r[2]);
    const uint32_t li = hl ? cidx(P, l[0], l[1], l[2]) : 0u;
    const uint32_t ri = hr ? cidx(P, r[0], r[1], r[2]) : 0u;
    const bool ol = hl && occ[li] != 0;
    const bool orr = hr && occ[ri] != 0;
    if (!ol && !orr) return false;
    float value = 0.0f, weight = 0.0f;
    if (ol) {
        value += solid[li];
        weight += 1.0f;
    }
    if (orr) {
        value += solid[ri];
        weight += 1.0f;
    }
    out = value / weight;
    return true;
}

// Settled value of face (i,j,k) of axis A: domain-face rule, periodic duplicate, solid rule, else the
// stage's own interior value `inner(i,j,k)`.
// An OUTFLOW domain face copies its interior neighbour. In the reference that copy and the neighbour's solid rule
// run in the same enforce kernel and the copy reads first (observed on B200, :1023-1024 vs :1036-1063), so after
// the force and advection stages the copy does NOT see the neighbour's solid rule. The projection kernel applies
// the solid rule itself before its enforce pass (:1465-1475), so there the copy does see it: OUTFLOW_SEES_SOLID.
template <int A, bool OUTFLOW_SEES_SOLID, class Inner>
__device__ __forceinline__ float settle(const StepParams& P, int i, int j, int k, const uint8_t* __restrict__ occ, const float* __restrict__ solid, Inner&& inner) {
    int c[3] = {i, j, k};
    const int n = axis_n(P, A);
    const SmokeSimulationFlowBoundaryFaceDesc lo = P.flow[2 * A], hi = P.flow[2 * A + 1];
    bool outflow_copy = false;
    if (!P.fper[A]) {
        if (c[A] == 0) {
            if (!(lo.type == kFlowOutflow && n > 0)) return face_comp(lo, A);
            c[A] = 1;
            outflow_copy = true;
        } else if (c[A] == n) {
            if (hi.type != kFlowOutflow) return face_comp(hi, A);
            c[A] = n - 1;
            outflow_copy = true;
        }
    } else if (c[A] == n) {
        c[A] = 0;
    }
    // an index that is itself a domain face (possible only when n == 1) takes no solid rule
    const bool domain_index = !P.fper[A] && (c[A] == 0 || c[A] == n);
    float v;
    if ((OUTFLOW_SEES_SOLID || !outflow_copy) && !domain_index && solid_face<A>(P, c[0], c[1], c[2], occ, solid, v)) return v;
    return inner(c[0], c[1], c[2]);
}

template <int A>
__device__ __forceinline__ const float* pick(const float* a, const float* b, const float* c) {
    return A == 0 ? a : (A == 1 ? b : c);
}
template <int A>
__device__ __forceinline__ float* pick(float* a, float* b, float* c) {
    return A == 0 ? a : (A == 1 ? b : c);
}

// Index of element (i, j, k) of a field of kind KIND (0-2 faces, 3-4 cells) in its padded copy (see PadField).
template <int KIND>
__device__ __forceinline__ uint32_t pad_index(const StepParams& P, int i, int j, int k) {
    const uint32_t px = P.nx + (KIND == 0) + 2 * kPad, py = P.ny + (KIND == 1) + 2 * kPad;
    return (static_cast<uint32_t>(k + kPad) * py + static_cast<uint32_t>(j + kPad)) * px + static_cast<uint32_t>(i + kPad);
}

// ------------------------------------------------------------------------------------------ forces
__global__ void __launch_bounds__(kThreads) vorticity_kernel(const __grid_constant__ StepParams P, const float* __restrict__ u, const float* __restrict__ v, const float* __restrict__ w, const uint8_t* __restrict__ occ, float* __restrict__ wx, float* __restrict__ wy, float* __restrict__ wz, float* __restrict__ wm) {
    pdl_begin();
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= P.n) return;
    int x, y, z;
    cell_xyz(P, q, x, y, z);
    const bool solid = occ[q] != 0;
    const float4 o = vorticity_at(u, v, w, x, y, z, P);  // also for solid cells: no load waits on occupancy
    wx[q] = solid ? 0.0f : o.x;
    wy[q] = solid ? 0.0f : o.y;
    wz[q] = solid ? 0.0f : o.z;
    wm[q] = solid ? 0.0f : o.w;
}

// |w| lookup with clamp (or wrap on periodic axes), no occupancy test (load_flow_cell, :202-226).
__device__ __forceinline__ float flow_cell(const float* __restrict__ f, int x, int y, int z, const StepParams& P) {
    if (x < 0 || x >= P.nx) x = P.fper[0] ? wrapi(x, P.nx) : (x < 0 ? 0 : P.nx - 1);
    if (y < 0 || y >= P.ny) y = P.fper[1] ? wrapi(y, P.ny) : (y < 0 ? 0 : P.ny - 1);
    if (z < 0 || z >= P.nz) z = P.fper[2] ? wrapi(z, P.nz) : (z < 0 ? 0 : P.nz - 1);
    return __ldg(f + cidx(P, x, y, z));
}

// f = user force; fluid cells add buoyancy (:910-918) and confinement eps*h*(N x w) (:920-948).
__global__ void __launch_bounds__(kThreads) cell_force_kernel(const __grid_constant__ StepParams P, const float* __restrict__ wx, const float* __restrict__ wy, const float* __restrict__ wz, const float* __restrict__ wm, const float* __restrict__ density, const float* __restrict__ temperature, const float* __restrict__ ufx,
                                                               const float* __restrict__ ufy, const float* __restrict__ ufz, const uint8_t* __restrict__ occ, float* __restrict__ fx, float* __restrict__ fy, float* __restrict__ fz,
                                                               const __grid_constant__ ScalarSources S) {
    pdl_begin();
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= P.n) return;
    // The scalar stage's sourced fields and their padded copies: t_tmp = T' + dt * src_T, T' being T with solid cells at
    // the solid temperature (the step-start apply_solid_temperature of :2001 folded in); d_tmp = rho + dt * src_rho
    // (add_source, :852-857). T and rho do not change between this stage and the scalar advection.
    if (S.t_tmp) {
        const float tv = occ[q] != 0 ? S.solid_t[q] : temperature[q];
        const float tt = tv + P.dt * S.ts[q], dd = density[q] + P.dt * S.ds[q];
        S.t_tmp[q] = tt;
        S.d_tmp[q] = dd;
        if (S.t_pad) {
            int x, y, z;
            cell_xyz(P, q, x, y, z);
            S.t_pad[pad_index<4>(P, x, y, z)] = tt;
            S.d_pad[pad_index<3>(P, x, y, z)] = dd;
        }
    }
    float ax = ufx[q], ay = ufy[q], az = ufz[q];
    if (occ[q] == 0) {
        int x, y, z;
        cell_xyz(P, q, x, y, z);
        ay += -P.alpha * density[q] + P.beta * (temperature[q] - P.ambient);
        const float h = P.h, hh = 0.5f * P.inv_h;
        float gx, gy, gz;
        if (x > 0 && x < P.nx - 1 && y > 0 && y < P.ny - 1 && z > 0 && z < P.nz - 1) {  // all six neighbours in range
            const uint32_t sy = P.nx, sz = static_cast<uint32_t>(P.nx) * P.ny;
            gx = hh * (__ldg(wm + q + 1) - __ldg(wm + q - 1));
            gy = hh * (__ldg(wm + q + sy) - __ldg(wm + q - sy));
            gz = hh * (__ldg(wm + q + sz) - __ldg(wm + q - sz));
        } else {
            gx = hh * (flow_cell(wm, x + 1, y, z, P) - flow_cell(wm, x - 1, y, z, P));
            gy = hh * (flow_cell(wm, x, y + 1, z, P) - flow_cell(wm, x, y - 1, z, P));
            gz = hh * (flow_cell(wm, x, y, z + 1, P) - flow_cell(wm, x, y, z - 1, P));
        }
        const float gmag = sqrtf(gx * gx + gy * gy + gz * gz);
        if (!(gmag < 1.0e-6f)) {
            const float inv = 1.0f / gmag;
            const float nxv = gx * inv, nyv = gy * inv, nzv = gz * inv;
            const float ox = wx[q], oy = wy[q], oz = wz[q];
            ax += P.epsilon * h * (nyv * oz - nzv * oy);
            ay += P.epsilon * h * (nzv * ox - nxv * oz);
            az += P.epsilon * h * (nxv * oy - nyv * ox);
        }
    }
    fx[q] = ax;
    fy[q] = ay;
    fz[q] = az;
}

template <int A>
__device__ __forceinline__ void face_force_one(const StepParams& P, uint32_t q, int i, int j, int k, const float* __restrict__ in, const float* __restrict__ f, const uint8_t* __restrict__ occ, const float* __restrict__ solid, float* __restrict__ out, float* __restrict__ pad) {
    // the settled value, also into the interior of the padded copy that the velocity advection reads
    auto put = [&](float v) {
        out[q] = v;
        if (pad) pad[pad_index<A>(P, i, j, k)] = v;
    };
    const int n = axis_n(P, A);
    const int s = A == 0 ? i : (A == 1 ? j : k);
    if (s > 0 && s < n) {
        // interior face: all loads first, then the rules (same values as the general path below)
        const uint32_t ri = cidx(P, i, j, k), li = ri - (A == 0 ? 1u : (A == 1 ? static_cast<uint32_t>(P.nx) : static_cast<uint32_t>(P.nx) * P.ny));
        const uint8_t ol = occ[li], orr = occ[ri];
        const float base = in[q], fl = f[li], fr = f[ri];
        if (ol != 0 || orr != 0) {
            float value = 0.0f, weight = 0.0f;
            if (ol != 0) {
                value += solid[li];
                weight += 1.0f;
            }
            if (orr != 0) {
                value += solid[ri];
                weight += 1.0f;
            }
            put(value / weight);
        } else {
            put(base + P.dt * (0.5f * (0.0f + fl + fr)));
        }
        return;
    }
    put(settle<A, false>(P, i, j, k, occ, solid, [&](int a, int b, int c) {
        const int s = A == 0 ? a : (A == 1 ? b : c);
        float sum = 0.0f, weight = 0.0f;
        int lc[3] = {a, b, c};
        if (s > 0) {
            lc[A] = s - 1;
            sum += f[cidx(P, lc[0], lc[1], lc[2])];
            weight += 1.0f;
        }
        if (s < n) {
            lc[A] = s;
            sum += f[cidx(P, lc[0], lc[1], lc[2])];
            weight += 1.0f;
        }
        const float base = in[fidx<A>(P, a, b, c)];
        return weight > 0.0f ? base + P.dt * (weight > 1.0f ? 0.5f * sum : sum) : base;  // exact halving
    }));
}

// Block ranges: [0, bu) -> x faces, [bu, bu+bv) -> y faces, rest -> z faces.
template <bool COLUMN>
__global__ void __launch_bounds__(kThreads) face_force_kernel(const __grid_constant__ StepParams P, const float* __restrict__ iu, const float* __restrict__ iv, const float* __restrict__ iw, const float* __restrict__ fx, const float* __restrict__ fy, const float* __restrict__ fz, const uint8_t* __restrict__ occ, const float* __restrict__ su,
                                                               const float* __restrict__ sv, const float* __restrict__ sw, float* __restrict__ ou, float* __restrict__ ov, float* __restrict__ ow, float* __restrict__ pu, float* __restrict__ pv, float* __restrict__ pw, unsigned bu, unsigned bv, int planes) {
    pdl_begin();
    const unsigned b = blockIdx.x;
    if (b < bu) {
        for_face_column<0, COLUMN>(P, b, planes, [&](uint32_t q, int i, int j, int k) { face_force_one<0>(P, q, i, j, k, iu, fx, occ, su, ou, pu); });
    } else if (b < bu + bv) {
        for_face_column<1, COLUMN>(P, b - bu, planes, [&](uint32_t q, int i, int j, int k) { face_force_one<1>(P, q, i, j, k, iv, fy, occ, sv, ov, pv); });
    } else {
        for_face_column<2, COLUMN>(P, b - bu - bv, planes, [&](uint32_t q, int i, int j, int k) { face_force_one<2>(P, q, i, j, k, iw, fz, occ, sw, ow, pw); });
    }
}

// ------------------------------------------------------------------------------------------ velocity advection
// Point (i, j, k) of this thread in block b of an nx x ny x nz grid of points covered by boxes of P.tile; false
// outside the grid. Boxes run x fastest, then y, then z.
__device__ __forceinline__ bool tile_point(const StepParams& P, unsigned b, int nx, int ny, int nz, int& i, int& j, int& k) {
    const int lx = P.tile[0], ly = P.tile[1], lz = P.tile[2];
    const unsigned ntx = (nx + (1 << lx) - 1) >> lx, nty = (ny + (1 << ly) - 1) >> ly;
    const unsigned r = b / ntx, bx = b - r * ntx, bz = r / nty, by = r - bz * nty;
    const unsigned t = threadIdx.x;
    i = static_cast<int>((bx << lx) + (t & ((1u << lx) - 1u)));
    j = static_cast<int>((by << ly) + ((t >> lx) & ((1u << ly) - 1u)));
    k = static_cast<int>((bz << lz) + (t >> (lx + ly)));
    return i < nx && j < ny && k < nz;
}
// Blocks of kThreads that cover an nx x ny x nz grid of points in the advection shape of P.
unsigned advect_blocks(const StepParams& P, int nx, int ny, int nz) {
    if (P.tile[0] < 0) return blocks_for(static_cast<uint64_t>(nx) * ny * nz);
    const uint64_t tx = 1u << P.tile[0], ty = 1u << P.tile[1], tz = 1u << P.tile[2];
    return static_cast<unsigned>(((nx + tx - 1) / tx) * ((ny + ty - 1) / ty) * ((nz + tz - 1) / tz));
}

template <int A, bool CUBIC, bool TILED, bool POW2>
__device__ __forceinline__ void advect_face_one(const StepParams& P, unsigned blk, const PadField& u, const PadField& v, const PadField& w, const uint8_t* __restrict__ occ, const float* __restrict__ solid, float* __restrict__ out) {
    int i, j, k;
    uint32_t q;
    if (TILED) {
        if (!tile_point(P, blk, fsx<A>(P), fsy<A>(P), fsz<A>(P), i, j, k)) return;
        q = fidx<A>(P, i, j, k);
    } else {
        q = blk * kThreads + threadIdx.x;
        if (q >= (A == 0 ? P.nu : (A == 1 ? P.nv : P.nw))) return;
        face_ijk<A>(P, q, i, j, k);
    }
    const PadField& src = A == 0 ? u : (A == 1 ? v : w);
    out[q] = settle<A, false>(P, i, j, k, occ, solid, [&](int a, int b, int c) {
        const float h = P.h;
        const float px = A == 0 ? static_cast<float>(a) * h : (static_cast<float>(a) + 0.5f) * h;
        const float py = A == 1 ? static_cast<float>(b) * h : (static_cast<float>(b) + 0.5f) * h;
        const float pz = A == 2 ? static_cast<float>(c) * h : (static_cast<float>(c) + 0.5f) * h;
        const float3 p = trace_rk2<POW2, A>(px, py, pz, a, b, c, u, v, w, occ, P);
        return sample_pad<A, CUBIC, POW2>(src, p.x, p.y, p.z, P);
    });
}

// Samples and traces read the padded copies of the velocity (ghost cells hold the boundary taps). Blocks
// [0, bu) advect u faces, [bu, bu + bv) v faces, the rest w faces, each in the shape P.tile selects. POW2: the cell
// size is a power of two, so grid coordinates are products instead of divisions (over_h, the same floats).
// Six blocks per SM (at most 42 registers): the gathers wait on L1/L2 latency, and the extra resident warps hide more
// of it than the few spilled registers cost (240 -> 224 us at 128^3 against the compiler's 64 registers, 4 blocks).
template <bool CUBIC, bool TILED, bool POW2>
__global__ void __launch_bounds__(kThreads, 6) advect_velocity_kernel(const __grid_constant__ StepParams P, const PadField u, const PadField v, const PadField w, const uint8_t* __restrict__ occ, const float* __restrict__ su, const float* __restrict__ sv, const float* __restrict__ sw, float* __restrict__ ou, float* __restrict__ ov,
                                                                    float* __restrict__ ow, unsigned bu, unsigned bv) {
    pdl_begin();
    const unsigned b = blockIdx.x;
    if (b < bu) advect_face_one<0, CUBIC, TILED, POW2>(P, b, u, v, w, occ, su, ou);
    else if (b < bu + bv) advect_face_one<1, CUBIC, TILED, POW2>(P, b - bu, u, v, w, occ, sv, ov);
    else advect_face_one<2, CUBIC, TILED, POW2>(P, b - bu - bv, u, v, w, occ, sw, ow);
}

// Padded copies (see PadField) of up to 3 fields in one launch: block z-range c * pz_blocks .. for field c; each
// thread fills kPadPlanes cells of one column (loads first, then stores), 32 x 8 columns per block.
constexpr int kPadPlanes = 4;
struct PadJob {
    const float* f[3];
    float* out[3];
    int kind[3];
    int count;
    int pz_blocks;  // blocks per field along z (kPadPlanes planes each)
};

template <int KIND>
__device__ __forceinline__ float pad_value(const StepParams& P, const float* __restrict__ f, int i, int j, int k) {
    const int fx = P.nx + (KIND == 0), fy = P.ny + (KIND == 1), fz = P.nz + (KIND == 2);
    if (i >= 0 && i < fx && j >= 0 && j < fy && k >= 0 && k < fz) return __ldg(f + (static_cast<uint32_t>(k) * fy + j) * fx + i);
    return boundary_tap<KIND>(f, i, j, k, P);
}

__global__ void __launch_bounds__(256) pad_kernel(const __grid_constant__ StepParams P, const __grid_constant__ PadJob J) {
    const int c = blockIdx.z / J.pz_blocks, kp0 = (blockIdx.z - c * J.pz_blocks) * kPadPlanes;
    if (c >= J.count) return;
    const int kind = c == 0 ? J.kind[0] : (c == 1 ? J.kind[1] : J.kind[2]);
    const int px = P.nx + (kind == 0) + 2 * kPad, py = P.ny + (kind == 1) + 2 * kPad, pz = P.nz + (kind == 2) + 2 * kPad;
    const int ip = blockIdx.x * 32 + threadIdx.x, jp = blockIdx.y * 8 + threadIdx.y;
    if (ip >= px || jp >= py || kp0 >= pz) return;
    const int i = ip - kPad, j = jp - kPad;
    const float* f = c == 0 ? J.f[0] : (c == 1 ? J.f[1] : J.f[2]);
    float* out = c == 0 ? J.out[0] : (c == 1 ? J.out[1] : J.out[2]);
    float v[kPadPlanes];
#pragma unroll
    for (int u = 0; u < kPadPlanes; ++u) {
        const int k = kp0 + u - kPad;
        switch (kind) {
        case 0: v[u] = pad_value<0>(P, f, i, j, k); break;
        case 1: v[u] = pad_value<1>(P, f, i, j, k); break;
        case 2: v[u] = pad_value<2>(P, f, i, j, k); break;
        case 3: v[u] = pad_value<3>(P, f, i, j, k); break;
        default: v[u] = pad_value<4>(P, f, i, j, k); break;
        }
    }
#pragma unroll
    for (int u = 0; u < kPadPlanes; ++u)
        if (kp0 + u < pz) out[(static_cast<uint32_t>(kp0 + u) * py + jp) * px + ip] = v[u];
}

// Ghost cells only, for padded copies whose interior the producing kernel wrote: thread g of field c (blockIdx.y)
// takes ghost cell g of the shell, enumerated as the 2 kPad whole z-planes, then in each interior plane the 2 kPad
// y-rows, then in each interior row the 2 kPad x-cells; its value is the boundary tap, as in pad_kernel.
__global__ void __launch_bounds__(256) pad_ghost_kernel(const __grid_constant__ StepParams P, const __grid_constant__ PadJob J) {
    pdl_begin();
    const int c = blockIdx.y;
    if (c >= J.count) return;
    const int kind = c == 0 ? J.kind[0] : (c == 1 ? J.kind[1] : J.kind[2]);
    const uint32_t fx = P.nx + (kind == 0), fy = P.ny + (kind == 1), fz = P.nz + (kind == 2);
    const uint32_t px = fx + 2 * kPad, py = fy + 2 * kPad;
    const uint32_t na = 2u * kPad * px * py, nb = fz * 2u * kPad * px, nc = fz * fy * 2u * kPad;
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= na + nb + nc) return;
    uint32_t ip, jp, kp;
    if (g < na) {  // whole ghost z-planes
        const uint32_t plane = g / (px * py), r = g - plane * px * py;
        kp = plane < static_cast<uint32_t>(kPad) ? plane : fz + plane;
        jp = r / px;
        ip = r - jp * px;
    } else if (g < na + nb) {  // ghost y-rows of the interior planes
        const uint32_t h = g - na, per = 2u * kPad * px, plane = h / per, r = h - plane * per, row = r / px;
        kp = kPad + plane;
        jp = row < static_cast<uint32_t>(kPad) ? row : fy + row;
        ip = r - row * px;
    } else {  // ghost x-cells of the interior rows
        const uint32_t h = g - na - nb, per = fy * 2u * kPad, plane = h / per, r = h - plane * per, row = r / (2u * kPad), xi = r - row * (2u * kPad);
        kp = kPad + plane;
        jp = kPad + row;
        ip = xi < static_cast<uint32_t>(kPad) ? xi : fx + xi;
    }
    const int i = static_cast<int>(ip) - kPad, j = static_cast<int>(jp) - kPad, k = static_cast<int>(kp) - kPad;
    const float* f = c == 0 ? J.f[0] : (c == 1 ? J.f[1] : J.f[2]);
    float* out = c == 0 ? J.out[0] : (c == 1 ? J.out[1] : J.out[2]);
    float v;
    switch (kind) {
    case 0: v = pad_value<0>(P, f, i, j, k); break;
    case 1: v = pad_value<1>(P, f, i, j, k); break;
    case 2: v = pad_value<2>(P, f, i, j, k); break;
    case 3: v = pad_value<3>(P, f, i, j, k); break;
    default: v = pad_value<4>(P, f, i, j, k); break;
    }
    out[(kp * py + jp) * px + ip] = v;
}

// ------------------------------------------------------------------------------------------ pressure rhs
// b = -(h^2/dt) div u* + sum of OUTFLOW face pressures; 0 at solid cells and at the anchor (:1304-1328).
template <bool COLUMN>
__global__ void __launch_bounds__(kThreads) rhs_kernel(const __grid_constant__ StepParams P, const float* __restrict__ u, const float* __restrict__ v, const float* __restrict__ w, const uint8_t* __restrict__ occ, const int32_t* __restrict__ anchor, float* __restrict__ rhs, int planes) {
    pdl_begin();
    for_column<COLUMN>(P, planes, [&](uint32_t q, int x, int y, int z) {
        // every load is issued before the anchor/solid test (the six faces of a cell always exist)
        const bool zero = static_cast<int32_t>(q) == __ldg(anchor) || occ[q] != 0;
        const float h = P.h;
        const float div = (u[fidx<0>(P, x + 1, y, z)] - u[fidx<0>(P, x, y, z)] + v[fidx<1>(P, x, y + 1, z)] - v[fidx<1>(P, x, y, z)] + w[fidx<2>(P, x, y, z + 1)] - w[fidx<2>(P, x, y, z)]) * P.inv_h;
        if (zero) {
            rhs[q] = 0.0f;
            return;
        }
        float bsum = 0.0f;
        if (x == 0 && P.flow[0].type == kFlowOutflow) bsum += P.flow[0].pressure;
        if (x == P.nx - 1 && P.flow[1].type == kFlowOutflow) bsum += P.flow[1].pressure;
        if (y == 0 && P.flow[2].type == kFlowOutflow) bsum += P.flow[2].pressure;
        if (y == P.ny - 1 && P.flow[3].type == kFlowOutflow) bsum += P.flow[3].pressure;
        if (z == 0 && P.flow[4].type == kFlowOutflow) bsum += P.flow[4].pressure;
        if (z == P.nz - 1 && P.flow[5].type == kFlowOutflow) bsum += P.flow[5].pressure;
        rhs[q] = -(h * h / P.dt) * div + bsum;
    });
}

// ------------------------------------------------------------------------------------------ projection
template <int A>
__device__ __forceinline__ void project_one(const StepParams& P, uint32_t q, int i, int j, int k, const float* __restrict__ in, const float* __restrict__ p, const double* __restrict__ p64, const uint8_t* __restrict__ occ, const float* __restrict__ solid, float* __restrict__ out, float* __restrict__ pad) {
    // the projected value, also into the interior of the padded copy that the scalar advection reads
    auto put = [&](float v) {
        out[q] = v;
        if (pad) pad[pad_index<A>(P, i, j, k)] = v;
    };
    const int s = A == 0 ? i : (A == 1 ? j : k);
    if (s > 0 && s < axis_n(P, A)) {
        // interior face: both cells exist unwrapped, so every load is issued before any rule is decided; the
        // values are those of the general path below (solid rule, else the gradient step)
        const uint32_t ri = cidx(P, i, j, k), li = ri - (A == 0 ? 1u : (A == 1 ? static_cast<uint32_t>(P.nx) : static_cast<uint32_t>(P.nx) * P.ny));
        const uint8_t ol = occ[li], orr = occ[ri];
        const float base = in[q];
        float g;
        if (p64 != nullptr) g = static_cast<float>(P.dt_over_h64 * (p64[ri] - p64[li]));
        else g = P.dt * (p[ri] - p[li]) / P.h;
        if (ol != 0 || orr != 0) {
            float value = 0.0f, weight = 0.0f;
            if (ol != 0) {
                value += solid[li];
                weight += 1.0f;
            }
            if (orr != 0) {
                value += solid[ri];
                weight += 1.0f;
            }
            put(value / weight);
        } else {
            put(base - g);
        }
        return;
    }
    put(settle<A, true>(P, i, j, k, occ, solid, [&](int a, int b, int c) {
        int l[3] = {a, b, c};
        int r[3] = {a, b, c};
        l[A] -= 1;
        const bool hl = resolve_flow(P, l[0], l[1], l[2]);
        const bool hr = resolve_flow(P, r[0], r[1], r[2]);
        const float base = in[fidx<A>(P, a, b, c)];
        if (!(hl && hr)) return base;
        if (p64 != nullptr) {  // FP64 solution of a refined solve: the gradient keeps its precision
            const double g = P.dt_over_h64 * (p64[cidx(P, r[0], r[1], r[2])] - p64[cidx(P, l[0], l[1], l[2])]);
            return base - static_cast<float>(g);
        }
        const float pr = p[cidx(P, r[0], r[1], r[2])];
        const float pl = p[cidx(P, l[0], l[1], l[2])];
        return base - P.dt * (pr - pl) / P.h;
    }));
}

template <bool COLUMN>
__global__ void __launch_bounds__(kThreads) project_kernel(const __grid_constant__ StepParams P, const float* __restrict__ iu, const float* __restrict__ iv, const float* __restrict__ iw, const float* __restrict__ p, const double* __restrict__ p64, const uint8_t* __restrict__ occ, const float* __restrict__ su, const float* __restrict__ sv, const float* __restrict__ sw, float* __restrict__ ou,
                                                            float* __restrict__ ov, float* __restrict__ ow, float* __restrict__ pu, float* __restrict__ pv, float* __restrict__ pw, unsigned bu, unsigned bv, int planes) {
    pdl_begin();
    const unsigned b = blockIdx.x;
    if (b < bu) {
        for_face_column<0, COLUMN>(P, b, planes, [&](uint32_t q, int i, int j, int k) { project_one<0>(P, q, i, j, k, iu, p, p64, occ, su, ou, pu); });
    } else if (b < bu + bv) {
        for_face_column<1, COLUMN>(P, b - bu, planes, [&](uint32_t q, int i, int j, int k) { project_one<1>(P, q, i, j, k, iv, p, p64, occ, sv, ov, pv); });
    } else {
        for_face_column<2, COLUMN>(P, b - bu - bv, planes, [&](uint32_t q, int i, int j, int k) { project_one<2>(P, q, i, j, k, iw, p, p64, occ, sw, ow, pw); });
    }
}

// ------------------------------------------------------------------------------------------ scalars
// Fluid cells: one back-trace, then both scalars sampled with their own boundary rules (:1221-1233).
// Solid cells: temperature = solid temperature (:1235-1241), density = 0 until the fill pass.
template <bool CUBIC, bool TILED, bool POW2>
__global__ void __launch_bounds__(kThreads) advect_scalars_kernel(const __grid_constant__ StepParams P, const PadField u, const PadField v, const PadField w, const uint8_t* __restrict__ occ, const PadField t_tmp, const PadField d_tmp, const float* __restrict__ solid_t, float* __restrict__ t, float* __restrict__ d) {
    pdl_begin();
    int x, y, z;
    uint32_t q;
    if (TILED) {
        if (!tile_point(P, blockIdx.x, P.nx, P.ny, P.nz, x, y, z)) return;
        q = cidx(P, x, y, z);
    } else {
        q = blockIdx.x * blockDim.x + threadIdx.x;
        if (q >= P.n) return;
        cell_xyz(P, q, x, y, z);
    }
    if (occ[q] != 0) {
        t[q] = solid_t[q];
        d[q] = 0.0f;
        return;
    }
    const float h = P.h;
    const float3 p = trace_rk2<POW2, 3>((static_cast<float>(x) + 0.5f) * h, (static_cast<float>(y) + 0.5f) * h, (static_cast<float>(z) + 0.5f) * h, x, y, z, u, v, w, occ, P);
    float tv, dv;
    sample_pad_scalars<CUBIC, POW2>(t_tmp, d_tmp, p.x, p.y, p.z, P, tv, dv);
    t[q] = tv;
    d[q] = dv;
}

__global__ void density_fill_kernel(const FillEntry* __restrict__ list, const uint32_t* __restrict__ count, float* __restrict__ d) {
    pdl_begin();
    const uint32_t n = *count;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const FillEntry e = list[t];
        d[e.cell] = e.source >= 0 ? d[e.source] : 0.0f;
    }
}

// ------------------------------------------------------------------------------------------ views
__global__ void __launch_bounds__(kThreads) views_kernel(const __grid_constant__ StepParams P, const float* __restrict__ u, const float* __restrict__ v, const float* __restrict__ w, const uint8_t* __restrict__ occ, float* __restrict__ cx, float* __restrict__ cy, float* __restrict__ cz, float* __restrict__ vm, float* __restrict__ wx, float* __restrict__ wy,
                                                          float* __restrict__ wz, float* __restrict__ wm, float* __restrict__ div, uint32_t groups) {
    pdl_begin();
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= P.n) return;
    int x, y, z;
    cell_xyz(P, q, x, y, z);
    if (groups & kViewsVelocity) {
        const float a = centred<0>(u, x, y, z, P);
        const float b = centred<1>(v, x, y, z, P);
        const float c = centred<2>(w, x, y, z, P);
        cx[q] = a;
        cy[q] = b;
        cz[q] = c;
        vm[q] = sqrtf(a * a + b * b + c * c);
    }
    if (!(groups & kViewsVorticity)) return;
    if (occ[q] != 0) {
        wx[q] = wy[q] = wz[q] = wm[q] = 0.0f;
        div[q] = 0.0f;
        return;
    }
    const float4 o = vorticity_at(u, v, w, x, y, z, P);
    wx[q] = o.x;
    wy[q] = o.y;
    wz[q] = o.z;
    wm[q] = o.w;
    div[q] = (u[fidx<0>(P, x + 1, y, z)] - u[fidx<0>(P, x, y, z)] + v[fidx<1>(P, x, y + 1, z)] - v[fidx<1>(P, x, y, z)] + w[fidx<2>(P, x, y, z + 1)] - w[fidx<2>(P, x, y, z)]) * P.inv_h;
}

// ------------------------------------------------------------------------------------------ occupancy-derived
__global__ void occupancy_float_kernel(uint32_t n, const uint8_t* __restrict__ occ, float* __restrict__ out) {
    pdl_begin();
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) out[q] = static_cast<float>(occ[q]);
}

__global__ void set_int_kernel(int32_t* p, int32_t v) {
    pdl_begin();
    *p = v;
}

// anchor = smallest fluid cell index (:1292-1302), into *anchor (set to n before). Warps take runs of 32 cells in ascending
// order and stop at the first one with a fluid cell or past an anchor already found, so a grid of one block per SM reads little
// more than the cells up to it (one atomic for each of the grid's warps took 25 us at 96x128x96, now 2.4).
__global__ void __launch_bounds__(kThreads) anchor_kernel(uint32_t n, const uint8_t* __restrict__ occ, int32_t* anchor) {
    pdl_begin();
    const uint32_t lane = threadIdx.x & 31u, warps = gridDim.x * (kThreads / 32);
    for (uint64_t first = 32ull * (blockIdx.x * (kThreads / 32) + threadIdx.x / 32); first < n; first += 32ull * warps) {
        int32_t found = lane == 0 ? *static_cast<volatile int32_t*>(anchor) : 0;
        found = __shfl_sync(0xffffffffu, found, 0);  // one value for the warp
        if (static_cast<int64_t>(first) >= found) return;
        const uint32_t fluid = __ballot_sync(0xffffffffu, first + lane < n && occ[first + lane] == 0);
        if (fluid == 0) continue;
        if (lane == 0) atomicMin(anchor, static_cast<int32_t>(first + __ffs(static_cast<int>(fluid)) - 1u));
        return;
    }
}

// Row code of the Poisson operator (:1343-1412): solid or anchor rows are identity (diag 1, no neighbours);
// a fluid row's diagonal counts fluid neighbours (anchor included, periodic wrap, repeats counted) plus OUTFLOW
// domain faces, at least 1; neighbour bits mark distinct fluid non-anchor neighbours other than the cell itself.
__global__ void __launch_bounds__(kThreads) stencil_code_kernel(const __grid_constant__ StepParams P, const uint8_t* __restrict__ occ, const int32_t* __restrict__ anchor_ptr, uint16_t* __restrict__ codes) {
    pdl_begin();
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= P.n) return;
    const int32_t anchor = *anchor_ptr;
    if (occ[q] != 0 || static_cast<int32_t>(q) == anchor) {
        codes[q] = static_cast<uint16_t>(1u << 8);
        return;
    }
    int c[3];
    cell_xyz(P, q, c[0], c[1], c[2]);
    const int n[3] = {P.nx, P.ny, P.nz};
    uint32_t diag = 0, mask = 0;
#pragma unroll
    for (int e = 0; e < 6; ++e) {
        const int a = e >> 1;
        int d[3] = {c[0], c[1], c[2]};
        d[a] += (e & 1) ? 1 : -1;
        if (d[a] < 0 || d[a] >= n[a]) {
            if (!P.fper[a]) {
                if (P.flow[e].type == kFlowOutflow) ++diag;
                continue;
            }
            d[a] = wrapi(d[a], n[a]);
        }
        const uint32_t nb = cidx(P, d[0], d[1], d[2]);
        if (occ[nb] != 0) continue;
        ++diag;
        if (static_cast<int32_t>(nb) == anchor || nb == q) continue;
        if ((e & 1) && n[a] == 2 && P.fper[a]) continue;  // same cell as the -a neighbour, kept once
        mask |= 1u << e;
    }
    if (diag == 0) diag = 1;
    codes[q] = static_cast<uint16_t>(mask | (diag << 8) | kCodeActive);
}

// Sources of FillEntry while the list is built: a cell whose 26 neighbours are all solid, and one without any fluid cell.
constexpr int32_t kFillDeep = -2, kFillNone = -1;

// v + d on a density axis of n cells, |d| < n, wrapped on a periodic one; false when there is no such cell.
__device__ __forceinline__ bool fill_axis(int& v, int d, int n, int per) {
    v += d;
    if (v < 0) {
        v += n;
        return per != 0;
    }
    if (v >= n) {
        v -= n;
        return per != 0;
    }
    return true;
}

// Cells of the 3 x 3 x 3 neighbourhood (bit 9 (dz + 1) + 3 (dy + 1) + dx + 1) at squared distance d2.
__host__ __device__ constexpr uint32_t fill_ring(int d2) {
    uint32_t m = 0;
    for (int i = 0; i < 27; ++i) {
        const int dx = i % 3 - 1, dy = i / 3 % 3 - 1, dz = i / 9 - 1;
        if (dx * dx + dy * dy + dz * dz == d2) m |= 1u << i;
    }
    return m;
}

// Nearest-fluid source of each solid cell (:1243-1290): first Chebyshev shell (radius 1, 2, ...) holding a fluid cell,
// smallest squared distance in it, first in (dz, dy, dx) scan order on ties, density periodicity.
// Three kernels split it by depth, because a warp per cell wastes lanes on a small shell and a thread per cell makes the deepest
// cell a serial chain. Rebuilding everything that depends on the occupancy, with a thread per cell throughout, a warp per cell
// throughout and split: a sphere of radius 12 in 96x128x96 564, 103 and 86 us; of radius 40 in 128^3 19.1, 8.1 and 3.6 ms; half
// of 128^3 solid at random 228, 717 and 138 us; walls of 8 cells there 823, 2667 and 768 us, a floor of 32 68, 119 and 36 ms;
// walls of one cell in 256^3 666, 986 and 398 us.
// The first one lists the solid cells, in no particular order (a warp's cells take one slot range), with the sources that shell
// 1 holds: thin walls and scattered solids end here, a thread per cell with its 26 loads in flight.
__global__ void __launch_bounds__(kThreads) fill_list_kernel(const __grid_constant__ StepParams P, const uint8_t* __restrict__ occ, const int32_t* __restrict__ anchor_ptr, FillEntry* __restrict__ list, uint32_t* __restrict__ count) {
    pdl_begin();
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    const bool solid = q < P.n && occ[q] != 0;
    const uint32_t solids = __ballot_sync(0xffffffffu, solid);
    if (solids == 0) return;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(count, static_cast<uint32_t>(__popc(solids)));
    base = __shfl_sync(0xffffffffu, base, 0);
    int32_t source = kFillNone;
    if (solid && *anchor_ptr < static_cast<int32_t>(P.n)) {  // at least one fluid cell exists
        int x, y, z;
        cell_xyz(P, q, x, y, z);
        int cx[3], cy[3], cz[3];
        bool ox[3], oy[3], oz[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            cx[k] = x;
            cy[k] = y;
            cz[k] = z;
            ox[k] = fill_axis(cx[k], k - 1, P.nx, P.dper[0]);
            oy[k] = fill_axis(cy[k], k - 1, P.ny, P.dper[1]);
            oz[k] = fill_axis(cz[k], k - 1, P.nz, P.dper[2]);
        }
        uint32_t fluid = 0;
#pragma unroll
        for (int i = 0; i < 27; ++i) {
            if (i == 13) continue;
            const int kx = i % 3, ky = i / 3 % 3, kz = i / 9;
            if (ox[kx] && oy[ky] && oz[kz] && occ[cidx(P, cx[kx], cy[ky], cz[kz])] == 0) fluid |= 1u << i;
        }
        constexpr uint32_t kFaces = fill_ring(1), kEdges = fill_ring(2);
        source = kFillDeep;
        if (fluid != 0) {
            const uint32_t nearest = (fluid & kFaces) ? fluid & kFaces : ((fluid & kEdges) ? fluid & kEdges : fluid);
            const int i = __ffs(static_cast<int>(nearest)) - 1;
            fill_axis(x, i % 3 - 1, P.nx, P.dper[0]);
            fill_axis(y, i / 3 % 3 - 1, P.ny, P.dper[1]);
            fill_axis(z, i / 9 - 1, P.nz, P.dper[2]);
            source = static_cast<int32_t>(cidx(P, x, y, z));
        }
    }
    if (solid) list[base + __popc(solids & ((1u << lane) - 1u))] = FillEntry{q, source};
    const uint32_t deep = __ballot_sync(0xffffffffu, source == kFillDeep);
    if (lane == 0 && deep != 0) atomicAdd(count + 1, static_cast<uint32_t>(__popc(deep)));
}

// The best cell of a shell so far: smallest squared distance, then first in scan order.
struct FillBest {
    long long d2;
    int dz, dy, dx;
    int32_t cell;
    __device__ __forceinline__ void take(long long d, int z, int y, int x, int32_t c) {
        const bool better = d != d2 ? d < d2 : (z != dz ? z < dz : (y != dy ? y < dy : x < dx));
        if (!better) return;
        d2 = d;
        dz = z;
        dy = y;
        dx = x;
        cell = c;
    }
};

// A look at the two faces of the cube of radius r across axis A (0 x, 1 y, 2 z) around the cell at c, shared by W lanes: the z
// faces whole, the y faces without their z edges, the x faces without any, so the three calls see each cell of the shell once.
// Offsets that leave the domain are cut off beforehand, on a periodic axis at |d| < n: a longer one is a cell that a shorter one
// has shown. A lane steps through rows and columns by W cells without a division.
template <int A, int W>
__device__ __forceinline__ void fill_faces(const StepParams& P, const uint8_t* __restrict__ occ, const int c[3], int r, uint32_t lane, FillBest& best) {
    constexpr int R = A == 2 ? 1 : 2, C = A == 0 ? 1 : 0;  // axes of the rows and of the columns
    const int n[3] = {P.nx, P.ny, P.nz};
    const uint32_t stride[3] = {1u, static_cast<uint32_t>(P.nx), static_cast<uint32_t>(P.nx) * P.ny};
    const int low[3] = {P.dper[0] ? 1 - P.nx : -c[0], P.dper[1] ? 1 - P.ny : -c[1], P.dper[2] ? 1 - P.nz : -c[2]};
    const int high[3] = {P.dper[0] ? P.nx - 1 : P.nx - 1 - c[0], P.dper[1] ? P.ny - 1 : P.ny - 1 - c[1], P.dper[2] ? P.nz - 1 : P.nz - 1 - c[2]};
    const bool minus = -r >= low[A], plus = r <= high[A];
    if (!minus && !plus) return;
    const int rr = A == 2 ? r : r - 1, rc = A == 0 ? r - 1 : r;
    const int row0 = imax(-rr, low[R]), col0 = imax(-rc, low[C]);
    const int rows = imin(rr, high[R]) - row0 + 1, cols = imin(rc, high[C]) - col0 + 1;
    int at[2] = {c[A], c[A]};
    fill_axis(at[0], minus ? -r : 0, n[A], P.dper[A]);
    fill_axis(at[1], plus ? r : 0, n[A], P.dper[A]);
    const uint32_t face[2] = {static_cast<uint32_t>(at[0]) * stride[A], static_cast<uint32_t>(at[1]) * stride[A]};
    int row = W > 1 ? static_cast<int>(lane) / cols : 0, col = static_cast<int>(lane) - row * cols;
    const int drow = W / cols, dcol = W - drow * cols;
    constexpr int kBatch = 2;  // two cells of either face in flight
    while (row < rows) {
        uint32_t q[kBatch];
        int d[kBatch][2];
        uint8_t s[kBatch][2];
        bool in[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            in[k] = row < rows;
            d[k][0] = row0 + row;
            d[k][1] = col0 + col;
            int y = c[R], x = c[C];
            fill_axis(y, d[k][0], n[R], P.dper[R]);
            fill_axis(x, d[k][1], n[C], P.dper[C]);
            q[k] = static_cast<uint32_t>(y) * stride[R] + static_cast<uint32_t>(x) * stride[C];
            s[k][0] = in[k] && minus ? occ[face[0] + q[k]] : 1;
            s[k][1] = in[k] && plus ? occ[face[1] + q[k]] : 1;
            row += drow;
            col += dcol;
            if (col >= cols) {
                col -= cols;
                ++row;
            }
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k)
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                if (s[k][side]) continue;
                int o[3];
                o[A] = side ? r : -r;
                o[R] = d[k][0];
                o[C] = d[k][1];
                const long long d2 = static_cast<long long>(r) * r + static_cast<long long>(o[R]) * o[R] + static_cast<long long>(o[C]) * o[C];
                best.take(d2, o[2], o[1], o[0], static_cast<int32_t>(face[side] + q[k]));
            }
    }
}

template <int W>
__device__ __forceinline__ void fill_shell(const StepParams& P, const uint8_t* __restrict__ occ, const int c[3], int r, uint32_t lane, FillBest& best) {
    fill_faces<2, W>(P, occ, c, r, lane, best);
    fill_faces<1, W>(P, occ, c, r, lane, best);
    fill_faces<0, W>(P, occ, c, r, lane, best);
}
__device__ __forceinline__ FillBest fill_nothing() { return FillBest{0x7fffffffffffffffll, 0, 0, 0, kFillNone}; }

// From this many deep cells on, shells 2 to kFillNearRadius are searched by a thread per cell: all its lanes have work there,
// a warp's do not (25, 15 and 9 cells a face in shell 2). With fewer, one thread's serial chain takes longer than the warps
// do: the rebuild with threads and with warps there takes 90 and 77 us with 12 000 deep cells (a floor of 4 in 64^3), 106 and 112
// with 28 000, 124 and 140 with 38 000, 190 and 260 with 77 000.
constexpr uint32_t kFillMany = 32768;
constexpr int kFillNearRadius = 4;
__global__ void __launch_bounds__(kThreads) fill_near_kernel(const __grid_constant__ StepParams P, const uint8_t* __restrict__ occ, FillEntry* __restrict__ list, const uint32_t* __restrict__ count) {
    pdl_begin();
    if (count[1] < kFillMany) return;
    const uint32_t entries = count[0];
    for (uint64_t e = blockIdx.x * kThreads + threadIdx.x; e < entries; e += static_cast<uint64_t>(gridDim.x) * kThreads) {
        if (list[e].source != kFillDeep) continue;
        int c[3];
        cell_xyz(P, list[e].cell, c[0], c[1], c[2]);
        FillBest best = fill_nothing();
        for (int r = 2; r <= kFillNearRadius && best.cell < 0; ++r) fill_shell<1>(P, occ, c, r, 0u, best);
        if (best.cell >= 0) list[e].source = best.cell;
    }
}

// The deep cells that are left, a warp per cell, its lanes sharing each shell: a cell at depth r has
// (2 r + 1)^3 neighbours to look at, one load latency after the other if a thread walks them, and the deepest cell decides the
// time. A warp takes every warps-th entry, since deep cells lie together in the list.
__global__ void __launch_bounds__(kThreads) fill_source_kernel(const __grid_constant__ StepParams P, const uint8_t* __restrict__ occ, FillEntry* __restrict__ list, const uint32_t* __restrict__ count) {
    pdl_begin();
    const uint32_t lane = threadIdx.x & 31u, warps = gridDim.x * (kThreads / 32), entries = count[0];
    const int max_radius = imax(P.nx, imax(P.ny, P.nz)), from = count[1] < kFillMany ? 2 : kFillNearRadius + 1;
    if (count[1] == 0) return;
    for (uint64_t first = blockIdx.x * (kThreads / 32) + threadIdx.x / 32; first < entries; first += 32ull * warps) {
        const uint64_t e = first + static_cast<uint64_t>(lane) * warps;
        FillEntry mine{0u, kFillNone};
        if (e < entries) mine = list[e];
        for (uint32_t deep = __ballot_sync(0xffffffffu, mine.source == kFillDeep); deep != 0; deep &= deep - 1u) {
            const int owner = __ffs(static_cast<int>(deep)) - 1;
            int c[3];
            cell_xyz(P, __shfl_sync(0xffffffffu, mine.cell, owner), c[0], c[1], c[2]);
            FillBest best = fill_nothing();
            for (int r = from; r <= max_radius; ++r) {
                fill_shell<32>(P, occ, c, r, lane, best);
                if (__any_sync(0xffffffffu, best.cell >= 0)) break;
            }
            for (int o = 16; o > 0; o >>= 1)
                best.take(__shfl_xor_sync(0xffffffffu, best.d2, o), __shfl_xor_sync(0xffffffffu, best.dz, o), __shfl_xor_sync(0xffffffffu, best.dy, o), __shfl_xor_sync(0xffffffffu, best.dx, o), __shfl_xor_sync(0xffffffffu, best.cell, o));
            if (lane == static_cast<uint32_t>(owner)) list[e].source = best.cell;
        }
    }
}

__global__ void fill_value_kernel(float* __restrict__ dst, float value, uint64_t count) {
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < count; i += static_cast<uint64_t>(gridDim.x) * blockDim.x) dst[i] = value;
}

}  // namespace

constexpr uint32_t kColumnCells = 600000, kColumnSlab = 16 * kThreads;
constexpr int kColumnPlanes = 4;

StepParams make_params(const SmokeSimulationConfig& cfg) {
    StepParams P{};
    P.nx = cfg.nx;
    P.ny = cfg.ny;
    P.nz = cfg.nz;
    P.h = cfg.cell_size;
    P.dt = cfg.dt;
    P.ambient = cfg.ambient_temperature;
    P.alpha = cfg.buoyancy_density_factor;
    P.beta = cfg.buoyancy_temperature_factor;
    P.epsilon = cfg.vorticity_confinement;
    P.cubic = cfg.scalar_advection_mode == SMOKE_SIMULATION_SCALAR_ADVECTION_MONOTONIC_CUBIC;
    const SmokeSimulationFlowBoundaryFaceDesc* fb = &cfg.flow_boundary.x_minus;
    const SmokeSimulationScalarBoundaryFaceDesc* db = &cfg.density_boundary.x_minus;
    const SmokeSimulationScalarBoundaryFaceDesc* tb = &cfg.temperature_boundary.x_minus;
    for (int e = 0; e < 6; ++e) {
        P.flow[e] = fb[e];
        P.den[e] = db[e];
        P.tem[e] = tb[e];
    }
    for (int a = 0; a < 3; ++a) {
        P.fper[a] = fb[2 * a].type == kFlowPeriodic && fb[2 * a + 1].type == kFlowPeriodic;
        P.dper[a] = db[2 * a].type == kScalarPeriodic && db[2 * a + 1].type == kScalarPeriodic;
        P.tper[a] = tb[2 * a].type == kScalarPeriodic && tb[2 * a + 1].type == kScalarPeriodic;
    }
    const uint32_t nx = cfg.nx, ny = cfg.ny, nz = cfg.nz;
    P.n = nx * ny * nz;
    P.nu = (nx + 1) * ny * nz;
    P.nv = nx * (ny + 1) * nz;
    P.nw = nx * ny * (nz + 1);
    P.inv_h = 1.0f / cfg.cell_size;
    {  // a normal power of two with a normal reciprocal: x * inv_h == x / h for every float x
        int e = 0;
        P.h_pow2 = std::isnormal(cfg.cell_size) && std::isnormal(P.inv_h) && std::frexp(cfg.cell_size, &e) == 0.5f && P.inv_h * cfg.cell_size == 1.0f;
    }
    P.dt_over_h64 = static_cast<double>(cfg.dt) / static_cast<double>(cfg.cell_size);
    P.div_nx = FastDiv(nx);
    P.div_ny = FastDiv(ny);
    P.div_slab = FastDiv(nx * ny);
    for (int a = 0; a < 3; ++a) {
        P.div_fx[a] = FastDiv(nx + (a == 0));
        P.div_fy[a] = FastDiv(ny + (a == 1));
    }
    set_advect_tile(P, 0);
    return P;
}

bool set_advect_tile(StepParams& P, int code) {
    if (code < 0 || code >= kAdvectTileCount) return false;
    for (int a = 0; a < 3; ++a) P.tile[a] = kAdvectTiles[code][a];
    return true;
}

// Cells of a column per thread in the projection, face-force and right-hand-side kernels (for_column). They are bound
// by instruction issue, a good part of it index arithmetic, which a column pays once: 256x384x256 face force 453 -> 333 us,
// projection 365 -> 271, right-hand side 142 -> 119; 128^3 34 -> 30, 30 -> 25, 13 -> 10. Two cells
// give half of that, 8 or 16 leave 97x141x83 too few threads (projection 20, 21, 26 and 41 us with 2, 4, 8 and 16).
// Where the line lies: the three kernels together, with one cell against columns, take 34 and 46 us at 32^3, 25.6 and 28.1 at
// 64^3, 29.9 and 28.6 at 72^3, 36.0 and 33.5 at 84^3, 38.1 and 34.5 at 88^3, 56 and 46 at 97x141x83. Columns win from about
// 370 000 cells; the line at kColumnCells keeps to the sizes where they win by a tenth or more. Planes below kColumnSlab cells
// would fill their blocks badly (16x16x2600 36.2 and 36.0). Vorticity and cell force got slower as
// columns (30 -> 40 and 22 -> 27 us at 97x141x83) and stay with one.
int column_planes(const StepParams& P) { return P.n >= kColumnCells && static_cast<uint32_t>(P.nx) * P.ny >= kColumnSlab ? std::max(kColumnPlanes, (P.nz + 65535) / 65535) : 0; }
dim3 column_grid(const StepParams& P, int planes) { return planes > 0 ? dim3(blocks_for(static_cast<uint64_t>(P.nx) * P.ny), (P.nz + planes - 1) / planes) : dim3(blocks_for(P.n)); }

// Blocks of the u and v faces and the whole grid of a kernel over all faces.
struct FaceBlocks {
    unsigned u, v;
    dim3 grid;
};
FaceBlocks face_blocks(const StepParams& P, int planes) {
    const uint64_t nx = P.nx, ny = P.ny;
    FaceBlocks B;
    B.u = planes > 0 ? blocks_for((nx + 1) * ny) : blocks_for(P.nu);
    B.v = planes > 0 ? blocks_for(nx * (ny + 1)) : blocks_for(P.nv);
    B.grid = planes > 0 ? dim3(B.u + B.v + blocks_for(nx * ny), (P.nz + planes) / planes) : dim3(B.u + B.v + blocks_for(P.nw));
    return B;
}

cudaError_t launch_vorticity(const StepParams& P, ConstFaces vel, const uint8_t* occ, float* wx, float* wy, float* wz, float* wmag, cudaStream_t s) {
    vorticity_kernel<<<blocks_for(P.n), kThreads, 0, s>>>(P, vel.u, vel.v, vel.w, occ, wx, wy, wz, wmag);
    return cudaGetLastError();
}

cudaError_t launch_cell_force(const StepParams& P, const float* wx, const float* wy, const float* wz, const float* wmag, const float* density, const float* temperature, const float* ufx, const float* ufy, const float* ufz, const uint8_t* occ, float* fx, float* fy, float* fz, cudaStream_t s, const ScalarSources& S) {
    launch_pdl(cell_force_kernel, dim3(blocks_for(P.n)), dim3(kThreads), 0, s, P, wx, wy, wz, wmag, density, temperature, ufx, ufy, ufz, occ, fx, fy, fz, S);
    return cudaGetLastError();
}

cudaError_t launch_face_force(const StepParams& P, ConstFaces in, const float* fx, const float* fy, const float* fz, const uint8_t* occ, ConstFaces solid, Faces out, cudaStream_t s, Faces pad) {
    const int planes = column_planes(P);
    const FaceBlocks B = face_blocks(P, planes);
    launch_pdl(planes > 0 ? face_force_kernel<true> : face_force_kernel<false>, B.grid, dim3(kThreads), 0, s, P, in.u, in.v, in.w, fx, fy, fz, occ, solid.u, solid.v, solid.w, out.u, out.v, out.w, pad.u, pad.v, pad.w, B.u, B.v, planes);
    return cudaGetLastError();
}

// Padded copy descriptor of field KIND stored at `pad`.
PadField pad_field(const StepParams& P, int kind, const float* raw, const float* pad) {
    const uint32_t fx = P.nx + (kind == 0), fy = P.ny + (kind == 1);
    PadField F{};
    F.p = pad;
    F.raw = raw;
    F.px = fx + 2 * kPad;
    F.pxy = F.px * (fy + 2 * kPad);
    return F;
}

size_t pad_count(const StepParams& P, int kind) {
    return static_cast<size_t>(P.nx + (kind == 0) + 2 * kPad) * (P.ny + (kind == 1) + 2 * kPad) * (P.nz + (kind == 2) + 2 * kPad);
}

cudaError_t launch_pads(const StepParams& P, int count, const int* kinds, const float* const* fields, float* const* pads, cudaStream_t s, int ghost_only) {
    if (count < 1 || count > 3) return cudaErrorInvalidValue;
    PadJob J{};
    J.count = count;
    J.pz_blocks = (P.nz + 1 + 2 * kPad + kPadPlanes - 1) / kPadPlanes;
    for (int c = 0; c < count; ++c) {
        J.f[c] = fields[c];
        J.out[c] = pads[c];
        J.kind[c] = kinds[c];
    }
    if (ghost_only) {  // the largest shell of the fields (faces of the x, y or z axis have one more layer)
        const uint32_t px = P.nx + 1 + 2 * kPad, py = P.ny + 1 + 2 * kPad, pz = P.nz + 1 + 2 * kPad;
        const uint64_t most = static_cast<uint64_t>(px) * py * pz - static_cast<uint64_t>(P.nx) * P.ny * P.nz;
        launch_pdl(pad_ghost_kernel, dim3(static_cast<unsigned>((most + 255) / 256), count), dim3(256), 0, s, P, J);
        return cudaGetLastError();
    }
    const dim3 grid((P.nx + 1 + 2 * kPad + 31) / 32, (P.ny + 1 + 2 * kPad + 7) / 8, J.pz_blocks * count);
    pad_kernel<<<grid, dim3(32, 8), 0, s>>>(P, J);
    return cudaGetLastError();
}

// The advection kernel instance <CUBIC, TILED, POW2> of P, from the 8 given in that binary order.
template <class K>
K pick_advect(const StepParams& P, K k000, K k001, K k010, K k011, K k100, K k101, K k110, K k111) {
    const K all[8] = {k000, k001, k010, k011, k100, k101, k110, k111};
    return all[(P.cubic ? 4 : 0) + (P.tile[0] >= 0 ? 2 : 0) + (P.h_pow2 ? 1 : 0)];
}

// The device's global nanosecond timer into *slot (one thread).
__global__ void time_stamp_kernel(unsigned long long* slot) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    *slot = t;
}

cudaError_t launch_time_stamp(unsigned long long* slot, cudaStream_t s) {
    time_stamp_kernel<<<1, 1, 0, s>>>(slot);
    return cudaGetLastError();
}

cudaError_t launch_advect_velocity(const StepParams& P, ConstFaces in, ConstFaces pad, const uint8_t* occ, ConstFaces solid, Faces out, cudaStream_t s) {
    const unsigned bu = advect_blocks(P, P.nx + 1, P.ny, P.nz), bv = advect_blocks(P, P.nx, P.ny + 1, P.nz), bw = advect_blocks(P, P.nx, P.ny, P.nz + 1);
    const PadField u = pad_field(P, 0, in.u, pad.u), v = pad_field(P, 1, in.v, pad.v), w = pad_field(P, 2, in.w, pad.w);
    auto kernel = pick_advect(P, advect_velocity_kernel<false, false, false>, advect_velocity_kernel<false, false, true>, advect_velocity_kernel<false, true, false>, advect_velocity_kernel<false, true, true>, advect_velocity_kernel<true, false, false>,
                              advect_velocity_kernel<true, false, true>, advect_velocity_kernel<true, true, false>, advect_velocity_kernel<true, true, true>);
    launch_pdl(kernel, dim3(bu + bv + bw), dim3(kThreads), 0, s, P, u, v, w, occ, solid.u, solid.v, solid.w, out.u, out.v, out.w, bu, bv);
    return cudaGetLastError();
}

cudaError_t launch_rhs(const StepParams& P, ConstFaces vel, const uint8_t* occ, const int32_t* anchor, float* rhs, cudaStream_t s) {
    const int planes = column_planes(P);
    launch_pdl(planes > 0 ? rhs_kernel<true> : rhs_kernel<false>, column_grid(P, planes), dim3(kThreads), 0, s, P, vel.u, vel.v, vel.w, occ, anchor, rhs, planes);
    return cudaGetLastError();
}

cudaError_t launch_project(const StepParams& P, ConstFaces in, const float* pressure, const double* pressure64, const uint8_t* occ, ConstFaces solid, Faces out, cudaStream_t s, Faces pad) {
    const int planes = column_planes(P);
    const FaceBlocks B = face_blocks(P, planes);
    launch_pdl(planes > 0 ? project_kernel<true> : project_kernel<false>, B.grid, dim3(kThreads), 0, s, P, in.u, in.v, in.w, pressure, pressure64, occ, solid.u, solid.v, solid.w, out.u, out.v, out.w, pad.u, pad.v, pad.w, B.u, B.v, planes);
    return cudaGetLastError();
}

cudaError_t launch_advect_scalars(const StepParams& P, ConstFaces vel, ConstFaces vel_pad, const uint8_t* occ, const float* t_tmp, const float* t_pad, const float* d_tmp, const float* d_pad, const float* solid_temperature, float* temperature, float* density, cudaStream_t s) {
    const PadField u = pad_field(P, 0, vel.u, vel_pad.u), v = pad_field(P, 1, vel.v, vel_pad.v), w = pad_field(P, 2, vel.w, vel_pad.w);
    const PadField t = pad_field(P, 4, t_tmp, t_pad), d = pad_field(P, 3, d_tmp, d_pad);
    auto kernel = pick_advect(P, advect_scalars_kernel<false, false, false>, advect_scalars_kernel<false, false, true>, advect_scalars_kernel<false, true, false>, advect_scalars_kernel<false, true, true>, advect_scalars_kernel<true, false, false>,
                              advect_scalars_kernel<true, false, true>, advect_scalars_kernel<true, true, false>, advect_scalars_kernel<true, true, true>);
    launch_pdl(kernel, dim3(advect_blocks(P, P.nx, P.ny, P.nz)), dim3(kThreads), 0, s, P, u, v, w, occ, t, d, solid_temperature, temperature, density);
    return cudaGetLastError();
}

cudaError_t launch_density_fill(const FillEntry* list, const uint32_t* count, float* density, int max_blocks, cudaStream_t s) {
    launch_pdl(density_fill_kernel, dim3(max_blocks), dim3(kThreads), 0, s, list, count, density);
    return cudaGetLastError();
}

cudaError_t launch_views(const StepParams& P, ConstFaces vel, const uint8_t* occ, float* cx, float* cy, float* cz, float* vmag, float* wx, float* wy, float* wz, float* wmag, float* div, uint32_t groups, cudaStream_t s) {
    views_kernel<<<blocks_for(P.n), kThreads, 0, s>>>(P, vel.u, vel.v, vel.w, occ, cx, cy, cz, vmag, wx, wy, wz, wmag, div, groups);
    return cudaGetLastError();
}

cudaError_t launch_occupancy_float(const StepParams& P, const uint8_t* occ, float* out, cudaStream_t s) {
    occupancy_float_kernel<<<blocks_for(P.n), kThreads, 0, s>>>(P.n, occ, out);
    return cudaGetLastError();
}

cudaError_t launch_anchor(const StepParams& P, const uint8_t* occ, int32_t* anchor, cudaStream_t s) {
    launch_pdl(set_int_kernel, dim3(1), dim3(1), 0, s, anchor, static_cast<int32_t>(P.n));
    launch_pdl(anchor_kernel, dim3(std::min(sm_count(), blocks_for(P.n))), dim3(kThreads), 0, s, P.n, occ, anchor);
    return cudaGetLastError();
}

cudaError_t launch_stencil_codes(const StepParams& P, const uint8_t* occ, const int32_t* anchor, uint16_t* codes, cudaStream_t s) {
    launch_pdl(stencil_code_kernel, dim3(blocks_for(P.n)), dim3(kThreads), 0, s, P, occ, anchor, codes);
    return cudaGetLastError();
}

cudaError_t launch_fill_build(const StepParams& P, const uint8_t* occ, const int32_t* anchor, FillEntry* list, uint32_t* count, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(count, 0, kFillCounts * sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    launch_pdl(fill_list_kernel, dim3(blocks_for(P.n)), dim3(kThreads), 0, s, P, occ, anchor, list, count);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const dim3 wave(std::min(sm_count() * 8u, blocks_for(P.n)));  // 8 blocks an SM; the entry count is on the device
    if (P.n > kFillMany) launch_pdl(fill_near_kernel, wave, dim3(kThreads), 0, s, P, occ, list, static_cast<const uint32_t*>(count));
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    launch_pdl(fill_source_kernel, wave, dim3(kThreads), 0, s, P, occ, list, static_cast<const uint32_t*>(count));
    return cudaGetLastError();
}

cudaError_t launch_fill_value(float* dst, float value, uint64_t count, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    const uint64_t want = (count + kThreads - 1) / kThreads;
    const unsigned grid = static_cast<unsigned>(want < 4096 ? want : 4096);
    fill_value_kernel<<<grid, kThreads, 0, s>>>(dst, value, count);
    return cudaGetLastError();
}

}  // namespace smoke_b200
