// The fixed-count conjugate-gradient solve (the reference's solver, backend-cuda.cu:1414-1418, 1788-1824) with the whole
// iteration state on the chip, for grids whose vectors fit there.
//
// Work is split as in the streaming kernel (pcg.cu, march.cuh): 32 x 8-cell columns, each block a balanced range of
// (column, plane) units with the planes of a column consecutive, one thread per cell of a plane, one block per SM
// (cooperative launch). Here a block keeps its range: w and s of a thread's cells live in registers, r (with a one-cell
// halo), p and the operator codes in shared memory; only the iterate x goes through L2, its update placed where the block
// waits for the others. Arithmetic and the order of the sums are the streaming kernel's (Chronopoulos-Gear CG, M = I:
// s = w + beta s, p = r + beta p, r -= alpha s, w = A r, x += alpha p; a thread's products in plane order, then the warp,
// the block, 8 groups of blocks), because 64 unconverged iterations carry a change of rounding in alpha into the whole field.
// One order differs: the streaming kernel adds the blocks' FP64 partials of a group as they arrive, this one in block order, so
// its answer does not vary. That moves a total by a few 2^-53, which alpha and beta, rounded to FP32, hardly ever see: the two
// kernels gave the same bits after 64 iterations in every comparison made, and are held to 1e-4 of the largest pressure.
//
// What bounds it: the exchange (one per iteration) on small grids; on large ones the latency of dependent instructions, with
// two warps on a scheduler (128x160x128: 25 us an iteration, 0.32 issued per scheduler and cycle; shared memory at 15 % of its
// rate, L2 at 5 %). A block needs from outside only
//  - the w of the cells next to its range (the halo's r and s follow from them by the same recurrences), and
//  - the other blocks' partial dot products.
// Both travel as 64-bit words {value, tag} that the reader polls: no fence, no atomic, one L2 round trip. The tag is the
// number of the exchange, unique over launches (PcgControl::epoch), and two copies alternate, because a block that
// publishes exchange k + 2 has seen every block's words of k + 1, which each published after reading its words of k.
// Every wait is bounded as in grid_sync.cuh.
#include <map>
#include <mutex>

#include "grid_sync.cuh"
#include "launch.h"
#include "march.cuh"
#include "smoke_b200_ext.h"

namespace smoke_b200 {
namespace {

using gsync::global_ns;
using gsync::warp_sum;
using zmarch::kThreads;
using zmarch::CX;
using zmarch::CY;

constexpr int kWarps = kThreads / 32;
constexpr int kSums = 2;              // (r, r) and (A r, r)
constexpr int kSumWords = 2 * kSums;  // 64-bit words of one block's published sums: {low half, tag}, {high half, tag} of each
constexpr int kSideWords = 2 * CX + 2 * CY;  // words of one unit's side faces: y-, y+ (32 each), x-, x+ (8 each)
constexpr int kPitch = CX + 2, kSlab = kPitch * (CY + 2);  // r in shared memory, a plane with its side halo

// (No memory clobbers: a word is valid by its tag alone, so nothing is ordered by these accesses, and the plane loops may
// overlap them with their shared-memory reads.)
__device__ __forceinline__ void put_word(unsigned long long* p, uint32_t value, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((static_cast<unsigned long long>(tag) << 32) | value));
}
__device__ __forceinline__ unsigned long long get_word(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void get_words(const unsigned long long* p, unsigned long long& a, unsigned long long& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p));
}
__device__ __forceinline__ uint32_t tag_of(unsigned long long v) { return static_cast<uint32_t>(v >> 32); }

// A wait's bound, and where giving up is recorded: the grid's abort word and the block's flag for waits of this kind. Halo
// waits and sum waits have a flag each, read behind a barrier after those waits and before a barrier that comes before the next
// ones of the kind, so every warp of the block reads the same value.
struct Wait {
    PcgControl* ctl;
    int* flag;
    unsigned long long timeout_ns;
};
// Whether a wait ends without its word: the bound ran out (then the grid's abort is raised) or another block gave up.
__device__ __noinline__ bool give_up(unsigned spins, unsigned long long t0, Wait w) {
    bool out = *reinterpret_cast<volatile int*>(&w.ctl->abort) != 0;
    if (!out && (spins >= gsync::kBarrierMaxSpins || global_ns() - t0 > w.timeout_ns)) {
        atomicExch(&w.ctl->abort, 1);
        out = true;
    }
    if (out) *w.flag = 1;
    return out;
}
// Polls *p until it carries `tag`; returns the last word seen once the wait gives up.
__device__ __noinline__ unsigned long long poll(const unsigned long long* p, uint32_t tag, Wait w) {
    const unsigned long long t0 = global_ns();
    for (unsigned spins = 1;; ++spins) {
        const unsigned long long v = get_word(p);
        if (tag_of(v) == tag || ((spins & 15u) == 0u && give_up(spins, t0, w))) return v;
    }
}

// All threads of the blocks of a cluster, with what they wrote (blocks that have left do not count). The solve starts with its
// blocks in step: the right-hand side reaches them at different times, and blocks that set out apart stay apart, each exchange
// waiting for the last one. At 32^3, where the same 16 SMs run the cluster every time, a solve took 286 us or 411 (half to nine
// tenths of a frame's, never one that followed a solve, whose right-hand side is in L2); with this barrier always 290.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct ResidentArgs {
    int nx, ny, nz;
    int per[3];
    PcgResidentPlan plan;
    const uint16_t* codes;
    const float* b;
    float* x;
    unsigned long long* exchange;
    PcgControl* ctl;
    int iterations;
    int withhold_block;
    int withhold_exchange;
    uint32_t barrier_timeout_ms;
};

// Shared memory of a block of `planes` planes in up to two column segments: r with its halo, p, the side halo's s, codes.
constexpr uint32_t resident_smem(int planes) { return static_cast<uint32_t>(4 * (kSlab * (planes + 4) + (kThreads + kSideWords) * planes) + 2 * kThreads * planes); }

static_assert(resident_smem(kPcgResidentPlanes) + 272u <= 227u * 1024u, "the largest block and its sums (FP64) fit");

// A halo cell's s and r, formed from the w its owner published, must be the owner's bit for bit, so every rounding of the
// recurrences is spelled out. (With the products left to the compiler's contraction the copies drifted apart by an ulp an
// iteration: 64 iterations at 64^3 ended 1.6e-5 from the exact ones instead of 9e-7.)
__device__ __forceinline__ void advance(float w, float fa, float fb, float& s, float& r) {
    s = __fmaf_rn(fb, s, w);
    r = __fmaf_rn(-fa, s, r);
}
// diag * r0 - active neighbours, in the order -x +x -y +y -z +z.
__device__ __forceinline__ float row_value(uint32_t code, float rm1, float r0, float r1, const float* r, int pitch) {
    const float xm = r[-1], xp = r[1], ym = r[-pitch], yp = r[pitch];
    float acc = __fmul_rn(static_cast<float>((code >> 8) & 7u), r0);
    if (code & 1u) acc = __fsub_rn(acc, xm);
    if (code & 2u) acc = __fsub_rn(acc, xp);
    if (code & 4u) acc = __fsub_rn(acc, ym);
    if (code & 8u) acc = __fsub_rn(acc, yp);
    if (code & 16u) acc = __fsub_rn(acc, rm1);
    if (code & 32u) acc = __fsub_rn(acc, r1);
    return acc;
}

// v, but not a loop invariant: what is computed from it stays out of the registers that live across iterations.
__device__ __forceinline__ int opaque(int v) {
    asm volatile("" : "+r"(v));
    return v;
}
// f(0) ... f(M - 1), each call compiled with its index a constant, so that arrays indexed by it stay in registers (a loop of
// 70 such bodies is past the compiler's unrolling limit).
template <int M, int I = 0, class F>
__device__ __forceinline__ void for_planes(F&& f) {
    if constexpr (M - I <= 16) {
#pragma unroll
        for (int i = 0; i < M - I; ++i) f(I + i);
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) f(I + i);
        for_planes<M, I + 16>(f);
    }
}

// T: the type of the dot products and scalars; M: planes of a block at most.
template <typename T, int M>
__global__ void __launch_bounds__(kThreads, 1) pcg_resident_kernel(const __grid_constant__ ResidentArgs A) {
    extern __shared__ __align__(16) float area[];
    __shared__ T red[kSums][kWarps];
    __shared__ double all[kPcgSumCopies][kSums];
    __shared__ int flag[2];  // a halo wait, a sum wait of this block gave up
    // test hook: this block never publishes, so the others' bounded waits run out and abort the solve
    if (A.withhold_block > 0 && static_cast<int>(blockIdx.x) == A.withhold_block - 1 && A.withhold_exchange == 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;  // a warp is a row of the column
    const uint32_t G = gridDim.x, total = A.plan.total;
    const uint32_t ua = static_cast<uint32_t>((static_cast<uint64_t>(blockIdx.x) * total) / G);
    const uint32_t ub = static_cast<uint32_t>((static_cast<uint64_t>(blockIdx.x + 1) * total) / G);
    const int m = static_cast<int>(ub - ua);                              // planes of this block
    const int col0 = static_cast<int>(ua / A.nz), za = static_cast<int>(ua - static_cast<uint32_t>(col0) * A.nz);
    const int m0 = min(m, A.nz - za);                                     // planes of its first column; the rest from the next
    const uint32_t slab = static_cast<uint32_t>(A.nx) * A.ny;
    const int m_max = A.plan.planes;
    float* const rs = area;                              // r: [planes, a halo plane at both ends of a segment][10][34]
    float* const ps = rs + kSlab * (m_max + 4);          // p: [planes][256]
    float* const hs = ps + kThreads * m_max;             // s of the side halo: [planes][80]
    uint16_t* const cs = reinterpret_cast<uint16_t*>(hs + kSideWords * m_max);  // codes: [planes][256]
    const unsigned long long timeout_ns = A.barrier_timeout_ms ? static_cast<unsigned long long>(A.barrier_timeout_ms) * 1000000ull : gsync::kBarrierTimeoutNs;
    const Wait halo_wait{A.ctl, &flag[0], timeout_ns}, sum_wait{A.ctl, &flag[1], timeout_ns};
    uint32_t phase = A.ctl->epoch;  // tag of the last exchange
    // geometry of the block's two columns
    struct Column {
        int x0, y0, ex, ey;
        int west, east, south, north;  // neighbouring columns (-1: domain wall)
    };
    const int ncx = A.plan.ncx, ncy = A.plan.ncy;
    auto column = [&](int col) {
        Column c;
        const int cx = col % ncx, cy = col / ncx;
        c.x0 = cx * CX;
        c.y0 = cy * CY;
        c.ex = min(CX, A.nx - c.x0);
        c.ey = min(CY, A.ny - c.y0);
        c.west = cx > 0 ? col - 1 : (A.per[0] ? col + ncx - 1 : -1);
        c.east = cx < ncx - 1 ? col + 1 : (A.per[0] ? col - (ncx - 1) : -1);
        c.south = cy > 0 ? col - ncx : (A.per[1] ? col + ncx * (ncy - 1) : -1);
        c.north = cy < ncy - 1 ? col + ncx : (A.per[1] ? col - ncx * (ncy - 1) : -1);
        return c;
    };
    const Column c0 = column(col0), c1 = column(m > m0 ? col0 + 1 : col0);
    auto seg = [&](int i) { return i < m0 ? 0 : 1; };
    auto plane_z = [&](int i) { return i < m0 ? za + i : i - m0; };
    auto rplane = [&](int i) { return i < m0 ? i + 1 : i + 3; };         // plane i's slot in rs
    const bool own0 = lane < c0.ex && warp < c0.ey, own1 = m > m0 && lane < c1.ex && warp < c1.ey;
    auto owns = [&](int k) { return k == 0 ? own0 : own1; };
    const uint32_t qa = (static_cast<uint32_t>(za) * A.ny + c0.y0 + warp) * A.nx + c0.x0 + lane;  // plane 0's cell
    const uint32_t qb = static_cast<uint32_t>(c1.y0 + warp) * A.nx + c1.x0 + lane;               // plane m0's cell
    auto cell = [&](int i) { return i < m0 ? qa + static_cast<uint32_t>(i) * slab : qb + static_cast<uint32_t>(i - m0) * slab; };
    // this thread's words among a plane's side words: its y face and x face in the two columns (-1: none); a column of one row
    // or one cell has both faces of that axis on it
    auto y_word = [&](const Column& c, bool own) { return !own ? -1 : (warp == 0 && c.south >= 0 ? lane : (warp == c.ey - 1 && c.north >= 0 ? CX + lane : -1)); };
    auto x_word = [&](const Column& c, bool own) { return !own ? -1 : (lane == 0 && c.west >= 0 ? 2 * CX + warp : (lane == c.ex - 1 && c.east >= 0 ? 2 * CX + CY + warp : -1)); };
    const int yw0 = y_word(c0, own0), yw1 = y_word(c1, own1), xw0 = x_word(c0, own0), xw1 = x_word(c1, own1);
    const bool thin = c0.ex == 1 || c0.ey == 1 || c1.ex == 1 || c1.ey == 1;
    const int slot = (warp + 1) * kPitch + lane + 1;
    float* const ra = rs + kSlab + slot;      // r of plane i < m0 at ra[i * kSlab], of a later one at rb[i * kSlab]
    float* const rb = ra + 2 * kSlab;
    // words of the current exchange: [sums of the blocks][side faces of the units][z faces]
    const size_t side_base = static_cast<size_t>(2) * G * kSumWords;
    const size_t z_base = side_base + static_cast<size_t>(2) * total * kSideWords;
    const uint32_t z_slots = 2 * G + 2 * static_cast<uint32_t>(ncx * ncy);
    auto sum_words = [&](uint32_t block) { return A.exchange + (static_cast<size_t>(phase & 1u) * G + block) * kSumWords; };
    auto side_words = [&](int col, int z) { return A.exchange + side_base + (static_cast<size_t>(phase & 1u) * total + static_cast<uint32_t>(col) * A.nz + z) * kSideWords; };
    auto z_words = [&](uint32_t s) { return A.exchange + z_base + (static_cast<size_t>(phase & 1u) * z_slots + s) * kThreads + tid; };
    // z faces: first and last plane of a block (read by the blocks before and after it in the same column), and, on a periodic
    // axis, planes 0 and nz - 1 of a column
    auto col_slot = [&](int col, int top) { return 2 * G + 2 * static_cast<uint32_t>(col) + top; };
    // the z-halo words of segment k: below its first plane, above its last one (-1: domain wall)
    auto z_slot = [&](int k, int top) -> int {
        const int col = col0 + k;
        if (top) {
            const int ze = k == 0 ? za + m0 : m - m0;  // one past the segment's last plane
            return ze < A.nz ? static_cast<int>(2 * (blockIdx.x + 1)) : (A.per[2] ? static_cast<int>(col_slot(col, 0)) : -1);
        }
        return k == 0 && za > 0 ? static_cast<int>(2 * (blockIdx.x - 1) + 1) : (A.per[2] ? static_cast<int>(col_slot(col, 1)) : -1);
    };
    auto halo_slot = [&](int k, int top) { return opaque(owns(k) ? z_slot(k, top) : -1); };
    constexpr int kItems = M < 24 ? 4 : 7;  // side words of a lane in flight
    // z-halo plane of segment k in rs
    auto z_plane = [&](int k, int top) { return k == 0 ? (top ? m0 + 1 : 0) : (top ? m + 3 : m0 + 2); };
    // side item j = 3 i + f of a warp: faces of plane i, f = 0 y-, 1 y+, 2 both x faces (lanes 0-7 x-, 8-15 x+). Returns the
    // neighbouring column (-1: none, or the lane has no cell), the word of its facing face and the slots here.
    auto side_item = [&](int j, int& word, int& rslot, int& hslot) {
        const int i = j / 3, f = j - 3 * i;
        if (i >= m) return -1;
        const Column& c = i < m0 ? c0 : c1;
        int col, u, v;
        if (f < 2) {
            col = lane < c.ex ? (f == 0 ? c.south : c.north) : -1;
            word = (f ^ 1) * CX + lane;
            hslot = f * CX + lane;
            u = lane + 1;
            v = f == 0 ? 0 : c.ey + 1;
        } else {
            const int hi = lane >> 3, y = lane & 7;
            col = lane < 16 && y < c.ey ? (hi == 0 ? c.west : c.east) : -1;
            word = 2 * CX + (hi ^ 1) * CY + y;
            hslot = 2 * CX + hi * CY + y;
            u = hi == 0 ? 0 : c.ex + 1;
            v = y + 1;
        }
        hslot += i * kSideWords;
        rslot = rplane(i) * kSlab + v * kPitch + u;
        return col;
    };

    // ------------------------------------------------------------ r = b with its halo, s = p = x = 0, codes
    if (tid < 2) flag[tid] = 0;
    for (int i = tid; i < kSlab * (m_max + 4); i += kThreads) rs[i] = 0.0f;
    __syncthreads();
    float w[M], s[M], sz[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
#pragma unroll
    for (int i = 0; i < M; ++i) w[i] = s[i] = 0.0f;
    for (int i = 0; i < m; ++i) {
        if (!owns(seg(i))) continue;
        rs[rplane(i) * kSlab + slot] = __ldg(A.b + cell(i));
        ps[i * kThreads + tid] = 0.0f;
        cs[i * kThreads + tid] = __ldg(A.codes + cell(i));
        A.x[cell(i)] = 0.0f;
    }
    for (int k = 0; k < (m > m0 ? 2 : 1); ++k)
        for (int top = 0; top < 2; ++top) {
            if (!owns(k) || z_slot(k, top) < 0) continue;
            const Column& c = k == 0 ? c0 : c1;
            int z = top ? (k == 0 ? za + m0 : m - m0) : (k == 0 ? za - 1 : -1);
            z += z < 0 ? A.nz : (z >= A.nz ? -A.nz : 0);
            rs[z_plane(k, top) * kSlab + slot] = __ldg(A.b + ((static_cast<uint32_t>(z) * A.ny + c.y0 + warp) * A.nx + c.x0 + lane));
        }
    for (int j = warp; j < 3 * m; j += kWarps) {
        int word, rslot, hslot;
        const int col = side_item(j, word, rslot, hslot);
        if (col < 0) continue;
        const int i = j / 3, f = j - 3 * i;
        const Column& c = i < m0 ? c0 : c1;
        int x = f < 2 ? c.x0 + lane : (lane < 8 ? c.x0 - 1 : c.x0 + c.ex), y = f == 0 ? c.y0 - 1 : (f == 1 ? c.y0 + c.ey : c.y0 + (lane & 7));
        x += x < 0 ? A.nx : (x >= A.nx ? -A.nx : 0);
        y += y < 0 ? A.ny : (y >= A.ny ? -A.ny : 0);
        rs[rslot] = __ldg(A.b + ((static_cast<uint32_t>(plane_z(i)) * A.ny + y) * A.nx + x));
        hs[hslot] = 0.0f;
    }
    cluster_sync();  // (the block alone where the launch is no cluster)

    // ------------------------------------------------------------ the solve: exchange 0 (the start), then one per iteration
    const T guard = static_cast<T>(1.0e-20);
    uint32_t status = SMOKE_B200_SOLVE_ITERATION_CAP;
    int it = 0;
    T bb = 0, rr = 0, gamma = 0, alpha = 0, beta = 0;
    for (bool first = true;; first = false) {
        const float fa = static_cast<float>(alpha), fb = static_cast<float>(beta);
        if (!first) {
            // the halo's w were published before the sums that set alpha and beta: the z faces' and the first group of the side
            // faces' are in flight while the own cells advance
            unsigned long long zv[2][2], v[kItems];
            // test hook: in one iteration (from 1) one block waits for faces with a tag that none carries
            const uint32_t tag = A.withhold_exchange == it + 1 && static_cast<int>(blockIdx.x) == A.withhold_block - 1 ? phase ^ 0x80000000u : phase;
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int top = 0; top < 2; ++top)
                    if (const int zs = M <= 9 ? halo_slot(k, top) : -1; zs >= 0) zv[k][top] = get_word(z_words(zs));
            const int j1 = opaque(warp);
            auto load_sides = [&](int j0) __attribute__((always_inline)) {
#pragma unroll
                for (int n = 0; n < kItems; ++n) {
                    const int j = j0 + n * kWarps;
                    int word, rslot, hslot;
                    const int col = side_item(j, word, rslot, hslot);
                    if (col >= 0) v[n] = get_word(side_words(col, plane_z(j / 3)) + word);
                }
            };
            if (M <= 9) load_sides(j1);
            {
                float* r = ra;
                bool own = own0;
                for_planes<M>([&](int i) __attribute__((always_inline)) {
                    if (i >= m) return;
                    if (i == m0) {
                        r = rb;
                        own = own1;
                    }
                    if (!own) return;
                    float rv = r[i * kSlab];
                    ps[i * kThreads + tid] = __fmaf_rn(fb, ps[i * kThreads + tid], rv);
                    advance(w[i], fa, fb, s[i], rv);
                    r[i * kSlab] = rv;
                });
            }
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int top = 0; top < 2; ++top) {
                    const int zs = halo_slot(k, top);
                    if (zs < 0) continue;
                    if (M > 9) zv[k][top] = get_word(z_words(zs));
                    if (tag_of(zv[k][top]) != tag) zv[k][top] = poll(z_words(zs), tag, halo_wait);
                    advance(__uint_as_float(static_cast<uint32_t>(zv[k][top])), fa, fb, sz[k][top], rs[z_plane(k, top) * kSlab + slot]);
                }
            for (int j0 = j1; j0 < 3 * m; j0 += kItems * kWarps) {
                if (M > 9 || j0 != j1) load_sides(j0);
#pragma unroll
                for (int n = 0; n < kItems; ++n) {
                    const int j = j0 + n * kWarps;
                    int word, rslot, hslot;
                    const int col = side_item(j, word, rslot, hslot);
                    if (col < 0) continue;
                    if (tag_of(v[n]) != tag) v[n] = poll(side_words(col, plane_z(j / 3)) + word, tag, halo_wait);
                    advance(__uint_as_float(static_cast<uint32_t>(v[n])), fa, fb, hs[hslot], rs[rslot]);
                }
            }
            __syncthreads();
        }
        // w = A r of the own cells, the faces' w published under a new tag; this thread's (r, r) and (w, r) in plane order
        T loc[kSums] = {0, 0};
        ++phase;
        {
            unsigned long long* const out = side_words(col0, za);  // units are consecutive: plane i's words 80 i further
            const float* r = ra;
            float rm1 = r[-kSlab], r0 = r[0];
            bool own = own0;
            int yw = yw0, xw = xw0;
            for_planes<M>([&](int i) __attribute__((always_inline)) {
                if (i >= m) return;
                if (i == m0) {  // the next column's first plane
                    r = rb;
                    rm1 = r[i * kSlab - kSlab];
                    r0 = r[i * kSlab];
                    own = own1;
                    yw = yw1;
                    xw = xw1;
                }
                const float r1 = r[i * kSlab + kSlab];
                if (own) {
                    const float v = row_value(cs[i * kThreads + tid], rm1, r0, r1, r + i * kSlab, kPitch);
                    w[i] = v;
                    loc[0] += static_cast<T>(r0) * static_cast<T>(r0);
                    loc[1] += static_cast<T>(v) * static_cast<T>(r0);
                    if (yw >= 0) put_word(out + i * kSideWords + yw, __float_as_uint(v), phase);
                    if (xw >= 0) put_word(out + i * kSideWords + xw, __float_as_uint(v), phase);
                }
                rm1 = r0;
                r0 = r1;
            });
            // the planes that end a range or (periodic axis) a column, formed once more with the same operations; and the second
            // faces of a thin column
            auto value = [&](int i) {
                const float* r = rs + rplane(i) * kSlab + slot;
                return __float_as_uint(row_value(cs[i * kThreads + tid], r[-kSlab], r[0], r[kSlab], r, kPitch));
            };
            for (int k = 0; k < 2; ++k) {
                if (!owns(k)) continue;
                const int lo = k == 0 ? 0 : m0, hi = k == 0 ? m0 - 1 : m - 1;
                if (lo == 0 && za > 0) put_word(z_words(2 * blockIdx.x), value(lo), phase);
                if (hi == m - 1 && plane_z(hi) < A.nz - 1) put_word(z_words(2 * blockIdx.x + 1), value(hi), phase);
                if (A.per[2] && plane_z(lo) == 0) put_word(z_words(col_slot(col0 + k, 0)), value(lo), phase);
                if (A.per[2] && plane_z(hi) == A.nz - 1) put_word(z_words(col_slot(col0 + k, 1)), value(hi), phase);
                if (!thin) continue;
                const Column& c = k == 0 ? c0 : c1;
                for (int i = lo; i <= hi; ++i) {
                    if (c.ey == 1 && c.north >= 0) put_word(out + i * kSideWords + CX + lane, value(i), phase);
                    if (c.ex == 1 && c.east >= 0) put_word(out + i * kSideWords + 2 * CX + CY + warp, value(i), phase);
                }
            }
        }
        // the block's sums in the precision of the reduction, published under the same tag
#pragma unroll
        for (int k = 0; k < kSums; ++k) {
            const T v = warp_sum(loc[k]);
            if (lane == 0) red[k][warp] = v;
        }
        __syncthreads();
        // a block whose halo is incomplete publishes no sums: no other block takes any that were formed from it, in the last
        // iteration either, after which nothing but those sums is waited for
        const bool halo_failed = *static_cast<volatile int*>(&flag[0]) != 0;
        if (warp == 0) {
            // 8 lanes per sum add the warps' partials; lanes 0 and 1 of them write the two halves
            static_assert(kWarps == 8 && kSums == 2, "8 lanes per sum");
            const int part = lane & 7, k = (lane >> 3) & 1;
            T t = red[k][part];
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            const double mine = static_cast<double>(t);
            if (lane < 16 && part < 2 && !halo_failed) put_word(sum_words(blockIdx.x) + 2 * k + part, part ? __double2hiint(mine) : __double2loint(mine), phase);
        }
        if (!first) {
            // while the other blocks' words travel: x += alpha p
            constexpr int kBatch = M < 14 ? M : 14;  // loads in flight
            for (int k = 0; k < 2; ++k) {
                if (!owns(k)) continue;
                const int lo = k == 0 ? 0 : m0, hi = k == 0 ? m0 : m;
                float* x = A.x + (k == 0 ? qa : qb);
                for (int i0 = lo; i0 < hi; i0 += kBatch) {
                    float v[kBatch];
                    const float* from = x;
                    uint32_t step = static_cast<uint32_t>(opaque(static_cast<int>(slab)));
#pragma unroll
                    for (int n = 0; n < kBatch; ++n) {
                        if (i0 + n < hi) v[n] = __ldcg(from);
                        from += step;
                    }
                    step = static_cast<uint32_t>(opaque(static_cast<int>(slab)));
#pragma unroll
                    for (int n = 0; n < kBatch; ++n) {
                        if (i0 + n < hi) __stcg(x, __fmaf_rn(fa, ps[(i0 + n) * kThreads + tid], v[n]));
                        x += step;
                    }
                }
            }
        }
        // every block's sums of the current tag (a round reads a block's words together, so the wait ends one round trip after
        // the last arrived): warp c adds those of the blocks c, c + 8, ... in FP64
        {
            double acc[kSums] = {0.0, 0.0};
            static_assert(kWarps == kPcgSumCopies, "one warp per group of blocks");
            for (uint32_t i = warp + 8u * lane; i < G; i += 256u) {
                const unsigned long long* p = sum_words(i);
                unsigned long long v[kSumWords];
                const unsigned long long t0 = global_ns();
                for (unsigned spins = 1;; ++spins) {
                    bool ok = true;
#pragma unroll
                    for (int k = 0; k < kSums; ++k) get_words(p + 2 * k, v[2 * k], v[2 * k + 1]);
#pragma unroll
                    for (int k = 0; k < kSumWords; ++k) ok = ok && tag_of(v[k]) == phase;
                    if (ok || ((spins & 15u) == 0u && give_up(spins, t0, sum_wait))) break;
                }
#pragma unroll
                for (int k = 0; k < kSums; ++k) acc[k] += __hiloint2double(static_cast<int>(v[2 * k + 1]), static_cast<int>(v[2 * k]));
            }
#pragma unroll
            for (int k = 0; k < kSums; ++k) {
                acc[k] = warp_sum(acc[k]);
                if (lane == 0) all[warp][k] = acc[k];
            }
        }
        __syncthreads();
        T sums[kSums] = {0, 0};
#pragma unroll
        for (int c = 0; c < kPcgSumCopies; ++c)
#pragma unroll
            for (int k = 0; k < kSums; ++k) sums[k] += static_cast<T>(all[c][k]);
        if (halo_failed || *static_cast<volatile int*>(&flag[1]) != 0) {
            status = SMOKE_B200_SOLVE_BARRIER_TIMEOUT;
            break;
        }
        const T gn = sums[0], dn = sums[1];
        rr = gn;
        if (first) {
            bb = gn;  // r = b
            if (!(bb > T(0))) {  // b = 0 (the solution is 0, as x is) or not finite
                it = A.iterations;
                if (!isfinite(bb)) status = SMOKE_B200_SOLVE_NOT_FINITE;
                rr = 0;
                break;
            }
        } else {
            ++it;
        }
        if (!isfinite(gn) || !isfinite(dn)) {
            status = SMOKE_B200_SOLVE_NOT_FINITE;
            break;
        }
        if (it >= A.iterations) break;
        if (first) {
            alpha = fabs(dn) > guard ? gn / dn : T(0);
        } else {
            beta = fabs(gamma) > guard ? gn / gamma : T(0);
            const T den = alpha != T(0) ? dn - beta * gn / alpha : dn;
            alpha = fabs(den) > guard ? gn / den : T(0);
        }
        gamma = gn;
    }
    if (blockIdx.x == 0 && tid == 0) {
        PcgStatusDevice st{};
        st.iterations = it;
        st.passes = 1;
        st.status = status;
        st.rhs_norm = sqrt(static_cast<double>(bb));
        st.relative_residual = bb > T(0) ? sqrt(static_cast<double>(rr) / static_cast<double>(bb)) : 0.0;
        st.true_relative_residual = -1.0;
        A.ctl->status = st;
        // the next launch's tags continue from here: every block read the epoch before its first words, which this block has
        // seen (or has given up on: then skip the tag of the exchange that may be under way)
        A.ctl->epoch = phase + 4u;
    }
}

// Grids of at most 16 blocks run as one thread-block cluster: its blocks are resident together by definition, and on
// neighbouring SMs, where a word is on its way for less time and one barrier starts them together (cluster_sync). 32^3, 16
// blocks, a step: 472 us without the cluster, 330 with it.
constexpr int kClusterBlocks = 16;

template <typename T, int M>
cudaError_t launch_one(const ResidentArgs& A, cudaStream_t s) {
    static std::mutex lock;
    static std::map<int, cudaError_t> configured;            // per device
    static std::map<std::pair<int, int>, bool> one_cluster;  // per device and block count
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(A.plan.blocks);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = resident_smem(A.plan.planes);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    bool cluster = false;
    {
        std::lock_guard<std::mutex> guard(lock);
        auto it = configured.find(dev);
        if (it == configured.end()) {
            e = cudaFuncSetAttribute(pcg_resident_kernel<T, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(resident_smem(M)));
            if (e == cudaSuccess) e = cudaFuncSetAttribute(pcg_resident_kernel<T, M>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            it = configured.emplace(dev, e).first;
        }
        if (it->second != cudaSuccess) return it->second;
        if (A.plan.blocks > 1 && A.plan.blocks <= kClusterBlocks) {
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim = {static_cast<unsigned>(A.plan.blocks), 1u, 1u};
            auto c = one_cluster.find({dev, A.plan.blocks});
            if (c == one_cluster.end()) {
                int clusters = 0;
                const bool ok = cudaOccupancyMaxActiveClusters(&clusters, pcg_resident_kernel<T, M>, &cfg) == cudaSuccess && clusters > 0;
                if (!ok) cudaGetLastError();  // a block count the device does not take as a cluster
                c = one_cluster.emplace(std::make_pair(dev, A.plan.blocks), ok).first;
            }
            cluster = c->second;
        }
    }
    if (!cluster) {
        attr[0] = cudaLaunchAttribute{};
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    }
    return cudaLaunchKernelEx(&cfg, pcg_resident_kernel<T, M>, A);
}

template <typename T>
cudaError_t launch_planes(const ResidentArgs& A, cudaStream_t s) {
    if (A.plan.planes <= 9) return launch_one<T, 9>(A, s);
    if (A.plan.planes <= 32) return launch_one<T, 32>(A, s);
    return launch_one<T, kPcgResidentPlanes>(A, s);
}

}  // namespace

PcgResidentPlan pcg_resident_plan(int nx, int ny, int nz, int sms) {
    PcgResidentPlan p{};
    p.ncx = (nx + CX - 1) / CX;
    p.ncy = (ny + CY - 1) / CY;
    p.total = static_cast<uint32_t>(p.ncx) * static_cast<uint32_t>(p.ncy) * static_cast<uint32_t>(nz);
    // the streaming kernel's blocks at one per SM: at least 8 planes each
    const uint32_t want = p.total / 8u > 0u ? p.total / 8u : 1u;
    p.blocks = static_cast<int>(want < static_cast<uint32_t>(sms) ? want : static_cast<uint32_t>(sms));
    p.planes = static_cast<int>((p.total + p.blocks - 1) / p.blocks);
    // at most two columns meet in a block when it has no more planes than a column
    if (p.planes > kPcgResidentPlanes || p.planes > nz) p.blocks = 0;
    return p;
}

size_t pcg_exchange_bytes(const PcgResidentPlan& p) {
    if (p.blocks == 0) return 0;
    const size_t z_slots = 2 * static_cast<size_t>(p.blocks) + 2 * static_cast<size_t>(p.ncx) * p.ncy;
    return 2 * (static_cast<size_t>(p.blocks) * kSumWords + static_cast<size_t>(p.total) * kSideWords + z_slots * kThreads) * sizeof(unsigned long long);
}

cudaError_t launch_pcg_resident(const StepParams& P, const PcgSettings& S, const PcgResidentPlan& plan, const uint16_t* codes, const float* b, float* x, const PcgWork& work, PcgControl* ctl, cudaStream_t s) {
    ResidentArgs A{};
    A.nx = P.nx;
    A.ny = P.ny;
    A.nz = P.nz;
    for (int a = 0; a < 3; ++a) A.per[a] = P.fper[a];
    A.plan = plan;
    A.codes = codes;
    A.b = b;
    A.x = x;
    A.exchange = work.exchange;
    A.ctl = ctl;
    A.iterations = S.max_iterations;
    A.withhold_block = S.withhold_block;
    A.withhold_exchange = S.withhold_exchange;
    A.barrier_timeout_ms = S.barrier_timeout_ms;
    const cudaError_t e = cudaMemsetAsync(ctl, 0, kPcgControlResetBytes, s);
    if (e != cudaSuccess) return e;
    return S.fp64 ? launch_planes<double>(A, s) : launch_planes<float>(A, s);
}

}  // namespace smoke_b200
