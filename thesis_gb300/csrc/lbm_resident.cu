// Many time steps of one D2Q9 lattice in one launch, the populations held in
// shared memory.
//
// A small 2D lattice is bound by launches, not by work: a 128 x 128 step is
// 1 MB of L2 traffic and 4 warps per SM, but a launch per step took 4.1 us.
// Up to 2728 nodes per SM, with their halo (about 415,000 nodes on 152 SMs, the
// largest square 632 x 632), both population buffers fit the shared memory, so
// one cooperative launch runs all the steps of an lbm_step call: every block
// keeps a rectangular tile with a one-node halo and gathers from it, and only
// the populations that cross a tile's edge travel through L2.  Bound by one
// message flight per step where tiles are small and by FP32 issue where they
// are large; us a step, a launch per step and here: 61 x 47 MRT 4.1 and 1.5,
// 128^2 reference BGK 4.1 and 1.6, 256^2 4.1 and 1.8, 1024 x 256 TRT 6.4 and 2.7.
//
// Roles.  The `compute` threads update the tile's nodes, the edge nodes
// first; warps of `comm` threads then send the edge's outgoing populations
// and fetch the halo of the next step while the inner nodes are updated.  A
// message is one 8-byte word {population bits, tag} written and read with
// single relaxed accesses, so its arrival needs no fence and no flag: the
// reader polls the word itself until it carries the tag of the state it
// wants.  A tile reads its messages from slots of its own
// (mail[parity][tile][link], numbered by tile_link), side by side for the lanes
// that poll them: 128^2, 1000 steps 1.88 -> 1.60 ms against slots by destination
// node.  Every link that crosses a tile edge is sent and awaited in both
// directions, blocked or not: neighbouring tiles then advance in lockstep,
// neither can be two states ahead of the other, and two parities of the mailbox
// suffice.  The first step takes its halo from the entry state in global memory,
// the last writes the state (and rho, u when asked) there.
//
// Layout.  Direction d of the node at tile index t = lx + 1 + pitch (ly + 1)
// sits at d * PLANE + t of a buffer: with PLANE fixed at compile time a
// gather is nine loads at immediate offsets from three row addresses, and no
// edge case: halo cells outside the lattice hold nothing, but the links from
// them are blocked and replaced by the node's own population.
//
// Node arithmetic, boundary closures and encodings are those of the one-node
// step kernels (h_finish in physics mode, update_node in reference mode): the
// same results, bit for bit.  Every wait is bounded; a wait that gives up
// sets *err, which the host reports, and all blocks leave.
#include "lbm_resident.h"

#include <algorithm>

#include "lbm_step_x2.cuh"

namespace lbm {

namespace {

constexpr int PLANE = 2944;              // halo'd tile nodes a buffer holds per direction (desc packs t in 12 bits)
constexpr int MAX_COMPUTE = 512, MAX_COMM = 128, MSGS = 8;  // threads; messages per comm thread

__device__ __forceinline__ unsigned long long mail_load(const unsigned long long *q) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(q) : "memory");
    return v;
}
__device__ __forceinline__ void mail_store(unsigned long long *q, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(q), "l"(v) : "memory");
}

__device__ __forceinline__ unsigned pop_bits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ unsigned pop_bits(__half v) { return (unsigned)__half_as_ushort(v); }
__device__ __forceinline__ void pop_from(unsigned b, float &v) { v = __uint_as_float(b); }
__device__ __forceinline__ void pop_from(unsigned b, __half &v) { v = __ushort_as_half((unsigned short)b); }
__device__ __forceinline__ float pop_value(float v) { return v; }
__device__ __forceinline__ float pop_value(__half v) { return __half2float(v); }

// Nodes of the perimeter of a w x h tile, and the j-th of them: bottom row,
// top row, then the side columns.
__host__ __device__ __forceinline__ int tile_edges(int w, int h) {
    return h == 1 ? w : (w == 1 ? h : 2 * (w + h) - 4);
}
__device__ __forceinline__ void tile_edge(int j, int w, int h, int &lx, int &ly) {
    if (j < w) {
        lx = j;
        ly = 0;
    } else if (h > 1 && j < 2 * w) {
        lx = j - w;
        ly = h - 1;
    } else {
        j -= h > 1 ? 2 * w : w;
        const int ih = h - 2;
        lx = j < ih ? 0 : w - 1;
        ly = 1 + (j < ih ? j : j - ih);
    }
}
// The i-th node in update order: the perimeter, then the inner rows.
__device__ __forceinline__ void tile_order(int i, int edges, int w, int h, int &lx, int &ly) {
    if (i < edges) {
        tile_edge(i, w, h, lx, ly);
    } else {
        lx = 1 + (i - edges) % (w - 2);
        ly = 1 + (i - edges) / (w - 2);
    }
}

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

template <bool V>
struct Bool {
    static constexpr bool value = V;
};

// D2Q9 directions by run-time index.
__device__ __forceinline__ int lattice_c2x(int d) { return d == 1 || d == 5 || d == 8 ? 1 : (d == 3 || d == 6 || d == 7 ? -1 : 0); }
__device__ __forceinline__ int lattice_c2y(int d) { return d == 2 || d == 5 || d == 6 ? 1 : (d == 4 || d == 7 || d == 8 ? -1 : 0); }
__device__ __forceinline__ int lattice_o2(int d) { return d <= 4 ? (d + 1) % 4 + 1 : (d + 1 - 4) % 4 + 5; }

// A tile's share of one axis: [axis_begin(i), axis_begin(i + 1)) of n nodes
// cut g ways.
__device__ __forceinline__ int axis_begin(int i, int n, int g) { return (int)((long long)i * n / g); }

// The number of the link in direction d that leaves a tw x th tile from (lx,
// ly), among 6 (tw + th): three directions per node of each side, top, bottom,
// right, left; a corner's diagonal belongs to its row.
__host__ __device__ __forceinline__ int tile_link(int lx, int ly, int d, int cx, int cy, int tw, int th) {
    if (ly + cy >= th) return (d == 2 ? 0 : d - 4) * tw + lx;                      // 2 5 6
    if (ly + cy < 0) return (3 + (d == 4 ? 0 : d - 6)) * tw + lx;                  // 4 7 8
    const int q = cx > 0 ? (d == 1 ? 0 : (d == 5 ? 1 : 2)) : 3 + (d == 3 ? 0 : d - 5);  // 1 5 8, 3 6 7
    return 6 * tw + q * th + ly;
}

template <int COLL, int ST, bool PHYS>
__global__ void __launch_bounds__(MAX_COMPUTE + MAX_COMM, 1) resident_kernel(const __grid_constant__ ResidentArgs a) {
    using L = Lat<9>;
    using S = Store<ST>;
    using T = typename S::T;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x;
    const DynGeom g{a.p.nx, a.p.ny, a.p.nz, a.p.pitch};
    const int nx = g.nx, ny = g.ny;
    const int bx = blockIdx.x % a.gx, by = blockIdx.x / a.gx;
    const int x0 = axis_begin(bx, nx, a.gx), y0 = axis_begin(by, ny, a.gy);
    const int tw = axis_begin(bx + 1, nx, a.gx) - x0, th = axis_begin(by + 1, ny, a.gy) - y0;
    const int nt = tw * th, edges = tile_edges(tw, th), pitch = tw + 2;
    T *buf0 = (T *)smem_raw, *buf1 = buf0 + 9 * PLANE;
    uint32_t *desc = (uint32_t *)(buf1 + 9 * PLANE);  // flag word | t << 20, in update order

    // a coordinate beyond the lattice: wrapped, or false
    auto inside = [&](int &x, int &y) -> bool {
        if (x >= 0 && x < nx && y >= 0 && y < ny) return true;
        if (!a.wrap) return false;
        x = x < 0 ? x + nx : (x >= nx ? x - nx : x);
        y = y < 0 ? y + ny : (y >= ny ? y - ny : y);
        return true;
    };
    for (int i = tid; i < nt; i += blockDim.x) {
        int lx, ly;
        tile_order(i, edges, tw, th, lx, ly);
        desc[i] = (__ldg(a.p.word + x0 + lx + nx * (y0 + ly)) & 0xFFFFFu) | ((unsigned)(lx + 1 + pitch * (ly + 1)) << 20);
    }
    // the entry state with its halo
    for (int i = tid; i < pitch * (th + 2); i += blockDim.x) {
        int x = x0 - 1 + i % pitch, y = y0 - 1 + i / pitch;
        if (!inside(x, y)) continue;
        const T *in = (const T *)a.p.fin[0] + x + (long long)g.pitch * y;
#pragma unroll
        for (int d = 0; d < 9; ++d) buf0[d * PLANE + i] = in[d * nx];
    }
    __syncthreads();

    const int edge_threads = min((edges + 31) / 32 * 32, a.compute);
    const int bar_threads = edge_threads + (int)blockDim.x - a.compute;

    if (tid < a.compute) {
        // the boundary record of this thread's first node, which it updates in
        // every step: three dependent loads and the conversions of its FP64
        // velocity off the steps' critical path
        SlotInfo slot;
        if (tid < nt && (desc[tid] & W_SPECIAL)) {
            const int t = desc[tid] >> 20;
            slot = load_slot<PHYS>(a.p, x0 - 1 + t % pitch + nx * (y0 - 1 + t / pitch));
        }
        // A node's streamed populations: pulled, or its own across a blocked link.
        auto gather = [&](const T *c, uint32_t w, T (&raw)[9]) {
            const T *lo = c - pitch, *hi = c + pitch;
            raw[0] = c[0];
            raw[1] = c[PLANE - 1];
            raw[2] = lo[2 * PLANE];
            raw[3] = c[3 * PLANE + 1];
            raw[4] = hi[4 * PLANE];
            raw[5] = lo[5 * PLANE - 1];
            raw[6] = lo[6 * PLANE + 1];
            raw[7] = hi[7 * PLANE + 1];
            raw[8] = hi[8 * PLANE - 1];
            if (w & 0x1FEu) {
#pragma unroll
                for (int d = 1; d < 9; ++d)
                    if ((w >> d) & 1u) raw[d] = c[(PHYS ? L::opp(d) : d) * PLANE];
            }
        };
        // One step of this thread's nodes; LAST writes to global memory.
        auto nodes = [&](const StepParams &p, const T *in, T *out, auto last_tag) {
            constexpr bool LAST = decltype(last_tag)::value;
            auto node_step = [&](int i, const SlotInfo *pre) {
                const uint32_t u = desc[i], w = u & 0xFFFFFu;
                const int t = u >> 20;
                T raw[9];
                gather(in + t, w, raw);
                int node = 0;
                if (LAST || (w & W_SPECIAL)) node = x0 - 1 + t % pitch + nx * (y0 - 1 + t / pitch);
                T res[9];
                if (w & W_FLUID) {
                    if constexpr (PHYS) {
                        f1 h[9];
#pragma unroll
                        for (int d = 0; d < 9; ++d) h[d] = f1(pop_value(raw[d]));
                        h_finish<9, COLL, ST, true, true, DynGeom>(p, g, node, w, h, pre);
#pragma unroll
                        for (int d = 0; d < 9; ++d) h_put<ST>(&res[d], h[d].v);
                    } else {
                        float f[9];
#pragma unroll
                        for (int d = 0; d < 9; ++d) f[d] = S::decode(raw[d], p.shift[d], p.inv_scale);
                        update_node<9, COLL, ST, false, true, DynGeom>(f, w, node, p, g, pre);
#pragma unroll
                        for (int d = 0; d < 9; ++d) res[d] = S::encode(f[d], p.shift[d], p.scale);
                    }
                } else if constexpr (PHYS) {
                    const float S0 = ST == LBM_STORE_F16S ? p.scale : 1.f;
#pragma unroll
                    for (int d = 0; d < 9; ++d) h_put<ST>(&res[d], -p.sigma * p.shift[d] * S0);
                } else {
                    // as the f-space kernels: +0 unshifted, where the above is -0
#pragma unroll
                    for (int d = 0; d < 9; ++d) res[d] = S::encode(0.f, p.shift[d], p.scale);
                }
                if constexpr (LAST) {
                    T *o = (T *)p.fout[0] + node % nx + (long long)g.pitch * (node / nx);
#pragma unroll
                    for (int d = 0; d < 9; ++d) o[d * nx] = res[d];
                } else {
#pragma unroll
                    for (int d = 0; d < 9; ++d) out[d * PLANE + t] = res[d];
                }
            };
            if (tid < nt) node_step(tid, &slot);
            if constexpr (!LAST) {
                // the perimeter lies in the first round: hand it over
                if (tid < edge_threads) {
                    __syncwarp();
                    bar_arrive(1, bar_threads);
                }
            }
            int i = tid + a.compute;
            if constexpr (PHYS && !LAST) {
                // the inner rounds two at a time on packed FP32x2
#pragma unroll 1
                for (; i + a.compute < nt; i += 2 * a.compute) {
                    const uint32_t ua = desc[i], ub = desc[i + a.compute];
                    if ((ua | ub) & W_SPECIAL) {
                        node_step(i, nullptr);
                        node_step(i + a.compute, nullptr);
                        continue;
                    }
                    const bool fa = ua & W_FLUID, fb = ub & W_FLUID;
                    const int ta = ua >> 20, tb = ub >> 20;
                    const T *ca = in + ta, *cb = in + tb;
                    T ra[9], rb[9];
                    gather(ca, ua, ra);
                    gather(cb, ub, rb);
                    f2 h[9];
#pragma unroll
                    for (int d = 0; d < 9; ++d) h[d] = f2(fa ? pop_value(ra[d]) : 0.f, fb ? pop_value(rb[d]) : 0.f);
                    h_pair_relax<9, COLL, ST, true>(p, 0, 0, fa, fb, h);
                    const float S0 = ST == LBM_STORE_F16S ? p.scale : 1.f;
#pragma unroll
                    for (int d = 0; d < 9; ++d) {
                        const float zero = -p.sigma * p.shift[d] * S0;
                        h_put<ST>(out + d * PLANE + ta, fa ? h[d].v.x : zero);
                        h_put<ST>(out + d * PLANE + tb, fb ? h[d].v.y : zero);
                    }
                }
            }
#pragma unroll 1
            for (; i < nt; i += a.compute) node_step(i, nullptr);
        };
#pragma unroll 1
        for (int s = 0; s < a.steps - 1; ++s) {
            nodes(a.p, s & 1 ? buf1 : buf0, s & 1 ? buf0 : buf1, Bool<false>{});
            if (__syncthreads_or(0)) return;
        }
        nodes(a.last, (a.steps - 1) & 1 ? buf1 : buf0, nullptr, Bool<true>{});
    } else {
        // This thread's messages: out_s / in_s the place in a buffer, out_m /
        // in_m the word in the mailbox.
        int out_s[MSGS], out_m[MSGS], in_s[MSGS], in_m[MSGS];
#pragma unroll
        for (int k = 0; k < MSGS; ++k) out_s[k] = in_s[k] = -1;
        // the links by number (tile_link)
#pragma unroll
        for (int k = 0; k < MSGS; ++k) {
            const int link = tid - a.compute + k * ((int)blockDim.x - a.compute);
            int m = link, lx, ly, d;
            if (m < 6 * tw) {
                const bool top = m < 3 * tw;
                const int j = top ? m : m - 3 * tw, q = j / tw;
                lx = j - q * tw;
                ly = top ? th - 1 : 0;
                d = top ? (q == 0 ? 2 : 4 + q) : (q == 0 ? 4 : 6 + q);  // 2 5 6, 4 7 8
            } else if (m < 6 * (tw + th)) {
                m -= 6 * tw;
                const bool right = m < 3 * th;
                const int j = right ? m : m - 3 * th, q = j / th;
                ly = j - q * th;
                lx = right ? tw - 1 : 0;
                d = right ? (q == 0 ? 1 : (q == 1 ? 5 : 8)) : (q == 0 ? 3 : 5 + q);  // 1 5 8, 3 6 7
                const int cy = lattice_c2y(d);
                if (ly + cy < 0 || ly + cy >= th) continue;
            } else {
                continue;
            }
            const int cx = lattice_c2x(d), cy = lattice_c2y(d);
            // out: direction d of (lx, ly) to the node at c_d
            int x = x0 + lx + cx, y = y0 + ly + cy;
            if (!inside(x, y)) continue;
            out_s[k] = d * PLANE + lx + 1 + pitch * (ly + 1);
            // the tile it lies in, and the link's number there, where it leaves in the
            // opposite direction
            const int o = lattice_o2(d);
            const int ox = lx + cx < 0 ? (bx + a.gx - 1) % a.gx : (lx + cx >= tw ? (bx + 1) % a.gx : bx);
            const int oy = ly + cy < 0 ? (by + a.gy - 1) % a.gy : (ly + cy >= th ? (by + 1) % a.gy : by);
            const int ox0 = axis_begin(ox, nx, a.gx), oy0 = axis_begin(oy, ny, a.gy);
            out_m[k] = (ox + a.gx * oy) * a.links + tile_link(x - ox0, y - oy0, o, -cx, -cy,
                                                              axis_begin(ox + 1, nx, a.gx) - ox0,
                                                              axis_begin(oy + 1, ny, a.gy) - oy0);
            // in: that direction over the same link, from the halo
            in_s[k] = o * PLANE + lx + cx + 1 + pitch * (ly + cy + 1);
            in_m[k] = (int)blockIdx.x * a.links + link;
        }
#pragma unroll 1
        for (int s = 0; s < a.steps - 1; ++s) {
            T *out = s & 1 ? buf0 : buf1;
            unsigned long long *mail = a.mail + (size_t)((s + 1) & 1) * (gridDim.x * a.links);
            const unsigned tag = a.tag + (unsigned)s + 1u;
            bar_sync(1, bar_threads);
#pragma unroll
            for (int k = 0; k < MSGS; ++k)
                if (out_s[k] >= 0)
                    mail_store(mail + out_m[k], ((unsigned long long)tag << 32) | pop_bits(out[out_s[k]]));
            unsigned need = 0;
#pragma unroll
            for (int k = 0; k < MSGS; ++k) need |= in_s[k] >= 0 ? 1u << k : 0u;
            bool bad = false;
            unsigned look = min(a.polls, 1023u);  // the next poll after which to look at the limit and at *err
#pragma unroll 1
            for (unsigned spin = 0; need; ++spin) {
                unsigned long long v[MSGS];
#pragma unroll
                for (int k = 0; k < MSGS; ++k)
                    if ((need >> k) & 1u) v[k] = mail_load(mail + in_m[k]);
#pragma unroll
                for (int k = 0; k < MSGS; ++k)
                    if (((need >> k) & 1u) && (unsigned)(v[k] >> 32) == tag) {
                        need &= ~(1u << k);
                        pop_from((unsigned)v[k], out[in_s[k]]);
                    }
                if (spin >= look) {
                    if (!need) break;
                    look += 1024u;
                    if (spin >= a.polls || *(volatile unsigned *)a.err) {
                        bad = true;
                        break;
                    }
                }
            }
            if (bad) *(volatile unsigned *)a.err = 1u;
            if (__syncthreads_or(bad)) return;
        }
    }
}

using ResidentKernel = void (*)(const ResidentArgs);

ResidentKernel resident_kernel_of(int coll, int st, int phys) {
#define R_CASE(C, S, P) \
    if (coll == C && st == S && (phys != 0) == P) return resident_kernel<C, S, P>;
    R_CASE(1, 0, false) R_CASE(2, 0, false) R_CASE(3, 0, false) R_CASE(1, 0, true) R_CASE(2, 0, true)
    R_CASE(3, 0, true) R_CASE(1, 1, true) R_CASE(2, 1, true) R_CASE(3, 1, true)
#undef R_CASE
    return nullptr;
}

}  // namespace

bool resident_plan(int nx, int ny, int elem, int sms, ResidentPlan *out) {
    const long long N = (long long)nx * ny;
    // tiles of at least RES_MIN_NODES nodes: smaller ones only add edges
    constexpr int RES_MIN_NODES = 96;
    if (N > (long long)sms * PLANE) return false;
    const long long want = std::min<long long>(sms, std::max<long long>(1, N / RES_MIN_NODES));
    // the cut with the least largest tile, an edge node (its messages)
    // counted as two nodes
    long long best = -1;
    int nt = 0, edges = 0;
    for (int gx = 1; gx <= want && gx <= nx; ++gx) {
        const int gy = (int)std::min<long long>(want / gx, ny);
        const int tw = (nx + gx - 1) / gx, th = (ny + gy - 1) / gy;
        if ((long long)(tw + 2) * (th + 2) > PLANE) continue;
        if (6 * (tw + th) > MAX_COMM * MSGS || tile_edges(tw, th) > MAX_COMPUTE) continue;
        const long long cost = (long long)tw * th + 2 * (tw + th);
        if (best < 0 || cost < best) {
            best = cost;
            out->gx = gx;
            out->gy = gy;
            nt = tw * th;
            edges = tile_edges(tw, th);
            out->links = 6 * (tw + th);
            out->comm = std::min(MAX_COMM, (out->links + 31) / 32 * 32);
        }
    }
    if (best < 0) return false;
    const int rounds = (nt + MAX_COMPUTE - 1) / MAX_COMPUTE;
    out->compute = std::max((nt + rounds - 1) / rounds, edges);
    out->compute = (out->compute + 31) / 32 * 32;
    out->smem = (size_t)PLANE * (18 * elem + 4);
    return true;
}

const void *resident_prepare(int coll, int st, int phys, const ResidentPlan &plan) {
    ResidentKernel k = resident_kernel_of(coll, st, phys);
    if (!k) return nullptr;
    int bps = 0;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plan.smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k, plan.compute + plan.comm, plan.smem) != cudaSuccess ||
        bps < 1) {
        cudaGetLastError();
        return nullptr;
    }
    return (const void *)k;
}

int resident_launch(const void *kern, const ResidentPlan &plan, const ResidentArgs &a, cudaStream_t s) {
    void *args[] = {(void *)&a};
    return (int)cudaLaunchCooperativeKernel(kern, dim3((unsigned)(plan.gx * plan.gy)),
                                            dim3((unsigned)(plan.compute + plan.comm)), args, plan.smem, s);
}

}  // namespace lbm
