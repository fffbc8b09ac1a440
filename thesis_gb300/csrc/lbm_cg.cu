// Colour-gradient two-phase D2Q9 on a periodic lattice (the reference's
// multiphase 2D path: gpuCollBgkwGC2D / gpuCollEnhancedBgkwGC2D,
// GpuCollision.cu:552-707; gpuStreaming2DCG, GpuStream.cu:30-158;
// gpuUpdateMacro2DCG, GpuUpdateMacro.cu:43-135; Laplace-law sums,
// Iterate.cu:496-499).
//
// The collision of a node needs the colour field phi = (rho_r - rho_b)/rho of
// its 8 (3x3 stencil) or 24 (5x5 stencil) neighbours after streaming.  One
// launch does a step: a block owns a tile of nodes, pulls both colours of each
// into registers, and of a ring of 1 (or 2) nodes around the tile pulls them
// only to form phi and rho; those meet in shared memory for the gradients,
// and the collision, perturbation and recolouring continue from the registers.
// State between steps: post-collision red and blue populations, SoA by
// direction, pull double buffer.  HBM-bound: 72 B of populations read and 72 B
// written per node in FP32; the ring's loads (1.33x with a 32 x 8 tile) are the
// neighbouring blocks' own and hit L2.  In practice the issue of about 900
// instructions per 32 nodes binds it (73 % of issue slots): 1024^2, FP32, 52 us
// a step in two launches that pulled twice, 40 us in one; F16S 54 and 42 us.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <new>
#include <string>
#include <vector>

#include "lbm_cg3.cuh"
#include "lbm_cg_store.cuh"
#include "lbm_device.cuh"
#include "thesis_lbm.h"

namespace lbm {
namespace {

template <class V>
struct CgArgs {
    CgSlots<9> s;            // lbm_cg_store.cuh
    float *R, *B;            // colour densities (output, when write_rb)
    float *rho, *ux, *uy;    // macroscopic output (when write_macro)
    int nx, ny;
    long long N;
    int write_macro, write_rb;
    CgModel<V> p;
};

// Tile of a block, 32 x TY nodes, one per thread, and the blocks per SM the step
// kernel is compiled for.  FP32 and 16-bit storage: TY = 8 at 40 registers (six
// blocks of 256 threads).  F64 is bound by FP64 operations and would spill 212
// to 384 bytes at 40; it takes 80 registers and one of two heights (cg_tile_f64).
constexpr int CG_TX = 32;
constexpr int cg_resident(int st, int ty) { return st == LBM_STORE_F64 ? (ty == 8 ? 3 : 6) : 6; }
// rest weights phi_k + theta_k alpha; in constant memory, where they cost an
// operand: as literals they change which products the compiler fuses, and so
// the last bits of a droplet's small velocities
__constant__ float c_phi[9] = {0.f, 0.2f, 0.2f, 0.2f, 0.2f, 0.05f, 0.05f, 0.05f, 0.05f};
__constant__ float c_teta[9] = {1.f, -0.2f, -0.2f, -0.2f, -0.2f, -0.05f, -0.05f, -0.05f, -0.05f};
__constant__ double c_phi_d[9] = {0., 0.2, 0.2, 0.2, 0.2, 0.05, 0.05, 0.05, 0.05};
__constant__ double c_teta_d[9] = {1., -0.2, -0.2, -0.2, -0.2, -0.05, -0.05, -0.05, -0.05};

template <class R> __device__ __forceinline__ R cg_rest_phi(int k) {
    if constexpr (sizeof(R) == 8) return c_phi_d[k];
    else return c_phi[k];
}
template <class R> __device__ __forceinline__ R cg_rest_teta(int k) {
    if constexpr (sizeof(R) == 8) return c_teta_d[k];
    else return c_teta[k];
}

__device__ __forceinline__ int wrapi(int a, int n) { return a < 0 ? a + n : (a >= n ? a - n : a); }

// PULL: gather from the neighbours (a time step); otherwise read the node's
// own populations (the first collision from a given post-stream state).  Node
// indices are unsigned 32-bit (fewer than 2^31 nodes), added to a base per
// direction that is the same for every thread: no 64-bit index per load.
template <int ST, bool PULL>
__device__ __forceinline__ void cg_gather(const CgArgs<typename CgStore<ST>::R> &a, int x, int y,
                                          typename CgStore<ST>::R (&r)[9], typename CgStore<ST>::R (&b)[9]) {
    using L = Lat<9>;
    using S = CgStore<ST>;
    using T = typename S::T;
    using R = typename S::R;
    const unsigned X[3] = {(unsigned)(x == 0 ? a.nx - 1 : x - 1), (unsigned)x, (unsigned)(x == a.nx - 1 ? 0 : x + 1)};
    const unsigned Y[3] = {(unsigned)a.nx * (unsigned)(y == 0 ? a.ny - 1 : y - 1), (unsigned)a.nx * (unsigned)y,
                           (unsigned)a.nx * (unsigned)(y == a.ny - 1 ? 0 : y + 1)};
#pragma unroll
    for (int d = 0; d < 9; ++d) {
        const unsigned s = PULL ? X[1 - L::cx(d)] + Y[1 - L::cy(d)] : X[1] + Y[1];
        S::load((const T *)a.s.in[d] + s, (const T *)a.s.in[9 + d] + s, (R)L::w(d), a.p.inv_scale, r[d], b[d]);
    }
}

template <int ST, int TY, bool PULL, bool HO, bool ENH>
__global__ void __launch_bounds__(CG_TX * TY, cg_resident(ST, TY)) cg_step_kernel(const CgArgs<typename CgStore<ST>::R> a) {
    using L = Lat<9>;
    using SP = CgStore<ST>;
    using T = typename SP::T;
    using R = typename SP::R;
    constexpr int H = HO ? 2 : 1, W = CG_TX + 2 * H, RING = 2 * H * W + 2 * H * TY;
    __shared__ R s_phi[(TY + 2 * H) * W];
    __shared__ R s_dn[ENH ? (TY + 2 * H) * W : 1];
    const int tid = threadIdx.x, lx = tid % CG_TX, ly = tid / CG_TX;
    const int x0 = blockIdx.x * CG_TX, y0 = blockIdx.y * TY, x = x0 + lx, y = y0 + ly;
    // colour field and density of tile position (cx, cy), from -H; past a
    // lattice face the position is the wrapped node's
    auto put = [&](int cx, int cy, R rr, R bb) {
        const R rho = rr + bb;
        const int c = (cy + H) * W + cx + H;
        s_phi[c] = (rr - bb) / rho;
        if (ENH) s_dn[c] = rho;
    };
    R f[9], r_r = 0, b_r = 0, jx = 0, jy = 0;
    {
        const bool own = x < a.nx && y < a.ny;
        if (x < a.nx + H && y < a.ny + H) {
            R r[9], b[9];
            cg_gather<ST, PULL>(a, own ? x : wrapi(x, a.nx), own ? y : wrapi(y, a.ny), r, b);
#pragma unroll
            for (int d = 0; d < 9; ++d) {
                f[d] = r[d] + b[d];
                r_r += r[d];
                b_r += b[d];
                if (L::cx(d)) jx += (R)L::cx(d) * f[d];
                if (L::cy(d)) jy += (R)L::cy(d) * f[d];
            }
            put(lx, ly, r_r, b_r);
        }
#pragma unroll 1
        for (int t = tid; t < RING; t += CG_TX * TY) {
            // rows below and above the tile, then the columns beside it
            int cx, cy;
            if (t < 2 * H * W) {
                const int row = t / W;
                cx = t % W - H;
                cy = row < H ? row - H : TY + row - H;
            } else {
                const int j = t - 2 * H * W, col = j / TY;
                cx = col < H ? col - H : CG_TX + col - H;
                cy = j % TY;
            }
            const int gx = x0 + cx, gy = y0 + cy;
            if (gx < a.nx + H && gy < a.ny + H) {
                R r[9], b[9];
                cg_gather<ST, PULL>(a, wrapi(gx, a.nx), wrapi(gy, a.ny), r, b);
                R rr = 0, bb = 0;
#pragma unroll
                for (int d = 0; d < 9; ++d) {
                    rr += r[d];
                    bb += b[d];
                }
                put(cx, cy, rr, bb);
            }
        }
        __syncthreads();
        if (!own) return;
    }
    const int node = x + a.nx * y;
    const R *phi = s_phi + (ly + H) * W + lx + H, *dn = s_dn + (ENH ? (ly + H) * W + lx + H : 0);
    const R rho = r_r + b_r;
    const R u = jx / rho, v = jy / rho;
    if (a.write_rb) {
        a.R[node] = (float)r_r;
        a.B[node] = (float)b_r;
    }
    if (a.write_macro) {
        a.rho[node] = (float)rho;
        a.ux[node] = (float)u;
        a.uy[node] = (float)v;
    }
    // colour and density gradients from the neighbours (GpuCollision.cu:112-281)
    R cgx = 0, cgy = 0, grx = 0, gry = 0;
    if (HO) {
        constexpr int hx[24] = {1, 0, -1, 0, 1, -1, -1, 1, 0, 1, 2, 2, 2, 2, 2, 1, 0, -1, -2, -2, -2, -2, -2, -1};
        constexpr int hy[24] = {0, 1, 0, -1, 1, 1, -1, -1, 2, 2, 2, 1, 0, -1, -2, -2, -2, -2, -2, -1, 0, 1, 2, 2};
        constexpr double hw[24] = {960., 960., 960., 960., 448., 448., 448., 448., 84., 32., 1., 32.,
                                   84.,  32.,  1.,   32.,  84.,  32.,  1.,   32.,  84., 32., 1., 32.};
#pragma unroll
        for (int k = 0; k < 24; ++k) {
            const int j = hx[k] + W * hy[k];
            const R w = (R)(hw[k] / 5040.0);
            const R a1 = w * phi[j], a2 = ENH ? w * dn[j] : (R)0;
            if (ENH) {
                grx += a2 * (R)hx[k];
                gry += a2 * (R)hy[k];
            }
            cgx += a1 * (R)hx[k];
            cgy += a1 * (R)hy[k];
        }
    } else {
#pragma unroll
        for (int k = 1; k < 9; ++k) {
            const int j = L::cx(k) + W * L::cy(k);
            const R w = k <= 4 ? (R)(4.0 / 12.0) : (R)(1.0 / 12.0);
            const R a1 = w * phi[j], a2 = ENH ? w * dn[j] : (R)0;
            if (ENH) {
                grx += a2 * (R)L::cx(k);
                gry += a2 * (R)L::cy(k);
            }
            cgx += a1 * (R)L::cx(k);
            cgy += a1 * (R)L::cy(k);
        }
    }
    const R r_visc = a.p.r_visc, b_visc = a.p.b_visc, beta = a.p.beta, A = a.p.A;
    const R mean_nu = (R)1 / (r_r / (rho * r_visc) + b_r / (rho * b_visc));
    const R omega_eff = (R)1 / ((R)3 * mean_nu + (R)0.5);
    const R mean_alpha = a.p.r_alpha * r_r / rho + a.p.b_alpha * b_r / rho;
    const R gnorm = sqrt(cgx * cgx + cgy * cgy);
    const R k_r = r_r / rho, k_b = b_r / rho, k_k = beta * r_r * b_r / rho;
    const R cu1 = u * u + v * v;
    const R G1 = (R)2 * u * grx, G2 = u * gry + v * grx, G4 = (R)2 * v * gry;
    const R ugr = u * grx + v * gry;
    const bool interface = gnorm > a.p.g_limit;
    // one reciprocal per node instead of two divisions per direction
    const R inv_g = interface ? (R)1 / gnorm : (R)0, inv_g2 = inv_g * inv_g;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const R cxk = (R)L::cx(k), cyk = (R)L::cy(k);
        const R wk = k == 0 ? (R)(4. / 9.) : (k <= 4 ? (R)(1. / 9.) : (R)(1. / 36.));
        R pert = 0, cosin = 0;
        if (interface) {
            const R pcg = cxk * cgx + cyk * cgy;
            if (k != 0) cosin = pcg * inv_g * (k <= 4 ? (R)1 : (R)0.70710678118654752);
            const R bk = k == 0 ? (R)(-4. / 27.) : (k <= 4 ? (R)(2. / 27.) : (R)(5. / 108.));
            pert = A * gnorm * (wk * (pcg * pcg) * inv_g2 - bk);
        }
        const R cu2 = u * cxk + v * cyk;
        const R rest = cg_rest_phi<R>(k) + cg_rest_teta<R>(k) * mean_alpha;
        R feq = rho * (rest + wk * ((R)3 * cu2 + (R)4.5 * cu2 * cu2 - (R)1.5 * cu1));
        if (ENH) {
            const R chi = k == 0 ? (R)(-8. / 3.) : (k <= 4 ? (R)(-1. / 6.) : (R)(1. / 12.));
            const R psi = k == 0 ? (R)0 : (k <= 4 ? (R)0.5 : (R)0.125);
            const R TC = G1 * (cxk * cxk) + (R)2 * G2 * (cxk * cyk) + G4 * (cyk * cyk);
            feq += mean_nu * (chi * ugr + psi * TC);
        }
        const R fp = omega_eff * feq + ((R)1 - omega_eff) * f[k] + pert;
        SP::store((T *)a.s.out[k] + (unsigned)node, (T *)a.s.out[9 + k] + (unsigned)node, (R)L::w(k), a.p.scale,
                  k_r * fp + k_k * cosin * rest, k_b * fp - k_k * cosin * rest);
    }
}

// Post-streaming red and blue populations (FP32, SoA) into storage slots.
template <int ST>
__global__ void cg_encode_kernel(const float *r, const float *b, void *out, int q, long long N, float scale) {
    using SP = CgStore<ST>;
    using T = typename SP::T;
    using R = typename SP::R;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)q * N) return;
    const int d = (int)(i / N);
    const R w = q == 9 ? (R)Lat<9>::w(d) : (R)Lat<19>::w(d);
    T *o = (T *)out;
    SP::store(o + i, o + (long long)q * N + i, w, (R)scale, (R)r[i], (R)b[i]);
}

// Storage slots back to red and blue populations (FP32, SoA).
template <int ST>
__global__ void cg_decode_kernel(const void *in, float *r, float *b, int q, long long N, float inv_scale) {
    using SP = CgStore<ST>;
    using T = typename SP::T;
    using R = typename SP::R;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)q * N) return;
    const int d = (int)(i / N);
    const R w = q == 9 ? (R)Lat<9>::w(d) : (R)Lat<19>::w(d);
    const T *s = (const T *)in;
    R rr, bb;
    SP::load(s + i, s + (long long)q * N + i, w, (R)inv_scale, rr, bb);
    r[i] = (float)rr;
    b[i] = (float)bb;
}

// FP64 Laplace-law sums: sum rho_r and count where chi >= c, sum rho_b and
// count where chi <= -c, max |u| (Iterate.cu:496-499, GpuUpdateMacro.cu:122-133).
constexpr int LAP_BLOCKS = 304, LAP_THREADS = 256;
__global__ void __launch_bounds__(LAP_THREADS)
cg_laplace_partial(const float *R, const float *B, const float *ux, const float *uy, const float *uz, long long n,
                   float c, double *partial) {
    double acc[5] = {0, 0, 0, 0, 0};
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double r = R[i], b = B[i], chi = (r - b) / (r + b);
        if (chi >= c) {
            acc[0] += r;
            acc[1] += 1;
        } else if (chi <= -c) {
            acc[2] += b;
            acc[3] += 1;
        }
        const double wz = uz ? (double)uz[i] : 0.0;
        const double um = sqrt((double)ux[i] * ux[i] + (double)uy[i] * uy[i] + wz * wz);
        acc[4] = um > acc[4] ? um : acc[4];
    }
    __shared__ double sm[LAP_THREADS][5];
#pragma unroll
    for (int k = 0; k < 5; ++k) sm[threadIdx.x][k] = acc[k];
    __syncthreads();
    if (threadIdx.x < 5) {
        double s = 0;
        for (int t = 0; t < LAP_THREADS; ++t)
            s = threadIdx.x == 4 ? (sm[t][4] > s ? sm[t][4] : s) : s + sm[t][threadIdx.x];
        partial[blockIdx.x * 5 + threadIdx.x] = s;
    }
}

__global__ void cg_laplace_final(const double *partial, double *out) {
    if (threadIdx.x >= 5) return;
    double s = 0;
    for (int bI = 0; bI < LAP_BLOCKS; ++bI) {
        const double v = partial[bI * 5 + threadIdx.x];
        s = threadIdx.x == 4 ? (v > s ? v : s) : s + v;
    }
    out[threadIdx.x] = s;
}

thread_local std::string g_cg_error;
int cg_fail(int code, const std::string &m) {
    g_cg_error = m;
    return code;
}

}  // namespace
}  // namespace lbm

using namespace lbm;

struct lbm_cg_handle_s {
    int n = 0, m = 0, h = 1, q = 9;  // D2Q9 (h = 1) or D3Q19
    long long N = 0;
    lbm_cg_params P{};
    int st = LBM_STORE_F32;          // population storage (lbm_cg_store.cuh)
    void *buf = nullptr;             // 2 buffers x 2 slots x q directions x N values
    float *R = nullptr, *B = nullptr, *rho = nullptr, *ux = nullptr, *uy = nullptr, *uz = nullptr;
    void *phi = nullptr, *dn = nullptr;  // 3D, two launches per step: colour field and density (arithmetic type)
    double *partial = nullptr, *sums = nullptr;
    int cur = 0;
    int sms = 1;
    int tile = 8;                    // 2D: rows of a block's tile
    int planes = 1;                  // 3D, one launch per step: planes a block marches over
    float scale = 1024.f;            // F16S: scale of the summed population's deviation
    cudaStream_t stream = nullptr;
    cudaEvent_t stepped = nullptr;  // after the last lbm_cg_step, on its stream
    size_t slot_bytes() const { return (size_t)q * (size_t)N * cg_elem_bytes(st); }
    void *buffer(int c) const { return (char *)buf + (size_t)c * 2 * slot_bytes(); }
};

template <class A>
static void cg_fill_common(const lbm_cg_handle_s *H, int from, int write_macro, int write_rb, A &a) {
    const size_t one = (size_t)H->N * cg_elem_bytes(H->st);
    for (int k = 0; k < 2 * H->q; ++k) {
        a.s.in[k] = (const char *)H->buffer(from) + k * one;
        a.s.out[k] = (char *)H->buffer(1 - from) + k * one;
    }
    a.R = H->R;
    a.B = H->B;
    a.rho = H->rho;
    a.ux = H->ux;
    a.uy = H->uy;
    a.nx = H->n;
    a.ny = H->m;
    a.N = H->N;
    a.write_macro = write_macro;
    a.write_rb = write_rb;
    using R = decltype(a.p.A);
    a.p = CgModel<R>{(R)H->P.r_alpha, (R)H->P.b_alpha, (R)H->P.r_viscosity, (R)H->P.b_viscosity, (R)H->P.beta,
                     (R)H->P.A, (R)H->P.g_limit, (R)H->scale, (R)(1.0f / H->scale)};
}

template <class R>
static CgArgs<R> cg_args(const lbm_cg_handle_s *H, int from, int write_macro, int write_rb) {
    CgArgs<R> a;
    memset(&a, 0, sizeof(a));
    cg_fill_common(H, from, write_macro, write_rb, a);
    return a;
}

template <class R>
static Cg3Args<R> cg3_args(const lbm_cg_handle_s *H, int from, int write_macro, int write_rb) {
    Cg3Args<R> a;
    memset(&a, 0, sizeof(a));
    cg_fill_common(H, from, write_macro, write_rb, a);
    a.phi = H->phi;
    a.dn = H->dn;
    a.uz = H->uz;
    a.nz = H->h;
    return a;
}

// Where a 3D step is one launch (cg3_step_kernel): FP32 storage with the
// 18-neighbour gradient.  F16S, whose ring pulls cost conversions, and F64, whose
// registers spill, are faster in two launches; us a step, two / one: 128^3 F16S
// 170 / 211, F64 2890 / 3560, FP32 185 / 162; 96 x 90 x 80 F16S 60.7 / 73.9, F64
// 1016 / 1154, FP32 68.7 / 60.1 (160 x 131 x 97 F16S with the enhanced
// equilibrium is the one measured the other way, 217 / 212).
static constexpr bool cg3_one_launch(int st, int high_order) { return st == LBM_STORE_F32 && !high_order; }

// The planes a block marches over: the cut along z with the fewest plane steps
// in a row, waves of resident blocks times a block's planes and the two it pulls
// for phi alone (256^3: 10 blocks along z, against 1 that leaves a third of the
// SMs' places empty, 1.41 against 1.22 ms).
static int cg3_planes(const lbm_cg_handle_s *H) {
    const long long tiles = (long long)((H->n + CG3_TX - 1) / CG3_TX) * ((H->m + CG3_TY - 1) / CG3_TY);
    const long long places = (long long)H->sms * CG3_RESIDENT;
    int planes = H->h;
    long long best = -1;
    for (int c = 1; c <= (H->h + 1) / 2; ++c) {
        const int k = (H->h + c - 1) / c;
        const long long cost = (tiles * c + places - 1) / places * (k + 2);
        if (best < 0 || cost < best) {
            best = cost;
            planes = k;
        }
    }
    return planes;
}

template <int ST, bool PULL>
static void cg3_launch_st(const lbm_cg_handle_s *H, int from, int write_macro, int write_rb, cudaStream_t s) {
    const auto a = cg3_args<typename CgStore<ST>::R>(H, from, write_macro, write_rb);
    if (!cg3_one_launch(ST, H->P.high_order)) {
        const dim3 grid((unsigned)((H->n + CG3_BLOCK - 1) / CG3_BLOCK), (unsigned)H->m, (unsigned)H->h);
        cg3_density_kernel<ST, PULL><<<grid, CG3_BLOCK, 0, s>>>(a);
        if (H->P.high_order) {
            if (H->P.enhanced) cg3_collide_kernel<ST, PULL, true, true><<<grid, CG3_BLOCK, 0, s>>>(a);
            else cg3_collide_kernel<ST, PULL, true, false><<<grid, CG3_BLOCK, 0, s>>>(a);
        } else if constexpr (!cg3_one_launch(ST, 0)) {
            if (H->P.enhanced) cg3_collide_kernel<ST, PULL, false, true><<<grid, CG3_BLOCK, 0, s>>>(a);
            else cg3_collide_kernel<ST, PULL, false, false><<<grid, CG3_BLOCK, 0, s>>>(a);
        }
        return;
    }
    if constexpr (cg3_one_launch(ST, 0)) {
        const dim3 grid((unsigned)((H->n + CG3_TX - 1) / CG3_TX), (unsigned)((H->m + CG3_TY - 1) / CG3_TY),
                        (unsigned)((H->h + H->planes - 1) / H->planes));
        if (H->P.enhanced) cg3_step_kernel<ST, PULL, true><<<grid, CG3_TX * CG3_TY, 0, s>>>(a, H->planes);
        else cg3_step_kernel<ST, PULL, false><<<grid, CG3_TX * CG3_TY, 0, s>>>(a, H->planes);
    }
}

template <int ST, int TY, bool PULL>
static void cg_launch_tile(const lbm_cg_handle_s *H, int from, int write_macro, int write_rb, cudaStream_t s) {
    const auto a = cg_args<typename CgStore<ST>::R>(H, from, write_macro, write_rb);
    const dim3 grid((unsigned)((H->n + CG_TX - 1) / CG_TX), (unsigned)((H->m + TY - 1) / TY));
    if (H->P.high_order) {
        if (H->P.enhanced) cg_step_kernel<ST, TY, PULL, true, true><<<grid, CG_TX * TY, 0, s>>>(a);
        else cg_step_kernel<ST, TY, PULL, true, false><<<grid, CG_TX * TY, 0, s>>>(a);
    } else {
        if (H->P.enhanced) cg_step_kernel<ST, TY, PULL, false, true><<<grid, CG_TX * TY, 0, s>>>(a);
        else cg_step_kernel<ST, TY, PULL, false, false><<<grid, CG_TX * TY, 0, s>>>(a);
    }
}

// Tile height of an F64 step: the one whose busiest SM has the least work, in
// nodes, a ring node (one pull, no collision) counted as a sixteenth.  us a
// step, plain gradient, two launches / TY = 8 / TY = 4: 1024^2 791 / 769 / 785,
// 500 x 400 160 / 164 / 156, 200 x 180 49.5 / 55.6 / 45.5, 130 x 97 37.1 / 33.1 /
// 20.7.
static int cg_tile_f64(const lbm_cg_handle_s *H) {
    auto busiest = [&](int ty) {
        const long long tiles = (long long)((H->n + CG_TX - 1) / CG_TX) * ((H->m + ty - 1) / ty);
        const int r = H->P.high_order ? 2 : 1, ring = 2 * r * (CG_TX + 2 * r + ty);
        return (tiles + H->sms - 1) / H->sms * (16 * CG_TX * ty + ring);
    };
    return busiest(8) <= busiest(4) ? 8 : 4;
}

template <int ST, bool PULL>
static void cg_launch_st(const lbm_cg_handle_s *H, int from, int write_macro, int write_rb, cudaStream_t s) {
    if constexpr (ST == LBM_STORE_F64) {
        if (H->tile == 4) return cg_launch_tile<ST, 4, PULL>(H, from, write_macro, write_rb, s);
    }
    cg_launch_tile<ST, 8, PULL>(H, from, write_macro, write_rb, s);
}

// One step (PULL) or the first collision from a given post-stream state.
template <bool PULL>
static void cg_any_launch(const lbm_cg_handle_s *H, int from, int write_macro, int write_rb, cudaStream_t s) {
    if (H->q == 19) {
        if (H->st == LBM_STORE_F16S) cg3_launch_st<LBM_STORE_F16S, PULL>(H, from, write_macro, write_rb, s);
        else if (H->st == LBM_STORE_F64) cg3_launch_st<LBM_STORE_F64, PULL>(H, from, write_macro, write_rb, s);
        else cg3_launch_st<LBM_STORE_F32, PULL>(H, from, write_macro, write_rb, s);
    } else {
        if (H->st == LBM_STORE_F16S) cg_launch_st<LBM_STORE_F16S, PULL>(H, from, write_macro, write_rb, s);
        else if (H->st == LBM_STORE_F64) cg_launch_st<LBM_STORE_F64, PULL>(H, from, write_macro, write_rb, s);
        else cg_launch_st<LBM_STORE_F32, PULL>(H, from, write_macro, write_rb, s);
    }
}

extern "C" {

const char *lbm_cg_last_error(void) { return g_cg_error.c_str(); }

static int cg_create(int n, int m, int h, const lbm_cg_params *P, lbm_cg_handle *out) {
    if (!P || !out) return cg_fail(LBM_ERR_INVALID, "null argument");
    *out = nullptr;
    if (n < 5 || m < 5 || h < 1 || m > 65535 || h > 65535 || (h > 1 && h < 5))
        return cg_fail(LBM_ERR_INVALID, "lattice must be at least 5 nodes along each axis (m, h <= 65535)");
    if ((long long)n * m * h >= (1ll << 31)) return cg_fail(LBM_ERR_INVALID, "more than 2^31 nodes");
    if (P->storage != LBM_STORE_F32 && P->storage != LBM_STORE_F16S && P->storage != LBM_STORE_F64)
        return cg_fail(LBM_ERR_INVALID, "colour-gradient storage must be F32, F16S or F64");
    if (!(P->r_viscosity > 0) || !(P->b_viscosity > 0)) return cg_fail(LBM_ERR_INVALID, "viscosities must be positive");
    lbm_cg_handle_s *H = new (std::nothrow) lbm_cg_handle_s();
    if (!H) return cg_fail(LBM_ERR_NOMEM, "out of host memory");
    H->n = n;
    H->m = m;
    H->h = h;
    H->q = h > 1 ? 19 : 9;
    H->N = (long long)n * m * h;
    H->P = *P;
    H->st = P->storage;
    {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&H->sms, cudaDevAttrMultiProcessorCount, dev);
        if (H->sms < 1) H->sms = 1;
        if (H->q == 19) H->planes = cg3_planes(H);
        else if (H->st == LBM_STORE_F64) H->tile = cg_tile_f64(H);
    }
    const size_t N = (size_t)H->N;
    const size_t rbytes = H->st == LBM_STORE_F64 ? sizeof(double) : sizeof(float);
    cudaError_t e = cudaMalloc((void **)&H->buf, 4 * H->slot_bytes());
    if (e == cudaSuccess) e = cudaMalloc((void **)&H->R, sizeof(float) * 6 * N);
    if (e == cudaSuccess && H->q == 19 && !cg3_one_launch(H->st, H->P.high_order))
        e = cudaMalloc((void **)&H->phi, rbytes * 2 * N);
    if (e == cudaSuccess) e = cudaMalloc((void **)&H->partial, sizeof(double) * (LAP_BLOCKS * 5 + 5));
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&H->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&H->stepped, cudaEventDisableTiming);
    if (e != cudaSuccess) {
        lbm_cg_destroy(H);
        return cg_fail(LBM_ERR_NOMEM, std::string("allocation: ") + cudaGetErrorString(e));
    }
    H->B = H->R + N;
    H->rho = H->R + 2 * N;
    H->ux = H->R + 3 * N;
    H->uy = H->R + 4 * N;
    H->uz = H->R + 5 * N;
    if (H->phi) H->dn = (char *)H->phi + rbytes * N;
    H->sums = H->partial + LAP_BLOCKS * 5;
    cudaMemset(H->R, 0, sizeof(float) * 6 * N);
    if (H->phi) cudaMemset(H->phi, 0, rbytes * 2 * N);
    *out = H;
    return LBM_OK;
}

int lbm_cg_create(int n, int m, const lbm_cg_params *P, lbm_cg_handle *out) { return cg_create(n, m, 1, P, out); }

int lbm_cg_create3d(int n, int m, int h, const lbm_cg_params *P, lbm_cg_handle *out) {
    if (h < 5) return cg_fail(LBM_ERR_INVALID, "lattice must be at least 5 nodes along each axis");
    return cg_create(n, m, h, P, out);
}

int lbm_cg_init(lbm_cg_handle H, const float *r_f, const float *b_f) {
    if (!H || !r_f || !b_f) return cg_fail(LBM_ERR_INVALID, "null argument");
    const size_t N = (size_t)H->N, Q = (size_t)H->q;
    // the given post-stream state goes to buffer 1 (through an FP32 staging
    // area in buffer 0, encoded into the storage); one collision without
    // streaming turns it into the post-collision state in buffer 0
    float *stage = (float *)H->buffer(0);
    const size_t fl = sizeof(float) * Q * N;
    float *stage_r = nullptr, *stage_b = nullptr;
    bool own = false;
    if (2 * fl <= 2 * H->slot_bytes()) {
        stage_r = stage;
        stage_b = stage + Q * N;
    } else {
        // F16S: buffer 0 holds fewer bytes than two FP32 colour sets
        cudaError_t e = cudaMalloc((void **)&stage_r, 2 * fl);
        if (e != cudaSuccess) return cg_fail(LBM_ERR_NOMEM, std::string("staging: ") + cudaGetErrorString(e));
        stage_b = stage_r + Q * N;
        own = true;
    }
    cudaError_t e = cudaMemcpyAsync(stage_r, r_f, fl, cudaMemcpyHostToDevice, H->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(stage_b, b_f, fl, cudaMemcpyHostToDevice, H->stream);
    if (e == cudaSuccess) {
        const unsigned blocks = (unsigned)((Q * N + 255) / 256);
        void *dst = H->buffer(1);
        if (H->st == LBM_STORE_F16S)
            cg_encode_kernel<LBM_STORE_F16S><<<blocks, 256, 0, H->stream>>>(stage_r, stage_b, dst, (int)Q, (long long)N, H->scale);
        else if (H->st == LBM_STORE_F64)
            cg_encode_kernel<LBM_STORE_F64><<<blocks, 256, 0, H->stream>>>(stage_r, stage_b, dst, (int)Q, (long long)N, H->scale);
        else
            cg_encode_kernel<LBM_STORE_F32><<<blocks, 256, 0, H->stream>>>(stage_r, stage_b, dst, (int)Q, (long long)N, H->scale);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(H->stream);
    if (own) cudaFree(stage_r);
    if (e != cudaSuccess) return cg_fail(LBM_ERR_CUDA, std::string("upload: ") + cudaGetErrorString(e));
    cg_any_launch<false>(H, 1, 1, 1, H->stream);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(H->stream);
    if (e != cudaSuccess) return cg_fail(LBM_ERR_CUDA, std::string("init: ") + cudaGetErrorString(e));
    H->cur = 0;
    return LBM_OK;
}

int lbm_cg_step(lbm_cg_handle H, int nsteps, int write_macro_last, void *stream) {
    if (!H || nsteps < 0) return cg_fail(LBM_ERR_INVALID, "invalid argument");
    cudaStream_t s = stream ? (cudaStream_t)stream : H->stream;
    for (int i = 0; i < nsteps; ++i) {
        const int last = i == nsteps - 1;  // the colour densities of the call's last step are kept
        cg_any_launch<true>(H, H->cur, write_macro_last && last, last, s);
        H->cur ^= 1;
    }
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaEventRecord(H->stepped, s);
    if (e != cudaSuccess) return cg_fail(LBM_ERR_CUDA, std::string("step: ") + cudaGetErrorString(e));
    return LBM_OK;
}

int lbm_cg_get_macro(lbm_cg_handle H, float *r_rho, float *b_rho, float *u, float *v) {
    if (!H) return cg_fail(LBM_ERR_INVALID, "null handle");
    cudaError_t e = cudaDeviceSynchronize();
    const size_t b = sizeof(float) * (size_t)H->N;
    if (e == cudaSuccess && r_rho) e = cudaMemcpy(r_rho, H->R, b, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && b_rho) e = cudaMemcpy(b_rho, H->B, b, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && u) e = cudaMemcpy(u, H->ux, b, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && v) e = cudaMemcpy(v, H->uy, b, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cg_fail(LBM_ERR_CUDA, std::string("read-back: ") + cudaGetErrorString(e));
    return LBM_OK;
}

int lbm_cg_get_macro3d(lbm_cg_handle H, float *r_rho, float *b_rho, float *u, float *v, float *w) {
    int rc = lbm_cg_get_macro(H, r_rho, b_rho, u, v);
    if (rc || !w) return rc;
    cudaError_t e = cudaMemcpy(w, H->uz, sizeof(float) * (size_t)H->N, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cg_fail(LBM_ERR_CUDA, std::string("read-back: ") + cudaGetErrorString(e));
    return LBM_OK;
}

int lbm_cg_get_populations(lbm_cg_handle H, float *r, float *b) {
    if (!H || !r || !b) return cg_fail(LBM_ERR_INVALID, "null argument");
    const size_t N = (size_t)H->N, Q = (size_t)H->q;
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return cg_fail(LBM_ERR_CUDA, std::string("read-back: ") + cudaGetErrorString(e));
    // decoded into the other buffer (free between steps) or a temporary
    const size_t fl = sizeof(float) * Q * N;
    float *tmp = nullptr;
    bool own = false;
    if (2 * fl <= 2 * H->slot_bytes()) {
        tmp = (float *)H->buffer(1 - H->cur);
    } else {
        e = cudaMalloc((void **)&tmp, 2 * fl);
        if (e != cudaSuccess) return cg_fail(LBM_ERR_NOMEM, std::string("read-back: ") + cudaGetErrorString(e));
        own = true;
    }
    const unsigned blocks = (unsigned)((Q * N + 255) / 256);
    const void *src = H->buffer(H->cur);
    const float inv = 1.0f / H->scale;
    if (H->st == LBM_STORE_F16S)
        cg_decode_kernel<LBM_STORE_F16S><<<blocks, 256, 0, H->stream>>>(src, tmp, tmp + Q * N, (int)Q, (long long)N, inv);
    else if (H->st == LBM_STORE_F64)
        cg_decode_kernel<LBM_STORE_F64><<<blocks, 256, 0, H->stream>>>(src, tmp, tmp + Q * N, (int)Q, (long long)N, inv);
    else
        cg_decode_kernel<LBM_STORE_F32><<<blocks, 256, 0, H->stream>>>(src, tmp, tmp + Q * N, (int)Q, (long long)N, inv);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(H->stream);
    if (e == cudaSuccess) e = cudaMemcpy(r, tmp, fl, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(b, tmp + Q * N, fl, cudaMemcpyDeviceToHost);
    if (own) cudaFree(tmp);
    if (e != cudaSuccess) return cg_fail(LBM_ERR_CUDA, std::string("read-back: ") + cudaGetErrorString(e));
    return LBM_OK;
}

int lbm_cg_laplace(lbm_cg_handle H, double *out) {
    if (!H || !out) return cg_fail(LBM_ERR_INVALID, "null argument");
    if (H->stepped) cudaStreamWaitEvent(H->stream, H->stepped, 0);
    cg_laplace_partial<<<LAP_BLOCKS, LAP_THREADS, 0, H->stream>>>(H->R, H->B, H->ux, H->uy, H->q == 19 ? H->uz : nullptr,
                                                                   H->N, (float)H->P.control_param, H->partial);
    cg_laplace_final<<<1, 32, 0, H->stream>>>(H->partial, H->sums);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, H->sums, sizeof(double) * 5, cudaMemcpyDeviceToHost, H->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(H->stream);
    if (e != cudaSuccess) return cg_fail(LBM_ERR_CUDA, std::string("laplace: ") + cudaGetErrorString(e));
    for (int k = 0; k < 5; ++k)
        if (!isfinite(out[k])) return cg_fail(LBM_DIVERGED, "non-finite colour-gradient field");
    return LBM_OK;
}

long long lbm_cg_nodes(lbm_cg_handle H) { return H ? H->N : -1; }

int lbm_cg_q(lbm_cg_handle H) { return H ? H->q : -1; }

void lbm_cg_destroy(lbm_cg_handle H) {
    if (!H) return;
    if (H->stream) cudaStreamSynchronize(H->stream);
    if (H->buf) cudaFree(H->buf);
    if (H->R) cudaFree(H->R);
    if (H->phi) cudaFree(H->phi);
    if (H->partial) cudaFree(H->partial);
    if (H->stepped) cudaEventDestroy(H->stepped);
    if (H->stream) cudaStreamDestroy(H->stream);
    delete H;
}

}  // extern "C"
