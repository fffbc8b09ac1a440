// 3x3 convolutions of the warm-start U-Net on the fifth-generation tensor
// cores (tcgen05.mma, accumulators in tensor memory, operands staged by
// tensor copies), for sm_100-class GPUs.
//
// Forward and data gradient (conv3x3_tc_kernel):
//
//   out[n, y, x0+m, co] = act(bias[co] + sum_{tap, ci} w[tap][co][ci] in[n, y+ky-1, x0+m+kx-1, ci])
//
// A tile is TC_M = 128 consecutive pixels of one image row: the GEMM's M.
// N = COUT output channels (16, 32, 64 or 128), K = 9 taps x cin, taken CHUNK
// (16, 32 or 64) input channels at a time; a job is one (tile, chunk).  The
// kernel is persistent: CTA b walks tiles b, b + gridDim.x, ...  Shared
// memory holds
//   B  every weight of the layer (9 taps x cin x COUT), loaded once, in the
//      K-major no-swizzle layout: core matrices of 8 rows x 16 bytes stored
//      as 128 contiguous bytes, byte ((t * KGall + j) * COUT + co) * 16 for
//      tap t, 8-channel group j, output channel co;
//   A  NS stages of input rows: one tensor copy per job brings the three
//      rows the taps read, TC_BOX = 136 pixels from x0 - 1 (zero fill outside
//      the image) x CHUNK channels, as K-major rows of 2 x CHUNK bytes with
//      the tensor copy's 128-, 64- or 32-byte swizzle.
// The tap's x shift kx is a start address kx rows further inside the same
// staged row: the hardware applies the swizzle to absolute shared-memory
// address bits, so a start moved by whole rows (or by 32 bytes for the next
// K = 16) reads the right elements with the descriptor's base offset 0.
//
// One thread of warp 4 issues the copies, one of warp 5 each job's
// 9 x CHUNK/16 MMAs (M = 128, N = COUT, K = 16, BF16 in, FP32 accumulate);
// warps 0-3 read finished tiles from NA tensor-memory accumulators (each warp
// its 32 lanes = 32 pixels), add the bias, apply ReLU and store BF16 (and FP32
// if asked), while the next tiles accumulate.  A job's fixed cost in the
// issuing threads is what bounds the level-0 layers, so they carry no division
// and no 64-bit index: tiles advance by carried coordinates (TileWalk), stages
// by counters.  Every wait is bounded: a wait that gives up sets *err, all
// roles stop, the copies and MMAs in flight finish, the tensor memory is freed
// and the kernel returns.
//
// Weight gradient (wgrad_tc_kernel): see its comment below.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace unet_tc {

constexpr int TC_M = 128;             // pixels per CTA (GEMM rows)
constexpr int TC_NP = TC_M + 2;       // staged pixels per row (halo)
constexpr long long TC_SPIN = 1ll << 26;  // bounded mbarrier polls

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor: start address, leading and stride byte
// offsets (all in 16-byte units), the fixed version field (bits 46-47 = 1),
// base offset 0 and layout type 0 (no swizzle).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator (bits 4-5 = 1), A
// and B BF16 (bits 7-9 = 1, 10-12 = 1), both K-major, N >> 3 at bit 17,
// M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Descriptors as halves: the start address sits in the low one, and offsets
// inside shared memory never carry out of its field.
struct Desc {
    uint32_t lo, hi;
    __device__ __forceinline__ Desc(uint64_t d) : lo((uint32_t)d), hi((uint32_t)(d >> 32)) {}
};
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, Desc a, uint32_t a_off, Desc b, uint32_t b_off, uint32_t idesc,
                                         uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %6, 0;\n\t"
        "mov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}\n" ::"r"(tmem_d),
        "r"(a.lo + a_off), "r"(a.hi), "r"(b.lo + b_off), "r"(b.hi), "r"(idesc), "r"(acc));
}

// The tiles blockIdx.x, blockIdx.x + gridDim.x, ... of a (image, row, segment)
// space with H rows and xt segments a row, as carried coordinates.
struct TileWalk {
    int xb, y, n, sx, sy, sn, xt, H, left;
    __device__ __forceinline__ TileWalk(int B, int H_, int xt_) : xt(xt_), H(H_) {
        const int first = blockIdx.x, step = gridDim.x, total = B * H * xt;
        xb = first % xt;
        y = first / xt % H;
        n = first / xt / H;
        sx = step % xt;
        sy = step / xt % H;
        sn = step / xt / H;
        left = total > first ? (total - 1 - first) / step + 1 : 0;
    }
    __device__ __forceinline__ void next() {
        xb += sx;
        const int cx = xb >= xt ? 1 : 0;
        xb -= cx ? xt : 0;
        y += sy + cx;
        const int cy = y >= H ? 1 : 0;
        y -= cy ? H : 0;
        n += sn + cy;
        --left;
    }
};
// A ring position of N slots: the slot, its barrier phase and, past the first
// round, the phase in which the slot was last released.
template <int N>
struct Ring {
    uint32_t slot = 0, round = 0;
    __device__ __forceinline__ void next() {
        if (++slot == N) {
            slot = 0;
            ++round;
        }
    }
};

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
                 : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}

// true once phase `parity` of the barrier has completed; false after
// TC_SPIN polls, or as soon as *stop (when given) is set
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, volatile int *stop = nullptr) {
    for (long long i = 0; i < TC_SPIN; ++i) {
        if (stop && (i & 1023) == 1023 && *stop) return false;
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// One lane of a converged warp.  The issuing warps run their loops with all
// lanes and elect the one that issues: control flow and operands then stay
// uniform in the compiler's eyes, and the descriptors reach the tensor core's
// uniform registers without a move per operand and instruction.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
    return p != 0;
}
// mbar_wait by a whole warp, the answer uniform
__device__ __forceinline__ bool mbar_wait_warp(uint32_t mbar, uint32_t parity, volatile int *stop) {
    return __all_sync(0xffffffffu, mbar_wait(mbar, parity, stop));
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 16 consecutive FP32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 16 columns without the wait, and the wait for all of them.
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// orders the loaded registers after the wait
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}
// 32 bytes in one store: a whole sector per thread
__device__ __forceinline__ void store32(void *p, const uint32_t (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

// 16 bytes global -> shared without a register round trip; src_bytes 0
// writes zeros (the source is then not read)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Swizzled K-major operand descriptor (tcgen05 layout types 2, 4, 6 for
// 128-, 64- and 32-byte rows): rows of ROWB bytes, 8-row groups 8 x ROWB
// bytes apart.  The hardware applies the swizzle to absolute shared-memory
// address bits, so a start address moved by whole rows (the tap shift) or by
// 32 bytes (the next K = 16) inside a swizzle atom reads the matching
// elements with base offset 0, as long as the tensor copy wrote the atoms at
// their absolute addresses.
template <int ROWB>
__device__ __forceinline__ uint64_t smem_desc_sw(uint32_t addr) {
    constexpr uint64_t layout = ROWB == 128 ? 2 : (ROWB == 64 ? 4 : 6);
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)((8 * ROWB) >> 4) << 32) | (1ull << 46) |
           (layout << 61);
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

// Tiled tensor copy of a 4-D box (c, x, y, n) into shared memory, completing
// on mbar.  The innermost coordinate c is a multiple of 8 channels (16 bytes).
__device__ __forceinline__ void tma_load4(uint32_t dst, const void *tmap, int c, int x, int y, int n, uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(dst),
        "l"(tmap), "r"(c), "r"(x), "r"(y), "r"(n), "r"(mbar)
        : "memory");
}

// Tiled tensor copy of a 4-D box from shared memory; elements outside the
// tensor are not written.  The issuing thread groups and awaits its copies.
__device__ __forceinline__ void tma_store4(const void *tmap, int c, int x, int y, int n, uint32_t src) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(tmap),
                 "r"(c), "r"(x), "r"(y), "r"(n), "r"(src)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void tma_store_read_wait() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

constexpr int TC_BOX = 136;  // staged pixels per row: x0 - 1 .. x0 + 134, a whole number of swizzle atoms

template <int COUT, int CHUNK, int NS>
struct TcSmem {
    // tensor-memory accumulators: a tile's MMAs wait for the epilogue of the
    // tile NA before it, so NA tiles overlap one accumulator round trip
    // (commit, epilogue, release); NA x COUT columns
    static constexpr int NA = 4 * COUT <= 512 ? 4 : 2;
    static constexpr int ROWB = CHUNK * 2;
    static constexpr int A_STAGE = 3 * TC_BOX * ROWB;
    static constexpr size_t bytes(int cin) {
        return 1024 + NS * (size_t)A_STAGE + 18 * (size_t)cin * COUT + 4 * COUT + 8 * (2 * NS + 2 * NA) + 16;
    }
};

// One finished tile of an epilogue warp: its 32 lanes of accumulator a to
// registers, 32 columns at a time, the accumulator released (barrier
// `release`) once all are read, then bias, ReLU and the stores.
// STAGED: the warp's 32 pixels go through `stage` (its own swizzled 32 x COUT
// tile in shared memory) and leave by one tensor copy: a thread's own stores
// are one sector in each of 32 lines, and their L1 wavefronts (512 of a
// 64-channel tile's 860) bound the level-0 layers with 32 and 64 outputs.
// MASK (data gradients): the output is the gradient before the layer below's
// ReLU, so it is zeroed where that layer's activation `act` (channels from
// act, stride act_cs) is not positive, and bsum gathers each channel's sum of
// the stored values over this lane's pixels, the bias gradient's share.
template <int COUT, bool MASK>
struct EpilogueMask {
    const __nv_bfloat16 *act = nullptr;
    int act_cs = 0;
    float bsum[MASK ? COUT : 1];
    // the tile's activations, and the next tile's on their way: a load takes
    // about a tile's time to arrive
    uint32_t m[MASK ? COUT / 16 : 1][8], ahead[MASK ? COUT / 16 : 1][8];
    __device__ __forceinline__ void take() {
        if constexpr (MASK) {
#pragma unroll
            for (int i = 0; i < COUT / 16; ++i)
#pragma unroll
                for (int k = 0; k < 8; ++k) m[i][k] = ahead[i][k];
        }
    }
    __device__ __forceinline__ void load(bool in, size_t pix) {
        if constexpr (MASK) {
#pragma unroll
            for (int i = 0; i < COUT / 16; ++i) {
                const void *p = act + pix * act_cs + 16 * i;
#pragma unroll
                for (int k = 0; k < 8; ++k) ahead[i][k] = 0u;
                if (in)
                    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                                 : "=r"(ahead[i][0]), "=r"(ahead[i][1]), "=r"(ahead[i][2]), "=r"(ahead[i][3]),
                                   "=r"(ahead[i][4]), "=r"(ahead[i][5]), "=r"(ahead[i][6]), "=r"(ahead[i][7])
                                 : "l"(p));
            }
        }
    }
};
template <int COUT, bool STAGED, bool MASK = false>
__device__ __forceinline__ void conv_epilogue(uint32_t tmem, uint32_t a, uint32_t release, const float *sbias,
                                              const CUtensorMap *tout, uint32_t stage, __nv_bfloat16 *out, int out_cs,
                                              int out_co, float *out32, int n, int y, int xb, int H, int W, int relu,
                                              EpilogueMask<COUT, MASK> *mask = nullptr) {
    constexpr int CW = COUT < 32 ? COUT : 32, RB = COUT * 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    fence_after();
    const int x = xb * TC_M + warp * 32 + lane;  // TMEM lane = GEMM row = pixel
    const size_t pix = ((size_t)n * H + y) * W + x;
    const uint32_t acc = tmem + ((uint32_t)(warp * 32) << 16) + a * COUT;
    if (STAGED) {
        if (lane == 0) tma_store_read_wait();  // the tile before has left the stage
        __syncwarp();
    }
#pragma unroll(MASK ? COUT / CW : 1)
    for (int c = 0; c < COUT; c += CW) {
        uint32_t r[CW / 16][16];
#pragma unroll
        for (int i = 0; i < CW / 16; ++i) tmem_ld16_async(acc + (uint32_t)(c + 16 * i), r[i]);
#pragma unroll
        for (int i = 0; i < CW / 16; ++i) tmem_wait(r[i]);
        if (c + CW == COUT) {
            // every column is in registers: the accumulator is free
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(release);
        }
#pragma unroll
        for (int q = 0; q < CW / 16; ++q) {
            float v[16];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 b4 = *(const float4 *)(sbias + c + 16 * q + 4 * i);
                v[4 * i] = __uint_as_float(r[q][4 * i]) + b4.x;
                v[4 * i + 1] = __uint_as_float(r[q][4 * i + 1]) + b4.y;
                v[4 * i + 2] = __uint_as_float(r[q][4 * i + 2]) + b4.z;
                v[4 * i + 3] = __uint_as_float(r[q][4 * i + 3]) + b4.w;
            }
            if (relu) {
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = fmaxf(v[i], 0.f);
            }
            if (STAGED || out) {
                uint32_t pk[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const __nv_bfloat162 h2 = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                    pk[i] = *(const uint32_t *)&h2;
                }
                if constexpr (MASK) {
                    // positive: sign clear and not zero (zero beyond the image)
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint32_t m = mask->m[c / 16 + q][i];
                        const __nv_bfloat162 mv = *(const __nv_bfloat162 *)&m;
                        const float2 mf = __bfloat1622float2(mv);
                        const __nv_bfloat162 pv = *(const __nv_bfloat162 *)&pk[i];
                        float2 pf = __bfloat1622float2(pv);
                        if (!(mf.x > 0.f)) {
                            pk[i] &= 0xFFFF0000u;
                            pf.x = 0.f;
                        }
                        if (!(mf.y > 0.f)) {
                            pk[i] &= 0x0000FFFFu;
                            pf.y = 0.f;
                        }
                        mask->bsum[c + 16 * q + 2 * i] += pf.x;
                        mask->bsum[c + 16 * q + 2 * i + 1] += pf.y;
                    }
                }
                if (STAGED) {
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        // the tensor copy's swizzle: 16-byte chunk index xor 128-byte line index
                        uint32_t off = (uint32_t)(lane * RB + 2 * (c + 16 * q) + 16 * k);
                        off ^= ((off >> 7) & (RB / 16 - 1)) << 4;
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + off), "r"(pk[4 * k]),
                                     "r"(pk[4 * k + 1]), "r"(pk[4 * k + 2]), "r"(pk[4 * k + 3])
                                     : "memory");
                    }
                } else if (x < W) {
                    store32(out + pix * out_cs + out_co + c + 16 * q, pk);
                }
            }
            if (!STAGED && out32 && x < W) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    uint32_t pk[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) pk[j] = __float_as_uint(v[8 * i + j]);
                    store32(out32 + pix * COUT + c + 16 * q + 8 * i, pk);
                }
            }
        }
    }
    if (STAGED) {
        fence_proxy_async();
        __syncwarp();
        if (lane == 0 && xb * TC_M + warp * 32 < W)
            tma_store4(tout, 0, xb * TC_M + warp * 32, y, n, stage);
    }
}

// Warp roles: warps 0-3 read the accumulators (each its 32 TMEM lanes) and
// store the outputs; one thread of warp 4 issues the tensor copies, one of
// warp 5 the MMAs.  Barriers (all counts 1 except acc_empty, 4):
//   full[s]      stage s holds its job's rows (tensor-copy bytes)
//   empty[s]     the MMAs that read stage s are done (tcgen05.commit)
//   acc_full[a]  accumulator a holds a finished tile (tcgen05.commit)
//   acc_empty[a] the four epilogue warps have read accumulator a
constexpr int CONV_THREADS = 192;
template <int COUT, int CHUNK, int NS>
__global__ void __launch_bounds__(CONV_THREADS, 1)
conv3x3_tc_kernel(const __grid_constant__ CUtensorMap tin, int cin, const __nv_bfloat16 *__restrict__ w,
                  const float *__restrict__ bias, __nv_bfloat16 *__restrict__ out, int out_cs, int out_co,
                  float *__restrict__ out32, int B, int H, int W, int relu, int *err) {
    static_assert(COUT % 16 == 0 && COUT <= 128 && (CHUNK == 16 || CHUNK == 32 || CHUNK == 64), "N, K chunk");
    static_assert(NS >= 2 && NS <= 4, "input stages");
    using SM = TcSmem<COUT, CHUNK, NS>;
    constexpr int ROWB = SM::ROWB, KG = CHUNK / 8;
    constexpr uint32_t A_STAGE = SM::A_STAGE;
    constexpr int NA = SM::NA;
    constexpr uint32_t COLS = NA * COUT < 32 ? 32 : NA * COUT;  // a power of two >= 32
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    unsigned char *smem = smem_raw + (base - raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int KGall = cin / 8, nch = cin / CHUNK;
    const uint32_t b_base = base + NS * A_STAGE;
    float *sbias = (float *)(smem + NS * A_STAGE + (size_t)18 * cin * COUT);
    uint64_t *bars = (uint64_t *)(sbias + COUT);
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * NS, accf0 = empty0 + 8 * NS, acce0 = accf0 + 8 * NA;
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * NS + 2 * NA);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    TileWalk walk(B, H, (W + TC_M - 1) / TC_M);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int k = 0; k < NS; ++k) {
            mbar_init(full0 + 8 * k, 1);
            mbar_init(empty0 + 8 * k, 1);
        }
        for (int a = 0; a < NA; ++a) {
            mbar_init(accf0 + 8 * a, 1);
            mbar_init(acce0 + 8 * a, 4);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < COUT) sbias[tid] = bias ? bias[tid] : 0.f;
    // every weight of the layer, no swizzle: byte ((t * KGall + j) * COUT + co) * 16
    for (int i = tid; i < 9 * KGall * COUT; i += CONV_THREADS) {
        const int tc = i / KGall, j = i % KGall, t = tc / COUT, co = tc % COUT;
        cp_async16(b_base + (uint32_t)(((t * KGall + j) * COUT + co) * 16), w + (size_t)i * 8, 16);
    }
    cp_async_commit();
    cp_async_wait<0>();
    fence_proxy_async();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    bool ok = true;

    if (warp == 4) {
        if (lane == 0) {
            Ring<NS> st;
            int issued = 0;
            for (; walk.left > 0 && ok; walk.next()) {
                for (int c = 0; c < nch; ++c) {
                    const uint32_t s = st.slot, fb = full0 + 8 * s;
                    if (st.round > 0 && !mbar_wait(empty0 + 8 * s, (st.round - 1) & 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(fb, A_STAGE);
                    tma_load4(base + s * A_STAGE, &tin, c * CHUNK, walk.xb * TC_M - 1, walk.y - 1, walk.n, fb);
                    st.next();
                    ++issued;
                }
            }
            if (!ok) {
                *abort_flag = 1;
                atomicExch(err, 1);
            }
            // the copies in flight land before the CTA leaves, whichever role
            // gave up: the last use of each stage
            for (int j = issued > NS ? issued - NS : 0; j < issued; ++j)
                mbar_wait(full0 + 8 * (uint32_t)(j % NS), (uint32_t)((j / NS) & 1));
        }
        __syncwarp();
    } else if (warp == 5) {
        constexpr uint32_t IDESC = idesc_bf16(TC_M, COUT);
        const bool leader = elect_one();
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        Ring<NS> st;
        Ring<NA> ac;
        const uint32_t tap_step = (uint32_t)(KGall * COUT);
        int committed = 0;
        for (int k = walk.left; k > 0 && ok; --k, ac.next()) {
            // the epilogue of tile k - NA has read the accumulator
            if (ac.round > 0 && !mbar_wait_warp(acce0 + 8 * ac.slot, (ac.round - 1) & 1, abort_flag)) {
                ok = false;
                break;
            }
            const uint32_t d = tm + ac.slot * COUT;
            for (int c = 0; c < nch; ++c) {
                const uint32_t s = st.slot;
                if (!mbar_wait_warp(full0 + 8 * s, st.round & 1, abort_flag)) {
                    ok = false;
                    break;
                }
                fence_after();
                const Desc da(smem_desc_sw<ROWB>(base + s * A_STAGE));
                const Desc db(smem_desc(b_base + (uint32_t)(c * KG * COUT * 16), COUT * 16, 128));
                if (leader) {
#pragma unroll
                    for (int t = 0; t < 9; ++t) {
#pragma unroll
                        for (int q = 0; q < KG / 2; ++q)
                            mma_bf16(d, da, (uint32_t)(((t / 3) * TC_BOX + t % 3) * ROWB / 16 + 2 * q), db,
                                     (uint32_t)t * tap_step + (uint32_t)(2 * q * COUT), IDESC,
                                     (c > 0 || t > 0 || q > 0) ? 1u : 0u);
                    }
                    mma_commit(empty0 + 8 * s);
                    if (c == nch - 1) mma_commit(accf0 + 8 * ac.slot);
                }
                st.next();
                ++committed;
            }
        }
        if (!ok) {
            *abort_flag = 1;
            if (leader) atomicExch(err, 1);
        }
        // no MMA or commit is in flight when the tensor memory is freed,
        // whichever role gave up: they complete in order, so the last commits
        // cover them all
        if (committed > 0)
            mbar_wait(empty0 + 8 * (uint32_t)((committed - 1) % NS), (uint32_t)(((committed - 1) / NS) & 1));
        const int done = committed / nch;  // finished tiles
        if (done > 0) mbar_wait(accf0 + 8 * (uint32_t)((done - 1) % NA), (uint32_t)(((done - 1) / NA) & 1));
        __syncwarp();
    } else {
        // epilogue warps: tile k from accumulator k % NA, 32 columns at a time
        Ring<NA> ac;
        for (; walk.left > 0; walk.next(), ac.next()) {
            const uint32_t a = ac.slot;
            const bool got = mbar_wait(accf0 + 8 * a, ac.round & 1, abort_flag);
            if (!__all_sync(0xffffffffu, got)) {
                ok = false;
                break;
            }
            conv_epilogue<COUT, false>(tmem, a, acce0 + 8 * a, sbias, nullptr, 0, out, out_cs, out_co, out32, walk.n,
                                       walk.y, walk.xb, H, W, relu);
        }
        if (!ok) {
            *abort_flag = 1;
            if (lane == 0) atomicExch(err, 1);
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
}

// The same convolution with a ring of input rows: a CTA takes a contiguous run
// of tiles in the order (image, row segment, y), y fastest, and keeps whole
// input rows (all cin channels, TC_BOX pixels) in NR ring slots, so a tile
// brings one new row where conv3x3_tc_kernel's stage brings three, and the
// tiles divide evenly over the CTAs.  A run crosses a few column segments; each
// costs two extra rows.  Chunks of CHUNK channels lie one after another in a
// slot, each a swizzled K-major tile of its own, and the MMAs run chunk, tap,
// K = 16, the order of conv3x3_tc_kernel, so the sums are the same.
// Barriers as there, with one full and empty barrier per slot: a slot is
// released by the commit of the last tile that reads its row.
template <int COUT, int CHUNK>
struct RowSmem {
    static constexpr int NA = 4 * COUT <= 512 ? 4 : 2;
    static constexpr int ROWB = CHUNK * 2, SUB = TC_BOX * ROWB;  // a chunk of a row; a whole number of swizzle atoms
    // outputs of 32 and 64 channels leave through shared memory (conv_epilogue)
    static constexpr bool STAGED = COUT == 32 || COUT == 64;
    static constexpr int STAGE = STAGED ? TC_M * COUT * 2 : 0;
    static constexpr size_t row_bytes(int cin) { return (size_t)TC_BOX * 2 * cin; }
    static constexpr size_t bytes(int cin, int nr) {
        return 1024 + STAGE + nr * row_bytes(cin) + 18 * (size_t)cin * COUT + 4 * COUT + 8 * (2 * nr + 2 * NA) + 16;
    }
};
constexpr int ROW_MAX = 8;  // most ring slots
// rows of partial bias gradients a kernel may leave, one per block, and their pitch
constexpr int BIAS_ROWS = 1216, BIAS_STRIDE = 64;

// A run of tiles in the order (n, xb, y), y fastest.
struct RunWalk {
    int y, xb, n, left, xt, H;
    __device__ __forceinline__ RunWalk(int B, int H_, int xt_) : xt(xt_), H(H_) {
        const long long total = (long long)B * H * xt;
        const int t0 = (int)(total * blockIdx.x / gridDim.x), t1 = (int)(total * (blockIdx.x + 1) / gridDim.x);
        left = t1 - t0;
        y = t0 % H;
        xb = t0 / H % xt;
        n = t0 / H / xt;
    }
    // tiles left in this column segment
    __device__ __forceinline__ int segment() const { return left < H - y ? left : H - y; }
    __device__ __forceinline__ void advance(int k) {
        left -= k;
        y += k;
        if (y == H) {
            y = 0;
            if (++xb == xt) {
                xb = 0;
                ++n;
            }
        }
    }
};
// Ring position with a run-time number of slots.
struct RowRing {
    int slot = 0, nr;
    uint32_t round = 0;
    __device__ __forceinline__ explicit RowRing(int n) : nr(n) {}
    __device__ __forceinline__ void next() {
        if (++slot == nr) {
            slot = 0;
            ++round;
        }
    }
};

template <int COUT, int CHUNK, bool MASK>
__global__ void __launch_bounds__(CONV_THREADS, 1)
conv3x3_rows_kernel(const __grid_constant__ CUtensorMap tin, const __grid_constant__ CUtensorMap tout, int cin, int nr, const __nv_bfloat16 *__restrict__ w,
                    const float *__restrict__ bias, __nv_bfloat16 *__restrict__ out, int out_cs, int out_co,
                    float *__restrict__ out32, const __nv_bfloat16 *__restrict__ act, int act_cs, float *__restrict__ db_rows,
                    int B, int H, int W, int relu, int *err) {
    static_assert(COUT % 16 == 0 && COUT <= 128 && (CHUNK == 16 || CHUNK == 32 || CHUNK == 64), "N, K chunk");
    using SM = RowSmem<COUT, CHUNK>;
    constexpr int ROWB = SM::ROWB, SUB = SM::SUB, KG = CHUNK / 8, NA = SM::NA;
    constexpr uint32_t COLS = NA * COUT < 32 ? 32 : NA * COUT;  // a power of two >= 32
    __shared__ float db_sum[MASK ? 4 : 1][MASK ? COUT : 1];
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw), stage0 = (raw + 1023u) & ~1023u, base = stage0 + SM::STAGE;
    unsigned char *smem = smem_raw + (base - raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int KGall = cin / 8, nch = cin / CHUNK;
    const uint32_t row = (uint32_t)(TC_BOX * 2 * cin), b_base = base + (uint32_t)nr * row;
    float *sbias = (float *)(smem + (size_t)nr * row + (size_t)18 * cin * COUT);
    uint64_t *bars = (uint64_t *)(sbias + COUT);
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * nr, accf0 = empty0 + 8 * nr, acce0 = accf0 + 8 * NA;
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * nr + 2 * NA);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    RunWalk walk(B, H, (W + TC_M - 1) / TC_M);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int k = 0; k < nr; ++k) {
            mbar_init(full0 + 8 * k, 1);
            mbar_init(empty0 + 8 * k, 1);
        }
        for (int a = 0; a < NA; ++a) {
            mbar_init(accf0 + 8 * a, 1);
            mbar_init(acce0 + 8 * a, 4);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < COUT) sbias[tid] = bias ? bias[tid] : 0.f;
    // every weight of the layer, as in conv3x3_tc_kernel
    for (int i = tid; i < 9 * KGall * COUT; i += CONV_THREADS) {
        const int tc = i / KGall, j = i % KGall, t = tc / COUT, co = tc % COUT;
        cp_async16(b_base + (uint32_t)(((t * KGall + j) * COUT + co) * 16), w + (size_t)i * 8, 16);
    }
    cp_async_commit();
    cp_async_wait<0>();
    fence_proxy_async();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    bool ok = true;

    if (warp == 4) {
        if (lane == 0) {
            RowRing st(nr);
            int issued = 0;
            while (walk.left > 0 && ok) {
                const int seg = walk.segment();
                for (int r = -1; r <= seg; ++r, st.next(), ++issued) {
                    const uint32_t s = (uint32_t)st.slot, fb = full0 + 8 * s;
                    if (st.round > 0 && !mbar_wait(empty0 + 8 * s, (st.round - 1) & 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(fb, row);
                    for (int c = 0; c < nch; ++c)
                        tma_load4(base + s * row + (uint32_t)(c * SUB), &tin, c * CHUNK, walk.xb * TC_M - 1,
                                  walk.y + r, walk.n, fb);
                }
                walk.advance(seg);
            }
            if (!ok) {
                *abort_flag = 1;
                atomicExch(err, 1);
            }
            // as in conv3x3_tc_kernel: the last use of each slot
            for (int j = issued > nr ? issued - nr : 0; j < issued; ++j)
                mbar_wait(full0 + 8 * (uint32_t)(j % nr), (uint32_t)((j / nr) & 1));
        }
        __syncwarp();
    } else if (warp == 5) {
        constexpr uint32_t IDESC = idesc_bf16(TC_M, COUT);
        const bool leader = elect_one();
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        RowRing st(nr);
        Ring<NA> ac;
        const uint32_t tap_step = (uint32_t)(KGall * COUT);
        int w0 = 0, w1 = 0, w2 = 0;  // slots of the tile's rows y - 1, y, y + 1
        int tiles = 0;               // tiles issued and committed
        auto take = [&]() -> bool {  // the next row of the ring becomes w2
            w0 = w1;
            w1 = w2;
            w2 = st.slot;
            const bool got = mbar_wait_warp(full0 + 8 * (uint32_t)st.slot, st.round & 1, abort_flag);
            st.next();
            return got;
        };
        while (walk.left > 0 && ok) {
            const int seg = walk.segment();
            ok = take() && take();
            for (int k = 0; k < seg && ok; ++k, ac.next()) {
                if (!take() ||
                    (ac.round > 0 && !mbar_wait_warp(acce0 + 8 * ac.slot, (ac.round - 1) & 1, abort_flag))) {
                    ok = false;
                    break;
                }
                fence_after();
                const uint32_t d = tm + ac.slot * COUT;
                for (int c = 0; c < nch; ++c) {
                    const uint32_t sub = (uint32_t)(c * SUB);
                    const Desc r0(smem_desc_sw<ROWB>(base + (uint32_t)w0 * row + sub)),
                        r1(smem_desc_sw<ROWB>(base + (uint32_t)w1 * row + sub)),
                        r2(smem_desc_sw<ROWB>(base + (uint32_t)w2 * row + sub));
                    const Desc db(smem_desc(b_base + (uint32_t)(c * KG * COUT * 16), COUT * 16, 128));
                    if (leader) {
#pragma unroll
                        for (int t = 0; t < 9; ++t) {
#pragma unroll
                            for (int q = 0; q < KG / 2; ++q)
                                mma_bf16(d, t < 3 ? r0 : (t < 6 ? r1 : r2), (uint32_t)((t % 3) * ROWB / 16 + 2 * q), db,
                                         (uint32_t)t * tap_step + (uint32_t)(2 * q * COUT), IDESC,
                                         (c > 0 || t > 0 || q > 0) ? 1u : 0u);
                        }
                    }
                }
                // row y - 1 has served; at a segment's end so have the others
                if (leader) {
                    mma_commit(empty0 + 8 * (uint32_t)w0);
                    if (k == seg - 1) {
                        mma_commit(empty0 + 8 * (uint32_t)w1);
                        mma_commit(empty0 + 8 * (uint32_t)w2);
                    }
                    mma_commit(accf0 + 8 * ac.slot);
                }
                ++tiles;
            }
            walk.advance(seg);
        }
        if (!ok) {
            *abort_flag = 1;
            if (leader) atomicExch(err, 1);
        }
        // as in conv3x3_tc_kernel; a tile's last commit is its accumulator's
        if (tiles > 0) mbar_wait(accf0 + 8 * (uint32_t)((tiles - 1) % NA), (uint32_t)(((tiles - 1) / NA) & 1));
        __syncwarp();
    } else {
        // epilogue warps: tile k from accumulator k % NA, 32 columns at a time
        Ring<NA> ac;
        EpilogueMask<COUT, MASK> mask;
        if constexpr (MASK) {
            mask.act = act;
            mask.act_cs = act_cs;
#pragma unroll
            for (int i = 0; i < COUT; ++i) mask.bsum[i] = 0.f;
        }
        RunWalk next = walk;
        auto load_next = [&]() {
            if constexpr (MASK) {
                const int x = next.xb * TC_M + warp * 32 + lane;
                mask.load(next.left > 0 && x < W, ((size_t)next.n * H + next.y) * W + x);
                if (next.left > 0) next.advance(1);
            }
        };
        load_next();
        for (; walk.left > 0; walk.advance(1), ac.next()) {
            mask.take();
            load_next();
            const bool got = mbar_wait(accf0 + 8 * ac.slot, ac.round & 1, abort_flag);
            if (!__all_sync(0xffffffffu, got)) {
                ok = false;
                break;
            }
            conv_epilogue<COUT, SM::STAGED, MASK>(tmem, ac.slot, acce0 + 8 * ac.slot, sbias, &tout,
                                                  stage0 + (uint32_t)warp * 64 * COUT, out, out_cs, out_co, out32, walk.n,
                                                  walk.y, walk.xb, H, W, relu, &mask);
        }
        if (SM::STAGED && lane == 0) tma_store_wait();
        if constexpr (MASK) {
            // channel sums of the warp's pixels, then (below) of the CTA's
            __syncwarp();
#pragma unroll
            for (int i = 0; i < COUT; ++i) {
                float v = mask.bsum[i];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == i % 32) db_sum[warp][i] = v;
            }
        }
        if (!ok) {
            *abort_flag = 1;
            if (lane == 0) atomicExch(err, 1);
        }
    }
    fence_before();
    __syncthreads();
    if constexpr (MASK) {
        if (tid < COUT)
            db_rows[(size_t)blockIdx.x * BIAS_STRIDE + tid] =
                (db_sum[0][tid] + db_sum[1][tid]) + (db_sum[2][tid] + db_sum[3][tid]);
    }
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
}

// dst[0..3] += (a, b, c, d) in one vector reduction; dst 16-byte aligned
__device__ __forceinline__ void red_add4(float *dst, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}

// Weight gradient on the tensor cores:
//
//   dw[ky][kx][co][ci] += sum_{n, y, x} dpre[n, y, x, co] in[n, y+ky-1, x+kx-1, ci]
//
// A job is one input row y and TC_M = 128 output pixels x0 .. x0+127: the
// GEMM's K.  Input row y meets output-gradient row y - ky + 1 in tap row ky.
// One tensor copy stages the output-gradient rows y-1, y, y+1 (128 pixels x
// CO channels each); the A operand stacks them along M as (row, co), so M
// row m holds channel m % CO of row y - 1 + m / CO, i.e. tap row
// ky = 2 - m / CO, in M_BLOCKS blocks of 128 (rows past 3 x CO read staging
// memory no result uses: the input row or the next stage).  A second copy
// stages the input row (TC_BOX pixels from x0 - 1) right after the three
// rows, for NC input channels: the B operand, whose tap shift
// kx is a start address kx pixel rows further.  Both operands are
// channel-contiguous per pixel, "MN-major" (the instruction descriptor's
// transpose bits), swizzled by their row bytes (2 x CO and 2 x NC): the
// leading byte offset steps between channel blocks along M (one staged row
// of 128 pixels), the stride byte offset between groups of 8 pixels along K.
// The accumulators D[block][kx] (128 lanes x NC columns) stay in tensor
// memory across all of a CTA's jobs and are added to dw at the end with
// 16-byte vector reductions (dw, cin and NC keep every group of four columns
// aligned); a layer wider than NC input channels is split over gridDim.y.
// One thread of warp 0 issues the copies (NS stages), one of warp 1 the MMAs;
// every wait is bounded.
template <int CO, int NC, int NS>
struct WgSmem {
    static constexpr int ROWB_A = CO * 2, ROWB_B = NC * 2;
    static constexpr int M_BLOCKS = 3 * CO > 128 ? 2 : 1;
    // The copy writes the three rows (A_ROWS bytes, a whole number of 1 KB
    // swizzle atoms) and B right after them; the MMAs of an M block read
    // 128 rows of CO channels from the stage start (A_SPAN bytes), so the
    // rows past 3 x CO fall on B or the next stage: in bounds, and they only
    // feed accumulator rows no result uses.  TAIL keeps the last stage's
    // span inside the allocation.
    static constexpr int A_ROWS = 3 * TC_M * ROWB_A;
    static constexpr int A_STAGE = A_ROWS;                        // offset of B in a stage
    static constexpr int A_SPAN = M_BLOCKS * 128 * TC_M * 2;
    static constexpr int B_STAGE = TC_BOX * ROWB_B;
    static constexpr int STAGE = (A_STAGE + B_STAGE + 1023) / 1024 * 1024;
    static constexpr int TAIL = A_SPAN > STAGE ? A_SPAN - STAGE : 0;
    static constexpr int BYTES = 1024 + NS * STAGE + TAIL + 16 * NS + 16;
    static constexpr int USED = M_BLOCKS * 3 * NC;
    static constexpr uint32_t COLS = USED <= 32 ? 32 : USED <= 64 ? 64 : USED <= 128 ? 128 : USED <= 256 ? 256 : 512;
};

// Swizzled MN-major operand descriptor: rows of ROWB bytes along K (one per
// pixel), lbo between channel blocks along M or N, 8-row groups 8 x ROWB
// bytes apart along K.
template <int ROWB>
__device__ __forceinline__ uint64_t smem_desc_sw_mn(uint32_t addr, uint32_t lbo) {
    constexpr uint64_t layout = ROWB == 128 ? 2 : (ROWB == 64 ? 4 : 6);
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((8 * ROWB) >> 4) << 32) | (1ull << 46) | (layout << 61);
}

template <int CO, int NC, int NS>
__global__ void __launch_bounds__(128, 1)
wgrad_tc_kernel(const __grid_constant__ CUtensorMap tdp, const __grid_constant__ CUtensorMap tin, int cin,
                float *__restrict__ dw, int B, int H, int W, int *err) {
    static_assert((CO == 16 || CO == 32 || CO == 64) && (NC == 16 || NC == 32 || NC == 64), "swizzle rows");
    using SM = WgSmem<CO, NC, NS>;
    constexpr int MB = SM::M_BLOCKS, ROWB_A = SM::ROWB_A, ROWB_B = SM::ROWB_B;
    constexpr uint32_t STAGE = SM::STAGE, A_STAGE = SM::A_STAGE, COLS = SM::COLS;
    static_assert(SM::USED <= 512, "accumulators fit in tensor memory");
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    unsigned char *smem = smem_raw + (base - raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ci0 = blockIdx.y * NC;
    uint64_t *bars = (uint64_t *)(smem + NS * STAGE + SM::TAIL);
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * NS;
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * NS);
    TileWalk walk(B, H, (W + TC_M - 1) / TC_M);
    const int jobs = walk.left;
    __shared__ volatile int abort_flag;  // a wait gave up
    __shared__ int status;               // 1: every MMA committed and complete

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int k = 0; k < NS; ++k) {
            mbar_init(full0 + 8 * k, 1);
            mbar_init(empty0 + 8 * k, 1);
        }
        abort_flag = 0;
        status = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    // kind::f16, BF16 operands, FP32 accumulator, A and B MN-major
    constexpr uint32_t IDESC = idesc_bf16(TC_M, NC) | (1u << 15) | (1u << 16);

    if (tid == 0) {
        bool ok = true;
        Ring<NS> st;
        int issued = 0;
        for (; walk.left > 0; walk.next(), st.next()) {
            const uint32_t s = st.slot, fb = full0 + 8 * s, dst = base + s * STAGE;
            if (st.round > 0 && !mbar_wait(empty0 + 8 * s, (st.round - 1) & 1, &abort_flag)) {
                ok = false;
                break;
            }
            mbar_expect_tx(fb, SM::A_ROWS + SM::B_STAGE);
            tma_load4(dst, &tdp, 0, walk.xb * TC_M, walk.y - 1, walk.n, fb);
            tma_load4(dst + A_STAGE, &tin, ci0, walk.xb * TC_M - 1, walk.y, walk.n, fb);
            ++issued;
        }
        if (!ok) {
            abort_flag = 1;
            atomicExch(err, 1);
        }
        // the copies in flight land before the CTA leaves, whichever role gave up
        for (int j = issued > NS ? issued - NS : 0; j < issued; ++j)
            mbar_wait(full0 + 8 * (uint32_t)(j % NS), (uint32_t)((j / NS) & 1));
    } else if (warp == 1) {
        bool ok = true;
        const bool leader = elect_one();
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        Ring<NS> st;
        int committed = 0;
        for (int j = 0; j < jobs; ++j, st.next()) {
            const uint32_t s = st.slot;
            if (!mbar_wait_warp(full0 + 8 * s, st.round & 1, &abort_flag)) {
                ok = false;
                break;
            }
            fence_after();
            const uint32_t a0 = base + s * STAGE;
            const Desc da(smem_desc_sw_mn<ROWB_A>(a0, TC_M * ROWB_A));
            const Desc db(smem_desc_sw_mn<ROWB_B>(a0 + A_STAGE, TC_BOX * ROWB_B));
            if (leader) {
#pragma unroll
                for (int ks = 0; ks < TC_M / 16; ++ks) {
#pragma unroll
                    for (int b = 0; b < MB; ++b) {
#pragma unroll
                        for (int kx = 0; kx < 3; ++kx)
                            mma_bf16(tm + (uint32_t)((b * 3 + kx) * NC), da,
                                     (uint32_t)((b * 128 * TC_M * 2 + 16 * ks * ROWB_A) / 16), db,
                                     (uint32_t)((16 * ks + kx) * ROWB_B / 16), IDESC, (j > 0 || ks > 0) ? 1u : 0u);
                    }
                }
                mma_commit(empty0 + 8 * s);
            }
            ++committed;
        }
        // the last commit covers every MMA (they complete in order)
        if (committed > 0 &&
            !mbar_wait_warp(empty0 + 8 * (uint32_t)((committed - 1) % NS), (uint32_t)(((committed - 1) / NS) & 1), nullptr))
            ok = false;
        if (leader) {
            if (!ok) {
                abort_flag = 1;
                atomicExch(err, 1);
            }
            status = ok && committed == jobs ? 1 : 0;
        }
    }
    __syncthreads();
    if (status && jobs > 0) {
        fence_after();
#pragma unroll
        for (int b = 0; b < MB; ++b) {
            const int m = b * 128 + warp * 32 + lane;  // TMEM lane of this thread in block b
            const int ky = 2 - m / CO, co = m % CO;
#pragma unroll 1
            for (int kx = 0; kx < 3; ++kx) {
#pragma unroll 1
                for (int c = 0; c < NC; c += 16) {
                    float v[16];
                    tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((b * 3 + kx) * NC + c), v);
                    if (ky >= 0) {
                        float *d = dw + ((size_t)(ky * 3 + kx) * CO + co) * cin + ci0 + c;
#pragma unroll
                        for (int i = 0; i < 16; i += 4) red_add4(d + i, v[i], v[i + 1], v[i + 2], v[i + 3]);
                    }
                }
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
}

}  // namespace unet_tc
