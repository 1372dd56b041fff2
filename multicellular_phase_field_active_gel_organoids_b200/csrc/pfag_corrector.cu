// Learned coarse-grid corrector: the kernels of a small convolutional network
// (3x3 convolutions, BF16 weights and activations, FP32 accumulation) on the
// 5th-generation tensor cores, for its inference and its training on the GPU.
// No counterpart in the reference (its step has no learned part).
//
// Layout.  An activation tensor is BF16 [B][H+2][W+2][C] (NHWC with a
// one-site zero halo, C a multiple of 8): the halo is the convolution's zero
// padding, so every tap of every pixel reads memory of the same sample.
// Pixels are numbered q = y*(W+2) + x inside a sample.  A weight tensor is
// BF16 [Cout][9][Cin] (tap t = (dy+1)*3 + (dx+1)), i.e. a [Cout][K] matrix with
// K = 9 Cin ordered (tap, channel).
//
// Forward (kc_conv_fwd): implicit GEMM D[q][co] = sum_k A[q][k] B[co][k] over
// tiles of 128 consecutive pixels of the rows 1..H of a sample (halo columns
// included; their outputs are written as zero), SUB tiles a stage.  The CTA
// stages the pixels q0 - (W+2) - 1 .. q0 + 128 SUB + (W+2) + 1 once in shared
// memory as [Cin/8][P][8] (16-byte rows: the canonical no-swizzle K-major
// core-matrix layout, 8 pixels x 8 channels per 128-byte core matrix); the A
// operand of tap t is the same buffer seen from pixel offset
// (W+2)+1 + dy*(W+2) + dx through its matrix descriptor, so there is no
// im2col copy.  One thread issues the 9 Cin/16 tcgen05.mma a tile (M = 128, N =
// Cout, K = 16) into a TMEM accumulator, tcgen05.commit arrives on an mbarrier,
// and each warp reads its 32 rows back with tcgen05.ld for the epilogue (bias,
// GELU, BF16 stores; the pre-activation is kept for training).  Two stages: one
// warp issues the MMAs of stage k while the others copy stage k + 1 and run the
// epilogue of stage k - 1 (mbarriers per stage: staged, MMAs done, accumulator
// read).  The GELU bounds it: a 32 -> 32 layer on 64 boxes of 128^2 takes 90 us
// (153 with one stage, one tile at a time and the three parts one after
// another), the 32 -> 16 layer without GELU 49 (89).
//
// Input gradient (the same kernel, EPI_DGRAD): the convolution of dz with the
// flipped, transposed weights, read straight from the forward layer's; the
// epilogue multiplies by GELU'(pre) of the layer below, so its dz is written at
// once (the separate pass took 51 us on 16 boxes of 128^2).
//
// Weight gradient (kc_conv_wgrad): dW[co][t][ci] = sum_q dZ[q][co] X[q+off_t][ci]
// as D[(dx, co)][ci] per tap row with M = 128 (zero-padded), N = Cin, K = pixels:
// both operands MN-major from the staged [C/8][pixels][8] buffers (a core
// matrix is 8 pixels x 8 channels either way), 3 accumulators of Cin columns
// that live in TMEM across all tiles of the CTA, added to dW at the end; two
// stages, so the next tile's copies and the bias sums run beside the MMAs (one
// stage, 9 accumulators with co alone on the rows, the bias sums of 32 threads
// before the MMAs: 120 us a 32 -> 32 layer on 16 boxes of 128^2, 38 so).
//
// Every wait on an mbarrier is bounded; a wait that runs out sets bit 0 of
// *err and the kernel skips the rest of its work (the host reports it).
#include "pfag_internal.cuh"
#include <cuda_bf16.h>
#include <cstdint>

namespace {

constexpr int KC_THREADS = 256;            // the warps that copy and run the epilogue
constexpr int KC_BLOCK = KC_THREADS + 32;   // and the one that issues the MMAs
// polls before a wait gives up (each suspends the thread for a while by itself)
constexpr long KC_SPIN_LIMIT = 1L << 22;

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// no-swizzle matrix descriptor (version 1): start, leading and stride byte offsets
__device__ __forceinline__ uint64_t mdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

// instruction descriptor of kind::f16: BF16 x BF16 -> F32, M = 128, N, majors
__host__ __device__ constexpr uint32_t idesc_bf16(int n, int a_mn, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// a, b: matrix descriptors as (base, start offset in 16-byte units): the start
// address is the descriptor's low field, so moving it is one 32-bit addition
// (building each descriptor anew kept the issuing thread at about 150 cycles an
// MMA, longer than the MMA)
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint32_t ao, uint64_t b, uint32_t bo,
                                         uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}\n"
        :
        : "r"(tmem_d), "r"((uint32_t)a + ao), "r"((uint32_t)(a >> 32)), "r"((uint32_t)b + bo),
          "r"((uint32_t)(b >> 32)), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t mbar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}

// bounded wait for the given phase parity; false if it ran out
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    for (long it = 0; it < KC_SPIN_LIMIT; it++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// warp 0 allocates `ncols` TMEM columns (a power of two >= 32) and publishes the address
__device__ __forceinline__ void tmem_alloc(uint32_t *slot, int ncols) {
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)),
                     "r"(ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
}

__device__ __forceinline__ void tmem_free(uint32_t taddr, int ncols) {
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 32 lanes x 16 columns of FP32 from TMEM (lane base encoded in taddr)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = __uint_as_float(r[k]);
}

__device__ __forceinline__ void cp16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
    return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

// Stage pixels [q_lo, q_lo + P) of a sample (zero outside [lo, hi)) as
// [C/8][ps][8]; consecutive threads take the chunks of one pixel, so a warp
// reads whole 32-byte sectors.
template <int C>
__device__ __forceinline__ void stage_pixels(unsigned char *dst, int ps, const __nv_bfloat16 *__restrict__ x,
                                             long sample_off, int q_lo, int P, int lo, int hi) {
    constexpr int CH = C / 8;
    for (int e = threadIdx.x; e < P * CH; e += KC_THREADS) {
        const int p = e / CH, c = e - p * CH;
        const int q = q_lo + p;
        unsigned char *d = dst + ((size_t)c * ps + p) * 16;
        if (q >= lo && q < hi) cp16(d, x + (sample_off + q) * C + c * 8);
        else *reinterpret_cast<uint4 *>(d) = make_uint4(0, 0, 0, 0);
    }
}

// 16 BF16 values to global memory; 32 bytes in one store where the address
// allows it (a warp's pixels are a whole sector or two apart either way, but
// half-sector stores take twice the requests)
__device__ __forceinline__ void store16(__nv_bfloat16 *dst, const uint32_t (&v)[8], bool wide) {
    if (wide) {
        asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                     "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                     : "memory");
    } else {
        reinterpret_cast<uint4 *>(dst)[0] = make_uint4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<uint4 *>(dst)[1] = make_uint4(v[4], v[5], v[6], v[7]);
    }
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 h = __halves2bfloat162(__float2bfloat16_rn(a), __float2bfloat16_rn(b));
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ float unpack_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float unpack_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

enum { EPI_LINEAR = 0, EPI_GELU = 1, EPI_DGRAD = 2, EPI_DGRAD_GELU = 3 };

// Y = act(conv3x3(X, W) + bias) on the padded layout (EPI_LINEAR, EPI_GELU; pre
// optional: the pre-activation, same layout as Y), or with w the forward
// layer's weights [CIN][9][COUT] the input gradient of X = dz (EPI_DGRAD), times
// GELU'(pre) of the layer below (EPI_DGRAD_GELU; pre is read).
// CIN, COUT in {16, 32}; SUB tiles of 128 pixels a stage, NST stages.
template <int CIN, int COUT, int EPI, int SUB, int NST>
__global__ void __launch_bounds__(KC_BLOCK, 2) kc_conv_fwd(const __nv_bfloat16 *__restrict__ x,
                                                             const __nv_bfloat16 *__restrict__ w,
                                                             const float *__restrict__ bias,
                                                             __nv_bfloat16 *__restrict__ y,
                                                             __nv_bfloat16 *__restrict__ pre, int B, int H, int W,
                                                             int wide, unsigned *__restrict__ err) {
    constexpr bool DGRAD = EPI == EPI_DGRAD || EPI == EPI_DGRAD_GELU;
    constexpr int TP = 128 * SUB, NCOL = 2 * SUB * COUT < 32 ? 32 : 2 * SUB * COUT;
    extern __shared__ __align__(128) unsigned char kc_smem[];
    // per stage: staged (every copying thread), its MMAs done, its accumulator read
    __shared__ __align__(8) unsigned long long bar_full[2], bar_done[2], bar_read[2];
    __shared__ uint32_t tmem_slot;
    __shared__ float sbias[COUT];
    const int Wp = W + 2, Q = (H + 2) * Wp;
    const int P = TP + 2 * Wp + 2;
    const int tiles_per = (H * Wp + TP - 1) / TP;
    const long ntiles = (long)B * tiles_per;
    unsigned char *ws = kc_smem;                                // weights [9 CIN/8][COUT][8]
    unsigned char *xs = kc_smem + (size_t)9 * CIN * COUT * 2;   // pixels [NST][CIN/8][P][8]
    const size_t xstage = (size_t)CIN / 8 * P * 16;
    if constexpr (DGRAD) {
        // wt[n][t][k] = w[k][8 - t][n]: chunk (t, k / 8) of row n at (chunk COUT + n) 16
        __nv_bfloat16 *wd = reinterpret_cast<__nv_bfloat16 *>(ws);
        for (int e = threadIdx.x; e < 9 * CIN * COUT; e += KC_BLOCK) {
            const int k = e / (9 * COUT), r = e - k * 9 * COUT, t = r / COUT, n = r - t * COUT;
            wd[(((8 - t) * (CIN / 8) + k / 8) * COUT + n) * 8 + k % 8] = w[e];
        }
    } else {
        // weights once: chunk c of row n at (c COUT + n) 16
        for (int e = threadIdx.x; e < 9 * CIN / 8 * COUT; e += KC_BLOCK) {
            const int c = e / COUT, n = e - c * COUT;
            cp16(ws + ((size_t)c * COUT + n) * 16, w + (size_t)n * 9 * CIN + c * 8);
        }
        if (threadIdx.x < COUT) sbias[threadIdx.x] = bias[threadIdx.x];
    }
    if (threadIdx.x == 0) {
        for (int st = 0; st < 2; st++) {
            mbar_init(smem_addr(&bar_full[st]), KC_THREADS);
            mbar_init(smem_addr(&bar_done[st]), 1);
            mbar_init(smem_addr(&bar_read[st]), KC_THREADS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tmem_alloc(&tmem_slot, NCOL);
    cp_wait();
    proxy_fence();                                                // the weights, for the MMAs
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = idesc_bf16(COUT, 0, 0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const auto load = [&](long tile, int st) {
        if (tile >= ntiles) return;
        const int b = (int)(tile / tiles_per), tb = (int)(tile - (long)b * tiles_per);
        stage_pixels<CIN>(xs + st * xstage, P, x, (long)b * Q, tb * TP - 1, P, 0, Q);   // q0 - Wp - 1, q0 = Wp + tb TP
    };
    const auto epilogue = [&](long tile, int acc, bool ok) {
        const int b = (int)(tile / tiles_per), tb = (int)(tile - (long)b * tiles_per);
        const long soff = (long)b * Q;
#pragma unroll 1
        for (int sub = warp >> 2; sub < SUB; sub += KC_THREADS / 128) {
            // row m = 32 (warp % 4) + lane of D (the loads run in every lane
            // whatever the wait gave: tcgen05.ld is warp-collective)
            const int q = Wp + tb * TP + 128 * sub + 32 * (warp & 3) + lane;
            const int yy = q / Wp, xx = q - yy * Wp;
            const bool in = q < (H + 1) * Wp, valid = ok && in && xx >= 1 && xx <= W;
#pragma unroll
            for (int h = 0; h < COUT / 16; h++) {
                const size_t o = (size_t)(soff + (in ? q : 0)) * COUT + 16 * h;
                uint32_t pr[8];
                if constexpr (EPI == EPI_DGRAD_GELU) {
                    const uint4 a = *reinterpret_cast<const uint4 *>(pre + o), c = *reinterpret_cast<const uint4 *>(pre + o + 8);
                    pr[0] = a.x; pr[1] = a.y; pr[2] = a.z; pr[3] = a.w;
                    pr[4] = c.x; pr[5] = c.y; pr[6] = c.z; pr[7] = c.w;
                }
                float v[16];
                tmem_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (acc * SUB + sub) * COUT + 16 * h, v);
                uint32_t out[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    float z[2], g[2];
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        z[i] = v[2 * k + i];
                        if constexpr (!DGRAD) z[i] += sbias[16 * h + 2 * k + i];
                        z[i] = valid ? z[i] : 0.0f;
                        g[i] = z[i];
                        if constexpr (EPI == EPI_GELU) g[i] = valid ? gelu(z[i]) : 0.0f;
                        if constexpr (EPI == EPI_DGRAD_GELU) {
                            const float p = i ? unpack_hi(pr[k]) : unpack_lo(pr[k]);
                            g[i] = valid ? __bfloat162float(__float2bfloat16_rn(z[i])) * gelu_grad(p) : 0.0f;
                        }
                    }
                    out[k] = pack2(g[0], g[1]);
                    if constexpr (!DGRAD) pr[k] = pack2(z[0], z[1]);
                }
                if (in) {
                    store16(y + o, out, wide != 0);
                    if constexpr (!DGRAD)
                        if (pre) store16(pre + o, pr, wide != 0);
                }
            }
        }
    };
    bool ok = true;
    int k = 0;                                                    // this CTA's stage counter
    if (threadIdx.x >= KC_THREADS) {
        // the MMA warp: stage k once it is staged and its accumulator (two, in turn) read
        int issued = -1;                                          // the last stage whose MMAs are under way
        for (long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, k++) {
            const int st = NST == 2 ? k & 1 : 0;
            ok = mbar_wait(smem_addr(&bar_full[st]), NST == 2 ? (k >> 1) & 1 : k & 1);
            if (ok && k >= 2) ok = mbar_wait(smem_addr(&bar_read[k & 1]), ((k - 2) >> 1) & 1);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            if (ok && lane == 0) {
                const uint64_t da = mdesc(smem_addr(xs + st * xstage), (uint32_t)P * 16, 128);
                const uint64_t db = mdesc(smem_addr(ws), COUT * 16, 128);
                const uint32_t acc = tmem + (k & 1) * SUB * COUT;
#pragma unroll
                for (int t = 0; t < 9; t++) {
                    const uint32_t off = 1 + (t / 3) * Wp + (t % 3 - 1);     // Wp + 1 + dy Wp + dx
#pragma unroll
                    for (int j = 0; j < CIN / 16; j++)
#pragma unroll
                        for (int sub = 0; sub < SUB; sub++)
                            mma_bf16(acc + sub * COUT, da, off + 2 * j * P + 128 * sub, db,
                                     (t * (CIN / 8) + 2 * j) * COUT, idesc, (t | j) != 0);
                }
                mma_commit(smem_addr(&bar_done[k & 1]));
            }
            if (ok) issued = k;
            __syncwarp();
        }
        // a wait elsewhere in the block that ran out may have ended it early: the
        // last MMAs still read shared memory and write TMEM, which the block gives up
        if (issued >= 0) ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&bar_done[issued & 1]), (issued >> 1) & 1)) && ok;
    } else {
        const auto finish = [&](long tile, int kk) {              // stage kk's epilogue, its MMAs done
            tc_fence_after();
            epilogue(tile, kk & 1, ok);
            tc_fence_before();
            mbar_arrive(smem_addr(&bar_read[kk & 1]));
        };
        const auto done = [&](int kk) { return mbar_wait(smem_addr(&bar_done[kk & 1]), (kk >> 1) & 1); };
        long prev = -1;                                           // tile whose accumulator waits for its epilogue
        load(blockIdx.x, 0);
        for (long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, k++) {
            cp_wait();
            proxy_fence();
            mbar_arrive(smem_addr(&bar_full[NST == 2 ? k & 1 : 0]));
            if constexpr (NST == 2) {
                // stage k - 1's MMAs are done: its buffer takes stage k + 1
                if (k > 0) ok = __all_sync(0xffffffffu, done(k - 1));
                if (ok) load(tile + gridDim.x, (k + 1) & 1);
                if (prev >= 0) finish(prev, k - 1);
                prev = tile;
            } else {
                ok = __all_sync(0xffffffffu, done(k));
                if (ok) load(tile + gridDim.x, 0);
                finish(tile, k);
            }
        }
        if (NST == 2 && k > 0 && ok) {
            ok = __all_sync(0xffffffffu, done(k - 1));
            finish(prev, k - 1);
        }
        cp_wait();
    }
    if (!ok && lane == 0) atomicOr(err, 1u);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem_free(tmem, NCOL);
}

// dW[co][t][ci] += sum_q dz[q][co] x[q + off_t][ci], db[co] += sum_q dz[q][co]
// (q over rows 1 .. H; dz zero on their halo sites).  CIN, COUT in {16, 32}; NST stages.  M = 128 holds the
// three column shifts of a tap row: with q' = q + dx, tap (dy, dx) is
// sum_q' dz[q' - dx][co] x[q' + dy Wp][ci], so dz is staged three times, shifted
// by one pixel each (rows dx COUT + co), and a tile takes 3 x 8 MMAs instead of
// 9 x 8 with three quarters of the rows empty.
template <int CIN, int COUT, int NST>
__global__ void __launch_bounds__(KC_BLOCK) kc_conv_wgrad(const __nv_bfloat16 *__restrict__ x,
                                                          const __nv_bfloat16 *__restrict__ dz,
                                                          float *__restrict__ dw, float *__restrict__ db, int B, int H,
                                                          int W, int vec, unsigned *__restrict__ err) {
    extern __shared__ __align__(128) unsigned char kc_smem[];
    __shared__ __align__(8) unsigned long long bar_full[2], bar_done[2];
    __shared__ uint32_t tmem_slot;
    __shared__ float sdb[COUT];
    constexpr int NCOL = 3 * CIN <= 64 ? 64 : 128;        // TMEM columns: 3 accumulators (tap rows) of CIN
    constexpr int CG = COUT / 8;
    const int Wp = W + 2, Q = (H + 2) * Wp;
    const int P = 128 + 2 * Wp + 2;
    const int tiles_per = (H * Wp + 127) / 128;
    const long ntiles = (long)B * tiles_per;
    constexpr size_t gstage = (size_t)16 * 128 * 16;
    unsigned char *gs = kc_smem;                             // dz [NST][16][128][8]: 3 shifts x co, padded to 128 rows
    unsigned char *xs = kc_smem + NST * gstage;              // x [NST][CIN/8][P][8]
    const size_t xstage = (size_t)CIN / 8 * P * 16;
    const int lane = threadIdx.x & 31;
    for (int e = threadIdx.x; e < NST * 16 * 128; e += KC_BLOCK)
        *reinterpret_cast<uint4 *>(gs + (size_t)e * 16) = make_uint4(0, 0, 0, 0);
    if (threadIdx.x < COUT) sdb[threadIdx.x] = 0.0f;
    if (threadIdx.x == 0) {
        for (int st = 0; st < 2; st++) {
            mbar_init(smem_addr(&bar_full[st]), KC_THREADS);
            mbar_init(smem_addr(&bar_done[st]), 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tmem_alloc(&tmem_slot, NCOL);
    proxy_fence();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = idesc_bf16(CIN, 1, 1);
    bool ok = true;
    int k = 0;
    if (threadIdx.x >= KC_THREADS) {
        int issued = -1;
        for (long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, k++) {
            const int st = NST == 2 ? k & 1 : 0;
            ok = mbar_wait(smem_addr(&bar_full[st]), NST == 2 ? (k >> 1) & 1 : k & 1);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            if (ok && lane == 0) {
                // A: dz^T (M = shift, co over 16 chunks of 8, K = 16 pixels), MN-major;
                // B: x shifted by tap row r (N = ci, K = 16 pixels), MN-major
                const uint64_t da = mdesc(smem_addr(gs + st * gstage), 128, 128 * 16);
                const uint64_t db = mdesc(smem_addr(xs + st * xstage), 128, (uint32_t)P * 16);
#pragma unroll
                for (int ks = 0; ks < 8; ks++)
#pragma unroll
                    for (int r = 0; r < 3; r++)
                        mma_bf16(tmem + (uint32_t)(r * CIN), da, ks * 16, db, 1 + r * Wp + ks * 16, idesc,
                                 (k == 0 && ks == 0) ? 0u : 1u);
                mma_commit(smem_addr(&bar_done[k & 1]));
            }
            if (ok) issued = k;
            __syncwarp();
        }
        // a wait elsewhere in the block that ran out may have ended it early: the
        // last MMAs still read shared memory and write TMEM, which the block gives up
        if (issued >= 0) ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&bar_done[issued & 1]), (issued >> 1) & 1)) && ok;
    } else {
        const auto load = [&](long tile, int st) {
            if (tile >= ntiles) return;
            const int b = (int)(tile / tiles_per), tb = (int)(tile - (long)b * tiles_per);
            const int q0 = Wp + tb * 128;
            stage_pixels<CIN>(xs + st * xstage, P, x, (long)b * Q, q0 - Wp - 1, P, 0, Q);
            // rows 1 .. H of dz only: its halo rows may hold anything
#pragma unroll
            for (int d = 0; d < 3; d++)
                stage_pixels<COUT>(gs + st * gstage + (size_t)d * CG * 128 * 16, 128, dz, (long)b * Q, q0 + 1 - d, 128, Wp,
                                   (H + 1) * Wp);
        };
        const auto done = [&](int kk) { return mbar_wait(smem_addr(&bar_done[kk & 1]), (kk >> 1) & 1); };
        float bsum[8];                                        // db partials: channels 8 (tid % CG) ..
#pragma unroll
        for (int i = 0; i < 8; i++) bsum[i] = 0.0f;
        // this thread's own copies of the unshifted dz hold the same channels of
        // some pixels (stage_pixels gives thread t chunk t % CG), complete after cp_wait
        const auto bias = [&](int st) {
            const unsigned char *g = gs + st * gstage + (size_t)(CG + threadIdx.x % CG) * 128 * 16;
#pragma unroll
            for (int p = threadIdx.x / CG; p < 128; p += KC_THREADS / CG) {
                const uint4 v = *reinterpret_cast<const uint4 *>(g + p * 16);
                bsum[0] += unpack_lo(v.x); bsum[1] += unpack_hi(v.x);
                bsum[2] += unpack_lo(v.y); bsum[3] += unpack_hi(v.y);
                bsum[4] += unpack_lo(v.z); bsum[5] += unpack_hi(v.z);
                bsum[6] += unpack_lo(v.w); bsum[7] += unpack_hi(v.w);
            }
        };
        load(blockIdx.x, 0);
        for (long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, k++) {
            const int st = NST == 2 ? k & 1 : 0;
            cp_wait();
            proxy_fence();
            mbar_arrive(smem_addr(&bar_full[st]));
            bias(st);
            if constexpr (NST == 2) {
                if (k > 0) ok = __all_sync(0xffffffffu, done(k - 1));
                if (ok) load(tile + gridDim.x, (k + 1) & 1);
            } else {
                ok = __all_sync(0xffffffffu, done(k));
                if (ok) load(tile + gridDim.x, 0);
            }
        }
        if (NST == 2 && k > 0 && ok) ok = __all_sync(0xffffffffu, done(k - 1));
        cp_wait();
#pragma unroll
        for (int i = 0; i < 8; i++) {
            for (int o = 16; o >= CG; o >>= 1) bsum[i] += __shfl_xor_sync(0xffffffffu, bsum[i], o);
            if (lane < CG) atomicAdd(&sdb[(threadIdx.x % CG) * 8 + i], bsum[i]);
        }
    }
    if (!ok && lane == 0) atomicOr(err, 1u);
    ok = __syncthreads_and(ok);
    tc_fence_after();
    if (ok && threadIdx.x < COUT) atomicAdd(&db[threadIdx.x], sdb[threadIdx.x]);
    // rows shift COUT + co of the accumulators: one warp per 32 rows
    if (ntiles > blockIdx.x && ok && threadIdx.x < 32 * ((3 * COUT + 31) / 32)) {
        const int row = threadIdx.x, d = row / COUT, co = row - d * COUT;
#pragma unroll 1
        for (int c0 = 0; c0 < 3 * CIN; c0 += 16) {
            float v[16];
            tmem_ld16(tmem + ((uint32_t)(32 * (threadIdx.x >> 5)) << 16) + (uint32_t)c0, v);
            if (row < 3 * COUT) {
                const int t = (c0 / CIN) * 3 + d, ci = c0 % CIN;
                float *o = dw + ((size_t)co * 9 + t) * CIN + ci;
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    if (vec) {
                        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(o + i), "f"(v[i]),
                                     "f"(v[i + 1]), "f"(v[i + 2]), "f"(v[i + 3])
                                     : "memory");
                    } else {
                        for (int e = 0; e < 4; e++) atomicAdd(o + i + e, v[i + e]);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem_free(tmem, NCOL);
}

// dz = dy * GELU'(pre) (or dy without activation), zero on the halo
template <int C>
__global__ void kc_act_bwd(const __nv_bfloat16 *__restrict__ dy, const __nv_bfloat16 *__restrict__ pre,
                           __nv_bfloat16 *__restrict__ dz, int B, int H, int W, int gelu_on) {
    const int Wp = W + 2, Q = (H + 2) * Wp;
    const long tot = (long)B * Q * C;
    for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (long)gridDim.x * blockDim.x) {
        const long px = e / C;
        const int q = (int)(px % Q), yy = q / Wp, xx = q - yy * Wp;
        float g = 0.0f;
        if (yy >= 1 && yy <= H && xx >= 1 && xx <= W) {
            g = __bfloat162float(dy[e]);
            if (gelu_on) g *= gelu_grad(__bfloat162float(pre[e]));
        }
        dz[e] = __float2bfloat16_rn(g);
    }
}

// wt[ci][t'][co] = w[co][8 - t'][ci]: the input gradient as a forward convolution
__global__ void kc_flip(const __nv_bfloat16 *__restrict__ w, __nv_bfloat16 *__restrict__ wt, int cin, int cout) {
    const int tot = cin * 9 * cout;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += gridDim.x * blockDim.x) {
        const int ci = e / (9 * cout), r = e - ci * 9 * cout, t = r / cout, co = r - t * cout;
        wt[e] = w[((size_t)co * 9 + (8 - t)) * cin + ci];
    }
}

__device__ __forceinline__ void adam_one(float *p, const float *g, float *m, float *v, __nv_bfloat16 *pb, int i,
                                         float mask, bool masked, float lr, float b1, float b2, float eps, float c1,
                                         float c2) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    float step = lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    if (masked) step *= mask;
    const float pi = p[i] - step;
    p[i] = pi;
    if (pb) pb[i] = __float2bfloat16_rn(pi);
}

// Adam on FP32 master weights, BF16 copies for the kernels; `mask` (optional)
// zeroes the update of padded entries.
__global__ void kc_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                        float *__restrict__ v, __nv_bfloat16 *__restrict__ pb, const float *__restrict__ mask, int n,
                        float lr, float b1, float b2, float eps, float c1, float c2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        adam_one(p, g, m, v, pb, i, mask ? mask[i] : 1.0f, mask != nullptr, lr, b1, b2, eps, c1, c2);
}

// The same for several tensors in one launch (blockIdx.y picks the tensor): a
// training step's ten updates took a launch of 2.8 us each.
constexpr int ADAM_MAX = 16;
struct AdamList {
    float *p[ADAM_MAX];
    const float *g[ADAM_MAX];
    float *m[ADAM_MAX], *v[ADAM_MAX];
    __nv_bfloat16 *pb[ADAM_MAX];
    int n[ADAM_MAX];
};
__global__ void kc_adam_list(AdamList L, float lr, float b1, float b2, float eps, float c1, float c2) {
    const int k = blockIdx.y;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L.n[k]; i += gridDim.x * blockDim.x)
        adam_one(L.p[k], L.g[k], L.m[k], L.v[k], L.pb[k], i, 1.0f, false, lr, b1, b2, eps, c1, c2);
}

// mean squared error over the valid sites and the first `nout` channels of
// out (padded, C channels) against target [B][H][W][nout] (FP32); writes the
// gradient into dout (padded, zero elsewhere) and adds the loss sum to *loss
// One thread per padded pixel: whole 32-byte stores, no division per channel
// (per element it took 29 us on 16 boxes of 128^2, 7 so).
template <int C>
__global__ void kc_mse(const __nv_bfloat16 *__restrict__ out, const float *__restrict__ target,
                       __nv_bfloat16 *__restrict__ dout, float *__restrict__ loss, int B, int H, int W, int nout,
                       float scale) {
    const int Wp = W + 2, Q = (H + 2) * Wp;
    const bool vec = ((uintptr_t)dout & 15) == 0;
    float acc = 0.0f;
    for (int b = blockIdx.y; b < B; b += gridDim.y) {
        for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < Q; q += gridDim.x * blockDim.x) {
            const int yy = q / Wp, xx = q - yy * Wp;
            const bool in = yy >= 1 && yy <= H && xx >= 1 && xx <= W;
            const size_t o = ((size_t)b * Q + q) * C;
            const float *t = target + (((size_t)b * H + (in ? yy - 1 : 0)) * W + (in ? xx - 1 : 0)) * nout;
            __align__(16) __nv_bfloat16 v[C];
#pragma unroll
            for (int ch = 0; ch < C; ch++) {
                float g = 0.0f;
                if (in && ch < nout) {
                    const float d = __bfloat162float(out[o + ch]) - t[ch];
                    acc += d * d;
                    g = 2.0f * d * scale;
                }
                v[ch] = __float2bfloat16_rn(g);
            }
            if (vec) {
#pragma unroll
                for (int h = 0; h < C / 8; h++)
                    reinterpret_cast<uint4 *>(dout + o)[h] = reinterpret_cast<const uint4 *>(v)[h];
            } else {
#pragma unroll
                for (int ch = 0; ch < C; ch++) dout[o + ch] = v[ch];
            }
        }
    }
    // one FP32 addition per block: thousands of small ones into the growing total
    // would lose its last bits
    __shared__ float part[8];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < 8; k++) t += part[k];
        atomicAdd(loss, (float)t);
    }
}

// The corrector's input on each cell's FFT box [xc-z+1, xc+z-2]^2:
// x0[n][1+i][1+j] = (phi, rho, s_v vx, s_v vy, 0 ...) scaled, BF16, 16 channels
template <typename real>
__global__ void kc_gather(const real *__restrict__ phi, const real *__restrict__ rho, const real *__restrict__ vx,
                          const real *__restrict__ vy, const int *__restrict__ xc, const int *__restrict__ yc, int N,
                          int z, int M, float s_phi, float s_rho, float s_v, __nv_bfloat16 *__restrict__ x0) {
    const int n = blockIdx.y;
    const int bi = xc[n] - z + 1, bj = yc[n] - z + 1, Mp = M + 2;
    const size_t NN = (size_t)N * N;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < M * M; e += gridDim.x * blockDim.x) {
        const int i = e / M, j = e - i * M;
        const size_t s = (size_t)n * NN + (size_t)(bi + i) * N + bj + j;
        const size_t b = (size_t)n * M * M + e;
        __align__(16) __nv_bfloat16 v[16];
        v[0] = __float2bfloat16_rn((float)phi[s] * s_phi);
        v[1] = __float2bfloat16_rn((float)rho[s] * s_rho);
        v[2] = __float2bfloat16_rn(vx ? (float)vx[b] * s_v : 0.0f);
        v[3] = __float2bfloat16_rn(vy ? (float)vy[b] * s_v : 0.0f);
#pragma unroll
        for (int k = 4; k < 16; k++) v[k] = __float2bfloat16_rn(0.0f);
        uint4 *d = reinterpret_cast<uint4 *>(x0 + (((size_t)n * Mp + 1 + i) * Mp + 1 + j) * 16);
        d[0] = reinterpret_cast<const uint4 *>(v)[0];
        d[1] = reinterpret_cast<const uint4 *>(v)[1];
    }
}

// phi += s_phi out[..0], rho += s_rho out[..1] on each cell's FFT box
template <typename real>
__global__ void kc_apply(const __nv_bfloat16 *__restrict__ out, real *__restrict__ phi, real *__restrict__ rho,
                         const int *__restrict__ xc, const int *__restrict__ yc, int N, int z, int M, float s_phi,
                         float s_rho) {
    const int n = blockIdx.y;
    const int bi = xc[n] - z + 1, bj = yc[n] - z + 1, Mp = M + 2;
    const size_t NN = (size_t)N * N;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < M * M; e += gridDim.x * blockDim.x) {
        const int i = e / M, j = e - i * M;
        const size_t s = (size_t)n * NN + (size_t)(bi + i) * N + bj + j;
        const __nv_bfloat16 *o = out + (((size_t)n * Mp + 1 + i) * Mp + 1 + j) * 16;
        phi[s] = phi[s] + (real)(s_phi * __bfloat162float(o[0]));
        rho[s] = rho[s] + (real)(s_rho * __bfloat162float(o[1]));
    }
}

template <int CIN, int COUT, int EPI, int SUB, int NST>
int launch_fwd_n(const void *x, const void *w, const float *bias, void *y, void *pre, int B, int H, int W, size_t smem,
                 unsigned *err, cudaStream_t s) {
    const int Wp = W + 2;
    const auto fn = kc_conv_fwd<CIN, COUT, EPI, SUB, NST>;
    PFAG_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const long ntiles = (long)B * ((H * Wp + 128 * SUB - 1) / (128 * SUB));
    const int grid = (int)std::min<long>(ntiles, 148L * (smem <= 112 * 1024 ? 2 : 1));
    const int wide = (((uintptr_t)y | (EPI <= EPI_GELU ? (uintptr_t)pre : 0)) & 31) == 0;
    fn<<<grid, KC_BLOCK, smem, s>>>((const __nv_bfloat16 *)x, (const __nv_bfloat16 *)w, bias, (__nv_bfloat16 *)y,
                                      (__nv_bfloat16 *)pre, B, H, W, wide, err);
    PFAG_CUDA_CHECK(cudaGetLastError());
    return PFAG_OK;
}
// two tiles a stage and two stages where they fit in 200 KB (boxes up to 597
// wide for 32 -> 32 channels, 633 for 32 -> 16, 1397 for 16 -> 32, 1433 for 16 ->
// 16), else one of each
template <int CIN, int COUT, int EPI>
int launch_fwd(const void *x, const void *w, const float *bias, void *y, void *pre, int B, int H, int W,
               unsigned *err, cudaStream_t s) {
    const int Wp = W + 2;
    const size_t ws = (size_t)9 * CIN * COUT * 2;
    const auto stage = [&](int sub) { return (size_t)CIN / 8 * (128 * sub + 2 * Wp + 2) * 16; };
    if (ws + stage(1) > 200 * 1024) { pfag_set_error("conv: box width %d too large for the staged tile", W); return PFAG_E_ARG; }
    if (ws + 2 * stage(2) <= 200 * 1024)
        return launch_fwd_n<CIN, COUT, EPI, 2, 2>(x, w, bias, y, pre, B, H, W, ws + 2 * stage(2), err, s);
    return launch_fwd_n<CIN, COUT, EPI, 1, 1>(x, w, bias, y, pre, B, H, W, ws + stage(1), err, s);
}

template <int CIN, int COUT, int NST>
int launch_wgrad_n(const void *x, const void *dz, float *dw, float *db, int B, int H, int W, size_t smem,
                   unsigned *err, cudaStream_t s) {
    const auto fn = kc_conv_wgrad<CIN, COUT, NST>;
    PFAG_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const long ntiles = (long)B * ((H * (W + 2) + 127) / 128);
    // one CTA per SM, each over many tiles
    const int grid = (int)std::min<long>(ntiles, 148L);
    const int vec = ((uintptr_t)dw & 15) == 0;
    fn<<<grid, KC_BLOCK, smem, s>>>((const __nv_bfloat16 *)x, (const __nv_bfloat16 *)dz, dw, db, B, H, W, vec, err);
    PFAG_CUDA_CHECK(cudaGetLastError());
    return PFAG_OK;
}
template <int CIN, int COUT>
int launch_wgrad(const void *x, const void *dz, float *dw, float *db, int B, int H, int W, unsigned *err,
                 cudaStream_t s) {
    const size_t stage = (size_t)16 * 128 * 16 + (size_t)CIN / 8 * (128 + 2 * (W + 2) + 2) * 16;
    if (stage > 200 * 1024) { pfag_set_error("conv: box width %d too large for the staged tile", W); return PFAG_E_ARG; }
    // two stages up to boxes 477 wide for 32 input channels, 1021 for 16
    if (2 * stage <= 200 * 1024) return launch_wgrad_n<CIN, COUT, 2>(x, dz, dw, db, B, H, W, 2 * stage, err, s);
    return launch_wgrad_n<CIN, COUT, 1>(x, dz, dw, db, B, H, W, stage, err, s);
}

}  // namespace

// ---- C ABI ------------------------------------------------------------------
extern "C" int pfag_conv3x3(const void *x, const void *w, const float *bias, void *y, void *pre, int B, int H, int W,
                            int cin, int cout, int gelu_on, unsigned *err, void *stream) {
    if (!x || !w || !bias || !y || !err || B < 1 || H < 1 || W < 1) { pfag_set_error("pfag_conv3x3: bad arguments"); return PFAG_E_ARG; }
    cudaStream_t s = (cudaStream_t)stream;
#define KC_FWD(ci, co)                                                                                         \
    if (cin == ci && cout == co)                                                                               \
        return gelu_on ? launch_fwd<ci, co, EPI_GELU>(x, w, bias, y, pre, B, H, W, err, s)                     \
                       : launch_fwd<ci, co, EPI_LINEAR>(x, w, bias, y, pre, B, H, W, err, s);
    KC_FWD(16, 32) KC_FWD(32, 32) KC_FWD(32, 16) KC_FWD(16, 16)
#undef KC_FWD
    pfag_set_error("pfag_conv3x3: channel pair %d -> %d not built (16/32 -> 16/32)", cin, cout);
    return PFAG_E_UNSUPPORTED;
}

extern "C" int pfag_conv3x3_dgrad(const void *dz, const void *w, const void *pre, void *dx, int B, int H, int W,
                                  int cin, int cout, int gelu_on, unsigned *err, void *stream) {
    if (!dz || !w || !dx || !err || (gelu_on && !pre) || B < 1 || H < 1 || W < 1) { pfag_set_error("pfag_conv3x3_dgrad: bad arguments"); return PFAG_E_ARG; }
    cudaStream_t s = (cudaStream_t)stream;
    void *pr = const_cast<void *>(pre);
#define KC_DG(ci, co)                                                                                          \
    if (cin == ci && cout == co)                                                                               \
        return gelu_on ? launch_fwd<co, ci, EPI_DGRAD_GELU>(dz, w, nullptr, dx, pr, B, H, W, err, s)           \
                       : launch_fwd<co, ci, EPI_DGRAD>(dz, w, nullptr, dx, nullptr, B, H, W, err, s);
    KC_DG(16, 32) KC_DG(32, 32) KC_DG(32, 16) KC_DG(16, 16)
#undef KC_DG
    pfag_set_error("pfag_conv3x3_dgrad: channel pair %d -> %d not built (16/32 -> 16/32)", cin, cout);
    return PFAG_E_UNSUPPORTED;
}

extern "C" int pfag_conv3x3_wgrad(const void *x, const void *dz, float *dw, float *db, int B, int H, int W, int cin,
                                  int cout, unsigned *err, void *stream) {
    if (!x || !dz || !dw || !db || !err || B < 1 || H < 1 || W < 1) { pfag_set_error("pfag_conv3x3_wgrad: bad arguments"); return PFAG_E_ARG; }
    cudaStream_t s = (cudaStream_t)stream;
#define KC_WG(ci, co) \
    if (cin == ci && cout == co) return launch_wgrad<ci, co>(x, dz, dw, db, B, H, W, err, s);
    KC_WG(16, 32) KC_WG(32, 32) KC_WG(32, 16) KC_WG(16, 16)
#undef KC_WG
    pfag_set_error("pfag_conv3x3_wgrad: channel pair %d -> %d not built", cin, cout);
    return PFAG_E_UNSUPPORTED;
}

extern "C" int pfag_conv_act_bwd(const void *dy, const void *pre, void *dz, int B, int H, int W, int c, int gelu_on,
                                 void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (c == 16) kc_act_bwd<16><<<592, 256, 0, s>>>((const __nv_bfloat16 *)dy, (const __nv_bfloat16 *)pre,
                                                    (__nv_bfloat16 *)dz, B, H, W, gelu_on);
    else if (c == 32) kc_act_bwd<32><<<592, 256, 0, s>>>((const __nv_bfloat16 *)dy, (const __nv_bfloat16 *)pre,
                                                         (__nv_bfloat16 *)dz, B, H, W, gelu_on);
    else { pfag_set_error("pfag_conv_act_bwd: %d channels", c); return PFAG_E_UNSUPPORTED; }
    PFAG_CUDA_CHECK(cudaGetLastError());
    return PFAG_OK;
}

extern "C" int pfag_conv_flip(const void *w, void *wt, int cin, int cout, void *stream) {
    kc_flip<<<64, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16 *)w, (__nv_bfloat16 *)wt, cin, cout);
    PFAG_CUDA_CHECK(cudaGetLastError());
    return PFAG_OK;
}

extern "C" int pfag_adam(float *p, const float *g, float *m, float *v, void *pb, const float *mask, int n, float lr,
                         float b1, float b2, float eps, int t, void *stream) {
    if (t < 1) { pfag_set_error("pfag_adam: step t >= 1"); return PFAG_E_ARG; }
    const float c1 = 1.0f - powf(b1, (float)t), c2 = 1.0f - powf(b2, (float)t);
    kc_adam<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(p, g, m, v, (__nv_bfloat16 *)pb, mask, n, lr, b1, b2,
                                                               eps, c1, c2);
    PFAG_CUDA_CHECK(cudaGetLastError());
    return PFAG_OK;
}

extern "C" int pfag_adam_list(int count, float *const *p, const float *const *g, float *const *m, float *const *v,
                              void *const *pb, const int *n, float lr, float b1, float b2, float eps, int t,
                              void *stream) {
    if (t < 1 || count < 1 || count > ADAM_MAX || !p || !g || !m || !v || !pb || !n) {
        pfag_set_error("pfag_adam_list: 1 to %d tensors, step t >= 1", ADAM_MAX);
        return PFAG_E_ARG;
    }
    AdamList L{};
    int most = 1;
    for (int k = 0; k < count; k++) {
        L.p[k] = p[k]; L.g[k] = g[k]; L.m[k] = m[k]; L.v[k] = v[k]; L.pb[k] = (__nv_bfloat16 *)pb[k]; L.n[k] = n[k];
        most = std::max(most, n[k]);
    }
    const float c1 = 1.0f - powf(b1, (float)t), c2 = 1.0f - powf(b2, (float)t);
    kc_adam_list<<<dim3((most + 255) / 256, count), 256, 0, (cudaStream_t)stream>>>(L, lr, b1, b2, eps, c1, c2);
    PFAG_CUDA_CHECK(cudaGetLastError());
    return PFAG_OK;
}

extern "C" int pfag_conv_mse(const void *out, const float *target, void *dout, float *loss, int B, int H, int W,
                             int c, int nout, float scale, void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    const int by = std::max(1, std::min(B, 65535));
    if (c == 16) kc_mse<16><<<dim3(std::max(1, std::min(((H + 2) * (W + 2) + 255) / 256, 296 / by)), by), 256, 0, s>>>(
        (const __nv_bfloat16 *)out, target, (__nv_bfloat16 *)dout, loss, B, H, W, nout, scale);
    else { pfag_set_error("pfag_conv_mse: %d channels", c); return PFAG_E_UNSUPPORTED; }
    PFAG_CUDA_CHECK(cudaGetLastError());
    return PFAG_OK;
}

extern "C" int pfag_corrector_gather(pfag_ctx *c, void *x0, float s_phi, float s_rho, float s_v) {
    if (!c || !x0) { pfag_set_error("pfag_corrector_gather: bad arguments"); return PFAG_E_ARG; }
    const dim3 g((c->M * c->M + 255) / 256, c->Ntot);
    if (c->prec == 64)
        kc_gather<double><<<g, 256, 0, c->stream>>>((const double *)c->phi, (const double *)c->rho,
                                                   (const double *)c->d_vx, (const double *)c->d_vy, c->d_xc, c->d_yc,
                                                   c->N, c->zone, c->M, s_phi, s_rho, s_v, (__nv_bfloat16 *)x0);
    else
        kc_gather<float><<<g, 256, 0, c->stream>>>((const float *)c->phi, (const float *)c->rho,
                                                  (const float *)c->d_vx, (const float *)c->d_vy, c->d_xc, c->d_yc,
                                                  c->N, c->zone, c->M, s_phi, s_rho, s_v, (__nv_bfloat16 *)x0);
    PFAG_CUDA_CHECK(cudaGetLastError());
    return PFAG_OK;
}

extern "C" int pfag_corrector_apply(pfag_ctx *c, const void *out, float s_phi, float s_rho) {
    if (!c || !out) { pfag_set_error("pfag_corrector_apply: bad arguments"); return PFAG_E_ARG; }
    if (c->path != PFAG_PATH_FUSED) { pfag_set_error("pfag_corrector_apply: fused path only"); return PFAG_E_UNSUPPORTED; }
    const dim3 g((c->M * c->M + 255) / 256, c->Ntot);
    if (c->prec == 64)
        kc_apply<double><<<g, 256, 0, c->stream>>>((const __nv_bfloat16 *)out, (double *)c->phi, (double *)c->rho,
                                                  c->d_xc, c->d_yc, c->N, c->zone, c->M, s_phi, s_rho);
    else
        kc_apply<float><<<g, 256, 0, c->stream>>>((const __nv_bfloat16 *)out, (float *)c->phi, (float *)c->rho,
                                                 c->d_xc, c->d_yc, c->N, c->zone, c->M, s_phi, s_rho);
    PFAG_CUDA_CHECK(cudaGetLastError());
    return pfag_fused_recentre(c);
}
