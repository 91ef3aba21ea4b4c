// mlp.cu — the learned orientation proposal network (include/mbs_mlp.h).
//
// 4 -> 128 -> 128 -> 128 -> 1 with erf GELU.  Every layer product runs on
// the 5th-generation tensor cores as BF16 x BF16 -> FP32: tcgen05.mma
// (M = 128, K = 16 per instruction) issued by one thread per CTA, both
// operands in shared memory in the K-major no-swizzle layout (8 x 16-byte
// core matrices), the accumulator in tensor memory, read back with tcgen05.ld.
//
// A training step is two kernels.  k_chain takes 16 samples per CTA through
// the whole forward and backward chain (activations stay in shared memory and
// registers; one MMA chain per layer); k_update forms the weight gradients,
// which sum over all samples, 16 columns per CTA, and applies Adam to them
// in the epilogue.  Operands cross between the two as images of the shared-
// memory tiles, so both kernels stage them with plain bulk copies.  The
// 128 -> 1 head is a per-sample dot product in FP32.  Master parameters,
// gradients and Adam moments are FP32.  All reductions run in a fixed order,
// so training is bitwise repeatable for a given seed.
//
// The step's operations are small (59 MFLOP at 256 samples); what bounds it is
// the chain of dependent passes.  As twenty launches (nine GEMMs and the
// element-wise and reduction kernels between them) a step of 256 samples took
// 134 us; as two with 32 samples per CTA 21 us; now, with 16, gelu and gelu'
// from one erf and each kernel's prologue beside the one before
// (programmatic dependent launch), 18 us; with the epoch's samples laid out in
// its shuffled order and the Adam state loaded under the products, 16 us.
#include "mbs_mlp.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>
#include <string>
#include <vector>

namespace mlp {

constexpr int kH = MBS_MLP_HIDDEN;   // 128
constexpr int kIn = MBS_MLP_IN;      // 4
constexpr int kInPad = 16;           // K of the first layer, padded for the MMA
constexpr int kTile = 128;           // M of one tcgen05.mma tile (batch rows padded to it)

// Flat parameter offsets (include/mbs_mlp.h)
constexpr int oW1 = 0, ob1 = oW1 + kH * kIn, oW2 = ob1 + kH, ob2 = oW2 + kH * kH;
constexpr int oW3 = ob2 + kH, ob3 = oW3 + kH * kH, ow4 = ob3 + kH, ob4 = ow4 + kH;
constexpr int kNParams = ob4 + 1;
static_assert(kNParams == MBS_MLP_N_PARAMS, "parameter layout");

using bf16 = __nv_bfloat16;

__device__ __forceinline__ float gelu(float z)
{
    return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f));
}

// GELU and its derivative from one erf.
__device__ __forceinline__ float gelu_both(float z, float &grad)
{
    const float e = 1.0f + erff(z * 0.70710678118654752f);
    grad = 0.5f * e + z * 0.39894228040143268f * expf(-0.5f * z * z);
    return 0.5f * z * e;
}

// Programmatic dependent launch: the next kernel of the stream may start its
// prologue; nothing global is touched before grid_wait (the kernels before
// have completed and their writes are visible then).
__device__ __forceinline__ void grid_release()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void grid_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ---- tcgen05 helpers --------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor, K-major without swizzle: start address,
// leading byte offset (between the two 8-element core matrices along K),
// stride byte offset (between 8-row groups), version 1, swizzle none.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16)
         | ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N and M of the tile.
__host__ __device__ constexpr uint32_t umma_idesc(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Byte offset of element (row, k) in a K-major no-swizzle tile whose rows hold
// kt elements: core matrix (row / 8, k / 8), 16 bytes per row inside it.
__device__ __forceinline__ uint32_t kmajor_off(int row, int k, int kt)
{
    return (uint32_t)((row >> 3) * (kt * 16) + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

// Bounded wait on an mbarrier phase (at most `limit` polls); false when it
// did not complete.
constexpr int kDefaultPollLimit = 1 << 22;

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase, int limit)
{
    for (int it = 0; it < limit; ++it) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred P1;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
                     "selp.b32 %0, 1, 0, P1;\n\t}"
                     : "=r"(done) : "r"(bar), "r"(phase) : "memory");
        if (done)
            return true;
    }
    return false;
}

// Watchdog of the tensor-core barrier waits: the device error flag, the
// poll limit, and (test hook) whether to leave out the MMAs and their
// commit, so that the wait runs out with no asynchronous operation pending.
struct Watch {
    int *err;
    int poll_limit;
    int skip_mma;
};

// ---- operand images ----------------------------------------------------
// A K-major tile of R rows and 128 k in its shared-memory layout (kmajor_off
// with kt = 128): 2,048 bytes per 8 rows.  Weights: the forward operand of
// layer l holds (row = output, k = input), the backward one (row = input,
// k = output).  Activations and gradients, transposed for the weight
// gradients: one image per 128 samples, (row = column of the layer, k = sample).
constexpr int kImg = kH * kTile;           // elements of a 128-row image
constexpr int kImgX = kInPad * kTile;      // of the input's 16-row image
struct Weights {
    bf16 *w1f;          // (output, input) with kt = 16
    bf16 *w2f, *w3f;    // forward
    bf16 *w2b, *w3b;    // backward
};
struct Images {
    bf16 *x0, *h1, *h2, *h3, *dz1, *dz2, *dz3;
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(1));
}

__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}

// kt / 16 MMAs over a staged tile pair (M = 128, N columns), then the commit;
// one thread.
__device__ __forceinline__ void mma_chain(uint32_t tmem, uint32_t a, uint32_t b, int kt, int N, bool accumulate,
                                          uint32_t bar)
{
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t idesc = umma_idesc(kTile, N), sbo = (uint32_t)kt * 16;
    for (int s = 0; s < kt / 16; ++s) {
        const uint64_t da = umma_desc(a + 256 * s, 128, sbo);
        const uint64_t db = umma_desc(b + 256 * s, 128, sbo);
        const uint32_t acc = (accumulate || s > 0) ? 1u : 0u;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "setp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     :: "r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(acc));
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(bar) : "memory");
}

// N accumulator columns (4 or 8) of the warp's 32 tensor-memory lanes.
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t ta, float *f)
{
    uint32_t v[N];
    if constexpr (N == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                     : "r"(ta));
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(ta));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i)
        f[i] = __uint_as_float(v[i]);
}

// ---- forward and backward chain of a CTA's samples -----------------------
// Samples per CTA: 16 in training (a step has few samples, and the element-wise
// work of a CTA is what its chain waits for), 32 in inference (each CTA loads
// all weights).  The weights are the M = 128 operand and the samples the N
// operand, so an accumulator row is a unit of the layer (tensor-memory lane)
// and its columns are the samples: every warp reads its lane quarter straight
// into registers, and a unit's consecutive samples are what the images hold.
// (Samples as the M operand filled 16 of 128 rows, eight times the MMA time,
// and their accumulators went through shared memory twice per layer.)
constexpr int kTrainRows = 16, kFwdRows = 32;
constexpr int kChainThreads = 512;   // warp = (lane quarter of the units, a quarter of the samples)

// shared memory: weight operands, sample tile, input tile, small arrays
template <bool kTrain, int kRows>
struct ChainSmem {
    static constexpr int W1 = 0, W2f = W1 + kH * kInPad * 2, W3f = W2f + 2 * kImg;
    static constexpr int W3b = W3f + 2 * kImg, W2b = W3b + (kTrain ? 2 * kImg : 0);
    static constexpr int H = W2b + (kTrain ? 2 * kImg : 0), X = H + kRows * kH * 2;
    static constexpr int vec = X + kRows * kInPad * 2, bar = vec + (4 * kH + 3 * kRows) * 4, bytes = bar + 64;
};
static_assert(ChainSmem<true, kTrainRows>::bytes <= 227 * 1024, "shared memory of one CTA");

struct ChainArgs {
    const float *q, *t;      // samples [n][4] and targets
    int n;                   // samples of this batch; the rows beyond are padding
    const float *params;
    Weights w;
    Images img;              // training only
    float *y, *dy;
    Watch watch;
};

template <bool kTrain, int kRows>
__global__ void __launch_bounds__(kChainThreads, 1) k_chain(ChainArgs a)
{
    using L = ChainSmem<kTrain, kRows>;
    constexpr int kV = kRows / 4;                          // samples of a thread
    extern __shared__ __align__(1024) unsigned char sm[];
    const uint32_t sbase = smem_u32(sm);
    float *sb = reinterpret_cast<float *>(sm + L::vec);    // b1, b2, b3, w4
    float *st = sb + 4 * kH, *sdy = st + kRows;
    const uint32_t bars = sbase + L::bar;                  // [0] MMA, [1] w1f, w2f, [2] w3f, [3] w3b, w2b
    uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + L::bar + 48);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r0 = blockIdx.x * kRows;
    const int unit = (warp & 3) * 32 + lane, s0 = (warp >> 2) * kV;   // this thread's accumulators
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(tslot)), "r"(32));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int i = 0; i < 4; ++i)
            mbar_init(bars + 8 * i);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (kTrain) {
        grid_release();
        grid_wait();
    }
    int failed = 0;
    if (tid == 0) {
        mbar_expect(bars + 8, kH * kInPad * 2 + 2 * kImg);
        bulk_load(sbase + L::W1, a.w.w1f, kH * kInPad * 2, bars + 8);
        bulk_load(sbase + L::W2f, a.w.w2f, 2 * kImg, bars + 8);
        mbar_expect(bars + 16, 2 * kImg);
        bulk_load(sbase + L::W3f, a.w.w3f, 2 * kImg, bars + 16);
        if (kTrain) {
            mbar_expect(bars + 24, 4 * kImg);
            bulk_load(sbase + L::W3b, a.w.w3b, 2 * kImg, bars + 24);
            bulk_load(sbase + L::W2b, a.w.w2b, 2 * kImg, bars + 24);
        }
        failed = *a.watch.err;   // a step before this one failed: nothing more is computed
    }
    if (tid < kRows) {   // a sample's input row: the quaternion, zeros to 16 columns
        const int r = r0 + tid;
        float4 qv = make_float4(0.f, 0.f, 0.f, 0.f);
        float tv = 0.f;
        if (r < a.n) {
            qv = make_float4(a.q[r * kIn], a.q[r * kIn + 1], a.q[r * kIn + 2], a.q[r * kIn + 3]);
            if (kTrain)
                tv = a.t[r];
        }
        st[tid] = tv;
        const bf16 z = __float2bfloat16(0.f);
        __align__(16) const bf16 v[8] = {__float2bfloat16(qv.x), __float2bfloat16(qv.y), __float2bfloat16(qv.z),
                                         __float2bfloat16(qv.w), z, z, z, z};
        *reinterpret_cast<uint4 *>(sm + L::X + kmajor_off(tid, 0, kInPad)) = *reinterpret_cast<const uint4 *>(v);
        *reinterpret_cast<uint4 *>(sm + L::X + kmajor_off(tid, 8, kInPad)) = make_uint4(0u, 0u, 0u, 0u);
    }
    for (int i = tid; i < 4 * kH; i += kChainThreads)
        sb[i] = a.params[i < kH ? ob1 + i : i < 2 * kH ? ob2 + i - kH : i < 3 * kH ? ob3 + i - 2 * kH : ow4 + i - 3 * kH];
    const float b4 = a.params[ob4];
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    bool ok = !__syncthreads_or(failed);
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tslot;
    uint32_t phase = 0;
    int loaded = 0;            // weight barriers waited for so far
    // One layer product W (128 x kt) times the staged samples: this thread's
    // accumulators.  `wbar`: the barrier of the weight operand.
    auto layer = [&](int woff, int soff, int kt, int wbar, float *v) {
        while (loaded < wbar && ok) {   // every thread: the MMA's own wait starts after it
            ++loaded;
            ok = mbar_wait(bars + 8 * loaded, 0, kDefaultPollLimit);
        }
        if (tid == 0 && ok && !a.watch.skip_mma)
            mma_chain(tmem, sbase + woff, sbase + soff, kt, kRows, false, bars);
        const bool done = mbar_wait(bars, phase, a.watch.poll_limit);
        phase ^= 1u;
        ok = __syncthreads_and(ok && done);
        if (!ok)
            return;
        asm volatile("tcgen05.fence::after_thread_sync;");
        tmem_ld<kV>(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)s0, v);
        asm volatile("tcgen05.fence::before_thread_sync;");
    };
    // This thread's values of a layer, BF16: into the sample tile (the next
    // product's operand) and, in training, into an image.
    auto put = [&](const float *v, bf16 *img, bool tile) {
        __align__(16) bf16 h[kV];
#pragma unroll
        for (int i = 0; i < kV; ++i) {
            h[i] = __float2bfloat16(v[i]);
            if (tile)
                *reinterpret_cast<bf16 *>(sm + L::H + kmajor_off(s0 + i, unit, kTile)) = h[i];
        }
        if (kTrain) {
            unsigned char *dst = reinterpret_cast<unsigned char *>(img + (size_t)(r0 / kTile) * kImg)
                               + kmajor_off(unit, (r0 & (kTile - 1)) + s0, kTile);
            if constexpr (kV == 4)
                *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(h);
            else
                *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(h);
        }
        if (tile) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
        }
    };
    float g1[kV], g2[kV], g3[kV], v[kV];   // gelu' of each layer
    auto forward = [&](float *g, int layer_no, bf16 *img) {
        const float bias = sb[layer_no * kH + unit];
        float h[kV];
#pragma unroll
        for (int i = 0; i < kV; ++i) {
            const float z = v[i] + bias;
            h[i] = kTrain ? gelu_both(z, g[i]) : gelu(z);
        }
        put(h, img, true);
    };
    auto backward = [&](const float *g, bf16 *img, bool tile) {
#pragma unroll
        for (int i = 0; i < kV; ++i)
            v[i] = v[i] * g[i];
        put(v, img, tile);
    };
    if (ok)
        layer(L::W1, L::X, kInPad, 1, v);
    if (ok) {
        forward(g1, 0, a.img.h1);
        layer(L::W2f, L::H, kH, 1, v);
    }
    if (ok) {
        forward(g2, 1, a.img.h2);
        layer(L::W3f, L::H, kH, 2, v);
    }
    if (ok) {
        forward(g3, 2, a.img.h3);
        // y = sum_j H3[j] w4[j] + b4: a warp per sample, fixed lane order
        for (int r = warp; r < kRows; r += kChainThreads / 32) {
            float s = 0.f;
            for (int j = lane; j < kH; j += 32)
                s = fmaf(__bfloat162float(*reinterpret_cast<const bf16 *>(sm + L::H + kmajor_off(r, j, kTile))),
                         sb[3 * kH + j], s);
#pragma unroll
            for (int w = 16; w > 0; w >>= 1)
                s += __shfl_xor_sync(0xffffffffu, s, w);
            if (lane == 0) {
                const float yv = s + b4;
                if (r0 + r < a.n)
                    a.y[r0 + r] = yv;
                // dy = 2 (y - t) / n (0 on padding rows)
                const float d = r0 + r < a.n ? 2.f * (yv - st[r]) / (float)a.n : 0.f;
                sdy[r] = d;
                if (kTrain)
                    a.dy[r0 + r] = d;
            }
        }
        __syncthreads();
    }
    if (kTrain && ok) {
        // dZ3 = dy w4 gelu'(Z3), dZ2 = (dZ3 W3) gelu'(Z2), dZ1 = (dZ2 W2) gelu'(Z1)
        const float w4 = sb[3 * kH + unit];
#pragma unroll
        for (int i = 0; i < kV; ++i)
            v[i] = sdy[s0 + i] * w4;
        backward(g3, a.img.dz3, true);
        layer(L::W3b, L::H, kH, 3, v);
        if (ok) {
            backward(g2, a.img.dz2, true);
            layer(L::W2b, L::H, kH, 3, v);
        }
        if (ok)
            backward(g1, a.img.dz1, false);
        if (tid < kInPad * (kRows / 8)) {   // the input's image: (column, 8 samples)
            const int col = tid & (kInPad - 1), rg = tid / kInPad;
            __align__(16) bf16 x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                x[i] = *reinterpret_cast<const bf16 *>(sm + L::X + kmajor_off(rg * 8 + i, col, kInPad));
            unsigned char *dst = reinterpret_cast<unsigned char *>(a.img.x0 + (size_t)(r0 / kTile) * kImgX);
            *reinterpret_cast<uint4 *>(dst + kmajor_off(col, (r0 & (kTile - 1)) + rg * 8, kTile)) =
                *reinterpret_cast<const uint4 *>(x);
        }
    }
    if (!ok && tid == 0) {
        atomicExch(a.watch.err, 1);
        mbar_wait(bars, phase ^ 1u, a.watch.poll_limit);   // any MMA in flight, bounded
        for (int i = loaded + 1; i <= (kTrain ? 3 : 2); ++i)
            mbar_wait(bars + 8 * i, 0, kDefaultPollLimit);  // copies in flight, bounded
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(32));
}

// ---- weight gradients and Adam -------------------------------------------
struct UpdateArgs {
    Images img;
    const float *dy;
    int bp;                  // padded samples (a multiple of 128)
    float *grad;             // plain gradients out (null: Adam)
    float *p, *m, *v;        // parameters and Adam moments
    float lr;
    const float *bc;         // bias corrections of step j at [2 j], [2 j + 1]
    const int *epoch;
    int steps_per_epoch, k;  // this step: epoch * steps_per_epoch + k
    Weights w;
    Watch watch;
};

// Adam state of N consecutive parameters (1, or 4 as vectors): loaded while the
// gradients are still being formed, then updated with the step's bias
// corrections and stored.
template <int N>
struct AdamState {
    float m[N], v[N], p[N];
    __device__ __forceinline__ void load(const UpdateArgs &a, int i)
    {
        if constexpr (N == 4) {
            const float4 x = *reinterpret_cast<const float4 *>(a.m + i);
            const float4 y = *reinterpret_cast<const float4 *>(a.v + i);
            const float4 z = *reinterpret_cast<const float4 *>(a.p + i);
            m[0] = x.x; m[1] = x.y; m[2] = x.z; m[3] = x.w;
            v[0] = y.x; v[1] = y.y; v[2] = y.z; v[3] = y.w;
            p[0] = z.x; p[1] = z.y; p[2] = z.z; p[3] = z.w;
        } else {
            m[0] = a.m[i];
            v[0] = a.v[i];
            p[0] = a.p[i];
        }
    }
    __device__ __forceinline__ void step(const UpdateArgs &a, int i, const float *g, float bc1, float bc2)
    {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float gi = g[k];
            const float mi = 0.9f * m[k] + 0.1f * gi;
            const float vi = 0.999f * v[k] + 0.001f * gi * gi;
            m[k] = mi;
            v[k] = vi;
            p[k] = p[k] - a.lr * (mi / bc1) / (sqrtf(vi / bc2) + 1e-8f);
        }
        if constexpr (N == 4) {
            *reinterpret_cast<float4 *>(a.m + i) = make_float4(m[0], m[1], m[2], m[3]);
            *reinterpret_cast<float4 *>(a.v + i) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4 *>(a.p + i) = make_float4(p[0], p[1], p[2], p[3]);
        } else {
            a.m[i] = m[0];
            a.v[i] = v[0];
            a.p[i] = p[0];
        }
    }
};

// CTAs: 8 of 16 columns each for dW3 = dZ3^T H2 and dW2 = dZ2^T H1, one for
// dW1 = dZ1^T X0, then the vectors, 32 entries a CTA: db3, db2, db1 (column
// sums of dZ) and the head's dw4, db4.  Both operands of a product are
// contiguous pieces of the images, copied 128 samples at a time into two
// stages; thread 0 copies and issues the MMAs.  The Adam update,
// a chain of divisions and a square root per parameter, takes half of the
// kernel's 6.7 us: four parameters per thread (1638 samples, 100 epochs: 11.60
// ms) rather than eight with 256 threads (11.82) or two with 1024 (12.19).
constexpr int kUpThreads = 512;
constexpr int kUpN = 16;
constexpr int kUpStage = 2 * kImg + kUpN * kTile * 2;
constexpr int kUpSmem = 2 * kUpStage + 64;
constexpr int kJobsW = kH / kUpN, kJobW1 = 2 * kJobsW, kJobBias = kJobW1 + 1, kJobHead = kJobBias + 3 * (kH / 32);
constexpr int kUpJobs = kJobHead + kH / 32 + 1;

__device__ __forceinline__ float image_at(const bf16 *img, int c, int row)
{
    return __bfloat162float(*reinterpret_cast<const bf16 *>(
        reinterpret_cast<const unsigned char *>(img + (size_t)(row / kTile) * kImg)
        + kmajor_off(c, row & (kTile - 1), kTile)));
}

template <bool kAdam>
__global__ void __launch_bounds__(kUpThreads) k_update(UpdateArgs a)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ float part[8][32];
    __shared__ int s_ok;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int job = blockIdx.x;
    float bc1 = 0.f, bc2 = 0.f;
    auto corrections = [&]() {
        if (kAdam) {
            const int j = (*a.epoch) * a.steps_per_epoch + a.k;
            bc1 = a.bc[2 * j];
            bc2 = a.bc[2 * j + 1];
        }
    };
    grid_release();
    const uint32_t sbase = smem_u32(sm), bars = sbase + 2 * kUpStage;   // full[2], MMA[2]
    uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + 2 * kUpStage + 48);
    if (job < kJobBias) {
        if (warp == 0) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                         :: "r"(smem_u32(tslot)), "r"(32));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        }
        if (tid == 0) {
            for (int i = 0; i < 4; ++i)
                mbar_init(bars + 8 * i);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
    }
    grid_wait();
    if (job >= kJobBias) {
        // vectors: 8 row groups g take rows g, g + 8, ... in turn, the group
        // sums are added in group order
        const int g = warp;
        float s = 0.f;
        int idx = -1;
        if (g >= 8)
            return;                            // 8 warps work, and wait for each other below
        if (job < kJobHead) {
            const int l = (job - kJobBias) / (kH / 32), c = (job - kJobBias) % (kH / 32) * 32 + lane;
            const bf16 *x = l == 0 ? a.img.dz3 : l == 1 ? a.img.dz2 : a.img.dz1;
            idx = (l == 0 ? ob3 : l == 1 ? ob2 : ob1) + c;
#pragma unroll 8
            for (int r = g; r < a.bp; r += 8)
                s += image_at(x, c, r);
        } else {
            const int j = (job - kJobHead) * 32 + lane;
            if (j <= kH) {
                idx = j < kH ? ow4 + j : ob4;
#pragma unroll 8
                for (int b = g; b < a.bp; b += 8)
                    s += j < kH ? a.dy[b] * image_at(a.img.h3, j, b) : a.dy[b];
            }
        }
        part[g][lane] = s;
        AdamState<1> ad;
        int failed = 0;
        if (g == 0)
            failed = *a.watch.err;
        if (g == 0 && idx >= 0 && kAdam) {
            ad.load(a, idx);
            corrections();
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (g == 0 && idx >= 0 && !failed) {
            float t = part[0][lane];
            for (int k = 1; k < 8; ++k)
                t += part[k][lane];
            if (kAdam)
                ad.step(a, idx, &t, bc1, bc2);
            else
                a.grad[idx] = t;
        }
        return;
    }
    const int l = job < kJobsW ? 3 : job < kJobW1 ? 2 : 1;
    const int n0 = l == 1 ? 0 : (job % kJobsW) * kUpN;
    const bf16 *A = l == 3 ? a.img.dz3 : l == 2 ? a.img.dz2 : a.img.dz1;
    const bf16 *B = l == 3 ? a.img.h2 : l == 2 ? a.img.h1 : a.img.x0;
    const size_t bstep = l == 1 ? kImgX : kImg;
    B += n0 * kTile;         // 8 rows of an image are 8 * 128 consecutive elements
    const int nblk = a.bp / kTile;
    int issued = 0, waited = 0, committed = 0;
    auto load = [&]() {
        const uint32_t d = sbase + (issued & 1) * kUpStage, bar = bars + 8 * (issued & 1);
        mbar_expect(bar, kUpStage);
        bulk_load(d, A + (size_t)issued * kImg, 2 * kImg, bar);
        bulk_load(d + 2 * kImg, B + (size_t)issued * bstep, kUpN * kTile * 2, bar);
        ++issued;
    };
    int failed = 0;
    if (tid == 0) {
        load();
        if (nblk > 1)
            load();
        failed = *a.watch.err;   // the chain or a step before it failed: nothing is stored
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    const bool run = !__syncthreads_or(failed);
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tslot;
    // accumulator row 32 (w % 4) + lane (the warp's lane quarter), columns
    // 4 (w / 4) .. + 3; their Adam state comes while the products run
    const int r = (warp & 3) * 32 + lane, cl = (warp >> 2) * 4, c = n0 + cl;
    const bool own = l != 1 || cl < kIn;       // dW1: the padding columns have no parameter
    const int i0 = l == 1 ? oW1 + r * kIn + c : (l == 3 ? oW3 : oW2) + r * kH + c;
    AdamState<4> ad;
    if (kAdam) {
        if (own)
            ad.load(a, i0);
        corrections();
    }
    if (tid == 0) {
        bool ok = run;
        for (int i = 0; i < nblk && ok; ++i) {
            ok = mbar_wait(bars + 8 * (i & 1), (i >> 1) & 1, kDefaultPollLimit);
            waited = i + 1;
            if (!ok)
                break;
            if (!a.watch.skip_mma) {
                const uint32_t d = sbase + (i & 1) * kUpStage;
                mma_chain(tmem, d, d + 2 * kImg, kTile, kUpN, i > 0, bars + 16 + 8 * (i & 1));
                committed = i + 1;
            }
            if (issued < nblk) {   // the stage is free once its MMAs are done
                ok = mbar_wait(bars + 16 + 8 * (i & 1), (i >> 1) & 1, a.watch.poll_limit);
                if (ok)
                    load();
            }
        }
        if (ok)
            ok = mbar_wait(bars + 16 + 8 * ((nblk - 1) & 1), ((nblk - 1) >> 1) & 1, a.watch.poll_limit);
        if (!ok) {
            atomicExch(a.watch.err, 1);
            for (int i = waited; i < issued; ++i)       // copies in flight, bounded
                mbar_wait(bars + 8 * (i & 1), (i >> 1) & 1, kDefaultPollLimit);
            if (committed > 0)                          // and MMAs
                mbar_wait(bars + 16 + 8 * ((committed - 1) & 1), ((committed - 1) >> 1) & 1, a.watch.poll_limit);
        }
        s_ok = ok;
    }
    __syncthreads();
    if (s_ok) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        float gv[4];
        tmem_ld<4>(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)cl, gv);
        if (own && !kAdam)
            *reinterpret_cast<float4 *>(a.grad + i0) = make_float4(gv[0], gv[1], gv[2], gv[3]);
        if (own && kAdam) {
            ad.step(a, i0, gv, bc1, bc2);
            __align__(8) bf16 h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                h[k] = __float2bfloat16(ad.p[k]);
            unsigned char *wf = reinterpret_cast<unsigned char *>(l == 1 ? a.w.w1f : l == 3 ? a.w.w3f : a.w.w2f);
            *reinterpret_cast<uint2 *>(wf + kmajor_off(r, c, l == 1 ? kInPad : kTile)) = *reinterpret_cast<const uint2 *>(h);
            if (l != 1) {
                unsigned char *wb = reinterpret_cast<unsigned char *>(l == 3 ? a.w.w3b : a.w.w2b);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    *reinterpret_cast<bf16 *>(wb + kmajor_off(c + k, r, kTile)) = h[k];
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(32));
}

// Weight operand images of the master parameters (W1's padding columns zero).
__global__ void k_refresh(const float *params, Weights w)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kH * kInPad) {
        const int r = i / kInPad, c = i - r * kInPad;
        *reinterpret_cast<bf16 *>(reinterpret_cast<unsigned char *>(w.w1f) + kmajor_off(r, c, kInPad)) =
            __float2bfloat16(c < kIn ? params[oW1 + r * kIn + c] : 0.f);
    }
    if (i < kH * kH) {
        const int r = i / kH, c = i - r * kH;
        const bf16 v2 = __float2bfloat16(params[oW2 + i]), v3 = __float2bfloat16(params[oW3 + i]);
        const uint32_t f = kmajor_off(r, c, kTile), b = kmajor_off(c, r, kTile);
        *reinterpret_cast<bf16 *>(reinterpret_cast<unsigned char *>(w.w2f) + f) = v2;
        *reinterpret_cast<bf16 *>(reinterpret_cast<unsigned char *>(w.w3f) + f) = v3;
        *reinterpret_cast<bf16 *>(reinterpret_cast<unsigned char *>(w.w2b) + b) = v2;
        *reinterpret_cast<bf16 *>(reinterpret_cast<unsigned char *>(w.w3b) + b) = v3;
    }
}

// Mean-squared loss of n samples, one CTA, fixed-order tree sum.
__global__ void __launch_bounds__(256) k_loss(const float *y, const float *t, int n, float *out)
{
    __shared__ float red[256];
    float s = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float d = y[i] - t[i];
        s = fmaf(d, d, s);
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w)
            red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        *out = red[0] / (float)max(n, 1);
}

// Start of a captured epoch: the epoch counter moves on (it starts at -1) and
// the samples are laid out in the epoch's shuffled order idx[epoch][n], so the
// steps read theirs without a chain of dependent loads.
__global__ void __launch_bounds__(1024) k_epoch(const float4 *q, const float *t, const int *idx, int n, int *epoch,
                                                float4 *sq, float *st)
{
    const int e = *epoch + 1;
    for (int i = threadIdx.x; i < n; i += 1024) {
        const int k = idx[(size_t)e * n + i];
        sq[i] = q[k];
        st[i] = t[k];
    }
    __syncthreads();
    if (threadIdx.x == 0)
        *epoch = e;
}

inline int pad_rows(int n) { return (n + kTile - 1) / kTile * kTile; }

}  // namespace mlp

using namespace mlp;

// Device memory of a training call that the network keeps for the next one (a
// cudaMalloc and cudaFree per call took 0.85 ms of a 13 ms fit).
constexpr size_t kBlockKeep = (size_t)64 << 20;

struct mbs_mlp {
    int device = 0;
    cudaStream_t stream = nullptr, upload = nullptr;   // upload: the training orders
    std::string err;
    float *params = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
    bf16 *wimg = nullptr;                 // weight operand images
    Weights w{};
    int step = 0;
    unsigned char *block = nullptr;       // a training call's device arrays, kept between calls
    size_t block_cap = 0;
    // samples for up to `cap` padded rows, activation images for `icap`
    int cap = 0, icap = 0;
    bf16 *acts = nullptr;
    Images img{};
    float *y = nullptr, *t = nullptr, *dy = nullptr, *q = nullptr;
    float *scalar = nullptr;
    int poll_limit = kDefaultPollLimit;   // mbs_mlp_set_watchdog
    int skip_mma = 0;
};

namespace {

int mfail(mbs_mlp *net, int code, const std::string &msg)
{
    if (net)
        net->err = msg;
    return code;
}

#define MK(expr, where)                                                          \
    do {                                                                         \
        cudaError_t e_ = (expr);                                                 \
        if (e_ != cudaSuccess)                                                   \
            return mfail(net, -3, std::string(where) + ": " + cudaGetErrorString(e_)); \
    } while (0)

void free_acts(mbs_mlp *net)
{
    void *ps[] = {net->y, net->t, net->dy, net->q};
    for (void *p : ps)
        cudaFree(p);
    net->y = net->t = net->dy = net->q = nullptr;
    net->cap = 0;
}

int ensure_acts(mbs_mlp *net, int rows)
{
    const int need = pad_rows(std::max(rows, 1));
    if (need <= net->cap)
        return 0;
    free_acts(net);
    MK(cudaMalloc((void **)&net->y, need * sizeof(float)), "cudaMalloc mlp");
    MK(cudaMalloc((void **)&net->t, need * sizeof(float)), "cudaMalloc mlp");
    MK(cudaMalloc((void **)&net->dy, need * sizeof(float)), "cudaMalloc mlp");
    MK(cudaMalloc((void **)&net->q, (size_t)need * kIn * sizeof(float)), "cudaMalloc mlp");
    net->cap = need;
    return 0;
}

// Activation and gradient images of a batch of `rows` samples.
int ensure_images(mbs_mlp *net, int rows)
{
    const int need = pad_rows(std::max(rows, 1));
    if (need <= net->icap)
        return 0;
    cudaFree(net->acts);
    net->acts = nullptr;
    net->icap = 0;
    const size_t one = (size_t)need * kH;
    MK(cudaMalloc((void **)&net->acts, (6 * one + (size_t)need * kInPad) * sizeof(bf16)), "cudaMalloc mlp");
    Images &g = net->img;
    g.h1 = net->acts;
    g.h2 = g.h1 + one;
    g.h3 = g.h2 + one;
    g.dz1 = g.h3 + one;
    g.dz2 = g.dz1 + one;
    g.dz3 = g.dz2 + one;
    g.x0 = g.dz3 + one;
    net->icap = need;
    return 0;
}

// Device flag set by a GEMM whose tensor-core barrier wait ran out (the
// third int of the network's scalar scratch).
int *mlp_err(mbs_mlp *net) { return reinterpret_cast<int *>(net->scalar) + 2; }

Watch watch(mbs_mlp *net) { return Watch{mlp_err(net), net->poll_limit, net->skip_mma}; }

// Reset before a call's kernels, checked after its final synchronisation.
int check_err(mbs_mlp *net)
{
    int e = 0;
    MK(cudaMemcpy(&e, mlp_err(net), sizeof(int), cudaMemcpyDeviceToHost), "D2H error flag");
    if (e) {
        cudaMemset(mlp_err(net), 0, sizeof(int));
        return mfail(net, -6, "tensor-core barrier wait timed out");
    }
    return 0;
}

// The kernels' dynamic shared-memory limits on this network's device (set
// before any graph capture: the training epoch is captured).
int set_attrs(mbs_mlp *net)
{
    const auto a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    MK(cudaFuncSetAttribute(k_chain<false, kFwdRows>, a, ChainSmem<false, kFwdRows>::bytes), "kernel attributes");
    MK(cudaFuncSetAttribute(k_chain<true, kTrainRows>, a, ChainSmem<true, kTrainRows>::bytes), "kernel attributes");
    MK(cudaFuncSetAttribute(k_update<false>, a, kUpSmem), "kernel attributes");
    MK(cudaFuncSetAttribute(k_update<true>, a, kUpSmem), "kernel attributes");
    return 0;
}

ChainArgs chain_args(mbs_mlp *net, int n)
{
    ChainArgs a{};
    a.q = net->q;
    a.t = net->t;
    a.n = n;
    a.params = net->params;
    a.w = net->w;
    a.img = net->img;
    a.y = net->y;
    a.dy = net->dy;
    a.watch = watch(net);
    return a;
}

// Forward pass of n samples already in net->q (device).
int forward_dev(mbs_mlp *net, int n)
{
    const ChainArgs a = chain_args(net, n);
    k_chain<false, kFwdRows><<<(n + kFwdRows - 1) / kFwdRows, kChainThreads, ChainSmem<false, kFwdRows>::bytes,
                               net->stream>>>(a);
    MK(cudaGetLastError(), "mlp forward launch");
    return 0;
}

// A launch whose prologue may overlap the kernel before it (grid_wait).
template <typename Args>
cudaError_t launch_dependent(cudaStream_t s, void (*kern)(Args), int grid, int threads, int smem, Args args)
{
    cudaLaunchAttribute at;
    std::memset(&at, 0, sizeof(at));
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, args);
}

// Forward and backward chain of a.n samples, then the gradients (adam false:
// into net->grad) or the updated parameters (u holds the step's constants).
int step_dev(mbs_mlp *net, const ChainArgs &a, UpdateArgs u, bool use_adam)
{
    const int bp = pad_rows(a.n);
    MK(launch_dependent(net->stream, k_chain<true, kTrainRows>, bp / kTrainRows, kChainThreads,
                        ChainSmem<true, kTrainRows>::bytes, a),
       "mlp chain launch");
    u.img = net->img;
    u.dy = net->dy;
    u.bp = bp;
    u.grad = net->grad;
    u.p = net->params;
    u.m = net->m;
    u.v = net->v;
    u.w = net->w;
    u.watch = watch(net);
    MK(launch_dependent(net->stream, use_adam ? k_update<true> : k_update<false>, kUpJobs, kUpThreads, kUpSmem, u),
       "mlp update launch");
    return 0;
}

int refresh(mbs_mlp *net)
{
    k_refresh<<<(kH * kH + 255) / 256, 256, 0, net->stream>>>(net->params, net->w);
    MK(cudaGetLastError(), "mlp refresh launch");
    return 0;
}

}  // namespace

extern "C" int mbs_mlp_create(mbs_mlp **out, int device, uint64_t seed)
{
    if (!out)
        return -1;
    *out = nullptr;
    mbs_mlp *net = new mbs_mlp();
    net->device = device;
    auto bail = [&](int rc) { mbs_mlp_destroy(net); return rc; };
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&net->stream, cudaStreamNonBlocking) != cudaSuccess
        || cudaStreamCreateWithFlags(&net->upload, cudaStreamNonBlocking) != cudaSuccess)
        return bail(-3);
    const size_t np = kNParams;
    if (cudaMalloc((void **)&net->params, np * 4) || cudaMalloc((void **)&net->grad, np * 4)
        || cudaMalloc((void **)&net->m, np * 4) || cudaMalloc((void **)&net->v, np * 4)
        || cudaMalloc((void **)&net->wimg, (kH * kInPad + 4 * kImg) * sizeof(bf16))
        || cudaMalloc((void **)&net->scalar, 16) || cudaMemset(net->scalar, 0, 16))
        return bail(-4);
    net->w = Weights{net->wimg, net->wimg + kH * kInPad, net->wimg + kH * kInPad + kImg,
                     net->wimg + kH * kInPad + 2 * kImg, net->wimg + kH * kInPad + 3 * kImg};
    if (set_attrs(net))
        return bail(-3);
    // uniform +-sqrt(6 / fan_in) weights, zero biases
    std::vector<float> p(np, 0.f);
    std::mt19937_64 rng(seed);
    auto fill = [&](int off, int count, int fan_in) {
        std::uniform_real_distribution<float> u(-std::sqrt(6.f / fan_in), std::sqrt(6.f / fan_in));
        for (int i = 0; i < count; ++i)
            p[off + i] = u(rng);
    };
    fill(oW1, kH * kIn, kIn);
    fill(oW2, kH * kH, kH);
    fill(oW3, kH * kH, kH);
    fill(ow4, kH, kH);
    const int rc = mbs_mlp_set_params(net, p.data());
    if (rc)
        return bail(rc);
    *out = net;
    return 0;
}

extern "C" int mbs_mlp_destroy(mbs_mlp *net)
{
    if (!net)
        return -1;
    cudaSetDevice(net->device);
    free_acts(net);
    void *ps[] = {net->params, net->grad, net->m, net->v, net->wimg, net->acts, net->scalar, net->block};
    for (void *p : ps)
        cudaFree(p);
    if (net->stream)
        cudaStreamDestroy(net->stream);
    if (net->upload)
        cudaStreamDestroy(net->upload);
    delete net;
    return 0;
}

extern "C" int mbs_mlp_set_watchdog(mbs_mlp *net, int poll_limit, int skip_mma)
{
    if (!net)
        return -1;
    net->poll_limit = poll_limit > 0 ? poll_limit : kDefaultPollLimit;
    net->skip_mma = skip_mma ? 1 : 0;
    return 0;
}

extern "C" const char *mbs_mlp_last_error(const mbs_mlp *net)
{
    return net ? net->err.c_str() : "null network";
}

extern "C" int mbs_mlp_get_params(mbs_mlp *net, float *params)
{
    if (!net || !params)
        return mfail(net, -1, "null argument");
    MK(cudaSetDevice(net->device), "cudaSetDevice");
    MK(cudaMemcpyAsync(params, net->params, kNParams * 4, cudaMemcpyDeviceToHost, net->stream), "D2H params");
    MK(cudaStreamSynchronize(net->stream), "sync");
    return 0;
}

extern "C" int mbs_mlp_set_params(mbs_mlp *net, const float *params)
{
    if (!net || !params)
        return mfail(net, -1, "null argument");
    MK(cudaSetDevice(net->device), "cudaSetDevice");
    MK(cudaMemcpyAsync(net->params, params, kNParams * 4, cudaMemcpyHostToDevice, net->stream), "H2D params");
    MK(cudaMemsetAsync(net->m, 0, kNParams * 4, net->stream), "memset");
    MK(cudaMemsetAsync(net->v, 0, kNParams * 4, net->stream), "memset");
    net->step = 0;
    int rc = refresh(net);
    if (rc)
        return rc;
    MK(cudaStreamSynchronize(net->stream), "sync");
    return 0;
}

extern "C" int mbs_mlp_forward(mbs_mlp *net, const float *q, int n, float *y)
{
    if (!net || n < 0 || (n > 0 && (!q || !y)))
        return mfail(net, -1, "bad arguments");
    if (n == 0)
        return 0;
    MK(cudaSetDevice(net->device), "cudaSetDevice");
    int rc = ensure_acts(net, n);
    if (rc)
        return rc;
    MK(cudaMemcpyAsync(net->q, q, (size_t)n * kIn * 4, cudaMemcpyHostToDevice, net->stream), "H2D q");
    if ((rc = forward_dev(net, n)))
        return rc;
    MK(cudaMemcpyAsync(y, net->y, (size_t)n * 4, cudaMemcpyDeviceToHost, net->stream), "D2H y");
    MK(cudaStreamSynchronize(net->stream), "sync");
    return check_err(net);
}

extern "C" int mbs_mlp_loss_grad(mbs_mlp *net, const float *q, const float *t, int n, float *loss,
                                 float *grad)
{
    if (!net || n <= 0 || !q || !t)
        return mfail(net, -1, "bad arguments");
    MK(cudaSetDevice(net->device), "cudaSetDevice");
    int rc = ensure_acts(net, n);
    if (rc || (rc = ensure_images(net, n)))
        return rc;
    MK(cudaMemcpyAsync(net->q, q, (size_t)n * kIn * 4, cudaMemcpyHostToDevice, net->stream), "H2D q");
    MK(cudaMemcpyAsync(net->t, t, (size_t)n * 4, cudaMemcpyHostToDevice, net->stream), "H2D t");
    if ((rc = step_dev(net, chain_args(net, n), UpdateArgs{}, false)))
        return rc;
    k_loss<<<1, 256, 0, net->stream>>>(net->y, net->t, n, net->scalar);
    MK(cudaGetLastError(), "loss launch");
    float l = 0.f;
    MK(cudaMemcpyAsync(&l, net->scalar, 4, cudaMemcpyDeviceToHost, net->stream), "D2H loss");
    if (grad)
        MK(cudaMemcpyAsync(grad, net->grad, kNParams * 4, cudaMemcpyDeviceToHost, net->stream), "D2H grad");
    MK(cudaStreamSynchronize(net->stream), "sync");
    if (loss)
        *loss = l;
    return check_err(net);
}

extern "C" int mbs_mlp_train(mbs_mlp *net, const float *q, const float *t, int n, int epochs,
                             int batch, float lr, uint64_t seed, float *final_loss)
{
    if (!net || n <= 0 || !q || !t || epochs < 0 || batch <= 0 || !(lr > 0.f))
        return mfail(net, -1, "bad arguments");
    MK(cudaSetDevice(net->device), "cudaSetDevice");
    batch = std::min(batch, n);
    int rc = ensure_acts(net, n);
    if (rc || (rc = ensure_images(net, batch)))
        return rc;
    cudaStream_t s = net->stream;
    // one epoch's steps: minibatches of `batch`, the last one shorter
    std::vector<int> sizes;
    for (int b0 = 0; b0 < n; b0 += batch)
        sizes.push_back(std::min(batch, n - b0));
    const size_t steps = (size_t)epochs * sizes.size();
    // one block (kept by the network up to kBlockKeep): samples, targets, the
    // same in the epoch's order, the orders, the bias corrections, the epoch
    // counter
    auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t bq = up((size_t)n * kIn * 4), bt = up((size_t)n * 4), bi = up((size_t)epochs * n * 4);
    const size_t bb = up(steps * 2 * 4);
    const size_t need = 2 * bq + 2 * bt + bi + bb + 256;
    cudaEvent_t ready = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    auto cleanup = [&]() {
        if (exec)
            cudaGraphExecDestroy(exec);
        if (graph)
            cudaGraphDestroy(graph);
        if (ready)
            cudaEventDestroy(ready);
        cudaStreamSynchronize(net->upload);   // it reads this call's host arrays
        cudaStreamSynchronize(s);
        if (net->block_cap > kBlockKeep) {
            cudaFree(net->block);
            net->block = nullptr;
            net->block_cap = 0;
        }
    };
    if (net->block_cap < need) {
        cudaFree(net->block);
        net->block = nullptr;
        net->block_cap = 0;
        if (cudaMalloc((void **)&net->block, need) == cudaSuccess)
            net->block_cap = need;
    }
    unsigned char *block = net->block;
    if (net->block_cap < need
        || cudaEventCreateWithFlags(&ready, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        cleanup();
        return mfail(net, -4, "cudaMalloc training set");
    }
    float *dq = (float *)block, *sq = (float *)(block + bq), *dt = (float *)(block + 2 * bq);
    float *st = (float *)(block + 2 * bq + bt), *dbc = (float *)(block + 2 * bq + 2 * bt + bi);
    int *didx = (int *)(block + 2 * bq + 2 * bt), *dstate = (int *)(block + 2 * bq + 2 * bt + bi + bb);
    // every step's Adam bias corrections
    std::vector<float> bc(steps * 2 + 2);
    for (size_t k = 0; k < steps; ++k) {
        const float step = (float)(net->step + 1 + (long long)k);
        bc[2 * k] = 1.f - std::pow(0.9f, step);
        bc[2 * k + 1] = 1.f - std::pow(0.999f, step);
    }
    const int before = -1;
    cudaError_t e = cudaMemcpyAsync(dq, q, (size_t)n * kIn * 4, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(dt, t, (size_t)n * 4, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && epochs > 0)
        e = cudaMemcpyAsync(dbc, bc.data(), steps * 2 * 4, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(dstate, &before, 4, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s);   // the host arrays are read before they go
    if (e != cudaSuccess) {
        cleanup();
        return mfail(net, -3, std::string("training upload: ") + cudaGetErrorString(e));
    }
    std::vector<int> order((size_t)epochs * n);   // outlives the uploads (cleanup waits)
    // One epoch (its shuffle, then two kernels per minibatch) captured once as a
    // graph and replayed per epoch.
    if (epochs > 0) {
        e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            const int spe = (int)sizes.size();
            k_epoch<<<1, 1024, 0, s>>>((const float4 *)dq, dt, didx, n, dstate, (float4 *)sq, st);
            ChainArgs ca = chain_args(net, batch);
            UpdateArgs ua{};
            ua.lr = lr;
            ua.bc = dbc;
            ua.epoch = dstate;
            ua.steps_per_epoch = spe;
            for (int k = 0, b0 = 0; k < spe && rc == 0; b0 += sizes[k], ++k) {
                ca.q = sq + (size_t)b0 * kIn;
                ca.t = st + b0;
                ca.n = sizes[k];
                ua.k = k;
                rc = step_dev(net, ca, ua, true);
            }
            const cudaError_t ec = cudaStreamEndCapture(s, &graph);
            if (e == cudaSuccess)
                e = ec;
        }
        if (e == cudaSuccess && rc == 0)
            e = cudaGraphInstantiate(&exec, graph, 0);
        // the epochs' shuffled orders, some epochs at a time on the upload
        // stream while the device trains on the ones before
        std::mt19937_64 rng(seed);
        std::vector<int> perm(n);
        const int some = std::max(1, 16384 / n);
        for (int e0 = 0; e0 < epochs && e == cudaSuccess && rc == 0; e0 += some) {
            const int e1 = std::min(epochs, e0 + some);
            for (int ep = e0; ep < e1; ++ep) {
                for (int i = 0; i < n; ++i)
                    perm[i] = i;
                std::shuffle(perm.begin(), perm.end(), rng);
                std::copy(perm.begin(), perm.end(), order.begin() + (size_t)ep * n);
            }
            e = cudaMemcpyAsync(didx + (size_t)e0 * n, order.data() + (size_t)e0 * n, (size_t)(e1 - e0) * n * 4,
                                cudaMemcpyHostToDevice, net->upload);
            if (e == cudaSuccess)
                e = cudaEventRecord(ready, net->upload);
            if (e == cudaSuccess)
                e = cudaStreamWaitEvent(s, ready, 0);
            for (int ep = e0; ep < e1 && e == cudaSuccess; ++ep)
                e = cudaGraphLaunch(exec, s);
        }
        if (e != cudaSuccess || rc) {
            cudaGetLastError();
            cleanup();
            if (rc)
                return rc;
            return mfail(net, -3, std::string("training graph: ") + cudaGetErrorString(e));
        }
    }
    if (rc == 0 && final_loss) {
        // loss over the whole set with the trained parameters
        e = cudaMemcpyAsync(net->q, dq, (size_t)n * kIn * 4, cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(net->t, dt, (size_t)n * 4, cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess && (rc = forward_dev(net, n)) == 0) {
            k_loss<<<1, 256, 0, s>>>(net->y, net->t, n, net->scalar);
            e = cudaMemcpyAsync(final_loss, net->scalar, 4, cudaMemcpyDeviceToHost, s);
        }
    }
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s);
    cleanup();
    if (rc)
        return rc;
    if (e != cudaSuccess)
        return mfail(net, -3, std::string("training: ") + cudaGetErrorString(e));
    if ((rc = check_err(net)) == 0)
        net->step += (int)steps;
    return rc;
}
