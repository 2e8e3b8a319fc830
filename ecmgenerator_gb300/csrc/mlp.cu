/*
 * mlp.cu -- the learned active-set proposal: a small MLP that, from an agent's
 * sorted neighbours and its preferred velocity, proposes which constraints
 * are active at the optimum of its ORCA linear program (ORCA.cpp:428-587).
 * The proposal is only a hint: the tick verifies it exactly and runs the full
 * incremental LP whenever the check fails (kernels.cu), so it never changes
 * the tick's results.
 *
 *   input  96 = 16 neighbours x (relative position / neighbour distance,
 *               relative velocity / 2, radius sum) + preferred velocity /
 *               LP radius, zero-padded from 82
 *   hidden 128 -> GELU -> 128 -> GELU
 *   output 160 classes (see ecmg_internal.h, kCls*)
 *
 * Inference: BF16 weights and activations on the 5th-generation tensor
 * cores (tcgen05.mma, FP32 accumulators in tensor memory), weights staged
 * once per CTA in shared memory in the MMA operand layout.  Training: FP32
 * master weights; forward and backward pass of a row tile in one kernel, every
 * contraction on the tensor cores with BF16 operands and FP32 accumulation
 * (k_train), the elementwise steps, softmax cross-entropy and Adam in FP32.
 * This translation unit is not part of the parity-critical arithmetic.
 */
#include "../../include/ecmg.h"
#include "ecmg_internal.h"

#include <cuda.h> /* CUtensorMap (the encoder is reached through the runtime) */
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

using namespace ecmg;

namespace {

constexpr int IN = kMlpIn, HID = kMlpHid, OUT = kMlpOut;
/* GELU (tanh form) and its derivative from one tanh.  Scalar operations: as
   pairs of products and sums the derivative came out an ulp apart here and
   there, which moves its BF16 product over a rounding line once in 70,000. */
__device__ __forceinline__ void gelu_both(float x, float* y, float* dy)
{
    const float k0 = 0.7978845608028654f, k1 = 0.044715f; /* sqrt(2/pi), tanh approximation */
    const float th = tanhf(k0 * (x + k1 * x * x * x));
    const float du = k0 * (1.0f + 3.0f * k1 * x * x);
    *y = 0.5f * x * (1.0f + th);
    *dy = 0.5f * (1.0f + th) + 0.5f * x * (1.0f - th * th) * du;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi); /* .x = lo (low half), .y = hi */
    return *reinterpret_cast<uint32_t*>(&v);
}

/* ------------------------------------------------------------------------
 * Inference on the 5th-generation tensor cores (tcgen05).  One CTA of
 * sixteen warps per SM, persistent over tiles of 128 agents, as four
 * independent pipelines: warps 4g .. 4g+3 run the tiles of pipeline g, each
 * with its own operand tile in shared memory, its own 128 tensor-memory
 * columns and its own named barrier, so that the epilogues of some
 * pipelines run while another's MMA chain occupies the tensor core (the
 * epilogues, not the tensor core, bound the kernel).  Per tile four chains
 * (M = 128; N = 128 / 128 / 128 + 32, layer 3 in two chains over the same
 * columns; K = 96 / 128 / 128 in steps of 16), each issued by the
 * pipeline's first thread and completed through its mbarrier (FP32
 * accumulators, 128 lanes x N columns).  Epilogue: warp w reads lanes
 * 32 (w mod 4) .. +31 (its rows) with tcgen05.ld, the load of the next 16
 * columns in flight while the current ones are used -- bias + GELU
 * (tanh.approx) + BF16 into the operand tile, or bias + argmax over the 160
 * outputs (first maximum wins).  The operand tile holds the features (one
 * TMA copy), then each hidden layer over the operand the previous chain has
 * finished reading; the next tile's copy is requested when the last chain
 * of a tile has completed.  Operands sit in shared memory in the canonical
 * K-major layout without swizzle: 8-row x 16-byte core matrices; the row
 * groups of one 8-column chunk are adjacent (stride byte offset 128), chunks
 * R x 16 bytes apart (leading byte offset) for an operand of R rows.  One
 * chunk of a 128-row feature tile is one 2 KB TMA box (8 columns x 128
 * rows).  Every wait is bounded (spin limit); on a timeout the pipeline sets
 * the error bit, waits for its copy and MMA chain in flight, and the CTA
 * frees its tensor memory and returns.
 * ---------------------------------------------------------------------- */
constexpr int kTile = 128;      /* agents per tile (MMA M) */
constexpr int kGroups = 4;      /* independent pipelines per CTA */
constexpr int kSlotCols = 128;  /* tensor-memory columns per pipeline (layer 3 runs as N = 128 + 32) */
constexpr int kTmemCols = kGroups * kSlotCols;
constexpr int kInferThreads = 128 * kGroups;
constexpr int kOutA = 128;      /* layer-3 outputs of the first chain */
constexpr int kSpinDefault = 1 << 22;

/* byte offset of element (r, k) of an [R x K] bf16 operand in that layout */
__host__ __device__ constexpr int tc_off(int r, int k, int R)
{
    return ((k >> 3) * (R >> 3) + (r >> 3)) * 128 + (r & 7) * 16 + (k & 7) * 2;
}

constexpr int kW1B = HID * IN * 2, kW2B = HID * HID * 2, kW3B = OUT * HID * 2; /* B operands: N rows x K */
constexpr int kWB = kW1B + kW2B + kW3B;
constexpr int kXB = kTile * IN * 2, kHB = kTile * HID * 2;
/* weights, one operand tile per pipeline (the feature tile, then each hidden
   tile over it), biases, tensor-memory address and barriers */
constexpr size_t kInferSmem = (size_t)kWB + kGroups * kHB + sizeof(float) * (2 * HID + OUT) + 128;
static_assert(kXB <= kHB, "a feature tile fits the pipeline's operand tile");
static_assert(kInferSmem <= 232448, "shared memory of one CTA");

/* shared-memory matrix descriptor (no swizzle) */
__device__ __forceinline__ uint64_t tc_sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46; /* descriptor version */
    return d;                /* base offset 0, relative LBO, layout type 0: no swizzle */
}

/* instruction descriptor, kind::f16: BF16 A and B (K-major), FP32 D */
__host__ __device__ constexpr uint32_t tc_idesc(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

/* D[tmem] (+)= A[M x K] * B[K x N], K-steps of 16 (two chunks), one thread;
   B is N rows of an operand packed with R rows (R = N, or a row block of a
   taller operand: chunks R x 16 bytes apart) */
__device__ __forceinline__ void tc_layer(uint32_t tmem, uint32_t a_saddr, uint32_t b_saddr, int K, int N, int R)
{
    const uint32_t id = tc_idesc(kTile, N);
    for (int ks = 0; ks < K / 16; ks++) {
        const uint64_t ad = tc_sdesc(a_saddr + ks * 2 * (kTile * 16), kTile * 16, 128);
        const uint64_t bd = tc_sdesc(b_saddr + ks * 2 * (R * 16), R * 16, 128);
        const uint32_t acc = ks > 0 ? 1u : 0u;
        asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(id), "r"(acc));
    }
}

__device__ __forceinline__ void tc_commit(uint32_t mbar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
                 : "memory");
}

/* bounded wait for the mbarrier phase with the given parity: false after
   `limit` polls.  Limits of at least 1024 poll with try_wait (which may
   suspend the thread for a while); smaller ones -- the diagnostic setting
   of ecmg_mlp_set_wait_limit -- with the non-blocking test_wait, so that a
   limit of one poll really gives up at once */
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, int limit = kSpinDefault)
{
    const bool blocking = limit >= 1024;
    for (int it = 0; it < limit; it++) {
        uint32_t ok;
        if (blocking)
            asm volatile(
                "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                : "=r"(ok)
                : "r"(mbar), "r"(parity)
                : "memory");
        else
            asm volatile(
                "{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                : "=r"(ok)
                : "r"(mbar), "r"(parity)
                : "memory");
        if (ok) return true;
    }
    return false;
}

/* 16 fp32 columns of this thread's lane, issued without waiting; the
   registers are valid after tmem_wait16 on them (the wait takes them as
   operands, so that no use is scheduled before it) */
__device__ __forceinline__ void tmem_issue16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait16(uint32_t (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15])
                 :
                 : "memory");
}
/* f(registers, column) over `cols` columns (a multiple of 32) in chunks of
   16, the load of each chunk in flight while the previous one is used */
template <class F>
__device__ __forceinline__ void tmem_chunks(uint32_t taddr, int cols, F&& f)
{
    uint32_t ra[16], rb[16];
    tmem_issue16(taddr, ra);
    tmem_wait16(ra);
#pragma unroll 1
    for (int c = 0; c < cols; c += 32) {
        tmem_issue16(taddr + (uint32_t)(c + 16), rb);
        f(ra, c);
        tmem_wait16(rb);
        const bool more = c + 32 < cols;
        if (more) tmem_issue16(taddr + (uint32_t)(c + 32), ra);
        f(rb, c + 16);
        if (more) tmem_wait16(ra);
    }
}

/* W [K x N] row-major FP32 -> BF16 B operand (N rows x K) in the tc layout */
__global__ void k_pack_tc(const float* W, int K, int N, unsigned char* out)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < K * N; i += gridDim.x * blockDim.x) {
        int n = i / K, k = i % K;
        *reinterpret_cast<__nv_bfloat16*>(out + tc_off(n, k, N)) = __float2bfloat16_rn(W[(size_t)k * N + n]);
    }
}

/* the 12 TMA boxes (8 columns x 128 rows) of the feature tile at row r0 */
__device__ __forceinline__ void tma_tile(const CUtensorMap* tm, uint32_t sdst, int r0, uint32_t mbar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"((uint32_t)kXB)
                 : "memory");
#pragma unroll 1
    for (int kc = 0; kc < IN / 8; kc++)
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
                "r"(sdst + (uint32_t)(kc * kTile * 16)),
            "l"(tm), "r"(kc * 8), "r"(r0), "r"(mbar)
            : "memory");
}

__device__ __forceinline__ float tanh_approx(float x)
{
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* GELU (tanh form) for inference of two values plus their biases: the
   hardware tanh approximation (relative error about 2^-11, below the BF16
   rounding of the activations); everything else two values per instruction,
   the epilogues being bound by their instruction count */
__device__ __forceinline__ uint32_t gelu_fast2(uint32_t z0, uint32_t z1, float b0, float b1)
{
    const float k0 = 0.7978845608028654f, k1 = 0.044715f;
    const float2 x = __fadd2_rn(make_float2(__uint_as_float(z0), __uint_as_float(z1)), make_float2(b0, b1));
    const float2 c = __fmul2_rn(make_float2(k1, k1), __fmul2_rn(x, x));
    const float2 u = __fmul2_rn(make_float2(k0, k0), __ffma2_rn(c, x, x));
    const float2 hx = __fmul2_rn(make_float2(0.5f, 0.5f), x);
    const float2 y = __ffma2_rn(hx, make_float2(tanh_approx(u.x), tanh_approx(u.y)), hx);
    return pack_bf16(y.x, y.y);
}

/* 32 consecutive fp32 columns of this thread's lane, one wait */
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v)
{
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                   "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                   "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory"); /* the registers are tied to the wait: no use before it */
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

/* barrier of one 4-warp group (ids 1 to 4; 0 is the CTA barrier) */
__device__ __forceinline__ void group_sync(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }
/* barrier of one group that also ORs a flag over its threads */
__device__ __forceinline__ bool group_any(bool v, int id)
{
    unsigned r;
    asm volatile(
        "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.or.pred q, %2, 128, p;\nselp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(r)
        : "r"((unsigned)v), "r"(id)
        : "memory");
    return r != 0;
}

/* class of every row of X [n, IN] (bf16, row-major); err |= errbit when a
   wait runs past `spin` polls (the CTA then drains and stops) */
__global__ void __launch_bounds__(kInferThreads, 1)
    k_mlp_infer(const __grid_constant__ CUtensorMap tmX, const int* n_ptr, int n_fixed, const unsigned char* wpack,
                const float* bias, unsigned char* cls, int* err, int errbit, int spin)
{
    extern __shared__ __align__(128) unsigned char sm[];
    unsigned char* sW1 = sm;
    unsigned char* sW2 = sW1 + kW1B;
    unsigned char* sW3 = sW2 + kW2B;
    unsigned char* sT = sW3 + kW3B; /* [kGroups][kHB] operand tiles */
    float* sb = reinterpret_cast<float*>(sT + kGroups * kHB);
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(sb + 2 * HID + OUT);
    uint64_t* s_mbar = reinterpret_cast<uint64_t*>(
        (reinterpret_cast<uintptr_t>(s_tmem + 2) + 7) & ~(uintptr_t)7); /* [g] MMA done, [kGroups + g] tile landed */
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = warp >> 2, quad = warp & 3, gt = tid & 127; /* pipeline, TMEM lane quarter, thread in group */
    const int bar_id = 1 + g;
    const int n = n_ptr ? *n_ptr : n_fixed;

    for (int i = tid; i < kWB / 16; i += blockDim.x)
        reinterpret_cast<uint4*>(sm)[i] = reinterpret_cast<const uint4*>(wpack)[i];
    for (int i = tid; i < 2 * HID + OUT; i += blockDim.x) sb[i] = bias[i];
    const uint32_t mbar0 = (uint32_t)__cvta_generic_to_shared(s_mbar);
    if (tid == 0) {
        for (int b = 0; b < 2 * kGroups; b++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar0 + 8u * b) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(s_tmem)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    /* from here on the groups run independent pipelines */
    const uint32_t tmem = *s_tmem + (uint32_t)(g * kSlotCols);
    const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
    const uint32_t aT = (uint32_t)__cvta_generic_to_shared(sT + g * kHB);
    unsigned char* tbuf = sT + g * kHB;
    const uint32_t aW1 = (uint32_t)__cvta_generic_to_shared(sW1), aW2 = (uint32_t)__cvta_generic_to_shared(sW2),
                   aW3 = (uint32_t)__cvta_generic_to_shared(sW3);
    const uint32_t mb_mma = mbar0 + 8u * (uint32_t)g, mb_x = mbar0 + 8u * (uint32_t)(kGroups + g);
    const int row = quad * 32 + lane;
    const int ntiles = (n + kTile - 1) / kTile;
    int tile = (int)blockIdx.x + g * (int)gridDim.x; /* group g: tiles blockIdx.x + (kGroups j + g) gridDim.x */
    uint32_t ph_mma = 0u, ph_x = 0u;
    bool mma_pending = false, x_pending = false, fail = false;

    auto wait = [&](uint32_t mb, uint32_t& ph, bool& pending) {
        const bool ok = mbar_wait(mb, ph, spin);
        fail = group_any(!ok, bar_id);
        if (!fail) {
            ph ^= 1u;
            pending = false;
        }
        tc_fence_after();
        return !fail;
    };
    /* the operands the group's threads wrote are visible to the tensor core
       and the accumulator has been read out; then the leader issues one
       chain */
    auto mma = [&](uint32_t w, int K, int N, int R) {
        fence_async_smem();
        tc_fence_before();
        group_sync(bar_id);
        tc_fence_after();
        if (gt == 0) {
            tc_layer(tmem, aT, w, K, N, R);
            tc_commit(mb_mma);
        }
        mma_pending = true;
    };
    /* bias + GELU + BF16 of the accumulator into the group's operand tile
       (the chain that read it has completed) */
    auto epi_hidden = [&](const float* bl) {
        tmem_chunks(lane_base, HID, [&](uint32_t (&r)[16], int c) {
            const float4* b4 = reinterpret_cast<const float4*>(bl + c); /* 16-byte aligned */
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const float4 ba = b4[2 * q], bb = b4[2 * q + 1];
                const uint32_t* v = r + 8 * q;
                uint4 u;
                u.x = gelu_fast2(v[0], v[1], ba.x, ba.y);
                u.y = gelu_fast2(v[2], v[3], ba.z, ba.w);
                u.z = gelu_fast2(v[4], v[5], bb.x, bb.y);
                u.w = gelu_fast2(v[6], v[7], bb.z, bb.w);
                *reinterpret_cast<uint4*>(tbuf + tc_off(row, c + 8 * q, kTile)) = u;
            }
        });
    };
    /* bias + running argmax over outputs [o0, o0 + cols); the first maximum wins */
    auto epi_argmax = [&](int o0, int cols, float& best, int& bi) {
        const float* bl = sb + 2 * HID + o0;
        tmem_chunks(lane_base, cols, [&](uint32_t (&r)[16], int c) {
            const float4* b4 = reinterpret_cast<const float4*>(bl + c); /* 16-byte aligned */
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
                const float4 b = b4[i / 4];
                const float2 za = __fadd2_rn(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])),
                                             make_float2(b.x, b.y));
                const float2 zb = __fadd2_rn(make_float2(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])),
                                             make_float2(b.z, b.w));
                if (za.x > best) { best = za.x; bi = o0 + c + i; }
                if (za.y > best) { best = za.y; bi = o0 + c + i + 1; }
                if (zb.x > best) { best = zb.x; bi = o0 + c + i + 2; }
                if (zb.y > best) { best = zb.y; bi = o0 + c + i + 3; }
            }
        });
    };

    if (tile < ntiles) {
        if (gt == 0) tma_tile(&tmX, aT, tile * kTile, mb_x);
        x_pending = true;
    }
    while (!fail && tile < ntiles) {
        if (!wait(mb_x, ph_x, x_pending)) break;
        mma(aW1, IN, HID, HID);
        if (!wait(mb_mma, ph_mma, mma_pending)) break;
        epi_hidden(sb);
        mma(aW2, HID, HID, HID);
        if (!wait(mb_mma, ph_mma, mma_pending)) break;
        epi_hidden(sb + HID);
        /* layer 3: outputs 0..127, read out, then 128..159 in the same columns */
        mma(aW3, HID, kOutA, OUT);
        if (!wait(mb_mma, ph_mma, mma_pending)) break;
        float best = -INFINITY;
        int bi = 0;
        epi_argmax(0, kOutA, best, bi);
        mma(aW3 + (uint32_t)(kOutA / 8) * 128u, HID, OUT - kOutA, OUT);
        if (!wait(mb_mma, ph_mma, mma_pending)) break;
        epi_argmax(kOutA, OUT - kOutA, best, bi);
        const int r = tile * kTile + row;
        if (r < n) cls[r] = (unsigned char)bi;
        /* the operand tile is free (the last chain has completed): the
           group's next features go into it */
        tile += kGroups * (int)gridDim.x;
        if (tile < ntiles) {
            if (gt == 0) tma_tile(&tmX, aT, tile * kTile, mb_x);
            x_pending = true;
        }
    }
    if (fail && gt == 0) atomicOr(err, errbit);
    /* nothing in flight may outlive the CTA: the group's copy and MMA chain
       are waited for (with the default bound) before tensor memory is freed */
    if (x_pending) (void)mbar_wait(mb_x, ph_x);
    if (mma_pending) (void)mbar_wait(mb_mma, ph_mma);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*s_tmem), "r"(kTmemCols) : "memory");
}

/* ------------------------------------------------------------------------
 * Training: one kernel for the forward and backward pass of a minibatch, one
 * that sums the gradients and takes the Adam step.
 *
 * k_train.  One CTA of sixteen warps per SM, persistent over tiles of 128
 * rows; a tile's activations never leave the SM.  The weights (BF16, 96 KB)
 * stay in shared memory as the B operands of the forward chains (K-major) and,
 * read along the other axis (MN-major), of the backward ones; likewise an
 * activation tile is the K-major A operand of the next layer and the MN-major
 * operand of its weight gradient, so that nothing is transposed or stored
 * twice.  Per tile, each chain issued by one thread and awaited by all:
 *   Z1 = X W1, Z2 = A1 W2, Z3 = A2 W3 (outputs 0..127, then 128..159)
 *   dA2 = dZ3 W3^T, then dW3 += A2^T dZ3
 *   dA1 = dZ2 W2^T, then dW2 += A1^T dZ2
 *   dW1^T += dZ1^T X
 * with FP32 accumulators: tensor-memory columns 0..127 for the Z's and dA's,
 * 128..511 for the three weight gradients, which stay there over all tiles of
 * the CTA.  Between the chains a thread owns 32 columns of one row in
 * registers: bias, GELU and its derivative (from one tanh; the derivative is
 * kept in FP32 for the backward pass), softmax cross-entropy, and the FP32
 * bias gradients, summed over a warp's rows by a transposing butterfly and
 * over tiles in registers.  dZ2 overwrites A2 and dZ1 overwrites A1 once
 * dW3 and dW2 have read them (a second mbarrier: the next stage's loads and
 * products run beside these chains).  A CTA writes its sums as one partial
 * gradient.
 *
 * What bounds it: the latency of the elementwise work between the chains
 * (accurate tanh, exp and quotients of 416 activations per row) at the four
 * warps per scheduler that the registers leave: of a tile's 35,000 cycles the
 * two activations take 8,700, the softmax 8,500, waiting for chains and
 * barriers 9,000; the scheduler issues in 44 % of them.  Four steps of 65,536
 * rows take 381 us; 505 with a 64-bit remainder per loaded chunk (5,400
 * cycles a tile), a divide per output (5,300), the weights loaded through
 * registers and a start that waits for the step before; 2,890 as 4 x 24 launches that passed
 * every activation, its transpose and its BF16 copy through memory, with a
 * two-block column sum for each bias gradient.
 * ---------------------------------------------------------------------- */
constexpr int OW1 = 0, OB1 = OW1 + IN * HID, OW2 = OB1 + HID, OB2 = OW2 + HID * HID, OW3 = OB2 + HID,
              OB3 = OW3 + HID * OUT, NPARAM = OB3 + OUT; /* W1 [IN x HID], b1, W2 [HID x HID], b2, W3 [HID x OUT], b3 */
constexpr int NWEIGHT = HID * (IN + HID + OUT);
constexpr int kTrThreads = 512, kTrCols = 512; /* tensor memory: all of it */
constexpr int kTrW3 = 128, kTrW2 = kTrW3 + OUT, kTrW1 = kTrW2 + HID; /* first columns of dW3, dW2, dW1^T */
static_assert(kTrW1 + IN == kTrCols, "the weight gradients fill the tensor memory");
constexpr int kZB = kTile * OUT * 2;
constexpr size_t kTrainSmem =
    (size_t)kWB + kXB + 2 * kHB + kZB + sizeof(float) * (2 * HID + OUT) + sizeof(int) * 2 * kTile + 64;
static_assert(kTrainSmem <= 232448, "shared memory of one CTA");
static_assert((4 * 2 + 4 * 8) * kTile * 4 <= kZB, "the softmax's exchange fits the dZ3 tile before it is written");

/* instruction descriptor with the major axes of A and B (1: MN-major) */
__host__ __device__ constexpr uint32_t tc_idesc_mn(int N, int amn, int bmn)
{
    return tc_idesc(kTile, N) | ((uint32_t)amn << 15) | ((uint32_t)bmn << 16);
}

/* D[tmem] (+)= A B over `steps` K-steps of 16, one thread.  K-major operand of
   R rows: chunks (8 columns) R x 16 bytes apart, a K-step is two chunks.
   MN-major (the same storage read along the other axis): the 8-column groups
   of the M or N axis are R x 16 bytes apart, the 8-row groups of the K axis
   128 bytes, a K-step is two of those. */
__device__ __forceinline__ void tc_chain(uint32_t tmem, uint32_t a, int ra, int amn, uint32_t b, int rb, int bmn,
                                         int n, int steps, bool add)
{
    const uint32_t id = tc_idesc_mn(n, amn, bmn);
    const uint32_t sa = amn ? 256u : 32u * (uint32_t)ra, sb = bmn ? 256u : 32u * (uint32_t)rb;
    const uint64_t da = amn ? tc_sdesc(a, 128, 16u * ra) : tc_sdesc(a, 16u * ra, 128);
    const uint64_t db = bmn ? tc_sdesc(b, 128, 16u * rb) : tc_sdesc(b, 16u * rb, 128);
    for (int ks = 0; ks < steps; ks++) {
        const uint32_t acc = add || ks > 0 ? 1u : 0u;
        asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(da + (uint64_t)(ks * (sa >> 4))), "l"(db + (uint64_t)(ks * (sb >> 4))), "r"(id), "r"(acc));
    }
}

/* eight columns each from taddr, taddr + 32, + 64 and + 96 */
__device__ __forceinline__ void tmem_ld8x4(uint32_t taddr, float (&v)[32])
{
    uint32_t r[32];
#pragma unroll
    for (int g = 0; g < 4; g++)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                     : "=r"(r[8 * g]), "=r"(r[8 * g + 1]), "=r"(r[8 * g + 2]), "=r"(r[8 * g + 3]), "=r"(r[8 * g + 4]),
                       "=r"(r[8 * g + 5]), "=r"(r[8 * g + 6]), "=r"(r[8 * g + 7])
                     : "r"(taddr + 32u * (uint32_t)g));
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                   "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]),
                   "+r"(r[23])
                 :
                 : "memory");
    asm volatile("" : "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]),
                 "+r"(r[31])
                 :
                 : "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8])
{
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
                 :
                 : "memory");
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}

/* sum of v[c] over the warp's lanes, for column c in lane c: at each step a
   lane keeps the half of the columns that its number points to */
__device__ __forceinline__ float warp_colsum(float (&v)[32])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; i++) {
            const float keep = up ? v[i + o] : v[i], give = up ? v[i] : v[i + o];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return v[0];
}

/* the same of 8 columns, for column c in the lanes c, c + 8, c + 16, c + 24 */
__device__ __forceinline__ float warp_colsum8(float (&v)[8])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 4; o; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; i++) {
            const float keep = up ? v[i + o] : v[i], give = up ? v[i] : v[i + o];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 8);
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
}

/* the row of X that row r of the minibatch is: r itself, or (draw) a hash of
   the step's seed (splitmix64) modulo n, by the quotient's estimate with inv =
   floor((2^64 - 1) / n), which is short by two at most */
__device__ __forceinline__ int train_row(int r, int n, unsigned long long inv, unsigned long long seed, int draw)
{
    if (!draw) return r;
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(r + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    unsigned long long m = z - __umul64hi(z, inv) * (unsigned long long)n;
    if (m >= (unsigned long long)n) m -= (unsigned long long)n;
    if (m >= (unsigned long long)n) m -= (unsigned long long)n;
    return (int)m;
}

__global__ void __launch_bounds__(kTrThreads, 1)
    k_train(const __nv_bfloat16* X, const unsigned char* y, int n, int B, unsigned long long inv,
            unsigned long long seed, int draw, const unsigned char* wpack, const float* P, float* part, float* part_loss, int* part_ok, int* err, int spin)
{
    extern __shared__ __align__(128) unsigned char sm[];
    unsigned char *sW1 = sm, *sW2 = sW1 + kW1B, *sW3 = sW2 + kW2B;
    unsigned char *sX = sW3 + kW3B, *sA1 = sX + kXB, *sA2 = sA1 + kHB, *sZ = sA2 + kHB;
    float* sb = reinterpret_cast<float*>(sZ + kZB); /* biases; at the end the bias gradients */
    int* s_row = reinterpret_cast<int*>(sb + 2 * HID + OUT); /* this tile's and the next one's rows of X */
    uint64_t* s_mbar = reinterpret_cast<uint64_t*>(s_row + 2 * kTile);
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(s_mbar + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quad = warp & 3, cg = warp >> 2; /* tensor-memory lane quarter, column group */
    const int row = quad * 32 + lane, c0 = cg * 32;

    /* the rows of a tile, by the last four warps (-1: beyond the batch) */
    const int ntiles = (B + kTile - 1) / kTile;
    auto set_rows = [&](int tile, int buf) {
        const int i = tid - (kTrThreads - kTile), r = tile * kTile + i;
        if (i < 0) return;
        const int x = tile < ntiles && r < B ? train_row(r, n, inv, seed, draw) : -1;
        s_row[buf * kTile + i] = x;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(y + max(x, 0)));
    };
    set_rows((int)blockIdx.x, 0);
    const uint32_t mb = (uint32_t)__cvta_generic_to_shared(s_mbar), mbw = mb + 8;
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbw) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(s_tmem)),
                     "r"(kTrCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;
    const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
    const uint32_t aW1 = (uint32_t)__cvta_generic_to_shared(sW1), aW2 = (uint32_t)__cvta_generic_to_shared(sW2),
                   aW3 = (uint32_t)__cvta_generic_to_shared(sW3), aX = (uint32_t)__cvta_generic_to_shared(sX),
                   aA1 = (uint32_t)__cvta_generic_to_shared(sA1), aA2 = (uint32_t)__cvta_generic_to_shared(sA2),
                   aZ = (uint32_t)__cvta_generic_to_shared(sZ);
    uint32_t ph = 0u, phw = 0u;
    bool pending = false, pending_w = false, fail = false;
    /* the tiles written and the accumulator read so far are visible to the
       tensor core; then one thread issues */
    auto ready = [&] {
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        pending = true;
        return tid == 0;
    };
    /* the weight-gradient chain has read this operand: a tile of the thread's
       own goes over it.  A thread whose wait runs out leaves the tile as it is
       and keeps the chain pending; the barrier before the next chain then
       stops the CTA, so that never more than one chain is outstanding on mbw
       and the drain below waits for that one.  False: stop. */
    auto over_tile = [&](unsigned char* t, const float (&v)[32], auto&& store) {
        const bool ok = mbar_wait(mbw, phw, spin);
        tc_fence_after();
        if (ok) {
            phw ^= 1u;
            pending_w = false;
            store(t, v);
        }
        fence_async_smem();
        tc_fence_before();
        fail = __syncthreads_or(!ok) != 0;
        tc_fence_after();
        return !fail;
    };
    auto wait = [&] {
        const bool ok = mbar_wait(mb, ph, spin);
        fail = __syncthreads_or(!ok) != 0;
        if (!fail) {
            ph ^= 1u;
            pending = false;
        }
        tc_fence_after();
        return !fail;
    };
    /* the 12 16-byte chunks of each of a tile's rows, three per thread.  They
       are loaded where the backward pass leaves registers, and take no branch,
       so that nothing waits for them before store_x (loaded earlier they were
       spilled, which waits); rows beyond the batch load the first row and are
       stored as zeros. */
    const bool wide = (reinterpret_cast<uintptr_t>(X) & 15) == 0;
    uint4 xr[3];
    auto load_x = [&](int buf) {
        if (!wide) return;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const int e = tid + i * kTrThreads, r = max(s_row[buf * kTile + e / 12], 0);
            xr[i] = __ldg(reinterpret_cast<const uint4*>(X + (size_t)r * IN + e % 12 * 8));
        }
    };
    auto store_x = [&](int buf) {
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const int e = tid + i * kTrThreads, r = s_row[buf * kTile + e / 12];
            uint4 x = make_uint4(0u, 0u, 0u, 0u);
            if (wide) {
                if (r >= 0) x = xr[i];
            } else if (r >= 0) {
                const unsigned short* h = reinterpret_cast<const unsigned short*>(X + (size_t)r * IN + e % 12 * 8);
                x = make_uint4(h[0] | (uint32_t)h[1] << 16, h[2] | (uint32_t)h[3] << 16, h[4] | (uint32_t)h[5] << 16,
                               h[6] | (uint32_t)h[7] << 16);
            }
            *reinterpret_cast<uint4*>(sX + tc_off(e / 12, (e % 12) * 8, kTile)) = x;
        }
    };
    auto pack8 = [](const float* v) {
        return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
    };
    auto store32 = [&](unsigned char* t, const float (&v)[32]) {
#pragma unroll
        for (int q = 0; q < 4; q++) *reinterpret_cast<uint4*>(t + tc_off(row, c0 + 8 * q, kTile)) = pack8(v + 8 * q);
    };
    /* z -> gelu(z) as BF16 into the tile, v -> the derivative */
    auto activate = [&](float (&v)[32], const float* bias, unsigned char* t) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            float a[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                float* x = v + 8 * q + i;
                gelu_both(*x + bias[c0 + 8 * q + i], &a[i], x);
            }
            *reinterpret_cast<uint4*>(t + tc_off(row, c0 + 8 * q, kTile)) = pack8(a);
        }
    };

    const float fb = (float)B, rfb = 1.0f / fb;
    float db1 = 0.0f, db2 = 0.0f, db3 = 0.0f, db3b = 0.0f, loss = 0.0f;
    int right = 0;
    bool add = false;
    int tile = (int)blockIdx.x, buf = 0;
    load_x(0);
    /* everything above reads the minibatch only; from here on the weights that
       the kernel before writes, and the partial gradients that it reads */
    asm volatile("griddepcontrol.wait;" ::: "memory");
    static_assert(kWB % (16 * kTrThreads) == 0, "whole 16-byte pieces per thread");
#pragma unroll
    for (int i = 0; i < kWB / (16 * kTrThreads); i++) {
        const int o = (i * kTrThreads + tid) * 16;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(sm + o)),
                     "l"(wpack + o)
                     : "memory");
    }
    for (int i = tid; i < 2 * HID + OUT; i += kTrThreads)
        sb[i] = i < HID ? P[OB1 + i] : (i < 2 * HID ? P[OB2 + i - HID] : P[OB3 + i - 2 * HID]);
    asm volatile("cp.async.wait_all;" ::: "memory");
    for (; tile < ntiles; tile += (int)gridDim.x, buf ^= 1) {
        store_x(buf);
        float g1[32], g2[32];
        if (ready()) {
            tc_chain(tmem, aX, kTile, 0, aW1, HID, 0, HID, IN / 16, false);
            tc_commit(mb);
        }
        const int xrow = s_row[buf * kTile + row];
        const bool valid = xrow >= 0;
        const int yy = (int)y[max(xrow, 0)];
        set_rows(tile + (int)gridDim.x, buf ^ 1);
        if (!wait()) break;
        tmem_ld32(lane_base + c0, g1);
        activate(g1, sb, sA1);
        if (ready()) {
            tc_chain(tmem, aA1, kTile, 0, aW2, HID, 0, HID, HID / 16, false);
            tc_commit(mb);
        }
        if (!wait()) break;
        tmem_ld32(lane_base + c0, g2);
        activate(g2, sb + HID, sA2);
        if (ready()) {
            tc_chain(tmem, aA2, kTile, 0, aW3, OUT, 0, kOutA, HID / 16, false);
            tc_commit(mb);
        }
        if (!wait()) break;
        /* the outputs of a thread: columns 32 g + 8 cg + 0..7, g = 0..4 */
        float z[32], zb[8];
        tmem_ld8x4(lane_base + cg * 8, z);
        if (ready()) { /* outputs 128..159, eight per column group */
            tc_chain(tmem, aA2, kTile, 0, aW3 + (uint32_t)(kOutA / 8) * 128u, OUT, 0, OUT - kOutA, HID / 16, false);
            tc_commit(mb);
        }
        if (!wait()) break;
        tmem_ld8(lane_base + cg * 8, zb);
        /* softmax cross-entropy of the row; its four column groups exchange
           through the dZ3 tile's memory */
        float* sx = reinterpret_cast<float*>(sZ);
        int* sxi = reinterpret_cast<int*>(sx + 4 * kTile);
        float mx = -INFINITY, zt = 0.0f;
        int am = -1;
        const int yl = yy < OUT && ((yy >> 3) & 3) == cg ? (yy >> 5) * 8 + (yy & 7) : -1;
        const float* b3 = sb + 2 * HID + 8 * cg;
#pragma unroll
        for (int i = 0; i < 32; i++) {
            z[i] += b3[(i >> 3) * 32 + (i & 7)];
            if (z[i] > mx) { mx = z[i]; am = i; }
            if (i == yl) zt = z[i];
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            zb[i] += b3[kOutA + i];
            if (zb[i] > mx) { mx = zb[i]; am = 32 + i; }
            if (32 + i == yl) zt = zb[i];
        }
        am = am < 0 ? 0 : (am >> 3) * 32 + 8 * cg + (am & 7);
        sx[cg * kTile + row] = mx;
        sxi[cg * kTile + row] = am;
        group_sync(1 + quad);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float m = sx[q * kTile + row];
            const int a = sxi[q * kTile + row];
            if (m > mx || (m == mx && a < am)) { mx = m; am = a; }
        }
        /* the sum of the exponentials as a warp with one output in 32 per lane
           takes it: five outputs in order, then halves of the lanes added */
        float4* ss = reinterpret_cast<float4*>(sxi + 4 * kTile);
        float p8[8];
#pragma unroll
        for (int i = 0; i < 32; i++) z[i] = expf(z[i] - mx);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            zb[i] = expf(zb[i] - mx);
            p8[i] = (((z[i] + z[i + 8]) + z[i + 16]) + z[i + 24]) + zb[i];
        }
        ss[2 * cg * kTile + row] = make_float4(p8[0], p8[1], p8[2], p8[3]);
        ss[(2 * cg + 1) * kTile + row] = make_float4(p8[4], p8[5], p8[6], p8[7]);
        group_sync(1 + quad);
        float4 h[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const float4 a0 = ss[q * kTile + row], a1 = ss[(2 + q) * kTile + row], a2 = ss[(4 + q) * kTile + row],
                         a3 = ss[(6 + q) * kTile + row];
            h[q] = make_float4((a0.x + a2.x) + (a1.x + a3.x), (a0.y + a2.y) + (a1.y + a3.y),
                               (a0.z + a2.z) + (a1.z + a3.z), (a0.w + a2.w) + (a1.w + a3.w));
        }
        const float se = ((h[0].x + h[1].x) + (h[0].z + h[1].z)) + ((h[0].y + h[1].y) + (h[0].w + h[1].w));
        /* the column group that holds the label counts the row */
        if (valid && yl >= 0) loss += -(zt - mx - logf(se));
        if (valid && cg == 0 && am == yy) right++;
        /* (e / se - [label]) / B, each quotient from the divisor's reciprocal
           and one residual step (Markstein; 1 <= se <= 160): correctly rounded
           while the residual is a normal number, down to some 1e-30, and off by
           a unit of the smallest number below; a row beyond the batch counts
           nothing */
        const float rse = 1.0f / se, rb = valid ? rfb : 0.0f;
        auto quotient = [](float x, float d, float rd) {
            const float q = x * rd;
            return __fmaf_rn(__fmaf_rn(-q, d, x), rd, q);
        };
        auto dz = [&](float e, int i) { return quotient(quotient(e, se, rse) - (i == yl ? 1.0f : 0.0f), fb, rb); };
#pragma unroll
        for (int i = 0; i < 32; i++) z[i] = dz(z[i], i);
#pragma unroll
        for (int i = 0; i < 8; i++) zb[i] = dz(zb[i], 32 + i);
        group_sync(1 + quad); /* the quarter's exchange has been read */
        __syncthreads();      /* and the other quarters': the tile may be written */
#pragma unroll
        for (int q = 0; q < 4; q++)
            *reinterpret_cast<uint4*>(sZ + tc_off(row, 32 * q + 8 * cg, kTile)) = pack8(z + 8 * q);
        *reinterpret_cast<uint4*>(sZ + tc_off(row, kOutA + cg * 8, kTile)) = pack8(zb);
        if (ready()) {
            tc_chain(tmem, aZ, kTile, 0, aW3, OUT, 1, HID, OUT / 16, false);
            tc_commit(mb);
            tc_chain(tmem + kTrW3, aA2, kTile, 1, aZ, kTile, 1, OUT, kTile / 16, add);
            tc_commit(mbw);
        }
        pending_w = true;
        db3 += warp_colsum(z);
        db3b += warp_colsum8(zb);
        if (!wait()) break;
        float d[32];
        tmem_ld32(lane_base + c0, d);
#pragma unroll
        for (int i = 0; i < 32; i++) d[i] *= g2[i];
        if (!over_tile(sA2, d, store32)) break; /* A2 is read by dW3 */
        pending = true;
        if (tid == 0) {
            tc_chain(tmem, aA2, kTile, 0, aW2, HID, 1, HID, HID / 16, false);
            tc_commit(mb);
            tc_chain(tmem + kTrW2, aA1, kTile, 1, aA2, kTile, 1, HID, kTile / 16, add);
            tc_commit(mbw);
        }
        pending_w = true;
        db2 += warp_colsum(d);
        if (!wait()) break;
        tmem_ld32(lane_base + c0, d);
#pragma unroll
        for (int i = 0; i < 32; i++) d[i] *= g1[i];
        if (!over_tile(sA1, d, store32)) break; /* A1 is read by dW2 */
        pending = true;
        if (tid == 0) {
            tc_chain(tmem + kTrW1, aA1, kTile, 1, aX, kTile, 1, IN, kTile / 16, add);
            tc_commit(mb);
        }
        load_x(buf ^ 1);
        db1 += warp_colsum(d);
        if (!wait()) break;
        add = true;
    }
    if (fail && tid == 0) atomicOr(err, 1);
    if (pending) (void)mbar_wait(mb, ph);
    if (pending_w) (void)mbar_wait(mbw, phw);
    if (!fail) {
        /* the CTA's partial gradient, in the order of part_param: a warp's
           stores are contiguous */
        float* G = part + (size_t)blockIdx.x * NPARAM;
        float v[32];
        for (int b = cg; b < (OUT + HID + IN) / 32; b += 4) {
            tmem_ld32(lane_base + kTrW3 + b * 32, v);
#pragma unroll
            for (int i = 0; i < 32; i += 4)
                *reinterpret_cast<float4*>(G + ((b * 8 + i / 4) * kTile + row) * 4) =
                    make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
        /* bias gradients: the four row quarters in order, through the dZ3 tile */
        float* sg = reinterpret_cast<float*>(sZ) + quad * (2 * HID + OUT);
        sg[c0 + lane] = db1;
        sg[HID + c0 + lane] = db2;
        sg[2 * HID + (lane >> 3) * 32 + 8 * cg + (lane & 7)] = db3;
        if (lane < 8) sg[2 * HID + kOutA + cg * 8 + lane] = db3b;
        float* sl = reinterpret_cast<float*>(sA1);
        int* sr = reinterpret_cast<int*>(sA2);
#pragma unroll
        for (int o = 16; o; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
        right = __reduce_add_sync(0xffffffffu, right);
        if (lane == 0) {
            sl[warp] = loss;
            sr[warp] = right;
        }
        __syncthreads();
        const float* s4 = reinterpret_cast<const float*>(sZ);
        constexpr int NB = 2 * HID + OUT;
        for (int i = tid; i < NB; i += kTrThreads)
            G[NWEIGHT + i] = (s4[i] + s4[NB + i]) + (s4[2 * NB + i] + s4[3 * NB + i]);
        if (tid == 0) {
            float l = 0.0f;
            int k = 0;
            for (int w = 0; w < kTrThreads / 32; w++) {
                l += sl[w];
                k += sr[w];
            }
            part_loss[blockIdx.x] = l;
            part_ok[blockIdx.x] = k;
        }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); /* k_reduce_adam */
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTrCols) : "memory");
}

/* the parameter that entry j of a partial gradient belongs to.  The weights'
   entries are tensor-memory columns dW3 | dW2 | dW1^T in fours, by lanes: a
   lane is the input unit of W3 and W2 and the output unit of W1; then the
   biases b1 | b2 | b3. */
__device__ __forceinline__ int part_param(int j)
{
    if (j >= NWEIGHT) {
        const int i = j - NWEIGHT;
        return i < HID ? OB1 + i : (i < 2 * HID ? OB2 + i - HID : OB3 + i - 2 * HID);
    }
    const int c = j / (4 * kTile) * 4 + (j & 3), l = (j >> 2) & (kTile - 1);
    if (c < OUT) return OW3 + l * OUT + c;
    if (c < OUT + HID) return OW2 + l * HID + c - OUT;
    return OW1 + (c - OUT - HID) * HID + l;
}

/* place of parameter i of the flat array in the packed weights (-1: a bias) */
__device__ __forceinline__ int pack_off(int i)
{
    if (i < OB1) return tc_off(i % HID, i / HID, HID);
    if (i < OW2) return -1;
    if (i < OB2) return kW1B + tc_off((i - OW2) % HID, (i - OW2) / HID, HID);
    if (i < OW3) return -1;
    if (i < OB3) return kW1B + kW2B + tc_off((i - OW3) % OUT, (i - OW3) / OUT, OUT);
    return -1;
}

__global__ void k_pack_all(const float* p, unsigned char* pack)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); /* k_train's start */
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NPARAM) return;
    const int o = pack_off(i);
    if (o >= 0) *reinterpret_cast<__nv_bfloat16*>(pack + o) = __float2bfloat16_rn(p[i]);
}

/* gradient = sum of the partial gradients (the same order on every run), then
   the Adam step on it (lr > 0) with the BF16 copy of the new weights.  Once a
   wait of k_train has run out (*err, until the host clears it) there is no
   whole gradient: this step and the ones queued behind it change nothing, and
   their loss and hits say so.  A warp
   sums an eighth of the partials of 128 parameters, four per lane; block 0 adds
   up the loss.  Bound by reading the partials (128 of 198 KB) out of L2, where
   k_train has just written them: 16-byte loads and 388 blocks, one wave, in
   place of 4-byte loads and 1,549 blocks, and the weights and moments loaded
   ahead of the sum (four training steps 417 -> 403 us). */
constexpr int kRedParams = 128;
constexpr int kNoStep = -1; /* hits of a step that was not taken */
static_assert(NPARAM % 4 == 0, "a partial gradient is read in fours");
__global__ void __launch_bounds__(256) k_reduce_adam(const float* part, int nparts, float* g, float* p, float* m,
                                                     float* v, unsigned char* pack, float lr, float b1, float b2,
                                                     float eps, float c1, float c2, const float* part_loss,
                                                     const int* part_ok, const int* err, float* loss, int* right)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); /* the next step's k_train */
    __shared__ float s[8][kRedParams];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int j = blockIdx.x * kRedParams + (int)threadIdx.x;
    const bool mine = threadIdx.x < kRedParams && j < NPARAM;
    const int i = mine ? part_param(j) : 0;
    /* after k_train's end, which comes after the last step's (the parameters
       and moments below) */
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (*err) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            *loss = __int_as_float(0x7fffffff); /* NaN */
            *right = kNoStep;
        }
        return;
    }
    float p0 = 0.0f, m0 = 0.0f, v0 = 0.0f;
    if (mine && lr > 0.0f) {
        p0 = p[i];
        m0 = m[i];
        v0 = v[i];
    }
    const int j4 = blockIdx.x * kRedParams + 4 * lane;
    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (j4 < NPARAM) {
#pragma unroll 8
        for (int q = w; q < nparts; q += 8) {
            const float4 x = *reinterpret_cast<const float4*>(part + (size_t)q * NPARAM + j4);
            a.x += x.x;
            a.y += x.y;
            a.z += x.z;
            a.w += x.w;
        }
    }
    *reinterpret_cast<float4*>(&s[w][4 * lane]) = a;
    __syncthreads();
    if (blockIdx.x == 0 && w == 7) {
        float l = 0.0f;
        int k = 0;
        for (int q = lane; q < nparts; q += 32) {
            l += part_loss[q];
            k += part_ok[q];
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        k = __reduce_add_sync(0xffffffffu, k);
        if (lane == 0) {
            *loss = l;
            *right = k;
        }
    }
    if (!mine) return;
    float gi = s[0][threadIdx.x];
#pragma unroll
    for (int q = 1; q < 8; q++) gi += s[q][threadIdx.x];
    g[i] = gi;
    if (!(lr > 0.0f)) return;
    const float mi = b1 * m0 + (1.0f - b1) * gi;
    const float vi = b2 * v0 + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pn = p0 - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pn;
    const int o = pack_off(i);
    if (o >= 0) *reinterpret_cast<__nv_bfloat16*>(pack + o) = __float2bfloat16_rn(pn);
}

}  // namespace

struct ecmg_mlp {
    float* p = nullptr;     /* FP32 master parameters */
    float* g = nullptr;     /* gradients */
    float* m = nullptr;     /* Adam first moment */
    float* v = nullptr;     /* Adam second moment */
    unsigned char* pack = nullptr; /* BF16 weights in the tensor-core operand layout (inference) */
    int* derr = nullptr;           /* inference error flag (ecmg_mlp_predict), and its page-locked copy */
    int* h_err = nullptr;
    int sms = 1;
    int spin = kSpinDefault;       /* polls of an mbarrier before the inference gives up */
    float* bias = nullptr;  /* b1 | b2 | b3 */
    int step = 0;
    bool packed = false;
    /* training (allocated by its first use): the partial gradients of up to
       one CTA per SM with their losses and hits, the BF16 operand copy of the
       weights, and per-step losses and hits; page-locked staging of what
       loss_grad and train read back */
    int parts = 0;
    float *part = nullptr, *part_loss = nullptr, *hist_loss = nullptr;
    int *part_ok = nullptr, *hist_ok = nullptr, *gerr = nullptr;
    unsigned char* tpack = nullptr;
    float* h_grad = nullptr;
    int hist = 0;
    cudaStream_t s = nullptr;
};

namespace ecmg {
/* used by the tick (ctx.cu) */
cudaError_t mlp_infer(ecmg_mlp* mlp, const void* X, const int* n_dev, int n_max, unsigned char* cls, cudaStream_t s,
                      int sms, int* err, int errbit);
cudaError_t mlp_pack(ecmg_mlp* mlp);
}  // namespace ecmg

cudaError_t ecmg::mlp_pack(ecmg_mlp* mm)
{
    /* outside any stream capture: the inference kernel's shared memory limit */
    cudaError_t ea = cudaFuncSetAttribute(k_mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInferSmem);
    if (ea != cudaSuccess) return ea;
    if (mm->packed) return cudaSuccess;
    k_pack_tc<<<64, 256, 0, mm->s>>>(mm->p + OW1, IN, HID, mm->pack);
    k_pack_tc<<<64, 256, 0, mm->s>>>(mm->p + OW2, HID, HID, mm->pack + kW1B);
    k_pack_tc<<<64, 256, 0, mm->s>>>(mm->p + OW3, HID, OUT, mm->pack + kW1B + kW2B);
    cudaMemcpyAsync(mm->bias, mm->p + OB1, sizeof(float) * HID, cudaMemcpyDeviceToDevice, mm->s);
    cudaMemcpyAsync(mm->bias + HID, mm->p + OB2, sizeof(float) * HID, cudaMemcpyDeviceToDevice, mm->s);
    cudaMemcpyAsync(mm->bias + 2 * HID, mm->p + OB3, sizeof(float) * OUT, cudaMemcpyDeviceToDevice, mm->s);
    cudaError_t e = cudaStreamSynchronize(mm->s);
    if (e == cudaSuccess) mm->packed = true;
    return e;
}

constexpr float kBeta1 = 0.9f, kBeta2 = 0.999f; /* Adam */

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

/* the driver's tensor-map encoder, reached through the runtime (no link
   against the driver library) */
static EncodeTiledFn tensor_map_encoder()
{
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
        cudaGetLastError();
    });
    return fn;
}

/* X [rows, IN] bf16 row-major as a 2D tensor; boxes of 8 columns x 128 rows,
   rows beyond `rows` read as zeros */
static cudaError_t feature_map(CUtensorMap* tm, const void* X, int rows)
{
    EncodeTiledFn enc = tensor_map_encoder();
    if (!enc) return cudaErrorNotSupported;
    const cuuint64_t dims[2] = {(cuuint64_t)IN, (cuuint64_t)(rows > 0 ? rows : 1)};
    const cuuint64_t strides[1] = {(cuuint64_t)IN * 2};
    const cuuint32_t box[2] = {8, (cuuint32_t)kTile};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(X), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t ecmg::mlp_infer(ecmg_mlp* mm, const void* X, const int* n_dev, int n_max, unsigned char* cls,
                            cudaStream_t s, int sms, int* err, int errbit)
{
    CUtensorMap tm;
    cudaError_t e = feature_map(&tm, X, n_max);
    if (e != cudaSuccess) return e;
    int tiles = (n_max + kTile - 1) / kTile;
    int grid = tiles < sms ? tiles : sms; /* one CTA per SM holds the weights once */
    if (grid < 1) grid = 1;
    k_mlp_infer<<<grid, kInferThreads, kInferSmem, s>>>(tm, n_dev, n_max, mm->pack, mm->bias, cls, err, errbit,
                                                         mm->spin);
    return cudaGetLastError();
}

extern "C" {

ecmg_status ecmg_mlp_create(unsigned long long seed, ecmg_mlp** out)
{
    if (!out) return ECMG_ERR_INVALID_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) {
        cudaGetLastError();
        return ECMG_ERR_NO_DEVICE;
    }
    ecmg_mlp* mm = new ecmg_mlp();
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&mm->sms, cudaDevAttrMultiProcessorCount, dev);
    bool ok = cudaStreamCreateWithFlags(&mm->s, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMalloc(&mm->p, sizeof(float) * NPARAM) == cudaSuccess &&
              cudaMalloc(&mm->g, sizeof(float) * NPARAM) == cudaSuccess &&
              cudaMalloc(&mm->m, sizeof(float) * NPARAM) == cudaSuccess &&
              cudaMalloc(&mm->v, sizeof(float) * NPARAM) == cudaSuccess &&
              cudaMalloc(&mm->pack, (size_t)kWB) == cudaSuccess &&
              cudaMalloc(&mm->derr, sizeof(int)) == cudaSuccess && cudaMemset(mm->derr, 0, sizeof(int)) == cudaSuccess &&
              cudaMallocHost(&mm->h_err, sizeof(int)) == cudaSuccess &&
              cudaMalloc(&mm->bias, sizeof(float) * (2 * HID + OUT)) == cudaSuccess;
    if (!ok) {
        ecmg_mlp_destroy(mm);
        return ECMG_ERR_CUDA;
    }
    /* He-style init from a 64-bit mixer of the seed (host, deterministic) */
    std::vector<float> h(NPARAM, 0.0f);
    unsigned long long st = seed * 0x9E3779B97F4A7C15ull + 1;
    auto rnd = [&]() {
        st += 0x9E3779B97F4A7C15ull;
        unsigned long long z = st;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0; /* U(-1,1) */
    };
    auto fill = [&](int off, int fan_in, int cnt) {
        double a = std::sqrt(3.0 * 2.0 / fan_in);
        for (int i = 0; i < cnt; i++) h[off + i] = (float)(a * rnd());
    };
    fill(OW1, IN, IN * HID);
    fill(OW2, HID, HID * HID);
    fill(OW3, HID, HID * OUT);
    cudaMemcpy(mm->p, h.data(), sizeof(float) * NPARAM, cudaMemcpyHostToDevice);
    cudaMemset(mm->m, 0, sizeof(float) * NPARAM);
    cudaMemset(mm->v, 0, sizeof(float) * NPARAM);
    *out = mm;
    return ECMG_OK;
}

ecmg_status ecmg_mlp_destroy(ecmg_mlp* mm)
{
    if (!mm) return ECMG_ERR_INVALID_ARG;
    if (mm->s) cudaStreamSynchronize(mm->s);
    void* ds[] = {mm->p, mm->g, mm->m, mm->v, mm->bias, mm->pack, mm->derr, mm->part, mm->part_loss, mm->hist_loss,
                  mm->part_ok, mm->hist_ok, mm->gerr, mm->tpack};
    for (void* d : ds)
        if (d) cudaFree(d);
    if (mm->h_grad) cudaFreeHost(mm->h_grad);
    if (mm->h_err) cudaFreeHost(mm->h_err);
    if (mm->s) cudaStreamDestroy(mm->s);
    delete mm;
    return ECMG_OK;
}

int ecmg_mlp_param_count(void) { return NPARAM; }

ecmg_status ecmg_mlp_get_params(ecmg_mlp* mm, float* host_out)
{
    if (!mm || !host_out) return ECMG_ERR_INVALID_ARG;
    cudaStreamSynchronize(mm->s);
    return cudaMemcpy(host_out, mm->p, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost) == cudaSuccess ? ECMG_OK
                                                                                                       : ECMG_ERR_CUDA;
}

ecmg_status ecmg_mlp_set_params(ecmg_mlp* mm, const float* host_in)
{
    if (!mm || !host_in) return ECMG_ERR_INVALID_ARG;
    for (int i = 0; i < NPARAM; i++)
        if (!std::isfinite(host_in[i])) return ECMG_ERR_INVALID_ARG;
    cudaStreamSynchronize(mm->s);
    if (cudaMemcpy(mm->p, host_in, sizeof(float) * NPARAM, cudaMemcpyHostToDevice) != cudaSuccess) return ECMG_ERR_CUDA;
    mm->packed = false;
    return ECMG_OK;
}

/* training scratch, and room for the losses of `steps` steps */
static ecmg_status ensure_train(ecmg_mlp* mm, int steps)
{
    if (!mm->part) {
        const size_t np = (size_t)mm->sms;
        bool ok = cudaMalloc(&mm->part_loss, sizeof(float) * np) == cudaSuccess &&
                  cudaMalloc(&mm->part_ok, sizeof(int) * np) == cudaSuccess &&
                  cudaMalloc(&mm->tpack, (size_t)kWB) == cudaSuccess &&
                  cudaMalloc(&mm->gerr, sizeof(int)) == cudaSuccess &&
                  cudaMemset(mm->gerr, 0, sizeof(int)) == cudaSuccess &&
                  cudaMallocHost(&mm->h_grad, sizeof(float) * (NPARAM + 2)) == cudaSuccess &&
                  /* outside any stream capture: the kernel's shared memory limit */
                  cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem) ==
                      cudaSuccess &&
                  cudaMalloc(&mm->part, sizeof(float) * np * NPARAM) == cudaSuccess;
        if (!ok) return ECMG_ERR_CUDA;
        mm->parts = mm->sms;
    }
    if (steps > mm->hist) {
        if (mm->hist_loss) cudaFree(mm->hist_loss);
        if (mm->hist_ok) cudaFree(mm->hist_ok);
        mm->hist_loss = nullptr;
        mm->hist_ok = nullptr;
        mm->hist = 0;
        if (cudaMalloc(&mm->hist_loss, sizeof(float) * (size_t)steps) != cudaSuccess ||
            cudaMalloc(&mm->hist_ok, sizeof(int) * (size_t)steps) != cudaSuccess)
            return ECMG_ERR_CUDA;
        mm->hist = steps;
    }
    return ECMG_OK;
}

/* forward and backward on B rows (the rows of X in order, or drawn with the
   seed), the gradient in mm->g and, for lr > 0, the Adam step; the summed
   loss and the hits go to entry `at` of the history.  Every contraction takes
   BF16 operands on the tensor cores and accumulates in FP32; the elementwise
   steps and the master weights are FP32. */
static cudaError_t train_step(ecmg_mlp* mm, const void* X, const unsigned char* y, int n, int B,
                              unsigned long long seed, int draw, int at, float lr, float c1, float c2)
{
    /* as few CTAs as give every one the same number of tiles: each writes a
       partial gradient of 198 KB (65,536 rows: 128 CTAs, not 152) */
    const int tiles = (B + kTile - 1) / kTile, rounds = (tiles + mm->parts - 1) / mm->parts;
    const int grid = (tiles + rounds - 1) / rounds;
    /* its start -- tensor memory, row indices, the first rows -- runs beside the
       end of the kernel before, whose weights it waits for (four steps 402 ->
       393 us, 3,001 rows 65 -> 62).  The reduction is launched the same way: its
       blocks are let in as the CTAs end, not before, where they would crowd on
       the SMs that have no tile (393 -> 381; let in before the partial gradients
       are written: 398) */
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kTrThreads);
    cfg.dynamicSmemBytes = kTrainSmem;
    cfg.stream = mm->s;
    cudaLaunchAttribute pdl{};
    pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &pdl;
    cfg.numAttrs = 1;
    const cudaError_t e =
        cudaLaunchKernelEx(&cfg, k_train, (const __nv_bfloat16*)X, y, n, B, ~0ull / (unsigned)n, seed, draw,
                           (const unsigned char*)mm->tpack, (const float*)mm->p, mm->part, mm->part_loss, mm->part_ok,
                           mm->gerr, mm->spin);
    if (e != cudaSuccess) return e;
    cfg.gridDim = dim3((NPARAM + kRedParams - 1) / kRedParams);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    return cudaLaunchKernelEx(&cfg, k_reduce_adam, (const float*)mm->part, grid, mm->g, mm->p, mm->m, mm->v, mm->tpack, lr,
                              kBeta1, kBeta2, 1e-8f, c1, c2, (const float*)mm->part_loss, (const int*)mm->part_ok,
                              (const int*)mm->gerr, mm->hist_loss + at, mm->hist_ok + at);
}

ecmg_status ecmg_mlp_loss_grad(ecmg_mlp* mm, const void* dev_x, const unsigned char* dev_y, int n, float* loss,
                               float* host_grad)
{
    if (!mm || !dev_x || !dev_y || n < 1) return ECMG_ERR_INVALID_ARG;
    if (ensure_train(mm, 1) != ECMG_OK) return ECMG_ERR_CUDA;
    k_pack_all<<<(NPARAM + 255) / 256, 256, 0, mm->s>>>(mm->p, mm->tpack);
    cudaError_t e = train_step(mm, dev_x, dev_y, n, n, 0, 0, 0, 0.0f, 1.0f, 1.0f);
    /* one wait for everything that is read back */
    float* h = mm->h_grad;
    int* herr = (int*)(h + NPARAM + 1);
    auto get = [&](void* dst, const void* src, size_t bytes) {
        if (e == cudaSuccess) e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, mm->s);
    };
    if (host_grad) get(h, mm->g, sizeof(float) * NPARAM);
    get(h + NPARAM, mm->hist_loss, sizeof(float));
    get(herr, mm->gerr, sizeof(int));
    if (e == cudaSuccess) e = cudaStreamSynchronize(mm->s);
    if (e != cudaSuccess) return ECMG_ERR_CUDA;
    if (*herr) {
        cudaMemsetAsync(mm->gerr, 0, sizeof(int), mm->s);
        return ECMG_ERR_BOUND;
    }
    if (loss) *loss = h[NPARAM] / (float)n;
    if (host_grad) std::memcpy(host_grad, h, sizeof(float) * NPARAM);
    return ECMG_OK;
}

ecmg_status ecmg_mlp_train(ecmg_mlp* mm, const void* dev_x, const unsigned char* dev_y, int n, int steps, int batch,
                           float lr, unsigned long long seed, float* host_loss, float* host_acc)
{
    if (!mm || !dev_x || !dev_y || n < 1 || steps < 0 || batch < 1 || !(lr > 0.0f)) return ECMG_ERR_INVALID_ARG;
    if (ensure_train(mm, std::max(1, steps)) != ECMG_OK) return ECMG_ERR_CUDA;
    k_pack_all<<<(NPARAM + 255) / 256, 256, 0, mm->s>>>(mm->p, mm->tpack);
    for (int it = 0; it < steps; it++) {
        const unsigned long long sd = seed + 0x51ED27ull * (unsigned long long)(mm->step + 1);
        mm->step++;
        const float c1 = 1.0f - powf(kBeta1, (float)mm->step), c2 = 1.0f - powf(kBeta2, (float)mm->step);
        if (train_step(mm, dev_x, dev_y, n, batch, sd, 1, it, lr, c1, c2) != cudaSuccess) return ECMG_ERR_CUDA;
    }
    mm->packed = false;
    /* the steps' losses and hits are read back together at the end */
    std::vector<int> ok(host_acc ? (size_t)steps : 0);
    int herr = 0;
    cudaError_t e = cudaSuccess;
    if (host_loss && steps)
        e = cudaMemcpyAsync(host_loss, mm->hist_loss, sizeof(float) * (size_t)steps, cudaMemcpyDeviceToHost, mm->s);
    if (e == cudaSuccess && host_acc && steps)
        e = cudaMemcpyAsync(ok.data(), mm->hist_ok, sizeof(int) * (size_t)steps, cudaMemcpyDeviceToHost, mm->s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&herr, mm->gerr, sizeof(int), cudaMemcpyDeviceToHost, mm->s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(mm->s);
    if (e != cudaSuccess) return ECMG_ERR_CUDA;
    if (herr) { /* the model has taken the steps before the wait that ran out */
        ok.resize((size_t)steps);
        cudaMemsetAsync(mm->gerr, 0, sizeof(int), mm->s);
        if (steps && (cudaMemcpyAsync(ok.data(), mm->hist_ok, sizeof(int) * (size_t)steps, cudaMemcpyDeviceToHost,
                                      mm->s) != cudaSuccess ||
                      cudaStreamSynchronize(mm->s) != cudaSuccess))
            return ECMG_ERR_CUDA;
        mm->step -= (int)std::count(ok.begin(), ok.end(), kNoStep);
    }
    for (int it = 0; it < steps; it++) {
        if (host_loss) host_loss[it] /= (float)batch;
        if (host_acc) host_acc[it] = herr && ok[it] == kNoStep ? NAN : (float)ok[it] / (float)batch;
    }
    return herr ? ECMG_ERR_BOUND : ECMG_OK;
}

ecmg_status ecmg_mlp_set_wait_limit(ecmg_mlp* mm, int polls)
{
    if (!mm || polls < 0) return ECMG_ERR_INVALID_ARG;
    mm->spin = polls > 0 ? polls : kSpinDefault;
    return ECMG_OK;
}

ecmg_status ecmg_mlp_predict(ecmg_mlp* mm, const void* dev_x, int n, unsigned char* dev_cls)
{
    if (!mm || !dev_x || !dev_cls || n < 0) return ECMG_ERR_INVALID_ARG;
    if (n == 0) return ECMG_OK;
    if (ecmg::mlp_pack(mm) != cudaSuccess) return ECMG_ERR_CUDA;
    if (ecmg::mlp_infer(mm, dev_x, nullptr, n, dev_cls, mm->s, mm->sms, mm->derr, 1) != cudaSuccess)
        return ECMG_ERR_CUDA;
    if (cudaMemcpyAsync(mm->h_err, mm->derr, sizeof(int), cudaMemcpyDeviceToHost, mm->s) != cudaSuccess ||
        cudaStreamSynchronize(mm->s) != cudaSuccess)
        return ECMG_ERR_CUDA;
    if (*mm->h_err == 0) return ECMG_OK;
    cudaMemsetAsync(mm->derr, 0, sizeof(int), mm->s); /* the flag is zero between calls */
    return ECMG_ERR_BOUND;
}

}  // extern "C"
