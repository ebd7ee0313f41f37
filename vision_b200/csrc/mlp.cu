// Radiance-cache MLP on the tcgen05 tensor cores (sm_100a).
//
// Network: 64 BF16 inputs -> 4 hidden layers of 64 (ReLU) -> 3 outputs, no
// biases.  Every layer is a tcgen05.mma.kind::f16 with BF16 operands in
// shared memory and the FP32 accumulator in tensor memory:
//   inference  (k_mlp_infer): one CTA per SM holding the forward weights once
//     and running kInferGroups independent 4-warp pipelines, each with its
//     own 96 tensor-memory columns (64 of accumulator, 32 of activations) and
//     two tile buffers; while a pipeline runs the five layers of one 128-row
//     tile, the TMA engine loads its next tile into the other buffer (128-byte
//     swizzle, rows past n zero-filled).  M=128 x N=64 (N=16 for the padded
//     output layer), K=64 as four K=16 steps.  Thread t of a pipeline owns
//     tile row t: after each layer it reads its accumulator row with
//     tcgen05.ld (32x32b), rounds to BF16, applies ReLU and writes the next
//     layer's operand row back to tensor memory with tcgen05.st (two BF16 per
//     column), where the MMA reads it; only the features and the weights come
//     from shared memory.
//   training   (k_mlp_train): the same forward pass keeping every layer's
//     BF16 input in shared memory; the relative-L2 loss gradient; the backward
//     data products dX = dZ W^T (M=128) masked by ReLU'; and the weight
//     gradients dW = X^T dZ as M=64 MMAs whose operands are the same
//     shared-memory tiles read MN-major, accumulated in tensor memory over all
//     tiles of the CTA and added to the global FP32 gradient once per CTA.
//   k_mlp_adam updates the FP32 master weights; k_mlp_pack rewrites the BF16
//   operand image (W as [out][in], read MN-major for the data gradients).
// Shared-memory operands use the canonical no-swizzle layout: 8-row x 16-byte
// core matrices, rows of a core matrix 16 B apart; for a K-major operand with
// R rows, core matrices along M/N are 128 B apart (SBO) and along K R*16 B
// apart (LBO); the same 128-row activation tile read MN-major has LBO = 128 B
// (next 8 batch rows) and SBO = 2048 B (next 8 features).
// Every wait on the MMA-completion mbarrier is bounded; on timeout the kernel
// records the error, skips the rest of its work, frees its tensor memory and
// returns.
#include "vs_mlp.h"
#include "vs_resident.h"

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cstdint>

namespace vs {

namespace {

constexpr int kTile = 128;
constexpr uint32_t kTileBytes = kTile * 64 * 2;       // 16 KB activation tile
constexpr uint32_t kPackBytes = kMlpPackElems * 2;     // 34,816 B
constexpr long long kWaitCycles = 4000000000ll;       // ~2 s at 1.9 GHz

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor, no swizzle, Blackwell version field.
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return static_cast<uint64_t>((saddr >> 4) & 0x3FFFu) | (static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16) |
           (static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor: BF16 x BF16 -> FP32, dense.
__host__ __device__ constexpr uint32_t idesc(int M, int N, int a_mn, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(a_mn) << 15) |
           (static_cast<uint32_t>(b_mn) << 16) | (static_cast<uint32_t>(N >> 3) << 17) |
           (static_cast<uint32_t>(M >> 4) << 24);
}

__device__ __forceinline__ void mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t id, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(id), "r"(accumulate));
}

// The same with the A operand in tensor memory (M = 128: lane = row, two K
// elements per 32-bit column).
__device__ __forceinline__ void mma_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t id, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b), "r"(id), "r"(accumulate));
}

__device__ __forceinline__ void commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
                 : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}

// Bounded wait on the phase parity of an mbarrier.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    long long t0 = clock64();
    for (;;) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
        if (clock64() - t0 > kWaitCycles) return false;
    }
}

// Issues the loads of 64 accumulator columns (four 32x32b.x16) and waits for
// them once.
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, float *v) {
    uint32_t r[64];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[16 * q + 0]), "=r"(r[16 * q + 1]), "=r"(r[16 * q + 2]), "=r"(r[16 * q + 3]),
              "=r"(r[16 * q + 4]), "=r"(r[16 * q + 5]), "=r"(r[16 * q + 6]), "=r"(r[16 * q + 7]),
              "=r"(r[16 * q + 8]), "=r"(r[16 * q + 9]), "=r"(r[16 * q + 10]), "=r"(r[16 * q + 11]),
              "=r"(r[16 * q + 12]), "=r"(r[16 * q + 13]), "=r"(r[16 * q + 14]), "=r"(r[16 * q + 15])
            : "r"(taddr + 16u * q));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(r[i]);
}

// The first 4 accumulator columns of this thread's row.
__device__ __forceinline__ float4 tmem_ld4(uint32_t taddr) {
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    return make_float4(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]), __uint_as_float(r[3]));
}

// Stores 32 columns of this thread's row and waits for the store.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
        "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&h);
}
// ReLU of a pair after rounding (the same value as rounding the ReLU; NaN
// gives 0 either way).
__device__ __forceinline__ uint32_t pack2_relu(float a, float b) {
    const __nv_bfloat162 h = __hmax2(__floats2bfloat162_rn(a, b), __nv_bfloat162(__ushort_as_bfloat16(0), __ushort_as_bfloat16(0)));
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ float bf_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf_hi(uint32_t u) { return __uint_as_float(u & 0xFFFF0000u); }

// Byte offset of 16-byte chunk kc (elements 8kc..8kc+7) of row r in a
// 128-row K-major tile.
__device__ __forceinline__ uint32_t tile_chunk(uint32_t r, uint32_t kc) {
    return kc * 2048u + (r >> 3) * 128u + (r & 7u) * 16u;
}

// Writes 64 values as BF16 into row r of a 128-row tile.
__device__ __forceinline__ void st_row64(uint8_t *tile, uint32_t r, const float *v) {
#pragma unroll
    for (int kc = 0; kc < 8; ++kc) {
        uint4 u = make_uint4(pack2(v[8 * kc], v[8 * kc + 1]), pack2(v[8 * kc + 2], v[8 * kc + 3]),
                             pack2(v[8 * kc + 4], v[8 * kc + 5]), pack2(v[8 * kc + 6], v[8 * kc + 7]));
        *reinterpret_cast<uint4 *>(tile + tile_chunk(r, kc)) = u;
    }
}

__device__ __forceinline__ void ld_row64_bf(const uint8_t *tile, uint32_t r, float *v) {
#pragma unroll
    for (int kc = 0; kc < 8; ++kc) {
        uint4 u = *reinterpret_cast<const uint4 *>(tile + tile_chunk(r, kc));
        v[8 * kc + 0] = bf_lo(u.x);
        v[8 * kc + 1] = bf_hi(u.x);
        v[8 * kc + 2] = bf_lo(u.y);
        v[8 * kc + 3] = bf_hi(u.y);
        v[8 * kc + 4] = bf_lo(u.z);
        v[8 * kc + 5] = bf_hi(u.z);
        v[8 * kc + 6] = bf_lo(u.w);
        v[8 * kc + 7] = bf_hi(u.w);
    }
}

// Row `row` of the global feature matrix (zeros past n).
__device__ __forceinline__ void ld_features(uint4 *f, const uint16_t *feat, uint64_t row, uint32_t n) {
    const uint4 *src = reinterpret_cast<const uint4 *>(feat + row * 64u);
#pragma unroll
    for (int kc = 0; kc < 8; ++kc) f[kc] = row < n ? __ldg(src + kc) : make_uint4(0, 0, 0, 0);
}

__device__ __forceinline__ void copy_to_smem(uint8_t *dst, const uint4 *src, uint32_t bytes) {
    for (uint32_t i = threadIdx.x; i < bytes / 16u; i += blockDim.x) reinterpret_cast<uint4 *>(dst)[i] = __ldg(src + i);
}

// Forward weight descriptors: layer l < 4 is [64 out][64 in] (LBO 1024), the
// output layer [16 out][64 in] (LBO 256); K step s advances 2 K-chunks.
__device__ __forceinline__ uint64_t w_fwd_desc(uint32_t wbase, int l, int s) {
    if (l < 4) return sdesc(wbase + l * 8192u + s * 2048u, 1024u, 128u);
    return sdesc(wbase + 4u * 8192u + s * 512u, 256u, 128u);
}
// The same image read for dX = dZ W^T: N = in, K = out, MN-major (the next 8
// out rows 128 B on, the next 8 in columns 1024 B or, in the output layer's
// image, 256 B on); K step s advances 16 out rows.
__device__ __forceinline__ uint64_t w_bwd_desc(uint32_t wbase, int l, int s) {
    if (l < 4) return sdesc(wbase + l * 8192u + s * 256u, 128u, 1024u);
    return sdesc(wbase + 4u * 8192u, 128u, 256u);
}
// A 128-row activation tile as a K-major operand, K step s.
__device__ __forceinline__ uint64_t tile_kdesc(uint32_t base, int s) { return sdesc(base + s * 4096u, 2048u, 128u); }
// The same tile read MN-major (features along M/N, batch rows along K), K step s.
__device__ __forceinline__ uint64_t tile_mndesc(uint32_t base, int s) { return sdesc(base + s * 256u, 128u, 2048u); }

struct TmemSlot {
    uint32_t addr;
};

__device__ __forceinline__ void tmem_alloc(uint32_t slot_saddr, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_saddr), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

// A 128-row feature tile written by TMA with the 128-byte swizzle (row r at
// 128 r, its 16-byte chunk c at (c ^ (r & 7)) * 16, 1024-byte aligned) as a
// K-major operand, K step s: SBO 1024 B between 8-row groups, the K=16 step
// 32 B further inside the swizzle atom, layout type SWIZZLE_128B.
__device__ __forceinline__ uint64_t tile_sw128_desc(uint32_t base, int s) {
    return sdesc(base + s * 32u, 16u, 1024u) | (2ull << 61);
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}

// One 2D tile of the feature tensor map into shared memory (no multicast),
// completing on `mbar` with its byte count.
__device__ __forceinline__ void tma_load_tile(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(map), "r"(x), "r"(y), "r"(mbar)
        : "memory");
}

// Named barrier over the 128 threads of pipeline g (barrier 1 + g), returning
// whether every thread passed true.
__device__ __forceinline__ bool group_sync_and(uint32_t g, bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, %2, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(r)
        : "r"(static_cast<uint32_t>(v)), "r"(1u + g)
        : "memory");
    return r != 0u;
}

// Five pipelines of 96 columns fill the 512 of tensor memory.  With the
// activations in shared memory instead (written by the epilogue, read by the
// next MMA) each tile moved 200 KB through shared memory, 1600 of the 2300
// cycles it took; here it moves 66 KB.
// 2,073,600 rows: 130 -> 106 us (bound now by the epilogues' latency and the
// conversions: ALU 51 %, tensor pipe 33 %, 2.7 TB/s).
constexpr uint32_t kInferGroups = 5;
constexpr uint32_t kInferCols = 96;
static_assert(kInferGroups * kInferCols <= 512u, "tensor memory columns");
constexpr uint32_t kInferThreads = 128u * kInferGroups;
constexpr uint32_t kInferBars = 3u * kInferGroups;  // per pipeline: two tile loads, one MMA
constexpr uint32_t kInferSmem = 1024u + kPackBytes + kInferGroups * 2u * kTileBytes + 8u * kInferBars + 16u;
static_assert(kInferSmem <= 232448u, "inference shared memory above the per-CTA limit");

__global__ void __launch_bounds__(kInferThreads, 1) k_mlp_infer(const __grid_constant__ CUtensorMap fmap, uint32_t n,
                                                                const uint4 *__restrict__ wpack,
                                                                float4 *__restrict__ out, int *err) {
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte alignment for the swizzled TMA destinations.
    const uint32_t raw = smem_u32(smem_raw);
    uint8_t *smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    uint8_t *w = smem;
    uint8_t *bufs = smem + kPackBytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(bufs + kInferGroups * 2u * kTileBytes);
    uint32_t *slot = reinterpret_cast<uint32_t *>(bars + kInferBars);
    const uint32_t tid = threadIdx.x, g = tid >> 7, gt = tid & 127u;
    if (tid < 32) tmem_alloc(smem_u32(slot), 512);
    if (tid == 0) {
        for (uint32_t i = 0; i < kInferBars; ++i) mbar_init(smem_u32(bars + i), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    copy_to_smem(w, wpack, kPackBytes);
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    // Pipeline g: accumulator columns [96 g, 96 g + 64), activation columns
    // [96 g + 64, 96 g + 96), tile buffers buf0 + {0, kTileBytes}, barriers
    // load[0], load[1], mma.
    const uint32_t tmem = *slot + kInferCols * g, act = tmem + 64u;
    const uint32_t lane = (gt & ~31u) << 16;
    const uint32_t wbase = smem_u32(w);
    const uint32_t buf0 = smem_u32(bufs + g * 2u * kTileBytes);
    const uint32_t mb_load = smem_u32(bars + 3u * g), mb_mma = mb_load + 16u;
    const uint32_t tiles = (n + kTile - 1) / kTile;
    const uint32_t stride = gridDim.x * kInferGroups;
    uint32_t tt = blockIdx.x * kInferGroups + g;
    uint32_t ph_load = 0u, ph_mma = 0u;  // parity bits (bit b: buffer b)
    bool pending[2] = {false, false};
    if (gt == 0 && tt < tiles) {
        mbar_expect_tx(mb_load, kTileBytes);
        tma_load_tile(buf0, &fmap, 0, static_cast<int>(tt * kTile), mb_load);
    }
    pending[0] = tt < tiles;
    bool ok = true;
    for (uint32_t k = 0; tt < tiles && ok; tt += stride, ++k) {
        const uint32_t cur = k & 1u, nxt = cur ^ 1u;
        const uint32_t buf = buf0 + cur * kTileBytes;
        // The other buffer held the previous tile, whose last MMA has
        // completed: load the next tile into it now.
        if (tt + stride < tiles) {
            if (gt == 0) {
                mbar_expect_tx(mb_load + 8u * nxt, kTileBytes);
                tma_load_tile(buf0 + nxt * kTileBytes, &fmap, 0, static_cast<int>((tt + stride) * kTile),
                              mb_load + 8u * nxt);
            }
            pending[nxt] = true;
        }
        bool done = mbar_wait(mb_load + 8u * cur, (ph_load >> cur) & 1u);
        ph_load ^= 1u << cur;
        pending[cur] = !done;
        ok = group_sync_and(g, done);
        if (!ok) break;
        const uint64_t row = static_cast<uint64_t>(tt) * kTile + gt;
        for (int l = 0; l < 5; ++l) {
            if (gt == 0) {
                const uint32_t id = l < 4 ? idesc(128, 64, 0, 0) : idesc(128, 16, 0, 0);
                if (l == 0) {
#pragma unroll
                    for (int s = 0; s < 4; ++s) mma(tmem, tile_sw128_desc(buf, s), w_fwd_desc(wbase, 0, s), id, s > 0);
                } else {
#pragma unroll
                    for (int s = 0; s < 4; ++s) mma_ta(tmem, act + 8u * s, w_fwd_desc(wbase, l, s), id, s > 0);
                }
                commit(mb_mma);
            }
            done = mbar_wait(mb_mma, ph_mma);
            ph_mma ^= 1u;
            fence_after();
            // The epilogue of a thread whose wait ran out is skipped; the
            // barrier that follows makes the pipeline agree to stop.
            if (done && l < 4) {
                float v[64];
                tmem_ld64(tmem + lane, v);
                uint32_t h[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) h[i] = pack2_relu(v[2 * i], v[2 * i + 1]);
                tmem_st32(act + lane, h);
            } else if (done) {
                const float4 v = tmem_ld4(tmem + lane);
                if (row < n) out[row] = make_float4(v.x, v.y, v.z, 0.0f);
            }
            fence_before();
            ok = group_sync_and(g, done);
            fence_after();
            if (!ok) break;
        }
    }
    // A pipeline that stopped early waits (bounded) for the loads it still
    // has in flight before the CTA releases its shared memory.
    for (uint32_t b = 0; b < 2; ++b)
        if (pending[b]) (void)mbar_wait(mb_load + 8u * b, (ph_load >> b) & 1u);
    if (!ok && gt == 0) atomicExch(err, 1);
    fence_before();
    __syncthreads();
    fence_after();
    if (tid < 32) tmem_free(*slot, 512);
}

// Training shared memory: the weight image, then per pipeline the input tile X0
// and the hidden activations H1..H4 and the output-gradient tile DO
// (128 x 16); barriers and slots.
constexpr uint32_t kTrainPipes = 2;
constexpr uint32_t kTrainThreads = 128u * kTrainPipes + 32u;
constexpr uint32_t kTrainPipeBytes = 5u * kTileBytes + 4096u;
constexpr uint32_t kOffPipe = kPackBytes;
constexpr uint32_t kOffBar = kOffPipe + kTrainPipes * kTrainPipeBytes;
constexpr uint32_t kTrainSmem = kOffBar + 128u;
constexpr uint32_t kTrainCols = 512;   // D of pipeline p: 64 p; dW0..dW3: 128 + 64 l; dW4: 384..399
static_assert(kTrainSmem <= 232448u, "training shared memory above the per-CTA limit");

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

// Adds four consecutive floats (16-byte aligned) to global memory.
__device__ __forceinline__ void red_add4(float *p, const float *v) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3])
                 : "memory");
}

// The forward pass, the loss gradient and the backward pass of one tile are
// ten dependent rounds of an MMA batch and an epilogue, each mostly latency.
// Two pipelines of 128 threads (one tile each) alternate, so one's epilogue
// runs under the other's MMAs, and a 65,536-sample step needs two passes over
// the tiles instead of four.  A ninth warp issues every MMA, in a fixed order,
// because both pipelines accumulate the weight gradients in the same columns.
// To fit two pipelines, a layer's gradient dZ overwrites the activations it
// was masked with, and the data gradient reads the forward weight image
// MN-major instead of a second, transposed copy.
// 65,536 samples: kernel 71 -> 34 us; four steps with their updates 424 -> 269 us.
__global__ void __launch_bounds__(kTrainThreads, 1) k_mlp_train(const uint16_t *__restrict__ feat,
                                                                const float4 *__restrict__ target, uint32_t n,
                                                                const uint4 *__restrict__ wpack, float loss_scale,
                                                                float *__restrict__ grad, double *loss, int *err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    // Barriers: ready[p] (the pipeline's 128 threads have written their
    // operands), done[p] (its MMA batch has completed).
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kOffBar);
    uint32_t *slot = reinterpret_cast<uint32_t *>(smem + kOffBar + 32);
    float *red = reinterpret_cast<float *>(smem + kOffBar + 48);
    const uint32_t tid = threadIdx.x, pipe = tid >> 7, gt = tid & 127u;
    if (tid < 32) tmem_alloc(smem_u32(slot), kTrainCols);
    if (tid == 0) {
        for (uint32_t p = 0; p < kTrainPipes; ++p) {
            mbar_init(smem_u32(bars + p), 128);
            mbar_init(smem_u32(bars + kTrainPipes + p), 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    copy_to_smem(smem, wpack, kPackBytes);
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *slot;
    const uint32_t wb = smem_u32(smem);
    const uint32_t tiles = (n + kTile - 1) / kTile;
    const uint32_t stride = gridDim.x * kTrainPipes;
    bool ok = true;
    float loss_acc = 0.0f;
    if (pipe == kTrainPipes) {
        // The issuing thread: rounds of both pipelines in turn (0..4: forward
        // layers, 5..9: backward layers 4..0).
        if (gt == 0) {
            uint32_t phase[kTrainPipes] = {0u, 0u};
            for (uint32_t base = blockIdx.x; base < tiles && ok; base += stride) {
                for (int round = 0; round < 10 && ok; ++round) {
#pragma unroll
                    for (uint32_t p = 0; p < kTrainPipes; ++p) {
                        if (!ok || base + p * gridDim.x >= tiles) continue;
                        ok = mbar_wait(smem_u32(bars + p), phase[p]);
                        if (!ok) continue;
                        phase[p] ^= 1u;
                        fence_after();
                        const uint32_t act = smem_u32(smem + kOffPipe + p * kTrainPipeBytes);
                        const uint32_t d = tmem + 64u * p;
                        if (round < 5) {
                            const uint32_t id = round < 4 ? idesc(128, 64, 0, 0) : idesc(128, 16, 0, 0);
#pragma unroll
                            for (int s = 0; s < 4; ++s)
                                mma(d, tile_kdesc(act + round * kTileBytes, s), w_fwd_desc(wb, round, s), id, s > 0);
                        } else {
                            // dW_l += X_l^T dZ_l, dX_l = dZ_l W_l^T; dZ_l lies in H_{l+1}'s tile (l = 4: DO).
                            const int l = 9 - round;
                            const uint32_t x = act + l * kTileBytes, dz = x + kTileBytes;
                            const uint32_t dw = tmem + 128u + 64u * l;
                            const uint32_t id_w = l == 4 ? idesc(64, 16, 1, 1) : idesc(64, 64, 1, 1);
                            const uint32_t first = base == blockIdx.x && p == 0u ? 1u : 0u;
#pragma unroll
                            for (int s = 0; s < 8; ++s)
                                mma(dw, tile_mndesc(x, s), tile_mndesc(dz, s), id_w, (!first || s > 0) ? 1u : 0u);
                            if (l == 4) {
                                mma(d, sdesc(dz, 2048u, 128u), w_bwd_desc(wb, 4, 0), idesc(128, 64, 0, 1), 0u);
                            } else if (l > 0) {
#pragma unroll
                                for (int s = 0; s < 4; ++s)
                                    mma(d, tile_kdesc(dz, s), w_bwd_desc(wb, l, s), idesc(128, 64, 0, 1), s > 0);
                            }
                        }
                        commit(smem_u32(bars + kTrainPipes + p));
                    }
                }
            }
        }
    } else {
        uint8_t *act = smem + kOffPipe + pipe * kTrainPipeBytes;
        uint8_t *DO = act + 5u * kTileBytes;
        const uint32_t ready = smem_u32(bars + pipe), done = smem_u32(bars + kTrainPipes + pipe);
        const uint32_t lane = (gt & ~31u) << 16;
        const uint32_t d = tmem + 64u * pipe + lane;
        uint32_t phase = 0u;
        // Publishes this thread's operand row and waits for the MMA batch.
        auto round_trip = [&]() {
            fence_async_smem();
            fence_before();
            mbar_arrive(ready);
            ok = __all_sync(0xffffffffu, mbar_wait(done, phase)) != 0;
            phase ^= 1u;
            fence_after();
        };
        uint32_t tt = blockIdx.x + pipe * gridDim.x;
        uint4 f[8];
        ld_features(f, feat, static_cast<uint64_t>(tt) * kTile + gt, n);
        for (; tt < tiles && ok; tt += stride) {
            const uint64_t row = static_cast<uint64_t>(tt) * kTile + gt;
            const bool valid = row < n;
#pragma unroll
            for (int kc = 0; kc < 8; ++kc) *reinterpret_cast<uint4 *>(act + tile_chunk(gt, kc)) = f[kc];
            // The next tile's row, in flight under this tile's rounds.
            ld_features(f, feat, row + static_cast<uint64_t>(stride) * kTile, n);
            const float4 t = valid ? __ldg(target + row) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            // Forward: layers 0..3 into H1..H4, output layer into registers.
            for (int l = 0; l < 4 && ok; ++l) {
                round_trip();
                if (!ok) break;
                float v[64];
                tmem_ld64(d, v);
#pragma unroll
                for (int i = 0; i < 64; ++i) v[i] = fmaxf(v[i], 0.0f);
                st_row64(act + (l + 1) * kTileBytes, gt, v);
            }
            if (!ok) break;
            round_trip();
            if (!ok) break;
            const float4 y4 = tmem_ld4(d);
            // Relative L2 loss (denominator without gradient) and its gradient.
            float go[3] = {0.0f, 0.0f, 0.0f};
            if (valid) {
                const float y[3] = {y4.x, y4.y, y4.z}, tv[3] = {t.x, t.y, t.z};
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    float e = y[c] - tv[c];
                    float den = y[c] * y[c] + 0.01f;
                    loss_acc += e * e / den;
                    go[c] = 2.0f * e / den * loss_scale;
                }
            }
            *reinterpret_cast<uint4 *>(DO + tile_chunk(gt, 0)) = make_uint4(pack2(go[0], go[1]), pack2(go[2], 0.0f), 0u, 0u);
            *reinterpret_cast<uint4 *>(DO + tile_chunk(gt, 1)) = make_uint4(0u, 0u, 0u, 0u);
            // Backward: dZ_{l-1} = dX_l where H_l > 0, written over H_l.
            for (int l = 4; l > 0 && ok; --l) {
                round_trip();
                if (!ok) break;
                float v[64], h[64];
                tmem_ld64(d, v);
                ld_row64_bf(act + l * kTileBytes, gt, h);
#pragma unroll
                for (int i = 0; i < 64; ++i) v[i] = h[i] > 0.0f ? v[i] : 0.0f;
                st_row64(act + l * kTileBytes, gt, v);
            }
            if (!ok) break;
            round_trip();
        }
    }
    fence_before();
    const bool all_ok = __syncthreads_and(ok) != 0;
    fence_after();
    // Weight gradients: rows of an M=64 accumulator live in lanes 16w..16w+15
    // of warp w's quarter (row 16w + t in lane 32w + t, t < 16); pipeline p's
    // warps add layers 2p and 2p + 1, pipeline 0's the output layer too.
    if (all_ok && pipe < kTrainPipes && blockIdx.x < tiles) {
        const uint32_t lane = (gt & ~31u) << 16;
        const uint32_t r = 16u * (gt >> 5) + (gt & 31u);
        const bool holder = (gt & 31u) < 16u;
        for (uint32_t l = 2u * pipe; l < 2u * pipe + 2u; ++l) {
            float v[64];
            tmem_ld64(tmem + lane + 128u + 64u * l, v);
            if (holder) {
#pragma unroll
                for (int c = 0; c < 64; c += 4) red_add4(grad + l * 4096u + r * 64u + c, v + c);
            }
        }
        if (pipe == 0) {
            const float4 v = tmem_ld4(tmem + lane + 384u);
            if (holder) {
                atomicAdd(grad + 4 * 4096 + r * 3, v.x);
                atomicAdd(grad + 4 * 4096 + r * 3 + 1, v.y);
                atomicAdd(grad + 4 * 4096 + r * 3 + 2, v.z);
            }
        }
    }
    // Loss reduction.
    if (pipe < kTrainPipes) {
        for (int o = 16; o > 0; o >>= 1) loss_acc += __shfl_xor_sync(0xffffffffu, loss_acc, o);
        if ((tid & 31u) == 0) red[tid >> 5] = loss_acc;
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (tid == 0) {
        double sum = 0.0;
        for (uint32_t w = 0; w < 4u * kTrainPipes; ++w) sum += static_cast<double>(red[w]);
        atomicAdd(loss, sum * loss_scale);
        if (!all_ok) atomicExch(err, 1);
    }
    if (tid < 32) tmem_free(tmem, kTrainCols);
}

// Packed-image offset (elements) of weight (l, in, out).
__device__ __forceinline__ uint32_t pack_offset(int l, uint32_t in, uint32_t out) {
    if (l < 4) return l * 4096u + (in >> 3) * 512u + (out >> 3) * 64u + (out & 7u) * 8u + (in & 7u);
    return 4u * 4096u + (in >> 3) * 128u + (out & 7u) * 8u + (in & 7u);
}
__device__ __forceinline__ void param_coords(uint32_t i, int &l, uint32_t &in, uint32_t &out) {
    if (i < 4u * 4096u) {
        l = static_cast<int>(i / 4096u);
        in = (i % 4096u) / 64u;
        out = i % 64u;
    } else {
        l = 4;
        in = (i - 4u * 4096u) / 3u;
        out = (i - 4u * 4096u) % 3u;
    }
}

__global__ void k_mlp_pack(const float *w, uint16_t *pack) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= static_cast<uint32_t>(kMlpParams)) return;
    int l;
    uint32_t in, out;
    param_coords(i, l, in, out);
    __nv_bfloat16 h = __float2bfloat16_rn(w[i]);
    uint16_t u = *reinterpret_cast<uint16_t *>(&h);
    pack[pack_offset(l, in, out)] = u;
}

__global__ void k_mlp_adam(float *w, float *m, float *v, const float *g, MlpAdam a, uint16_t *pack) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= static_cast<uint32_t>(kMlpParams)) return;
    float gi = g[i];
    float mi = a.beta1 * m[i] + (1.0f - a.beta1) * gi;
    float vi = a.beta2 * v[i] + (1.0f - a.beta2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    float mh = mi / (1.0f - powf(a.beta1, static_cast<float>(a.step)));
    float vh = vi / (1.0f - powf(a.beta2, static_cast<float>(a.step)));
    float wi = w[i] - a.lr * mh / (sqrtf(vh) + a.eps);
    w[i] = wi;
    int l;
    uint32_t in, out;
    param_coords(i, l, in, out);
    __nv_bfloat16 h = __float2bfloat16_rn(wi);
    uint16_t u = *reinterpret_cast<uint16_t *>(&h);
    pack[pack_offset(l, in, out)] = u;
}

}  // namespace

cudaError_t mlp_pack(const MlpState &s, cudaStream_t st) {
    k_mlp_pack<<<(kMlpParams + 255) / 256, 256, 0, st>>>(s.w, s.pack);
    return cudaGetLastError();
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library).
static cudaError_t encode_fn(PFN_cuTensorMapEncodeTiled_v12000 *out) {
    static std::atomic<PFN_cuTensorMapEncodeTiled_v12000> found{nullptr};
    *out = found.load();
    if (*out) return cudaSuccess;
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q);
    if (e != cudaSuccess) return e;
    if (q != cudaDriverEntryPointSuccess || !fn) return cudaErrorSymbolNotFound;
    *out = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    found.store(*out);
    return cudaSuccess;
}

// The feature matrix (n rows of 64 BF16, 128-byte rows, 16-byte aligned) as a
// TMA tensor map with 128-row x 64-column boxes and the 128-byte swizzle.
static cudaError_t feature_map(const uint16_t *feat, uint32_t n, CUtensorMap *map) {
    PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    cudaError_t e = encode_fn(&encode);
    if (e != cudaSuccess) return e;
    if (reinterpret_cast<uintptr_t>(feat) & 15u) return cudaErrorMisalignedAddress;
    cuuint64_t dims[2] = {64u, n};
    cuuint64_t strides[1] = {128u};
    cuuint32_t box[2] = {64u, static_cast<cuuint32_t>(kTile)};
    cuuint32_t elem[2] = {1u, 1u};
    CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t *>(feat), dims, strides,
                                box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t mlp_infer(const MlpState &s, const uint16_t *feat, uint32_t n, float4 *out, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    cudaError_t e = allow_shared<k_mlp_infer>(kInferSmem);
    if (e != cudaSuccess) return e;
    CUtensorMap map;
    e = feature_map(feat, n, &map);
    if (e != cudaSuccess) return e;
    int sms = 0;
    e = device_sms(&sms);
    if (e != cudaSuccess) return e;
    const uint32_t tiles = (n + kTile - 1) / kTile;
    uint32_t grid = static_cast<uint32_t>(sms);
    const uint32_t need = (tiles + kInferGroups - 1) / kInferGroups;
    if (grid > need) grid = need;
    k_mlp_infer<<<grid, kInferThreads, kInferSmem, st>>>(map, n, reinterpret_cast<const uint4 *>(s.pack), out, s.err);
    return cudaGetLastError();
}

cudaError_t mlp_train_step(const MlpState &s, const uint16_t *feat, const float4 *target, uint32_t n, MlpAdam adam,
                           bool update, cudaStream_t st) {
    cudaError_t e = allow_shared<k_mlp_train>(kTrainSmem);
    if (e != cudaSuccess) return e;
    // The loss follows the gradient: one clear for both.
    e = cudaMemsetAsync(s.grad, 0, kMlpGradBytes, st);
    if (e != cudaSuccess) return e;
    if (n > 0) {
        int sms = 0;
        e = device_sms(&sms);
        if (e != cudaSuccess) return e;
        uint32_t tiles = (n + kTile - 1) / kTile;
        uint32_t grid = static_cast<uint32_t>(sms);
        if (grid > tiles) grid = tiles;
        k_mlp_train<<<grid, kTrainThreads, kTrainSmem, st>>>(feat, target, n, reinterpret_cast<const uint4 *>(s.pack),
                                                   adam.loss_scale, s.grad, s.loss, s.err);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (update) {
        k_mlp_adam<<<(kMlpParams + 255) / 256, 256, 0, st>>>(s.w, s.m, s.v, s.grad, adam, s.pack);
        e = cudaGetLastError();
    }
    return e;
}

}  // namespace vs
