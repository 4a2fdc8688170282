// BF16 GEMM on the 5th-generation tensor cores (tcgen05, FP32 accumulators in tensor memory, operands brought in by
// TMA) for the warm-start MLP's forward and backward passes: C[M][N] (f32) = sum_k A(m, k) B(n, k), each operand
// either K-major (stored [rows][K], K contiguous) or MN-major (stored [K][rows], the M or N index contiguous), with
// row strides for padded storage and an optional split of K into slices summed afterwards in slice order.
//
// Structure (one persistent CTA per SM, 128 x 256 output tiles, 64-wide K blocks):
//   warp 0, one thread -- producer: per K block, waits until its stage of a shared-memory ring is free and
//                         issues the TMA tile loads of A (16 KB) and B (32 KB) into it (128-byte swizzle), counted on
//                         the stage's `full` mbarrier by transaction bytes;
//   warp 1             -- allocates 512 TMEM columns (two 128 x 256 FP32 accumulators); one thread issues, per K
//                         block, four tcgen05.mma (K = 16 each) and commits them to the stage's `empty` mbarrier (the
//                         stage is reusable once the MMAs have read it), and after a tile's last block commits to the
//                         accumulator's `full` mbarrier;
//   the other warps    -- epilogue: wait for an accumulator, read it with tcgen05.ld (each warp the 32 TMEM lanes of
//                         its quadrant, the warps of a quadrant taking its columns in turn), do what the product is
//                         for (store FP32 rows; add a bias and activate; an Adam step), and release the accumulator;
//                         the other accumulator is meanwhile being filled with the next tile.
// Tiles are visited M-fastest, so the CTAs working at the same time share B tiles (the weights) in L2. Every
// mbarrier wait is bounded; a wait that gives up sets *err, the CTA stops issuing work, waits (bounded) for the TMA
// loads and MMAs it started, frees its tensor memory and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <cstdint>
#include <mutex>

#include "../../include/taral_pdhg.h"
#include "mlp.cuh"

namespace taral {
namespace tc {

using mlp::AdamStep;
using mlp::adam_step;
using mlp::bf16;
using mlp::gelu;
constexpr int TM = 128, TK = 64;  // tile rows and K block; the tile's columns TN are a template parameter (256, 128 or 64)
constexpr int kBytesA = TM * TK * 2;
// Shared memory of a CTA: the ring and, per epilogue warp, a chunk of 32 rows of the accumulator (+ alignment slack)
template <class E>
constexpr int smem_bytes(int tn) {
    return E::kStages * (kBytesA + tn * TK * 2) + E::kWarps * 32 * E::kStride * 4 + 1024;
}
constexpr int kSpinLimit = 1 << 24;

// Instruction descriptor of tcgen05.mma kind::f16: F32 accumulate (bits 4-5 = 1), A and B BF16 (bits 7-9, 10-12 =
// 1), A MN-major (bit 15), B MN-major (bit 16), N >> 3 in bits 17-22, M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t idesc(int tn, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u) |
           (uint32_t(tn >> 3) << 17) | (uint32_t(TM >> 4) << 24);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

// Shared-memory descriptor of a tile in the 128-byte swizzle (version 1, layout SWIZZLE_128B = 2). K-major: rows of
// 128 B (64 K elements), 8-row atoms 1024 B apart (stride byte offset), leading byte offset unused (1). MN-major:
// rows of 128 B along M / N (64 elements) for one k, 8-k atoms 1024 B apart (stride byte offset) and 64-element M /
// N atoms `mn_atom` bytes apart (leading byte offset). Offsets in 16-byte units.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr, uint32_t lbo_bytes) {
    return uint64_t((saddr >> 4) & 0x3FFF) | (uint64_t((lbo_bytes >> 4) & 0x3FFF) << 16) |
           (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61);
}

__device__ __forceinline__ bool wait_parity(uint32_t bar, uint32_t parity) {
    for (int i = 0; i < kSpinLimit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

struct GemmShape {
    int M, N, K;
    int m_tiles, n_tiles, slices, kb_per_slice, kb_total;
    int a_mn, b_mn;
};

// Epilogues: what becomes of a warp's chunk of the product, 32 rows x kCols columns staged in shared memory with row
// stride kStride. rows(chunk, row0, col0, M, N, slice): the chunk starts at row row0 and column col0 of the product.
struct EpiTile {  // C, or with K slices the partial of slice s at C + s * M * ldc
    static constexpr int kStages = 4, kWarps = 8, kCtas = 1, kCols = 32, kStride = 33;
    float* C;
    int ldc;
    __device__ __forceinline__ void rows(const float* chunk, int lane, int row0, int col0, int M, int N, int slice) const {
        float* out = C + size_t(slice) * size_t(M) * ldc;
        const int col = col0 + lane;  // a lane per column: every store is 32 consecutive floats of a row
        if (col >= N) return;
#pragma unroll 8
        for (int i = 0; i < 32; ++i)
            if (row0 + i < M) out[size_t(row0 + i) * ldc + col] = chunk[i * 33 + lane];
    }
};
// A layer's output: Z = C + b and, for a hidden layer, H = bf16(gelu(Z)) (the last layer: H NULL).
struct EpiLayer {
    static constexpr int kStages = 4, kWarps = 8, kCtas = 1, kCols = 32, kStride = 33;
    const float* b;
    float* Z;
    bf16* H;
    int ld;
    __device__ __forceinline__ void rows(const float* chunk, int lane, int row0, int col0, int M, int N, int) const {
        const int col = col0 + lane;
        if (col >= N) return;
        const float bc = b[col];
#pragma unroll 4
        for (int i = 0; i < 32; ++i)
            if (row0 + i < M) {
                const float z = chunk[i * 33 + lane] + bc;
                const size_t at = size_t(row0 + i) * ld + col;
                Z[at] = z;
                if (H) H[at] = __float2bfloat16(gelu(z));
            }
    }
};
// A weight gradient consumed where it is formed: Adam on the FP32 masters W with the moments m, v (all three in the blocked
// layout of mlp.cuh, with `groups` column groups), and the bf16 copy Wb (row stride ldb, a multiple of 16). What bounds it
// is memory: 26 bytes a weight (masters and moments read and written, the copy written); storing the gradient and reading
// it back would add 8. Row-major masters, whose tile rows are 1 KB pieces 528 KB apart, took 570 us on 68M weights
// (3.1 TB/s) whatever the loads in flight.
struct EpiAdam {
    static constexpr int kStages = 2, kWarps = 16, kCtas = 2, kCols = 16, kStride = 0;  // straight from registers
    float *W, *m, *v;
    bf16* Wb;
    int groups, ldb;
    AdamStep s;
    // row: this lane's row of the product, g: its 16 gradients from column col0
    __device__ __forceinline__ void row(const uint32_t (&g)[16], int r, int col0, int M) const {
        if (r >= M || col0 >= 16 * groups) return;
        const size_t at = mlp::blocked_at(r, col0, groups);
        uint32_t out[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float4 w = __ldcs(reinterpret_cast<const float4*>(W + at + 128 * k)), a = __ldcs(reinterpret_cast<const float4*>(m + at + 128 * k)),
                   q = __ldcs(reinterpret_cast<const float4*>(v + at + 128 * k));
            adam_step(s, __uint_as_float(g[4 * k]), w.x, a.x, q.x), adam_step(s, __uint_as_float(g[4 * k + 1]), w.y, a.y, q.y);
            adam_step(s, __uint_as_float(g[4 * k + 2]), w.z, a.z, q.z), adam_step(s, __uint_as_float(g[4 * k + 3]), w.w, a.w, q.w);
            __stcs(reinterpret_cast<float4*>(W + at + 128 * k), w), __stcs(reinterpret_cast<float4*>(m + at + 128 * k), a);
            __stcs(reinterpret_cast<float4*>(v + at + 128 * k), q);
            const __nv_bfloat162 lo = __floats2bfloat162_rn(w.x, w.y), hi = __floats2bfloat162_rn(w.z, w.w);
            out[2 * k] = reinterpret_cast<const uint32_t&>(lo), out[2 * k + 1] = reinterpret_cast<const uint32_t&>(hi);
        }
        uint4* to = reinterpret_cast<uint4*>(Wb + size_t(r) * ldb + col0);  // a whole 32-byte sector at once
        to[0] = make_uint4(out[0], out[1], out[2], out[3]), to[1] = make_uint4(out[4], out[5], out[6], out[7]);
    }
};

// The product A B^T of every (m tile, n tile, K slice) work item into the epilogue.
template <class E, int TN>
__global__ void __launch_bounds__(64 + 32 * E::kWarps, E::kCtas) k_umma_gemm(const __grid_constant__ CUtensorMap mapA,
                                                                      const __grid_constant__ CUtensorMap mapB, GemmShape g,
                                                                      const E epi, int* err) {
    constexpr int kStages = E::kStages, kBytesB = TN * TK * 2, kStageBytes = kBytesA + kBytesB;
    constexpr uint32_t kTmemCols = 2 * TN;  // two accumulators
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2], drain;
    __shared__ uint32_t tmem_sh;
    __shared__ int failed;
    const uint32_t s0 = smem_u32(smem_raw), pad = (1024u - (s0 & 1023u)) & 1023u;
    const uint32_t ring = s0 + pad;  // 1024-byte aligned: the swizzle pattern is a function of the address bits
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int items = g.m_tiles * g.n_tiles * g.slices;

    if (tid == 0) {
        failed = 0;
        for (int s = 0; s < kStages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[s])));
        }
        for (int a = 0; a < 2; ++a) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&acc_full[a])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&acc_empty[a])), "r"(32 * E::kWarps));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&drain)));
        asm volatile("fence.mbarrier_init.release.cluster;");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mapA)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mapB)) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_sh;
    auto stopped = [&] { return *reinterpret_cast<volatile int*>(&failed) != 0; };  // set by another role's thread

    auto item_coords = [&](int item, int& m0, int& n0, int& kb0, int& kb1, int& slice) {
        const int mt = item % g.m_tiles, rest = item / g.m_tiles;
        slice = rest % g.slices;
        m0 = mt * TM, n0 = (rest / g.slices) * TN;
        kb0 = slice * g.kb_per_slice;
        kb1 = min(kb0 + g.kb_per_slice, g.kb_total);
    };

    if (warp == 0) {
        if (lane == 0) {  // producer
            uint32_t it = 0;
            for (int item = blockIdx.x; item < items && !stopped(); item += gridDim.x) {
                int m0, n0, kb0, kb1, slice;
                item_coords(item, m0, n0, kb0, kb1, slice);
                for (int kb = kb0; kb < kb1; ++kb, ++it) {
                    const uint32_t s = it % kStages, use = it / kStages;
                    if (use > 0 && !wait_parity(smem_u32(&empty[s]), (use - 1) & 1)) {
                        atomicOr(&failed, 1);
                        break;
                    }
                    const uint32_t fb = smem_u32(&full[s]), a = ring + s * kStageBytes, b = a + kBytesA;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb),
                                 "r"(uint32_t(kStageBytes))
                                 : "memory");
                    const int k0 = kb * TK;
                    if (g.a_mn) {  // [K][M] storage: two boxes of 64 M x 64 K
                        tma_load(a, &mapA, m0, k0, fb);
                        tma_load(a + 8192, &mapA, m0 + 64, k0, fb);
                    } else {  // [M][K] storage: one box of 64 K x 128 M
                        tma_load(a, &mapA, k0, m0, fb);
                    }
                    if (g.b_mn) {  // [K][N]: boxes of 64 N x 64 K
                        for (int j = 0; j < TN / 64; ++j) tma_load(b + 8192 * j, &mapB, n0 + 64 * j, k0, fb);
                    } else {  // [N][K]: one box of 64 K x TN
                        tma_load(b, &mapB, k0, n0, fb);
                    }
                }
            }
            // drain: every stage this thread filled has been consumed or its loads have landed before exit
            const uint32_t issued = it;
            for (uint32_t q = issued > kStages ? issued - kStages : 0; q < issued; ++q)
                wait_parity(smem_u32(&full[q % kStages]), (q / kStages) & 1);
        }
    } else if (warp == 1) {
        if (lane == 0) {  // MMA issuer
            const uint32_t id = idesc(TN, g.a_mn != 0, g.b_mn != 0);
            const uint32_t lbo_a = g.a_mn ? 8192u : 16u, lbo_b = g.b_mn ? 8192u : 16u;
            const uint32_t kstep_a = g.a_mn ? 2048u : 32u, kstep_b = g.b_mn ? 2048u : 32u;  // 16 K elements
            uint32_t it = 0, tile = 0;
            bool ok = true;
            for (int item = blockIdx.x; item < items && ok && !stopped(); item += gridDim.x, ++tile) {
                int m0, n0, kb0, kb1, slice;
                item_coords(item, m0, n0, kb0, kb1, slice);
                const uint32_t acc = tile & 1, use = tile >> 1;
                if (use > 0 && !wait_parity(smem_u32(&acc_empty[acc]), (use - 1) & 1)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
                const uint32_t d = tmem + acc * TN;
                for (int kb = kb0; kb < kb1; ++kb, ++it) {
                    const uint32_t s = it % kStages;
                    if (!wait_parity(smem_u32(&full[s]), (it / kStages) & 1)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    const uint32_t a = ring + s * kStageBytes, b = a + kBytesA;
#pragma unroll
                    for (int ks = 0; ks < TK / 16; ++ks) {
                        const uint64_t ad = sw128_desc(a + ks * kstep_a, lbo_a), bd = sw128_desc(b + ks * kstep_b, lbo_b);
                        const uint32_t accumulate = (kb > kb0 || ks > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
                            "l"(ad), "l"(bd), "r"(id), "r"(accumulate));
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                     smem_u32(&empty[s]))
                                 : "memory");
                }
                if (!ok) break;
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(&acc_full[acc]))
                             : "memory");
            }
            if (!ok) atomicOr(&failed, 1);
            // every MMA this thread issued has completed before the tensor memory is freed
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&drain))
                         : "memory");
            if (!wait_parity(smem_u32(&drain), 0)) atomicOr(&failed, 1);
        }
    } else {  // epilogue, warps from 2: TMEM lanes 32 (warp % 4) .. + 31, every (kWarps / 4)-th chunk of 32 columns
        const int q = warp & 3, part = (warp - 2) / 4;
        uint32_t tile = 0;
        for (int item = blockIdx.x; item < items; item += gridDim.x, ++tile) {
            int m0, n0, kb0, kb1, slice;
            item_coords(item, m0, n0, kb0, kb1, slice);
            const uint32_t acc = tile & 1, use = tile >> 1;
            if (stopped() || !wait_parity(smem_u32(&acc_full[acc]), use & 1)) {
                atomicOr(&failed, 1);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            // lane l holds row (m0 + 32 q + l) of each chunk of columns; unless the epilogue takes it from there, the chunk
            // goes through this warp's tile in shared memory, for accesses to consecutive elements of a row
            float* tile_sm = reinterpret_cast<float*>(smem_raw + pad + kStages * kStageBytes) + (warp - 2) * 32 * E::kStride;
#pragma unroll 1
            for (int cb = part; cb < TN / E::kCols; cb += E::kWarps / 4) {
                uint32_t r[E::kCols];
                const uint32_t taddr = tmem + (uint32_t(q * 32) << 16) + acc * TN + uint32_t(cb * E::kCols);
                if constexpr (E::kCols == 32) {
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                          "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                          "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
                          "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                        : "r"(taddr));
                } else {
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                          "=r"(r[15])
                        : "r"(taddr));
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if constexpr (E::kStride == 0) {
                    epi.row(r, m0 + q * 32 + lane, n0 + cb * E::kCols, g.M);
                } else {
#pragma unroll
                    for (int i = 0; i < E::kCols; ++i) tile_sm[lane * E::kStride + i] = __uint_as_float(r[i]);  // banks (lane + i) % 32
                    __syncwarp();
                    epi.rows(tile_sm, lane, m0 + q * 32, n0 + cb * E::kCols, g.M, g.N, slice);
                    __syncwarp();
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[acc])) : "memory");
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 1) {
        __syncwarp();  // the warp converged for the .sync.aligned dealloc
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
    }
    if (tid == 0 && failed) atomicExch(err, 1);
}

// Sum of the slice partials in slice order (deterministic): C[r][c] = sum_s ws[s][r][c].
__global__ void k_sum_slices(int M, int N, int ldc, int slices, const float* __restrict__ ws, float* __restrict__ C) {
    const size_t total = size_t(M) * N;
    for (size_t e = size_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += size_t(gridDim.x) * blockDim.x) {
        const size_t r = e / size_t(N), c = e % size_t(N), at = r * size_t(ldc) + c;
        float s = 0.f;
        for (int q = 0; q < slices; ++q) s += ws[size_t(q) * size_t(M) * ldc + at];
        C[at] = s;
    }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link-time dependency on the driver library).
static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// A bf16 matrix stored row-major [rows][ld] (cols <= ld used), read in boxes of 64 columns x box_rows rows with the
// 128-byte swizzle; out-of-range elements read as zero.
static bool make_map(CUtensorMap* m, const void* base, int rows, int cols, int ld, int box_rows) {
    const auto fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {cuuint64_t(cols), cuuint64_t(rows)};
    const cuuint64_t strides[1] = {cuuint64_t(ld) * 2};
    const cuuint32_t box[2] = {64u, cuuint32_t(box_rows)};
    const cuuint32_t estr[2] = {1u, 1u};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Checks, tensor maps and launch of sum_k A(m, k) B(n, k) into `epi`. a_mn = 0: A stored [M][lda] (K contiguous); 1:
// [K][lda] (M contiguous); likewise b_mn for B with N. lda, ldb multiples of 8 (16-byte rows), A and B 16-byte aligned.
// *slices: K slices asked for in, used out. err: device int set to 1 when a completion wait gave up (the result is then
// undefined).
template <class E, int TN>
static int launch_tiles(int M, int N, int K, const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, const E& epi,
                       int* slices, int* err, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || K <= 0 || !A || !B || !err) return TARAL_ERR_INPUT;
    if (lda % 8 || ldb % 8 || lda < (a_mn ? M : K) || ldb < (b_mn ? N : K)) return TARAL_ERR_INPUT;
    if (reinterpret_cast<uintptr_t>(A) % 16 || reinterpret_cast<uintptr_t>(B) % 16) return TARAL_ERR_INPUT;
    CUtensorMap ma, mb;
    const bool okA = a_mn ? make_map(&ma, A, K, M, lda, 64) : make_map(&ma, A, M, K, lda, TM);
    const bool okB = b_mn ? make_map(&mb, B, K, N, ldb, 64) : make_map(&mb, B, N, K, ldb, TN);
    if (!okA || !okB) return TARAL_ERR_CUDA;
    constexpr int smem = smem_bytes<E>(TN);
    static_assert(E::kCtas * (smem + 1024) <= 228 * 1024 && E::kCtas * 2 * TN <= 512, "shared and tensor memory of an SM");
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TARAL_ERR_CUDA;
    {  // the shared-memory opt-in is a per-device attribute of the kernel: set once on every device used
        static std::mutex mu;
        static bool configured[64] = {};
        std::lock_guard<std::mutex> lock(mu);
        if (!configured[dev]) {
            if (cudaFuncSetAttribute(k_umma_gemm<E, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
                return TARAL_ERR_CUDA;
            configured[dev] = true;
        }
    }
    GemmShape g;
    g.M = M, g.N = N, g.K = K, g.a_mn = a_mn, g.b_mn = b_mn;
    g.m_tiles = (M + TM - 1) / TM, g.n_tiles = (N + TN - 1) / TN;
    g.kb_total = (K + TK - 1) / TK;
    const int ask = *slices < 1 ? 1 : *slices > g.kb_total ? g.kb_total : *slices;
    g.kb_per_slice = (g.kb_total + ask - 1) / ask;
    g.slices = *slices = (g.kb_total + g.kb_per_slice - 1) / g.kb_per_slice;  // every slice holds at least one K block
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int items = g.m_tiles * g.n_tiles * g.slices;
    sms *= E::kCtas;
    k_umma_gemm<E, TN><<<items < sms ? items : sms, 64 + 32 * E::kWarps, smem, stream>>>(ma, mb, g, epi, err);
    return cudaGetLastError() == cudaSuccess ? TARAL_OK : TARAL_ERR_CUDA;
}

// 256 columns a tile, or 64 where that leaves most of the GPU idle: with fewer than a quarter of the SMs at work a product
// lasts as long as one tile's epilogue, which 64 columns cut to a quarter (512 x 512 weights, 64 rows: layer 19.9 -> 9.7
// us, Adam 29.4 -> 10.9 us).
template <class E>
static int launch_gemm(int M, int N, int K, const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, const E& epi,
                       int* slices, int* err, cudaStream_t stream) {
    const int64_t items = int64_t((M + TM - 1) / TM) * ((N + 255) / 256) * (*slices < 1 ? 1 : *slices);
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (items <= sms / 4) return launch_tiles<E, 64>(M, N, K, A, lda, a_mn, B, ldb, b_mn, epi, slices, err, stream);
    return launch_tiles<E, 256 / E::kCtas>(M, N, K, A, lda, a_mn, B, ldb, b_mn, epi, slices, err, stream);
}

// C[M][N] (row stride ldc) = sum_k A(m, k) B(n, k), operands as for launch_gemm. slices > 1: K split into that many
// slices whose partials go to ws (slices * M * ldc floats) and are summed in order into C.
int gemm_umma(int M, int N, int K, const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, float* C,
              int ldc, int slices, float* ws, int* err, cudaStream_t stream) {
    if (!C || ldc < N || (slices > 1 && !ws)) return TARAL_ERR_INPUT;
    const int kb = (K + TK - 1) / TK;
    const bool split = slices > 1 && kb > 1;
    int used = slices;
    const int rc = launch_gemm(M, N, K, A, lda, a_mn, B, ldb, b_mn, EpiTile{split ? ws : C, ldc}, &used, err, stream);
    if (rc != TARAL_OK || !split) return rc;
    k_sum_slices<<<592, 256, 0, stream>>>(M, N, ldc, used, ws, C);
    return cudaGetLastError() == cudaSuccess ? TARAL_OK : TARAL_ERR_CUDA;
}

// The partials alone (see gemm_umma): *slices slices asked for in, written out; a single slice is the product itself.
int gemm_partials(int M, int N, int K, const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, float* ws,
                  int* slices, int* err, cudaStream_t stream) {
    return launch_gemm(M, N, K, A, lda, a_mn, B, ldb, b_mn, EpiTile{ws, N}, slices, err, stream);
}

// Z (M x N) = A W + b with A [M][K] and W [K][ldw], and H = bf16(gelu(Z)) unless H is NULL.
int gemm_layer(int M, int N, int K, const void* A, const void* W, int ldw, const float* b, float* Z, bf16* H, int* err,
               cudaStream_t stream) {
    int one = 1;
    return launch_gemm(M, N, K, A, K, 0, W, ldw, 1, EpiLayer{b, Z, H, N}, &one, err, stream);
}

// Adam on W (M x N; W, m and v blocked, the copy Wb with row stride ldw) with the gradient sum_k A(k, m) B(k, n), both
// operands stored [K][..].
int gemm_adam(int M, int N, int K, const void* A, int lda, const void* B, int ldb, float* W, float* m, float* v, bf16* Wb,
              int ldw, const AdamStep& s, int* err, cudaStream_t stream) {
    int one = 1;
    if (ldw % 16) return TARAL_ERR_INPUT;
    return launch_gemm(M, N, K, A, lda, 1, B, ldb, 1, EpiAdam{W, m, v, Wb, mlp::blocked_groups(N), ldw, s}, &one, err, stream);
}

int gemm_tc(int M, int N, int K, const void* A, const void* Bt, float* C, int* err, cudaStream_t stream) {
    if (K % 8) return TARAL_ERR_INPUT;
    return gemm_umma(M, N, K, A, K, 0, Bt, K, 0, C, N, 1, nullptr, err, stream);
}

}  // namespace tc
}  // namespace taral

// C (M x N, f32) = A (M x K, bf16, row-major) * Bt (N x K, bf16, row-major)^T on the tcgen05 tensor cores.
// K must be a multiple of 8 and A, Bt 16-byte aligned. err: device int, set to 1 when an MMA completion wait gave
// up (the result is then undefined).
extern "C" int taral_gemm_bf16_tc(int M, int N, int K, const void* A, const void* Bt, float* C, int* err,
                                  void* stream) {
    return taral::tc::gemm_tc(M, N, K, A, Bt, C, err, static_cast<cudaStream_t>(stream));
}

// The general form: operand layouts, row strides and split-K (see gemm_umma).
extern "C" int taral_gemm_bf16_umma(int M, int N, int K, const void* A, int lda, int a_mn, const void* B, int ldb,
                                    int b_mn, float* C, int ldc, int slices, float* ws, int* err, void* stream) {
    return taral::tc::gemm_umma(M, N, K, A, lda, a_mn, B, ldb, b_mn, C, ldc, slices, ws, err,
                                static_cast<cudaStream_t>(stream));
}
