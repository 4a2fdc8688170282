// Learned warm start: a small MLP (in -> hidden x depth, GELU -> out) trained and evaluated on the GPU with this
// file's own BF16 tensor-core kernels (include/taral_pdhg.h, part 7). It maps a scenario's 256-dim price/capacity
// perturbation to an initial (x, y) for the PDHG solve. No counterpart in the reference.
//
// Layout: weights W_l bf16 [in_l][out_l] row-major (with FP32 master copies and Adam moments), biases FP32.
// Forward per layer: C = H_{l-1} W_l (GEMM, FP32 accumulate), Z = C + b, H = bf16(gelu(Z)) (last layer: Y = Z).
// Backward: dW = H_{l-1}^T dZ, db = sum_b dZ, dH_{l-1} = dZ W_l^T, dZ = dH * gelu'(Z); loss = mean (Y - T)^2.
//
// GEMMs: for every layer whose input width is a multiple of 8 (and whose dZ rows are 16-byte multiples: the output
// gradient of the last layer is stored with its row stride rounded up to 8) all three GEMMs run on the tcgen05 tensor
// cores through TMA (mlp_tc.cu) from one bf16 copy of W, its rows padded to 8 elements: the forward C = H W (W read
// MN-major) with bias and activation in its epilogue, dH_prev = dZ W^T (W K-major, K split into slices summed in
// order) and dW = H_prev^T dZ (both operands MN-major), which in training ends in the Adam step itself, so that the
// weight gradient never reaches memory. Any other layer uses mma.sync m16n8k16 (bf16 x bf16 -> f32), 128 x 128 x 32 CTA
// tiles, 8 warps of 64 x 32, operands staged in shared memory and fed with ldmatrix; A may be stored transposed (TA:
// A = X^T) and B as [N][K] (TB: B = W^T); split-K writes per-slice partials that a second kernel adds in slice order
// (deterministic).
//
// A training step at 64 x 132,001 outputs (68M weights) took 1.5 ms with separate kernels for the transposed copy, the
// gathered targets, the residual, the column sums, the weight gradients and Adam, and a host synchronisation per step;
// what bounds it is the 26 bytes per weight of Adam plus two reads of the bf16 copy.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <random>
#include <string>
#include <vector>

#include "../../include/taral_pdhg.h"
#include "mlp.cuh"
#include "staging.hpp"

namespace taral {
namespace tc {
using mlp::AdamStep;
using mlp::bf16;
int gemm_partials(int M, int N, int K, const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, float* ws,
                  int* slices, int* err, cudaStream_t stream);
int gemm_layer(int M, int N, int K, const void* A, const void* W, int ldw, const float* b, float* Z, bf16* H, int* err,
               cudaStream_t stream);
int gemm_adam(int M, int N, int K, const void* A, int lda, const void* B, int ldb, float* W, float* m, float* v, bf16* Wb,
              int ldw, const AdamStep& s, int* err, cudaStream_t stream);
int gemm_umma(int M, int N, int K, const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, float* C,
              int ldc, int slices, float* ws, int* err, cudaStream_t stream);
}
namespace mlp {

struct MlpError {
    std::string msg;
};
#define MK(call)                                                                                          \
    do {                                                                                                  \
        cudaError_t e_ = (call);                                                                          \
        if (e_ != cudaSuccess) throw MlpError{std::string(#call) + ": " + cudaGetErrorString(e_)};      \
    } while (0)

constexpr int BM = 128, BN = 128, BK = 32, PAD = 8;

__device__ __forceinline__ void ldsm_x4(const bf16* p, uint32_t (&r)[4]) {
    uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// C[z][M][N] = sum over k in slice z of op(A)[m][k] op(B)[k][n].
//   TA = false: A stored [M][K];  TA = true: A stored [K][M] (op(A) = stored^T).
//   TB = false: B stored [K][N];  TB = true: B stored [N][K].
// VEC: every dimension is a multiple of 8 and the pointers are 16-byte aligned (8-element vector loads).
template <bool TA, bool TB, bool VEC>
__global__ void __launch_bounds__(256) k_gemm(int M, int N, int K, int kslice, const bf16* __restrict__ A,
                                              const bf16* __restrict__ B, float* __restrict__ C) {
    __shared__ __align__(16) bf16 As[BM][BK + PAD];
    __shared__ __align__(16) bf16 Bs[BN][BK + PAD];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wm = warp >> 2, wn = warp & 3;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int kb = blockIdx.z * kslice, ke = min(K, kb + kslice);
    float acc[4][4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
    const bf16 zero = __float2bfloat16(0.f);
    for (int k0 = kb; k0 < ke; k0 += BK) {
        // ---- A tile: As[m][k]
        for (int v = tid; v < BM * BK / 8; v += 256) {
            if (!TA) {
                const int r = v / (BK / 8), c8 = (v % (BK / 8)) * 8, gm = m0 + r, gk = k0 + c8;
                if (VEC && gm < M && gk + 8 <= ke) {
                    *reinterpret_cast<uint4*>(&As[r][c8]) = *reinterpret_cast<const uint4*>(A + size_t(gm) * K + gk);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) As[r][c8 + e] = (gm < M && gk + e < ke) ? A[size_t(gm) * K + gk + e] : zero;
                }
            } else {
                const int kk = v / (BM / 8), m8 = (v % (BM / 8)) * 8, gk = k0 + kk, gm = m0 + m8;
                if (VEC && gk < ke && gm + 8 <= M) {
                    uint4 q = *reinterpret_cast<const uint4*>(A + size_t(gk) * M + gm);
                    const bf16* e8 = reinterpret_cast<const bf16*>(&q);
#pragma unroll
                    for (int e = 0; e < 8; ++e) As[m8 + e][kk] = e8[e];
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) As[m8 + e][kk] = (gk < ke && gm + e < M) ? A[size_t(gk) * M + gm + e] : zero;
                }
            }
        }
        // ---- B tile: Bs[n][k]
        for (int v = tid; v < BN * BK / 8; v += 256) {
            if (TB) {
                const int r = v / (BK / 8), c8 = (v % (BK / 8)) * 8, gn = n0 + r, gk = k0 + c8;
                if (VEC && gn < N && gk + 8 <= ke) {
                    *reinterpret_cast<uint4*>(&Bs[r][c8]) = *reinterpret_cast<const uint4*>(B + size_t(gn) * K + gk);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) Bs[r][c8 + e] = (gn < N && gk + e < ke) ? B[size_t(gn) * K + gk + e] : zero;
                }
            } else {
                const int kk = v / (BN / 8), n8 = (v % (BN / 8)) * 8, gk = k0 + kk, gn = n0 + n8;
                if (VEC && gk < ke && gn + 8 <= N) {
                    uint4 q = *reinterpret_cast<const uint4*>(B + size_t(gk) * N + gn);
                    const bf16* e8 = reinterpret_cast<const bf16*>(&q);
#pragma unroll
                    for (int e = 0; e < 8; ++e) Bs[n8 + e][kk] = e8[e];
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) Bs[n8 + e][kk] = (gk < ke && gn + e < N) ? B[size_t(gk) * N + gn + e] : zero;
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int ks = 0; ks < BK; ks += 16) {
            uint32_t a[4][4], b[4][2];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) ldsm_x4(&As[wm * 64 + mi * 16 + (lane & 15)][ks + (lane >> 4) * 8], a[mi]);
#pragma unroll
            for (int nj = 0; nj < 2; ++nj) {
                uint32_t r[4];
                ldsm_x4(&Bs[wn * 32 + nj * 16 + (lane & 7) + (lane >> 4) * 8][ks + ((lane >> 3) & 1) * 8], r);
                b[2 * nj][0] = r[0], b[2 * nj][1] = r[1], b[2 * nj + 1][0] = r[2], b[2 * nj + 1][1] = r[3];
            }
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) mma_bf16(acc[mi][ni], a[mi], b[ni]);
        }
        __syncthreads();
    }
    float* Cz = C + size_t(blockIdx.z) * M * N;
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
            const int row = m0 + wm * 64 + mi * 16 + (lane >> 2), col = n0 + wn * 32 + ni * 8 + (lane & 3) * 2;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int rr = row + 8 * h;
                if (rr < M) {
                    if (col < N) Cz[size_t(rr) * N + col] = acc[mi][ni][2 * h];
                    if (col + 1 < N) Cz[size_t(rr) * N + col + 1] = acc[mi][ni][2 * h + 1];
                }
            }
        }
}

// C = sum over slices s of P[s] (fixed order).
__global__ void k_splitk_sum(size_t count, int slices, const float* __restrict__ P, float* __restrict__ C) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < count; i += size_t(gridDim.x) * blockDim.x) {
        float s = 0.f;
        for (int z = 0; z < slices; ++z) s += P[size_t(z) * count + i];
        C[i] = s;
    }
}

// Z = C + b; H = bf16(gelu(Z)) (act) or Y = Z (no act, H may be NULL).
__global__ void k_bias_act(int rows, int cols, const float* __restrict__ C, const float* __restrict__ b,
                           float* __restrict__ Z, bf16* __restrict__ H, int act) {
    const size_t n = size_t(rows) * cols;
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        const float z = C[i] + b[i % cols];
        Z[i] = z;
        if (H) H[i] = __float2bfloat16(act ? gelu(z) : z);
    }
}

// A bias vector's Adam step, taken where its gradient is formed (b NULL: the gradient only).
struct BiasStep {
    float *b, *m, *v;
    AdamStep s;
};
__device__ __forceinline__ void bias_step(const BiasStep& t, int j, float g, float* db) {
    db[j] = g;
    if (t.b) adam_step(t.s, g, t.b[j], t.m[j], t.v[j]);
}

// A CTA takes COLS columns: threads (x, y) = (column, row modulo blockDim / COLS), rows in chunks of kRowChunk. grad(r)
// is the gradient at row r of the thread's column, formed by the thread that owns the entry; the columns are then summed
// in row order by one thread each from shared memory (column_smem bytes), as a loop over the rows would, without reading
// the gradients back from memory.
constexpr int kRowChunk = 256;
constexpr int kLossCols = 32, kHiddenCols = 16;
inline size_t column_smem(int rows, int cols) { return size_t(std::min(rows, kRowChunk)) * size_t(cols + 1) * sizeof(float); }
template <int COLS, class Grad>
__device__ __forceinline__ float column_sums(int rows, bool in, float* sh, Grad grad) {
    const int tx = threadIdx.x % COLS, ty = threadIdx.x / COLS, step = blockDim.x / COLS;
    float sum = 0.f;
    for (int r0 = 0; r0 < rows; r0 += kRowChunk) {
        const int n = min(kRowChunk, rows - r0);
        if (in) {
#pragma unroll 4
            for (int r = ty; r < n; r += step) sh[r * (COLS + 1) + tx] = grad(r0 + r);
        }
        __syncthreads();
        if (ty == 0 && in) {
#pragma unroll 8
            for (int r = 0; r < n; ++r) sum += sh[r * (COLS + 1) + tx];
        }
        __syncthreads();
    }
    return sum;  // in the threads with y = 0
}

// The output gradient: with r = Y - T, G = 2 r / (rows cols): dY = bf16(G), db = column sums of G, and the CTA's sum of
// r^2 in part[CTA]. idx: the row of T that belongs to row r (NULL: r itself).
__global__ void __launch_bounds__(256) k_loss_grad(int rows, int cols, int ldy, const float* __restrict__ Y,
                                                   const float* __restrict__ T, const int* __restrict__ idx,
                                                   bf16* __restrict__ dY, float* __restrict__ db, BiasStep bias,
                                                   double* __restrict__ part) {
    extern __shared__ float sh[];
    __shared__ double warps[8];
    const int j = blockIdx.x * kLossCols + threadIdx.x % kLossCols;
    const float scale = 2.f / (float(rows) * float(cols));
    double s = 0;
    const float g = column_sums<kLossCols>(rows, j < cols, sh, [&](int r) {
        const size_t t = size_t(idx ? __ldg(idx + r) : r) * cols + j;
        const float e = __ldg(Y + size_t(r) * cols + j) - __ldg(T + t);
        dY[size_t(r) * ldy + j] = __float2bfloat16(e * scale);  // row stride ldy >= cols (padded for TMA)
        s += double(e) * double(e);
        return e * scale;
    });
    if (threadIdx.x < kLossCols && j < cols) bias_step(bias, j, g, db);
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int w = 0; w < 8; ++w) t += warps[w];
        part[blockIdx.x] = t;
    }
}

// A hidden layer's gradient: dH = the sum of the slices of P in order, dZ = bf16(dH gelu'(Z)), db = column sums of
// dH gelu'(Z). 1,024 threads on 16 columns: with 64 rows every thread has one entry, whose slices (74 behind the output
// layer) are its whole latency.
__global__ void __launch_bounds__(1024) k_hidden_grad(int rows, int cols, int slices, const float* __restrict__ P,
                                                      const float* __restrict__ Z, bf16* __restrict__ dZ,
                                                      float* __restrict__ db, BiasStep bias) {
    extern __shared__ float sh[];
    const int j = blockIdx.x * kHiddenCols + threadIdx.x % kHiddenCols;
    const size_t count = size_t(rows) * cols;
    const float g = column_sums<kHiddenCols>(rows, j < cols, sh, [&](int r) {
        const size_t at = size_t(r) * cols + j;
        const float z0 = __ldg(Z + at);
        float d = 0.f;
        int z = 0;
        for (; z + 16 <= slices; z += 16) {
            float p[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) p[e] = __ldg(P + size_t(z + e) * count + at);
#pragma unroll
            for (int e = 0; e < 16; ++e) d += p[e];
        }
#pragma unroll 8
        for (; z < slices; ++z) d += __ldg(P + size_t(z) * count + at);
        const float e = d * gelu_grad(z0);
        dZ[at] = __float2bfloat16(e);
        return e;
    });
    if (threadIdx.x < kHiddenCols && j < cols) bias_step(bias, j, g, db);
}


__global__ void k_to_bf16(size_t n, const float* __restrict__ src, bf16* __restrict__ dst) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        dst[i] = __float2bfloat16(src[i]);
}

// Adam on row-major FP32 masters with a stored gradient, for a layer whose dW runs on mma.sync; refreshes the bf16 copy
// (row stride ldb).
__global__ void k_adam(int rows, int cols, int ldb, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, bf16* __restrict__ wb, AdamStep s) {
    for (int r = blockIdx.y; r < rows; r += gridDim.y)
        for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < cols; j += gridDim.x * blockDim.x) {
            const size_t at = size_t(r) * cols + j;
            adam_step(s, g[at], w[at], m[at], v[at]);
            wb[size_t(r) * ldb + j] = __float2bfloat16(w[at]);
        }
}

// Row-major P (rows x cols) into the masters W (blocked or row-major) and their bf16 copy, and back.
__global__ void k_set_weights(int rows, int cols, int groups, int ldb, const float* __restrict__ P, float* __restrict__ W,
                              bf16* __restrict__ wb) {
    for (int r = blockIdx.y; r < rows; r += gridDim.y)
        for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < cols; j += gridDim.x * blockDim.x) {
            const float w = P[size_t(r) * cols + j];
            W[groups ? blocked_at(r, j, groups) : size_t(r) * cols + j] = w;
            wb[size_t(r) * ldb + j] = __float2bfloat16(w);
        }
}
__global__ void k_get_weights(int rows, int cols, int groups, const float* __restrict__ W, float* __restrict__ P) {
    for (int r = blockIdx.y; r < rows; r += gridDim.y)
        for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < cols; j += gridDim.x * blockDim.x)
            P[size_t(r) * cols + j] = W[blocked_at(r, j, groups)];
}

// The dataset rows idx[0 .. rows) as bf16 operand rows.
__global__ void k_gather_rows(int cols, const int* __restrict__ idx, const float* __restrict__ src, bf16* __restrict__ dst) {
    const float* from = src + size_t(idx[blockIdx.x]) * cols;
    for (int c = threadIdx.x; c < cols; c += blockDim.x) dst[size_t(blockIdx.x) * cols + c] = __float2bfloat16(from[c]);
}

static int grid1(size_t n) { return int(std::max<size_t>(1, std::min<size_t>((n + 255) / 256, 148 * 16))); }

struct Layer {
    int in = 0, out = 0;
    float *W = nullptr, *b = nullptr, *gW = nullptr, *gb = nullptr, *mW = nullptr, *vW = nullptr, *mb = nullptr,
          *vb = nullptr;
    bf16* Wb = nullptr;   // W as bf16
    int ldw = 0;          // row stride of Wb
    bool tc = false;      // the GEMMs run on tcgen05 (ldw is out rounded up to 16), else on mma.sync (ldw = out)
    bool fused = false;   // Adam in the epilogue of dW: W, mW, vW blocked (mlp.cuh), else row-major
    float* Z = nullptr;  // pre-activation [batch][out]
    bf16* H = nullptr;   // activation [batch][out] (GEMM operand of the next layer)
};

struct Mlp {
    int in_dim = 0, hidden = 0, depth = 0, out_dim = 0, max_batch = 0;
    std::vector<Layer> L;
    bf16* Xb = nullptr;  // input batch
    float *Xf = nullptr, *Tf = nullptr, *C = nullptr, *ws = nullptr;
    bf16 *dYb = nullptr, *dZb[2] = {nullptr, nullptr};  // hidden layers' dZ, in turn
    int ldy = 0;  // row stride of dYb: the output width, rounded up to 8 when the last layer's backward runs on tcgen05
    double* part = nullptr;
    int* d_perm = nullptr;  // an epoch's order of the dataset
    int* d_err = nullptr;  // set by the tcgen05 GEMM when a completion wait gave up
    float *DX = nullptr, *DT = nullptr;  // dataset
    int dcount = 0;
    size_t ws_count = 0;
    int64_t steps = 0;
    cudaStream_t s = nullptr;
    std::vector<void*> allocs;
    Staging host;  // large transfers from and to the caller's arrays
    std::string err;

    template <class U>
    U* alloc(size_t n) {
        void* p = nullptr;
        cudaError_t e = cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(U));
        if (e != cudaSuccess) throw MlpError{std::string("cudaMalloc: ") + cudaGetErrorString(e)};
        allocs.push_back(p);
        return static_cast<U*>(p);
    }
    ~Mlp() {
        if (s) cudaStreamSynchronize(s);
        for (void* p : allocs) cudaFree(p);
        if (s) cudaStreamDestroy(s);
    }

    void create(int in, int hid, int dep, int out, int mb) {
        in_dim = in, hidden = hid, depth = dep, out_dim = out, max_batch = mb;
        MK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        int prev = in;
        for (int l = 0; l <= depth; ++l) {
            Layer y;
            y.in = prev, y.out = l < depth ? hidden : out;
            y.tc = y.in % 8 == 0;
            y.ldw = y.tc ? (y.out + 15) / 16 * 16 : y.out;
            y.fused = y.tc && (l == depth || y.out % 8 == 0);
            const size_t nw = y.fused ? blocked_size(y.in, y.out) : size_t(y.in) * y.out;
            y.W = alloc<float>(nw), y.gW = alloc<float>(size_t(y.in) * y.out), y.mW = alloc<float>(nw), y.vW = alloc<float>(nw);
            y.Wb = alloc<bf16>(size_t(y.in) * y.ldw);
            MK(cudaMemsetAsync(y.W, 0, nw * sizeof(float), s));  // the padding of the blocks is updated along with them
            y.b = alloc<float>(y.out), y.gb = alloc<float>(y.out), y.mb = alloc<float>(y.out), y.vb = alloc<float>(y.out);
            y.Z = alloc<float>(size_t(mb) * y.out), y.H = alloc<bf16>(size_t(mb) * y.out);
            MK(cudaMemsetAsync(y.mW, 0, nw * sizeof(float), s));
            MK(cudaMemsetAsync(y.vW, 0, nw * sizeof(float), s));
            MK(cudaMemsetAsync(y.mb, 0, y.out * sizeof(float), s));
            MK(cudaMemsetAsync(y.vb, 0, y.out * sizeof(float), s));
            L.push_back(y);
            prev = y.out;
        }
        size_t widest = std::max<size_t>(size_t(out), size_t(hid));
        Xb = alloc<bf16>(size_t(mb) * in), Xf = alloc<float>(size_t(mb) * in), Tf = alloc<float>(size_t(mb) * out);
        ldy = L[depth].tc ? (out + 7) / 8 * 8 : out;
        C = alloc<float>(size_t(mb) * widest), dYb = alloc<bf16>(size_t(mb) * ldy);
        for (bf16*& d : dZb) d = alloc<bf16>(size_t(mb) * hid);
        part = alloc<double>(size_t(loss_ctas())), d_err = alloc<int>(1);
        MK(cudaMemsetAsync(d_err, 0, sizeof(int), s));
        ws_count = size_t(64) * mb * hid;  // split-K partials of dH = dZ W^T (K = out)
        ws = alloc<float>(ws_count);
        size_t largest = size_t(mb) * out;
        for (const Layer& y : L) largest = std::max(largest, size_t(y.in) * y.out);
        host.prepare(largest * sizeof(float));
        MK(cudaStreamSynchronize(s));
    }

    int64_t param_count() const {
        int64_t n = 0;
        for (const Layer& y : L) n += int64_t(y.in) * y.out + y.out;
        return n;
    }

    // C[M][N] = op(A) op(B); split-K (slices > 1) through the workspace.
    template <bool TA, bool TB>
    void gemm(int M, int N, int K, const bf16* A, const bf16* B, float* out, int slices = 1) {
        bool vec = M % 8 == 0 && N % 8 == 0 && K % 8 == 0 && (reinterpret_cast<uintptr_t>(A) % 16 == 0) &&
                   (reinterpret_cast<uintptr_t>(B) % 16 == 0);
        int kslice = (K + slices - 1) / slices;
        kslice = (kslice + BK - 1) / BK * BK;
        slices = (K + kslice - 1) / kslice;
        float* dst = slices > 1 ? ws : out;
        if (slices > 1 && size_t(slices) * M * N > ws_count) throw MlpError{"split-K workspace too small"};
        dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, slices);
        if (vec) k_gemm<TA, TB, true><<<grid, 256, 0, s>>>(M, N, K, kslice, A, B, dst);
        else k_gemm<TA, TB, false><<<grid, 256, 0, s>>>(M, N, K, kslice, A, B, dst);
        if (slices > 1) k_splitk_sum<<<grid1(size_t(M) * N), 256, 0, s>>>(size_t(M) * N, slices, ws, out);
        MK(cudaGetLastError());
    }

    static dim3 grid2(const Layer& y) {  // kernels over the entries of a weight matrix
        return dim3(unsigned(std::min(64, (y.out + 255) / 256)), unsigned(std::min(y.in, 592)));
    }

    int loss_ctas() const { return (out_dim + kLossCols - 1) / kLossCols; }

    void check_tc() {  // after a stream synchronisation: did a tcgen05 GEMM give up waiting?
        int e = 0;
        MK(cudaMemcpyAsync(&e, d_err, sizeof(int), cudaMemcpyDeviceToHost, s));
        MK(cudaStreamSynchronize(s));
        if (e) {
            MK(cudaMemsetAsync(d_err, 0, sizeof(int), s));
            throw MlpError{"tcgen05 GEMM: an MMA completion wait timed out"};
        }
    }

    void tc_check(int rc) {
        if (rc != TARAL_OK) throw MlpError{std::string("tcgen05 GEMM launch: ") + cudaGetErrorString(cudaGetLastError())};
    }

    void forward(int batch) {  // Xb -> L[l].Z, L[l].H ; output Z of the last layer is Y
        const bf16* in = Xb;
        for (int l = 0; l <= depth; ++l) {
            Layer& y = L[l];
            if (y.tc) {
                tc_check(taral::tc::gemm_layer(batch, y.out, y.in, in, y.Wb, y.ldw, y.b, y.Z, l < depth ? y.H : nullptr, d_err, s));
            } else {
                gemm<false, false>(batch, y.out, y.in, in, y.Wb, C);
                k_bias_act<<<grid1(size_t(batch) * y.out), 256, 0, s>>>(batch, y.out, C, y.b, y.Z, l < depth ? y.H : nullptr,
                                                                        l < depth ? 1 : 0);
            }
            in = y.H;
        }
        MK(cudaGetLastError());
    }

    // Needs forward(batch); the target of row r is row idx[r] of T (idx NULL: r). step NULL: fills gW, gb. Otherwise the
    // Adam step is taken on every layer: its dH_prev first, which reads the old weights.
    void backward(int batch, const float* T, const int* idx, const AdamStep* step) {
        auto bias = [&](Layer& y) { return step ? BiasStep{y.b, y.mb, y.vb, *step} : BiasStep{}; };
        Layer& top = L[depth];
        k_loss_grad<<<loss_ctas(), 256, column_smem(batch, kLossCols), s>>>(batch, top.out, ldy, top.Z, T, idx, dYb, top.gb,
                                                                            bias(top), part);
        const bf16* dZ = dYb;
        int ldz = ldy;  // row stride of dZ
        for (int l = depth; l >= 0; --l) {
            Layer& y = L[l];
            const bf16* Hprev = l > 0 ? L[l - 1].H : Xb;
            // tcgen05 when the operands fit TMA (16-byte rows): dH_prev = dZ W^T reads both operands K-major, dW = H_prev^T
            // dZ both MN-major; mma.sync otherwise
            const bool tc = y.tc && ldz % 8 == 0;
            bf16* next = dZb[l & 1];
            if (l > 0) {
                Layer& p = L[l - 1];
                int slices;
                const float* partials = ws;
                if (tc) {
                    const int tiles = ((batch + 127) / 128) * ((y.in + 255) / 256);
                    const size_t per_slice = size_t(batch) * y.in;
                    slices = int(std::max<size_t>(1, std::min<size_t>(std::max(1, 148 / tiles), ws_count / per_slice)));
                    tc_check(taral::tc::gemm_partials(batch, y.in, y.out, dZ, ldz, 0, y.Wb, y.ldw, 0, ws, &slices, d_err, s));
                } else {
                    gemm<false, true>(batch, y.in, y.out, dZ, y.Wb, C, std::max(1, std::min(64, y.out / 2048)));
                    slices = 1, partials = C;
                }
                k_hidden_grad<<<(p.out + kHiddenCols - 1) / kHiddenCols, 1024, column_smem(batch, kHiddenCols), s>>>(
                    batch, p.out, slices, partials, p.Z, next, p.gb, bias(p));
            }
            if (y.fused && step) {
                tc_check(taral::tc::gemm_adam(y.in, y.out, batch, Hprev, y.in, dZ, ldz, y.W, y.mW, y.vW, y.Wb, y.ldw, *step, d_err, s));
            } else {
                if (tc) tc_check(taral::tc::gemm_umma(y.in, y.out, batch, Hprev, y.in, 1, dZ, ldz, 1, y.gW, y.out, 1, nullptr, d_err, s));
                else gemm<true, false>(y.in, y.out, batch, Hprev, dZ, y.gW);  // dW = H_prev^T dZ
                if (step) {
                    k_adam<<<grid2(y), 256, 0, s>>>(y.in, y.out, y.ldw, y.W, y.gW, y.mW, y.vW, y.Wb, *step);
                }
            }
            dZ = next, ldz = hidden;
        }
        MK(cudaGetLastError());
    }

    double loss(int batch) {  // of the last backward(batch); synchronises
        std::vector<double> h(static_cast<size_t>(loss_ctas()));
        MK(cudaMemcpyAsync(h.data(), part, h.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        MK(cudaStreamSynchronize(s));
        double t = 0;
        for (double v : h) t += v;
        return t / (double(batch) * L[depth].out);
    }

    AdamStep next_step(float lr) {
        ++steps;
        const float b1 = 0.9f, b2 = 0.999f;
        return {lr, b1, b2, 1e-8f, 1.f - std::pow(b1, float(steps)), 1.f - std::pow(b2, float(steps))};
    }

    void load_input(int batch, const float* x_host) {
        MK(cudaMemcpyAsync(Xf, x_host, size_t(batch) * in_dim * sizeof(float), cudaMemcpyHostToDevice, s));
        k_to_bf16<<<grid1(size_t(batch) * in_dim), 256, 0, s>>>(size_t(batch) * in_dim, Xf, Xb);
    }
};

}  // namespace mlp
}  // namespace taral

// ================================================================================================ C ABI
using taral::mlp::Mlp;
using taral::mlp::MlpError;

struct taral_mlp {
    Mlp m;
};

#define MLP_GUARD(h, ...)                                     \
    try {                                                     \
        __VA_ARGS__;                                          \
        return TARAL_OK;                                      \
    } catch (const MlpError& e) {                             \
        (h)->m.err = e.msg;                                   \
        return e.msg.find("cudaMalloc") != std::string::npos ? TARAL_ERR_ALLOC : TARAL_ERR_CUDA; \
    } catch (const std::bad_alloc&) {                         \
        return TARAL_ERR_ALLOC;                               \
    }

extern "C" int taral_mlp_create(int in_dim, int hidden, int depth, int out_dim, int max_batch, taral_mlp** out) {
    if (!out || in_dim <= 0 || hidden <= 0 || depth < 0 || out_dim <= 0 || max_batch <= 0) return TARAL_ERR_INPUT;
    *out = nullptr;
    int dev = 0;
    if (cudaGetDeviceCount(&dev) != cudaSuccess || dev == 0) return TARAL_ERR_NO_DEVICE;
    auto* h = new taral_mlp;
    try {
        h->m.create(in_dim, hidden, depth, out_dim, max_batch);
    } catch (const MlpError& e) {
        delete h;
        return e.msg.find("cudaMalloc") != std::string::npos ? TARAL_ERR_ALLOC : TARAL_ERR_CUDA;
    }
    *out = h;
    return TARAL_OK;
}

extern "C" int64_t taral_mlp_param_count(const taral_mlp* h) { return h ? h->m.param_count() : 0; }

// Parameter layout: for each layer W (in x out, row-major) then b (out).
extern "C" int taral_mlp_set_params(taral_mlp* h, const float* params) {
    if (!h || !params) return TARAL_ERR_INPUT;
    MLP_GUARD(h, {
        Mlp& m = h->m;
        const float* p = params;
        for (auto& y : m.L) {
            size_t nw = size_t(y.in) * y.out;
            MK(m.host.copy(y.gW, p, nw * sizeof(float), cudaMemcpyHostToDevice, m.s));  // gW: the row-major form
            taral::mlp::k_set_weights<<<m.grid2(y), 256, 0, m.s>>>(y.in, y.out, y.fused ? taral::mlp::blocked_groups(y.out) : 0,
                                                                   y.ldw, y.gW, y.W, y.Wb);
            p += nw;
            MK(m.host.copy(y.b, p, y.out * sizeof(float), cudaMemcpyHostToDevice, m.s));
            p += y.out;
        }
        MK(cudaStreamSynchronize(m.s));
    })
}

extern "C" int taral_mlp_get_params(taral_mlp* h, float* params) {
    if (!h || !params) return TARAL_ERR_INPUT;
    MLP_GUARD(h, {
        Mlp& m = h->m;
        float* p = params;
        for (auto& y : m.L) {
            size_t nw = size_t(y.in) * y.out;
            if (y.fused)
                taral::mlp::k_get_weights<<<m.grid2(y), 256, 0, m.s>>>(y.in, y.out, taral::mlp::blocked_groups(y.out), y.W, y.gW);
            MK(m.host.copy(p, y.fused ? y.gW : y.W, nw * sizeof(float), cudaMemcpyDeviceToHost, m.s));
            p += nw;
            MK(m.host.copy(p, y.b, y.out * sizeof(float), cudaMemcpyDeviceToHost, m.s));
            p += y.out;
        }
        MK(cudaStreamSynchronize(m.s));
    })
}

extern "C" int taral_mlp_forward(taral_mlp* h, int batch, const float* x, float* y) {
    if (!h || !x || !y || batch <= 0 || batch > h->m.max_batch) return TARAL_ERR_INPUT;
    MLP_GUARD(h, {
        Mlp& m = h->m;
        m.load_input(batch, x);
        m.forward(batch);
        MK(m.host.copy(y, m.L[m.depth].Z, size_t(batch) * m.out_dim * sizeof(float), cudaMemcpyDeviceToHost, m.s));
        MK(cudaStreamSynchronize(m.s));
        m.check_tc();
    })
}

extern "C" int taral_mlp_gradients(taral_mlp* h, int batch, const float* x, const float* target, double* loss,
                                   float* grads) {
    if (!h || !x || !target || batch <= 0 || batch > h->m.max_batch) return TARAL_ERR_INPUT;
    MLP_GUARD(h, {
        Mlp& m = h->m;
        m.load_input(batch, x);
        MK(m.host.copy(m.Tf, target, size_t(batch) * m.out_dim * sizeof(float), cudaMemcpyHostToDevice, m.s));
        m.forward(batch);
        m.backward(batch, m.Tf, nullptr, nullptr);
        const double l = m.loss(batch);
        m.check_tc();
        if (loss) *loss = l;
        if (grads) {
            float* p = grads;
            for (auto& y : m.L) {
                size_t nw = size_t(y.in) * y.out;
                MK(m.host.copy(p, y.gW, nw * sizeof(float), cudaMemcpyDeviceToHost, m.s));
                p += nw;
                MK(m.host.copy(p, y.gb, y.out * sizeof(float), cudaMemcpyDeviceToHost, m.s));
                p += y.out;
            }
            MK(cudaStreamSynchronize(m.s));
        }
    })
}

extern "C" int taral_mlp_set_dataset(taral_mlp* h, int count, const float* x, const float* target) {
    if (!h || count <= 0 || !x || !target) return TARAL_ERR_INPUT;
    MLP_GUARD(h, {
        Mlp& m = h->m;
        if (m.DX) throw MlpError{"dataset already set"};
        m.DX = m.alloc<float>(size_t(count) * m.in_dim), m.DT = m.alloc<float>(size_t(count) * m.out_dim);
        MK(m.host.copy(m.DX, x, size_t(count) * m.in_dim * sizeof(float), cudaMemcpyHostToDevice, m.s));
        MK(m.host.copy(m.DT, target, size_t(count) * m.out_dim * sizeof(float), cudaMemcpyHostToDevice, m.s));
        m.d_perm = m.alloc<int>(size_t(count));
        MK(cudaStreamSynchronize(m.s));
        m.dcount = count;
    })
}

// Adam over the dataset: `epochs` passes of shuffled mini-batches (the last partial batch is dropped).
extern "C" int taral_mlp_train(taral_mlp* h, int epochs, int batch, float lr, uint64_t seed, double* last_loss) {
    if (!h || epochs <= 0 || batch <= 0 || batch > h->m.max_batch || !h->m.DX || h->m.dcount < batch)
        return TARAL_ERR_INPUT;
    MLP_GUARD(h, {
        Mlp& m = h->m;
        std::mt19937_64 rng(seed);
        std::vector<int> perm(m.dcount);
        double loss = 0;
        for (int e = 0; e < epochs; ++e) {
            for (int i = 0; i < m.dcount; ++i) perm[i] = i;
            std::shuffle(perm.begin(), perm.end(), rng);
            MK(cudaMemcpyAsync(m.d_perm, perm.data(), perm.size() * sizeof(int), cudaMemcpyHostToDevice, m.s));
            for (int b0 = 0; b0 + batch <= m.dcount; b0 += batch) {
                taral::mlp::k_gather_rows<<<batch, 128, 0, m.s>>>(m.in_dim, m.d_perm + b0, m.DX, m.Xb);
                m.forward(batch);
                const taral::mlp::AdamStep step = m.next_step(lr);
                m.backward(batch, m.DT, m.d_perm + b0, &step);
            }
        }
        loss = m.loss(batch);  // the last step's
        m.check_tc();
        if (last_loss) *last_loss = loss;
    })
}

extern "C" const char* taral_mlp_last_error(const taral_mlp* h) { return h ? h->m.err.c_str() : "NULL mlp"; }
extern "C" void taral_mlp_destroy(taral_mlp* h) { delete h; }

// Standalone GEMM on device buffers (test hook): C[M][N] (f32) = op(A) op(B), bf16 operands, per the TA/TB rules
// of k_gemm; slices > 1 uses split-K through a caller-provided workspace of slices * M * N floats.
extern "C" int taral_gemm_bf16(int M, int N, int K, int ta, int tb, const void* A, const void* B, float* C,
                               int slices, float* workspace, void* stream) {
    using namespace taral::mlp;
    if (M <= 0 || N <= 0 || K <= 0 || !A || !B || !C || slices < 1 || (slices > 1 && !workspace)) return TARAL_ERR_INPUT;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    bool vec = M % 8 == 0 && N % 8 == 0 && K % 8 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0 &&
               reinterpret_cast<uintptr_t>(B) % 16 == 0;
    int kslice = (K + slices - 1) / slices;
    kslice = (kslice + BK - 1) / BK * BK;
    slices = (K + kslice - 1) / kslice;
    float* dst = slices > 1 ? workspace : C;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, slices);
    const bf16* a = static_cast<const bf16*>(A);
    const bf16* b = static_cast<const bf16*>(B);
#define LAUNCH(TA_, TB_)                                                                       \
    if (vec) k_gemm<TA_, TB_, true><<<grid, 256, 0, s>>>(M, N, K, kslice, a, b, dst);          \
    else k_gemm<TA_, TB_, false><<<grid, 256, 0, s>>>(M, N, K, kslice, a, b, dst);
    if (!ta && !tb) { LAUNCH(false, false) }
    else if (ta && !tb) { LAUNCH(true, false) }
    else if (!ta && tb) { LAUNCH(false, true) }
    else { LAUNCH(true, true) }
#undef LAUNCH
    if (slices > 1) k_splitk_sum<<<grid1(size_t(M) * N), 256, 0, s>>>(size_t(M) * N, slices, workspace, C);
    return cudaGetLastError() == cudaSuccess ? TARAL_OK : TARAL_ERR_CUDA;
}
