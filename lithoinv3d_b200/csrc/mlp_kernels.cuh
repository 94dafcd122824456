// BF16 tensor-core kernels of the warm-start MLP (training and inference),
// FP32 accumulation.  No reference counterpart: the reference has no learned
// component.
//
// GEMM: C[M x N] = A[M x K] . B[K x N], bf16 operands, fp32 accumulators,
// mma.sync m16n8k16.  A is stored row-major [M][K] (A_T = false) or as its
// transpose [K][M] (A_T = true); B row-major [K][N] (B_T = false) or as [N][K]
// (B_T = true).  Tiles stay in the stored layout in shared memory and the
// fragments are read with ldmatrix, transposing on the fly where the stored
// layout differs from the fragment's -- so the forward Y = X W^T, the input
// gradient dX = dY W and the weight gradient dW = dY^T X use one kernel.
// M and N must be multiples of 128 and K of 32 (the network pads its
// layers); every operand row starts on a 16-byte boundary.
//
// Three square CTA tiles, K through a ring of cp.async stages: 128 (8 warps of
// 64 x 32, 2 stages of 32), 64 (8 warps of 32 x 16, 4 stages of 32) and 32
// (4 warps of 16 x 16, 8 stages of 64: K a multiple of 64).  An element's products are added in the
// same order in all of them, so the choice is one of speed alone (mma_tile).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace litho_b200 {
namespace mlp {

constexpr int kBM = 128, kBN = 128, kBK = 32;  // granules of M, N and K
// Shared-memory row lengths (bf16 elements): +8 keeps ldmatrix rows on
// different banks and 16-byte aligned.  Tiles are stored [BT][kBK] or [kBK][BT].
template <int BT>
struct MmaShape {
    static constexpr int kThreads = BT == 32 ? 128 : 256;
    static constexpr int kStages = BT == 128 ? 2 : BT == 64 ? 4 : 8;
    static constexpr int kBK = BT == 32 ? 64 : 32;
    static constexpr int kWarpsN = BT == 32 ? 2 : 4;
    static constexpr int kWM = BT / 2, kWN = BT / kWarpsN;  // warp tile (two warp rows)
    static constexpr int kMI = kWM / 16, kNI = kWN / 8;
    static constexpr int kRowMK = kBK + 8, kRowKM = BT + 8;
    static constexpr int kTile = BT * kRowMK > kBK * kRowKM ? BT * kRowMK : kBK * kRowKM;
    static constexpr int kRing = kStages * 2 * kTile;  // elements: A and B tiles of every stage
    static constexpr int kSmem = kRing * 2;            // bytes
};

// A kernel launched with programmatic stream serialisation (launch_next) may
// be put on the SMs before the kernels ahead of it in the stream are done.
// Every kernel of the training chain calls this before its first access to
// memory: it lets the next one on in turn, and waits until the work ahead is
// complete and visible.  Without that launch attribute it does nothing.
__device__ __forceinline__ void wait_for_stream() {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
}

enum Epilogue {
    EPI_F32 = 0,        // C fp32
    EPI_BIAS_RELU = 1,  // bf16 relu(C + bias[n])
    EPI_BIAS_F32 = 2,   // fp32 C + bias[n]
    EPI_BF16 = 3,       // bf16 C
    EPI_BF16_RELU_BWD = 4,  // bf16 C where the forward's activation was positive, else 0
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(smem)), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_addr(p)));
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Loads one operand tile (BT rows of the M or N side x kBK of K) into shared
// memory in its stored layout.  TRANS = stored [K][MN]: kBK rows of BT.
template <int BT, bool TRANS>
__device__ __forceinline__ void load_tile(__nv_bfloat16* sm, const __nv_bfloat16* __restrict__ g, int ld, int mn0,
                                          int k0) {
    using Sh = MmaShape<BT>;
#pragma unroll
    for (int i = 0; i < BT * Sh::kBK / 8 / Sh::kThreads; ++i) {
        const int c = (int)threadIdx.x + i * Sh::kThreads;
        if (!TRANS) {  // [mn][k]: BT rows x kBK / 8 chunks of 8
            const int row = c / (Sh::kBK / 8), col = (c % (Sh::kBK / 8)) * 8;
            cp_async16(sm + row * Sh::kRowMK + col, g + (size_t)(mn0 + row) * ld + k0 + col);
        } else {  // [k][mn]: kBK rows x BT / 8 chunks of 8
            const int row = c / (BT / 8), col = (c % (BT / 8)) * 8;
            cp_async16(sm + row * Sh::kRowKM + col, g + (size_t)(k0 + row) * ld + mn0 + col);
        }
    }
}

// One CTA tile at (m0, n0): acc = A . B over nk steps of kBK, every element's
// products added in ascending k.  lda / ldb: row lengths (elements) of A and
// B as stored; ring: MmaShape<BT>::kRing elements of shared memory.
template <int BT, bool A_T, bool B_T>
__device__ __forceinline__ void mma_tile_sum(float (&acc)[MmaShape<BT>::kMI][MmaShape<BT>::kNI][4],
                                             __nv_bfloat16* ring, int nk, const __nv_bfloat16* __restrict__ A, int lda,
                                             int m0, const __nv_bfloat16* __restrict__ B, int ldb, int n0) {
    using Sh = MmaShape<BT>;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp / Sh::kWarpsN) * Sh::kWM, wn = (warp % Sh::kWarpsN) * Sh::kWN;
#pragma unroll
    for (int i = 0; i < Sh::kMI; ++i)
#pragma unroll
        for (int j = 0; j < Sh::kNI; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.f;
    auto fill = [&](int kt) {
        __nv_bfloat16* st = ring + (kt % Sh::kStages) * 2 * Sh::kTile;
        load_tile<BT, A_T>(st, A, lda, m0, kt * Sh::kBK);
        load_tile<BT, !B_T>(st + Sh::kTile, B, ldb, n0, kt * Sh::kBK);
    };
#pragma unroll
    for (int kt = 0; kt < Sh::kStages - 1; ++kt) {
        if (kt < nk) fill(kt);
        cp_async_commit();
    }
    const int r = lane & 7, mat = lane >> 3;  // ldmatrix: row within 8x8 matrix, matrix index
    for (int kt = 0; kt < nk; ++kt) {
        // stage kt has landed, and every warp is done with stage kt - 1, which is refilled
        cp_async_wait<Sh::kStages - 2>();
        __syncthreads();
        if (kt + Sh::kStages - 1 < nk) fill(kt + Sh::kStages - 1);
        cp_async_commit();
        const __nv_bfloat16* a = ring + (kt % Sh::kStages) * 2 * Sh::kTile;
        const __nv_bfloat16* b = a + Sh::kTile;
#pragma unroll
        for (int kk = 0; kk < Sh::kBK; kk += 16) {
            uint32_t af[Sh::kMI][4];
#pragma unroll
            for (int i = 0; i < Sh::kMI; ++i) {
                const int mrow = wm + i * 16;
                if (!A_T)  // stored [m][k]: matrices (m+0,k+0) (m+8,k+0) (m+0,k+8) (m+8,k+8)
                    ldsm_x4(af[i], a + (mrow + r + 8 * (mat & 1)) * Sh::kRowMK + kk + 8 * (mat >> 1));
                else  // stored [k][m], transposed on load
                    ldsm_x4_t(af[i], a + (kk + r + 8 * (mat >> 1)) * Sh::kRowKM + mrow + 8 * (mat & 1));
            }
            uint32_t bf[Sh::kNI][2];
#pragma unroll
            for (int j = 0; j < Sh::kNI; j += 2) {
                const int ncol = wn + j * 8;
                uint32_t t4[4];
                if (B_T)  // stored [n][k]: matrices (n+0,k+0) (n+0,k+8) (n+8,k+0) (n+8,k+8)
                    ldsm_x4(t4, b + (ncol + r + 8 * (mat >> 1)) * Sh::kRowMK + kk + 8 * (mat & 1));
                else  // stored [k][n], transposed on load
                    ldsm_x4_t(t4, b + (kk + r + 8 * (mat & 1)) * Sh::kRowKM + ncol + 8 * (mat >> 1));
                bf[j][0] = t4[0]; bf[j][1] = t4[1];
                bf[j + 1][0] = t4[2]; bf[j + 1][1] = t4[3];
            }
#pragma unroll
            for (int i = 0; i < Sh::kMI; ++i)
#pragma unroll
                for (int j = 0; j < Sh::kNI; ++j) mma_bf16(acc[i][j], af[i], bf[j][0], bf[j][1]);
        }
    }
}

// Calls f(row, col, c0, c1) for the thread's pairs of neighbouring columns of
// the tile at (m0, n0).
template <int BT, typename F>
__device__ __forceinline__ void mma_tile_each(const float (&acc)[MmaShape<BT>::kMI][MmaShape<BT>::kNI][4], int m0,
                                              int n0, F f) {
    using Sh = MmaShape<BT>;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // c0,c1 at (row g, cols 2q, 2q+1), c2,c3 at row g + 8
    const int row0 = m0 + (warp / Sh::kWarpsN) * Sh::kWM + (lane >> 2);
    const int col0 = n0 + (warp % Sh::kWarpsN) * Sh::kWN + 2 * (lane & 3);
#pragma unroll
    for (int i = 0; i < Sh::kMI; ++i)
#pragma unroll
        for (int j = 0; j < Sh::kNI; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) f(row0 + i * 16 + 8 * h, col0 + j * 8, acc[i][j][2 * h], acc[i][j][2 * h + 1]);
}

// y: the forward's activations [M][ldc], read by EPI_BF16_RELU_BWD alone.
template <int BT, bool A_T, bool B_T, int EPI>
__global__ void __launch_bounds__(MmaShape<BT>::kThreads)
    k_gemm_bf16(int K, const __nv_bfloat16* __restrict__ A, int lda, const __nv_bfloat16* __restrict__ B, int ldb,
                const float* __restrict__ bias, float* __restrict__ Cf, __nv_bfloat16* __restrict__ Cb, int ldc,
                const __nv_bfloat16* __restrict__ y) {
    using Sh = MmaShape<BT>;
    extern __shared__ __align__(16) __nv_bfloat16 ring[];
    wait_for_stream();
    const int m0 = blockIdx.y * BT, n0 = blockIdx.x * BT;
    float acc[Sh::kMI][Sh::kNI][4];
    mma_tile_sum<BT, A_T, B_T>(acc, ring, K / Sh::kBK, A, lda, m0, B, ldb, n0);
    mma_tile_each<BT>(acc, m0, n0, [&](int row, int col, float v0, float v1) {
        if (EPI == EPI_BIAS_RELU || EPI == EPI_BIAS_F32) {
            v0 += bias[col];
            v1 += bias[col + 1];
        }
        if (EPI == EPI_BIAS_RELU || EPI == EPI_BF16 || EPI == EPI_BF16_RELU_BWD) {
            __nv_bfloat162 o;
            o.x = __float2bfloat16(EPI == EPI_BIAS_RELU ? fmaxf(v0, 0.f) : v0);
            o.y = __float2bfloat16(EPI == EPI_BIAS_RELU ? fmaxf(v1, 0.f) : v1);
            if (EPI == EPI_BF16_RELU_BWD) {
                const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(y + (size_t)row * ldc + col);
                if (!(__bfloat162float(a.x) > 0.f)) o.x = __float2bfloat16(0.f);
                if (!(__bfloat162float(a.y) > 0.f)) o.y = __float2bfloat16(0.f);
            }
            *reinterpret_cast<__nv_bfloat162*>(Cb + (size_t)row * ldc + col) = o;
        } else {
            *reinterpret_cast<float2*>(Cf + (size_t)row * ldc + col) = make_float2(v0, v1);
        }
    });
}

// Rows of x [][n] fp32 (rows[r], or r itself) -> bf16 [batch][n_pad] (n_pad a
// multiple of 4): padding columns and the batch's rows from n_rows on are
// zero.  Four columns per thread; vec: every row of x starts on a 16-byte
// boundary.
__global__ void k_load_input(int n_rows, int batch, int n, int n_pad, bool vec, const float* __restrict__ x,
                             const long long* __restrict__ rows, __nv_bfloat16* __restrict__ y) {
    wait_for_stream();
    const size_t i = 4 * (blockIdx.x * (size_t)blockDim.x + threadIdx.x);
    if (i >= (size_t)batch * n_pad) return;
    const int r = (int)(i / n_pad), c = (int)(i % n_pad);
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (r < n_rows) {
        const float* p = x + (size_t)(rows ? rows[r] : r) * n + c;
        if (vec && c < n) {  // n is a multiple of 4
            const float4 q = *reinterpret_cast<const float4*>(p);
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (c + k < n) v[k] = p[k];
        }
    }
    __nv_bfloat162 o[2];
    o[0].x = __float2bfloat16(v[0]); o[0].y = __float2bfloat16(v[1]);
    o[1].x = __float2bfloat16(v[2]); o[1].y = __float2bfloat16(v[3]);
    *reinterpret_cast<uint2*>(y + i) = *reinterpret_cast<const uint2*>(o);
}

// Loss: 0.5 * mean over (row, col < n_valid) of (pred - target)^2 with the
// gradient w.r.t. pred (bf16, padding columns zero) and per-block sums.  Row
// r's target is row target_rows[r], or r itself.
__global__ void k_mse(int rows, int cols, int n_valid, const float* __restrict__ pred, const float* __restrict__ target,
                      const long long* __restrict__ target_rows, int ld_target, __nv_bfloat16* __restrict__ dpred,
                      float* __restrict__ block_loss) {
    wait_for_stream();
    __shared__ float red[256];
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const float inv = 1.f / ((float)rows * (float)n_valid);
    float l = 0.f;
    if (i < (size_t)rows * cols) {
        const int r = (int)(i / cols), c = (int)(i % cols);
        float d = 0.f;
        if (c < n_valid) {
            d = pred[i] - target[(size_t)(target_rows ? target_rows[r] : r) * ld_target + c];
            l = 0.5f * d * d * inv;
        }
        dpred[i] = __float2bfloat16(d * inv);
    }
    red[threadIdx.x] = l;
    __syncthreads();
    for (int k = blockDim.x / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) block_loss[blockIdx.x] = red[0];
}

// ReLU backward in place on the bf16 gradient: dz = dy * (y > 0).
__global__ void k_relu_bwd(size_t n, const __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ dy) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < n && !(__bfloat162float(y[i]) > 0.f)) dy[i] = __float2bfloat16(0.f);
}

// Bias gradient: column sums of dY [rows][ld] (bf16) over 32 columns from c0,
// returned by the block's first 32 threads.  The block stages
// 128 rows at a time so that the loads overlap; each column's rows are then
// added in order by one thread.  rows is a multiple of 128; st: 128 x 32.
__device__ __forceinline__ float colsum32(int rows, int ld, int c0, const __nv_bfloat16* __restrict__ dy,
                                          __nv_bfloat16 (&st)[128][32]) {
    float s = 0.f;
    for (int r0 = 0; r0 < rows; r0 += 128) {
        __syncthreads();
        for (int c = threadIdx.x; c < 128 * 4; c += blockDim.x) {  // 128 rows of 4 16-byte chunks
            const int row = c >> 2, col = (c & 3) * 8;
            *reinterpret_cast<uint4*>(&st[row][col]) =
                *reinterpret_cast<const uint4*>(dy + (size_t)(r0 + row) * ld + c0 + col);
        }
        __syncthreads();
        if (threadIdx.x < 32) {
#pragma unroll 16
            for (int r = 0; r < 128; ++r) s += __bfloat162float(st[r][threadIdx.x]);
        }
    }
    return s;
}

__global__ void __launch_bounds__(128) k_colsum(int rows, int cols, const __nv_bfloat16* __restrict__ dy,
                                                float* __restrict__ out) {
    __shared__ __align__(16) __nv_bfloat16 st[128][32];
    const int c0 = blockIdx.x * 32;
    const float s = colsum32(rows, cols, c0, dy, st);
    if (threadIdx.x < 32) out[c0 + threadIdx.x] = s;
}

// Adam on one fp32 master weight (Kingma & Ba, 2015, with bias correction
// c1 = 1 - b1^t, c2 = 1 - b2^t); returns the new weight.
struct Adam {
    float lr, b1, b2, eps, c1, c2;
};
__device__ __forceinline__ float adam_update(const Adam& k, float w, float g, float& m1, float& m2) {
    const float a = k.b1 * m1 + (1.f - k.b1) * g, b = k.b2 * m2 + (1.f - k.b2) * g * g;
    m1 = a;
    m2 = b;
    return w - k.lr * (a / k.c1) / (sqrtf(b / k.c2) + k.eps);
}

// n weights; refreshes the bf16 copy wb when given.
__global__ void k_adam(size_t n, float* __restrict__ w, const float* __restrict__ gw, float* __restrict__ m1,
                       float* __restrict__ m2, Adam k, __nv_bfloat16* __restrict__ wb) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float a = m1[i], b = m2[i];
    const float v = adam_update(k, w[i], gw[i], a, b);
    m1[i] = a;
    m2[i] = b;
    w[i] = v;
    if (wb) wb[i] = __float2bfloat16(v);
}

// Parameter gradients of several layers in one launch, and with UPDATE the
// Adam step on them: gradients then stay in registers.  Blocks
// [tile0, tile0 + (out / 64) (in / 64)) of a layer form 64 x 64 tiles of
// dW = dZ^T X; the next out / 32 blocks its bias gradients.
// The optimiser's state is 26 bytes per weight and sets the floor (21 us at
// 6.5 TB/s for 5.4e6 weights); what the kernel waits for is the latency of
// state loads and divisions, so 8 warps share a tile (4 warps: 53 us, 8: 43),
// the state is prefetched into L2 while the products run and rows are updated
// 16 bytes a thread.  One launch, because narrow layers are a fraction of a
// wave each (separate products, column sums and updates: 220 us).
struct LayerGrad {
    const __nv_bfloat16 *dz, *x;  // [batch][out], [batch][in]
    float *w, *gw, *mw, *vw, *b, *gb, *mb, *vb;
    __nv_bfloat16* wb;
    int in, out, block0;
};
constexpr int kGradLayers = 16;  // per launch
struct LayerGrads {
    LayerGrad layer[kGradLayers];
    int n;
};

template <bool UPDATE>
__global__ void __launch_bounds__(MmaShape<64>::kThreads)
    k_layer_grads(const __grid_constant__ LayerGrads L, int batch, Adam k) {
    using Sh = MmaShape<64>;
    __shared__ __align__(16) __nv_bfloat16 ring[Sh::kRing];
    wait_for_stream();
    int l = 0;
    while (l + 1 < L.n && (int)blockIdx.x >= L.layer[l + 1].block0) ++l;
    const LayerGrad& g = L.layer[l];
    const int t = (int)blockIdx.x - g.block0, tx = g.in / 64, tiles = tx * (g.out / 64);
    if (t < tiles) {
        const int m0 = (t / tx) * 64, n0 = (t % tx) * 64;
        const int row0 = (int)threadIdx.x / 16, col0 = ((int)threadIdx.x % 16) * 4;  // update: rows of 64, 16 per pass
        if (UPDATE)  // the optimiser's state on its way from DRAM while the products run
            for (int c = threadIdx.x; c < 3 * 64 * 2; c += Sh::kThreads) {
                const float* p = c < 128 ? g.w : c < 256 ? g.mw : g.vw;
                p += (size_t)(m0 + (c & 127) / 2) * g.in + n0 + (c & 1) * 32;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
            }
        float acc[Sh::kMI][Sh::kNI][4];
        // A = dZ stored [batch][out] = [K][M]; B = X [batch][in] = [K][N]
        mma_tile_sum<64, true, false>(acc, ring, batch / Sh::kBK, g.dz, g.out, m0, g.x, g.in, n0);
        if (!UPDATE) {
            mma_tile_each<64>(acc, m0, n0, [&](int row, int col, float v0, float v1) {
                *reinterpret_cast<float2*>(g.gw + (size_t)row * g.in + col) = make_float2(v0, v1);
            });
            return;
        }
        // through shared memory, so that state rows are read and written 16 bytes a thread
        constexpr int kRow = 68;
        static_assert(64 * kRow * sizeof(float) <= Sh::kRing * sizeof(__nv_bfloat16), "the tile fits the ring");
        float* tile = reinterpret_cast<float*>(ring);
        __syncthreads();
        mma_tile_each<64>(acc, 0, 0, [&](int row, int col, float v0, float v1) {
            *reinterpret_cast<float2*>(tile + row * kRow + col) = make_float2(v0, v1);
        });
        __syncthreads();
#pragma unroll 2
        for (int r = row0; r < 64; r += 16) {
            const size_t i = (size_t)(m0 + r) * g.in + n0 + col0;
            const float4 d = *reinterpret_cast<const float4*>(tile + r * kRow + col0);
            float4 w = *reinterpret_cast<const float4*>(g.w + i), m = *reinterpret_cast<const float4*>(g.mw + i),
                   v = *reinterpret_cast<const float4*>(g.vw + i);
            w.x = adam_update(k, w.x, d.x, m.x, v.x);
            w.y = adam_update(k, w.y, d.y, m.y, v.y);
            w.z = adam_update(k, w.z, d.z, m.z, v.z);
            w.w = adam_update(k, w.w, d.w, m.w, v.w);
            *reinterpret_cast<float4*>(g.w + i) = w;
            *reinterpret_cast<float4*>(g.mw + i) = m;
            *reinterpret_cast<float4*>(g.vw + i) = v;
            __nv_bfloat162 o[2];
            o[0].x = __float2bfloat16(w.x);
            o[0].y = __float2bfloat16(w.y);
            o[1].x = __float2bfloat16(w.z);
            o[1].y = __float2bfloat16(w.w);
            *reinterpret_cast<uint2*>(g.wb + i) = *reinterpret_cast<const uint2*>(o);
        }
    } else {
        const int c = (t - tiles) * 32 + (int)threadIdx.x;
        const float s = colsum32(batch, g.out, (t - tiles) * 32, g.dz,
                                 *reinterpret_cast<__nv_bfloat16(*)[128][32]>(ring));
        if (threadIdx.x >= 32) return;
        if (!UPDATE) {
            g.gb[c] = s;
        } else {
            float m = g.mb[c], v = g.vb[c];
            g.b[c] = adam_update(k, g.b[c], s, m, v);
            g.mb[c] = m;
            g.vb[c] = v;
        }
    }
}

}  // namespace mlp
}  // namespace litho_b200
