// Warm-start MLP: training and inference on the device with the BF16
// tensor-core kernels of mlp_kernels.cuh.  No reference counterpart (the
// reference's L-BFGS-B starts from the model's own parameters with a
// steepest-descent first step, lbfgsb_optimizer.cpp:35-38, 162).
//
// Network: n_in -> width (ReLU) x depth -> n_out, fp32 master weights with
// Adam, bf16 copies for the GEMMs, fp32 accumulation.  Layer widths are
// padded to multiples of 128 (the GEMM tile); padded output columns carry
// zero targets and are masked out of the loss.
#include "../../include/litho_gpu.h"
#include "mlp_kernels.cuh"
#include "per_device.hpp"
#include "tc_gemm.cuh"
#include "tc_gemm_tma.cuh"

#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

using litho_b200::PerDevice;
using namespace litho_b200::mlp;

namespace {

int cdiv_i(long long a, long long b) { return static_cast<int>((a + b - 1) / b); }
int pad128(int n) { return cdiv_i(n, 128) * 128; }

template <typename T>
struct Buf {
    T* p = nullptr;
    size_t n = 0;
    Buf() = default;
    Buf(const Buf&) = delete;
    Buf& operator=(const Buf&) = delete;
    Buf(Buf&& o) noexcept : p(o.p), n(o.n) {
        o.p = nullptr;
        o.n = 0;
    }
    ~Buf() {
        if (p) cudaFree(p);
    }
    cudaError_t alloc(size_t count) {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
        cudaError_t e = cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T));
        if (e == cudaSuccess) {
            n = count;
            e = cudaMemset(p, 0, std::max<size_t>(count, 1) * sizeof(T));
        }
        return e;
    }
};

constexpr int kQueued = 32;  // training batches launched before the host waits

struct Layer {
    int in = 0, out = 0;  // padded dims
    Buf<float> w, b, gw, gb, mw, vw, mb, vb;
    Buf<__nv_bfloat16> wb;  // bf16 copy [out][in]
    Buf<__nv_bfloat16> act;  // bf16 output activation [batch][out] (hidden layers)
    Buf<__nv_bfloat16> dz;   // bf16 gradient of the output before the ReLU [batch][out]
};

}  // namespace

struct lf_mlp {
    int device = 0;
    cudaStream_t stream = nullptr;
    int n_in = 0, n_in_pad = 0, width = 0, depth = 0, n_out = 0, n_out_pad = 0, batch = 0;
    std::vector<Layer> layers;  // depth hidden + 1 output
    Buf<__nv_bfloat16> xb;  // input (bf16)
    Buf<float> pred, loss_blocks;
    int n_loss = 0;           // loss blocks of one batch; loss_blocks holds kQueued batches
    float* h_loss = nullptr;  // pinned: the loss blocks, then the GEMM error flag
    Buf<long long> rows;      // row numbers of the queued batches, and their pinned host copy
    long long* h_rows = nullptr;
    int step = 0;
    int engine = LF_GEMM_AUTO;  // lf_mlp_set_engine: per GEMM, TMA-fed tcgen05 for deep K, mma.sync otherwise
    std::string err;
};

#define MLP_TRY(m, expr)                                                       \
    do {                                                                       \
        cudaError_t e_ = (expr);                                               \
        if (e_ != cudaSuccess) {                                               \
            (m)->err = std::string(#expr) + ": " + cudaGetErrorString(e_);     \
            return LF_ECUDA;                                                   \
        }                                                                      \
    } while (0)

static lf_status mlp_check_launch(lf_mlp* m) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        m->err = std::string("kernel launch: ") + cudaGetErrorString(e);
        return LF_ECUDA;
    }
    return LF_OK;
}

// Raises the kernel's dynamic shared-memory limit on the current device.
template <typename... P>
static cudaError_t allow_smem(PerDevice& limit, void (*kernel)(P...), int bytes) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    return limit.once(dev, [&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); });
}

// One GEMM on `stream`: the tcgen05 kernel (K a multiple of 64; 128 x 256
// tiles when N allows, else 128 x 128) or the warp-level mma.sync kernel
// (K a multiple of 32).
template <bool A_T, bool B_T, int EPI, int BN>
static cudaError_t gemm_tc(cudaStream_t stream, int M, int N, int K, const __nv_bfloat16* A, int lda,
                           const __nv_bfloat16* B, int ldb, const float* bias, float* Cf, __nv_bfloat16* Cb, int ldc) {
    static PerDevice limit;  // per instantiation
    const cudaError_t e = allow_smem(limit, k_gemm_tc<A_T, B_T, EPI, BN>, TcShape<BN>::kSmem);
    if (e != cudaSuccess) return e;
    dim3 grid(N / BN, M / kBM);
    k_gemm_tc<A_T, B_T, EPI, BN><<<grid, kTcThreads, TcShape<BN>::kSmem, stream>>>(M, N, K, A, lda, B, ldb, bias, Cf,
                                                                                  Cb, ldc);
    return cudaPeekAtLastError();  // left for the caller's launch check
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (the
// library does not link the driver library itself).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

// 2-D tensor map of a row-major bf16 array [rows][cols] with row length ld
// (elements): boxes of 64 columns x box_rows rows, 128-byte swizzle.
static bool bf16_map(CUtensorMap* map, const void* base, int rows, int cols, int ld, int box_rows) {
    const auto encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {64u, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1u, 1u};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// One GEMM on the TMA-fed, warp-specialised tcgen05 kernel (tc_gemm_tma.cuh).
template <bool A_T, bool B_T, int EPI, int BN>
static cudaError_t gemm_tma(cudaStream_t stream, int M, int N, int K, const __nv_bfloat16* A, int lda,
                            const __nv_bfloat16* B, int ldb, const float* bias, float* Cf, __nv_bfloat16* Cb, int ldc) {
    static PerDevice limit;
    const cudaError_t e = allow_smem(limit, k_gemm_tma<A_T, B_T, EPI, BN>, TmaShape<BN>::kSmem);
    if (e != cudaSuccess) return e;
    CUtensorMap mapA, mapB;
    const bool okA = A_T ? bf16_map(&mapA, A, K, M, lda, 64) : bf16_map(&mapA, A, M, K, lda, kBM);
    const bool okB = B_T ? bf16_map(&mapB, B, N, K, ldb, BN) : bf16_map(&mapB, B, K, N, ldb, 64);
    if (!okA || !okB) return cudaErrorInvalidValue;
    dim3 grid(N / BN, M / kBM);
    k_gemm_tma<A_T, B_T, EPI, BN><<<grid, kTmaThreads, TmaShape<BN>::kSmem, stream>>>(M, N, K, mapA, mapB, bias, Cf,
                                                                                     Cb, ldc);
    return cudaPeekAtLastError();
}

// LF_GEMM_AUTO: the TMA-fed tcgen05 kernel where a deep reduction has enough
// 128 x 128 output tiles to fill a third of the SMs, the mma.sync kernel
// otherwise: its 32 x 32 tiles spread a small product over the whole chip,
// where one tcgen05 tile is a serial chain of K / 16 instructions on one SM.
// Measured on B200, microseconds of a blocking call (20 of them its own),
// mma.sync against tcgen05: 256 x 512 x 8192 39 / 90, 512 x 1024 x 8192
// 79 / 91, 768 x 1024 x 8192 111 / 91, 2048 x 2048 x 8192 295 / 97; at K = 2048
// 256 x 512 22 / 54, 1024 x 1024 41 / 54, 2048 x 2048 88 / 56.  The line is that
// of K = 8192; at K = 2048 the sizes cross between 64 and 256 tiles, so the
// least of the products it sends to tcgen05 there are faster on mma.sync.  Below
// K = 2048 tcgen05 stays behind (14.0 against 8.9 TFLOP/s at K = 512).
constexpr int kAutoTmaMinK = 2048, kAutoTmaMinTiles = 48;
static int auto_engine(int M, int N, int K) {
    const bool tma = K >= kAutoTmaMinK && K % kTcBK == 0 && (long long)(M / kBM) * (N / kBN) >= kAutoTmaMinTiles;
    return tma ? LF_GEMM_TCGEN05_TMA : LF_GEMM_MMA_SYNC;
}

// The mma.sync kernel's CTA tile: the largest that still gives every SM a
// tile, 32 for what is smaller than that (a 256 x 512 layer is 8 tiles of 128
// on 148 SMs, 128 tiles of 32).  Kernel times on B200: 256 x 512 x 512 9.5 ->
// 3.8 us (tiles of 128, of 32), 256 x 512 x 1408 26 -> 6.9 us, 256 x 512 x 8192
// 27 us (87 us in 128 x 256 tiles of the tcgen05 kernel); 1024 x 1024 x 1024
// 36 -> 26 us a blocking call with tiles of 64.
constexpr int kSms = 148;
static int mma_tile(int M, int N, int K) {
    if ((long long)(M / 128) * (N / 128) >= kSms) return 128;
    return (long long)(M / 64) * (N / 64) >= kSms || K % MmaShape<32>::kBK ? 64 : 32;
}

// Launches a kernel that calls wait_for_stream: its blocks may be placed while
// the work ahead in the stream drains: 1.5 us less per kernel, 152 -> 134 us for
// the 12 kernels of a step of the 8192 -> 512 x 4 -> 1313 network.  Errors are
// left for the caller's launch check too.
template <typename... P, typename... A>
static cudaError_t launch_next(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                               A... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <int BT, bool A_T, bool B_T, int EPI>
static cudaError_t launch_mma(cudaStream_t stream, int M, int N, int K, const __nv_bfloat16* A, int lda,
                              const __nv_bfloat16* B, int ldb, const float* bias, float* Cf, __nv_bfloat16* Cb,
                              int ldc, const __nv_bfloat16* y) {
    using Sh = MmaShape<BT>;
    if (Sh::kSmem > 48 * 1024) {
        static PerDevice limit;
        const cudaError_t e = allow_smem(limit, k_gemm_bf16<BT, A_T, B_T, EPI>, Sh::kSmem);
        if (e != cudaSuccess) return e;
    }
    return launch_next(k_gemm_bf16<BT, A_T, B_T, EPI>, dim3(N / BT, M / BT), Sh::kThreads, Sh::kSmem, stream, K, A, lda,
                       B, ldb, bias, Cf, Cb, ldc, y);
}

template <bool A_T, bool B_T, int EPI>
static cudaError_t gemm_mma(cudaStream_t stream, int M, int N, int K, const __nv_bfloat16* A, int lda,
                            const __nv_bfloat16* B, int ldb, const float* bias, float* Cf, __nv_bfloat16* Cb, int ldc,
                            const __nv_bfloat16* y = nullptr) {
    switch (mma_tile(M, N, K)) {
    case 128: return launch_mma<128, A_T, B_T, EPI>(stream, M, N, K, A, lda, B, ldb, bias, Cf, Cb, ldc, y);
    case 64: return launch_mma<64, A_T, B_T, EPI>(stream, M, N, K, A, lda, B, ldb, bias, Cf, Cb, ldc, y);
    default: return launch_mma<32, A_T, B_T, EPI>(stream, M, N, K, A, lda, B, ldb, bias, Cf, Cb, ldc, y);
    }
}

template <bool A_T, bool B_T, int EPI>
static cudaError_t gemm_on(int engine, cudaStream_t stream, int M, int N, int K, const __nv_bfloat16* A, int lda,
                           const __nv_bfloat16* B, int ldb, const float* bias, float* Cf, __nv_bfloat16* Cb, int ldc) {
    if (engine == LF_GEMM_AUTO) engine = auto_engine(M, N, K);
    if (engine == LF_GEMM_TCGEN05_TMA) {
        if (N % 256 == 0)
            return gemm_tma<A_T, B_T, EPI, 256>(stream, M, N, K, A, lda, B, ldb, bias, Cf, Cb, ldc);
        return gemm_tma<A_T, B_T, EPI, 128>(stream, M, N, K, A, lda, B, ldb, bias, Cf, Cb, ldc);
    }
    if (engine == LF_GEMM_TCGEN05) {
        if (N % 256 == 0)
            return gemm_tc<A_T, B_T, EPI, 256>(stream, M, N, K, A, lda, B, ldb, bias, Cf, Cb, ldc);
        return gemm_tc<A_T, B_T, EPI, 128>(stream, M, N, K, A, lda, B, ldb, bias, Cf, Cb, ldc);
    }
    return gemm_mma<A_T, B_T, EPI>(stream, M, N, K, A, lda, B, ldb, bias, Cf, Cb, ldc);
}

template <bool A_T, bool B_T, int EPI>
static void gemm(lf_mlp* m, int M, int N, int K, const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb,
                 const float* bias, float* Cf, __nv_bfloat16* Cb, int ldc) {
    cudaError_t e = gemm_on<A_T, B_T, EPI>(m->engine, m->stream, M, N, K, A, lda, B, ldb, bias, Cf, Cb, ldc);
    if (e != cudaSuccess && m->err.empty()) m->err = std::string("gemm launch: ") + cudaGetErrorString(e);
}

// Waits for the stream; then the losses of the last n batches into losses[n],
// and the tensor-core GEMM error flag (an mbarrier wait that expired), read
// and cleared, where `tc`.
static lf_status finish(lf_mlp* m, int n, float* losses, bool tc) {
    unsigned int flag = 0;
    float* h_flag = m->h_loss + (size_t)kQueued * m->n_loss;
    if (losses)
        MLP_TRY(m, cudaMemcpyAsync(m->h_loss, m->loss_blocks.p, sizeof(float) * n * m->n_loss, cudaMemcpyDeviceToHost,
                                   m->stream));
    if (tc)
        MLP_TRY(m, cudaMemcpyFromSymbolAsync(h_flag, g_tc_gemm_error, sizeof(flag), 0, cudaMemcpyDeviceToHost,
                                             m->stream));
    MLP_TRY(m, cudaStreamSynchronize(m->stream));
    for (int b = 0; losses && b < n; ++b) {
        double s = 0.0;
        for (int i = 0; i < m->n_loss; ++i) s += m->h_loss[(size_t)b * m->n_loss + i];
        losses[b] = static_cast<float>(s);
    }
    if (tc) std::memcpy(&flag, h_flag, sizeof(flag));
    if (flag) {
        const unsigned int zero = 0;
        MLP_TRY(m, cudaMemcpyToSymbol(g_tc_gemm_error, &zero, sizeof(zero)));
        m->err = "tensor-core GEMM: an mbarrier wait expired";
        return LF_ETIMEOUT;
    }
    return LF_OK;
}

extern "C" lf_status lf_mlp_create(int device, int n_in, int width, int depth, int n_out, int batch, unsigned seed,
                                   lf_mlp** out) {
    if (!out) return LF_EINVAL;
    *out = nullptr;
    if (n_in <= 0 || width <= 0 || width % 128 != 0 || depth < 1 || n_out <= 0 || batch <= 0 || batch % 128 != 0)
        return LF_EINVAL;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        return LF_ECUDA;
    }
    auto* m = new (std::nothrow) lf_mlp();
    if (!m) return LF_ENOMEM;
    m->device = device;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete m;
        return LF_ECUDA;
    }
    m->n_in = n_in;
    m->n_in_pad = pad128(n_in);
    m->width = pad128(width);
    m->depth = depth;
    m->n_out = n_out;
    m->n_out_pad = pad128(n_out);
    m->batch = batch;
    m->layers.resize(depth + 1);
    std::mt19937_64 rng(seed);
    lf_status st = LF_OK;
    for (int l = 0; l <= depth && st == LF_OK; ++l) {
        Layer& L = m->layers[l];
        L.in = l == 0 ? m->n_in_pad : m->width;
        L.out = l == depth ? m->n_out_pad : m->width;
        const int in_real = l == 0 ? n_in : width, out_real = l == depth ? n_out : width;
        const size_t nw = (size_t)L.in * L.out;
        // He initialisation for ReLU layers (N(0, 2/fan_in)); the output layer
        // starts small; padded rows/columns stay zero
        std::vector<float> w(nw, 0.f);
        std::normal_distribution<float> nd(0.f, std::sqrt(2.f / in_real) * (l == depth ? 0.1f : 1.f));
        for (int o = 0; o < out_real; ++o)
            for (int i = 0; i < in_real; ++i) w[(size_t)o * L.in + i] = nd(rng);
        std::vector<__nv_bfloat16> wb(nw);
        for (size_t i = 0; i < nw; ++i) wb[i] = __float2bfloat16(w[i]);
        cudaError_t e = cudaSuccess;
        for (Buf<float>* b : {&L.w, &L.gw, &L.mw, &L.vw})
            if (e == cudaSuccess) e = b->alloc(nw);
        for (Buf<float>* b : {&L.b, &L.gb, &L.mb, &L.vb})
            if (e == cudaSuccess) e = b->alloc(L.out);
        if (e == cudaSuccess) e = L.wb.alloc(nw);
        if (e == cudaSuccess && l < depth) e = L.act.alloc((size_t)batch * L.out);
        if (e == cudaSuccess) e = L.dz.alloc((size_t)batch * L.out);
        if (e == cudaSuccess) e = cudaMemcpy(L.w.p, w.data(), nw * sizeof(float), cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(L.wb.p, wb.data(), nw * sizeof(__nv_bfloat16), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) st = LF_ECUDA;
    }
    if (st == LF_OK) {
        m->n_loss = cdiv_i((long long)batch * m->n_out_pad, 256);
        if (m->xb.alloc((size_t)batch * m->n_in_pad) != cudaSuccess ||
            m->pred.alloc((size_t)batch * m->n_out_pad) != cudaSuccess ||
            m->loss_blocks.alloc((size_t)kQueued * m->n_loss) != cudaSuccess ||
            m->rows.alloc((size_t)kQueued * batch) != cudaSuccess ||
            cudaMallocHost(&m->h_loss, sizeof(float) * ((size_t)kQueued * m->n_loss + 1)) != cudaSuccess ||
            cudaMallocHost(&m->h_rows, sizeof(long long) * (size_t)kQueued * batch) != cudaSuccess)
            st = LF_ECUDA;
    }
    if (st != LF_OK) {
        lf_mlp_destroy(m);
        return st;
    }
    *out = m;
    return LF_OK;
}

extern "C" void lf_mlp_destroy(lf_mlp* m) {
    if (!m) return;
    cudaSetDevice(m->device);
    cudaStreamSynchronize(m->stream);
    cudaStreamDestroy(m->stream);
    if (m->h_loss) cudaFreeHost(m->h_loss);
    if (m->h_rows) cudaFreeHost(m->h_rows);
    delete m;
}

extern "C" const char* lf_mlp_last_error(lf_mlp* m) { return m ? m->err.c_str() : "null network"; }

// The batch's input, n rows of d_x [][n_in] fp32 (device), the given ones or
// the first -> padded bf16 [batch][n_in_pad].
static lf_status load_input(lf_mlp* m, const float* d_x, int n, const long long* d_rows = nullptr) {
    const bool vec = m->n_in % 4 == 0 && reinterpret_cast<uintptr_t>(d_x) % 16 == 0;
    launch_next(k_load_input, cdiv_i((long long)m->batch * m->n_in_pad, 4 * 256), 256, 0, m->stream, n, m->batch,
                m->n_in, m->n_in_pad, vec, d_x, d_rows, m->xb.p);
    return mlp_check_launch(m);
}

static lf_status forward(lf_mlp* m) {
    const __nv_bfloat16* x = m->xb.p;
    for (int l = 0; l <= m->depth; ++l) {
        Layer& L = m->layers[l];
        if (l < m->depth) {
            gemm<false, true, EPI_BIAS_RELU>(m, m->batch, L.out, L.in, x, L.in, L.wb.p, L.in, L.b.p, nullptr, L.act.p,
                                            L.out);
            x = L.act.p;
        } else {
            gemm<false, true, EPI_BIAS_F32>(m, m->batch, L.out, L.in, x, L.in, L.wb.p, L.in, L.b.p, m->pred.p, nullptr,
                                           L.out);
        }
    }
    return mlp_check_launch(m);
}

static bool on_mma(const lf_mlp* m, int M, int N, int K) {
    return m->engine == LF_GEMM_MMA_SYNC || (m->engine == LF_GEMM_AUTO && auto_engine(M, N, K) == LF_GEMM_MMA_SYNC);
}

// Loss (blocks of queue slot `slot`) and parameter gradients for one batch
// (targets: rows of d_y [][n_out] fp32, the given ones or the first); with
// `update` the gradients go straight into the Adam step.
static lf_status backward(lf_mlp* m, const float* d_y, const Adam* update, const long long* d_rows = nullptr,
                          int slot = 0) {
    launch_next(k_mse, m->n_loss, 256, 0, m->stream, m->batch, m->n_out_pad, m->n_out, m->pred.p, d_y, d_rows, m->n_out,
                m->layers[m->depth].dz.p, m->loss_blocks.p + (size_t)slot * m->n_loss);
    for (int l = m->depth; l > 0; --l) {
        // dZ below: dH [batch][in] = dZ W (A = dZ [batch][out], B = W [out][in] = [K][N]), through the ReLU
        Layer &L = m->layers[l], &P = m->layers[l - 1];
        if (on_mma(m, m->batch, L.in, L.out)) {
            gemm_mma<false, false, EPI_BF16_RELU_BWD>(m->stream, m->batch, L.in, L.out, L.dz.p, L.out, L.wb.p, L.in,
                                                      nullptr, nullptr, P.dz.p, L.in, P.act.p);
        } else {
            gemm<false, false, EPI_BF16>(m, m->batch, L.in, L.out, L.dz.p, L.out, L.wb.p, L.in, nullptr, nullptr,
                                         P.dz.p, L.in);
            const size_t n = (size_t)m->batch * L.in;
            k_relu_bwd<<<cdiv_i(n, 256), 256, 0, m->stream>>>(n, P.act.p, P.dz.p);
        }
    }
    bool grouped = true;
    for (const Layer& L : m->layers) grouped = grouped && on_mma(m, L.out, L.in, m->batch);
    if (grouped) {
        for (int l0 = 0; l0 <= m->depth; l0 += kGradLayers) {
            LayerGrads G{};
            G.n = std::min(kGradLayers, m->depth + 1 - l0);
            int blocks = 0;
            for (int l = 0; l < G.n; ++l) {
                Layer& L = m->layers[l0 + l];
                G.layer[l] = {L.dz.p, l0 + l == 0 ? m->xb.p : m->layers[l0 + l - 1].act.p, L.w.p, L.gw.p, L.mw.p,
                              L.vw.p, L.b.p, L.gb.p, L.mb.p, L.vb.p, L.wb.p, L.in, L.out, blocks};
                blocks += (L.in / 64) * (L.out / 64) + L.out / 32;
            }
            launch_next(update ? k_layer_grads<true> : k_layer_grads<false>, blocks, MmaShape<64>::kThreads, 0,
                        m->stream, G, m->batch, update ? *update : Adam{});
        }
    } else {
        for (int l = m->depth; l >= 0; --l) {
            Layer& L = m->layers[l];
            const __nv_bfloat16* xin = l == 0 ? m->xb.p : m->layers[l - 1].act.p;
            // dW [out][in] = dZ^T X: A = dZ stored [batch][out] = [K][M]; B = X [batch][in] = [K][N]
            gemm<true, false, EPI_F32>(m, L.out, L.in, m->batch, L.dz.p, L.out, xin, L.in, nullptr, L.gw.p, nullptr,
                                       L.in);
            k_colsum<<<L.out / 32, 128, 0, m->stream>>>(m->batch, L.out, L.dz.p, L.gb.p);
            if (!update) continue;
            const size_t nw = (size_t)L.in * L.out;
            k_adam<<<cdiv_i(nw, 256), 256, 0, m->stream>>>(nw, L.w.p, L.gw.p, L.mw.p, L.vw.p, *update, L.wb.p);
            k_adam<<<cdiv_i(L.out, 256), 256, 0, m->stream>>>(L.out, L.b.p, L.gb.p, L.mb.p, L.vb.p, *update, nullptr);
        }
    }
    return mlp_check_launch(m);
}

// Whether no GEMM of a training step runs on the tcgen05 kernels.
static bool trains_on_mma(const lf_mlp* m) {
    for (const Layer& L : m->layers)
        if (!on_mma(m, m->batch, L.out, L.in) || !on_mma(m, m->batch, L.in, L.out) || !on_mma(m, L.out, L.in, m->batch))
            return false;
    return true;
}

// Queues one training step.
static lf_status queue_step(lf_mlp* m, const float* d_x, const float* d_y, const long long* d_rows, int slot,
                            float lr) {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float t = (float)(m->step + 1);
    const Adam adam{lr, b1, b2, eps, 1.f - std::pow(b1, t), 1.f - std::pow(b2, t)};
    lf_status st = load_input(m, d_x, m->batch, d_rows);
    if (st == LF_OK) st = forward(m);
    if (st == LF_OK) st = backward(m, d_y, &adam, d_rows, slot);
    if (st == LF_OK) ++m->step;
    return st;
}

extern "C" lf_status lf_mlp_train_step(lf_mlp* m, const float* d_x, const float* d_y, float lr, float* loss) {
    if (!m || !d_x || !d_y || !(lr > 0.f)) return LF_EINVAL;
    cudaSetDevice(m->device);
    const lf_status st = queue_step(m, d_x, d_y, nullptr, 0, lr);
    const bool tc = m->engine != LF_GEMM_MMA_SYNC;
    return st == LF_OK && (loss || tc) ? finish(m, 1, loss, tc) : st;
}

extern "C" lf_status lf_mlp_train_rows(lf_mlp* m, const float* d_x, const float* d_y, long long n_rows,
                                       const long long* rows, int n_batches, float lr, float* losses) {
    if (!m || !d_x || !d_y || n_rows < 0 || n_batches < 0 || (n_batches > 0 && (!rows || !losses)) || !(lr > 0.f))
        return LF_EINVAL;
    for (long long i = 0; i < (long long)n_batches * m->batch; ++i)
        if (rows[i] < 0 || rows[i] >= n_rows) return LF_EINVAL;
    cudaSetDevice(m->device);
    // A tcgen05 product may give up on a wait: its batch is the last one then, as
    // in single steps, so such networks are checked after every batch (their
    // steps take far longer than the 20 us of a check).
    const int queue = trains_on_mma(m) ? kQueued : 1;
    for (int b0 = 0; b0 < n_batches; b0 += queue) {
        const int nb = std::min(queue, n_batches - b0);
        const size_t n = (size_t)nb * m->batch;
        std::memcpy(m->h_rows, rows + (size_t)b0 * m->batch, sizeof(long long) * n);
        MLP_TRY(m, cudaMemcpyAsync(m->rows.p, m->h_rows, sizeof(long long) * n, cudaMemcpyHostToDevice, m->stream));
        lf_status st = LF_OK;
        for (int b = 0; b < nb && st == LF_OK; ++b)
            st = queue_step(m, d_x, d_y, m->rows.p + (size_t)b * m->batch, b, lr);
        const lf_status done = finish(m, nb, losses + b0, m->engine != LF_GEMM_MMA_SYNC);  // always: h_rows is reused
        if (st != LF_OK || done != LF_OK) return st != LF_OK ? st : done;
    }
    return LF_OK;
}

extern "C" lf_status lf_mlp_predict(lf_mlp* m, const float* d_x, int rows, float* d_y) {
    if (!m || rows < 0 || (rows > 0 && (!d_x || !d_y))) return LF_EINVAL;
    cudaSetDevice(m->device);
    for (int r0 = 0; r0 < rows; r0 += m->batch) {
        const int nr = std::min(m->batch, rows - r0);
        lf_status st = load_input(m, d_x + (size_t)r0 * m->n_in, nr);
        if (st == LF_OK) st = forward(m);
        if (st != LF_OK) return st;
        MLP_TRY(m, cudaMemcpy2DAsync(d_y + (size_t)r0 * m->n_out, sizeof(float) * m->n_out, m->pred.p,
                                     sizeof(float) * m->n_out_pad, sizeof(float) * m->n_out, nr,
                                     cudaMemcpyDeviceToDevice, m->stream));
    }
    return finish(m, 0, nullptr, m->engine != LF_GEMM_MMA_SYNC);
}

// Parameters in the unpadded order: for each layer W [out][in] then b [out].
static size_t param_count(const lf_mlp* m) {
    size_t n = 0;
    for (int l = 0; l <= m->depth; ++l) {
        const int in = l == 0 ? m->n_in : (m->width), out = l == m->depth ? m->n_out : m->width;
        n += (size_t)in * out + out;
    }
    return n;
}

extern "C" lf_status lf_mlp_param_count(lf_mlp* m, size_t* n) {
    if (!m || !n) return LF_EINVAL;
    *n = param_count(m);
    return LF_OK;
}

// which: 0 weights, 1 gradients of the last lf_mlp_gradients.
static lf_status copy_params(lf_mlp* m, int which, float* host) {
    size_t k = 0;
    for (int l = 0; l <= m->depth; ++l) {
        Layer& L = m->layers[l];
        const int in = l == 0 ? m->n_in : m->width, out = l == m->depth ? m->n_out : m->width;
        const float* w = which == 0 ? L.w.p : L.gw.p;
        const float* b = which == 0 ? L.b.p : L.gb.p;
        MLP_TRY(m, cudaMemcpy2DAsync(host + k, sizeof(float) * in, w, sizeof(float) * L.in, sizeof(float) * in, out,
                                     cudaMemcpyDeviceToHost, m->stream));
        k += (size_t)in * out;
        MLP_TRY(m, cudaMemcpyAsync(host + k, b, sizeof(float) * out, cudaMemcpyDeviceToHost, m->stream));
        k += out;
    }
    MLP_TRY(m, cudaStreamSynchronize(m->stream));
    return LF_OK;
}

extern "C" lf_status lf_mlp_get_params(lf_mlp* m, float* host) {
    if (!m || !host) return LF_EINVAL;
    cudaSetDevice(m->device);
    return copy_params(m, 0, host);
}

extern "C" lf_status lf_mlp_set_params(lf_mlp* m, const float* host) {
    if (!m || !host) return LF_EINVAL;
    cudaSetDevice(m->device);
    size_t k = 0;
    for (int l = 0; l <= m->depth; ++l) {
        Layer& L = m->layers[l];
        const int in = l == 0 ? m->n_in : m->width, out = l == m->depth ? m->n_out : m->width;
        std::vector<float> w((size_t)L.in * L.out, 0.f);
        for (int o = 0; o < out; ++o)
            std::memcpy(&w[(size_t)o * L.in], host + k + (size_t)o * in, sizeof(float) * in);
        k += (size_t)in * out;
        std::vector<__nv_bfloat16> wb(w.size());
        for (size_t i = 0; i < w.size(); ++i) wb[i] = __float2bfloat16(w[i]);
        std::vector<float> b(L.out, 0.f);
        std::memcpy(b.data(), host + k, sizeof(float) * out);
        k += out;
        MLP_TRY(m, cudaMemcpy(L.w.p, w.data(), sizeof(float) * w.size(), cudaMemcpyHostToDevice));
        MLP_TRY(m, cudaMemcpy(L.wb.p, wb.data(), sizeof(__nv_bfloat16) * wb.size(), cudaMemcpyHostToDevice));
        MLP_TRY(m, cudaMemcpy(L.b.p, b.data(), sizeof(float) * b.size(), cudaMemcpyHostToDevice));
        for (Buf<float>* z : {&L.mw, &L.vw, &L.mb, &L.vb})
            MLP_TRY(m, cudaMemset(z->p, 0, sizeof(float) * z->n));
    }
    m->step = 0;
    return LF_OK;
}

// Loss and parameter gradients (no update) of one batch, gradients in the
// parameter order of lf_mlp_get_params.
extern "C" lf_status lf_mlp_gradients(lf_mlp* m, const float* d_x, const float* d_y, float* loss, float* host_grads) {
    if (!m || !d_x || !d_y) return LF_EINVAL;
    cudaSetDevice(m->device);
    lf_status st = load_input(m, d_x, m->batch);
    if (st == LF_OK) st = forward(m);
    if (st == LF_OK) st = backward(m, d_y, nullptr);
    if (st == LF_OK) st = finish(m, 1, loss, m->engine != LF_GEMM_MMA_SYNC);
    if (st == LF_OK && host_grads) st = copy_params(m, 1, host_grads);
    return st;
}

extern "C" lf_status lf_set_device_wait_limit(long long polls) {
    const long long v = polls < 0 ? kTcWaitLimit : polls;
    return cudaMemcpyToSymbol(g_tc_stage_wait_limit, &v, sizeof(v)) == cudaSuccess ? LF_OK : LF_ECUDA;
}

extern "C" lf_status lf_mlp_set_engine(lf_mlp* m, int engine) {
    if (!m || (engine != LF_GEMM_TCGEN05 && engine != LF_GEMM_MMA_SYNC && engine != LF_GEMM_TCGEN05_TMA &&
               engine != LF_GEMM_AUTO))
        return LF_EINVAL;
    m->engine = engine;
    return LF_OK;
}

extern "C" lf_status lf_gemm_bf16(int engine, int a_trans, int b_trans, int epilogue, int M, int N, int K,
                                  const void* A, int lda, const void* B, int ldb, const float* bias, void* C, int ldc,
                                  void* stream) {
    if (engine == LF_GEMM_AUTO) engine = auto_engine(M, N, K);
    const bool tc = engine == LF_GEMM_TCGEN05 || engine == LF_GEMM_TCGEN05_TMA;
    if ((!tc && engine != LF_GEMM_MMA_SYNC) || M <= 0 || N <= 0 || K <= 0 || M % kBM ||
        N % kBN || K % (tc ? kTcBK : kBK) || !A || !B || !C ||
        (epilogue != EPI_F32 && epilogue != EPI_BF16 && epilogue != EPI_BIAS_RELU && epilogue != EPI_BIAS_F32) ||
        ((epilogue == EPI_BIAS_RELU || epilogue == EPI_BIAS_F32) && !bias) || lda % 8 || ldb % 8 || ldc % 2 ||
        (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) % 16)
        return LF_EINVAL;
    // minimum row lengths of the stored operands
    if (lda < (a_trans ? M : K) || ldb < (b_trans ? K : N) || ldc < N) return LF_EINVAL;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const auto* a = static_cast<const __nv_bfloat16*>(A);
    const auto* b = static_cast<const __nv_bfloat16*>(B);
    float* cf = static_cast<float*>(C);
    __nv_bfloat16* cb = static_cast<__nv_bfloat16*>(C);
    cudaError_t e = cudaSuccess;
#define LF_GEMM_CASE(AT, BT)                                                                                          \
    if (!!a_trans == AT && !!b_trans == BT) {                                                                        \
        switch (epilogue) {                                                                                          \
        case EPI_F32: e = gemm_on<AT, BT, EPI_F32>(engine, st, M, N, K, a, lda, b, ldb, bias, cf, nullptr, ldc); break; \
        case EPI_BF16: e = gemm_on<AT, BT, EPI_BF16>(engine, st, M, N, K, a, lda, b, ldb, bias, nullptr, cb, ldc); break; \
        case EPI_BIAS_RELU:                                                                                          \
            e = gemm_on<AT, BT, EPI_BIAS_RELU>(engine, st, M, N, K, a, lda, b, ldb, bias, nullptr, cb, ldc);          \
            break;                                                                                                   \
        default: e = gemm_on<AT, BT, EPI_BIAS_F32>(engine, st, M, N, K, a, lda, b, ldb, bias, cf, nullptr, ldc); break; \
        }                                                                                                            \
    }
    LF_GEMM_CASE(false, false)
    LF_GEMM_CASE(false, true)
    LF_GEMM_CASE(true, false)
    LF_GEMM_CASE(true, true)
#undef LF_GEMM_CASE
    if (e != cudaSuccess) return LF_ECUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return LF_ECUDA;
    if (tc) {
        unsigned int flag = 0;
        if (cudaMemcpyFromSymbol(&flag, g_tc_gemm_error, sizeof(flag)) != cudaSuccess) return LF_ECUDA;
        if (flag) {
            const unsigned int zero = 0;
            cudaMemcpyToSymbol(g_tc_gemm_error, &zero, sizeof(zero));
            return LF_ETIMEOUT;
        }
    }
    return LF_OK;
}
