// lf_forward_noalloc: the single-body gz + TMI forward for callers that
// cannot allocate device memory.
//
// Who needs it: code that runs where cudaMalloc is unavailable or forbidden --
// inside a host framework that owns every device allocation through its own
// pool, in a process whose memory budget is fixed up front, or in a plugin
// called from a real-time loop that must not allocate.  Such callers already
// hold their inputs and outputs in device memory and pass those pointers in.
//
// What it uses instead of allocations: one file-scope __device__ scratch array
// of kNoallocScratchBytes (8 MiB).  Every GPU that loads this library holds it
// until the process exits.  The library looks up its device address once per
// device with cudaGetSymbolAddress, on the first call made on that device, and
// keeps it for the life of the process: a cudaDeviceReset of that device
// invalidates the kept address, so calling this entry point after a device
// reset is not supported.  All calls share the array and every call
// overwrites the regions it reads (nothing in it has to start at zero), except
// the error flag, which each call clears first; calls that overlap on the GPU
// (two streams, two threads) race on it: serialise them.
//
// Every call reads its error flag back into host memory and waits for its
// stream, neither of which is legal while the stream is being captured into a
// CUDA graph: the entry point refuses a capturing stream (LF_EINVAL) instead of
// invalidating the caller's capture.  An error already pending on the calling
// thread when the call starts (a failed launch of the caller's own) is left in
// place and reported as LF_ECUDA before any work is queued.
//
// The kernels are the library's FP64 forward (facet constants, station-tiled
// pair kernel, chunk reduction) specialised to one group.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <mutex>

#include "../../include/litho_gpu.h"

namespace {
#include "kernels_fp64.cuh"
}  // namespace

namespace {

constexpr size_t kNoallocScratchBytes = size_t(8) << 20;
constexpr size_t kNoallocScratchDoubles = kNoallocScratchBytes / sizeof(double);
constexpr int kMaxDevices = 64;

// The only scratch this entry point uses.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocScratchBytes];

std::mutex g_mutex;
void* g_scratch_addr[kMaxDevices] = {nullptr};

// Device address of g_noalloc_scratch on `dev` (looked up once per device,
// with that device current).
cudaError_t scratch_address(int dev, double** out) {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_scratch_addr[dev] = p;
    }
    *out = static_cast<double*>(g_scratch_addr[dev]);
    return cudaSuccess;
}

struct SingleGroup {
    double gscale;  // G * rho * 1e3 * 1e5
    double mscale;  // amp * 100 / (4 pi)
    litho_b200::d3 mdir, fdir;
};

// Facet constants of one group; triangle indices are bounds-checked against
// nv (a bad facet is marked invalid and raises the error flag).
__global__ void k_na_prep(int nv, const double* __restrict__ xyz, int nt, const int32_t* __restrict__ tri,
                          SingleGroup g, double* __restrict__ fc, int* __restrict__ err) {
    using namespace litho_b200;
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nt) return;
    int ia = tri[3 * f], ib = tri[3 * f + 1], ic = tri[3 * f + 2];
    double out[NFC];
    if (ia < 0 || ia >= nv || ib < 0 || ib >= nv || ic < 0 || ic >= nv) {
        atomicExch(err, 1);
        for (int k = 0; k < NFC; ++k) out[k] = 0.0;
        out[FC_AREA2] = -1.0;
    } else {
        const d3 v[3] = {mk3(xyz[3 * ia], xyz[3 * ia + 1], xyz[3 * ia + 2]),
                         mk3(xyz[3 * ib], xyz[3 * ib + 1], xyz[3 * ib + 2]),
                         mk3(xyz[3 * ic], xyz[3 * ic + 1], xyz[3 * ic + 2])};
        face_consts_fwd(v, g.mdir, g.fdir, out);
    }
    store_face_fwd(out, fc + (size_t)f * NFC);
}

// Station-tiled pair kernel over uniform facet chunks of `cs` facets.
template <int FT>
__global__ void __launch_bounds__(128) k_na_forward(int ns, const double* __restrict__ sta, int nt, int cs,
                                                    const double* __restrict__ fc, double* __restrict__ part_gz,
                                                    double* __restrict__ part_tmi) {
    using namespace litho_b200;
    __shared__ __align__(16) double sm[NFC * FT];
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    int chunk = blockIdx.y;
    int fb = chunk * cs, fe = min(nt, fb + cs);
    forward_fp64_block<true, true, FT>(sm, s, s < ns, sta, fc, fb, fe, part_gz + (size_t)chunk * ns,
                                       part_tmi + (size_t)chunk * ns);
}

__global__ void k_na_reduce(int ns, int nch, const double* __restrict__ part_gz, const double* __restrict__ part_tmi,
                            SingleGroup g, double* __restrict__ gz, double* __restrict__ tmi) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= ns) return;
    double tg = 0.0, tt = 0.0;
    for (int c = 0; c < nch; ++c) {
        tg += part_gz[(size_t)c * ns + s];
        tt += part_tmi[(size_t)c * ns + s];
    }
    if (gz) gz[s] = tg * g.gscale;
    if (tmi) tmi[s] = -g.mscale * tt;
}

}  // namespace

extern "C" lf_status lf_forward_noalloc(int nv, const double* d_xyz, int nt, const int32_t* d_tri, int ns,
                                        const double* d_sta, double density_gcc, double susceptibility_si,
                                        double inc_deg, double dec_deg, double field_nt, double* d_gz,
                                        double* d_tmi, void* stream) {
    if (nv < 3 || nt < 1 || ns < 1 || !d_xyz || !d_tri || !d_sta || (!d_gz && !d_tmi)) return LF_EINVAL;
    if (!std::isfinite(density_gcc) || !std::isfinite(susceptibility_si) || !std::isfinite(inc_deg) ||
        !std::isfinite(dec_deg) || !std::isfinite(field_nt))
        return LF_EINVAL;
    // Scratch layout (doubles): [0, 32) error flag and padding, 38 per facet
    // (the documented limit; its record takes the first NFC * nt of them),
    // then gz and TMI chunk partials 2 * nch * ns.
    const size_t head = 32;
    static_assert(litho_b200::NFC <= 38, "the documented size limit counts 38 doubles per facet");
    const size_t fcSize = (size_t)38 * nt;
    if (head + fcSize + 2 * (size_t)ns > kNoallocScratchDoubles) return LF_EINVAL;
    const size_t room = (kNoallocScratchDoubles - head - fcSize) / (2 * (size_t)ns);
    int sBlocks = (ns + 127) / 128;
    int wantChunks = (148 * 4 + sBlocks - 1) / sBlocks;
    int cs = (nt + wantChunks - 1) / wantChunks;
    if (cs < 64) cs = 64;
    int nch = (nt + cs - 1) / cs;
    if ((size_t)nch > room) {
        nch = static_cast<int>(room);
        cs = (nt + nch - 1) / nch;
        nch = (nt + cs - 1) / cs;
    }
    // An error left pending by earlier work of the caller is theirs: report it
    // without clearing it, before queueing anything.
    if (cudaPeekAtLastError() != cudaSuccess) return LF_ECUDA;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) return LF_ECUDA;
    if (cap != cudaStreamCaptureStatusNone) return LF_EINVAL;  // host read-back and sync cannot be captured
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return LF_ECUDA;
    double* base = nullptr;
    if (scratch_address(dev, &base) != cudaSuccess) return LF_ECUDA;
    int* err = reinterpret_cast<int*>(base);
    double* fc = base + head;
    double* partG = fc + fcSize;
    double* partM = partG + (size_t)nch * ns;

    // magnetisation and scales as MagneticForward / GravityForward build them
    const double pi = litho_b200::kPi;
    double I = inc_deg * pi / 180.0, D = dec_deg * pi / 180.0, cI = std::cos(I);
    SingleGroup g;
    g.fdir = {cI * std::cos(D), cI * std::sin(D), -std::sin(I)};
    double amp = std::fabs(susceptibility_si * field_nt / 100.0);
    g.mdir = (susceptibility_si * field_nt / 100.0 < 0.0) ? litho_b200::d3{-g.fdir.x, -g.fdir.y, -g.fdir.z} : g.fdir;
    if (amp < litho_b200::kEps) g.mdir = g.fdir;
    g.mscale = amp * 100.0 / (4.0 * pi);
    g.gscale = 6.67430e-11 * density_gcc * 1000.0 * 1e5;

    if (cudaMemsetAsync(err, 0, sizeof(int), st) != cudaSuccess) return LF_ECUDA;
    k_na_prep<<<(nt + 127) / 128, 128, 0, st>>>(nv, d_xyz, nt, d_tri, g, fc, err);
    dim3 grid(sBlocks, nch);
    k_na_forward<32><<<grid, 128, 0, st>>>(ns, d_sta, nt, cs, fc, partG, partM);
    k_na_reduce<<<(ns + 255) / 256, 256, 0, st>>>(ns, nch, partG, partM, g, d_gz, d_tmi);
    if (cudaGetLastError() != cudaSuccess) return LF_ECUDA;
    int hErr = 0;
    if (cudaMemcpyAsync(&hErr, err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess) return LF_ECUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return LF_ECUDA;
    return hErr ? LF_EINVAL : LF_OK;
}
