// bt_step_noalloc: one step of the reference update that performs no device
// allocation at all.
//
// Who needs this: callers that may not call cudaMalloc — code that runs while
// a CUDA stream is being captured into a graph (allocation is not a stream
// operation and breaks the capture), host applications whose framework has
// already reserved (almost) all device memory for its own pool, and
// plugin hosts that forbid libraries from allocating behind their back. Such a
// caller owns every input and output buffer and passes them in; this entry
// point needs no handle and allocates nothing.
//
// The step itself is the library's generic update (single_step_kernel,
// bt_step_single.cuh: the arithmetic of the kernels that the handle-based API
// runs for FP64 and for steps that carry pulses). Its scratch, the per-CTA sums
// of M(t), lives in the file-scope array below instead of in memory allocated by
// bt_create. Every GPU that loads the library holds that array until the process
// exits.
//
// Sharing: all calls on a device use the same array. Each call writes what its
// second kernel reads, so sequential calls are independent. Calls whose kernels
// overlap on the GPU (different streams, or different host threads, without
// ordering between them) race on the array and give wrong results: order them on
// one stream.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>

#include <cudaTypedefs.h>

#include "../../include/bt.h"
#include "bt_internal.h"

namespace {

constexpr size_t SCRATCH_BYTES = 3 * sizeof(double) * bt::SINGLE_CTAS;

// The scratch of every allocation-free call on this device (58 KB).
static __device__ __align__(256) unsigned char g_noalloc_scratch[SCRATCH_BYTES];

constexpr int MAX_DEVICES = 64;
std::mutex g_setup_mutex;
// per device: the device address of the array and the id of the context it
// was looked up in (a cudaDeviceReset ends that context; the module is loaded
// again in the next one and the array may move)
unsigned char* g_scratch_addr[MAX_DEVICES] = {};
unsigned long long g_scratch_ctx[MAX_DEVICES] = {};

// unique id of the calling thread's current context (0 when there is none or
// the driver cannot say)
unsigned long long current_context_id() {
    static PFN_cuCtxGetCurrent_v4000 get_current = nullptr;
    static PFN_cuCtxGetId_v12000 get_id = nullptr;
    static bool looked = false;
    if (!looked) {
        cudaDriverEntryPointQueryResult q;
        void* p = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 4000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<PFN_cuCtxGetCurrent_v4000>(p);
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<PFN_cuCtxGetId_v12000>(p);
        looked = true;
    }
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS)
        return 0;
    return id;
}

// Set-up, once per device and context, with that device current: the
// host-side name of a __device__ array is only a stand-in; the address a
// kernel may use comes from cudaGetSymbolAddress (which also creates the
// device's context on a first call).
// The look-up is not a stream operation; a call whose look-up would fall
// inside a stream capture is refused (cudaErrorStreamCaptureUnsupported), so
// the rule that the first call on a device precedes any capture is enforced.
cudaError_t scratch_for_current_device(cudaStream_t stream, unsigned char** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    const unsigned long long ctx = current_context_id();
    if (!g_scratch_addr[dev] || ctx == 0 || ctx != g_scratch_ctx[dev]) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone)
            return cudaErrorStreamCaptureUnsupported;
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_scratch_addr[dev] = static_cast<unsigned char*>(p);
        g_scratch_ctx[dev] = current_context_id();
    }
    *out = g_scratch_addr[dev];
    return cudaSuccess;
}

template <typename T>
void fill(const bt_config& c, bt::StepParams<T>& P, const void* const in[3], void* const out[3], const void* vx,
          const void* vy, const void* vz, unsigned char* scratch, double* sums) {
    constexpr double SMALL = 1.0e-50;
    std::memset(&P, 0, sizeof(P));
    P.nx = c.nx; P.ny = c.ny; P.nz = c.nz;
    for (int k = 0; k < 3; ++k) {
        P.in[k] = static_cast<const T*>(in[k]);
        P.out[k] = static_cast<T*>(out[k]);
    }
    P.vx = static_cast<const T*>(vx);
    P.vy = static_cast<const T*>(vy);
    P.vz = static_cast<const T*>(vz);
    const double dTime = c.dt;
    P.hx = (T)(dTime / c.dx); P.hy = (T)(dTime / c.dy); P.hz = (T)(dTime / c.dz);
    P.hxx = (T)(dTime / (c.dx * c.dx)); P.hyy = (T)(dTime / (c.dy * c.dy)); P.hzz = (T)(dTime / (c.dz * c.dz));
    const double Bx = c.main_field[0], By = c.main_field[1], Bz = c.main_field[2];
    const double anb = std::sqrt(Bx * Bx + By * By + Bz * Bz);
    const double an[3] = {Bx / anb, By / anb, Bz / anb};
    for (int k = 0; k < 3; ++k) {
        P.an[k] = (T)an[k];
        P.peqn[k] = (T)(c.p_eq * an[k]);
    }
    P.axis = -1;
    for (int k = 0; k < 3; ++k)
        if (an[k] == 1.0 && an[(k + 1) % 3] == 0.0 && an[(k + 2) % 3] == 0.0) P.axis = k;
    P.b = (T)(dTime * c.gamma);
    P.dx = (T)c.dx; P.dy = (T)c.dy; P.dz = (T)c.dz;
    const double D = c.d_pore;
    P.dpp = (T)(2.0 * (D * D) / (D + D + SMALL));
    P.dps = (T)(2.0 * (SMALL * D) / (SMALL + D + SMALL));
    for (int f = 0; f < 64; ++f) {
        double ct1 = 1.0 / c.t1, ct2 = 1.0 / c.t2;
        const double d3[3] = {c.dx, c.dy, c.dz};
        for (int b = 0; b < 6; ++b)
            if (f & (1 << b)) {
                ct1 += c.rho1 / d3[b / 2];
                ct2 += c.rho2 / d3[b / 2];
            }
        P.dtt1[f] = (T)(dTime * (1.0 / (1.0 / ct1)));
        P.dtt2[f] = (T)(dTime * (1.0 / (1.0 / ct2)));
    }
    P.diffusion = c.diffusion ? 1 : 0;
    P.box[0] = c.buffer[0]; P.box[1] = c.nx - c.buffer[0];
    P.box[2] = c.buffer[1]; P.box[3] = c.ny - c.buffer[1];
    P.box[4] = c.buffer[2]; P.box[5] = c.nz - c.buffer[2];
    P.dxd = c.dx; P.dyd = c.dy; P.dzd = c.dz;
    P.partials = reinterpret_cast<double*>(scratch);
    P.mt = sums;
}

}  // namespace

extern "C" int bt_step_noalloc(const bt_config* cfg, const uint8_t* mask, const void* vx, const void* vy,
                               const void* vz, const void* mx_in, const void* my_in, const void* mz_in, void* mx_out,
                               void* my_out, void* mz_out, double* sums, void* stream) {
    if (!cfg || !mask || !mx_in || !my_in || !mz_in || !mx_out || !my_out || !mz_out || !sums) return BT_E_ARG;
    const bt_config& c = *cfg;
    if (c.scheme != BT_SCHEME_REFERENCE || (c.precision != BT_F32 && c.precision != BT_F64)) return BT_E_ARG;
    if (c.nx <= 0 || c.ny <= 0 || c.nz <= 0 || !(c.dt > 0) || !(c.dx > 0) || !(c.dy > 0) || !(c.dz > 0))
        return BT_E_ARG;
    for (int a = 0; a < 3; ++a)
        if (c.buffer[a] < 0 || 2 * c.buffer[a] > (a == 0 ? c.nx : a == 1 ? c.ny : c.nz)) return BT_E_ARG;
    // one field per call, advection on or off: a batched config (a q-sweep)
    // is not accepted, so no caller mistakes one stepped member for the batch
    if (c.batch > 1 || c.batch < 0 || (c.velocity != 0 && c.velocity != 1)) return BT_E_ARG;
    // a single step has no earlier step to have set non-copy ghost layers
    // (the first step of a run reads copies): copy faces only
    if (c.boundary[0] != BT_BC_COPY || c.boundary[1] != BT_BC_COPY || c.boundary[2] != BT_BC_COPY) return BT_E_ARG;
    if (c.velocity == 1 && (!vx || !vy || !vz)) return BT_E_ARG;
    const long long nvox = (long long)c.nx * c.ny * c.nz;
    if (nvox > BT_NOALLOC_MAX_VOXELS) {
        std::fprintf(stderr,
                     "bt_step_noalloc: %d x %d x %d = %lld voxels exceeds the allocation-free limit of %d voxels "
                     "(use bt_create / bt_run for larger grids)\n",
                     c.nx, c.ny, c.nz, nvox, BT_NOALLOC_MAX_VOXELS);
        return BT_E_SIZE;
    }
    // the grid's size in column tiles of 32 x 8, z split to fill the SMs, no empty
    // z-chunk: a caller's limit
    const int gx = (c.nx + bt::TX - 1) / bt::TX, gy = (c.ny + bt::TY - 1) / bt::TY;
    const long long tiles = (long long)gx * gy;
    int zsplit = 1;
    if (tiles < 1216) zsplit = (int)std::min<long long>((1216 + tiles - 1) / tiles, std::max(1, c.nz / 8));
    zsplit = std::max(1, std::min(zsplit, c.nz));
    while ((c.nz + zsplit - 1) / zsplit > 1024) zsplit++;
    const int zchunk = (c.nz + zsplit - 1) / zsplit;
    zsplit = (c.nz + zchunk - 1) / zchunk;
    if (tiles * zsplit > BT_NOALLOC_MAX_BLOCKS) {
        std::fprintf(stderr, "bt_step_noalloc: grid of %lld blocks exceeds the allocation-free limit of %d\n",
                     tiles * zsplit, BT_NOALLOC_MAX_BLOCKS);
        return BT_E_SIZE;
    }
    unsigned char* scratch = nullptr;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const cudaError_t se = scratch_for_current_device(s, &scratch);
    if (se == cudaErrorStreamCaptureUnsupported) {
        std::fprintf(stderr,
                     "bt_step_noalloc: the first call on a device looks up its scratch array and must come before "
                     "any stream capture\n");
        return BT_E_ARG;
    }
    if (se != cudaSuccess) return BT_E_CUDA;
    const void* in[3] = {mx_in, my_in, mz_in};
    void* out[3] = {mx_out, my_out, mz_out};
    const int prec = c.vector_mult == 1 ? 1 : 0;
    const int vel = c.velocity == 1 ? 1 : 0;
    cudaError_t e;
    if (c.precision == BT_F64) {
        bt::StepParams<double> P;
        fill<double>(c, P, in, out, vx, vy, vz, scratch, sums);
        e = bt::launch_single<double>(P, mask, c.grad, vel, prec, s);
    } else {
        bt::StepParams<float> P;
        fill<float>(c, P, in, out, vx, vy, vz, scratch, sums);
        e = bt::launch_single<float>(P, mask, c.grad, vel, prec, s);
    }
    return e == cudaSuccess ? BT_OK : BT_E_CUDA;
}
