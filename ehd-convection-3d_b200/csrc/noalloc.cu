// noalloc.cu -- the Poisson solve and E field on caller-owned device buffers,
// for callers that cannot allocate device memory.
//
// Some callers of this library run where device allocation is not theirs to
// do: a host framework that owns every allocation on the GPU through its own
// pool, a process that must not grow its footprint after start-up, or code
// between the launches of another library's pipeline where a cudaMalloc would
// synchronise the device.  ehd_poisson_noalloc serves them: it solves the same
// discrete Poisson problem as the time step (FFT in x and y, FP64 tridiagonal
// solve in z, E = -grad(phi)) on device arrays the caller passes in, and keeps
// its working storage in one file-scope device array of fixed size instead of
// allocating.  It calls no cudaMalloc, cudaFree or other allocating routine,
// on the device or on the host.
//
// A call is seven launches: the tables in one, the five of the solve, phi and E
// in one, each waiting on the one before as the step's do.  With 13 launches
// (tables, three memsets, an E kernel of one warp a block, phi in place) a call
// at 96 x 96 x 65 took 64 us, so 38 (109 before that with the one-thread-per-mode
// FP64 sweep).
//
// The array costs EHD_NOALLOC_SCRATCH_BYTES of device memory on each GPU the
// entry point is used on, until the process exits.  Under CUDA's lazy module
// loading (the default) the driver commits it when the first call on a device
// looks up its address, so that first call is itself a device allocation by
// the driver: make it at start-up, before any stream capture.  With
// CUDA_MODULE_LOADING=EAGER the array is committed on every GPU when the
// library's module loads.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>

#include "common.cuh"
#include "ehd.h"
#include "kernels.h"

namespace ehd {
namespace {

// The working storage.  In host code this name is a host-side stand-in, not a
// device address: host code obtains the address with cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_noalloc_scratch[EHD_NOALLOC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
std::mutex g_mu;
// per device: the array's address and the context it was looked up in (a
// cudaDeviceReset makes a new primary context, where the module reloads and
// the array may move)
void *g_scratch_addr[kMaxDevices] = {};
CUcontext g_scratch_ctx[kMaxDevices] = {};
// the context in which the z solve's shared-memory attribute was set: its need
// grows with NZ, so it is set by the first call outside a capture, whatever that
// call's NZ, for a deeper one inside a capture
CUcontext g_zmeet_ctx[kMaxDevices] = {};
bool g_zmeet_set[kMaxDevices] = {};

// The calling thread's current driver context, through the runtime's driver
// entry point (the library links only the runtime).
CUcontext current_context() {
    using Fn = CUresult (*)(CUcontext *);
    static Fn fn = nullptr;
    static bool looked_up = false;
    if (!looked_up) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult st{};
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &st) ==
                cudaSuccess && st == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<Fn>(p);
        looked_up = true;
    }
    CUcontext c = nullptr;
    if (fn && fn(&c) != CUDA_SUCCESS) c = nullptr;
    return c;
}

size_t align256(size_t b) { return (b + 255) / 256 * 256; }

bool only_235(int n) {
    if (n < 1) return false;
    for (int f : {2, 3, 5})
        while (n % f == 0) n /= f;
    return n == 1;
}

FftPlan plan_of(int n) {
    FftPlan p{};
    p.n = n;
    while (n % 4 == 0) { p.rad[p.nrad++] = 4; n /= 4; }
    while (n % 2 == 0) { p.rad[p.nrad++] = 2; n /= 2; }
    while (n % 3 == 0) { p.rad[p.nrad++] = 3; n /= 3; }
    while (n % 5 == 0) { p.rad[p.nrad++] = 5; n /= 5; }
    return p;
}

// Everything the solve reads before writing, in one launch: the twiddles
// exp(-2 pi i k / n) of both axes, the zero reference charge, and the Thomas
// pivots per mode, the same table as the context's (api.cu):
// beta = 2 + (kx^2 + ky^2) dz^2, cp_0 = -1/beta, cp_i = 1/(-beta - cp_{i-1}),
// the first `rows` of them (one thread a mode, the thread's number also that
// of a twiddle or reference).
__global__ void setup_kernel(double2 *twx, double2 *twy, double *qmean, double *cpt, int nx, int ny,
                             int nz, int rows, double lx, double ly, double dz) {
    const int nxh = nx / 2 + 1;
    const int modes = nxh * ny;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int stride = gridDim.x * blockDim.x;
    for (int k = m; k < nx + ny; k += stride) {
        const bool xa = k < nx;
        const int i = xa ? k : k - nx;
        double s, c;
        sincospi(-2.0 * (double)i / (double)(xa ? nx : ny), &s, &c);
        (xa ? twx : twy)[i] = make_double2(c, s);
    }
    for (int k = m; k < 2 * nz; k += stride) qmean[k] = 0.0;
    if (m >= modes) return;
    const int j = m / nxh, i = m - j * nxh;
    const double kx = (double)i * 2.0 * M_PI / lx;
    const double ky = (j <= ny / 2 ? (double)j : (double)j - ny) * 2.0 * M_PI / ly;
    const double beta = 2.0 + (kx * kx + ky * ky) * dz * dz;
    double prev = 0.0;
    for (int z = 0; z < rows; ++z) {
        prev = 1.0 / (-beta - prev);
        cpt[(size_t)z * modes + m] = prev;
    }
}

// phi = phi00(z) + phi' (phi00 carries V and 0 on the electrodes, phi' is zero
// there) and E = -grad(phi), central differences with the electrode copy of
// Ez (gpu_efield, gpu_bc, poisson.cu:44-73), from phi' of the planes 1..NZ-2
// in scratch (phip points a plane before them).
__global__ void fields_kernel(const double *__restrict__ phip, const double *__restrict__ phi00,
                              double *__restrict__ phi, double *__restrict__ ex,
                              double *__restrict__ ey, double *__restrict__ ez, int nx, int ny,
                              int nz, double inv2dx, double inv2dy, double inv2dz) {
    step_enter();
    // runs over a plane: rows alone would be short blocks on narrow grids
    const int xy = blockIdx.x * blockDim.x + threadIdx.x, z = blockIdx.y;
    if (xy >= nx * ny) return;
    const int y = xy / nx, x = xy - y * nx;
    auto p = [&](int xx, int yy, int zz) {
        return zz == 0 || zz == nz - 1 ? 0.0
                                       : __ldg(phip + (size_t)xx + (size_t)nx * ((size_t)yy + (size_t)ny * zz));
    };
    const int xm = x == 0 ? nx - 1 : x - 1, xp = x == nx - 1 ? 0 : x + 1;
    const int ym = y == 0 ? ny - 1 : y - 1, yp = y == ny - 1 ? 0 : y + 1;
    const int zc = z < 1 ? 1 : (z > nz - 2 ? nz - 2 : z);
    const size_t i = (size_t)x + (size_t)nx * ((size_t)y + (size_t)ny * z);
    phi[i] = phi00[z] + p(x, y, z);
    ex[i] = (p(xm, y, z) - p(xp, y, z)) * inv2dx;
    ey[i] = (p(x, ym, z) - p(x, yp, z)) * inv2dy;
    ez[i] = ((phi00[zc - 1] + p(x, y, zc - 1)) - (phi00[zc + 1] + p(x, y, zc + 1))) * inv2dz;
}

}  // namespace
}  // namespace ehd

using namespace ehd;

extern "C" int ehd_poisson_noalloc(const ehd_params *p, const double *q, double *phi,
                                   double *ex, double *ey, double *ez, void *stream) {
    if (!p || !q || !phi || !ex || !ey || !ez)
        return set_error(EHD_ERR_INVALID, "ehd_poisson_noalloc: NULL argument");
    if (p->nx < 1 || p->ny < 1 || p->nz < 4 || !only_235(p->nx) || !only_235(p->ny) ||
        !(p->dx > 0) || !(p->dy > 0) || !(p->dz > 0) || !(p->lx > 0) || !(p->ly > 0) ||
        !(p->eps > 0))
        return set_error(EHD_ERR_INVALID, "ehd_poisson_noalloc: invalid grid or parameters");
    const int nx = p->nx, ny = p->ny, nz = p->nz;
    const int nxh = nx / 2 + 1, pitch = (nxh + 15) / 16 * 16;
    const size_t modes = (size_t)nxh * ny;
    // scratch layout
    const size_t b_spec = align256(sizeof(double2) * (size_t)(nz - 2) * ny * pitch);
    const size_t b_cpt = align256(sizeof(double) * modes * (size_t)(nz - 2));
    const size_t b_dpw = align256(sizeof(double2) * modes * (size_t)(nz - 2));
    const size_t b_twx = align256(sizeof(double2) * nx), b_twy = align256(sizeof(double2) * ny);
    const size_t b_row = align256(sizeof(double) * (size_t)(nz - 2) * ny);
    const size_t b_z = align256(sizeof(double) * nz);
    const size_t b_qm = align256(sizeof(double) * 2 * nz);
    const size_t total = b_spec + b_cpt + b_dpw + b_twx + b_twy + b_row + 3 * b_z + b_qm;
    if (total > EHD_NOALLOC_SCRATCH_BYTES || (long long)nx * ny * nz > (1LL << 31))
        return set_error(EHD_ERR_INVALID,
                         "ehd_poisson_noalloc: the grid needs more working storage than the "
                         "EHD_NOALLOC_SCRATCH_BYTES (64 MiB) the entry point has; use ehd_poisson");
    // the shared-memory FFT limits of the context path apply as well
    if ((size_t)2 * nx * 16 > 200 * 1024 || (size_t)2 * ny * 16 > 200 * 1024)
        return set_error(EHD_ERR_INVALID, "ehd_poisson_noalloc: nx or ny too large");

    {
        // an error left pending by the caller's earlier work is reported as
        // such, and left pending (not consumed by this call's launch checks)
        const cudaError_t pending = cudaPeekAtLastError();
        if (pending != cudaSuccess)
            return set_error(EHD_ERR_CUDA, "ehd_poisson_noalloc: a CUDA error from earlier work "
                                           "is pending; nothing was launched");
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return set_error(EHD_ERR_CUDA, "ehd_poisson_noalloc: no usable current device");
    unsigned char *base = nullptr;
    cudaStream_t s = (cudaStream_t)stream;
    {
        // first call on this device (in this context): the device address of
        // the array
        std::lock_guard<std::mutex> lk(g_mu);
        const CUcontext ctx = current_context();
        if (!g_scratch_addr[dev] || g_scratch_ctx[dev] != ctx) {
            void *ptr = nullptr;
            if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || !ptr)
                return set_error(EHD_ERR_CUDA, "ehd_poisson_noalloc: cudaGetSymbolAddress failed");
            g_scratch_addr[dev] = ptr;
            g_scratch_ctx[dev] = ctx;
        }
        base = (unsigned char *)g_scratch_addr[dev];
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        if ((!g_zmeet_set[dev] || g_zmeet_ctx[dev] != ctx) &&
            cudaStreamIsCapturing(s, &st) == cudaSuccess && st == cudaStreamCaptureStatusNone) {
            if (prepare_zmeet<double>() != cudaSuccess)
                return set_error(EHD_ERR_CUDA, "ehd_poisson_noalloc: kernel set-up failed");
            g_zmeet_set[dev] = true;
            g_zmeet_ctx[dev] = ctx;
        }
    }
    PoissonArgs a{};
    a.nx = nx;
    a.ny = ny;
    a.nz = nz;
    a.nxh = nxh;
    a.pitch = pitch;
    {
        int rows = 16;
        while (rows > 1 && (size_t)2 * rows * nx * 16 > 64 * 1024) rows >>= 1;
        int cols = 8;
        while (cols > 1 && (size_t)2 * cols * ny * 16 > 160 * 1024) cols >>= 1;
        a.rows_per_block = rows;
        a.cols_per_block = cols;
    }
    a.px = plan_of(nx);
    a.py = plan_of(ny);
    unsigned char *cur = base;
    a.spec = cur;                       cur += b_spec;
    double *cpt = (double *)cur;        cur += b_cpt;
    a.dpw = (double2 *)cur;             cur += b_dpw;
    double2 *twx = (double2 *)cur;      cur += b_twx;
    double2 *twy = (double2 *)cur;      cur += b_twy;
    a.rowsum = (double *)cur;           cur += b_row;
    a.planesum = (double *)cur;         cur += b_z;
    a.phi00 = (double *)cur;            cur += b_z;
    a.ez00 = (double *)cur;             cur += b_z;
    double *qmean = (double *)cur;      cur += b_qm;
    a.cpt = cpt;
    a.twx = twx;
    a.twy = twy;
    a.q = q;
    a.qmean = qmean;
    // phi' of the interior planes into the sweep's scratch, which is free by then
    // (16 bytes a mode and plane; the solve writes plane z at phip + z NX NY)
    double *phip = (double *)a.dpw - (size_t)nx * ny;
    a.phip = phip;
    a.eps = p->eps;
    a.voltage = p->voltage;
    a.dz = p->dz;
    a.lx = p->lx;
    a.ly = p->ly;

    // the two-sided z solve reads the pivots of half the planes
    const int piv = zmeet_modes(nz, sizeof(double)) > 0 ? (nz - 2) / 2 : nz - 2;
    setup_kernel<<<(unsigned)((modes + 127) / 128), 128, 0, s>>>(twx, twy, qmean, cpt, nx, ny, nz, piv,
                                                                  p->lx, p->ly, p->dz);
    if (cudaGetLastError() != cudaSuccess)
        return set_error(EHD_ERR_CUDA, "ehd_poisson_noalloc: the table kernel failed to launch");
    if (launch_poisson<double>(a, s) != cudaSuccess)
        return set_error(EHD_ERR_CUDA, "ehd_poisson_noalloc: Poisson kernels failed to launch");
    if (step_launch(fields_kernel, dim3((nx * ny + 255) / 256, nz), 256, 0, s, phip, a.phi00, phi,
                    ex, ey, ez, nx, ny, nz, 0.5 / p->dx, 0.5 / p->dy, 0.5 / p->dz) != cudaSuccess)
        return set_error(EHD_ERR_CUDA, "ehd_poisson_noalloc: the field kernel failed to launch");
    return EHD_OK;
}
