// noalloc.cu -- charge deposition of reference Points that allocates nothing.
//
// Some callers cannot allocate device memory at the point where they need a
// deposit: a host framework that owns a fixed device-memory budget and hands
// plugins only the buffers it has already sized, or a time-critical loop
// that must not call cudaMalloc/cudaFree because those may synchronise the
// whole device.  pic_deposit_points_noalloc serves them: the caller passes
// the particles and the output grids, and the one scratch buffer the
// deposit needs (the 64-bit fixed-point node accumulators) is a file-scope
// __device__ array of fixed size that every GPU loading this library keeps
// until the process exits.
//
// The arithmetic is the library's own deposit: the cell of a Point is
// (int)(x*(1/dx)), the FP32 in-cell offset is the FP64 remainder, each axis
// offset is rounded to 20 bits and the four corner weights are exact 40-bit
// products summed in 64-bit integers -- so the result is bit-for-bit the
// final_mesh / rho that pic_import_points + pic_charge_deposition produce.
#include <cuda.h>
#include <cuda_runtime.h>

#include <mutex>
#include <string>

#include "pic_internal.h"

namespace picb200 {
namespace {

// 2^19 nodes = 4 MiB of accumulators, e.g. up to 724 x 724 nodes.
constexpr int64_t kNoAllocMaxNodes = 1ll << 19;
constexpr int kMaxDevices = 64;

__device__ __align__(256) unsigned long long g_noalloc_acc[kNoAllocMaxNodes];

std::mutex g_mu;
// Per device: the device address of the scratch array and the unique id of
// the CUDA context it was looked up in.  The address belongs to the module
// as loaded into that context; after cudaDeviceReset the next primary
// context loads the module again, possibly at another address, so a change
// of context id means a new lookup.
struct ScratchSlot {
    unsigned long long ctx_id;
    unsigned long long* addr;
};
ScratchSlot g_slot[kMaxDevices] = {};

using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

// The current context's unique id through the driver entry points (no link
// against libcuda); 0 when the driver cannot tell, which disables the cache.
unsigned long long current_context_id() {
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static bool looked_up = false;
    if (!looked_up) {
        looked_up = true;
        cudaDriverEntryPointQueryResult q1, q2;
        void* f1 = nullptr;
        void* f2 = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f1, cudaEnableDefault, &q1) == cudaSuccess &&
            q1 == cudaDriverEntryPointSuccess &&
            cudaGetDriverEntryPoint("cuCtxGetId", &f2, cudaEnableDefault, &q2) == cudaSuccess &&
            q2 == cudaDriverEntryPointSuccess) {
            get_current = reinterpret_cast<CtxGetCurrentFn>(f1);
            get_id = reinterpret_cast<CtxGetIdFn>(f2);
        }
        cudaGetLastError();
    }
    if (!get_current || !get_id) return 0;
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS) return 0;
    return id;
}

// Device address of the scratch array on the current device (the host-side
// name of the array is not a device address), looked up with the device
// current once per device and context.
int scratch_address(unsigned long long** out) {
    int dev = 0;
    PIC_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(PIC_ERR_NO_DEVICE, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_mu);
    // 0 before the runtime has made the device's primary context current: the
    // lookup below does that, and the id is read again after it
    const unsigned long long id = current_context_id();
    ScratchSlot& slot = g_slot[dev];
    if (!slot.addr || id == 0 || slot.ctx_id != id) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_acc);
        if (e != cudaSuccess) {
            slot.addr = nullptr;
            return fail(PIC_ERR_CUDA, std::string("cudaGetSymbolAddress(g_noalloc_acc): ") +
                                          cudaGetErrorString(e));
        }
        slot.addr = static_cast<unsigned long long*>(p);
        slot.ctx_id = current_context_id();
    }
    *out = slot.addr;
    return PIC_OK;
}

__global__ void k_na_clear(ulonglong2* acc, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) acc[i] = make_ulonglong2(0ull, 0ull);
}

__device__ __forceinline__ uint32_t na_axis(float f) {
    const float t = __fadd_rn(__fmul_rn(f, (float)(1u << kAxisBits)), 12582912.0f);
    return __float_as_uint(t) - 0x4B400000u;
}

// A point's cell and axis weights, or cell -1.
struct NaPoint {
    int gx, gy;
    uint32_t ax, ay;
};

__device__ __forceinline__ NaPoint na_point(const pic_point* __restrict__ pts, int64_t i, int64_t n, int nx, int ny,
                                            double inv_dx, double inv_dy) {
    NaPoint p{-1, 0, 0u, 0u};
    if (i >= n || pts[i].pointer == -1) return p;
    const double sx = pts[i].x * inv_dx, sy = pts[i].y * inv_dy;
    if (!(sx >= 0.0 && sy >= 0.0 && sx < (double)nx && sy < (double)ny)) return p;
    p.gx = (int)sx;
    p.gy = (int)sy;
    const float one_below = 0x1.fffffep-1f;
    p.ax = na_axis(fminf((float)(sx - p.gx), one_below));
    p.ay = na_axis(fminf((float)(sy - p.gy), one_below));
    return p;
}

constexpr uint32_t kNaOne = 1u << kAxisBits;

// Points in any order: what bounds the deposit is the atomics, four a point, and
// of those the 32-byte sectors that a warp's additions fall into (about 150 per
// nanosecond).  So lanes that add to one sector do it with one instruction.
//
// Grids whose cells fit into the scratch four words each, where they have points
// enough: a cell's corner sums
// are a sector, four lanes a point add to it, and k_na_finish_cells gathers a
// node from its four cells.  Where cells have many points each, blocks add to
// one of `copies` of the array in turn (additions to one sector wait for each
// other).
__global__ void __launch_bounds__(256) k_na_deposit_cells(const pic_point* __restrict__ pts, int64_t n, int nx, int ny,
                                                          double inv_dx, double inv_dy, unsigned long long* acc,
                                                          int copies) {
    const NaPoint p = na_point(pts, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, n, nx, ny, inv_dx, inv_dy);
    const int cell = p.gx < 0 ? -1 : p.gy * nx + p.gx, lane = threadIdx.x & 31;
    acc += (int64_t)(blockIdx.x & (copies - 1)) * nx * ny * 4 + (lane & 3);
#pragma unroll
    for (int h = 0; h < 4; ++h) {  // 8 points at a time, a lane a corner
        const int from = 8 * h + (lane >> 2);
        const int q = __shfl_sync(0xffffffffu, cell, from);
        const uint32_t px = __shfl_sync(0xffffffffu, p.ax, from), py = __shfl_sync(0xffffffffu, p.ay, from);
        const unsigned long long wx = lane & 1 ? px : kNaOne - px;
        if (q >= 0) atomicAdd(acc + (int64_t)q * 4, wx * (lane & 2 ? py : kNaOne - py));
    }
}

// Larger grids, or fewer points: a word a node; the two nodes of a cell's row are neighbours,
// two lanes a point.
__global__ void __launch_bounds__(256) k_na_deposit_nodes(const pic_point* __restrict__ pts, int64_t n, int nx, int ny,
                                                          double inv_dx, double inv_dy, unsigned long long* acc) {
    const NaPoint p = na_point(pts, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, n, nx, ny, inv_dx, inv_dy);
    const int GX = nx + 1, node = p.gx < 0 ? -1 : p.gy * GX + p.gx, lane = threadIdx.x & 31;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int from = 16 * h + (lane >> 1);
        const int q = __shfl_sync(0xffffffffu, node, from);
        const uint32_t px = __shfl_sync(0xffffffffu, p.ax, from), py = __shfl_sync(0xffffffffu, p.ay, from);
        if (q < 0) continue;
        const unsigned long long wx = lane & 1 ? px : kNaOne - px;
        unsigned long long* to = acc + q + (lane & 1);
        atomicAdd(to, wx * (kNaOne - py));
        atomicAdd(to + GX, wx * py);
    }
}

__device__ __forceinline__ void na_store(unsigned long long sum, int64_t i, double qscale, double chrg,
                                         double* final_mesh, double* rho) {
    const double f = (double)sum * qscale;
    final_mesh[i] = f;
    if (rho) rho[i] += f * chrg;
}

__global__ void k_na_finish_cells(const unsigned long long* acc, int nx, int ny, int copies, double qscale, double chrg,
                                  double* final_mesh, double* rho) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, GX = nx + 1;
    if (i >= GX * (ny + 1)) return;
    const int gy = i / GX, gx = i - gy * GX;
    unsigned long long sum = 0;
    for (int r = 0; r < copies; ++r) {
        const unsigned long long* a = acc + (int64_t)r * nx * ny * 4;
#pragma unroll
        for (int c = 0; c < 4; ++c) {  // the node is corner c of cell (gx - (c & 1), gy - (c >> 1))
            const int x = gx - (c & 1), y = gy - (c >> 1);
            if (x >= 0 && x < nx && y >= 0 && y < ny) sum += a[((int64_t)y * nx + x) * 4 + c];
        }
    }
    na_store(sum, i, qscale, chrg, final_mesh, rho);
}

__global__ void k_na_finish_nodes(const unsigned long long* acc, int64_t nodes, double qscale, double chrg,
                                  double* final_mesh, double* rho) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nodes) na_store(acc[i], i, qscale, chrg, final_mesh, rho);
}

}  // namespace
}  // namespace picb200

using namespace picb200;

extern "C" int pic_deposit_points_noalloc(const pic_point* dev_points, int64_t n, int32_t nx,
                                          int32_t ny, double xmax, double ymax,
                                          const pic_species_desc* species, double surf_area,
                                          double epsilon, double* dev_final_mesh,
                                          double* dev_rho, void* cuda_stream) {
    if (n < 0 || (n > 0 && !dev_points) || !species || !dev_final_mesh)
        return fail(PIC_ERR_ARG, "pic_deposit_points_noalloc: null pointer or negative count");
    if (nx < 1 || ny < 1 || !(xmax > 0) || !(ymax > 0) || !(epsilon > 0) ||
        !(species->sim_count > 0))
        return fail(PIC_ERR_CONFIG, "pic_deposit_points_noalloc: bad grid or species description");
    const int64_t GX = (int64_t)nx + 1, nodes = GX * ((int64_t)ny + 1);
    if (nodes > kNoAllocMaxNodes)
        return fail(PIC_ERR_CAPACITY,
                    "pic_deposit_points_noalloc: grid of " + std::to_string(nodes) +
                        " nodes exceeds the fixed scratch of " + std::to_string(kNoAllocMaxNodes) +
                        " nodes");
    unsigned long long* acc = nullptr;
    PIC_TRY(scratch_address(&acc));
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    const double dx = xmax / nx, dy = ymax / ny;
    const double surf = surf_area > 0 ? surf_area : xmax * ymax;
    // updateWeighingFactor, src/particles.cpp:303-305
    const double weighing = species->actual_count * surf / (species->sim_count * dx * dy * dx * dy);
    const double qscale = kChargeUnit * (dx * dy) * weighing;  // as the context's flush rounds it
    const double chrg = -species->charge / epsilon;  // RhoKernel, src/interpolation.cpp:164-170
    const int64_t cells = (int64_t)nx * ny;
    const auto blocks = [](int64_t k) { return (unsigned)((k + 255) / 256); };
    // Cells where they fit and have three points each: clearing and gathering four
    // words a cell costs more than the additions of fewer.  Measured, us a call, four
    // scattered additions a point / nodes in pairs / cells: 4M points on 300 x 280
    // cells 112 / 81 / 62, on 32 x 32 (16 copies) 628 / 415 / 64, 1M on 300 x 280 40 / 32 /
    // 30; on 700 x 700, too large for cells, 109 / 81.  The three launches alone, without
    // the host's part of the call: 3,000 points on 362 x 362 5.2 / 5.1 / 6.3, 100,000 6.9 / 6.0 /
    // 7.0, 300,000 (2.3 a cell) 11.6 / 8.8 / 9.1, 1M 27 / 18 / 16; on 200 x 200 100,000 (2.5)
    // 7.1 / 6.0 / 6.1, 200,000 10.0 / 7.9 / 7.2; on 100 x 100 20,000 5.3 / 5.0 / 5.1, 30,000 6.0 /
    // 5.3 / 5.2.
    const bool by_cell = cells * 4 <= kNoAllocMaxNodes && n >= 3 * cells;
    int copies = 1;  // up to 16, while the cells have 64 points each a copy
    while (by_cell && copies < 16 && cells * 8 * copies <= kNoAllocMaxNodes && n >= cells * 128 * copies) copies *= 2;
    const int64_t words = by_cell ? cells * 4 * copies : nodes;
    k_na_clear<<<blocks((words + 1) / 2), 256, 0, st>>>(reinterpret_cast<ulonglong2*>(acc), (words + 1) / 2);
    if (by_cell) {
        if (n > 0)
            k_na_deposit_cells<<<blocks(n), 256, 0, st>>>(dev_points, n, nx, ny, 1.0 / dx, 1.0 / dy, acc, copies);
        k_na_finish_cells<<<blocks(nodes), 256, 0, st>>>(acc, nx, ny, copies, qscale, chrg, dev_final_mesh, dev_rho);
    } else {
        if (n > 0) k_na_deposit_nodes<<<blocks(n), 256, 0, st>>>(dev_points, n, nx, ny, 1.0 / dx, 1.0 / dy, acc);
        k_na_finish_nodes<<<blocks(nodes), 256, 0, st>>>(acc, nodes, qscale, chrg, dev_final_mesh, dev_rho);
    }
    PIC_CUDA(cudaGetLastError());
    return PIC_OK;
}
