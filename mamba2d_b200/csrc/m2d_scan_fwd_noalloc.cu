// Forward scan for callers that cannot hand the library a workspace buffer.
//
// The regular forward entry point needs a scratch region (the per-CTA ring that carries the last
// row of one band of image rows to the first row of the next band) and expects the caller to
// allocate it.  Some callers have no way to do that: a host runtime that binds this library behind
// a fixed "inputs in, outputs out" plugin signature has no slot for an extra buffer; a service that
// carved up all device memory at start-up has no allocator left to ask; and code running inside a
// latency-critical loop must not call cudaMalloc, which can synchronise the whole device.  For
// them this file keeps the ring in a file-scope __device__ array of fixed size, so the call needs
// nothing but the inputs and the output.
//
// Cost and limits of that choice:
//   - every GPU on which this library is loaded holds M2D_NOALLOC_SCRATCH_BYTES (32 MiB) of
//     device memory from load until the process exits;
//   - problems whose ring would not fit are rejected with M2D_ERR_TOO_LARGE;
//   - all calls on one device share the one array.  Only its first word (the status word the
//     kernels share with the regular entry point's workspace layout) has to start at zero, and the
//     call clears it itself; every other slot is written before it is read within a call, and what
//     an earlier call left behind is never read.  But two calls that overlap in time on the same
//     GPU -- different streams, or different host threads -- would overwrite each other's slots
//     and produce wrong results.  Serialise them (one stream, or events between streams);
//   - the first call on each device looks up the array's device address
//     (cudaGetSymbolAddress) and caches it; make that first call before starting any stream
//     capture on that device.
#include <mutex>

#include "launch.cuh"

namespace m2d {

// In host code this name is only a handle for the runtime's symbol table, not a device address:
// it must go through cudaGetSymbolAddress before a kernel can be given a pointer to it.
static __device__ __align__(256) unsigned char g_noalloc_ring[M2D_NOALLOC_SCRATCH_BYTES];

static std::mutex g_ring_mutex;
static float4* g_ring_ptr[kMaxDevices] = {};   // device address of g_noalloc_ring on each device

// Device address of the ring on the CURRENT device; looked up once per device.
static int ring_address(float4** out) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return M2D_ERR_LAUNCH;
    std::lock_guard<std::mutex> lock(g_ring_mutex);
    if (g_ring_ptr[dev] == nullptr) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_ring) != cudaSuccess || p == nullptr) {
            cudaGetLastError();
            return M2D_ERR_LAUNCH;
        }
        g_ring_ptr[dev] = static_cast<float4*>(p);
    }
    *out = g_ring_ptr[dev];
    return M2D_OK;
}

// The plan of the regular entry where its scratch fits the array, else the fastest that does: fewer CTAs with more warps and
// longer bands, or no chains of CTAs.
static Plan plan_noalloc(const m2d_scan_desc* d) {
    const Plan p = plan_fwd(d);
    return p.scratch <= M2D_NOALLOC_SCRATCH_BYTES ? p : make_plan_fwd(d, M2D_NOALLOC_SCRATCH_BYTES);
}

}  // namespace m2d

extern "C" uint64_t m2d_scan_fwd_noalloc_need(const m2d_scan_desc* d) {
    if (m2d::check_desc(d, false, false) != M2D_OK) return 0;
    return m2d::plan_noalloc(d).scratch;
}

extern "C" int m2d_scan_fwd_noalloc(const m2d_scan_desc* d, void* stream) {
    int rc = m2d::check_desc(d, false, true);
    if (rc != M2D_OK) return rc;
    if (!d->y) return M2D_ERR_NULL;
    if (d->flags & M2D_SCAN_WS_CLEARED) return M2D_ERR_FLAGS;      // the scratch is not the caller's
    const m2d::Plan pl = m2d::plan_noalloc(d);
    if (pl.scratch > M2D_NOALLOC_SCRATCH_BYTES) return M2D_ERR_TOO_LARGE;   // decided before any device work
    float4* ring = nullptr;
    rc = m2d::ring_address(&ring);
    if (rc != M2D_OK) return rc;
    return m2d::launch_forward(d, pl, reinterpret_cast<char*>(ring), static_cast<cudaStream_t>(stream));
}
