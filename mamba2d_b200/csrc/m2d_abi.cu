// C-ABI housekeeping: version, status strings and the process-wide flag of failed waits.
#include "launch.cuh"

namespace m2d {

int* wait_failure_flag() {
    static std::mutex m;
    static int* flag = nullptr;
    std::lock_guard<std::mutex> lock(m);
    if (!flag && device_index() >= 0) {
        // (an allocation is not part of anything that may be under capture on this thread)
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        void* p = nullptr;
        if (cudaHostAlloc(&p, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
            flag = static_cast<int*>(p);
            *flag = 0;
        } else {
            cudaGetLastError();
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
    }
    return flag;
}

// What the host has seen of that word: failures so far, and whether one has not been taken yet.
static std::mutex g_seen_mutex;
static int64_t g_seen = 0;
static bool g_pending = false;

static bool look_at_flag() {        // false: there is no word
    int* f = wait_failure_flag();
    if (f && __atomic_exchange_n(f, 0, __ATOMIC_ACQ_REL) != 0) {
        ++g_seen;
        g_pending = true;
    }
    return f != nullptr;
}

}  // namespace m2d

extern "C" int m2d_take_wait_failure(void) {
    std::lock_guard<std::mutex> lock(m2d::g_seen_mutex);
    m2d::look_at_flag();
    const bool was = m2d::g_pending;
    m2d::g_pending = false;
    return was ? 1 : 0;
}

extern "C" int64_t m2d_wait_failure_mark(void) {
    std::lock_guard<std::mutex> lock(m2d::g_seen_mutex);
    return m2d::look_at_flag() ? m2d::g_seen : -1;
}

extern "C" int m2d_abi_version(void) { return M2D_ABI_VERSION; }

extern "C" const char* m2d_strerror(int status) {
    switch (status) {
        case M2D_OK: return "ok";
        case M2D_ERR_NULL: return "a required pointer is NULL";
        case M2D_ERR_DTYPE: return "unknown dtype";
        case M2D_ERR_SHAPE: return "bad shape: need B,E,N >= 1 and H,W >= 2";
        case M2D_ERR_UNSUPPORTED_N: return "state size N > 16 is not supported";
        case M2D_ERR_PITCH: return "BT/BL/C pixel pitch smaller than N";
        case M2D_ERR_WORKSPACE: return "workspace missing, too small or not 256-byte aligned";
        case M2D_ERR_LAUNCH: return "CUDA launch failed";
        case M2D_ERR_ABI: return "descriptor size does not match this library";
        case M2D_ERR_TOO_LARGE: return "problem exceeds the fixed capacity of this entry point";
        case M2D_ERR_FLAGS: return "unknown bit in desc->flags";
        default: return "unknown status";
    }
}
