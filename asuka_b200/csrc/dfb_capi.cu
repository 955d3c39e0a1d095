// Library-level C ABI entry points: version and error reporting.
#include <stdarg.h>
#include <stdio.h>

#include <atomic>

#include "../../include/dfb.h"
#include "dfb_internal.h"

namespace dfb {
static thread_local char g_msg[512] = "";
static std::atomic<long> g_launches{0};

void count_launches(long n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

void clear_error() { g_msg[0] = '\0'; }

int set_error(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_msg, sizeof(g_msg), fmt, ap);
    va_end(ap);
    return code;
}

int set_cuda_error(const char* what, cudaError_t e) {
    snprintf(g_msg, sizeof(g_msg), "%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e));
    return DFB_ERR_CUDA;
}
}  // namespace dfb

extern "C" int dfb_version(void) { return 100; }

extern "C" const char* dfb_last_error(void) { return dfb::g_msg; }

extern "C" long dfb_launch_count(void) { return dfb::g_launches.load(std::memory_order_relaxed); }

extern "C" int dfb_fork(void* main_stream, void* const* streams, int nstreams) {
    dfb::clear_error();
    if (nstreams < 0 || (nstreams > 0 && !streams)) return dfb::set_error(DFB_ERR_INVALID, "invalid arguments to dfb_fork");
    cudaEvent_t ev;
    cudaError_t e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (e != cudaSuccess) return dfb::set_cuda_error("dfb_fork", e);
    e = cudaEventRecord(ev, (cudaStream_t)main_stream);
    for (int i = 0; i < nstreams && e == cudaSuccess; ++i) e = cudaStreamWaitEvent((cudaStream_t)streams[i], ev, 0);
    cudaEventDestroy(ev);
    return e == cudaSuccess ? DFB_OK : dfb::set_cuda_error("dfb_fork", e);
}

extern "C" int dfb_join(void* main_stream, void* const* streams, int nstreams) {
    dfb::clear_error();
    if (nstreams < 0 || (nstreams > 0 && !streams)) return dfb::set_error(DFB_ERR_INVALID, "invalid arguments to dfb_join");
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < nstreams && e == cudaSuccess; ++i) {
        cudaEvent_t ev;
        e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
        if (e != cudaSuccess) break;
        e = cudaEventRecord(ev, (cudaStream_t)streams[i]);
        if (e == cudaSuccess) e = cudaStreamWaitEvent((cudaStream_t)main_stream, ev, 0);
        cudaEventDestroy(ev);
    }
    return e == cudaSuccess ? DFB_OK : dfb::set_cuda_error("dfb_join", e);
}
