// Library-wide state and the small informational entry points of ogle_cuda.h.
#include <atomic>
#include <cstdlib>

#include "common.cuh"

namespace ogle {
int read_tc_error();
int clear_tc_error();
void set_role_wait_limit(long polls);
std::atomic<uint64_t> g_launch_count{0};
static thread_local char g_last_error[256] = "";
void set_last_error(cudaError_t e) {
    const char* s = cudaGetErrorString(e);
    int i = 0;
    for (; s[i] && i < 255; ++i) g_last_error[i] = s[i];
    g_last_error[i] = 0;
}
namespace {
// -1: not set by the caller. The environment, when it names a value, wins over the caller.
std::atomic<int> g_overlapped{-1};
}
bool overlapped_launches_enabled(bool asked_for) {
    // measured 5 % faster at one image per step, nothing at 32, 1-2 % slower at 256: off unless the
    // environment or the caller (a session whose tensors are small) turns it on
    static const int env = [] { const char* e = getenv("OGLE_PDL"); return e ? (e[0] == '1' ? 1 : 0) : -1; }();
    if (env >= 0) return env == 1;
    return asked_for || g_overlapped.load(std::memory_order_relaxed) == 1;
}
void set_overlapped_launches(int on) { g_overlapped.store(on ? 1 : 0, std::memory_order_relaxed); }
void set_last_error(const char* s) {
    int i = 0;
    for (; s[i] && i < 255; ++i) g_last_error[i] = s[i];
    g_last_error[i] = 0;
}
namespace { thread_local OgleContraction g_contraction = {}; }
void note_contraction(int form, int ranges, int n_tile, bool overlapped) { g_contraction = {form, ranges, n_tile, overlapped ? 1 : 0}; }
}  // namespace ogle

extern "C" {

int ogle_cuda_last_contraction(OgleContraction* out) {
    if (!out) return OGLE_ERR_INVALID;
    *out = ogle::g_contraction;
    return OGLE_OK;
}

const char* ogle_cuda_status_string(int status) {
    switch (status) {
        case OGLE_OK: return "ok";
        case OGLE_ERR_INVALID: return "invalid argument";
        case OGLE_ERR_UNSUPPORTED: return "unsupported (outside what the reference defines)";
        case OGLE_ERR_CUDA: return "CUDA call failed";
        case OGLE_ERR_ALIGNMENT: return "pointer or stride not 16-byte aligned";
        case OGLE_ERR_DEVICE: return "no sm_100 device";
        case OGLE_ERR_TIMEOUT: return "bounded device-side wait gave up";
        default: return "unknown status";
    }
}

const char* ogle_cuda_build_info(void) { return "ogle_cuda 0.1 sm_100a"; }

uint64_t ogle_cuda_launch_count(void) { return ogle::g_launch_count.load(std::memory_order_relaxed); }

const char* ogle_cuda_last_error(void) { return ogle::g_last_error; }

int ogle_cuda_device_status(void) {
    if (cudaDeviceSynchronize() != cudaSuccess) return OGLE_ERR_CUDA;
    const int v = ogle::read_tc_error();
    return v == 0 ? OGLE_OK : (v < 0 ? OGLE_ERR_CUDA : OGLE_ERR_TIMEOUT);
}

int ogle_cuda_device_status_detail(void) {
    if (cudaDeviceSynchronize() != cudaSuccess) return OGLE_ERR_CUDA;
    return ogle::read_tc_error();
}

int ogle_cuda_set_overlapped_launches(int on) {
    ogle::set_overlapped_launches(on);
    return OGLE_OK;
}

int ogle_cuda_set_wait_limit(long polls) {
    ogle::set_role_wait_limit(polls);
    return OGLE_OK;
}

int ogle_cuda_clear_device_status(void) { return ogle::clear_tc_error() == 0 ? OGLE_OK : OGLE_ERR_CUDA; }

}  // extern "C"
