// evp_green.cu's C entries on the CPU (host_cuda_fake.hpp), with a launch that throws, fails or succeeds.
#include "host_cuda_fake.hpp"

#include "evp_green.cu"

#include <stdexcept>

static std::string g_message;
static int g_launch;  // 0: works; 1: throws, as a length that fits no block does; 2: a launch error

namespace evp {
void set_last_error(const std::string& m) { g_message = m; }
void fft_configure() {}
FftPlan1D make_plan(int n) {
    FftPlan1D p{};
    p.n = n;
    return p;
}
cudaMemPool_t solver_pool() { return (cudaMemPool_t)8; }
cudaMemPool_t operator_pool() { return (cudaMemPool_t)8; }
void release_pools() {}
void launch_green_apply(const Dev&, const FftPlan1D&, const FftPlan1D&, const FftPlan1D&, const double*, double*, const double*,
                        const double*, cudaStream_t) {
    if (g_launch == 1) throw std::runtime_error("FFT pencils of length 256 do not fit one block");
    if (g_launch == 2) fake::last = cudaErrorInvalidConfiguration;
}
}  // namespace evp

extern "C" {
// One call of an entry; fail: an entry of the runtime that fails at its first call, or "".  Returns the status,
// -100 when an exception left the entry; *left counts the device allocations that were not freed.
int green_call(int noalloc, int n1, int n2, int n3, int launch, const char* fail, int* left) {
    fake::reset();
    g_message.clear();
    g_launch = launch;
    fake::fail_call = fail;
    fake::fail_at = 0;
    double c[81] = {}, x = 0.0;
    int rc;
    try {
        rc = noalloc ? evp_green_apply_noalloc(&x, &x, n1, n2, n3, c, c, nullptr) : evp_green_apply(&x, &x, n1, n2, n3, c, c, nullptr);
    } catch (...) {
        rc = -100;
    }
    *left = (int)fake::device.size();
    return rc;
}
const char* green_message(void) { return g_message.c_str(); }
}
