// evp_engine.cu's error paths on the CPU (host_cuda_fake.hpp): two members that need different kernels in
// every pass, so that a pass forks onto the auxiliary streams inside the capture.
#include "host_cuda_fake.hpp"

#include "evp_engine.cu"

namespace evp {
static int g_throw;  // a launch that throws inside the capture
void member_jobs_voxel(const Dev& d, MemberJobs& mj) {
    for (int k : {(int)BK_CORR, (int)BK_NEWTON}) {
        mj.job[0][k] = Job{0, 0, 1, 1, 1, 1};
        mj.variant[0][k] = d.nsys;
        mj.threads[0][k] = 32;
    }
}
void member_jobs_fft(const Dev& d, const FftPlan1D&, const FftPlan1D&, const FftPlan1D&, int, MemberJobs& mj) {
    for (int k : {(int)BK_XFWD, (int)BK_YFWD, (int)BK_ZGREEN, (int)BK_YINV, (int)BK_XINV}) {
        mj.job[0][k] = Job{0, 0, 1, 1, 1, 1};
        mj.variant[0][k] = d.nsys;
        mj.threads[0][k] = 32;
    }
}
void launch_batched_voxel(const BatchLaunch&, const BatchParams&, cudaStream_t) {
    if (g_throw) throw std::runtime_error("a launcher's exception");
}
void launch_batched_fft(const BatchLaunch&, const BatchParams&, cudaStream_t) {}
void launch_control(const BatchSolve*, int, int*, cudaStream_t) {}
}  // namespace evp

// One engine whose first launch fails in `call` at its n-th use (or in a launcher: "throw"), then a second launch that
// must work.  Returns -1 when the call was not reached, 0 when all is well, else what was wrong: 1 no exception,
// 2 the stream was left in capture, 4 the second launch failed, 8 a stream, event or graph was left behind.
extern "C" int engine_case(const char* call, int n) {
    using namespace evp;
    fake::reset();
    int bad = 0;
    bool reached = false;
    {
        Engine eng((cudaStream_t)16);
        std::vector<Engine::Member> m(2);
        for (int i = 0; i < 2; i++) {
            std::memset(&m[i], 0, sizeof(m[i]));
            m[i].e.d.nsys = i + 1;
        }
        eng.set_members(m);
        fake::calls.clear();
        g_throw = std::string(call) == "throw";
        fake::fail_call = call;
        fake::fail_at = n;
        bool threw = false;
        try {
            eng.launch(2, nullptr);
        } catch (std::exception&) {
            threw = true;
        }
        reached = g_throw || fake::calls[call] > n;
        g_throw = 0;
        fake::fail_call.clear();
        if (reached && !threw) bad |= 1;
        if (fake::capturing) bad |= 2;
        try {
            eng.launch(2, nullptr);
        } catch (std::exception&) {
            bad |= 4;
        }
    }
    if (!fake::device.empty() || !fake::streams.empty() || !fake::events.empty()) bad |= 8;
    return reached ? bad : -1;
}
