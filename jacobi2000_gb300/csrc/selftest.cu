// Self-test of the bounded device-side waits: the production mbarrier wait
// (tc::mbar_wait) with a caller-chosen limit, on a barrier that nothing
// arrives on (or, as the control case, one that its own thread completes).
// The kernel gives up, sets the error flag and returns; the host reads the
// flag with the check every batch call uses and reports JC_DEVICE_TIMEOUT.
// No kernel is left running and the context stays usable.
#include <cstring>
#include <vector>

#include "runtime.hpp"
#include "tc.cuh"

namespace jc {

namespace {

__global__ void wait_selftest_kernel(int satisfy, unsigned long long limit_ns, int* err) {
    __shared__ uint64_t bar;
    __shared__ int cta_failed;
    if (threadIdx.x == 0) {
        tc::mbar_init(&bar, 1);
        tc::fence_barrier_init();
        cta_failed = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0 && satisfy) tc::mbar_arrive(&bar);
    // every thread of the CTA waits on phase 0; when the limit runs out the
    // first to notice sets the CTA flag and the others return at once
    tc::mbar_wait(&bar, 0, err, &cta_failed, limit_ns);
    __syncthreads();
}

}  // namespace

void selftest_device_wait(int satisfy, unsigned limit_us) {
    if (limit_us < 1 || limit_us > 2000000u) throw Error(JC_BAD_ARGUMENT, "limit_us must be in [1, 2000000]");
    int* flag = nullptr;
    cuda_check(cudaMalloc(&flag, sizeof(int)), "cudaMalloc", JC_OVER_BUDGET);
    struct Free {
        int* p;
        ~Free() { cudaFree(p); }
    } guard{flag};
    cuda_check(cudaMemset(flag, 0, sizeof(int)), "cudaMemset");
    wait_selftest_kernel<<<1, 64>>>(satisfy, (unsigned long long)limit_us * 1000ull, flag);
    cuda_check(cudaGetLastError(), "wait self-test launch");
    check_wait_flag(flag, nullptr);
}

// The same wait running out in a device call of `m`, as far as the model can tell: it
// sets the model's flag, on the model's stream, and nothing is read back.
void selftest_model_wait(Model& m, unsigned limit_us) {
    if (limit_us < 1 || limit_us > 2000000u) throw Error(JC_BAD_ARGUMENT, "limit_us must be in [1, 2000000]");
    wait_selftest_kernel<<<1, 64, 0, m.stream>>>(0, (unsigned long long)limit_us * 1000ull, m.wait_flag());
    cuda_check(cudaGetLastError(), "wait self-test launch");
}

// The projection of one 100 x 60 state by a cluster of eight CTAs, one unit's total
// of pass `pass` unsent (to the cluster's first CTA alone when one_peer). CTAs whose
// sums are not whole must store nothing: that is all of them, or in the last pass the
// first alone, which holds the instance's scalars and units 0 to 3 of segment 0.
void selftest_projection_wait(int pass, int one_peer, unsigned limit_us) {
    if (limit_us < 1 || limit_us > 2000000u) throw Error(JC_BAD_ARGUMENT, "limit_us must be in [1, 2000000]");
    if (pass < -1 || pass > 2) throw Error(JC_BAD_ARGUMENT, "pass must be in [-1, 2]");
    constexpr int nx = 100, ny = 60, n = nx * ny;
    DeviceArena a;
    Dims d{};
    d.C = 3;
    for (float& v : d.norm_std) v = 1.0f;
    d.norm_depth = d.energy_r_max = 1.0f;
    d.g = 9.81f;
    std::vector<float> x(3 * n), y(3 * n);
    for (int i = 0; i < 3 * n; i++) x[i] = 0.001f * (float)(i % 97);
    InstDev I{};
    I.nx = nx;
    I.ny = ny;
    I.flags = JC_PROJECT_MASS | JC_PROJECT_ENERGY;
    I.state = a.alloc_n<float>(x.size());
    const ProjSlot s0{0.5, 1.0, 0.0, 1.0};
    ProjSlot s1;
    Pack p{};
    p.n_inst = 1;
    p.max_inst_cells = n;
    p.inst = a.alloc_n<InstDev>(1);
    p.proj = a.alloc_n<ProjSlot>(1);
    p.err = a.alloc_n<int>(1);
    cuda_check(cudaMemset(p.err, 0, sizeof(int)), "cudaMemset");
    cuda_check(cudaMemcpy(p.inst, &I, sizeof(I), cudaMemcpyHostToDevice), "H2D", JC_MAP);
    cuda_check(cudaMemcpy(p.proj, &s0, sizeof(s0), cudaMemcpyHostToDevice), "H2D", JC_MAP);
    cuda_check(cudaMemcpy(I.state, x.data(), x.size() * sizeof(float), cudaMemcpyHostToDevice), "H2D", JC_MAP);
    projection_selftest(d, p, pass, one_peer, (unsigned long long)limit_us * 1000ull, nullptr);
    cuda_check(cudaMemcpy(y.data(), I.state, y.size() * sizeof(float), cudaMemcpyDeviceToHost), "D2H", JC_MAP);
    cuda_check(cudaMemcpy(&s1, p.proj, sizeof(s1), cudaMemcpyDeviceToHost), "D2H", JC_MAP);
    bool state_kept = true, slot_kept = std::memcmp(&s0, &s1, sizeof(s0)) == 0;
    for (int i = 0; i < 3 * n; i++) {
        const int cell = i % n;
        if (pass == 2 && one_peer && !(cell < 4096 && cell % 512 < 128)) continue;
        if (std::memcmp(&x[i], &y[i], sizeof(float)) != 0) state_kept = false;
    }
    if ((pass >= 0) != state_kept || (pass >= 0) != slot_kept)
        throw Error(JC_CUDA_ERROR, pass >= 0 ? "the projection stored results of sums that are not whole"
                                             : "the projection stored nothing");
    check_wait_flag(p.err, nullptr);
}

}  // namespace jc
