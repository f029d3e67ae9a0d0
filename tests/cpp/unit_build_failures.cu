// build_units over a CUDA runtime whose calls are faked (fake_cudart.cpp): no kernel runs, and one
// call at a time fails.  After a failure nothing more is queued -- what comes next works by what the
// failed step was to compute --, the status tells an allocation from a CUDA error, and nothing is
// left allocated.  Prints "ok <allocations> <calls>".
#include "../../opensubdiv_gb300/csrc/unit_build.cu"

#include <cstdarg>
#include <cstdlib>

extern "C" {
extern int fake_allocations, fake_fail_allocation, fake_live;
extern int fake_calls, fake_fail_call, fake_failed;
extern int fake_launches_after_failure;
int fake_allocate(void **p, size_t bytes);
void fake_release(void *p);
void fake_reset(int fail_allocation, int fail_call);
}

namespace gb300 {
std::atomic<uint64_t> g_launches{0};
int fail(int code, const char *, ...) { return code; }
int ok() { return GB300_OK; }
int check_cuda(cudaError_t e, const char *) {
    return e == cudaSuccess                 ? GB300_OK
           : e == cudaErrorMemoryAllocation ? GB300_ERR_OUT_OF_MEMORY
                                            : GB300_ERR_CUDA;
}
int check_launch(const char *who) { return check_cuda(cudaGetLastError(), who); }
int num_sms() { return 152; }
int scratch_alloc(void **p, size_t bytes, cudaStream_t, const char *who) {
    return check_cuda((cudaError_t)fake_allocate(p, bytes), who);
}
void scratch_free(void *p, cudaStream_t) { fake_release(p); }
}  // namespace gb300

static int run(int fail_allocation, int fail_call, bool &built) {
    fake_reset(fail_allocation, fail_call);
    static int some[4] = {};
    gb300::UnitTable t;
    void *owned[2];
    const int st = gb300::build_units(70000, some, some, some, (const float *)some, 0, t, owned,
                                      "build_units");
    built = owned[0] && owned[1];
    if (!built && (owned[0] || owned[1] || t.numSlices)) return -1;
    for (void *p : owned) cudaFree(p);
    return st;
}

#define CHECK(x)                                                                             \
    if (!(x)) {                                                                              \
        printf("%s, allocation %d call %d: status %d, %d live, %d launches\n", #x, a, c, st, \
               fake_live, fake_launches_after_failure);                                      \
        return 1;                                                                            \
    }

int main() {
    int a = -1, c = -1;
    bool built = false;
    int st = run(a, c, built);
    CHECK(st == GB300_OK && built && fake_live == 0);
    const int allocations = fake_allocations, calls = fake_calls;
    for (a = 0; a < allocations; ++a) {
        st = run(a, c, built);
        CHECK(fake_failed && !built && fake_live == 0 && fake_launches_after_failure == 0);
        CHECK(st == GB300_ERR_OUT_OF_MEMORY);
    }
    a = -1;
    for (c = 0; c < calls; ++c) {
        st = run(a, c, built);
        CHECK(fake_failed && !built && fake_live == 0 && fake_launches_after_failure == 0);
        CHECK(st == GB300_ERR_CUDA);
    }
    printf("ok %d %d\n", allocations, calls);
    return 0;
}
