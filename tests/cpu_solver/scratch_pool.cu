// Host-only check of the scratch buffers that the plans of a device share (owner.cu): who gets which buffer, and
// behind which event.  The runtime's calls are stand-ins: an event is passed once the test says so.  Prints JSON for the
// test to check.  Kernels are not run: there is no GPU (with one the program says so and stops).
#include <cuda_runtime.h>
#include <cstdlib>

static bool passed = true;  // all recorded work is done
static long waits = 0, live = 0;
static cudaError_t fake_malloc(void **p, size_t)
{
    *p = malloc(1);
    live++;
    return cudaSuccess;
}
template <class T> static cudaError_t fake_malloc(T **p, size_t n) { return fake_malloc((void **)p, n); }
static cudaError_t fake_free(const void *p)
{
    if (p) live--;
    free((void *)p);
    return cudaSuccess;
}
static cudaError_t fake_wait()
{
    if (!passed) waits++;
    return cudaSuccess;
}
static cudaError_t fine() { return cudaSuccess; }
#define cudaMalloc fake_malloc
#define cudaFree fake_free
#define cudaMemcpyAsync(...) fine()
#define cudaMemcpy(...) fine()
#define cudaMemsetAsync(...) fine()
#define cudaStreamSynchronize(s) fine()
#define cudaStreamWaitEvent(a, b, c) fake_wait()
#define cudaEventQuery(e) (passed ? cudaSuccess : cudaErrorNotReady)
#define cudaEventRecord(a, b) fine()
#define cudaEventSynchronize(e) fake_wait()
#define cudaEventCreateWithFlags(e, f) fine()
#define cudaEventDestroy(e) fine()
#define cudaGetLastError() fine()
#include "../../fmbem_gpu_c_gb300/csrc/owner.cu"
#undef cudaGetDeviceCount
#include <cstdio>

// what owner.cu takes from the rest of the library
namespace fmm {
int raise_smem_limit(const void *, size_t, size_t *) { return 0; }
cudaError_t dev_alloc(Plan *, void **p, size_t n) { return fake_malloc(p, n); }
void direction_classes(const Plan *, int, int, std::vector<int> &, std::vector<int> &) {}
int ensure_whole_tables(Plan *) { return 0; }
} // namespace fmm
void fmm_set_error(const char *, ...) {}

using namespace fmm;

static int use(Plan *P)  // one call's translations: the buffer that they got
{
    void *part = nullptr;
    if (pool_take(P, PART_CAP, &part) || pool_give(P)) return -1;
    return P->own_scratch;
}

int main()
{
    int n = 0;
    if (cudaGetDeviceCount(&n) == cudaSuccess && n > 0) {
        printf("{\"gpu\": %d}\n", n);
        return 0;
    }
    const int most = (int)(POOL_CAP / PART_CAP);
    std::vector<Plan *> plans;
    for (int i = 0; i <= most; i++) plans.push_back(new Plan());
    printf("{\"gpu\": 0, \"most\": %d, \"one_by_one\": [", most);
    for (int i = most; i >= 0; i--) printf("%s%d", i < most ? ", " : "", use(plans[i]));
    const long held = live;
    passed = false;
    printf("], \"held\": %ld, \"together\": [", held);
    for (int i = 0; i < most; i++) printf("%s%d", i ? ", " : "", use(plans[i]));
    printf("], \"again\": [");
    waits = 0;
    for (int i = 0; i < most; i++) printf("%s%d", i ? ", " : "", use(plans[i]));
    printf("], \"again_waits\": %ld, ", waits);
    waits = 0;
    const int shared = use(plans[most]);  // one plan more than buffers
    printf("\"over\": %d, \"over_waits\": %ld, ", shared, waits);
    int at = 0;
    for (int i = 0; i < most; i++)
        if (plans[i]->own_scratch == shared) at = i;
    waits = 0;
    use(plans[at]);  // the plan whose buffer that was
    printf("\"displaced_waits\": %ld, ", waits);
    // a plan that goes, and another at its address
    Plan *gone = plans[1];
    pool_leave(gone);
    waits = 0;
    use(gone);
    printf("\"next_waits\": %ld, ", waits);
    for (Plan *P : plans) {
        pool_leave(P);
        delete P;
    }
    printf("\"live\": %ld}\n", live);
    return 0;
}
