// Host-only check of what the translations without atomics (owner.cu) hold after a failed allocation: the runtime's
// calls are stand-ins on host memory, of which the n-th allocation fails, for every n in turn.  A later attempt has to
// succeed, and after free_owner() nothing may be left.  Prints JSON for the test to check.  Kernels are not run:
// there is no GPU (with one the program says so and stops).
#include <cuda_runtime.h>
#include <cstdlib>
#include <cstring>

static long live = 0, fail_in = 0, calls = 0;
static cudaError_t fake_malloc(void **p, size_t n)
{
    calls++;
    if (fail_in > 0 && --fail_in == 0) return cudaErrorMemoryAllocation;
    *p = calloc(1, n ? n : 1);
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
static cudaError_t fake_copy(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t = 0)
{
    memcpy(d, s, n);
    return cudaSuccess;
}
static cudaError_t fake_set(void *d, int v, size_t n, cudaStream_t)
{
    memset(d, v, n);
    return cudaSuccess;
}
static cudaError_t fine() { return cudaSuccess; }
#define cudaMalloc fake_malloc
#define cudaFree fake_free
#define cudaMemcpyAsync fake_copy
#define cudaMemcpy fake_copy
#define cudaMemsetAsync fake_set
#define cudaStreamSynchronize(s) fine()
#define cudaStreamWaitEvent(a, b, c) fine()
#define cudaEventQuery(e) fine()
#define cudaEventRecord(a, b) fine()
#define cudaEventSynchronize(e) fine()
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
void direction_classes(const Plan *, int, int nkeys, std::vector<int> &cls, std::vector<int> &rep)
{
    cls.assign(nkeys, 0);
    rep.assign(1, 0);
}
int ensure_whole_tables(Plan *P)
{
    return P->rot32_whole || fake_malloc((void **)&P->rot32_whole, 64) == cudaSuccess ? 0 : FMM_ERR_CUDA;
}
} // namespace fmm
void fmm_set_error(const char *, ...) {}

using namespace fmm;
static void nothing(Plan *, int, int) {}
static void nothing(Plan *) {}

int main()
{
    int n = 0;
    if (cudaGetDeviceCount(&n) == cudaSuccess && n > 0) {
        printf("{\"gpu\": %d}\n", n);
        return 0;
    }
    printf("{\"gpu\": 0, \"runs\": [");
    bool first = true;
    for (int type : {OWN_FP64, OWN_FF, OWN_FP32})
        for (int at = 1;; at++) {
            Plan *P = new Plan();
            std::vector<int> ints(4096, 0);
            std::vector<short> shorts(4096, 0);
            std::vector<unsigned char> bytes(4096, 0);
            P->lmin = 2;
            P->lmax = 4;
            P->pmax = 12;
            P->pleaf = 8;
            for (int l = 2; l <= 4; l++) {
                LevelDev &L = P->lev[l];
                L.nb = 8 * l;
                L.p = 16 - 2 * l;
                L.num_sr = 40 * l;
                L.parent = L.sr_beg = L.child_beg = L.child_list = L.sr_src = ints.data();
                L.sr_dir = shorts.data();
                L.octant = bytes.data();
            }
            const long before = live;
            calls = 0;
            fail_in = at;
            const int st = translate_owner(P, type, nothing, nothing);
            const bool failed = fail_in == 0;
            fail_in = 0;
            const int again = translate_owner(P, type, nothing, nothing);
            free_owner(P);
            fake_free(P->rot32_whole);
            printf("%s{\"type\": %d, \"at\": %d, \"failed\": %d, \"status\": %d, \"again\": %d, \"left\": %ld}", first ? "" : ", ", type, at,
                   failed ? 1 : 0, st, again, live - before);
            first = false;
            delete P;
            if (!failed) break;  // fewer allocations than `at`
        }
    printf("]}\n");
    return 0;
}
