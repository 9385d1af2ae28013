// Host-only check that the lists and work units of the batched passes (batched.cu) are on the device when the
// functions that make them return: the plans' streams do not wait for the default stream, on which a copy from
// pageable memory may go on after cudaMemcpy.  The runtime's calls are stand-ins on host memory; a copy counts as
// under way until its stream is waited for.  Prints JSON for the test to check.  Kernels are not run: there is no GPU
// (with one the program says so and stops).
#include <cuda_runtime.h>
#include <cstdlib>
#include <cstring>

static long under_way = 0, copies = 0;
static cudaError_t fake_malloc(void **p, size_t n)
{
    *p = calloc(1, n ? n : 1);
    return cudaSuccess;
}
template <class T> static cudaError_t fake_malloc(T **p, size_t n) { return fake_malloc((void **)p, n); }
static cudaError_t fake_free(const void *p)
{
    free((void *)p);
    return cudaSuccess;
}
static cudaError_t fake_copy(void *d, const void *s, size_t n, cudaMemcpyKind)
{
    memcpy(d, s, n);
    under_way++;
    copies++;
    return cudaSuccess;
}
static cudaError_t fake_sync(cudaStream_t s)
{
    if (s == 0 || s == cudaStreamLegacy) under_way = 0;
    return cudaSuccess;
}
static cudaError_t fine() { return cudaSuccess; }
#define cudaMalloc fake_malloc
#define cudaFree fake_free
#define cudaMemcpy fake_copy
#define cudaStreamSynchronize fake_sync
#define cudaGetLastError() fine()
#include "../../fmbem_gpu_c_gb300/csrc/batched.cu"
#include <cstdio>

// what batched.cu takes from the rest of the library, unused here
namespace fmm {
int raise_smem_limit(const void *, size_t, size_t *) { return 0; }
cudaError_t dev_alloc(Plan *, void **p, size_t n) { return fake_malloc(p, n); }
int launch_pass32(Plan *, int, int, int, cudaStream_t) { return 0; }
} // namespace fmm
void fmm_set_error(const char *, ...) {}

using namespace fmm;

int main()
{
    int n = 0;
    if (cudaGetDeviceCount(&n) == cudaSuccess && n > 0) {
        printf("{\"gpu\": %d}\n", n);
        return 0;
    }
    printf("{\"gpu\": 0, \"left\": [");
    for (int form = 0; form < 2; form++) {
        RcrList L;
        const int nkeys = 8;
        L.key_beg.assign(1, 0);
        for (int d = 0; d < nkeys; d++) {
            for (int i = 0; i < 5; i++) L.dst_rank.push_back(i);
            L.key_beg.push_back(5 * (d + 1));
            L.key_w.push_back(0);
            L.cls_of_key.push_back(d & 1);
        }
        L.ndst_rank = 5;
        RcrPass ps = {};
        ps.p = ps.pin = ps.pout = 9;
        std::vector<int> off(10, 0);
        const int a = ensure_items(L, form, 20, 0);
        const long left = under_way;
        const int b = ensure_units(off, L.form[form], form == FORM_FOLDED, ps);
        printf("%s[%d, %ld, %d, %ld]", form ? ", " : "", a, left, b, under_way);
    }
    printf("], \"copies\": %ld}\n", copies);
    return 0;
}
