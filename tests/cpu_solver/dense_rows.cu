// Host-only check of where the dense tensor-core passes (tc_dense.cu) copy a source row from: prints JSON lines for
// the test to check.  Nothing runs on a GPU.
#include "../../fmbem_gpu_c_gb300/csrc/tc_dense.cu"
#include <cstdio>

// what tc_dense.cu takes from the rest of the library, unused here
namespace fmm {
int raise_smem_limit(const void *, size_t, size_t *) { return 0; }
cudaError_t dev_alloc(Plan *, void **, size_t) { return cudaErrorNotSupported; }
RcrList *pass32_desc(Plan *, int, int, int, RcrPass &) { return nullptr; }
int gen_dense_rcr(Plan *, int, int, const int *, int, double2 *) { return 0; }
void direction_classes(const Plan *, int, int, std::vector<int> &, std::vector<int> &) {}
} // namespace fmm
void fmm_set_error(const char *, ...) {}

int main()
{
    const int rows[] = {-1, 0, 1, 33554431, 33554432, 40000001, 268435457, 2147483647};
    for (int row : rows)
        for (int P2 : {16, 25, 196, 256})
            for (int c0 : {0, 9, 49})
                for (int cnt : {7, 15, 16}) {
                    const fmm::RowCopy c = fmm::row_copy(row, P2, c0, cnt);
                    printf("[%d, %d, %d, %d, %llu, %d]\n", row, P2, c0, cnt, c.from, c.n);
                }
    return 0;
}
