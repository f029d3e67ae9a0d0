// The rule for the unit layout's rows (units_rows) on the host: "n regular length stride offset batch ->
// way" over a grid, one line each.
#include "../../opensubdiv_gb300/csrc/stencils_units.cu"

namespace gb300 {
std::atomic<uint64_t> g_launches{0};
int fail(int code, const char *, ...) { return code; }
int ok() { return GB300_OK; }
int check_cuda(cudaError_t, const char *) { return GB300_OK; }
int check_launch(const char *) { return GB300_OK; }
int num_sms() { return 152; }
int status_word_address(int **) { return GB300_OK; }
}  // namespace gb300

int main() {
    for (int n : {65536, 262143, 262144, 524288, 1 << 20, 3 << 19, 2 << 20, 4 << 20, 8600000})
        for (int regular = 0; regular < 2; ++regular)
            for (int length = 1; length <= 33; ++length)
                for (int gap = 0; gap <= 12; ++gap)
                    for (int offset = 0; offset < 8; ++offset)
                        for (int batch = 0; batch < 2; ++batch) {
                            gb300::UnitTable t;
                            t.numStencils = n;
                            t.numSlices = n / 200;
                            t.regular = regular;
                            const int stride = length + gap;
                            const float *dst = (const float *)(uintptr_t)(1024 + 4 * offset);
                            printf("%d %d %d %d %d %d %d\n", n, regular, length, stride, offset,
                                   batch, (int)gb300::units_rows(t, dst, stride, length,
                                                                 (long long)n * stride * 4, batch));
                        }
    return 0;
}
