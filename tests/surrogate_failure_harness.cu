// The surrogate with a tensor-map encoder that fails on request, on the host
// (tests/test_gpu_surrogate_failures.py). Test infrastructure only.
#include <cuda.h>
#include <cuda_runtime.h>

#include <string>

namespace hidem {
thread_local std::string g_nocontext_error;
}

static int g_left = 1 << 30;  // encodings until one fails
static void *g_real;
static CUresult failing_encode(CUtensorMap *m, CUtensorMapDataType t, cuuint32_t rank, void *base, const cuuint64_t *dims,
                               const cuuint64_t *strides, const cuuint32_t *box, const cuuint32_t *es,
                               CUtensorMapInterleave il, CUtensorMapSwizzle sw, CUtensorMapL2promotion l2,
                               CUtensorMapFloatOOBfill fill) {
    if (g_left-- <= 0) return CUDA_ERROR_INVALID_VALUE;
    return reinterpret_cast<decltype(&failing_encode)>(g_real)(m, t, rank, base, dims, strides, box, es, il, sw, l2, fill);
}
static cudaError_t failing_entry_point(const char *name, void **p, unsigned long long flags,
                                       cudaDriverEntryPointQueryResult *q) {
    const cudaError_t e = cudaGetDriverEntryPoint(name, &g_real, flags, q);
    *p = reinterpret_cast<void *>(&failing_encode);
    return e;
}
#define cudaGetDriverEntryPoint failing_entry_point
#include "../hidem_b200/csrc/surrogate.cu"
#undef cudaGetDriverEntryPoint

// the encodings one training step takes
extern "C" int step_encodings(hidem_surrogate *s) {
    g_left = 1 << 30;
    if (hidem_surrogate_train(s, 1, nullptr) != HIDEM_OK) return -1;
    const int used = (1 << 30) - g_left;
    g_left = 1 << 30;
    return used;
}

// One training step whose encoding number `fail` (from 0) fails. 0: it was refused, and once the
// surrogate's stream is idle no side stream has work left; else what is wrong.
extern "C" int failed_step(hidem_surrogate *s, int fail) {
    g_left = fail;
    double loss = 0;
    const hidem_status st = hidem_surrogate_train(s, 1, &loss);
    g_left = 1 << 30;
    cudaStreamSynchronize(s->stream);
    int left = 0;
    for (size_t l = 0; l < s->side.size(); ++l)
        if (cudaStreamQuery(s->side[l]) != cudaSuccess) left |= 1 << l;
    return st != HIDEM_ERR_CUDA ? -1 : left;
}
