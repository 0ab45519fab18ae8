// late_error.cu -- the solve (PART 0) and the gradient vector flow (PART 1) with a
// host-side fake: once the call has read its control word, the word's error field
// is set on the device, as a sweep launched after that read would set it.
#include <cuda_runtime.h>

namespace {
size_t g_ctrl_bytes = 0, g_error_offset = 0;
int g_reads = 0, g_fail_after = 0;   // 0: never

cudaError_t fake_memcpy(void *dst, const void *src, size_t n, cudaMemcpyKind kind, cudaStream_t st)
{
    cudaError_t e = cudaMemcpyAsync(dst, src, n, kind, st);
    if (e == cudaSuccess && kind == cudaMemcpyDeviceToHost && n == g_ctrl_bytes && ++g_reads == g_fail_after)
        e = cudaMemsetAsync((char *)const_cast<void *>(src) + g_error_offset, 1, 4, st);
    return e;
}
}  // namespace

#define cudaMemcpyAsync fake_memcpy
#if PART == 0
#include "maxflow.cu"
typedef m16::MfCtrl Ctrl;
#else
#include "gvf.cu"
typedef m16::GvfCtrl Ctrl;
#endif

// the next call's control word is marked failed after `reads` reads of it (0: never)
extern "C" void fail_after(int reads)
{
    g_ctrl_bytes = sizeof(Ctrl);
    g_error_offset = offsetof(Ctrl, error);
    g_reads = 0;
    g_fail_after = reads;
}
