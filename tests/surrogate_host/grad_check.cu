// mtg_surrogate_loss_grad on the CPU, with the runtime calls and the network's
// launches replaced: the caller's gradient and loss are written when the call succeeds
// and left alone when a bounded wait of the kernels ran out.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>

namespace fake {
template <class T>
cudaError_t alloc(T **p, size_t n) { return (*p = (T *)malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
inline cudaError_t release(void *p) { return free(p), cudaSuccess; }
inline cudaError_t copy(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { return memcpy(d, s, n), cudaSuccess; }
inline cudaError_t fill(void *p, int v, size_t n, cudaStream_t) { return memset(p, v, n), cudaSuccess; }
inline cudaError_t ok(...) { return cudaSuccess; }
}  // namespace fake
#define cudaMalloc fake::alloc
#define cudaMallocHost fake::alloc
#define cudaFree fake::release
#define cudaMemcpyAsync fake::copy
#define cudaMemsetAsync fake::fill
#define cudaSetDevice fake::ok
#define cudaStreamSynchronize fake::ok
#include "surrogate.cu"

static int timeout_bit = 0;
namespace mtg {
namespace mlp {
int backward_parts(int) { return 3; }
cudaError_t launch_forward_tc(const Weights &, const float *, const int *, int, const float *, float *, float *, int *,
                              cudaStream_t) { return cudaSuccess; }
cudaError_t launch_backward_tc(const Weights &, const float *, const int *, const float *, const float *, int,
                               const float *, const float *, float *, float *loss_part, int *err, cudaStream_t) {
    for (int k = 0; k < 3; k++) loss_part[k] = 4.0f;
    *err |= timeout_bit;
    return cudaSuccess;
}
cudaError_t launch_grad_sum(const float *, int, float *grad, cudaStream_t) {
    for (int i = 0; i < kParams; i++) grad[i] = 7.0f;
    return cudaSuccess;
}
uint32_t tc_default_spin() { return 1; }
}  // namespace mlp
}  // namespace mtg
int mtg_internal_fail(int code, const char *) { return code; }

int main() {
    static mtg_surrogate s;
    int err = 0;
    s.err = &err;
    std::vector<float> staging(mlp::kParams);
    s.grad = staging.data();
    for (float &v : s.h_ynorm) v = 1.0f;
    std::vector<float> X(5 * mlp::kIn, 1.0f), T(5 * mlp::kOut, 1.0f), g(mlp::kParams, -1.0f);
    double loss = -1.0;
    timeout_bit = kErrTimeout;
    const int rc = mtg_surrogate_loss_grad(&s, X.data(), T.data(), 5, &loss, g.data());
    int touched = 0;
    for (float v : g) touched += v != -1.0f;
    printf("timeout: rc %d touched %d loss %g err %d\n", rc, touched, loss, err);
    timeout_bit = 0;
    const int rc2 = mtg_surrogate_loss_grad(&s, X.data(), T.data(), 5, &loss, g.data());
    touched = 0;
    for (float v : g) touched += v == 7.0f;
    printf("success: rc %d written %d loss %g\n", rc2, touched, loss);
    return 0;
}
