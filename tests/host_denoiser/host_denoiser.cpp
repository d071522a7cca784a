// Test harness: the denoiser's host code (vviewer_gb300/csrc/denoise.cu,
// compiled for the host) on a device of the test's own, whose memory can run
// out and whose kernels only look at the addresses they are given.
#include <cstdlib>
#include <cstring>

#include "denoise_kernels.cuh"
#include "internal.h"

static size_t g_total = 0, g_used = 0;
static int g_bad = 0; // kernels launched on memory that is not there
static struct { char *p; size_t n; } g_live[256];

static void use(const void *p)
{
    bool there = false;
    for (auto &e : g_live)
        there |= e.p && (char *)p >= e.p && (char *)p < e.p + e.n;
    g_bad += !there;
}

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n)
{
    if (g_used + n > g_total)
        return cudaErrorMemoryAllocation;
    for (auto &e : g_live)
        if (!e.p) {
            e = {(char *)std::malloc(n), n};
            *p = e.p;
            g_used += n;
            return cudaSuccess;
        }
    return cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void *p)
{
    for (auto &e : g_live)
        if (e.p == p) {
            g_used -= e.n;
            std::free(p);
            e = {nullptr, 0};
        }
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind kind)
{
    use(kind == cudaMemcpyHostToDevice ? d : s);
    if (!g_bad)
        std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind kind, cudaStream_t)
{
    return cudaMemcpy(d, s, n, kind);
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t)
{
    use(d);
    if (!g_bad)
        std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "out of memory"; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = g_total - g_used; *t = g_total; return cudaSuccess; }
}

namespace vvpt {
bool reclaim_pools() { return false; }
}

namespace vvdn {
bool conv3x3(const ConvArgs &a, cudaStream_t, uint32_t *, ConvKernels) { use(a.in); if (!a.rgba) use(a.out); return true; }
bool conv3x3_concat(const ConvArgs &a, cudaStream_t, uint32_t *, ConvKernels) { use(a.in); use(a.coarse); use(a.out); return true; }
void inject_wait_timeout() {}
void conv3x3_wgrad(const bf16 *d, int, const bf16 *x, int, int, int, int, float *dw, float *db, cudaStream_t, uint32_t *, long)
{
    use(d), use(x), use(dw), use(db);
}
void sum_grads(const float *g, size_t, float *s, size_t, cudaStream_t) { use(g), use(s); }
void prepare_weights(const float *, const WeightTable &, bf16 *, bf16 *, cudaStream_t) {}
void pack_features(const float *, const float *, const float *, bf16 *x, int, cudaStream_t) { use(x); }
void avgpool2(const bf16 *i, bf16 *o, int, int, int, int, cudaStream_t) { use(i), use(o); }
void upcat(const bf16 *c, int, const bf16 *s, int, bf16 *o, int, int, int, cudaStream_t) { use(c), use(s), use(o); }
void upcat_backward(const bf16 *c, int, int, bf16 *a, bf16 *b, int, int, int, cudaStream_t) { use(c), use(a), use(b); }
void pool_backward_combine(const bf16 *s, const bf16 *p, const bf16 *e, bf16 *d, int, int, int, int, cudaStream_t) { use(s), use(p), use(e), use(d); }
void l1_loss(const float *o, int, const float *, bf16 *d, float *l, int, cudaStream_t) { use(o), use(d), use(l); }
void adam(float *p, const float *g, size_t, float *, float *, size_t, float, float, float, float, int, cudaStream_t) { use(p), use(g); }
void unpack_output(const float *y, int, float *, int, cudaStream_t) { use(y); }
}

// calls[k]: 0 apply, 1 gradients, on a w x h image with `room[k]` MiB of free
// device memory; status[k] its status, bad[k] whether kernels ran on memory
// that is not there.
extern "C" void host_denoiser_calls(int n, const int *calls, const int *w, const int *h, const int *room, int *status, int *bad)
{
    vvpt_ctx ctx;
    vvpt_denoiser *dn = nullptr;
    g_total = (size_t)1 << 30;
    if (vvpt_denoiser_create(&ctx, 1, &dn) != VVPT_OK)
        return;
    uint64_t np = 0;
    vvpt_denoiser_num_params(dn, &np);
    float *host = (float *)std::malloc(np * sizeof(float));
    alignas(16) float image[4] = {};
    for (int k = 0; k < n; k++) {
        g_total = g_used + ((size_t)room[k] << 20);
        g_bad = 0;
        vvpt_denoise_batch b{};
        b.radiance = b.albedo = b.normal = b.target = image;
        b.count = 1, b.width = (uint32_t)w[k], b.height = (uint32_t)h[k];
        status[k] = calls[k] ? vvpt_denoiser_gradients(dn, &b, host, np, nullptr)
                             : vvpt_denoiser_apply(dn, image, image, image, image, (uint32_t)w[k], (uint32_t)h[k]);
        bad[k] = g_bad;
    }
    std::free(host);
    vvpt_denoiser_destroy(dn);
}
