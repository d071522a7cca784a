// Test harness: the weight and bias gradient of denoise_kernels.cu on device
// arrays of the test's own (`g`: kGradCopies copies of the weights' and then
// the bias's gradient, stride floats apart), so that each instantiation can be
// compared with 64-bit sums of the same BF16 inputs. Built with
// denoise_kernels.cu.
#include "denoise_kernels.cuh"

extern "C" __attribute__((visibility("default"))) int device_wgrad(const void *dout, int cout, const void *in, int cin,
                                                                   int n, int h, int w, float *g, int stride)
{
    const vvdn::bf16 *d = static_cast<const vvdn::bf16 *>(dout), *x = static_cast<const vvdn::bf16 *>(in);
    vvdn::wgrad_mma_sync(d, cout, x, cin, n, h, w, g, g + 9 * cin * cout, nullptr, stride);
    vvdn::sum_grads(g, stride, g, 9 * cin * cout + cout, nullptr);
    const cudaError_t launch = cudaGetLastError(), sync = cudaDeviceSynchronize();
    return (int)(launch != cudaSuccess ? launch : sync);
}
