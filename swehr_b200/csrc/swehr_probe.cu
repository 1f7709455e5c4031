/*
 * swehr_probe.cu -- device-peak probes for the benchmark's roofline (not part
 * of the SWEHR C ABI; built into libswehr_probe.so beside libswehr.so).
 *
 * swehr_probe_fp64_peak: the FP64 vector-pipe ceiling of this GPU, measured.
 * Every thread runs eight independent fused multiply-add chains (enough
 * independent work to cover the pipe's latency at full occupancy) on a grid
 * of eight resident blocks per SM; the value reported is the best of a few
 * timed launches, in TFLOP/s (an FMA counts two floating-point operations).
 * The step kernels' arithmetic is FP64 division, square root and exp/pow
 * sequences that all run on this pipe, so this is the compute roof they are
 * held against (tensor cores are not used by the stencil).
 */
#include <cuda_runtime.h>

#include "swehr_ctx.h"
#include "swehr_ieee.h"

static const int PROBE_THREADS = 256;
static const int PROBE_CHAINS = 8;

__global__ void __launch_bounds__(PROBE_THREADS) k_fp64_fma(double *out, int iters, double b, double c)
{
    double a[PROBE_CHAINS];
#pragma unroll
    for (int k = 0; k < PROBE_CHAINS; k++) a[k] = 1.0 + 1e-3 * (threadIdx.x + k);
    for (int it = 0; it < iters; it++) {
#pragma unroll
        for (int k = 0; k < PROBE_CHAINS; k++) a[k] = fma(a[k], b, c);
    }
    double s = 0;
#pragma unroll
    for (int k = 0; k < PROBE_CHAINS; k++) s += a[k];
    if (s == 12345.678) out[blockIdx.x] = s;   /* keeps the chains live; never true */
}

extern "C" int swehr_probe_fp64_peak(double *tflops)
{
    if (!tflops) return 1;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 2;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 2;
    double *out = nullptr;
    if (cudaMalloc(&out, (size_t)sms * 8 * sizeof(double)) != cudaSuccess) return 3;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int grid = sms * 8, iters = 4096;
    double best = 0;
    for (int rep = 0; rep < 6; rep++) {
        cudaEventRecord(e0);
        k_fp64_fma<<<grid, PROBE_THREADS>>>(out, iters, 0.999999, 1e-7);
        cudaEventRecord(e1);
        cudaEventSynchronize(e1);
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        const double flops = 2.0 * grid * PROBE_THREADS * (double)iters * PROBE_CHAINS;
        if (rep > 0 && ms > 0) {
            const double tf = flops / (ms * 1e-3) / 1e12;
            if (tf > best) best = tf;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    const cudaError_t err = cudaGetLastError();
    *tflops = best;
    return err == cudaSuccess ? 0 : 4;
}

/* swehr_probe_ieee: the branch-free sequences of swehr_ieee.h beside the
 * plain operators and the bodies of swehr_math.h, element by
 * element, for the tests.  op: 0 a/b, 1 root of a, 2 exp(a), 3 a^b, 4
 * cos(atan a), 5 a/b of small a, 6 a/b of any small a, 7 exp(a) down to zero;
 * host arrays of n doubles.  refused: 1 where the operands are
 * not ones the sequences take. */
__global__ void k_ieee(int op, const double *__restrict__ a, const double *__restrict__ b, long long n, double *fast,
                       double *plain, double *refused)
{
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const double x = a[q], y = b[q];
        bool ok = true;
        switch (op) {
        case 0: fast[q] = sw_quot(x, y, sw_rcp(y)); plain[q] = x / y; ok = sw_mid_or_zero(x) && sw_mid_pos(y); break;
        case 1: fast[q] = sw_sqrt_mid(x); plain[q] = sw_sqrt_pow(x); ok = sw_mid_pos(x) || sw_zero(x); break;
        case 2: fast[q] = sw_exp_mid(x, 0.0); plain[q] = sw_exp(x); ok = sw_exp_fits(x); break;
        case 3: fast[q] = sw_pow_mid(x, y, &ok); plain[q] = sw_pow(x, y); break;
        case 4: fast[q] = sw_cos_atan_mid(x, &ok); plain[q] = sw_cos_atan(x); break;
        case 5: fast[q] = sw_quot(x, y, sw_rcp(y)); plain[q] = x / y; ok = sw_low_or_zero(x) && sw_mid_depth(y); break;
        case 6: fast[q] = sw_quot_tiny(x, y, sw_rcp(y)); plain[q] = x / y; ok = sw_small(x) && sw_mid_depth(y); break;
        default: fast[q] = sw_exp_gone(x) ? 0.0 : sw_exp_mid(x, 0.0); plain[q] = sw_exp(x); ok = sw_exp_gone(x); break;
        }
        refused[q] = !ok;
    }
}

extern "C" int swehr_probe_ieee(int op, const double *a, const double *b, long long n, double *fast, double *plain,
                                double *refused)
{
    if (!a || !b || !fast || !plain || !refused || n < 1 || op < 0 || op > 7) return 1;
    const size_t bytes = (size_t)n * sizeof(double);
    double *d = nullptr;
    if (cudaMalloc(&d, 5 * bytes) != cudaSuccess) return 2;
    cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
    k_ieee<<<592, 256>>>(op, d, d + n, n, d + 2 * n, d + 3 * n, d + 4 * n);
    cudaMemcpy(fast, d + 2 * n, bytes, cudaMemcpyDeviceToHost);
    cudaMemcpy(plain, d + 3 * n, bytes, cudaMemcpyDeviceToHost);
    cudaMemcpy(refused, d + 4 * n, bytes, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

/* swehr_probe_give_up: the flag that a wait on the device sets when it gives
 * up, set from the host, for the tests of what follows it. */
extern "C" int swehr_probe_give_up(swehr_ctx *c)
{
    const int32_t one = 1;
    return c && cudaMemcpy(&c->d_ctl->dev_error, &one, sizeof one, cudaMemcpyHostToDevice) == cudaSuccess ? 0 : 1;
}
