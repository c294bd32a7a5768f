/*
 * Throughput probes and the operand-layout self-test of the tensor pipes (measurement
 * entry points; no assembly kernel uses them).
 */
#include <cuda_runtime.h>
#include "igab_device.cuh"
#include "igab_tc.cuh"

namespace {

/* ---------------------------------------------------------------- self-test
 * One CTA: A (128 x 32) and B (96 x 32) of small exact values in the operand
 * layout, D = A B^T with M 128 / N 96 (4 k-steps) into columns 0-95 and, for
 * a narrow shape, A B[0:32]^T with M 128 / N 32 into columns 96-127 (first
 * k-step overwrite, then accumulate), and with negate-A on k-steps 2-3 into
 * columns 128-159.  out[128][160] receives columns 0-159. */
__global__ void __launch_bounds__(128) k_tc_selftest(float *out, int *status)
{
    __shared__ __align__(128) unsigned char sm[16384 + 12288];
    __shared__ unsigned long long bar;
    __shared__ unsigned int tbase;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char *A = sm, *B = sm + 16384;
    for (int idx = tid; idx < 128 * 32; idx += 128) {
        const int m = idx / 32, k = idx % 32;
        *reinterpret_cast<float *>(A + tc_off(m, k)) = (float)((m * 5 + k * 3) % 13 - 6) * 0.5f;
    }
    for (int idx = tid; idx < 96 * 32; idx += 128) {
        const int n = idx / 32, k = idx % 32;
        *reinterpret_cast<float *>(B + tc_off(n, k)) = (float)((n * 7 + k) % 11 - 5) * 0.25f;
    }
    if (tid == 0) {
        tc_mbar_init(&bar, 1);
        tc_fence_mbar_init();
    }
    if (warp == 0) tc_alloc(&tbase, 256);
    tc_fence_proxy_async();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tm = tbase;
    if (tid == 0) {
        const uint32_t sa = tc_smem_u32(A), sb = tc_smem_u32(B);
        for (int kk = 0; kk < 4; kk++)
            tc_mma_tf32(tm, tc_sdesc(sa + kk * TC_KSTEP_BYTES), tc_sdesc(sb + kk * TC_KSTEP_BYTES),
                        tc_idesc_tf32(128, 96), kk > 0);
        for (int kk = 0; kk < 4; kk++)
            tc_mma_tf32(tm + 96, tc_sdesc(sa + kk * TC_KSTEP_BYTES), tc_sdesc(sb + kk * TC_KSTEP_BYTES),
                        tc_idesc_tf32(128, 32), kk > 0);
        /* negate-A: columns 128-159 = A B[0:32]^T for k-steps 0-1 minus it for k-steps 2-3 */
        for (int kk = 0; kk < 4; kk++)
            tc_mma_tf32(tm + 128, tc_sdesc(sa + kk * TC_KSTEP_BYTES), tc_sdesc(sb + kk * TC_KSTEP_BYTES),
                        tc_idesc_tf32(128, 32, kk >= 2), kk > 0);
        tc_commit(&bar);
    }
    __syncthreads();
    if (tid == 0 && !tc_mbar_wait(&bar, 0)) atomicOr(status, 1);
    __syncthreads();
    tc_fence_after_sync();
    for (int part = 0; part < 10; part++) {
        float v[16];
        tc_ld16(tm + ((uint32_t)(32 * warp) << 16) + 16u * part, v);
        for (int i = 0; i < 16; i++) out[(32 * warp + lane) * 160 + 16 * part + i] = v[i];
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after_sync();
        tc_dealloc(tm, 256);
    }
}

/* ---------------------------------------------------------------- peak probe
 * One CTA per SM, one thread issues `reps` back-to-back tcgen05.mma kind::tf32
 * M 128 x N n x K 8 into one accumulator (operands: zeros in shared memory). */
template <int N>
__global__ void __launch_bounds__(128) k_tc_peak(int reps, int *status)
{
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ unsigned long long bar;
    __shared__ unsigned int tb;
    const int tid = threadIdx.x, warp = tid >> 5;
    for (int i = tid; i < 49152 / 4; i += blockDim.x) reinterpret_cast<float *>(sm)[i] = 0.f;
    if (tid == 0) {
        tc_mbar_init(&bar, 1);
        tc_fence_mbar_init();
    }
    if (warp == 0) tc_alloc(&tb, 256);
    tc_fence_proxy_async();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tm = tb;
    if (tid == 0) {
        const uint32_t sa = tc_smem_u32(sm), sb = sa + 16384;
        for (int r = 0; r < reps; r++)
            tc_mma_tf32(tm, tc_sdesc(sa + (r & 3) * TC_KSTEP_BYTES), tc_sdesc(sb + (r & 3) * TC_KSTEP_BYTES),
                        tc_idesc_tf32(128, N), r > 0);
        tc_commit(&bar);
        if (!tc_mbar_wait(&bar, 0)) atomicOr(status, 1);
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after_sync();
        tc_dealloc(tm, 256);
    }
}

template <int N>
int tc_peak_run(int nsm, double *tflops)
{
    const int reps = 4096;
    const size_t smem = 200000;   /* one CTA per SM */
    int *st = nullptr;
    IGAB_CUDA_TRY(cudaMalloc((void **)&st, sizeof(int)));
    cudaError_t e = cudaMemset(st, 0, sizeof(int));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tc_peak<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaEvent_t a = nullptr, b = nullptr;
    if (e == cudaSuccess) e = cudaEventCreate(&a);
    if (e == cudaSuccess) e = cudaEventCreate(&b);
    if (e == cudaSuccess) {
        k_tc_peak<N><<<nsm, 128, smem>>>(reps, st);   /* warm-up */
        cudaEventRecord(a);
        k_tc_peak<N><<<nsm, 128, smem>>>(reps, st);
        cudaEventRecord(b);
        e = cudaEventSynchronize(b);
    }
    float ms = 0.f;
    int hs = 0;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, a, b);
    if (e == cudaSuccess) e = cudaMemcpy(&hs, st, sizeof(int), cudaMemcpyDeviceToHost);
    if (a) cudaEventDestroy(a);
    if (b) cudaEventDestroy(b);
    cudaFree(st);
    if (e != cudaSuccess) {
        igab_set_error("igab_tc_peak: %s", cudaGetErrorString(e));
        return IGAB_ERR_CUDA;
    }
    if (hs) {
        igab_set_error("igab_tc_peak: completion wait timed out");
        return IGAB_ERR_CUDA;
    }
    *tflops = 2.0 * 128 * N * 8 * (double)reps * nsm / (ms * 1e-3) / 1e12;
    return 0;
}

__device__ __forceinline__ void dmma(double &c0, double &c1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

/* FP64 tensor-pipe issue rate: every warp issues back-to-back mma.sync m8n8k4 f64 on
 * eight independent accumulator pairs (512 flops per warp instruction) */
__global__ void __launch_bounds__(256) k_dmma_peak(int reps, double *sink)
{
    double c[8][2];
#pragma unroll
    for (int i = 0; i < 8; i++) c[i][0] = c[i][1] = 0.0;
    const double a = 1.0 + 1e-9 * threadIdx.x, b = 0.999;
    for (int r = 0; r < reps; r++) {
#pragma unroll
        for (int i = 0; i < 8; i++) dmma(c[i][0], c[i][1], a, b);
    }
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < 8; i++) s += c[i][0] + c[i][1];
    if (s == -12345.0) sink[0] = s;   /* keeps the chains live */
}

} /* namespace */

extern "C" int igab_tc_peak(int device, int n_cols, double *tflops)
{
    if (!tflops) {
        igab_set_error("igab_tc_peak: null output");
        return IGAB_ERR_ARG;
    }
    IGAB_CUDA_TRY(cudaSetDevice(device));
    int nsm = 0;
    IGAB_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device));
    switch (n_cols) {
    case 32: return tc_peak_run<32>(nsm, tflops);
    case 96: return tc_peak_run<96>(nsm, tflops);
    case 256: return tc_peak_run<256>(nsm, tflops);
    default:
        igab_set_error("igab_tc_peak: n_cols must be 32, 96 or 256");
        return IGAB_ERR_ARG;
    }
}

extern "C" int igab_tc_selftest(int device, float *out_host)
{
    if (!out_host) {
        igab_set_error("igab_tc_selftest: null output");
        return IGAB_ERR_ARG;
    }
    IGAB_CUDA_TRY(cudaSetDevice(device));
    float *d_out = nullptr;
    int *d_st = nullptr;
    IGAB_CUDA_TRY(cudaMalloc((void **)&d_out, 128 * 160 * sizeof(float)));
    cudaError_t e = cudaMalloc((void **)&d_st, sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(d_st, 0, sizeof(int));
    if (e == cudaSuccess) {
        k_tc_selftest<<<1, 128>>>(d_out, d_st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    int st = 0;
    if (e == cudaSuccess) e = cudaMemcpy(out_host, d_out, 128 * 160 * sizeof(float), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&st, d_st, sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(d_out);
    cudaFree(d_st);
    if (e != cudaSuccess) {
        igab_set_error("igab_tc_selftest: %s", cudaGetErrorString(e));
        return IGAB_ERR_CUDA;
    }
    if (st) {
        igab_set_error("igab_tc_selftest: tensor-core completion wait timed out");
        return IGAB_ERR_CUDA;
    }
    return 0;
}

int igab_launch_dmma_peak(double *tflops)
{
    int dev = 0, nsm = 0;
    IGAB_CUDA_TRY(cudaGetDevice(&dev));
    IGAB_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    double *sink = nullptr;
    IGAB_CUDA_TRY(cudaMalloc((void **)&sink, sizeof(double)));
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaError_t err = cudaEventCreate(&e0);
    if (err == cudaSuccess) err = cudaEventCreate(&e1);
    const int reps = 1 << 13;
    const unsigned nblk = (unsigned)nsm * 4u;   /* 32 warps per SM */
    float best = 1e30f;
    if (err == cudaSuccess) {
        k_dmma_peak<<<nblk, 256>>>(reps, sink);   /* warm-up */
        for (int rep = 0; rep < 3 && err == cudaSuccess; rep++) {
            cudaEventRecord(e0);
            k_dmma_peak<<<nblk, 256>>>(reps, sink);
            cudaEventRecord(e1);
            err = cudaEventSynchronize(e1);
            float ms = 0.f;
            if (err == cudaSuccess) err = cudaEventElapsedTime(&ms, e0, e1);
            if (err == cudaSuccess && ms < best) best = ms;
        }
        if (err == cudaSuccess) err = cudaGetLastError();
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(sink);
    if (err != cudaSuccess) {
        igab_set_error("igab_dmma_peak: %s", cudaGetErrorString(err));
        return IGAB_ERR_CUDA;
    }
    const double flops = 512.0 * 8.0 * reps * (double)nblk * 8.0;   /* per warp instruction x chains x warps */
    *tflops = flops / (best * 1e-3) / 1e12;
    return 0;
}
