// Kernels of the device-resident brick-world service. Built with
// --fmad=false: the thermal source and the atlas quantisation are plain
// float products and quotients that must round like the reference's host
// loops (native/src/aero_lbm_simulation_bridge.cpp).
#include "brick_world_cell.cuh"

namespace aero {
namespace bw {

namespace {

constexpr int kBlock = 256;

__global__ void __launch_bounds__(kBlock) fill_kernel(FillArgs a, CellFields out) {
    const long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (cell < (long long)a.n * a.n * a.n) fill_cell(a, out, cell);
}

__global__ void __launch_bounds__(kBlock) sync_kernel(SyncArgs a) {
    const long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int bits = 0;
    if (cell < a.cells) {
        float* f = a.flow + cell * kFlowChannels;
        float v[4] = {f[0], f[1], f[2], f[3]};
        bits = sync_cell(a, cell, v);
        *reinterpret_cast<float4*>(f) = make_float4(v[0], v[1], v[2], v[3]);
    }
    or_flag(a.flag, bits);
}

__global__ void __launch_bounds__(kBlock) publish_kernel(PublishArgs a) {
    const long long res = a.res;
    const long long samples = res * res * res;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= samples) return;
    long long src = i;
    if (a.dense_n > 0) {
        const long long n = a.dense_n;
        const int ax = (int)(i / (res * res)), ay = (int)((i / res) % res), az = (int)(i % res);
        const long long gx = min((long long)n - 1, (long long)ax * a.stride);
        const long long gy = min((long long)n - 1, (long long)ay * a.stride);
        const long long gz = min((long long)n - 1, (long long)az * a.stride);
        src = (gx * n + gy) * n + gz;
    }
    const float* f = a.src + src * kFlowChannels;
    reinterpret_cast<short4*>(a.out)[i] = pack_sample(f, a.velocity_scale);
}

unsigned blocks_for(long long count) { return (unsigned)((count + kBlock - 1) / kBlock); }

}  // namespace

cudaError_t launch_fill(const FillArgs& a, const CellFields& out, cudaStream_t s) {
    const long long cells = (long long)a.n * a.n * a.n;
    if (cells <= 0) return cudaSuccess;
    fill_kernel<<<blocks_for(cells), kBlock, 0, s>>>(a, out);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_sync(const SyncArgs& a, cudaStream_t s) {
    if (a.cells <= 0) return cudaSuccess;
    sync_kernel<<<blocks_for(a.cells), kBlock, 0, s>>>(a);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_publish(const PublishArgs& a, cudaStream_t s) {
    const long long samples = (long long)a.res * a.res * a.res;
    if (samples <= 0) return cudaSuccess;
    publish_kernel<<<blocks_for(samples), kBlock, 0, s>>>(a);
    count_launch();
    return cudaGetLastError();
}

}  // namespace bw
}  // namespace aero
