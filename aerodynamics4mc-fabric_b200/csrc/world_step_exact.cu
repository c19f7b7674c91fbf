// Kernels of a brick world's tick (world_step.cuh). Built with --fmad=false.
#include "world_step.cuh"

#include "brick_world_cell.cuh"

namespace aero {
namespace {

constexpr int kBlock = 128;

struct InputJobs {
    WorldInputs j[kWorldChunk];
};
struct StepJobs {
    WorldStep j[kWorldChunk];
};
struct OutputJobs {
    WorldOutput j[kWorldChunk];
};
// the parameter space of a launch
static_assert(sizeof(InputJobs) <= 32764 && sizeof(StepJobs) <= 32764 && sizeof(OutputJobs) <= 32764, "too many bricks per launch");

// Inputs of each cell and, from the reference temperature it has just
// written, the temperature nudge of the same cell.
__global__ void __launch_bounds__(kBlock) world_inputs_kernel(const __grid_constant__ InputJobs jobs) {
    const WorldInputs& w = jobs.j[blockIdx.y];
    const long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (cell == 0) *w.flag = 0;
    if (cell >= (long long)w.fill.n * w.fill.n * w.fill.n) return;
    bw::fill_cell(w.fill, w.out, cell);
    if (w.nudge.t) thermal_nudge_cell(w.nudge, cell);
}

template <int kParity>
__global__ void __launch_bounds__(kBlock) world_step_kernel(const __grid_constant__ StepJobs jobs) {
    const WorldStep& w = jobs.j[blockIdx.y];
    const PadGeom G = w.a.g;
    const long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (cell >= (long long)G.nx * G.ny * G.nz) return;
    int x, y, z;
    cell_coords(G, cell, x, y, z);
    step_ip_cell<StoreF32, true, kParity>(w.f, w.a, G, cell, x, y, z, nullptr);
}

__global__ void __launch_bounds__(256) world_face_fill_kernel(const __grid_constant__ StepJobs jobs) {
    const WorldStep& w = jobs.j[blockIdx.y];
    face_fill_cell<StoreF32>(w.f, w.a, blockIdx.x * blockDim.x + threadIdx.x);
}

// Output of the streamed state, air and surface temperature, static
// constraints and the flow flags in one pass; one atomic per block, and none
// where the word has the bits.
__global__ void __launch_bounds__(kBlock) world_output_kernel(const __grid_constant__ OutputJobs jobs) {
    const WorldOutput& w = jobs.j[blockIdx.y];
    const PadGeom G = w.a.g;
    const long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int bits = 0;
    if (cell < w.sync.cells) {
        int x, y, z;
        cell_coords(G, cell, x, y, z);
        float o[4];
        macro_ip_cell<StoreF32, true>(w.f, w.a, G, cell, x, y, z, 1.0f, o);
        bits = bw::sync_cell(w.sync, cell, o);
        *reinterpret_cast<float4*>(w.sync.flow + cell * bw::kFlowChannels) = make_float4(o[0], o[1], o[2], o[3]);
    }
    const int after = __syncthreads_or(bits & bw::kFlagAfter), before = __syncthreads_or(bits & bw::kFlagBefore);
    if (threadIdx.x == 0) {
        const int all = (after ? bw::kFlagAfter : 0) | (before ? bw::kFlagBefore : 0);
        if (all & ~*reinterpret_cast<volatile int*>(w.sync.flag)) atomicOr(w.sync.flag, all);
    }
}

__global__ void __launch_bounds__(kBlock) world_atlas_kernel(const float* __restrict__ f, const __grid_constant__ IpArgs a,
                                                             bw::PublishArgs p) {
    const long long res = p.res;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= res * res * res) return;
    const PadGeom G = a.g;
    const int x = min(G.nx - 1, (int)(i / (res * res)) * p.stride), y = min(G.ny - 1, (int)((i / res) % res) * p.stride),
              z = min(G.nz - 1, (int)(i % res) * p.stride);
    float o[4];
    macro_ip_cell<StoreF32, true>(f, a, G, ((long long)x * G.ny + y) * G.nz + z, x, y, z, 1.0f, o);
    reinterpret_cast<short4*>(p.out)[i] = bw::pack_sample(o, p.velocity_scale);
}

unsigned blocks_for(long long n, int block) { return (unsigned)((n + block - 1) / block); }
long long cells_of(const PadGeom& g) { return (long long)g.nx * g.ny * g.nz; }

}  // namespace

cudaError_t launch_world_inputs(const WorldInputs* jobs, int n, cudaStream_t s) {
    if (n < 1 || n > kWorldChunk) return cudaErrorInvalidValue;
    InputJobs p;
    for (int i = 0; i < n; ++i) p.j[i] = jobs[i];
    const long long cells = (long long)jobs[0].fill.n * jobs[0].fill.n * jobs[0].fill.n;
    world_inputs_kernel<<<dim3(blocks_for(cells, kBlock), (unsigned)n), kBlock, 0, s>>>(p);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_world_step(const WorldStep* jobs, int n, int parity, cudaStream_t s) {
    if (n < 1 || n > kWorldChunk) return cudaErrorInvalidValue;
    StepJobs p;
    for (int i = 0; i < n; ++i) p.j[i] = jobs[i];
    const dim3 grid(blocks_for(cells_of(jobs[0].a.g), kBlock), (unsigned)n);
    step_timer_begin(s);
    if (parity == 0) world_step_kernel<0><<<grid, kBlock, 0, s>>>(p);
    else world_step_kernel<1><<<grid, kBlock, 0, s>>>(p);
    step_timer_end(s);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_world_face_fill(const WorldStep* jobs, int n, cudaStream_t s) {
    if (n < 1 || n > kWorldChunk) return cudaErrorInvalidValue;
    StepJobs p;
    for (int i = 0; i < n; ++i) p.j[i] = jobs[i];
    const long long links = face_fill_count(jobs[0].a.g, jobs[0].a.fill_faces);
    world_face_fill_kernel<<<dim3(blocks_for(links, 256), (unsigned)n), 256, 0, s>>>(p);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_world_output(const WorldOutput* jobs, int n, cudaStream_t s) {
    if (n < 1 || n > kWorldChunk) return cudaErrorInvalidValue;
    OutputJobs p;
    for (int i = 0; i < n; ++i) p.j[i] = jobs[i];
    world_output_kernel<<<dim3(blocks_for(jobs[0].sync.cells, kBlock), (unsigned)n), kBlock, 0, s>>>(p);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_world_atlas(const float* f, const IpArgs& a, const bw::PublishArgs& p, cudaStream_t s) {
    const long long samples = (long long)p.res * p.res * p.res;
    if (samples <= 0) return cudaSuccess;
    world_atlas_kernel<<<blocks_for(samples, kBlock), kBlock, 0, s>>>(f, a, p);
    count_launch();
    return cudaGetLastError();
}

}  // namespace aero
