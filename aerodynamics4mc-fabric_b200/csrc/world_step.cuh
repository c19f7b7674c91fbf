// One tick of a brick world as launches over all of its bricks: the passes of
// a runtime-mode call (inputs, temperature nudge and update, step, face
// pre-fill, output and dynamic refresh), each one launch per kWorldChunk
// bricks of one size instead of one launch per brick. A brick's arguments
// travel in the launch's parameter space, indexed by blockIdx.y.
//
// The bricks are small (64^3 fills a third of the chip, 16^3 a few SMs) and a
// brick's call is about ten launches, so a tick of eight 64^3 bricks spent 400
// of 1080 us between kernels and one of 27 16^3 bricks 1000 of 1900 us on the
// host (tick and atlases); together they take 730 us and, by the host's speed,
// 560 to 610.
#pragma once

#include "brick_world.cuh"
#include "d3q27_inplace.cuh"
#include "thermal.cuh"

namespace aero {

struct WorldInputs {
    bw::FillArgs fill;
    CellFields out;
    ThermalNudgeArgs nudge;  // t null: no temperature transport
    int* flag;               // cleared for the refresh of the same tick
};
struct WorldStep {
    float* f;
    IpArgs a;
};
struct WorldOutput {
    const float* f;
    IpArgs a;
    bw::SyncArgs sync;
};

// All on n <= kWorldChunk bricks of one size; FP32 populations in the
// reference's order.
cudaError_t launch_world_inputs(const WorldInputs* jobs, int n, cudaStream_t s);
cudaError_t launch_world_step(const WorldStep* jobs, int n, int parity, cudaStream_t s);
cudaError_t launch_world_face_fill(const WorldStep* jobs, int n, cudaStream_t s);
cudaError_t launch_world_output(const WorldOutput* jobs, int n, cudaStream_t s);
// A context's strided output quantised straight into a packed atlas (p.out;
// p.stride, p.res, p.velocity_scale set).
cudaError_t launch_world_atlas(const float* f, const IpArgs& a, const bw::PublishArgs& p, cudaStream_t s);

}  // namespace aero
