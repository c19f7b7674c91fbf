// Discrete adjoint of the D3Q27 brick step with checkpointed recomputation.
//
// Forward model (per call n = 1..N, two population buffers, pull layout):
//   s_1 = C(feq(1, u_in))                     fluid cells, initial equilibrium
//   s_n = C(P(s_{n-1}))                       n >= 2
//   u_probe = j / clamp(rho) of P(s_N)        the brick step's velocity output
// where P pulls each direction from its source cell (periodic faces wrap;
// solid sources and bounce-back faces return the cell's own opposite
// population; velocity faces supply feq(1, u_in)), and C is the factorised
// cumulant collision with Smagorinsky SGS, Boussinesq buoyancy along +z from a
// static temperature field, and a per-cell body-force field (adjoint27.cuh).
// Loss L = sum over probes of |u_probe - target|^2.
//
// Reverse sweep: lambda_N is seeded at the probe cells; for n = N..1 one
// launch per call recomputes the cell's collision from s_{n-1} (or the initial
// equilibrium), applies its transposed Jacobian to lambda_n, accumulates the
// body-force gradient of the cell in FP64, and scatters the pre-collision
// adjoint along the transposed pull (every population slot is read by exactly
// one fluid cell, so the scatter needs no atomics); velocity-face pulls and
// the initial equilibrium accumulate the inflow gradient in FP64. States are
// checkpointed every K calls during the forward run and recomputed segment by
// segment, but for the last two segments, whose states the forward run leaves
// in the sweep's buffers (K = 1 stores every state and recomputes nothing).
// At 64^3, 200 calls, K = 20: 25 us a forward call and 72 us a call of the
// sweep (49 and 140 before the pull classification and the kept segments).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/aero_lbm_b200.h"
#include "adjoint27.cuh"
#include "d3q27_kernels.cuh"
#include "runtime_internal.h"

namespace aero {
namespace adj {
namespace {

struct Geo {
    int nx, ny, nz;
    long long cells;
    int kind[6];  // per face: 1 periodic, 2 bounce-back, 4 velocity
    const uint2* links;  // pull classification of every cell (adj_links_kernel)
};

// Pull classification of a fluid cell, built once per brick (the mask and the
// face kinds never change): x holds one bit per direction whose source is
// solid or outside a bounce-back face (plus kLinkSolid on solid cells), y one
// bit per direction whose source is outside a velocity face.
// The rules run 27 times per cell and launch otherwise: as branches they took
// 32 of the forward launch's 50 us and about 70 of the reverse launch's 115
// us at 64^3 (the initial call, which pulls nothing, ran in 18 and 43 us).
// With the two words every population is one load or store at an address
// formed by selects.
constexpr unsigned kLinkSolid = 1u << 31;

__global__ void adj_links_kernel(Geo G, const uint8_t* __restrict__ solid, uint2* __restrict__ links) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= G.cells) return;
    unsigned bounce = solid[i] ? kLinkSolid : 0u, inflow = 0u;
    int c[3];
    cell_xyz32(i, G.ny, G.nz, c[0], c[1], c[2]);
    const int n[3] = {G.nx, G.ny, G.nz};
    for (int q = 0; q < 27; ++q) {
        // periodic axes wrap; then the first out-of-range axis in the order
        // x-, x+, y-, y+, z-, z+ names the face
        int s[3] = {c[0] - q_cx(q), c[1] - q_cy(q), c[2] - q_cz(q)};
        int face = -1;
        for (int a = 0; a < 3; ++a) {
            if (s[a] >= 0 && s[a] < n[a]) continue;
            const int fid = 2 * a + (s[a] < 0 ? 0 : 1);
            if (G.kind[fid] == kHydroPeriodic) s[a] = s[a] < 0 ? s[a] + n[a] : s[a] - n[a];
            else if (face < 0) face = fid;
        }
        if (face >= 0) {
            if (G.kind[face] == kHydroVelocity) inflow |= 1u << q;
            else bounce |= 1u << q;
        } else if (solid[((long long)s[0] * G.ny + s[1]) * G.nz + s[2]]) {
            bounce |= 1u << q;
        }
    }
    links[i] = make_uint2(bounce, inflow);
}

// Cell index of the neighbour along -c_q: one term per axis. A coordinate
// that leaves the brick wraps; a link that leaves by a face that is not
// periodic never uses the index.
struct Neighbours {
    unsigned X[3], Y[3], Z[3];
    __device__ __forceinline__ Neighbours(const Geo& G, int x, int y, int z) {
        const unsigned row = (unsigned)G.nz, slab = (unsigned)G.ny * row;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int sx = x + k - 1, sy = y + k - 1, sz = z + k - 1;
            X[k] = (unsigned)(sx < 0 ? sx + G.nx : (sx >= G.nx ? sx - G.nx : sx)) * slab;
            Y[k] = (unsigned)(sy < 0 ? sy + G.ny : (sy >= G.ny ? sy - G.ny : sy)) * row;
            Z[k] = (unsigned)(sz < 0 ? sz + G.nz : (sz >= G.nz ? sz - G.nz : sz));
        }
    }
    __device__ __forceinline__ unsigned source(int q) const { return X[1 - q_cx(q)] + Y[1 - q_cy(q)] + Z[1 - q_cz(q)]; }
};

// The population a pull of direction q reads: the source cell's, or after a
// bounce the cell's own opposite one.
// I: unsigned where every slot index of a state fits 32 bits, else 64 bits.
template <class I>
__device__ __forceinline__ I link_slot(const Geo& G, const Neighbours& nb, unsigned own, unsigned i, int q) {
    const I bounced = (I)q_opp(q) * (I)G.cells + i, pulled = (I)q * (I)G.cells + nb.source(q);
    return (own >> q) & 1u ? bounced : pulled;
}

// Streamed populations of a fluid cell.
template <class I, class T>
__device__ __forceinline__ void pull_cell(const Geo& G, const T* __restrict__ s, long long i, const Neighbours& nb, uint2 w,
                                          const T (&uin)[3], T (&p)[27]) {
    const unsigned own = w.x | w.y;
#pragma unroll
    for (int q = 0; q < 27; ++q) p[q] = s[link_slot<I>(G, nb, own, (unsigned)i, q)];
    if (w.y) {
#pragma unroll
        for (int q = 0; q < 27; ++q)
            if ((w.y >> q) & 1u) p[q] = feq_t<T>(q, T(1), uin[0], uin[1], uin[2]);
    }
}

__device__ __forceinline__ void cell_xyz(const Geo& G, long long i, int& x, int& y, int& z) {
    cell_xyz32(i, G.ny, G.nz, x, y, z);
}

template <class T>
struct StepArgs {
    Geo G;
    CollideParams cp;
    const float* temperature;  // cells or null
    const float* force;        // 3 x cells (SoA) or null
    T uin[3];
    const T* src;
    T* dst;
};

template <class T>
__device__ __forceinline__ void cell_force(const StepArgs<T>& A, long long i, T& t, T& fx, T& fy, T& fz) {
    t = A.temperature ? T(A.temperature[i]) : T(0);
    fx = fy = fz = T(0);
    if (A.force) {
        fx = T(A.force[i]);
        fy = T(A.force[A.G.cells + i]);
        fz = T(A.force[2 * A.G.cells + i]);
    }
}

// One forward call: init (kInit, collide the equilibrium) or pull + collide.
template <class T, bool kInit, class I>
__global__ void __launch_bounds__(128) adj_step_kernel(StepArgs<T> A) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.G.cells) return;
    T* __restrict__ dst = A.dst;
    const uint2 w = A.G.links[i];
    if (w.x & kLinkSolid) {
#pragma unroll
        for (int q = 0; q < 27; ++q) dst[(I)q * (I)A.G.cells + (unsigned)i] = wq<T>(q);
        return;
    }
    T p[27];
    if (kInit) {
#pragma unroll
        for (int q = 0; q < 27; ++q) p[q] = feq_t<T>(q, T(1), A.uin[0], A.uin[1], A.uin[2]);
    } else {
        int x, y, z;
        cell_xyz(A.G, i, x, y, z);
        pull_cell<I>(A.G, A.src, i, Neighbours(A.G, x, y, z), w, A.uin, p);
    }
    T t, fx, fy, fz;
    cell_force(A, i, t, fx, fy, fz);
    T fo[27];
    CollideTape<T> tape;
    collide_fwd<T>(p, A.cp, t, fx, fy, fz, fo, tape);
#pragma unroll
    for (int q = 0; q < 27; ++q) dst[(I)q * (I)A.G.cells + (unsigned)i] = fo[q];
}

// Probe velocities of P(s) and the loss sum (FP64).
template <class T>
__global__ void adj_probe_kernel(Geo G, const T* __restrict__ s, T ux_in, T uy_in, T uz_in, int nprobe,
                                 const long long* __restrict__ cells, const float* __restrict__ target,
                                 float* __restrict__ out_u, double* __restrict__ probe_loss) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nprobe) return;
    const long long i = cells[k];
    int x, y, z;
    cell_xyz(G, i, x, y, z);
    const T uin[3] = {ux_in, uy_in, uz_in};
    T p[27], u[3], rc;
    bool rf;
    pull_cell<unsigned long long>(G, s, i, Neighbours(G, x, y, z), G.links[i], uin, p);
    probe_velocity<T>(p, u, rc, rf);
    double l = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double d = (double)u[a] - (double)target[3 * k + a];
        l += d * d;
        out_u[3 * k + a] = (float)u[a];
    }
    probe_loss[k] = l;
}

// Scatter of a pre-collision adjoint along the transposed pull; velocity-face
// pulls add to the inflow gradient. Every fluid cell's slot of the output is
// the source of exactly one pull of the forward step (a neighbour's slot
// pull, or the cell's own bounce-back), except the slot (opp q, cell) of a
// direction q that the cell pulls from a velocity face: nothing reads that
// population, so its adjoint is zero, written here. With kAccumulate false
// the launch therefore writes every fluid slot of lam_prev exactly once and
// needs no clearing pass (solid cells' slots are never read).
template <bool kAccumulate, class I>
__device__ __forceinline__ void scatter(const Geo& G, long long i, const Neighbours& nb, uint2 w, const float (&lam)[27],
                                        const float (&uin)[3], float* __restrict__ lam_prev, double (&du)[3]) {
    const unsigned own = w.x | w.y;
    if (w.y) {
#pragma unroll
        for (int q = 0; q < 27; ++q) {
            if (!((w.y >> q) & 1u)) continue;
            float d[3];
            dfeq_du<float>(q, 1.0f, uin[0], uin[1], uin[2], d);
            du[0] += (double)lam[q] * d[0];
            du[1] += (double)lam[q] * d[1];
            du[2] += (double)lam[q] * d[2];
        }
    }
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        float* slot = lam_prev + link_slot<I>(G, nb, own, (unsigned)i, q);
        const bool inflow = (w.y >> q) & 1u;
        if (!kAccumulate) *slot = inflow ? 0.0f : lam[q];
        else if (!inflow) *slot += lam[q];
    }
}

// Block sum of the per-thread inflow-gradient parts, added to this block's
// own slot (launches are serial on the stream, so the sum over blocks and
// calls is formed in a fixed order: the result is deterministic).
__device__ __forceinline__ void add_du(double (&du)[3], double* __restrict__ du_part) {
    __shared__ double sh[3][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        double v = du[a];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) sh[a][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            double t = 0.0;
            for (int w = 0; w < nw; ++w) t += sh[a][w];
            du_part[3 * blockIdx.x + a] += t;
        }
    }
}

// lambda_N at the probe cells: dL/du through the probe observable, scattered.
// One warp per probe: the pulls of different cells read different slots, so
// only probes of one cell share slots; the first of them adds all of its
// cell's probes in order, the others do nothing. Inflow-gradient parts go to
// the probe's own entry of du_probe. (As one thread over all probes, each
// waiting for the last one's loads, the 64 probes of a 64^3 brick took 1056
// us.)
__global__ void adj_seed_kernel(Geo G, const float* __restrict__ s, float ux_in, float uy_in, float uz_in, int nprobe,
                                const long long* __restrict__ cells, const float* __restrict__ target,
                                float* __restrict__ lam, double* __restrict__ du_probe) {
    const int first = blockIdx.x;
    const long long i = cells[first];
    bool earlier = false;
    for (int k = threadIdx.x; k < first; k += 32) earlier |= cells[k] == i;
    double du[3] = {0.0, 0.0, 0.0};
    if (!__any_sync(0xffffffffu, earlier) && threadIdx.x == 0) {
        int x, y, z;
        cell_xyz(G, i, x, y, z);
        const float uin[3] = {ux_in, uy_in, uz_in};
        const Neighbours nb(G, x, y, z);
        const uint2 w = G.links[i];
        float p[27], u[3], rc;
        bool rf;
        pull_cell<unsigned long long>(G, s, i, nb, w, uin, p);
        probe_velocity<float>(p, u, rc, rf);
        for (int k = first; k < nprobe; ++k) {
            if (cells[k] != i) continue;
            const float lu[3] = {2.0f * (u[0] - target[3 * k]), 2.0f * (u[1] - target[3 * k + 1]),
                                 2.0f * (u[2] - target[3 * k + 2])};
            float lp[27];
            probe_velocity_vjp<float>(u, rc, rf, lu, lp);
            scatter<true, unsigned long long>(G, i, nb, w, lp, uin, lam, du);
        }
    }
    if (threadIdx.x == 0)
        for (int a = 0; a < 3; ++a) du_probe[3 * first + a] = du[a];
}

// One reverse call: lambda_n (cell-local read) -> lambda_{n-1} (scatter),
// body-force gradient of the cell, inflow gradient.
// Latency-bound (long scoreboard) at 20 warps per SM, the most that its
// registers allow. Of the block sizes that keep 20 warps, 320 threads measured
// best where the grid fills the chip (64^3, sweep per call: 72 us against 74
// of 128, 78 of 64 and 72 of 640 threads); below about one and a half waves
// the smaller blocks spread better (48^3: 36.5 us with 320 threads, 33.9 with
// 128; 56^3: 44.9 and 46.2), so rev_threads_for draws the line there.
constexpr int kRevThreads = 320, kRevThreadsSmall = 128;
int rev_threads_for(long long cells) {
    const long long wave = 2LL * kRevThreads * device_sms();
    return 2 * cells >= 3 * wave ? kRevThreads : kRevThreadsSmall;
}
template <bool kInit, class I>
__global__ void __launch_bounds__(kRevThreads, 2) adj_reverse_kernel(StepArgs<float> A, const float* __restrict__ lam_n,
                                                          float* __restrict__ lam_prev, double* __restrict__ grad_f,
                                                          double* __restrict__ du_part) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double du[3] = {0.0, 0.0, 0.0};
    const uint2 w = i < A.G.cells ? A.G.links[i] : make_uint2(kLinkSolid, 0u);
    if (!(w.x & kLinkSolid)) {
        int x, y, z;
        cell_xyz(A.G, i, x, y, z);
        const Neighbours nb(A.G, x, y, z);
        float p[27];
        if (kInit) {
#pragma unroll
            for (int q = 0; q < 27; ++q) p[q] = feq_t<float>(q, 1.0f, A.uin[0], A.uin[1], A.uin[2]);
        } else {
            pull_cell<I>(A.G, A.src, i, nb, w, A.uin, p);
        }
        float t, fx, fy, fz;
        cell_force(A, i, t, fx, fy, fz);
        float fo[27];
        CollideTape<float> tape;
        collide_fwd<float, false>(p, A.cp, t, fx, fy, fz, fo, tape);
        float lo[27], li[27], lf[3];
#pragma unroll
        for (int q = 0; q < 27; ++q) lo[q] = lam_n[(long long)q * A.G.cells + i];
        collide_vjp<float>(tape, A.cp, lo, li, lf);
        // one thread per entry, one launch after the other: the sums keep their
        // order, and an addition in L2 needs no load to wait for
        atomicAdd(grad_f + i, (double)lf[0]);
        atomicAdd(grad_f + A.G.cells + i, (double)lf[1]);
        atomicAdd(grad_f + 2 * A.G.cells + i, (double)lf[2]);
        if (kInit) {
#pragma unroll
            for (int q = 0; q < 27; ++q) {
                float d[3];
                dfeq_du<float>(q, 1.0f, A.uin[0], A.uin[1], A.uin[2], d);
                du[0] += (double)li[q] * d[0];
                du[1] += (double)li[q] * d[1];
                du[2] += (double)li[q] * d[2];
            }
        } else {
            scatter<false, I>(A.G, i, nb, w, li, A.uin, lam_prev, du);
        }
    }
    add_du(du, du_part);
}

// ------------------------------------------------------------------ host side
struct Brick {
    AeroLbmB200AdjointConfig cfg{};
    Geo geo{};
    CollideParams cp{};
    long long cells = 0;
    size_t state_elems = 0;
    void* block = nullptr;     // one allocation: the arrays below up to the inflow-gradient parts
    uint8_t* solid = nullptr;
    float* temperature = nullptr;
    float* force = nullptr;
    float* st[2] = {nullptr, nullptr};
    double* st64[2] = {nullptr, nullptr};
    void* sweep = nullptr;     // one block: the checkpoint and segment states
    std::vector<float*> ckpt;  // ckpt[j] = s_{jK} for j >= 1 (index 0 unused)
    std::vector<float*> seg;   // two sets of K - 1 segment states
    cudaStream_t side = nullptr;  // recomputation stream (overlaps the reverse launches)
    float* lam[2] = {nullptr, nullptr};
    double* grad_f = nullptr;
    double* probe_loss = nullptr;  // per probe
    double* du_part = nullptr;     // 3 x reverse blocks: inflow-gradient parts of the reverse launches
    double* du_probe = nullptr;    // 3 x probes: those of the seed
    uint2* links = nullptr;        // pull classification
    int rev_blocks = 0, rev_threads = 0;
    int nprobe = 0;
    long long* probe_cells = nullptr;
    float* probe_target = nullptr;
    float* probe_u = nullptr;
    double fwd_ms = 0.0, rev_ms = 0.0, recompute_ms = 0.0, total_ms = 0.0;
    int fwd_steps = 0, rev_steps = 0;

    ~Brick() {
        for (void* p : {block, sweep, (void*)st64[0], (void*)st64[1], (void*)probe_loss, (void*)du_probe, (void*)probe_cells,
                        (void*)probe_target, (void*)probe_u})
            if (p) cudaFree(p);
        if (side) cudaStreamDestroy(side);
    }
};

std::mutex g_adj_mutex;
std::map<long long, Brick*> g_adj;
long long g_next_adj = 1;
std::string g_adj_error;

bool adj_ok(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return true;
    g_adj_error = std::string(what) + ": " + cudaGetErrorString(e);
    return false;
}

CollideParams params_of(const AeroLbmB200AdjointConfig& c) {
    CollideParams p{};
    const float nu = std::min(std::max((c.tau - 0.5f) / 3.0f, 1.0e-8f), (0.95f - 0.5f) / 3.0f);
    p.tau_shear_base = std::min(std::max(0.5f + 3.0f * nu, kTauMin), kTauMax);
    p.tau_normal_base = p.tau_shear_base;
    p.nu0 = std::max(1e-6f, nu);
    p.sgs_c2 = c.smagorinsky_c * c.smagorinsky_c;
    p.sgs_nut_cap = 5.0f * p.nu0;
    p.sgs_bulk = 0.30f;
    p.buoy_beta = c.buoyancy_beta;
    p.buoy_fmax = 0.02f;
    p.max_speed = 0.57735026919f * 0.60f;
    p.enable_sgs = c.smagorinsky_c > 0.0f ? 1 : 0;
    p.enable_buoyancy = c.buoyancy_beta != 0.0f ? 1 : 0;
    p.gravity_axis = 2;
    return p;
}

template <class T>
StepArgs<T> step_args(const Brick& b, const float* inflow, const T* src, T* dst) {
    StepArgs<T> a{};
    a.G = b.geo;
    a.cp = b.cp;
    a.temperature = b.temperature;
    a.force = b.force;
    a.uin[0] = T(inflow[0]);
    a.uin[1] = T(inflow[1]);
    a.uin[2] = T(inflow[2]);
    a.src = src;
    a.dst = dst;
    return a;
}

size_t aligned(size_t bytes) { return (bytes + 255) / 256 * 256; }

// Slot indices of a state fit 32 bits (one address operation less per load).
bool narrow(const Brick& b) { return b.state_elems < (1ull << 32); }

unsigned blocks_for(long long n, int t) { return (unsigned)((n + t - 1) / t); }

template <class T>
bool launch_step(const Brick& b, const float* inflow, bool init, const T* src, T* dst, cudaStream_t s) {
    const StepArgs<T> a = step_args<T>(b, inflow, src, dst);
    const unsigned blocks = blocks_for(b.cells, 128);
    if (init) adj_step_kernel<T, true, unsigned long long><<<blocks, 128, 0, s>>>(a);
    else if (narrow(b)) adj_step_kernel<T, false, unsigned><<<blocks, 128, 0, s>>>(a);
    else adj_step_kernel<T, false, unsigned long long><<<blocks, 128, 0, s>>>(a);
    count_launch();
    return adj_ok(cudaGetLastError(), "adjoint forward step");
}

float elapsed(cudaEvent_t a, cudaEvent_t b) {
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, a, b);
    return ms;
}

bool upload_force(Brick& b, const float* force_soa, cudaStream_t s) {
    if (!force_soa) return adj_ok(cudaMemsetAsync(b.force, 0, 3 * b.cells * sizeof(float), s), "force clear");
    return adj_ok(cudaMemcpyAsync(b.force, force_soa, 3 * b.cells * sizeof(float), cudaMemcpyHostToDevice, s), "force upload");
}

Brick* find_brick(long long h) {
    auto it = g_adj.find(h);
    return it == g_adj.end() ? nullptr : it->second;
}

}  // namespace
}  // namespace adj
}  // namespace aero

using namespace aero;
using namespace aero::adj;

extern "C" {

AERO_LBM_B200_EXPORT void aero_lbm_b200_adjoint_default_config(AeroLbmB200AdjointConfig* c) {
    if (!c) return;
    *c = AeroLbmB200AdjointConfig{};
    c->nx = c->ny = c->nz = 64;
    c->face_kind[0] = c->face_kind[1] = AERO_LBM_HYDRO_BOUNDARY_VELOCITY_DIRICHLET;
    c->face_kind[2] = c->face_kind[3] = AERO_LBM_HYDRO_BOUNDARY_PERIODIC;
    c->face_kind[4] = AERO_LBM_HYDRO_BOUNDARY_BOUNCE_BACK;
    c->face_kind[5] = AERO_LBM_HYDRO_BOUNDARY_VELOCITY_DIRICHLET;
    c->tau = 0.55f;
    c->smagorinsky_c = 0.1f;
    c->buoyancy_beta = 1e-4f;
    c->steps = 200;
    c->checkpoint_every = 20;
}

AERO_LBM_B200_EXPORT int aero_lbm_b200_adjoint_create(const AeroLbmB200AdjointConfig* cfg, const uint8_t* obstacle,
                                                      const float* temperature, long long* out_handle) {
    std::lock_guard<std::mutex> lk(g_adj_mutex);
    g_adj_error.clear();
    if (!cfg || !obstacle || !out_handle || cfg->nx <= 0 || cfg->ny <= 0 || cfg->nz <= 0 || cfg->steps < 1 ||
        cfg->checkpoint_every < 1 || !(cfg->tau > 0.5f) || cfg->smagorinsky_c < 0.0f) {
        g_adj_error = "adjoint_create: invalid config (dims > 0, steps >= 1, checkpoint_every >= 1, tau > 0.5)";
        return 0;
    }
    for (int f = 0; f < 6; ++f) {
        const int k = cfg->face_kind[f];
        if (k != AERO_LBM_HYDRO_BOUNDARY_PERIODIC && k != AERO_LBM_HYDRO_BOUNDARY_BOUNCE_BACK &&
            k != AERO_LBM_HYDRO_BOUNDARY_VELOCITY_DIRICHLET) {
            g_adj_error = "adjoint_create: face kinds must be periodic, bounce-back or velocity";
            return 0;
        }
        if ((k == AERO_LBM_HYDRO_BOUNDARY_PERIODIC) != (cfg->face_kind[f ^ 1] == AERO_LBM_HYDRO_BOUNDARY_PERIODIC)) {
            g_adj_error = "adjoint_create: a periodic face needs a periodic opposite face";
            return 0;
        }
    }
    auto* b = new Brick();
    b->cfg = *cfg;
    b->cells = (long long)cfg->nx * cfg->ny * cfg->nz;
    b->state_elems = (size_t)b->cells * 27;
    b->cp = params_of(*cfg);
    const size_t n = (size_t)b->cells;
    b->rev_threads = rev_threads_for(b->cells);
    b->rev_blocks = (int)blocks_for(b->cells, b->rev_threads);
    // the brick's arrays are slices of one block (ten allocations otherwise)
    struct Slice {
        void** to;
        size_t bytes;
    };
    const std::vector<Slice> slices = {{(void**)&b->st[0], b->state_elems * sizeof(float)},
                                       {(void**)&b->st[1], b->state_elems * sizeof(float)},
                                       {(void**)&b->lam[0], b->state_elems * sizeof(float)},
                                       {(void**)&b->lam[1], b->state_elems * sizeof(float)},
                                       {(void**)&b->grad_f, 3 * n * sizeof(double)},
                                       {(void**)&b->du_part, 3 * (size_t)b->rev_blocks * sizeof(double)},
                                       {(void**)&b->links, n * sizeof(uint2)},
                                       {(void**)&b->force, 3 * n * sizeof(float)},
                                       {(void**)&b->temperature, temperature ? n * sizeof(float) : 0},
                                       {(void**)&b->solid, n}};
    size_t total = 0;
    for (const Slice& x : slices) total += aligned(x.bytes);
    bool ok = adj_ok(cudaMalloc(&b->block, total), "adjoint alloc");
    char* next = static_cast<char*>(b->block);
    for (const Slice& x : slices) {
        if (!ok || !x.bytes) continue;
        *x.to = next;
        next += aligned(x.bytes);
    }
    const cudaStream_t s = current_stream();
    if (ok && temperature)
        ok = adj_ok(cudaMemcpyAsync(b->temperature, temperature, n * sizeof(float), cudaMemcpyHostToDevice, s), "temperature upload");
    if (ok) ok = adj_ok(cudaMemcpyAsync(b->solid, obstacle, n, cudaMemcpyHostToDevice, s), "mask upload");
    if (!ok) {
        cudaStreamSynchronize(s);
        delete b;
        return 0;
    }
    b->geo.nx = cfg->nx;
    b->geo.ny = cfg->ny;
    b->geo.nz = cfg->nz;
    b->geo.cells = b->cells;
    for (int f = 0; f < 6; ++f) b->geo.kind[f] = cfg->face_kind[f];
    b->geo.links = b->links;
    adj_links_kernel<<<blocks_for(b->cells, 256), 256, 0, s>>>(b->geo, b->solid, b->links);
    count_launch();
    if (!adj_ok(cudaGetLastError(), "adjoint links") || !adj_ok(cudaStreamSynchronize(s), "adjoint links")) {
        delete b;
        return 0;
    }
    const long long h = g_next_adj++;
    g_adj[h] = b;
    *out_handle = h;
    return 1;
}

AERO_LBM_B200_EXPORT int aero_lbm_b200_adjoint_set_probes(long long handle, int count, const int* cells, const float* targets) {
    std::lock_guard<std::mutex> lk(g_adj_mutex);
    g_adj_error.clear();
    Brick* b = find_brick(handle);
    if (!b || count < 1 || !cells || !targets) {
        g_adj_error = "adjoint_set_probes: unknown handle, no probes or null arrays";
        return 0;
    }
    std::vector<long long> c(count);
    std::vector<uint8_t> solid(b->cells);
    if (!adj_ok(cudaMemcpy(solid.data(), b->solid, b->cells, cudaMemcpyDeviceToHost), "mask read")) return 0;
    for (int k = 0; k < count; ++k) {
        if (cells[k] < 0 || cells[k] >= b->cells || solid[cells[k]]) {
            g_adj_error = "adjoint_set_probes: probe " + std::to_string(k) + " is outside the brick or solid";
            return 0;
        }
        c[k] = cells[k];
    }
    for (void* p : {(void*)b->probe_cells, (void*)b->probe_target, (void*)b->probe_u, (void*)b->probe_loss, (void*)b->du_probe})
        if (p) cudaFree(p);
    b->probe_cells = nullptr;
    b->du_probe = nullptr;
    b->probe_target = b->probe_u = nullptr;
    b->probe_loss = nullptr;
    b->nprobe = 0;
    if (!adj_ok(cudaMalloc(&b->probe_cells, count * sizeof(long long)), "probe alloc") ||
        !adj_ok(cudaMalloc(&b->probe_target, 3 * count * sizeof(float)), "probe alloc") ||
        !adj_ok(cudaMalloc(&b->probe_u, 3 * count * sizeof(float)), "probe alloc") ||
        !adj_ok(cudaMalloc(&b->probe_loss, count * sizeof(double)), "probe alloc") ||
        !adj_ok(cudaMalloc(&b->du_probe, 3 * (size_t)count * sizeof(double)), "probe alloc") ||
        !adj_ok(cudaMemcpy(b->probe_cells, c.data(), count * sizeof(long long), cudaMemcpyHostToDevice), "probe upload") ||
        !adj_ok(cudaMemcpy(b->probe_target, targets, 3 * count * sizeof(float), cudaMemcpyHostToDevice), "probe upload"))
        return 0;
    b->nprobe = count;
    return 1;
}

// Forward run (no checkpoints kept): loss and probe velocities. precision 0
// runs the FP32 model the gradient is taken of, 1 the same model in FP64.
AERO_LBM_B200_EXPORT int aero_lbm_b200_adjoint_forward(long long handle, const float* force_soa, const float* inflow,
                                                       int precision, double* out_loss, float* out_probe_u) {
    std::lock_guard<std::mutex> lk(g_adj_mutex);
    g_adj_error.clear();
    Brick* b = find_brick(handle);
    if (!b || !inflow || b->nprobe < 1 || (precision != 0 && precision != 1)) {
        g_adj_error = "adjoint_forward: unknown handle, null inflow, no probes or bad precision";
        return 0;
    }
    cudaStream_t s = current_stream();
    if (!upload_force(*b, force_soa, s)) return 0;
    const int N = b->cfg.steps;
    const Geo G = b->geo;
    if (precision == 0) {
        if (!launch_step<float>(*b, inflow, true, nullptr, b->st[0], s)) return 0;
        int cur = 0;
        for (int n = 2; n <= N; ++n) {
            if (!launch_step<float>(*b, inflow, false, b->st[cur], b->st[cur ^ 1], s)) return 0;
            cur ^= 1;
        }
        adj_probe_kernel<float><<<blocks_for(b->nprobe, 64), 64, 0, s>>>(G, b->st[cur], inflow[0], inflow[1], inflow[2],
                                                                          b->nprobe, b->probe_cells, b->probe_target,
                                                                          b->probe_u, b->probe_loss);
    } else {
        for (int k = 0; k < 2; ++k)
            if (!b->st64[k] && !adj_ok(cudaMalloc(&b->st64[k], b->state_elems * sizeof(double)), "fp64 state alloc")) return 0;
        if (!launch_step<double>(*b, inflow, true, nullptr, b->st64[0], s)) return 0;
        int cur = 0;
        for (int n = 2; n <= N; ++n) {
            if (!launch_step<double>(*b, inflow, false, b->st64[cur], b->st64[cur ^ 1], s)) return 0;
            cur ^= 1;
        }
        adj_probe_kernel<double><<<blocks_for(b->nprobe, 64), 64, 0, s>>>(G, b->st64[cur], inflow[0], inflow[1], inflow[2],
                                                                           b->nprobe, b->probe_cells, b->probe_target,
                                                                           b->probe_u, b->probe_loss);
    }
    count_launch();
    if (!adj_ok(cudaGetLastError(), "probe kernel")) return 0;
    std::vector<double> pl(b->nprobe);
    if (!adj_ok(cudaMemcpyAsync(pl.data(), b->probe_loss, b->nprobe * sizeof(double), cudaMemcpyDeviceToHost, s), "loss read"))
        return 0;
    if (out_probe_u &&
        !adj_ok(cudaMemcpyAsync(out_probe_u, b->probe_u, 3 * b->nprobe * sizeof(float), cudaMemcpyDeviceToHost, s), "probe read"))
        return 0;
    if (!adj_ok(cudaStreamSynchronize(s), "forward sync")) return 0;
    double loss = 0.0;
    for (double v : pl) loss += v;
    if (out_loss) *out_loss = loss;
    return 1;
}

// Loss and its gradient with respect to the body-force field (3 x cells, SoA,
// FP64) and the inflow vector (3, FP64): forward run with checkpoints, then
// the reverse sweep segment by segment.
AERO_LBM_B200_EXPORT int aero_lbm_b200_adjoint_gradient(long long handle, const float* force_soa, const float* inflow,
                                                        double* out_loss, double* out_grad_force, double* out_grad_inflow) {
    std::lock_guard<std::mutex> lk(g_adj_mutex);
    g_adj_error.clear();
    Brick* b = find_brick(handle);
    if (!b || !inflow || b->nprobe < 1) {
        g_adj_error = "adjoint_gradient: unknown handle, null inflow or no probes";
        return 0;
    }
    const auto t0 = std::chrono::steady_clock::now();
    cudaStream_t s = current_stream();
    const int N = b->cfg.steps, K = b->cfg.checkpoint_every;
    const Geo G = b->geo;
    const size_t bytes = b->state_elems * sizeof(float);
    // checkpoint and segment states, allocated at the first gradient call
    // (forward-only use needs neither) as slices of one block: 47 allocations
    // of a 64^3 brick's 28 MB took most of that call
    if (!b->sweep) {
        const int segments = (N + K - 1) / K;
        const size_t slices = (size_t)segments - 1 + 2 * (size_t)std::max(0, K - 1);
        const size_t slice = aligned(bytes);
        if (!b->side && !adj_ok(cudaStreamCreateWithFlags(&b->side, cudaStreamNonBlocking), "side stream")) return 0;
        if (!adj_ok(cudaMalloc(&b->sweep, std::max<size_t>(1, slices) * slice), "checkpoint and segment alloc")) {
            b->sweep = nullptr;
            return 0;
        }
        char* next = static_cast<char*>(b->sweep);
        auto take = [&] {
            float* p = reinterpret_cast<float*>(next);
            next += slice;
            return p;
        };
        b->ckpt.assign(segments, nullptr);
        for (int j = 1; j < segments; ++j) b->ckpt[j] = take();
        b->seg.clear();
        for (int j = 0; j < 2 * std::max(0, K - 1); ++j) b->seg.push_back(take());
    }
    cudaEvent_t ev[6];
    for (auto& e : ev) cudaEventCreate(&e);
    const size_t du_bytes = 3 * (size_t)b->rev_blocks * sizeof(double);
    bool ok = upload_force(*b, force_soa, s) && adj_ok(cudaMemsetAsync(b->du_part, 0, du_bytes, s), "clear") &&
              adj_ok(cudaMemsetAsync(b->grad_f, 0, 3 * b->cells * sizeof(double), s), "clear");
    // forward run. A checkpoint is written by its own launch, and so are the
    // states of the last two segments: their two buffer sets are idle until
    // the sweep reverses those segments, so these need no recomputation.
    const int segments = (N + K - 1) / K;
    const int per = std::max(0, K - 1);
    auto kept = [&](int n) -> float* {  // where s_n stays for the sweep (null: nowhere)
        const int j = n / K, m = n - j * K;
        if (n >= N) return nullptr;
        if (m == 0) return b->ckpt[j];
        return j >= segments - 2 ? b->seg[(size_t)(segments - 1 - j) * per + m - 1] : nullptr;
    };
    cudaEventRecord(ev[0], s);
    float* state = kept(1) ? kept(1) : b->st[0];
    int cur = 0;
    ok = ok && launch_step<float>(*b, inflow, true, nullptr, state, s);
    for (int n = 2; ok && n <= N; ++n) {
        float* dst = kept(n);
        if (!dst) dst = b->st[cur ^= 1];
        ok = launch_step<float>(*b, inflow, false, state, dst, s);
        state = dst;
    }
    cudaEventRecord(ev[1], s);
    // loss and the seed of lambda_N
    if (ok) {
        adj_probe_kernel<float><<<blocks_for(b->nprobe, 64), 64, 0, s>>>(G, state, inflow[0], inflow[1], inflow[2],
                                                                          b->nprobe, b->probe_cells, b->probe_target,
                                                                          b->probe_u, b->probe_loss);
        count_launch();
        ok = adj_ok(cudaMemsetAsync(b->lam[0], 0, bytes, s), "lambda clear");
    }
    if (ok) {
        adj_seed_kernel<<<b->nprobe, 32, 0, s>>>(G, state, inflow[0], inflow[1], inflow[2], b->nprobe, b->probe_cells,
                                                 b->probe_target, b->lam[0], b->du_probe);
        count_launch();
        ok = adj_ok(cudaGetLastError(), "seed kernel");
    }
    // reverse sweep over segments: segment j covers calls jK+1 .. min((j+1)K, N)
    // and needs s_{jK} .. s_{(j+1)K-1} (s_0 = the initial equilibrium). The
    // states of segment j - 1 are recomputed on the side stream, into the
    // other of two buffer sets, while segment j is reversed on s: the
    // recomputation reads only checkpoint j - 1, so the two run side by side.
    int lc = 0;
    double rec_ms = 0.0, rev_ms = 0.0;
    cudaStream_t s2 = b->side;
    std::vector<cudaEvent_t> evw(segments), evr(segments), eve(segments);  // on s: before / after the wait, after the reverse
    cudaEvent_t rec_done[2], rev_done[2], fwd_done;
    bool rev_used[2] = {false, false};
    for (int k = 0; k < segments; ++k) {
        cudaEventCreate(&evw[k]);
        cudaEventCreate(&evr[k]);
        cudaEventCreate(&eve[k]);
    }
    for (int k = 0; k < 2; ++k) {
        cudaEventCreateWithFlags(&rec_done[k], cudaEventDisableTiming);
        cudaEventCreateWithFlags(&rev_done[k], cudaEventDisableTiming);
    }
    cudaEventCreateWithFlags(&fwd_done, cudaEventDisableTiming);
    // the side stream starts after the forward (force field, checkpoints)
    ok = ok && adj_ok(cudaEventRecord(fwd_done, s), "sweep fork") && adj_ok(cudaStreamWaitEvent(s2, fwd_done, 0), "sweep fork");
    auto recompute = [&](int j, int set) {
        const int first = j * K + 1, last = std::min((j + 1) * K, N);
        if (rev_used[set] && !adj_ok(cudaStreamWaitEvent(s2, rev_done[set], 0), "segment reuse")) return false;
        const float* prev = j > 0 ? b->ckpt[j] : nullptr;
        for (int m = 1; m <= last - first; ++m) {
            float* dst = b->seg[(size_t)set * per + m - 1];
            if (!(m == 1 && j == 0 ? launch_step<float>(*b, inflow, true, nullptr, dst, s2)
                                   : launch_step<float>(*b, inflow, false, prev, dst, s2)))
                return false;
            prev = dst;
        }
        return adj_ok(cudaEventRecord(rec_done[set], s2), "segment done");
    };
    for (int j = segments - 1, idx = 0; ok && j >= 0; --j, ++idx) {
        const int set = idx % 2;
        if (j > 0 && j - 1 < segments - 2) ok = recompute(j - 1, set ^ 1);
        const int first = j * K + 1, last = std::min((j + 1) * K, N);
        // states[m] = s_{jK + m} for m = 1 .. last - first (s_{jK} = ckpt[j])
        std::vector<const float*> states(last - first + 1, nullptr);
        states[0] = j > 0 ? b->ckpt[j] : nullptr;
        for (int m = 1; m <= last - first; ++m) states[m] = b->seg[(size_t)set * per + m - 1];
        ok = ok && adj_ok(cudaEventRecord(evw[idx], s), "sweep event") && (j >= segments - 2 || adj_ok(cudaStreamWaitEvent(s, rec_done[set], 0), "segment wait")) &&
             adj_ok(cudaEventRecord(evr[idx], s), "sweep event");
        for (int n = last; ok && n >= first; --n) {
            const int m = n - first;  // input state of call n is states[m]
            StepArgs<float> a = step_args<float>(*b, inflow, states[m], nullptr);
            // the reverse launch writes every fluid slot of lam[lc ^ 1] (scatter)
            const unsigned blocks = b->rev_blocks;
            const int threads = b->rev_threads;
            float *lam = b->lam[lc], *prev = b->lam[lc ^ 1];
            if (n == 1) adj_reverse_kernel<true, unsigned long long><<<blocks, threads, 0, s>>>(a, lam, prev, b->grad_f, b->du_part);
            else if (narrow(*b)) adj_reverse_kernel<false, unsigned><<<blocks, threads, 0, s>>>(a, lam, prev, b->grad_f, b->du_part);
            else adj_reverse_kernel<false, unsigned long long><<<blocks, threads, 0, s>>>(a, lam, prev, b->grad_f, b->du_part);
            count_launch();
            ok = adj_ok(cudaGetLastError(), "reverse kernel");
            lc ^= 1;
        }
        ok = ok && adj_ok(cudaEventRecord(eve[idx], s), "sweep event") && adj_ok(cudaEventRecord(rev_done[set], s), "sweep event");
        rev_used[set] = true;
    }
    if (ok) ok = adj_ok(cudaStreamSynchronize(s), "sweep sync");
    for (int k = 0; ok && k < segments; ++k) {
        rec_ms += elapsed(evw[k], evr[k]);
        rev_ms += elapsed(evr[k], eve[k]);
    }
    for (int k = 0; k < segments; ++k) {
        cudaEventDestroy(evw[k]);
        cudaEventDestroy(evr[k]);
        cudaEventDestroy(eve[k]);
    }
    for (int k = 0; k < 2; ++k) {
        cudaEventDestroy(rec_done[k]);
        cudaEventDestroy(rev_done[k]);
    }
    cudaEventDestroy(fwd_done);
    std::vector<double> pl(b->nprobe), du(3 * ((size_t)b->rev_blocks + b->nprobe));
    if (ok) ok = adj_ok(cudaMemcpyAsync(pl.data(), b->probe_loss, b->nprobe * sizeof(double), cudaMemcpyDeviceToHost, s),
                        "loss read") &&
                 adj_ok(cudaMemcpyAsync(du.data(), b->du_part, du_bytes, cudaMemcpyDeviceToHost, s), "gradient read") &&
                 adj_ok(cudaMemcpyAsync(du.data() + 3 * (size_t)b->rev_blocks, b->du_probe, 3 * (size_t)b->nprobe * sizeof(double),
                                        cudaMemcpyDeviceToHost, s), "gradient read");
    if (ok && out_grad_force)
        ok = adj_ok(cudaMemcpyAsync(out_grad_force, b->grad_f, 3 * b->cells * sizeof(double), cudaMemcpyDeviceToHost, s),
                    "gradient read");
    if (ok) ok = adj_ok(cudaStreamSynchronize(s), "gradient sync");
    if (ok) {
        b->fwd_ms = elapsed(ev[0], ev[1]);
        b->recompute_ms = rec_ms;
        b->rev_ms = rev_ms;
        b->fwd_steps = N;
        b->rev_steps = N;
        b->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }
    for (auto& e : ev) cudaEventDestroy(e);
    if (!ok) return 0;
    double loss = 0.0, gu[3] = {0.0, 0.0, 0.0};
    for (double v : pl) loss += v;
    for (size_t k = 0; k < du.size(); ++k) gu[k % 3] += du[k];
    if (out_loss) *out_loss = loss;
    if (out_grad_inflow) {
        out_grad_inflow[0] = gu[0];
        out_grad_inflow[1] = gu[1];
        out_grad_inflow[2] = gu[2];
    }
    return 1;
}

// Device times of the last gradient call: forward (with checkpoint copies),
// segment recomputation and reverse launches, per call, and the wall time.
AERO_LBM_B200_EXPORT int aero_lbm_b200_adjoint_timing(long long handle, double* fwd_ms_per_step, double* recompute_ms_per_step,
                                                      double* rev_ms_per_step, double* total_ms) {
    std::lock_guard<std::mutex> lk(g_adj_mutex);
    Brick* b = find_brick(handle);
    if (!b || b->fwd_steps == 0) return 0;
    if (fwd_ms_per_step) *fwd_ms_per_step = b->fwd_ms / b->fwd_steps;
    if (recompute_ms_per_step) *recompute_ms_per_step = b->recompute_ms / b->rev_steps;
    if (rev_ms_per_step) *rev_ms_per_step = b->rev_ms / b->rev_steps;
    if (total_ms) *total_ms = b->total_ms;
    return 1;
}

AERO_LBM_B200_EXPORT void aero_lbm_b200_adjoint_destroy(long long handle) {
    std::lock_guard<std::mutex> lk(g_adj_mutex);
    auto it = g_adj.find(handle);
    if (it == g_adj.end()) return;
    cudaStreamSynchronize(current_stream());
    delete it->second;
    g_adj.erase(it);
}

AERO_LBM_B200_EXPORT const char* aero_lbm_b200_adjoint_last_error(void) { return g_adj_error.c_str(); }

// One cell's collision and its vector-Jacobian product on the host CPU
// (precision 0 float, 1 double), for checking the reverse sweep against
// finite differences without a GPU.
AERO_LBM_B200_EXPORT int aero_lbm_b200_adjoint_collide_vjp_host(int precision, const AeroLbmB200AdjointConfig* cfg,
                                                                const double* f_in, double temperature,
                                                                const double* cell_force, const double* lam_out,
                                                                double* f_out, double* lam_in, double* lam_force) {
    if (!cfg || !f_in || !cell_force || !lam_out || !f_out || !lam_in || !lam_force) return 0;
    const CollideParams cp = params_of(*cfg);
    if (precision == 0) {
        float f[27], fo[27], lo[27], li[27], lf[3];
        for (int q = 0; q < 27; ++q) { f[q] = (float)f_in[q]; lo[q] = (float)lam_out[q]; }
        CollideTape<float> t;
        collide_fwd<float>(f, cp, (float)temperature, (float)cell_force[0], (float)cell_force[1], (float)cell_force[2], fo, t);
        collide_vjp<float>(t, cp, lo, li, lf);
        for (int q = 0; q < 27; ++q) { f_out[q] = fo[q]; lam_in[q] = li[q]; }
        for (int a = 0; a < 3; ++a) lam_force[a] = lf[a];
    } else {
        double f[27], fo[27], lo[27], li[27], lf[3];
        for (int q = 0; q < 27; ++q) { f[q] = f_in[q]; lo[q] = lam_out[q]; }
        CollideTape<double> t;
        collide_fwd<double>(f, cp, temperature, cell_force[0], cell_force[1], cell_force[2], fo, t);
        collide_vjp<double>(t, cp, lo, li, lf);
        for (int q = 0; q < 27; ++q) { f_out[q] = fo[q]; lam_in[q] = li[q]; }
        for (int a = 0; a < 3; ++a) lam_force[a] = lf[a];
    }
    return 1;
}

}  // extern "C"
