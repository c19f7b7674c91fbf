"""A tick of the brick world in which one thing fails, on the CPU: the service
(brick_world.cu) is linked against fakes of the CUDA runtime and of the solver,
which note the calls and return the failures. A failed joint launch costs the
bricks of that launch their contexts and no others; a tick that ends early at a
brick it cannot prepare has stepped the bricks in front of it."""
from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import aero_b200

CSRC = Path(__file__).resolve().parents[1] / "aerodynamics4mc-fabric_b200" / "csrc"

SOLVER = r"""
#include <map>
#include "runtime_internal.h"
namespace aero {
static std::map<long long, Context*> live;
static std::string error;
static long long failing = 0;
static int stepped_together = 0;
Context::~Context() {}
const std::string& last_error() { return error; }
void set_error(const std::string& m) { error = m; }
void clear_error() { error.clear(); }
std::recursive_mutex& runtime_mutex() { static std::recursive_mutex m; return m; }
cudaStream_t current_stream() { return nullptr; }
bool cuda_ok(cudaError_t e, const char* what) { if (e != cudaSuccess) error = what; return e == cudaSuccess; }
Context* find_context(long long key) { auto it = live.find(key); return it == live.end() ? nullptr : it->second; }
void halo_batch_begin() {}
bool halo_batch_flush() { return true; }
bool output_device(Context&, OutBox, int, float, float*) { return true; }
bool world_atlas(Context&, const bw::PublishArgs&, bool* done) { *done = false; return true; }
bool step_rect_device(long long key, int nx, int ny, int nz, const DeviceFill&) {
    Context*& c = live[key];
    if (!c) c = new Context;
    c->nx = nx; c->ny = ny; c->nz = nz;
    c->initialized = true;
    return true;
}
bool world_step_ready(const Context* c, int, int, int) { return c != nullptr; }
bool world_step_batch(const std::vector<WorldStepJob>& jobs) {
    error.clear();
    for (const WorldStepJob& j : jobs)
        if (failing && j.ctx == find_context(failing)) { error = "injected"; return false; }
    for (const WorldStepJob& j : jobs) *j.sync.flag = bw::kFlagBefore | bw::kFlagAfter;
    stepped_together += (int)jobs.size();
    return true;
}
namespace bw {
cudaError_t launch_fill(const FillArgs&, const CellFields&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_sync(const SyncArgs& a, cudaStream_t) { *a.flag = kFlagBefore | kFlagAfter; return cudaSuccess; }
cudaError_t launch_publish(const PublishArgs&, cudaStream_t) { return cudaSuccess; }
}
}
extern "C" {
void aero_lbm_release_context(long long key) { aero::live.erase(key); }
void fake_fail(long long key) { aero::failing = key; }
int fake_live() { return (int)aero::live.size(); }
int fake_stepped_together() { return aero::stepped_together; }
}
"""

RUNTIME = r"""
#include <cstdlib>
#include <cstring>
static int fail_malloc = 0;
extern "C" {
void fake_fail_malloc(int on) { fail_malloc = on; }
int cudaMalloc(void** p, size_t n) { *p = fail_malloc ? nullptr : calloc(1, n); return *p ? 0 : 2; }
int cudaMallocHost(void** p, size_t n) { *p = calloc(1, n); return 0; }
int cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(1, n); return 0; }
int cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return 0; }
int cudaFree(void* p) { free(p); return 0; }
int cudaFreeHost(void* p) { free(p); return 0; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int, void*) { memcpy(d, s, n); return 0; }
int cudaMemsetAsync(void* d, int v, size_t n, void*) { memset(d, v, n); return 0; }
int cudaStreamSynchronize(void*) { return 0; }
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 1; }
#define OK(name) int name(...) { return 1; }
#define TEXT(name) const char* name(...) { return ""; }
OK(aero_lbm_benchmark_default_config) OK(aero_lbm_benchmark_reset_config) OK(aero_lbm_benchmark_set_config)
OK(aero_lbm_clear_d3q27_f16_boundary_shell_rect) OK(aero_lbm_context_realtime_cached_initialized)
OK(aero_lbm_exchange_halo_layers_rect) OK(aero_lbm_init_rect) OK(aero_lbm_patch_d3q27_f16_static_cells_rect)
OK(aero_lbm_set_d3q27_f16_boundary_shell_rect) OK(aero_lbm_set_realtime_solver_mode) OK(aero_lbm_shutdown)
OK(aero_lbm_step_rect_cached) TEXT(aero_lbm_last_error) TEXT(aero_lbm_memory_info) TEXT(aero_lbm_runtime_info)
TEXT(aero_lbm_timing_info)
}
"""


@pytest.fixture(scope="module")
def fakes(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("fakes")
    (d / "solver.cu").write_text(SOLVER)
    (d / "runtime.cpp").write_text(RUNTIME)
    flags = ["-std=c++17", "-O0", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
             f"-I{CSRC}", f"-I{CSRC.parents[1] / 'include'}", "-c"]
    units = [(d / "solver.cu", nvcc, flags), (CSRC / "brick_world.cu", nvcc, flags),
             (CSRC / "brick_world_deltas.cpp", nvcc, ["-x", "cu", *flags]), (d / "runtime.cpp", "g++", ["-fPIC", "-w", "-c"])]
    builds = [(subprocess.Popen([tool, *f, str(src), "-o", str(d / (src.name + ".o"))], stderr=subprocess.PIPE, text=True))
              for src, tool, f in units]
    for b in builds:
        assert b.wait() == 0, b.stderr.read()
    # the fakes' own cuda functions also where a process has loaded the real ones
    subprocess.run(["g++", "-shared", "-o", str(d / "fakes.so"), *[str(d / (u[0].name + ".o")) for u in units], "-Wl,--no-undefined,-Bsymbolic"],
                   check=True)
    return aero_b200.load_library(d / "fakes.so")


def world(lib, coords):
    n = 4
    svc = aero_b200.BrickWorldService(lib)
    svc.ensure_world(1, n)
    svc.set_hints(1, coords)
    for c in coords:
        add(svc, c)
    return svc


def add(svc, c):
    n = svc.n
    svc.upload_static(1, c, np.zeros((n, n, n), np.uint8))
    svc.upload_dynamic(1, c, np.full((n, n, n, 4), 0.01, np.float32), np.zeros((n, n, n), np.float32))


def test_failed_launch_keeps_the_other_launches(fakes):
    coords = [(2 * k, 0, 0) for k in range(40)]
    svc = world(fakes, coords)
    try:
        svc.step(1, 1)  # each brick's first call on its own
        before = fakes.fake_stepped_together()
        svc.step(1, 1)
        assert fakes.fake_stepped_together() - before == 40 and fakes.fake_live() == 40
        fakes.fake_fail(ctypes.c_longlong(-36))  # context keys count down from -1: the 36th brick
        before = fakes.fake_stepped_together()
        with pytest.raises(RuntimeError, match="injected"):
            svc.step(1, 1)
        assert fakes.fake_live() == 32
        assert fakes.fake_stepped_together() - before == 32
        fakes.fake_fail(ctypes.c_longlong(0))
        before = fakes.fake_stepped_together()
        svc.step(1, 1)  # the lost ones start again on their own
        assert fakes.fake_stepped_together() - before == 32 and fakes.fake_live() == 40
    finally:
        svc.release()


def test_early_end_steps_the_bricks_in_front(fakes):
    svc = world(fakes, [(0, 0, 0), (2, 0, 0), (4, 0, 0)])
    try:
        svc.step(1, 1)
        svc.set_hints(1, [(0, 0, 0), (2, 0, 0), (4, 0, 0), (6, 0, 0)])
        add(svc, (6, 0, 0))
        before = fakes.fake_stepped_together()
        fakes.fake_fail_malloc(1)
        with pytest.raises(RuntimeError):
            svc.step(1, 1)
        fakes.fake_fail_malloc(0)
        assert fakes.fake_stepped_together() - before == 3
        svc.step(1, 1)
        assert fakes.fake_live() == 4
    finally:
        fakes.fake_fail_malloc(0)
        svc.release()
