"""A refused kernel launch ends the call with an error, whichever way the chunks are launched.

The host runtime (csrc/sp_runtime.cu, sp_tuning.cu, sp_server.cu hold no kernels) is compiled
with the host compiler against a stand-in for the CUDA runtime that keeps device memory on the
host and refuses what the case names: the step launch, or the step kernel's opt-in to its
dynamic shared memory.  Every refusal must come back as a status, once: the next call starts
clean, and what was created is destroyed."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "stochasticphysics_b200" / "csrc"
CUDA_INCLUDE = Path("/usr/local/cuda/include")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>
#include "sp_runtime.h"

static std::string refuse;
static thread_local cudaError_t last = cudaSuccess;
static int streams = 0, graphs = 0;
static cudaError_t set(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
extern "C" {
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "refused"; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
    return set(refuse == "attribute" ? cudaErrorInvalidValue : cudaSuccess);
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) { std::memset(p, 0, sizeof *p); p->multiProcessorCount = 148; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { ++streams; *s = reinterpret_cast<cudaStream_t>(8); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { --streams; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { ++graphs; *g = reinterpret_cast<cudaGraph_t>(8); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* g, cudaGraph_t, unsigned long long) { ++graphs; *g = reinterpret_cast<cudaGraphExec_t>(8); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { --graphs; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { --graphs; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(8); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { std::free(p); return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = size_t(1) << 34; return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = reinterpret_cast<cudaMemPool_t>(8); return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 1; return cudaSuccess; }
}

namespace sp {
static DeviceOnce once;
const KernelSet& kernel_set(int, int, int, int, int inject) {
    static KernelSet k;
    static const KernelSet none;
    k.valid = true;
    k.D = k.Mn = k.OUT = 3;
    k.real_bytes = 8;
    k.init = [](const EnsDev*, const RawParticles&, unsigned long long, cudaStream_t) {};
    k.step[0] = [](const EnsDev*, const TileDesc*, int, int, int, cudaStream_t) {
        if (refuse == "step") set(cudaErrorLaunchOutOfResources);
    };
    k.reduce = [](const EnsDev*, int, int, int, cudaStream_t) {};
    k.field = [](const EnsDev*, int, unsigned long long, int, cudaStream_t) {};
    k.prepare = [] { allow_dynamic_smem(reinterpret_cast<const void*>(8), 90000, once); };
    return inject ? none : k;
}
RawParticles provided_raw(const double*, unsigned long long) { return {}; }
double* provide_particles(sp_context*, const sp_ensemble_desc&, cudaStream_t) { return nullptr; }
unsigned long long upload_increments(sp_context*, const double*, void*, int, size_t, size_t, size_t, cudaStream_t) { return 0; }
void launch_commit(const EnsDev*, int, cudaStream_t) {}
void launch_bump_targets(const EnsDev*, int, cudaStream_t) {}
void launch_set_target(EnsCtl*, unsigned long long, cudaStream_t) {}
void launch_field_window(const FieldParams&, double, unsigned long long, unsigned long long, double*, cudaStream_t) {}
double measure_fma_peak(int, int, cudaStream_t) { return 0; }
void launch_debug_normals(unsigned long long, unsigned long long, unsigned long long, unsigned long long, unsigned long long, int, int, double*, cudaStream_t) {}
}  // namespace sp

int main(int, char** argv) {
    const std::string how = argv[1];
    std::vector<double> one(64, 1.0);
    sp_ensemble_desc d;
    std::memset(&d, 0, sizeof d);
    d.abi_version = SP_ABI_VERSION;
    d.problem = SP_PROBLEM_NEEL;
    d.solver = SP_SOLVER_HEUN_STRONG;
    d.precision = SP_PRECISION_FP64;
    d.noise = SP_NOISE_PHILOX;
    d.oversampling = 100;
    d.number_of_steps = how == "graph" ? 1000000 : 1000;
    d.timestep = 1e-12;
    d.n_particles = 4;
    sp_particles& q = d.particles;
    q.magnetic_radius = q.saturation_magnetisation = q.damping_constant = q.gyromagnetic_ratio = q.anisotropy_constant =
        q.hydrodynamic_radius = q.viscosity = q.orientation = q.magnetisation = one.data();
    sp_context* ctx = nullptr;
    if (sp_create(&ctx, 0) != SP_OK) return 1;
    const auto call = [&]() -> int {
        if (how == "ensemble") {
            sp_ensemble* e = nullptr;
            sp_status s = sp_ensemble_create(ctx, &d, &e);
            if (s == SP_OK) s = sp_ensemble_advance(e, 900, nullptr);
            sp_ensemble_destroy(e);
            return s;
        }
        if (how == "server") {
            sp_server* srv = nullptr;
            uint64_t id = 0;
            if (sp_server_create(ctx, nullptr, &srv) != SP_OK || sp_server_submit(srv, &d, &id) != SP_OK) return -1;
            const sp_status s = sp_server_wait(srv, id, 20000.0, nullptr, nullptr, nullptr);
            sp_server_destroy(srv);
            return s;
        }
        return sp_simulate(ctx, &d, nullptr, nullptr);
    };
    refuse = argv[2];
    const int first = call();
    const std::string text = first == SP_OK ? "" : sp_last_error();
    refuse = "";
    const int second = call();
    sp_destroy(ctx);
    std::printf("%d %d %d %d %s\n", first, second, streams, graphs, text.c_str());
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None or not (CUDA_INCLUDE / "cuda_runtime.h").exists():
        pytest.skip("no g++ or no CUDA headers")
    d = tmp_path_factory.mktemp("launch")
    (d / "t.cpp").write_text(PROGRAM)
    sources = [str(d / "t.cpp")] + [str(CSRC / f) for f in ("sp_runtime.cu", "sp_tuning.cu", "sp_server.cu")]
    subprocess.run([cxx, "-x", "c++", "-std=c++17", "-O1", "-pthread", "-I", str(CUDA_INCLUDE), "-I", str(CSRC), "-o",
                    str(d / "t")] + sources, check=True)
    return d / "t"


@pytest.mark.parametrize("refused", ["step", "attribute", "nothing"])
@pytest.mark.parametrize("how", ["direct", "graph", "ensemble", "server"])
def test_refused_launch_is_reported_once(program, how, refused):
    out = subprocess.run([str(program), how, refused], check=True, capture_output=True, text=True, timeout=60).stdout
    first, second, streams, graphs, text = (out.rstrip("\n") + " ").split(" ", 4)
    assert (int(first) != 0) == (refused != "nothing"), out
    assert int(second) == 0, "an error reported once came back in the next call"
    assert int(streams) == 0 and int(graphs) == 0
    if refused != "nothing":
        assert "refused" in text
