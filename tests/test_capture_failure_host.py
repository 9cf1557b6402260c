"""A capture of step graphs that fails halfway (``batch.cu`` compiled here and linked
with stand-ins for the CUDA runtime and for the launches; no GPU is used). Whatever
call fails, and in whichever step of the capture, the case's step number, buffer
parity and lists of support sites are afterwards what they were: a failed capture of
the two step graphs is an error of the run, a failed capture of the 16-step graph
leaves the run to the step graphs."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "life_gb300", "csrc")

DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include <string>
#include "lbm_kernels.h"
#include "life_internal.h"
using namespace life;

// ---- stand-ins ----
static int calls, fail_at, captures, launched_one, launched_chain;

static bool capturing;
static cudaError_t hit() { return capturing && ++calls == fail_at ? cudaErrorMemoryAllocation : cudaSuccess; }

extern "C" {
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = true; captures++; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { const cudaError_t e = hit(); capturing = false; *g = nullptr; return e; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    capturing = true;
    const cudaError_t e = hit();
    capturing = false;
    if (e == cudaSuccess) *x = reinterpret_cast<cudaGraphExec_t>((size_t)captures);
    return e;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
    if ((size_t)x <= 2) launched_one++;
    else launched_chain++;
    return cudaSuccess;
}
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t*, size_t* n) { *n = 0; return cudaSuccess; }
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType* t) { *t = cudaGraphNodeTypeKernel; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return hit(); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return hit(); }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* f, cudaEvent_t, cudaEvent_t) { *f = 0; return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 1; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
// the object's own registration and launch stubs
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 1; }  // (skips the launch)
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t*, const void*) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
int life_case_create(const LifeCaseParams*, const LifeBodyDesc*, int32_t, LifeCase**) { return LIFE_ERR_INVALID; }
int life_case_destroy(LifeCase*) { return LIFE_OK; }
const char* life_last_error(void) { return ""; }
}
namespace life {
int set_error(int code, const std::string&) { return code; }
int cuda_fail(cudaError_t, const char*) { return LIFE_ERR_CUDA; }
int ensure_steps(LifeCase*, int, int) { return LIFE_OK; }
LatDev lattice_view(const LifeCase*, int) { return LatDev{}; }
cudaError_t launch_outlet(const LatDev&, double*, cudaStream_t) { return hit(); }
cudaError_t launch_record(const LifeCase*, int, cudaStream_t) { return hit(); }
cudaError_t launch_perimeter(const void*, void*, const LatDev&, int, cudaStream_t) { return hit(); }
cudaError_t launch_step_lowp(const void*, void*, const LatDev&, int, cudaStream_t) { return hit(); }
cudaError_t launch_interior_f64(const double*, double*, const LatDev&, int, cudaStream_t) { return hit(); }
cudaError_t launch_interior_lowp(const void*, void*, const LatDev&, int, cudaStream_t) { return hit(); }
cudaError_t launch_interior_batch_f64(const BatchLatCase*, const int*, int, int, int, int, int, cudaStream_t) { return hit(); }
cudaError_t launch_interior_batch_lowp(int, const BatchLatCase*, const int*, int, int, int, int, int, cudaStream_t) { return hit(); }
int batch_blocks_per_sm_f64(int) { return 1; }
int batch_blocks_per_sm_lowp(int, int) { return 1; }
}  // namespace life
int ibm_forces(LifeCase*, int, const void*, cudaStream_t) { return hit() == cudaSuccess ? LIFE_OK : LIFE_ERR_CUDA; }
int ibm_apply(LifeCase* c, int, const void*, void*, cudaStream_t) {
    if (hit() != cudaSuccess) return LIFE_ERR_CUDA;
    swap_site_lists(c->W);
    return hit() == cudaSuccess ? LIFE_OK : LIFE_ERR_CUDA;
}

// ---- the runs ----
static int bad;
static void expect(bool ok, const char* what, int at) {
    if (!ok && bad++ < 10) printf("failing call %d: %s\n", at, what);
}
static LifeCase* make(long long* s0, long long* s1) {
    LifeCase* c = new LifeCase();
    c->Nx = c->Ny = 64;
    c->obj.hasIBM = true;
    c->W.sites = s0;
    c->W.sites_prev = s1;
    return c;
}
int main() {
    static long long l0[1], l1[1];
    // the calls of the two step graphs' captures, and of the 16-step graph's
    calls = fail_at = 0;
    LifeCase* c = make(l0, l1);
    expect(case_graph_steps(c, 2, nullptr, nullptr) == LIFE_OK, "plain run", 0);
    const int two = calls;
    expect(case_graph_steps(c, 64, nullptr, nullptr) == LIFE_OK && launched_chain == 4, "plain chain", 0);
    const int all = calls;
    expect(two > 20 && all - two > 160, "calls counted", 0);
    int failed = 0;
    for (int at = 1; at <= all; at++) {
        calls = captures = launched_one = launched_chain = 0;
        fail_at = at;
        c = make(l0, l1);
        const int rc = case_graph_steps(c, 2, nullptr, nullptr);
        if (at <= two) {
            failed++;
            expect(rc != LIFE_OK, "a failed capture of the step graphs is an error", at);
            expect(c->t == 0 && c->cur == 0 && c->W.sites == l0 && c->W.sites_prev == l1, "view after the error", at);
            // and the case can be stepped again
            captures = 0;
            expect(case_graph_steps(c, 3, nullptr, nullptr) == LIFE_OK && c->t == 3 && c->cur == 1 && c->W.sites == l1, "later run", at);
        } else {
            expect(rc == LIFE_OK && c->t == 2 && c->W.sites == l0, "step graphs", at);
            const int r2 = case_graph_steps(c, 65, nullptr, nullptr);
            expect(r2 == LIFE_OK, "a failed 16-step graph is no error", at);
            expect(c->t == 67 && c->cur == 1 && c->W.sites == l1 && c->W.sites_prev == l0, "view after the run", at);
            expect(launched_chain == 0 && launched_one == 67, "steps one by one", at);
        }
    }
    printf("%d %d %d\n", all, failed, bad);
    return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cxx = shutil.which("g++")
    if not os.path.exists(nvcc) or not cxx:
        pytest.skip("nvcc or g++ not found")
    d = tmp_path_factory.mktemp("capture")
    src, obj, exe = d / "driver.cpp", d / "batch.o", d / "driver"
    src.write_text(DRIVER)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    inc = ["-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I", cuda]
    for cmd in ([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", *inc[:4], "-c",
                 os.path.join(CSRC, "batch.cu"), "-o", str(obj)],
                [cxx, "-O1", "-std=c++17", *inc, str(src), str(obj), "-o", str(exe)]):
        res = subprocess.run(cmd, capture_output=True, text=True)
        assert res.returncode == 0, res.stderr[-3000:]
    return str(exe)


def test_failed_capture_leaves_the_case_as_it_was(driver):
    res = subprocess.run([driver], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stderr
    total, failed, bad = map(int, res.stdout.split()[-3:])
    assert bad == 0, res.stdout
    assert total > 180 and failed > 20
