"""asv_evaluate when a CUDA call fails midway: it returns an error only after the
copies from the caller's arrays have ended, on whichever stream they run.  The
host code is built against stand-ins of the CUDA calls it makes, of which the
n-th copy, event or launch fails."""
import os
import subprocess

SRC = r"""
#include "asv.h"
#include "asv_eval.cuh"
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

static int calls, fail_at;                     // fallible calls of the evaluation, the one that fails
static std::vector<cudaStream_t> in_flight;    // streams with a copy from the caller's arrays queued
static char streams[8];
static int nstream;
static bool counting;
static cudaError_t step() { return counting && ++calls == fail_at ? cudaErrorUnknown : cudaSuccess; }

extern "C" {
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaErrorUnknown; }
const char *cudaGetErrorString(cudaError_t) { return "stand-in"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)&streams[nstream++]; return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return cudaStreamCreateWithFlags(s, 0); }
cudaError_t cudaStreamGetPriority(cudaStream_t, int *p) { *p = 0; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)&streams[7]; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return step(); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return step(); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { *p = calloc(1, n); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t st)
{
    if (step() != cudaSuccess) return cudaErrorUnknown;
    if (k == cudaMemcpyHostToDevice) in_flight.push_back(st);
    else memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
    for (size_t i = 0; i < in_flight.size();) {
        if (in_flight[i] == st) in_flight.erase(in_flight.begin() + i); else i++;
    }
    return cudaSuccess;
}
}
size_t asv_eval_sbound_words(int, int, int) { return 64; }
int asv_launch_eval_range_init(int *, cudaStream_t) { return step() ? -1 : 0; }
int asv_launch_eval_range(const int32_t *, const int32_t *, long long, int *, cudaStream_t) { return step() ? -1 : 0; }
int asv_launch_eval_sbound(const int32_t *, int, int, int, unsigned *, cudaStream_t) { return step() ? -1 : 0; }
int asv_launch_eval(const int32_t *, const int32_t *, int, int, int, int, int, unsigned *, int *, int *, const unsigned *,
                    unsigned long long *, cudaStream_t) { return step() ? -1 : 0; }

int main()
{
    asv_ctx *ctx = nullptr;
    if (asv_create(nullptr, &ctx) != ASV_OK) return 1;
    std::vector<int32_t> a(2 * 3 * 4), b(2 * 3 * 4);
    asv_eval e;
    int errors = 0;
    counting = true;
    for (fail_at = 1; fail_at < 64; fail_at++) {
        calls = 0;
        const asv_status s = asv_evaluate(ctx, a.data(), b.data(), 4, 3, 2, &e);
        if (s == ASV_OK && calls < fail_at) { printf("%d failing calls\n", errors); return errors > 8 ? 0 : 2; }
        errors += s != ASV_OK;
        // (a call whose result the evaluation need not look at may fail and change nothing)
        if (s != ASV_OK && !in_flight.empty()) { printf("call %d failed: copies still under way\n", fail_at); return 3; }
        in_flight.clear();
    }
    return 4;
}
"""


def test_no_copy_outlives_a_failed_call(tmp_path):
    from anisotropic_supervoxel_gb300 import _build
    src, exe = tmp_path / "eval_errors.cpp", str(tmp_path / "eval_errors")
    src.write_text(SRC)
    inc = [f for d in (_build.CSRC, _build.INCLUDE, os.path.join(_build.CUDA_HOME, "include")) for f in ("-I", d)]
    # the rest of the library's calls stay unresolved: none is made here
    subprocess.run(["g++", "-std=c++17", "-O1", *inc, str(src), os.path.join(_build.CSRC, "asv_api.cpp"), "-o", exe,
                    "-Wl,--unresolved-symbols=ignore-all"], check=True)
    p = subprocess.run([exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout
