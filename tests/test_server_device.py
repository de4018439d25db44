"""Where the server's device memory comes from (CPU, against a fake CUDA runtime).

The server of a device may be used from threads that have another device current, or
none yet: whatever a submission allocates has to be on the server's device, the
caller's device has to stay as it was, and a submission whose tables exist allocates
nothing. csrc/server.cu has no kernels, so it is compiled by the host compiler and
linked to a runtime that records every allocation's device.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "qtctreconstruction_b200", "csrc")
CUDA_INCLUDE = "/usr/local/cuda/include"

FAKE = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>
#include <vector>
#include "ctb200.h"
#include "ctb_internal.h"

static thread_local int current = 0;
static std::mutex mu;
static std::map<char*, std::pair<size_t, int>> blocks;  // allocation -> bytes, device
static int allocations = 0, wrong = 0;

static int device_of(const void* p) {
    std::lock_guard<std::mutex> lk(mu);
    auto it = blocks.upper_bound(const_cast<char*>(static_cast<const char*>(p)));
    if (it == blocks.begin()) return -1;
    --it;
    return static_cast<const char*>(p) < it->first + it->second.first ? it->second.second : -1;
}
extern "C" {
cudaError_t cudaSetDevice(int d) { current = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof *p);
    p->major = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t bytes) {
    *p = std::calloc(1, bytes);
    std::lock_guard<std::mutex> lk(mu);
    blocks[static_cast<char*>(*p)] = {bytes, current};
    ++allocations;
    if (current != 1) ++wrong;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::mutex> lk(mu);
    blocks.erase(static_cast<char*>(p));
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) { *p = std::calloc(1, bytes); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = size_t(1) << 30; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    a->type = cudaMemoryTypeHost;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaLaunchHostFunc(cudaStream_t, cudaHostFn_t f, void* p) { f(p); return cudaSuccess; }
}
namespace ctb {
static int used_elsewhere = 0;  // tables a kernel would use on another device
std::vector<float2> filter_table(const PadGeom&, int, bool) { return std::vector<float2>(16); }
std::vector<float2> fft_twiddle_table(int) { return std::vector<float2>(16); }
FiltLayout filt_layout(int sq, int) { return FiltLayout{sq, 8, sq + 16}; }
cudaError_t launch_trig(const float* deg, int, const Trig& t, cudaStream_t) {
    for (const void* p : {static_cast<const void*>(deg), static_cast<const void*>(t.cs),
                          static_cast<const void*>(t.order), static_cast<const void*>(t.end)})
        used_elsewhere += device_of(p) != 1;
    return cudaSuccess;
}
BpJob make_bp_job(const float4*, int, int, const FiltLayout&, int, Trig t, const float4*, int, float*, int, int) {
    used_elsewhere += device_of(t.order) != 1;
    return BpJob{};
}
FiltJob make_filt_job(const float*, int, int, const PadGeom&, const FiltLayout&, const float2* Hc, const float4*, int,
                      float, float4*) {
    used_elsewhere += device_of(Hc) != 1;
    return FiltJob{};
}
void bp_number_items(BpBatch&, int, int) {}
int bp_default_variant(int, int, int, int) { return 0; }
cudaError_t launch_filter_batch(const FiltBatch&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_backproject_batch(const BpBatch&, int, unsigned*, unsigned*, cudaStream_t, bool) {
    return cudaSuccess;
}
}  // namespace ctb

static int failures = 0;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); ++failures; } } while (0)

int main() {
    ctb_server_config cfg{};
    cfg.device = 1;
    cfg.memory_budget = size_t(64) << 20;
    cfg.copy_threads = 1;
    cfg.staging_bytes = 1 << 20;
    ctb_server* s = nullptr;
    if (ctb_server_create(&cfg, &s) != CTB_OK) return 2;
    std::vector<float> sino(1 << 20), out(1 << 20);
    auto round = [&](int count, int na) {
        std::vector<uint64_t> ids;
        for (int k = 0; k < count; ++k) {
            ctb_request r{};
            r.sino = sino.data();
            r.out = out.data();
            r.depth = 1;
            r.num_angles = na + k;
            r.bins = 17 + 8 * (k % 4);
            r.output_size = 16;
            r.flags = CTB_REQ_DEVICE;
            uint64_t id = 0;
            CHECK(ctb_server_submit(s, &r, &id) == CTB_OK);
            CHECK(current == 0);
            ids.push_back(id);
        }
        for (uint64_t id : ids) {
            CHECK(ctb_server_wait(s, id, 10000.0) == CTB_OK);
            CHECK(ctb_server_release(s, id) == CTB_OK);
        }
    };
    std::thread([&] { round(8, 30); }).join();  // a thread with device 0 current builds the tables
    const int before = allocations;
    std::thread([&] { round(64, 5000); }).join();
    CHECK(allocations == before);
    CHECK(wrong == 0);
    CHECK(ctb::used_elsewhere == 0);
    ctb_server_destroy(s);
    CHECK(blocks.empty());
    return failures ? 1 : 0;
}
"""


def test_allocations_are_on_the_servers_device(tmp_path):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    fake, exe = tmp_path / "fake.cpp", tmp_path / "server_device"
    fake.write_text(FAKE)
    cmd = ["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-I" + CUDA_INCLUDE,
           "-x", "c++", str(fake), os.path.join(CSRC, "server.cu"), os.path.join(CSRC, "host_math.cpp"),
           "-o", str(exe), "-lpthread"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
