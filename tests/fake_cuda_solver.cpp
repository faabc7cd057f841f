// The solver's host code (csrc/solver.cpp) over a fake CUDA runtime in host
// memory and fakes of the launches that the scenario reaches: what becomes of
// the force scratch when a call fails half way. Exit code 0: sound.
#include "../include/foilcfd_step.h"
#include "kernels.h"

#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
std::map<const void*, size_t> sizes;
long long links = 0;        // length of the next force list
bool failTables = false;    // the next build fails after its lists have grown
int failMemset = -1;        // the memset that fails, counted down
int problems = 0;

void check(bool ok, const char* what) {
    if (ok) return;
    std::printf("FAILED: %s\n", what);
    ++problems;
}
cudaError_t take(void** p, size_t n) {
    *p = std::malloc(n);
    std::memset(*p, 0xff, n);   // device memory starts with anything
    sizes[*p] = n;
    return cudaSuccess;
}
cudaError_t give(void* p) {
    sizes.erase(p);
    std::free(p);
    return cudaSuccess;
}
} // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return take(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return take(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return take(p, n); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaFreeHost(void* p) { return give(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return give(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memmove(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memmove(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
    if (failMemset >= 0 && failMemset-- == 0) return cudaErrorLaunchFailure;
    std::memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

namespace fcfd {
bool is_device_pointer(const void*) { return false; }
void GeomScratch::release() {}
cudaError_t launch_fill(float*, long long, float, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_reset(Storage, void*, void*, const std::uint8_t*, LevelDims, float, float, unsigned, cudaStream_t) {
    return cudaSuccess;
}
size_t force_scratch_bytes(int count) { return (1 + 3 * static_cast<size_t>((count + 63) / 64)) * sizeof(double); }
cudaError_t build_level_tables(LevelDims, const std::uint8_t*, LevelTables& t, GeomScratch&, cudaStream_t) {
    t.linkCount = links;
    if (links > t.linkRoom) {
        cudaFree(t.linkCells);
        cudaFree(t.linkMasks);
        t.linkRoom = links + links / 8 + 1;
        cudaMalloc(reinterpret_cast<void**>(&t.linkCells), t.linkRoom * 4);
        cudaMalloc(reinterpret_cast<void**>(&t.linkMasks), t.linkRoom * 4);
    }
    if (failTables) {
        failTables = false;
        return cudaErrorLaunchFailure;
    }
    return cudaSuccess;
}
cudaError_t launch_force(Storage, const ForceList& l, cudaStream_t) {
    check(l.count == links, "the list is the last field's");
    check(sizes.count(l.scratch) && sizes[l.scratch] >= force_scratch_bytes(l.count), "scratch holds the list's partial sums");
    unsigned ticket;
    std::memcpy(&ticket, l.scratch, sizeof ticket);
    check(ticket == 0, "the ticket starts at zero");
    for (int k = 0; k < 3; ++k) l.out[k] = 0.0;
    return cudaSuccess;
}
} // namespace fcfd

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    const fcfd_dims d{16, 12, 4};
    fcfd_scaling sc{};
    sc.tau = 0.55f;
    sc.u_lat = 0.05f;
    std::vector<std::uint8_t> flags(16 * 12 * 4, 0);
    char err[256] = "";
    fcfd_solver* s = fcfd_create();
    double f[3];
    auto set = [&](long long n) { links = n; return fcfd_set_flags(s, flags.data(), flags.size()); };
    links = 10;
    check(fcfd_init(s, &d, &sc, flags.data(), flags.size(), nullptr, nullptr, err, sizeof err) == 0, err);
    check(fcfd_force_now(s, f) == 0, "force of the first field");
    if (what == "tables") {          // the list grew, then the build failed
        failTables = true;
        check(set(1000) != 0, "a failed build is reported");
    } else if (what == "memset") {   // the scratch grew, its clearing failed
        failMemset = 0;
        check(set(1000) != 0, "a failed clearing is reported");
    } else if (what != "grow") {
        check(false, "scenario");
    }
    check(set(1000) == 0, "the same field again");
    check(fcfd_force_now(s, f) == 0, "force of the longer list");
    check(set(10) == 0 && fcfd_force_now(s, f) == 0, "a short list again");
    fcfd_destroy(s);
    return problems;
}
