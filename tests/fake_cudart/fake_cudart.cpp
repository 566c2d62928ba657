// A stand-in for the CUDA runtime under the library's own host code (dsmd_core.cu, dsmd_edges.cu): device memory is host memory,
// kernels are named but do not run, and any launch can be refused. The few kernels that report to the host are played: the end of
// a list build, the end of an edge search and displacement checks, with the gate that they close. Test infrastructure only.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <utility>
#include <vector>

#include "dsmd_force.cuh"

namespace {

std::map<const void*, std::string>& kernels() {   // (registered while the library's globals are constructed)
    static std::map<const void*, std::string> by_address;
    return by_address;
}
std::vector<std::string> log_;                 // launches, copies and waits, in the order of the calls
std::string refused;                           // launches of kernels with this in their name fail ...
int refuse_after = 0;                          // ... from this one on
cudaError_t last = cudaSuccess;
unsigned need_stride = 0;                      // what list builds find
bool outside = false, check_outside = false;   // an atom outside, found by list builds and by displacement checks
bool gate_closed = false;
int copies_until_failure = -1;
std::set<std::pair<const char*, const char*>> pinned_ranges;

void post(dsmd::Mail* mail, const double* v, int n, unsigned long long seq) {
    for (int k = 0; k < n; ++k) {
        unsigned long long bits;
        std::memcpy(&bits, v + k, sizeof(bits));
        mail->word[2 * k] = (bits >> 32 << 32) | (seq & 0xFFFFFFFFull);
        mail->word[2 * k + 1] = (bits << 32) | (seq & 0xFFFFFFFFull);
    }
}

void report_check(const dsmd::DisplacementReport& r) {
    if (gate_closed && r.gate2 < dsmd::kGateOpen) return;
    const double out[2] = {0.0, check_outside ? 1.0 : 0.0};
    gate_closed = check_outside;
    post(r.mail, out, 2, r.seq);
}

cudaError_t launch(const std::string& name, void** args) {
    if (!refused.empty() && name.find(refused) != std::string::npos && refuse_after-- <= 0) {
        log_.push_back("refused " + name);
        return last = cudaErrorLaunchOutOfResources;
    }
    log_.push_back("launch " + name);
    if (name.find("k_build_done") != std::string::npos) {
        const unsigned stride = *static_cast<unsigned*>(args[2]);
        const double out[4] = {outside ? 1.0 : 0.0, 0.0, need_stride ? static_cast<double>(need_stride == ~0u ? stride + 1 : need_stride) : 0.0, 0.0};
        gate_closed = outside || out[2] > stride;
        post(*static_cast<dsmd::Mail**>(args[3]), out, 4, *static_cast<unsigned long long*>(args[4]));
    } else if (name.find("k_post_displacement") != std::string::npos) {
        report_check(*static_cast<dsmd::DisplacementReport*>(args[0]));
    } else if (name.find("k_pack") != std::string::npos) {
        const auto& r = *static_cast<dsmd::DisplacementReport*>(args[23]);
        if (r.ticket) report_check(r);
    }
    return cudaSuccess;
}

}  // namespace

extern "C" {

// -- for the tests ----------------------------------------------------------------------------------------------------
void fake_reset() {
    log_.clear();
    refused.clear();
    refuse_after = 0;
    last = cudaSuccess;
    need_stride = 0;
    outside = check_outside = gate_closed = false;
    copies_until_failure = -1;
    pinned_ranges.clear();
}
void fake_refuse(const char* name, int after) { refused = name; refuse_after = after; }
void fake_build_finds(unsigned stride, int atoms_outside) { need_stride = stride; outside = atoms_outside != 0; }   // ~0: always a longer row
void fake_check_finds(int atoms_outside) { check_outside = atoms_outside != 0; }
void fake_pin(const char* p, size_t bytes) { pinned_ranges.insert({p, p + bytes}); }
void fake_fail_copy(int after) { copies_until_failure = after; }
int fake_log_size() { return static_cast<int>(log_.size()); }
const char* fake_log(int k) { return log_[k].c_str(); }

// -- runtime ----------------------------------------------------------------------------------------------------------
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 1; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { kernels()[host] = name; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
    *g = *b = dim3(1);
    *m = 0;
    *static_cast<void**>(s) = nullptr;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t) { return launch(kernels()[f], args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void** args) { return launch(kernels()[f], args); }
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(1, n + 16); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (copies_until_failure >= 0 && copies_until_failure-- == 0) {
        log_.push_back("failed copy");
        return last = cudaErrorUnknown;
    }
    for (const auto& r : pinned_ranges)   // as the runtime does: by where the copy starts
        if (s >= r.first && s < r.second) {
            if (static_cast<const char*>(s) + n > r.second) return last = cudaErrorInvalidValue;
            log_.push_back("queued copy");
        }
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* n) { *n = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { log_.push_back("wait"); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { log_.push_back("wait"); return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return last; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorLaunchOutOfResources ? "refused" : "error"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    *a = cudaPointerAttributes{};
    a->type = cudaMemoryTypeUnregistered;
    for (const auto& r : pinned_ranges)
        if (p >= r.first && p < r.second) a->type = cudaMemoryTypeHost;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { *a = cudaFuncAttributes{}; a->ptxVersion = a->binaryVersion = 100; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 1; return cudaSuccess; }

}  // extern "C"

// -- force kernels ----------------------------------------------------------------------------------------------------
namespace dsmd {

template <int COPIES, bool ENERGY, int ORDER>
cudaError_t launch_pair(const PairParams&, const ForceArgs& a, bool, unsigned, bool, cudaStream_t) {
    return launch(a.list_settled ? "k_pair early" : "k_pair", nullptr);
}

template <int ORDER>
cudaError_t launch_step(const PairParams&, const ForceArgs&, const Grid&, const StepArgs&, const DisplacementReport& r, bool, unsigned, cudaStream_t) {
    const cudaError_t e = launch("k_step", nullptr);
    if (e == cudaSuccess && r.ticket) report_check(r);
    return e;
}

template cudaError_t launch_pair<0, false, 0>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
template cudaError_t launch_pair<0, false, 2>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
template cudaError_t launch_pair<0, true, 0>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
template cudaError_t launch_pair<0, true, 2>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
template cudaError_t launch_pair<1, false, 0>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
template cudaError_t launch_pair<1, true, 0>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
template cudaError_t launch_pair<kEwaldCopiesMost, false, 2>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
template cudaError_t launch_pair<kEwaldCopiesMost, true, 2>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
template cudaError_t launch_step<0>(const PairParams&, const ForceArgs&, const Grid&, const StepArgs&, const DisplacementReport&, bool, unsigned, cudaStream_t);
template cudaError_t launch_step<2>(const PairParams&, const ForceArgs&, const Grid&, const StepArgs&, const DisplacementReport&, bool, unsigned, cudaStream_t);

}  // namespace dsmd
