// A CUDA runtime that runs no kernel, for the library's host code on a machine without a GPU:
// linked with the library's objects in place of the runtime. Device memory is host memory,
// copies are copies, launches are recorded; the n-th allocation from now can be made to fail.
// A few launches leave what the host loops wait for: a solve is done after `passes` residuals.
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "resident.cuh"

namespace {
std::map<const void*, std::string> names;   // kernels by their host stubs
std::map<const void*, int> limits;          // dynamic shared memory allowed, by kernel
std::vector<std::string> log_;
std::string joined;
int fail_in = 0, lowered = 0, refused = 0, passes = 2, seen = 0, null_exchange = 0, give_up = 0;

cudaError_t allocate(void** p, size_t n) {
  *p = nullptr;
  if (fail_in > 0 && --fail_in == 0) return cudaErrorMemoryAllocation;
  *p = calloc(1, n ? n : 1);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}

cudaError_t launch(const void* f, void** args, size_t smem) {
  const std::string& n = names[f];
  log_.push_back(n);
  auto is = [&](const char* s) { return n.find(s) != std::string::npos; };
  if ((int)smem > (limits.count(f) ? limits[f] : 48 * 1024)) {
    ++refused;
    return cudaErrorInvalidValue;
  }
  if (is("k_residual_fast") || is("k_na_residual")) {
    ib3d::SolveCtl* ctl = *static_cast<ib3d::SolveCtl**>(args[is("k_na_residual") ? 8 : 9]);
    ctl->last_res = 1.0;
    if (++seen % passes == 0) ctl->done = 1;
  } else if (is("k_sor64")) {
    (*static_cast<ib3d::SolveCtl**>(args[is("k_sor64_fast") ? 6 : 7]))->done = 1;
  } else if (is("k_resident32")) {
    const ib3d::Resident32& a = *static_cast<ib3d::Resident32*>(args[0]);
    null_exchange += a.xch == nullptr;
    if (give_up) *a.err = 1;
  } else if (is("k_resident64")) {
    const ib3d::Resident64& a = *static_cast<ib3d::Resident64*>(args[0]);
    null_exchange += a.xch == nullptr || a.errs == nullptr || a.pc_out == nullptr;
    if (give_up) *a.err = 1;
  }
  return cudaSuccess;
}
}  // namespace

extern "C" {
// ---- what the tests read and set
void fake_fail_in(int n) { fail_in = n; }        // the n-th allocation from now fails
int fake_pending_failure() { return fail_in; }
int fake_lowered() { return lowered; }           // limits set below an earlier one
int fake_refused() { return refused; }           // launches above their kernel's limit
int fake_null_exchange() { return null_exchange; }
void fake_give_up(int on) { give_up = on; }      // on-chip sweeps report a wait that ran out
unsigned fake_quad_item(unsigned block, unsigned threads, unsigned t) { return ib3d::quad_item(block, threads, t); }
const char* fake_launches() {                    // kernels launched since the last call
  joined.clear();
  for (const auto& s : log_) joined += s + "\n";
  log_.clear();
  return joined.c_str();
}

// ---- the runtime
cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return allocate(p, n); }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  if (!d || !s) return cudaErrorInvalidValue;
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemset(void* d, int v, size_t n) {
  if (!d) return cudaErrorInvalidValue;
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
  if (limits.count(f) && v < limits[f]) ++lowered;
  limits[f] = v;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static void* mem = calloc(1, 32 << 20);
  *p = mem;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3, dim3, void** args, size_t smem, cudaStream_t) {
  return launch(f, args, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  return launch(f, args, c->dynamicSmemBytes);
}

// ---- what nvcc's host code calls
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* stub, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names[stub] = name;
}
static size_t pushed_smem;
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t smem, struct CUstream_st*) {
  pushed_smem = smem;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  *g = *b = dim3(1);
  *smem = pushed_smem;
  *static_cast<void**>(st) = nullptr;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* stub) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(stub));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void** args, size_t smem, cudaStream_t) {
  return launch(reinterpret_cast<const void*>(k), args, smem);
}
}
