// The host side of fne_cg_* on a stand-in for the CUDA runtime: no device, no
// kernel runs.  A graph launch writes the state that the script names for it
// where the graph's last kernel would, and the calls are written to a log.
// Built and read by test_cg_host.py.
#include "../fenics_nonlinear_energies_b200/csrc/fne_krylov.cu"

#include <cstdio>
#include <cstdlib>
#include <cstring>

namespace fne {
std::string g_text;
int set_error(int code, const std::string& msg) {
  g_text = msg;
  return code;
}
}  // namespace fne

namespace {
std::vector<std::string> calls;             // graph launches, waits, event records, frees
std::vector<double> residual;               // ||r||^2 after graph k; -1: this one reports the stop
cudaError_t last = cudaSuccess;
int launches = 0, graphs = 0, fail_graph = -1, fail_wait = -1, waits = 0, capturing = 0;
fne::CgState* host_state = nullptr;
int chunk = 0, handles = 0;
std::vector<void*> events;
std::string name_of(cudaEvent_t e) {
  for (size_t k = 0; k < events.size(); ++k)
    if (events[k] == (void*)e) return k == 2 ? "done" : "ev" + std::to_string(k);
  return "?";
}
}  // namespace

#ifndef __CUDA_ARCH__  // (the compiler's device pass brings its own)
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return (*p = std::calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) {
  if (p) calls.push_back("free");
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(1, n);
  host_state = static_cast<fne::CgState*>(*p);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  calls.push_back("copy");
  return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return std::memset(p, v, n), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  events.push_back(*e = (cudaEvent_t)std::malloc(1));
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return calls.push_back("record " + name_of(e)), cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  calls.push_back("wait " + name_of(e));
  return name_of(e) != "done" && waits++ == fail_wait ? last = cudaErrorLaunchFailure : cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  return *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone, cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)std::malloc(1), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = (cudaGraph_t)std::malloc(1), cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  chunk = (launches - 1) / 2;  // two kernels an iteration and the state kernel went into the graph
  launches = 0;
  return *e = (cudaGraphExec_t)std::malloc(1), cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return calls.push_back("destroy graph"), cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
  if (graphs == fail_graph) return last = cudaErrorLaunchFailure;
  const double rr = residual[std::min<size_t>(graphs, residual.size() - 1)];
  fne::CgState s = host_state[(graphs + 1) & 1];
  if (!s.stop) {
    s.it = s.its = (graphs + 1) * chunk;
    s.maxit = 1000000;
    s.rr0 = 1.0;
    s.tol2 = 1e-12;
    s.rr = rr;
    s.stop = rr == -1.0;
  }
  host_state[graphs++ & 1] = s;
  launches += 2 * chunk + 1;
  calls.push_back("graph");
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "scripted failure"; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { return *n = 2, cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  return *n = 2, cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return ++launches, cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return ++launches, cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
  *g = *b = dim3(1), *m = 0, *static_cast<cudaStream_t*>(s) = nullptr;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return ++launches, cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { return *k = (cudaKernel_t)f, cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { return reinterpret_cast<void**>(&handles); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
char __cudaInitModule(void**) { return 1; }
}
#endif

// usage: chunk, graph launch that fails (-1: none), wait that fails (-1), whether the solve's stream is being captured,
// residual after each graph ... (the last for all that follow; -1: stop; nan)
int main(int argc, char** argv) {
  fail_graph = std::atoi(argv[2]);
  fail_wait = std::atoi(argv[3]);
  for (int k = 5; k < argc; ++k) residual.push_back(std::atof(argv[k]));
  const int64_t idx[4] = {0, 1, 2, 3};
  const double v[4] = {1, 1, 1, 1};
  double x[4];
  fne_cg* c = nullptr;
  int32_t its = 0, why = 0;
  if (fne_cg_create(4, 4, idx, idx, 0, std::atoi(argv[1]), &c) != FNE_OK) return 2;
  fne_cg_set_matrix(c, v, nullptr);
  calls.clear();
  launches = 0;
  capturing = std::atoi(argv[4]);
  const int rc = fne_cg_solve(c, v, x, 1e-6, 1000000, &its, &why, nullptr);
  int64_t told = -1;
  fne_cg_launches(c, &told);
  std::printf("%d %d %d %d\n", rc, its, launches, (int)told);
  for (const auto& s : calls) std::printf("%s,", s.c_str());
  calls.clear();
  fne_cg_destroy(c);
  std::printf("\n%s,%s\n", calls[0].c_str(), calls[1].c_str());
  return 0;
}
