// A stand-in for the CUDA runtime and NVRTC that runs nothing and records
// everything: the library's own objects are linked against it (see
// __init__.py), so that the host side of a call -- which kernels it launches,
// with which grids, attributes and generated constants -- runs and is tested
// without a GPU. Memory is never touched; a "compiled" kernel is its source.
#include <cuda.h>
#include <cuda_runtime.h>
#include <nvrtc.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>

#define API extern "C" __attribute__((visibility("default")))

namespace {
struct Kernel {
  std::string name, defines;   // JSON members of the NCA_ constants
  int aux_word = -1;           // of a generated kernel: which argument word is its counters' address
};
std::mutex mu;
std::string log_text;
std::map<const void*, Kernel*> runtime_kernels;
int resident = 4;   // CTAs per SM that every occupancy query answers
thread_local dim3 call_grid, call_block;
thread_local size_t call_smem;
thread_local cudaStream_t call_stream;

void record(const std::string& line) {
  std::lock_guard<std::mutex> lk(mu);
  log_text += line + "\n";
}
void record_launch(const Kernel* k, dim3 g, dim3 b, size_t smem, const unsigned long long* words = nullptr) {
  record("{\"launch\": \"" + k->name + "\", \"grid\": [" + std::to_string(g.x) + ", " + std::to_string(g.y) + ", " +
         std::to_string(g.z) + "], \"block\": " + std::to_string(b.x) + ", \"smem\": " + std::to_string(smem) +
         (words && k->aux_word >= 0 ? ", \"aux\": " + std::to_string(words[k->aux_word]) : "") + ", \"consts\": {" + k->defines + "}}");
}
// "#define NCA_NAME <integer>" lines of a source as JSON members
std::string constants(const char* src) {
  std::string out;
  std::set<std::string> seen;
  for (const char* p = strstr(src, "#define NCA_"); p; p = strstr(p + 1, "#define NCA_")) {
    const char* n = p + 8;
    const char* e = n;
    while (*e && *e != ' ' && *e != '(' && *e != '\n') ++e;
    if (*e != ' ') continue;
    char* end;
    const long long v = strtoll(e + 1, &end, 10);
    if (end == e + 1 || (*end != '\n' && *end != 'u' && *end != '\0')) continue;
    const std::string name(n, e);
    if (!seen.insert(name).second) continue;
    out += (out.empty() ? "\"" : ", \"") + name + "\": " + std::to_string(v);
  }
  return out;
}

CUresult module_load(CUmodule* m, const void* image) {
  *m = (CUmodule) new std::string((const char*)image);
  return CUDA_SUCCESS;
}
CUresult module_function(CUfunction* f, CUmodule m, const char* name) {
  auto* k = new Kernel{name, constants(((std::string*)m)->c_str())};
  const size_t at = k->defines.find("\"NCA_W_AUX\": ");
  if (at != std::string::npos) k->aux_word = atoi(k->defines.c_str() + at + 13);
  *f = (CUfunction)k;
  return CUDA_SUCCESS;
}
CUresult launch(CUfunction f, unsigned gx, unsigned gy, unsigned gz, unsigned bx, unsigned by, unsigned bz, unsigned smem,
                CUstream, void** args, void**) {
  record_launch((const Kernel*)f, dim3(gx, gy, gz), dim3(bx, by, bz), smem, (const unsigned long long*)args[0]);
  return CUDA_SUCCESS;
}
CUresult func_attribute(CUfunction, CUfunction_attribute, int) { return CUDA_SUCCESS; }
CUresult occupancy(int* n, CUfunction, int, size_t) {
  *n = resident;
  return CUDA_SUCCESS;
}
CUresult error_string(CUresult, const char** s) {
  *s = "fake";
  return CUDA_SUCCESS;
}
CUresult tensor_map(CUtensorMap* m, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                    const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                    CUtensorMapFloatOOBfill) {
  memset(m, 0, sizeof(*m));
  return CUDA_SUCCESS;
}
}  // namespace

// ---- the log, for the tests -----------------------------------------------------
API const char* fake_log() {
  static std::string copy;
  std::lock_guard<std::mutex> lk(mu);
  copy = log_text;
  log_text.clear();
  return copy.c_str();
}
API void fake_resident(int n) { resident = n; }

// ---- host stubs of compiled kernels -----------------------------------------------
API void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
API void __cudaRegisterFatBinaryEnd(void**) {}
API void __cudaUnregisterFatBinary(void**) {}
API void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
API void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  std::lock_guard<std::mutex> lk(mu);
  runtime_kernels[host] = new Kernel{name, "", -1};
}
API unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
  call_grid = g; call_block = b; call_smem = smem; call_stream = s;
  return 0;
}
API cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = call_grid; *b = call_block; *smem = call_smem; *(cudaStream_t*)s = call_stream;
  return cudaSuccess;
}
API cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* host) {
  std::lock_guard<std::mutex> lk(mu);
  *k = (cudaKernel_t)runtime_kernels[host];
  return cudaSuccess;
}
API cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void**, size_t smem, cudaStream_t) {
  record_launch((const Kernel*)k, g, b, smem);
  return cudaSuccess;
}

// ---- runtime ------------------------------------------------------------------------
API cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
API cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrComputeCapabilityMajor ? 10
       : a == cudaDevAttrComputeCapabilityMinor ? 3 : 1 << 16;
  return cudaSuccess;
}
API cudaError_t cudaGetLastError() { return cudaSuccess; }
API const char* cudaGetErrorString(cudaError_t) { return "fake"; }
API cudaError_t cudaMalloc(void** p, size_t n) { *p = malloc(n); return cudaSuccess; }
API cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
API cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = (cudaMemPool_t)malloc(1); return cudaSuccess; }
API cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
API cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
  record("{\"scratch\": " + std::to_string(n) + "}");
  *p = malloc(n);
  return cudaSuccess;
}
API cudaError_t cudaFreeAsync(void* p, cudaStream_t) { free(p); return cudaSuccess; }
API cudaError_t cudaMemsetAsync(void* p, int, size_t n, cudaStream_t) {
  record("{\"memset\": " + std::to_string(n) + ", \"at\": " + std::to_string((unsigned long long)p) + "}");
  return cudaSuccess;
}
API cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
API cudaError_t cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) {
  return cudaSuccess;
}
API cudaError_t cudaMemcpyFromSymbolAsync(void*, const void*, size_t, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
API cudaError_t cudaMemcpyToSymbolAsync(const void*, const void*, size_t, size_t, cudaMemcpyKind, cudaStream_t) {
  return cudaSuccess;
}
API cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = (void*)s; return cudaSuccess; }
API cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::string name;
  {
    std::lock_guard<std::mutex> lk(mu);
    name = runtime_kernels[f]->name;
  }
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize)
    record("{\"smem_limit\": " + std::to_string(v) + ", \"kernel\": \"" + name + "\"}");
  return cudaSuccess;
}
API cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = resident; return cudaSuccess; }
API cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = resident;
  return cudaSuccess;
}
API cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
API cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
API cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
API cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
API cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }   // all alike: the first wins
API cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
API cudaError_t cudaStreamGetId(cudaStream_t s, unsigned long long* id) { *id = (unsigned long long)s; return cudaSuccess; }
API cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
API cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)malloc(1); return cudaSuccess; }
API cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
API cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
API cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
API cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
API cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
API cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
API cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
API cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** fn, unsigned, unsigned long long,
                                                 cudaDriverEntryPointQueryResult* q) {
  static const std::map<std::string, void*> table = {
      {"cuModuleLoadData", (void*)module_load},       {"cuModuleGetFunction", (void*)module_function},
      {"cuLaunchKernel", (void*)launch},              {"cuFuncSetAttribute", (void*)func_attribute},
      {"cuOccupancyMaxActiveBlocksPerMultiprocessor", (void*)occupancy},
      {"cuGetErrorString", (void*)error_string},      {"cuTensorMapEncodeTiled", (void*)tensor_map}};
  auto it = table.find(name);
  *fn = it == table.end() ? nullptr : it->second;
  *q = *fn ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}

// ---- NVRTC: the "cubin" of a source is the source -------------------------------------
API nvrtcResult nvrtcVersion(int* a, int* b) { *a = *b = 0; return NVRTC_SUCCESS; }
API nvrtcResult nvrtcCreateProgram(nvrtcProgram* p, const char* src, const char*, int, const char* const*, const char* const*) {
  record("{\"compile\": " + std::to_string(strlen(src)) + "}");
  *p = (nvrtcProgram) new std::string(src);
  return NVRTC_SUCCESS;
}
API nvrtcResult nvrtcCompileProgram(nvrtcProgram, int, const char* const*) { return NVRTC_SUCCESS; }
API nvrtcResult nvrtcDestroyProgram(nvrtcProgram* p) { delete (std::string*)*p; return NVRTC_SUCCESS; }
API const char* nvrtcGetErrorString(nvrtcResult) { return "fake"; }
API nvrtcResult nvrtcGetProgramLogSize(nvrtcProgram, size_t* n) { *n = 0; return NVRTC_SUCCESS; }
API nvrtcResult nvrtcGetProgramLog(nvrtcProgram, char*) { return NVRTC_SUCCESS; }
API nvrtcResult nvrtcGetCUBINSize(nvrtcProgram p, size_t* n) { *n = ((std::string*)p)->size() + 1; return NVRTC_SUCCESS; }
API nvrtcResult nvrtcGetCUBIN(nvrtcProgram p, char* out) {
  memcpy(out, ((std::string*)p)->c_str(), ((std::string*)p)->size() + 1);
  return NVRTC_SUCCESS;
}
