// Shared host-side plumbing of libncgb300: error state, dtype table, CUDA
// driver entry points (resolved through cudart, so the library loads on a
// machine without libcuda.so.1), and device properties.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/ncgb300.h"

namespace nca {

// Internal error: thrown inside the library, converted to a status code at the
// C ABI boundary (no exception crosses it).
struct Error : std::runtime_error {
  int code;
  Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

[[noreturn]] void fail(int code, const char* fmt, ...);
void set_last_error(const std::string& msg);
void clear_last_error();
// message of the last failed call on this thread (valid until the next call)
const std::string& last_error();

// Runs f, mapping exceptions to status codes.
template <class F>
int32_t guarded(F&& f) {
  try {
    clear_last_error();
    f();
    return NCA_OK;
  } catch (const Error& e) {
    set_last_error(e.what());
    return e.code;
  } catch (const std::bad_alloc&) {
    set_last_error("host allocation failed");
    return NCA_ERR_OOM;
  } catch (const std::exception& e) {
    set_last_error(e.what());
    return NCA_ERR_INVALID;
  } catch (...) {
    set_last_error("unknown error");
    return NCA_ERR_INVALID;
  }
}

void check_cuda(cudaError_t e, const char* what);
void check_cu(CUresult r, const char* what);

// ---- dtypes ----------------------------------------------------------------
struct DTypeInfo {
  const char* name;
  const char* ctype;   // C type in generated device code (storage type)
  int size;
  bool is_float;       // float32/float64/bfloat16/float16
  bool is_signed;
  bool device_ok;      // usable on the device path
};
const DTypeInfo& dtinfo(int dt);
bool dtype_valid(int dt);
// float32 stands in for the 16-bit float storage types in arithmetic
inline int arith_dtype(int dt) { return (dt == NCA_BFLOAT16 || dt == NCA_FLOAT16) ? NCA_FLOAT32 : dt; }
// op_traits<T>::sum_type (src/lib/ncarray/op_traits.hh:72-76,380-410); 16-bit floats -> float32
int sum_dtype(int dt);

// ---- driver API through cudart -----------------------------------------------
struct Driver {
  CUresult (*cuModuleLoadData)(CUmodule*, const void*);
  CUresult (*cuModuleGetFunction)(CUfunction*, CUmodule, const char*);
  CUresult (*cuLaunchKernel)(CUfunction, unsigned, unsigned, unsigned, unsigned, unsigned,
                             unsigned, unsigned, CUstream, void**, void**);
  CUresult (*cuFuncSetAttribute)(CUfunction, CUfunction_attribute, int);
  CUresult (*cuOccupancyMaxActiveBlocksPerMultiprocessor)(int*, CUfunction, int, size_t);
  CUresult (*cuGetErrorString)(CUresult, const char**);
  CUresult (*cuTensorMapEncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                     const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                     const cuuint32_t*, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion,
                                     CUtensorMapFloatOOBfill);
};
const Driver& drv();

// Number of kernels this library has launched (all entry points).
void count_launch(int64_t n = 1);
int64_t launch_count();

// Current device (initialising its primary context) and its SM count.
int current_device();
int sm_count(int dev);

// Stream-ordered scratch (cudaMallocAsync) freed at scope exit on the same stream.
struct StreamScratch {
  void* ptr = nullptr;
  cudaStream_t stream = nullptr;
  StreamScratch() = default;
  StreamScratch(size_t bytes, cudaStream_t s);
  ~StreamScratch();
  StreamScratch(const StreamScratch&) = delete;
  StreamScratch& operator=(const StreamScratch&) = delete;
};

// `n` arrival counters, all zero, for a kernel on stream `s` that leaves them
// zero; null where the caller has to zero counters of its own.
uint32_t* arrival_counters(int64_t n, cudaStream_t s);
// The same for a kernel that may leave any count: counters that no earlier
// launch has used since they were zeroed. The launch is made while `held` is.
struct FreshCounters {
  uint32_t* ptr = nullptr;
  std::unique_lock<std::mutex> held;
};
FreshCounters fresh_counters(int64_t n, cudaStream_t s);

// ---- chunk tables of the batched kernels --------------------------------------
// Bytes per chunk: a CTA's share of the batch in whole slabs, between 128 and
// 384 KiB; 512 KiB from 2 MiB a CTA on. Larger chunks have fewer ends (trees,
// counts) and leave more of the last round idle: 2000 arrays, 2.2 GB, at 128 /
// 256 / 384 / 512 / 1024 KiB 597 / 551 / 530 / 525 / 530 us; 600 arrays through
// the general form, 0.66 GB, at 64 / 128 / 256 / 384 KiB 254 / 216 / 201 / 197.
// Small batches: 160 arrays (352 KB a CTA) at 64 / 128 / 256 / 384 / 512 KiB
// 68 / 62 / 56 / 54 / 58 us, 40 arrays at 64 / 128 / 512 KiB 25 / 20 / 33.
inline long long chunk_bytes_for(long long total, long long ctas, long long slab) {
  const long long per = total / ctas;
  if (per >= 2 * 1024 * 1024) return 512 * 1024;
  return std::min<long long>(384 * 1024, std::max<long long>(128 * 1024, per / slab * slab));
}
// Stable order by descending size, in linear time: 64 classes per power of two.
template <class C, class F>
void order_chunks(std::vector<C>& chunks, F bytes) {
  auto cls = [&](const C& c) {
    const unsigned long long b = (unsigned long long)std::max<long long>(bytes(c), 0) + 64;
    int lg = 63 - __builtin_clzll(b);
    return lg * 64 + (int)((b >> (lg - 6)) & 63);
  };
  std::vector<int> start(64 * 64 + 1, 0);
  for (const C& c : chunks) ++start[(size_t)(64 * 64 - 1 - cls(c)) + 1];
  for (size_t k = 1; k < start.size(); ++k) start[k] += start[k - 1];
  std::vector<C> out(chunks.size());
  for (const C& c : chunks) out[(size_t)start[(size_t)(64 * 64 - 1 - cls(c))]++] = c;
  chunks.swap(out);
}

}  // namespace nca
