// 2-D histogram binning of float32 (x, y) points with optional float32 weights.
//
// The reference has only an internal scatter-add (`dest[idx[i]] += src[i]`,
// src/lib/ncarray/device/kernels.cuh:660-680, host/elementwise.hh:482-505) and
// no public histogram API; this file adds one.
// Binning rule (the oracle restates it bit for bit): in float32,
//   fx = floor((x - x_lo) * sx),  sx = (float)(nbx / (x_hi - x_lo))   (same for y)
// and the point is kept only if 0 <= fx < nbx and 0 <= fy < nby (NaN dropped).
// counts (uint64) are exact; weights are summed per bin with float32 partial
// sums whose rounding errors are collected exactly (compensated), combined as
// sums of three floats, and added to the float32 output once at the end.
//
// A bin grid of more than a few thousand bins does not fit in shared memory
// and global atomics on it run at the L2 atomic rate, far below HBM speed.
// The partitioned path therefore reads the points once and the much smaller
// per-tile records once:
//   1. sample: one block of 1024 points in 32 estimates how many points fall
//      in each tile of TB consecutive bins; each tile gets a bucket with 25 %
//      slack (the total is bounded, so the scratch is sized on the host);
//   2. scatter: every CTA bins a chunk of points, orders the chunk's (bin
//      within tile: uint16, weight: float32) records by tile in shared memory
//      and appends each tile's run to its bucket with coalesced stores (one
//      global atomic per tile and chunk reserves the space); records that do
//      not fit in their bucket are added with global atomics directly;
//   3. accumulate: a persistent grid splits the concatenated buckets into
//      equal record ranges; a CTA counts each tile piece of its range into a
//      shared-memory copy of the tile (uint32 counts, float32 sums and
//      compensation terms: the value returned by the float atomic gives the
//      exact rounding error of each addition via TwoSum) and stores the piece;
//   4. combine: every bin adds its tile's pieces in a fixed order (uint64
//      counts, three-float weights) to the outputs.
// Passes 1 and 2 are in tiles.cuh.
// Small inputs and grids with too many tiles use direct global atomics.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <mutex>
#include <string>

#include "common.hpp"
#include "tiles.cuh"

namespace {

using namespace nca_tiles;

constexpr int THREADS = 256;
constexpr int ACC_THREADS = 1024;

static __device__ int g_hist_status;   // NCA_ERR_TIMEOUT after a wait that ran out

struct Bins {
  float xl, yl, sx, sy, fnx, fny;
  int nbx, nby;
};

__device__ __forceinline__ int bin_of(const Bins& B, float x, float y) {
  const float fx = floorf(__fmul_rn(__fsub_rn(x, B.xl), B.sx));
  const float fy = floorf(__fmul_rn(__fsub_rn(y, B.yl), B.sy));
  if (!(fx >= 0.0f && fx < B.fnx && fy >= 0.0f && fy < B.fny)) return -1;
  return (int)fy * B.nbx + (int)fx;
}

// The same bin for grids of at most 2^22 bins (the partitioned path), without
// float-to-int conversions: the floor of v in [0, 2^23) is the low mantissa
// bits of v + 2^23 rounded toward zero, and v >= 0 / v < n (integer n) accept
// exactly the values whose floor floorf(v) does.
__device__ __forceinline__ unsigned tile_bin_of(const Bins& B, float x, float y) {
  const float fx = __fmul_rn(__fsub_rn(x, B.xl), B.sx);
  const float fy = __fmul_rn(__fsub_rn(y, B.yl), B.sy);
  if (!(fx >= 0.0f && fx < B.fnx && fy >= 0.0f && fy < B.fny)) return NO_BIN;
  const unsigned ix = (unsigned)__float_as_int(__fadd_rz(fx, 8388608.0f)) & 0x7fffffu;
  const unsigned iy = (unsigned)__float_as_int(__fadd_rz(fy, 8388608.0f)) & 0x7fffffu;
  return iy * (unsigned)B.nbx + ix;
}

// ---- direct path: global atomics per point -------------------------------------
template <bool WEIGHTED>
__global__ void __launch_bounds__(THREADS)
hist2d_direct_kernel(const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ w,
                     long long n, Bins B, unsigned long long* __restrict__ counts, double* __restrict__ wacc) {
  const long long stride = (long long)gridDim.x * THREADS;
  for (long long i = (long long)blockIdx.x * THREADS + threadIdx.x; i < n; i += stride) {
    const int b = bin_of(B, __ldcs(x + i), __ldcs(y + i));
    if (b >= 0) {
      atomicAdd(counts + b, 1ull);
      if (WEIGHTED) atomicAdd(wacc + b, (double)__ldcs(w + i));
    }
  }
}

__global__ void __launch_bounds__(THREADS) wsum_finish_kernel(const double* __restrict__ wacc, float* __restrict__ wsum,
                                                               long long nb) {
  for (long long i = (long long)blockIdx.x * THREADS + threadIdx.x; i < nb; i += (long long)gridDim.x * THREADS)
    wsum[i] = __double2float_rn((double)wsum[i] + wacc[i]);
}

// the points as a source of the partition passes
template <bool WEIGHTED>
struct Points {
  static constexpr int NA = WEIGHTED ? 3 : 2;
  static constexpr bool VAL = WEIGHTED;
  const float *x, *y, *w;
  Bins B;
  unsigned long long* counts;
  double* wacc;
  __device__ __forceinline__ const unsigned* array(int k) const {
    return reinterpret_cast<const unsigned*>(k == 0 ? x : k == 1 ? y : w);
  }
  __device__ __forceinline__ unsigned bin(unsigned a, unsigned b) const {
    return tile_bin_of(B, __uint_as_float(a), __uint_as_float(b));
  }
  __device__ __forceinline__ void direct(unsigned bn, unsigned word) const {
    atomicAdd(counts + bn, 1ull);
    if (WEIGHTED) atomicAdd(wacc + bn, (double)__uint_as_float(word));
  }
};

// ---- pass 3: per-tile shared-memory histograms of record ranges -------------------
template <bool WEIGHTED>
__device__ __forceinline__ void acc_record(unsigned* c, float* s, float* e, unsigned l, float wv) {
  atomicAdd(&c[l], 1u);
  if (WEIGHTED) {
    const float old = atomicAdd(&s[l], wv);       // s[l] became fl(old + wv)
    const float sum = __fadd_rn(old, wv);
    const float bb = __fsub_rn(sum, old);
    const float err = __fadd_rn(__fsub_rn(old, __fsub_rn(sum, bb)), __fsub_rn(wv, bb));
    if (err != 0.f) atomicAdd(&e[l], err);
  }
}

template <bool WEIGHTED>
__device__ __forceinline__ void acc_vec(unsigned* c, float* s, float* e, uint4 q, float4 w0, float4 w1) {
  acc_record<WEIGHTED>(c, s, e, q.x & 0xffffu, w0.x);
  acc_record<WEIGHTED>(c, s, e, q.x >> 16, w0.y);
  acc_record<WEIGHTED>(c, s, e, q.y & 0xffffu, w0.z);
  acc_record<WEIGHTED>(c, s, e, q.y >> 16, w0.w);
  acc_record<WEIGHTED>(c, s, e, q.z & 0xffffu, w1.x);
  acc_record<WEIGHTED>(c, s, e, q.z >> 16, w1.y);
  acc_record<WEIGHTED>(c, s, e, q.w & 0xffffu, w1.z);
  acc_record<WEIGHTED>(c, s, e, q.w >> 16, w1.w);
}

template <bool WEIGHTED>
__device__ __forceinline__ void acc_range(unsigned* c, float* s, float* e, const unsigned short* __restrict__ rec_bin,
                                          const float* __restrict__ rec_w, long long a, long long b) {
  // records [a, b) of the record arrays; bucket starts are multiples of 8
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  long long a8 = (a + 7) & ~7ll;
  if (a8 > b) a8 = b;
  const long long nv = (b - a8) >> 3, b8 = a8 + (nv << 3);
  for (long long r = a + threadIdx.x; r < a8; r += ACC_THREADS)
    acc_record<WEIGHTED>(c, s, e, rec_bin[r], WEIGHTED ? rec_w[r] : 0.f);
  for (long long r = b8 + threadIdx.x; r < b; r += ACC_THREADS)
    acc_record<WEIGHTED>(c, s, e, rec_bin[r], WEIGHTED ? rec_w[r] : 0.f);
  const uint4* vb = reinterpret_cast<const uint4*>(rec_bin + a8);
  const float4* vw = reinterpret_cast<const float4*>(WEIGHTED ? rec_w + a8 : nullptr);
  long long v = threadIdx.x;
  for (; v + ACC_THREADS < nv; v += 2 * ACC_THREADS) {
    const uint4 q0 = __ldcs(vb + v), q1 = __ldcs(vb + v + ACC_THREADS);
    float4 w0 = z4, w1 = z4, w2 = z4, w3 = z4;
    if (WEIGHTED) {
      w0 = __ldcs(vw + 2 * v);
      w1 = __ldcs(vw + 2 * v + 1);
      w2 = __ldcs(vw + 2 * (v + ACC_THREADS));
      w3 = __ldcs(vw + 2 * (v + ACC_THREADS) + 1);
    }
    acc_vec<WEIGHTED>(c, s, e, q0, w0, w1);
    acc_vec<WEIGHTED>(c, s, e, q1, w2, w3);
  }
  if (v < nv) {
    const uint4 q0 = __ldcs(vb + v);
    float4 w0 = z4, w1 = z4;
    if (WEIGHTED) {
      w0 = __ldcs(vw + 2 * v);
      w1 = __ldcs(vw + 2 * v + 1);
    }
    acc_vec<WEIGHTED>(c, s, e, q0, w0, w1);
  }
}

template <bool WEIGHTED>
__global__ void __launch_bounds__(ACC_THREADS)
tile_accumulate_kernel(int nv, const long long* __restrict__ off, const long long* __restrict__ PV,
                       const unsigned short* __restrict__ rec_bin, const float* __restrict__ rec_w,
                       unsigned* __restrict__ pc, float* __restrict__ ps, float* __restrict__ pe, long long nbins) {
  extern __shared__ __align__(128) unsigned char sm[];
  unsigned* c = reinterpret_cast<unsigned*>(sm);
  float* s = reinterpret_cast<float*>(sm + TB * 4);
  float* e = reinterpret_cast<float*>(sm + TB * 8);
  const int G = gridDim.x, g = blockIdx.x;
  const long long R = PV[nv];
  const long long S1 = range_start(R, g + 1, G);
  long long pos = range_start(R, g, G);
  int v = 0;
  while (pos < S1) {
    while (PV[v + 1] <= pos) ++v;                // pos < R = PV[nv], so v < nv
    const int t = v;
    const long long tend = PV[t + 1] < S1 ? PV[t + 1] : S1;
    const int width = (int)(nbins - (long long)t * TB < TB ? nbins - (long long)t * TB : TB);   // the last tile may be short
    for (int i = threadIdx.x; i < width; i += ACC_THREADS) {
      c[i] = 0u;
      if (WEIGHTED) { s[i] = 0.f; e[i] = 0.f; }
    }
    __syncthreads();
    acc_range<WEIGHTED>(c, s, e, rec_bin, rec_w, off[t] + (pos - PV[t]), off[t] + (tend - PV[t]));
    pos = tend;
    __syncthreads();
    const long long slot = (long long)(g + t) * TB;
    for (int i = threadIdx.x; i < width; i += ACC_THREADS) {
      pc[slot + i] = c[i];
      if (WEIGHTED) {
        ps[slot + i] = s[i];
        pe[slot + i] = e[i];
      }
    }
    __syncthreads();
  }
}

// A weight sum as three floats: additions to the first two keep their rounding
// errors exactly, the third collects what the second loses. With n terms and
// partial sums up to M it is off by at most about n^3 M 2^-72, less than the
// n M 2^-53 of a float64 sum for n up to 700; a bin has at most a piece per
// accumulating CTA, one an SM.
struct Sum3 {
  float hi, mid, lo;
  // a = rn(a + b); returns the error of that addition
  static __device__ __forceinline__ float two_sum(float& a, float b) {
    const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    a = s;
    return e;
  }
  __device__ __forceinline__ void add(float a, float b) {
    const float ea = two_sum(hi, a), eb = two_sum(mid, b);
    lo = __fadd_rn(lo, __fadd_rn(eb, two_sum(mid, ea)));
  }
  __device__ __forceinline__ void add(const Sum3& o) {
    add(o.hi, o.mid);
    lo = __fadd_rn(lo, o.lo);
  }
  // a sum that left float32's range stays outside it
  __device__ __forceinline__ bool finite() const { return fabsf(hi) < __int_as_float(0x7f800000); }
  // the sum as a float, off by half a unit in the last place
  __device__ __forceinline__ float get() {
    const float e = two_sum(hi, mid);
    return __fadd_rn(hi, __fadd_rn(e, lo));
  }
};

// ---- pass 4: add the pieces of every bin's tile to the outputs ----------------------
// A block takes 4 * THREADS / CG bins of one tile, four a thread, and splits the
// tile's pieces over CG groups of threads, merged in a fixed order: with few
// tiles one has pieces from many CTAs, and a loop over them is a chain of load
// latency (CG = 8 from 8 pieces a tile on: 64 x 64 bins, 2^20 weighted points 54
// us a call with CG = 4, 48 with 8; 1024 x 1024 bins have 2-3 pieces a tile,
// CG = 1). The sharing CTAs come from the prefix pass and the weights are sums
// of three floats (Sum3): 64-bit divisions and float64 adds and conversions per
// bin were most of the pass (50-65 us for 1024 x 1024 weighted bins, 20-22 with
// pairs of floats; with three a call takes the same time within 1 us). The
// output's old value is one more term: 2^20 points added to 2048 x 2048 bins
// 160 -> 134 us a call without float64 arithmetic for it.
template <bool WEIGHTED, int CG>
__global__ void __launch_bounds__(THREADS)
tile_combine_kernel(long long nbins, int G, const long long* __restrict__ PV,
                    const unsigned* __restrict__ pc, const float* __restrict__ ps, const float* __restrict__ pe,
                    const double* __restrict__ wacc, unsigned long long* __restrict__ counts,
                    float* __restrict__ wsum, int ntiles, const int2* __restrict__ ctas) {
  static_assert(TB % (4 * THREADS) == 0, "a block's bins lie in one tile");
  constexpr int Q = THREADS / CG;   // threads per group, four bins each
  constexpr int LOADS = WEIGHTED ? 4 : 8;
  __shared__ int s_bad;
  __shared__ unsigned long long scn[CG > 1 ? CG - 1 : 1][CG > 1 ? Q : 1][4];
  __shared__ Sum3 sw[CG > 1 && WEIGHTED ? CG - 1 : 1][CG > 1 && WEIGHTED ? Q : 1][4];
  const int q = threadIdx.x % Q, grp = threadIdx.x / Q;
  const long long bin0 = (long long)blockIdx.x * 4 * Q;
  const int t = (int)(bin0 / TB);
  const long long R = PV[ntiles];
  const int s_first = ctas[t].x, s_last = ctas[t].y;
  if (CG > 1) {
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
  }
  const long long bin = bin0 + 4 * q;
  unsigned long long cn[4] = {0, 0, 0, 0};
  Sum3 ws[4] = {};
  // past the last bin the pieces hold whatever the scratch held before: such
  // values are neither stored nor asked whether they are finite
  const int nb = (int)(nbins - bin < 4 ? nbins - bin : 4);
  auto slot_of = [&](int g) { return (long long)(g + t) * TB + (bin - (long long)t * TB); };
  uint4 pcv[LOADS];
  float4 psv[LOADS], pev[LOADS];
  auto load = [&](int u, int g) {
    pcv[u] = *reinterpret_cast<const uint4*>(pc + slot_of(g));
    if (WEIGHTED) {
      psv[u] = *reinterpret_cast<const float4*>(ps + slot_of(g));
      pev[u] = *reinterpret_cast<const float4*>(pe + slot_of(g));
    }
  };
  auto add = [&](int u) {
    cn[0] += pcv[u].x; cn[1] += pcv[u].y; cn[2] += pcv[u].z; cn[3] += pcv[u].w;
    if (WEIGHTED) {
      ws[0].add(psv[u].x, pev[u].x);
      ws[1].add(psv[u].y, pev[u].y);
      ws[2].add(psv[u].z, pev[u].z);
      ws[3].add(psv[u].w, pev[u].w);
    }
  };
  // (an empty range stored no piece)
  auto empty = [&](int g) { return R < G && range_start(R, g, G) == range_start(R, g + 1, G); };
  int g = s_first + grp;
  if (R >= G)
    for (; g + (LOADS - 1) * CG <= s_last; g += LOADS * CG) {   // LOADS pieces' loads in flight
#pragma unroll
      for (int u = 0; u < LOADS; ++u) load(u, g + u * CG);
#pragma unroll
      for (int u = 0; u < LOADS; ++u) add(u);
    }
  for (; g <= s_last; g += CG)
    if (!empty(g)) { load(0, g); add(0); }
  bool finite = true;
#pragma unroll
  for (int k = 0; k < 4; ++k) finite &= ws[k].finite() | (k >= nb);
  if (CG > 1) {
    if (!finite) s_bad = 1;
    if (grp > 0) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        scn[grp - 1][q][k] = cn[k];
        if (WEIGHTED) sw[grp - 1][q][k] = ws[k];
      }
    }
    __syncthreads();
    if (grp > 0) return;
#pragma unroll
    for (int u = 0; u < CG - 1; ++u)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        cn[k] += scn[u][q][k];
        if (WEIGHTED) ws[k].add(sw[u][q][k]);
      }
#pragma unroll
    for (int k = 0; k < 4; ++k) finite &= ws[k].finite() | (k >= nb);
    if (s_bad) finite = false;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k >= nb) break;
    counts[bin + k] += cn[k];
    if (WEIGHTED) {
      const float w0 = wsum[bin + k];
      double d = wacc[bin + k];
      if (finite && d == 0.0) {   // the value that is there is one more term
        Sum3 all = ws[k];
        all.add(w0, 0.f);
        if (all.finite()) {
          wsum[bin + k] = all.get();
          continue;
        }
      }
      double p = ((double)ws[k].hi + (double)ws[k].mid) + (double)ws[k].lo;
      if (!finite) {   // sums beyond float32: the pieces again in float64
        p = 0.0;
        for (int g = s_first; g <= s_last; ++g)
          if (!empty(g)) p += (double)ps[slot_of(g) + k] + (double)pe[slot_of(g) + k];
      }
      wsum[bin + k] = __double2float_rn((double)w0 + (d + p));
    }
  }
}

}  // namespace

namespace nca {
// NCA_OK or the error a histogram kernel recorded since the last read (cleared)
int hist_read_status(cudaStream_t s) {
  int v = 0, zero = 0;
  check_cuda(cudaMemcpyFromSymbolAsync(&v, g_hist_status, sizeof(int), 0, cudaMemcpyDeviceToHost, s), "status read");
  check_cuda(cudaMemcpyToSymbolAsync(g_hist_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, s), "status clear");
  check_cuda(cudaStreamSynchronize(s), "status sync");
  return v;
}

// address of the status word on the current device
static int* hist_status_word() {
  static std::mutex mu;
  static int* addr[64] = {nullptr};
  const int dev = current_device();
  if (dev < 0 || dev >= 64) fail(NCA_ERR_LIMIT, "device %d", dev);
  std::lock_guard<std::mutex> lk(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    check_cuda(cudaGetSymbolAddress(&p, g_hist_status), "status word address");
    addr[dev] = static_cast<int*>(p);
  }
  return addr[dev];
}
}  // namespace nca

extern "C" int32_t nca_hist2d(const float* x, const float* y, const float* w, int64_t n, int32_t nbx, int32_t nby,
                              double x_lo, double x_hi, double y_lo, double y_hi, uint64_t* counts, float* wsum,
                              void* stream) {
  return nca::guarded([&] {
    using namespace nca;
    if (n < 0) fail(NCA_ERR_INVALID, "negative point count");
    if (nbx <= 0 || nby <= 0 || (int64_t)nbx * nby > (1ll << 30)) fail(NCA_ERR_SHAPE, "bin grid %d x %d out of range", nbx, nby);
    if (!(x_hi > x_lo) || !(y_hi > y_lo)) fail(NCA_ERR_INVALID, "empty bin range");
    if (!counts) fail(NCA_ERR_INVALID, "null counts");
    if (n > 0 && (!x || !y)) fail(NCA_ERR_INVALID, "null coordinates");
    if ((w == nullptr) != (wsum == nullptr)) fail(NCA_ERR_INVALID, "weights and wsum go together");
    if (n == 0) return;
    Bins B;
    B.xl = (float)x_lo;
    B.yl = (float)y_lo;
    B.sx = (float)((double)nbx / (x_hi - x_lo));
    B.sy = (float)((double)nby / (y_hi - y_lo));
    B.fnx = (float)nbx;
    B.fny = (float)nby;
    B.nbx = nbx;
    B.nby = nby;
    cudaStream_t s = (cudaStream_t)stream;
    const int dev = current_device();
    const int sms = sm_count(dev);
    const long long nbins = (long long)nbx * nby;
    const long long ntiles = (nbins + TB - 1) / TB;
    const bool weighted = w != nullptr;
    unsigned long long* cnt = (unsigned long long*)counts;
    // the bulk copies of the partitioned path need 16-byte aligned point arrays
    const bool aligned = ((uintptr_t)x % 16 == 0) && ((uintptr_t)y % 16 == 0) && (!weighted || (uintptr_t)w % 16 == 0);
    // NCA_HIST_PATH=direct forces the direct path (tests and measurements)
    const char* hp = getenv("NCA_HIST_PATH");
    const std::string path = hp ? hp : "";
    if (ntiles > MAX_TILES || n < (1 << 20) || !aligned || path == "direct") {
      StreamScratch acc(weighted ? (size_t)nbins * sizeof(double) : 0, s);
      double* wacc = (double*)acc.ptr;
      if (weighted) check_cuda(cudaMemsetAsync(wacc, 0, (size_t)nbins * sizeof(double), s), "memset weights");
      const long long grid = std::min<long long>((n + THREADS - 1) / THREADS, (long long)sms * 8);
      if (weighted) hist2d_direct_kernel<true><<<(unsigned)grid, THREADS, 0, s>>>(x, y, w, n, B, cnt, wacc);
      else hist2d_direct_kernel<false><<<(unsigned)grid, THREADS, 0, s>>>(x, y, nullptr, n, B, cnt, nullptr);
      check_cuda(cudaGetLastError(), "hist2d launch");
      count_launch();
      if (weighted) {
        wsum_finish_kernel<<<(unsigned)std::min<long long>((nbins + THREADS - 1) / THREADS, (long long)sms * 8),
                             THREADS, 0, s>>>(wacc, wsum, nbins);
        check_cuda(cudaGetLastError(), "wsum finish launch");
        count_launch();
      }
      return;
    }
    // partitioned path, at most 2^30 points per pass so that record indices
    // fit in 31 bits; longer inputs add up pass by pass
    auto pass = [&](const float* x, const float* y, const float* w, long long n) {
      // persistent accumulate grid: as many CTAs as fit with the tile in shared memory
      const size_t smem = weighted ? (size_t)TB * 12 : (size_t)TB * 4;
      const void* acc_fn = weighted ? (const void*)tile_accumulate_kernel<true> : (const void*)tile_accumulate_kernel<false>;
      check_cuda(cudaFuncSetAttribute(acc_fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "smem attribute");
      int per_sm = 0;
      check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, acc_fn, ACC_THREADS, smem), "occupancy");
      if (per_sm < 1) per_sm = 1;
      // Unweighted, a CTA's records should outnumber the bins it clears and stores
      // (2^20 points into 100 x 100 bins 38 us, 44 with every CTA). Weighted points
      // that crowd into few bins are bound by the chains of adds to one address, so
      // every CTA takes a share of them (2^20 points in one of 128 x 128 bins 241
      // us, 485 with 65 CTAs; spread evenly 54 either way).
      const int G = (int)(weighted ? (long long)sms * per_sm
                                   : std::max<long long>(1, std::min<long long>((long long)sms * per_sm, n / std::min<long long>(TB, nbins) + 1)));
      const long long nslots = (long long)(G + ntiles) * TB;
      const size_t bytes = 4 * 256 + Buckets::bytes(n, ntiles, weighted) + (size_t)nslots * (weighted ? 12 : 4);
      StreamScratch scratch(bytes, s);
      StreamScratch acc(weighted ? (size_t)nbins * sizeof(double) : 0, s);
      double* wacc = (double*)acc.ptr;
      if (weighted) check_cuda(cudaMemsetAsync(wacc, 0, (size_t)nbins * sizeof(double), s), "memset weights");
      char* p = (char*)(((uintptr_t)scratch.ptr + 255) & ~(uintptr_t)255);
      Buckets bk;
      bk.take(p, n, ntiles, weighted);
      unsigned* pc = carve<unsigned>(p, nslots);
      float* ps = weighted ? carve<float>(p, nslots) : nullptr;
      float* pe = weighted ? carve<float>(p, nslots) : nullptr;
      int* status = hist_status_word();
      if (weighted) partition(Points<true>{x, y, w, B, cnt, wacc}, n, (int)ntiles, bk, G, status, sms, s);
      else partition(Points<false>{x, y, nullptr, B, cnt, nullptr}, n, (int)ntiles, bk, G, status, sms, s);
      const float* rw = (const float*)bk.rec_val;
      if (weighted)
        tile_accumulate_kernel<true><<<G, ACC_THREADS, smem, s>>>((int)ntiles, bk.off, bk.PV, bk.rec_bin, rw, pc, ps, pe,
                                                                  nbins);
      else
        tile_accumulate_kernel<false><<<G, ACC_THREADS, smem, s>>>((int)ntiles, bk.off, bk.PV, bk.rec_bin, nullptr, pc, nullptr,
                                                                   nullptr, nbins);
      auto combine = [&](auto kernel, int cg) {
        const long long per = 4 * THREADS / cg;
        kernel<<<(unsigned)((nbins + per - 1) / per), THREADS, 0, s>>>(nbins, G, bk.PV, pc, ps, pe, wacc, cnt, wsum, (int)ntiles,
                                                                       bk.ctas);
      };
      if (G >= 8 * ntiles) {
        if (weighted) combine(tile_combine_kernel<true, 8>, 8);
        else combine(tile_combine_kernel<false, 8>, 8);
      } else {
        if (weighted) combine(tile_combine_kernel<true, 1>, 1);
        else combine(tile_combine_kernel<false, 1>, 1);
      }
      check_cuda(cudaGetLastError(), "hist2d launches");
      count_launch(6);
    };
    for (long long s0 = 0; s0 < n; s0 += (1ll << 30)) {
      const long long len = std::min<long long>(n - s0, 1ll << 30);
      pass(x + s0, y + s0, weighted ? w + s0 : nullptr, len);
    }
  });
}
