// Partition passes for a bin grid that fits neither in shared memory nor in
// the L2 atomic rate (the 2-D histogram, hist.cu):
//   1. sample: one block of 1024 elements in 32 estimates how many land in
//      each tile of TB consecutive bins; a tile's bucket gets 25 % slack;
//   2. scatter: every CTA takes a chunk of elements, orders their records by
//      tile in shared memory and appends each tile's run to its bucket with
//      coalesced stores (one global atomic per tile and chunk reserves the
//      space); records past their bucket's capacity are added directly with
//      global atomics;
//   3. the caller accumulates record ranges tile by tile in shared memory and
//      combines the pieces.
// The points as their source (all arrays are 4-byte elements):
//   VAL          records carry a weight
//   NA           arrays read per element: x, y and the weight
//   array(k)     base of array k
//   bin(a, b)    bin of the words a of x and b of y, or NO_BIN
//   direct(bin, word)  adds a record with global atomics
#pragma once
#include <cstdint>

#include "common.hpp"
#include "mbar.cuh"

namespace nca_tiles {

constexpr int TB_LOG2 = 14;
constexpr int TB = 1 << TB_LOG2;        // bins per tile (local index fits in uint16)
constexpr int MAX_TILES = 256;          // 4 Mi bins
constexpr int SAMPLE = 32;              // 1 block of 1024 elements in SAMPLE is counted in pass 1
constexpr int SCAN_THREADS = 256;       // one-block scans over the tiles
constexpr int SLACK = 2048;             // records of slack per bucket
constexpr int FPAD = 16;                // fill counters 128 bytes apart (uint64)
constexpr int EPAD = 32;                // estimate counters 128 bytes apart (uint32)
static_assert(MAX_TILES == SCAN_THREADS, "one tile per thread of a scan");
constexpr unsigned NO_BIN = 0xffffffffu;
constexpr unsigned long long kWaitNs = 2000000000ull;   // bound of every mbarrier wait

// The scatter pass: threads per CTA and elements per chunk (8 a thread, two
// 16-byte words of each array).
constexpr int ST = 512, CHUNK = 8 * ST;

// Exclusive prefix sums of the values v(t) of n <= SCAN_THREADS tiles by one
// block: out[t] for t < n and out[n] = total.
template <class F>
__device__ __forceinline__ void block_scan(int n, F v, long long* out) {
  __shared__ long long sc[SCAN_THREADS];
  const int t = threadIdx.x;
  const long long a = t < n ? v(t) : 0;
  sc[t] = a;
  __syncthreads();
  for (int d = 1; d < SCAN_THREADS; d <<= 1) {
    const long long u = t >= d ? sc[t - d] : 0;
    __syncthreads();
    sc[t] += u;
    __syncthreads();
  }
  if (t < n) out[t] = sc[t] - a;
  if (t == SCAN_THREADS - 1) out[n] = sc[t];
}

// ---- pass 1: sampled tile counts ----------------------------------------------------
template <class Src>
__global__ void __launch_bounds__(256) tile_sample_kernel(Src src, long long n, int ntiles, unsigned* __restrict__ est) {
  __shared__ unsigned cnt[MAX_TILES];
  for (int t = threadIdx.x; t < ntiles; t += 256) cnt[t] = 0;
  __syncthreads();
  // the sample: every SAMPLE-th block of 1024 consecutive elements, a CTA at a time
  const long long nblk = (n + 1023) / 1024, ns = (nblk + SAMPLE - 1) / SAMPLE;
  for (long long s = blockIdx.x; s < ns; s += gridDim.x) {
    unsigned a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long i = s * SAMPLE * 1024 + k * 256 + threadIdx.x;
      const long long j = i < n ? i : n - 1;
      a[k] = __ldg(src.array(0) + j);
      b[k] = __ldg(src.array(1) + j);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned bin = src.bin(a[k], b[k]);
      if (bin != NO_BIN && s * SAMPLE * 1024 + k * 256 + threadIdx.x < n) atomicAdd(&cnt[bin >> TB_LOG2], 1u);
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < ntiles; t += 256)
    if (cnt[t]) atomicAdd(est + (long long)t * EPAD, cnt[t]);
}

__device__ __forceinline__ long long bucket_cap(const unsigned* __restrict__ est, int t) {
  const long long e = est[(long long)t * EPAD];
  return ((e * (SAMPLE * 5 / 4) + 7) & ~7ll) + SLACK;
}

// capacity and offset of every bucket; capacities are multiples of 8 records
// so every bucket starts 16-byte aligned
static __global__ void __launch_bounds__(SCAN_THREADS)
tile_plan_kernel(const unsigned* __restrict__ est, int ntiles, long long* __restrict__ off, long long* __restrict__ cap,
                 unsigned long long* __restrict__ fill) {
  block_scan(ntiles, [&](int t) { return bucket_cap(est, t); }, off);
  if ((int)threadIdx.x < ntiles) {
    cap[threadIdx.x] = bucket_cap(est, threadIdx.x);
    fill[(long long)threadIdx.x * FPAD] = 0;
  }
}

// CTA g of G takes records [R g / G, R (g + 1) / G) of the concatenated
// buckets; its piece of tile t is partial slot g + t, which is unique because
// both g and t grow along the concatenation.
__device__ __forceinline__ long long range_start(long long R, int g, int G) { return R * g / G; }

// the first and last CTA whose ranges meet [lo, hi) (hi > lo)
__device__ __forceinline__ void range_ctas(long long R, int G, long long lo, long long hi, int& first, int& last) {
  int g = (int)(lo * G / R);
  while (g > 0 && range_start(R, g, G) > lo) --g;
  while (g + 1 < G && range_start(R, g + 1, G) <= lo) ++g;
  first = g;
  g = (int)((hi - 1) * G / R);
  while (g + 1 < G && range_start(R, g + 1, G) <= hi - 1) ++g;
  last = g;
}

// stored records per bucket, their exclusive prefix sum PV (PV[ntiles] = total)
// and the first and last accumulating CTA of each tile (last < first: none)
static __global__ void __launch_bounds__(SCAN_THREADS)
tile_prefix_kernel(int ntiles, const long long* __restrict__ cap, const unsigned long long* __restrict__ fill,
                   long long* __restrict__ PV, int G, int2* __restrict__ ctas) {
  __shared__ long long sp[SCAN_THREADS + 1];
  block_scan(ntiles, [&](int t) {
    const long long f = (long long)fill[(long long)t * FPAD];
    return f < cap[t] ? f : cap[t];
  }, sp);
  __syncthreads();
  const int t = threadIdx.x;
  if (t == 0) PV[ntiles] = sp[ntiles];
  if (t >= ntiles) return;
  PV[t] = sp[t];
  int f = 0, l = -1;
  if (sp[t + 1] > sp[t]) range_ctas(sp[ntiles], G, sp[t], sp[t + 1], f, l);
  ctas[t] = make_int2(f, l);
}

// ---- pass 2: scatter elements into buckets ------------------------------------------
// A persistent grid walks the chunks. Bulk copies fetch a chunk's arrays into
// shared memory; once every thread has its 8 elements in registers the buffer
// is free, and the next chunk's copies run under this one. Tile counts are
// shared-memory adds, scanned by the warps that have tiles; every record then
// takes its staged position from its tile's running position (a shared-memory
// add that returns it) and consecutive threads write consecutive records.
// Elements without a bin count as one more tile behind the others, so nothing
// branches on them. Waits are bounded (2 s of %globaltimer): on a timeout the
// CTA records NCA_ERR_TIMEOUT in *status, waits for its copy in flight and
// stops. Bound: shared memory (72 % of its data pipe) and the four barriers of a
// chunk. 2^26 weighted points into 64 tiles 300 -> 237 us (0.75 of the measured
// copy rate) against a double buffer, 2048-point chunks of 256 threads, 4-byte
// shared loads, ranks kept in registers and a second scan; 16-byte global loads
// without the bulk copies at 3 CTAs per SM: 259.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

template <class Src>
__host__ __device__ constexpr int scatter_smem() { return Src::NA * CHUNK * 4 + CHUNK * (Src::VAL ? 8 : 4) + 16; }

template <class Src>
__global__ void __launch_bounds__(ST, Src::VAL ? 2 : 3)
tile_scatter_kernel(Src src, long long n, int ntiles, const long long* __restrict__ off, const long long* __restrict__ cap,
                    unsigned long long* __restrict__ fill, unsigned short* __restrict__ rec_bin,
                    unsigned* __restrict__ rec_val, int* __restrict__ status) {
  constexpr int NA = Src::NA;
  constexpr uint32_t ABYTES = CHUNK * 4;
  extern __shared__ __align__(128) unsigned char sm[];
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
  const uint4* buf = reinterpret_cast<const uint4*>(sm);              // [NA][CHUNK / 4]
  uint2* stage2 = reinterpret_cast<uint2*>(sm + NA * ABYTES);         // (bin, value) in tile order
  unsigned* stage1 = reinterpret_cast<unsigned*>(sm + NA * ABYTES);   // bins only
  const uint32_t bar = sbase + scatter_smem<Src>() - 16;
  __shared__ unsigned cnt[MAX_TILES + 32];
  __shared__ unsigned pos[MAX_TILES + 32];  // next staged position of each tile
  __shared__ uint2 tinfo[MAX_TILES];        // (record index - staged position, end of the stored part)
  __shared__ unsigned wpre[MAX_TILES / 32 + 1];
  __shared__ unsigned s_total;
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const unsigned none = (unsigned)ntiles << TB_LOG2;    // the bin of an element without one
  const long long nfull = n / CHUNK, nchunks = (n + CHUNK - 1) / CHUNK;
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < MAX_TILES + 32) cnt[tid] = 0;
  __syncthreads();
  auto issue = [&](long long ch) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(NA * ABYTES) : "memory");
#pragma unroll
    for (int k = 0; k < NA; ++k) bulk_load(sbase + k * ABYTES, src.array(k) + ch * CHUNK, ABYTES, bar);
  };
  long long ch = blockIdx.x;
  if (tid == 0 && ch < nfull) issue(ch);
  uint32_t phase = 0;
  bool failed = false;
  for (; ch < nchunks; ch += gridDim.x, phase ^= 1u) {
    unsigned bins[8], val[8];
    const bool full = ch < nfull;
    const bool ok = !full || nca_dev::mbar_wait(bar, phase, kWaitNs);
    if (full && ok) {
      uint4 a[2], b[2], v[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        a[h] = buf[h * ST + tid];
        b[h] = buf[CHUNK / 4 + h * ST + tid];
        if (Src::VAL) v[h] = buf[2 * (CHUNK / 4) + h * ST + tid];
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        bins[4 * h] = src.bin(a[h].x, b[h].x);
        bins[4 * h + 1] = src.bin(a[h].y, b[h].y);
        bins[4 * h + 2] = src.bin(a[h].z, b[h].z);
        bins[4 * h + 3] = src.bin(a[h].w, b[h].w);
        if (Src::VAL) {
          val[4 * h] = v[h].x;
          val[4 * h + 1] = v[h].y;
          val[4 * h + 2] = v[h].z;
          val[4 * h + 3] = v[h].w;
        }
      }
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const long long i = ch * CHUNK + k * ST + tid;
        bins[k] = NO_BIN;
        val[k] = 0;
        if (!full && i < n) {
          bins[k] = src.bin(__ldcs(src.array(0) + i), __ldcs(src.array(1) + i));
          if (Src::VAL) val[k] = __ldcs(src.array(2) + i);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      bins[k] = min(bins[k], none);
      atomicAdd(&cnt[bins[k] >> TB_LOG2], 1u);
    }
    if (__syncthreads_or(ok ? 0 : 1)) { failed = true; break; }
    // the chunk is in registers: fetch the next one
    if (tid == 0 && ch + gridDim.x < nfull) issue(ch + gridDim.x);
    // exclusive scan of the tile counts by the warps that have tiles
    unsigned v0 = 0, v = 0;
    if (wp * 32 <= ntiles) {
      v0 = v = cnt[tid];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += u;
      }
      if (lane == 31) wpre[wp] = v;
    }
    __syncthreads();
    unsigned lo = 0;
    unsigned long long p = 0;
    if (tid <= ntiles) {
      lo = v - v0;
      for (int u = 0; u < wp; ++u) lo += wpre[u];
      pos[tid] = lo;
      cnt[tid] = 0;
      if (tid == ntiles) s_total = lo;
      // the tile's run in its bucket; where it lies is needed only after the staging
      else if (v0) p = atomicAdd(fill + (long long)tid * FPAD, (unsigned long long)v0);
    }
    __syncthreads();
    // stage the records in tile order
    unsigned j[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) j[k] = atomicAdd(&pos[bins[k] >> TB_LOG2], 1u);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (Src::VAL) stage2[j[k]] = make_uint2(bins[k], val[k]);
      else stage1[j[k]] = bins[k];
    }
    if (tid < ntiles && v0) {
      // positions [p, p + v0) are this CTA's; the part below the capacity is
      // always written, so every position below min(fill, cap) holds a record
      const long long room = cap[tid] - (long long)p;
      const unsigned avail = room <= 0 ? 0u : (room >= (long long)v0 ? v0 : (unsigned)room);
      tinfo[tid] = make_uint2((unsigned)(off[tid] + (long long)p) - lo, lo + avail);
    }
    __syncthreads();
    // consecutive threads write consecutive records of a tile's run
    const unsigned total = s_total;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const unsigned q = tid + k * ST;
      if (q >= total) break;
      const uint2 r = Src::VAL ? stage2[q] : make_uint2(stage1[q], 0u);
      const uint2 ti = tinfo[r.x >> TB_LOG2];
      if (q < ti.y) {
        rec_bin[ti.x + q] = (unsigned short)(r.x & (TB - 1));
        if (Src::VAL) rec_val[ti.x + q] = r.y;
      } else {
        src.direct(r.x, r.y);
      }
    }
  }
  if (failed && tid == 0) {
    atomicExch(status, 7 /* NCA_ERR_TIMEOUT */);
    nca_dev::mbar_wait(bar, phase, kWaitNs / 2);   // the copy in flight
  }
}

template <typename T>
T* carve(char*& p, long long count) {
  T* r = reinterpret_cast<T*>(p);
  p += ((size_t)count * sizeof(T) + 255) & ~(size_t)255;
  return r;
}

// Scratch of the partition passes of n elements into ntiles tiles: the sample
// has at most nsamp elements, so the capacities add up to at most 1.25 *
// SAMPLE * nsamp + (SLACK + 8) per bucket.
inline long long max_records(long long n, long long ntiles) {
  const long long nsamp = (((n + 1023) / 1024 + SAMPLE - 1) / SAMPLE) * 1024;
  return (long long)(SAMPLE * 5 / 4) * nsamp + (long long)(SLACK + 8) * ntiles;
}

struct Buckets {
  long long *off, *cap, *PV;
  unsigned long long* fill;
  unsigned* est;
  unsigned* rec_val;
  unsigned short* rec_bin;
  int2* ctas;
  static size_t bytes(long long n, long long ntiles, bool val) {
    return 9 * 256 + (size_t)(ntiles + 1) * 8 * 4 + (size_t)ntiles * FPAD * 8 + (size_t)ntiles * EPAD * 4 +
           (size_t)max_records(n, ntiles) * (val ? 6 : 2);
  }
  void take(char*& p, long long n, long long ntiles, bool val) {
    off = carve<long long>(p, ntiles + 1);
    cap = carve<long long>(p, ntiles + 1);
    PV = carve<long long>(p, ntiles + 1);
    ctas = carve<int2>(p, ntiles);
    fill = carve<unsigned long long>(p, ntiles * FPAD);
    est = carve<unsigned>(p, ntiles * EPAD);
    rec_val = val ? carve<unsigned>(p, max_records(n, ntiles)) : nullptr;
    rec_bin = carve<unsigned short>(p, max_records(n, ntiles));
  }
};

// passes 1 and 2 and the prefix of the stored records for G accumulating CTAs (4 launches)
template <class Src>
void partition(const Src& src, long long n, int ntiles, const Buckets& b, int G, int* status, int sms, cudaStream_t s) {
  using namespace nca;
  check_cuda(cudaMemsetAsync(b.est, 0, (size_t)ntiles * EPAD * 4, s), "memset estimates");
  const long long sblk = ((n + 1023) / 1024 + SAMPLE - 1) / SAMPLE;
  tile_sample_kernel<Src><<<(unsigned)(sblk < sms * 8 ? sblk : sms * 8), 256, 0, s>>>(src, n, ntiles, b.est);
  tile_plan_kernel<<<1, SCAN_THREADS, 0, s>>>(b.est, ntiles, b.off, b.cap, b.fill);
  constexpr int smem = scatter_smem<Src>();
  check_cuda(cudaFuncSetAttribute((const void*)tile_scatter_kernel<Src>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
             "smem attribute");
  int per_sm = 0;
  check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)tile_scatter_kernel<Src>, ST, smem), "occupancy");
  const long long chunks = (n + CHUNK - 1) / CHUNK, grid = (long long)sms * (per_sm < 1 ? 1 : per_sm);
  tile_scatter_kernel<Src><<<(unsigned)(chunks < grid ? chunks : grid), ST, smem, s>>>(src, n, ntiles, b.off, b.cap, b.fill,
                                                                                       b.rec_bin, b.rec_val, status);
  tile_prefix_kernel<<<1, SCAN_THREADS, 0, s>>>(ntiles, b.cap, b.fill, b.PV, G, b.ctas);
}

}  // namespace nca_tiles
