// 3-D stencils: dst[c] = src[c] + dt * sum_o w[o] * src[c + o] over the 3x3x3
// neighbourhood with zero halo. Replaces ncarray's device-only Stencil<3>
// (src/lib/ncarray/expression/stencil.hh:58-255), whose NVRTC kernel reloads
// every neighbour from global memory per output (jit/device/rtcompiler.hh:187-385).
//
// GB300 design: each CTA owns a TX x TY column of outputs and marches along z.
// One elected thread streams z-planes (TX + 2*HX) x (TY + 2) x 1 into a ring of
// NST shared-memory stages with TMA (cp.async.bulk.tensor.3d) completing on
// mbarriers; the tensor map's out-of-bounds zero fill supplies the halo. The
// x origin of every box is x0 - HX with HX = 16 / sizeof(T), so it stays on a
// 16-byte boundary. Every thread owns 4 consecutive x outputs of one y row and
// keeps three rolling accumulators: plane p adds its dz = +1 / 0 / -1
// in-plane partial sums to outputs p-1, p, p+1, so each plane is read from
// shared memory once. Waits are bounded (2 s of %globaltimer); on timeout the
// CTA stops, records NCA_ERR_TIMEOUT in a status word, drains its copies in
// flight (bounded too) and returns.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include <mutex>
#include <unordered_map>

#include "common.hpp"
#include "mbar.cuh"
#include "tune.hpp"

namespace {

// tile shapes (x, y) of the TMA kernel; each has (TX / 4) * TY = THREADS threads
constexpr int NST = 4, THREADS = 256;
constexpr int kTiles[3][2] = {{64, 16}, {128, 8}, {32, 32}};
constexpr unsigned long long kWaitNs = 2000000000ull;

static __device__ int g_stencil_status;
__device__ int g_jit_status;   // set by JIT kernels (kind 7) whose bounded waits give up

template <class T>
struct Weights {
  T w[27];
  T dt;
};

template <class T> __host__ __device__ constexpr int halo_x() { return 16 / (int)sizeof(T); }
template <class T, int TX> __host__ __device__ constexpr int box_w() { return TX + 2 * halo_x<T>(); }
template <class T, int TX, int TY> __host__ __device__ constexpr int stage_bytes() {
  return ((box_w<T, TX>() * (TY + 2) * (int)sizeof(T)) + 127) / 128 * 128;
}


using nca_dev::mbar_wait;

template <class T, int TX, int TY>
__device__ __forceinline__ void issue_plane(const CUtensorMap* tmap, uint32_t dst, uint32_t bar, int x, int y, int z) {
  constexpr uint32_t bytes = (uint32_t)(box_w<T, TX>() * (TY + 2) * sizeof(T));
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(reinterpret_cast<unsigned long long>(tmap)), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

// 6 consecutive row values starting at column c0 - 1 (c0 is 16-byte aligned)
template <class T>
__device__ __forceinline__ void load_row(const T* row, int c0, T* v) {
  v[0] = row[c0 - 1];
  if constexpr (sizeof(T) == 4) {
    const float4 m = *reinterpret_cast<const float4*>(row + c0);
    v[1] = m.x; v[2] = m.y; v[3] = m.z; v[4] = m.w;
  } else {
    const double2 m0 = *reinterpret_cast<const double2*>(row + c0);
    const double2 m1 = *reinterpret_cast<const double2*>(row + c0 + 2);
    v[1] = m0.x; v[2] = m0.y; v[3] = m1.x; v[4] = m1.y;
  }
  v[5] = row[c0 + 4];
}

template <class T>
__device__ __forceinline__ T fmaT(T a, T b, T c) {
  if constexpr (sizeof(T) == 4) return __fmaf_rn(a, b, c); else return __fma_rn(a, b, c);
}

// MODE 0: any 27 weights; 1: 7-point star (weights of offsets with two or
// three non-zero components are zero); 2: isotropic 27-point (the weight of an
// offset depends only on how many of its components are non-zero: w[13] for
// none, w[12] for one, w[9] for two, w[0] for three), evaluated per plane from
// the in-plane centre, face and corner sums (12 instead of 27 FMAs a point).
template <class T, int MODE, int TX, int TY>
__global__ void __launch_bounds__(THREADS)
stencil_tma_kernel(const __grid_constant__ CUtensorMap tmap, T* __restrict__ out, int nx, int ny, int nz,
                   int zt, const __grid_constant__ Weights<T> W) {
  extern __shared__ __align__(128) unsigned char smem[];
  static_assert((TX / 4) * TY == THREADS, "a tile has one thread per 4 outputs");
  constexpr int BW = box_w<T, TX>(), HX = halo_x<T>(), SB = stage_bytes<T, TX, TY>();
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + NST * SB);
  const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, z0 = blockIdx.z * zt;
  const int zend = min(z0 + zt, nz);
  const int nplanes = zend - z0 + 2;  // planes z0-1 .. zend
  const int ty = threadIdx.x / (TX / 4), tx4 = (threadIdx.x % (TX / 4)) * 4;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const uint32_t bbase = (uint32_t)__cvta_generic_to_shared(bars);
  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; ++s)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bbase + 8 * s) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  int issued = 0;
  if (threadIdx.x == 0) {
    for (; issued < NST && issued < nplanes; ++issued)
      issue_plane<T, TX, TY>(&tmap, sbase + issued * SB, bbase + 8 * issued, x0 - HX, y0 - 1, z0 - 1 + issued);
  }
  // acc_a: output p-1 (missing only plane p's dz=+1 part), acc_b: output p
  // (has plane p-1's dz=-1 part), cen: centre value of output p-1
  T acc_a[4], acc_b[4], cen[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) { acc_a[j] = acc_b[j] = cen[j] = T(0); }
  const int x = x0 + tx4, y = y0 + ty;
  const bool active = x < nx && y < ny;
  bool timed_out = false;
  int i = 0;
  for (; i < nplanes; ++i) {
    const int st = i % NST;
    const bool ok = mbar_wait(bbase + 8 * st, (uint32_t)((i / NST) & 1), kWaitNs);
    if (ok) {
      const T* plane = reinterpret_cast<const T*>(smem + st * SB);
      const int c0 = HX + tx4;
      T v[3][6];
      load_row(plane + (ty + 1) * BW, c0, v[1]);
      if constexpr (MODE == 1) {
#pragma unroll
        for (int r = 0; r < 3; r += 2) {
          const T* row = plane + (ty + r) * BW;
          if constexpr (sizeof(T) == 4) {
            const float4 m = *reinterpret_cast<const float4*>(row + c0);
            v[r][1] = m.x; v[r][2] = m.y; v[r][3] = m.z; v[r][4] = m.w;
          } else {
            const double2 m0 = *reinterpret_cast<const double2*>(row + c0);
            const double2 m1 = *reinterpret_cast<const double2*>(row + c0 + 2);
            v[r][1] = m0.x; v[r][2] = m0.y; v[r][3] = m1.x; v[r][4] = m1.y;
          }
        }
      } else {
        load_row(plane + ty * BW, c0, v[0]);
        load_row(plane + (ty + 2) * BW, c0, v[2]);
      }
      // partial sums of this plane for dz = -1 (output p+1), 0 (output p), +1 (output p-1)
      T pm[4], p0[4], pp[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if constexpr (MODE == 2) {
          // in-plane centre C, faces F and corners K of output column j
          const T C = v[1][j + 1];
          const T F = ((v[1][j] + v[1][j + 2]) + v[0][j + 1]) + v[2][j + 1];
          const T K = (v[0][j] + v[0][j + 2]) + (v[2][j] + v[2][j + 2]);
          p0[j] = fmaT(W.w[9], K, fmaT(W.w[12], F, W.w[13] * C));
          const T q = fmaT(W.w[0], K, fmaT(W.w[9], F, W.w[12] * C));
          pm[j] = q;
          pp[j] = q;
        } else if constexpr (MODE == 1) {
          pm[j] = pp[j] = T(0);   // the z terms are added below
          T s = W.w[13] * v[1][j + 1];
          s = fmaT(W.w[12], v[1][j], s);
          s = fmaT(W.w[14], v[1][j + 2], s);
          s = fmaT(W.w[10], v[0][j + 1], s);
          p0[j] = fmaT(W.w[16], v[2][j + 1], s);
        } else {
          T s0 = T(0), s1 = T(0), s2 = T(0);
#pragma unroll
          for (int oy = 0; oy < 3; ++oy)
#pragma unroll
            for (int ox = 0; ox < 3; ++ox) {
              const T u = v[oy][j + ox];
              s0 = fmaT(W.w[0 * 9 + oy * 3 + ox], u, s0);
              s1 = fmaT(W.w[1 * 9 + oy * 3 + ox], u, s1);
              s2 = fmaT(W.w[2 * 9 + oy * 3 + ox], u, s2);
            }
          pm[j] = s0; p0[j] = s1; pp[j] = s2;
        }
      }
      const int p = z0 - 1 + i;
      // output p-1 is complete
      if (active && i >= 2) {
        T o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          o[j] = fmaT(W.dt, MODE == 1 ? fmaT(W.w[22], v[1][j + 1], acc_a[j]) : acc_a[j] + pp[j], cen[j]);
        T* dst = out + ((size_t)(p - 1) * ny + y) * nx + x;
        if constexpr (sizeof(T) == 4) {
          *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
          reinterpret_cast<double2*>(dst)[0] = make_double2(o[0], o[1]);
          reinterpret_cast<double2*>(dst)[1] = make_double2(o[2], o[3]);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        // output p: now lacks only plane p+1 (star: plane p-1's part is its centre value)
        acc_a[j] = MODE == 1 ? fmaT(W.w[4], cen[j], p0[j]) : acc_b[j] + p0[j];
        acc_b[j] = pm[j];              // output p+1: plane p's dz=-1 part
        cen[j] = v[1][j + 1];          // centre of output p
      }
    }
    if (__syncthreads_or(ok ? 0 : 1)) { timed_out = true; break; }
    if (threadIdx.x == 0 && issued < nplanes) {
      issue_plane<T, TX, TY>(&tmap, sbase + st * SB, bbase + 8 * st, x0 - HX, y0 - 1, z0 - 1 + issued);
      ++issued;
    }
  }
  if (timed_out && threadIdx.x == 0) {
    atomicExch(&g_stencil_status, (int)NCA_ERR_TIMEOUT);
    for (int k = i; k < issued; ++k) mbar_wait(bbase + 8 * (k % NST), (uint32_t)((k / NST) & 1), kWaitNs / 2);
  }
}

// ---- three Jacobi steps per pass (float32) ------------------------------------------
// nca_stencil3d_iterate moves the grid through HBM once per step, 8 bytes a
// point, and the one-step kernel above already runs at 0.97 of the measured
// copy rate (512^3, 7 points: 163 us a step), so only fewer passes help. This
// kernel advances three steps while a plane of a tile is on the chip:
// a CTA of NW warps owns a tile of 128 x (NW * R) columns, halo included, and
// marches along z. TMA streams the planes into a ring of T3_NST stages; a warp
// holds R whole 128-column rows (lane l the columns 4l..4l+3), so the x
// neighbours come from two shuffles and the y neighbours inside a warp from
// registers; the rows next to a warp's cross shared memory. The three steps of
// an iteration are independent: step k + 1 takes the plane that step k
// completed in the iteration before, so one barrier per plane suffices (the
// exchange is double-buffered by parity). y, z and centre terms are packed
// float32 pairs, x terms (across the pairs) scalars on their halves: 1071 us
// for ten steps of 512^3 against 1327 with scalars only (at 16 x 2 rows: 1118).
// The rolling accumulators add the same terms in the same order as the
// one-step kernel, so the results equal three single steps bit for bit. Values
// outside the grid are zeroed after every step (the zero halo); the tile's
// outer three rows and columns are recomputed by the neighbouring tiles. x
// tiles advance by 120 columns (480 bytes: boxes start on 16-byte boundaries).
// Bound: instruction issue (about 10 a point and step with the recomputed halo
// and the tiles' overhang of 512, 0.55 of the issue slots). Star 14 warps x 3
// rows, isotropic 12 x 2 (register-bound): ten steps of 512^3 float32 1702 ->
// 1071 us (7 points), 1700 -> 1615 us (27); (64, 64, 64) 83 -> 53, 103 -> 48;
// (200, 300, 400) 342 -> 241, 430 -> 351.
constexpr int T3_K = 3, T3_EX = 128, T3_HX = 4;
constexpr int T3_TX = T3_EX - 2 * T3_HX;
constexpr int T3_NST = 4;
constexpr int T3_LAG = 2 * T3_K + 2;   // iterations from a plane's arrival to the output of the plane 5 below it
template <int NW, int R>
struct T3 {   // sizes of a CTA of NW warps
  static constexpr int EY = NW * R, TY = EY - 2 * T3_K;
  static constexpr int STAGE = T3_EX * EY * 4;
  static constexpr int XB = NW * 2 * T3_EX * 4;                        // one exchange buffer
  static constexpr int SMEM = T3_NST * STAGE + 2 * (T3_K - 1) * XB + T3_NST * 8;
};

template <int V> struct IntC { static constexpr int value = V; };
// the step's weights as packed pairs: kernel parameters that the packed
// instructions read from the constant bank instead of registers
struct Pairs {
  float2 dt, z0, z1, c, y0, y1;   // star; isotropic: z0, z1, c, y0 = the weights by distance class 3, 2, 0, 1
  float x0, x1;
};
struct Row4 { float2 a, b; };   // four consecutive columns

__device__ __forceinline__ unsigned long long u2(float2 a) { return *reinterpret_cast<unsigned long long*>(&a); }
__device__ __forceinline__ float2 f2(unsigned long long a) { return *reinterpret_cast<float2*>(&a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(u2(a)), "l"(u2(b)), "l"(u2(c)));
  return f2(d);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(u2(a)), "l"(u2(b)));
  return f2(d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(u2(a)), "l"(u2(b)));
  return f2(d);
}
__device__ __forceinline__ Row4 row4(float4 m) { return Row4{make_float2(m.x, m.y), make_float2(m.z, m.w)}; }
__device__ __forceinline__ Row4 zero4() { return Row4{make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }

// one step's rolling state of a thread's rows: a (the output one plane back,
// lacking the newest plane), b (isotropic form: the older plane's part of the
// current output) and c, the centre values of the plane before
template <int R>
struct Step3 { Row4 a[R], b[R], c[R]; };

// adds a plane (rows r[0..R-1] with the rows above and below) to a step's
// state and returns the completed output rows of the plane before
template <int MODE, int R>
__device__ __forceinline__ void step_plane(Step3<R>& S, const Row4* r, const Row4& top, const Row4& bot,
                                           const Pairs& W, Row4* o) {
  const float2 dt = W.dt;
  if constexpr (MODE == 1) {
    const float2 wz0 = W.z0, wz1 = W.z1, wc = W.c, wy0 = W.y0, wy1 = W.y1;
    const float wx0 = W.x0, wx1 = W.x1;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const Row4 v = r[i];
      const Row4 up = i == 0 ? top : r[i > 0 ? i - 1 : 0], dn = i == R - 1 ? bot : r[i < R - 1 ? i + 1 : i];
      const float lf = __shfl_up_sync(0xffffffffu, v.b.y, 1), rt = __shfl_down_sync(0xffffffffu, v.a.x, 1);
      o[i].a = fma2(dt, fma2(wz1, v.a, S.a[i].a), S.c[i].a);
      o[i].b = fma2(dt, fma2(wz1, v.b, S.a[i].b), S.c[i].b);
      float2 sa = mul2(wc, v.a), sb = mul2(wc, v.b);
      // x neighbours sit across the pairs: scalar FMAs on the halves, no repacking
      sa = make_float2(__fmaf_rn(wx0, lf, sa.x), __fmaf_rn(wx0, v.a.x, sa.y));
      sb = make_float2(__fmaf_rn(wx0, v.a.y, sb.x), __fmaf_rn(wx0, v.b.x, sb.y));
      sa = make_float2(__fmaf_rn(wx1, v.a.y, sa.x), __fmaf_rn(wx1, v.b.x, sa.y));
      sb = make_float2(__fmaf_rn(wx1, v.b.y, sb.x), __fmaf_rn(wx1, rt, sb.y));
      sa = fma2(wy0, up.a, sa);
      sb = fma2(wy0, up.b, sb);
      sa = fma2(wy1, dn.a, sa);
      sb = fma2(wy1, dn.b, sb);
      // the older plane's term: its centre is the value kept for the output
      S.a[i].a = fma2(wz0, S.c[i].a, sa);
      S.a[i].b = fma2(wz0, S.c[i].b, sb);
      S.c[i] = v;
    }
  } else {
    // isotropic: per row the sum of the two x neighbours; F and K as in the one-step kernel
    auto xsum = [](const Row4& v) {
      const float lf = __shfl_up_sync(0xffffffffu, v.b.y, 1), rt = __shfl_down_sync(0xffffffffu, v.a.x, 1);
      return Row4{make_float2(__fadd_rn(lf, v.a.y), __fadd_rn(v.a.x, v.b.x)),
                  make_float2(__fadd_rn(v.a.y, v.b.y), __fadd_rn(v.b.x, rt))};
    };
    const float2 w0 = W.c, w1 = W.y0, w2 = W.z1, w3 = W.z0;
    Row4 xu = xsum(top), xc = xsum(r[0]);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const Row4 v = r[i];
      const Row4 up = i == 0 ? top : r[i > 0 ? i - 1 : 0], dn = i == R - 1 ? bot : r[i < R - 1 ? i + 1 : i];
      const Row4 xd = xsum(dn);
      const float2 Fa = add2(add2(xc.a, up.a), dn.a), Fb = add2(add2(xc.b, up.b), dn.b);
      const float2 Ka = add2(xu.a, xd.a), Kb = add2(xu.b, xd.b);
      const float2 pa = fma2(w2, Ka, fma2(w1, Fa, mul2(w0, v.a))), pb = fma2(w2, Kb, fma2(w1, Fb, mul2(w0, v.b)));
      const float2 qa = fma2(w3, Ka, fma2(w2, Fa, mul2(w1, v.a))), qb = fma2(w3, Kb, fma2(w2, Fb, mul2(w1, v.b)));
      o[i].a = fma2(dt, add2(S.a[i].a, qa), S.c[i].a);
      o[i].b = fma2(dt, add2(S.a[i].b, qb), S.c[i].b);
      S.a[i].a = add2(S.b[i].a, pa);
      S.a[i].b = add2(S.b[i].b, pb);
      S.b[i].a = qa;
      S.b[i].b = qb;
      S.c[i] = v;
      xu = xc;
      xc = xd;
    }
  }
}

template <int MODE, int NW, int R>
__global__ void __launch_bounds__(32 * NW, 1)
stencil_tma3_kernel(const __grid_constant__ CUtensorMap tmap, float* __restrict__ out, int nx, int ny, int nz, int zt,
                    const __grid_constant__ Pairs W) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int EY = T3<NW, R>::EY, STAGE = T3<NW, R>::STAGE, XB = T3<NW, R>::XB;
  __shared__ volatile int failed;   // a bounded wait ran out
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  unsigned char* const xbuf = smem + T3_NST * STAGE;   // [parity][step][warp][2 rows]
  const uint32_t bbase = sbase + T3_NST * STAGE + 2 * (T3_K - 1) * XB;
  const int x0 = blockIdx.x * T3_TX - T3_HX, y0 = blockIdx.y * T3<NW, R>::TY - T3_K, z0 = blockIdx.z * zt;
  const int zend = min(z0 + zt, nz);
  const int nin = zend - z0 + 2 * T3_K;       // planes read: z0-3 .. zend+2
  const int nit = zend - z0 + T3_LAG;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    failed = 0;
    for (int s = 0; s < T3_NST; ++s)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bbase + 8 * s) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int k = threadIdx.x; k < 2 * (T3_K - 1) * XB / 16; k += 32 * NW)
    reinterpret_cast<float4*>(xbuf)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  auto issue = [&](int k) {   // input plane k of the march into its stage
    const uint32_t bar = bbase + 8 * (k % T3_NST);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)STAGE) : "memory");
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(sbase + (k % T3_NST) * STAGE), "l"(reinterpret_cast<unsigned long long>(&tmap)), "r"(x0), "r"(y0),
        "r"(z0 - T3_K + k), "r"(bar) : "memory");
  };
  int issued = 0;
  if (threadIdx.x == 0)
    for (; issued < T3_NST && issued < nin; ++issued) issue(issued);
  Step3<R> S[T3_K];
  Row4 P[T3_K][R];   // the plane each step takes this iteration
#pragma unroll
  for (int k = 0; k < T3_K; ++k)
#pragma unroll
    for (int i = 0; i < R; ++i) S[k].a[i] = S[k].b[i] = S[k].c[i] = P[k][i] = zero4();
  const int gx = x0 + 4 * lane, gy = y0 + warp * R;
  // rows inside the grid (rin) and rows this thread stores (rout)
  const bool xin = gx >= 0 && gx < nx;
  unsigned rin = 0, rout = 0;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = warp * R + i;
    if (xin && gy + i >= 0 && gy + i < ny) rin |= 1u << i;
    if (((rin >> i) & 1u) && lane > 0 && lane < 31 && row >= T3_K && row < EY - T3_K) rout |= 1u << i;
  }
  const bool inside = x0 >= 0 && x0 + T3_EX <= nx && y0 >= 0 && y0 + EY <= ny;   // no masks in x and y
  // the rows above and below this warp's in the exchange buffers (a tile's
  // first and last warp read their own: halo rows whose values are not used)
  const int above = (warp > 0 ? (warp - 1) * 2 + 1 : 0) * 32 + lane;
  const int below = (warp < NW - 1 ? (warp + 1) * 2 : warp * 2) * 32 + lane;
  // one iteration; PAR: its parity. The steps run last to first: a step's old
  // centre rows are dead when the step before it emits its plane, so over two
  // iterations (unrolled below) every row stays in the registers it was
  // computed in.
  auto iterate = [&](int i, auto PAR) {
    constexpr int par = decltype(PAR)::value;
    const int st = i % T3_NST;
    const bool has = i < nin;
    const bool ok = !has || mbar_wait(bbase + 8 * st, (uint32_t)((i / T3_NST) & 1), kWaitNs);
    const float4* xr = reinterpret_cast<const float4*>(xbuf + (par ^ 1) * (T3_K - 1) * XB);
    float4* xw = reinterpret_cast<float4*>(xbuf + par * (T3_K - 1) * XB) + warp * 64 + lane;
    // (after the last input plane the stage holds an older one: finite values that no output uses)
    const float4* plane = reinterpret_cast<const float4*>(smem + st * STAGE) + lane;
    Row4 top[T3_K], bot[T3_K];
    auto read = [&](int k) {   // step k's input rows from shared memory
      if (k > 0) {
        top[k] = row4(xr[(k - 1) * (XB / 16) + above]);
        bot[k] = row4(xr[(k - 1) * (XB / 16) + below]);
        return;
      }
      top[0] = row4(plane[(warp > 0 ? warp * R - 1 : 0) * 32]);
      bot[0] = row4(plane[(warp < NW - 1 ? warp * R + R : warp * R) * 32]);
#pragma unroll
      for (int q = 0; q < R; ++q) P[0][q] = row4(plane[(warp * R + q) * 32]);
    };
    // the isotropic form has the registers to read everything first (a 512^3
    // step 162 us against 172); the star form reads per step (107 against 120)
    if (MODE == 2)
#pragma unroll
      for (int k = T3_K - 1; k >= 0; --k) read(k);
#pragma unroll
    for (int k = T3_K - 1; k >= 0; --k) {
      Row4 o[R];
      if (MODE != 2) read(k);
      step_plane<MODE, R>(S[k], P[k], top[k], bot[k], W, o);
      if (k < T3_K - 1) {
        const int p = z0 - T3_K + i - 1 - 2 * k;   // the plane step k + 1 completed
        if (p < 0 || p >= nz) {
          asm volatile("");   // a branch (CTA-uniform), not a select per value
#pragma unroll
          for (int q = 0; q < R; ++q) o[q] = zero4();
        } else if (!inside) {
          asm volatile("");
#pragma unroll
          for (int q = 0; q < R; ++q)
            if (!((rin >> q) & 1u)) o[q] = zero4();
        }
        xw[k * (XB / 16)] = make_float4(o[0].a.x, o[0].a.y, o[0].b.x, o[0].b.y);
        xw[k * (XB / 16) + 32] = make_float4(o[R - 1].a.x, o[R - 1].a.y, o[R - 1].b.x, o[R - 1].b.y);
#pragma unroll
        for (int q = 0; q < R; ++q) P[k + 1][q] = o[q];
      } else if (i >= T3_LAG && i < nit) {
        float* dst = out + ((size_t)(z0 + i - T3_LAG) * ny + gy) * nx + gx;
#pragma unroll
        for (int q = 0; q < R; ++q)
          if ((rout >> q) & 1u)
            *reinterpret_cast<float4*>(dst + (size_t)q * nx) = make_float4(o[q].a.x, o[q].a.y, o[q].b.x, o[q].b.y);
      }
    }
    // the plane's barrier: its stage is read, the exchanged rows are written
    if (!ok) failed = 1;
    __syncthreads();
    if (threadIdx.x == 0 && ok && issued < nin) { issue(issued); ++issued; }
  };
  int i = 0;
#pragma unroll 1
  for (; i < nit && !failed; i += 2) {   // a wait that ran out ends the march after at most one more plane
    iterate(i, IntC<0>());
    iterate(i + 1, IntC<1>());
  }
  if (failed && threadIdx.x == 0) {
    atomicExch(&g_stencil_status, (int)NCA_ERR_TIMEOUT);
    for (int k = max(0, i - 2); k < issued; ++k) mbar_wait(bbase + 8 * (k % T3_NST), (uint32_t)((k / T3_NST) & 1), kWaitNs / 2);
  }
}

// Any shape: one thread per output, neighbours read through L1/L2.
template <class T>
__global__ void __launch_bounds__(THREADS)
stencil_direct_kernel(const T* __restrict__ src, T* __restrict__ out, int nx, int ny, int nz,
                      const __grid_constant__ Weights<T> W) {
  const long long n = (long long)nx * ny * nz;
  for (long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x; id < n; id += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(id % nx), y = (int)((id / nx) % ny), z = (int)(id / ((long long)nx * ny));
    T pz[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int dz = 0; dz < 3; ++dz) {
      const int zz = z + dz - 1;
      if (zz < 0 || zz >= nz) continue;
#pragma unroll
      for (int oy = 0; oy < 3; ++oy) {
        const int yy = y + oy - 1;
        if (yy < 0 || yy >= ny) continue;
#pragma unroll
        for (int ox = 0; ox < 3; ++ox) {
          const int xx = x + ox - 1;
          if (xx < 0 || xx >= nx) continue;
          pz[dz] = fmaT(W.w[dz * 9 + oy * 3 + ox], __ldg(src + ((long long)zz * ny + yy) * nx + xx), pz[dz]);
        }
      }
    }
    const T acc = (pz[2] + pz[0]) + pz[1];
    out[id] = fmaT(W.dt, acc, src[id]);
  }
}

struct Grid3 {
  int nz, ny, nx, dtype;
  const void* base;
  void* mut;
};

Grid3 check_grid(const nca_view* v, const char* what) {
  using namespace nca;
  if (!v) fail(NCA_ERR_INVALID, "%s: null view", what);
  if (v->ndim != 3) fail(NCA_ERR_SHAPE, "%s: stencil grids are 3-D (got %d dims)", what, v->ndim);
  if (v->dtype != NCA_FLOAT32 && v->dtype != NCA_FLOAT64)
    fail(NCA_ERR_DTYPE, "%s: stencil grids are float32 or float64", what);
  if (v->pointer_axis >= 0) fail(NCA_ERR_UNSUPPORTED, "%s: pointer axes are not supported", what);
  const int64_t isz = dtinfo(v->dtype).size;
  if (v->strides[2] != isz || v->strides[1] != isz * v->shape[2] || v->strides[0] != isz * v->shape[2] * v->shape[1])
    fail(NCA_ERR_UNSUPPORTED, "%s: stencil grids must be C-contiguous", what);
  for (int d = 0; d < 3; ++d)
    if (v->shape[d] <= 0 || v->shape[d] >= (1 << 30)) fail(NCA_ERR_SHAPE, "%s: extent out of range", what);
  int64_t off = v->offsets[0] + v->offsets[1] + v->offsets[2];
  if (!v->data) fail(NCA_ERR_INVALID, "%s: null data", what);
  Grid3 g{(int)v->shape[0], (int)v->shape[1], (int)v->shape[2], v->dtype, (const char*)v->data + off,
          (char*)v->data + off};
  return g;
}

template <class T>
Weights<T> make_weights(const double* w27, double dt) {
  Weights<T> W;
  for (int i = 0; i < 27; ++i) W.w[i] = (T)w27[i];
  W.dt = (T)dt;
  return W;
}

bool star7(const double* w) {
  for (int i = 0; i < 27; ++i) {
    const int dz = i / 9, oy = (i / 3) % 3, ox = i % 3;
    const int nz = (dz != 1) + (oy != 1) + (ox != 1);
    if (nz >= 2 && w[i] != 0.0) return false;
  }
  return true;
}

// the weight of every offset depends only on its number of non-zero components
bool isotropic27(const double* w) {
  const double cls[4] = {w[13], w[12], w[9], w[0]};
  for (int i = 0; i < 27; ++i) {
    const int dz = i / 9, oy = (i / 3) % 3, ox = i % 3;
    const int nz = (dz != 1) + (oy != 1) + (ox != 1);
    if (w[i] != cls[nz]) return false;
  }
  return true;
}

bool tma_ok(const Grid3& g) {
  // row pitch and plane pitch must be multiples of 16 bytes and the x extent a
  // multiple of 4 (each thread stores 4 aligned outputs)
  return g.nx % 4 == 0 && ((uintptr_t)g.base % 16) == 0 && nca::drv().cuTensorMapEncodeTiled != nullptr;
}

// tensor map of a grid with boxes of bx x by x 1 points
template <class T>
void encode_box(CUtensorMap* m, const Grid3& g, int bx, int by) {
  const cuuint64_t dims[3] = {(cuuint64_t)g.nx, (cuuint64_t)g.ny, (cuuint64_t)g.nz};
  const cuuint64_t strides[2] = {(cuuint64_t)g.nx * sizeof(T), (cuuint64_t)g.nx * g.ny * sizeof(T)};
  const cuuint32_t box[3] = {(cuuint32_t)bx, (cuuint32_t)by, 1u};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  nca::check_cu(nca::drv().cuTensorMapEncodeTiled(
                    m, sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3,
                    const_cast<void*>(g.base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE),
                "cuTensorMapEncodeTiled");
}

template <class T, int TX, int TY>
void launch_tma(const Grid3& src, const Grid3& dst, const Weights<T>& W, int mode, int zt, cudaStream_t s) {
  CUtensorMap m;
  encode_box<T>(&m, src, box_w<T, TX>(), TY + 2);
  dim3 grid((src.nx + TX - 1) / TX, (src.ny + TY - 1) / TY, (src.nz + zt - 1) / zt);
  const size_t smem = NST * stage_bytes<T, TX, TY>() + NST * 8;
  if (mode == 1)
    stencil_tma_kernel<T, 1, TX, TY><<<grid, THREADS, smem, s>>>(m, (T*)dst.mut, src.nx, src.ny, src.nz, zt, W);
  else if (mode == 2)
    stencil_tma_kernel<T, 2, TX, TY><<<grid, THREADS, smem, s>>>(m, (T*)dst.mut, src.nx, src.ny, src.nz, zt, W);
  else
    stencil_tma_kernel<T, 0, TX, TY><<<grid, THREADS, smem, s>>>(m, (T*)dst.mut, src.nx, src.ny, src.nz, zt, W);
  nca::check_cuda(cudaGetLastError(), "stencil launch");
  nca::count_launch();
}

template <class T>
void launch_tile(int tile, const Grid3& src, const Grid3& dst, const Weights<T>& W, int mode, int zt, cudaStream_t s) {
  switch (tile) {
    case 1: launch_tma<T, kTiles[1][0], kTiles[1][1]>(src, dst, W, mode, zt, s); break;
    case 2: launch_tma<T, kTiles[2][0], kTiles[2][1]>(src, dst, W, mode, zt, s); break;
    default: launch_tma<T, kTiles[0][0], kTiles[0][1]>(src, dst, W, mode, zt, s); break;
  }
}

// Tile shape and z-march depth: the autotuner's cached choice for this
// (dtype, stencil form, grid size class), else the built-in heuristic; in
// search mode a miss times every (tile, depth) candidate on this call first.
template <class T>
void tma_schedule(const Grid3& src, const Grid3& dst, const Weights<T>& W, int mode, cudaStream_t s, int& tile,
                  int& zt) {
  using namespace nca;
  tile = 0;
  zt = src.nz >= 256 ? 32 : (src.nz >= 64 ? 16 : 8);
  const std::string key = std::string("stencil3d|") + (sizeof(T) == 4 ? "f32" : "f64") + "|" + std::to_string(mode) +
                          "|" + size_class(src.nz) + "x" + size_class(src.ny) + "x" + size_class(src.nx);
  std::vector<int> v;
  if (tune_get(key, v) && v.size() == 2 && v[0] >= 0 && v[0] < 3 && v[1] >= 1) {
    tile = v[0];
    zt = v[1];
    return;
  }
  if (!tune_should_search(s)) return;
  std::vector<std::pair<int, int>> cands;
  for (int t = 0; t < 3; ++t)
    for (int z : {8, 16, 32, 64})
      if (z <= std::max(8, src.nz)) cands.push_back({t, z});
  const int best = tune_pick(s, (int)cands.size(), [&](int i) {
    launch_tile<T>(cands[(size_t)i].first, src, dst, W, mode, cands[(size_t)i].second, s);
  });
  tile = cands[(size_t)best].first;
  zt = cands[(size_t)best].second;
  tune_put(key, {tile, zt});
}

template <class T>
void launch_one(const Grid3& src, const Grid3& dst, const Weights<T>& W, int mode, cudaStream_t s) {
  using namespace nca;
  const int dev = current_device();
  if (tma_ok(src) && tma_ok(dst)) {
    int tile = 0, zt = 8;
    tma_schedule<T>(src, dst, W, mode, s, tile, zt);
    launch_tile<T>(tile, src, dst, W, mode, zt, s);
    return;
  } else {
    const long long n = (long long)src.nx * src.ny * src.nz;
    const long long blocks = std::min<long long>((n + THREADS - 1) / THREADS, (long long)sm_count(dev) * 32);
    stencil_direct_kernel<T><<<(unsigned)blocks, THREADS, 0, s>>>((const T*)src.base, (T*)dst.mut, src.nx, src.ny,
                                                                  src.nz, W);
  }
  check_cuda(cudaGetLastError(), "stencil launch");
  count_launch();
}

// z chunks of a three-step pass: one CTA per SM at a time, and every chunk
// marches T3_LAG + 2 planes more than it stores, so the split with the fewest
// planes end to end. Returns those planes; zt and rounds of resident CTAs.
template <int NW, int R>
int64_t split3(const Grid3& g, int sms, int& zt, int64_t& rounds) {
  const int64_t tiles = (int64_t)((g.nx + T3_TX - 1) / T3_TX) * ((g.ny + T3<NW, R>::TY - 1) / T3<NW, R>::TY);
  int64_t best = -1;
  for (int c = 1; c <= g.nz && c <= 4 * sms; ++c) {
    const int d = (g.nz + c - 1) / c;
    const int64_t r = (tiles * ((g.nz + d - 1) / d) + sms - 1) / sms, cost = r * (d + T3_LAG + 2);
    if (best < 0 || cost < best) { best = cost; zt = d; rounds = r; }
  }
  return best;
}

template <int MODE, int NW, int R>
void launch3_as(const Grid3& src, const Grid3& dst, const Weights<float>& W, cudaStream_t s) {
  using namespace nca;
  CUtensorMap m;
  encode_box<float>(&m, src, T3_EX, T3<NW, R>::EY);
  const int tx = (src.nx + T3_TX - 1) / T3_TX, ty = (src.ny + T3<NW, R>::TY - 1) / T3<NW, R>::TY;
  int zt = src.nz;
  int64_t rounds = 1;
  split3<NW, R>(src, sm_count(current_device()), zt, rounds);
  auto two = [](float v) { return make_float2(v, v); };
  Pairs p{};
  p.dt = two(W.dt);
  p.c = two(W.w[13]);
  if (MODE == 1) {
    p.z0 = two(W.w[4]); p.z1 = two(W.w[22]); p.y0 = two(W.w[10]); p.y1 = two(W.w[16]);
    p.x0 = W.w[12]; p.x1 = W.w[14];
  } else {
    p.y0 = two(W.w[12]); p.z1 = two(W.w[9]); p.z0 = two(W.w[0]);
  }
  auto fn = stencil_tma3_kernel<MODE, NW, R>;
  check_cuda(cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, T3<NW, R>::SMEM), "smem attribute");
  fn<<<dim3(tx, ty, (src.nz + zt - 1) / zt), 32 * NW, T3<NW, R>::SMEM, s>>>(m, (float*)dst.mut, src.nx, src.ny, src.nz, zt, p);
  check_cuda(cudaGetLastError(), "stencil launch");
  count_launch();
}

// Whether a three-step pass is shorter than three single steps: both are
// estimated, in us. A pass takes its planes end to end, 0.93 us each for 7
// points and 0.82 for 27 (1.13 and 0.94 where only one round of CTAs runs, which
// nothing overlaps). A single step takes a start, a CTA's march and what the
// CTAs of an SM issue together, or the bytes if those take longer. What tiles of
// 120 columns and 36 or 18 rows waste on a narrow grid, and the 10 extra planes
// of a chunk on a flat one, decides: three steps against one pass, 7 points / 27,
// (1, 2048, 2048) 43 against 74 / 55 against 129; (4, 2048, 2048) 80, 92 / 103,
// 156; (8, 2048, 2048) 135, 123 / 160, 207; (16, 2048, 2048) 261, 183 / 302, 307;
// (8, 8, 100000) 49, 103 / 68, 89; (29, 437, 340) 31, 23 / 37, 25; (64, 64, 64)
// 25, 14 / 31, 12; (512, 512, 512) 511, 300 / 510, 481. The single step's numbers
// are fitted to 170 grids of 1 to 512 planes, both weights: its estimate is off
// by 5 % on average, and the rule takes the slower form on nine thin grids, by
// 9 % at most ((3, 16, 148) 13.4 against 12.3), costing 0.2 % on average. With
// the march and the issue taken as the longer of the two, without the start, 47
// of the 340 took a form slower by more than 3 %, up to 1.5 times.
bool three_pays(const Grid3& g, int mode, int sms, int tile, int zt1) {
  const bool star = mode == 1;
  int zt = g.nz;
  int64_t rounds = 1;
  const double planes = (double)(star ? split3<14, 3>(g, sms, zt, rounds) : split3<12, 2>(g, sms, zt, rounds));
  const double pass = 1.5 + planes * (star ? 0.93 + 0.2 / (double)rounds : 0.82 + 0.12 / (double)rounds);
  const int d = std::min(zt1, g.nz) + 2;
  const int64_t n = (int64_t)((g.nx + kTiles[tile][0] - 1) / kTiles[tile][0]) *
                    ((g.ny + kTiles[tile][1] - 1) / kTiles[tile][1]) * ((g.nz + zt1 - 1) / zt1);
  double work;
  if (n <= 4 * (int64_t)sms) {   // every CTA at once
    const double r = (double)((n + sms - 1) / sms);
    work = star ? 3.1 + 0.2 * d + 0.1 * d * r : 3.1 + 0.25 * d + 0.155 * d * r;
  } else {
    const double r = (double)n / sms;
    work = star ? 2.5 + 0.16 * d * r : 4.7 + 0.19 * d * r;
  }
  const double bytes = (star ? 1.5 : 2.0) + (double)g.nx * g.ny * g.nz * 8.0 / 6.7e6;
  return pass < 3.0 * std::max(work, bytes);
}

void launch3(const Grid3& src, const Grid3& dst, const Weights<float>& W, int mode, cudaStream_t s) {
  if (mode == 1) launch3_as<1, 14, 3>(src, dst, W, s);
  else launch3_as<2, 12, 2>(src, dst, W, s);
}

void run(const nca_view* a, const nca_view* b, const double* w27, double dt, int iters, cudaStream_t s) {
  using namespace nca;
  if (!w27) fail(NCA_ERR_INVALID, "null weights");
  if (iters < 0) fail(NCA_ERR_INVALID, "negative iteration count");
  Grid3 ga = check_grid(a, "a"), gb = check_grid(b, "b");
  if (ga.nx != gb.nx || ga.ny != gb.ny || ga.nz != gb.nz || ga.dtype != gb.dtype)
    fail(NCA_ERR_SHAPE, "stencil grids differ in shape or dtype");
  const size_t bytes = (size_t)ga.nx * ga.ny * ga.nz * dtinfo(ga.dtype).size;
  const char *pa = (const char*)ga.base, *pb = (const char*)gb.base;
  if (pa < pb + bytes && pb < pa + bytes) fail(NCA_ERR_INVALID, "stencil source and destination overlap");
  const int mode = star7(w27) ? 1 : isotropic27(w27) ? 2 : 0;
  // steps 1 .. iters-1 three at a time where the three-step kernel applies and pays
  // (each pass moves the result to the other grid, and three single steps do
  // too); the last step runs alone, so that afterwards the two grids hold the
  // last two iterates, as when every step runs alone
  bool three = ga.dtype == NCA_FLOAT32 && mode != 0 && iters > T3_K && tma_ok(ga) && tma_ok(gb);
  if (three) {
    int tile = 0, zt = 8;
    tma_schedule<float>(ga, gb, make_weights<float>(w27, dt), mode, s, tile, zt);
    three = three_pays(ga, mode, sm_count(current_device()), tile, zt);
  }
  bool from_a = true;
  for (int it = 0; it < iters; from_a = !from_a) {
    const Grid3& src = from_a ? ga : gb;
    const Grid3& dst = from_a ? gb : ga;
    if (three && iters - 1 - it >= T3_K) {
      launch3(src, dst, make_weights<float>(w27, dt), mode, s);
      it += T3_K;
      continue;
    }
    ++it;
    if (ga.dtype == NCA_FLOAT32) launch_one<float>(src, dst, make_weights<float>(w27, dt), mode, s);
    else launch_one<double>(src, dst, make_weights<double>(w27, dt), mode, s);
  }
}

}  // namespace

namespace {
// Arrival counters of kernels whose last CTA merges the partial results, one
// block of them per stream (see stream_words). Zero when the module loads.
constexpr int ARR_STREAMS = 64, ARR_N = 4096, FRESH_N = 16384;
__device__ uint32_t g_arrivals[ARR_STREAMS][ARR_N];
__device__ uint32_t g_fresh[ARR_STREAMS][FRESH_N];
}  // namespace

namespace nca {
// address of the status word of JIT kernels on the current device
int* jit_status_word() {
  static std::mutex mu;
  static int* addr[64] = {nullptr};
  const int dev = current_device();
  if (dev < 0 || dev >= 64) fail(NCA_ERR_LIMIT, "device %d", dev);
  std::lock_guard<std::mutex> lk(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    check_cuda(cudaGetSymbolAddress(&p, g_jit_status), "status word address");
    addr[dev] = static_cast<int*>(p);
  }
  return addr[dev];
}

// Kernels of one stream run one after the other, so a block of counters that
// every kernel leaves zero (its last CTA resets what it used) serves all of a
// stream's kernels without a memset before each: (4096, 16384) float32 summed
// over axis 0 59.7 -> 54.9 us. Streams are told apart by their id, which no
// later stream gets again. Null, and the caller zeroes words of its own: for a
// stream under capture (its graph may run on several streams at once), past
// the first ARR_STREAMS streams of a device and above ARR_N words.
//
// Kernels with bounded waits may stop early and leave any count behind, so
// every launch of theirs takes the next counters of the stream's other block,
// and a block that is used up is zeroed as a whole. ((256, 1, 16, 256) transposed
// float32 with a sum and a maximum: 12.4 us with a memset before each launch, 18.7
// with counters under a mark of the launch that a compare and swap had to install,
// 12.5 so; (8, 5, 7, 9) 9.1, 6.2, 6.1.)
struct StreamBlocks {
  uint32_t *plain = nullptr, *fresh = nullptr;
  int64_t next = 0;
  std::mutex m;   // held from taking fresh counters to their launch
};
static StreamBlocks* stream_blocks(cudaStream_t stream) {
  static std::mutex mu;
  static StreamBlocks blocks[64][ARR_STREAMS];
  static std::unordered_map<unsigned long long, int> slots[64];
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamIsCapturing(stream, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone ||
      cudaStreamGetId(stream, &id) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  const int dev = current_device();
  if (dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(mu);
  auto it = slots[dev].find(id);
  if (it == slots[dev].end()) {
    const int k = (int)slots[dev].size();
    if (k >= ARR_STREAMS) return nullptr;
    void *p = nullptr, *f = nullptr;
    check_cuda(cudaGetSymbolAddress(&p, g_arrivals), "arrival counters");
    check_cuda(cudaGetSymbolAddress(&f, g_fresh), "fresh counters");
    blocks[dev][k].plain = static_cast<uint32_t*>(p) + (size_t)k * ARR_N;
    blocks[dev][k].fresh = static_cast<uint32_t*>(f) + (size_t)k * FRESH_N;
    it = slots[dev].emplace(id, k).first;
  }
  return &blocks[dev][it->second];
}
uint32_t* arrival_counters(int64_t n, cudaStream_t stream) {
  StreamBlocks* b = n <= ARR_N ? stream_blocks(stream) : nullptr;
  return b ? b->plain : nullptr;
}
FreshCounters fresh_counters(int64_t n, cudaStream_t stream) {
  FreshCounters c;
  StreamBlocks* b = n <= FRESH_N ? stream_blocks(stream) : nullptr;
  if (!b) return c;
  c.held = std::unique_lock<std::mutex>(b->m);
  if (b->next + n > FRESH_N) {
    check_cuda(cudaMemsetAsync(b->fresh, 0, FRESH_N * sizeof(uint32_t), stream), "fresh counters");
    b->next = 0;
  }
  c.ptr = b->fresh + b->next;
  b->next += n;
  return c;
}

// reads and clears the stencil status word (synchronises the stream)
int stencil_read_status(cudaStream_t s) {
  int v = 0, zero = 0;
  check_cuda(cudaMemcpyFromSymbolAsync(&v, g_stencil_status, sizeof(int), 0, cudaMemcpyDeviceToHost, s), "status read");
  check_cuda(cudaMemcpyToSymbolAsync(g_stencil_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, s), "status clear");
  check_cuda(cudaStreamSynchronize(s), "status sync");
  return v;
}
}  // namespace nca

namespace {
// One thread waits, through the bounded-wait helper every pipeline kernel
// uses, on an mbarrier that expects one arrival which never comes (no copy is
// issued, so none is in flight); after limit_ns it records NCA_ERR_TIMEOUT in
// the stencil status word and returns.
__global__ void wait_probe_kernel(unsigned long long limit_ns) {
  __shared__ __align__(8) unsigned long long bar;
  if (threadIdx.x != 0) return;
  const uint32_t b = (uint32_t)__cvta_generic_to_shared(&bar);
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  if (!mbar_wait(b, 0u, limit_ns)) atomicExch(&g_stencil_status, (int)NCA_ERR_TIMEOUT);
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(b) : "memory");
}
}  // namespace

extern "C" int32_t nca_wait_probe(double limit_s, void* stream) {
  return nca::guarded([&] {
    using namespace nca;
    if (!(limit_s >= 1e-3 && limit_s <= 2.0)) fail(NCA_ERR_INVALID, "limit %g s: 0.001 .. 2 s", limit_s);
    wait_probe_kernel<<<1, 32, 0, (cudaStream_t)stream>>>((unsigned long long)(limit_s * 1e9));
    check_cuda(cudaGetLastError(), "wait probe launch");
    count_launch();
  });
}

extern "C" int32_t nca_stencil3d(const nca_view* src, const nca_view* dst, const double* weights27, double dt,
                                 void* stream) {
  return nca::guarded([&] { run(src, dst, weights27, dt, 1, (cudaStream_t)stream); });
}

extern "C" int32_t nca_stencil3d_iterate(const nca_view* a, const nca_view* b, const double* weights27, double dt,
                                         int32_t iters, void* stream) {
  return nca::guarded([&] { run(a, b, weights27, dt, iters, (cudaStream_t)stream); });
}
