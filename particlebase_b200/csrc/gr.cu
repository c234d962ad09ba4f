// Radial distribution function: pair counts per distance bin.
//
// Replaces cudaCalcGR::calcgr (cudaCalcGR.cu:85-116) with the pair kernel
// calcF_IJpairWithBlock5_F4<calcGR_F4> (kerneltemplate.hh:423-512,
// kernelinline.hh:433-449): every unordered pair of atoms, minimum image,
// bin j = trunc(r / rstep + 1/2), counted when 0 < j < rnum.  The reference
// walks every pair of cell blocks (makePairInfo, cudaCalcGR.cu:43-83), so the
// work is all pairs whatever rmax is.  Here a task is 256 atoms i against 64
// atoms j; each CTA takes many tasks and keeps one shared-memory histogram,
// which it adds to the global counts with 64-bit integer atomics at its end, so
// the result does not depend on scheduling.
//
// Arithmetic: FP32 round-to-nearest with no fused multiply-add, r^2 =
// (dx^2 + dy^2) + dz^2, and the exact minimum image (the coordinate above the
// box middle moved down by L first): x = fl(fl(sqrt(r^2) inv) + 1/2), bin
// trunc(x).  The oracle restates exactly these operations.  Two pairs go
// through packed FP32x2 instructions, which round each half as the scalar ones.
// x grows with r^2, so "x < rnum" is a comparison of r^2 with the largest r^2
// that passes (found on the host by bisection).  The bin comes from an
// approximate square root, and is computed exactly where that one's error could
// change it (near a half-integer: one pair in a thousand at 840 bins).
//
// Bound by instruction issue: 27 instructions a pair of a lane, 74 % of the issue
// slots; the shared-memory atomics take 44 % of that pipe.  32,000 atoms, 840
// bins, out to half the box: 0.53 ms.  It was 0.93 ms when every CTA had one tile
// pair of 128 x 128 atoms (one global atomic per bin and CTA) and a pair took an
// IEEE square root and a scalar minimum image.
#include <cmath>
#include <cstring>

#include "md.cuh"
#include "tma.cuh"

namespace pb {
namespace {

constexpr int kGrThreads = 128;
constexpr uint32_t kGrI = 2 * kGrThreads;  // atoms i of a task, two per thread
constexpr uint32_t kGrJ = 64;              // atoms j of a task
constexpr uint32_t kGrRatio = kGrI / kGrJ;
constexpr float kGrFar = 1e30f;
// a CTA's 32-bit counts are added to the global ones before they can wrap
constexpr uint32_t kGrFlush = 0xffffffffu / (kGrI * kGrJ);

// Binning of one distance: x_max = rnum, lim = 1/2 less the error of the
// approximate x, cap = largest r^2 that is counted.
struct GrBins {
  float inv, cap, lim, mz;  // mz: -0
  uint32_t rnum;
};

__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Packed sum of two FP32 pairs, and their product, each half rounded once.  The
// product is a fused multiply-add of -0 that the compiler cannot see through:
// it contracts a packed product and sum, even with their rounding named.
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }

__device__ __forceinline__ float2 mul2(float2 a, float2 b, float minus_zero) {
  return __ffma2_rn(a, b, make_float2(minus_zero, minus_zero));
}

// Counts four pairs.  The rare exact bins share one branch; a pair out of range
// adds to a counter of its lane that nobody reads (a branch around the atomic
// took more).
__device__ __forceinline__ void count_pairs(const GrBins &g, const float (&r2)[4], uint32_t hist,
                                            uint32_t idle) {
  constexpr float kRound = 12582912.0f;  // 1.5 x 2^23: adding it rounds to an integer
  uint32_t b[4];
  float off = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float x = __fmul_rn(sqrt_approx(r2[k]), g.inv);
    const float m = __fadd_rn(x, kRound);
    b[k] = __float_as_uint(m) - __float_as_uint(kRound);
    off = fmaxf(off, fabsf(__fsub_rn(x, __fsub_rn(m, kRound))));  // NaN, of r2 = inf, drops out
  }
  if (off > g.lim) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      b[k] = (uint32_t)__fadd_rn(__fmul_rn(__fsqrt_rn(r2[k]), g.inv), 0.5f);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(r2[k] <= g.cap ? hist + 4u * b[k] : idle)
                 : "memory");
}

// Minimum-image component of two pairs: xi - xj, or the smaller of
// (xi - L) - xj and xi - (xj - L) where that exceeds half the box.  n, nl hold
// -xj and -(xj - L).  Without the comparison (kMin) the smallest of the three is
// the same number unless |xi - xj| is within rounding of half the box; the
// caller takes it only when such pairs lie beyond the counted range.
template <bool kMin>
__device__ __forceinline__ float2 image2(float2 xi, float2 xil, float2 n, float2 nl, float h) {
  const float2 d = add2(xi, n), a = add2(xil, n), b = add2(xi, nl);
  if (kMin)
    return make_float2(fminf(fminf(fabsf(d.x), fabsf(a.x)), fabsf(b.x)),
                       fminf(fminf(fabsf(d.y), fabsf(a.y)), fabsf(b.y)));
  return make_float2(fabsf(d.x) > h ? fminf(fabsf(a.x), fabsf(b.x)) : d.x,
                     fabsf(d.y) > h ? fminf(fabsf(a.y), fabsf(b.y)) : d.y);
}

// An atom i: its position, and the same moved down by L.
struct AtomI {
  float x, y, z, xl, yl, zl;
};

// One task's pairs of this thread; kDiag: only j >= first.
template <bool kMin, bool kDiag>
__device__ __forceinline__ void task(const GrBins &g, const AtomI (&a)[2],
                                     const float (&sj)[6][kGrJ], const uint32_t (&first)[2],
                                     float3 h, uint32_t hist) {
  const uint32_t idle = hist + 4u * (g.rnum + (threadIdx.x & 31u));
#pragma unroll 4
  for (uint32_t j = 0; j < kGrJ; j += 2) {
    float2 c[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) c[k] = *reinterpret_cast<const float2 *>(&sj[k][j]);
    float r2[4];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float2 dx = image2<kMin>(make_float2(a[k].x, a[k].x), make_float2(a[k].xl, a[k].xl),
                                     c[0], c[1], h.x);
      const float2 dy = image2<kMin>(make_float2(a[k].y, a[k].y), make_float2(a[k].yl, a[k].yl),
                                     c[2], c[3], h.y);
      const float2 dz = image2<kMin>(make_float2(a[k].z, a[k].z), make_float2(a[k].zl, a[k].zl),
                                     c[4], c[5], h.z);
      const float2 q = add2(add2(mul2(dx, dx, g.mz), mul2(dy, dy, g.mz)), mul2(dz, dz, g.mz));
      r2[2 * k] = kDiag && j < first[k] ? INFINITY : q.x;
      r2[2 * k + 1] = kDiag && j + 1 < first[k] ? INFINITY : q.y;
    }
    count_pairs(g, r2, hist, idle);
  }
}

template <bool kMin>
__global__ void __launch_bounds__(kGrThreads, 7)
    k_gr(const float4 *__restrict__ r, uint32_t N, float Lx, float Ly, float Lz, GrBins g,
         uint64_t ntask, uint32_t TI, uint32_t TJ, unsigned long long *counts) {
  extern __shared__ uint32_t hist[];  // rnum bins (bin 0 is not counted), and the idle counters
  __shared__ __align__(16) float sj[6][kGrJ];  // -x, -(x - L), and so for y, z
  const uint32_t base = smem_u32(hist);
  const float3 h = make_float3(0.5f * Lx, 0.5f * Ly, 0.5f * Lz);
  for (uint32_t b = threadIdx.x; b < g.rnum; b += kGrThreads) hist[b] = 0u;
  uint32_t done = 0;
  // row I of tasks holds J = ratio I .. TJ - 1; rows I and TI - 1 - I together
  // have W tasks whatever I is
  const uint32_t W = 2 * TJ - kGrRatio * TI + kGrRatio;
  for (uint64_t q = blockIdx.x; q < ntask; q += gridDim.x) {
    const uint32_t row = (uint32_t)(q / W), off = (uint32_t)(q % W);
    const uint32_t len = TJ - kGrRatio * row, back = TI - 1 - row;
    if (off >= len && back == row) continue;  // the middle row has no partner
    const uint32_t I = off < len ? row : back;
    const uint32_t J = kGrRatio * I + (off < len ? off : off - len);
    __syncthreads();
    if (done == kGrFlush) {
      for (uint32_t b = threadIdx.x; b < g.rnum; b += kGrThreads) {
        if (b > 0 && hist[b]) atomicAdd(&counts[b], (unsigned long long)hist[b]);
        hist[b] = 0u;
      }
      done = 0;
    }
    ++done;
    if (threadIdx.x < kGrJ) {
      const uint32_t j = J * kGrJ + threadIdx.x;
      const float4 p = j < N ? r[j] : make_float4(kGrFar, kGrFar, kGrFar, 0.f);
      sj[0][threadIdx.x] = -p.x;
      sj[1][threadIdx.x] = -__fsub_rn(p.x, Lx);
      sj[2][threadIdx.x] = -p.y;
      sj[3][threadIdx.x] = -__fsub_rn(p.y, Ly);
      sj[4][threadIdx.x] = -p.z;
      sj[5][threadIdx.x] = -__fsub_rn(p.z, Lz);
    }
    __syncthreads();
    AtomI a[2];
    uint32_t first[2];  // j from which a thread's pairs count (j > i)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t i = I * kGrI + k * kGrThreads + threadIdx.x;
      const float4 p = i < N ? r[i] : make_float4(-kGrFar, -kGrFar, -kGrFar, 0.f);
      first[k] = i >= J * kGrJ ? i - J * kGrJ + 1 : 0u;
      a[k] = AtomI{p.x, p.y, p.z, __fsub_rn(p.x, Lx), __fsub_rn(p.y, Ly), __fsub_rn(p.z, Lz)};
    }
    if (J < kGrRatio * (I + 1))
      task<kMin, true>(g, a, sj, first, h, base);
    else
      task<kMin, false>(g, a, sj, first, h, base);
  }
  __syncthreads();
  for (uint32_t b = threadIdx.x; b < g.rnum; b += kGrThreads)
    if (b > 0 && hist[b]) atomicAdd(&counts[b], (unsigned long long)hist[b]);
}

// x of a squared distance, each operation rounded to FP32.
float gr_x(float r2, float inv) {
  volatile float s = std::sqrt(r2);
  volatile float m = s * inv;
  volatile float x = m + 0.5f;
  return x;
}

// Largest r^2 whose x lies below rnum (x never decreases with r^2).
float gr_cap(float inv, uint32_t rnum) {
  uint32_t lo = 0u, hi = 0x7f800000u;  // bits of 0 (x = 1/2) and of infinity
  while (hi - lo > 1) {
    const uint32_t mid = lo + (hi - lo) / 2;
    float r2;
    std::memcpy(&r2, &mid, 4);
    if (gr_x(r2, inv) < (float)rnum) lo = mid; else hi = mid;
  }
  float r2;
  std::memcpy(&r2, &lo, 4);
  return r2;
}

}  // namespace

uint32_t gr_max_bins() { return 16384; }

cudaError_t launch_gr(const float4 *r, uint32_t N, const float L[3], float inv, uint32_t rnum,
                      unsigned long long *counts, cudaStream_t s) {
  if (N == 0 || rnum == 0) return cudaSuccess;
  const uint32_t TI = (N + kGrI - 1) / kGrI, TJ = (N + kGrJ - 1) / kGrJ;
  const uint64_t ntask = (uint64_t)((TI + 1) / 2) * (2 * TJ - kGrRatio * TI + kGrRatio);
  // both x carry at most 3 roundings of 2^-24 and the approximate square root
  // 2^-23: their difference stays below 4 x 2^-23 of x
  // (a flushed subnormal r^2 must lie in bin 0 as well, else every bin is exact)
  const float lim = inv < 1e18f ? 0.5f - (float)rnum * 4.8e-7f - 1e-6f : -1.0f;
  const GrBins g{inv, gr_cap(inv, rnum), lim, -0.0f, rnum};
  const size_t smem = sizeof(uint32_t) * (rnum + 32u);
  // pairs half a box apart in some axis are not counted: r^2 above cap, by far
  // more than the rounding of either form of the minimum image
  const float h = 0.5f * std::fmin(L[0], std::fmin(L[1], L[2])) * 0.9999f;
  auto kern = g.cap < h * h ? k_gr<true> : k_gr<false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 1, per = 1;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
    return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kGrThreads, smem)) !=
      cudaSuccess)
    return e;
  const uint64_t slots = (uint64_t)sms * (per > 0 ? per : 1);
  kern<<<(uint32_t)(ntask < slots ? ntask : slots), kGrThreads, smem, s>>>(
      r, N, L[0], L[1], L[2], g, ntask, TI, TJ, counts);
  return cudaGetLastError();
}

}  // namespace pb
