// Lennard-Jones pair forces over the cell list.
//
// Replaces cudaParticleMD::calcForce (cudaParticleMD.cu:24-69):
// calcF_IJpairWithBlock_F4<MDpairForce<potentialLJ>> on a (cells x 27) grid
// writing 27 partial-force planes tmp81N, followed by reduce27_F4
// (kerneltemplate.hh:229-294, kerneltemplate.hh:523-565, kernelinline.hh:86-96,
// kernelfuncs.cu:935-949).  The physics is the reference's: truncated,
// unshifted LJ, F_i = sum_{j != i, r < rc} 24 eps (s/r)^6 (2 (s/r)^6 - 1) / r^2
// (r_i - r_j) with the minimum image, over the 27-cell stencil.  No 81 N
// scratch: each atom's force is summed in registers and written once.
//
// Work items.  One CTA of 8 warps computes one work item = (system, x-y column
// of cells, run of z cells [z0, z1)), at most about 8 tiles of 16 consecutive
// (z-sorted) home atoms; at density 0.84 the shared memory makes it 7 cells of 14
// atoms, 7 tiles.  It stages the 3 x 3 neighbour columns over z cells
// [z0 - 1, z1] (periodic halo cells included) in shared memory by bulk copies
// of the sorted positions (bounded wait), then a warp takes a tile and waits
// for no other.  Four CTAs share an SM, so one's staging overlaps another's
// computation.  What bounds it is instruction issue (70 % of the slots at 1M
// atoms, shared memory 61 %).  Per home atom 188 warp instructions; when they were 186,
// staging took 30, block tables and tile set-up 23, phase 1 56, phase 2 77.  Longer runs stage fewer halo cells
// per home atom and shorter ones fit more CTAs: 4, 5, 6 and 7 cells of 14 atoms
// took 0.362, 0.322, 0.284 and 0.268 ms at 1M atoms; 9 cells, at three CTAs per
// SM, 0.293; CTAs of 16 warps over 14 cells 0.281.  A persistent kernel with
// producer warps that tested quads of candidates with FMAs took 0.325 ms.
//
// Coordinate frame.  Positions are absolute FP32 coordinates.  Each item moves
// all staged atoms into one frame by subtracting 0 or L per axis: a neighbour
// image below the box (atoms near the top face) and, in items on the top face,
// every non-wrapped atom, get x - L.  The subtraction only ever applies to
// coordinates >= L/2, where it is exact (Sterbenz), so displacements x_i - x_j
// in the frame are the minimum-image displacements with no rounding beyond
// the subtraction itself, even in a 190-sigma box.  Work items are laid out
// so that a top-face item's cells all lie above the box middle (a column that
// fits one run rounds only the image above its top).
//
// Stage.  Each staged column is one z-sorted array padded with far atoms
// (coordinates 1e30) to a multiple of 8 slots.  A slot holds the exact frame
// position and type (16 B), and an approximate record of four fp16 values (8 B):
// the position relative to the item's centre in units of the longest cell edge,
// and its squared norm; with several types also the indicators of its type.
//
// Phase 1, on the tensor cores.  The candidates of a tile are the blocks of 8
// whose z range meets [zmin - rc, zmax + rc].  One mma.sync m16n8k8 (fp16
// operands, FP32 sums) gives 16 x 8 values
// |x_j|^2 - 2 x_i . x_j + (|x_i|^2 - bound), whose sign says whether the pair
// may be within rc.  `bound` exceeds rc^2 by what the rounding of the records
// can change (from the home atom's own norm), so the hits are a superset of the
// pairs inside the cutoff: about 4 % more.  With several types the indicators'
// share of the product lowers the bound to that pair of types' own cutoff.
// mma.sync and not tcgen05: a tile shares its window with no other, its product
// has a depth of 8, and 52 of them take 11 % of the tensor pipe; the work is in
// reading their signs.  A lane owns 2 home atoms x 2 candidates of each block
// and lists the candidates that may be near either of its two.
//
// Phase 2.  Each lane walks its list (lane-minor in shared memory).  It fetches
// the exact position once, evaluates the pairs with both its home atoms
// (neighbours in z, sharing most candidates: 1.42 sphere volumes for 2) in
// packed FP32x2 arithmetic, each home atom one half, and applies the exact
// cutoff 0 < r^2 < rc^2 (the self pair has r^2 = 0).  Two shuffles combine the 4
// lanes of an atom.  Bit strings in registers instead of lists cost 51
// instructions a step against 38 (0.364 against 0.325 ms with the staging of
// that version); evening out the lists of neighbouring lanes gained nothing.
//
// Every sum runs in candidate order within a lane and in a fixed order over
// the lanes, and windows and blocks depend on the item alone, so a system's
// forces do not depend on scheduling or on the other systems of a batch.  An
// item whose stage exceeds its capacity computes from global memory instead
// (slower) and raises a status bit; so does an item with a home atom out of the
// range of the records (an open box, hundreds of sigma outside), without the bit.
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "force_common.cuh"

namespace pb {
namespace {

constexpr int kTile = 16;         // home atoms per tile (rows of one mma)
constexpr int kTabBlocks = 96;    // blocks in a warp's table at once
constexpr uint32_t kTabBytes = kTabBlocks * 4;
// Hits a lane lists before they are evaluated: as many as leave the shared
// memory for the CTAs per SM that the registers allow.
__host__ __device__ constexpr uint32_t list_len(int nt) { return nt > 1 ? 36u : 28u; }
// Per warp: the table of block starts, and the lanes' lists of hits.
__host__ __device__ constexpr uint32_t warp_bytes(int nt) { return kTabBytes + list_len(nt) * 64u; }
constexpr float kMaxNorm = 30000.f;  // largest norm of a home atom in fp16 records

// One work item: its staged columns and the constants of its frame.
template <int NT>
struct Stage {
  uint32_t c0[10];        // first slot of each column's region (multiples of 8); c0[9] = end
  uint32_t e0[9], e1[9], e2[9];  // ends of its low image, middle run and high image
  float sx[9], sy[9];     // frame shift of each column (0 or L)
  float szl, szm, szh;    // frame shift of the low image, the middle run, the high image
  float cx, cy, cz, scale;  // centre and scale of the fp16 records
  float rcw;              // half-width of the z windows
  float rs, rs2, rs_dl;   // rc (of the longest-ranged pair) in record units: for the bounds
  uint32_t home_g0, hb, H, ntile;  // home atoms: first sorted slot, first stage slot, count
  uint32_t kbase[9];
  int z0, nz, nseg, periodic, overflow;
  int shifted;            // some frame shift is not zero
  int one;                // the system has one type, whatever the launch is compiled for
  uint32_t nmax;          // largest norm staged (float bits, non-negative)
  LJLocal<NT> lj;
  // several types: what the bound of a pair of types lies below the longest
  // one, per type of home atom as fp16 for candidate types 0 .. 3
  uint2 cut[NT > 1 ? NT : 1];
  float4 lj4[NT > 1 ? NT * NT : 1];  // {sigma^2, 24 eps, bits of rc^2 less one, 0} per type pair
};

// Slots of a stage for `cap` staged atoms: every column rounds up to whole
// blocks, and one block of far atoms pads the block tables.  A multiple of 16,
// which keeps every part of the shared memory below on a 16-byte boundary.
__host__ __device__ __forceinline__ uint32_t padded_slots(uint32_t cap) {
  return ((cap + 15u) & ~15u) + 9u * 8u + 8u;
}
static_assert(warp_bytes(1) % 16 == 0 && warp_bytes(2) % 16 == 0, "tables are read 16 bytes at a time");

// Bytes per slot of the type indicators, and of everything: exact position,
// fp16 record, type indicators, and a share of the block's z range.
__host__ __device__ constexpr uint32_t type_bytes(int nt) { return nt > 2 ? 8u : (nt > 1 ? 4u : 0u); }
__host__ __device__ constexpr uint32_t slot_bytes(int nt) { return 25u + type_bytes(nt); }

// Dynamic shared memory of one CTA: the stage, and the warps' tables and lists.
__host__ __device__ __forceinline__ uint32_t smem_bytes(uint32_t cap, int warps, int nt) {
  return padded_slots(cap) * slot_bytes(nt) + (uint32_t)warps * warp_bytes(nt);
}

// Coefficient of w^k in cos(pi sqrt(w) / 2).
constexpr double cos_term(int k) {
  double t = 1.0;
  for (int j = 1; j <= k; ++j)
    t *= -3.14159265358979323846 * 3.14159265358979323846 / 4 / (2 * j * (2 * j - 1));
  return t;
}

template <int K = 0>
__device__ __forceinline__ double cos_sum(double w) {
  constexpr double t = cos_term(K);
  if constexpr (K == 8)
    return t;
  else
    return fma(cos_sum<K + 1>(w), w, t);
}

// f0 cos(pi r / 2 rc) / r of the soft-core force: the cosine's Taylor series in (r / rc)^2, in
// FP64 (its terms up to the 8th leave 6e-13 inside the range), takes no root and no quotient.
template <int M>
__device__ __forceinline__ float soft_core(const LJLocal<M> &lj, float r2) {
  return lj.sc_f0 * (float)cos_sum((double)r2 * lj.sc_w) * rsqrtf(r2);
}

// MODE kModeCapped: relaxation force of the steepest-descent path, with the
// pair distance floored at sigma/2 so that overlapping random starts give
// finite forces.  MODE kModeSoftCore: the soft-core force of potentialSC
// (kernelinline.hh:136-158) as MDpairForce applies it (kerneltemplate.hh:530-564):
// f0 cos(r / rc * pi / 2) times the unit vector, zero beyond rc.
template <int NT, bool ENERGY, typename Acc, int MODE = kModeLJ>
struct PairAcc {
  Acc fx = 0, fy = 0, fz = 0, pe = 0, pes = 0, vir = 0;
  uint32_t n = 0;
  template <int M>
  __device__ __forceinline__ void add(const LJLocal<M> &lj, int k, float dx, float dy, float dz,
                                      float r2) {
    if (MODE == kModeSoftCore) {
      const float f = soft_core(lj, r2);
      fx += (Acc)(f * dx);
      fy += (Acc)(f * dy);
      fz += (Acc)(f * dz);
      return;
    }
    if (MODE == kModeCapped) r2 = fmaxf(r2, 0.25f * lj.s2[k]);
    const float inv = rcp_approx(r2);
    const float sr2 = lj.s2[k] * inv;
    const float sr6 = sr2 * sr2 * sr2;
    const float f = lj.e24[k] * sr6 * fmaf(2.0f, sr6, -1.0f) * inv;
    fx += (Acc)(f * dx);
    fy += (Acc)(f * dy);
    fz += (Acc)(f * dz);
    if (ENERGY) {
      const float u = lj.e4[k] * sr6 * (sr6 - 1.0f);
      pe += (Acc)(0.5f * u);
      pes += (Acc)(0.5f * (u - lj.ush[k]));
      vir += (Acc)(0.5f * f * r2);
      ++n;
    }
  }
};

// Packed force sums of phase 2 (FP32): one half per home atom of the lane.
struct Force2 {
  float2 fx = {0.f, 0.f}, fy = {0.f, 0.f}, fz = {0.f, 0.f};
};

// Global-memory path (stage overflow): lanes are 32 consecutive home atoms,
// candidates of one z cell of one column, frame shifts applied per pair.
template <int NT, bool ENERGY, bool SELF, typename Acc, int MODE>
__device__ __forceinline__ void global_range(const float4 *__restrict__ P, uint32_t jb,
                                             uint32_t je, float xi, float yi, float zi, int ti,
                                             float sx, float sy, float sz, uint32_t self,
                                             const LJLocal<NT> &lj,
                                             PairAcc<NT, ENERGY, Acc, MODE> &a) {
  for (uint32_t j = jb; j < je; ++j) {
    const float4 q = P[j];
    const float dx = xi - (q.x - sx), dy = yi - (q.y - sy), dz = zi - (q.z - sz);
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const int k = NT == 1 ? 0 : ti * NT + __float_as_int(q.w);
    if (r2 < lj.rc2[k] && (!SELF || j != self)) a.add(lj, k, dx, dy, dz, r2);
  }
}


// 0 < r2 < rc2 by one unsigned comparison: floats that are not negative order
// as their bits, r2 = 0 wraps to the largest value and NaNs lie above every rc2.
// The bound of a pair that does not interact (rc2 = 0) is 0: nothing lies below.
__device__ __forceinline__ bool inside(float r2, uint32_t rc2_less_1) {
  return __float_as_uint(r2) - 1u < rc2_less_1;
}

__device__ __forceinline__ uint32_t less_1(float rc2) {
  return rc2 > 0.0f ? __float_as_uint(rc2) - 1u : 0u;
}

// D = A B + C of one m16n8k8 product, fp16 operands and FP32 sums.
__device__ __forceinline__ void mma_16x8x8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b,
                                           const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, "
      "{%7, %8, %9, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(b), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}

__device__ __forceinline__ uint4 lds_u4(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(a)
               : "memory");
  return v;
}

// Stage reads: the stage is read-only once handed over, so the compiler may
// schedule them freely.
__device__ __forceinline__ uint32_t lds_stage(uint32_t a) {
  uint32_t v;
  asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ float2 unpack_half2(uint32_t u) {
  return __half22float2(*reinterpret_cast<const __half2 *>(&u));
}

__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// LJ tables of the item's system (one warp).
template <int NT, int MODE>
__device__ __forceinline__ void load_lj(const ForceBufs &b, const SysDesc &S, Stage<NT> &d) {
  const LJTable &T = b.lj[S.lj];
  const float sc = 1.0f / fmaxf(fmaxf(S.g.len[0], S.g.len[1]), S.g.len[2]);
  const int lane = threadIdx.x & 31;
  const float most = MODE == kModeSoftCore ? b.sc_rc * b.sc_rc : kFar;
  float rc2max = 0.f;
  for (int t = lane; t < NT * NT; t += 32) {
    const int k = t / NT * T.nt + t % NT;
    // (a cutoff that is not a number is none; the soft core has its own range)
    const float rc2 = MODE == kModeSoftCore || T.rc2[k] > 0.0f ? fminf(T.rc2[k], most) : 0.0f;
    d.lj.s2[t] = T.s2[k];
    d.lj.e24[t] = T.e24[k];
    d.lj.e4[t] = T.e4[k];
    d.lj.rc2[t] = rc2;
    d.lj.ush[t] = T.ushift[k];
    if (NT > 1)
      d.lj4[t] = make_float4(T.s2[k], T.e24[k], __uint_as_float(less_1(rc2)), 0.f);
    rc2max = fmaxf(rc2max, rc2);
  }
  // non-negative floats order as their bits
  rc2max = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(rc2max)));
  if (NT > 1 && lane < NT) {
    float c[4];
    for (int k = 0; k < 4; ++k) {
      const float rc2 = k < T.nt && lane < T.nt ? fminf(T.rc2[lane * T.nt + k], most) : rc2max;
      // rounded down, so that no pair inside its cutoff is lost
      c[k] = (rc2max - rc2) * sc * sc * (1.0f - 1.0f / 512.0f);
    }
    d.cut[lane] = make_uint2(pack_half2(c[0], c[1]), pack_half2(c[2], c[3]));
  }
  if (lane == 0) {
    if (MODE == kModeSoftCore) {
      d.lj.sc_w = 1.0 / ((double)b.sc_rc * b.sc_rc);
      d.lj.sc_f0 = b.sc_f0;
    }
    d.one = T.nt == 1;
    d.rcw = sqrtf(rc2max) * 1.00001f + 1e-5f;
    const float rs = sqrtf(rc2max) * sc * 1.00001f;
    d.rs = rs;
    d.rs2 = rc2max * sc * sc + 1e-4f;
    d.rs_dl = rs * (1.05f / 512.0f);
  }
}

// Lays out the stage of work item `it` and starts its copies (one warp): runs
// of the sorted positions go to their slots by bulk copies that complete on
// `full`, and far atoms pad the columns.
template <int NT>
__device__ __forceinline__ void plan_stage(const ForceBufs &b, const ForceItem &it, Stage<NT> &d,
                                           float4 *E, uint64_t *full) {
  const int lane = threadIdx.x & 31;
  const SysDesc &S = b.sys[it.sys];
  const int z0 = it.z0, z1 = it.z1, nz = S.g.n[2];
  const bool per = S.g.periodic != 0;
  uint32_t nl = 0, nm = 0, nh = 0, gl = 0, gm = 0, gh = 0, home0 = 0, home1 = 0;
  if (lane < 9) {
    const uint32_t kb = it.kbase[lane];
    d.kbase[lane] = kb;
    if (per || kb != kNoCell) {  // no column past an open face
      // the z cells of a column are consecutive keys: its staged cells are one
      // run, plus an image of the top (bottom) cell below (above) it
      const uint32_t zl = (uint32_t)max(z0 - 1, 0), zh = (uint32_t)min(z1 + 1, nz);
      gm = b.start[kb + zl];
      nm = b.start[kb + zh] - gm;
      if (per && z0 == 0) {
        gl = b.start[kb + nz - 1];
        nl = b.start[kb + nz] - gl;
      }
      if (per && z1 == nz) {
        gh = b.start[kb];
        nh = b.start[kb + 1] - gh;
      }
      if (lane == 4) {
        home0 = b.start[kb + z0];
        home1 = b.start[kb + z1];
      }
    }
  }
  const uint32_t n = nl + nm + nh, slots = (n + 7u) & ~7u;
  uint32_t incl = slots, atoms = n;
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
    atoms += __shfl_xor_sync(0xffffffffu, atoms, o);
  }
  const uint32_t first = incl - slots;
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 8);
  // the system's own capacity decides: the same path alone or batched
  const uint32_t H = __shfl_sync(0xffffffffu, home1 - home0, 4);
  const uint32_t ntile = (H + kTile - 1) / kTile;
  const bool overflow = total + 8u > padded_slots(S.cap) || ntile > (uint32_t)kWinCap;
  const bool copy = !overflow && !(b.test_flags & 1u);  // test hook: the copies never arrive
  if (copy && lane == 0) mbar_arrive_expect_tx(full, 16u * atoms);
  __syncwarp();
  if (lane < 9) {
    if (copy) {
      if (nl) bulk_g2s(E + first, b.rs + gl, 16u * nl, full);
      if (nm) bulk_g2s(E + first + nl, b.rs + gm, 16u * nm, full);
      if (nh) bulk_g2s(E + first + nl + nm, b.rs + gh, 16u * nh, full);
      for (uint32_t k = first + n; k < first + slots; ++k)
        E[k] = make_float4(kFar, kFar, kFar, 0.f);
    }
    d.c0[lane] = first;
    d.e0[lane] = first + nl;
    d.e1[lane] = first + nl + nm;
    d.e2[lane] = first + n;
  } else if (copy && lane < 17) {
    E[total + (uint32_t)lane - 9u] = make_float4(kFar, kFar, kFar, 0.f);
  }
  if (lane == 4) {
    d.c0[9] = total;
    d.home_g0 = home0;
    d.H = H;
    d.hb = first + nl + (home0 - gm);
    d.ntile = ntile;
    d.overflow = overflow;
    if (overflow) {
      d.ntile = min((H + 31) / 32, (uint32_t)kWinCap);
      atomicOr(&b.status[it.sys], kStatusSmemOverflow);
    }
  }
}

// Frame shifts and constants of the item (one warp).
template <int NT>
__device__ __forceinline__ void plan_frame(const ForceBufs &b, const ForceItem &it, Stage<NT> &d) {
  const int lane = threadIdx.x & 31;
  const Grid &g = b.sys[it.sys].g;
  const int z0 = it.z0, z1 = it.z1, nz = g.n[2];
  const bool per = g.periodic != 0;
  // an item on the top face works in the frame shifted down by L, where the
  // shifts of its atoms (all in the upper half) are exact; a whole column
  // keeps the unshifted frame and rounds only the image above its top
  const float Fx = per && it.cx == g.n[0] - 1 ? g.L[0] : 0.0f;
  const float Fy = per && it.cy == g.n[1] - 1 ? g.L[1] : 0.0f;
  const float Fz = per && z1 == nz && z0 > 0 ? g.L[2] : 0.0f;
  float sx = 0.f, sy = 0.f;
  if (lane < 9 && per) {
    const int ax = it.cx + lane / 3 - 1, ay = it.cy + lane % 3 - 1;
    const int wx = ax < 0 ? -1 : (ax >= g.n[0] ? 1 : 0);
    const int wy = ay < 0 ? -1 : (ay >= g.n[1] ? 1 : 0);
    // frame: F = L on the top face; staged = x + w L - F, so the shift is F - w L
    // (an open box has no images and no frame shift)
    sx = Fx - (float)wx * g.L[0];
    sy = Fy - (float)wy * g.L[1];
  }
  if (lane < 9) {
    d.sx[lane] = sx;
    d.sy[lane] = sy;
  }
  const bool any = __any_sync(0xffffffffu, sx != 0.f || sy != 0.f);
  if (lane == 0) {
    d.szm = Fz;
    d.szl = per ? Fz + g.L[2] : Fz;  // image z0 - 1 wraps below when z0 == 0
    d.szh = per ? Fz - g.L[2] : Fz;  // image z1 wraps above when z1 == nz
    d.shifted = any || (per && (z0 == 0 || z1 == nz));
    d.cx = g.lo[0] + ((float)it.cx + 0.5f) * g.len[0] - Fx;
    d.cy = g.lo[1] + ((float)it.cy + 0.5f) * g.len[1] - Fy;
    d.cz = g.lo[2] + 0.5f * (float)(z0 + z1) * g.len[2] - Fz;
    d.scale = 1.0f / fmaxf(fmaxf(g.len[0], g.len[1]), g.len[2]);
    d.z0 = z0;
    d.nz = nz;
    d.nseg = z1 - z0;
    d.periodic = per;
    d.nmax = 0u;
  }
}

// Opens the z windows of an item whose staged columns are not all sorted by z (one warp).
// Cells are sorted, and so are runs of them, except that cell 0 also takes the atoms more
// than a cell above the top of the box (open boundaries, or positions not wrapped); an
// image joins its run at the other two seams.  The atoms on either side of a seam are read
// from global memory, so that no other warp waits and nothing is kept for the tiles.
template <int NT>
__device__ __forceinline__ void check_order(const ForceBufs &b, const ForceItem &it, Stage<NT> &d) {
  const int lane = threadIdx.x & 31, seam = lane / 9;
  const Grid &g = b.sys[it.sys].g;
  const int z0 = it.z0, z1 = it.z1, nz = g.n[2];
  const bool per = g.periodic != 0;
  if (z0 > 1 && z1 < nz) return;
  const uint32_t kb = it.kbase[lane % 9];
  const bool there = seam == 0 ? per && z0 == 0 : seam == 1 ? z0 <= 1 : per && z1 == nz;
  bool drop = false;
  if (lane < 27 && there && (per || kb != kNoCell)) {
    const uint32_t kl = kb + (uint32_t)max(z0 - 1, 0), kh = kb + (uint32_t)min(z1 + 1, nz);
    // the cells before the seam and after it
    const uint32_t a0 = seam == 0 ? kb + nz - 1 : kl, a1 = seam == 0 ? kb + nz : seam == 1 ? kb + 1 : kh;
    const uint32_t c0 = seam == 0 ? kl : seam == 1 ? kb + 1 : kb, c1 = seam == 2 ? kb + 1 : kh;
    const uint32_t sa = b.start[a0], ea = b.start[a1], sc = b.start[c0], ec = b.start[c1];
    if (sa < ea && sc < ec) {
      const float up = seam == 1 ? 0.0f : g.L[2];  // by an image below, or of one above
      // (a NaN, last in cell 0, may hide atoms that are out of order before it)
      drop = !(b.rs[ea - 1].z - (seam == 0 ? up : 0.0f) <= b.rs[sc].z + (seam == 2 ? up : 0.0f));
    }
  }
  if (__any_sync(0xffffffffu, drop) && lane == 0) d.rcw = kFar;
}

// Moves the staged atoms into the item's frame, a warp per column (x - 0 is x,
// so unshifted atoms pass unchanged).
template <int NT, int kWarps>
__device__ __forceinline__ void shift_stage(const Stage<NT> &d, float4 *E) {
  for (int c = threadIdx.x >> 5; c < 9; c += kWarps) {
    const float sx = d.sx[c], sy = d.sy[c];
    const uint32_t e0 = d.e0[c], e1 = d.e1[c], e2 = d.e2[c];
    for (uint32_t u = d.c0[c] + (threadIdx.x & 31); u < e2; u += 32) {
      float4 q = E[u];
      q.x -= sx;
      q.y -= sy;
      q.z -= u < e0 ? d.szl : (u < e1 ? d.szm : d.szh);
      E[u] = q;
    }
  }
}

// fp16 records and block z ranges of the stage, all threads of the CTA.  An
// atom with a non-finite coordinate (a simulation that has blown up) becomes a
// far atom, and makes the z range of its block NaN, which no window excludes.
// Far atoms have infinite or NaN records: no hit, or one that the exact test
// drops.
template <int NT, int kWarps>
__device__ __forceinline__ void make_records(Stage<NT> &d, float4 *E, uint2 *Hf, uint32_t *Ht, float *zb) {
  const uint32_t total = d.c0[9];
  const float cx = d.cx, cy = d.cy, cz = d.cz, sc = d.scale;
  float nmax = 0.f;
  for (uint32_t u = threadIdx.x; u < total + 8u; u += kWarps * 32) {
    const float4 q = E[u];
    const uint32_t xy = pack_half2((q.x - cx) * sc, (q.y - cy) * sc);
    const float2 r = unpack_half2(xy);
    const float zr = (q.z - cz) * sc, z = __half2float(__float2half_rn(zr));
    const float n = fmaf(r.x, r.x, fmaf(r.y, r.y, z * z));
    Hf[u] = make_uint2(xy, pack_half2(zr, n));
    if (NT > 1) {
      const uint32_t ty = (uint32_t)__float_as_int(q.w), one = ty & 1u ? 0x3c000000u : 0x3c00u;
      const uint32_t lo = ty < 2u ? one : 0u, hi = ty >= 2u && ty < 4u ? one : 0u;
      if (NT == 2)
        Ht[u] = lo;
      else
        reinterpret_cast<uint2 *>(Ht)[u] = make_uint2(lo, hi);
    }
    const float far = fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fabsf(q.z));
    if (far < 1e29f && !isnan(n))
      nmax = fmaxf(nmax, n);
    else
      E[u] = make_float4(kFar, kFar, kFar, q.w);
    const uint32_t k = u & 7u;
    // q.z - q.z is 0, or NaN where z is not finite
    if (k == 0u || k == 7u) zb[(u >> 3) * 2u + (k >> 2)] = q.z + (q.z - q.z);
  }
  const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(nmax));
  if ((threadIdx.x & 31) == 0) atomicMax(&d.nmax, m);
}

// Whether a home atom of the item lies out of the range of the fp16 records (far outside
// its cell); all threads of the CTA.  A norm out of that range is stored as infinity or
// as what it is.
template <int NT, int kWarps>
__device__ __noinline__ bool home_out_of_range(const Stage<NT> &d, const float4 *E, const uint2 *Hf) {
  bool out = false;
  for (uint32_t u = d.hb + threadIdx.x; u < d.hb + d.H; u += kWarps * 32)
    out = out || (unpack_half2(Hf[u].y).y > kMaxNorm && fabsf(E[u].x) < 1e29f);
  return __syncthreads_or(out);
}

// One tile of 16 home atoms (one warp); energy sums (pe, shifted pe, virial,
// pairs) are added to `ce`.
template <int NT, bool ENERGY, typename Acc, int MODE>
__device__ __forceinline__ void tile_forces(const ForceBufs &b, const Stage<NT> &d,
                                            const float4 *E, const uint2 *Hf, const uint32_t *Ht,
                                            const float *zb, uint32_t tile, uint32_t *tab, double *ce) {
  constexpr bool kSum32 = std::is_same<Acc, float>::value;
  const int lane = threadIdx.x & 31;
  const uint32_t g = (uint32_t)lane >> 2, t = (uint32_t)lane & 3u;
  const uint32_t H = d.H, h0 = tile * kTile, hb = d.hb + h0;
  // home atoms of this lane: rows g and g + 8 of the mma hold the neighbouring
  // atoms 2 g and 2 g + 1 of the tile, which share most of their candidates
  const bool va = h0 + 2 * g < H, vb = h0 + 2 * g + 1 < H;
  const uint32_t sa = hb + (va ? 2 * g : 0u), sb = hb + (vb ? 2 * g + 1 : 0u);
  float4 pa = E[sa], pb = E[sb];
  if (!va) pa.x = pa.y = pa.z = kNoAtom;
  if (!vb) pb.x = pb.y = pb.z = kNoAtom;
  // the particle index of the force store, fetched now so that its latency
  // passes during the pair loops (lane t = 0 stores atom a, t = 1 atom b)
  const uint32_t pi = (t == 0 && va) || (t == 1 && vb)
                          ? __ldg(b.pid + d.home_g0 + h0 + 2 * g + t) : 0u;

  // operands of the distance product: A rows (-2 x, -2 y, -2 z, 1), C the
  // rows' squared norm less the bound
  const uint2 ha = Hf[sa], hbv = Hf[sb];
  uint32_t a0 = 0u, a1 = 0u;
  float C[4];
  {
    const float2 axy = unpack_half2(ha.x), bxy = unpack_half2(hbv.x);
    const float az = unpack_half2(ha.y).x, bz = unpack_half2(hbv.y).x;
    if (t == 0) {
      a0 = pack_half2(-2.f * axy.x, -2.f * axy.y);
      a1 = pack_half2(-2.f * bxy.x, -2.f * bxy.y);
    } else if (t == 1) {
      a0 = pack_half2(-2.f * az, 1.f);
      a1 = pack_half2(-2.f * bz, 1.f);
    } else if (NT > 1) {
      const uint2 ca = d.cut[__float_as_int(pa.w)], cb = d.cut[__float_as_int(pb.w)];
      a0 = t == 2 ? ca.x : ca.y;
      a1 = t == 2 ? cb.x : cb.y;
    }
    // bound of a home atom: a partner within rc lies at most rc farther from the centre, at
    // `far`; rounding the two records moves the points by at most 2^-10 far, and the
    // stored norm by 2^-11 far^2 (5 % more of both, and 1e-4 in rs2, for the sums' own
    // rounding).  No atom farther away widens it.
    const auto row = [&](float n) {
      const float far = sqrt_approx(n) + d.rs;
      return n - fmaf(far, fmaf(far, 1.05f * (1.0f / 2048.0f + 1.0f / 1048576.0f), d.rs_dl), d.rs2);
    };
    C[0] = C[1] = va ? row(fmaf(axy.x, axy.x, fmaf(axy.y, axy.y, az * az))) : kFar;
    C[2] = C[3] = vb ? row(fmaf(bxy.x, bxy.x, fmaf(bxy.y, bxy.y, bz * bz))) : kFar;
  }
  const uint32_t eb = smem_u32(E) + 32u * t;  // candidate 2 t of a block
  // B operand: candidate g; lanes t >= 2 hold its type indicators (one type:
  // their A operand is zero, and they repeat the record)
  const bool types = NT > 1 && t >= 2;
  const uint32_t stride = types ? type_bytes(NT) : 8u;
  const uint32_t hbase = (types ? smem_u32(Ht) : smem_u32(Hf)) + stride * g +
                         (stride == 8u ? 4u * (t & 1u) : 0u);
  const uint32_t tb = smem_u32(tab);
  const uint32_t lbase = tb + kTabBytes + 2u * (uint32_t)lane;   // this lane's list, entry k at + 64 k
  const uint32_t far = d.c0[9];

  PairAcc<NT, ENERGY, Acc, MODE> acca, accb;
  Force2 acc;
  const float2 m1 = make_float2(-1.0f, -1.0f);
  const int ta = NT == 1 ? 0 : __float_as_int(pa.w) * NT;
  const int tbt = NT == 1 ? 0 : __float_as_int(pb.w) * NT;
  float2 s2 = make_float2(d.lj.s2[0], d.lj.s2[0]);
  float2 e24 = make_float2(d.lj.e24[0], d.lj.e24[0]);
  float2 e4 = make_float2(d.lj.e4[0], d.lj.e4[0]);
  uint32_t rca = less_1(d.lj.rc2[0]), rcb = rca;  // bits of rc^2, less one
  float4 l0a, l1a, l0b, l1b;
  if (NT == 2) {
    l0a = d.lj4[ta];
    l1a = d.lj4[ta + 1];
    l0b = d.lj4[tbt];
    l1b = d.lj4[tbt + 1];
  }

  // the tile's z window (all z when its first atom is a far one, or the columns are not
  // sorted: check_order)
  const float z0 = E[hb].z, z1 = E[hb + min((uint32_t)kTile, H - h0) - 1].z;
  const float zlo = z0 < 1e29f ? z0 - d.rcw : -kFar, zhi = z1 + d.rcw;
  const uint32_t blocks = d.c0[9] >> 3;
  for (uint32_t blk = 0; blk < blocks;) {
    // table: first slots of the blocks in the window; far blocks pad it to a
    // multiple of 4
    __syncwarp();
    uint32_t nt = 0;
    for (; blk < blocks && nt <= (uint32_t)kTabBlocks - 36u; blk += 32) {
      const uint32_t i = blk + (uint32_t)lane;
      const float2 z = reinterpret_cast<const float2 *>(zb)[min(i, blocks)];
      const bool in = i < blocks && !(z.y < zlo) && !(z.x > zhi);
      const uint32_t m = __ballot_sync(0xffffffffu, in);
      if (in) tab[nt + __popc(m & ((1u << lane) - 1u))] = 8u * i;
      nt += __popc(m);
    }
    const uint32_t cb4 = (nt + 3u) & ~3u;
    if (lane < 4 && nt + lane < cb4) tab[nt + lane] = far;
    __syncwarp();
    uint32_t u = 0;
    do {
      // phase 1: until all blocks are tested or some lane's list is nearly full
      uint32_t oa = lbase;
      for (; u < cb4; u += 4) {
        if (__any_sync(0xffffffffu, oa > lbase + 64u * (list_len(NT) - 8u))) break;
        const uint4 o4 = lds_u4(tb + 4u * u);
        const uint32_t o[4] = {o4.x, o4.y, o4.z, o4.w};
        uint32_t B[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) B[j] = lds_stage(hbase + (NT == 2 ? stride : 8u) * o[j]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float D[4];
          mma_16x8x8(D, a0, a1, B[j], C);
          if ((__float_as_uint(D[0]) | __float_as_uint(D[2])) & 0x80000000u) {
            sts_u16(oa, o[j]);
            oa += 64u;
          }
          if ((__float_as_uint(D[1]) | __float_as_uint(D[3])) & 0x80000000u) {
            sts_u16(oa, o[j] + 1u);
            oa += 64u;
          }
        }
      }
      __syncwarp();
      // phase 2: the exact pairs of every hit; a lane past its last one takes a far atom
      // (two per round, for independent work)
      const uint32_t lend =
          lbase + 64u * ((__reduce_max_sync(0xffffffffu, (oa - lbase) >> 6) + 1u) & ~1u);
      for (uint32_t la = lbase; la < lend; la += 128u) {
        float4 q[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t e = la + 64u * j < oa ? lds_u16(la + 64u * j) : far;
          q[j] = lds_f4(eb + 16u * e);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 dx = make_float2(pa.x - q[j].x, pb.x - q[j].x);
          const float2 dy = make_float2(pa.y - q[j].y, pb.y - q[j].y);
          const float2 dz = make_float2(pa.z - q[j].z, pb.z - q[j].z);
          const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
          const int tj = NT == 1 ? 0 : __float_as_int(q[j].w);
          if (NT == 2) {
            // both candidate types' parameters wait in registers
            const bool k = tj != 0;
            s2 = make_float2(k ? l1a.x : l0a.x, k ? l1b.x : l0b.x);
            e24 = make_float2(k ? l1a.y : l0a.y, k ? l1b.y : l0b.y);
            rca = __float_as_uint(k ? l1a.z : l0a.z);
            rcb = __float_as_uint(k ? l1b.z : l0b.z);
          } else if (NT > 2) {
            const float4 la = d.lj4[ta + tj], lb = d.lj4[tbt + tj];
            s2 = make_float2(la.x, lb.x);
            e24 = make_float2(la.y, lb.y);
            rca = __float_as_uint(la.z);
            rcb = __float_as_uint(lb.z);
          }
          const bool ina = inside(r2.x, rca), inb = inside(r2.y, rcb);
          float2 f, r2c = r2, sr6;
          if constexpr (MODE == kModeSoftCore) {
            f = sr6 = make_float2(0.0f, 0.0f);
            if (ina || inb)  // (short ranges: seldom in any lane)
              f = make_float2(soft_core(d.lj, r2.x), soft_core(d.lj, r2.y));
          } else {
            if (MODE == kModeCapped) {
              const float2 fl = __fmul2_rn(make_float2(0.25f, 0.25f), s2);
              r2c = make_float2(fmaxf(r2.x, fl.x), fmaxf(r2.y, fl.y));
            }
            const float2 inv = make_float2(rcp_approx(r2c.x), rcp_approx(r2c.y));
            const float2 sr2 = __fmul2_rn(s2, inv);
            sr6 = __fmul2_rn(__fmul2_rn(sr2, sr2), sr2);
            const float2 tt = __ffma2_rn(__fadd2_rn(e24, e24), sr6, make_float2(-e24.x, -e24.y));
            f = __fmul2_rn(__fmul2_rn(tt, sr6), inv);
          }
          f.x = ina ? f.x : 0.0f;
          f.y = inb ? f.y : 0.0f;
          if constexpr (kSum32) {
            acc.fx = __ffma2_rn(f, dx, acc.fx);
            acc.fy = __ffma2_rn(f, dy, acc.fy);
            acc.fz = __ffma2_rn(f, dz, acc.fz);
          } else {
            const float2 gx = __fmul2_rn(f, dx), gy = __fmul2_rn(f, dy), gz = __fmul2_rn(f, dz);
            acca.fx += (Acc)gx.x;
            acca.fy += (Acc)gy.x;
            acca.fz += (Acc)gz.x;
            accb.fx += (Acc)gx.y;
            accb.fy += (Acc)gy.y;
            accb.fz += (Acc)gz.y;
          }
          if (ENERGY) {
            const int ka = ta + tj, kb = tbt + tj;
            if (NT > 1) e4 = make_float2(d.lj.e4[ka], d.lj.e4[kb]);
            float2 u = __fmul2_rn(__fmul2_rn(e4, sr6), __fadd2_rn(sr6, m1));
            u.x = ina ? u.x : 0.0f;
            u.y = inb ? u.y : 0.0f;
            // (a pair's half share is taken at the end: a power of two)
            acca.pe += (Acc)u.x;
            accb.pe += (Acc)u.y;
            if (NT > 1) {  // one type: from pe and the count, at the end
              acca.pes += (Acc)(ina ? u.x - d.lj.ush[ka] : 0.0f);
              accb.pes += (Acc)(inb ? u.y - d.lj.ush[kb] : 0.0f);
            }
            // f is zero outside the cutoff, where r^2 may be +inf
            acca.vir += (Acc)(ina ? f.x * r2c.x : 0.0f);
            accb.vir += (Acc)(inb ? f.y * r2c.y : 0.0f);
            acca.n += (uint32_t)ina + (uint32_t)inb;
          }
        }
      }
    } while (u < cb4);
  }
  // the 4 lanes of an atom
  using Sum = typename std::conditional<kSum32, float, Acc>::type;
  Sum v[6] = {(Sum)acca.fx, (Sum)acca.fy, (Sum)acca.fz, (Sum)accb.fx, (Sum)accb.fy, (Sum)accb.fz};
  if constexpr (kSum32) {
    v[0] = acc.fx.x;
    v[1] = acc.fy.x;
    v[2] = acc.fz.x;
    v[3] = acc.fx.y;
    v[4] = acc.fy.y;
    v[5] = acc.fz.y;
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    v[k] += __shfl_xor_sync(0xffffffffu, v[k], 1);
    v[k] += __shfl_xor_sync(0xffffffffu, v[k], 2);
  }
  if (t == 0 && va) b.F[pi] = make_float4((float)v[0], (float)v[1], (float)v[2], 0.0f);
  if (t == 1 && vb) b.F[pi] = make_float4((float)v[3], (float)v[4], (float)v[5], 0.0f);
  if (ENERGY) {
    double e[4] = {warp_sum((double)(acca.pe + accb.pe)), warp_sum((double)(acca.pes + accb.pes)),
                   warp_sum((double)(acca.vir + accb.vir)), (double)warp_sum(acca.n + accb.n)};
    // (the same sum when the system runs beside others of more types)
    if (NT == 1 || d.one) e[1] = e[0] - e[3] * (double)d.lj.ush[0];
    for (int k = 0; k < 3; ++k) e[k] *= 0.5;
    if (lane == 0)
      for (int k = 0; k < 4; ++k) ce[k] += e[k];
  }
}

// Global-memory path of an item whose stage does not fit: task t covers the
// groups of 32 consecutive home atoms t, t + ntask, ...; lanes are atoms.
template <int NT, bool ENERGY, typename Acc, int MODE>
__device__ __noinline__ void task_global(const ForceBufs &b, const Stage<NT> &d, uint32_t t,
                                         uint32_t ntask, double *ce) {
  const int lane = threadIdx.x & 31;
  const int nseg = d.nseg, z0 = d.z0, nz = d.nz;
  const uint32_t H = d.H;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (uint32_t gi = t; gi * 32 < H; gi += ntask) {
    const uint32_t h = gi * 32 + lane;
    const bool valid = h < H;
    const uint32_t gh = d.home_g0 + (valid ? h : H - 1);
    // home cell (staged index k in [1, nseg]) of this lane, and the warp's span
    int lo = 1, hi = nseg;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (b.start[d.kbase[4] + (uint32_t)(z0 - 1 + mid)] <= gh) lo = mid; else hi = mid - 1;
    }
    const int kmin = __reduce_min_sync(0xffffffffu, lo);
    const int kmax = __reduce_max_sync(0xffffffffu, lo);
    const float4 p = b.rs[gh];
    const float xi = p.x - d.sx[4], yi = p.y - d.sy[4], zi = p.z - d.szm;
    const int ti = NT == 1 ? 0 : __float_as_int(p.w);
    PairAcc<NT, ENERGY, Acc, MODE> acc;
    for (int c = 0; c < 9; ++c) {
      if (!d.periodic && d.kbase[c] == kNoCell) continue;  // no column past an open face
      const float sx = d.sx[c], sy = d.sy[c];
      for (int k = kmin - 1; k <= kmax + 1; ++k) {
        const int zr = z0 - 1 + k, zc = (zr + nz) % nz;
        if (!d.periodic && (zr < 0 || zr >= nz)) continue;
        const uint32_t key = d.kbase[c] + (uint32_t)zc;
        const float sz = zr < 0 ? d.szl : (zr >= nz ? d.szh : d.szm);
        if (c == 4)
          global_range<NT, ENERGY, true, Acc, MODE>(b.rs, b.start[key], b.start[key + 1], xi, yi,
                                                    zi, ti, sx, sy, sz, gh, d.lj, acc);
        else
          global_range<NT, ENERGY, false, Acc, MODE>(b.rs, b.start[key], b.start[key + 1], xi,
                                                     yi, zi, ti, sx, sy, sz, 0, d.lj, acc);
      }
    }
    if (valid) b.F[b.pid[gh]] = make_float4((float)acc.fx, (float)acc.fy, (float)acc.fz, 0.0f);
    if (ENERGY) {
      s[0] += warp_sum(valid ? (double)acc.pe : 0.0);
      s[1] += warp_sum(valid ? (double)acc.pes : 0.0);
      s[2] += warp_sum(valid ? (double)acc.vir : 0.0);
      s[3] += (double)warp_sum(valid ? acc.n : 0u);
    }
  }
  if (ENERGY && lane == 0)
    for (int k = 0; k < 4; ++k) ce[k] += s[k];
}

// ---- the kernel ---------------------------------------------------------------

template <int NT, bool ENERGY, typename Acc, int kWarps, int MODE>
__global__ void __launch_bounds__(kWarps * 32,
                                  (NT == 1 && !ENERGY && std::is_same<Acc, float>::value && MODE != kModeSoftCore ? 32 : 24) / kWarps)
    k_force(const __grid_constant__ ForceBufs b) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ Stage<NT> d;
  __shared__ uint64_t full;
  __shared__ double cle[ENERGY ? kWarps : 1][4];  // energy sums of the warps
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const ForceItem &it = b.items[blockIdx.x];
  const uint32_t sys = it.sys;
  // what no kernel of a step writes is read ahead of the wait for the cell build
  if (warp == 1) {
    plan_frame<NT>(b, it, d);
  } else if (warp == 2) {
    load_lj<NT, MODE>(b, b.sys[sys], d);
  } else if (threadIdx.x == 0) {
    mbar_init(&full, 1);
    mbar_fence_init();
  }
  pdl_enter();
  if (b.steps_left != nullptr && b.steps_left[sys] == 0) {
    // a system whose step budget is spent keeps its state
    if (ENERGY && threadIdx.x < 4) b.partials[(size_t)blockIdx.x * 4 + threadIdx.x] = 0.0;
    return;
  }
  const uint32_t slots = padded_slots((uint32_t)b.cap);
  float4 *E = reinterpret_cast<float4 *>(smem_raw);
  uint2 *Hf = reinterpret_cast<uint2 *>(smem_raw + (size_t)slots * 16u);
  uint32_t *Ht = reinterpret_cast<uint32_t *>(smem_raw + (size_t)slots * 24u);
  float *zb = reinterpret_cast<float *>(smem_raw + (size_t)slots * (slot_bytes(NT) - 1u));
  uint32_t *tab = reinterpret_cast<uint32_t *>(smem_raw + (size_t)slots * slot_bytes(NT)) +
                  warp * (warp_bytes(NT) / 4);
  if (warp == 0) {
    __syncwarp();
    plan_stage<NT>(b, it, d, E, &full);
  } else if (warp == 2) {
    check_order<NT>(b, it, d);
  }
  __syncthreads();
  if (!d.overflow) {
    bool ok = lane != 0 || mbar_wait_or_abort(&full, 0u, &kNeverAbort,
                                              b.wait_polls ? b.wait_polls : kWaitPolls);
    ok = __syncthreads_and(ok);
    if (!ok) {
      // the copies did not arrive: report it, and give them one more bounded
      // wait before the shared memory they write is released
      if (threadIdx.x == 0) {
        atomicOr(&b.status[sys], kStatusWaitTimeout);
        if (!(b.test_flags & 1u)) mbar_wait_bounded(&full, 0u);
      }
      // not what an earlier call left there
      if (ENERGY && threadIdx.x < 4) b.partials[(size_t)blockIdx.x * 4 + threadIdx.x] = 0.0;
      return;
    }
    if (d.shifted) {
      shift_stage<NT, kWarps>(d, E);
      __syncthreads();
    }
    make_records<NT, kWarps>(d, E, Hf, Ht, zb);
    __syncthreads();
  }
  // home atoms out of the range of fp16 records (far outside their cells): global path
  const bool global =
      d.overflow || (__uint_as_float(d.nmax) > kMaxNorm && home_out_of_range<NT, kWarps>(d, E, Hf));
  const uint32_t ntile = d.ntile;
  double *ce = cle[ENERGY ? warp : 0];
  if (ENERGY && lane == 0)
    for (int k = 0; k < 4; ++k) ce[k] = 0.0;
  for (uint32_t k = warp; k < ntile; k += kWarps) {
    if (!global)
      tile_forces<NT, ENERGY, Acc, MODE>(b, d, E, Hf, Ht, zb, k, tab, ce);
    else
      task_global<NT, ENERGY, Acc, MODE>(b, d, k, ntile, ce);
  }
  if (ENERGY) {  // the item's sums in the order of its warps
    __syncthreads();
    if (threadIdx.x < 4) {
      double v = 0.0;
      for (int k = 0; k < kWarps; ++k) v += cle[k][threadIdx.x];
      b.partials[(size_t)blockIdx.x * 4 + threadIdx.x] = v;
    }
  }
}

// Warps of a CTA: the default, and a small one.
constexpr int kWarpsDefault = 8, kWarpsSmall = 4;

template <int NT, bool E, typename Acc, int kWarps, int MODE = kModeLJ>
cudaError_t launch_w(const ForceBufs &b, cudaStream_t s) {
  const size_t smem = smem_bytes((uint32_t)b.cap, kWarps, NT);
  auto kern = k_force<NT, E, Acc, kWarps, MODE>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  return launch_pdl(kern, dim3(b.nitems), dim3(kWarps * 32), smem, s, b);
}

template <int NT, bool E, typename Acc>
cudaError_t launch_t(const ForceBufs &b, int threads, cudaStream_t s) {
  return threads == 128 ? launch_w<NT, E, Acc, kWarpsSmall>(b, s)
                        : launch_w<NT, E, Acc, kWarpsDefault>(b, s);
}

template <int NT>
cudaError_t launch_nt(const ForceBufs &b, bool energy, bool acc64, int threads, cudaStream_t s) {
  if (energy) {
    return acc64 ? launch_t<NT, true, double>(b, threads, s)
                 : launch_t<NT, true, float>(b, threads, s);
  }
  return acc64 ? launch_t<NT, false, double>(b, threads, s)
               : launch_t<NT, false, float>(b, threads, s);
}

template <int MODE>
cudaError_t launch_mode(const ForceBufs &b, int nt_max, cudaStream_t s) {
  if (b.nitems == 0) return cudaSuccess;
  switch (nt_max) {
    case 1: return launch_w<1, false, float, kWarpsDefault, MODE>(b, s);
    case 2: return launch_w<2, false, float, kWarpsDefault, MODE>(b, s);
    case 3: case 4: return launch_w<4, false, float, kWarpsDefault, MODE>(b, s);
    default: return launch_w<8, false, float, kWarpsDefault, MODE>(b, s);
  }
}

}  // namespace

int force_max_segment() { return kMaxSeg; }

int force_max_capacity() {
  // largest staged-atom capacity whose shared memory fits one CTA
  uint32_t cap = 64;
  while (smem_bytes(cap + 64, kWarpsDefault, kMaxTypes) <= 180u * 1024u) cap += 64;
  return (int)cap;
}

// Static shared memory of a CTA, at most: the stage record, and the energy sums.
static int static_bytes(int nt, bool energy) {
  const size_t st = nt <= 1 ? sizeof(Stage<1>) : nt <= 2 ? sizeof(Stage<2>)
                    : nt <= 4 ? sizeof(Stage<4>) : sizeof(Stage<8>);
  return (int)st + (energy ? kWarpsDefault : 1) * 4 * 8 + 64;
}

int force_smem_per_cta(int cap, int nt) {
  // (1.5 KB over the stage record: runs that would fill the last of it leave a stage no
  // headroom)
  return (int)smem_bytes((uint32_t)cap, kWarpsDefault, nt) + static_bytes(nt, false) + 1536;
}

int force_smem_limit(int nt) {
  // the CTAs per SM that the registers allow (one type 4, several 3) share its
  // 228 KB, less 1 KB per CTA reserved by the driver
  return (nt <= 1 ? 56 : 74) * 1024;
}

int force_capacity_room(int nt) {
  // With one type the launches with energies have fewer CTAs per SM by their registers and
  // more shared memory each; and a one-type system may run beside systems of many types,
  // whose slots are larger.
  const auto fits = [](uint32_t cap, int k, bool energy) {
    return (int)smem_bytes(cap, kWarpsDefault, k) + static_bytes(k, energy) <= force_smem_limit(k);
  };
  uint32_t cap = 64;
  while (fits(cap + 16, nt, nt > 1) && (nt > 1 || fits(cap + 16, kMaxTypes, false))) cap += 16;
  return (int)cap;
}

cudaError_t launch_force_capped(const ForceBufs &b, int nt_max, cudaStream_t s) {
  return launch_mode<kModeCapped>(b, nt_max, s);
}

cudaError_t launch_force_softcore(const ForceBufs &b, int nt_max, cudaStream_t s) {
  return launch_mode<kModeSoftCore>(b, nt_max, s);
}

cudaError_t launch_force(const ForceBufs &b, int nt_max, bool energy, bool acc64,
                         int block_threads, cudaStream_t s) {
  if (b.nitems == 0) return cudaSuccess;
  switch (nt_max) {
    case 1: return launch_nt<1>(b, energy, acc64, block_threads, s);
    case 2: return launch_nt<2>(b, energy, acc64, block_threads, s);
    case 3: case 4: return launch_nt<4>(b, energy, acc64, block_threads, s);
    default: return launch_nt<8>(b, energy, acc64, block_threads, s);
  }
}

}  // namespace pb
