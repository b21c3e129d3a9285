// Barnes-Hut walk + Hernquist halo + kick-drift (+ star formation) on sm_100a.
//
// Semantics follow `main` in src/physics/shaders/nbody_bh.wgsl:64-181 per
// particle: own-leaf density, softened opening test
//   accept  <=>  size^2 < theta^2 (r^2 + eps^2)  ||  size^2 < eps^2 / 4,
// monopole G M r / (r^2 + eps^2)^(3/2), leaf direct sum with j != i, halo,
// v += a dt, gas drag, x += v dt, pad and specific-energy writes.
//
// Execution is warp-cooperative: a warp owns 32 Morton-consecutive particles
// (one per lane) and walks the union of their frontiers, but each lane applies
// exactly its own particle's acceptance decisions (a lane is active for a node
// only if it opened every ancestor), so the per-particle interaction set equals
// the reference's thread-per-particle stack walk.
//   * The stack holds child ranges (children of a BFS node are contiguous) with
//     the mask of lanes that opened the parent. Each round pops up to four
//     ranges and stages their children into shared memory by one coalesced load
//     (one child per lane, structure of arrays), so the round's stack, ballot and
//     staging work is shared by up to 32 children.
//   * Children are tested two at a time with sm_100's packed FP32x2 FMA/ADD/MUL;
//     accumulation is predicated, not branched (a child a lane does not take gets
//     r^2 + eps^2 = +inf, so rsqrt gives 0).
//   * Opened leaves are queued and summed in windows of up to 96 source pairs, by
//     subgroups of 8 particles with 4 lanes each (leaf_flush).
//   * Warps are persistent and take work items from an atomic counter (load
//     balance across the dense core); per-item FP64 partials of the
//     diagnostics replace a block-wide barrier.
//   * Walk group size: a work item is 32, 16, 8 or 4 Morton-consecutive
//     particles (LPP = 1, 2, 4 or 8 lanes per particle). With LPP > 1 the lanes of a
//     particle split the round's slot pairs between them (items of 8 or 4 also the
//     leaf pairs) and add their partial sums by shuffles at the end, so a
//     small galaxy keeps more warps busy and each warp walks the union of
//     fewer frontiers. A 32-particle walk group (layout, diagnostics) holds LPP
//     items. The split changes the order of the force sums, so results change
//     at the rounding level (inside the force tolerance) between group sizes;
//     each galaxy carries its own LPP, so it gets the same arithmetic alone or
//     in a pool.
//   * Over a batch, every group belongs to one galaxy and walks that galaxy's
//     tree with its own Params; warps steal groups across all galaxies.
//   * Walk split (one galaxy): a small galaxy's walk is as long as its densest
//     work item. With wsplit = S > 1 each item is walked by S warps over
//     disjoint parts of the tree (the nodes of one level dealt out in turn, with
//     their subtrees; the levels above belong to part 0), and the last of the S
//     to finish adds their sums in part order and integrates. Every interaction
//     happens once, as in the unsplit walk; only the order of the sums changes.
#pragma once
#include "common.cuh"

namespace gs {

constexpr int kWalkThreads = 128;
constexpr int kWalkWarps = kWalkThreads / 32;
constexpr int kPartials = 6;  // e_diag, e_true, px, py, pz, mass
#ifndef GS_WALK_RANGES
#define GS_WALK_RANGES 4
#endif
constexpr int kWalkRanges = GS_WALK_RANGES;  // child ranges popped and tested per round (1..4)
static_assert(kWalkRanges >= 1 && kWalkRanges <= 4, "a round stages at most one child per lane");
// ranges; a round explores kWalkRanges paths, each leaving <= 7 pending ranges per depth
constexpr int kWalkStack = 8 * 11 * kWalkRanges;
// Resident blocks per SM the walk is compiled for. Walk groups of 32: 7, the most that 31.7
// KB of staging per block let onto an SM, at 72 registers per thread (6 at 80 registers:
// walk of 524288 particles 953 -> 968 us; compensated sums need the 80: 306 -> 290 us on a
// sphere of 200003). Smaller groups walk small galaxies, which do not fill the SMs, and
// run with fewer spills and more loads in flight at more registers: full step at 7 / 6
// / 5 blocks in us: 4096 particles 62.1 / 61.2 / 60.0, 16384 106.0 / 101.1 / 101.8, 25000 133 / 131 / 124
// (groups of 8); 60001 163 / 157 / 164, 100000 310 / 308 / 303 (groups of 16). The launch
// tuning accepts 1..8 blocks per SM; no more are launched than the resident ones.
constexpr int kWalkBlocksPerSM = 8;  // the tuning's largest value
constexpr int kWalkResident = 7;
template <int LPP, bool COMP>
constexpr int walk_resident() {
  return LPP >= 4 ? 5 : LPP == 2 || COMP ? 6 : kWalkResident;
}
constexpr uint32_t kWalkGroup = 32;             // particles per walk group (layout, diagnostics)
constexpr uint32_t kWalkParts = 8;              // partial-sum slots per walk group (the largest LPP)
// with the walk group chosen by size, galaxies of at most this many particles
// walk in groups of 8 / 16 particles (measured crossovers of the step time on a
// B200 with the split below: 8 is fastest up to 32768 particles, 16 at 65536,
// 16 and 32 tie at 131072, 32 from 150000 on)
constexpr uint32_t kWalkAuto8 = 45000;
constexpr uint32_t kWalkAuto16 = 100000;
// a split walk splits at the first tree level of at least this many nodes per split
constexpr uint32_t kSplitMinNodes = 4;
// with the walk split chosen by size, a lone galaxy of at most this many
// particles walks each work item in 4 / 2 parts (measured: 4 parts fastest at
// 4096-8192 particles, 2 and 4 tie at 16384, none from 32768 on)
constexpr uint32_t kSplitAuto4 = 12000;
constexpr uint32_t kSplitAuto2 = 24000;

// nbody_bh.wgsl:206-213
__device__ inline uint32_t pcg(uint32_t v0) {
  uint32_t v = v0 * 747796405u + 2891336453u;
  v = ((v >> ((v >> 28u) + 4u)) ^ v) * 277803737u;
  return (v >> 22u) ^ v;
}
__device__ inline float rand01(uint32_t i, uint32_t salt) {
  return __fdiv_rn(__uint2float_rn(pcg(i ^ (salt * 0x9E3779B9u))), 4294967296.0f);
}
// nbody_bh.wgsl:216-227 (Kroupa inverse CDF)
__device__ inline float imf_sample(float u1, float u2) {
  const float a0 = powf(0.08f, -0.3f), b0 = powf(0.5f, -0.3f);
  const float lowInt = __fdiv_rn(__fsub_rn(a0, b0), 0.3f);
  const float a1 = powf(0.5f, -1.3f), b1 = powf(100.0f, -1.3f);
  const float hiInt = __fdiv_rn(__fmul_rn(0.5f, __fsub_rn(a1, b1)), 1.3f);
  if (u1 < __fdiv_rn(lowInt, __fadd_rn(lowInt, hiInt)))
    return powf(__fsub_rn(a0, __fmul_rn(u2, __fsub_rn(a0, b0))), -1.0f / 0.3f);
  return powf(__fsub_rn(a1, __fmul_rn(u2, __fsub_rn(a1, b1))), -1.0f / 1.3f);
}
__device__ inline uint32_t wgsl_u32(float x) {
  if (!(x > 0.0f)) return 0u;
  if (x >= 4294967296.0f) return 0xffffffffu;
  return (uint32_t)x;
}

// star_formation (nbody_bh.wgsl:229-268) on one particle, in registers.
// p1 = (vel, pad), s = stellar record.
__device__ inline void star_formation_one(const gs_params& P, uint32_t i, float4& p1, float4& s) {
  const uint32_t salt = wgsl_u32(__fmul_rn(P.time, 977.0f)) + 1u;
  if (p1.w < -0.5f) {
    const float density = __fsub_rn(-p1.w, 1.0f);
    if (density > P.sfDensity && P.sfEff > 0.0f) {
      const float prob = __fmul_rn(__fmul_rn(P.sfEff, P.sfDt),
                                   fminf(__fsqrt_rn(__fdiv_rn(density, fmaxf(P.sfDensity, 1e-6f))), 3.0f));
      if (rand01(i, salt) < prob) {
        const float m = imf_sample(rand01(i, salt + 7u), rand01(i, salt + 13u));
        s = make_float4(m, __fmul_rn(P.time, P.agingRate), rand01(i, salt + 29u), 0.0f);
        p1.w = 0.0f;
      }
    }
  } else if (s.x >= 8.0f) {
    const float ageMyr = __fsub_rn(__fmul_rn(P.time, P.agingRate), s.y);
    const float tMS = __fmul_rn(10000.0f, powf(s.x, -2.5f));
    const float tGiant = __fadd_rn(__fmul_rn(tMS, 0.12f), 15.0f);
    if (ageMyr > __fadd_rn(__fadd_rn(__fadd_rn(tMS, tGiant), 15.0f), 30.0f)) {
      s = make_float4(-1.0f, 0.0f, s.z, 0.7f);
      p1.w = -1.0f;
      p1.x = __fadd_rn(p1.x, __fmul_rn(__fsub_rn(rand01(i, salt + 41u), 0.5f), 2.0f));
      p1.y = __fadd_rn(p1.y, __fmul_rn(__fsub_rn(rand01(i, salt + 43u), 0.5f), 2.0f));
      p1.z = __fadd_rn(p1.z, __fmul_rn(__fsub_rn(rand01(i, salt + 47u), 0.5f), 2.0f));
    }
  }
}

struct WalkArgs {
  const float4* __restrict__ pin;   // 2 float4 per particle, tree (sorted) order
  float4* __restrict__ pout;
  float4* __restrict__ stellar;     // in place, used when SF is fused
  const float4* __restrict__ cm;    // node com.xyz, mass
  const WalkInfo* __restrict__ info;
  DevState* st;                     // per-slot states
  float* __restrict__ energy;       // e_i
  float4* __restrict__ dbg_acc;     // optional {ax, ay, az, phi} (G applied)
  float* __restrict__ dbg_dens;
  double* __restrict__ partials;    // [walk items][kPartials], a galaxy's from its SegDesc item0
  unsigned* work;                   // [0] next group, [1] finished warps (self-resetting)
  Layout L;                         // galaxies and the group -> galaxy map
  uint32_t pool_n, node_pool;       // particle and node pool sizes (memory-safety bounds)
  SegDesc seg0;                     // the only galaxy, for the one-galaxy instantiation
  // split walks (one galaxy, seg0.wsplit > 1): the tree levels of the split, the
  // per-split partial sums [3][wsplit][split_stride] (float4: ax pair, ay pair;
  // az pair, potential pair; density, self weight) and the arrivals per work item
  const TreeMeta* meta;
  float4* split_buf;
  unsigned* split_arrive;           // zero between launches (the last arrival resets it)
  uint32_t split_stride;
};

// Opened leaves wait in a per-warp queue until they hold kLeafFlush source pairs
// (or the walk ends); their direct sums then run over windows of up to
// kLeafWindow staged pairs (see leaf_flush).
#ifndef GS_LEAF_WINDOW
#define GS_LEAF_WINDOW 96
#endif
#ifndef GS_LEAF_FLUSH
#define GS_LEAF_FLUSH 72
#endif
constexpr int kLeafWindow = GS_LEAF_WINDOW;
constexpr int kLeafFlush = GS_LEAF_FLUSH;
constexpr uint32_t kLeafMax = 16;  // particles of a queued leaf (larger ones are summed at once)
static_assert(kLeafWindow % 32 == 0 && kLeafWindow <= 128, "a lane stages whole pairs; 7-bit pair indices");
// a queue entry packs the first particle and the count: particle indices have 27 bits
constexpr int kLeafCountShift = 27;

// Per-warp shared staging.
struct WalkSmem {
  // {first child | (count-1) << 29, lane mask}, above kWalkRanges empty entries (mask
  // 0) that a round reads when fewer ranges are left
  uint2 stack[kWalkRanges + kWalkStack];
  uint2 q[kLeafFlush + 32];         // opened leaves: {first | (count-1) << 27, opening mask}
  union {
    struct {
      // staged child ranges, pair-interleaved so a packed test reads two 128-bit
      // words: cxy[4p..4p+3] = {x(2p), x(2p+1), y(2p), y(2p+1)}, czm likewise {z, m}
      __align__(16) float cxy[16 * kWalkRanges];
      __align__(16) float czm[16 * kWalkRanges];
      float cthr[8 * kWalkRanges];  // accepted where r^2 + eps^2 (groups of 32) or theta^2 times it is larger
    };
    uint2 pinfo[kLeafWindow];       // a window's source pairs: {first source | both << 31, opening mask}
  };
  // staged leaf sources, pair-interleaved the same way
  __align__(16) float lxy[4 * kLeafWindow];
  __align__(16) float lzm[4 * kLeafWindow];
  // the window's pairs of one subgroup: byte offset of the pair in lxy | opening mask << 24
  uint32_t list[kLeafWindow + 4];
};

// Reciprocal square root for the walk's r^2 + eps^2, which is never subnormal
// (eps^2 is zero or at least the smallest normal float, and zero softening adds
// that smallest normal instead): the flush-to-zero form gives the same result as
// rsqrtf there and issues fewer instructions.
__device__ __forceinline__ float rsqrt_walk(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ inline float2 f2(float a) { return make_float2(a, a); }

// Packed sums of a particle: acceleration / G and sum of m / r.
struct Sums {
  float2 ax, ay, az, pt;
};

// One packed step of a direct sum (nbody_bh.wgsl:117-131): the two staged sources
// of the pair whose {x, x, y, y} lie `at` bytes into lxy against the particle at -p,
// with e0 and e1 the softening each source gets (+inf: r^2 + eps^2 is +inf, rsqrt
// gives 0 and every term vanishes, as r is finite).
template <typename Smem>
__device__ __forceinline__ void pair_step(const Smem& S, uint32_t at, float2 px, float2 py, float2 pz, float e0, float e1, Sums& s) {
  const float4 jxy = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(S.lxy) + at);
  const float4 jzm = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(S.lzm) + at);
  const float2 jx = make_float2(jxy.x, jxy.y), jy = make_float2(jxy.z, jxy.w);
  const float2 jz = make_float2(jzm.x, jzm.y), jm = make_float2(jzm.z, jzm.w);
  const float2 ex = __fadd2_rn(jx, px), ey = __fadd2_rn(jy, py), ez = __fadd2_rn(jz, pz);
  // the softening enters through two scalar FMAs: no register pair to fill for it
  const float2 e2 = __ffma2_rn(ex, ex, __ffma2_rn(ey, ey, make_float2(fmaf(ez.x, ez.x, e0), fmaf(ez.y, ez.y, e1))));
  const float2 ri = make_float2(rsqrt_walk(e2.x), rsqrt_walk(e2.y));
  const float2 mr = __fmul2_rn(jm, ri);
  const float2 ff = __fmul2_rn(__fmul2_rn(mr, ri), ri);
  s.ax = __ffma2_rn(ex, ff, s.ax);
  s.ay = __ffma2_rn(ey, ff, s.ay);
  s.az = __ffma2_rn(ez, ff, s.az);
  s.pt = __fadd2_rn(s.pt, mr);
}

// Direct sum of one staged chunk of k sources of a leaf of more than kLeafMax
// particles, for the lanes in `me`. A particle served by LPP lanes splits the
// source pairs: lane `sub` takes pairs sub, sub + LPP, ... With soft (eps^2 a normal
// float) the self pair is included (zero force at r = 0; its potential is removed
// once at the end of the walk); otherwise the particle's own source jself is skipped.
// A source past k is staged as a massless zero.
template <int LPP, typename Smem>
__device__ __forceinline__ void leaf_sum(const Smem& S, uint32_t k, uint32_t jself, bool me, bool soft, float2 px,
                                         float2 py, float2 pz, float eps2, Sums& s, uint32_t sub) {
  // One softening for all of the lane's pairs: with a test per pair, a step of 150000 particles half
  // of which are at one place took 12.3 ms instead of 10.9, and 25.1 instead of 22.7 with all
  // positions NaN (one leaf).
  if (soft) {
    const float e = me ? eps2 : INFINITY;
    for (uint32_t j = 2 * sub; j < k; j += 2 * LPP) pair_step(S, 8 * j, px, py, pz, e, e, s);
  } else {
    for (uint32_t j = 2 * sub; j < k; j += 2 * LPP) {
      const bool u0 = me && j != jself, u1 = me && j + 1 < k && j + 1 != jself;
      pair_step(S, 8 * j, px, py, pz, u0 ? eps2 : INFINITY, u1 ? eps2 : INFINITY, s);
    }
  }
}

// Direct sums of the queued leaves (nq of them, qp source pairs in all).
//
// What bounds it: an opened leaf is opened by a third of the item's 32 particles, so
// a sum in which every lane takes every source of the leaf wastes two thirds of its
// issue slots (a 32-particle item ran 453 packed steps for 162 useful ones per lane on
// the 524288-particle disk, theta 0.5). Here the item's particles form subgroups of 8 Morton neighbours, and
// the warp takes one subgroup at a time: 8 particles x 4 lanes, the lanes of a
// particle splitting the source pairs that some particle of the subgroup takes part
// in: 281 steps (subgroups of 16: 352, of 4: 229 with twice the subgroups to set up).
// The price is one list of the subgroup's pairs and one sum over the 4 lanes per
// subgroup and window, so leaves are queued until a window is nearly full (windows of
// 64 pairs: walk 1027 us, of 96: 1000 us, of 32: 1103 us; 96 fills the shared memory
// of 7 blocks per SM). Against the leaf-by-leaf sums it replaced: walk of that disk
// 1091 -> 1000 us (49.7 -> 47.3 thousand warp instructions per item), the collision of
// 524288 1140 -> 1087 us, 16384 particles (items of 8) 87 -> 75 us.
//
// A window: each lane turns its queued leaf into source pairs (a leaf of odd count
// ends in a massless zero), then stages whole pairs, so the loads of a window are in
// flight together and the staging stores are 128 bits wide.
// Items of 8 or 4 particles are one subgroup: no list, and the lanes' partial sums stay
// where the rest of the walk keeps them.
template <int LPP, typename Smem>
__device__ __forceinline__ void leaf_flush(Smem& S, const float4* __restrict__ pin, uint32_t nq, uint32_t qp,
                                           uint32_t gbeg, int lane, bool soft, float eps2, float nx, float ny,
                                           float nz, Sums& s) {
  constexpr uint32_t G = 32 / LPP, SUBT = G < 8 ? G : 8, SH = 32 / SUBT, NSUB = G / SUBT;
  constexpr uint32_t SMASK = (1u << SUBT) - 1u;
  constexpr uint32_t W = kLeafWindow, kPer = W / 32;  // pairs a lane stages
  const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
  const uint32_t tl = lane % SUBT, share = lane / SUBT;
  for (uint32_t w0 = 0; w0 < qp; w0 += W) {
    __syncwarp();  // the queue is written; the staging is no longer read
    uint32_t run = 0;
    for (uint32_t e0 = 0; e0 < nq; e0 += 32) {
      const bool has = e0 + lane < nq;
      const uint2 en = has ? S.q[e0 + lane] : make_uint2(0u, 0u);
      const uint32_t first = en.x & ((1u << kLeafCountShift) - 1u), cnt = (en.x >> kLeafCountShift) + 1u;
      const uint32_t np = has ? (cnt + 1u) >> 1 : 0u;
      uint32_t incl = np;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += y;
      }
      // the leaf's pairs [klo, khi) lie in the window, pair k at window position at + k
      const int at = (int)(run + incl - np - w0);
      const int klo = max(0, -at), khi = min((int)np, (int)W - at);
      const uint32_t kn = khi > klo ? (uint32_t)(khi - klo) : 0u;
#pragma unroll
      for (uint32_t k = 0; k < kLeafMax / 2; k++)
        if (k - (uint32_t)klo < kn) S.pinfo[at + (int)k] = make_uint2((first + 2 * k) | 0x80000000u, en.y);
      if ((cnt & 1u) && np - 1u - (uint32_t)klo < kn) S.pinfo[at + (int)np - 1].x = first + 2 * (np - 1u);
      run += __shfl_sync(full, incl, 31);
    }
    __syncwarp();
    const uint32_t nw = min(W, qp - w0);
    uint32_t pm[kPer];
    float4 A[kPer], B[kPer];
    // all loads first (no branches): slots past the window repeat its last pair and
    // no list names them; a missing second source is the first with no mass
#pragma unroll
    for (uint32_t r = 0; r < kPer; r++) {
      const uint32_t t = lane + 32 * r;
      const uint2 pi = S.pinfo[min(t, nw - 1)];
      const float4* src = pin + 2 * (size_t)(pi.x & 0x7fffffffu);
      const bool both = pi.x >> 31;
      A[r] = __ldg(src);
      B[r] = __ldg(src + (both ? 2 : 0));
      B[r].w = both ? B[r].w : 0.f;
      pm[r] = t < nw ? pi.y : 0u;
    }
#pragma unroll
    for (uint32_t r = 0; r < kPer; r++) {
      const uint32_t t = lane + 32 * r;
      *reinterpret_cast<float4*>(&S.lxy[4 * t]) = make_float4(A[r].x, B[r].x, A[r].y, B[r].y);
      *reinterpret_cast<float4*>(&S.lzm[4 * t]) = make_float4(A[r].z, B[r].z, A[r].w, B[r].w);
    }
#pragma unroll 1
    for (uint32_t g = 0; g < NSUB; g++) {
      uint32_t n = nw;
      if (NSUB > 1) {  // the subgroup's pairs, in window order, padded with a pair nobody takes
        n = 0;
#pragma unroll
        for (uint32_t r = 0; r < kPer; r++) {
          const uint32_t m = (pm[r] >> (SUBT * g)) & SMASK;
          const uint32_t b = __ballot_sync(full, m != 0u);
          if (m) S.list[n + __popc(b & below)] = (16 * (lane + 32 * r)) | (m << 24);
          n += __popc(b);
        }
        // no pair of this subgroup's: leave before the padding, which the next subgroup's list
        // would overwrite with no ordering of the two
        if (n == 0) continue;
        if (lane < (int)SH) S.list[n + lane] = 0u;
      }
      __syncwarp();
      const float2 px = f2(NSUB > 1 ? __shfl_sync(full, nx, SUBT * g + tl) : nx);
      const float2 py = f2(NSUB > 1 ? __shfl_sync(full, ny, SUBT * g + tl) : ny);
      const float2 pz = f2(NSUB > 1 ? __shfl_sync(full, nz, SUBT * g + tl) : nz);
      Sums z;
      if (NSUB > 1) z.ax = z.ay = z.az = z.pt = f2(0.f);
      else z = s;
      if (soft) {
        const uint32_t bit = NSUB > 1 ? 0x1000000u << tl : 1u << tl;
#pragma unroll 2
        for (uint32_t j0 = 0; j0 < n; j0 += SH) {
          uint32_t at, m;
          if (NSUB > 1) {
            m = S.list[j0 + share];
            at = m & 0xffffffu;
          } else {
            const uint32_t t = min(j0 + share, n - 1);
            at = 16 * t;
            m = j0 + share < n ? S.pinfo[t].y : 0u;
          }
          const float e = m & bit ? eps2 : INFINITY;
          pair_step(S, at, px, py, pz, e, e, z);
        }
      } else {  // the particle's own source is left out
        const uint32_t self = gbeg + SUBT * g + tl;
        for (uint32_t j0 = 0; j0 < n; j0 += SH) {
          uint32_t t = min(j0 + share, n - 1), m;
          if (NSUB > 1) {
            m = S.list[j0 + share];
            t = (m & 0xffffffu) >> 4;
            m >>= 24;
          } else {
            m = j0 + share < n ? S.pinfo[t].y : 0u;
          }
          const uint32_t fx = S.pinfo[t].x, f = fx & 0x7fffffffu;
          const bool me = (m >> tl) & 1u;
          pair_step(S, 16 * t, px, py, pz, me && f != self ? eps2 : INFINITY,
                    me && (fx >> 31) && f + 1 != self ? eps2 : INFINITY, z);
        }
      }
      if (NSUB > 1) {  // add the shares; the particle's own lane keeps the result
        float v[4] = {z.ax.x + z.ax.y, z.ay.x + z.ay.y, z.az.x + z.az.y, z.pt.x + z.pt.y};
#pragma unroll
        for (int k = 0; k < 4; k++) {
#pragma unroll
          for (uint32_t o = SUBT; o < 32; o <<= 1) v[k] += __shfl_xor_sync(full, v[k], o);
        }
        if (lane / SUBT == g) {
          s.ax.x += v[0];
          s.ay.x += v[1];
          s.az.x += v[2];
          s.pt.x += v[3];
        }
        __syncwarp();  // the list is no longer read
      } else {
        s = z;
      }
    }
  }
}

// Kahan step on packed pairs: s + x with the lost low-order part kept in c
// (c holds the negated error; the compensated total is s - c).
__device__ __forceinline__ void kahan_add2(float2& s, float2& c, float2 x) {
  const float2 y = __ffma2_rn(c, f2(-1.0f), x);   // x - c
  const float2 t = __fadd2_rn(s, y);
  c = __ffma2_rn(y, f2(-1.0f), __ffma2_rn(s, f2(-1.0f), t));  // (t - s) - y
  s = t;
}

// All ones if a > b (ordered: NaN gives 0), else 0, as one compare-and-set.
__device__ inline uint32_t set_gt_mask(float a, float b) {
  uint32_t r;
  asm("set.gt.u32.f32 %0, %1, %2;" : "=r"(r) : "f"(a), "f"(b));
  return r;
}

// The largest x >= 0, infinity included, for which theta2 * x > s2 does not hold in FP32 (the
// product grows with x): x > open_threshold(s2, theta2) decides like theta2 * x > s2 for every x.
// It is infinity where nothing is accepted: a size beyond 1.8e19 (its square overflows), theta2 = 0.
// Otherwise searched on the bits, from around s2 / theta2.
__device__ __noinline__ float open_threshold(float s2, float theta2) {
  if (!(theta2 * INFINITY > s2)) return INFINITY;
  uint32_t lo = 0u, hi = 0x7f7fffffu;  // holds not at lo
  if (!(theta2 * __uint_as_float(hi) > s2)) return __uint_as_float(hi);
  const uint32_t q = __float_as_uint(s2 / theta2);
  if (q - 8u < 0x7f000000u) {
    if (!(theta2 * __uint_as_float(q - 4u) > s2)) lo = q - 4u;
    if (theta2 * __uint_as_float(q + 4u) > s2) hi = q + 4u;
  }
  while (hi - lo > 1u) {
    const uint32_t mid = lo + (hi - lo) / 2u;
    if (theta2 * __uint_as_float(mid) > s2) hi = mid;
    else lo = mid;
  }
  return __uint_as_float(lo);
}

// Transpose of the 32 x 32 bit matrix held one row per lane: afterwards bit j
// of lane i is bit i of lane j (five butterfly stages of 16, 8, 4, 2, 1 bits). The
// stages of 16 and 8 bits are one byte permutation each, the others a rotation and a
// bit select.
__device__ __forceinline__ uint32_t warp_transpose(uint32_t x, int lane) {
  x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), lane & 16 ? 0x3276 : 0x5410);
  x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), lane & 8 ? 0x3715 : 0x6240);
#pragma unroll
  for (int j = 4; j >= 1; j >>= 1) {
    const uint32_t m = j == 4 ? 0x0F0F0F0Fu : j == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    // the bits a rotation wraps around fall on the kept ones
    const uint32_t keep = lane & j ? ~m : m, in = __funnelshift_l(y, y, lane & j ? 32 - j : j);
    x = (x & keep) | (in & ~keep);
  }
  return x;
}

// ONE: the layout holds a single galaxy, whose descriptor comes with the
// kernel parameters instead of a per-group lookup. COMP: far-field (monopole)
// contributions are accumulated with compensation, blocked by round: a round's
// terms (at most 32 per lane) are summed plainly and each round's sum is added to
// the particle's total with a Kahan step; near-field leaf sums add plainly into
// the same totals.
// LPP: lanes per particle (walk group of 32 / LPP particles); a launch walks the
// galaxies whose SegDesc wlpp field equals LPP and skips the others' work items.
template <bool SF, bool DBG, bool ONE, bool COMP, int LPP>
__global__ void __launch_bounds__(kWalkThreads, walk_resident<LPP, COMP>()) walk_kernel(WalkArgs a) {
  static_assert(LPP == 1 || LPP == 2 || LPP == 4 || LPP == 8, "lanes per particle");
  constexpr uint32_t G = 32 / LPP;                         // particles per work item
  constexpr int NPP = 16 / LPP;                            // slot pairs a lane tests in a full round
  constexpr unsigned GMASK = G == 32 ? 0xffffffffu : (1u << G) - 1u;
  constexpr uint32_t kStride = LPP;                        // work items per walk group
  griddep_wait();  // launched with a programmatic dependency: predecessors' writes first
  __shared__ WalkSmem smem_all[kWalkWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t pl = lane % G;    // the lane's particle within the item
  const uint32_t sub = lane / G;   // its share of the slot pairs and leaf sources
  // slots whose pairs this lane tests: pairs sub, sub + LPP, ... (bits 2pp, 2pp + 1)
  const uint32_t mine = LPP == 1   ? 0xffffffffu
                        : LPP == 2 ? (0x33333333u << (2 * sub))
                        : LPP == 4 ? (0x03030303u << (2 * sub))
                                   : (0x00030003u << (2 * sub));
  WalkSmem& S = smem_all[warp];
  // splits per work item (1, 2, 4, 8): a lone galaxy walked in groups of 16 or
  // fewer (the 32-particle build, the large galaxies' walk, carries no split code)
  const uint32_t NS = ONE && LPP > 1 ? a.seg0.wsplit : 1u;
  const uint32_t nitems = a.L.groups * kStride * NS;
  const unsigned full = 0xffffffffu;

  const uint32_t below = (1u << lane) - 1u, lanebit = 1u << pl;
  // Walk groups of 32 test size^2 < theta^2 (r^2 + eps^2) as r^2 + eps^2 > thr(size^2), with the
  // threshold (open_threshold) that makes every decision the same. A tree's sizes are the
  // root's over powers of two, so its size^2 share a mantissa, and the threshold's bits
  // are size^2's plus one number for all of them; other sizes (uploaded trees) are
  // searched for. It saves a packed multiply per pair; a warp of smaller groups walks too
  // few pairs to earn back the set-up (walk of 524288 particles 972 -> 951 us; of 60001, in
  // groups of 16, 99 -> 101) and multiplies by theta^2. Where theta^2 is zero (or NaN) nothing is
  // accepted: the multiplier is then the smallest normal float, so that an inactive lane's infinite
  // distance and a dummy are far as ever, and thr_zero makes every other threshold infinite.
  constexpr bool kThr = LPP == 1;
  float theta2, thr_zero = 0.f;
  uint32_t root_s2 = 0, thr_add = 0, thr_range = 0, thr_slot = 0xffffffffu;
  auto threshold_of = [&](const SegDesc& g) {
    const float theta = __ldg(&a.st[g.slot].p.theta);
    theta2 = theta * theta;
    if (!kThr) {
      thr_zero = theta2 > 0.f ? 0.f : INFINITY;
      if (!(theta2 > 0.f)) theta2 = 1.17549435e-38f;
      return;
    }
    root_s2 = __float_as_uint(a.info[g.node_off].s2);
    thr_add = __float_as_uint(open_threshold(__uint_as_float(root_s2), theta2)) - root_s2;
    // both ends far from subnormals and infinity: size^2 within [2^-95, 2^93), the shift within 2^+-16
    thr_range = root_s2 - 0x10000000u < 0x5e000000u && thr_add + 0x08000000u < 0x10000000u ? 0x5e000000u : 0u;
  };
  if (ONE) threshold_of(a.seg0);
  if (lane < kWalkRanges) S.stack[lane] = make_uint2(0u, 0u);

  while (true) {
    uint32_t c = 0;  // grab the next work item of the schedule
    if (lane == 0) c = atomicAdd(&a.work[0], 1u);
    c = __shfl_sync(full, c, 0);
    if (c >= nitems) break;
    const uint32_t ksp = c % NS, cq = c / NS;  // split ksp of work item cq
    const uint32_t gcur = cq / kStride, part = cq % kStride;
    const SegDesc sd = ONE ? a.seg0 : a.L.segs[a.L.seg_of_group[gcur]];
    if (!ONE && sd.wlpp != LPP) continue;  // a galaxy of another group size
    DevState* const sst = a.st + sd.slot;
    const gs_params& P = sst->p;  // read-only during the walk; fields loaded where used
    const float eps2p = __ldg(&P.epsilon2);
    const float qe2 = 0.25f * eps2p;
    // Self pairs may be summed and removed afterwards when softened. Softening below
    // the smallest normal float counts as none, so every r^2 + eps^2 below is a
    // normal number (or +inf, or NaN from non-finite input), for which the
    // flush-to-zero rsqrt gives the same result as the non-flushing one.
    const bool soft = eps2p >= 1.17549435e-38f;
    // Without softening a node test at r = 0 (a particle's own one-particle leaf)
    // would weigh rsqrt(0) = inf by 0 (NaN): the distances add the smallest
    // normal float instead, which moves no r^2 above 1e-30 by more than a
    // rounding step, and such a node is opened as before.
    const float eps2 = soft ? eps2p : 1.17549435e-38f;
    if (!ONE && sd.slot != thr_slot) {  // a warp's next item is mostly of the same galaxy
      threshold_of(sd);
      thr_slot = sd.slot;
    }
    const uint32_t seg_end = sd.off + sd.n;
    const uint32_t gbeg = sd.off + (gcur - sd.group0) * kWalkGroup + part * G, gend = gbeg + G;
    const uint32_t i = gbeg + pl;
    const bool valid = i < seg_end;
    // The particle's record is read again for the integration at the end, so only its
    // negated position stays live through the walk.
    float4 p0 = make_float4(0.f, 0.f, 0.f, 0.f), p1 = p0;
    if (valid) p0 = a.pin[2 * (size_t)i];
    const float2 px = f2(-p0.x), py = f2(-p0.y), pz = f2(-p0.z);  // negated: r = q + (-p)
    Sums F = {f2(0.f), f2(0.f), f2(0.f), f2(0.f)};
    float2 cax = f2(0.f), cay = f2(0.f), caz = f2(0.f), cpt = f2(0.f);  // COMP only
    float dens = 0.f, selfw = 0.f;
    unsigned long long nmono = 0, npair = 0, nvisit = 0;
    uint32_t nq = 0, qp = 0;  // queued leaves, their source pairs
    const unsigned all = __ballot_sync(full, valid) & GMASK;  // the item's particles (lanes of share 0)

    // Split walk: the first level of at least kSplitMinNodes nodes per split is
    // the split level; split k owns its nodes j with j = k mod NS (counted from
    // the level's start) and their subtrees, and split 0 also every contribution
    // of the levels above, which the other splits test (to reach their own
    // nodes) without adding.
    uint32_t up_end = 0u, win_end = 0u;
    bool idle = false;
    if (NS > 1) {
      const TreeMeta* m = a.meta + sd.slot;
      const uint32_t nl = min(m->num_levels, (uint32_t)kDepths);
      up_end = win_end = 0xffffffffu;
      for (uint32_t l = 1; l < nl; l++) {
        const uint32_t cnt = m->level_count[l];
        if (cnt >= kSplitMinNodes * NS) {
          up_end = sd.node_off + m->level_start[l];
          win_end = up_end + cnt;
          break;
        }
      }
      idle = ksp > 0 && up_end == 0xffffffffu;  // no such level: split 0 walks the whole tree
    }

    int sp = 0;
    if (lane == 0) S.stack[kWalkRanges] = make_uint2(sd.node_off, all);  // the root: range {node_off, 1}
    sp = idle ? 0 : 1;
    uint32_t budget = 4u * sd.node_cap + 1024u;
    while (true) {
      if (qp >= (uint32_t)kLeafFlush || (sp == 0 && qp > 0)) {
        leaf_flush<LPP>(S, a.pin, nq, qp, gbeg, lane, soft, eps2, px.x, py.x, pz.x, F);
        nq = qp = 0;
      }
      if (sp == 0) break;
      __syncwarp();
      // pop up to kWalkRanges ranges; their children are staged and tested together
      const int nr = min(sp, kWalkRanges);
      const uint2* const top = &S.stack[kWalkRanges + sp - 1];
      sp -= nr;
      uint32_t masks[kWalkRanges];  // lanes that opened each popped range's parent
#pragma unroll
      for (int r = 0; r < kWalkRanges; r++) masks[r] = top[-r].y;
      if (--budget == 0) {
        if (lane == 0) raise_err(sst, GS_DERR_STACK);
        break;
      }
      // Stage range r in lanes 8r..8r+7: one child per lane; slots past a range's
      // count hold massless dummies. Massless and sub-softening children
      // (size^2 < eps^2/4, always accepted, nbody_bh.wgsl:112) get size^2 = -inf,
      // so the per-lane test is one compare with the child's threshold.
      bool own = false, isleaf = false, massive = false, skip = false;
      uint32_t cnode = 0, cchild = 0, ccnt = 0;  // this lane's slot: node, first child or particle, count
      uint32_t act = 0;                          // and the particles that opened its parent
      float csize = 1.f;
      if (lane < 8 * kWalkRanges) {
        const uint32_t c = lane & 7;
        const uint2 e = top[-(lane >> 3)];
        const uint32_t rs = e.x & 0x1fffffffu;
        act = e.y;
        // slots past the count (and empty entries) load a node of the range (the first of
        // the pool) and are made dummies like massless nodes, with no children to go on to
        bool real = e.y != 0u && c <= e.x >> 29, counted = true;
        cnode = rs + min(c, e.x >> 29);
        if (NS > 1 && real) {
          if (cnode < up_end) counted = ksp == 0;                                    // levels above the split
          else if (cnode < win_end && ((cnode - up_end) & (NS - 1)) != ksp) real = false;  // another split's
        }
        float4 q = __ldg(&a.cm[cnode]);
        const uint4 w = __ldg(reinterpret_cast<const uint4*>(a.info) + cnode);  // WalkInfo
        cchild = w.y;
        ccnt = real ? w.z & ~kLeafBit : 0u;
        csize = __uint_as_float(w.w);
        const bool heavy = real && q.w != 0.0f;
        isleaf = real && (w.z & kLeafBit);
        massive = heavy && counted;
        skip = isleaf && !counted;
        own = isleaf && heavy && cchild < gend && cchild + ccnt > gbeg;
        const float s2 = __uint_as_float(w.x);
        // never opened: massless and dummies (which contribute nothing, far away and
        // massless), and sub-softening children
        float thr = -INFINITY;
        if (heavy && !(s2 < qe2)) {
          thr = kThr ? __uint_as_float(w.x + thr_add) : s2 + thr_zero;
          if (kThr && (((w.x ^ root_s2) & 0x7fffffu) || w.x - 0x10000000u >= thr_range)) thr = open_threshold(s2, theta2);
        }
        if (!heavy) q = make_float4(1e30f, 1e30f, 1e30f, 0.f);
        const int st = 4 * (lane >> 1) + (lane & 1);
        S.cxy[st] = q.x;
        S.cxy[st + 2] = q.y;
        S.czm[st] = q.z;
        S.czm[st + 2] = counted ? q.w : 0.0f;  // tested for opening, adds nothing
        S.cthr[lane] = thr;
      }
      const unsigned ownmask = __ballot_sync(full, own);  // leaves holding our particles
      const unsigned leafmask = __ballot_sync(full, isleaf);
      const unsigned massmask = DBG ? __ballot_sync(full, massive) : 0u;
      const unsigned skipm = NS > 1 ? __ballot_sync(full, skip) : 0u;  // opened leaves another split sums
      __syncwarp();
      // eps^2 per range; a lane inactive for a range adds +inf: it accepts every child, and
      // adds nothing as rsqrt gives 0, and so it sets no open bit (nor does a slot past a
      // range's count, a dummy with the threshold -inf). A NaN distance (the lane's own position
      // or a centre of mass) or threshold fails the compare and does set one, in ranges the
      // lane is inactive for and at dummies too: these are dropped below
      float e2[kWalkRanges];
#pragma unroll
      for (int r = 0; r < kWalkRanges; r++) e2[r] = masks[r] & lanebit ? eps2 : INFINITY;
      uint32_t obits = 0;  // children this lane does not accept, bit = slot
      // COMP: the round's far-field terms (at most 32 per lane) are summed plainly,
      // then the round's sum joins the particle's total in one Kahan step
      float2 rax = f2(0.f), ray = f2(0.f), raz = f2(0.f), rpt = f2(0.f);
#pragma unroll
      for (int kk = 0; kk < NPP; kk++) {
        // a range's pairs are tested only if the range was popped (one check per range)
        if ((kk * LPP) % 4 == 0 && kk * LPP >= 4 * nr) break;
        const int pp = (int)sub + kk * LPP;
        const int c = 2 * pp;
        // the pair's range pp >> 2: (kk * LPP) >> 2 for shares below 4, one more above
        const float er = LPP < 8 ? e2[(kk * LPP) >> 2] : (sub >= 4 ? e2[2 * kk + 1] : e2[2 * kk]);
        const float4 qxy = *reinterpret_cast<const float4*>(&S.cxy[2 * c]);
        const float4 qzm = *reinterpret_cast<const float4*>(&S.czm[2 * c]);
        const float2 qx = make_float2(qxy.x, qxy.y), qy = make_float2(qxy.z, qxy.w);
        const float2 qz = make_float2(qzm.x, qzm.y), qm = make_float2(qzm.z, qzm.w);
        const float2 thr = *reinterpret_cast<const float2*>(&S.cthr[c]);
        const float2 rx = __fadd2_rn(qx, px), ry = __fadd2_rn(qy, py), rz = __fadd2_rn(qz, pz);
        const float2 d2 = __ffma2_rn(rx, rx, __ffma2_rn(ry, ry, __ffma2_rn(rz, rz, f2(er))));
        // all ones where the child is accepted; an accepted child keeps r^2 + eps^2,
        // any other gets +inf, so rsqrt makes its terms exactly 0
        const float2 td = kThr ? d2 : __fmul2_rn(f2(theta2), d2);
        const uint32_t ax_ = set_gt_mask(td.x, thr.x), ay_ = set_gt_mask(td.y, thr.y);
        obits |= (~ax_ & (1u << c)) | (~ay_ & (2u << c));
        const float2 dsel = make_float2(__uint_as_float((__float_as_uint(d2.x) & ax_) | (0x7f800000u & ~ax_)),
                                        __uint_as_float((__float_as_uint(d2.y) & ay_) | (0x7f800000u & ~ay_)));
        const float2 rinv = make_float2(rsqrt_walk(dsel.x), rsqrt_walk(dsel.y));
        const float2 mr = __fmul2_rn(qm, rinv);
        const float2 f = __fmul2_rn(__fmul2_rn(mr, rinv), rinv);
        if (COMP) {
          rax = __ffma2_rn(rx, f, rax);
          ray = __ffma2_rn(ry, f, ray);
          raz = __ffma2_rn(rz, f, raz);
          rpt = __fadd2_rn(rpt, mr);
        } else {
          F.ax = __ffma2_rn(rx, f, F.ax);
          F.ay = __ffma2_rn(ry, f, F.ay);
          F.az = __ffma2_rn(rz, f, F.az);
          F.pt = __fadd2_rn(F.pt, mr);  // sum of m/r; potential = -G * sum
        }
      }
      if (COMP) {
        kahan_add2(F.ax, cax, rax);
        kahan_add2(F.ay, cay, ray);
        kahan_add2(F.az, caz, raz);
        kahan_add2(F.pt, cpt, rpt);
      }
      if (DBG) {
        uint32_t keep = 0;  // the slots this lane tests, of the ranges it is active for
#pragma unroll
        for (int r = 0; r < kWalkRanges; r++)
          if (masks[r] & lanebit) keep |= 0xffu << (8 * r);
        keep &= mine;
        nvisit += __popc(massmask & keep);
        nmono += __popc(massmask & keep & ~obits);
      }
      for (uint32_t bb = ownmask; bb; bb &= bb - 1) {  // own-leaf density (nbody_bh.wgsl:93-95)
        const uint32_t cc = __ffs(bb) - 1;
        const uint32_t lf = __shfl_sync(full, cchild, cc), cnt = __shfl_sync(full, ccnt, cc);
        const float sz = __shfl_sync(full, csize, cc);
        // the slot's own mask: the stack entry it came from is overwritten by this round's pushes
        if ((__shfl_sync(full, act, cc) & lanebit) && (i - lf) < cnt) {
          dens = (float)cnt / (sz * sz * sz);
          // the leaf's direct sum includes the particle itself (softened walks)
          if (((obits & ~skipm) >> cc) & 1u) selfw += 1.0f;
        }
      }
      if (!__any_sync(full, obits != 0u)) continue;
      // Every slot's open mask at once: lane c's col holds the lanes that open
      // slot c (the transpose of the 32 x 32 bit matrix whose rows are the lanes'
      // obits), so each slot's lane can act on its own child in parallel. Only
      // the share that tests slot c has its bits: shifted down, they are the
      // item's particle mask, of which those that opened the slot's parent count.
      const uint32_t col = (warp_transpose(obits, lane) >> ((((uint32_t)lane >> 1) % LPP) * G)) & act;
      const uint32_t om = __ballot_sync(full, col != 0u);  // children opened by some particle
      // opened internal children: each slot's lane writes its child range and open
      // mask to the stack, in slot order (prefix positions)
      if (om & ~leafmask) {
        // a galaxy's child ranges stay in its node range by construction (build,
        // upload check); the walk itself only guards the pool bounds. A refused range
        // (a dummy has no children) stays off the stack.
        const bool push = col != 0u && !isleaf;
        const bool ok = push && cchild > cnode && ccnt - 1u < 8u && cchild <= a.node_pool - ccnt;
        if (push && !ok) raise_err(sst, GS_DERR_TREE);
        const uint32_t okm = __ballot_sync(full, ok);
        const int np = __popc(okm);
        if (sp + np > kWalkStack) {  // not for depth <= 10 trees
          if (lane == 0) raise_err(sst, GS_DERR_STACK);
        } else {
          if (ok)
            S.stack[kWalkRanges + sp + __popc(okm & below)] = make_uint2(cchild | ((ccnt - 1u) << 29), col);
          sp += np;
        }
      }
      // Opened leaves: those of at most kLeafMax particles join the queue, in slot
      // order; larger ones (coincident particles at the deepest level) are summed
      // at once, in chunks of 32.
      const uint32_t leafc = om & leafmask & ~skipm;
      if (leafc) {
        const bool mine_leaf = (leafc >> lane) & 1u;
        // empty (adds nothing), large, or past the particle pool: not for the queue
        const bool odd = mine_leaf && (ccnt - 1u >= kLeafMax || cchild > a.pool_n - ccnt);
        const uint32_t oddm = __ballot_sync(full, odd), goodm = leafc & ~oddm;
        const bool good = mine_leaf && !odd;
        if (good) S.q[nq + __popc(goodm & below)] = make_uint2(cchild | ((ccnt - 1u) << kLeafCountShift), col);
        nq += __popc(goodm);
        qp += __reduce_add_sync(full, good ? (ccnt + 1u) >> 1 : 0u);
        if (DBG) {
          for (uint32_t bb = leafc; bb; bb &= bb - 1) {
            const uint32_t cc = __ffs(bb) - 1;
            const unsigned open = __shfl_sync(full, col, cc);
            const uint32_t lf = __shfl_sync(full, cchild, cc), cnt = __shfl_sync(full, ccnt, cc);
            if (sub == 0 && ((open >> pl) & 1u)) npair += cnt - (i - lf < cnt ? 1u : 0u);
          }
        }
        for (uint32_t bb = oddm; bb; bb &= bb - 1) {
          const uint32_t cc = __ffs(bb) - 1;
          const unsigned open = __shfl_sync(full, col, cc);
          const uint32_t lf = __shfl_sync(full, cchild, cc), cnt = __shfl_sync(full, ccnt, cc);
          if (cnt > a.pool_n || lf > a.pool_n - cnt) {
            if (lane == 0) raise_err(sst, GS_DERR_TREE);
            continue;
          }
          for (uint32_t b0 = 0; b0 < cnt; b0 += 32) {
            const uint32_t k = min(32u, cnt - b0);
            __syncwarp();
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (lane < (int)k) v = __ldg(&a.pin[2 * (size_t)(lf + b0 + lane)]);
            const int se = 4 * (lane >> 1) + (lane & 1);
            S.lxy[se] = v.x;
            S.lxy[se + 2] = v.y;
            S.lzm[se] = v.z;
            S.lzm[se + 2] = v.w;
            __syncwarp();
            leaf_sum<LPP>(S, k, i - (lf + b0), (open >> pl) & 1u, soft, px, py, pz, eps2, F, sub);
          }
        }
      }
    }
    if (COMP) {  // fold the compensations into the sums
      F.ax = __ffma2_rn(cax, f2(-1.0f), F.ax);
      F.ay = __ffma2_rn(cay, f2(-1.0f), F.ay);
      F.az = __ffma2_rn(caz, f2(-1.0f), F.az);
      F.pt = __ffma2_rn(cpt, f2(-1.0f), F.pt);
    }
    if (LPP > 1) {  // add the shares of each particle (lanes pl, pl + G, ...), fixed order
#pragma unroll
      for (uint32_t o = G; o < 32; o <<= 1) {
        F.ax = __fadd2_rn(F.ax, make_float2(__shfl_xor_sync(full, F.ax.x, o), __shfl_xor_sync(full, F.ax.y, o)));
        F.ay = __fadd2_rn(F.ay, make_float2(__shfl_xor_sync(full, F.ay.x, o), __shfl_xor_sync(full, F.ay.y, o)));
        F.az = __fadd2_rn(F.az, make_float2(__shfl_xor_sync(full, F.az.x, o), __shfl_xor_sync(full, F.az.y, o)));
        F.pt = __fadd2_rn(F.pt, make_float2(__shfl_xor_sync(full, F.pt.x, o), __shfl_xor_sync(full, F.pt.y, o)));
        selfw += __shfl_xor_sync(full, selfw, o);
      }
    }
    if (DBG) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        nmono += __shfl_xor_sync(full, nmono, o);
        npair += __shfl_xor_sync(full, npair, o);
        nvisit += __shfl_xor_sync(full, nvisit, o);
      }
      if (lane == 0) {
        atomicAdd(&sst->counters[0], nmono);
        atomicAdd(&sst->counters[1], npair);
        atomicAdd(&sst->counters[2], nvisit);
      }
    }
    if (NS > 1) {
      // Each split leaves its sums in split_buf; the last split of the item to
      // arrive adds them in split order (the same sums whatever the arrival order)
      // and finishes the item. No split waits for another.
      const uint32_t li = i - sd.off;
      const size_t st = a.split_stride;
      float4* const B = a.split_buf;
      const float4 o0 = make_float4(F.ax.x, F.ax.y, F.ay.x, F.ay.y), o1 = make_float4(F.az.x, F.az.y, F.pt.x, F.pt.y);
      const float4 o2 = make_float4(dens, selfw, 0.f, 0.f);
      if (valid && sub == 0) {
        B[(size_t)ksp * st + li] = o0;
        B[(size_t)(NS + ksp) * st + li] = o1;
        B[(size_t)(2 * NS + ksp) * st + li] = o2;
      }
      __threadfence();
      __syncwarp();
      unsigned* const arrive = a.split_arrive + (size_t)(gcur - sd.group0) * kStride + part;
      unsigned prev = 0;
      if (lane == 0) prev = atomicAdd(arrive, 1u);
      prev = __shfl_sync(full, prev, 0);
      if (prev != NS - 1) continue;  // another split finishes this item
      __threadfence();
      if (lane == 0) *arrive = 0u;   // every split of the item has arrived: ready for the next launch
      if (valid && sub == 0) {
        float4 u0 = o0, u1 = o1, u2 = o2;
        for (uint32_t k = 0; k < NS; k++) {
          float4 v0 = o0, v1 = o1, v2 = o2;
          if (k != ksp) {
            v0 = __ldcg(B + (size_t)k * st + li);
            v1 = __ldcg(B + (size_t)(NS + k) * st + li);
            v2 = __ldcg(B + (size_t)(2 * NS + k) * st + li);
          }
          if (k == 0) {
            u0 = v0;
            u1 = v1;
            u2 = v2;
          } else {
            u0 = make_float4(u0.x + v0.x, u0.y + v0.y, u0.z + v0.z, u0.w + v0.w);
            u1 = make_float4(u1.x + v1.x, u1.y + v1.y, u1.z + v1.z, u1.w + v1.w);
            u2 = make_float4(fmaxf(u2.x, v2.x), u2.y + v2.y, 0.f, 0.f);  // the own leaf is found once or equal
          }
        }
        F.ax = make_float2(u0.x, u0.y);
        F.ay = make_float2(u0.z, u0.w);
        F.az = make_float2(u1.x, u1.y);
        F.pt = make_float2(u1.z, u1.w);
        dens = u2.x;
        selfw = u2.y;
      }
    }
    if (valid) {
      p0 = a.pin[2 * (size_t)i];
      p1 = a.pin[2 * (size_t)i + 1];
    }
    if (soft && selfw != 0.0f) F.pt.x -= selfw * p0.w * rsqrtf(eps2);

    double e_diag = 0, e_true = 0, mx = 0, my = 0, mz = 0, ms = 0;
    if (valid && sub == 0) {
      const float G = P.G;
      float fx = (F.ax.x + F.ax.y) * G, fy = (F.ay.x + F.ay.y) * G, fz = (F.az.x + F.az.y) * G;
      const float pot = -(F.pt.x + F.pt.y) * G;
      if (DBG) {
        a.dbg_acc[i] = make_float4(fx, fy, fz, pot);
        a.dbg_dens[i] = dens;
      }
      // Hernquist halo(s), nbody_bh.wgsl:147-157
      float potHalo = 0.0f;
      if (P.haloMass > 0.0f) {
        for (uint32_t h = 0; h < P.haloCount && h < 2; h++) {
          const float* cc = h == 0 ? P.haloC1 : P.haloC2;
          const float dx = p0.x - cc[0], dy = p0.y - cc[1], dz = p0.z - cc[2];
          const float rlen = fmaxf(sqrtf(dx * dx + dy * dy + dz * dz), 1e-6f);
          const float ra = rlen + P.haloA;
          const float k = G * P.haloMass / (ra * ra * rlen);
          fx -= dx * k;
          fy -= dy * k;
          fz -= dz * k;
          potHalo -= G * P.haloMass / ra;
        }
      }
      // kick (nbody_bh.wgsl:161), gas drag (:166-171), drift (:173)
      float vx = fmaf(fx, P.dt, p1.x), vy = fmaf(fy, P.dt, p1.y), vz = fmaf(fz, P.dt, p1.z);
      const bool gas = p1.w < -0.5f;
      if (gas && P.gasDrag > 0.0f) {
        const float hx = -p0.y, hy = p0.x, hz = 1e-6f;
        const float il = rsqrtf(hx * hx + hy * hy + hz * hz);
        const float ux = hx * il, uy = hy * il, uz = hz * il;
        const float vp = vx * ux + vy * uy + vz * uz;
        const float damp = expf(-P.gasDrag * P.dt);
        const float qx = vp * ux, qy = vp * uy, qz = vp * uz;
        vx = qx + (vx - qx) * damp;
        vy = qy + (vy - qy) * damp;
        vz = qz + (vz - qz) * damp;
      }
      const float4 o0 = make_float4(fmaf(vx, P.dt, p0.x), fmaf(vy, P.dt, p0.y), fmaf(vz, P.dt, p0.z), p0.w);
      float4 o1 = make_float4(vx, vy, vz, gas ? -(1.0f + dens) : 0.0f);
      const float e = 0.5f * (vx * vx + vy * vy + vz * vz) + 0.5f * pot + potHalo;
      a.energy[i] = e;
      const double m = p0.w;
      e_diag = e;
      e_true = m * (double)e;
      mx = m * vx;
      my = m * vy;
      mz = m * vz;
      ms = m;
      if (SF && !sst->sf_off) {
        float4 s = a.stellar[i];
        const float4 s_old = s;
        star_formation_one(P, i - sd.off, o1, s);
        if (s.x != s_old.x || s.y != s_old.y || s.z != s_old.z || s.w != s_old.w) a.stellar[i] = s;
      }
      a.pout[2 * (size_t)i] = o0;
      a.pout[2 * (size_t)i + 1] = o1;
    }
    // per-group partial sums of the diagnostics (fixed order, no atomics)
    double v[kPartials] = {e_diag, e_true, mx, my, mz, ms};
#pragma unroll
    for (int k = 0; k < kPartials; k++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(full, v[k], o);
    }
    if (lane < kPartials) {
      double pv = v[0];
#pragma unroll
      for (int k = 1; k < kPartials; k++)
        if (lane == k) pv = v[k];
      a.partials[((size_t)sd.item0 + (gcur - sd.group0) * LPP + part) * kPartials + lane] = pv;
    }
  }
  // the last warp to finish resets the work counters for the next launch
  if (lane == 0) {
    const unsigned total = gridDim.x * kWalkWarps;
    __threadfence();
    if (atomicAdd(&a.work[1], 1u) == total - 1) {
      a.work[0] = 0;
      a.work[1] = 0;
    }
  }
}

}  // namespace gs
