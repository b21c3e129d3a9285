// The on-device rebuild of one small galaxy as a single kernel on one thread-block
// cluster: bounding box, Morton codes, stable radix sort, gather, central tracking,
// BFS numbering and node COMs, with the results of the kernels it replaces
// (bbox, codes, four onesweep passes, gather, track, flags, scan, emit, leaves)
// bit for bit.
//
// What bounds it: latency. Up to 32768 particles those ten to eleven kernels take 3 to 5
// us each inside a step graph (16 us for the COM cascade, whose levels each cost three
// round trips to L2) while moving a few MB. Here the sorted keys, the positions and the
// COMs stay in the shared memory of up to 16 blocks of 256 or 512 threads, and a
// cluster barrier (about 0.6 us) stands where a launch boundary stood. Blocks are as
// small as the particles allow, because a block-wide phase costs every warp its
// instructions: 1024 threads per block took 46 us where 256 take 33 (4096 particles).
//
// Block r owns the sorted positions [r P, (r + 1) P) of the galaxy, P a power of two.
//   * Sort: four 8-bit LSD passes. A warp ranks its keys by ballots, each block stores
//     its digit counts into every other block's shared memory, and each key is stored
//     straight into the block that owns its position.
//   * Tree: the closed-form BFS numbering of build.cuh. The nodes a block starts at one
//     depth are contiguous in the level, so the blocks exchange twelve counts.
//   * COMs: a node whose particles lie in one block is summed there, level by level with
//     block barriers. Only the last node a block starts at each depth can reach into
//     the next block; those (at most 15 per level) are summed by block 0 at the end from
//     children it fetches for all levels at once.
#pragma once
#include <cooperative_groups.h>

#include "build.cuh"
#include "common.cuh"
#include "morton.cuh"
#include "sort.cuh"

namespace gs {

constexpr int kFuseCtas = 16;              // largest cluster
constexpr uint32_t kFusePer = 4;           // most particles per thread
constexpr int kFuseWarps = 16;             // most warps of a block
constexpr uint32_t kFuseMax = 32768;       // 16 blocks of 512 threads
constexpr int kFuseStrad = kDepths * kFuseCtas;  // nodes that can span blocks

// Threads per block, particles per block and blocks for a galaxy of n particles.
// kFuseMax is where the 16 SMs of one cluster stop paying against all 148: full step in
// us, one cluster / separate kernels: 1000 particles 49 / 78, 4096 64 / 97, 8192 84 / 117, 16384
// 114 / 142, 32768 161 / 183, and 60001 (16 blocks of 1024 threads) 180 / 174.
struct FuseShape {
  uint32_t threads, log2p, ctas;
};
inline FuseShape fuse_shape(uint32_t n) {
  FuseShape f;
  f.log2p = 8;
  while (((uint64_t)kFuseCtas << f.log2p) < n) f.log2p++;
  f.threads = f.log2p <= 10 ? 256u : 512u;
  f.ctas = 1;
  while (((uint64_t)f.ctas << f.log2p) < n) f.ctas *= 2;
  return f;
}

struct FuseArgs {
  const float4* __restrict__ pin;   // 2 float4 per particle
  float4* __restrict__ pout;
  const float4* __restrict__ sin;
  float4* __restrict__ sout;
  uint32_t* __restrict__ keys;      // sorted codes
  uint32_t* __restrict__ vals;      // gather permutation (pool indices)
  MortonFrame* frames;
  DevState* st;
  BuildBuffers b;
  SegDesc sd;
  uint32_t log2p;                   // log2 of the particles per block
  int advance_time, track;
};

// What block 0 needs of every block to sum the nodes that span blocks.
struct FusePub {
  uint32_t cnt[kCounters];          // nodes started per depth, leaves
  uint32_t first[kDepths];          // depth d + 1 nodes started before the first depth d node
  uint32_t last[kDepths];           // packed entry of the last node started at depth d
  uint32_t span;                    // bit d: the last node started at depth d reaches the next block
  uint32_t first_leaf;              // slot of the first leaf start (~0: none)
};

// Fixed part of the shared memory; the per-particle arrays follow it.
struct FuseSmem {
  union {
    uint16_t wcnt[kFuseWarps][256]; // digit counts per warp
    float4 ch[8 * kFuseStrad];      // children of the spanning nodes
  };
  uint32_t tots[kFuseCtas][256];    // digit counts of every block (each block writes its row everywhere)
  uint32_t poff[2][256];            // digit offsets of each half of the warps
  uint32_t base[256];
  int red[kFuseWarps][6];
  int boxes[kFuseCtas][6];          // bounding box of every block (likewise)
  uint32_t cnts[kFuseCtas][kCounters];  // node counts of every block (likewise)
  MortonFrame frame;
  float size[kDepths];
  long long central[2];
  uint32_t wc[kFuseWarps][6];       // packed node counts per warp
  FusePub pub;                      // read by every block
  FusePub pubs[kFuseCtas];
  uint32_t off[kFuseCtas][kCounters];  // nodes started by earlier blocks, per depth
  uint32_t ls[kDepths + 1], lc[kDepths + 1], lbase[kDepths + 1];
  uint32_t overflow;
  uint32_t bits[kFusePer * kFuseWarps];  // leaf starts
  uint32_t lastpos[kDepths];  // last start with D <= d: (its rank + 1) << 1 | (a depth d node starts there)
  uint32_t wpre[kFusePer * kFuseWarps];  // leaf starts before each word of bits
  uint32_t nstart;
  uint32_t run[6];                  // packed counts of the start chunks emitted so far
  uint32_t par[kFuseStrad];         // spanning nodes: place among the children of their parent
  uint4 sm[kFuseStrad];             // spanning nodes: {node, child base, children, leaf start}
  float4 scom[kFuseStrad];
};

// bytes of shared memory for P = 1 << log2p particles per block:
//   R0 (8 P + 512)  key/value buffer 0, later the codes with halos and their shared digits
//   R1 (8 P + 512)  key/value buffer 1, later the nodes' packed entries
//   R2 (16 P)       sorted positions
//   R3 (8 P + 1024) node COMs (the first P / 2 + 64 nodes; further ones stay in L2)
__host__ __device__ inline uint32_t fuse_com_cap(uint32_t log2p) { return (1u << log2p) / 2 + 64; }
inline size_t fuse_smem(uint32_t log2p) {
  const size_t P = (size_t)1 << log2p;
  return sizeof(FuseSmem) + 2 * (8 * P + 512) + 16 * P + 16 * (size_t)fuse_com_cap(log2p);
}
// A node's packed entry: leaf bit, slot of a leaf's first particle, first child
// (index among the depth d + 1 nodes the block starts).
__device__ __forceinline__ uint32_t fuse_entry(bool leaf, uint32_t slot, uint32_t j0) {
  return (leaf ? 0x80000000u : 0u) | (slot << 16) | j0;
}
static_assert(kFusePer * 32 * kFuseWarps <= 4096, "12 bits of leaf slot, 16 of child index");

// T: threads per block (256 or 512); P is at least T, at most 4 T.
template <int MODE, int T>
__global__ void __launch_bounds__(T, 1) fused_rebuild_kernel(FuseArgs a) {
  constexpr uint32_t W = T / 32, PARTS = T / 256, WP = W / PARTS;  // PARTS threads per digit, WP warps each
  namespace cg = cooperative_groups;
  griddep_wait();  // launched with a programmatic dependency: predecessors' writes first
  extern __shared__ __align__(16) unsigned char fuse_raw[];
  FuseSmem& S = *reinterpret_cast<FuseSmem*>(fuse_raw);
  cg::cluster_group cl = cg::this_cluster();
  const uint32_t rank = cl.block_rank(), C = cl.num_blocks();
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t lp = a.log2p, P = 1u << lp, n = a.sd.n, off = a.sd.off;
  const uint32_t base = rank << lp, cntp = base < n ? min(P, n - base) : 0u;  // this block's particles
  unsigned char* const R0 = fuse_raw + sizeof(FuseSmem);
  unsigned char* const R1 = R0 + 8 * (size_t)P + 512;
  float4* const s_pos = reinterpret_cast<float4*>(R1 + 8 * (size_t)P + 512);
  float4* const s_com = s_pos + P;
  uint2* const kv0 = reinterpret_cast<uint2*>(R0);
  uint2* const kv1 = reinterpret_cast<uint2*>(R1);
  DevState* const st = a.st + a.sd.slot;
  const unsigned full = 0xffffffffu;
  cl.barrier_arrive();  // a block's shared memory may be written once it runs

  // ---- bounding box of the finite particles (bbox_kernel) ------------------------------
  // A warp owns 32 K consecutive particles, lane-striped: the stable order of the sort.
  const uint32_t K = P / T;
  float x[kFusePer], y[kFusePer], z[kFusePer];
  int mn[3], mx[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    mn[k] = float_to_ordered(INFINITY);
    mx[k] = float_to_ordered(-INFINITY);
  }
#pragma unroll
  for (uint32_t k = 0; k < kFusePer; k++) {
    const uint32_t slot = warp * (32 * K) + k * 32 + lane;
    x[k] = y[k] = z[k] = 0.f;
    if (k < K && slot < cntp) {
      const float4 p = a.pin[2 * (size_t)(off + base + slot)];
      x[k] = p.x;
      y[k] = p.y;
      z[k] = p.z;
      if (isfinite(p.x) && isfinite(p.y) && isfinite(p.z)) {
        const int e[3] = {float_to_ordered(p.x), float_to_ordered(p.y), float_to_ordered(p.z)};
#pragma unroll
        for (int c = 0; c < 3; c++) {
          mn[c] = min(mn[c], e[c]);
          mx[c] = max(mx[c], e[c]);
        }
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 3; c++) {
    mn[c] = __reduce_min_sync(full, mn[c]);
    mx[c] = __reduce_max_sync(full, mx[c]);
  }
  if (lane == 0)
    for (int c = 0; c < 3; c++) {
      S.red[warp][c] = mn[c];
      S.red[warp][3 + c] = mx[c];
    }
  if (tid < 2) S.central[tid] = st->central[tid];
  __syncthreads();
  cl.barrier_wait();
  if (tid < 6) {
    int v = S.red[0][tid];
    for (uint32_t w = 1; w < W; w++) v = tid < 3 ? min(v, S.red[w][tid]) : max(v, S.red[w][tid]);
    for (uint32_t r = 0; r < C; r++) cl.map_shared_rank(&S.boxes[rank][0], r)[tid] = v;
  }
  cl.sync();
  if (warp == 0) {
    float fmn[3], fmx[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const uint32_t r = min(lane, C - 1);
      fmn[c] = ordered_to_float(__reduce_min_sync(full, S.boxes[r][c]));
      fmx[c] = ordered_to_float(__reduce_max_sync(full, S.boxes[r][3 + c]));
    }
    if (lane == 0) S.frame = frame_from_bbox(fmn, fmx);
    __syncwarp();
    if (lane < kDepths) S.size[lane] = __double2float_rn(ldexp(S.frame.size, -(int)lane));
  }
  if (tid == 0) {
    if (rank == 0) {
      a.frames[a.sd.slot] = S.frame;
      if (a.advance_time) {
        st->p.time = __double2float_rn(st->sim_time);
        st->sim_time = __dadd_rn(st->sim_time, (double)st->p.dt);
      }
    }
  }
  __syncthreads();

  // ---- codes and the four sort passes --------------------------------------------------
  uint32_t key[kFusePer], val[kFusePer], rk[kFusePer];
  {
    const MortonFrame f = S.frame;
#pragma unroll
    for (uint32_t k = 0; k < kFusePer; k++) {
      const uint32_t slot = warp * (32 * K) + k * 32 + lane;
      key[k] = val[k] = 0u;
      if (k < K && slot < cntp) {
        key[k] = morton_code(f, x[k], y[k], z[k]);
        val[k] = base + slot;
      }
    }
  }
  const unsigned lt_mask = (1u << lane) - 1u;
#pragma unroll 1
  for (int pass = 0; pass < kSortPasses; pass++) {
    const int shift = 8 * pass;
    if (pass > 0) {
      const uint2* src = pass & 1 ? kv0 : kv1;
#pragma unroll
      for (uint32_t k = 0; k < kFusePer; k++) {
        const uint32_t slot = warp * (32 * K) + k * 32 + lane;
        if (k < K && slot < cntp) {
          const uint2 e = src[slot];
          key[k] = e.x;
          val[k] = e.y;
        }
      }
    }
    uint32_t* const zero = reinterpret_cast<uint32_t*>(&S.wcnt[0][0]);
#pragma unroll
    for (uint32_t k = 0; k < W * 128 / T; k++) zero[tid + k * T] = 0u;
    __syncthreads();
    {
#pragma unroll
      for (uint32_t k = 0; k < kFusePer; k++) {
        if (k < K) {
          const bool valid = warp * (32 * K) + k * 32 + lane < cntp;
          const uint32_t d = (key[k] >> shift) & 255u;
          // lanes with the same digit, by eight ballots (a match instruction takes longer)
          unsigned peers = __ballot_sync(full, valid);
#pragma unroll
          for (int b = 0; b < 8; b++) {
            const unsigned bal = __ballot_sync(full, (d >> b) & 1u);
            peers &= (d >> b) & 1u ? bal : ~bal;
          }
          const uint32_t before = valid ? S.wcnt[warp][d] : 0u;
          rk[k] = before + __popc(peers & lt_mask);
          __syncwarp();
          if (valid && (uint32_t)(__ffs(peers) - 1) == lane) S.wcnt[warp][d] = (uint16_t)(before + __popc(peers));
          __syncwarp();
        }
      }
    }
    __syncthreads();
    const uint32_t dg = tid / PARTS, part = tid % PARTS;
    {
      uint32_t run = 0;
#pragma unroll
      for (uint32_t w = 0; w < WP; w++) {
        const uint32_t c = S.wcnt[part * WP + w][dg];
        S.wcnt[part * WP + w][dg] = (uint16_t)run;
        run += c;
      }
      uint32_t incl = run;
#pragma unroll
      for (uint32_t o = 1; o < PARTS; o <<= 1) {
        const uint32_t t = __shfl_up_sync(full, incl, o);
        if (part >= o) incl += t;
      }
      S.poff[part][dg] = incl - run;
      const uint32_t total = __shfl_sync(full, incl, (lane / PARTS) * PARTS + PARTS - 1);
      for (uint32_t r = part; r < C; r += PARTS) cl.map_shared_rank(&S.tots[rank][0], r)[dg] = total;
    }
    cl.sync();  // every block's digit counts have arrived
    uint32_t all = 0, before = 0;
    for (uint32_t r = part; r < C; r += PARTS) {
      const uint32_t c = S.tots[r][dg];
      all += c;
      before += r < rank ? c : 0u;
    }
#pragma unroll
    for (uint32_t o = 1; o < PARTS; o <<= 1) {
      all += __shfl_xor_sync(full, all, o);
      before += __shfl_xor_sync(full, before, o);
    }
    // exclusive scan over the digits: PARTS equal copies of each lie side by side
    uint32_t incl = all;
#pragma unroll
    for (uint32_t o = PARTS; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(full, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) S.red[warp][0] = (int)incl;
    __syncthreads();
    uint32_t pre = 0;
#pragma unroll 8
    for (uint32_t w = 0; w < W; w++) pre += w < warp ? (uint32_t)S.red[w][0] : 0u;
    if (part == 0) S.base[dg] = before + pre + incl - all;
    __syncthreads();
    uint2* const dst = pass & 1 ? kv1 : kv0;
    {
#pragma unroll
      for (uint32_t k = 0; k < kFusePer; k++) {
        if (k < K && warp * (32 * K) + k * 32 + lane < cntp) {
          const uint32_t d = (key[k] >> shift) & 255u;
          const uint32_t pos = S.base[d] + S.poff[warp / WP][d] + S.wcnt[warp][d] + rk[k];
          cl.map_shared_rank(dst, min(pos >> lp, C - 1))[pos & (P - 1)] =
              make_uint2(key[k], val[k]);
        }
      }
    }
    cl.sync();  // the keys have arrived; counts and sources may be overwritten
  }

  // ---- gather, tracking (gather_kernel, track_kernel) ----------------------------------
  for (uint32_t slot = tid; slot < cntp; slot += T) {
    const uint2 e = kv1[slot];
    const uint32_t i = off + base + slot;
    if (e.y >= n) {  // impossible for a permutation
      raise_err(st, GS_DERR_LOOKBACK);
      continue;
    }
    const uint32_t s = off + e.y;
    const float4 q0 = a.pin[2 * (size_t)s], q1 = a.pin[2 * (size_t)s + 1], sv = a.sin[s];
    a.keys[i] = e.x;
    a.vals[i] = s;
    a.pout[2 * (size_t)i] = q0;
    a.pout[2 * (size_t)i + 1] = q1;
    a.sout[i] = sv;
    s_pos[slot] = q0;
    if (a.track) {
      for (int h = 0; h < 2; h++) {
        if (S.central[h] != (long long)s) continue;
        st->central[h] = i;
        if (h < (int)st->p.haloCount) {
          const float q[3] = {q0.x, q0.y, q0.z};
          float* dst = h == 0 ? st->p.haloC1 : st->p.haloC2;
          for (int k = 0; k < 3; k++) {
            const double hc = st->halo_c[h][k];
            const double nv = __dadd_rn(hc, __dmul_rn(__dsub_rn((double)q[k], hc), 0.1));
            st->halo_c[h][k] = nv;
            dst[k] = __double2float_rn(nv);
          }
        }
      }
    }
  }

  // ---- leaf and start depths (tree_flags_kernel) ---------------------------------------
  uint32_t* const s_code = reinterpret_cast<uint32_t*>(R0);           // codes of [base - 16, base + P + 16)
  int8_t* const s_c16 = reinterpret_cast<int8_t*>(s_code + P + 32);   // cpd(j, j + 16) of [base - 16, base + P)
  int8_t* const s_m4 = s_c16 + P + 32;                                // its maxima over four
  uint8_t* const dlb = reinterpret_cast<uint8_t*>(s_m4 + P + 32);     // D | L << 4 of [base, base + P)
  for (uint32_t k = tid; k < P + 32; k += T) {
    const int g = (int)base - 16 + (int)k;
    uint32_t c = 0;
    if (g >= 0 && g < (int)n) {
      const uint32_t r = (uint32_t)g >> lp;
      c = (r == rank ? kv1 : cl.map_shared_rank(kv1, r))[(uint32_t)g & (P - 1)].x;
    }
    s_code[k] = c;
  }
  __syncthreads();
  for (uint32_t k = tid; k < P + 16; k += T) {
    const int j = (int)base - 16 + (int)k;
    s_c16[k] = (j >= 0 && j + 16 < (int)n) ? (int8_t)cpd(s_code[k], s_code[k + 16]) : (int8_t)-1;
  }
  for (uint32_t k = tid; k < (P >> 5); k += T) S.bits[k] = 0u;
  if (tid < kDepths) S.lastpos[tid] = 0u;
  __syncthreads();
  for (uint32_t k = tid; k < P + 12; k += T)
    s_m4[k] = max(max(s_c16[k], s_c16[k + 1]), max(s_c16[k + 2], s_c16[k + 3]));
  __syncthreads();
  // The particles that start nodes are those with D <= L (the leaf starts).
#pragma unroll 1
  for (uint32_t c0 = 0; c0 < P; c0 += T) {
    const uint32_t loc = c0 + tid;
    bool starts = false;
    if (loc < cntp) {
      int D = 0;
      if (base + loc > 0) {
        const uint32_t x0 = s_code[loc + 15], x1 = s_code[loc + 16];
        D = x0 == x1 ? 11 : cpd(x0, x1) + 1;
      }
      const int M = max(max(max((int)s_m4[loc], (int)s_m4[loc + 4]), max((int)s_m4[loc + 8], (int)s_m4[loc + 12])),
                        (int)s_c16[loc + 16]);
      const int L = min(kMaxLevel, M + 1);
      starts = D <= L;
      dlb[loc] = (uint8_t)(D | (L << 4));
    }
    const uint32_t bal = __ballot_sync(full, starts);
    if (lane == 0) S.bits[loc >> 5] = bal;
  }
  __syncthreads();
  if (warp == 0) {  // starts before each word
    uint32_t run = 0;
    for (uint32_t w0 = 0; w0 < (P >> 5); w0 += 32) {
      const uint32_t v = w0 + lane < (P >> 5) ? __popc(S.bits[w0 + lane]) : 0u;
      uint32_t incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(full, incl, o);
        if ((int)lane >= o) incl += t;
      }
      if (w0 + lane < (P >> 5)) S.wpre[w0 + lane] = run + incl - v;
      run += __shfl_sync(full, incl, 31);
    }
    if (lane == 0) S.nstart = run;
  } else if (warp == 1) {
    if (lane < kCounters) S.pub.cnt[lane] = 0u;
    if (lane < 6) S.run[lane] = 0u;
  }
  __syncthreads();
  // counts per depth, and the last start of depth <= d
#pragma unroll 1
  for (uint32_t c0 = 0; c0 < P; c0 += T) {
    const uint32_t loc = c0 + tid;
    const uint32_t word = S.bits[loc >> 5];
    const bool starts = (word >> lane) & 1u;
    if (!__any_sync(full, starts)) continue;
    const uint32_t dl = starts ? dlb[loc] : 0u;
    const uint32_t rk1 = S.wpre[loc >> 5] + __popc(word & lt_mask) + 1;
    const int D = dl & 15, L = dl >> 4;
    uint32_t mc = 0, ml = 0;  // lane d keeps depth d's count and last start
#pragma unroll
    for (int d = 0; d < kDepths; d++) {
      const uint32_t in = __ballot_sync(full, starts && D <= d && d <= L);
      const uint32_t le = __ballot_sync(full, starts && D <= d);
      const int top = 31 - __clz(le);
      const uint32_t lr = __shfl_sync(full, rk1, top & 31);
      if ((int)lane == d) {
        mc = __popc(in);
        ml = le ? lr << 1 | ((in >> top) & 1u) : 0u;
      }
    }
    if (lane == 11) mc = __popc(word);
    if (lane < kCounters && mc) atomicAdd(&S.pub.cnt[lane], mc);
    if (lane < kDepths && ml) atomicMax(&S.lastpos[lane], ml);
  }
  __syncthreads();
  if (tid < C * kCounters)
    cl.map_shared_rank(&S.cnts[rank][0], tid / kCounters)[tid % kCounters] = S.pub.cnt[tid % kCounters];
  cl.sync();  // every block's node counts have arrived, and its codes are read
  if (tid < kCounters) {  // counts -> offsets of each block, level totals
    uint32_t run = 0;
    for (uint32_t r = 0; r < C; r++) {
      S.off[r][tid] = run;
      run += S.cnts[r][tid];
    }
    if (tid < kDepths) S.lc[tid] = run;
    else S.lc[kDepths] = run;  // leaves
  }
  __syncthreads();
  if (warp == 0) {  // lane d: level d
    const uint32_t lc = lane < kDepths ? S.lc[lane] : 0u, cn = lane < kDepths ? S.pub.cnt[lane] : 0u;
    uint32_t ls = lc, lb = cn;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const uint32_t t = __shfl_up_sync(full, ls, o), u = __shfl_up_sync(full, lb, o);
      if ((int)lane >= o) {
        ls += t;
        lb += u;
      }
    }
    const uint32_t nodes = __shfl_sync(full, ls, kDepths - 1);
    if (lane <= kDepths) {  // exclusive; lane kDepths has the totals
      S.ls[lane] = ls - lc;
      S.lbase[lane] = lb - cn;
    }
    uint32_t dn = 0;  // start depth of the next block's first particle
    if (cntp == P && base + P < n) {
      const uint32_t c0 = s_code[P + 15], c1 = s_code[P + 16];
      dn = c0 == c1 ? 11u : (uint32_t)cpd(c0, c1) + 1u;
    }
    // the depth d group open at the block's end is a node this block started (not
    // one of an earlier block, nor a leaf of less depth) and goes on in the next block
    const uint32_t span = __ballot_sync(full, lane < kDepths && dn > lane && (S.lastpos[min(lane, 10u)] & 1u));
    uint32_t fl = ~0u;
    for (uint32_t w0 = 0; w0 < (P >> 5) && fl == ~0u; w0 += 32) {
      const uint32_t v = w0 + lane < (P >> 5) ? S.bits[w0 + lane] : 0u;
      const uint32_t some = __ballot_sync(full, v != 0u);
      if (some) {
        const int w = __ffs(some) - 1;
        fl = 32 * (w0 + w) + __ffs(__shfl_sync(full, v, w)) - 1;
      }
    }
    const uint32_t levels = 32 - __clz(__ballot_sync(full, lc != 0u));
    if (lane == 0) {
      S.overflow = nodes > a.sd.node_cap ? 1u : 0u;
      S.pub.span = span;
      S.pub.first_leaf = fl;
    }
    if (rank == 0) {
      TreeMeta* const m = a.b.meta + a.sd.slot;
      if (lane <= kDepths) {
        m->level_start[lane] = ls - lc;
        m->level_count[lane] = lc;
      }
      if (lane == 0) {
        m->num_nodes = nodes;
        m->num_levels = levels;
        m->num_leaves = S.lc[kDepths];
        m->overflow = nodes > a.sd.node_cap ? 1u : 0u;
        m->root_size = S.frame.size;
        if (nodes > a.sd.node_cap) raise_err(st, GS_DERR_NODES);
      }
    }
  }
  if (tid < kDepths) {
    S.pub.first[tid] = tid < kMaxLevel ? S.pub.cnt[tid + 1] : 0u;
    S.pub.last[tid] = 0u;
  }
  __syncthreads();
  if (S.overflow) {  // the same in every block
    cl.sync();
    return;
  }

  // ---- node indices, parents, child bases, leaf lists (tree_emit_kernel) ----------------
  uint32_t* const s_nd = reinterpret_cast<uint32_t*>(R1);  // the block's nodes, by depth then order
  const uint32_t no = a.sd.node_off;
  const uint32_t nd_cap = (8 * P + 512) / 4;               // at most 1.59 P + 10 nodes start in a block
  uint16_t* const s_start = reinterpret_cast<uint16_t*>(s_com);  // slots of the starts (the COMs come later)
#pragma unroll 1
  for (uint32_t loc = tid; loc < cntp; loc += T) {
    const uint32_t word = S.bits[loc >> 5];
    if ((word >> lane) & 1u) s_start[S.wpre[loc >> 5] + __popc(word & lt_mask)] = (uint16_t)loc;
  }
  __syncthreads();
#pragma unroll 1
  for (uint32_t c0 = 0; c0 < S.nstart; c0 += T) {
    const bool has = c0 + tid < S.nstart;
    const uint32_t loc = has ? s_start[c0 + tid] : 0u, dl = has ? dlb[loc] : 15u;  // none: D = 15
    const int D = dl & 15, L = dl >> 4;
    uint32_t ex[6];  // packed counts before this start: depths 2w (low half) and 2w + 1
#pragma unroll
    for (int w = 0; w < 6; w++) {
      const uint32_t v = (D <= 2 * w && 2 * w <= L ? 1u : 0u) | (D <= 2 * w + 1 && 2 * w + 1 <= L ? 0x10000u : 0u);
      uint32_t incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(full, incl, o);
        if ((int)lane >= o) incl += t;
      }
      ex[w] = incl - v;
      if (lane == 31) S.wc[warp][w] = incl;
    }
    __syncthreads();
    if (warp < 6) {
      const uint32_t v = lane < W ? S.wc[lane][warp] : 0u;
      uint32_t incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(full, incl, o);
        if ((int)lane >= o) incl += t;
      }
      const uint32_t before = S.run[warp];
      __syncwarp();
      if (lane < W) S.wc[lane][warp] = before + incl - v;
      if (lane == 31) S.run[warp] = before + incl;
    }
    __syncthreads();
    if (has) {
#pragma unroll
      for (int w = 0; w < 6; w++) ex[w] += S.wc[warp][w];
      const uint32_t i = off + base + loc, lr = c0 + tid;
      // mortonTree.js:127: an internal node with numNodes + 8 > maxNodes would be a leaf
#pragma unroll
      for (int d = 0; d < kDepths; d++) {
        if (D <= d && d <= L) {
          const uint32_t j = (ex[d >> 1] >> (16 * (d & 1))) & 0xffffu;  // among the block's depth d nodes
          const uint32_t j1 = d < kMaxLevel ? (ex[(d + 1) >> 1] >> (16 * ((d + 1) & 1))) & 0xffffu : 0u;
          const uint32_t nl = S.ls[d] + S.off[rank][d] + j, nn = no + nl;
          a.b.node_start[nn] = i;
          a.b.depth[nn] = (uint8_t)d;
          a.b.child_base[nn] = no + (d < kMaxLevel ? S.ls[d + 1] + S.off[rank][d + 1] + j1 : S.ls[kDepths]);
          int32_t par = -1;
          if (d > 0) {
            const uint32_t jp = (ex[(d - 1) >> 1] >> (16 * ((d - 1) & 1))) & 0xffffu;
            par = (int32_t)(no + S.ls[d - 1] + S.off[rank][d - 1] + jp + (D <= d - 1 ? 1u : 0u) - 1u);
          }
          a.b.parent[nn] = par;
          const uint32_t ent = fuse_entry(d == L, loc, j1);
          const uint32_t ln = S.lbase[d] + j;
          if (ln < nd_cap) s_nd[ln] = ent;
          else raise_err(st, GS_DERR_NODES);
          if (j == 0) S.pub.first[d] = j1;
          if (j + 1 == S.pub.cnt[d]) S.pub.last[d] = ent;
          if (d == L) {
            a.b.leaf_node[off + S.off[rank][11] + lr] = nn;
            a.b.leaf_start[off + S.off[rank][11] + lr] = i;
          }
          if (d < L && nl + 1 + 8 > a.sd.max_nodes) raise_err(st, GS_DERR_NODES);
        }
      }
    }
    __syncthreads();  // the next chunk rewrites the warps' counts
  }
  if (tid < sizeof(FusePub) / 4)  // block 0 sums the spanning nodes
    reinterpret_cast<uint32_t*>(cl.map_shared_rank(&S.pubs[rank], 0))[tid] =
        reinterpret_cast<const uint32_t*>(&S.pub)[tid];
  __syncthreads();

  // ---- COMs of the nodes inside the block (tree_leaves_kernel's arithmetic) -------------
  const uint32_t com_cap = fuse_com_cap(lp), mine = S.lbase[kDepths], span = S.pub.span;
  for (uint32_t ln = tid; ln < min(mine, nd_cap); ln += T) {  // leaves
    const uint32_t ent = s_nd[ln];
    if (!(ent >> 31)) continue;
    int d = 0;
    while (ln >= S.lbase[d + 1]) d++;
    const uint32_t j = ln - S.lbase[d];
    if (j + 1 == S.pub.cnt[d] && ((span >> d) & 1u)) continue;  // reaches into the next block
    const uint32_t lo = (ent >> 16) & 0x7fffu;
    uint32_t w = (lo + 1) >> 5, hi = cntp;
    uint32_t b = w < (cntp + 31) / 32 ? S.bits[w] & (0xffffffffu << ((lo + 1) & 31)) : 0u;
    while (!b && ++w < (cntp + 31) / 32) b = S.bits[w];
    if (b) hi = min(hi, 32 * w + __ffs(b) - 1);
    ComSum<false> sum;
    for (uint32_t k0 = lo; k0 < hi; k0 += 4) {
      float4 q[4];
#pragma unroll
      for (uint32_t k = 0; k < 4; k++) q[k] = s_pos[min(k0 + k, hi - 1)];
#pragma unroll
      for (uint32_t k = 0; k < 4; k++)
        if (k0 + k < hi) sum.add(q[k]);
    }
    const float4 c = sum.mean();
    const float size = S.size[d];
    const uint32_t nn = no + S.ls[d] + S.off[rank][d] + j;
    if (ln < com_cap) s_com[ln] = c;
    a.b.cm[nn] = c;
    a.b.info[nn] = walk_info(size, off + base + lo, kLeafBit | (hi - lo));
  }
  __syncthreads();
  for (int d = kMaxLevel - 1; d >= 0; d--) {
    if (S.lc[d + 1] == 0) continue;  // nothing below, in any block
    const uint32_t cd = S.pub.cnt[d], strad = (span >> d) & 1u;
    const float size = S.size[d];
    for (uint32_t j = tid; j + strad < cd; j += T) {
      const uint32_t ln = S.lbase[d] + j;
      const uint32_t ent = s_nd[ln];
      if (ent >> 31) continue;
      const uint32_t j0 = ent & 0xffffu, j1 = j + 1 < cd ? s_nd[ln + 1] & 0xffffu : S.pub.cnt[d + 1];
      const uint32_t nc = j1 - j0, cb = no + S.ls[d + 1] + S.off[rank][d + 1] + j0;
      if (nc == 0 || nc > 8) {
        raise_err(st, GS_DERR_NODES);  // impossible for a correct numbering
        continue;
      }
      ComSum<MODE == kComF64> sum;
      const uint32_t lc = S.lbase[d + 1] + j0;
      float4 q[8];  // loads together, sums in slot order
#pragma unroll
      for (uint32_t k = 0; k < 8; k++) {
        const uint32_t kk = min(k, nc - 1);
        q[k] = lc + kk < com_cap ? s_com[lc + kk] : __ldcg(&a.b.cm[cb + kk]);
      }
#pragma unroll
      for (uint32_t k = 0; k < 8; k++)
        if (k < nc) sum.add(q[k]);
      const float4 c = sum.mean();
      const uint32_t nn = no + S.ls[d] + S.off[rank][d] + j;
      if (ln < com_cap) s_com[ln] = c;
      a.b.cm[nn] = c;
      a.b.info[nn] = walk_info(size, cb, nc);
    }
    __syncthreads();
  }

  // ---- nodes that span blocks, by block 0 ----------------------------------------------
  cl.sync();  // every block's nodes and tables are written
  if (rank == 0) {
    for (uint32_t e = tid; e < kFuseStrad; e += T) {
      const uint32_t d = e / kFuseCtas, r = e % kFuseCtas;
      const FusePub& p = S.pubs[r];
      uint4 m = make_uint4(0u, 0u, 0u, ~0u);  // no spanning node
      if (r < C && ((p.span >> d) & 1u)) {
        m.x = no + S.ls[d] + S.off[r][d] + p.cnt[d] - 1;
        const uint32_t ent = p.last[d];
        if (ent >> 31) {  // a leaf: up to the next leaf start
          const uint32_t lo = (r << lp) + ((ent >> 16) & 0x7fffu);
          uint32_t hi = n;
          for (uint32_t q = r + 1; q < C; q++)
            if (S.pubs[q].first_leaf != ~0u) {
              hi = (q << lp) + S.pubs[q].first_leaf;
              break;
            }
          ComSum<false> sum;
          for (uint32_t k0 = lo; k0 < hi; k0 += kComChunk) {
            float4 q[kComChunk];
#pragma unroll
            for (int k = 0; k < kComChunk; k++)
              q[k] = __ldcg(&a.pout[2 * (size_t)(off + min(k0 + k, hi - 1))]);
#pragma unroll
            for (int k = 0; k < kComChunk; k++)
              if (k0 + k < hi) sum.add(q[k]);
          }
          S.scom[e] = sum.mean();
          m.y = off + lo;
          m.z = kLeafBit | (hi - lo);
          m.w = 1u;
        } else {
          const uint32_t j0 = ent & 0xffffu;
          uint32_t nc = p.cnt[d + 1] - j0;
          for (uint32_t q = r + 1; q < C; q++) {
            nc += S.pubs[q].first[d];
            if (S.pubs[q].cnt[d]) break;
          }
          m.y = no + S.ls[d + 1] + S.off[r][d + 1] + j0;
          m.z = min(nc, 8u);
          m.w = 0u;
          if (nc == 0 || nc > 8) raise_err(st, GS_DERR_NODES);  // impossible for a correct numbering
        }
      }
      S.sm[e] = m;
      if (m.w != ~0u && d > 0) {  // its parent spans blocks too: the last one of depth d - 1 started so far
        uint32_t q = r;
        while (q > 0 && !((S.pubs[q].span >> (d - 1)) & 1u)) q--;
        S.par[e] = (d - 1) * kFuseCtas + q;
      }
    }
    __syncthreads();
    constexpr uint32_t kChild = (8 * kFuseStrad + T - 1) / T;
    float4 child[kChild];  // all their children, loads together
#pragma unroll
    for (uint32_t q = 0; q < kChild; q++) {
      const uint32_t k = tid + q * T;
      const uint4 m = k < 8 * kFuseStrad ? S.sm[k >> 3] : make_uint4(0u, 0u, 0u, ~0u);
      if (m.w == 0u && (k & 7) < m.z) child[q] = __ldcg(&a.b.cm[m.y + (k & 7)]);
    }
#pragma unroll
    for (uint32_t q = 0; q < kChild; q++) {
      const uint32_t k = tid + q * T;
      if (k < 8 * kFuseStrad) S.ch[k] = child[q];  // slots past a node's children are not read
    }
    __syncthreads();
    if (warp == 0) {
      for (int d = kDepths - 1; d >= 0; d--) {
        const uint32_t e = d * kFuseCtas + lane;
        const uint4 m = lane < kFuseCtas ? S.sm[e] : make_uint4(0u, 0u, 0u, ~0u);
        if (!__any_sync(full, m.w != ~0u)) continue;
        if (m.w != ~0u) {
          float4 c;
          if (m.w == 1u) {
            c = S.scom[e];
          } else {
            ComSum<MODE == kComF64> sum;
            float4 q[8];
#pragma unroll
            for (uint32_t k = 0; k < 8; k++) q[k] = S.ch[8 * e + min(k, m.z - 1)];
#pragma unroll
            for (uint32_t k = 0; k < 8; k++)
              if (k < m.z) sum.add(q[k]);
            c = sum.mean();
          }
          a.b.cm[m.x] = c;
          a.b.info[m.x] = walk_info(S.size[d], m.y, m.z);
          if (d > 0) {
            const uint32_t pe = S.par[e], k = m.x - S.sm[pe].y;
            if (S.sm[pe].w == 0u && k < 8u) S.ch[8 * pe + k] = c;
          }
        }
        __syncwarp();
      }
    }
  }
  cl.sync();  // no block leaves while block 0 reads its tables
}

}  // namespace gs
