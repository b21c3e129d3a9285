// Node numbering and COMs of a rebuild in one kernel, a block per build tile of 1024
// sorted particles (galaxies too large for the one-cluster rebuild, and pools).
//
// What bounds it: latency. Numbering and COMs as two kernels (tree_emit_kernel, then
// tree_leaves_kernel, whose threads carry every node to its parent over global
// memory) took 8 and 25 us at any size: a node's COM, its parent's arrival counter and the
// siblings' COMs are three dependent round trips to L2 per level. Here a node whose
// particles lie in the tile is summed by the block, level by level, from shared memory;
// only a node that spans tiles takes arrivals over global memory, and such nodes
// lie at the upper levels. With the flags joined to the gather, full step in us before /
// after: 60001 particles (theta 0.7) 168.5 / 162.9, 100000 320 / 313, sphere of 200003 369 / 358, 524288
// 1109 / 1098, 2^20 2197 / 2184. What is left is the chain of arrivals to the root.
//
// A spanning node: the tile that starts it knows its first child cb, the tile in which it
// ends the child after its last, ce (both galaxy-local, cb >= 1), and its children finish
// in any tile between. Its arrival counter gets +1 per finished child, +cb from the first
// tile and -ce from the last: it is zero when all have arrived and not before, since k
// children without the others leave k > 0, with cb k + cb > 0, and with ce at
// most k - ce <= -cb < 0. Whoever brings it to zero sums the children in slot order and
// arrives at the next parent. No tile waits, and the counter ends at zero.
#pragma once
#include "build.cuh"
#include "common.cuh"

namespace gs {

constexpr uint32_t kTileComs = kFlagTile / 2 + 64;       // COMs kept in shared memory
constexpr uint32_t kTileNodes = 2 * kFlagTile + 128;     // at most 1.59 x 1024 + 10 nodes start in a tile

struct TileTreeSmem {
  float4 pos[kFlagTile];
  float4 com[kTileComs];
  uint32_t nd[kTileNodes];          // nodes by depth, then order: leaf bit, slot << 16, first child
  uint32_t start[kFlagTile + 1];    // the starts: slot | D << 16 | L << 24; then the tile's end
  uint32_t bits[kFlagTile / 32], wpre[kFlagTile / 32], nstart;
  uint32_t wc[kFlagThreads / 32][6], run[6];
  uint32_t ls[kDepths + 1], off[kCounters], cnt[kCounters], lbase[kDepths + 1];
  uint32_t first[kDepths];          // depth d + 1 nodes before the first start with D <= d
  uint32_t found, span;             // bit d: such a start exists; the last depth d node spans tiles
  uint32_t last[kDepths];           // entry of the last depth d node
  uint32_t open, overflow, dnext;
  float size[kDepths];
};

// Adds to the arrival counter of spanning node `up` (galaxy-local, depth d); the arrival
// that completes it sums its children and goes on to its parent.
template <int MODE>
__device__ __forceinline__ void tile_arrive(const BuildBuffers& b, const float* size, uint32_t no, uint32_t up, int d,
                                            int add, DevState* st) {
  while (true) {
    const int old = (int)cuda::atomic_ref<uint32_t, cuda::thread_scope_device>(b.arrive[no + up])
                        .fetch_add((uint32_t)add, cuda::memory_order_acq_rel);
    if (old + add != 0) return;
    const uint32_t cb = __ldcg(&b.child_base[no + up]);
    const uint32_t ce = __ldcg(&b.info[no + up].child);  // left there by the tile it ends in
    const int32_t pp = __ldcg(&b.parent[no + up]);
    const uint32_t nc = no + ce - cb;
    if (nc == 0 || nc > 8 || d < 0) {
      raise_err(st, GS_DERR_NODES);  // impossible for a correct numbering
      return;
    }
    float4 q[8];
#pragma unroll
    for (uint32_t k = 0; k < 8; k++) q[k] = __ldcg(&b.cm[cb + min(k, nc - 1)]);
    ComSum<MODE == kComF64> sum;
#pragma unroll
    for (uint32_t k = 0; k < 8; k++)
      if (k < nc) sum.add(q[k]);
    b.cm[no + up] = sum.mean();
    b.info[no + up] = walk_info(size[d], cb, nc);
    if (pp < 0) return;
    up = (uint32_t)pp - no;
    d--;
    add = 1;
  }
}

template <int MODE>
__global__ void __launch_bounds__(kFlagThreads)
    tree_tile_kernel(BuildBuffers b, Layout Lo, const float4* __restrict__ pos, DevState* sts) {
  griddep_wait();  // launched with a programmatic dependency: predecessors' writes first
  __shared__ TileTreeSmem S;
  constexpr uint32_t T = kFlagThreads, W = T / 32, P = kFlagTile;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tile = blockIdx.x;
  const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
  const SegDesc sd = Lo.segs[Lo.seg_of_flag_tile[tile]];
  DevState* const st = sts + sd.slot;
  const uint32_t seg_end = sd.off + sd.n, base = sd.off + (tile - sd.flag_tile0) * P;
  const uint32_t cntp = min(P, seg_end - base), no = sd.node_off;
  const bool last_tile = base + P >= seg_end;
  const TreeMeta& m = b.meta[sd.slot];
  uint32_t dl4[P / T];
  float4 p4[P / T];
#pragma unroll
  for (uint32_t q = 0; q < P / T; q++) {  // loads together
    const uint32_t k = q * T + tid;
    dl4[q] = k < cntp ? b.dl[base + k] : 15u;  // none: D = 15
    p4[q] = pos[2 * (size_t)(base + min(k, cntp - 1))];
  }
  if (tid < kCounters) {
    S.off[tid] = b.blk_offs[(size_t)tile * kTileWords + tid];
    S.cnt[tid] = b.blk_counts[(size_t)tile * kTileWords + tid];
  } else if (tid >= 32 && tid < 32 + kDepths + 1) {
    S.ls[tid - 32] = m.level_start[tid - 32];
  } else if (tid >= 64 && tid < 64 + kDepths) {
    S.size[tid - 64] = __double2float_rn(ldexp(m.root_size, -(int)(tid - 64)));
    S.last[tid - 64] = 0u;
  } else if (tid == 96) {
    // a node that ends just where the tile begins (its first start has D <= d) spans nothing
    S.open = b.blk_offs[(size_t)tile * kTileWords + kCounters] & ((1u << (b.dl[base] & 15u)) - 1u);
    S.overflow = m.overflow;
    S.dnext = last_tile ? 0u : b.dl[base + P] & 15u;
    S.found = S.span = 0u;
  } else if (tid >= 128 && tid < 128 + 6) {
    S.run[tid - 128] = 0u;
  }

  // ---- the starts (D <= L), as a list in order -------------------------------------------
  uint32_t bal[P / T];
#pragma unroll
  for (uint32_t q = 0; q < P / T; q++) {
    S.pos[q * T + tid] = p4[q];
    bal[q] = __ballot_sync(full, (dl4[q] & 15u) <= dl4[q] >> 4);
    if (lane == 0) S.bits[q * W + warp] = bal[q];
  }
  __syncthreads();
  if (S.overflow) return;
  if (warp == 0) {
    const uint32_t v = __popc(S.bits[lane]);
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(full, incl, o);
      if ((int)lane >= o) incl += t;
    }
    S.wpre[lane] = incl - v;
    if (lane == 31) S.nstart = incl;
  } else if (warp == 1) {
    const uint32_t cn = lane < kDepths ? S.cnt[lane] : 0u;
    uint32_t lb = cn;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const uint32_t t = __shfl_up_sync(full, lb, o);
      if ((int)lane >= o) lb += t;
    }
    if (lane <= kDepths) S.lbase[lane] = lb - cn;
  }
  __syncthreads();
#pragma unroll
  for (uint32_t q = 0; q < P / T; q++)
    if ((bal[q] >> lane) & 1u)
      S.start[S.wpre[q * W + warp] + __popc(bal[q] & below)] =
          (q * T + tid) | (dl4[q] & 15u) << 16 | (dl4[q] >> 4) << 24;
  const uint32_t nstart = S.nstart, dnext = S.dnext;
  if (tid == 0) S.start[nstart] = cntp;
  __syncthreads();
  for (uint32_t d = warp; d < kDepths; d += W) {  // per depth: first and last start with D <= d
    uint32_t before = 0;
    bool hit = false;
    for (uint32_t k0 = 0; k0 < nstart && !hit; k0 += 32) {
      const uint32_t D = k0 + lane < nstart ? (S.start[k0 + lane] >> 16) & 15u : 15u;
      const uint32_t le = __ballot_sync(full, D <= d), eq = __ballot_sync(full, D == d + 1);
      hit = le != 0u;
      before += __popc(hit ? eq & ((le & (0u - le)) - 1u) : eq);
    }
    bool spans = false;
    for (int k0 = ((int)nstart - 1) & ~31; k0 >= 0 && hit; k0 -= 32) {
      const uint32_t x = k0 + lane < nstart ? S.start[k0 + lane] : 15u << 16;
      const uint32_t le = __ballot_sync(full, ((x >> 16) & 15u) <= d);
      if (!le) continue;
      spans = dnext > d && __shfl_sync(full, x >> 24, 31 - __clz(le)) > d;  // an internal node that goes on in the next tile
      break;
    }
    if (lane == 0) {
      S.first[d] = before;
      if (hit) atomicOr(&S.found, 1u << d);
      if (spans) atomicOr(&S.span, 1u << d);
    }
  }
  // ---- node indices, parents, child bases, leaf lists (tree_emit_kernel); leaf COMs -------
#pragma unroll 1
  for (uint32_t c0 = 0; c0 < nstart; c0 += T) {
    const bool has = c0 + tid < nstart;
    const uint32_t sv = has ? S.start[c0 + tid] : 15u << 16, loc = sv & 0xffffu;  // none: D = 15
    const int D = (sv >> 16) & 15, L = sv >> 24;
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
      const uint32_t run = S.run[warp];
      __syncwarp();
      if (lane < W) S.wc[lane][warp] = run + incl - v;
      if (lane == 31) S.run[warp] = run + incl;
    }
    __syncthreads();
    if (has) {
#pragma unroll
      for (int w = 0; w < 6; w++) ex[w] += S.wc[warp][w];
      const uint32_t i = base + loc, lr = sd.off + S.off[11] + c0 + tid;
      uint32_t leaf_ln = 0, leaf_nn = 0;
#pragma unroll
      for (int d = 0; d < kDepths; d++) {
        if (D <= d && d <= L) {
          const uint32_t j = (ex[d >> 1] >> (16 * (d & 1))) & 0xffffu;  // among the tile's depth d nodes
          const uint32_t j1 = d < kMaxLevel ? (ex[(d + 1) >> 1] >> (16 * ((d + 1) & 1))) & 0xffffu : 0u;
          const uint32_t nl = S.ls[d] + S.off[d] + j, nn = no + nl;
          b.node_start[nn] = i;
          b.depth[nn] = (uint8_t)d;
          b.child_base[nn] = no + (d < kMaxLevel ? S.ls[d + 1] + S.off[d + 1] + j1 : S.ls[kDepths]);
          int32_t par = -1;
          if (d > 0) {
            const uint32_t jp = (ex[(d - 1) >> 1] >> (16 * ((d - 1) & 1))) & 0xffffu;
            par = (int32_t)(no + S.ls[d - 1] + S.off[d - 1] + jp + (D <= d - 1 ? 1u : 0u) - 1u);
          }
          b.parent[nn] = par;
          const uint32_t ent = (d == L ? 0x80000000u : 0u) | (loc << 16) | j1;
          const uint32_t ln = S.lbase[d] + j;
          if (ln < kTileNodes) S.nd[ln] = ent;
          else raise_err(st, GS_DERR_NODES);
          if (j + 1 == S.cnt[d]) S.last[d] = ent;
          if (d == L) {
            leaf_ln = ln;
            leaf_nn = nn;
          }
          // mortonTree.js:127: an internal node with numNodes + 8 > maxNodes would be a leaf
          if (d < L && nl + 1 + 8 > sd.max_nodes) raise_err(st, GS_DERR_NODES);
        }
      }
      // the start's leaf: up to the next start
      b.leaf_node[lr] = leaf_nn;
      b.leaf_start[lr] = i;
      const uint32_t hi = S.start[c0 + tid + 1] & 0xffffu;
      ComSum<false> sum;
      for (uint32_t k0 = loc; k0 < hi; k0 += 4) {
        float4 q[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) q[k] = S.pos[min(k0 + k, hi - 1)];
#pragma unroll
        for (uint32_t k = 0; k < 4; k++)
          if (k0 + k < hi) sum.add(q[k]);
      }
      uint32_t end = base + hi;
      if (c0 + tid + 1 == nstart && dnext > (uint32_t)L) {  // it goes on in the next tile
        // its end first, past tiles without a start by their counts, then by the flags, then its
        // records, both kComChunk loads at a time: one particle per trip, its flag before its
        // record, took 11.2 ms for the rebuild of 100000 particles half of which are at one
        // place, 2.6 ms so (sphere of 200003: 88 -> 86 us)
        const uint32_t from = end;
        for (uint32_t x = tile + 1; end < seg_end && b.blk_counts[(size_t)x * kTileWords + kMaxLevel + 1] == 0; x++)
          end += P;
        for (bool more = end < seg_end; more; more = more && end < seg_end) {
          uint32_t f[kComChunk];
#pragma unroll
          for (uint32_t k = 0; k < kComChunk; k++) f[k] = end + k < seg_end ? b.dl[end + k] : 0u;
#pragma unroll
          for (uint32_t k = 0; k < kComChunk; k++) {
            more = more && (f[k] & 15u) > f[k] >> 4;  // past the galaxy: 0, a start
            end += more ? 1u : 0u;
          }
        }
        end = min(end, seg_end);
        for (uint32_t k0 = from; k0 < end; k0 += kComChunk) {
          float4 q[kComChunk];
#pragma unroll
          for (uint32_t k = 0; k < kComChunk; k++) q[k] = pos[2 * (size_t)min(k0 + k, end - 1)];
#pragma unroll
          for (uint32_t k = 0; k < kComChunk; k++)
            if (k0 + k < end) sum.add(q[k]);
        }
      }
      const float4 c = sum.mean();
      if (leaf_ln < kTileComs) S.com[leaf_ln] = c;
      b.cm[leaf_nn] = c;
      b.info[leaf_nn] = walk_info(S.size[L], i, kLeafBit | (end - i));
    }
    __syncthreads();  // the next chunk rewrites the warps' counts
  }
  __syncthreads();

  // ---- COMs of the internal nodes inside the tile ------------------------------------------
  const uint32_t span = S.span;
  for (int d = kMaxLevel - 1; d >= 0; d--) {
    if (S.cnt[d + 1] == 0) continue;  // no node of this depth has all its children here
    const uint32_t cd = S.cnt[d], strad = (span >> d) & 1u;
    const float size = S.size[d];
    for (uint32_t j = tid; j + strad < cd; j += T) {
      const uint32_t ln = S.lbase[d] + j;
      const uint32_t ent = S.nd[ln];
      if (ent >> 31) continue;
      const uint32_t j0 = ent & 0xffffu, j1 = j + 1 < cd ? S.nd[ln + 1] & 0xffffu : S.cnt[d + 1];
      const uint32_t nc = j1 - j0, cb = no + S.ls[d + 1] + S.off[d + 1] + j0;
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
        q[k] = lc + kk < kTileComs ? S.com[lc + kk] : __ldcg(&b.cm[cb + kk]);
      }
#pragma unroll
      for (uint32_t k = 0; k < 8; k++)
        if (k < nc) sum.add(q[k]);
      const float4 c = sum.mean();
      const uint32_t nn = no + S.ls[d] + S.off[d] + j;
      if (ln < kTileComs) S.com[ln] = c;
      b.cm[nn] = c;
      b.info[nn] = walk_info(size, cb, nc);
    }
    __syncthreads();
  }

  // ---- arrivals at the nodes that span tiles ----------------------------------------------
  // at most 8 children of a node of an earlier tile and 8 of one that goes on, per depth
  if (tid < 16 * kMaxLevel) {
    const int d = 1 + tid / 16;
    const uint32_t k = tid % 16, f = S.first[d - 1], cn = S.cnt[d];
    const bool goes_on = (span >> (d - 1)) & 1u;
    const uint32_t j0 = goes_on ? S.last[d - 1] & 0xffffu : cn;
    const bool early = k < 8;
    const uint32_t j = early ? k : j0 + k - 8;
    const bool finished = !(j + 1 == cn && ((span >> d) & 1u));
    if (j < cn && finished && (early ? k < f : j >= f))
      tile_arrive<MODE>(b, S.size, no, S.ls[d - 1] + S.off[d - 1] + (early ? 0u : S.cnt[d - 1]) - 1, d - 1, 1, st);
  }
  if (tid < kMaxLevel) {  // nodes this tile starts that go on
    const int d = tid;
    if ((span >> d) & 1u)
      tile_arrive<MODE>(b, S.size, no, S.ls[d] + S.off[d] + S.cnt[d] - 1, d,
                        (int)(S.ls[d + 1] + S.off[d + 1] + (S.last[d] & 0xffffu)), st);
  } else if (tid >= 32 && tid < 32 + kMaxLevel) {  // nodes of earlier tiles that end here, or just after
    const int d = tid - 32;
    if (((S.open >> d) & 1u) && (((S.found >> d) & 1u) || dnext <= (uint32_t)d)) {
      const uint32_t n = S.ls[d] + S.off[d] - 1, ce = S.ls[d + 1] + S.off[d + 1] + S.first[d];
      b.info[no + n].child = ce;
      tile_arrive<MODE>(b, S.size, no, n, d, -(int)ce, st);
    }
  }
}

}  // namespace gs
