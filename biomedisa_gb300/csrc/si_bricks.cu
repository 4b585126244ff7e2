// Brick walker: the random walk of si_walk, reorganised so that every step
// reads its neighbourhood record from and counts its hit into SHARED memory.
//
// The crop is cut into core bricks of 10^3 voxels. A walker is processed by the
// CTA of the core brick that holds it, inside the 16^3 extended box of that
// brick (4 voxels of halo below, 2 above): the CTA loads the box's packed
// neighbourhood records with one TMA tensor copy, counts hits in a shared
// 16^3 counter array, and the walker advances until it leaves the box or ends
// its walk. Leaving walkers keep their state (position, step counter) and are
// re-bucketed for the next round; each round sorts all live walkers by
// (label slot, core brick) with a counting sort. Hits of a box are flushed to
// the global uint32 hit maps once per visit; the step that leaves a box adds
// its hit with a global atomic.
//
// Per-step semantics, randomness (Philox counter (t/4, seed pos, axis, label))
// and hence the integer hit maps are exactly those of si_walk
// (pycuda_small.py:138-257 semantics): integer sums do not depend on the order
// in which walkers or steps are processed.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <atomic>
#include <cstring>
#include <mutex>
#include <vector>

#include "si_common.cuh"
#include "si_internal.h"
#include "si_tma.cuh"

namespace si {
namespace {

constexpr int kCore = 10;   // core brick edge
constexpr int kLo = 4;      // halo below the core (even: TMA x alignment)
constexpr int kExt = 16;    // extended box edge (kLo + kCore + 2)
constexpr int kExtVox = kExt * kExt * kExt;
constexpr int kAdvThreads = 512;
constexpr uint32_t kChunk = 4096;  // sorted walkers per work ticket
constexpr int kScanBlock = 1024;   // elements per scan block (256 threads x 4)

// Threads of a CTA of float walker pairs, 3 CTAs per SM: a record is 8 registers
// a walker, and at 256 threads (80 registers) they spill (117x141x133, walk of
// 9.75e9 steps: 64.0 ms; 192 threads and 96 registers 57.8 ms, 128 x 5 60.4,
// 256 x 2 59.3).
constexpr int kFloatThreads = 192;

// Device counters of a sorted walk.
enum WalkCtr {
  kCtrLive = 0,    // walkers live after the last scan = states of the next sweep
  kCtrIn = 1,      // states the next scatter reads
  kCtrSweeps = 2,  // sweeps that ran
  kCtrOver = 3,    // round limit hit with live walkers
  kCtrWords = 4
};

struct BrickGeom {
  int Zc, Yc, Xc;
  int edge;  // brick edge used for bucketing
  int nbz, nby, nbx;
  uint32_t nb;   // bricks per label
  uint32_t label_step, brick_step;  // bucket = label slot * label_step + brick * brick_step
  uint32_t F;    // Yc * Xc
  uint32_t Xp;   // record row pitch (even)
  FastDiv by_F, by_X, by_edge;
};

// Walker state: x = position (crop linear index), y = seed index,
// z = step counter t, w = end of its walk (24 bits) | label slot << 24.
__device__ __forceinline__ bool live(const uint4& s) { return s.z != (s.w & 0xFFFFFFu); }

__device__ __forceinline__ void coords(const BrickGeom& g, uint32_t pos, int& z, int& y, int& x) {
  z = (int)g.by_F(pos);
  const uint32_t r = pos - (uint32_t)z * g.F;
  y = (int)g.by_X(r);
  x = (int)(r - (uint32_t)y * (uint32_t)g.Xc);
}

__device__ __forceinline__ uint32_t bucket_of(const BrickGeom& g, const uint4& s) {
  int z, y, x;
  coords(g, s.x, z, y, x);
  const uint32_t brick = (g.by_edge((uint32_t)z) * (uint32_t)g.nby + g.by_edge((uint32_t)y)) * (uint32_t)g.nbx +
                         g.by_edge((uint32_t)x);
  return (s.w >> 24) * g.label_step + brick * g.brick_step;
}

template <bool kFirst>
__device__ __forceinline__ bool fetch_state(uint64_t i, uint64_t n, const uint4* __restrict__ states,
                                            const SeedRec* __restrict__ seeds, uint32_t ns, int sorw, uint4& s) {
  if (i >= n) return false;
  if (kFirst) {
    const uint32_t w = (uint32_t)(i / ns);
    const uint32_t sidx = (uint32_t)(i - (uint64_t)w * ns);
    const SeedRec sd = seeds[sidx];
    s = make_uint4(sd.pos, sidx, w * (uint32_t)sorw, ((w + 1u) * (uint32_t)sorw) | (seed_slot(sd.meta) << 24));
    return true;
  }
  s = states[i];
  return live(s);
}

// Count (kScatter = false) or scatter (true) live walkers into buckets, with
// warp aggregation of equal keys. Scatter: counts are cursors relative to
// offsets, or absolute ones (offsets null).
template <bool kFirst, bool kScatter>
__global__ void __launch_bounds__(256) bucket_kernel(const uint4* __restrict__ states_in, uint64_t n,
                                                     const SeedRec* __restrict__ seeds, uint32_t ns, int sorw,
                                                     BrickGeom g, uint32_t* __restrict__ counts,
                                                     const uint32_t* __restrict__ offsets,
                                                     uint4* __restrict__ states_out,
                                                     const uint32_t* __restrict__ n_dev = nullptr) {
  if (n_dev) n = *n_dev;  // the count lives on the device (device-side sweep loop)
  const int lane = threadIdx.x & 31;
  // four states a thread, so that their loads and cursor atomics overlap (a
  // walker's load, atomic and store one after the other bound this pass)
  constexpr int N = 4;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += N * stride) {
    uint4 s[N];
    bool ok[N];
    uint32_t key[N], peers[N], at[N];
#pragma unroll
    for (int k = 0; k < N; ++k)
      ok[k] = fetch_state<kFirst>(base + k * stride + lane, n, states_in, seeds, ns, sorw, s[k]);
#pragma unroll
    for (int k = 0; k < N; ++k) {
      key[k] = ok[k] ? bucket_of(g, s[k]) : 0u;
      const uint32_t act = __ballot_sync(0xffffffffu, ok[k]);
      at[k] = peers[k] = 0u;
      if (ok[k]) {
        peers[k] = __match_any_sync(act, key[k]);
        if (lane == __ffs(peers[k]) - 1) at[k] = atomicAdd(&counts[key[k]], (uint32_t)__popc(peers[k]));
      }
    }
    if (kScatter) {
#pragma unroll
      for (int k = 0; k < N; ++k)
        if (ok[k]) {
          const uint32_t b = __shfl_sync(peers[k], at[k], __ffs(peers[k]) - 1);
          states_out[(offsets ? offsets[key[k]] : 0u) + b + __popc(peers[k] & ((1u << lane) - 1u))] = s[k];
        }
    }
  }
}

// Three-phase exclusive scan of n uint32 counts into offsets[0..n], total into
// offsets[n] and *total.
__global__ void __launch_bounds__(256) scan_sums_kernel(const uint32_t* __restrict__ in, uint32_t n,
                                                        uint32_t* __restrict__ sums) {
  __shared__ uint32_t red[8];
  const uint32_t b0 = blockIdx.x * kScanBlock;
  uint32_t v = 0;
  for (uint32_t i = b0 + threadIdx.x; i < min(b0 + kScanBlock, n); i += blockDim.x) v += in[i];
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < 8; ++w) t += red[w];
    sums[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(1024) scan_top_kernel(uint32_t* __restrict__ sums, uint32_t nblocks) {
  __shared__ uint32_t part[1024];
  const uint32_t per = (nblocks + 1023) / 1024;
  const uint32_t beg = threadIdx.x * per, end = min(beg + per, nblocks);
  uint32_t s = 0;
  for (uint32_t i = beg; i < end; ++i) s += sums[i];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {
    const uint32_t v = threadIdx.x >= (unsigned)off ? part[threadIdx.x - off] : 0u;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  uint32_t run = threadIdx.x ? part[threadIdx.x - 1] : 0u;
  for (uint32_t i = beg; i < end; ++i) {
    const uint32_t c = sums[i];
    sums[i] = run;
    run += c;
  }
}

__global__ void __launch_bounds__(256) scan_apply_kernel(const uint32_t* __restrict__ in, uint32_t n,
                                                         const uint32_t* __restrict__ sums,
                                                         uint32_t* __restrict__ out, uint32_t* __restrict__ total) {
  __shared__ uint32_t warp_tot[8];
  const uint32_t b0 = blockIdx.x * kScanBlock;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // each thread owns 4 consecutive elements
  const uint32_t i0 = b0 + threadIdx.x * 4;
  uint32_t v[4];
  uint32_t tsum = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = (i0 + k < n) ? in[i0 + k] : 0u;
    tsum += v[k];
  }
  uint32_t incl = tsum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[wid] = incl;
  __syncthreads();
  uint32_t wbase = 0;
  for (int w = 0; w < wid; ++w) wbase += warp_tot[w];
  uint32_t run = sums[blockIdx.x] + wbase + incl - tsum;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (i0 + k < n) out[i0 + k] = run;
    run += v[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) {
    out[n] = run;
    *total = run;
  }
}

// Packed records with an even row pitch (TMA needs 16-byte row strides).
__global__ void __launch_bounds__(256) pack_pitched_kernel(const uint8_t* __restrict__ img, BrickGeom g,
                                                           uint2* __restrict__ rec) {
  const uint64_t V = (uint64_t)g.Zc * g.Yc * g.Xp;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < V; i += stride) {
    const int x = (int)(i % g.Xp);
    const uint64_t zy = i / g.Xp;
    const int y = (int)(zy % g.Yc);
    const int z = (int)(zy / g.Yc);
    uint2 r = make_uint2(0u, 0u);
    if (z > 0 && y > 0 && x > 0 && z < g.Zc - 1 && y < g.Yc - 1 && x < g.Xc - 1) {
      const size_t p = ((size_t)z * g.Yc + y) * g.Xc + x;
      uint32_t mask = 0;
      mask |= (z + 1 >= g.Zc - 1) ? 1u : 0u;
      mask |= (z - 1 <= 0) ? 2u : 0u;
      mask |= (y + 1 >= g.Yc - 1) ? 4u : 0u;
      mask |= (y - 1 <= 0) ? 8u : 0u;
      mask |= (x + 1 >= g.Xc - 1) ? 16u : 0u;
      mask |= (x - 1 <= 0) ? 32u : 0u;
      r.x = (uint32_t)img[p + g.F] | ((uint32_t)img[p - g.F] << 8) | ((uint32_t)img[p + g.Xc] << 16) |
            ((uint32_t)img[p - g.Xc] << 24);
      r.y = (uint32_t)img[p + 1] | ((uint32_t)img[p - 1] << 8) | (mask << 16) | ((uint32_t)img[p] << 24);
    }
    rec[i] = r;
  }
}

__device__ __forceinline__ float byte_p23(uint32_t w, uint32_t k) {
  return __int_as_float((int)__byte_perm(w, 0x4B000000u, 0x7540u + k));
}

__device__ __forceinline__ uint32_t pick(const U4& r, uint32_t sub) {
  return sub == 0u ? r.x : (sub == 1u ? r.y : (sub == 2u ? r.z : r.w));
}

// Advance all sorted live walkers, chunk by chunk (persistent CTAs).
__global__ void __launch_bounds__(kAdvThreads, 4) brick_advance_kernel(
    const __grid_constant__ CUtensorMap rec_map, BrickGeom g, uint4* __restrict__ states,
    const uint32_t* __restrict__ offsets, uint32_t nbt, uint32_t n_live, uint32_t* __restrict__ chunk_ctr, const SeedRec* __restrict__ seeds, uint32_t k0, uint32_t k1,
    uint32_t* __restrict__ hits, uint32_t* __restrict__ err, uint32_t wait_lim) {
  extern __shared__ __align__(128) uint8_t smem[];
  uint2* s_rec = reinterpret_cast<uint2*>(smem);
  uint32_t* s_hits = reinterpret_cast<uint32_t*>(smem + kExtVox * sizeof(uint2));
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ uint32_t s_chunk, s_bucket, s_end, s_next;
  const int tid = threadIdx.x;
  const size_t V = (size_t)g.F * g.Zc;
  if (tid == 0) mbar_init(&s_bar, 1);
  __syncthreads();
  uint32_t phase = 0;
  for (;;) {
    if (tid == 0) s_chunk = atomicAdd(chunk_ctr, 1u);
    __syncthreads();
    const uint64_t c0 = (uint64_t)s_chunk * kChunk;
    if (c0 >= n_live) break;
    const uint64_t c1w = c0 + kChunk;
    const uint32_t c1 = c1w < (uint64_t)n_live ? (uint32_t)c1w : n_live;
    uint32_t p = (uint32_t)c0;
    while (p < c1) {
      if (tid == 0) {
        // bucket holding sorted position p: last b with offsets[b] <= p
        uint32_t lo = 0, hi = nbt;  // offsets has nbt + 1 entries, offsets[nbt] = n_live
        while (hi - lo > 1) {
          const uint32_t mid = (lo + hi) >> 1;
          if (offsets[mid] <= p) lo = mid; else hi = mid;
        }
        s_bucket = lo;
        s_end = min(offsets[lo + 1], c1);
        s_next = p;
      }
      __syncthreads();
      const uint32_t bucket = s_bucket;
      const uint32_t seg_end = s_end;
      const uint32_t slot = bucket / g.nb;
      const uint32_t brick = bucket - slot * g.nb;
      const int bx = (int)(brick % (uint32_t)g.nbx);
      const int by = (int)((brick / (uint32_t)g.nbx) % (uint32_t)g.nby);
      const int bz = (int)(brick / ((uint32_t)g.nbx * (uint32_t)g.nby));
      const int ex0 = bx * kCore - kLo, ey0 = by * kCore - kLo, ez0 = bz * kCore - kLo;
      if (tid == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&s_bar, kExtVox * sizeof(uint2));
        tma_load_box(s_rec, &rec_map, ex0, ey0, ez0, &s_bar);
      }
      for (int i = tid; i < kExtVox; i += kAdvThreads) s_hits[i] = 0u;
      const bool done = mbar_wait_bounded(&s_bar, phase, wait_lim);
      if (__syncthreads_or(!done)) {
        // gave up: wait (bounded) for the box copy still in flight before the
        // CTA's shared memory goes away, then report
        if (tid == 0) {
          mbar_wait_bounded(&s_bar, phase, kDrainWaitLimit);
          atomicOr(err, 1u);
        }
        return;
      }
      phase ^= 1u;
      uint32_t* __restrict__ hl = hits + (size_t)slot * V;
      for (;;) {
        const uint32_t w = atomicAdd(&s_next, 1u);
        if (w >= seg_end) break;
        uint4 st = states[w];
        const SeedRec sd = seeds[st.y];
        const float c = sd.c;
        const float b23 = __fadd_rn(sd.b, 8388608.0f);
        const uint32_t axis = seed_axis(sd.meta), label = seed_label(sd.meta);
        int z, y, x;
        coords(g, st.x, z, y, x);
        uint32_t l = ((uint32_t)(z - ez0) << 8) | ((uint32_t)(y - ey0) << 4) | (uint32_t)(x - ex0);
        uint32_t t = st.z;
        const uint32_t te = st.w & 0xFFFFFFu;
        uint32_t blk = t >> 2;
        U4 rr = philox4x32_10(U4{blk, sd.pos, axis, label}, k0, k1);
        bool left = false;
        uint32_t gpos = st.x;
        while (t < te) {
          if ((t >> 2) != blk) {
            blk = t >> 2;
            rr = philox4x32_10(U4{blk, sd.pos, axis, label}, k0, k1);
          }
          const uint32_t bits = pick(rr, t & 3u);
          const uint2 r = s_rec[l];
          float d, w0, w1, w2, w3, w4, w5;
          d = __fsub_rn(b23, byte_p23(r.x, 0)); w0 = edge_weight(__fmul_rn(d, d), c);
          d = __fsub_rn(b23, byte_p23(r.x, 1)); w1 = edge_weight(__fmul_rn(d, d), c);
          d = __fsub_rn(b23, byte_p23(r.x, 2)); w2 = edge_weight(__fmul_rn(d, d), c);
          d = __fsub_rn(b23, byte_p23(r.x, 3)); w3 = edge_weight(__fmul_rn(d, d), c);
          d = __fsub_rn(b23, byte_p23(r.y, 0)); w4 = edge_weight(__fmul_rn(d, d), c);
          d = __fsub_rn(b23, byte_p23(r.y, 1)); w5 = edge_weight(__fmul_rn(d, d), c);
          const float c1 = __fadd_rn(w0, w1);
          const float c2 = __fadd_rn(c1, w2);
          const float c3 = __fadd_rn(c2, w3);
          const float c4 = __fadd_rn(c3, w4);
          const float c5 = __fadd_rn(c4, w5);
          const float rnd = __fmul_rn(c5, u01_from_bits(bits));
          int dir = (int)(w0 <= rnd) + (int)(c1 <= rnd) + (int)(c2 <= rnd) + (int)(c3 <= rnd) + (int)(c4 <= rnd);
          if (rnd == 0.0f) dir = 0;
          ++t;
          if ((r.y >> (16 + dir)) & 1u) continue;  // refused: the step counts, nothing is hit
          const uint32_t shift = (uint32_t)(2 - (dir >> 1)) * 4u;  // z: 8, y: 4, x: 0
          const uint32_t coord = (l >> shift) & 15u;
          const bool plus = (dir & 1) == 0;
          if (plus ? coord == 15u : coord == 0u) {
            // the move leaves the box: global hit, walker continues next round
            const int zz = ez0 + (int)(l >> 8) + (dir == 0) - (dir == 1);
            const int yy = ey0 + (int)((l >> 4) & 15u) + (dir == 2) - (dir == 3);
            const int xx = ex0 + (int)(l & 15u) + (dir == 4) - (dir == 5);
            gpos = (uint32_t)zz * g.F + (uint32_t)yy * (uint32_t)g.Xc + (uint32_t)xx;
            atomicAdd(&hl[gpos], 1u);
            left = true;
            break;
          }
          l = plus ? l + (1u << shift) : l - (1u << shift);
          atomicAdd(&s_hits[l], 1u);
        }
        st.z = t;
        if (left) st.x = gpos;
        states[w] = st;
      }
      __syncthreads();
      // flush the box counters
      for (int i = tid; i < kExtVox; i += kAdvThreads) {
        const uint32_t v = s_hits[i];
        if (v) {
          const int zz = ez0 + (i >> 8), yy = ey0 + ((i >> 4) & 15), xx = ex0 + (i & 15);
          atomicAdd(&hl[(size_t)zz * g.F + (size_t)yy * g.Xc + xx], v);
        }
      }
      __syncthreads();
      p = seg_end;
    }
  }
}

// ---------------------------------------------------------------------------
// Sorted sweep: every live walker advances exactly min(K, steps left) steps over
// the packed records in global memory (uniform work per thread). Walkers are
// counting-sorted by (label slot, 6^3 brick) between sweeps, so the threads
// resident at any moment work on a compact slab of the volume and its records
// and hit counters stay in L2.
// ---------------------------------------------------------------------------
// Walkers still live after their K steps are counted into next_counts by
// (label slot, brick): the counting pass of the next sort, fused (warp
// aggregation of equal keys; walkers of a warp come from few buckets).
template <bool kFloat>
__global__ void __launch_bounds__(256) sweep_kernel(const void* __restrict__ packed, BrickGeom g,
                                                    uint4* __restrict__ states, uint32_t K,
                                                    const SeedRec* __restrict__ seeds, uint32_t k0, uint32_t k1,
                                                    uint32_t* __restrict__ hits, uint32_t* __restrict__ next_counts,
                                                    const uint32_t* __restrict__ ctrs) {
  const uint32_t n_live = ctrs[kCtrLive];
  __shared__ int32_t s_delta[6];
  if (threadIdx.x < 6) {
    const int32_t F = (int32_t)g.F, X = g.Xc;
    s_delta[threadIdx.x] = threadIdx.x == 0 ? F : threadIdx.x == 1 ? -F : threadIdx.x == 2 ? X
                           : threadIdx.x == 3 ? -X : threadIdx.x == 4 ? 1 : -1;
  }
  __syncthreads();
  const size_t V = (size_t)g.F * g.Zc;
  const uint32_t stride = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  const uint64_t nz = f2_negzero();
  // next sweep's bucket counts, warp-aggregated (whole warps call this)
  auto count = [&](bool alive, const uint4& st) {
    const uint32_t act = __ballot_sync(0xffffffffu, alive);
    if (alive) {
      const uint32_t key = bucket_of(g, st);
      const uint32_t peers = __match_any_sync(act, key);
      if (lane == __ffs(peers) - 1) atomicAdd(&next_counts[key], (uint32_t)__popc(peers));
    }
  };
  // warp-uniform trip count, so the counting below runs with full warps
  const uint32_t i_end = (n_live + 31u) & ~31u;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < i_end; i += stride) {
    bool alive = false;
    uint4 st = make_uint4(0u, 0u, 0u, 0u);
    if (i < n_live) {
      st = states[i];
      const SeedRec sd = seeds[st.y];
      const uint32_t te = st.w & 0xFFFFFFu;
      const uint32_t t_end = min(st.z + K, te);
      uint32_t* __restrict__ hl = hits + (size_t)(st.w >> 24) * V;
      st.x = walk_steps<kFloat>(packed, st.x, st.z, t_end, sd.c, sd.b, sd.pos, seed_axis(sd.meta),
                                seed_label(sd.meta), k0, k1, hl, s_delta, nz);
      st.z = t_end;
      states[i] = st;
      alive = t_end != te;
    }
    count(alive, st);
  }
}

// The same sweep with N consecutive walkers per thread (walk_steps_multi);
// kMinBlocks CTAs of kThreads per SM.
template <bool kFloat, int N, int kThreads, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
    sweep_multi_kernel(const void* __restrict__ packed, BrickGeom g, uint4* __restrict__ states, uint32_t K,
                       const SeedRec* __restrict__ seeds, uint32_t k0, uint32_t k1, uint32_t* __restrict__ hits,
                       uint32_t* __restrict__ next_counts, const uint32_t* __restrict__ ctrs) {
  const uint32_t n_live = ctrs[kCtrLive];
  __shared__ int32_t s_delta[6];
  if (threadIdx.x < 6) {
    const int32_t F = (int32_t)g.F, X = g.Xc;
    s_delta[threadIdx.x] = threadIdx.x == 0 ? F : threadIdx.x == 1 ? -F : threadIdx.x == 2 ? X
                           : threadIdx.x == 3 ? -X : threadIdx.x == 4 ? 1 : -1;
  }
  __syncthreads();
  const size_t V = (size_t)g.F * g.Zc;
  const uint32_t stride = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  const uint64_t nz = f2_negzero();
  // consecutive walkers (same bucket order: neighbours in the volume); the
  // trip count is warp-uniform so the counting runs with full warps
  const uint32_t n_groups = (n_live + (uint32_t)N - 1u) / (uint32_t)N;
  const uint32_t i_end = (n_groups + 31u) & ~31u;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < i_end; i += stride) {
    uint4 st[N];
    bool alive[N];
    uint32_t te[N];
    PairWalker W[N];
#pragma unroll
    for (int w = 0; w < N; ++w) {
      st[w] = make_uint4(0u, 0u, 0u, 0u);
      alive[w] = false;
      te[w] = 0u;
      W[w] = pair_walker(0u, 0u, 0u, 0.0f, 0.0f, 0u, 0u, 0u, hits);  // no steps without a walker
    }
    if (i < n_groups) {
#pragma unroll
      for (int w = 0; w < N; ++w) {
        const uint32_t idx = (uint32_t)N * i + (uint32_t)w;
        if (idx < n_live) {
          st[w] = states[idx];
          const SeedRec sd = seeds[st[w].y];
          te[w] = st[w].w & 0xFFFFFFu;
          W[w] = pair_walker(st[w].x, st[w].z, min(st[w].z + K, te[w]), sd.c, sd.b, sd.pos,
                             seed_axis(sd.meta), seed_label(sd.meta), hits + (size_t)(st[w].w >> 24) * V);
        }
      }
      walk_steps_multi<kFloat, N>(packed, W, k0, k1, s_delta, nz);
#pragma unroll
      for (int w = 0; w < N; ++w) {
        const uint32_t idx = (uint32_t)N * i + (uint32_t)w;
        if (idx < n_live) {
          st[w].x = W[w].pos;
          st[w].z = W[w].t_end;
          states[idx] = st[w];
          alive[w] = W[w].t_end != te[w];
        }
      }
    }
#pragma unroll
    for (int w = 0; w < N; ++w) {
      const uint32_t act = __ballot_sync(0xffffffffu, alive[w]);
      if (alive[w]) {
        const uint32_t key = bucket_of(g, st[w]);
        const uint32_t peers = __match_any_sync(act, key);
        if (lane == __ffs(peers) - 1) atomicAdd(&next_counts[key], (uint32_t)__popc(peers));
      }
    }
  }
}

// ---- host side ----
struct ScratchLayout {
  size_t rec, states0, states1, counts, offsets, sums, ctrs, total;
};

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

ScratchLayout layout(const BrickGeom& g, uint64_t max_walks, int nol) {
  ScratchLayout L{};
  const uint64_t nbt = (uint64_t)g.nb * nol;
  const uint64_t nblocks = (nbt + kScanBlock - 1) / kScanBlock;
  size_t off = 0;
  L.rec = off;
  off = align_up(off + (size_t)g.Zc * g.Yc * g.Xp * sizeof(uint2), 256);
  L.states0 = off;
  off = align_up(off + max_walks * sizeof(uint4), 256);
  L.states1 = off;
  off = align_up(off + max_walks * sizeof(uint4), 256);
  L.counts = off;
  off = align_up(off + (nbt + 1) * sizeof(uint32_t), 256);
  L.offsets = off;
  off = align_up(off + (nbt + 1) * sizeof(uint32_t), 256);
  L.sums = off;
  off = align_up(off + (nblocks + 1) * sizeof(uint32_t), 256);
  L.ctrs = off;  // [0] n_live, [1] chunk counter, [2] error flag
  off = align_up(off + 4 * sizeof(uint32_t), 256);
  L.total = off;
  return L;
}

BrickGeom make_geom(int Zc, int Yc, int Xc, int edge = kCore) {
  BrickGeom g{};
  g.Zc = Zc;
  g.Yc = Yc;
  g.Xc = Xc;
  g.edge = edge;
  g.nbz = (Zc + edge - 1) / edge;
  g.nby = (Yc + edge - 1) / edge;
  g.nbx = (Xc + edge - 1) / edge;
  g.nb = (uint32_t)g.nbz * g.nby * g.nbx;
  g.label_step = g.nb;
  g.brick_step = 1u;
  g.F = (uint32_t)Yc * Xc;
  g.Xp = (uint32_t)((Xc + 1) & ~1);
  g.by_F = FastDiv(g.F);
  g.by_X = FastDiv((uint32_t)Xc);
  g.by_edge = FastDiv((uint32_t)edge);
  return g;
}

int advance_blocks_per_sm() {
  static std::atomic<int> cached_dev[64];  // per device (the shared-memory opt-in is per device); 0 = not yet set
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  int cached = cached_dev[dev].load(std::memory_order_acquire);
  if (!cached) {
    const int smem = kExtVox * (int)(sizeof(uint2) + sizeof(uint32_t));
    cudaFuncSetAttribute(brick_advance_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, brick_advance_kernel, kAdvThreads, smem) != cudaSuccess ||
        n < 1)
      n = 1;
    cached = n;
    cached_dev[dev].store(n, std::memory_order_release);
  }
  return cached;
}

}  // namespace
}  // namespace si

using namespace si;

extern "C" int si_walk_bricks_scratch(int Zc, int Yc, int Xc, uint64_t max_walks, int nol,
                                      unsigned long long* bytes) {
  clear_error();
  if (!bytes || Zc < 3 || Yc < 3 || Xc < 3 || nol < 1 || nol > 256)
    return set_error(SI_ERR_ARG, "si_walk_bricks_scratch: bad arguments");
  *bytes = layout(make_geom(Zc, Yc, Xc), max_walks, nol).total;
  return SI_OK;
}

extern "C" int si_walk_bricks(const void* work, int Zc, int Yc, int Xc, const si_seed_t* seeds,
                              const uint32_t* n_seeds, uint32_t max_seeds, int nbrw, int sorw, uint64_t key,
                              uint32_t* hits, int nol, void* scratch, unsigned long long scratch_bytes,
                              int* rounds_out, void* stream) {
  clear_error();
  if (!work || !seeds || !n_seeds || !hits || !scratch) return set_error(SI_ERR_ARG, "si_walk_bricks: null pointer");
  if (Zc < 3 || Yc < 3 || Xc < 3 || nol < 1 || nol > 256) return set_error(SI_ERR_ARG, "si_walk_bricks: bad dims");
  if ((uint64_t)Zc * Yc * Xc > 0xFFFFFFFFull) return set_error(SI_ERR_LIMIT, "si_walk_bricks: volume above 2^32");
  if (nbrw < 0 || sorw < 0 || (uint64_t)nbrw * (uint64_t)sorw >= (1ull << 24))
    return set_error(SI_ERR_LIMIT, "si_walk_bricks: nbrw*sorw must be below 2^24");
  cudaStream_t st = as_stream(stream);
  if (rounds_out) *rounds_out = 0;
  uint32_t ns = 0;
  if (cudaMemcpyAsync(&ns, n_seeds, sizeof(uint32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return set_error(SI_ERR_CUDA, "si_walk_bricks: reading the seed count failed");
  ns = ns < max_seeds ? ns : max_seeds;
  const uint64_t walks = (uint64_t)ns * (uint64_t)nbrw;
  if (walks == 0 || sorw == 0) return SI_OK;
  if (walks >= 0xFFFFFFFFull) return set_error(SI_ERR_LIMIT, "si_walk_bricks: more than 2^32 walks");
  const BrickGeom g = make_geom(Zc, Yc, Xc);
  const ScratchLayout L = layout(g, walks, nol);
  if (scratch_bytes < L.total)
    return set_error(SI_ERR_ARG, "si_walk_bricks: scratch of %llu bytes, %llu needed", scratch_bytes,
                     (unsigned long long)L.total);
  uint8_t* base = static_cast<uint8_t*>(scratch);
  uint2* rec = reinterpret_cast<uint2*>(base + L.rec);
  uint4* states[2] = {reinterpret_cast<uint4*>(base + L.states0), reinterpret_cast<uint4*>(base + L.states1)};
  uint32_t* counts = reinterpret_cast<uint32_t*>(base + L.counts);
  uint32_t* offsets = reinterpret_cast<uint32_t*>(base + L.offsets);
  uint32_t* sums = reinterpret_cast<uint32_t*>(base + L.sums);
  uint32_t* ctrs = reinterpret_cast<uint32_t*>(base + L.ctrs);
  const uint32_t nbt = g.nb * (uint32_t)nol;
  const uint32_t nblocks = (nbt + kScanBlock - 1) / kScanBlock;
  const SeedRec* sd = reinterpret_cast<const SeedRec*>(seeds);

  EncodeTiledFn enc = encode_fn();
  if (!enc) return set_error(SI_ERR_CUDA, "si_walk_bricks: cuTensorMapEncodeTiled unavailable");
  CUtensorMap map;
  std::memset(&map, 0, sizeof(map));
  const cuuint64_t dims[3] = {(cuuint64_t)g.Xc, (cuuint64_t)g.Yc, (cuuint64_t)g.Zc};
  const cuuint64_t strides[2] = {(cuuint64_t)g.Xp * sizeof(uint2), (cuuint64_t)g.Xp * g.Yc * sizeof(uint2)};
  const cuuint32_t box[3] = {kExt, kExt, kExt};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult cr = enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, rec, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) return set_error(SI_ERR_CUDA, "si_walk_bricks: tensor map encoding failed (%d)", (int)cr);

  const int sms = sm_count();
  const int gb = sms * 8;
  pack_pitched_kernel<<<sms * 16, 256, 0, st>>>(static_cast<const uint8_t*>(work), g, rec);
  if (cudaMemsetAsync(ctrs, 0, 4 * sizeof(uint32_t), st) != cudaSuccess)
    return set_error(SI_ERR_CUDA, "si_walk_bricks: memset failed");
  const int smem = kExtVox * (int)(sizeof(uint2) + sizeof(uint32_t));
  const int adv_grid = sms * advance_blocks_per_sm();
  const uint32_t k0 = (uint32_t)key, k1 = (uint32_t)(key >> 32);
  int cur = 0;
  int rounds = 0;
  uint64_t n_prev = walks;  // entries of the previous round (round 0: virtual (seed, walk) pairs)
  for (;; ++rounds) {
    const bool first = rounds == 0;
    if (cudaMemsetAsync(counts, 0, (size_t)(nbt + 1) * sizeof(uint32_t), st) != cudaSuccess)
      return set_error(SI_ERR_CUDA, "si_walk_bricks: memset failed");
    if (first)
      bucket_kernel<true, false><<<gb, 256, 0, st>>>(nullptr, n_prev, sd, ns, sorw, g, counts, nullptr, nullptr);
    else
      bucket_kernel<false, false><<<gb, 256, 0, st>>>(states[cur], n_prev, sd, ns, sorw, g, counts, nullptr,
                                                      nullptr);
    scan_sums_kernel<<<nblocks, 256, 0, st>>>(counts, nbt, sums);
    scan_top_kernel<<<1, 1024, 0, st>>>(sums, nblocks);
    scan_apply_kernel<<<nblocks, 256, 0, st>>>(counts, nbt, sums, offsets, ctrs);
    uint32_t live_now = 0;
    if (cudaMemcpyAsync(&live_now, ctrs, sizeof(uint32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return set_error(SI_ERR_CUDA, "si_walk_bricks: round %d: %s", rounds, cudaGetErrorString(cudaGetLastError()));
    if (live_now == 0) break;
    if (cudaMemsetAsync(counts, 0, (size_t)(nbt + 1) * sizeof(uint32_t), st) != cudaSuccess)
      return set_error(SI_ERR_CUDA, "si_walk_bricks: memset failed");
    const int nxt = first ? 0 : 1 - cur;
    if (first)
      bucket_kernel<true, true><<<gb, 256, 0, st>>>(nullptr, n_prev, sd, ns, sorw, g, counts, offsets,
                                                    states[nxt]);
    else
      bucket_kernel<false, true><<<gb, 256, 0, st>>>(states[cur], n_prev, sd, ns, sorw, g, counts, offsets,
                                                     states[nxt]);
    cur = nxt;
    if (cudaMemsetAsync(ctrs + 1, 0, sizeof(uint32_t), st) != cudaSuccess)
      return set_error(SI_ERR_CUDA, "si_walk_bricks: memset failed");
    brick_advance_kernel<<<adv_grid, kAdvThreads, smem, st>>>(map, g, states[cur], offsets, nbt, live_now, ctrs + 1,
                                                               sd, k0, k1, hits, ctrs + 2, wait_limit());
    const int rc = check_launch("si_walk_bricks: advance");
    if (rc) return rc;
    n_prev = live_now;
    if (rounds > 100000) return set_error(SI_ERR_LIMIT, "si_walk_bricks: no convergence");
  }
  uint32_t err = 0;
  if (cudaMemcpyAsync(&err, ctrs + 2, sizeof(uint32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return set_error(SI_ERR_CUDA, "si_walk_bricks: final sync failed");
  if (err) return set_error(SI_ERR_CUDA, "si_walk_bricks: a TMA wait timed out");
  if (rounds_out) *rounds_out = rounds;
  return check_launch("si_walk_bricks");
}

namespace si {
namespace {
constexpr uint64_t kBatchWalks = 1ull << 25;  // default walks per seed range of si_walk_sorted
// Sort bricks. Their labels follow one another in the sorted order, so walkers that
// run at the same time share records and add to different maps (label by label the
// same bricks came round again for every label, and all walkers of a moment added
// to one map: 128^3 41.5 ms, now 41.0). Default edge, 4 to 8: about kBrickWalks walks
// per brick, but no fewer than kBucketWalks live ones per bucket. Smaller bricks keep
// a dense set of walkers closer together; of a sparse one a CTA then spans too many,
// and counting and scanning buckets that hold a walker or two costs more than it
// orders. Walks in ms at edges 4 / 6 / 8: 176x224x208, 9 labels, 2.4 walks a voxel 309 /
// 317 / 333, 400x512x512, 9 labels, 2.1 a voxel in seven ranges 4268 / 4164 / 4140, 128^3,
// 3 labels, 1.0 41.4 / 41.0 / 41.3, 419x492x462, 3 labels, 0.5 713 / 698 / 692.
constexpr int kSortEdge = 6;  // of batches
constexpr int kMinSortEdge = 4, kMaxSortEdge = 8;
constexpr double kBrickWalks = 160.0, kBucketWalks = 20.0;
// Default sweep length: 128 steps for walks of kLongWalk steps and more, 32 for shorter
// ones. Longer sweeps share the sort's cost among more steps, but let the walkers
// spread further between sorts. Walks of 4000 steps, 48 / 64 / 96 / 128 / 256
// steps a sweep: 128^3 44.4 / 43.2 / 42.0 / 41.4 / 42.0 ms, 419x492x462 873 /
// 855 / 838 / 834 / 843 ms. Speed does not put the line at kLongWalk: 128 steps are the
// fastest at every length. 32 / 64 / 128 / 256 steps a sweep, 240x250x230 uint8: walks of
// 252 steps 18.3 / 17.2 / 16.6 / 17.0 ms, 500 36.1 / 33.5 / 32.4 / 33.0, 1000 71.9 / 66.9 /
// 64.3 / 65.4, 2000 143 / 133 / 128 / 130 (uint16 alike; 40x36x33, 500 steps 0.58 / 0.48 /
// 0.45 / 0.42). Below it the default stays the 32 steps that callers who count sweeps or
// limit their number (si_walk_sorted_set_round_limit) know; sweep_steps = 128 gains 8 to
// 11 % there, and the batch tuner tries it.
constexpr int kLongWalk = 1000;
int default_sweep_steps(int sorw) { return sorw >= kLongWalk ? 128 : 32; }
std::atomic<unsigned long long> g_range_walks{0};  // 0 = kBatchWalks (si_walk_sorted_set_range)
std::atomic<int> g_sweep_pairs{1};  // sweep kernel mode (si_walk_sorted_set_pairs)
std::atomic<int> g_device_loop{1};  // 1: device-side sweep loop (si_walk_sorted_set_loop)
std::atomic<unsigned long long> g_round_limit{0};  // 0 = kRoundLimit (si_walk_sorted_set_round_limit)
constexpr uint64_t kRoundLimit = 1ull << 24;

uint32_t round_limit() {
  const unsigned long long v = g_round_limit.load(std::memory_order_relaxed);
  return (uint32_t)std::min<uint64_t>(v ? v : kRoundLimit, 0xFFFFFFFFull);
}

// ---------------------------------------------------------------------------
// Scan of the sorted walkers' bucket sizes: offsets receives every bucket's
// first place (the scatter's cursors), counts is zeroed as it is read (the
// sweep adds the next round's sizes), the counters move on to the next round.
// With the memsets and the counter update inside, a round is three launches
// for up to kScanOne buckets and five above; it was eight.
// ---------------------------------------------------------------------------
struct ScanArgs {
  uint32_t* counts;
  uint32_t n;
  uint32_t* offsets;
  uint32_t* ctrs;
  uint32_t limit;                    // most sweeps (round_limit)
  int cond;                          // 1: set the loop condition
  cudaGraphConditionalHandle handle;
};

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

// Exclusive scan over the CTA's threads (whole warps, at most 1024 threads);
// total receives the sum. Two barriers.
__device__ __forceinline__ uint32_t cta_exclusive(uint32_t v, uint32_t* s_warp, uint32_t& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t incl = warp_inclusive(v);
  if (lane == 31) s_warp[wid] = incl;
  __syncthreads();
  const uint32_t w = warp_inclusive(lane < nw ? s_warp[lane] : 0u);
  total = __shfl_sync(0xffffffffu, w, 31);
  const uint32_t before = __shfl_sync(0xffffffffu, w, wid ? wid - 1 : 0);
  __syncthreads();
  return (wid ? before : 0u) + incl - v;
}

__device__ __forceinline__ uint4 load_counts(const ScanArgs& a, uint32_t i0) {
  if (i0 + 4u <= a.n) return *reinterpret_cast<const uint4*>(a.counts + i0);
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (i0 < a.n) v.x = a.counts[i0];
  if (i0 + 1u < a.n) v.y = a.counts[i0 + 1u];
  if (i0 + 2u < a.n) v.z = a.counts[i0 + 2u];
  return v;
}

// Places four buckets from i0 (a multiple of 4; offsets and counts are padded
// to one), whose predecessors hold `run` walkers.
__device__ __forceinline__ void place_buckets(const ScanArgs& a, uint32_t i0, const uint4& v, uint32_t run) {
  if (i0 >= a.n) return;
  *reinterpret_cast<uint4*>(a.offsets + i0) = make_uint4(run, run + v.x, run + v.x + v.y, run + v.x + v.y + v.z);
  *reinterpret_cast<uint4*>(a.counts + i0) = make_uint4(0u, 0u, 0u, 0u);
}

// The sweep that just ran had ctrs[kCtrLive] states; the next has `live`.
__device__ __forceinline__ void next_round(const ScanArgs& a, uint32_t live) {
  const uint32_t prev = a.ctrs[kCtrLive];
  const uint32_t sweeps = a.ctrs[kCtrSweeps] + (prev ? 1u : 0u);
  a.ctrs[kCtrIn] = prev;
  a.ctrs[kCtrSweeps] = sweeps;
  a.ctrs[kCtrLive] = live;
  if (a.cond) {
    const bool over = live != 0u && sweeps >= a.limit;
    if (over) a.ctrs[kCtrOver] = 1u;
    cudaGraphSetConditional(a.handle, (live != 0u && !over) ? 1u : 0u);
  }
}

// The whole scan in one CTA. Above kScanOne buckets its serial tiles of 4096
// (about 1 us each) cost more than the two launches it saves.
constexpr uint32_t kScanOne = 16384;
__global__ void __launch_bounds__(1024) walk_scan_one_kernel(ScanArgs a) {
  __shared__ uint32_t s_warp[32];
  uint32_t carry = 0;
  uint4 v = load_counts(a, threadIdx.x * 4u);
  for (uint32_t b0 = 0; b0 < a.n; b0 += 4096u) {
    const uint32_t i0 = b0 + threadIdx.x * 4u;
    const uint4 next = load_counts(a, i0 + 4096u);  // the next tile's counts on their way
    uint32_t tile;
    place_buckets(a, i0, v, carry + cta_exclusive(v.x + v.y + v.z + v.w, s_warp, tile));
    carry += tile;
    v = next;
  }
  if (threadIdx.x == 0) next_round(a, carry);
}

// Three launches for many buckets: sums of 1024 buckets a CTA, their scan, the
// places.
__global__ void __launch_bounds__(256) walk_scan_sums_kernel(ScanArgs a, uint32_t* __restrict__ sums) {
  __shared__ uint32_t s_warp[32];
  const uint4 v = load_counts(a, blockIdx.x * kScanBlock + threadIdx.x * 4u);
  uint32_t total;
  cta_exclusive(v.x + v.y + v.z + v.w, s_warp, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) walk_scan_top_kernel(ScanArgs a, uint32_t* __restrict__ sums,
                                                             uint32_t nblocks) {
  __shared__ uint32_t s_warp[32];
  uint32_t carry = 0;
  for (uint32_t b0 = 0; b0 < nblocks; b0 += 1024u) {
    const uint32_t b = b0 + threadIdx.x;
    const uint32_t v = b < nblocks ? sums[b] : 0u;
    uint32_t tile;
    const uint32_t run = carry + cta_exclusive(v, s_warp, tile);
    if (b < nblocks) sums[b] = run;
    carry += tile;
  }
  if (threadIdx.x == 0) next_round(a, carry);
}

__global__ void __launch_bounds__(256) walk_scan_place_kernel(ScanArgs a, const uint32_t* __restrict__ sums) {
  __shared__ uint32_t s_warp[32];
  const uint32_t i0 = blockIdx.x * kScanBlock + threadIdx.x * 4u;
  const uint4 v = load_counts(a, i0);
  uint32_t total;
  place_buckets(a, i0, v, sums[blockIdx.x] + cta_exclusive(v.x + v.y + v.z + v.w, s_warp, total));
}

// A stream of this device for capturing loop bodies (never executes work).
cudaStream_t capture_stream() {
  static std::mutex mu;
  static cudaStream_t streams[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  std::lock_guard<std::mutex> lock(mu);
  if (!streams[dev] && cudaStreamCreateWithFlags(&streams[dev], cudaStreamNonBlocking) != cudaSuccess)
    streams[dev] = nullptr;
  return streams[dev];
}

// An executable graph holding one WHILE node whose body is what enqueue(s, h)
// puts on stream s (recorded by stream capture). The condition starts at 1
// on every launch; a kernel of the body sets it with cudaGraphSetConditional.
template <class F>
int build_while_graph(F&& enqueue, cudaGraphExec_t* exec) {
  cudaStream_t cs = capture_stream();
  if (!cs) return set_error(SI_ERR_CUDA, "si_walk_sorted: no capture stream");
  cudaGraph_t graph = nullptr;
  if (cudaGraphCreate(&graph, 0) != cudaSuccess) return set_error(SI_ERR_CUDA, "si_walk_sorted: graph create");
  int rc = SI_OK;
  cudaGraphConditionalHandle h;
  cudaGraphNodeParams cp = {};
  cudaGraphNode_t node;
  if (cudaGraphConditionalHandleCreate(&h, graph, 1, cudaGraphCondAssignDefault) != cudaSuccess) {
    rc = set_error(SI_ERR_CUDA, "si_walk_sorted: conditional handle: %s", cudaGetErrorString(cudaGetLastError()));
  } else {
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    if (cudaGraphAddNode(&node, graph, nullptr, nullptr, 0, &cp) != cudaSuccess)
      rc = set_error(SI_ERR_CUDA, "si_walk_sorted: while node: %s", cudaGetErrorString(cudaGetLastError()));
  }
  if (rc == SI_OK) {
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    if (cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed) != cudaSuccess) {
      rc = set_error(SI_ERR_CUDA, "si_walk_sorted: capture: %s", cudaGetErrorString(cudaGetLastError()));
    } else {
      enqueue(cs, h);
      cudaGraph_t captured = nullptr;
      if (cudaStreamEndCapture(cs, &captured) != cudaSuccess)
        rc = set_error(SI_ERR_CUDA, "si_walk_sorted: capture end: %s", cudaGetErrorString(cudaGetLastError()));
      else if (cudaGraphInstantiate(exec, graph, 0) != cudaSuccess)
        rc = set_error(SI_ERR_CUDA, "si_walk_sorted: instantiate: %s", cudaGetErrorString(cudaGetLastError()));
    }
  }
  cudaGraphDestroy(graph);
  return rc;
}

uint64_t range_walks() {
  const unsigned long long v = g_range_walks.load(std::memory_order_relaxed);
  return v ? (uint64_t)v : kBatchWalks;
}

// Scratch of a sorted walk (byte offsets).
struct SortLayout {
  size_t vols, states0, states1, counts, offsets, sums, ctrs, total;
};

SortLayout sort_layout(uint64_t nbt, uint64_t max_walks, size_t vol_bytes) {
  SortLayout L{};
  const uint64_t nblocks = (nbt + kScanBlock - 1) / kScanBlock;
  size_t off = 0;
  L.vols = off;
  off = align_up(off + vol_bytes, 256);
  L.states0 = off;
  off = align_up(off + max_walks * sizeof(uint4), 256);
  L.states1 = off;
  off = align_up(off + max_walks * sizeof(uint4), 256);
  L.counts = off;
  off = align_up(off + nbt * sizeof(uint32_t), 256);
  L.offsets = off;
  off = align_up(off + nbt * sizeof(uint32_t), 256);
  L.sums = off;
  off = align_up(off + nblocks * sizeof(uint32_t), 256);
  L.ctrs = off;
  off = align_up(off + kCtrWords * sizeof(uint32_t), 256);
  L.total = off;
  return L;
}

struct WalkBuffers {
  uint4* states[2];
  uint32_t *counts, *offsets, *sums, *ctrs;
  uint32_t nbt, nblocks;
};

WalkBuffers walk_buffers(void* scratch, const SortLayout& L, uint32_t nbt) {
  uint8_t* b = static_cast<uint8_t*>(scratch);
  WalkBuffers w{};
  w.states[0] = reinterpret_cast<uint4*>(b + L.states0);
  w.states[1] = reinterpret_cast<uint4*>(b + L.states1);
  w.counts = reinterpret_cast<uint32_t*>(b + L.counts);
  w.offsets = reinterpret_cast<uint32_t*>(b + L.offsets);
  w.sums = reinterpret_cast<uint32_t*>(b + L.sums);
  w.ctrs = reinterpret_cast<uint32_t*>(b + L.ctrs);
  w.nbt = nbt;
  w.nblocks = (nbt + kScanBlock - 1) / kScanBlock;
  return w;
}

void walk_scan(cudaStream_t s, const WalkBuffers& w, const ScanArgs& a) {
  if (w.nbt <= kScanOne) {
    walk_scan_one_kernel<<<1, 1024, 0, s>>>(a);
    return;
  }
  walk_scan_sums_kernel<<<w.nblocks, 256, 0, s>>>(a, w.sums);
  walk_scan_top_kernel<<<1, 1024, 0, s>>>(a, w.sums, w.nblocks);
  walk_scan_place_kernel<<<w.nblocks, 256, 0, s>>>(a, w.sums);
}

// One range of walks from their start to their end. first(s): counts the
// virtual walks; start(s, out): scatters them; scatter(s, in, out): the live
// states of the last sweep into the sorted order; sweep(s, states): K steps of
// every state, the live ones counted. Device loop: the executable graph it
// launches is added to execs (destroy it after the stream has run it).
template <class First, class Start, class Scatter, class Sweep>
int run_range(cudaStream_t st, const WalkBuffers& w, ScanArgs a, bool device_loop, const char* what,
              std::vector<cudaGraphExec_t>& execs, First first, Start start, Scatter scatter, Sweep sweep) {
  a.cond = 0;
  first(st);
  walk_scan(st, w, a);
  start(st, w.states[0]);
  if (device_loop) {
    sweep(st, w.states[0]);
    walk_scan(st, w, a);
    int rc = check_launch(what);
    if (rc) return rc;
    // two rounds per loop iteration: states[0] -> states[1] -> states[0]
    cudaGraphExec_t exec = nullptr;
    rc = build_while_graph(
        [&](cudaStream_t cs, cudaGraphConditionalHandle h) {
          for (int half = 0; half < 2; ++half) {
            scatter(cs, w.states[half], w.states[1 - half]);
            sweep(cs, w.states[1 - half]);
            ScanArgs b = a;
            b.cond = half;
            b.handle = h;
            walk_scan(cs, w, b);
          }
        },
        &exec);
    if (rc) return rc;
    execs.push_back(exec);
    return cudaGraphLaunch(exec, st) == cudaSuccess ? SI_OK : set_error(SI_ERR_CUDA, "%s: graph launch failed", what);
  }
  for (int cur = 0;; cur = 1 - cur) {
    uint32_t c[kCtrWords];
    if (cudaMemcpyAsync(c, w.ctrs, sizeof(c), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return set_error(SI_ERR_CUDA, "%s: %s", what, cudaGetErrorString(cudaGetLastError()));
    if (c[kCtrLive] == 0) return SI_OK;
    if (c[kCtrSweeps] >= a.limit) return set_error(SI_ERR_LIMIT, "%s: no convergence within %u sweeps", what, a.limit);
    if (c[kCtrIn] != 0) scatter(st, w.states[1 - cur], w.states[cur]);
    sweep(st, w.states[cur]);
    walk_scan(st, w, a);
    const int rc = check_launch(what);
    if (rc) return rc;
  }
}

// Waits for the walk and reads its counters.
int finish_walk(cudaStream_t st, const WalkBuffers& w, std::vector<cudaGraphExec_t>& execs, uint32_t limit, int rc,
                const char* what, int* rounds_out) {
  uint32_t c[kCtrWords] = {};
  if (cudaMemcpyAsync(c, w.ctrs, sizeof(c), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    rc = rc ? rc : set_error(SI_ERR_CUDA, "%s: %s", what, cudaGetErrorString(cudaGetLastError()));
  for (cudaGraphExec_t e : execs) cudaGraphExecDestroy(e);
  if (rc) return rc;
  if (c[kCtrOver]) return set_error(SI_ERR_LIMIT, "%s: no convergence within %u sweeps", what, limit);
  if (rounds_out) *rounds_out = (int)c[kCtrSweeps];
  return check_launch(what);
}
}  // namespace
}  // namespace si

namespace si {
namespace {
BrickGeom sort_geom(int Zc, int Yc, int Xc, int nol, int edge) {
  BrickGeom g = make_geom(Zc, Yc, Xc, edge);
  g.label_step = 1u;
  g.brick_step = (uint32_t)nol;
  return g;
}

uint64_t sort_bytes(int Zc, int Yc, int Xc, uint64_t walks, int nol, int edge) {
  return sort_layout((uint64_t)make_geom(Zc, Yc, Xc, edge).nb * (uint64_t)nol, walks, 0).total;
}

// The default sort edge for this many walks; kSortEdge where the preferred one has too
// many buckets or does not fit in `bytes`. More walks prefer no larger edge, so what
// si_walk_sorted_scratch asks for is enough for any fewer.
int default_sort_edge(int Zc, int Yc, int Xc, uint64_t walks, int nol, unsigned long long bytes) {
  const double V = (double)Zc * Yc * Xc, n = (double)std::max<uint64_t>(walks, 1);
  const double live = std::min(n, (double)range_walks());
  const double want = std::cbrt(std::max(kBrickWalks * V / n, kBucketWalks * nol * V / live));
  const int edge = want >= kMaxSortEdge ? kMaxSortEdge : std::max(kMinSortEdge, (int)std::lround(want));
  const bool counts = (uint64_t)make_geom(Zc, Yc, Xc, edge).nb * (uint64_t)nol < 0xFFFFFFFFull;
  return counts && sort_bytes(Zc, Yc, Xc, walks, nol, edge) <= bytes ? edge : kSortEdge;
}
}  // namespace
}  // namespace si

extern "C" int si_walk_sorted_scratch(int Zc, int Yc, int Xc, uint64_t max_walks, int nol, int sort_edge,
                                      unsigned long long* bytes) {
  clear_error();
  if (!bytes || Zc < 3 || Yc < 3 || Xc < 3 || nol < 1 || nol > 256 || sort_edge < 0 || sort_edge > 1024)
    return set_error(SI_ERR_ARG, "si_walk_sorted_scratch: bad arguments");
  *bytes = sort_bytes(Zc, Yc, Xc, max_walks, nol, sort_edge > 0 ? sort_edge : kSortEdge);
  if (sort_edge <= 0) {
    const int edge = default_sort_edge(Zc, Yc, Xc, max_walks, nol, ~0ull);
    *bytes = std::max<unsigned long long>(*bytes, sort_bytes(Zc, Yc, Xc, max_walks, nol, edge));
  }
  return SI_OK;
}

extern "C" int si_walk_sorted_set_range(unsigned long long walks_per_range) {
  clear_error();
  g_range_walks.store(walks_per_range, std::memory_order_relaxed);
  return SI_OK;
}

extern "C" int si_walk_sorted_set_pairs(int pairs) {
  clear_error();
  if (pairs < 0 || pairs > 3) return set_error(SI_ERR_ARG, "si_walk_sorted_set_pairs: 0 to 3");
  g_sweep_pairs.store(pairs, std::memory_order_relaxed);
  return SI_OK;
}

extern "C" int si_walk_sorted_set_loop(int device_loop) {
  clear_error();
  if (device_loop < 0 || device_loop > 1) return set_error(SI_ERR_ARG, "si_walk_sorted_set_loop: 0 or 1");
  g_device_loop.store(device_loop, std::memory_order_relaxed);
  return SI_OK;
}

extern "C" int si_walk_sorted_set_round_limit(unsigned long long sweeps) {
  clear_error();
  g_round_limit.store(sweeps, std::memory_order_relaxed);
  return SI_OK;
}

extern "C" int si_walk_sorted(const void* packed, int work_is_float, int Zc, int Yc, int Xc,
                              const si_seed_t* seeds, const uint32_t* n_seeds, uint32_t max_seeds, int nbrw,
                              int sorw, uint64_t key, uint32_t* hits, int nol, int sweep_steps, int sort_edge,
                              void* scratch, unsigned long long scratch_bytes, int* rounds_out, void* stream) {
  clear_error();
  if (!packed || !seeds || !n_seeds || !hits || !scratch) return set_error(SI_ERR_ARG, "si_walk_sorted: null pointer");
  if (Zc < 3 || Yc < 3 || Xc < 3 || nol < 1 || nol > 256) return set_error(SI_ERR_ARG, "si_walk_sorted: bad dims");
  if ((uint64_t)Zc * Yc * Xc > 0xFFFFFFFFull) return set_error(SI_ERR_LIMIT, "si_walk_sorted: volume above 2^32");
  if (nbrw < 0 || sorw < 0 || (uint64_t)nbrw * (uint64_t)sorw >= (1ull << 24))
    return set_error(SI_ERR_LIMIT, "si_walk_sorted: nbrw*sorw must be below 2^24");
  const bool default_steps = sweep_steps <= 0;
  if (default_steps) sweep_steps = default_sweep_steps(sorw);
  if (sort_edge > 1024) return set_error(SI_ERR_ARG, "si_walk_sorted: sort_edge above 1024");
  cudaStream_t st = as_stream(stream);
  if (rounds_out) *rounds_out = 0;
  uint32_t ns = 0;
  if (cudaMemcpyAsync(&ns, n_seeds, sizeof(uint32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return set_error(SI_ERR_CUDA, "si_walk_sorted: reading the seed count failed");
  ns = ns < max_seeds ? ns : max_seeds;
  const uint64_t walks = (uint64_t)ns * (uint64_t)nbrw;
  if (walks == 0 || sorw == 0) return SI_OK;
  if (walks >= 0xFFFFFFFFull) return set_error(SI_ERR_LIMIT, "si_walk_sorted: more than 2^32 walks");
  if (sort_edge <= 0)  // less than kSortEdge takes is refused below, whatever the default
    sort_edge = scratch_bytes < sort_bytes(Zc, Yc, Xc, walks, nol, kSortEdge)
                    ? kSortEdge
                    : default_sort_edge(Zc, Yc, Xc, walks, nol, scratch_bytes);
  const BrickGeom g = sort_geom(Zc, Yc, Xc, nol, sort_edge);
  if ((uint64_t)g.nb * (uint64_t)nol >= 0xFFFFFFFFull) return set_error(SI_ERR_LIMIT, "si_walk_sorted: too many buckets");
  const uint32_t nbt = g.nb * (uint32_t)nol;
  const SortLayout L = sort_layout(nbt, walks, 0);
  if (scratch_bytes < L.total)
    return set_error(SI_ERR_ARG, "si_walk_sorted: scratch of %llu bytes, %llu needed", scratch_bytes,
                     (unsigned long long)L.total);
  const WalkBuffers w = walk_buffers(scratch, L, nbt);
  const SeedRec* sd_all = reinterpret_cast<const SeedRec*>(seeds);
  const int sms = sm_count();
  const int gb = sms * 8;
  const uint32_t k0 = (uint32_t)key, k1 = (uint32_t)(key >> 32);
  // Seeds are walked in consecutive ranges of about range_walks() walks, each
  // to completion. Seeds come in slice order, so a range is a compact slab and
  // a sweep's records and hit counters stay closer to L2 than when every seed
  // of the volume is live at once (measured: +6 % on a 400x512x512 volume,
  // +19 % on 1024^3). Hits are integer sums of independent walks: the result
  // does not depend on the ranges.
  const uint64_t per_range = range_walks();
  const uint64_t nbatch = std::max<uint64_t>(1, (walks + per_range / 2) / per_range);
  // walkers per thread: mode 0 -> 1, 1 -> 2, 2 -> 3, 3 -> 4
  const int mode = g_sweep_pairs.load(std::memory_order_relaxed);
  // walks of which the SMs hold one per thread. A sweep of so few is bound by its
  // launches and tail as well: twice the steps, 3.39 and 3.21 ms on 40x36x33.
  const uint64_t resident = (uint64_t)sms * 768;
  if (default_steps && sorw >= kLongWalk && walks <= resident) sweep_steps *= 2;
  const uint32_t limit = round_limit();
  const bool device_loop = g_device_loop.load(std::memory_order_relaxed) != 0;
  const ScanArgs a{w.counts, nbt, w.offsets, w.ctrs, limit, 0, {}};
  const uint32_t K = (uint32_t)sweep_steps;
  if (cudaMemsetAsync(w.ctrs, 0, kCtrWords * sizeof(uint32_t), st) != cudaSuccess ||
      cudaMemsetAsync(w.counts, 0, (size_t)nbt * sizeof(uint32_t), st) != cudaSuccess)
    return set_error(SI_ERR_CUDA, "si_walk_sorted: memset failed");
  std::vector<cudaGraphExec_t> execs;
  int rc = SI_OK;
  for (uint64_t bidx = 0; bidx < nbatch && rc == SI_OK; ++bidx) {
    const uint32_t sa = (uint32_t)((uint64_t)ns * bidx / nbatch), se = (uint32_t)((uint64_t)ns * (bidx + 1) / nbatch);
    if (se == sa) continue;
    const SeedRec* sd = sd_all + sa;
    const uint32_t ns_b = se - sa;
    const uint64_t n0 = (uint64_t)ns_b * (uint64_t)nbrw;
    // One group of walkers per thread: CTAs start in the sorted order, so that
    // those running at any moment share a compact part of the volume. (A grid of
    // 8 CTAs per SM that strides over the walkers: 419x492x462 915 ms, this one
    // 857 ms; 176x224x208 with labels on all axes 370 and 332 ms.) Walks that
    // do not fill the SMs once go out in small CTAs, spread more evenly; where a
    // thread for each is resident at once, each gets one, as two in a thread wait
    // for the slower of their loads: 40x36x33, 95 thousand walks, pairs in CTAs of
    // 256 4.5 ms, of 64 4.2 ms (3.78 with the later sweeps), single 3.39 ms. One a
    // thread as well where walks or sweeps are no multiple of four steps: walkers off
    // the blocks of four random words do not advance together, so two of a thread
    // follow one another (128^3, 999 steps: uint8 24.2 and 20.7 ms, uint16 28.5 and 21.4).
    const bool unaligned = (((uint32_t)sorw | K) & 3u) != 0u;
    const bool single = mode == 1 && (n0 <= resident || unaligned);
    const bool few = mode == 1 && !single && n0 <= 2 * resident;
    const uint64_t per = single ? 1u : (uint64_t)mode + 1;
    const int tpb = few ? 64 : mode == 3 || single ? 128 : mode == 1 && work_is_float ? kFloatThreads : 256;
    const uint32_t blocks = (uint32_t)(((n0 + per - 1) / per + tpb - 1) / tpb);
    const uint32_t sort_blocks = (uint32_t)std::min<uint64_t>(gb, (n0 + 255) / 256);
    auto sweep = [&](cudaStream_t s, uint4* states) {
#define SI_SWEEP(KERNEL) KERNEL<<<blocks, tpb, 0, s>>>(packed, g, states, K, sd, k0, k1, hits, w.counts, w.ctrs)
#define SI_SWEEPS(F)                                   \
  do {                                                 \
    if (mode == 3)                                     \
      SI_SWEEP((sweep_multi_kernel<F, 4, 128, 3>));    \
    else if (mode == 2)                                \
      SI_SWEEP((sweep_multi_kernel<F, 3, 256, 2>));    \
    else if (single)                                   \
      SI_SWEEP((sweep_multi_kernel<F, 1, 128, 6>));    \
    else if (few)                                      \
      SI_SWEEP((sweep_multi_kernel<F, 2, 64, F ? 9 : 12>)); \
    else if (mode == 1)                                \
      SI_SWEEP((sweep_multi_kernel<F, 2, F ? kFloatThreads : 256, 3>)); \
    else                                               \
      SI_SWEEP(sweep_kernel<F>);                       \
  } while (0)
      if (work_is_float)
        SI_SWEEPS(true);
      else
        SI_SWEEPS(false);
#undef SI_SWEEPS
#undef SI_SWEEP
    };
    rc = run_range(
        st, w, a, device_loop, "si_walk_sorted", execs,
        [&](cudaStream_t s) {
          bucket_kernel<true, false><<<sort_blocks, 256, 0, s>>>(nullptr, n0, sd, ns_b, sorw, g, w.counts, nullptr,
                                                                 nullptr);
        },
        [&](cudaStream_t s, uint4* out) {
          bucket_kernel<true, true><<<sort_blocks, 256, 0, s>>>(nullptr, n0, sd, ns_b, sorw, g, w.offsets, nullptr, out);
        },
        [&](cudaStream_t s, uint4* in, uint4* out) {
          bucket_kernel<false, true><<<sort_blocks, 256, 0, s>>>(in, 0, sd, ns_b, sorw, g, w.offsets, nullptr, out,
                                                                 w.ctrs + kCtrIn);
        },
        sweep);
  }
  return finish_walk(st, w, execs, limit, rc, "si_walk_sorted", rounds_out);
}

// ===========================================================================
// Batched sorted sweeps: many volumes (uneven sizes, any label counts, uint8
// or float32 records) walked together. A walker state carries its volume in
// the top 8 bits of the step counter (t < 2^24), buckets are
// (volume, label slot, brick) ranges of one global bucket space, and every
// sweep launch advances the walkers of all volumes. Hit maps, randomness and
// results per volume are exactly those of si_walk_sorted on that volume alone.
// ===========================================================================
namespace si {
namespace {

struct VolDesc {
  const void* packed;
  uint32_t* hits;
  const SeedRec* seeds;
  uint32_t F;       // Yc * Xc
  int Zc, Yc, Xc;
  int nby, nbx;     // bricks per row / column
  uint32_t nb;      // bricks per label
  uint32_t nol;
  uint32_t bucket0; // first bucket of this volume
  uint64_t walk0;   // first global walk index of this volume (round 0)
  uint32_t ns;      // seeds
  int is_float;
  FastDiv by_F, by_X;
};

__device__ __forceinline__ uint32_t bvol(const uint4& s) { return s.z >> 24; }
__device__ __forceinline__ uint32_t bstep(const uint4& s) { return s.z & 0xFFFFFFu; }
__device__ __forceinline__ bool blive(const uint4& s) { return bstep(s) != (s.w & 0xFFFFFFu); }

__device__ __forceinline__ uint32_t bbucket(const VolDesc& v, const FastDiv& by_edge, const uint4& s) {
  const uint32_t z = v.by_F(s.x);
  const uint32_t r = s.x - z * v.F;
  const uint32_t y = v.by_X(r);
  const uint32_t x = r - y * (uint32_t)v.Xc;
  const uint32_t brick = (by_edge(z) * (uint32_t)v.nby + by_edge(y)) * (uint32_t)v.nbx + by_edge(x);
  return v.bucket0 + (s.w >> 24) + brick * v.nol;
}

template <bool kFirst>
__device__ __forceinline__ bool bfetch(uint64_t i, uint64_t n, const uint4* __restrict__ states,
                                       const VolDesc* __restrict__ vols, int n_vols, int sorw, uint4& s) {
  if (i >= n) return false;
  if (kFirst) {
    // volume holding global walk i (volumes are few: linear search)
    int v = 0;
    while (v + 1 < n_vols && vols[v + 1].walk0 <= i) ++v;
    const VolDesc& d = vols[v];
    const uint64_t j = i - d.walk0;
    const uint32_t w = (uint32_t)(j / d.ns);
    const uint32_t sidx = (uint32_t)(j - (uint64_t)w * d.ns);
    const SeedRec sd = d.seeds[sidx];
    s = make_uint4(sd.pos, sidx, (w * (uint32_t)sorw) | ((uint32_t)v << 24),
                   ((w + 1u) * (uint32_t)sorw) | (seed_slot(sd.meta) << 24));
    return true;
  }
  s = states[i];
  return blive(s);
}

template <bool kFirst, bool kScatter>
__global__ void __launch_bounds__(256) bbucket_kernel(const uint4* __restrict__ states_in, uint64_t n,
                                                      const VolDesc* __restrict__ vols, int n_vols, int sorw,
                                                      FastDiv edge, uint32_t* __restrict__ counts,
                                                      uint4* __restrict__ states_out,
                                                      const uint32_t* __restrict__ n_dev = nullptr) {
  if (n_dev) n = *n_dev;  // the count lives on the device (device-side sweep loop)
  const int lane = threadIdx.x & 31;
  constexpr int N = 4;  // states a thread, as in bucket_kernel
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += N * stride) {
    uint4 s[N];
    bool ok[N];
    uint32_t key[N], peers[N], at[N];
#pragma unroll
    for (int k = 0; k < N; ++k)
      ok[k] = bfetch<kFirst>(base + k * stride + lane, n, states_in, vols, n_vols, sorw, s[k]);
#pragma unroll
    for (int k = 0; k < N; ++k) {
      key[k] = ok[k] ? bbucket(vols[bvol(s[k])], edge, s[k]) : 0u;
      const uint32_t act = __ballot_sync(0xffffffffu, ok[k]);
      at[k] = peers[k] = 0u;
      if (ok[k]) {
        peers[k] = __match_any_sync(act, key[k]);
        if (lane == __ffs(peers[k]) - 1) at[k] = atomicAdd(&counts[key[k]], (uint32_t)__popc(peers[k]));
      }
    }
    if (kScatter) {
#pragma unroll
      for (int k = 0; k < N; ++k)
        if (ok[k]) {
          const uint32_t b = __shfl_sync(peers[k], at[k], __ffs(peers[k]) - 1);
          states_out[b + __popc(peers[k] & ((1u << lane) - 1u))] = s[k];
        }
    }
  }
}

// One sweep of the batched walkers of the volumes of one record kind: every CTA
// takes N * kThreads consecutive walkers of ONE volume, so that its geometry and
// record pointer are the same for all threads, as in sweep_multi_kernel (a
// kernel whose threads looked up their own walker's volume, record kind
// included, took 106 registers, 2 CTAs per SM: 222 ms of sweeps for 6 uint16
// volumes of 64..144 voxels an edge, this one 148 ms). After the scatter a
// bucket's cursor stands at its end, so the cursor before a volume's first
// bucket is where the volume's walkers start.
template <bool kFloat, int N, int kThreads, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks) bsweep_kernel(const VolDesc* __restrict__ vols, int n_vols,
                                                                 uint32_t nbt, const uint32_t* __restrict__ cursors,
                                                                 uint4* __restrict__ states, uint32_t K, uint32_t k0,
                                                                 uint32_t k1, FastDiv edge,
                                                                 uint32_t* __restrict__ next_counts) {
  static_assert(kThreads >= 128, "two volumes a thread, at most 256");
  constexpr uint32_t kSpan = (uint32_t)kThreads * (uint32_t)N;
  __shared__ uint32_t s_warp[32];
  __shared__ int32_t s_delta[6];
  __shared__ VolDesc d;
  __shared__ uint32_t s_first, s_n;
  {
    uint32_t beg[2], end[2], ctas[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int v = 2 * (int)threadIdx.x + k;
      beg[k] = end[k] = 0u;
      if (v < n_vols && (vols[v].is_float != 0) == kFloat) {
        beg[k] = v ? cursors[vols[v].bucket0 - 1u] : 0u;
        end[k] = cursors[(v + 1 < n_vols ? vols[v + 1].bucket0 : nbt) - 1u];
      }
      ctas[k] = (end[k] - beg[k] + kSpan - 1u) / kSpan;
    }
    if (threadIdx.x == 0) s_n = 0u;
    uint32_t total;
    uint32_t before = cta_exclusive(ctas[0] + ctas[1], s_warp, total);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (blockIdx.x >= before && blockIdx.x - before < ctas[k]) {
        const uint32_t at = (blockIdx.x - before) * kSpan;
        s_first = beg[k] + at;
        s_n = min(kSpan, end[k] - beg[k] - at);
        d = vols[2 * threadIdx.x + (unsigned)k];
        const int32_t F = (int32_t)d.F;
        s_delta[0] = F; s_delta[1] = -F; s_delta[2] = d.Xc; s_delta[3] = -d.Xc; s_delta[4] = 1; s_delta[5] = -1;
      }
      before += ctas[k];
    }
    __syncthreads();
  }
  const uint32_t n = s_n;
  if (n == 0u) return;  // beyond the last walker
  const int lane = threadIdx.x & 31;
  const uint64_t nz = f2_negzero();
  const uint32_t first = s_first;
  uint4 st[N];
  bool alive[N];
  uint32_t te[N];
  PairWalker W[N];
#pragma unroll
  for (int w = 0; w < N; ++w) {
    const uint32_t j = threadIdx.x * (uint32_t)N + (uint32_t)w;
    st[w] = make_uint4(0u, 0u, 0u, 0u);
    alive[w] = false;
    te[w] = 0u;
    W[w] = pair_walker(0u, 0u, 0u, 0.0f, 0.0f, 0u, 0u, 0u, nullptr);  // no steps without a walker
    if (j < n) {
      st[w] = states[first + j];
      const SeedRec sd = d.seeds[st[w].y];
      const uint32_t t = bstep(st[w]);
      te[w] = st[w].w & 0xFFFFFFu;
      W[w] = pair_walker(st[w].x, t, min(t + K, te[w]), sd.c, sd.b, sd.pos, seed_axis(sd.meta), seed_label(sd.meta),
                         d.hits + (size_t)(st[w].w >> 24) * ((size_t)d.F * d.Zc));
    }
  }
  walk_steps_multi<kFloat, N>(d.packed, W, k0, k1, s_delta, nz);
#pragma unroll
  for (int w = 0; w < N; ++w) {
    const uint32_t j = threadIdx.x * (uint32_t)N + (uint32_t)w;
    if (j < n) {
      st[w].x = W[w].pos;
      st[w].z = W[w].t_end | (st[w].z & 0xFF000000u);
      states[first + j] = st[w];
      alive[w] = W[w].t_end != te[w];
    }
    const uint32_t act = __ballot_sync(0xffffffffu, alive[w]);
    if (alive[w]) {
      const uint32_t key = bbucket(d, edge, st[w]);
      const uint32_t peers = __match_any_sync(act, key);
      if (lane == __ffs(peers) - 1) atomicAdd(&next_counts[key], (uint32_t)__popc(peers));
    }
  }
}

}  // namespace
}  // namespace si

namespace {
// host helper: descriptors, bucket totals, scratch layout
struct BatchPlan {
  std::vector<si::VolDesc> vols;
  uint64_t walks = 0;
  uint32_t nbt = 0;
  bool any_u8 = false, any_float = false;
  si::SortLayout layout{};
};

int make_batch_plan(const si_volume_t* vols, int n_vols, int nbrw, int edge, const uint32_t* ns_host,
                    BatchPlan& P) {
  P.vols.resize(n_vols);
  uint64_t bucket = 0, walk = 0;
  for (int v = 0; v < n_vols; ++v) {
    const si_volume_t& in = vols[v];
    if (!in.packed || !in.hits || !in.seeds || !in.n_seeds || in.Zc < 3 || in.Yc < 3 || in.Xc < 3 || in.nol < 1 ||
        in.nol > 256)
      return si::set_error(SI_ERR_ARG, "si_walk_sorted_batch: bad volume %d", v);
    if ((uint64_t)in.Zc * in.Yc * in.Xc > 0xFFFFFFFFull)
      return si::set_error(SI_ERR_LIMIT, "si_walk_sorted_batch: volume %d above 2^32 voxels", v);
    si::VolDesc& d = P.vols[v];
    d.packed = in.packed;
    d.hits = in.hits;
    d.seeds = reinterpret_cast<const si::SeedRec*>(in.seeds);
    d.Zc = in.Zc;
    d.Yc = in.Yc;
    d.Xc = in.Xc;
    d.F = (uint32_t)in.Yc * (uint32_t)in.Xc;
    const int nbz = (in.Zc + edge - 1) / edge;
    d.nby = (in.Yc + edge - 1) / edge;
    d.nbx = (in.Xc + edge - 1) / edge;
    d.nb = (uint32_t)nbz * d.nby * d.nbx;
    d.nol = (uint32_t)in.nol;
    d.bucket0 = (uint32_t)bucket;
    d.walk0 = walk;
    d.ns = ns_host ? (ns_host[v] < in.max_seeds ? ns_host[v] : in.max_seeds) : in.max_seeds;
    d.is_float = in.work_is_float;
    (in.work_is_float ? P.any_float : P.any_u8) = true;
    d.by_F = si::FastDiv(d.F);
    d.by_X = si::FastDiv((uint32_t)in.Xc);
    bucket += (uint64_t)d.nb * in.nol;
    walk += (uint64_t)d.ns * (uint64_t)nbrw;
  }
  if (bucket >= 0xFFFFFFFFull) return si::set_error(SI_ERR_LIMIT, "si_walk_sorted_batch: too many buckets");
  if (walk >= 0xFFFFFFFFull) return si::set_error(SI_ERR_LIMIT, "si_walk_sorted_batch: more than 2^32 walks");
  P.walks = walk;
  P.nbt = (uint32_t)bucket;
  P.layout = si::sort_layout(P.nbt, P.walks, n_vols * sizeof(si::VolDesc));
  return SI_OK;
}
}  // namespace

extern "C" int si_walk_sorted_batch_scratch(const si_volume_t* vols, int n_vols, int nbrw, int sort_edge,
                                            unsigned long long* bytes) {
  clear_error();
  if (!vols || !bytes || n_vols < 1 || n_vols > 256 || nbrw < 0 || sort_edge < 0 || sort_edge > 1024)
    return set_error(SI_ERR_ARG, "si_walk_sorted_batch_scratch: bad arguments");
  BatchPlan P;
  const int rc = make_batch_plan(vols, n_vols, nbrw, sort_edge > 0 ? sort_edge : kSortEdge, nullptr, P);
  if (rc) return rc;
  *bytes = P.layout.total;
  return SI_OK;
}

extern "C" int si_walk_sorted_batch(const si_volume_t* vols, int n_vols, int nbrw, int sorw, uint64_t key,
                                    int sweep_steps, int sort_edge, void* scratch, unsigned long long scratch_bytes,
                                    int* rounds_out, void* stream) {
  clear_error();
  if (!vols || !scratch || n_vols < 1 || n_vols > 256) return set_error(SI_ERR_ARG, "si_walk_sorted_batch: bad args");
  if (nbrw < 0 || sorw < 0 || (uint64_t)nbrw * (uint64_t)sorw >= (1ull << 24))
    return set_error(SI_ERR_LIMIT, "si_walk_sorted_batch: nbrw*sorw must be below 2^24");
  if (sweep_steps <= 0) sweep_steps = default_sweep_steps(sorw);
  if (sort_edge <= 0) sort_edge = kSortEdge;
  if (sort_edge > 1024) return set_error(SI_ERR_ARG, "si_walk_sorted_batch: sort_edge above 1024");
  cudaStream_t st = as_stream(stream);
  if (rounds_out) *rounds_out = 0;
  std::vector<uint32_t> ns(n_vols, 0);
  for (int v = 0; v < n_vols; ++v) {
    if (!vols[v].n_seeds) return set_error(SI_ERR_ARG, "si_walk_sorted_batch: volume %d has no seed count", v);
    if (cudaMemcpyAsync(&ns[v], vols[v].n_seeds, sizeof(uint32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess)
      return set_error(SI_ERR_CUDA, "si_walk_sorted_batch: reading seed counts failed");
  }
  if (cudaStreamSynchronize(st) != cudaSuccess)
    return set_error(SI_ERR_CUDA, "si_walk_sorted_batch: reading seed counts failed");
  BatchPlan P;
  int rc = make_batch_plan(vols, n_vols, nbrw, sort_edge, ns.data(), P);
  if (rc) return rc;
  if (P.walks == 0 || sorw == 0) return SI_OK;
  BatchPlan Pmax;  // scratch is sized for max_seeds
  rc = make_batch_plan(vols, n_vols, nbrw, sort_edge, nullptr, Pmax);
  if (rc) return rc;
  if (scratch_bytes < Pmax.layout.total)
    return set_error(SI_ERR_ARG, "si_walk_sorted_batch: scratch of %llu bytes, %llu needed", scratch_bytes,
                     (unsigned long long)Pmax.layout.total);
  // layout of the max-seed plan; the actual walks fit in it
  const WalkBuffers w = walk_buffers(scratch, Pmax.layout, P.nbt);
  VolDesc* d_vols = reinterpret_cast<VolDesc*>(static_cast<uint8_t*>(scratch) + Pmax.layout.vols);
  if (cudaMemcpyAsync(d_vols, P.vols.data(), n_vols * sizeof(VolDesc), cudaMemcpyHostToDevice, st) != cudaSuccess)
    return set_error(SI_ERR_CUDA, "si_walk_sorted_batch: descriptor upload failed");
  const int sms = sm_count();
  const uint32_t k0 = (uint32_t)key, k1 = (uint32_t)(key >> 32), K = (uint32_t)sweep_steps;
  const FastDiv by_edge((uint32_t)sort_edge);
  // walker pairs unless mode 0
  const bool pairs = g_sweep_pairs.load(std::memory_order_relaxed) != 0;
  const uint32_t sort_blocks = (uint32_t)std::min<uint64_t>((uint64_t)sms * 8, (P.walks + 255) / 256);
  auto sweep = [&](cudaStream_t s, uint4* states) {
// every volume's last CTA may be partly filled
#define SI_BSWEEP(F, N, T, MIN)                                                                                  \
  bsweep_kernel<F, N, T, MIN><<<(uint32_t)((P.walks + N * T - 1) / (N * T)) + (uint32_t)n_vols, T, 0, s>>>(       \
      d_vols, n_vols, P.nbt, w.offsets, states, K, k0, k1, by_edge, w.counts)
    if (P.any_u8) {
      if (pairs)
        SI_BSWEEP(false, 2, 256, 3);
      else
        SI_BSWEEP(false, 1, 256, 5);
    }
    if (P.any_float) {
      if (pairs)
        SI_BSWEEP(true, 2, kFloatThreads, 3);
      else
        SI_BSWEEP(true, 1, 256, 5);
    }
#undef SI_BSWEEP
  };
  const uint32_t limit = round_limit();
  const ScanArgs a{w.counts, P.nbt, w.offsets, w.ctrs, limit, 0, {}};
  if (cudaMemsetAsync(w.ctrs, 0, kCtrWords * sizeof(uint32_t), st) != cudaSuccess ||
      cudaMemsetAsync(w.counts, 0, (size_t)P.nbt * sizeof(uint32_t), st) != cudaSuccess)
    return set_error(SI_ERR_CUDA, "si_walk_sorted_batch: memset failed");
  std::vector<cudaGraphExec_t> execs;
  rc = run_range(
      st, w, a, g_device_loop.load(std::memory_order_relaxed) != 0, "si_walk_sorted_batch", execs,
      [&](cudaStream_t s) {
        bbucket_kernel<true, false><<<sort_blocks, 256, 0, s>>>(nullptr, P.walks, d_vols, n_vols, sorw, by_edge,
                                                                w.counts, nullptr);
      },
      [&](cudaStream_t s, uint4* out) {
        bbucket_kernel<true, true><<<sort_blocks, 256, 0, s>>>(nullptr, P.walks, d_vols, n_vols, sorw, by_edge,
                                                               w.offsets, out);
      },
      [&](cudaStream_t s, uint4* in, uint4* out) {
        bbucket_kernel<false, true><<<sort_blocks, 256, 0, s>>>(in, 0, d_vols, n_vols, sorw, by_edge, w.offsets, out,
                                                                w.ctrs + kCtrIn);
      },
      sweep);
  return finish_walk(st, w, execs, limit, rc, "si_walk_sorted_batch", rounds_out);
}
