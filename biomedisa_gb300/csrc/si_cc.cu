// Outlier removal ("clean") and hole filling ("fill") of label volumes on
// the device, after biomedisa/features/remove_outlier.py:67-141. Both rest on
// 6-connected component labelling by union-find over x-runs (maximal runs of
// same-class voxels along x), each run named by its first voxel:
//   * a mask pass packs a row's classes into words of 32 voxels (fill: voxels
//     of label k; clean: first voxels of runs), one coalesced read of the
//     volume;
//   * a merge pass joins the runs of neighbouring rows (-y, -z): two runs
//     overlap in one interval, which is found, and merged, once, at its first
//     voxel. Roots are hung under the smaller root with atomicMin, so a parent
//     index never increases and every parent chain strictly decreases (find
//     and merge loops end after at most `index` iterations);
//   * a count pass points every run at its root, the smallest voxel index of
//     its component (= the component's first voxel in C order, which is the
//     order in which scipy.ndimage.label numbers components), and adds up run
//     lengths, one atomic per distinct root per warp.
// Passes after the first work on words and runs, not voxels: a 256^3 volume is
// 0.5 M words and, with 1 % speckle, 0.1 to 0.6 M runs a label. Labelling every
// voxel took 1.2 ms a label of fill and 0.8 ms for clean there (rows walked by
// one thread each, four passes over 4-byte parents and sizes); runs take
// 0.07 and 0.13 ms. Launches and the chains of the union-find bound them now.
// Scratch: int32 parent[V], uint32 size[V] (entries of run starts only), one
// word per 32 voxels of a row, a small info block.
#include <algorithm>
#include <climits>
#include <cstdint>

#include "si_common.cuh"
#include "si_internal.h"

namespace si {
namespace {

struct CcInfo {
  int zmin, zmax, ymin, ymax, xmin, xmax;
  unsigned count;            // voxels of the label
  unsigned pad;
  unsigned long long best;   // largest component of the complement: size << 32 | ~first voxel
};

// Words of 32 voxels: row r = z * Y + y has W of them.
struct Words {
  int Z, Y, X, W;
  uint32_t n;  // Z * Y * W, at most 2^31 - 1
  int lanes, lg;  // lanes (a power of two) of a warp that take a word together
  FastDiv by_W, by_Y;
};

// A lane's place among words that a warp takes `lanes` lanes each: 32, and so one
// word a warp, but for rows of 16 voxels and less (kShort), of which it takes
// several (clean of 3000x700x3 noise took 1.60 ms a word a warp, 0.55 ms so).
template <bool kShort>
struct WordLane {
  int sub, first;  // lane within the word, first lane of the word
  int lg;
  unsigned low;    // the word's bits
  __device__ __forceinline__ explicit WordLane(const Words& g) {
    const int lane = threadIdx.x & 31, lanes = kShort ? g.lanes : 32;
    lg = kShort ? g.lg : 5;
    sub = lane & (lanes - 1);
    first = lane - sub;
    low = 0xFFFFFFFFu >> (32 - lanes);
  }
  __device__ __forceinline__ unsigned ballot(bool p) const { return (__ballot_sync(0xffffffffu, p) >> first) & low; }
};

// f(i, i < g.n) for the words of a warp, whole warps together.
template <bool kShort, class F>
__device__ __forceinline__ void for_word_lanes(const Words& g, const WordLane<kShort>& l, F f) {
  const uint32_t stride = (gridDim.x * blockDim.x) >> l.lg;
  for (uint32_t i0 = ((blockIdx.x * blockDim.x + threadIdx.x) & ~31u) >> l.lg; i0 < g.n; i0 += stride) {
    const uint32_t i = i0 + ((uint32_t)l.first >> l.lg);
    f(i, !kShort || i < g.n);
  }
}

__device__ __forceinline__ int uf_find(const int* L, int p) {
  const volatile int* vl = L;
  int q = vl[p];
  while (q != p) {
    p = q;
    q = vl[p];
  }
  return p;
}

// find with path halving: each visited node is re-pointed at its grandparent
// (an ancestor, so atomicMin keeps parents monotone and links intact)
__device__ __forceinline__ int uf_find_halve(int* L, int p) {
  const volatile int* vl = L;
  while (true) {
    const int q = vl[p];
    if (q == p) return p;
    const int r = vl[q];
    if (r == q) return q;
    atomicMin(&L[p], r);
    p = r;
  }
}

__device__ __forceinline__ void uf_merge(int* L, int a, int b) {
  while (true) {
    a = uf_find_halve(L, a);
    b = uf_find_halve(L, b);
    if (a == b) return;
    if (a < b) {
      const int t = a;
      a = b;
      b = t;
    }
    const int old = atomicMin(&L[a], b);  // hang root a under b
    if (old == a) return;
    a = old;  // a stopped being a root meanwhile: join its new parent with b
  }
}

inline int grid_for(int64_t n) {
  const int64_t want = (n + 255) / 256, cap = (int64_t)sm_count() * 16;
  return (int)(want < cap ? (want > 0 ? want : 1) : cap);
}

// Adds len to size[root] for the lanes with a run, one atomic per distinct
// root of the warp (whole warps call this).
__device__ __forceinline__ void count_run(unsigned* size, int root, unsigned len, bool active) {
  const unsigned act = __ballot_sync(0xffffffffu, active);
  if (!active) return;
  const unsigned same = __match_any_sync(act, root);
  const unsigned sum = __reduce_add_sync(same, len);
  if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&size[root], sum);
}

// ---- clean: components of all labels at once (same-label connectivity) ----
// starts[word]: first voxels of the runs. x = 0 always is one.

// First voxel of the run that holds bit `bit` of word w of a row.
__device__ __forceinline__ int start_of(const unsigned* __restrict__ row, int w, int bit) {
  unsigned m = row[w] & (0xFFFFFFFFu >> (31 - bit));
  while (m == 0u) m = row[--w];
  return 32 * w + 31 - __clz(m);
}

template <bool kShort>
__global__ void __launch_bounds__(256) clean_starts_kernel(const uint8_t* __restrict__ lab, Words g, int skip,
                                                           unsigned* __restrict__ starts, int* __restrict__ L,
                                                           unsigned* __restrict__ size) {
  const WordLane<kShort> l(g);
  for_word_lanes(g, l, [&](uint32_t i, bool has) {
    const int64_t r = has ? g.by_W(i) : 0u;
    const int w = (int)(i - (uint32_t)r * (uint32_t)g.W), x = 32 * w + l.sub;
    const int64_t v = r * g.X + x;
    const bool in = has && x < g.X;
    const int c = in ? lab[v] : -1;
    int left = __shfl_up_sync(0xffffffffu, c, 1);
    if (l.sub == 0) left = w ? lab[v - 1] : -1;  // short rows have one word
    const bool first = in && c != left;
    const unsigned m = l.ballot(first);
    if (l.sub == 0 && has) starts[i] = m;
    if (first && c != skip) {
      L[v] = (int)v;
      size[v] = 0u;
    }
  });
}

// A lane merges where its run and the neighbouring row's begin to overlap.
template <bool kShort>
__global__ void __launch_bounds__(256) clean_merge_kernel(const uint8_t* __restrict__ lab, Words g, int skip,
                                                          const unsigned* __restrict__ starts, int* L) {
  const WordLane<kShort> l(g);
  for_word_lanes(g, l, [&](uint32_t i, bool has) {
    const int64_t r = has ? g.by_W(i) : 0u;
    const int w = (int)(i - (uint32_t)r * (uint32_t)g.W), x = 32 * w + l.sub;
    const int64_t v = r * g.X + x;
    const bool in = has && x < g.X;
    const int c = in ? lab[v] : skip;
    const unsigned m = has ? starts[i] : 0u;
    const int y = (int)((uint32_t)r - g.by_Y((uint32_t)r) * (uint32_t)g.Y);
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
      const bool row = dir == 0 ? y > 0 : r >= g.Y;
      if (kShort ? !__any_sync(0xffffffffu, row) : !row) continue;  // the same for the whole warp
      const int64_t dr = dir == 0 ? 1 : g.Y, dv = dr * g.X;
      const bool eq = in && row && c != skip && lab[v - dv] == c;
      const unsigned e = l.ballot(eq);
      bool left = l.sub ? (e >> (l.sub - 1)) & 1u : false;
      // the first voxel of a word, in a run that comes from the word before
      if (l.sub == 0 && eq && !(m & 1u)) left = lab[v - dv - 1] == c;
      if (eq && (((m >> l.sub) & 1u) || !left))
        uf_merge(L, (int)(r * g.X) + start_of(starts + r * g.W, w, l.sub),
                 (int)((r - dr) * g.X) + start_of(starts + (r - dr) * g.W, w, l.sub));
    }
  });
}

// One thread per word.
__global__ void __launch_bounds__(256) clean_count_kernel(const uint8_t* __restrict__ lab, Words g, int skip,
                                                          const unsigned* __restrict__ starts, int* L,
                                                          unsigned* __restrict__ size) {
  const uint32_t stride = gridDim.x * blockDim.x, n = (g.n + 31u) & ~31u;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int64_t r = i < g.n ? g.by_W(i) : 0u;
    const int w = (int)(i - (uint32_t)r * (uint32_t)g.W);
    unsigned m = i < g.n ? starts[i] : 0u;
    while (__any_sync(0xffffffffu, m != 0u)) {
      int root = -1;
      unsigned len = 0u;
      if (m) {
        const int x = 32 * w + __ffs(m) - 1;
        m &= m - 1u;
        const int v = (int)(r * g.X) + x;
        if (lab[v] != skip) {
          int end = g.X;  // the next run's first voxel
          if (m) {
            end = 32 * w + __ffs(m) - 1;
          } else {
            for (int k = w + 1; k < g.W; ++k) {
              const unsigned q = starts[r * g.W + k];
              if (q) {
                end = 32 * k + __ffs(q) - 1;
                break;
              }
            }
          }
          len = (unsigned)(end - x);
          root = uf_find(L, v);
          L[v] = root;
        }
      }
      count_run(size, root, len, root >= 0);
    }
  }
}

__global__ void __launch_bounds__(256) clean_max_kernel(const uint8_t* __restrict__ lab, Words g, int skip,
                                                        const unsigned* __restrict__ starts,
                                                        const int* __restrict__ L, const unsigned* __restrict__ size,
                                                        unsigned* __restrict__ big) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < g.n; i += stride) {
    const int64_t r = g.by_W(i);
    const int w = (int)(i - (uint32_t)r * (uint32_t)g.W);
    for (unsigned m = starts[i]; m; m &= m - 1u) {
      const int v = (int)(r * g.X) + 32 * w + __ffs(m) - 1;
      const int c = lab[v];
      if (c == skip || L[v] != v) continue;
      const unsigned s = size[v];
      if (s > *static_cast<volatile unsigned*>(&big[c])) atomicMax(&big[c], s);
    }
  }
}

// remove_outlier.py:85-97: keep components with size > threshold * largest
template <bool kShort>
__global__ void __launch_bounds__(256) clean_write_kernel(const uint8_t* __restrict__ lab, Words g, int skip,
                                                          const unsigned* __restrict__ starts,
                                                          const int* __restrict__ L,
                                                          const unsigned* __restrict__ size,
                                                          const unsigned* __restrict__ big, double threshold,
                                                          uint8_t* __restrict__ out) {
  const WordLane<kShort> l(g);
  for_word_lanes(g, l, [&](uint32_t i, bool has) {
    if (!has) return;
    const int64_t r = g.by_W(i);
    const int w = (int)(i - (uint32_t)r * (uint32_t)g.W), x = 32 * w + l.sub;
    if (x >= g.X) return;
    const int64_t v = r * g.X + x;
    const int c = lab[v];
    bool keep = true;
    if (c != skip) {
      const int root = L[(int)(r * g.X) + start_of(starts + r * g.W, w, l.sub)];
      keep = (double)size[root] > threshold * (double)big[c];
    }
    out[v] = keep ? (uint8_t)c : (uint8_t)0;
  });
}

// ---- fill: one label at a time inside its grown bounding box ----
__global__ void fill_info_init_kernel(CcInfo* info) {
  info->zmin = info->ymin = info->xmin = INT_MAX;
  info->zmax = info->ymax = info->xmax = -1;
  info->count = 0u;
  info->best = 0ull;
}

// mask[word]: voxels of label k; their bounding box and number. One warp per
// row, eight words at a time (the loads of a word are 32 bytes: latency bounds
// this pass; 256^3: 52 us with a division per word and four at a time).
__global__ void __launch_bounds__(256) fill_mask_kernel(const uint8_t* __restrict__ img, Words g, int k,
                                                        unsigned* __restrict__ mask, CcInfo* info) {
  __shared__ int s_lo[3], s_hi[3];
  __shared__ unsigned s_count;
  if (threadIdx.x < 3) {
    s_lo[threadIdx.x] = INT_MAX;
    s_hi[threadIdx.x] = -1;
  }
  if (threadIdx.x == 0) s_count = 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint32_t rows = (uint32_t)g.Z * (uint32_t)g.Y, stride = gridDim.x * (blockDim.x >> 5);
  int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {-1, -1, -1};
  unsigned cnt = 0u;
  constexpr int N = 8;
  for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += stride) {
    const uint8_t* row = img + (int64_t)r * g.X;
    unsigned* out = mask + (int64_t)r * g.W;
    unsigned any = 0u;
    for (int w0 = 0; w0 < g.W; w0 += N) {
      int c[N];
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const int x = 32 * (w0 + j) + lane;
        c[j] = x < g.X ? row[x] : -1;
      }
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const unsigned m = __ballot_sync(0xffffffffu, c[j] == k);
        const int w = w0 + j;
        if (lane == j && w < g.W) out[w] = m;
        if (m) {
          lo[2] = min(lo[2], 32 * w + __ffs(m) - 1);
          hi[2] = max(hi[2], 32 * w + 31 - __clz(m));
          cnt += __popc(m);
          any = 1u;
        }
      }
    }
    if (any) {
      const int z = (int)g.by_Y(r), y = (int)(r - (uint32_t)z * (uint32_t)g.Y);
      lo[0] = min(lo[0], z);
      hi[0] = max(hi[0], z);
      lo[1] = min(lo[1], y);
      hi[1] = max(hi[1], y);
    }
  }
  if (lane == 0 && cnt) {
    for (int a = 0; a < 3; ++a) {
      atomicMin(&s_lo[a], lo[a]);
      atomicMax(&s_hi[a], hi[a]);
    }
    atomicAdd(&s_count, cnt);
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_count) {
    atomicMin(&info->zmin, s_lo[0]);
    atomicMax(&info->zmax, s_hi[0]);
    atomicMin(&info->ymin, s_lo[1]);
    atomicMax(&info->ymax, s_hi[1]);
    atomicMin(&info->xmin, s_lo[2]);
    atomicMax(&info->xmax, s_hi[2]);
    atomicAdd(&info->count, s_count);
  }
}

// The bounding box grown by one voxel and clamped (remove_outlier.py:57-63),
// and the complement of the label inside it, as words. Words of the volume
// that the box does not touch are empty.
struct Complement {
  Words g;
  const unsigned* mask;
  int z0, z1, y0, y1, x0, x1;  // inclusive; empty when z1 < z0
  __device__ __forceinline__ Complement(const Words& g_, const unsigned* m, const CcInfo* info) : g(g_), mask(m) {
    z0 = max(info->zmin - 1, 0);
    y0 = max(info->ymin - 1, 0);
    x0 = max(info->xmin - 1, 0);
    z1 = min(info->zmax + 1, g.Z - 1);
    y1 = min(info->ymax + 1, g.Y - 1);
    x1 = min(info->xmax + 1, g.X - 1);
    if (info->count == 0u) {
      z0 = 0;
      z1 = -1;
    }
  }
  __device__ __forceinline__ bool has_row(int z, int y) const { return z >= z0 && z <= z1 && y >= y0 && y <= y1; }
  // bits of word w that lie in the box
  __device__ __forceinline__ unsigned span(int w) const {
    const int a = max(x0 - 32 * w, 0), b = min(x1 - 32 * w, 31);
    if (a > 31 || b < 0 || a > b) return 0u;
    return (0xFFFFFFFFu >> (31 - b)) & (0xFFFFFFFFu << a);
  }
  __device__ __forceinline__ unsigned word(int64_t r, int w) const { return ~mask[r * g.W + w] & span(w); }
  // word w and whether the voxel before it is in the complement too
  __device__ __forceinline__ unsigned word(int64_t r, int w, unsigned& carry) const {
    carry = w ? word(r, w - 1) >> 31 : 0u;
    return word(r, w);
  }
  // x of the first voxel of the run that holds bit `bit` of word w
  __device__ __forceinline__ int start_of(int64_t r, int w, int bit) const {
    unsigned gaps = ~word(r, w) & ~(0xFFFFFFFFu << bit);
    while (gaps == 0u) {
      if (w == 0) return 0;
      gaps = ~word(r, --w);
    }
    return 32 * w + 32 - __clz(gaps);
  }
  // x behind the last voxel of that run
  __device__ __forceinline__ int end_of(int64_t r, int w, int bit) const {
    unsigned gaps = ~word(r, w) & (0xFFFFFFFFu << bit);
    while (gaps == 0u) {
      if (++w >= g.W) return 32 * w;  // the span ends every run before X
      gaps = ~word(r, w);
    }
    return 32 * w + __ffs(gaps) - 1;
  }
};

// f(r, z, y, w, inside) for every word of the volume, whole warps together.
template <class F>
__device__ __forceinline__ void for_words(const Words& g, const Complement& c, F f) {
  const uint32_t stride = gridDim.x * blockDim.x, n = (g.n + 31u) & ~31u;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint32_t r = i < g.n ? g.by_W(i) : 0u;
    const int w = (int)(i - r * (uint32_t)g.W), z = (int)g.by_Y(r), y = (int)(r - (uint32_t)z * (uint32_t)g.Y);
    f((int64_t)r, z, y, w, i < g.n && c.has_row(z, y));
  }
}

__global__ void __launch_bounds__(256) fill_init_kernel(Words g, const unsigned* __restrict__ mask,
                                                        const CcInfo* __restrict__ info, int* __restrict__ L,
                                                        unsigned* __restrict__ size) {
  const Complement c(g, mask, info);
  for_words(g, c, [&](int64_t r, int, int, int w, bool inside) {
    if (!inside) return;
    unsigned carry;
    const unsigned m = c.word(r, w, carry);
    for (unsigned s = m & ~((m << 1) | carry); s; s &= s - 1u) {
      const int v = (int)(r * g.X) + 32 * w + __ffs(s) - 1;
      L[v] = v;
      size[v] = 0u;
    }
  });
}

__global__ void __launch_bounds__(256) fill_merge_kernel(Words g, const unsigned* __restrict__ mask,
                                                         const CcInfo* __restrict__ info, int* L) {
  const Complement c(g, mask, info);
  for_words(g, c, [&](int64_t r, int z, int y, int w, bool inside) {
    if (!inside) return;
    unsigned carry;
    const unsigned m = c.word(r, w, carry);
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
      if (dir == 0 ? y == c.y0 : z == c.z0) continue;  // connectivity does not leave the box
      const int64_t rn = r - (dir == 0 ? 1 : g.Y);
      unsigned carry_n;
      const unsigned o = m & c.word(rn, w, carry_n);
      for (unsigned s = o & ~((o << 1) | (carry & carry_n)); s; s &= s - 1u) {
        const int bit = __ffs(s) - 1;
        uf_merge(L, (int)(r * g.X) + c.start_of(r, w, bit), (int)(rn * g.X) + c.start_of(rn, w, bit));
      }
    }
  });
}

__global__ void __launch_bounds__(256) fill_count_kernel(Words g, const unsigned* __restrict__ mask,
                                                         const CcInfo* __restrict__ info, int* L,
                                                         unsigned* __restrict__ size) {
  const Complement c(g, mask, info);
  for_words(g, c, [&](int64_t r, int, int, int w, bool inside) {
    unsigned s = 0u;
    if (inside) {
      unsigned carry;
      const unsigned m = c.word(r, w, carry);
      s = m & ~((m << 1) | carry);
    }
    while (__any_sync(0xffffffffu, s != 0u)) {
      int root = -1;
      unsigned len = 0u;
      if (s) {
        const int bit = __ffs(s) - 1, x = 32 * w + bit, v = (int)(r * g.X) + x;
        s &= s - 1u;
        len = (unsigned)(c.end_of(r, w, bit) - x);
        root = uf_find(L, v);
        L[v] = root;
      }
      count_run(size, root, len, root >= 0);
    }
  });
}

// Largest component (the smallest first voxel among the largest).
__global__ void __launch_bounds__(256) fill_max_kernel(Words g, const unsigned* __restrict__ mask, CcInfo* info,
                                                       const int* __restrict__ L,
                                                       const unsigned* __restrict__ size) {
  const Complement c(g, mask, info);
  unsigned long long best = 0ull;
  for_words(g, c, [&](int64_t r, int, int, int w, bool inside) {
    if (!inside) return;
    unsigned carry;
    const unsigned m = c.word(r, w, carry);
    for (unsigned s = m & ~((m << 1) | carry); s; s &= s - 1u) {
      const int v = (int)(r * g.X) + 32 * w + __ffs(s) - 1;
      if (L[v] != v) continue;
      const unsigned long long key = ((unsigned long long)size[v] << 32) | (unsigned)~v;
      best = key > best ? key : best;
    }
  });
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
    best = other > best ? other : best;
  }
  if ((threadIdx.x & 31) == 0 && best > *static_cast<volatile unsigned long long*>(&info->best))
    atomicMax(&info->best, best);
}

// remove_outlier.py:124-141. The largest entry of [label size, component
// sizes in first-voxel order] (first maximum) stays as it is, components
// larger than threshold * label size stay, the rest of the box becomes k; if
// the label itself is the largest entry its own voxels become 0.
__global__ void __launch_bounds__(256) fill_write_kernel(uint8_t* img, Words g, int k,
                                                         const unsigned* __restrict__ mask,
                                                         const CcInfo* __restrict__ info, const int* __restrict__ L,
                                                         const unsigned* __restrict__ size, double threshold) {
  const Complement c(g, mask, info);
  const int lane = threadIdx.x & 31;
  const unsigned count = info->count;
  const unsigned long long top = info->best;
  const bool label_biggest = count >= (unsigned)(top >> 32);
  const int best = (int)~(unsigned)top;
  const double limit = threshold * (double)count;
  for_words(g, c, [&](int64_t r, int, int, int w, bool inside) {
    unsigned fill = 0u, zero = 0u;
    if (inside) {
      const unsigned m = c.word(r, w);
      if (label_biggest) zero = mask[r * g.W + w];
      for (unsigned s = m & ~(m << 1); s; s &= s - 1u) {  // the word's pieces of runs
        const int bit = __ffs(s) - 1;
        const int root = L[(int)(r * g.X) + c.start_of(r, w, bit)];
        const bool keep = (!label_biggest && root == best) || (double)size[root] > limit;
        if (!keep) {
          const unsigned gaps = ~m & (0xFFFFFFFFu << bit);
          fill |= (0xFFFFFFFFu << bit) & (gaps ? (gaps & (0u - gaps)) - 1u : 0xFFFFFFFFu);
        }
      }
    }
    // the warp writes the changed words one after the other, a voxel a lane
    unsigned todo = __ballot_sync(0xffffffffu, (fill | zero) != 0u);
    const long long base = (long long)(r * g.X) + 32 * w;
    while (todo) {
      const int j = __ffs(todo) - 1;
      todo &= todo - 1u;
      const unsigned f = __shfl_sync(0xffffffffu, fill, j), q = __shfl_sync(0xffffffffu, zero, j);
      const long long b = __shfl_sync(0xffffffffu, base, j);
      if ((f >> lane) & 1u) img[b + lane] = (uint8_t)k;
      if ((q >> lane) & 1u) img[b + lane] = 0;
    }
  });
}

Words words_of(int Z, int Y, int X) {
  // One voxel a row: the rows of a plane are a row (same voxels in the same order,
  // same neighbours), and so for planes of one row.
  for (int k = 0; k < 2 && X == 1; ++k) {
    X = Y;
    Y = Z;
    Z = 1;
  }
  Words g{};
  g.Z = Z;
  g.Y = Y;
  g.X = X;
  g.W = (X + 31) / 32;
  g.n = (uint32_t)((int64_t)Z * Y * g.W);
  g.lg = 5;
  while (g.lg > 0 && (1 << (g.lg - 1)) >= X) --g.lg;
  g.lanes = 1 << g.lg;
  g.by_W = FastDiv((uint32_t)g.W);
  g.by_Y = FastDiv((uint32_t)Y);
  return g;
}

}  // namespace
}  // namespace si

using namespace si;

// info block (256 bytes), 256 maxima, one word per 32 voxels of a row, size,
// parent
static uint64_t cc_scratch_need(int Z, int Y, int X) {
  return (uint64_t)Z * Y * X * 8 + 256 * sizeof(unsigned) + 256 + (uint64_t)Z * Y * ((X + 31) / 32) * sizeof(unsigned);
}

extern "C" int si_cc_scratch_bytes(int Z, int Y, int X, uint64_t* bytes) {
  clear_error();
  if (!bytes || Z < 1 || Y < 1 || X < 1) return set_error(SI_ERR_ARG, "si_cc_scratch_bytes: bad arguments");
  *bytes = cc_scratch_need(Z, Y, X);
  return 0;
}

static int cc_check(const char* who, const void* a, int Z, int Y, int X, void* scratch, uint64_t scratch_bytes) {
  if (!a || !scratch) return set_error(SI_ERR_ARG, "%s: null pointer", who);
  if (Z < 1 || Y < 1 || X < 1) return set_error(SI_ERR_ARG, "%s: bad shape", who);
  const int64_t V = (int64_t)Z * Y * X;
  if (V > 0x7fffffffLL) return set_error(SI_ERR_ARG, "%s: more than 2^31 - 1 voxels", who);
  if (scratch_bytes < cc_scratch_need(Z, Y, X) || (uintptr_t)scratch % 16)
    return set_error(SI_ERR_ARG, "%s: scratch too small or misaligned", who);
  return 0;
}

// The scratch's parts: info block first (aligned), then the arrays.
struct CcScratch {
  CcInfo* info;
  unsigned *big, *words, *size;
  int* L;
  CcScratch(void* scratch, const Words& g) {
    uint8_t* b = static_cast<uint8_t*>(scratch);
    info = reinterpret_cast<CcInfo*>(b);
    big = reinterpret_cast<unsigned*>(b + 256);
    words = big + 256;
    size = words + g.n;
    L = reinterpret_cast<int*>(size + (int64_t)g.Z * g.Y * g.X);
  }
};

extern "C" int si_clean(const uint8_t* labels, uint8_t* out, int Z, int Y, int X, double threshold, int skip_label,
                        void* scratch, uint64_t scratch_bytes, void* stream) {
  clear_error();
  if (int rc = cc_check("si_clean", labels, Z, Y, X, scratch, scratch_bytes)) return rc;
  if (!out) return set_error(SI_ERR_ARG, "si_clean: null output");
  const Words g = words_of(Z, Y, X);
  const CcScratch c(scratch, g);
  cudaStream_t st = as_stream(stream);
  const int per_warp = grid_for((int64_t)g.n * g.lanes), per_thread = grid_for(g.n);
  if (cudaMemsetAsync(c.big, 0, 256 * sizeof(unsigned), st) != cudaSuccess)
    return set_error(SI_ERR_CUDA, "si_clean: memset failed");
  const bool sh = g.lanes < 32;
  (sh ? clean_starts_kernel<true> : clean_starts_kernel<false>)<<<per_warp, 256, 0, st>>>(labels, g, skip_label,
                                                                                          c.words, c.L, c.size);
  (sh ? clean_merge_kernel<true> : clean_merge_kernel<false>)<<<per_warp, 256, 0, st>>>(labels, g, skip_label, c.words,
                                                                                        c.L);
  clean_count_kernel<<<per_thread, 256, 0, st>>>(labels, g, skip_label, c.words, c.L, c.size);
  clean_max_kernel<<<per_thread, 256, 0, st>>>(labels, g, skip_label, c.words, c.L, c.size, c.big);
  (sh ? clean_write_kernel<true> : clean_write_kernel<false>)<<<per_warp, 256, 0, st>>>(
      labels, g, skip_label, c.words, c.L, c.size, c.big, threshold, out);
  return check_launch("si_clean");
}

extern "C" int si_fill(uint8_t* img, int Z, int Y, int X, double threshold, const int* label_list, int n_labels,
                       void* scratch, uint64_t scratch_bytes, void* stream) {
  clear_error();
  if (int rc = cc_check("si_fill", img, Z, Y, X, scratch, scratch_bytes)) return rc;
  if (n_labels < 0 || (n_labels > 0 && !label_list)) return set_error(SI_ERR_ARG, "si_fill: bad label list");
  const Words g = words_of(Z, Y, X);
  const CcScratch c(scratch, g);
  cudaStream_t st = as_stream(stream);
  const int mask_grid = std::min(grid_for((int64_t)g.Z * g.Y * 32), sm_count() * 8), per_thread = grid_for(g.n);
  for (int i = 0; i < n_labels; ++i) {
    const int k = label_list[i];
    if (k < 0 || k > 255) return set_error(SI_ERR_ARG, "si_fill: label %d outside 0..255", k);
    fill_info_init_kernel<<<1, 1, 0, st>>>(c.info);
    fill_mask_kernel<<<mask_grid, 256, 0, st>>>(img, g, k, c.words, c.info);
    fill_init_kernel<<<per_thread, 256, 0, st>>>(g, c.words, c.info, c.L, c.size);
    fill_merge_kernel<<<per_thread, 256, 0, st>>>(g, c.words, c.info, c.L);
    fill_count_kernel<<<per_thread, 256, 0, st>>>(g, c.words, c.info, c.L, c.size);
    fill_max_kernel<<<per_thread, 256, 0, st>>>(g, c.words, c.info, c.L, c.size);
    fill_write_kernel<<<per_thread, 256, 0, st>>>(img, g, k, c.words, c.info, c.L, c.size, threshold);
  }
  return check_launch("si_fill");
}
