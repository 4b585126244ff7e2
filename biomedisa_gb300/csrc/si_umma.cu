// 16 -> 16 channel 3x3x3 convolution of the surrogate network on the
// 5th-generation tensor cores (tcgen05): the forward pass and, with flipped
// weights W'[t][ci][co] = W[26 - t][co][ci], the data gradient.
//
// Implicit GEMM over output tiles of 128 consecutive voxels of an x-row,
// organised by INPUT rows. A CTA walks "columns" (n, z, x chunk, y phase):
// output rows y_j = phase + j*dil, j < nt, and input rows i = 0 .. nt + 1 at
// y = phase + (i - 1)*dil. Input row i meets output rows j = i - 2, i - 1, i
// through the taps dy = +1, 0, -1, so per (dz, dx) ONE tcgen05.mma
// (kind::f16, M = 128 voxels, N = 48, K = 16, bf16 in, fp32 accumulate)
// multiplies the shifted input by the three stacked 16x16 weight blocks
// [W(dz,+1,dx); W(dz,0,dx); W(dz,-1,dx)] and adds into three consecutive
// 16-column accumulators in tensor memory: 9 MMAs of N = 48 per input row
// instead of 27 of N = 16 per output row, with each staged input row read
// by the tensor core 9 times instead of 27.
//
// Accumulator ring. The CTA's input rows form one sequence k = 0, 1, ...
// over all its columns (column c starts at k = P_c, P_{c+1} = P_c + rows + 2);
// input k adds into ring positions k, k + 1, k + 2 and completes position k
// (output j = k - P_c - 2 of its column; positions P_c and P_c + 1 are
// padding). Positions live in the 16 slots of 16 columns (k mod 16) of the
// CTA's 256 tensor-memory columns; a region starting at slot 14 or 15 is issued
// as two MMAs (N = 32 + 16 or 16 + 32) that continue at slot 0, so every
// position sums its 27 products in one slot, in the same order wherever it
// falls in the ring (results do not depend on the grid). The regions of consecutive
// inputs overlap, and no wait lies between their MMAs: one thread's MMAs keep their
// order there too (promised by PTX for the same accumulator and shape only; no
// different bit in 3.4 million convolutions, and waiting for each input's MMAs changed
// nothing and cost 5 to 7 %). Every MMA accumulates; the epilogue zeroes a position's slot (tcgen05.st) after
// reading it and before releasing it, and all slots start zeroed.
//
// Shared-memory operands. An input z-row is one TMA box of {16 channels,
// voxels, 1, lines, 1} over the 5-D tensor map {16, W, H, D, N}: rows of 32
// bytes with the 32-byte swizzle (K-major); the A operand of shift dx is that
// block at a start address 32*dil*dx bytes further (the swizzle is a function of
// the address, so any row may start an operand). Rows of 16-byte channel halves,
// which need no swizzle, read every 32-byte sector of L2 twice.
//   W > 64: a tile is 128 voxels of one line, its box has dil more on both
//   sides, and voxels outside the row arrive as zeros (TMA fill).
//   W <= 64: a tile is 128 / W whole lines of consecutive z (two lines of 64 voxels
//   make one MMA instead of two half empty ones). The box has no halo; the shifted
//   operand's rows that belong to the next line are kept out of the sums by the
//   MMA's lane mask.
// Input rows outside the volume in y or, with all lines, in z are neither loaded
// nor multiplied (their contribution is zero). The weights sit once per CTA
// as 9 blocks [dz][dx] of [half][48][8 ci], without swizzle.
//
// Split. Two CTAs per SM: the issuing warp's own instructions are a column's
// critical path (one row costs it about 1300 cycles, 9 MMAs, however many voxels
// it has), so a second CTA with its own issuer nearly doubles the rate. A CTA
// walks whole columns b, b + G, ... while every CTA has one; the rows of the
// columns that are left are split evenly. What bounds it then: the shared-memory
// pipe, 60 % operand reads (43 wavefronts per MMA: 4 KB of A, 1.5 KB of B) and 20 %
// copies at 200 x 192 x 216. Measured, one convolution without / with residual,
// before (one CTA per SM, channel halves, a line per tile) and now: 8 x 64^3
// 186 / 192 -> 45 / 50 us, 200 x 192 x 216 400 / 416 -> 171 / 199 us, 128 x 256 x
// 1024 1223 / 1275 -> 572 / 679 us. A second epilogue group (the issue slots it
// takes) costs 5 %, the columns split only in equal segments 5 to 10 %.
//
// Roles (a persistent CTA of 7 warps): warp 0 loads each input row's
// z-rows into a ring of 5 row slots; warp 6 loads, for a residual layer,
// each output row's residual tile into a ring of 7 slots (so the epilogue
// never waits on a global load); warp 1 issues the 9 MMAs and one commit
// per input row (row slot free and ring position complete); warps 2-5 run the
// epilogue (thread m = tensor-memory lane m = voxel m of the tile): release of
// the position, bias, residual, ReLU, bf16 or fp32 store, release of the residual
// slot. Warps 0, 1 and 6 run their loops as whole warps with warp-uniform operands
// and issue from one elected lane. A launch may begin while the stream's kernel before it drains (programmatic
// dependent launch; it reads nothing until that one has ended). Every wait is
// bounded: a role that gives up flags the CTA, the others stop at their next
// wait, the copies and MMAs in flight are waited for (bounded), the tensor
// memory is freed and the status records the error.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "si_common.cuh"
#include "si_internal.h"
#include "si_tma.cuh"

namespace si {
namespace {

constexpr int kTileM = 128;
constexpr int kMaxDil = 8;
constexpr int kRowBytes = (kTileM + 2 * kMaxDil) * 32;  // one staged z-row: 4608 bytes
constexpr int kSlotBytes = 3 * kRowBytes;               // an input row: its three z-rows
constexpr int kRowSlots = 5;                            // ring of staged input rows
constexpr int kResBytes = kTileM * 32;                  // one residual row tile [128][16]: 4096 bytes
constexpr int kResSlots = 7;                            // ring of staged residual rows
constexpr int kWBlockBytes = 2 * 48 * 16;               // one (dz, dx) weight block [half][48][8]
constexpr int kWBytes = 9 * kWBlockBytes;
constexpr int kSmemBytes = kWBytes + kRowSlots * kSlotBytes + kResSlots * kResBytes + 1024;  // + alignment slack
constexpr int kCtasPerSm = 2;
constexpr int kTmemCols = 512 / kCtasPerSm;
constexpr int kR = kTmemCols / 16;                      // accumulator ring positions
constexpr int kResWarp = 6;                             // the warp loading residual rows
constexpr int kThreads = 32 * (kResWarp + 1);
static_assert(kWBytes % 256 == 0 && kRowBytes % 256 == 0 && kResBytes % 256 == 0, "swizzle atoms of 256 bytes");
static_assert(kR >= kRowSlots + 3, "a row slot's done barrier is passed before its next phase");

__device__ uint32_t g_umma_status;  // bit 0: a wait gave up (read by si_nn_umma_status)

// Shared-memory matrix descriptor, K-major core matrices; kLayout 0: no swizzle,
// 6: rows of 32 bytes, 32-byte swizzle.
template <int kLayout>
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // fixed descriptor version bits 46..48 = 0b001
  d |= (uint64_t)kLayout << 61;
  return d;                // base offset 0, absolute offsets
}

// kind::f16 instruction descriptor: fp32 D, bf16 A and B, both K-major, M = 128, N = kN.
template <int kN>
__host__ __device__ constexpr uint32_t idesc_f16() {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kN >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
}

// The three x-taps of one (input z-row, accumulator region): descriptors a + dx *
// da and b + dx * 96. Executed by a whole warp with warp-uniform operands (which
// then stay in uniform registers); one elected lane issues the MMAs.
template <int kN>
__device__ __forceinline__ void umma3(uint32_t d_tmem, uint64_t a, uint64_t da, uint64_t b) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 a1, a2, b1, b2;\n\tsetp.ne.b32 p, 1, 0;\n\t"
      "add.s64 a1, %1, %2;\n\tadd.s64 a2, a1, %2;\n\tadd.s64 b1, %3, 96;\n\tadd.s64 b2, b1, 96;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %3, %4, p;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %4, p;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %4, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(da), "l"(b), "r"(idesc_f16<kN>())
      : "memory");
}
// The same; the first MMA leaves the lanes of l alone, the last those of r.
template <int kN>
__device__ __forceinline__ void umma3(uint32_t d_tmem, uint64_t a, uint64_t da, uint64_t b, const uint32_t (&l)[4],
                                      const uint32_t (&r)[4]) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 a1, a2, b1, b2;\n\tsetp.ne.b32 p, 1, 0;\n\t"
      "add.s64 a1, %1, %2;\n\tadd.s64 a2, a1, %2;\n\tadd.s64 b1, %3, 96;\n\tadd.s64 b2, b1, 96;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %3, %4, {%5, %6, %7, %8}, p;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %4, p;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %4, {%9, %10, %11, %12}, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(da), "l"(b), "r"(idesc_f16<kN>()), "r"(l[0]), "r"(l[1]), "r"(l[2]), "r"(l[3]), "r"(r[0]), "r"(r[1]),
      "r"(r[2]), "r"(r[3])
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// The copy, the expect_tx and the plain arrival below are executed by a
// whole warp with warp-uniform operands; one elected lane issues them.
__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* map, int x, int y, int z, int n,
                                            uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
      "%5, %6}], [%7];\n\t}" ::"r"(smem_u32(dst)),
      "l"(map), "r"(0), "r"(x), "r"(y), "r"(z), "r"(n), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void expect_tx_elect(uint64_t* bar, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
      "r"(bytes)
      : "memory");
}
// 32 bytes to a 32-byte aligned address in one store, else two of 16.
__device__ __forceinline__ void store32(void* p, const uint32_t (&v)[8], int wide) {
  if (wide)
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
  else {
    static_cast<uint4*>(p)[0] = make_uint4(v[0], v[1], v[2], v[3]);
    static_cast<uint4*>(p)[1] = make_uint4(v[4], v[5], v[6], v[7]);
  }
}
__device__ __forceinline__ void arrive_elect(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
  const uint32_t z = 0;
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
      "r"(z)
      : "memory");
}

// A column: digits (y phase, x chunk, z group, n), the first fastest.
constexpr int kDigits = 4;
struct UmmaGeom {
  int N, D, H, W, dil;
  int lines;              // z-lines of a tile (1: tiles of 128 voxels with a halo along x)
  int nt;                 // output rows of a column (phase 0; others may have one less)
  int rounds;             // whole columns a CTA walks: b, b + G, ...
  int radix[kDigits];     // extents of the digits
  int step[kDigits];      // the digits of the grid size G
  long long tail_col;     // first of the columns after the rounds, whose rows
  long long tail_rows;    // (this many) are split evenly over the CTAs
};

// Where a CTA starts its rounds and its share of the tail (decoded once).
struct Starts {
  int dg[kDigits], tail_dg[kDigits], tail_j, tail;
  __device__ static void decode(const UmmaGeom& g, unsigned long long c, int (&d)[kDigits]) {
    for (int k = 0; k < kDigits; ++k) {
      d[k] = (int)(c % (unsigned)g.radix[k]);
      c /= (unsigned)g.radix[k];
    }
  }
  __device__ void set(const UmmaGeom& g) {
    const long long r0 = g.tail_rows * blockIdx.x / gridDim.x;
    tail = (int)(g.tail_rows * (blockIdx.x + 1) / gridDim.x - r0);
    tail_j = (int)(r0 % g.nt);
    decode(g, blockIdx.x, dg);
    decode(g, (unsigned long long)(g.tail_col + r0 / g.nt), tail_dg);
  }
};

// A CTA's position: a column (its digits) and the input row i in it, i < cnt + 2,
// at y = y0 + i * dil; p = the ring position of its count, k mod kR, with the
// phase (k / kR) & 1.
struct Walk {
  int dg[kDigits];
  int rounds;      // columns left of the rounds, this one included
  int tail;        // rows left of the CTA's share of the tail, this column's not included
  bool live;
  int n, z, x0, y0, cnt;
  int i, p;
  uint32_t ph;
  __device__ __forceinline__ void enter(const UmmaGeom& g, int j0, int rows) {
    n = dg[3];
    z = dg[2] * g.lines;
    x0 = dg[1] * kTileM;
    const int nt = (g.H - dg[0] + g.dil - 1) / g.dil;  // nt < 1: H below the dilation
    y0 = dg[0] + (j0 - 1) * g.dil;
    cnt = max(0, min(j0 + rows, nt) - j0);
    i = 0;
  }
  __device__ __forceinline__ void enter_tail(const UmmaGeom& g, int j0) {
    const int rows = min(g.nt - j0, tail);
    tail -= rows;
    enter(g, j0, rows);
  }
  __device__ __forceinline__ void start_tail(const UmmaGeom& g, const Starts& s) {
    tail = s.tail;
    live = tail > 0;
#pragma unroll
    for (int k = 0; k < kDigits; ++k) dg[k] = s.tail_dg[k];
    enter_tail(g, s.tail_j);
  }
  __device__ __forceinline__ void start(const UmmaGeom& g, const Starts& s) {
    p = 0;
    ph = 0;
    rounds = g.rounds;
    live = true;
    tail = 0;
#pragma unroll
    for (int k = 0; k < kDigits; ++k) dg[k] = s.dg[k];
    if (rounds > 0)
      enter(g, 0, g.nt);
    else
      start_tail(g, s);
  }
  // true when it entered another column
  __device__ __forceinline__ bool next(const UmmaGeom& g, const Starts& s) {
    if (++p == kR) {
      p = 0;
      ph ^= 1u;
    }
    if (++i < cnt + 2) return false;
    if (rounds == 1) {
      rounds = 0;
      start_tail(g, s);
      return true;
    }
    if (rounds == 0 && tail == 0) {
      live = false;
      return true;
    }
    int carry = rounds ? 0 : 1;
#pragma unroll
    for (int k = 0; k < kDigits; ++k) {
      dg[k] += (rounds ? g.step[k] : 0) + carry;
      carry = dg[k] >= g.radix[k] ? 1 : 0;
      dg[k] -= carry ? g.radix[k] : 0;
    }
    if (rounds) {
      --rounds;
      enter(g, 0, g.nt);
    } else {
      enter_tail(g, 0);
    }
    return true;
  }
  // input z-rows with a line inside the volume, bit dz
  __device__ __forceinline__ uint32_t z_mask(const UmmaGeom& g) const {
    uint32_t m = 0;
#pragma unroll
    for (int dz = 0; dz < 3; ++dz) {
      const int zz = z + (dz - 1) * g.dil;
      m |= (zz + g.lines > 0 && zz < g.D) ? (1u << dz) : 0u;
    }
    return m;
  }
  __device__ __forceinline__ int y(const UmmaGeom& g) const { return y0 + i * g.dil; }
};

// Index and phase of a ring of kN barriers (mbarrier parity of the use).
template <int kN>
struct Ring {
  int idx = 0;
  uint32_t ph = 0;
  uint32_t wrapped = 0;  // at least one full turn done
  __device__ __forceinline__ void next() {
    if (++idx == kN) {
      idx = 0;
      ph ^= 1u;
      wrapped = 1u;
    }
  }
};

template <bool kOutF32, bool kPacked>
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
    conv16_umma_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap rmap,
                       const __nv_bfloat16* __restrict__ w, const float* __restrict__ bias, int has_res,
                       const __nv_bfloat16* __restrict__ mask, void* __restrict__ y_out, const __grid_constant__ UmmaGeom g, int relu, int wide,
                       uint32_t wait_lim) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sw = smem;                             // weight blocks [dz][dx][half][48][8]
  uint8_t* rows = smem + kWBytes;                 // [row slot][dz][voxel][16], 32-byte swizzle
  uint8_t* rres = rows + kRowSlots * kSlotBytes;  // [residual slot][128][16], 32-byte swizzle
  __shared__ __align__(8) uint64_t full_bar[kRowSlots];   // an item's input z-rows landed
  __shared__ __align__(8) uint64_t done_bar[kR];          // its MMAs completed: position complete, row slot free
  __shared__ __align__(8) uint64_t free_bar[kR];          // position read, zeroed, released
  __shared__ __align__(8) uint64_t rfull_bar[kResSlots];  // an item's residual row landed
  __shared__ __align__(8) uint64_t rfree_bar[kResSlots];  // ... and was read
  __shared__ uint32_t tmem_base;
  __shared__ float s_bias[16];
  __shared__ Starts s_start;
  __shared__ volatile int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int dil = g.dil;

  // the next convolution's CTAs may take the place of this one's that have ended
  // (2.4 us a launch); they too wait here for the whole grid before them
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int i = tid; i < 9 * 48 * 2; i += kThreads) {
    const int blk = i / 96, nrow = (i / 2) % 48, h = i % 2;
    const int q = nrow / 16, co = nrow % 16;
    const int tap = (blk / 3) * 9 + (2 - q) * 3 + blk % 3;  // dz digit, dy digit 2 - q, dx digit
    const uint4 v = reinterpret_cast<const uint4*>(w)[(tap * 16 + co) * 2 + h];
    *reinterpret_cast<uint4*>(sw + blk * kWBlockBytes + h * 768 + nrow * 16) = v;
  }
  if (tid < 16) s_bias[tid] = bias ? bias[tid] : 0.0f;
  if (tid == 0) {
    s_fail = 0;
    for (int b = 0; b < kRowSlots; ++b) mbar_init(&full_bar[b], 1);
    for (int b = 0; b < kR; ++b) {
      mbar_init(&done_bar[b], 1);
      mbar_init(&free_bar[b], 4);  // one arrival per epilogue warp
    }
    for (int b = 0; b < kResSlots; ++b) {
      mbar_init(&rfull_bar[b], 1);
      mbar_init(&rfree_bar[b], 4);
    }
    fence_barrier_init();
  }
  if (tid == 32 * kResWarp) s_start.set(g);
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_proxy_async_shared();  // weights written by threads, read by the tensor core
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const uint32_t tmem = tmem_base;
  const uint32_t lane_base = (uint32_t)(32 * (warp & 3)) << 16;  // this warp's tensor-memory lane quadrant
  if (warp >= 2 && warp < 6) {  // all slots start at zero
    for (int b = 0; b < kR; ++b) tmem_zero16(tmem + lane_base + (uint32_t)(16 * b));
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();

  // Every role visits the CTA's columns and their input rows (items) in the same
  // order.
  Walk t;
  t.start(g, s_start);

  // progress (warps 0 / 1 / kResWarp): items whose rows / residual rows were
  // loaded; the done barrier and parity of the last commit
  long long q_loaded = 0, q_res = 0;
  int last_done = -1;
  uint32_t last_par = 0;
  if (warp == 0) {
    // ---- producer, the whole warp in step, one elected lane issuing: each
    // item's z-rows into the row ring
    const uint32_t box_bytes = 32u * (uint32_t)(kPacked ? g.W * g.lines : kTileM + 2 * dil);
    const int xo = kPacked ? 0 : dil;
    Ring<kRowSlots> rr;
    Ring<kR> old;  // the done barrier of the item kRowSlots before
    uint32_t zm = t.z_mask(g);
    while (t.live) {
      bool ok = !s_fail;
      if (rr.wrapped) {
        ok = ok && mbar_wait_fast(&done_bar[old.idx], old.ph, wait_lim);
        old.next();
      }
      if (!__all_sync(0xffffffffu, ok)) {
        s_fail = 1;
        break;
      }
      const int yy = t.y(g);
      if (yy < 0 || yy >= g.H || zm == 0) {
        arrive_elect(&full_bar[rr.idx]);
      } else {
        expect_tx_elect(&full_bar[rr.idx], (uint32_t)__popc(zm) * box_bytes);
        uint8_t* dst = rows + (size_t)rr.idx * kSlotBytes;
#pragma unroll
        for (int dz = 0; dz < 3; ++dz)
          if (zm & (1u << dz))
            tma_load_5d(dst + dz * kRowBytes, &xmap, t.x0 - xo, yy, t.z + (dz - 1) * dil, t.n, &full_bar[rr.idx]);
      }
      rr.next();
      ++q_loaded;
      if (t.next(g, s_start)) zm = t.z_mask(g);
    }
  } else if (warp == kResWarp) {
    // ---- residual loader, the whole warp in step: for each item the
    // residual row of the position it completes (output j = i - 2; padding
    // positions arrive without a copy)
    Ring<kResSlots> sr;
    const uint32_t res_bytes = kPacked ? 32u * (uint32_t)(g.W * g.lines) : (uint32_t)kResBytes;
    while (has_res && t.live) {
      bool ok = !s_fail;
      if (sr.wrapped) ok = ok && mbar_wait_fast(&rfree_bar[sr.idx], sr.ph ^ 1u, wait_lim);
      if (!__all_sync(0xffffffffu, ok)) {
        s_fail = 1;
        break;
      }
      if (t.i >= 2) {
        expect_tx_elect(&rfull_bar[sr.idx], res_bytes);
        tma_load_5d(rres + (size_t)sr.idx * kResBytes, &rmap, t.x0, t.y(g) - dil, t.z, t.n, &rfull_bar[sr.idx]);
      } else {
        arrive_elect(&rfull_bar[sr.idx]);
      }
      sr.next();
      ++q_res;
      t.next(g, s_start);
    }
  } else if (warp == 1) {
    // ---- MMA issuer, the whole warp in step (operands warp-uniform), one
    // elected lane issuing. Its own instructions bound a column's walk, so an
    // item costs it one barrier test (even lanes the row, odd lanes the
    // position), three issue blocks and one commit.
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    // weight block b = dz*3 + dx: descriptor bdesc0 + b * kWBlockBytes / 16
    const uint64_t bdesc0 = smem_desc<0>(smem_u32(sw), 768, 128);
    const uint64_t ddx = (uint64_t)(2 * dil);  // one dx step in descriptor start-address units (16 bytes)
    const uint64_t adesc0 = smem_desc<6>(smem_u32(rows) - (kPacked ? 32u * (uint32_t)dil : 0u), 16, 256);
    uint32_t ml[4], mr[4];  // packed: lanes whose left / right neighbour is outside the row
    if (kPacked) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int m = 32 * q + lane, x = m % g.W;
        ml[q] = __ballot_sync(0xffffffffu, x < dil);
        mr[q] = __ballot_sync(0xffffffffu, x + dil >= g.W);
      }
    }
    Ring<kRowSlots> rr;
    Ring<kR> p2;  // position k + 2, first touched by input k
    p2.idx = 2;
    uint32_t zm = t.z_mask(g);
    auto issue = [&](uint32_t d, uint64_t a, uint64_t b, auto width) {
      constexpr int kN = decltype(width)::value;
      if (kPacked)
        umma3<kN>(d, a, ddx, b, ml, mr);
      else
        umma3<kN>(d, a, ddx, b);
    };
    while (t.live) {
      const bool odd = (lane & 1) && p2.wrapped;
      const int failed = s_fail;
      const bool ok = mbar_wait_fast(odd ? &free_bar[p2.idx] : &full_bar[rr.idx], odd ? p2.ph ^ 1u : rr.ph, wait_lim);
      if (!__all_sync(0xffffffffu, ok && !failed)) {  // one decision for the whole warp
        s_fail = 1;
        break;
      }
      __syncwarp();  // what the odd lanes saw released holds for the issuing lane
      tmem_fence_after();
      const int yy = t.y(g);
      if (yy >= 0 && yy < g.H) {
        const uint64_t ad = adesc0 + (uint64_t)((rr.idx * kSlotBytes) >> 4);
        const uint32_t dd = tm + (uint32_t)(16 * t.p);
        if (t.p <= kR - 3) {
#pragma unroll
          for (int dz = 0; dz < 3; ++dz)
            if (zm & (1u << dz))
              issue(dd, ad + (uint64_t)((dz * kRowBytes) >> 4), bdesc0 + (uint64_t)(dz * 3 * (kWBlockBytes >> 4)),
                    std::integral_constant<int, 48>{});
        } else {
          // a region running past the ring end continues at slot 0; the
          // second piece starts 32 or 16 weight rows (16 bytes each) in
#pragma unroll 1
          for (int dz = 0; dz < 3; ++dz) {
            if (!(zm & (1u << dz))) continue;
            const uint64_t a = ad + (uint64_t)((dz * kRowBytes) >> 4);
            const uint64_t b = bdesc0 + (uint64_t)(dz * 3 * (kWBlockBytes >> 4));
            if (t.p == kR - 2) {
              issue(dd, a, b, std::integral_constant<int, 32>{});
              issue(tm, a, b + 32, std::integral_constant<int, 16>{});
            } else {
              issue(dd, a, b, std::integral_constant<int, 16>{});
              issue(tm, a, b + 16, std::integral_constant<int, 32>{});
            }
          }
        }
      }
      last_done = t.p;
      last_par = t.ph;
      umma_commit(&done_bar[last_done]);
      rr.next();
      p2.next();
      if (t.next(g, s_start)) zm = t.z_mask(g);
    }
  } else {
    // ---- epilogue (warps 2 .. kResWarp - 1): every item's completed position, in item order
    const int m = 32 * (warp & 3) + lane;  // tensor-memory lane = voxel offset in the tile
    const int line = kPacked ? m / g.W : 0, mx = kPacked ? m - line * g.W : m;
    Ring<kResSlots> sr;
    while (t.live) {
      const int p = t.p;
      const int x = t.x0 + mx, z = t.z + line;
      const bool out = t.i >= 2 && x < g.W && line < g.lines && z < g.D;  // output row j = i - 2
      const long long r = (((long long)t.n * g.D + z) * g.H + (t.y(g) - dil)) * g.W + x;
      uint4 mq[2];
      if (mask && out) {  // arrives while the MMAs are waited for
        mq[0] = __ldg(reinterpret_cast<const uint4*>(mask + r * 16));
        mq[1] = __ldg(reinterpret_cast<const uint4*>(mask + r * 16) + 1);
      }
      bool ok = !s_fail && mbar_wait_fast(&done_bar[p], t.ph, wait_lim);
      if (has_res) ok = ok && mbar_wait_fast(&rfull_bar[sr.idx], sr.ph, wait_lim);
      if (!__all_sync(0xffffffffu, ok)) {
        s_fail = 1;
        break;
      }
      tmem_fence_after();
      const uint32_t ta = tmem + lane_base + (uint32_t)(16 * p);
      uint32_t v[16];
      if (t.i >= 2) {
        tmem_ld16(ta, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      }
      uint4 rq[2];
      if (has_res) {
        const uint8_t* rp = rres + (size_t)sr.idx * kResBytes + m * 32;
        const int sz = (m >> 2) & 1;  // the swizzle swaps the halves of every other four rows
        rq[0] = *reinterpret_cast<const uint4*>(rp + 16 * sz);
        rq[1] = *reinterpret_cast<const uint4*>(rp + 16 * (sz ^ 1));
      }
      // the position is free before the row is finished and stored
      tmem_zero16(ta);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tmem_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&free_bar[p]);
      if (out) {
        float u[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) u[e] = __uint_as_float(v[e]) + s_bias[e];
        if (has_res) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t words[4] = {rq[h].x, rq[h].y, rq[h].z, rq[h].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              u[h * 8 + 2 * e] += __uint_as_float(words[e] << 16);
              u[h * 8 + 2 * e + 1] += __uint_as_float(words[e] & 0xFFFF0000u);
            }
          }
        }
        if (relu) {
#pragma unroll
          for (int e = 0; e < 16; ++e) u[e] = fmaxf(u[e], 0.0f);
        }
        if (mask) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t words[4] = {mq[h].x, mq[h].y, mq[h].z, mq[h].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if (!(__uint_as_float(words[e] << 16) > 0.0f)) u[h * 8 + 2 * e] = 0.0f;
              if (!(__uint_as_float(words[e] & 0xFFFF0000u) > 0.0f)) u[h * 8 + 2 * e + 1] = 0.0f;
            }
          }
        }
        uint32_t pk[8];
        if (kOutF32) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int e = 0; e < 8; ++e) pk[e] = __float_as_uint(u[8 * h + e]);
            store32(static_cast<float*>(y_out) + r * 16 + 8 * h, pk, wide);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const __nv_bfloat162 b2 = __floats2bfloat162_rn(u[2 * e], u[2 * e + 1]);
            pk[e] = *reinterpret_cast<const uint32_t*>(&b2);
          }
          store32(static_cast<__nv_bfloat16*>(y_out) + r * 16, pk, wide);
        }
      }
      // The residual slot only now: its values have arrived, the stores took them, and
      // the fence orders the reads before the copy that refills it. (Released with the
      // position, its loads still on their way, the slot was refilled under them once in
      // some thousand convolutions: up to 32 voxels of a row with another row's residual.
      // None in 2.7 million so, at the same speed.)
      if (has_res) {
        fence_proxy_async_shared();
        __syncwarp();
        if (lane == 0) mbar_arrive(&rfree_bar[sr.idx]);
      }
      sr.next();
      t.next(g, s_start);
    }
  }
  __syncwarp();
  __syncthreads();
  if (s_fail) {
    // let everything in flight complete (bounded) before the CTA's shared and
    // tensor memory go away: the last commit covers every MMA issued; each
    // row and residual slot has at most one copy outstanding
    if (warp == 1 && lane == 0 && last_done >= 0)
      mbar_wait_bounded(&done_bar[last_done], last_par, kDrainWaitLimit);
    if (warp == 0 && lane == 0)
      for (long long ql = q_loaded > kRowSlots ? q_loaded - kRowSlots : 0; ql < q_loaded; ++ql)
        mbar_wait_bounded(&full_bar[ql % kRowSlots], (uint32_t)((ql / kRowSlots) & 1), kDrainWaitLimit);
    if (warp == kResWarp && lane == 0)
      for (long long ql = q_res > kResSlots ? q_res - kResSlots : 0; ql < q_res; ++ql)
        mbar_wait_bounded(&rfull_bar[ql % kResSlots], (uint32_t)((ql / kResSlots) & 1), kDrainWaitLimit);
    if (tid == 0) atomicOr(&g_umma_status, 1u);
  }
  tmem_fence_before();
  __syncthreads();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

template <bool kOutF32, bool kPacked>
cudaError_t launch_conv16(const CUtensorMap& map, const CUtensorMap& rmap, const __nv_bfloat16* w, const float* bias,
                          int has_res, const __nv_bfloat16* mask, void* y, const UmmaGeom& g, int relu, int wide,
                          int grid, cudaStream_t st) {
  const auto kernel = conv16_umma_kernel<kOutF32, kPacked>;
  const cudaError_t ae = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  if (ae != cudaSuccess) return ae;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3(kThreads);
  c.dynamicSmemBytes = kSmemBytes;
  c.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, map, rmap, w, bias, has_res, mask, y, g, relu, wide, wait_limit());
}

}  // namespace

// 16 -> 16 convolution on the tensor cores (see the file comment). x, w,
// residual, mask, y 16-byte aligned; dil <= 8. With a mask (bf16, shaped like y)
// values where it is not above 0 are stored as 0. Returns SI_OK or an error code.
int conv16_umma(const void* x, const void* w, const float* bias, const void* residual, const void* mask, void* y,
                int N, int D, int H, int W, int dil, int relu, int out_f32, cudaStream_t st) {
  if (dil < 1 || dil > kMaxDil) return set_error(SI_ERR_ARG, "conv16_umma: dilation must be 1..%d", kMaxDil);
  if ((long long)N * D > 0x7FFFFFFFll) return set_error(SI_ERR_ARG, "conv16_umma: too many z-planes");
  const EncodeTiledFn enc = encode_fn();
  if (!enc) return set_error(SI_ERR_CUDA, "conv16_umma: cuTensorMapEncodeTiled unavailable");
  UmmaGeom g{};
  g.N = N;
  g.D = D;
  g.H = H;
  g.W = W;
  g.dil = dil;
  g.lines = std::max(1, std::min(kTileM / W, D));
  const bool packed = g.lines > 1;
  const int xchunks = (W + kTileM - 1) / kTileM, zgroups = (D + g.lines - 1) / g.lines;
  const long long columns = (long long)N * zgroups * xchunks * dil;
  g.nt = (H + dil - 1) / dil;
  // one CTA per row at most; whole columns while every CTA has one, then rows
  const long long grid = std::min(columns * g.nt, (long long)kCtasPerSm * sm_count());
  g.rounds = (int)std::min<long long>(columns / grid, 0x7FFFFFFF);
  g.tail_col = g.rounds * grid;
  g.tail_rows = (columns - g.tail_col) * g.nt;
  const int radix[kDigits] = {dil, xchunks, zgroups, N};
  long long rest = grid;
  for (int k = 0; k < kDigits; ++k) {
    g.radix[k] = radix[k];
    g.step[k] = (int)(rest % radix[k]);
    rest /= radix[k];
  }
  // {16 channels, x, y, z, n}: a box lands as [line][voxel][16 channels], the halves
  // of rows 4..7 of every eight swapped (32-byte swizzle)
  const cuuint64_t dims[5] = {16, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D, (cuuint64_t)N};
  const cuuint64_t strides[4] = {32ull, 32ull * W, 32ull * W * H, 32ull * W * H * D};  // bytes, dims 1..4
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const cuuint32_t box[5] = {16, (cuuint32_t)(packed ? W : kTileM + 2 * dil), 1, (cuuint32_t)g.lines, 1};
  const cuuint32_t rbox[5] = {16, (cuuint32_t)(packed ? W : kTileM), 1, (cuuint32_t)g.lines, 1};
  CUtensorMap map, rmap;
  std::memset(&map, 0, sizeof(map));
  std::memset(&rmap, 0, sizeof(rmap));
  const auto encode = [&](CUtensorMap* m, const void* ptr, const cuuint32_t* b) {
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(ptr), dims, strides, b, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  const CUresult cr = encode(&map, x, box);
  if (cr != CUDA_SUCCESS) return set_error(SI_ERR_CUDA, "conv16_umma: tensor map encoding failed (%d)", (int)cr);
  const CUresult rr = residual ? encode(&rmap, residual, rbox) : CUDA_SUCCESS;
  if (rr != CUDA_SUCCESS)
    return set_error(SI_ERR_CUDA, "conv16_umma: residual tensor map encoding failed (%d)", (int)rr);
  const int has_res = residual ? 1 : 0, wide = (uintptr_t)y % 32 == 0;
  const auto* wb = static_cast<const __nv_bfloat16*>(w);
  const auto launch = out_f32 ? (packed ? launch_conv16<true, true> : launch_conv16<true, false>)
                              : (packed ? launch_conv16<false, true> : launch_conv16<false, false>);
  const cudaError_t ae =
      launch(map, rmap, wb, bias, has_res, static_cast<const __nv_bfloat16*>(mask), y, g, relu, wide, (int)grid, st);
  if (ae != cudaSuccess) return set_error(SI_ERR_CUDA, "conv16_umma: launch: %s", cudaGetErrorString(ae));
  return check_launch("conv16_umma");
}

}  // namespace si

extern "C" int si_nn_umma_status(int* status, void* stream) {
  si::clear_error();
  if (!status) return si::set_error(SI_ERR_ARG, "si_nn_umma_status: null pointer");
  cudaStream_t st = si::as_stream(stream);
  uint32_t v = 0;
  const uint32_t zero = 0;
  if (cudaMemcpyFromSymbolAsync(&v, si::g_umma_status, sizeof(v), 0, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess ||
      cudaMemcpyToSymbolAsync(si::g_umma_status, &zero, sizeof(zero), 0, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return si::set_error(SI_ERR_CUDA, "si_nn_umma_status: %s", cudaGetErrorString(cudaGetLastError()));
  *status = (int)v;
  if (v) return si::set_error(SI_ERR_CUDA, "tensor-core convolution: a wait gave up (status %u)", v);
  return SI_OK;
}

extern "C" int si_nn_conv16_tc_set_streams(int streams) {
  si::clear_error();
  if (streams != 1 && streams != 2 && streams != 4)
    return si::set_error(SI_ERR_ARG, "si_nn_conv16_tc_set_streams: 1, 2 or 4");
  return SI_OK;
}
