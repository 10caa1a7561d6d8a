// Prefill matmul on the 5th-generation tensor cores: out[m, n] = sum_k x[m, k] * bf16(q[n, k] * s + b).
//
// Arithmetic contract (the reference's prefill form, cuda/kernels/qmm_prefill.cu:1,115-118): every weight is rounded once
// to bf16, w = bf16(fma(q, s, b)) with q exact, then ONE fp32 accumulation chain runs over all of K in 16-input steps
// (tcgen05.mma, accumulator in tensor memory).  Any chunking of the rows gives the same bits; they are not the decode
// kernel's bits (that one keeps the affine terms in fp32).
//
// Two blocks (a cluster on one SM pair) share a tile of 256 output columns x up to 192 rows of x, "swap-AB": the
// dequantised weights are the MMA's A operand (M = 256, 128 columns a block), the rows of x its B operand (N, half of them
// in each block's shared memory), cta_group::2.  What bounds it is the tensor pipe, so everything else is kept below its
// pace (2 N cycles a stage of 64 inputs):
//   * A lives in TENSOR MEMORY: conversion warps hold their codes as m16n8k16 fragments already, one tcgen05.st.16x128b.x8 a
//     warp and stage puts 16 columns x 64 inputs in place.  With A in shared memory (the first version: one block, 128 x 256
//     tiles) a stage moved 105 KB through a port of 128 bytes a cycle, 823 cycles for 512 cycles of math; now it moves
//     33 KB for 384 cycles of math;
//   * the pair halves the bytes of x each SM brings in and reads;
//   * two accumulators of 192 columns alternate between tiles (384 of the 512 tensor-memory columns; two 64-column stages of
//     A take the rest, four beside accumulators of 128), so a tile's drain runs under the next tile's math;
//   * N is chosen per call, or per expert, so that tiles fill the SM pairs in whole waves (see pf_rows).
//
// The kernel is persistent: tiles are dealt round-robin to at most one cluster an SM pair, and every producer runs on into
// the next tile.  Rings: packed units (bulk copies, one super-block a block), x (tensor-map boxes), A stages.  Roles of a block: warp 0 loads x, warp 1 owns tensor memory and, in the first block of the pair,
// issues the MMAs, warp 2 loads packed units, warps 4-19 are two groups of eight conversion warps that take alternate
// stages, warps 20-27 drain the finished accumulator.  Barriers the MMA warp waits on live in the first block; the second
// block's copies and conversion warps signal them across the pair.
// Measured, one projection by CUDA events from a graph (in brackets in us: one block a tile with A in shared memory): 2048 rows,
// 17408 x 5120 240 us = 1522 TFLOP/s (335), 5120 x 17408 238 us (402), 1024 x 5120 20 us (53); 391 rows, 17408 x 5120 54 us
// (90); 64 rows, 6144 x 5120 17 us (45).  The tensor pipe is active in 92 % of the cycles of the first of these.  cuBLAS does
// 8192^3 in bf16 at 1696 TFLOP/s here, 1427 over seconds: both are bound by power.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <mutex>

#include "../../include/tensorfold_b200.h"
#include "tf_layout.h"
#include "tf_ptx.cuh"

namespace tf {

int fail_moe(int code, const char* msg);
int cuda_fail_moe(cudaError_t e, const char* what);
int* device_error_word();          // tf_api.cu: the current device's error word (null before tf_init)

namespace {

constexpr int PF_COLS = 128;       // output columns of a block (half of the pair's MMA M)
constexpr int PF_ROWS = 192;       // rows of x a tile may hold (MMA N)
constexpr int PF_GROUP_ROWS = 128; // pairs a plan item may hold in the expert form
constexpr int PF_STAGE_K = 128;    // inputs a stage: long enough that barrier traffic stays small beside the conversion
constexpr int PF_XHALF = PF_ROWS / 2 * 128;        // a block's half of the rows, 64 inputs (128 bytes a row)
constexpr int PF_X_BYTES = 2 * PF_XHALF;
constexpr int PF_W_BYTES = 10240;  // packed units of a stage: two g64 units (9216 B) or four g32 units (10240 B)
constexpr int PF_NX = 4;           // stages of x in flight
constexpr int PF_NW = 10;          // packed-unit slots: 90 KB in flight an SM cover HBM's latency when experts stream once
constexpr int PF_A_COLS = 64;      // tensor-memory columns of a stage of A
constexpr int PF_TMEM_COLS = 512;  // two accumulators, then stages of A: two beside 192-column accumulators, four beside 128
constexpr int PF_THREADS = 896;    // 28 warps: x loads, MMA, unit loads, (idle), 2 x 8 conversion, 8 drain
constexpr int PF_CONV0 = 4;        // first conversion warp
constexpr int PF_DRAIN0 = 20;      // first drain warp (multiples of 4: tensor-memory lane groups go by warp % 4)
constexpr int PF_W_OFF = PF_NX * PF_X_BYTES, PF_BAR_OFF = PF_W_OFF + PF_NW * PF_W_BYTES;
constexpr int PF_BARS = 2 * PF_NX + 2 * PF_NW + 4;
constexpr int PF_SMEM = PF_BAR_OFF + PF_BARS * 8 + 16 + 1024 /* alignment slack */;
static_assert(2 * PF_ROWS + 2 * PF_A_COLS <= PF_TMEM_COLS && 2 * 128 + 4 * PF_A_COLS <= PF_TMEM_COLS, "tensor memory");
static_assert(PF_XHALF % 1024 == 0, "x tiles stay 1024-byte aligned for the 128-byte swizzle");
static_assert(PF_NX == 4, "a stage of A (two or four of them) is released by the barrier of its x stage");
static_assert(PF_SMEM <= 232448, "fits the opt-in shared memory of a block");

struct PrefillParams {
  const uint32_t* w;
  int64_t sb_stride;
  int N, K, M;
  int rows;                   // rows of a tile (a multiple of 16, at most PF_ROWS); the x map's boxes hold half of them
  int acc_cols;               // columns of an accumulator: 128 or 192, at least `rows`
  void* out;
  int64_t ldo;
  int out_f32;
  int* err;
  // grouped form (items != null): a tile is plan item (expert, first, count <= rows) x 256 columns; row r of it is row
  // first + r of x, which holds the rows in member order, and of out, or with members row members[first + r] of out
  const int* items;
  const int* counts;
  const int* members;
  int64_t expert_stride;
  int experts;                // experts the table holds (grouped form)
  int epi;                    // 0 store, 1 relu^2, 2 SwiGLU over gate/up rows interleaved in tiles of 16 (out: N / 2 columns)
  float limit;
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// After a wait that gave up: copies in flight land before the shared memory is released.
__device__ __forceinline__ void let_copies_land() {
  for (int i = 0; i < 64; ++i) __nanosleep(20000);
}

__device__ __forceinline__ float pf_bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float pf_swiglu(float g, float u, float limit) {
  float gv = pf_bf16r(g), uv = pf_bf16r(u);
  if (limit > 0.f) {
    gv = fminf(gv, limit);
    uv = fminf(fmaxf(uv, -limit), limit);
  }
  return pf_bf16r(gv / (1.f + expf(-gv))) * uv;
}

__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_byte_addr) {
  // K-major, 128-byte swizzle: rows 128 B apart inside an 8-row atom, atoms 1024 B apart (SBO), LBO unused (1),
  // descriptor version 1, layout type 2 (SWIZZLE_128B)
  const uint32_t lo = ((smem_byte_addr >> 4) & 0x3FFFu) | (1u << 16);
  const uint32_t hi = 64u | (1u << 14) | (2u << 29);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}

// One 16-input step of a stage: A [256 x 16] from tensor memory (128 lanes of each block), B [N x 16] from both blocks'
// shared memory.  Issued by one thread.
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrives on the barrier at this address in both blocks of the pair once every MMA issued so far is done.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}

// Bounded wait by a whole warp.  The polling loop stays out of line: the roles' loops share the
// instruction caches, and a role that misses there waits hundreds of cycles for a handful of instructions.
__device__ __noinline__ bool poll(uint32_t bar, uint32_t parity, const volatile int* abort_flag) {
#pragma unroll 1
  for (uint32_t i = 0; i < WAIT_POLLS; ++i) {
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity), "r"(20000u)
                 : "memory");
    if (done) return true;
    if ((i & 255u) == 255u && *abort_flag) return false;
  }
  return false;
}
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, const volatile int* abort_flag) {
  if (__all_sync(0xFFFFFFFFu, mbar32_try_wait(bar, parity))) return true;
  return __all_sync(0xFFFFFFFFu, poll(bar, parity, abort_flag));
}

// Sixteen columns of output x 64 inputs: register 4 s + j of a lane is its A-fragment register j of 16-input step s.
__device__ __forceinline__ void tmem_store_a(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// True in one lane of the warp.
__device__ __forceinline__ bool elect() {
  uint32_t one;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xFFFFFFFF;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(one));
  return one != 0;
}

// The address of a barrier in the first block of the pair.
__device__ __forceinline__ uint32_t in_first(const void* p) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"(smem_addr(p)));
  return remote;
}
__device__ __forceinline__ void arrive_first(uint32_t remote) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}
// Tensor-map copies into this block's shared memory that complete on a barrier of the first block.
__device__ __forceinline__ void pair_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
               "l"(map), "r"(bar), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tmem_load16(uint32_t taddr, float (&v)[2][8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=f"(v[0][0]), "=f"(v[0][1]), "=f"(v[0][2]), "=f"(v[0][3]), "=f"(v[0][4]), "=f"(v[0][5]), "=f"(v[0][6]), "=f"(v[0][7]),
        "=f"(v[1][0]), "=f"(v[1][1]), "=f"(v[1][2]), "=f"(v[1][3]), "=f"(v[1][4]), "=f"(v[1][5]), "=f"(v[1][6]), "=f"(v[1][7])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Eight lanes each hold eight rows of one column; afterwards each holds eight columns of one row, as bf16: lane l of the
// group gets row l.  Rows are rounded and paired first, so three exchanges of two words do it.
__device__ __forceinline__ uint4 transpose8(const float (&v)[8], int lane) {
  uint32_t p[4];                                             // rows 2 i, 2 i + 1 of this lane's column
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    p[i] = *reinterpret_cast<const uint32_t*>(&t);
  }
  // neighbouring columns: an even lane keeps rows 2 i of both, an odd lane rows 2 i + 1
  const bool odd = lane & 1;
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    const uint32_t got = __shfl_xor_sync(0xFFFFFFFFu, __byte_perm(p[i], p[i + 1], odd ? 0x5410 : 0x7632), 1);
    p[i] = odd ? __byte_perm(got, p[i], 0x7610) : __byte_perm(p[i], got, 0x5410);
    p[i + 1] = odd ? __byte_perm(got, p[i + 1], 0x7632) : __byte_perm(p[i + 1], got, 0x7610);
  }
  // then a 4 x 4 transpose of (column pair, row pair) words over the other two lane bits
#pragma unroll
  for (int bit = 1; bit <= 2; bit <<= 1) {
    const bool upper = lane & (2 * bit);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i & bit) continue;
      const uint32_t got = __shfl_xor_sync(0xFFFFFFFFu, upper ? p[i] : p[i | bit], 2 * bit);
      if (upper) p[i] = got;
      else p[i | bit] = got;
    }
  }
  return make_uint4(p[0], p[1], p[2], p[3]);
}

template <int GS>
__global__ void __launch_bounds__(PF_THREADS, 1) prefill_kernel(const __grid_constant__ CUtensorMap tmx, const PrefillParams p) {
  constexpr int S = GS / 16;                                 // k16 steps a group
  constexpr int UNITS = PF_STAGE_K / GS;                     // units a stage (2 for g64, 4 for g32)
  constexpr int WPL = words_per_lane(4, GS);
  constexpr int UNITW = unit_words(4, GS);
  static_assert(UNITS * UNITW * 4 <= PF_W_BYTES, "slot holds a stage's packed units");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + PF_BAR_OFF);     // first block: the pair's rows of x have landed and its 16
                                                    // conversion warps have stored their A
  uint64_t* empty = full + PF_NX;                   // the MMAs that read the stage (x and A) are done
  uint64_t* w_full = empty + PF_NX;                 // packed units landed (bulk copy)
  uint64_t* w_empty = w_full + PF_NW;               // the 8 conversion warps of the stage's group have read the slot
  uint64_t* acc_full = w_empty + PF_NW;             // [2] every MMA of a tile is done
  uint64_t* acc_empty = acc_full + 2;               // [2] first block: the 16 drain warps of the pair have read the accumulator
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
  const int half = blockIdx.x & 1, pair_id = blockIdx.x >> 1, pairs_in_grid = gridDim.x >> 1;     // (clusters are blocks 2 i, 2 i + 1)
  const int nstages = (p.K + PF_STAGE_K - 1) / PF_STAGE_K;
  const int total_units = p.K / GS;
  const int nsb = (p.N + PF_COLS - 1) / PF_COLS, ncp = (nsb + 1) / 2;
  const bool grouped = p.items != nullptr;
  const int a_stages = p.acc_cols > 128 ? 2 : 4;
  const uint32_t a_col0 = 2 * p.acc_cols;

  auto give_up = [&](int code) {
    if (lane == 0) {
      *abort_flag = code;
      atomicCAS(p.err, 0, code);
    }
  };

  if (tid == 0) {
    for (int i = 0; i < PF_NX; ++i) mbar_init(full + i, 17), mbar_init(empty + i, 1);
    for (int i = 0; i < PF_NW; ++i) mbar_init(w_full + i, 1), mbar_init(w_empty + i, 8);
    for (int i = 0; i < 2; ++i) mbar_init(acc_full + i, 1), mbar_init(acc_empty + i, 16);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(PF_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();                                            // the pair's barriers exist before either block signals the other
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();

  // Tiles = pairs of column blocks x row tiles (plan items in the grouped form), columns fastest, dealt round-robin to the
  // clusters.  Every role of both blocks walks the same (tile, stage) sequence, so a running stage count g names the ring
  // slots and their phases without any exchange between the roles.
  if (grouped) pdl_wait();                                   // the plan may be the previous kernel's output
  const int row_tiles = grouped ? p.counts[0] : (p.M + p.rows - 1) / p.rows;
  const int tiles = ncp * row_tiles;
  const int my_tiles = pair_id < tiles ? (tiles - pair_id + pairs_in_grid - 1) / pairs_in_grid : 0;
  const int total = my_tiles * nstages;                      // stages this block runs

  struct Tile {
    int sb;                                                  // this block's super-block (past the last one: nothing is stored)
    int m0, rows_here, n;                                    // first row (of members in the grouped form), rows, MMA N
    const uint32_t* w;                                       // this block's units
  };
  auto tile_at = [&](int it) {
    const int t = pair_id + it * pairs_in_grid;
    const int y = t / ncp;
    Tile ti;
    ti.sb = 2 * (t - y * ncp) + half;
    ti.w = p.w + static_cast<int64_t>(min(ti.sb, nsb - 1)) * p.sb_stride;
    if (grouped) {
      const int* item = p.items + 3 * y;
      // an item that names an expert outside the table runs against expert 0 with no rows (nothing is stored) and is
      // reported: every role still walks the same tile sequence, and nothing is read past the table
      const int expert = __ldg(item);
      const bool known = expert >= 0 && expert < p.experts;
      if (!known && threadIdx.x == 0) atomicCAS(p.err, 0, ERR_BAD_ITEM);
      ti.w += static_cast<int64_t>(known ? expert : 0) * p.expert_stride;
      ti.m0 = __ldg(item + 1);
      ti.rows_here = known ? min(p.rows, __ldg(item + 2)) : 0;
    } else {
      ti.m0 = y * p.rows;
      ti.rows_here = min(p.rows, p.M - ti.m0);
    }
    ti.n = max(16, (ti.rows_here + 15) & ~15);
    return ti;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ x tiles (L2 -> shared): this block's half of the rows
    if (!grouped) pdl_wait();                                // x may be the previous kernel's output
    bool ok = true;
    int slot = 0;
    uint32_t phase = 1;                                      // parity of the `empty` phase that frees the slot (first round: passes)
    const uint32_t bytes = p.rows * 128;                     // both blocks' copies of 64 inputs
    const uint32_t full0 = in_first(full), full32 = smem_addr(full), empty32 = smem_addr(empty), smem32 = smem_addr(smem);
    for (int it = 0; it < my_tiles && ok; ++it) {
      const Tile ti = tile_at(it);
      const int y = ti.m0 + half * (ti.n / 2);               // (a box may reach past the share: those rows are not multiplied)
#pragma unroll 1
      for (int ls = 0; ls < nstages; ++ls) {
        ok = warp_wait(empty32 + 8 * slot, phase, abort_flag);
        if (!ok) break;
        const uint32_t bar = full0 + 8 * slot, dst = smem32 + slot * PF_X_BYTES;
        const int k0 = ls * PF_STAGE_K;
        const bool both = p.K - k0 > 64;
        if (elect()) {
          if (half == 0) mbar32_expect_tx(full32 + 8 * slot, both ? 2 * bytes : bytes);
          pair_load_2d(dst, &tmx, k0, y, bar);
          if (both) pair_load_2d(dst + PF_XHALF, &tmx, k0 + 64, y, bar);
        }
        __syncwarp();
        if (++slot == PF_NX) slot = 0, phase ^= 1u;
      }
    }
    if (!ok) give_up(ERR_WAIT_EMPTY);
    if (!ok) let_copies_land();
  } else if (warp == 2) {
    // ------------------------------------------------------------------ packed units (HBM -> shared, bulk copies)
    // The units may be the previous kernel's output too.  The wait costs 0.35 to 0.5 us a launch (a layer of 1984 hidden at 744
    // rows, seven launches, 119 -> 123 us); bringing the first units to L2 before it gained nothing.
    if (!grouped) pdl_wait();
    bool ok = true;
    int slot = 0;
    uint32_t phase = 1;
    const uint32_t w_full32 = smem_addr(w_full), w_empty32 = smem_addr(w_empty), smem32 = smem_addr(smem + PF_W_OFF);
    for (int it = 0; it < my_tiles && ok; ++it) {
      const uint32_t* w = tile_at(it).w;
#pragma unroll 1
      for (int ls = 0; ls < nstages; ++ls, w += UNITS * UNITW) {
        ok = warp_wait(w_empty32 + 8 * slot, phase, abort_flag);
        if (!ok) break;
        const uint32_t bytes = min(UNITS, total_units - ls * UNITS) * UNITW * 4;
        if (elect()) {
          mbar32_expect_tx(w_full32 + 8 * slot, bytes);
          bulk_load32(smem32 + slot * PF_W_BYTES, w, bytes, w_full32 + 8 * slot);
        }
        __syncwarp();
        if (++slot == PF_NW) slot = 0, phase ^= 1u;
      }
    }
    if (!ok) give_up(ERR_WAIT_EMPTY);
    if (!ok) let_copies_land();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issue (one thread of the first block)
    if (half == 0) {
      // The tensor pipe's queue is short, so this warp must stay ahead of it: one barrier a stage, eight MMAs a barrier,
      // and addresses that are the same in every lane (elect.sync lets the compiler keep them in uniform registers, which it
      // does not do in a loop behind `lane == 0`).
      const uint32_t full32 = smem_addr(full), empty32 = smem_addr(empty), acc_full32 = smem_addr(acc_full);
      const uint64_t bd0 = umma_desc(smem_addr(smem));
      const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, tmem_base, 0);
      const int whole = p.K / PF_STAGE_K;                      // stages of 128 inputs; K may end with half of one
      bool ok = true;
      int slot = 0;
      uint32_t phase = 0, a_slot = 0;
      for (int it = 0; it < my_tiles && ok; ++it) {
        const uint32_t n8 = __shfl_sync(0xFFFFFFFFu, static_cast<uint32_t>(tile_at(it).n >> 3), 0);
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (n8 << 17) | ((256u >> 4) << 24);
        const uint32_t acc = tmem + static_cast<uint32_t>((it & 1) * p.acc_cols);
        // the accumulator's last tile must have been drained
        if (it >= 2) ok = warp_wait(smem_addr(acc_empty + (it & 1)), ((it >> 1) - 1) & 1, abort_flag);
#pragma unroll 1
        for (int ls = 0; ls < nstages && ok; ++ls) {
          ok = warp_wait(full32 + 8 * slot, phase, abort_flag);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a = tmem + a_col0 + a_slot * PF_A_COLS;
          const uint64_t bd = bd0 + slot * (PF_X_BYTES >> 4);
          if (elect()) {
            umma_pair(acc, a, bd, idesc, ls != 0 ? 1u : 0u);   // 16 inputs: 8 columns of A, 32 bytes inside the swizzle atom
#pragma unroll
            for (int q = 1; q < 4; ++q) umma_pair(acc, a + 8 * q, bd + 2 * q, idesc, 1u);
            if (ls < whole || p.K % PF_STAGE_K > 64) {
#pragma unroll
              for (int q = 0; q < 4; ++q) umma_pair(acc, a + 32 + 8 * q, bd + (PF_XHALF >> 4) + 2 * q, idesc, 1u);
            }
            umma_commit_pair(empty32 + 8 * slot);
            if (ls == nstages - 1) umma_commit_pair(acc_full32 + 8 * (it & 1));
          }
          __syncwarp();
          a_slot = (a_slot + 1) & (a_stages - 1);
          if (++slot == PF_NX) slot = 0, phase ^= 1u;
        }
      }
      if (!ok) give_up(ERR_WAIT_FULL);
    }
  } else if (warp >= PF_CONV0 && warp < PF_DRAIN0) {
    // ------------------------------------------------------------------ conversion: packed codes -> bf16 A stage in tensor memory
    // A warp owns 16 output columns (tile pair tp, half h) of every stage its group takes; its lanes hold the codes as
    // A fragments, which is how tcgen05.st.16x128b lays them down (lane = output column, 32-bit column = two inputs).
    const int cw = warp - PF_CONV0, group = cw >> 3, dw = cw & 7, tp = dw & 3, h = dw >> 2, g8 = lane >> 2;
    const __nv_bfloat162 k128 = __floats2bfloat162_rn(128.f, 128.f);
    const uint32_t a_lane = tmem_base + (static_cast<uint32_t>(32 * tp + 16 * h) << 16) + a_col0;
    const uint32_t full0 = in_first(full);
    const uint32_t w_off = smem_addr(smem + PF_W_OFF) + ((tp * 32 + lane) * WPL + h * S) * 4;
    const uint32_t sb_off = smem_addr(smem + PF_W_OFF) + (TILE_PAIRS * 32 * WPL + tp * 32 + g8 * 4 + h * 2) * 4;
    bool ok = true;
    int sw = group, ls = group % nstages;
    uint32_t pw = 0;
    for (int i = group; i < total; i += 2) {                   // i = the block's running stage count
      ok = warp_wait(smem_addr(w_full + sw), pw, abort_flag);
      if (!ok) {
        give_up(ERR_WAIT_FULL);
        break;
      }
      const int units_here = total_units - ls * UNITS;         // (of UNITS: K may end inside the stage)
      uint32_t frag[2][16];
#pragma unroll
      for (int u = 0; u < UNITS; ++u) {
        const uint32_t at = sw * PF_W_BYTES + u * UNITW * 4;
        uint32_t wd[S];
        if constexpr (S == 4) {
          const uint4 v = lds128(w_off + at);
          wd[0] = v.x, wd[1] = v.y, wd[2] = v.z, wd[3] = v.w;
        } else {
          const uint2 v = lds64(w_off + at);
          wd[0] = v.x, wd[1] = v.y;
        }
        uint2 sbw = lds64(sb_off + at);                        // columns g8 and g8 + 8 of the half
        // past the end of K x is zero (the tensor map fills it) and the weights must be finite: scales and biases of
        // zero give zero weights
        if (u > 0 && u >= units_here) sbw = make_uint2(0u, 0u);
        __nv_bfloat162 sc[2], bi[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint32_t v = r == 0 ? sbw.x : sbw.y, s2 = __byte_perm(v, 0u, 0x1010), b2 = __byte_perm(v, 0u, 0x3232);
          sc[r] = *reinterpret_cast<const __nv_bfloat162*>(&s2);
          bi[r] = *reinterpret_cast<const __nv_bfloat162*>(&b2);
        }
#pragma unroll
        for (int sidx = 0; sidx < S; ++sidx)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t v = lop3_and_or(wd[sidx] >> (4 * j), 0x000F000Fu, 0x43004300u);
            const __nv_bfloat162 q2 = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&v), k128);       // exact code
            const __nv_bfloat162 w2 = __hfma2(q2, sc[j & 1], bi[j & 1]);                            // one rounding
            frag[u * S / 4][(u * S % 4 + sidx) * 4 + j] = *reinterpret_cast<const uint32_t*>(&w2);
          }
      }
      __syncwarp();
      if (elect()) mbar_arrive(w_empty + sw);                // the slot's words are in registers
      if (i >= a_stages) {                                     // the MMAs that read the A stage's last contents are done
        const int before = i - a_stages;
        ok = warp_wait(smem_addr(empty + before % PF_NX), (before / PF_NX) & 1, abort_flag);
        if (!ok) {
          give_up(ERR_WAIT_EMPTY);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      const uint32_t a = a_lane + (i & (a_stages - 1)) * PF_A_COLS;
      tmem_store_a(a, frag[0]);
      if (units_here * GS > 64) tmem_store_a(a + 32, frag[1]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (elect()) arrive_first(full0 + 8 * (i % PF_NX));
      sw += 2;
      if (sw >= PF_NW) sw -= PF_NW, pw ^= 1u;
      ls += 2;
      while (ls >= nstages) ls -= nstages;
    }
  } else if (warp >= PF_DRAIN0) {
    // ------------------------------------------------------------------ drain: tensor memory -> global, a tile behind
    if (!grouped) pdl_wait();                                  // nothing is written before the previous kernel is done
    const int lg = warp & 3, part = (warp - PF_DRAIN0) >> 2;   // this warp may touch TMEM lanes [32 lg, 32 lg + 32)
    const uint32_t acc_empty0 = in_first(acc_empty);
    for (int it = 0; it < my_tiles; ++it) {
      const Tile ti = tile_at(it);
      const int ab = it & 1, rows_here = ti.rows_here, m0 = ti.m0, sb = ti.sb;
      const bool done = warp_wait(smem_addr(acc_full + ab), (it >> 1) & 1, abort_flag);
      if (!done) {
        give_up(ERR_WAIT_FULL);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (*abort_flag != 0) break;
      // Sixteen rows of x a pass, passes in turn between the two warps of a lane group.  A lane holds its output column for
      // them; each group of eight lanes transposes 8 x 8 blocks in registers, so that a lane writes eight neighbouring
      // columns of one row as 16 bytes.
      const bool swiglu = p.epi == 2;
      const int col = swiglu ? sb * (PF_COLS / 2) + lg * 16 + (lane & 15) : sb * PF_COLS + lg * 32 + lane;
      const int ncols = swiglu ? p.N / 2 : p.N;
      const bool live = sb < nsb && col < ncols;
      const bool wide = !p.out_f32 && (ncols & 7) == 0 && (p.ldo & 7) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
      const uint32_t acc = tmem_base + (static_cast<uint32_t>(lg * 32) << 16) + static_cast<uint32_t>(ab * p.acc_cols);
      // v[j] = output column `col` of row rr + j
      auto store8 = [&](const float (&v)[8], int rr) {
        if (wide) {
          const uint4 o = transpose8(v, lane);                 // columns col - l8 .. col - l8 + 7 of row rr + l8
          const int r = rr + (lane & 7);
          if (live && r < rows_here) {
            const int64_t m = p.members != nullptr ? p.members[m0 + r] : m0 + r;
            *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.out) + m * p.ldo + (col - (lane & 7))) = o;
          }
        } else if (live) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (rr + j < rows_here) {
              const int64_t m = p.members != nullptr ? p.members[m0 + rr + j] : m0 + rr + j;
              if (p.out_f32) reinterpret_cast<float*>(p.out)[m * p.ldo + col] = v[j];
              else reinterpret_cast<__nv_bfloat16*>(p.out)[m * p.ldo + col] = __float2bfloat16_rn(v[j]);
            }
          }
        }
      };
#pragma unroll 1
      for (int r0 = 16 * part; r0 < rows_here; r0 += 32) {
        float v[2][8];
        tmem_load16(acc + r0, v);
        if (swiglu) {
          // lanes 0-15 hold gate columns, 16-31 the up columns of the same outputs: lanes below 16 take rows 0-7 of the
          // pass, the others rows 8-15
          const bool low = lane < 16;
          float w[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float got = __shfl_xor_sync(0xFFFFFFFFu, low ? v[1][j] : v[0][j], 16);
            w[j] = pf_swiglu(low ? v[0][j] : got, low ? got : v[1][j], p.limit);
          }
          store8(w, r0 + (low ? 0 : 8));
        } else {
          if (p.epi == 1) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float u = fmaxf(pf_bf16r(v[j >> 3][j & 7]), 0.f);
              v[j >> 3][j & 7] = u * u;
            }
          }
          store8(v[0], r0);
          if (r0 + 8 < rows_here) store8(v[1], r0 + 8);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) arrive_first(acc_empty0 + 8 * ab);
    }
  }

  // Neither block leaves (its tensor memory, shared memory and barriers stay in use) before both are done.
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(PF_TMEM_COLS) : "memory");
  }
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
  static EncodeTiled fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(sym);
  });
  return fn;
}

}  // namespace

namespace {

int g_pairs[64] = {};              // clusters of the prefill kernel a device runs at once (set by prefill_configure)

template <int GS>
cudaError_t launch_pairs(const CUtensorMap& map, const PrefillParams& p, int clusters, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * clusters);
  cfg.blockDim = dim3(PF_THREADS);
  cfg.dynamicSmemBytes = PF_SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = 2, attrs[0].val.clusterDim.y = 1, attrs[0].val.clusterDim.z = 1;
  // the next kernel's blocks may take an SM as soon as this one's last wave leaves it and set up there; they read and write
  // global memory, weights among it, only once this one is done (the caller is not asked whether they are settled)
  attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, prefill_kernel<GS>, map, p);
}

template <int GS>
cudaError_t configure_pairs(int* clusters) {
  cudaError_t e = cudaFuncSetAttribute(prefill_kernel<GS>, cudaFuncAttributeMaxDynamicSharedMemorySize, PF_SMEM);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2);
  cfg.blockDim = dim3(PF_THREADS);
  cfg.dynamicSmemBytes = PF_SMEM;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2, attr.val.clusterDim.y = 1, attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaOccupancyMaxActiveClusters(clusters, prefill_kernel<GS>, &cfg);
}

// Rows of a tile for an (n, m) call: the fewest cycles, waves of tiles times a tile's pace.  A stage of 64 inputs takes
// 2 rows cycles of math, but no less than the conversion of its weights (PF_CONVERT cycles); ties go to the larger tile,
// which converts the weights fewer times.
constexpr int PF_CONVERT = 240;
int pf_rows(int n, int m, int clusters) {
  const int64_t ncp = (n + 2 * PF_COLS - 1) / (2 * PF_COLS);
  int best = 16;
  int64_t cost = INT64_MAX;
  for (int rows = 16; rows <= PF_ROWS; rows += 16) {
    const int64_t waves = (ncp * ((m + rows - 1) / rows) + clusters - 1) / clusters;
    const int64_t c = waves * (2 * rows > PF_CONVERT ? 2 * rows : PF_CONVERT);
    if (c <= cost) cost = c, best = rows;
  }
  return best;
}

int resident_pairs() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  return g_pairs[dev];
}

}  // namespace

cudaError_t prefill_configure(int device) {
  int a = 0, b = 0;
  cudaError_t e = configure_pairs<64>(&a);
  if (e == cudaSuccess) e = configure_pairs<32>(&b);
  if (e == cudaSuccess && (a < 1 || b < 1)) e = cudaErrorLaunchOutOfResources;
  if (e == cudaSuccess && device >= 0 && device < 64) g_pairs[device] = a < b ? a : b;
  return e;
}

int encode_rows(CUtensorMap* map, const void* x, int64_t ldx, int rows, int k, int box_rows) {
  EncodeTiled encode = encode_fn();
  if (encode == nullptr) return fail_moe(TF_ERR_UNSUPPORTED, "prefill: the driver does not export cuTensorMapEncodeTiled");
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ldx) * 2};
  const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? TF_OK : fail_moe(TF_ERR_ARG, "prefill: cuTensorMapEncodeTiled refused the input tensor");
}

}  // namespace tf

using namespace tf;

extern "C" int tf_qmm_prefill_act(const void* x, int64_t ldx, int m, const void* tiled, int64_t sb_stride, int n, int k, int gs,
                                  void* out, int64_t ldo, int out_f32, int epi, float limit, void* stream);

extern "C" int tf_qmm_prefill(const void* x, int64_t ldx, int m, const void* tiled, int64_t sb_stride, int n, int k, int gs,
                              void* out, int64_t ldo, int out_f32, void* stream) {
  return tf_qmm_prefill_act(x, ldx, m, tiled, sb_stride, n, k, gs, out, ldo, out_f32, 0, 0.f, stream);
}

extern "C" int tf_qmm_prefill_act(const void* x, int64_t ldx, int m, const void* tiled, int64_t sb_stride, int n, int k, int gs,
                                  void* out, int64_t ldo, int out_f32, int epi, float limit, void* stream) {
  if (gs != 32 && gs != 64) return fail_moe(TF_ERR_UNSUPPORTED, "tf_qmm_prefill: 4-bit weights with groups of 32 or 64");
  if (m < 1 || n < 1 || k < gs || k % gs) return fail_moe(TF_ERR_ARG, "tf_qmm_prefill: K must be a positive multiple of the group");
  if (epi < 0 || epi > 2 || (epi == 2 && n % 32) || (epi != 0 && out_f32)) return fail_moe(TF_ERR_ARG, "tf_qmm_prefill: bad epilogue");
  if (!x || !tiled || !out || ldo < (epi == 2 ? n / 2 : n) || ldx < k) return fail_moe(TF_ERR_ARG, "tf_qmm_prefill: null pointer or short rows");
  if (reinterpret_cast<uintptr_t>(x) % 16 || ldx % 8) return fail_moe(TF_ERR_ALIGN, "tf_qmm_prefill: x rows must start on 16-byte boundaries");
  if (reinterpret_cast<uintptr_t>(tiled) % 16) return fail_moe(TF_ERR_ALIGN, "tf_qmm_prefill: tiled weights must be 16-byte aligned");
  int* err = device_error_word();
  if (err == nullptr) return fail_moe(TF_ERR_STATE, "tf_qmm_prefill: tf_init has not been called for the current device");
  const int clusters = resident_pairs();
  if (clusters < 1) return fail_moe(TF_ERR_STATE, "tf_qmm_prefill: tf_init has not been called for the current device");
  PrefillParams p = {};
  p.rows = pf_rows(n, m, clusters);
  p.acc_cols = p.rows > 128 ? 192 : 128;
  CUtensorMap map;
  if (int rc = encode_rows(&map, x, ldx, m, k, p.rows / 2)) return rc;
  p.w = static_cast<const uint32_t*>(tiled);
  p.sb_stride = sb_stride > 0 ? sb_stride : static_cast<int64_t>(k / gs) * unit_words(4, gs);
  p.N = n, p.K = k, p.M = m;
  p.out = out, p.ldo = ldo, p.out_f32 = out_f32;
  p.err = err;
  p.epi = epi, p.limit = limit;
  const int64_t tiles = static_cast<int64_t>((n + 2 * PF_COLS - 1) / (2 * PF_COLS)) * ((m + p.rows - 1) / p.rows);
  if (tiles > (1 << 24)) return fail_moe(TF_ERR_ARG, "tf_qmm_prefill: too many tiles");
  const int grid = static_cast<int>(tiles < clusters ? tiles : clusters);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = gs == 64 ? launch_pairs<64>(map, p, grid, s) : launch_pairs<32>(map, p, grid, s);
  return e == cudaSuccess ? TF_OK : cuda_fail_moe(e, "tf_qmm_prefill");
}

namespace tf {
namespace {

// dst[pos, :] = src[row(members[pos]), :] for every planned pair: the rows of a grouped call in member order, so an item's
// rows are contiguous.  A warp a row, four 16-byte copies in flight a lane: bound by the writes (66 MB for 12288 pairs of
// 2688: 14 us).  Fetching the rows inside the matmul with gather copies of four rows was slower by far (a copy that is
// not the same in every lane costs about 100 cycles to issue, 25 of them a stage).
__global__ void __launch_bounds__(256) gather_rows_kernel(const __nv_bfloat16* __restrict__ src, int64_t ld, const int* __restrict__ items,
                                                          const int* __restrict__ counts, const int* __restrict__ members, int slots,
                                                          int pairs, int k, __nv_bfloat16* __restrict__ dst) {
  const int lane = threadIdx.x & 31, pos = blockIdx.x * 8 + (threadIdx.x >> 5);
  // members past the items hold no pair; a plan may list its items in any order
  __shared__ int ends[8];
  int end = 0;
  for (int i = threadIdx.x, n = counts[0]; i < n; i += 256) end = max(end, items[3 * i + 1] + items[3 * i + 2]);
  end = __reduce_max_sync(0xFFFFFFFFu, end);
  if (lane == 0) ends[threadIdx.x >> 5] = end;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) end = max(end, ends[w]);
  if (pos >= min(pairs, end)) return;
  const int pair = members[pos];
  if (pair < 0 || pair >= pairs) return;
  const int64_t row = slots > 0 ? pair / slots : pair;
  const uint4* s4 = reinterpret_cast<const uint4*>(src + row * ld);
  uint4* d4 = reinterpret_cast<uint4*>(dst + static_cast<int64_t>(pos) * k);
  const int chunks = k / 8;
  for (int i = lane; i < chunks; i += 128) {
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i + 32 * j < chunks) v[j] = s4[i + 32 * j];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i + 32 * j < chunks) d4[i + 32 * j] = v[j];
  }
}

}  // namespace
}  // namespace tf

extern "C" int tf_moe_gather(const void* x, int64_t ldx, int slots, const int* items, const int* counts, const int* members, int pairs,
                             int k, void* sorted, void* stream) {
  if (!x || !items || !counts || !members || !sorted || slots < 0 || pairs < 1 || k < 8 || k % 8 || ldx < k)
    return fail_moe(TF_ERR_ARG, "tf_moe_gather: null pointer or bad sizes");
  if (reinterpret_cast<uintptr_t>(x) % 16 || ldx % 8 || reinterpret_cast<uintptr_t>(sorted) % 16)
    return fail_moe(TF_ERR_ALIGN, "tf_moe_gather: rows must start on 16-byte boundaries");
  gather_rows_kernel<<<(pairs + 7) / 8, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), ldx, items, counts, members, slots, pairs, k, static_cast<__nv_bfloat16*>(sorted));
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TF_OK : cuda_fail_moe(e, "tf_moe_gather");
}

extern "C" int tf_moe_experts_sorted(const void* sorted, int64_t ldx, const void* tiled, int64_t expert_stride, int experts, int n, int k,
                                     int gs, const int* items, const int* counts, const int* members, int pairs, int max_items, void* out,
                                     int64_t ldo, int out_f32, int epi, float limit, void* stream) {
  if (experts < 1) return fail_moe(TF_ERR_ARG, "tf_moe_experts_prefill: the table holds at least one expert");
  if (gs != 32 && gs != 64) return fail_moe(TF_ERR_UNSUPPORTED, "tf_moe_experts_prefill: 4-bit weights with groups of 32 or 64");
  if (n < 1 || k < gs || k % gs || k % 8 || pairs < 1 || max_items < 1 || max_items > 65535)
    return fail_moe(TF_ERR_ARG, "tf_moe_experts_prefill: bad sizes");
  if (epi < 0 || epi > 2 || (epi == 2 && n % 32) || (epi != 0 && out_f32)) return fail_moe(TF_ERR_ARG, "tf_moe_experts_prefill: bad epilogue");
  if (!sorted || !tiled || !items || !counts || !out || ldo < (epi == 2 ? n / 2 : n) || ldx < k)
    return fail_moe(TF_ERR_ARG, "tf_moe_experts_prefill: null pointer or short rows");
  if (reinterpret_cast<uintptr_t>(sorted) % 16 || ldx % 8 || reinterpret_cast<uintptr_t>(tiled) % 16)
    return fail_moe(TF_ERR_ALIGN, "tf_moe_experts_prefill: rows and units must start on 16-byte boundaries");
  int* err = device_error_word();
  const int clusters = resident_pairs();
  if (err == nullptr || clusters < 1) return fail_moe(TF_ERR_STATE, "tf_moe_experts_prefill: tf_init has not been called for the current device");
  CUtensorMap map;
  if (int rc = encode_rows(&map, sorted, ldx, pairs, k, PF_GROUP_ROWS / 2)) return rc;
  PrefillParams p = {};
  p.w = static_cast<const uint32_t*>(tiled);
  p.sb_stride = static_cast<int64_t>(k / gs) * unit_words(4, gs);
  p.N = n, p.K = k, p.M = pairs;
  p.rows = p.acc_cols = PF_GROUP_ROWS;
  p.out = out, p.ldo = ldo, p.out_f32 = out_f32;
  p.err = err;
  p.items = items, p.counts = counts, p.members = members;
  p.expert_stride = expert_stride;
  p.experts = experts;
  p.epi = epi, p.limit = limit;
  const int64_t tiles = static_cast<int64_t>((n + 2 * PF_COLS - 1) / (2 * PF_COLS)) * max_items;   // upper bound: the plan says how many
  const int grid = static_cast<int>(tiles < clusters ? tiles : clusters);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = gs == 64 ? launch_pairs<64>(map, p, grid, s) : launch_pairs<32>(map, p, grid, s);
  return e == cudaSuccess ? TF_OK : cuda_fail_moe(e, "tf_moe_experts_prefill");
}

extern "C" int tf_moe_experts_prefill(const void* x, int64_t ldx, int slots, const void* tiled, int64_t expert_stride,
                                      int experts, int n, int k, int gs, const int* items, const int* counts,
                                      const int* members, int pairs, int max_items, void* sorted, void* out, int64_t ldo,
                                      int out_f32, int epi, float limit, void* stream) {
  if (!members) return fail_moe(TF_ERR_ARG, "tf_moe_experts_prefill: null pointer");
  if (int rc = tf_moe_gather(x, ldx, slots, items, counts, members, pairs, k, sorted, stream)) return rc;
  return tf_moe_experts_sorted(sorted, k, tiled, expert_stride, experts, n, k, gs, items, counts, members, pairs, max_items, out, ldo,
                               out_f32, epi, limit, stream);
}
