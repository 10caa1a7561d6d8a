// Row-exact affine matmul for 17 and more rows (batched verify windows) on the 5th-generation tensor cores.
//
// The arithmetic is qmm_tiled.cuh's, bit for bit: per K slice and per group in order, P' = sum of x * (q + C) as one chain
// of 16-input MMA steps from zero, acc = fma(xs, b - C s, fma(P', s, acc)); slices added in slice order; one rounding.
// (tcgen05.mma with K = 16 accumulates a step exactly as mma.sync.m16n8k16 does: the tests demand equal bits.)
//
// What bounds the tiled kernel there is mma.sync and the conversion it repeats for every row tile: a dense layer of 48 rows
// took 365 us for 30 us of weight bytes.  Here the weights are the UMMA A operand (128 output columns), the rows of x the B
// operand (N), and three groups of warps work on different groups of inputs at the same time:
//   * conversion warps turn packed codes into A fragments (q + 128, one three-input logic op a pair) and store them to
//     tensor memory with tcgen05.st.16x128b, whose lane layout is the fragment's;
//   * one warp issues the MMAs of a group into a product buffer P' of N columns (no accumulation across groups: the affine
//     step is per group, in fp32);
//   * epilogue warps (a thread owns one output column and all rows of the tile) read P' back and apply the affine step
//     into registers with packed fp32 fmas.
// A block holds two 128-column super-blocks side by side, which halves the bytes of x it pulls from L2 a weight byte, and
// is persistent: work items (row tile, two super-blocks, K slice) are dealt round-robin and every ring runs on across items.
// Row tiles come first in the item order, so the tiles that share weights run at the same time and find them in L2.  Slices
// meet in global memory as in qmm_stream.cuh: the warp that counts itself in last adds them in slice order.
// Blocks never wait for one another.  `count` is zero before and after every launch.
// What bounds it now is the chain inside a block, not memory and not the tensor pipe (12 % of active cycles at 48 rows): a pair
// of groups (one a super-block) takes about 1200 cycles, at 16 rows nearly as many as at 48 (17408 x 5120 in one slice, 80 pairs
// one after another: 53.2 us at 16 rows, 54.6 at 48, 62.0 at 64), so it is waits and round trips through tensor memory rather
// than the epilogue's arithmetic.  Code is kept short (the slice sum is a loop over sixteen rows), since a first pass over it is
// fetched from L2.
// Measured from graphs, weights past L2, sums given (4 bits, groups of 64; the tiled kernel in brackets): 48 rows, 17408 x 5120
// 37.3 us (66.0), 5120 x 17408 50.0 (77.7), 6144 x 5120 31.9 (38.9), 5120 x 6144 34.2 (44.6); 256 rows, 17408 x 5120 140 us
// (254), 5120 x 17408 227 (305).
#pragma once

#include "qmm_tiled.cuh"

namespace tf {

struct WindowParams {
  const float* xs;            // optional [M, KG] group sums
  const uint32_t* w;
  int64_t sb_stride;
  void* out;                  // [M, N] bf16 or fp32
  int64_t ldo;
  float* part;                // [row tiles][nsb][sk][4][ROWS * 32] slices; unused when sk == 1
  int* count;                 // [row tiles][nsb][4]
  int M, N, KG, sk, nsb;
  int row_tiles, tile_rows;   // rows of a tile: a multiple of 16, at most ROWS
  int items, out_f32;
  int* err;
};

template <int BITS, int GS, int ROWS>
struct WindowGeo {
  static constexpr int THREADS = 640;                       // copy, MMA, 2 sums; 2 x 4 conversion; 2 x 4 epilogue warps
  static constexpr int G = 128 / GS, S = GS / 16;
  static constexpr int WPL = words_per_lane(BITS, GS), UNITW = unit_words(BITS, GS);
  static constexpr int XHALF = ROWS * XHALF_ROW;
  static constexpr int X_OFF = 0, W_OFF = 2 * XHALF;
  static constexpr int W_BYTES = G * UNITW * 4;
  static constexpr int XS_OFF = W_OFF + 2 * W_BYTES;
  static constexpr int STAGE = (XS_OFF + ROWS * G * 4 + 1023) / 1024 * 1024;
  static constexpr int NST_A = 222 * 1024 / STAGE;
  static constexpr int NST = NST_A > 8 ? 8 : NST_A;
  static constexpr int ACOLS = GS / 2;                      // tensor-memory columns of a group of A
  static constexpr int AS = GS == 128 ? 2 : 4;              // A buffers a super-block
  static constexpr int PS = ROWS == 32 ? 4 : 2;             // product buffers a super-block
  static constexpr int P_COL0 = 2 * AS * ACOLS;
  static constexpr int BARS = 3 * NST + 4 * AS + 4 * PS;
  static constexpr int SMEM = NST * STAGE + BARS * 8 + 16 + 1024;
  static_assert(NST >= 3 && SMEM <= 227 * 1024, "fits the shared memory of an SM");
  static_assert(P_COL0 + 2 * PS * ROWS <= 512, "fits tensor memory");
  static_assert(XHALF % 1024 == 0 && W_BYTES % 16 == 0 && XS_OFF % 16 == 0, "stage parts stay aligned");
};

__device__ __forceinline__ uint64_t window_desc(uint32_t addr) {
  // K-major, 128-byte swizzle: rows 128 B apart inside an 8-row atom, atoms 1024 B apart
  const uint32_t lo = ((addr >> 4) & 0x3FFFu) | (1u << 16), hi = 64u | (1u << 14) | (2u << 29);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}
__device__ __forceinline__ void window_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void window_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool window_elect() {
  uint32_t one;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xFFFFFFFF;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(one));
  return one != 0;
}
// Sixteen output columns x 32 inputs: register 4 s + j is A-fragment register j of step s.
__device__ __forceinline__ void window_store_a(uint32_t t, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(t), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void window_load16(uint32_t t, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(t)
      : "memory");
}
// Bounded wait by a whole warp: one quick test, then polls that may suspend in hardware.  (Out of line the loop would be
// shorter still, but a call does not get along with setmaxnreg's register budget.)
__device__ __forceinline__ bool window_poll(uint32_t bar, uint32_t parity, uint32_t abort_word) {
#pragma unroll 1
  for (uint32_t i = 0; i < WAIT_POLLS; ++i) {
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity), "r"(20000u)
                 : "memory");
    if (done) return true;
    if ((i & 255u) == 255u) {
      uint32_t gone;
      asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(gone) : "r"(abort_word));
      if (gone) return false;
    }
  }
  return false;
}
__device__ __forceinline__ bool window_wait(uint32_t bar, uint32_t parity, uint32_t abort_word) {
  if (__all_sync(0xFFFFFFFFu, mbar32_try_wait(bar, parity))) return true;
  return __all_sync(0xFFFFFFFFu, window_poll(bar, parity, abort_word));
}
// The registers of earlier loads may be read after this; it takes them as operands so that no use moves above it.
__device__ __forceinline__ void window_landed(uint32_t (&v)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]),
                 "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])::"memory");
}

template <int BITS, int GS, int ROWS>
__global__ void __launch_bounds__(640, 1) qmm_window_kernel(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ WindowParams p) {
  using Geo = WindowGeo<BITS, GS, ROWS>;
  constexpr int G = Geo::G, S = Geo::S, WPL = Geo::WPL, UNITW = Geo::UNITW, NST = Geo::NST, AS = Geo::AS, PS = Geo::PS;
  constexpr float OFFSET = code_offset(BITS);
  static_assert(!Fmt<BITS>::SPLIT, "one plane of codes an MMA");

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem32 = (smem_addr(smem_raw) + 1023u) & ~1023u;
  const uint32_t full32 = smem32 + NST * Geo::STAGE;        // weights and x of a stage have landed
  const uint32_t empty32 = full32 + 8 * NST;                // conversion and epilogue warps and the MMAs are done with it
  const uint32_t sums32 = empty32 + 8 * NST;                // the stage's group sums are written
  const uint32_t a_full32 = sums32 + 8 * NST;               // [2][AS] a group of A is in tensor memory
  const uint32_t a_empty32 = a_full32 + 16 * AS;            // [2][AS] the MMAs that read it are done
  const uint32_t p_full32 = a_empty32 + 16 * AS;            // [2][PS] a group's products are in tensor memory
  const uint32_t p_empty32 = p_full32 + 16 * PS;            // [2][PS] the epilogue warps have read them
  const uint32_t tmem32 = p_empty32 + 16 * PS, abort32 = tmem32 + 4;

  const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
  if (tid == 0) {
    auto init = [](uint32_t bar, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(n) : "memory"); };
    for (int i = 0; i < NST; ++i) init(full32 + 8 * i, 2), init(empty32 + 8 * i, 17), init(sums32 + 8 * i, 2);
    for (int i = 0; i < 2 * AS; ++i) init(a_full32 + 8 * i, 4), init(a_empty32 + 8 * i, 1);
    for (int i = 0; i < 2 * PS; ++i) init(p_full32 + 8 * i, 1), init(p_empty32 + 8 * i, 4);
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(abort32), "r"(0) : "memory");
    mbar_fence_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tmem32) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, lds32(tmem32), 0);
  pdl_launch_dependents();

  auto give_up = [&](int code) {
    if (lane == 0) {
      asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(abort32), "r"(code) : "memory");
      atomicCAS(p.err, 0, code);
    }
  };
  struct Item {
    int sb0, lanes, slice, tile, g_first, per, nst, m0, rows, n;
  };
  auto item_at = [&](int i) {
    Item it;
    const int j = i / p.row_tiles;
    it.tile = i - j * p.row_tiles;
    it.slice = j % p.sk;
    it.sb0 = (j / p.sk) * 2;
    it.lanes = min(2, p.nsb - it.sb0);
    it.g_first = static_cast<int>(static_cast<unsigned>(it.slice * p.KG) / static_cast<unsigned>(p.sk));   // (fits: the host checks)
    it.per = static_cast<int>(static_cast<unsigned>((it.slice + 1) * p.KG) / static_cast<unsigned>(p.sk)) - it.g_first;
    it.nst = (it.per + G - 1) / G;
    it.m0 = it.tile * p.tile_rows;
    it.rows = min(p.tile_rows, p.M - it.m0);
    it.n = (it.rows + 15) & ~15;
    return it;
  };
  const int step = gridDim.x;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");     // 128 x 48 + 256 x 72 + 256 x 144 = 640 x 96, the launch's registers
    if (warp == 0) {
      // ---------------------------------------------------------------- copies: units (bulk) and rows of x (tensor map)
      auto issue_w = [&](const Item& it, int st, int slot) {
        if (lane == 0) {
          const int ng = min(G, it.per - st * G);
          const uint32_t* src = p.w + static_cast<int64_t>(it.sb0) * p.sb_stride + (static_cast<int64_t>(it.g_first) + static_cast<int64_t>(st) * G) * UNITW;
          const uint32_t bar = full32 + 8 * slot, dst = smem32 + slot * Geo::STAGE + Geo::W_OFF;
          mbar32_expect_tx(bar, it.lanes * ng * UNITW * 4);
          for (int kw = 0; kw < it.lanes; ++kw) bulk_load32(dst + kw * Geo::W_BYTES, src + kw * p.sb_stride, ng * UNITW * 4, bar);
        }
      };
      auto issue_x = [&](const Item& it, int st, int slot) {
        if (lane == 0) {
          const int ng = min(G, it.per - st * G), boxes = (ng * GS + 63) / 64;
          const uint32_t bar = full32 + 8 * slot, dst = smem32 + slot * Geo::STAGE + Geo::X_OFF;
          mbar32_expect_tx(bar, boxes * Geo::XHALF);
          const int k0 = (it.g_first + st * G) * GS;
          for (int b = 0; b < boxes; ++b) tma_load_2d32(dst + b * Geo::XHALF, &tmx, k0 + 64 * b, it.m0, bar);
        }
      };
      {                                                      // the first weights never depend on the previous kernel
        int gst = 0;
        for (int i = blockIdx.x; i < p.items && gst < NST; i += step) {
          const Item it = item_at(i);
          for (int st = 0; st < it.nst && gst < NST; ++st, ++gst) issue_w(it, st, gst);
        }
      }
      pdl_wait();
      bool ok = true;
      int gst = 0, slot = 0;
      uint32_t phase = 1;
      for (int i = blockIdx.x; i < p.items && ok; i += step) {
        const Item it = item_at(i);
        for (int st = 0; st < it.nst; ++st, ++gst) {
          if (gst >= NST) {
            ok = window_wait(empty32 + 8 * slot, phase, abort32);
            if (!ok) {
              give_up(ERR_WAIT_EMPTY);
              break;
            }
            issue_w(it, st, slot);
          }
          issue_x(it, st, slot);
          if (++slot == NST) slot = 0, phase ^= 1;
        }
      }
      if (!ok)
        for (int i = 0; i < 64; ++i) __nanosleep(20000);     // copies in flight land before the shared memory is released
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issue
      bool ok = true;
      int slot = 0;
      uint32_t phase = 0, j[2] = {0, 0};
      for (int i = blockIdx.x; i < p.items && ok; i += step) {
        const Item it = item_at(i);
        const uint32_t n8 = __shfl_sync(0xFFFFFFFFu, static_cast<uint32_t>(it.n >> 3), 0);
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (n8 << 17) | ((128u >> 4) << 24);
        for (int st = 0; st < it.nst && ok; ++st) {
          ok = window_wait(full32 + 8 * slot, phase, abort32);
          const int ng = min(G, it.per - st * G);
          const uint64_t bd = window_desc(smem32 + slot * Geo::STAGE + Geo::X_OFF);
          for (int u = 0; u < ng && ok; ++u) {
#pragma unroll
            for (int kw = 0; kw < 2; ++kw) {
              if (kw >= it.lanes || !ok) continue;
              const uint32_t as = j[kw] % AS, ps = j[kw] % PS;
              ok = window_wait(a_full32 + 8 * (kw * AS + as), (j[kw] / AS) & 1, abort32);
              if (ok && j[kw] >= PS) ok = window_wait(p_empty32 + 8 * (kw * PS + ps), (j[kw] / PS - 1) & 1, abort32);
              if (!ok) continue;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              const uint32_t a = tmem + (kw * AS + as) * Geo::ACOLS, d = tmem + Geo::P_COL0 + (kw * PS + ps) * ROWS;
              if (window_elect()) {
#pragma unroll
                for (int s = 0; s < S; ++s) {
                  const int k16 = u * S + s;                 // 16-input step of the stage
                  window_mma(d, a + 8 * s, bd + (k16 >> 2) * (Geo::XHALF >> 4) + (k16 & 3) * 2, idesc, s != 0);
                }
                window_commit(a_empty32 + 8 * (kw * AS + as));
                window_commit(p_full32 + 8 * (kw * PS + ps));
                if (u == ng - 1 && kw == it.lanes - 1) window_commit(empty32 + 8 * slot);
              }
              __syncwarp();
              ++j[kw];
            }
          }
          if (++slot == NST) slot = 0, phase ^= 1;
        }
      }
      if (!ok) give_up(ERR_WAIT_FULL);
    } else {
      // ---------------------------------------------------------------- group sums of x (two warps, every other row tile)
      pdl_wait();
      bool ok = true;
      int slot = 0;
      uint32_t phase = 0;
      const int w2 = warp - 2;
      const uint32_t xrow = (lane & 7) * XHALF_ROW;
      const uint32_t sw0 = (((lane >> 3) ^ (lane & 7)) << 4), sw1 = (((4 | (lane >> 3)) ^ (lane & 7)) << 4);
      constexpr int NV = (ROWS * G + 63) / 64;
      for (int i = blockIdx.x; i < p.items && ok; i += step) {
        const Item it = item_at(i);
        float v[NV];
        auto fetch = [&](int st) {                           // given sums: on their way while the stage's copies are
#pragma unroll
          for (int e = 0; e < NV; ++e) {
            const int idx = e * 64 + w2 * 32 + lane, u = idx / ROWS, r = idx % ROWS;
            v[e] = 0.f;
            if (u < G && st * G + u < it.per && r < it.rows)
              v[e] = p.xs[static_cast<int64_t>(it.m0 + r) * p.KG + it.g_first + st * G + u];
          }
        };
        if (p.xs != nullptr) fetch(0);
        for (int st = 0; st < it.nst; ++st) {
          ok = window_wait(full32 + 8 * slot, phase, abort32);
          if (!ok) {
            give_up(ERR_WAIT_FULL);
            break;
          }
          const int ng = min(G, it.per - st * G);
          const uint32_t sp32 = smem32 + slot * Geo::STAGE, xs32 = sp32 + Geo::XS_OFF;
          if (p.xs != nullptr) {
#pragma unroll
            for (int e = 0; e < NV; ++e) {
              const int idx = e * 64 + w2 * 32 + lane;
              if (idx < ROWS * G) asm volatile("st.shared.f32 [%0], %1;" ::"r"(xs32 + idx * 4), "f"(v[e]) : "memory");
            }
          } else {
            for (int u = 0; u < ng; ++u) {
#pragma unroll 2
              for (int mt = w2; mt < it.n / 8; mt += 2) {
                float d[4];
                ones_mma_group<GS, Geo::XHALF>(d, sp32 + Geo::X_OFF, xrow, sw0, sw1, mt, u * GS);
                if (lane < 4)
                  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(xs32 + (u * ROWS + mt * 8 + 2 * lane) * 4), "f"(d[0]), "f"(d[1])
                               : "memory");
              }
            }
          }
          __syncwarp();
          if (lane == 0) mbar32_arrive(sums32 + 8 * slot);
          if (p.xs != nullptr && st + 1 < it.nst) fetch(st + 1);
          if (++slot == NST) slot = 0, phase ^= 1;
        }
      }
    }
  } else if (warp < 12) {
    // ------------------------------------------------------------------ conversion: packed codes -> A in tensor memory
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    const int kw = (warp - 4) >> 2, tp = warp & 3;
    const uint32_t w_off = Geo::W_OFF + kw * Geo::W_BYTES + (tp * 32 + lane) * WPL * 4;
    const uint32_t a_lane = tmem + kw * AS * Geo::ACOLS + (static_cast<uint32_t>(tp * 32) << 16);
    bool ok = true;
    int slot = 0;
    uint32_t phase = 0, j = 0;
    for (int i = blockIdx.x; i < p.items && ok; i += step) {
      const Item it = item_at(i);
      for (int st = 0; st < it.nst && ok; ++st) {
        ok = window_wait(full32 + 8 * slot, phase, abort32);
        const int ng = kw < it.lanes ? min(G, it.per - st * G) : 0;
        for (int u = 0; u < ng && ok; ++u) {
          const uint32_t src = smem32 + slot * Geo::STAGE + w_off + u * (UNITW * 4);
          uint32_t wd[WPL];
          if constexpr (WPL % 4 == 0) {
#pragma unroll
            for (int e = 0; e < WPL; e += 4) {
              const uint4 v = lds128(src + e * 4);
              wd[e] = v.x, wd[e + 1] = v.y, wd[e + 2] = v.z, wd[e + 3] = v.w;
            }
          } else if constexpr (WPL % 2 == 0) {
#pragma unroll
            for (int e = 0; e < WPL; e += 2) {
              const uint2 v = lds64(src + e * 4);
              wd[e] = v.x, wd[e + 1] = v.y;
            }
          } else {
#pragma unroll
            for (int e = 0; e < WPL; ++e) wd[e] = lds32(src + e * 4);
          }
          const uint32_t as = j % AS;
          if (j >= AS) ok = window_wait(a_empty32 + 8 * (kw * AS + as), (j / AS - 1) & 1, abort32);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int s = 0; s < S; s += 2) {                 // 32 inputs a store
              uint32_t r[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) r[e] = pair_reg<BITS, GS, false>(wd, (h * S + s) * 4 + e);
              window_store_a(a_lane + as * Geo::ACOLS + (static_cast<uint32_t>(16 * h) << 16) + 8 * s, r);
            }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar32_arrive(a_full32 + 8 * (kw * AS + as));
          ++j;
        }
        __syncwarp();
        if (ok && lane == 0) mbar32_arrive(empty32 + 8 * slot);
        if (++slot == NST) slot = 0, phase ^= 1;
      }
    }
    if (!ok) give_up(ERR_WAIT_FULL);
  } else {
    // ------------------------------------------------------------------ epilogue: the affine step, and the item's output
    asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
    const int kw = (warp - 12) >> 2, tp = warp & 3;
    const uint32_t sb_off = Geo::W_OFF + kw * Geo::W_BYTES + (TILE_PAIRS * 32 * WPL + affine_index(tp * 32 + lane)) * 4;
    const uint32_t p_lane = tmem + Geo::P_COL0 + kw * PS * ROWS + (static_cast<uint32_t>(tp * 32) << 16);
    bool ok = true;
    int slot = 0;
    uint32_t phase = 0, j = 0;
    uint64_t acc[ROWS / 2];                                  // rows 2 i, 2 i + 1 of this thread's column
    for (int i = blockIdx.x; i < p.items && ok; i += step) {
      const Item it = item_at(i);
      const bool active = kw < it.lanes;
#pragma unroll
      for (int e = 0; e < ROWS / 2; ++e) acc[e] = 0;
      for (int st = 0; st < it.nst && ok; ++st) {
        ok = window_wait(sums32 + 8 * slot, phase, abort32);
        const int ng = active ? min(G, it.per - st * G) : 0;
        const uint32_t sp32 = smem32 + slot * Geo::STAGE;
        for (int u = 0; u < ng && ok; ++u) {
          const uint32_t sb = lds32(sp32 + sb_off + u * (UNITW * 4));
          const float s = bf16_lo(sb), c = fmaf(-OFFSET, s, bf16_hi(sb));
          const uint64_t ss = pack2(s, s), cc = pack2(c, c);
          const uint32_t xs32 = sp32 + Geo::XS_OFF + u * ROWS * 4;
          const uint32_t ps = j % PS;
          ok = window_wait(p_full32 + 8 * (kw * PS + ps), (j / PS) & 1, abort32);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int q0 = 0; q0 < ROWS / 16; q0 += 2) {        // 32 rows of products in flight
            if (16 * q0 < it.n) {
              uint32_t v[2][16];
              window_load16(p_lane + ps * ROWS + 16 * q0, v[0]);
              const bool both = q0 + 1 < ROWS / 16 && 16 * (q0 + 1) < it.n;
              if (both) window_load16(p_lane + ps * ROWS + 16 * (q0 + 1), v[1]);
              window_landed(v[0]);
              if (both) window_landed(v[1]);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                if (q0 + h >= ROWS / 16 || (h == 1 && !both)) break;
                const int q = q0 + h;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const uint4 x4 = lds128(xs32 + (16 * q + 4 * e) * 4);
                  acc[8 * q + 2 * e] = fma2p(pack2u(x4.x, x4.y), cc, fma2p(pack2u(v[h][4 * e], v[h][4 * e + 1]), ss, acc[8 * q + 2 * e]));
                  acc[8 * q + 2 * e + 1] =
                      fma2p(pack2u(x4.z, x4.w), cc, fma2p(pack2u(v[h][4 * e + 2], v[h][4 * e + 3]), ss, acc[8 * q + 2 * e + 1]));
                }
              }
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar32_arrive(p_empty32 + 8 * (kw * PS + ps));
          ++j;
        }
        __syncwarp();
        if (ok && lane == 0) mbar32_arrive(empty32 + 8 * slot);
        if (++slot == NST) slot = 0, phase ^= 1;
      }
      if (!ok || !active) continue;

      pdl_wait();                                            // nothing is written before the previous kernel is done
      const int sb = it.sb0 + kw;
      const int n = sb * SB_COLS + tp * 32 + lane;
      auto store = [&](int row, float f) {
        const int64_t o = (it.m0 + row) * p.ldo + n;
        if (p.out_f32) reinterpret_cast<float*>(p.out)[o] = f;
        else reinterpret_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(f);
      };
      if (p.sk > 1) {
        // rows 4 q .. 4 q + 3 of column `lane` of the quarter: float4 q * 32 + lane
        const int64_t quad = (static_cast<int64_t>(it.tile) * p.nsb + sb) * p.sk;
        float4* base = reinterpret_cast<float4*>(p.part) + (quad * 4 + tp) * (ROWS * 8) + lane;
        constexpr int64_t SLICE = 4 * ROWS * 8;
        float4* dst = base + it.slice * SLICE;
#pragma unroll
        for (int q = 0; q < ROWS / 4; ++q)
          if (4 * q < it.n) {
            float4 f;
            unpack2(acc[2 * q], f.x, f.y), unpack2(acc[2 * q + 1], f.z, f.w);
            __stcg(dst + q * 32, f);
          }
        __threadfence();                                     // the slice is visible before this warp counts itself in
        __syncwarp();
        int* counter = p.count + (static_cast<int64_t>(it.tile) * p.nsb + sb) * 4 + tp;
        int seen = 0;
        if (lane == 0) seen = atomicAdd(counter, 1);
        seen = __shfl_sync(0xFFFFFFFFu, seen, 0);
        if (seen == p.sk - 1) {
          __threadfence();                                   // the other warps' slices are visible before they are read
#pragma unroll 1
          for (int q0 = 0; q0 < it.n / 4; q0 += 4) {         // sixteen rows a turn, sixteen loads in flight a lane
            const float4* src = base + q0 * 32;
            float4 f[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) f[q] = __ldcg(src + q * 32);
            int s = 1;
#pragma unroll 1
            for (; s + 4 <= p.sk; s += 4) {                  // slice order ((s0 + s1) + s2) + ...
              float4 g[4][4];
#pragma unroll
              for (int t = 0; t < 4; ++t)
#pragma unroll
                for (int q = 0; q < 4; ++q) g[t][q] = __ldcg(src + (s + t) * SLICE + q * 32);
#pragma unroll
              for (int t = 0; t < 4; ++t)
#pragma unroll
                for (int q = 0; q < 4; ++q) f[q].x += g[t][q].x, f[q].y += g[t][q].y, f[q].z += g[t][q].z, f[q].w += g[t][q].w;
            }
#pragma unroll 1
            for (; s < p.sk; ++s)
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const float4 g = __ldcg(src + s * SLICE + q * 32);
                f[q].x += g.x, f[q].y += g.y, f[q].z += g.z, f[q].w += g.w;
              }
            if (n < p.N) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const float v[4] = {f[q].x, f[q].y, f[q].z, f[q].w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                  if (4 * (q0 + q) + e < it.rows) store(4 * (q0 + q) + e, v[e]);
              }
            }
          }
          if (lane == 0) *counter = 0;                       // the next launch finds the counter at zero again
        }
      } else if (n < p.N) {
#pragma unroll
        for (int e = 0; e < ROWS / 2; ++e) {
          float f[2];
          unpack2(acc[e], f[0], f[1]);
          if (2 * e < it.rows) store(2 * e, f[0]);
          if (2 * e + 1 < it.rows) store(2 * e + 1, f[1]);
        }
      }
    }
    if (!ok) give_up(ERR_WAIT_SUMS);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

}  // namespace tf
