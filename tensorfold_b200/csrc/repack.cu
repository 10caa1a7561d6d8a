// Load-time repack: stored MLX rows <-> tiled units (tf_layout.h), one block per (128 columns, run of groups).
//
// A unit and the stored words it comes from are the same size: GS * BITS / 32 = WPL words a row and group, 128 rows.  So a
// block brings the RUN = GROUPS * WPL words of its 128 rows into shared memory with coalesced loads (a run is about 128
// bytes), permutes the codes from one shared buffer into another, and stores with coalesced stores; unpack is the mirror
// image.  The bound is memory, every word crosses HBM once each way, so the permutation must stay cheap: a thread makes
// whole lanes (pack) or whole rows (unpack), so positions are compile-time constants, codes move in pairs (inputs 2 i,
// 2 i + 1 are neighbours in the stored row and the two halves of one lane word), and 4-bit codes, the common width, move
// four bytes at a time with byte permutes.
// Measured from graphs, 17408 x 5120 in groups of 64 (pack / unpack): 4 bits 29 / 22 us (3.5 / 4.6 TB/s), 8 bits 51 / 49 us (3.7 /
// 3.9), 3 bits 45 / 39 us (1.7 / 2.0), 2 bits 21 / 22, 5 bits 63 / 50, 6 bits 54 / 54.  One thread an output word, gathering its
// codes from global memory, took 252 / 289 us at 4 bits.
#include <algorithm>
#include <type_traits>

#include "../../include/tensorfold_b200.h"
#include "tf_layout.h"

#include <cuda_runtime.h>

namespace tf {

int fail_moe(int code, const char* msg);          // tf_api.cu: sets the thread's error text
int cuda_fail_moe(cudaError_t e, const char* what);

namespace {

constexpr int REPACK_THREADS = 128;               // one thread a column (unpack) or a lane of the four tile pairs (pack)

template <int BITS, int GS>
struct RepackGeo {
  static constexpr int WPL = words_per_lane(BITS, GS), UNITW = unit_words(BITS, GS), S = GS / 16;
  static constexpr int WA = Fmt<BITS>::WA, WB = Fmt<BITS>::WB, PAIRS = pairs_per_lane(GS);
  static constexpr int WORDS_A = PAIRS * WA / 16;                        // lane words of plane A; the rest are plane B
  // groups a block takes: runs of about 128 bytes a row (64 for 2 bits and groups of 32, whose affine words fill the rest)
  static constexpr int GROUPS = WPL >= 32 ? 1 : WPL == 2 ? 8 : 32 / WPL;
  static constexpr int RUN = GROUPS * WPL;
  static constexpr int VEC = WPL % 4 == 0 ? 4 : 1;                       // words a global access moves (rows are then 16-byte aligned)
  // Strides in words that keep eight neighbouring rows, or the lanes of eight neighbouring columns, on distinct banks;
  // rows keep at least one spare word (a funnel shift reads one past the last).
  static constexpr int ROW = VEC == 4 ? RUN + 4 : (RUN + 1) | 1;
  static constexpr int QUAD = 4 * WPL + (WPL % 2 == 0 ? 4 : 0);          // the four lanes of a column, in unpack's shared units
  static constexpr int UNIT = 32 * QUAD + AFFINE_WORDS;
};

template <int VEC>
using Vec = std::conditional_t<VEC == 4, uint4, uint32_t>;

// Global accesses of VEC words; `wide`: the tensor starts on a 16-byte boundary (a view of a larger buffer may not).
template <int VEC>
__device__ __forceinline__ Vec<VEC> fetch(const uint32_t* p, bool wide) {
  if constexpr (VEC == 4) {
    if (!wide) return make_uint4(p[0], p[1], p[2], p[3]);
  }
  return *reinterpret_cast<const Vec<VEC>*>(p);
}
template <int VEC>
__device__ __forceinline__ void put(uint32_t* p, Vec<VEC> v, bool wide) {
  if constexpr (VEC == 4) {
    if (!wide) {
      p[0] = v.x, p[1] = v.y, p[2] = v.z, p[3] = v.w;
      return;
    }
  }
  *reinterpret_cast<Vec<VEC>*>(p) = v;
}

// Codes 2 i and 2 i + 1 of a run of stored words, in the low BITS and the next BITS bits (garbage above).
template <int BITS>
__device__ __forceinline__ uint32_t stored_pair(const uint32_t* run, int i) {
  const int bit = 2 * BITS * i, w = bit >> 5, sh = bit & 31;
  if constexpr (32 % (2 * BITS) == 0) return run[w] >> sh;
  else return __funnelshift_r(run[w], run[w + 1], sh);
}

// The words of one lane (4 g + t of a tile pair) for one group: `rows` points at the group's first word of column g.
template <int BITS, int GS>
__device__ __forceinline__ void lane_words(const uint32_t* rows, int t, uint32_t (&out)[RepackGeo<BITS, GS>::WPL]) {
  using Geo = RepackGeo<BITS, GS>;
  constexpr int S = Geo::S, WA = Geo::WA, WB = Geo::WB;
  if constexpr (BITS == 4) {
    // word h S + s holds byte t (a pair of codes) of words 2 s and 2 s + 1 of columns g and g + 8 of half h
    const uint32_t pick = t | ((t + 4) << 4);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int s = 0; s < S; s += 2) {
        const uint4 a = *reinterpret_cast<const uint4*>(rows + 16 * h * Geo::ROW + 2 * s);
        const uint4 b = *reinterpret_cast<const uint4*>(rows + (16 * h + 8) * Geo::ROW + 2 * s);
        auto word = [&](uint32_t a0, uint32_t b0, uint32_t a1, uint32_t b1) {
          const uint32_t x = __byte_perm(__byte_perm(a0, b0, pick), __byte_perm(a1, b1, pick), 0x5410);
          const uint32_t lo = x & 0x0F0F0F0Fu, hi = (x >> 4) & 0x0F0F0F0Fu;
          return __byte_perm(lo | (lo >> 4), hi | (hi >> 4), 0x6420);
        };
        out[h * S + s] = word(a.x, b.x, a.y, b.y);
        out[h * S + s + 1] = word(a.z, b.z, a.w, b.w);
      }
  } else {
#pragma unroll
    for (int i = 0; i < Geo::WPL; ++i) out[i] = 0u;
#pragma unroll
    for (int p = 0; p < Geo::PAIRS; ++p) {
      const int j = p & 3, s = (p >> 2) % S, h = (p >> 2) / S;
      const uint32_t pair = stored_pair<BITS>(rows + (16 * h + 8 * (j & 1)) * Geo::ROW, 8 * s + 4 * (j >> 1) + t);
      auto insert = [&](int word, int slot, int width, int shift) {
        const uint32_t mask = (1u << width) - 1u;
        out[word] |= ((pair >> shift) & mask) << (slot * width) | ((pair >> (BITS + shift)) & mask) << (16 + slot * width);
      };
      insert(p / (16 / WA), p % (16 / WA), WA, 0);
      if constexpr (WB > 0) insert(Geo::WORDS_A + p / (16 / WB), p % (16 / WB), WB, WA);
    }
  }
}

template <int BITS, int GS>
__global__ void __launch_bounds__(REPACK_THREADS) pack_kernel(const uint32_t* __restrict__ words, const uint16_t* __restrict__ scales,
                                                              const uint16_t* __restrict__ biases, const uint32_t* __restrict__ words2,
                                                              const uint16_t* __restrict__ scales2, const uint16_t* __restrict__ biases2,
                                                              int n, int kg, uint32_t* __restrict__ tiled, bool wide_words, bool wide_tiled) {
  using Geo = RepackGeo<BITS, GS>;
  constexpr int WPL = Geo::WPL, UNITW = Geo::UNITW, RUN = Geo::RUN, VEC = Geo::VEC;
  __shared__ __align__(16) uint32_t rows[SB_COLS * Geo::ROW];
  __shared__ __align__(16) uint32_t units[Geo::GROUPS * UNITW];
  const int runs = (kg + Geo::GROUPS - 1) / Geo::GROUPS, tid = threadIdx.x;
  const int g0 = blockIdx.x % runs * Geo::GROUPS, groups = min(Geo::GROUPS, kg - g0);
  const int64_t sb = blockIdx.x / runs, wpr = static_cast<int64_t>(kg) * WPL;
  // With a second source the packed rows interleave 16 rows of the first with 16 rows of the second (gate and up): packed
  // row r comes from source (r / 16) % 2, row (r / 32) * 16 + r % 16.
  auto source = [&](int64_t& row) -> bool {
    if (words2 == nullptr) return false;
    const bool second = (row >> 4) & 1;
    row = (row >> 5) * 16 + (row & 15);
    return second;
  };
#pragma unroll 8
  for (int i = tid; i < SB_COLS * RUN / VEC; i += REPACK_THREADS) {
    const int c = i / (RUN / VEC), w = i % (RUN / VEC) * VEC;
    int64_t row = sb * SB_COLS + c;
    Vec<VEC> v = {};                                                     // rows past n pack as zero codes
    if (row < n && w < groups * WPL) {
      const uint32_t* src = source(row) ? words2 : words;
      v = fetch<VEC>(src + row * wpr + static_cast<int64_t>(g0) * WPL + w, wide_words);
    }
    *reinterpret_cast<Vec<VEC>*>(rows + c * Geo::ROW + w) = v;
  }
  for (int i = tid; i < SB_COLS * groups; i += REPACK_THREADS) {
    const int c = i / groups, u = i % groups;
    int64_t row = sb * SB_COLS + c;
    uint32_t v = 0u;
    if (row < n) {
      const bool second = source(row);
      const int64_t at = row * kg + g0 + u;
      v = static_cast<uint32_t>((second ? scales2 : scales)[at]) | (static_cast<uint32_t>((second ? biases2 : biases)[at]) << 16);
    }
    units[u * UNITW + TILE_PAIRS * 32 * WPL + affine_index(c)] = v;
  }
  __syncthreads();
  const int tp = tid >> 5, lane = tid & 31;
  for (int u = 0; u < groups; ++u) {
    uint32_t mine[WPL];
    lane_words<BITS, GS>(rows + (32 * tp + (lane >> 2)) * Geo::ROW + u * WPL, lane & 3, mine);
    Vec<VEC>* dst = reinterpret_cast<Vec<VEC>*>(units + u * UNITW + tid * WPL);
#pragma unroll
    for (int i = 0; i < WPL / VEC; ++i) {
      if constexpr (VEC == 4) dst[i] = make_uint4(mine[4 * i], mine[4 * i + 1], mine[4 * i + 2], mine[4 * i + 3]);
      else dst[i] = mine[i];
    }
  }
  __syncthreads();
  uint32_t* out = tiled + (sb * kg + g0) * UNITW;                             // (a unit is a multiple of 16 bytes)
  for (int i = tid; i < groups * UNITW / 4; i += REPACK_THREADS)
    put<4>(out + 4 * i, reinterpret_cast<const uint4*>(units)[i], wide_tiled);
}

template <int BITS, int GS>
__global__ void __launch_bounds__(REPACK_THREADS) unpack_kernel(const uint32_t* __restrict__ tiled, int n, int kg,
                                                                uint32_t* __restrict__ words, uint16_t* __restrict__ scales,
                                                                uint16_t* __restrict__ biases, bool wide_words, bool wide_tiled) {
  using Geo = RepackGeo<BITS, GS>;
  constexpr int WPL = Geo::WPL, UNITW = Geo::UNITW, UNIT = Geo::UNIT, RUN = Geo::RUN, WA = Geo::WA, WB = Geo::WB, S = Geo::S;
  constexpr int VEC = Geo::VEC, CODE_WORDS = TILE_PAIRS * 32 * WPL;
  __shared__ __align__(16) uint32_t units[Geo::GROUPS * UNIT];               // the four lanes of a column QUAD words apart
  __shared__ __align__(16) uint32_t rows[SB_COLS * Geo::ROW];
  const int runs = (kg + Geo::GROUPS - 1) / Geo::GROUPS, tid = threadIdx.x;
  const int g0 = blockIdx.x % runs * Geo::GROUPS, groups = min(Geo::GROUPS, kg - g0);
  const int64_t sb = blockIdx.x / runs, wpr = static_cast<int64_t>(kg) * WPL;
  const uint32_t* src = tiled + (sb * kg + g0) * UNITW;
#pragma unroll 8
  for (int i = tid; i < groups * UNITW / 4; i += REPACK_THREADS) {
    const int u = 4 * i / UNITW, w = 4 * i % UNITW;                          // (four words of a quad, or of the affine part)
    const int at = w < CODE_WORDS ? w / (4 * WPL) * Geo::QUAD + w % (4 * WPL) : 32 * Geo::QUAD + w - CODE_WORDS;
    *reinterpret_cast<uint4*>(units + u * UNIT + at) = fetch<4>(src + 4 * i, wide_tiled);
  }
  __syncthreads();
  if constexpr (BITS == 4) {
    // Half a block a group: a thread takes columns c and c + 8.  Word h S + s of lane t holds the byte pairs (slots 0, 2 of
    // column c, slots 1, 3 of column c + 8) that go to byte t of words 2 s and 2 s + 1 of those rows.
    const int g = tid & 7, h = (tid >> 3) & 1, tp = (tid >> 4) & 3;
    for (int u = tid >> 6; u < groups; u += 2) {
      const uint32_t* quad = units + u * UNIT + (8 * tp + g) * Geo::QUAD + h * S;
      uint32_t* row = rows + (32 * tp + 16 * h + g) * Geo::ROW + u * WPL;
#pragma unroll
      for (int s = 0; s < S; s += 2) {
        uint32_t e[4][2], o[4][2];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const uint2 v = *reinterpret_cast<const uint2*>(quad + t * WPL + s);
          const uint32_t vv[2] = {v.x, v.y};
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint32_t even = vv[i] & 0x0F0F0F0Fu, odd = (vv[i] >> 4) & 0x0F0F0F0Fu;
            e[t][i] = even | (even >> 12), o[t][i] = odd | (odd >> 12);      // bytes 0 and 1: slots 0, 2 and slots 1, 3
          }
        }
        auto gather = [&](const uint32_t (&x)[4][2], int i, uint32_t& first, uint32_t& second) {
          const uint32_t ab = __byte_perm(x[0][i], x[1][i], 0x5140), cd = __byte_perm(x[2][i], x[3][i], 0x5140);
          first = __byte_perm(ab, cd, 0x5410), second = __byte_perm(ab, cd, 0x7632);
        };
        uint4 a, b;
        gather(e, 0, a.x, a.y), gather(e, 1, a.z, a.w);
        gather(o, 0, b.x, b.y), gather(o, 1, b.z, b.w);
        *reinterpret_cast<uint4*>(row + 2 * s) = a;
        *reinterpret_cast<uint4*>(row + 8 * Geo::ROW + 2 * s) = b;
      }
    }
  } else {
    const int g = tid & 7, r8 = (tid >> 3) & 1, h = (tid >> 4) & 1, tp = tid >> 5;
    for (int u = 0; u < groups; ++u) {
      const uint32_t* quad = units + u * UNIT + (8 * tp + g) * Geo::QUAD;
      uint32_t mine[WPL + 1] = {};
#pragma unroll
      for (int i = 0; i < GS / 2; ++i) {                                     // pair i: inputs 2 i and 2 i + 1
        const int s = i >> 3, t = i & 3, p = (h * S + s) * 4 + r8 + 2 * ((i >> 2) & 1);
        const uint32_t* lw = quad + t * WPL;
        const uint32_t a = lw[p / (16 / WA)] >> (p % (16 / WA) * WA);
        uint32_t lo = a & ((1u << WA) - 1u), hi = (a >> 16) & ((1u << WA) - 1u);
        if constexpr (WB > 0) {
          const uint32_t b = lw[Geo::WORDS_A + p / (16 / WB)] >> (p % (16 / WB) * WB);
          lo |= (b & ((1u << WB) - 1u)) << WA, hi |= ((b >> 16) & ((1u << WB) - 1u)) << WA;
        }
        const uint32_t pair = lo | (hi << BITS);
        const int bit = 2 * BITS * i;
        mine[bit >> 5] |= pair << (bit & 31);
        if ((bit & 31) + 2 * BITS > 32) mine[(bit >> 5) + 1] |= pair >> (32 - (bit & 31));
      }
      Vec<VEC>* dst = reinterpret_cast<Vec<VEC>*>(rows + tid * Geo::ROW + u * WPL);
#pragma unroll
      for (int i = 0; i < WPL / VEC; ++i) {
        if constexpr (VEC == 4) dst[i] = make_uint4(mine[4 * i], mine[4 * i + 1], mine[4 * i + 2], mine[4 * i + 3]);
        else dst[i] = mine[i];
      }
    }
  }
  __syncthreads();
  const int cols = static_cast<int>(min(static_cast<int64_t>(SB_COLS), n - sb * SB_COLS));
  for (int i = tid; i < cols * (RUN / VEC); i += REPACK_THREADS) {
    const int c = i / (RUN / VEC), w = i % (RUN / VEC) * VEC;
    if (w < groups * WPL)
      put<VEC>(words + (sb * SB_COLS + c) * wpr + static_cast<int64_t>(g0) * WPL + w,
               *reinterpret_cast<const Vec<VEC>*>(rows + c * Geo::ROW + w), wide_words);
  }
  for (int i = tid; i < cols * groups; i += REPACK_THREADS) {
    const int c = i / groups, u = i % groups;
    const uint32_t v = units[u * UNIT + 32 * Geo::QUAD + affine_index(c)];
    const int64_t at = (sb * SB_COLS + c) * kg + g0 + u;
    scales[at] = static_cast<uint16_t>(v & 0xFFFFu);
    biases[at] = static_cast<uint16_t>(v >> 16);
  }
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

bool format_known(int bits, int gs) {
  return (bits == 2 || bits == 3 || bits == 4 || bits == 5 || bits == 6 || bits == 8) && (gs == 32 || gs == 64 || gs == 128);
}

struct Sources {
  const void *words, *scales, *biases, *words2, *scales2, *biases2;
};

// One block a (super-block, run of groups), runs fastest.
template <int BITS, int GS>
int grid_of(int n, int kg) {
  constexpr int GROUPS = RepackGeo<BITS, GS>::GROUPS;
  return (kg + GROUPS - 1) / GROUPS * ((n + SB_COLS - 1) / SB_COLS);
}

template <int BITS, int GS>
void launch_pack(const Sources& f, int n, int kg, uint32_t* tiled, cudaStream_t s) {
  pack_kernel<BITS, GS><<<grid_of<BITS, GS>(n, kg), REPACK_THREADS, 0, s>>>(
      static_cast<const uint32_t*>(f.words), static_cast<const uint16_t*>(f.scales), static_cast<const uint16_t*>(f.biases),
      static_cast<const uint32_t*>(f.words2), static_cast<const uint16_t*>(f.scales2), static_cast<const uint16_t*>(f.biases2), n, kg,
      tiled, aligned16(f.words) && aligned16(f.words2), aligned16(tiled));
}

template <int BITS, int GS>
void launch_unpack(const uint32_t* tiled, int n, int kg, uint32_t* words, uint16_t* scales, uint16_t* biases, cudaStream_t s) {
  unpack_kernel<BITS, GS><<<grid_of<BITS, GS>(n, kg), REPACK_THREADS, 0, s>>>(tiled, n, kg, words, scales, biases, aligned16(words), aligned16(tiled));
}

#define TF_EACH_GROUP(CALL, B) \
  if (gs == 32) CALL(B, 32);   \
  else if (gs == 64) CALL(B, 64); \
  else CALL(B, 128);
#define TF_EACH_FORMAT(CALL)                  \
  switch (bits) {                             \
    case 2: TF_EACH_GROUP(CALL, 2) break;     \
    case 3: TF_EACH_GROUP(CALL, 3) break;     \
    case 4: TF_EACH_GROUP(CALL, 4) break;     \
    case 5: TF_EACH_GROUP(CALL, 5) break;     \
    case 6: TF_EACH_GROUP(CALL, 6) break;     \
    default: TF_EACH_GROUP(CALL, 8) break;    \
  }

int shape_error(const char* who, int n, int k, int bits, int gs) {
  if (!format_known(bits, gs)) return fail_moe(TF_ERR_ARG, who);
  if (n < 1 || k < gs || k % gs || (static_cast<int64_t>(k) * bits) % 32) return fail_moe(TF_ERR_ARG, who);
  return TF_OK;
}

int pack_units(const Sources& f, int n, int k, int bits, int gs, void* tiled, void* stream, const char* who) {
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  uint32_t* units = static_cast<uint32_t*>(tiled);
  const int kg = k / gs;
#define TF_CALL(B, G) launch_pack<B, G>(f, n, kg, units, s)
  TF_EACH_FORMAT(TF_CALL)
#undef TF_CALL
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TF_OK : cuda_fail_moe(e, who);
}

}  // namespace

}  // namespace tf

using namespace tf;

extern "C" {

int tf_pack(const void* words, const void* scales, const void* biases, int n, int k, int bits, int gs, void* tiled, void* stream) {
  if (int rc = shape_error("tf_pack: an affine format, whole groups and words", n, k, bits, gs)) return rc;
  if (!words || !scales || !biases || !tiled) return fail_moe(TF_ERR_ARG, "tf_pack: null pointer");
  return pack_units({words, scales, biases, nullptr, nullptr, nullptr}, n, k, bits, gs, tiled, stream, "tf_pack");
}

int tf_pack_pair(const void* words_a, const void* scales_a, const void* biases_a, const void* words_b, const void* scales_b,
                 const void* biases_b, int n_each, int k, int bits, int gs, void* tiled, void* stream) {
  if (n_each < 16 || n_each % 16)
    return fail_moe(TF_ERR_ARG, "tf_pack_pair: rows in whole 16-row tiles");
  if (int rc = shape_error("tf_pack_pair: an affine format, whole groups and words", 2 * n_each, k, bits, gs)) return rc;
  if (!words_a || !scales_a || !biases_a || !words_b || !scales_b || !biases_b || !tiled)
    return fail_moe(TF_ERR_ARG, "tf_pack_pair: null pointer");
  return pack_units({words_a, scales_a, biases_a, words_b, scales_b, biases_b}, 2 * n_each, k, bits, gs, tiled, stream, "tf_pack_pair");
}

int tf_unpack(const void* tiled, int n, int k, int bits, int gs, void* words, void* scales, void* biases, void* stream) {
  if (int rc = shape_error("tf_unpack: an affine format, whole groups and words", n, k, bits, gs)) return rc;
  if (!words || !scales || !biases || !tiled) return fail_moe(TF_ERR_ARG, "tf_unpack: null pointer");
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int kg = k / gs;
#define TF_CALL(B, G)                                                                                          \
  launch_unpack<B, G>(static_cast<const uint32_t*>(tiled), n, kg, static_cast<uint32_t*>(words), static_cast<uint16_t*>(scales), \
                      static_cast<uint16_t*>(biases), s)
  TF_EACH_FORMAT(TF_CALL)
#undef TF_CALL
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TF_OK : cuda_fail_moe(e, "tf_unpack");
}

}  // extern "C"
