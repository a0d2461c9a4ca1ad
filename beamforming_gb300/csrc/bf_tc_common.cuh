// bf_tc_common.cuh -- what the tensor-core kernels share: the tile and its row
// map, the unpack of raw E bytes into operand words, and the epilogue of one
// accumulator.
#pragma once

#include "bf_internal.h"
#include "bf_ptx.cuh"

namespace bf {
namespace {

constexpr int kTT = 64;                 // times per tile
constexpr int kBM = 128;                // GEMM rows per tile
constexpr int kKC = 128;                // K bytes per TMA box / swizzle atom (64 dishes x re/im)
constexpr int kSub = 2;                 // boxes per pipeline stage
constexpr int kStageK = kSub * kKC;     // K bytes per stage (128 dishes x re/im): 8 MMAs
static_assert(kSub == 2, "mma_ts_stage8 issues the eight MMAs of two W boxes");
constexpr int kRawBox = kTT * kKC;      // raw E per box: 64 times x 64 dishes x 2 pol
constexpr int kRawBytes = kSub * kRawBox;
constexpr int kStageCols = kStageK / 4;  // TMEM columns per unpacked stage
constexpr int kDigSlots = 2;            // digit-row slots (one per tile in flight)
// Offset correction: one extra MMA per tile, issued first (it also clears the
// accumulator) or, with row sums (RowSums), last, multiplies a constant A tile by
// the tile's digit rows.  The constant row holds -2^-6, -2^-2, -4, -64, -256 at K = 0..4 (again at 16..20,
// so the 32-byte swizzle cannot move them), the digit row of n holds d0..d3 and
// 4 d4, all times 2^-9, with sum_k W[n][k] = d0 + 16 d1 + 256 d2 + 4096 d3 + 65536 d4, so it
// adds -2^-15 sum_k W[n][k] = -8 sum_k W[n][k] 2^-18 exactly.
constexpr uint32_t kDigitScaleLo = 0xE8C8A888u;  // E4M3 -2^-6, -2^-2, -4, -64
constexpr uint32_t kDigitScaleHi = 0x000000F8u;  // E4M3 -256
constexpr int kConstABytes = kBM * kDigitRow;

// Position in a ring of n slots: slot index and the parity of the pass over the ring.
struct Ring {
  uint32_t idx = 0, phase = 0, n;
  __device__ explicit Ring(int n_) : n(static_cast<uint32_t>(n_)) {}
  __device__ __forceinline__ void advance() {
    if (++idx == n) {
      idx = 0;
      phase ^= 1u;
    }
  }
};

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

// (c << 8) | (sat(re) << 4) | sat(im): two integers saturated to [0, 15] and
// packed as the nibbles of one byte below the bytes of c.
__device__ __forceinline__ uint32_t pack_u4x2(uint32_t re, uint32_t im, uint32_t c) {
  uint32_t r;
  asm("cvt.pack.sat.u4.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(re), "r"(im), "r"(c));
  return r;
}

// GEMM row r (0..31) of a lane quarter q <-> time and polarization of the tile.
// The epilogue's loads give thread (g, c) = (lane / 4, lane % 4) the four rows
// g, g + 8, g + 16, g + 24, so those hold four consecutive bytes of J: four
// times of one polarization (Jlinear, arraysizes.hxx:92; quarter q holds 32
// times of polarization q % 2), or two times of both (J2linear,
// arraysizes.hxx:103; 16 times).  Which of the four sits in which row depends
// on g through `swap`, which spreads the raw rows that 8 lanes of the unpack
// read together over all 8 positions of the 128-byte swizzle (no bank
// conflicts); the epilogue undoes it with one byte permute.
template <bool kJ2>
struct RowMap {
  __device__ static __forceinline__ uint32_t swap(uint32_t g) { return kJ2 ? 2u * (g >> 2) : g >> 1; }
  __device__ static __forceinline__ uint32_t time(uint32_t q, uint32_t r) {
    const uint32_t g = r & 7u, j = (r >> 3) ^ swap(g);
    return kJ2 ? 16u * q + 2u * g + (j >> 1) : 32u * (q >> 1) + 4u * g + j;
  }
  __device__ static __forceinline__ uint32_t pol(uint32_t q, uint32_t r) {
    return kJ2 ? ((r >> 3) ^ swap(r & 7u)) & 1u : q & 1u;
  }
};

// Byte offset of 16-byte chunk j of row r in a 128B-swizzled tile (TMA layout).
__device__ __forceinline__ uint32_t sw128_offset(uint32_t r, uint32_t j) {
  return (r >> 3) * 1024u + (r & 7u) * 128u + ((j ^ (r & 7u)) << 4);
}

// Byte offsets of the eight 16-byte chunks of row t of a raw box, computed once:
// the swizzle's exclusive-or would cost the integer pipe 8 operations per box.
struct UnpackRow {
  uint32_t at[8];
  __device__ __forceinline__ explicit UnpackRow(uint32_t t) {
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) at[j] = sw128_offset(t, j);
  }
};

// One raw E box (64 times x 64 dishes x 2 polarizations, 128-byte swizzle) in
// shared memory -> the 128 operand bytes of this lane's row, of the polarization
// that `sel` picks (0x6420: even bytes, 0x7531: odd ones).  Returns
// the sum of those 128 nibbles with kSums.
template <bool kSums>
__device__ __forceinline__ uint32_t unpack_box(uint32_t raw, const UnpackRow &row, uint32_t sel, uint32_t (&out)[32]) {
  uint32_t e[16];  // this row's polarization, dishes 4m..4m+3 of the box in word m
#pragma unroll
  for (uint32_t j = 0; j < 8; ++j) {
    // 16-byte chunk j: dishes 8j..8j+7, bytes [d0p0 d0p1 d1p0 d1p1 ...]
    uint4 w;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w)
                 : "r"(raw + row.at[j]));
    e[2 * j] = prmt(w.x, w.y, sel);
    e[2 * j + 1] = prmt(w.z, w.w, sel);
  }
  const uint32_t msk = 0x0F0F0F0Fu;
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    out[2 * m] = (e[m] >> 4) & msk;  // real nibbles u (E4M3 bytes = u * 2^-9)
    out[2 * m + 1] = e[m] & msk;     // imaginary nibbles
  }
  if (!kSums) return 0;
  uint32_t s[2] = {0, 0};  // byte sums of 16 words: at most 240
#pragma unroll
  for (int m = 0; m < 16; ++m) s[m >> 3] += out[2 * m] + out[2 * m + 1];
  return __dp4a(s[0], 0x01010101u, __dp4a(s[1], 0x01010101u, 0u));
}

// The A tile of the offset MMA: 128 rows of 32 bytes (32-byte swizzle), one tile
// per accumulator.  Words 0, 1, 4 and 5 of a row hold the digit scales; words 2
// and 3 of its first 16 bytes take -- against kDigitScaleLo in the digit rows --
// the sum of the row's nibbles u as base-16 digits, from the two parts of its
// K stages (or boxes) that the unpack warps of its lane quarter take.
template <int kTiles>
__device__ __forceinline__ void fill_offset_tiles(uint8_t *sA) {
  for (int i = threadIdx.x; i < kTiles * kConstABytes / 4; i += blockDim.x) {
    const int w = i & 3;
    reinterpret_cast<uint32_t *>(sA)[i] = w == 0 ? kDigitScaleLo : w == 1 ? kDigitScaleHi : 0u;
  }
}

// One unpack warp's walk over the tiles: it takes the K stages kpos, kpos +
// groups, ... of tile after tile, and hands over its rows' sums at the end of each.
struct RowSums {
  uint32_t *at;  // this lane's word in the first tile
  int tile = 0, kpos;
  uint32_t sum = 0;  // < 2^16: at most 2 * 2048 nibbles
  __device__ RowSums(uint8_t *sA, int group, int part, int row)
      : at(reinterpret_cast<uint32_t *>(sA) + row * (kDigitRow / 4) + ((row >> 2) & 1) * 4 + 2 + part), kpos(group) {}
  // After each stage (and once before the first: with fewer stages a tile than
  // groups a warp has none of some tiles).  `free` waits for the MMAs of the tile
  // two before, `arrive` tells the issuer.
  template <class Free, class Arrive>
  __device__ __forceinline__ bool settle(int nk, int ntiles, Free free, Arrive arrive) {
    while (kpos >= nk && tile < ntiles) {
      if (!free(tile)) return false;
      uint32_t w = (sum | (sum << 8)) & 0x00FF00FFu;
      w = (w | (w << 4)) & 0x0F0F0F0Fu;
      at[(tile & 1) * (kConstABytes / 4)] = w;
      fence_proxy_async_smem();
      __syncwarp();
      arrive(tile);
      sum = 0;
      ++tile;
      kpos -= nk;
    }
    return true;
  }
};

// The epilogue of one accumulator for one warp: lane quarter q of the tile's
// rows and a range of its 8-beam column chunks.  Thread (g, cb) = (lane / 4,
// lane % 4) takes rows g, g + 8, g + 16, g + 24 (four consecutive bytes of J,
// RowMap) of every fourth beam.
template <bool kJ2, bool kAdler>
struct EpilogueTile {
  const float *gcur;  // written by the launch before this one: plain loads (grid_wait)
  uint8_t *jrow;  // the thread's bytes for beam b0 + cb
  int64_t bstride;
  int blim;
  int nbytes;     // of the thread's 4 bytes, those inside the row
  uint32_t osel;  // the rows' bytes into J's order
  bool wide, bytes;

  __device__ __forceinline__ EpilogueTile(const TcProblem &P, int f, int pass, int tt, int q, int lane) {
    const uint32_t g = static_cast<uint32_t>(lane) >> 2, cb = static_cast<uint32_t>(lane) & 3u;
    osel = 0x3210u ^ (0x1111u * RowMap<kJ2>::swap(g));
    const int b0 = pass * P.nb_pass;
    // 2^18 G[f][b0 ..] (zero beyond B): the accumulator ends at 2^-18 raw
    // exactly and the power-of-two scaling is exact, so (2^18 G) * (2^-18 raw)
    // rounds like G * raw (cpu.cxx:37)
    gcur = P.gs + static_cast<int64_t>(f) * P.npass * P.nb_pass + b0 + cb;
    // huge or non-finite gains of this frequency: requantise with the
    // narrowing of cpu.cxx:38 (tile-uniform branch, normally not taken)
    wide = P.gwide[f] != 0;
    const int64_t bj = static_cast<int64_t>(b0 + static_cast<int>(cb)) * P.F + f;  // beam row b0 + cb
    int64_t at;  // the thread's 4 bytes in the J row
    if constexpr (!kJ2) {
      at = static_cast<int64_t>(tt) * kTT + RowMap<kJ2>::time(q, 8 * RowMap<kJ2>::swap(g) + g);
      jrow = P.J + (bj * 2 + (q & 1)) * P.rpitch + at;
      bstride = static_cast<int64_t>(P.F) * 2 * P.rpitch;
    } else {
      at = 2 * (static_cast<int64_t>(tt) * kTT + 16 * q + 2 * static_cast<int>(g));
      jrow = P.J + bj * P.rpitch + at;
      bstride = static_cast<int64_t>(P.F) * P.rpitch;
    }
    nbytes = static_cast<int>(max(int64_t(0), min(int64_t(4), P.rlen - at)));
    bytes = P.bytes != 0;
    blim = P.B - b0 - static_cast<int>(cb);              // beam offsets below this exist
  }

  // The J words of 8 beams (one chunk: beams 8 c + cb and 8 c + 4 + cb, four rows
  // each) from their accumulators and scaled gains.  What bounds the epilogue
  // is the issue rate and above all the integer pipe, so the arithmetic runs
  // two values to an instruction on the float pipe: acc = 2^-18 raw exactly;
  // x = (2^18 G) acc is one IEEE multiply, equal to G * raw (cpu.cxx:37); then
  // x 2^-149 + 8 2^-149 is rounded once, to a multiple of the smallest
  // subnormal, so its bit pattern is the integer lrint(x) + 8 (ties to even:
  // 8 is even), a large positive integer above the range and a negative one
  // below it.  The saturating pack clamps that to [0, 15] -- the nibble that
  // ucomplex4 stores (icomplex4.hxx:33) -- and the one value below the lower
  // clamp of cpu.cxx:38, nibble 0 (-8), becomes 1 (-7) for eight nibbles at once.
  // With a 4x4 byte transpose across lanes and scalar clamps and conversions
  // the epilogue took 86 instructions for 32 rows x 8 beams, now about 55:
  // full chunk 956 -> 886 us, wide array 812 -> 780 us, 128-problem batch
  // 376 -> 355 us (one-CTA kernel).
  template <bool kWide>
  __device__ __forceinline__ void words(const uint32_t (&r)[16], float g0, float g1, uint32_t (&w)[2]) const {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float gn = k ? g1 : g0;
      uint32_t x = 0;
      if constexpr (!kWide) {
        const uint64_t g2 = f32x2(__float_as_uint(gn), __float_as_uint(gn));
        const uint64_t tiny = f32x2(1u, 1u), eight = f32x2(8u, 8u);  // 2^-149 and 8 2^-149
#pragma unroll
        for (int j = 3; j >= 0; --j) {
          const int at = 4 * k + 2 * (j & 1) + 8 * (j >> 1);
          const uint64_t y = fma_f32x2(mul_f32x2(g2, f32x2(r[at], r[at + 1])), tiny, eight);
          x = pack_u4x2(static_cast<uint32_t>(y), static_cast<uint32_t>(y >> 32), x);
        }
        // bit 3 of a nibble of z: the nibble of x is zero
        const uint32_t z = ~(((x & 0x77777777u) + 0x77777777u) | x) & 0x88888888u;
        x += z >> 3;
      } else {
#pragma unroll
        for (int j = 3; j >= 0; --j) {
          const int at = 4 * k + 2 * (j & 1) + 8 * (j >> 1);
          x = pack_u4x2(static_cast<uint32_t>(requant_narrow(__fmul_rn(gn, __uint_as_float(r[at]))) + 8),
                        static_cast<uint32_t>(requant_narrow(__fmul_rn(gn, __uint_as_float(r[at + 1]))) + 8), x);
        }
      }
      w[k] = prmt(x, 0u, osel);
    }
  }

  // The fused adler32 sums of one tile: word h of the thread's chunk number cc
  // sits at byte position base + cc * step + h * half (mod 65521), so the tile
  // needs only a0 = sum of its bytes, a1 = sum cc * (bytes of chunk cc), a2 = sum
  // of the second words' bytes, a3 = sum k * byte_k within words; then
  // sum i d_i = base a0 + step a1 + half a2 + a3 (32-bit sums per tile:
  // bytes <= 255, at most 24 words; the products are taken in 64 bits).
  struct Sums {
    uint32_t a0 = 0, a1 = 0, a2 = 0, a3 = 0;
  };

  // Stores a chunk's words at dst (beam 8 c + cb) and counts them.  kFull: every
  // beam and time of the warp's share exists.
  template <bool kFull>
  __device__ __forceinline__ void put(uint8_t *dst, int c, int cc, const uint32_t (&w)[2], Sums &a) const {
    if constexpr (kFull) {
      __stcs(reinterpret_cast<uint32_t *>(dst), w[0]);
      __stcs(reinterpret_cast<uint32_t *>(dst + 4 * bstride), w[1]);
    } else if (!bytes) {  // rows are multiples of 4 bytes
      if (nbytes > 0 && 8 * c < blim) __stcs(reinterpret_cast<uint32_t *>(dst), w[0]);
      if (nbytes > 0 && 8 * c + 4 < blim) __stcs(reinterpret_cast<uint32_t *>(dst + 4 * bstride), w[1]);
    } else {
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < nbytes && 8 * c + 4 * k < blim) dst[4 * k * bstride + i] = static_cast<uint8_t>(w[k] >> (8 * i));
    }
    if constexpr (kAdler) {  // only the bytes stored count
      const uint32_t in = kFull || nbytes == 4 ? 0xFFFFFFFFu : (1u << (8 * nbytes)) - 1u;
      const uint32_t w0 = kFull || 8 * c < blim ? w[0] & in : 0u;
      const uint32_t w1 = kFull || 8 * c + 4 < blim ? w[1] & in : 0u;
      const uint32_t s1 = __dp4a(w1, 0x01010101u, 0u);
      const uint32_t s01 = __dp4a(w0, 0x01010101u, s1);
      a.a0 += s01;
      a.a1 += static_cast<uint32_t>(cc) * s01;
      a.a2 += s1;
      a.a3 = __dp4a(w1, 0x03020100u, __dp4a(w0, 0x03020100u, a.a3));
    }
  }

  __device__ __forceinline__ void add(const TcProblem &P, int c_begin, const Sums &a, unsigned long long &ad_s1,
                                      unsigned long long &ad_s2) const {
    if constexpr (kAdler) {
      const uint64_t off = static_cast<uint64_t>((jrow + static_cast<int64_t>(8 * c_begin) * bstride) - P.jbase);
      const uint32_t base = static_cast<uint32_t>(off % kAdlerMod);
      const uint32_t half = static_cast<uint32_t>(static_cast<uint64_t>(4 * bstride) % kAdlerMod);
      const uint32_t step = static_cast<uint32_t>(static_cast<uint64_t>(8 * bstride) % kAdlerMod);
      ad_s1 += a.a0;
      ad_s2 += static_cast<unsigned long long>(base) * a.a0 + static_cast<unsigned long long>(step) * a.a1 +
               static_cast<unsigned long long>(half) * a.a2 + a.a3;
    }
  }

  // Chunks [c_begin, c_end) of the accumulator at acc_addr, with up to kC loads
  // in flight at once: a tensor-memory load takes ~500 cycles beside a busy
  // tensor core, and the accumulator is free once the last one is in registers
  // (`release`).  `wait` waits for the accumulator.  The rare narrowing requantisation is a loop of its own: inlined
  // in every chunk its code (~300 instructions each) would push the epilogue
  // out of the instruction cache.
  template <int kC, class Wait, class Release>
  __device__ __forceinline__ bool run(const TcProblem &P, uint32_t acc_addr, int c_begin, int c_end,
                                      unsigned long long &ad_s1, unsigned long long &ad_s2, Wait wait,
                                      Release release) const {
    Sums a;
    bool ok;
    if (!wide) {
      ok = __all_sync(0xffffffffu, !bytes && nbytes == 4 && 8 * c_end - 4 < blim)
               ? chunks<kC, true>(acc_addr, c_begin, c_end, a, wait, release)
               : chunks<kC, false>(acc_addr, c_begin, c_end, a, wait, release);
    } else {
      ok = wait();
      uint8_t *dst = jrow + static_cast<int64_t>(8 * c_begin) * bstride;  // beam 8 c + cb of chunk c
#pragma unroll 1
      for (int c = c_begin; ok && c < c_end; ++c) {
        uint32_t r[16], w[2];
        tmem_ld_rows4_x2(acc_addr + 16u * c, r);
        tmem_ld_wait(r);
        words<true>(r, gcur[8 * c], gcur[8 * c + 4], w);
        put<false>(dst, c, c - c_begin, w, a);
        dst += 8 * bstride;
      }
      if (ok) release();
    }
    add(P, c_begin, a, ad_s1, ad_s2);
    return ok;
  }

  template <int kC, bool kFull, class Wait, class Release>
  __device__ __forceinline__ bool chunks(uint32_t acc_addr, int c_begin, int c_end, Sums &a, Wait &wait,
                                         Release &release) const {
    uint8_t *dst = jrow + static_cast<int64_t>(8 * c_begin) * bstride;  // beam 8 c + cb of chunk c
    if (!wait()) return false;
    int c = c_begin;
    for (; c + kC <= c_end; c += kC) {
      group<kC, kFull>(acc_addr, c, c_begin, dst, a, [&]() {
        if (c + kC == c_end) release();
      });
    }
    if constexpr (kC > 1) {
#pragma unroll 1
      for (; c < c_end; ++c) {
        group<1, kFull>(acc_addr, c, c_begin, dst, a, [&]() {
          if (c + 1 == c_end) release();
        });
      }
    }
    if (c_begin == c_end) release();
    return true;
  }

  // kC chunks from c: all their loads in flight, then `loaded`, then their words.
  template <int kC, bool kFull, class Loaded>
  __device__ __forceinline__ void group(uint32_t acc_addr, int c, int c_begin, uint8_t *&dst, Sums &a,
                                        Loaded loaded) const {
    uint32_t r[kC][16];
    float g[2 * kC];
#pragma unroll
    for (int i = 0; i < kC; ++i) tmem_ld_rows4_x2(acc_addr + 16u * (c + i), r[i]);
#pragma unroll
    for (int i = 0; i < kC; ++i) {
      g[2 * i] = gcur[8 * (c + i)];
      g[2 * i + 1] = gcur[8 * (c + i) + 4];
    }
#pragma unroll
    for (int i = 0; i < kC; ++i) tmem_ld_wait(r[i]);  // the first waits for all; each ties its registers to the wait
    loaded();
#pragma unroll
    for (int i = 0; i < kC; ++i) {
      uint32_t w[2];
      words<false>(r[i], g[2 * i], g[2 * i + 1], w);
      put<kFull>(dst, c + i, c + i - c_begin, w, a);
      dst += 8 * bstride;
    }
  }
};

// A warp's adler32 sums into the device sums: one pair of atomics.
__device__ __forceinline__ void add_adler(unsigned long long *sums, unsigned long long s1, unsigned long long s2,
                                          int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  if (lane == 0) {
    atomicAdd(sums, s1);
    atomicAdd(sums + 1, s2);
  }
}

}  // namespace
}  // namespace bf
