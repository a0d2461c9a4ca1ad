// bf_tc.cu -- the beamformer on the 5th-generation tensor cores (tcgen05).
//
// The complex sum of cpu.cxx:26-35 becomes one real GEMM per frequency:
//
//   rows    m = (t, p)      128 per tile: 64 times x 2 polarizations
//   columns n = (b, re|im)  2 * beams (<= 192 per pass)
//   depth   k = (d, re|im)  2 * dishes
//
//   [Jre]   [ Ar  -Ai ] [Ere]
//   [Jim] = [ Ai   Ar ] [Eim]      summed over d
//
// Operands are 8-bit floats (E4M3).  A byte holding an unsigned nibble u in
// [0, 15] is, read as E4M3, exactly u * 2^-9 (exponent field 0 or 1: the
// subnormal and the first normal binade share the step 2^-9).  So the raw
// ucomplex4 nibbles (value x stored as u = x + 8) become tensor-core operands
// with one AND per 4 values.  The offset goes into the accumulator with one extra
// MMA per tile (digit rows of the row sums of W times a constant tile, see
// kDigitScaleLo):
//
//   acc[n] = 2^-18 (-8 sum_k W[n][k] + sum_k u_k W[n][k])
//          = 2^-18 sum_k (u_k - 8) W[n][k] = 2^-18 raw
//
// W holds the integers Ar, -Ai, Ai in [-8, 8] in the same form, w * 2^-9 (a sign
// and the low nibble), or for wide passes w + 8 in [0, 16], when the extra MMA
// also takes off 8 sum_k u_k (see bf_prep_weights).  Every partial sum is an
// integer multiple of 2^-18 below 2^2 in magnitude (ndishes <= 2048: at most 20
// significant bits), exact in the f32 accumulator.  As normal numbers (w itself) the products are just
// as exact, but the codes' exponent bits toggle from column to column, and the
// chip runs at its power limit: the full chunk took 745 us with them, 719
// with subnormals (the wide array 743, 726; sustained).  The
// requantisation clamp(lrint(G * float(raw)), -7, 7) of cpu.cxx:37-39 is one
// IEEE multiply by 2^18 G (exactly G * raw) and a round-half-even step.
//
// Warp roles (one CTA per SM, persistent over tiles; warp numbers for the
// layout of 8 epilogue warps, 480 threads; with 12 epilogue warps, 608
// threads, the roles after the epilogue move up by four):
//   warps 0-7    epilogue: TMEM accumulator -> registers (four rows of a beam to a
//                thread) -> requantise (multiply, convert, saturating nibble pack)
//                -> 32-bit stores of 4 consecutive bytes of J
//   warp  8      E producer: TMA of raw E boxes into a deep ring released by the unpack
//   warp  9      TMEM allocator and MMA issuer (A operand from TMEM)
//   warp  10     W producer: TMA of each tile's digit rows and of the W slice of
//                each K stage, released by the MMA
//   warps 11-14  unpack (groups of four take K stages in turn): raw E bytes ->
//                de-interleaved E4M3 operand rows written straight into tensor
//                memory (tcgen05.st); no shared-memory operand
//
// It runs passes of at most 16 beams (two CTAs per SM), and wider ones only where
// the device has no room for a cluster of two SMs (bf_tc_pair.cu takes them).
//
// Launches with four or more unpacked stages in TMEM (beam passes of at most
// 64 beams) run two unpack groups, which take the stages in turn, and one more
// warp, the W forwarder: it arrives on a stage's a_full once that stage's W slot
// has landed, so the unpack warps carry no W hand-over, and the W producer
// reuses a slot as soon as the tensor core has finished the stage that used it.
//
// Which of the tile's 64 times and 2 polarizations a GEMM row (TMEM lane) holds:
// RowMap.  TMEM columns: accumulators at [0, N) and [256, 256 + N), unpacked
// E stages (64 columns = 256 K bytes each) in the remaining columns.
#include "bf_internal.h"
#include "bf_once.h"
#include "bf_tc_common.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <cudaTypedefs.h>

namespace bf {
namespace {

// Warp layout: kEpiWarps epilogue warps, the three single-thread roles, then
// kUnpackGroups groups of four unpack warps.  A warp reaches TMEM lanes
// 32 * (warp % 4) .. + 31 only, so every role that touches TMEM rows comes in
// fours covering the four lane quarters.  Twelve epilogue warps suit short K
// (ndishes <= 512: the epilogue paces the tiles), eight suit long K (the
// unpack does, and more epilogue warps take its issue slots).
template <int kEpiWarps_, int kUnpackGroups_>
struct Roles {
  static constexpr int kEpiWarps = kEpiWarps_;
  static constexpr int kUnpackGroups = kUnpackGroups_;
  static constexpr bool kForwarder = kUnpackGroups > 1;  // W-landed forwarder warp
  static constexpr int kEpiThreads = 32 * kEpiWarps;
  static constexpr int kEpiParts = kEpiWarps / 4;  // column parts: each read by four warps (one per lane quarter)
  static constexpr int kEProdWarp = kEpiWarps;
  static constexpr int kMmaWarp = kEpiWarps + 1;
  static constexpr int kWProdWarp = kEpiWarps + 2;
  static constexpr int kUnpackWarp0 = kEpiWarps + 3;
  static constexpr int kFwdWarp = kUnpackWarp0 + 4 * kUnpackGroups;
  static constexpr int kThreads = 32 * (kFwdWarp + (kForwarder ? 1 : 0));
};
constexpr int kAccCols = 256;           // TMEM column offset of the second accumulator
// Beam passes of at most kHalfPass beams run the half-SM layout: 4 epilogue
// warps, 256 TMEM columns (second accumulator at column 128) and at most
// kSmemLimitHalf bytes of shared memory, so that two CTAs share each SM and
// each SM has two MMA issuers, two unpack chains and two epilogues.
constexpr int kAccColsHalf = 128;
constexpr int kSmemLimitHalf = 115712;  // half of the SM's 228 KiB less the 1 KiB each block reserves
constexpr int kSmemLimit = 232448;      // 227 KiB opt-in per block
constexpr int kMaxStages = 8;
constexpr int kMaxWSlots = 6;
constexpr int kMinRaw = 4;
constexpr int kMaxRaw = 16;


struct TcParams {
  TcProblem one;            // the problem of a plain launch
  const TcProblem *table;   // grouped launch: nprob problems in device memory, by tile_begin
  int nprob;
  int ntiles;
  int nk;                   // K stages per tile (every problem has the same dishes)
  int max_nb_pass;          // sizes the W slots, gain buffers and TMEM layout
  int stages;               // unpacked-operand stages in TMEM
  int wslots;               // W slots in smem
  int raw;                  // raw E slots in smem
  int test_stall;           // nonzero: the producers issue nothing (failure-path test)
  int groups;               // unpack groups (2: with the W forwarder; needs stages >= 4)
  int half;                 // nonzero: the half-SM layout (two CTAs per SM)
  int *err;
};

// Tiles of a CTA.  A plain launch strides them over the grid.  A grouped
// launch gives each CTA a contiguous range, so that it stays with one problem
// for many tiles: every change of problem costs each role a tensor-map
// acquire and a cold descriptor, and with strided tiles almost every tile of
// a large batch belongs to another problem.
struct TileRange {
  int first, end, step;
  template <bool kGrouped>
  __device__ __forceinline__ static TileRange of(const TcParams &p) {
    if constexpr (kGrouped) {
      const int64_t n = p.ntiles, g = gridDim.x, b = blockIdx.x;
      return {static_cast<int>(b * n / g), static_cast<int>((b + 1) * n / g), 1};
    } else {
      return {static_cast<int>(blockIdx.x), p.ntiles, static_cast<int>(gridDim.x)};
    }
  }
  __device__ __forceinline__ uint32_t count() const {
    return first < end ? static_cast<uint32_t>((end - 1 - first) / step + 1) : 0u;
  }
};

// Problem of a tile and the tile's index inside it; a CTA's tiles only grow,
// so a grouped launch walks the table forward from the last problem seen.
template <bool kGrouped>
struct ProblemCursor {
  int idx = -1;
  __device__ __forceinline__ const TcProblem &at(const TcParams &p, int tile, int &lt) {
    if constexpr (!kGrouped) {
      lt = tile;
      return p.one;
    } else {
      if (idx < 0) {  // first tile: binary search
        int lo = 0, hi = p.nprob - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (p.table[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
        }
        idx = lo;
      }
      while (idx + 1 < p.nprob && p.table[idx + 1].tile_begin <= tile) ++idx;
      lt = tile - p.table[idx].tile_begin;
      return p.table[idx];
    }
  }
};

// Coordinates (beam pass, 64-time block, frequency) of a CTA's tiles.  A plain
// launch visits tiles blockIdx.x, + gridDim.x, ...: the cursor adds the grid
// size in the same mixed radix (npass, ntt, F) instead of dividing by the
// run-time sizes for every tile (two divisions cost ~40 instructions, and
// every role of the CTA pays them).  A grouped launch may change problem from
// one tile to the next, so it divides.
struct TileCursor {
  int pass = 0, tt = 0, f = 0;  // current tile (plain launches)
  int dp = 0, dt = 0, df = 0;   // gridDim.x in the same radix
  template <bool kGrouped>
  __device__ __forceinline__ void start(const TcParams &p) {
    if constexpr (!kGrouped) {
      const int np = p.one.npass, nt = p.one.ntt;
      const int b = static_cast<int>(blockIdx.x), g = static_cast<int>(gridDim.x);
      pass = b % np;
      tt = (b / np) % nt;
      f = b / (np * nt);
      dp = g % np;
      dt = (g / np) % nt;
      df = g / (np * nt);
    }
  }
  // Coordinates of tile lt of problem P; then steps to the CTA's next tile.
  template <bool kGrouped>
  __device__ __forceinline__ void take(const TcProblem &P, int lt, int &pass_, int &tt_, int &f_) {
    if constexpr (kGrouped) {
      pass_ = lt % P.npass;
      tt_ = (lt / P.npass) % P.ntt;
      f_ = lt / (P.npass * P.ntt);
    } else {
      pass_ = pass;
      tt_ = tt;
      f_ = f;
      pass += dp;
      int c = pass >= P.npass;
      pass -= c ? P.npass : 0;
      tt += dt + c;
      c = tt >= P.ntt;
      tt -= c ? P.ntt : 0;
      f += df + c;
    }
  }
};

struct SmemPlan {
  int wbox, wbytes, dbytes;
  int off_w, off_a, off_d, off_r, off_bar, nbar, total;
};

__host__ __device__ inline SmemPlan smem_plan(int stages, int wslots, int raw, int nb_pass) {
  SmemPlan s{};
  s.wbox = 2 * nb_pass * kKC;
  s.wbytes = kSub * s.wbox;
  s.dbytes = (2 * nb_pass * kDigitRow + 1023) / 1024 * 1024;
  s.off_w = 0;
  s.off_a = s.off_w + wslots * s.wbytes;  // constant A tile of the offset MMA
  s.off_d = s.off_a + 2 * kConstABytes;       // digit-row slots
  s.off_r = s.off_d + kDigSlots * s.dbytes;
  s.off_bar = s.off_r + raw * kRawBytes;
  // raw_full[R], raw_empty[R], w_full[SW], w_empty[SW], a_full[S], empty[S], accfull[2], accempty[2],
  // d_full[2], d_empty[2], rs_full[2]
  s.nbar = 2 * raw + 2 * wslots + 2 * stages + 4 + 2 * kDigSlots + 2;
  s.total = s.off_bar + 8 * s.nbar + 16;
  return s;
}

// TMEM column of unpacked stage i: the columns left over after the two accumulators.
__host__ __device__ inline uint32_t stage_col(int i, int ncols, int per_half, int acc_cols) {
  return i < per_half ? static_cast<uint32_t>(ncols + kStageCols * i)
                      : static_cast<uint32_t>(acc_cols + ncols + kStageCols * (i - per_half));
}

template <bool kGrouped, bool kJ2, int kEpiW, bool kAdler, int kGroups, bool kHalf>
__global__ void __launch_bounds__(Roles<kEpiW, kGroups>::kThreads, kHalf ? 2 : 1)
    bf_form_beams_tc(const __grid_constant__ TcParams p) {
  using RL = Roles<kEpiW, kGroups>;
  constexpr int kAcc = kHalf ? kAccColsHalf : kAccCols;  // TMEM column of the second accumulator
  constexpr int kEpiThreads = RL::kEpiThreads, kEpiParts = RL::kEpiParts, kEProdWarp = RL::kEProdWarp;
  constexpr int kMmaWarp = RL::kMmaWarp, kWProdWarp = RL::kWProdWarp, kUnpackWarp0 = RL::kUnpackWarp0;
  constexpr int kUnpackGroups = RL::kUnpackGroups;
  constexpr bool kSums = !kHalf;  // passes of the half-SM layout are too narrow for W + 8 (tc_w_offset)
  extern __shared__ uint8_t smem_dyn[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  const int S = p.stages, SW = p.wslots, R = p.raw;
  const SmemPlan sp = smem_plan(S, SW, R, p.max_nb_pass);
  uint8_t *sW = smem + sp.off_w;
  uint8_t *sA = smem + sp.off_a;
  uint8_t *sD = smem + sp.off_d;
  uint8_t *sR = smem + sp.off_r;
  const uint32_t bar0 = smem_u32(smem + sp.off_bar);
  auto raw_full = [&](int r) { return bar0 + 8u * r; };
  auto raw_empty = [&](int r) { return bar0 + 8u * (R + r); };
  auto w_full = [&](int s) { return bar0 + 8u * (2 * R + s); };
  auto w_empty = [&](int s) { return bar0 + 8u * (2 * R + SW + s); };
  auto a_full = [&](int s) { return bar0 + 8u * (2 * R + 2 * SW + s); };
  auto empty = [&](int s) { return bar0 + 8u * (2 * R + 2 * SW + S + s); };
  auto accfull = [&](int i) { return bar0 + 8u * (2 * R + 2 * SW + 2 * S + i); };
  auto accempty = [&](int i) { return bar0 + 8u * (2 * R + 2 * SW + 2 * S + 2 + i); };
  auto d_full = [&](int i) { return bar0 + 8u * (2 * R + 2 * SW + 2 * S + 4 + i); };
  auto d_empty = [&](int i) { return bar0 + 8u * (2 * R + 2 * SW + 2 * S + 4 + kDigSlots + i); };
  auto rs_full = [&](int i) { return bar0 + 8u * (2 * R + 2 * SW + 2 * S + 4 + 2 * kDigSlots + i); };
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(smem + sp.off_bar + 8 * sp.nbar);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // known to be warp-uniform
  const int lane = threadIdx.x & 31;
  const int ncols = 2 * p.max_nb_pass;                 // accumulator columns reserved (largest GEMM N)
  const int per_half = (kAcc - ncols) / kStageCols;  // unpacked stages beside each accumulator

  // Each producer sets up its own barriers and starts its copies at once; the
  // other warps meet while those are under way.
  if (warp == kEProdWarp) {
    for (int i = lane; i < 2 * R; i += 32) mbar_init(raw_full(i), i < R ? 1 : 128);
    if (!kGrouped && lane == 0) tma_prefetch_desc(&p.one.tm_e);
  } else if (warp == kWProdWarp) {
    for (int i = lane; i < 2 * SW; i += 32) mbar_init(w_full(i), 1);
    if (lane < 2 * kDigSlots) mbar_init(d_full(lane), 1);
    if (!kGrouped && lane == 0) {
      tma_prefetch_desc(&p.one.tm_w);
      tma_prefetch_desc(&p.one.tm_d);
    }
  } else if (warp == 0) {
    if (lane < 2 * S) mbar_init(a_full(lane), lane < S ? 128 + (RL::kForwarder ? 1 : 0) : 1);  // one group (+ forwarder)
    if (lane < 4) mbar_init(accfull(lane), lane < 2 ? 1 : kEpiThreads);
    if (lane < 2) mbar_init(rs_full(lane), 4 * kUnpackGroups);
  }
  static_assert(2 * kMaxStages <= 32, "one lane per stage barrier");
  fence_barrier_init();
  __syncwarp();  // a producer's lane 0 uses barriers that its other lanes set up, and waits for no other warp
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(tmem_holder), 2 * kAcc);
    tmem_relinquish();
  }
  fill_offset_tiles<kSums ? 2 : 1>(sA);
  fence_proxy_async_smem();
  grid_launch_next();
  grid_wait();
  tc_fence_before();
  if (warp == kEProdWarp || warp == kWProdWarp)
    cta_arrive(RL::kThreads);
  else
    cta_sync(RL::kThreads);
  tc_fence_after();
  const uint32_t tmem_base = warp == kEProdWarp || warp == kWProdWarp ? 0u : *tmem_holder;  // the producers need none
  int *err = p.err;

  if (warp == kEProdWarp) {
    // ------------------------------------------------------------ E producer
    if (lane == 0 && !p.test_stall) {
      const uint64_t pol_e = policy_evict_first();
      Ring rr(R);
      uint32_t issued = 0;
      bool ok = true;
      const TcProblem *seen = nullptr;
      TileCursor cur;
      cur.start<kGrouped>(p);
      const TileRange tr = TileRange::of<kGrouped>(p);
      ProblemCursor<kGrouped> pc;
      for (int tile = tr.first; ok && tile < tr.end; tile += tr.step) {
        int lt;
        const TcProblem &P = pc.at(p, tile, lt);
        if (kGrouped && &P != seen) {  // a table entry the host rewrites between launches
          tensormap_acquire(&P.tm_e);
          seen = &P;
        }
        int pass, tt, f;
        cur.take<kGrouped>(P, lt, pass, tt, f);
        (void)pass;
        for (int ks = 0; ks < p.nk; ++ks, rr.advance(), ++issued) {
          const int r = static_cast<int>(rr.idx);
          if (!mbar_wait(raw_empty(r), rr.phase ^ 1u, err, kDevTimeoutEmpty)) {
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(raw_full(r), kRawBytes);
#pragma unroll
          for (int h = 0; h < kSub; ++h)
            tma_load_3d(smem_u32(sR + r * kRawBytes + h * kRawBox), &P.tm_e, raw_full(r), (ks * kSub + h) * kKC, f,
                        tt * kTT, pol_e);
        }
      }
      // Let the copies already issued land before the CTA exits.  Also when
      // this thread saw no error: another role's error can end the consumers
      // before they waited for the last copies.  On a clean run these waits
      // return at once.
      for (uint32_t k = (issued >= static_cast<uint32_t>(R) ? issued - R : 0); k < issued; ++k)
        mbar_wait_drain(raw_full(static_cast<int>(k % R)), (k / R) & 1u);
    }
  } else if (warp == kWProdWarp) {
    // ------------------------------------------------------------ W producer
    if (lane == 0 && !p.test_stall) {
      const uint64_t pol_w = policy_evict_last();
      Ring wr(SW), dr(kDigSlots);
      uint32_t it = 0, dit = 0;
      bool ok = true;
      const TcProblem *seen = nullptr;
      TileCursor cur;
      cur.start<kGrouped>(p);
      const TileRange tr = TileRange::of<kGrouped>(p);
      ProblemCursor<kGrouped> pc;
      for (int tile = tr.first; ok && tile < tr.end; tile += tr.step) {
        int lt;
        const TcProblem &P = pc.at(p, tile, lt);
        if (kGrouped && &P != seen) {  // a table entry the host rewrites between launches
          tensormap_acquire(&P.tm_w);
          tensormap_acquire(&P.tm_d);
          seen = &P;
        }
        int pass, tt, f;
        cur.take<kGrouped>(P, lt, pass, tt, f);
        (void)tt;
        const int wbox = 2 * P.nb_pass * kKC;
        {  // the tile's digit rows, for the offset MMA
          const int ds = static_cast<int>(dr.idx);
          if (!mbar_wait(d_empty(ds), dr.phase ^ 1u, err, kDevTimeoutEmpty)) {
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(d_full(ds), 2 * P.nb_pass * kDigitRow);
          tma_load_3d(smem_u32(sD + ds * sp.dbytes), &P.tm_d, d_full(ds), 0, pass * 2 * P.nb_pass, f, pol_w);
          dr.advance();
          ++dit;
        }
        for (int ks = 0; ks < p.nk; ++ks, ++it, wr.advance()) {
          const int s = static_cast<int>(wr.idx);
          if constexpr (RL::kForwarder) {
            // the slot held sequence it - SW: free once the tensor core finished
            // that stage (its commit on empty).  SW <= S, so the stage's next use
            // (sequence it - SW + S) is not loaded yet and the barrier cannot be a
            // phase past the one waited for.
            if (it >= static_cast<uint32_t>(SW)) {
              const uint32_t j = it - static_cast<uint32_t>(SW);
              if (!mbar_wait(empty(static_cast<int>(j % static_cast<uint32_t>(S))), (j / static_cast<uint32_t>(S)) & 1u,
                             err, kDevTimeoutEmpty)) {
                ok = false;
                break;
              }
            }
          } else if (!mbar_wait(w_empty(s), wr.phase ^ 1u, err, kDevTimeoutEmpty)) {
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(w_full(s), kSub * wbox);
#pragma unroll
          for (int h = 0; h < kSub; ++h)
            tma_load_3d(smem_u32(sW + s * sp.wbytes + h * wbox), &P.tm_w, w_full(s), (ks * kSub + h) * kKC,
                        pass * 2 * P.nb_pass, f, pol_w);
        }
      }
      // as in the E producer: drain on every exit, not only after an own error
      for (uint32_t k = (it >= static_cast<uint32_t>(SW) ? it - SW : 0); k < it; ++k)
        mbar_wait_drain(w_full(static_cast<int>(k % SW)), (k / SW) & 1u);
      for (uint32_t k = (dit >= static_cast<uint32_t>(kDigSlots) ? dit - kDigSlots : 0); k < dit; ++k)
        mbar_wait_drain(d_full(static_cast<int>(k % kDigSlots)), (k / kDigSlots) & 1u);
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMA issuer
    // The whole warp runs the loop and waits together; one elected lane issues.
    // Kept warp-uniform, the descriptors, the stage addresses and the loop live
    // in uniform registers, which is where tcgen05.mma takes them from.  Inside
    // a single-lane branch every operand of every MMA was moved there first: a
    // stage of 8 MMAs then cost 401 cycles at N <= 64 without commit and wait
    // and 715 with them, against 163 / 257 (N = 32 / 64, the tensor core's own
    // 128 / 256) and 309 / 365 in this form (152 SMs, 400 stages, clock64).
    {
      Ring ar(S), wr(SW), dr(kDigSlots);
      const uint64_t a_off = smem_desc_sw32(smem_u32(sA));
      const uint64_t w_desc0 = smem_desc_sw128(smem_u32(sW));
      uint32_t local = 0;
      uint32_t nstage = 0, ndig = 0, nacc = 0;  // commits issued on empty, d_empty, accfull
      bool ok = true;
      const TileRange tr = TileRange::of<kGrouped>(p);
      ProblemCursor<kGrouped> pc;
      for (int tile = tr.first; ok && tile < tr.end; tile += tr.step, ++local) {
        int lt;
        const TcProblem &P = pc.at(p, tile, lt);
        const uint32_t idesc = idesc_e4m3_f32(kBM, 2 * P.nb_pass);
        const int wbox = 2 * P.nb_pass * kKC;
        const uint32_t ab = local & 1u;
        const uint32_t aph = (local >> 1) & 1u;
        if (!__all_sync(0xffffffffu, mbar_wait(accempty(ab), aph ^ 1u, err, kDevTimeoutAccEmpty))) break;
        const int ds = static_cast<int>(dr.idx);
        if (!__all_sync(0xffffffffu, mbar_wait(d_full(ds), dr.phase, err, kDevTimeoutFull))) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + ab * kAcc;
        // the offset MMA: -8 sum_k W[n][k] 2^-18, with the row sums also
        // -8 sum_k u[m][k] 2^-18, which are there last
        auto offset_mma = [&]() {
          mma_f8f6f4(d_tmem, a_off + (kSums ? ab * (kConstABytes >> 4) : 0u), smem_desc_sw32(smem_u32(sD + ds * sp.dbytes)), idesc,
                     kSums ? 1u : 0u);
          mma_commit(d_empty(ds));
        };
        if constexpr (!kSums) {
          if (elect_one()) offset_mma();
          ++ndig;  // with its commit: the tile may end early
        }
        __syncwarp();
        for (int ks = 0; ks < p.nk; ++ks, ar.advance(), wr.advance()) {
          const int s = static_cast<int>(ar.idx);
          const int sw = static_cast<int>(wr.idx);
          // the unpack arrives on a_full only once this stage's W slot has landed too
          if (!__all_sync(0xffffffffu, mbar_wait(a_full(s), ar.phase, err, kDevTimeoutUnpacked))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_tmem = tmem_base + stage_col(s, ncols, per_half, kAcc);
          const uint64_t b_desc = w_desc0 + static_cast<uint64_t>((sw * sp.wbytes) >> 4);
          if (elect_one()) {
            mma_ts_stage8(d_tmem, a_tmem, b_desc, b_desc + static_cast<uint64_t>(wbox >> 4), idesc, !kSums || ks > 0);
            mma_commit(empty(s));  // also frees the W slot: the unpack passes it on
          }
          __syncwarp();
          ++nstage;
        }
        if (!ok) break;
        if constexpr (kSums) {
          if (!__all_sync(0xffffffffu, mbar_wait(rs_full(ab), aph, err, kDevTimeoutUnpacked))) break;
          tc_fence_after();
        }
        if constexpr (kSums) {
          if (elect_one()) offset_mma();
          ++ndig;
        }
        if (elect_one()) mma_commit(accfull(ab));
        __syncwarp();
        dr.advance();
        ++nacc;
      }
      // A commit's arrival is an asynchronous write into this CTA's shared
      // memory, and nothing waits for the last ones on each stage and digit
      // slot: wait for the last phase committed on every barrier (bounded)
      // before the CTA can exit.  On the error path this also lets the MMAs
      // already issued finish before the tensor memory is freed.
      const uint32_t uS = static_cast<uint32_t>(S), uD = static_cast<uint32_t>(kDigSlots);
      for (uint32_t k = nstage > uS ? nstage - uS : 0; k < nstage; ++k)
        mbar_wait_drain(empty(static_cast<int>(k % uS)), (k / uS) & 1u);
      for (uint32_t k = ndig > uD ? ndig - uD : 0; k < ndig; ++k)
        mbar_wait_drain(d_empty(static_cast<int>(k % uD)), (k / uD) & 1u);
      for (uint32_t k = nacc > 2u ? nacc - 2u : 0u; k < nacc; ++k)
        mbar_wait_drain(accfull(static_cast<int>(k & 1u)), (k >> 1) & 1u);
      __syncwarp();
    }
  } else if (RL::kForwarder && warp == RL::kFwdWarp) {
    // ------------------------------------------------------------ W forwarder
    // Sequence it's a_full gets one arrival from here once its W slot has
    // landed, after the previous use of that a_full slot (it - S) completed.
    if (lane == 0 && !p.test_stall) {
      const uint32_t total = TileRange::of<kGrouped>(p).count() * static_cast<uint32_t>(p.nk);
      const uint32_t uS = static_cast<uint32_t>(S), uSW = static_cast<uint32_t>(SW);
      for (uint32_t it = 0; it < total; ++it) {
        if (!mbar_wait(w_full(static_cast<int>(it % uSW)), (it / uSW) & 1u, err, kDevTimeoutFull)) break;
        if (it >= uS &&
            !mbar_wait(a_full(static_cast<int>((it - uS) % uS)), ((it - uS) / uS) & 1u, err, kDevTimeoutUnpacked))
          break;
        mbar_arrive(a_full(static_cast<int>(it % uS)));
      }
    }
  } else if (warp >= kUnpackWarp0) {
    // ------------------------------------------------------------ unpack
    // Group g takes the K stages with it % kUnpackGroups == g.  Each lane fills
    // one GEMM row: it reads the raw row of its time, which holds both
    // polarizations, and keeps its own (RowMap).
    const int group = (warp - kUnpackWarp0) >> 2;
    const int q = warp & 3;
    const uint32_t pp = RowMap<kJ2>::pol(q, lane);
    const uint32_t tl = RowMap<kJ2>::time(q, lane);
    const uint32_t lane_addr = static_cast<uint32_t>(32 * q) << 16;
    const UnpackRow row(tl);
    const uint32_t sel = pp ? 0x7531u : 0x6420u;  // odd or even bytes: polarization 1 or 0
    // this CTA's K stages: its tiles (TileRange) times nk
    const uint32_t my_tiles = TileRange::of<kGrouped>(p).count();
    const uint32_t total = my_tiles * static_cast<uint32_t>(p.nk);
    // W slots: the tensor core's release of an operand stage (empty) also ends
    // its use of that stage's W slot, so the lead lane of the group handling
    // sequence it frees the W slot of sequence it - S when it sees the stage
    // free, and waits for the W slot of sequence it before its a_full arrival.
    // With SW >= S (the planner's rule) the releases of each slot come in
    // order for any number of groups: the release of sequence j precedes the
    // a_full arrival of j + S, and the next use of its slot, j + SW, is
    // released only after the tensor core consumed j + SW >= j + S.
    const bool wlead = warp == kUnpackWarp0 + 4 * group && lane == 0;
    Ring rr(R), ar(S), wr(SW);
    int relslot = ((group - S) % SW + SW) % SW;  // W slot of sequence it - S
    for (int g = 0; g < group; ++g) {
      rr.advance();
      ar.advance();
      wr.advance();
    }
    RowSums rs(sA, group, group, 32 * q + lane);
    auto rs_free = [&](int tile) {
      return __all_sync(0xffffffffu, mbar_wait(accfull(tile & 1), ((tile >> 1) & 1) ^ 1, err, kDevTimeoutAccFull));
    };
    auto rs_arrive = [&](int tile) {
      if (lane == 0) mbar_arrive(rs_full(tile & 1));
    };
    bool ok = !kSums || rs.settle(p.nk, static_cast<int>(my_tiles), rs_free, rs_arrive);
    for (uint32_t it = group; ok && it < total; it += kUnpackGroups) {
      {
        const int r = static_cast<int>(rr.idx);
        const int s = static_cast<int>(ar.idx);
        if (!__all_sync(0xffffffffu, mbar_wait(raw_full(r), rr.phase, err, kDevTimeoutFull))) {
          ok = false;  // the warp leaves together
          break;
        }
        const uint32_t col = tmem_base + lane_addr + stage_col(s, ncols, per_half, kAcc);
        // the whole stage goes to registers first, so that only the tensor-memory
        // stores wait for the tensor core to release the stage
        uint32_t out[kSub][32];
#pragma unroll
        for (int h = 0; h < kSub; ++h) rs.sum += unpack_box<kSums>(smem_u32(sR) + r * kRawBytes + h * kRawBox, row, sel, out[h]);
        // the raw slot is in registers now; the next TMA into it is an async-proxy
        // write after these generic reads, so order them across proxies first
        fence_proxy_async_smem();
        mbar_arrive(raw_empty(r));
        if (!__all_sync(0xffffffffu, mbar_wait(empty(s), ar.phase ^ 1u, err, kDevTimeoutEmpty))) {
          ok = false;
          break;
        }
        // the stores first: the W-slot hand-over runs while they drain
#pragma unroll
        for (int h = 0; h < kSub; ++h) tmem_st_32x32b_x32(col + 32 * h, out[h]);
        if constexpr (!RL::kForwarder) {
          if (it >= static_cast<uint32_t>(S) && wlead) mbar_arrive(w_empty(relslot));  // sequence it - S is done
          if (wlead && !mbar_wait(w_full(static_cast<int>(wr.idx)), wr.phase, err, kDevTimeoutFull)) ok = false;
        }
        tmem_st_wait();
        if (!__all_sync(0xffffffffu, ok)) break;
        tc_fence_before();
        mbar_arrive(a_full(s));
        if constexpr (kSums) {
          rs.kpos += kUnpackGroups;
          ok = rs.settle(p.nk, static_cast<int>(my_tiles), rs_free, rs_arrive);
        }
      }
#pragma unroll
      for (int g = 0; g < kUnpackGroups; ++g) {
        rr.advance();
        ar.advance();
        wr.advance();
        relslot = relslot + 1 == SW ? 0 : relslot + 1;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // Warp w reads TMEM lane quarter w % 4 and column part w / 4.
    const int q = warp & 3;
    const int part = warp >> 2;
    const uint32_t lane_addr = static_cast<uint32_t>(32 * q) << 16;

    // The warps of the epilogue share no barrier: each reads its chunks' gains
    // straight from the scaled-gain rows gs = 2^18 G (L1-resident) and waits for
    // the accumulator on its own, so a slow warp does not hold up the others.
    uint32_t local = 0;
    // fused adler32 (kAdler): this lane's sums of the J bytes it stores,
    // sum d_i and sum i d_i with the byte position i taken mod 65521
    unsigned long long ad_s1 = 0, ad_s2 = 0;
    TileCursor cur;
    cur.start<kGrouped>(p);
    const TileRange tr = TileRange::of<kGrouped>(p);
    ProblemCursor<kGrouped> pc;
    for (int tile = tr.first; tile < tr.end; tile += tr.step, ++local) {
      int lt;
      const TcProblem &P = pc.at(p, tile, lt);
      int pass, tt, f;
      cur.take<kGrouped>(P, lt, pass, tt, f);
      const uint32_t ab = local & 1u;
      const uint32_t aph = (local >> 1) & 1u;
      const EpilogueTile<kJ2, kAdler> et(P, f, pass, tt, q, lane);
      const int nchunk = P.nb_pass / 8;
      const bool ok = et.template run<2>(
          P, tmem_base + ab * kAcc + lane_addr, part * nchunk / kEpiParts, (part + 1) * nchunk / kEpiParts, ad_s1, ad_s2,
          [&]() {
            const bool full = __all_sync(0xffffffffu, mbar_wait(accfull(ab), aph, err, kDevTimeoutAccFull));
            tc_fence_after();
            return full;
          },
          [&]() {
            tc_fence_before();
            mbar_arrive(accempty(ab));
          });
      if (!ok) break;
    }
    if constexpr (kAdler) add_adler(p.one.adler, ad_s1, ad_s2, lane);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(*tmem_holder, 2 * kAcc);
  }
}

// The E4M3 codes of v * 2^-9 (a sign bit and |v|) of four stored nibbles u = v + 8.
__device__ __forceinline__ uint32_t w_codes(uint32_t u) {
  const uint32_t x = u ^ 0x08080808u;                // two's complement nibbles
  const uint32_t n = (x >> 3) & 0x01010101u;         // 1 where negative
  return ((x ^ (n * 15u)) + n) | (n << 7);           // 15 - x + 1 there
}
__device__ __forceinline__ uint32_t w_negate(uint32_t codes) {  // zero stays zero
  return codes ^ (((codes & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) & 0x80808080u);
}

// Builds the E4M3 operand W[f][n][k] and the digit rows of the row sums
// sum_k W[f][n][k] from A[f][b][d].
//   n = 2*b + cj                   (cj: 0 = real output, 1 = imaginary output)
//   k = 8*(d/4)  + 4*c  + d%4      (c:  0 = real input,  1 = imaginary input)
// W = Ar, -Ai for the real output and Ai, Ar for the imaginary output, stored as
// E4M3 (W + 8) * 2^-9, all codes 0..16.  The accumulator is then too large by
// 8 sum_k u_k in every column of a row, which the unpack sums and the offset MMA
// takes off (RowSums).  Signed codes are as exact and need no sums, but the
// chip runs at its power limit and operands whose sign changes from column to
// column cost the most of it: the full chunk (f=84 t=32768 b=96 d=512) took 716 us
// with them and 661 so, at 1.40 and 1.63 GHz; the wide array 731 and 690.
//
// One warp per beam: both of its rows hold the same numbers, so a lane turns 16
// dishes into the codes of Ar, Ai and -Ai four bytes at a time and stores 32
// bytes of each row.  Bound by the bytes of W (f=16 b=512 d=1024: 33.5 MB and
// 8.4 MB of A); a warp per row and a byte per load took 42 us there, this 14.4
// (f=16 b=96 d=512: 9.1 and 4.5 us, launch included).
constexpr int kPrepBeams = 8;  // beams per 256-thread block

template <bool kOffset, bool kCopy>
__global__ void __launch_bounds__(32 * kPrepBeams) bf_prep_weights(const uint8_t *A,
                                                                    uint8_t *__restrict__ W,
                                                                    uint8_t *__restrict__ dig,
                                                                    const float *G, float *__restrict__ gs,
                                                                    int *__restrict__ gwide, int B, int D, int Dk,
                                                                    int nw, int nw_pad, int a_layout,
                                                                    unsigned long long *adler,
                                                                    uint8_t *__restrict__ A_copy,
                                                                    float *__restrict__ G_copy) {
  grid_launch_next();
  grid_wait();
  if (adler && blockIdx.x == 0 && threadIdx.x < 2) adler[threadIdx.x] = 0;
  const int beams = nw_pad / 2;
  const int fblocks = (beams + kPrepBeams - 1) / kPrepBeams;  // blocks per frequency
  const int f = static_cast<int>(blockIdx.x) / fblocks;
  const int b = (static_cast<int>(blockIdx.x) % fblocks) * kPrepBeams + static_cast<int>(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (static_cast<int>(blockIdx.x) % fblocks == 0) {  // the frequency's scaled gains: 2^18 G, zero past B
    // |raw| <= 128 D, so with |G| * 128 D < 2^30 every product G * raw stays
    // below 2^31 and the plain requantisation is exact; otherwise (or for a
    // non-finite gain) the frequency takes the narrowing one of cpu.cxx:38
    const float wide_at = 1073741824.0f / (128.0f * static_cast<float>(D));
    int wide = 0;
    for (int i = threadIdx.x; i < beams; i += blockDim.x) {
      const float g = i < B ? G[static_cast<int64_t>(f) * B + i] : 0.0f;
      if (kCopy && G_copy && i < B) G_copy[static_cast<int64_t>(f) * B + i] = g;
      gs[static_cast<int64_t>(f) * beams + i] = 262144.0f * g;
      wide |= !(fabsf(g) < wide_at);
    }
    wide = __syncthreads_or(wide);
    if (threadIdx.x == 0) gwide[f] = wide;
  }
  if (b >= beams) return;  // the whole warp
  int s_re = 0, s_im = 0;  // sums of Ar and Ai
  if (b < nw / 2) {
    const uint8_t *row = A + (static_cast<int64_t>(f) * B + b) * D;  // linear layout
    const bool vec = a_layout == kALinear && b < B && D % 16 == 0 && (reinterpret_cast<uintptr_t>(A) & 15u) == 0;
    // rows 2 b and 2 b + 1 of 2 Dk bytes, Dk a multiple of 8: 16-byte aligned
    uint4 *w0 = reinterpret_cast<uint4 *>(W + (static_cast<int64_t>(f) * nw + 2 * b) * (2 * Dk));
    uint4 *w1 = w0 + Dk / 8;
    for (int i = lane; i < (Dk + 15) / 16; i += 32) {  // dishes 16 i .. 16 i + 15
      uint32_t w[4];
      if (vec) {
        const uint4 q = reinterpret_cast<const uint4 *>(row)[i];
        w[0] = q.x, w[1] = q.y, w[2] = q.z, w[3] = q.w;
        if (kCopy && A_copy) reinterpret_cast<uint4 *>(A_copy + (static_cast<int64_t>(f) * B + b) * D)[i] = q;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          w[j] = 0;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int d = 16 * i + 4 * j + k;
            int re = 0, im = 0;
            if (b < B && d < D) load_a(A, a_layout, f, b, d, B, D, re, im);
            const uint32_t byte = static_cast<uint32_t>(((re + 8) << 4) | (im + 8));  // as stored
            w[j] |= byte << (8 * k);
            if (kCopy && A_copy && b < B && d < D)
              A_copy[(static_cast<int64_t>(f) * B + b) * D + d] = static_cast<uint8_t>(byte);
          }
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // 8 dishes: 16 bytes of each row
        if (16 * i + 8 * h >= Dk) break;
        uint32_t re[2], im[2], ni[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t ur = (w[2 * h + j] >> 4) & 0x0F0F0F0Fu, ui = w[2 * h + j] & 0x0F0F0F0Fu;
          s_re += static_cast<int>(__dp4a(ur, 0x01010101u, 0u)) - 32;
          s_im += static_cast<int>(__dp4a(ui, 0x01010101u, 0u)) - 32;
          if constexpr (kOffset) {  // the stored nibbles are Ar + 8 and Ai + 8
            re[j] = ur;
            im[j] = ui;
            ni[j] = 0x10101010u - ui;
          } else {
            re[j] = w_codes(ur);
            im[j] = w_codes(ui);
            ni[j] = w_negate(im[j]);
          }
        }
        w0[2 * i + h] = make_uint4(re[0], ni[0], re[1], ni[1]);
        w1[2 * i + h] = make_uint4(im[0], re[0], im[1], re[1]);
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s_re += __shfl_xor_sync(0xffffffffu, s_re, o);
    s_im += __shfl_xor_sync(0xffffffffu, s_im, o);
  }
  if (lane < 2) {  // row 2 b + lane
    // s = sum_k W[n][k], |s| <= 16 D <= 2^15, in balanced base-16 digits
    // d0..d3 in [-8, 7] and d4 in {-1, 0, 1}; the digit row holds the E4M3
    // codes of d0, d1, d2, d3, 4 d4 (see kDigitScaleLo)
    uint32_t d03 = 0;
    int rest = lane == 0 ? s_re - s_im : s_im + s_re;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = rest & 15;
      const int dj = r >= 8 ? r - 16 : r;
      rest = (rest - dj) >> 4;
      const int av = dj < 0 ? -dj : dj;
      d03 |= static_cast<uint32_t>(av | (dj < 0 ? 0x80 : 0x00)) << (8 * j);
    }
    const uint32_t d4 = rest == 0 ? 0u : (rest > 0 ? 0x04u : 0x84u);  // 4 * d4: +-4 or 0
    uint4 *row = reinterpret_cast<uint4 *>(dig + (static_cast<int64_t>(f) * nw_pad + 2 * b + lane) * kDigitRow);
    row[0] = make_uint4(d03, d4, kOffset ? kDigitScaleLo : 0u, kOffset ? kDigitScaleLo : 0u);
    row[1] = make_uint4(0u, 0u, 0u, 0u);
  }
}
static_assert(kDigitRow == 32, "two 16-byte stores per digit row");

PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn() {
  // initialised once, thread-safely (the server thread encodes maps too)
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
    return nullptr;
  }();
  return fn;
}

bool make_map(CUtensorMap *m, const void *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides,
              const cuuint32_t *box, CUtensorMapSwizzle swz) {
  auto fn = get_encode_fn();
  if (!fn) return false;
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, const_cast<void *>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

int g_test_stall = 0;
std::atomic<int> g_test_one_cta{0};

}  // namespace

int num_sms() {
  static AskedOnce<int> asked;
  int n = 1;
  (void)asked.get(&n, [](int *k) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    return e != cudaSuccess ? e : cudaDeviceGetAttribute(k, cudaDevAttrMultiProcessorCount, dev);
  });
  return n;
}

void tc_set_test_stall(int on) { g_test_stall = on; }
void tc_set_test_one_cta(int on) { g_test_one_cta.store(on); }

void tc_plan_beams(int64_t B, int *nb_pass, int *npass, int granule) {
  // at most 96 beams (192 accumulator columns) per pass, so that two
  // accumulators and at least two unpacked stages fit the 512 TMEM columns;
  // several passes are balanced in steps of `granule` beams
  const int64_t b8 = (B + 7) / 8 * 8;
  const int64_t np = (b8 + 95) / 96;
  const int64_t nbp = np == 1 ? b8 : ((b8 + np - 1) / np + granule - 1) / granule * granule;
  *nb_pass = static_cast<int>(nbp);
  *npass = static_cast<int>((b8 + nbp - 1) / nbp);
}

bool tc_supported(const bf_dims &d) {
  if (d.npolarizations != 2) return false;
  if (d.ndishes <= 0 || d.ndishes % 8 != 0) return false;  // TMA row strides: 2*D multiple of 16 bytes
  if (d.ntimes <= 0 || d.ntimes % 16 != 0) return false;   // TMA store row strides: T multiple of 16 bytes
  if (d.nbeams <= 0 || d.nfrequencies <= 0) return false;
  // ndishes <= 2048 keeps |sum_k W[n][k]| <= 2^15, the range of the offset-correction digits
  if (d.ntimes > (1ll << 31) || d.nfrequencies > (1 << 20) || d.nbeams > (1 << 16) || d.ndishes > 2048)
    return false;
  return true;
}

// 16 bytes of E from byte `off`, `valid` of them (the rest 0).  Unaligned words
// where all of them lie inside the array, else byte by byte.
__device__ __forceinline__ uint4 load16_any(const uint8_t *E, int64_t off, int valid, int64_t avail) {
  uint32_t w[4];
  if (valid >= 16 && off >= 4 && off + 20 <= avail) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(E + off);
    const uint32_t *p = reinterpret_cast<const uint32_t *>(at & ~uintptr_t(3));
    const uint32_t sh = 8u * static_cast<uint32_t>(at & 3u);
    uint32_t v[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) v[i] = p[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __funnelshift_r(v[i], v[i + 1], sh);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w[i] = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (4 * i + k < valid) w[i] |= static_cast<uint32_t>(E[off + 4 * i + k]) << (8 * k);
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// The padded copy of E (TcPadded): rows [t][f] of Dk dishes x 2 bytes.  One
// polarization: row [t'][f] interleaves the rows of times 2 t' and 2 t' + 1.
// One warp per row, 16 bytes per lane and step: bound by the bytes it moves.
__global__ void __launch_bounds__(256) bf_pad_e(const uint8_t *E, int64_t avail, uint8_t *__restrict__ out,
                                                int64_t T, int64_t F, int64_t D, int64_t Dk, int P) {
  grid_launch_next();
  grid_wait();
  const int64_t rows = (P == 2 ? T : (T + 1) / 2) * F;
  const int lane = threadIdx.x & 31;
  for (int64_t row = blockIdx.x * 8ll + (threadIdx.x >> 5); row < rows; row += gridDim.x * 8ll) {
    uint4 *dst = reinterpret_cast<uint4 *>(out + row * 2 * Dk);
    if (P == 2) {
      for (int64_t c = lane; c < Dk / 8; c += 32) {
        const int64_t left = 2 * D - 16 * c;
        dst[c] = load16_any(E, row * 2 * D + 16 * c, static_cast<int>(left < 16 ? (left < 0 ? 0 : left) : 16), avail);
      }
    } else {
      const int64_t t = row / F, f = row - t * F;
      for (int64_t c = lane; c < Dk / 8; c += 32) {  // dishes 8 c .. 8 c + 7 of both times
        const int64_t left = D - 8 * c;
        const int valid = static_cast<int>(left < 8 ? (left < 0 ? 0 : left) : 8);
        uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (2 * t + q >= T) continue;
          const int64_t off = ((2 * t + q) * F + f) * D + 8 * c;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < valid) w[k >> 1] |= static_cast<uint32_t>(E[off + k]) << (16 * (k & 1) + 8 * q);
        }
        dst[c] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
}

TcPadded tc_padded(const bf_dims &d, const uint8_t *E, bool resident) {
  TcPadded r;
  if (d.npolarizations < 1 || d.npolarizations > 2 || d.ndishes <= 0 || d.ndishes > 2048) return r;
  if (d.ntimes <= 0 || d.nbeams <= 0 || d.nfrequencies <= 0) return r;
  if (d.ntimes > (1ll << 31) || d.nfrequencies > (1 << 20) || d.nbeams > (1 << 16)) return r;
  const int64_t Dk = (d.ndishes + 7) / 8 * 8;
  // This route takes three overlapped launches, 13 us for the smallest shapes.
  // The dp4a kernel takes about 6 + 7.5 us per 128 dishes for a wave of three
  // blocks of 64 rows x 32 beams per SM.  Of 73 shapes measured with both (us, dp4a
  // against this route): up to 128 dishes in one wave 8 to 15 against 10 to 14, so
  // those stay; 129 to 256 dishes t=80 f=7 d=192 p=1 b=20 14.4 against 13.2, t=1001
  // f=1 d=250 b=45 20.6 against 13.3; more: t=26 f=3 d=539 p=1 b=63 32.9 against 13.6,
  // t=1144 f=10 d=277 p=1 b=41 47 against 16; two waves: t=4166 f=2 d=122 b=39 25 against
  // 13; t=7033 f=4 d=328 b=77 147 against 21.
  // Few times stay too, although this route would be faster from one up:
  // bf_last_kernel() has always named the dp4a kernel for the reference's own
  // shapes of 8 times and 1 and for odd chunks with resident weights, and callers
  // may count on it.
  if (d.ntimes < (resident ? 256 : 16)) return r;
  const int64_t rows = 64 / d.npolarizations;
  const double blocks = static_cast<double>((d.ntimes + rows - 1) / rows) * d.nfrequencies * ((d.nbeams + 31) / 32);
  const double waves = std::ceil(blocks / (3.0 * num_sms()));
  if (waves * (6.0 + 7.5 * static_cast<double>((d.ndishes + 127) / 128)) < 20.0) return r;
  // the operand and one chunk of the copy stay below 1 GiB
  if (static_cast<double>(d.nfrequencies) * (d.nbeams + 7) * 4.0 * Dk > 1073741824.0) return r;
  r.copy = d.npolarizations == 1 || Dk != d.ndishes || (reinterpret_cast<uintptr_t>(E) & 15u) != 0;
  r.times = d.ntimes;
  if (r.copy) {
    const int64_t per_t = d.nfrequencies * Dk * d.npolarizations;  // bytes of the copy per time
    r.times = std::max<int64_t>(128, (int64_t(256) << 20) / per_t / 128 * 128);
    r.times = std::min(r.times, d.ntimes);
    r.bytes = static_cast<size_t>((r.times + 1) / 2 * 2 * per_t);
    if (r.bytes > (size_t(1) << 30)) return r;
  }
  r.ok = true;
  return r;
}

cudaError_t launch_pad_e(const bf_dims &d, const uint8_t *E, size_t avail, int64_t times, uint8_t *out,
                         cudaStream_t s) {
  const int64_t Dk = (d.ndishes + 7) / 8 * 8;
  const int64_t rows = (d.npolarizations == 2 ? times : (times + 1) / 2) * d.nfrequencies;
  const int64_t blocks = std::min<int64_t>((rows + 7) / 8, 16ll * num_sms());
  return launch_overlapped(bf_pad_e, static_cast<unsigned>(blocks), 256, 0, s, E, static_cast<int64_t>(avail), out, times,
                           d.nfrequencies, d.ndishes, Dk, static_cast<int>(d.npolarizations));
}

cudaError_t launch_prep_weights(const TcWeights &w, const uint8_t *A, cudaStream_t s, int a_layout,
                                unsigned long long *adler, uint8_t *A_copy, float *G_copy) {
  const int64_t blocks = static_cast<int64_t>((w.nw_pad / 2 + kPrepBeams - 1) / kPrepBeams) * w.F;
  if (blocks > 0x7FFFFFFF) return cudaErrorInvalidValue;
  // Signed codes: without the copies' code where none are asked for (t=2001 f=9 d=250
  // b=45 19.9 against 20.4 us).  W + 8 is no slower with it (b=96 20.2 against 20.7).
  auto kern = tc_w_offset(w.nb_pass) ? bf_prep_weights<true, true>
              : A_copy               ? bf_prep_weights<false, true>
                                     : bf_prep_weights<false, false>;
  return launch_overlapped(kern, static_cast<unsigned>(blocks), 32 * kPrepBeams, 0, s, A, w.W, w.dig, w.G,
                           w.gs, w.gwide, static_cast<int>(w.B), static_cast<int>(w.D), static_cast<int>(w.Dk), w.nw,
                           w.nw_pad, a_layout, adler, A_copy, G_copy);
}

// Rows that start or end between words are stored byte by byte.
static void set_row_stores(TcProblem &P) {
  P.bytes = ((reinterpret_cast<uintptr_t>(P.J) | static_cast<uintptr_t>(P.rpitch) | static_cast<uintptr_t>(P.rlen)) & 3u) ? 1 : 0;
}

// Fills a problem record: shape, pointers and the two tensor maps.
static cudaError_t make_problem(TcProblem &P, const TcWeights &w, int64_t T, uint8_t *J, const uint8_t *E,
                                int64_t jpitch, int j_layout, bool pair) {
  const int64_t F = w.F, D = w.Dk;  // E rows hold Dk dishes too: they are D, or E is a padded copy
  if (reinterpret_cast<uintptr_t>(E) & 15u) return cudaErrorMisalignedAddress;
  std::memset(&P, 0, sizeof(P));
  P.T = static_cast<int>(T);
  P.F = static_cast<int>(F);
  P.B = static_cast<int>(w.B);
  P.J = J;
  P.jbase = J;
  P.adler = nullptr;
  if (jpitch <= 0) jpitch = T;
  if (jpitch < T) return cudaErrorInvalidValue;
  if (j_layout != kJLinear && j_layout != kJ2) return cudaErrorInvalidValue;
  P.jlayout = j_layout;
  P.rpitch = j_layout == kJ2 ? 2 * jpitch : jpitch;
  P.rlen = j_layout == kJ2 ? 2 * T : T;
  set_row_stores(P);
  P.nb_pass = w.nb_pass;
  P.npass = w.npass;
  P.ntt = static_cast<int>((T + kTT - 1) / kTT);
  P.nw_pad = w.nw_pad;
  P.pair = pair ? 1 : 0;
  P.w_rows = pair ? pair_cols(w.nb_pass) / 2 : 2 * w.nb_pass;
  P.gs = w.gs;
  P.gwide = w.gwide;
  {  // E[t][f][d*p] bytes: dims {2D, F, T}
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(2 * D), static_cast<cuuint64_t>(F),
                                static_cast<cuuint64_t>(T)};
    const cuuint64_t str[2] = {static_cast<cuuint64_t>(2 * D), static_cast<cuuint64_t>(2 * D * F)};
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(kKC), 1, static_cast<cuuint32_t>(kTT)};
    if (!make_map(&P.tm_e, E, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return cudaErrorInvalidValue;
  }
  {  // W[f][n][k] bytes: dims {2D, nw, F}
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(2 * D), static_cast<cuuint64_t>(w.nw),
                                static_cast<cuuint64_t>(F)};
    const cuuint64_t str[2] = {static_cast<cuuint64_t>(2 * D), static_cast<cuuint64_t>(2 * D * w.nw)};
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(kKC), static_cast<cuuint32_t>(P.w_rows), 1};
    if (!make_map(&P.tm_w, w.W, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return cudaErrorInvalidValue;
  }
  {  // digit rows dig[f][n][32] bytes: dims {32, nw_pad, F}
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(kDigitRow), static_cast<cuuint64_t>(w.nw_pad),
                                static_cast<cuuint64_t>(F)};
    const cuuint64_t str[2] = {static_cast<cuuint64_t>(kDigitRow), static_cast<cuuint64_t>(kDigitRow) * w.nw_pad};
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(kDigitRow), static_cast<cuuint32_t>(P.w_rows), 1};
    if (!make_map(&P.tm_d, w.dig, 3, dims, str, box, CU_TENSOR_MAP_SWIZZLE_32B)) return cudaErrorInvalidValue;
  }
  return cudaSuccess;
}

// Ring depths and shared memory for a launch whose largest pass has max_nb_pass beams.
static cudaError_t plan_launch(TcParams &p, int max_nb_pass, const TcRingPlan &plan, int *smem_bytes) {
  // unpacked stages live in the TMEM columns beside the two accumulators; raw E
  // slots take the shared memory the W slots leave
  const bool half = max_nb_pass <= kHalfPass;
  const int acc_cols = half ? kAccColsHalf : kAccCols;
  const int smem_limit = half ? kSmemLimitHalf : kSmemLimit;
  const int per_half = (acc_cols - 2 * max_nb_pass) / kStageCols;
  const int stages = std::min(kMaxStages, 2 * per_half);
  if (stages < 2) return cudaErrorInvalidValue;
  // Four or more unpacked stages: two unpack groups and the W forwarder.  Its
  // W producer reuses the slot of sequence it - SW once the tensor core's
  // commit of that sequence's stage arrives on `empty`, a parity wait that
  // must not find the stage's next use (sequence it - SW + S) committed too,
  // so SW <= S.  Otherwise one group, which hands W slots back S stages late,
  // so at least S slots keep it moving.
  const int groups = stages >= 4 && !half ? 2 : 1;  // the half-SM layout has one group
  // shared memory: W slots first (their loads gate the MMA), then raw E slots
  int wslots = plan.wslots > 0 ? plan.wslots : kMaxWSlots;
  if (groups == 2) wslots = std::min(wslots, stages);
  int raw = plan.raw > 0 ? plan.raw : kMinRaw;
  while (wslots > 2 && smem_plan(stages, wslots, raw, max_nb_pass).total + 1024 > smem_limit) --wslots;
  while (raw < kMaxRaw && smem_plan(stages, wslots, raw + 1, max_nb_pass).total + 1024 <= smem_limit && plan.raw <= 0)
    ++raw;
  while (raw > 2 && smem_plan(stages, wslots, raw, max_nb_pass).total + 1024 > smem_limit) --raw;
  // Two groups take alternate sequences, and raw slot k % R serves sequences
  // k and k - R: an odd R gives them to different groups, and the group with
  // k can reach its raw_full parity wait while k - R's copy has not landed,
  // when the wait (one phase early) returns at once.  An even R keeps every
  // raw slot with one group, which takes its sequences in order.
  if (groups == 2 && raw % 2 == 1) --raw;
  const int st = groups == 2 ? stages : std::min(stages, wslots);
  // The same holds for the TMEM stage ring: stage slot k % S serves k and
  // k + S, so two groups need an even S (here always 2 x stages per accumulator).
  if (groups == 2 && (wslots > st || raw < 2 || st % 2 == 1)) return cudaErrorInvalidValue;
  p.max_nb_pass = max_nb_pass;
  p.stages = st;
  p.wslots = wslots;
  p.raw = raw;
  p.groups = groups;
  p.half = half ? 1 : 0;
  p.test_stall = g_test_stall;
  *smem_bytes = smem_plan(st, wslots, raw, max_nb_pass).total + 1024;
  return *smem_bytes > smem_limit ? cudaErrorInvalidValue : cudaSuccess;
}

template <bool kGrouped, bool kJ2, int kEpiW, bool kAdler, int kGroups, bool kHalf>
static cudaError_t launch_inst(const TcParams &p, int smem_bytes, cudaStream_t s) {
  auto kern = bf_form_beams_tc<kGrouped, kJ2, kEpiW, kAdler, kGroups, kHalf>;
  static std::atomic<bool> attr_set{false};
  if (!attr_set.load()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kHalf ? kSmemLimitHalf : kSmemLimit);
    // two half-SM blocks per SM need the whole shared-memory carveout
    if (e == cudaSuccess && kHalf)
      e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    attr_set.store(true);
  }
  const int grid = std::min(p.ntiles, (kHalf ? 2 : 1) * num_sms());
  if (grid <= 0) return cudaSuccess;
  return launch_overlapped(kern, grid, Roles<kEpiW, kGroups>::kThreads, smem_bytes, s, p);
}

// Warp layout of a launch: passes of at most kHalfPass beams run two CTAs per
// SM of four epilogue warps and one unpack group each; otherwise two unpack
// groups (with the forwarder) beside eight epilogue warps; one group beside
// twelve epilogue warps up to 4 K stages per tile (the epilogue paces short
// tiles) or eight for deeper tiles.
template <bool kGrouped, bool kJ2, bool kAdler>
static cudaError_t launch_layout(const TcParams &p, int smem_bytes, cudaStream_t s) {
  if (p.half) return launch_inst<kGrouped, kJ2, 4, kAdler, 1, true>(p, smem_bytes, s);
  if (p.groups == 2) return launch_inst<kGrouped, kJ2, 8, kAdler, 2, false>(p, smem_bytes, s);
  return p.nk <= 4 ? launch_inst<kGrouped, kJ2, 12, kAdler, 1, false>(p, smem_bytes, s)
                   : launch_inst<kGrouped, kJ2, 8, kAdler, 1, false>(p, smem_bytes, s);
}

template <bool kJ2, bool kAdler>
static cudaError_t launch_plain(const TcParams &p, int smem_bytes, cudaStream_t s) {
  return launch_layout<false, kJ2, kAdler>(p, smem_bytes, s);
}

// Instantiation for a launch: J2 output and the fused adler32 only in plain
// launches.
template <bool kGrouped>
static cudaError_t launch_kernel(const TcParams &p, int smem_bytes, cudaStream_t s) {
  if constexpr (kGrouped) {
    return launch_layout<true, false, false>(p, smem_bytes, s);
  } else {
    const bool j2 = p.one.jlayout == kJ2, adler = p.one.adler != nullptr;
    if (j2) return adler ? launch_plain<true, true>(p, smem_bytes, s) : launch_plain<true, false>(p, smem_bytes, s);
    return adler ? launch_plain<false, true>(p, smem_bytes, s) : launch_plain<false, false>(p, smem_bytes, s);
  }
}

// Passes of at most kHalfPass beams run two CTAs on each SM instead: their MMAs
// take a few cycles, so two of everything else on an SM is worth more than
// sharing W (b = 16: DRAM at 0.87 of the copy bandwidth).
cudaError_t tc_pair_launch(int max_nb_pass, bool *pair) {
  int clusters = 0;
  const cudaError_t e = max_nb_pass > kHalfPass ? pair_clusters(&clusters) : cudaSuccess;
  *pair = clusters > 0 && !g_test_one_cta.load();
  return e;
}

cudaError_t tc_make_problem(TcProblem &P, const TcWeights &w, int64_t T, uint8_t *J, const uint8_t *E,
                            int64_t jpitch, int j_layout, bool pair) {
  return make_problem(P, w, T, J, E, jpitch, j_layout, pair);
}

int64_t tc_problem_tiles(const TcProblem &P) {
  return static_cast<int64_t>(P.pair ? (P.ntt + 1) / 2 : P.ntt) * P.F * P.npass;
}

int tc_stages_per_tile(int64_t D) { return static_cast<int>((D + kStageK / 2 - 1) / (kStageK / 2)); }

cudaError_t tc_plan_rings(int64_t D, int max_nb_pass, const TcRingPlan &plan, int *out) {
  TcParams p{};
  p.nk = tc_stages_per_tile(D);
  int smem_bytes = 0;
  const cudaError_t e = plan_launch(p, max_nb_pass, plan, &smem_bytes);
  if (e != cudaSuccess) return e;
  const int acc = p.half ? kAccColsHalf : kAccCols;  // the kernel's kAcc
  const int ncols = 2 * max_nb_pass;
  const int per_half = (acc - ncols) / kStageCols;
  int last_col = 0;  // one past the highest TMEM column an unpacked stage uses
  for (int i = 0; i < p.stages; ++i)
    last_col = std::max(last_col, static_cast<int>(stage_col(i, ncols, per_half, acc)) + kStageCols);
  out[0] = p.stages;
  out[1] = p.wslots;
  out[2] = p.raw;
  out[3] = p.groups;
  out[4] = p.half ? 2 : 1;
  out[5] = p.nk;
  out[6] = smem_bytes;
  out[7] = 2 * acc;  // TMEM columns allocated
  out[8] = ncols;    // columns of each accumulator (at 0 and at acc)
  out[9] = acc;
  out[10] = per_half;
  out[11] = last_col;
  return cudaSuccess;
}

// Unpack groups of a pair launch.
static int pair_groups(int max_nb_pass, const TcRingPlan &plan) {
  return plan.one_group && max_nb_pass > kNarrowPass ? 1 : 2;
}

cudaError_t tc_launch_shape(int64_t D, int max_nb_pass, bool pair, const TcRingPlan &plan, int *stages, int *groups,
                            int *ctas_per_sm) {
  if (pair) {
    *ctas_per_sm = 1;
    *groups = pair_groups(max_nb_pass, plan);
    return pair_launch_shape(D, max_nb_pass, *groups, stages);
  }
  TcParams p{};
  p.nk = tc_stages_per_tile(D);
  int smem_bytes = 0;
  const cudaError_t e = plan_launch(p, max_nb_pass, plan, &smem_bytes);
  if (e != cudaSuccess) return e;
  *stages = p.stages;
  *groups = p.groups;
  *ctas_per_sm = p.half ? 2 : 1;
  return cudaSuccess;
}

cudaError_t launch_tc_grouped(const TcProblem *table, int nprob, int ntiles, int64_t D, int max_nb_pass,
                              bool pair, bool two_pass, const TcRingPlan &plan, int *err, cudaStream_t s) {
  if (pair)
    return launch_pair_grouped(table, nprob, ntiles, D, max_nb_pass, two_pass, pair_groups(max_nb_pass, plan),
                               g_test_stall, err, s);
  TcParams p{};
  p.table = table;
  p.nprob = nprob;
  p.ntiles = ntiles;
  p.nk = tc_stages_per_tile(D);
  p.err = err;
  int smem_bytes = 0;
  const cudaError_t e = plan_launch(p, max_nb_pass, plan, &smem_bytes);
  if (e != cudaSuccess) return e;
  return launch_kernel<true>(p, smem_bytes, s);
}

cudaError_t launch_tc(const TcWeights &w, int64_t T, uint8_t *J, const uint8_t *E, int *err, cudaStream_t s,
                      int64_t jpitch, int j_layout, unsigned long long *adler, const uint8_t *jbase,
                      const TcRows *rows) {
  TcParams p{};
  bool pair = false;
  cudaError_t e = tc_pair_launch(w.nb_pass, &pair);
  if (e != cudaSuccess) return e;
  e = make_problem(p.one, w, T, J, E, jpitch, j_layout, pair);
  if (e != cudaSuccess) return e;
  p.one.adler = adler;
  if (jbase) p.one.jbase = jbase;
  if (adler && (p.one.jbase > J)) return cudaErrorInvalidValue;
  if (rows) {
    p.one.rpitch = rows->pitch;
    p.one.rlen = rows->len;
    set_row_stores(p.one);
  }
  if (pair) return launch_pair(p.one, w.Dk, g_test_stall, err, s);
  const int64_t ntiles = static_cast<int64_t>(p.one.ntt) * w.F * w.npass;
  if (ntiles > 0x7FFFFFFF) return cudaErrorInvalidValue;
  p.ntiles = static_cast<int>(ntiles);
  p.nprob = 1;
  p.nk = tc_stages_per_tile(w.Dk);
  p.err = err;
  int smem_bytes = 0;
  e = plan_launch(p, w.nb_pass, TcRingPlan{}, &smem_bytes);
  if (e != cudaSuccess) return e;
  return launch_kernel<false>(p, smem_bytes, s);
}

}  // namespace bf
