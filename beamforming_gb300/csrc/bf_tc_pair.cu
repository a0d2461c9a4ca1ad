// bf_tc_pair.cu -- the tensor-core beamformer on pairs of SMs (cta_group::2).
//
// Same GEMM, operands and epilogue as bf_tc.cu (see there for the arithmetic),
// but two CTAs of a cluster work on one tile of 128 times: each unpacks its own
// 64 times into its own tensor memory and requantises them, and one thread of
// the leader issues every MMA for both (M = 256).  Each CTA holds one half of
// the W rows, so W costs a CTA half the shared memory: a frequency's whole W
// (b = 96, d = 512: 96 KB) stays resident and is loaded once per frequency
// instead of once per tile, and the tensor cores read half as many bytes of it
// from shared memory.  In the one-CTA kernel W went through shared memory
// twice per tile (TMA write, MMA read), 3072 of the ~4600 cycles of shared-memory
// traffic a tile needs at 128 B per cycle, against 3072 cycles of MMA work.
//
// Tiles of a cluster are contiguous: beam pass fastest, then time, then
// frequency (then problem).  W stage ks of a new (problem, frequency, pass) is
// loaded as soon as the tensor cores finished the last tile that used slot ks.
// Where W does not fit (deep K, or more passes than fit) the slots are an ordinary
// ring.  A problem of two passes (97 to 128 beams) keeps the W of both, and where
// the tile's K stages all fit in tensor memory (ndishes <= 512 there) the second
// pass reads the operand that was unpacked for the first, whose E is then neither
// loaded nor unpacked again: f=64 d=512 b=128, 32768 times, 956 -> 707 us (581 at
// twice the measured bf16 rate), 128 problems of 8192 times 496 -> 330.
//
// Warp roles of each CTA (kEpiW epilogue warps):
//   epilogue     as in bf_tc.cu
//   E producer   TMA of raw E boxes
//   MMA          leader: issues for both CTAs.  Peer: tells the leader when its
//                own W stages and digit rows have landed
//   W producer   TMA of this CTA's half of W and of the digit rows
//   unpack       8 warps: two groups of four that take stages in turn, or (batches
//                of passes wider than 64 beams) one group in which two warps per
//                lane quarter take one box of each stage.  With two stages in
//                tensor memory a stage must be stored, announced and waited for
//                within the 768 cycles of the other's MMAs; two groups overlap
//                the rest of their work (664 against 703 us on the full chunk
//                in short bursts).  More warps only contend for the integer pipe
//                (16 unpack warps 712, 12 epilogue warps 693 us).
#include "bf_internal.h"
#include "bf_once.h"
#include "bf_tc_common.cuh"

#include <algorithm>
#include <atomic>

namespace bf {
namespace {

constexpr int kPairAcc = 256;        // TMEM column of the second accumulator
constexpr int kPairCols = 512;       // TMEM columns of a CTA: all
constexpr int kPairSmem = 232448;    // 227 KiB opt-in per block
constexpr int kPairMaxRaw = 16;
constexpr int kPairMaxStages = 8;
constexpr int kEpiW = 8;       // epilogue warps
constexpr int kEpiChunks = 2;  // chunks of 8 beams in flight per epilogue warp
constexpr int kUnpackWarps = 8;
constexpr int kPairThreads = 32 * (kEpiW + kUnpackWarps + 3);

struct PairParams {
  TcProblem one;            // the problem of a plain launch
  const TcProblem *table;   // grouped launch: nprob problems in device memory, by tile_begin
  int nprob;
  int ntiles;               // tile pairs
  int nk;                   // K stages per tile
  int ncols;                // widest GEMM N of the launch (a multiple of 32)
  int stages, wslots, raw;  // TMEM stages, W slots, raw E slots
  int sets;                 // passes whose W (unless streamed) and digit rows stay resident
  int share;                // nonzero: the passes of a tile share its unpacked operand
  int test_stall;
  int *err;
};

struct PairSmem {
  int wbytes, dbytes;
  int off_a, off_d, off_r, off_bar, nbar, total;
};

__host__ __device__ inline PairSmem pair_smem(int stages, int wslots, int raw, int ncols) {
  PairSmem s{};
  s.wbytes = kSub * (ncols / 2) * kKC;  // this CTA's half of the rows
  s.dbytes = (ncols / 2 * kDigitRow + 1023) / 1024 * 1024;
  s.off_a = wslots * s.wbytes;
  s.off_d = s.off_a + 2 * kConstABytes;
  s.off_r = s.off_d + kDigSlots * s.dbytes;
  s.off_bar = s.off_r + raw * kRawBytes;
  // raw_full[R] raw_empty[R] w_full[SW] w_peer[SW] w_empty[SW] a_full[S] empty[S] accfull[2] accempty[2]
  // d_full[2] d_peer[2] d_empty[2] rs_full[2] cut_done
  s.nbar = 2 * raw + 3 * wslots + 2 * stages + 4 + 3 * kDigSlots + 3;
  s.total = s.off_bar + 8 * s.nbar + 32;  // + the TMEM address and the leader's commit counts
  return s;
}

// A cluster's tiles, one by one.
template <bool kGrouped>
struct PairCursor {
  const TcProblem *P;
  int idx = 0, pass, tp, f, ntp;
  __device__ __forceinline__ PairCursor(const PairParams &p, int first) : P(&p.one) {
    int lt = first;
    if constexpr (kGrouped) {
      int lo = 0, hi = p.nprob - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (p.table[mid].tile_begin <= first) lo = mid; else hi = mid - 1;
      }
      idx = lo;
      P = p.table + lo;
      lt -= P->tile_begin;
    }
    ntp = (P->ntt + 1) >> 1;
    pass = lt % P->npass;
    tp = (lt / P->npass) % ntp;
    f = lt / (P->npass * ntp);
  }
  // This is the first (last) of its tiles with these W and digit rows, `n` tiles
  // after the start (before the end) of the cluster's range: those of up to `sets`
  // passes stay for a frequency.  They are given back together and only where
  // tiles follow, so the releases of all slots run through the ring in rounds
  // (drain_commits), although a range that starts with an odd pass loads that first
  // -- unless a failed wait cuts it short (cut_commits).
  __device__ __forceinline__ bool first_of_w(int n, int sets) const { return P->npass > sets || n < P->npass || tp == 0; }
  __device__ __forceinline__ bool last_of_w(int n, int sets) const {
    return P->npass > sets || (tp + 1 == ntp && n > P->npass - pass);
  }
  // This tile's operand is unpacked for it (and not for the pass before), and
  // free after it.
  __device__ __forceinline__ bool first_of_a(bool share, bool range_first) const { return !share || pass == 0 || range_first; }
  __device__ __forceinline__ bool last_of_a(bool share, bool range_last) const { return !share || pass + 1 == P->npass || range_last; }
  __device__ __forceinline__ void next(const PairParams &p) {
    if (++pass < P->npass) return;
    pass = 0;
    if (++tp < ntp) return;
    tp = 0;
    ++f;
    if constexpr (kGrouped) {
      if (f == P->F && idx + 1 < p.nprob) {
        f = 0;
        P = p.table + ++idx;
        ntp = (P->ntt + 1) >> 1;
      }
    }
  }
  // beams of this tile's pass (a multiple of 8) and its GEMM N (a multiple of 32)
  __device__ __forceinline__ int beams() const { return min(P->nb_pass, (P->B + 7) / 8 * 8 - pass * P->nb_pass); }
  __device__ __forceinline__ int n() const { return (2 * beams() + 31) & ~31; }
};

// Commits the leader issued, for the exits of both CTAs (in the shared memory of each).
struct Commits {
  uint32_t nstage, nw, ndig, nacc;  // on empty, w_empty, d_empty, accfull
  uint32_t cut;                     // a failed wait ended a tile: cut_done too
  uint32_t w1, d1;                  // then: of nw and ndig, on the second resident W, the second digit slot
};

// `w1` and `d1` of an issuer whose tile `cut` a failed wait ended: its walk over the
// tiles once more, on the failure path alone.  (Counting slot by slot as the commits
// are issued: the wide array 698 -> 714 us in one form, t=8208 f=21 d=328 b=41 34.6 ->
// 35.0 in another.)  One lane.
template <bool kGrouped>
__device__ __noinline__ void cut_commits(const PairParams &p, int first, int cut, int end, Commits &c) {
  uint32_t w = 0, d = 0;  // of the tiles before
  int it = 0, dit = 0;    // slots loaded
  int w_at[2] = {0, 0}, d_at[2] = {0, 0};
  const int nk = p.nk, SW = p.wslots;
  PairCursor<kGrouped> cur(p, first);
#pragma unroll 1
  for (int tile = first; tile <= cut; ++tile, cur.next(p)) {
    const bool odd = cur.pass & 1;
    if (cur.first_of_w(tile - first, p.sets)) {
      (odd ? w_at[1] : w_at[0]) = it % SW;
      (odd ? d_at[1] : d_at[0]) = dit % kDigSlots;
      it += nk;
      ++dit;
    }
    const bool last = cur.last_of_w(end - tile, p.sets);
    // the cut tile's: what is left of the counts
    const uint32_t tw = tile == cut ? c.nw - w : last ? static_cast<uint32_t>(nk) : 0u;
    const uint32_t td = tile == cut ? c.ndig - d : last ? 1u : 0u;
    w += tw;
    d += td;
    if (SW >= nk && (odd ? w_at[1] : w_at[0]) != 0) c.w1 += tw;
    if ((odd ? d_at[1] : d_at[0]) != 0) c.d1 += td;
  }
}

static_assert(sizeof(Commits) + 4 <= 32, "they fit behind the TMEM address (pair_smem)");

// A CTA's exit: waits (bounded) for the last phase that the leader committed on each
// barrier, one to a lane.  `bw`, `ba`, `bc`: the first W, stage and accumulator barrier.
// A function, for leader and peer: inlined, its waits push the kernel's loops out of
// the instruction cache (t=8208 f=21 d=328 b=41 34.3 -> 35.1 us).
__device__ __noinline__ void drain_commits(uint32_t bw, uint32_t ba, uint32_t bc, int S, int SW, int nk,
                                           const Commits &n) {
#pragma unroll 1
  for (int i = threadIdx.x & 31; i < S + SW + 2 * kDigSlots + 1; i += 32) {
    // slot `at` of a ring that `count` commits went round
    const int w = i - S, d = w - SW, a = d - kDigSlots;
    uint32_t bar = ba + 8u * (S + i), count = n.nstage;
    int ring = S, at = i;
    if (w >= 0) bar = bw + 8u * (2 * SW + w), count = n.nw, ring = SW, at = w;
    if (d >= 0) bar = bc + 64u + 8u * d, count = n.ndig, ring = kDigSlots, at = d;
    if (a >= 0) bar = bc + 8u * a, count = n.nacc, ring = 2, at = a;
    if (a >= 2) bar = bc + 96u, count = n.cut, ring = 1, at = 0;
    if (n.cut && w >= 0 && d < 0) {  // each resident W by itself, its slots in order
      ring = SW < nk ? SW : nk;
      count = w < ring ? n.nw - n.w1 : n.w1;
      at = w < ring ? w : w - ring;
    } else if (n.cut && d >= 0 && a < 0) {
      count = d ? n.d1 : n.ndig - n.d1, ring = 1, at = 0;
    }
    const uint32_t done = (count + ring - 1 - at) / ring;
    if (done) mbar_wait_drain(bar, (done - 1u) & 1u);
  }
  __syncwarp();
}

// Operands to unpack for tiles first .. end - 1 (first < end).
template <bool kGrouped>
__device__ __forceinline__ int operands_of(const PairParams &p, int first, int end) {
  if (!p.share) return end - first;
  auto span = [](int a, int b, int np) { return (b - 1) / np - a / np + 1; };  // a < b
  if constexpr (!kGrouped) return span(first, end, p.one.npass);
  int n = 0;
  for (int i = PairCursor<kGrouped>(p, first).idx; i < p.nprob; ++i) {
    const int t0 = p.table[i].tile_begin, t1 = i + 1 < p.nprob ? p.table[i + 1].tile_begin : p.ntiles;
    if (t0 >= end) break;
    n += span(max(first, t0) - t0, min(end, t1) - t0, p.table[i].npass);
  }
  return n;
}

// TMEM column of unpacked stage i: the columns left beside the two accumulators.
__host__ __device__ inline uint32_t pair_stage_col(uint32_t i, int ncols, int per_half, int cols) {
  return static_cast<uint32_t>(ncols) + i * static_cast<uint32_t>(cols) +
         (i < static_cast<uint32_t>(per_half) ? 0u : static_cast<uint32_t>(kPairAcc - per_half * cols));
}

template <bool kGrouped, bool kJ2, bool kAdler, int kGroups, bool kSums>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
    bf_form_beams_pair(const __grid_constant__ PairParams p) {
  constexpr int kUnpackWarp0 = kEpiW, kEProdWarp = kEpiW + kUnpackWarps, kMmaWarp = kEProdWarp + 1;
  constexpr int kWProdWarp = kEProdWarp + 2;
  constexpr int kEpiParts = kEpiW / 4;
  constexpr int kStageWarps = kUnpackWarps / kGroups;  // unpack warps of a stage
  constexpr int kBoxes = kSub * 4 / kStageWarps;       // boxes of it each of them takes
  extern __shared__ uint8_t smem_dyn[];
  // the same offset in both CTAs of the cluster
  uint8_t *smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
  const int S = p.stages, SW = p.wslots, R = p.raw, nk = p.nk;
  const PairSmem sp = pair_smem(S, SW, R, p.ncols);
  uint8_t *sW = smem, *sA = smem + sp.off_a, *sD = smem + sp.off_d, *sR = smem + sp.off_r;
  const uint32_t bar0 = smem_u32(smem + sp.off_bar);
  auto raw_full = [&](int r) { return bar0 + 8u * r; };
  auto raw_empty = [&](int r) { return bar0 + 8u * (R + r); };
  const uint32_t bw = bar0 + 16u * R;
  auto w_full = [&](int s) { return bw + 8u * s; };
  auto w_peer = [&](int s) { return bw + 8u * (SW + s); };
  auto w_empty = [&](int s) { return bw + 8u * (2 * SW + s); };
  const uint32_t ba = bw + 24u * SW;
  auto a_full = [&](int s) { return ba + 8u * s; };
  auto empty = [&](int s) { return ba + 8u * (S + s); };
  const uint32_t bc = ba + 16u * S;
  auto accfull = [&](int i) { return bc + 8u * i; };
  auto accempty = [&](int i) { return bc + 16u + 8u * i; };
  auto d_full = [&](int i) { return bc + 32u + 8u * i; };
  auto d_peer = [&](int i) { return bc + 48u + 8u * i; };
  auto d_empty = [&](int i) { return bc + 64u + 8u * i; };
  auto rs_full = [&](int i) { return bc + 80u + 8u * i; };
  const uint32_t cut_done = bc + 96u;  // the MMAs of a tile that a failed wait cut short
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(smem + sp.off_bar + 8 * sp.nbar);
  Commits *counts = reinterpret_cast<Commits *>(tmem_holder + 1);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // known to be warp-uniform
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const int ncols = p.ncols;
  const int per_half = (kPairAcc - ncols) / kStageCols;

  // Each producer sets up its own barriers and starts its copies without waiting
  // for the CTAs of the pair to meet (setup_sync, some 2700 cycles in).
  if (warp == kEProdWarp) {
    for (int i = lane; i < 2 * R; i += 32) mbar_init(raw_full(i), i < R ? 1 : kStageWarps);
    if (!kGrouped && lane == 0) tma_prefetch_desc(&p.one.tm_e);
  } else if (warp == kWProdWarp) {
    for (int i = lane; i < 3 * SW; i += 32) mbar_init(w_full(i), 1);
    if (lane < 3 * kDigSlots) mbar_init(d_full(0) + 8u * lane, 1);
    if (!kGrouped && lane == 0) {
      tma_prefetch_desc(&p.one.tm_w);
      tma_prefetch_desc(&p.one.tm_d);
    }
  } else if (warp == 0) {
    // a_full, accempty (the leader's): the unpack warps of a stage, the epilogue
    // warps, in both CTAs
    if (lane < 2 * S) mbar_init(a_full(lane), lane < S ? 2 * kStageWarps : 1);
    if (lane < 4) mbar_init(accfull(lane), lane < 2 ? 1 : 2 * kEpiW);
    if (lane < 2) mbar_init(rs_full(lane), 2 * kUnpackWarps);
    if (lane == 0) *counts = Commits{};
    if (lane == 0) mbar_init(cut_done, 1);
  }
  fence_barrier_init();
  __syncwarp();  // a producer's lane 0 uses barriers that its other lanes set up, and waits for no other warp
  if (warp == kMmaWarp) {
    tmem_alloc_pair(smem_u32(tmem_holder), kPairCols);
    tmem_relinquish_pair();
  }
  fill_offset_tiles<kSums ? 2 : 1>(sA);
  fence_proxy_async_smem();
  grid_launch_next();
  grid_wait();
  auto setup_sync = [&]() {
    tc_fence_before();
    cluster_sync();
    tc_fence_after();
  };
  static_assert(2 * kPairMaxStages <= 32, "one lane per stage barrier");
  int *err = p.err;

  const int64_t ncl = gridDim.x >> 1, cl = blockIdx.x >> 1;
  const int first = static_cast<int>(cl * p.ntiles / ncl), end = static_cast<int>((cl + 1) * p.ntiles / ncl);
  const bool stream_w = SW < nk;  // W slots are an ordinary ring
  const int sets = p.sets;
  const bool share = !kSums && p.share != 0;

  if (warp == kEProdWarp) {
    // ------------------------------------------------------------ E producer
    const uint64_t pol_e = policy_evict_first();
    Ring rr(R);
    uint32_t issued = 0;
    bool ok = !p.test_stall;
    cluster_arrive();
    const TcProblem *seen = nullptr;
    PairCursor<kGrouped> cur(p, first);
    for (int tile = first; ok && tile < end; ++tile, cur.next(p)) {
      if (!cur.first_of_a(share, tile == first)) continue;
      if (kGrouped && cur.P != seen) {  // a table entry the host rewrites between launches
        tensormap_acquire(&cur.P->tm_e);
        seen = cur.P;
      }
      for (int ks = 0; ks < nk; ++ks, rr.advance(), ++issued) {
        const int r = static_cast<int>(rr.idx);
        ok = __all_sync(0xffffffffu, mbar_wait(raw_empty(r), rr.phase ^ 1u, err, kDevTimeoutEmpty));
        if (!ok) break;
        if (lane == 0) {
          mbar_arrive_expect_tx(raw_full(r), kRawBytes);
#pragma unroll
          for (int h = 0; h < kSub; ++h)
            tma_load_3d(smem_u32(sR + r * kRawBytes + h * kRawBox), &cur.P->tm_e, raw_full(r), (ks * kSub + h) * kKC,
                        cur.f, (2 * cur.tp + rank) * kTT, pol_e);
        }
        __syncwarp();
      }
    }
    cluster_wait();
    // let the copies already issued land before the CTA exits, on every exit
    for (uint32_t k = (issued >= static_cast<uint32_t>(R) ? issued - R : 0); k < issued; ++k)
      mbar_wait_drain(raw_full(static_cast<int>(k % R)), (k / R) & 1u);
  } else if (warp == kWProdWarp) {
    // ------------------------------------------------------------ W producer
    const uint64_t pol_w = policy_evict_last();
    Ring wr(SW), dr(kDigSlots);
    uint32_t it = 0, dit = 0;
    bool ok = !p.test_stall;
    cluster_arrive();
    const TcProblem *seen = nullptr;
    PairCursor<kGrouped> cur(p, first);
    for (int tile = first; ok && tile < end; ++tile, cur.next(p)) {
      const bool fresh = cur.first_of_w(tile - first, sets);
      if (fresh || stream_w) {
        if (kGrouped && cur.P != seen) {
          tensormap_acquire(&cur.P->tm_w);
          tensormap_acquire(&cur.P->tm_d);
          seen = cur.P;
        }
        const int row0 = cur.pass * 2 * cur.P->nb_pass + rank * (cur.n() / 2);
        const int wbox = cur.P->w_rows * kKC;
        if (fresh) {  // the digit rows, for the offset MMA
          const int ds = static_cast<int>(dr.idx);
          ok = __all_sync(0xffffffffu, mbar_wait(d_empty(ds), dr.phase ^ 1u, err, kDevTimeoutEmpty));
          if (!ok) break;
          if (lane == 0) {
            mbar_arrive_expect_tx(d_full(ds), cur.P->w_rows * kDigitRow);
            tma_load_3d(smem_u32(sD + ds * sp.dbytes), &cur.P->tm_d, d_full(ds), 0, row0, cur.f, pol_w);
          }
          dr.advance();
          ++dit;
        }
        for (int ks = 0; ks < nk; ++ks, ++it, wr.advance()) {
          const int s = static_cast<int>(wr.idx);
          ok = __all_sync(0xffffffffu, mbar_wait(w_empty(s), wr.phase ^ 1u, err, kDevTimeoutEmpty));
          if (!ok) break;
          if (lane == 0) {
            mbar_arrive_expect_tx(w_full(s), kSub * wbox);
#pragma unroll
            for (int h = 0; h < kSub; ++h)
              tma_load_3d(smem_u32(sW + s * sp.wbytes + h * wbox), &cur.P->tm_w, w_full(s), (ks * kSub + h) * kKC,
                          row0, cur.f, pol_w);
          }
          __syncwarp();
        }
      }
    }
    cluster_wait();
    for (uint32_t k = (it >= static_cast<uint32_t>(SW) ? it - SW : 0); k < it; ++k)
      mbar_wait_drain(w_full(static_cast<int>(k % SW)), (k / SW) & 1u);
    for (uint32_t k = (dit >= static_cast<uint32_t>(kDigSlots) ? dit - kDigSlots : 0); k < dit; ++k)
      mbar_wait_drain(d_full(static_cast<int>(k % kDigSlots)), (k / kDigSlots) & 1u);
  } else if (warp == kMmaWarp && rank == 1) {
    // ------------------------------------- peer: this CTA's W and digits landed
    setup_sync();
    if (lane == 0 && !p.test_stall) {
      Ring wr(SW), dr(kDigSlots);
      bool ok = true;
      PairCursor<kGrouped> cur(p, first);
      for (int tile = first; ok && tile < end; ++tile, cur.next(p)) {
        const bool fresh = cur.first_of_w(tile - first, sets);
        if (fresh) {
          if (!mbar_wait(d_full(dr.idx), dr.phase, err, kDevTimeoutFull)) break;
          mbar_arrive_cluster(map_cta(d_peer(dr.idx), 0));
          dr.advance();
        }
        if (fresh || stream_w) {
          for (int ks = 0; ks < nk; ++ks, wr.advance()) {
            if (!mbar_wait(w_full(wr.idx), wr.phase, err, kDevTimeoutFull)) {
              ok = false;
              break;
            }
            mbar_arrive_cluster(map_cta(w_peer(wr.idx), 0));
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMA issuer
    // Warp-uniform, one elected lane issues (see bf_tc.cu).  The tensor core
    // idles whenever a stage costs this warp more than its MMAs take, so the
    // loop of the common tile -- resident W, neither loaded nor given back --
    // holds nothing but the wait, the MMAs and the commit.
    setup_sync();
    const uint32_t tmem_base = *tmem_holder;
    Ring ar(S), wr(SW), dr(kDigSlots);
    const uint64_t a_off = smem_desc_sw32(smem_u32(sA));
    const uint64_t w_desc0 = smem_desc_sw128(smem_u32(sW));
    const uint32_t w_step = static_cast<uint32_t>(sp.wbytes) >> 4;
    uint32_t local = 0;
    uint32_t nstage = 0, nw = 0, ndig = 0, nacc = 0;  // commits issued on empty, w_empty, d_empty, accfull
    bool ok = true;
    int w_at[2] = {0, 0}, d_at[2] = {0, 0};  // first W slot and digit slot of even and odd passes
    Ring a0(S);                              // the first stage of the tile's operand
    PairCursor<kGrouped> cur(p, first);
    int tile = first;
    for (; ok && tile < end; ++tile, ++local, cur.next(p)) {
      const uint32_t idesc = idesc_e4m3_f32(2 * kBM, static_cast<uint32_t>(cur.n()));
      const uint32_t wbox = static_cast<uint32_t>(cur.P->w_rows * kKC) >> 4;
      const bool fresh = cur.first_of_w(tile - first, sets), last = cur.last_of_w(end - tile, sets);
      const bool new_a = cur.first_of_a(share, tile == first), last_a = cur.last_of_a(share, tile + 1 == end);
      const bool odd = cur.pass & 1;
      if (new_a) a0 = ar; else ar = a0;
      if (fresh) (odd ? w_at[1] : w_at[0]) = stream_w ? 0 : static_cast<int>(wr.idx);
      if (fresh) (odd ? d_at[1] : d_at[0]) = static_cast<int>(dr.idx);
      const int w0 = odd ? w_at[1] : w_at[0], ds = odd ? d_at[1] : d_at[0];
      const uint32_t ab = local & 1u;
      if (!__all_sync(0xffffffffu, mbar_wait(accempty(ab), ((local >> 1) & 1u) ^ 1u, err, kDevTimeoutAccEmpty))) break;
      if (fresh && !__all_sync(0xffffffffu, mbar_wait(d_full(ds), dr.phase, err, kDevTimeoutFull) &&
                                                mbar_wait(d_peer(ds), dr.phase, err, kDevTimeoutFull)))
        break;
      if (fresh) dr.advance();
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + ab * kPairAcc;
      // the offset MMA: -8 sum_k W[n][k] 2^-18, with the row sums also
      // -8 sum_k u[m][k] 2^-18, which are there last
      auto offset_mma = [&]() {
        mma_f8f6f4_pair(d_tmem, a_off + (kSums ? ab * (kConstABytes >> 4) : 0u), smem_desc_sw32(smem_u32(sD + ds * sp.dbytes)), idesc,
                        kSums ? 1u : 0u);
        if (last) mma_commit_pair(d_empty(ds));
      };
      if constexpr (!kSums) {
        if (elect_one()) offset_mma();
        ndig += last ? 1u : 0u;  // with its commit: the tile may end early
      }
      __syncwarp();
      if (!fresh && !last && !stream_w) {
        uint64_t b_desc = w_desc0 + static_cast<uint32_t>(w0) * w_step;
        for (int ks = 0; ks < nk; ++ks, b_desc += w_step) {
          const uint32_t bar = a_full(ar.idx);
          if (new_a && !__all_sync(0xffffffffu, mbar_wait(bar, ar.phase, err, kDevTimeoutUnpacked))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_tmem = tmem_base + pair_stage_col(ar.idx, ncols, per_half, kStageCols);
          if (elect_one()) {
            mma_ts_box_pair(d_tmem, a_tmem, b_desc, idesc, !kSums || ks > 0);
            mma_ts_box_pair(d_tmem, a_tmem + 32, b_desc + wbox, idesc, 1u);
            if (last_a) mma_commit_pair(bar + 8u * S);  // empty
          }
          __syncwarp();
          nstage += last_a ? 1u : 0u;
          ar.advance();
        }
      } else {
        const bool reload = fresh || stream_w, release = last || stream_w;
        for (int ks = 0; ks < nk; ++ks, ar.advance()) {
          // the parity of a W slot's current load: resident slots (SW == nk) step
          // with the loads, not with the tiles
          const int sw = stream_w ? static_cast<int>(wr.idx) : w0 + ks;
          if (reload && !__all_sync(0xffffffffu, mbar_wait(w_full(sw), wr.phase, err, kDevTimeoutFull) &&
                                                     mbar_wait(w_peer(sw), wr.phase, err, kDevTimeoutFull))) {
            ok = false;
            break;
          }
          const uint32_t bar = a_full(ar.idx);
          if (new_a && !__all_sync(0xffffffffu, mbar_wait(bar, ar.phase, err, kDevTimeoutUnpacked))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_tmem = tmem_base + pair_stage_col(ar.idx, ncols, per_half, kStageCols);
          const uint64_t b_desc = w_desc0 + static_cast<uint32_t>(sw) * w_step;
          if (elect_one()) {
            mma_ts_box_pair(d_tmem, a_tmem, b_desc, idesc, !kSums || ks > 0);
            mma_ts_box_pair(d_tmem, a_tmem + 32, b_desc + wbox, idesc, 1u);
            if (last_a) mma_commit_pair(bar + 8u * S);  // empty
            if (release) mma_commit_pair(w_empty(sw));
          }
          __syncwarp();
          nstage += last_a ? 1u : 0u;
          nw += release ? 1u : 0u;
          if (reload) wr.advance();
        }
      }
      if (!ok) break;
      if constexpr (kSums) {
        if (!__all_sync(0xffffffffu, mbar_wait(rs_full(ab), (local >> 1) & 1u, err, kDevTimeoutUnpacked))) break;
        tc_fence_after();
      }
      if constexpr (kSums) {
        if (elect_one()) offset_mma();
        ndig += last ? 1u : 0u;
      }
      if (elect_one()) mma_commit_pair(accfull(ab));
      __syncwarp();
      ++nacc;
    }
    // A tile that a failed wait cut short has MMAs that no commit covers (the offset
    // MMA, stages that the next pass would read too): one more commit does.
    const uint32_t cut = tile < end ? 1u : 0u;
    if (cut && elect_one()) mma_commit_pair(cut_done);
    __syncwarp();
    // A commit's arrival is an asynchronous write into both CTAs' shared memory:
    // wait for the last phase committed on every barrier before the CTAs can exit,
    // here and, from the counts, in the peer.
    if (lane == 0) {
      *counts = Commits{nstage, nw, ndig, nacc, cut, 0u, 0u};
      if (cut) cut_commits<kGrouped>(p, first, tile, end, *counts);
      const uint32_t at = map_cta(smem_u32(counts), 1);
      st_cluster_u32(at, nstage);
      st_cluster_u32(at + 4, nw);
      st_cluster_u32(at + 8, ndig);
      st_cluster_u32(at + 12, nacc);
      st_cluster_u32(at + 16, cut);
      if (cut) {
        st_cluster_u32(at + 20, counts->w1);
        st_cluster_u32(at + 24, counts->d1);
      }
    }
    __syncwarp();
    drain_commits(bw, ba, bc, S, SW, nk, *counts);
  } else if (warp >= kUnpackWarp0 && warp < kEProdWarp) {
    // ------------------------------------------------------------ unpack
    // Each lane fills one GEMM row: it reads the raw row of its time, which
    // holds both polarizations, and keeps its own (RowMap).  The groups take
    // stages in turn (R and S are multiples of their number, so a slot always
    // belongs to one group).
    setup_sync();
    const uint32_t tmem_base = *tmem_holder;
    const int group = (warp - kUnpackWarp0) / kStageWarps;
    const int box0 = ((warp - kUnpackWarp0) % kStageWarps >> 2) * kBoxes;
    const int q = warp & 3;
    const UnpackRow row(RowMap<kJ2>::time(q, lane));
    const uint32_t sel = RowMap<kJ2>::pol(q, lane) ? 0x7531u : 0x6420u;  // odd or even bytes
    const uint32_t lane_addr = static_cast<uint32_t>(32 * q) << 16;
    const int operands = kSums ? end - first : operands_of<kGrouped>(p, first, end);
    const uint32_t total = static_cast<uint32_t>(operands) * static_cast<uint32_t>(nk);
    Ring rr(R), ar(S);
    for (int g = 0; g < group; ++g) {
      rr.advance();
      ar.advance();
    }
    const int my_tiles = end - first;
    RowSums rs(sA, group, (warp - kUnpackWarp0) >> 2, 32 * q + lane);
    auto rs_free = [&](int tile) {
      return __all_sync(0xffffffffu, mbar_wait(accfull(tile & 1), ((tile >> 1) & 1) ^ 1, err, kDevTimeoutAccFull));
    };
    auto rs_arrive = [&](int tile) {
      if (lane == 0) mbar_arrive_cluster(map_cta(rs_full(tile & 1), 0));
    };
    bool live = !kSums || rs.settle(nk, my_tiles, rs_free, rs_arrive);
    for (uint32_t it = group; live && it < total; it += kGroups) {
      const int r = static_cast<int>(rr.idx);
      const int s = static_cast<int>(ar.idx);
      if (!__all_sync(0xffffffffu, mbar_wait(raw_full(r), rr.phase, err, kDevTimeoutFull))) break;
      // box by box: the first box's words are made before the stage is free, the
      // others' while the stores of the one before are under way
      const uint32_t raw = smem_u32(sR) + static_cast<uint32_t>(r * kRawBytes + box0 * kRawBox);
      const uint32_t col = tmem_base + lane_addr + pair_stage_col(s, ncols, per_half, kStageCols) + 32u * box0;
      bool free = true;
#pragma unroll
      for (int h = 0; h < kBoxes; ++h) {
        uint32_t out[32];
        rs.sum += unpack_box<kSums>(raw + h * kRawBox, row, sel, out);
        if (h == 0) free = __all_sync(0xffffffffu, mbar_wait(empty(s), ar.phase ^ 1u, err, kDevTimeoutEmpty));
        if (!free) break;
        tmem_st_32x32b_x32(col + 32 * h, out);
      }
      if (!free) break;
      // the next TMA into the slot is an async-proxy write after these generic reads
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(raw_empty(r));
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster_relaxed(map_cta(a_full(s), 0));
      if constexpr (kSums) {
        rs.kpos += kGroups;
        live = rs.settle(nk, my_tiles, rs_free, rs_arrive);
      }
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        rr.advance();
        ar.advance();
      }
    }
  } else if (warp < kEpiW) {
    // ------------------------------------------------------------ epilogue
    // Warp w reads TMEM lane quarter w % 4 and column part w / 4.  The warps
    // share no barrier: a slow one does not hold up the others.
    const int q = warp & 3;
    const int part = warp >> 2;
    setup_sync();
    const uint32_t tmem_base = *tmem_holder;
    const uint32_t lane_addr = static_cast<uint32_t>(32 * q) << 16;
    uint32_t local = 0;
    unsigned long long ad_s1 = 0, ad_s2 = 0;  // fused adler32 (kAdler): sums of the J bytes this lane stores
    PairCursor<kGrouped> cur(p, first);
    for (int tile = first; tile < end; ++tile, ++local, cur.next(p)) {
      const uint32_t ab = local & 1u;
      const EpilogueTile<kJ2, kAdler> et(*cur.P, cur.f, cur.pass, 2 * cur.tp + rank, q, lane);
      const int nchunk = cur.beams() / 8;
      const bool ok = et.template run<kEpiChunks>(
          *cur.P, tmem_base + ab * kPairAcc + lane_addr, part * nchunk / kEpiParts, (part + 1) * nchunk / kEpiParts,
          ad_s1, ad_s2,
          [&]() {
            const bool full = __all_sync(0xffffffffu, mbar_wait(accfull(ab), (local >> 1) & 1u, err, kDevTimeoutAccFull));
            tc_fence_after();
            return full;
          },
          [&]() {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster_relaxed(map_cta(accempty(ab), 0));
          });
      if (!ok) break;
    }
    if constexpr (kAdler) add_adler(p.one.adler, ad_s1, ad_s2, lane);
  }

  // Both CTAs meet once more: neither frees tensor memory or exits while the
  // other's threads or the leader's MMAs may still reach into it.  What can still
  // come after that are the arrivals of the leader's last commits at the peer's
  // own barriers, which the peer waits for here.
  __syncwarp();
  tc_fence_before();
  cluster_sync();
  if (warp == kMmaWarp) {
    if (rank == 1) drain_commits(bw, ba, bc, S, SW, nk, *counts);
    tc_fence_after();
    tmem_dealloc_pair(*tmem_holder, kPairCols);
  }
}

// Ring depths and shared memory of a launch whose widest GEMM N is ncols.
cudaError_t plan_pair(PairParams &p, int64_t D, int max_nb_pass, bool two_pass, int groups, int *smem_bytes) {
  p.nk = tc_stages_per_tile(D);
  p.ncols = pair_cols(max_nb_pass);
  const int ncols = p.ncols;
  int stages = std::min(kPairMaxStages, 2 * ((kPairAcc - ncols) / kStageCols));
  stages -= stages % groups;  // so does a TMEM stage
  if (stages < 2) return cudaErrorInvalidValue;
  // W resident (all nk slots) where at least 64 KB of raw E slots fit beside it,
  // else as many slots as that leaves: a W load takes ~2400 cycles from the
  // commit that frees its slot to the peer's word that it landed
  auto total = [&](int w, int r) { return pair_smem(stages, w, r, ncols).total + 1024; };
  int wslots = p.nk;
  if (total(wslots, 4) > kPairSmem) {
    wslots = 2;
    while (wslots < p.nk - 1 && total(wslots + 1, 4) <= kPairSmem) ++wslots;
  }
  // two passes' W where that leaves as much: neither is loaded per tile then
  // (f=32 d=256 b=192, 16384 times: 191 -> 164 us)
  if (two_pass && total(2 * p.nk, 4) <= kPairSmem) wslots = 2 * p.nk;
  p.sets = wslots < p.nk ? kDigSlots : std::min(kDigSlots, wslots / p.nk);
  // a tile's whole operand fits the TMEM stages: its passes take it in turn
  // (with row sums, one per tile of the accumulator, they do not)
  p.share = two_pass && p.nk <= stages && !tc_w_offset(max_nb_pass) ? 1 : 0;
  int raw = 2;
  while (raw < kPairMaxRaw && total(wslots, raw + 1) <= kPairSmem) ++raw;
  raw -= raw % groups;  // a raw slot stays with one unpack group
  p.stages = stages;
  p.wslots = wslots;
  p.raw = raw;
  *smem_bytes = total(wslots, raw);
  return *smem_bytes > kPairSmem ? cudaErrorInvalidValue : cudaSuccess;
}

template <bool kGrouped, bool kJ2, bool kAdler, int kGroups, bool kSums>
cudaError_t launch_inst(const PairParams &p, int smem_bytes, cudaStream_t s) {
  auto kern = bf_form_beams_pair<kGrouped, kJ2, kAdler, kGroups, kSums>;
  static std::atomic<bool> attr_set{false};
  if (!attr_set.load()) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem);
    if (e != cudaSuccess) return e;
    attr_set.store(true);
  }
  int clusters = 0;
  const cudaError_t e = pair_clusters(&clusters);
  if (e != cudaSuccess) return e;
  if (clusters <= 0) return cudaErrorInvalidConfiguration;
  const int grid = 2 * std::min(p.ntiles, clusters);
  if (grid <= 0) return cudaSuccess;
  return launch_overlapped(kern, grid, kPairThreads, smem_bytes, s, p);
}

template <bool kSums>
cudaError_t launch_plain(const PairParams &p, int smem_bytes, cudaStream_t s) {
  const bool adler = p.one.adler != nullptr;
  if (p.one.jlayout == kJ2)
    return adler ? launch_inst<false, true, true, 2, kSums>(p, smem_bytes, s)
                 : launch_inst<false, true, false, 2, kSums>(p, smem_bytes, s);
  return adler ? launch_inst<false, false, true, 2, kSums>(p, smem_bytes, s)
               : launch_inst<false, false, false, 2, kSums>(p, smem_bytes, s);
}

}  // namespace

int pair_cols(int nb_pass) { return (2 * nb_pass + 31) / 32 * 32; }

cudaError_t pair_clusters(int *n) {
  static AskedOnce<int> asked;
  return asked.get(n, [](int *k) {
    int dev = 0, sms = 0;
    auto kern = bf_form_beams_pair<false, false, false, 2, true>;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = kPairSmem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(k, kern, &cfg);
    *k = std::min(*k, sms / 2);
    if (e != cudaSuccess) (void)cudaGetLastError();
    return e;
  });
}

cudaError_t pair_launch_shape(int64_t D, int max_nb_pass, int groups, int *stages) {
  PairParams p{};
  int smem_bytes = 0;
  const cudaError_t e = plan_pair(p, D, max_nb_pass, false, groups, &smem_bytes);
  *stages = p.stages;
  return e;
}

cudaError_t pair_plan(int64_t D, int max_nb_pass, bool two_pass, int groups, int *out) {
  PairParams p{};
  int smem_bytes = 0;
  const cudaError_t e = plan_pair(p, D, max_nb_pass, two_pass, groups, &smem_bytes);
  if (e != cudaSuccess) return e;
  const int per_half = (kPairAcc - p.ncols) / kStageCols;  // the kernel's
  uint32_t last_col = 0;
  for (int i = 0; i < p.stages; ++i)
    last_col = std::max(last_col, pair_stage_col(i, p.ncols, per_half, kStageCols) + kStageCols);
  const int v[12] = {p.stages, p.wslots, p.raw,    p.sets,   p.share,  p.nk,
                     smem_bytes, kPairCols, p.ncols, kPairAcc, per_half, static_cast<int>(last_col)};
  std::copy(v, v + 12, out);
  return cudaSuccess;
}

cudaError_t launch_pair(const TcProblem &one, int64_t D, int test_stall, int *err, cudaStream_t s) {
  PairParams p{};
  p.one = one;
  p.nprob = 1;
  const int64_t ntiles = tc_problem_tiles(one);
  if (ntiles > 0x7FFFFFFF) return cudaErrorInvalidValue;
  p.ntiles = static_cast<int>(ntiles);
  p.err = err;
  p.test_stall = test_stall;
  int smem_bytes = 0;
  const cudaError_t e = plan_pair(p, D, one.nb_pass, one.npass == 2, 2, &smem_bytes);
  if (e != cudaSuccess) return e;
  return tc_w_offset(one.nb_pass) ? launch_plain<true>(p, smem_bytes, s) : launch_plain<false>(p, smem_bytes, s);
}

cudaError_t launch_pair_grouped(const TcProblem *table, int nprob, int ntiles, int64_t D, int max_nb_pass, bool two_pass,
                                int groups, int test_stall, int *err, cudaStream_t s) {
  PairParams p{};
  p.table = table;
  p.nprob = nprob;
  p.ntiles = ntiles;
  p.err = err;
  p.test_stall = test_stall;
  int smem_bytes = 0;
  const cudaError_t e = plan_pair(p, D, max_nb_pass, two_pass, groups, &smem_bytes);
  if (e != cudaSuccess) return e;
  if (groups == 1) return launch_inst<true, false, false, 1, true>(p, smem_bytes, s);  // only beside two TMEM stages
  return tc_w_offset(max_nb_pass) ? launch_inst<true, false, false, 2, true>(p, smem_bytes, s)
                                  : launch_inst<true, false, false, 2, false>(p, smem_bytes, s);
}

}  // namespace bf
