// Trellis-decode product on the 5th-generation tensor cores (tcgen05 + TMEM), for 9 rows and more.
//
//   Y[t, n] = bf16( svh[n] * H128( sum_k Q[n, k] * Xh[t, k] )[n] (+ residual[t, n]) )
//
// "Swap-AB": the decoded weight block is the UMMA A operand (128 weight rows = the span of one output Hadamard), the
// activations are the B operand (TN tokens), so the fp32 accumulator sits in TMEM as [lane = weight row][column = token].
// Weights are decoded once per CTA and reused by all TN tokens of the tile.
//
// Warp roles (DW + 3 warps, DW = 8 or 16 decode warps):
//   warps 0..DW-1  decode: packed words (shared memory) -> fp16 codes -> A tile in the canonical K-major 128-byte-swizzled UMMA
//                  layout, in teams of four (eight) warps that take the stages in turn; later the epilogue
//   warp DW        producer X: TMA tiles of Xh [tokens x 64] (128-byte swizzle)
//   warp DW+1      MMA issuer: one elected thread; it also owns the TMEM allocation
//   warp DW+2      producer W: bulk copies of the packed words, several stages ahead
//
// A stage holds an A tile and the X tile it meets, with one "full" and one "empty" barrier for both.  What bounded the loop before
// was one thread: with a barrier pair per operand, addresses converted and ring positions divided out at each use, the issuer took
// 950 clocks per 64 columns of K whatever the number of tokens.  Now up to 128 tokens the decode warps' instructions bound it (550
// clocks at 16 tokens and 4 bits: 52 issued per 256 weights and scheduler, in 66 % of the clocks).
//
// A pair of CTAs (kPair, cta_group::2: two weight blocks, the tokens of a tile shared): each CTA loads half of the X tile and the
// tensor cores read both halves.  A 512-token tile streams 64 KB of X per 64 columns of K, and that many bytes out of the L2 for
// every SM at a time took 1700 clocks where the products take 1050; in pairs 1050 it is.  34816 x 5120 at 2048 tokens, 4 bits: 692
// -> 566 us (1.29 PFLOP/s); at 8192 tokens 2246 us.
//
// Split of K (ksplit CTAs of a cluster): for few tokens and short N, where row blocks alone leave SMs idle.  Sums meet over
// distributed shared memory in rank order.
// (The reference engine's counterparts are WMMA kernels whose decoded fragments are shared through LDS, reference:
// third_party/libr4d/r4d_gemm_trellis_nt_m256.hip:1-60; nothing is shared with them.)
#include "sm100_ptx.cuh"
#include "trellis_decode.cuh"

namespace r4dxb {
namespace {

constexpr int kSlabK = 64;                      // K of an A or X tile = one 128-byte swizzle row of fp16
constexpr int kATileBytes = 128 * kSlabK * 2;   // 16 KiB
constexpr int kSmemLimit = 227 * 1024;          // of a CTA that has an SM to itself
constexpr int kSmemHalf = 113 * 1024;           // of two that share one
constexpr int kExtra = 2048;                    // alignment slack and barriers

template <int KB, int TN, int DW, bool kPair>
struct Shape {
  static constexpr int kHalves = TN > 256 ? 2 : 1;          // one MMA covers at most 256 token columns
  static constexpr int kMmaN = TN / kHalves;
  static constexpr int kXRows = kPair ? kMmaN / 2 : kMmaN;  // token rows of a half that this CTA loads
  static constexpr int kXTileBytes = kHalves * kXRows * kSlabK * 2;
  static constexpr int kWordsBytes = 1024 * KB;             // packed words of a slab: 4 k-tiles x 8 n-tiles x 8 KB words
  static constexpr int kBudget = (DW == 8 ? kSmemHalf : kSmemLimit) - kExtra;
  static constexpr int kStageBytes = kATileBytes + kXTileBytes;
  static constexpr bool Fits(int stages, int slots) { return stages * kStageBytes + slots * kWordsBytes <= kBudget; }
  // (with two stages a team, a team decodes while the products of its other stage run)
  static constexpr int kStages = DW == 8 ? (Fits(4, 6) ? 4 : 2) : (Fits(8, 8) ? 8 : (Fits(4, 4) ? 4 : 2));
  // The stages and word slots that a team fills and empties are its own (a barrier that passed from team to team would show a team
  // that is ahead the parity it waits for one phase early), so the ring depths are multiples of the team count.
  static constexpr int kTeams = kStages < DW / 4 ? kStages : DW / 4;
  static constexpr int kTeamWarps = DW / kTeams;
  static constexpr int kSlotsFit = (kBudget - kStages * kStageBytes) / kWordsBytes / kTeams * kTeams;
  static constexpr int kSlots = kSlotsFit < 16 ? kSlotsFit : 16;
  static constexpr uint32_t kTmemCols = TN <= 32 ? 32 : (TN <= 64 ? 64 : (TN <= 128 ? 128 : (TN <= 256 ? 256 : 512)));
  // Epilogue staging, in the (by then drained) rings: [token][weight row] floats.  From 128 tokens a lane finishes 32 rows of one
  // token (row stride 144 floats: the two tokens of a quarter-warp's loads lie in different banks), below a warp takes one token.
  static constexpr bool kWide = TN >= 128;
  static constexpr int kEpiStride = kWide ? 144 : 132;
  static constexpr int kEpiBytes = 32 * kEpiStride * 4;                      // per group of four epilogue warps
  static constexpr int kChunk = TN < 256 ? TN : 256;                         // token columns that meet at a time when K is split
  static constexpr int kEpiGroups = DW / 4 * kEpiBytes, kEpiChunk = kChunk * kEpiStride * 4;
  static constexpr int kRings = kStages * kStageBytes + kSlots * kWordsBytes;
  static constexpr int kEpi = DW == 16 && kEpiChunk > kEpiGroups ? kEpiChunk : kEpiGroups;
  static constexpr int kTotal = (kRings > kEpi ? kRings : kEpi) + kExtra;
  static_assert(kSlots >= kTeams && kTotal <= kBudget + kExtra, "shared memory budget");
  static_assert((2 * kStages + 2 * kSlots + 1) * 8 + 16 <= 1024, "barrier block");
  static_assert(!kPair || kMmaN % 32 == 0, "token columns of a paired product");
};

// Reduce-scatter epilogue (tensor-parallel prefill): instead of its own output tensor, the row-parallel product
// stores every partial row into the receive buffer of the rank that owns the row (rows are dealt out in
// contiguous blocks of rows_per_rank), over NVLink peer mappings, tile by tile as the epilogue produces them;
// one system-scope counter per owner collects the arrivals of every CTA on every rank.
struct RsArgs {
  __nv_bfloat16* recv[8];      // peer-mapped receive buffers, indexed by owner rank: [world(src)][rows_per_rank][N]
  unsigned* cnt[8];            // peer-mapped arrival counters, indexed by owner rank
  int world, rank, rows_per_rank;
};

// Grouped experts: the rows of xh are the (row, expert) pairs sorted by expert; a token tile is one expert's next TN rows.
// offsets [E + 1] and perm [pairs] come from the routing plan, tiles / ntiles from the tile list kernel.
struct GroupArgs {
  const int* offsets;
  const int* perm;             // sorted position -> pair id = output row
  const int* tiles;            // [2 * max_tiles]: (local expert, first sorted row)
  const int* ntiles;
  long long words;             // packed words per expert
  int max_tiles;               // grid height: an upper bound on the tile count
};

struct ProductArgs {
  const uint32_t* words;
  const __half* svh;
  __nv_bfloat16* y;
  const __nv_bfloat16* residual;
  int T, N, K;
  int* status;
  RsArgs rs;
  GroupArgs g;
};

template <int CW>
__device__ __forceinline__ void TmemLoadColumns(uint32_t taddr, uint32_t (&v)[CW]) {
  if constexpr (CW == 32) ptx::TmemLoad32x32(taddr, v);
  else ptx::TmemLoad32x16(taddr, v);
}

// Where the outputs of token t of row block nb go.
template <bool kGrouped>
__device__ __forceinline__ __nv_bfloat16* OutRow(const ProductArgs& a, int t, int nb) {
  if constexpr (kGrouped) return a.y + static_cast<size_t>(__ldg(a.g.perm + t)) * a.N + nb * 128;
  if (a.rs.world > 0) {
    const int owner = t / a.rs.rows_per_rank, tl = t - owner * a.rs.rows_per_rank;
    return a.rs.recv[owner] + (static_cast<size_t>(a.rs.rank) * a.rs.rows_per_rank + tl) * a.N + nb * 128;
  }
  return a.y + static_cast<size_t>(t) * a.N + nb * 128;
}

// The rows of a tile whose wait ran out: NaN instead of what they held before.
template <bool kGrouped>
__device__ __noinline__ void FillNan(const ProductArgs& a, int t0, int t_end) {
  for (int t = t0 + (threadIdx.x >> 5); t < t_end; t += blockDim.x >> 5)
    *reinterpret_cast<uint2*>(OutRow<kGrouped>(a, t, blockIdx.x) + (threadIdx.x & 31) * 4) = make_uint2(0x7FC07FC0u, 0x7FC07FC0u);
}

template <int KB, int TN, int DW, bool kPair, bool kGrouped>
__global__ void __launch_bounds__((DW + 3) * 32, DW == 8 ? 2 : 1)
TrellisProductKernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ ProductArgs a) {
  using S = Shape<KB, TN, DW, kPair>;
  constexpr int kStages = S::kStages, kSlots = S::kSlots, kTeams = S::kTeams, kTeamWarps = S::kTeamWarps;
  extern __shared__ unsigned char smem_dyn[];
  // 1024-byte alignment: required by the swizzled UMMA / TMA tiles
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kTotal - kExtra);
  uint64_t* full = bars;                    // [kStages] A decoded and X landed -> MMA (the second CTA of a pair: X landed)
  uint64_t* empty = full + kStages;         // [kStages] products done -> decode, producer X
  uint64_t* wfull = empty + kStages;        // [kSlots]  producer W -> decode
  uint64_t* wempty = wfull + kSlots;        // [kSlots]  decode -> producer W
  uint64_t* accum = wempty + kSlots;        // [1]       MMA -> epilogue
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t smem_at = ptx::SmemAddr(smem), full_at = ptx::SmemAddr(full), empty_at = ptx::SmemAddr(empty);
  const uint32_t wfull_at = ptx::SmemAddr(wfull), wempty_at = ptx::SmemAddr(wempty), slots_at = smem_at + kStages * S::kStageBytes;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = blockIdx.x;                 // 128-row weight block
  const int prank = kPair ? nb & 1 : 0;      // place in the pair; the first one issues the products
  const int T = a.T, N = a.N, K = a.K;
  const uint32_t* words = a.words;
  const __half* svh = a.svh;
  int t0 = blockIdx.y * TN;                  // first token of the tile
  int t_end = T;                             // rows at and past t_end are not stored
  if constexpr (kGrouped) {
    if (static_cast<int>(blockIdx.y) >= __ldg(a.g.ntiles)) return;       // the whole CTA, before any barrier exists
    const int e = __ldg(a.g.tiles + 2 * blockIdx.y);
    t0 = __ldg(a.g.tiles + 2 * blockIdx.y + 1);
    t_end = __ldg(a.g.offsets + e + 1);
    words += static_cast<long long>(e) * a.g.words;
    svh += static_cast<size_t>(e) * N;
  }
  // this CTA's steps of K (a stage each): all, or an even share where the CTAs of a cluster split K
  const int ksplit = gridDim.z, krank = blockIdx.z;
  const int all_steps = K / kSlabK;
  const int step0 = krank * all_steps / ksplit, steps = (krank + 1) * all_steps / ksplit - step0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::MbarInit(&full[s], !kPair ? kTeamWarps + 1 : (prank == 0 ? 2 * (kTeamWarps + 1) : 1));
      ptx::MbarInit(&empty[s], 1);
    }
    for (int s = 0; s < kSlots; ++s) {
      ptx::MbarInit(&wfull[s], 1);
      ptx::MbarInit(&wempty[s], kTeamWarps);
    }
    ptx::MbarInit(accum, 1);
    *abort_flag = 0;
    ptx::MbarFenceInit();
  }
  if (warp == DW + 1) {
    if constexpr (kPair) {
      ptx::TmemAllocPair(tmem_slot, S::kTmemCols);
      ptx::TmemRelinquishPair();
    } else {
      ptx::TmemAlloc(tmem_slot, S::kTmemCols);
      ptx::TmemRelinquish();
    }
  }
  if (warp == DW && lane == 0) ptx::PrefetchTensorMap(&tmap_x);
  ptx::TcFenceBefore();
  __syncthreads();
  if constexpr (kPair) ptx::ClusterSync();   // the partner's barriers exist before anything arrives at them
  ptx::TcFenceAfter();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == DW) {
    // ---------------- producer X ----------------
    if (ptx::ElectOne()) {
      int s = 0;
      uint32_t phase = 1;
      for (int it = 0; it < steps; ++it) {
        if (!ptx::MbarWaitAt(empty_at + s * 8, phase, abort_flag, 1)) break;
        ptx::MbarArriveExpectTxAt(full_at + s * 8, S::kXTileBytes);
        const uint32_t dst = smem_at + s * S::kStageBytes + kATileBytes;
#pragma unroll
        for (int h = 0; h < S::kHalves; ++h)
          ptx::TmaLoad2DAt(dst + h * (S::kXRows * kSlabK * 2), &tmap_x, full_at + s * 8, (step0 + it) * kSlabK,
                           t0 + h * S::kMmaN + prank * S::kXRows);
        if (++s == kStages) { s = 0; phase ^= 1u; }
      }
    }
  } else if (warp == DW + 2) {
    // ---------------- producer W ----------------
    if (ptx::ElectOne()) {
      constexpr size_t kStepWords = S::kWordsBytes / 4;
      const uint32_t* src = words + static_cast<size_t>(nb) * (K / kSlabK) * (S::kWordsBytes / 4) + step0 * kStepWords;
      int s = 0;
      uint32_t phase = 1;
      for (int it = 0; it < steps; ++it) {
        if (!ptx::MbarWaitAt(wempty_at + s * 8, phase, abort_flag, 7)) break;
        ptx::MbarArriveExpectTxAt(wfull_at + s * 8, S::kWordsBytes);
        ptx::BulkLoadAt(slots_at + s * S::kWordsBytes, src, S::kWordsBytes, wfull_at + s * 8);
        src += kStepWords;
        if (++s == kSlots) { s = 0; phase ^= 1u; }
      }
    }
  } else if (warp == DW + 1) {
    // ---------------- MMA issuer ----------------
    if (ptx::ElectOne()) {
      int s = 0;
      uint32_t phase = 0;
      if (kPair && prank == 1) {
        // the second CTA of a pair: pass on that its X tiles have landed
        const uint32_t leader_full = ptx::MapToRank(full_at, ptx::ClusterRank() & ~1u);
        for (int it = 0; it < steps; ++it) {
          if (!ptx::MbarWaitAt(full_at + s * 8, phase, abort_flag, 2)) break;
          ptx::MbarArriveRemote(leader_full + s * 8);
          if (++s == kStages) { s = 0; phase ^= 1u; }
        }
      } else {
        constexpr uint32_t idesc = ptx::UmmaInstrDescF16(kPair ? 256 : 128, S::kMmaN, false);
        const uint64_t da0 = ptx::UmmaDescSw128(smem_at), db0 = ptx::UmmaDescSw128(smem_at + kATileBytes);     // (the address is the low field, in units of 16 bytes)
        const uint16_t pair_mask = kPair ? static_cast<uint16_t>(3u << (ptx::ClusterRank() & ~1u)) : 0;
        uint32_t accumulate = 0;
        bool ok = true, ready = false;       // ready: this stage was seen full while the last one's products were queued
        int it = 0;
        while (it < steps && ok) {
#pragma unroll                               // (a round of the ring at a time: stage addresses are constants)
          for (int st = 0; st < kStages; ++st) {
            if (it == steps) break;
            if (!ready) ok = ptx::MbarWaitAt(full_at + st * 8, phase, abort_flag, 3);
            if (!ok) break;
            ptx::TcFenceAfter();
#pragma unroll
            for (int h = 0; h < S::kHalves; ++h)
#pragma unroll
              for (int k = 0; k < kSlabK / 16; ++k) {
                const uint64_t da = da0 + (st * S::kStageBytes + k * 32) / 16;
                const uint64_t db = db0 + (st * S::kStageBytes + h * (S::kXRows * kSlabK * 2) + k * 32) / 16;
                if constexpr (kPair) ptx::UmmaF16Pair(tmem_base + h * S::kMmaN, da, db, idesc, k > 0 ? 1u : accumulate);
                else ptx::UmmaF16(tmem_base + h * S::kMmaN, da, db, idesc, k > 0 ? 1u : accumulate);
              }
            accumulate = 1;
            ++it;
            // (the next stage is looked at before the commit, which holds the thread up until the products are under way; past the
            // last one the answer is not used)
            ready = ptx::MbarTestWaitAt(full_at + (st + 1) % kStages * 8, st + 1 == kStages ? phase ^ 1u : phase);
            if constexpr (kPair) ptx::UmmaCommitPairAt(empty_at + st * 8, pair_mask);
            else ptx::UmmaCommitAt(empty_at + st * 8);       // frees the stage once these products have read it
          }
          phase ^= 1u;
        }
        if (ok) {                            // accumulator complete
          if constexpr (kPair) ptx::UmmaCommitPairAt(ptx::SmemAddr(accum), pair_mask);
          else ptx::UmmaCommit(accum);
        }
      }
    }
  } else {
    // ---------------- decode warps ----------------
    // a slab is 32 tiles (4 k-tiles x 8 n-tiles); a warp takes 8 / kTeamWarps of the n-tiles
    // lane slot: row (lane % 16) of the 16-row n-tile, K half (lane / 16) -> conflict-free 16-byte stores
    constexpr int kNTiles = 8 / kTeamWarps, NW = 8 * KB;
    const int row_in_tile = lane & 15, khalf = lane >> 4;
    const int team = warp / kTeamWarps, j0 = warp % kTeamWarps * kNTiles;
    TrellisLane<KB> tl;
    tl.Init(2 * row_in_tile + khalf);
    const uint32_t arrive_at = kPair ? ptx::MapToRank(full_at, ptx::ClusterRank() & ~1u) : full_at;
    const int r0 = j0 * 16 + row_in_tile;
    unsigned char* at0 = smem + (r0 >> 3) * 1024 + (r0 & 7) * 128;
    bool ok = true;
    int s = team, sw = team;
    uint32_t phase = 1, wphase = 0;
    for (int it = team; it < steps; it += kTeams) {
      ok = ptx::MbarWaitAt(wfull_at + sw * 8, wphase, abort_flag, 4) && ptx::MbarWaitAt(empty_at + s * 8, phase, abort_flag, 5);
      if (!ok) break;
      unsigned char* at = at0 + s * S::kStageBytes;
      const uint32_t* tw0 = reinterpret_cast<const uint32_t*>(smem + kStages * S::kStageBytes + sw * S::kWordsBytes) + j0 * NW;
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        const int chunk = ((kt * 2 + khalf) ^ (row_in_tile & 7)) << 4;         // 16-byte chunk inside the 128-byte row
#pragma unroll
        for (int j = 0; j < kNTiles; ++j) {
          const uint32_t* tw = tw0 + (kt * 8 + j) * NW;
          uint32_t hi, lo;
          tl.Window(tw[tl.i0], tw[tl.i1], (KB == 4) ? 0u : tw[tl.i2], hi, lo);
          __half2 w[4];
          TrellisDecode8<KB>(hi, lo, w);
          *reinterpret_cast<uint4*>(at + j * 2048 + chunk) = *reinterpret_cast<const uint4*>(w);
        }
      }
      ptx::FenceProxyAsyncShared();          // generic-proxy stores -> visible to the tensor core (async proxy)
      __syncwarp();
      if (lane == 0) {
        if constexpr (kPair) ptx::MbarArriveRemote(arrive_at + s * 8);
        else ptx::MbarArriveAt(arrive_at + s * 8);
        ptx::MbarArriveAt(wempty_at + sw * 8);
      }
      if ((s += kTeams) >= kStages) { s -= kStages; phase ^= 1u; }
      if ((sw += kTeams) >= kSlots) { sw -= kSlots; wphase ^= 1u; }
    }

    // ---------------- epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31 ----------------
    // Groups of four warps take 32-column chunks round-robin; a group stages its chunk through its own transpose buffer, which
    // lives in the rings (every stage has drained by now).
    if (ok) ok = ptx::MbarWait(accum, 0, abort_flag, 6);
    ptx::TcFenceAfter();
    constexpr int kGroups = DW / 4;
    constexpr int CW = TN < 32 ? 16 : 32;    // columns per TMEM load
    const int q = warp & 3, grp = warp >> 2;
    const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    auto out_row = [&](int t) { return OutRow<kGrouped>(a, t, nb); };
    auto to_row = [&](int t, int r, uint2 v) { *reinterpret_cast<uint2*>(out_row(t) + r) = v; };
    // four outputs (rows r ..) of token t: residual and rounding
    auto round4 = [&](int t, int r, float o0, float o1, float o2, float o3) {
      if (a.residual != nullptr) {
        const uint2 rv = *reinterpret_cast<const uint2*>(a.residual + static_cast<size_t>(t) * N + nb * 128 + r);
        o0 += BfLo(rv.x); o1 += BfHi(rv.x); o2 += BfLo(rv.y); o3 += BfHi(rv.y);
      }
      return make_uint2(PackBf16(o0, o1), PackBf16(o2, o3));
    };
    const float inv_sqrt = 0.08838834764831845f;
    // Tokens [c, c + kTokens) of the tile out of their sums: `load(c, row)` gives four weight rows of a token, `store(t, row, v)`
    // takes four outputs.
    constexpr int kTokens = S::kWide ? 8 : 1;
    auto finish = [&](int c, int c_end, auto load, auto store) {
      if constexpr (S::kWide) {
        // a lane has rows 16 i + 4 p + e (i < 8, e < 4) of one token: five Hadamard stages in registers, two between lanes
        const int p = lane & 3;
        c += lane >> 2;
        const int ct = min(c, c_end - 1);    // (lanes past the end repeat the last token)
        float v[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 f = load(ct, 16 * i + 4 * p);
          v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
        }
        float2 w[16];                        // (both halves of a pair per instruction from the second stage on)
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = make_float2(v[2 * i] + v[2 * i + 1], v[2 * i] - v[2 * i + 1]);
#pragma unroll
        for (int m = 1; m < 16; m <<= 1)
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (!(i & m)) {
              const float2 x = w[i], z = w[i | m];
              w[i] = ptx::Add2(x, z);
              w[i | m] = ptx::Fma2(z, make_float2(-1.f, -1.f), x);
            }
#pragma unroll
        for (int m = 1; m < 4; m <<= 1) {
          const float sign = (lane & m) ? -1.f : 1.f;
#pragma unroll
          for (int i = 0; i < 16; ++i)
            w[i] = ptx::Fma2(w[i], make_float2(sign, sign),
                             make_float2(__shfl_xor_sync(0xffffffffu, w[i].x, m), __shfl_xor_sync(0xffffffffu, w[i].y, m)));
        }
        __syncwarp();                        // (every lane has its sums: `store` may put the outputs in their place)
        if (c < c_end) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = 16 * i + 4 * p;
            const uint2 sv = *reinterpret_cast<const uint2*>(svh + nb * 128 + r);
            const __half2 s01 = *reinterpret_cast<const __half2*>(&sv.x), s23 = *reinterpret_cast<const __half2*>(&sv.y);
            store(t0 + c, r, round4(t0 + c, r, w[2 * i].x * inv_sqrt * __low2float(s01), w[2 * i].y * inv_sqrt * __high2float(s01),
                                    w[2 * i + 1].x * inv_sqrt * __low2float(s23), w[2 * i + 1].y * inv_sqrt * __high2float(s23)));
          }
        }
      } else {
        const float4 p = load(c, lane * 4);
        float f[4] = {p.x, p.y, p.z, p.w};
        WarpFwht128(f);
        const uint2 sv = *reinterpret_cast<const uint2*>(svh + nb * 128 + lane * 4);
        const __half2 s01 = *reinterpret_cast<const __half2*>(&sv.x), s23 = *reinterpret_cast<const __half2*>(&sv.y);
        store(t0 + c, lane * 4, round4(t0 + c, lane * 4, f[0] * inv_sqrt * __low2float(s01), f[1] * inv_sqrt * __high2float(s01),
                                       f[2] * inv_sqrt * __low2float(s23), f[3] * inv_sqrt * __high2float(s23)));
      }
    };
    const int tile_end = min(TN, t_end - t0);            // tokens of this tile
    if (DW == 16 && ksplit > 1) {
      // K was split: the CTAs of the cluster lay their sums side by side in shared memory, a chunk of token columns at a time, and
      // each finishes its share of the tokens, adding up over distributed shared memory in rank order
      float* sums = reinterpret_cast<float*>(smem);
      for (int c0 = 0; c0 < tile_end; c0 += S::kChunk) {
        const int c_end = min(c0 + S::kChunk, tile_end);
        for (int cc = c0 + grp * CW; cc < c_end; cc += kGroups * CW) {
          uint32_t v[CW];
          if (ok) {
            TmemLoadColumns<CW>(tmem_lane + cc, v);
            ptx::TmemLoadWait();
          }
#pragma unroll
          for (int c = 0; c < CW; ++c)       // (a wait that ran out shows as NaN)
            sums[(cc - c0 + c) * S::kEpiStride + q * 32 + lane] = ok ? __uint_as_float(v[c]) : __int_as_float(0x7FC00000);
        }
        ptx::ClusterSync();
        for (int c = c0 + (warp * ksplit + krank) * kTokens; c < c_end; c += DW * ksplit * kTokens)
          finish(c, c_end, [&](int ct, int row) {
            float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int r = 0; r < ksplit; ++r) {
              const float4 x = ptx::LoadRemote4(smem_at + ((ct - c0) * S::kEpiStride + row) * 4, kPair ? 2 * r + prank : r);
              f.x += x.x; f.y += x.y; f.z += x.z; f.w += x.w;
            }
            return f;
          }, to_row);
        ptx::ClusterSync();
      }
    } else {
      // Two buffers a group where they fit: a warp loads its next columns while others finish theirs.  Wide tiles: the rounded rows
      // of a token replace its sums and leave as one bulk copy of 256 bytes (stores of a lane's rows, 32 bytes of eight tokens
      // each, took half of the epilogue: 27k of 115k clocks a tile at 512 tokens).
      constexpr int kBuffers = 2 * S::kEpiGroups <= S::kRings ? 2 : 1;
      const bool bulk = S::kWide && a.rs.world == 0 && (reinterpret_cast<uintptr_t>(a.y) & 15) == 0;
      int buf = 0;
      for (int c0 = grp * 32; c0 < tile_end; c0 += kGroups * 32, buf ^= kBuffers - 1) {
        float* epi = reinterpret_cast<float*>(smem + (grp * kBuffers + buf) * S::kEpiBytes);
        if (ok) {
          uint32_t v[CW];
          TmemLoadColumns<CW>(tmem_lane + c0, v);
          ptx::TmemLoadWait();
#pragma unroll
          for (int c = 0; c < CW; ++c) epi[c * S::kEpiStride + q * 32 + lane] = __uint_as_float(v[c]);
        }
        if (kBuffers == 2 && bulk) ptx::BulkStoreWaitRead();      // (the copies out of the other buffer, before anyone writes there)
        asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
        const int c_end = min(c0 + CW, tile_end);
        auto load = [&](int ct, int row) { return *reinterpret_cast<const float4*>(epi + (ct - c0) * S::kEpiStride + row); };
        if (bulk) {
          const int c = c0 + q * kTokens;
          if (ok && c < c_end) {
            finish(c, c_end, load, [&](int t, int r, uint2 v) {
              *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(epi + (t - t0 - c0) * S::kEpiStride) + r) = v;
            });
            ptx::FenceProxyAsyncShared();
            __syncwarp();
            if (lane < kTokens && c + lane < c_end) {
              ptx::BulkStore(out_row(t0 + c + lane), ptx::SmemAddr(epi + (c + lane - c0) * S::kEpiStride), 256);
              ptx::BulkStoreCommit();
            }
            if (kBuffers == 1) ptx::BulkStoreWaitRead();
          }
        } else if (ok) {
          for (int c = c0 + q * kTokens; c < c_end; c += 4 * kTokens) finish(c, c_end, load, to_row);
        }
        if (kBuffers == 1) asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
      }
      if (bulk) ptx::BulkStoreWait();
    }
    if (!kGrouped && a.rs.world > 0) {
      // every partial row of this tile is on its way: publish them, then count this CTA in at each owner it wrote to
      // (also when a wait ran out: the peers must not wait for a CTA that gave up; the status word tells the host)
      __threadfence_system();
      asm volatile("bar.sync 6, %0;" ::"r"(DW * 32) : "memory");
      if (threadIdx.x == 0) {
        const int t_last = min(t0 + TN, T) - 1;
        for (int o = t0 / a.rs.rows_per_rank; o <= t_last / a.rs.rows_per_rank; ++o) atomicAdd_system(a.rs.cnt[o], 1u);
      }
    }
  }
  if (DW == 16 && warp >= DW && ksplit > 1) {
    // the other warps take part in the cluster's barriers
    __syncwarp();
    for (int c0 = 0; c0 < min(TN, t_end - t0); c0 += S::kChunk) {
      ptx::ClusterSync();
      ptx::ClusterSync();
    }
  }

  // ---------------- teardown ----------------
  ptx::TcFenceBefore();
  __syncthreads();
  if (*abort_flag != 0) {
    FillNan<kGrouped>(a, t0, min(t0 + TN, t_end));
    // give copies that may still be in flight time to land before the shared memory goes away
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    if (threadIdx.x == 0) atomicExch(a.status, *abort_flag);
  }
  if constexpr (kPair) ptx::ClusterSync();   // neither CTA of a pair leaves or frees tensor memory while the other still reads
  if (warp == DW + 1) {
    if constexpr (kPair) ptx::TmemDeallocPair(tmem_base, S::kTmemCols);
    else ptx::TmemDealloc(tmem_base, S::kTmemCols);
  }
}

template <int KB, int TN, int DW, bool kPair, bool kGrouped>
int Launch(const void* xh, const ProductArgs& a, int ksplit, cudaStream_t stream) {
  using S = Shape<KB, TN, DW, kPair>;
  static_assert(DW == 8 || kGrouped || S::kTotal >= ptx::kProductAlone, "CTAs of a cluster wait for each other with tensor memory in hand");
  CUtensorMap tmap;
  const int rc = MakeTensorMap2D16(&tmap, xh, static_cast<uint64_t>(a.T), static_cast<uint64_t>(a.K), S::kXRows, kSlabK, false);
  if (rc) return rc;
  auto kern = TrellisProductKernel<KB, TN, DW, kPair, kGrouped>;
  const cudaError_t ea = AllowAllSharedMemory(kern);
  if (ea != cudaSuccess) return static_cast<int>(ea);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.N / 128, kGrouped ? a.g.max_tiles : (a.T + TN - 1) / TN, ksplit);
  cfg.blockDim = dim3((DW + 3) * 32, 1, 1);
  cfg.dynamicSmemBytes = S::kTotal;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kPair ? 2 : 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = ksplit;
  cfg.attrs = attr;
  cfg.numAttrs = kPair || ksplit > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tmap, a);
  ++g_launch_count;
  return static_cast<int>(e);
}

template <int KB>
int LaunchTile(const void* xh, const ProductArgs& a, int tn, int ksplit, cudaStream_t s) {
  // wide tiles in pairs of weight blocks, where there is an even number of them and the cluster stays within eight CTAs
  const bool pair = a.N % 256 == 0 && ksplit <= 4;
  // few tokens and more row blocks than SMs: eight decode warps, so that two CTAs share an SM and the second half of the blocks does
  // not wait for the first (34816 x 5120: 16 tokens 63 against 61 us at 4 bits, 64 tokens 88 against 76 at 5 bits)
  const bool two = ksplit == 1 && (a.N / 128) * ((a.T + tn - 1) / tn) > 148;
  switch (tn) {
    case 16: return two ? Launch<KB, 16, 8, false, false>(xh, a, ksplit, s) : Launch<KB, 16, 16, false, false>(xh, a, ksplit, s);
    case 32: return two ? Launch<KB, 32, 8, false, false>(xh, a, ksplit, s) : Launch<KB, 32, 16, false, false>(xh, a, ksplit, s);
    case 64: return two ? Launch<KB, 64, 8, false, false>(xh, a, ksplit, s) : Launch<KB, 64, 16, false, false>(xh, a, ksplit, s);
    case 128: return Launch<KB, 128, 16, false, false>(xh, a, ksplit, s);
    case 192: return Launch<KB, 192, 16, false, false>(xh, a, ksplit, s);
    case 256: return pair ? Launch<KB, 256, 16, true, false>(xh, a, ksplit, s) : Launch<KB, 256, 16, false, false>(xh, a, ksplit, s);
    case 384: return pair ? Launch<KB, 384, 16, true, false>(xh, a, ksplit, s) : Launch<KB, 384, 16, false, false>(xh, a, ksplit, s);
    case 512: return pair ? Launch<KB, 512, 16, true, false>(xh, a, ksplit, s) : Launch<KB, 512, 16, false, false>(xh, a, ksplit, s);
    default: return R4DXB_BAD_ARG;
  }
}

int LaunchKb(const void* xh, const ProductArgs& a, int kb, int tn, int ksplit, cudaStream_t s) {
  switch (kb) {
    case 3: return LaunchTile<3>(xh, a, tn, ksplit, s);
    case 4: return LaunchTile<4>(xh, a, tn, ksplit, s);
    case 5: return LaunchTile<5>(xh, a, tn, ksplit, s);
    default: return R4DXB_BAD_ARG;
  }
}

template <int KB>
int LaunchGrouped(const void* xh, const ProductArgs& a, int tn, int decode_warps, cudaStream_t s) {
  // eight decode warps: 352 threads per CTA, so two CTAs share an SM and one tile's prologue and epilogue overlap the
  // other's main loop (an expert tile has little K: the fixed part of a CTA is most of its time)
  if (decode_warps == 8) {
    switch (tn) {
      case 16: return Launch<KB, 16, 8, false, true>(xh, a, 1, s);
      case 32: return Launch<KB, 32, 8, false, true>(xh, a, 1, s);
      case 64: return Launch<KB, 64, 8, false, true>(xh, a, 1, s);
      case 96: return Launch<KB, 96, 8, false, true>(xh, a, 1, s);
      case 128: return Launch<KB, 128, 8, false, true>(xh, a, 1, s);
      default: return R4DXB_BAD_ARG;
    }
  }
  switch (tn) {
    case 16: return Launch<KB, 16, 16, false, true>(xh, a, 1, s);
    case 32: return Launch<KB, 32, 16, false, true>(xh, a, 1, s);
    case 64: return Launch<KB, 64, 16, false, true>(xh, a, 1, s);
    case 96: return Launch<KB, 96, 16, false, true>(xh, a, 1, s);
    case 128: return Launch<KB, 128, 16, false, true>(xh, a, 1, s);
    case 256: return Launch<KB, 256, 16, false, true>(xh, a, 1, s);
    default: return R4DXB_BAD_ARG;
  }
}

ProductArgs MakeArgs(const void* w, const void* svh, void* y, const void* residual, int T, int N, int K, int* status) {
  ProductArgs a = {};
  a.words = static_cast<const uint32_t*>(w);
  a.svh = static_cast<const __half*>(svh);
  a.y = static_cast<__nv_bfloat16*>(y);
  a.residual = static_cast<const __nv_bfloat16*>(residual);
  a.T = T;
  a.N = N;
  a.K = K;
  a.status = status;
  return a;
}

}  // namespace

int g_grouped_decode_warps = 0;      // 0: by tile size (r4dxb_set_gemm_decode_warps)

int TrellisProduct(const void* w, const void* svh, const void* xh, void* y, const void* residual, int T, int N, int K, int kb, int tn,
                   int ksplit, int* status, cudaStream_t s) {
  return LaunchKb(xh, MakeArgs(w, svh, y, residual, T, N, K, status), kb, tn, ksplit, s);
}

}  // namespace r4dxb

using namespace r4dxb;

extern "C" {

/* Grouped experts on the tensor cores (prefill and wide batches of the mixture-of-experts block):
 * y[perm[p]] = svh[e] * H128(xh[p] Q_e^T); max_tiles >= P / tn + E bounds the grid. */
int r4dxb_trellis_gemm_grouped(const void* words, const void* svh, const void* xh, void* y, const int* offsets, const int* perm,
                               const int* tiles, const int* ntiles, int max_tiles, int P, int E, int N, int K, int kb, int tn,
                               int* status, void* stream) {
  if (P < 1 || E < 1 || N % 128 || K % 128 || max_tiles < 1 || max_tiles > 65535) return R4DXB_BAD_ARG;
  ProductArgs a = MakeArgs(words, svh, y, nullptr, P, N, K, status);
  a.g.offsets = offsets;
  a.g.perm = perm;
  a.g.tiles = tiles;
  a.g.ntiles = ntiles;
  a.g.words = static_cast<long long>(N / 16) * (K / 16) * 8 * kb;
  a.g.max_tiles = max_tiles;
  // us a block of 512 experts (hidden 2048) with eight / sixteen decode warps: 600 rows 786 / 1018, 2048 rows 1000 / 1228, 4096 rows
  // (tiles of 128) 1368 / 1558
  const int dw = g_grouped_decode_warps ? g_grouped_decode_warps : (tn <= 128 ? 8 : 16);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (kb) {
    case 3: return LaunchGrouped<3>(xh, a, tn, dw, s);
    case 4: return LaunchGrouped<4>(xh, a, tn, dw, s);
    case 5: return LaunchGrouped<5>(xh, a, tn, dw, s);
    default: return R4DXB_BAD_ARG;
  }
}

/* Row-parallel product with the reduce-scatter in its epilogue: partial row t goes to rank t / rows_per_rank, into
 * recv[owner] + (rank * rows_per_rank + t % rows_per_rank) * N (bf16), and every CTA adds 1 to cnt[owner] for each
 * owner its token tile touches, after its rows are visible at system scope.  recv / cnt: `world` peer-mapped pointers. */
int r4dxb_trellis_gemm_rs(const void* w, const void* svh, const void* xh, int T, int N, int K, int kb, int tn, int* status,
                          void* const* recv, void* const* cnt, int world, int rank, int rows_per_rank, void* stream) {
  if (T < 1 || N % 128 || K % 128 || world < 2 || world > 8 || rank < 0 || rank >= world || rows_per_rank < 1 ||
      static_cast<long long>(rows_per_rank) * world < T)
    return R4DXB_BAD_ARG;
  ProductArgs a = MakeArgs(w, svh, nullptr, nullptr, T, N, K, status);
  for (int p = 0; p < world; ++p) {
    a.rs.recv[p] = static_cast<__nv_bfloat16*>(recv[p]);
    a.rs.cnt[p] = static_cast<unsigned*>(cnt[p]);
  }
  a.rs.world = world;
  a.rs.rank = rank;
  a.rs.rows_per_rank = rows_per_rank;
  return LaunchKb(xh, a, kb, tn, 1, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
