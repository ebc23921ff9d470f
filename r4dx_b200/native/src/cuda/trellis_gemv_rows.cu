// Trellis-decode weight-streaming product for 1..8 activation rows on mma.sync, the weights decoded straight into its operands.
//
//   y[t, n] = bf16( svh[n] * H128( sum_k Q[n, k] * xh[t, k] )[n] (+ residual[t, n]) ),  xh = fp16(H128(suh (.) act(x)))
//
// Operands are those of the prompt path's tcgen05 product: code values as the format defines them (one fp16 rounding), fp16 rows,
// products and sums in fp32.  One m16n8k16 takes 256 weights times up to eight rows, so a weight costs its state's extraction, a
// multiply, a byte sum, half a byte permute and half a multiply-add, whatever the row count.
// (The hash bytes themselves as 8-bit operands, with rows of two signed digits, need neither byte sum nor packing, but multiply
// by code values that are not rounded, and the digits of a row share one exponent: 2.2e-4 of a product against 64 bits where this
// form and the tcgen05 product have 2.0e-4.)
//
// What bounds it: instructions.  Per 256 weights a warp issues 8 extractions, 8 multiplies, 8 byte sums, 4 permutes, 4 multiply-adds
// and one MMA, 41 clocks of a scheduler by themselves.  us at 2 / 4 / 8 rows, 4 bits, L2 flushed, against the CUDA-core kernel
// (trellis_gemv.cu): 34816 x 5120 50 / 50 / 54 (64 / 80 / 118), 5120 x 17408 34 / 34 / 35 (44 / 67 / 98), 16384 x 5120
// 30 / 30 / 30 (40 / 47 / 69), 5120 x 6144 19 / 19 / 19 (22 / 26 / 39).  (The 8-bit form took 44 / 44 / 56, 32 / 32 / 36.)
//
// One row: no MMA but fp16 multiply-adds in the order of the CUDA-core kernel, whose rounding it keeps (up to 3 of 34816 outputs
// differ, by one bf16 step: the fp32 sums are added up in another order).  Multiplies, byte sums and fp16 multiply-adds share a pipe,
// 24 of them per 256 weights at two clocks, with 4 bits 20 of them (every second byte sum runs elsewhere): 40 of the 50 clocks that the
// loop takes.  us at one row, 4 / 5 bits, L2 flushed (CUDA-core kernel): 34816 x 5120 46 / 54 (53 / 62), 5120 x 17408 32 / 36 (37 / 43),
// 16384 x 5120 28 / 32 (32 / 38), 5120 x 6144 18 / 19.5 (19 / 21).  ops/kernels.py:one_row_split says where it serves.
//
// Grouped mode (mixture-of-experts blocks with a few rows per expert): a CTA serves one 128-row block of one tile of the routing
// plan, up to eight rows of one expert; the rows are those of the planned pairs in expert order.  A block of 512
// experts (top 10, hidden 2048) takes 261 / 478 / 620 us at 17 / 64 / 200 rows of x where the tcgen05 tiles of 16 rows take 339 /
// 626 / 798: most experts have one or two rows, and decoding their weights is the work.  (Tiles of four rows: 261 / 478 / 755; with
// most rows routed to a dozen experts they took 329 / 628 us at 64 / 200 rows, these 277 / 452, the tcgen05 tiles 320 / 458.)
//
// Two launches: TrellisRowsInputKernel writes the transformed rows once (every CTA would otherwise repeat the transform: at 8 rows
// of 5120 columns that was 74k of 103k clocks), then one CTA per (128-row block, K slice) streams words
// through a ring of bulk copies - filled before the wait for the rows - and `ksplit` CTAs of a cluster add up over
// distributed shared memory in rank order.
#include <cooperative_groups.h>

#include "sm100_ptx.cuh"
#include "trellis_decode.cuh"

namespace cg = cooperative_groups;

namespace r4dxb {
namespace {

constexpr int kTeamWarps = 4;            // warps that share one K block
constexpr int kTeams = 4;
constexpr int kConsumerWarps = kTeamWarps * kTeams;
constexpr int kThreads = (kConsumerWarps + 1) * 32;
constexpr int kSums = 2 * kTeams;        // partial sums of a row inside a CTA
constexpr int kMaxStages = 6;
// The teams take the K blocks in turn, so with six stages a stage passes from one team to another.  A barrier per stage would then
// alias: a team that never waited for a stage's phase 0 finds the parity of its phase 1 satisfied while the copies of phase 0 are
// still on their way.  Block b therefore signals through barrier b % kBarriers: all blocks of a barrier belong to one team, which
// (like the producer) waits for its phases in order.
constexpr int kBarriers = 12;
static_assert(kBarriers % kTeams == 0 && kBarriers >= kMaxStages, "the blocks of a barrier belong to one team, and at most one of them is in flight");
constexpr int kMaxSiblings = 3;

struct RowsArgs {
  const __nv_bfloat16* x;
  const __nv_bfloat16* residual;
  const __nv_bfloat16* norm_w;           // prologue mode 1
  float eps;
  int T, K, kblocks_per_cta, stages, act;
  const __half* xh;                      // [siblings][T][K], the k-tiles of every 128 columns in StoredTile order
  // one to three weights that read the same rows through the same prologue; blockIdx.y runs over all their row blocks
  // grouped mode
  const int* g_offsets;                  // [E + 1] into g_perm
  const int* g_perm;                     // pair of each sorted position = output row; its input row is pair / g_xdiv
  const int* g_tiles;                    // (expert, first sorted position) per tile, *g_ntiles of them
  const int* g_ntiles;
  int g_experts, g_xdiv, g_tile_rows;
  long long g_words;                     // words of one expert
  int* status;                           // receives 700 + role code (390: split-K hand-off) when a bounded wait ran out
  int count;
  struct Weight {
    const uint32_t* words;
    const __half* suh;
    const __half* svh;
    __nv_bfloat16* y;
    int N, nb_end;                       // row blocks [previous nb_end, nb_end) belong to this weight
  } w[kMaxSiblings];
};

struct Ctl {                             // control block at the start of dynamic shared memory
  uint64_t full[kBarriers], empty[kBarriers];   // of block b % kBarriers
  uint64_t red_bar;                      // split-K partials have landed
  uint64_t xfull;                        // rows have landed
  int abort_flag;
  int pad;
  uint32_t fill[10];
};
static_assert(sizeof(Ctl) % 128 == 0, "what follows the control block is 128-byte aligned");

// Place of a k-tile inside its 128 columns of a stored row: the four k-tiles that a quad of lanes reads together (see the main
// loop) lie side by side, 32 bytes each.
__host__ __device__ constexpr int StoredTile(int kt) { return ((kt >> 1) & 1) * 4 + (kt >> 2) * 2 + (kt & 1); }

// bytes between two rows in shared memory: neighbouring rows start 16 bytes apart modulo the banks
__host__ __device__ constexpr int XStride(int kslice) { return kslice * 2 + 16; }

__device__ __forceinline__ void ConsumerSync() { asm volatile("bar.sync 1, %0;" ::"r"(kConsumerWarps * 32) : "memory"); }

__device__ __forceinline__ void MmaF16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float SumSquares8(const uint4& v) {
  return BfLo(v.x) * BfLo(v.x) + BfHi(v.x) * BfHi(v.x) + BfLo(v.y) * BfLo(v.y) + BfHi(v.y) * BfHi(v.y) +
         BfLo(v.z) * BfLo(v.z) + BfHi(v.z) * BfHi(v.z) + BfLo(v.w) * BfLo(v.w) + BfHi(v.w) * BfHi(v.w);
}

// Sum of squares of one eighth of a row (warps 0..7 of a CTA); the eighths are added in order, as in the CUDA-core kernel's
// prologue.
__device__ __forceinline__ float EighthSumSquares(const __nv_bfloat16* row, int K, int warp, int lane) {
  const int kw = (K / 8 + 7) & ~7;    // columns per warp, a multiple of 8
  const int k_lo = warp * kw, k_hi = min(K, k_lo + kw);
  float ss = 0.f;
  for (int k = k_lo + lane * 8; k < k_hi; k += 256) ss += SumSquares8(*reinterpret_cast<const uint4*>(row + k));
  return WarpSum(ss);
}
__device__ __forceinline__ float RowRms(const float* eighths, int K, float eps) {
  float ss = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) ss += eighths[w];
  return rsqrtf(ss / K + eps);
}

// four columns of act(x) * suh, before the Hadamard transform
template <int PRO>
__device__ __forceinline__ void Activate(uint2 xv, uint2 uv, uint2 wv, uint2 sv, float r, int act, float (&v)[4]) {
  if constexpr (PRO == 2) {
    const uint32_t p01 = PackBf16(GateAct(BfLo(xv.x), act) * BfLo(uv.x), GateAct(BfHi(xv.x), act) * BfHi(uv.x));
    const uint32_t p23 = PackBf16(GateAct(BfLo(xv.y), act) * BfLo(uv.y), GateAct(BfHi(xv.y), act) * BfHi(uv.y));
    v[0] = BfLo(p01); v[1] = BfHi(p01); v[2] = BfLo(p23); v[3] = BfHi(p23);
  } else {
    v[0] = BfLo(xv.x); v[1] = BfHi(xv.x); v[2] = BfLo(xv.y); v[3] = BfHi(xv.y);
    if constexpr (PRO == 1) {
      // same rounding point as the standalone norm kernel: the normalised row is a bf16 tensor
      const uint32_t p01 = PackBf16(v[0] * r * (1.f + BfLo(wv.x)), v[1] * r * (1.f + BfHi(wv.x)));
      const uint32_t p23 = PackBf16(v[2] * r * (1.f + BfLo(wv.y)), v[3] * r * (1.f + BfHi(wv.y)));
      v[0] = BfLo(p01); v[1] = BfHi(p01); v[2] = BfLo(p23); v[3] = BfHi(p23);
    }
  }
  const __half2 s01 = *reinterpret_cast<const __half2*>(&sv.x), s23 = *reinterpret_cast<const __half2*>(&sv.y);
  v[0] *= __low2float(s01); v[1] *= __high2float(s01); v[2] *= __low2float(s23); v[3] *= __high2float(s23);
}

// The transformed rows of a launch: grid (T, parts, weights), a warp takes up to kInBlocks 128-column blocks.
constexpr int kInWarps = 16;
constexpr int kInBlocks = 2;
inline int InputParts(int K) { return (K / 128 + kInWarps * kInBlocks - 1) / (kInWarps * kInBlocks); }
// Grouped: grid (pairs, parts), t = sorted position.  A chain of latencies: the signs and norm weights, which no kernel writes,
// are requested before the wait for the previous kernel and all of a warp's activations at once after it.
template <int PRO, bool kGrouped>
__global__ void __launch_bounds__(kInWarps * 32) TrellisRowsInputKernel(RowsArgs a, __half* xh) {
  __shared__ float red[8];
  const int t = blockIdx.x, sib = blockIdx.z, T = a.T, K = a.K;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const __half* suh = a.w[sib].suh;
  int xrow = t;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if constexpr (kGrouped) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (t >= __ldg(a.g_offsets + a.g_experts)) return;       // (pairs of experts that live elsewhere)
    const int lo = LastAtOrBelow(a.g_offsets, a.g_experts, t);
    suh += static_cast<size_t>(lo) * K;
    xrow = __ldg(a.g_perm + t) / a.g_xdiv;
  }
  const int b0 = blockIdx.y * warps * kInBlocks + warp, blocks = K / 128;      // this warp's blocks: b0, b0 + warps, ..
  uint2 sv[kInBlocks], nv[kInBlocks], xv[kInBlocks], uv[kInBlocks];
#pragma unroll
  for (int i = 0; i < kInBlocks; ++i) {
    const int k = min(b0 + i * warps, blocks - 1) * 128 + lane * 4;
    sv[i] = *reinterpret_cast<const uint2*>(suh + k);
    nv[i] = PRO == 1 ? *reinterpret_cast<const uint2*>(a.norm_w + k) : make_uint2(0u, 0u);
  }
  const __nv_bfloat16* xin = a.x + static_cast<size_t>(xrow) * (PRO == 2 ? 2 * static_cast<size_t>(K) : K);
  if constexpr (!kGrouped) asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
  for (int i = 0; i < kInBlocks; ++i) {
    const int k = min(b0 + i * warps, blocks - 1) * 128 + lane * 4;
    xv[i] = *reinterpret_cast<const uint2*>(xin + k);
    uv[i] = PRO == 2 ? *reinterpret_cast<const uint2*>(xin + K + k) : make_uint2(0u, 0u);
  }
  float r = 0.f;
  if constexpr (PRO == 1) {
    if (warp < 8) {
      const float ss = EighthSumSquares(xin, K, warp, lane);
      if (lane == 0) red[warp] = ss;
    }
    __syncthreads();
    r = RowRms(red, K, a.eps);
  }
  __half* dst = xh + (static_cast<size_t>(sib) * T + t) * K + StoredTile(lane >> 2) * 16 + (lane & 3) * 4;
#pragma unroll
  for (int i = 0; i < kInBlocks; ++i) {
    if (b0 + i * warps >= blocks) break;
    float v[4];
    Activate<PRO>(xv[i], uv[i], nv[i], sv[i], r, a.act, v);
    WarpFwht128(v);
    const float inv_sqrt = 0.08838834764831845f;   // 1 / sqrt(128)
    const __half2 o01 = __floats2half2_rn(v[0] * inv_sqrt, v[1] * inv_sqrt), o23 = __floats2half2_rn(v[2] * inv_sqrt, v[3] * inv_sqrt);
    uint2 ov;
    ov.x = *reinterpret_cast<const uint32_t*>(&o01);
    ov.y = *reinterpret_cast<const uint32_t*>(&o23);
    *reinterpret_cast<uint2*>(dst + (b0 + i * warps) * 128) = ov;
  }
}

// two code values of a row of a tile (positions J, J + 1) as an operand register
template <int KB, int J>
__device__ __forceinline__ uint32_t Code2(const uint32_t (&w)[3]) {
  const __half2 q = TrellisCode2<KB>(TrellisRow<KB>::template State<J>(w[2], w[1], w[0]), TrellisRow<KB>::template State<J + 1>(w[2], w[1], w[0]));
  return *reinterpret_cast<const uint32_t*>(&q);
}

// The 16 code values of a row of a tile times the 16 columns x, onto the partial sums of its two halves: one fp16 multiply-add per
// pair, the eight columns of a half in order.
template <int KB>
__device__ __forceinline__ void RowDot(const uint32_t (&w)[3], const uint4& xlo, const uint4& xhi, __half2 (&h)[2]) {
  const uint32_t x[8] = {xlo.x, xlo.y, xlo.z, xlo.w, xhi.x, xhi.y, xhi.z, xhi.w};
#define R4DXB_STEP(I)                                                                                          \
  {                                                                                                           \
    const uint32_t q = Code2<KB, 2 * I>(w);                                                                    \
    h[I / 4] = __hfma2(*reinterpret_cast<const __half2*>(&q), *reinterpret_cast<const __half2*>(&x[I]), h[I / 4]); \
  }
  R4DXB_STEP(0) R4DXB_STEP(1) R4DXB_STEP(2) R4DXB_STEP(3) R4DXB_STEP(4) R4DXB_STEP(5) R4DXB_STEP(6) R4DXB_STEP(7)
#undef R4DXB_STEP
}

template <int KB, int TMAX, bool kGrouped = false>
__global__ void __launch_bounds__(kThreads, TMAX > 4 && !kGrouped ? 1 : 2) TrellisRowsKernel(RowsArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int ksplit = gridDim.x;
  const int krank = blockIdx.x;            // == rank inside the cluster
  int nb = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int sidx = 0;                            // the weight this CTA serves
  while (sidx + 1 < a.count && nb >= a.w[sidx].nb_end) ++sidx;
  if (sidx > 0) nb -= a.w[sidx - 1].nb_end;
  const int N = a.w[sidx].N, K = a.K;
  int T = a.T, start = 0;                  // rows of this CTA, the first one's place in xh
  const uint32_t* words = a.w[sidx].words;
  const __half* svh = a.w[sidx].svh;
  if constexpr (kGrouped) {
    if (static_cast<int>(blockIdx.z) >= __ldg(a.g_ntiles)) return;       // the whole CTA (a cluster of one), before any barrier exists
    const int e = __ldg(a.g_tiles + 2 * blockIdx.z);
    start = __ldg(a.g_tiles + 2 * blockIdx.z + 1);
    T = min(a.g_tile_rows, __ldg(a.g_offsets + e + 1) - start);
    words += static_cast<size_t>(e) * a.g_words;
    svh += static_cast<size_t>(e) * N;
  }
  // K blocks are dealt out as evenly as the count allows (17 blocks over 4 CTAs: 4, 4, 4, 5); shared memory is laid
  // out for the longest slice
  const int kslice = a.kblocks_per_cta * 128;
  const int kb_lo = krank * (K / 128) / ksplit;
  const int my_blocks = (krank + 1) * (K / 128) / ksplit - kb_lo;
  constexpr int NW = 8 * KB;
  constexpr int kStageBytes = 8 * 8 * NW * 4;     // 8 k-tiles x 8 n-tiles
  // A stage is two bulk copies of four k-tiles each, 64 bytes apart modulo the banks; a quad reads two k-tiles of either half, so
  // its words spread over all banks.  (Padding every k-tile took eight copies of 1 KB, and the copy engine then delivered
  // 8 bytes per clock and SM: 53k instead of 35k clocks for the main loop of 40 blocks.)
  constexpr int kTileBytes = 8 * NW * 4;
  constexpr int kHalfSlot = 4 * kTileBytes + 64;
  constexpr int kStageSlot = 2 * kHalfSlot;

  const int xstride = XStride(kslice);
  Ctl* ctl = reinterpret_cast<Ctl*>(smem_raw);
  float* loc = reinterpret_cast<float*>(smem_raw + sizeof(Ctl));                     // [kSums][TMAX][128] sums of (k-tile half, team)
  float* part = loc + kSums * TMAX * 128;                                             // [ksplit][TMAX][128] (used on cluster rank 0)
  unsigned char* xs = reinterpret_cast<unsigned char*>(part + (ksplit > 1 ? ksplit : 0) * TMAX * 128);   // rows: [TMAX][xstride]
  unsigned char* wst = xs + static_cast<size_t>(TMAX) * xstride;                     // [stages][kStageSlot]
  uint64_t* red_bar = &ctl->red_bar;
  volatile int* abort_flag = &ctl->abort_flag;
  const uint32_t full_at = ptx::SmemAddr(ctl->full), wst_at = ptx::SmemAddr(wst);      // (the empty barriers follow the full ones)

  if (threadIdx.x == 0) {
    for (int s = 0; s < kBarriers; ++s) {
      ptx::MbarInit(&ctl->full[s], 1);
      ptx::MbarInit(&ctl->empty[s], kTeamWarps);
    }
    ptx::MbarInit(red_bar, ksplit * kConsumerWarps);
    ptx::MbarInit(&ctl->xfull, 1);
    *abort_flag = 0;
    ptx::MbarFenceInit();
  }
  __syncthreads();
  // Cluster rendezvous, split in two: arrive now, wait only just before the first remote write, so
  // the weight stream overlaps with it.  It guarantees that rank 0's reduction
  // barrier is initialised before any peer CTA touches it.
  if (ksplit > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  // let the next kernel in the stream begin its own launch and weight prefetch
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == kConsumerWarps) {
    // ---------------- producer: this CTA's words through the stage ring, the rows once the ring is full ----------------
    if (lane == 0) {
      const unsigned char* src = reinterpret_cast<const unsigned char*>(words) +
                                 (static_cast<size_t>(nb) * (K / 128) + static_cast<size_t>(kb_lo)) * kStageBytes;
      int s = 0, b = 0;            // stage and barrier of block `it`
      int eb = 0;                  // barrier of the block that held the stage before, and the parity of its release
      uint32_t ephase = 0;
      for (int it = 0; it <= my_blocks; ++it) {
        if (it == min(a.stages, my_blocks)) {
          asm volatile("griddepcontrol.wait;" ::: "memory");
          ptx::MbarArriveExpectTx(&ctl->xfull, T * my_blocks * 256);
          const __half* xsrc = a.xh + (static_cast<size_t>(sidx) * T + start) * K + kb_lo * 128;
          for (int t = 0; t < T; ++t)
            ptx::BulkLoad(xs + static_cast<size_t>(t) * xstride, xsrc + static_cast<size_t>(t) * K, my_blocks * 256, &ctl->xfull);
        }
        if (it == my_blocks) break;
        if (it >= a.stages) {
          if (!ptx::MbarWaitAt(full_at + (kBarriers + eb) * 8, ephase, abort_flag, 1)) break;
          if (++eb == kBarriers) { eb = 0; ephase ^= 1u; }
        }
        ptx::MbarArriveExpectTxAt(full_at + b * 8, kStageBytes);
        ptx::BulkLoadAt(wst_at + s * kStageSlot, src, kStageBytes / 2, full_at + b * 8);
        ptx::BulkLoadAt(wst_at + s * kStageSlot + kHalfSlot, src + kStageBytes / 2, kStageBytes / 2, full_at + b * 8);
        src += kStageBytes;
        if (++s == a.stages) s = 0;
        if (++b == kBarriers) b = 0;
      }
    }
  } else {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    bool ok = ptx::MbarWait(&ctl->xfull, 0, abort_flag, 3);

    // ---------------- main loop: a team of four warps takes every fourth K block ----------------
    // a warp has four of the block's k-tiles and four of its n-tiles;
    // lane (g, c): rows g and g + 8 of an n-tile, the 16 columns of its k-tile, four of them per MMA (the contraction index of
    // the fragments maps to columns alike in both operands); column g of the product = row g of x
    const int team = warp / kTeamWarps, w4 = warp % kTeamWarps;
    const int kq = w4 & 1, nt0 = (w4 >> 1) * 4;
    // stage index and barrier parity advance by counting: a division by the run-time ring depth per 128-wide
    // K block would cost as much as decoding a dozen weights
    int s = team, b = team;
    uint32_t phase = 0;
    while (s >= a.stages) s -= a.stages;
    auto next_block = [&] {
      __syncwarp();
      if (lane == 0) ptx::MbarArriveAt(full_at + (kBarriers + b) * 8);
      s += kTeams;
      while (s >= a.stages) s -= a.stages;
      b += kTeams;
      if (b >= kBarriers) { b -= kBarriers; phase ^= 1u; }
    };
    float* mine = loc + (team * 2 + kq) * TMAX * 128 + nt0 * 16;
    if constexpr (TMAX == 1) {
      // One row: nothing to contract, so a lane takes a row of an n-tile (lanes 16..31 that of the next n-tile) times the 64 columns
      // of half a K block.  Sums of 16 products in fp16 (the even or the odd columns of one half of four k-tiles), the rest in fp32.
      TrellisRow<KB> row;
      row.Init(lane & 15);
      float acc[2] = {0.f, 0.f};
      const unsigned char* xrow = xs + kq * 64;
      for (int it = team; it < my_blocks && ok; it += kTeams) {
        ok = ptx::MbarWaitAt(full_at + b * 8, phase, abort_flag, 2);
        if (!ok) break;
        const unsigned char* st = wst + s * kStageSlot + kq * kHalfSlot + (nt0 + (lane >> 4)) * (NW * 4);
        __half2 h[2][2];
#pragma unroll
        for (int i = 0; i < 2; ++i) h[i][0] = h[i][1] = __float2half2_rn(0.f);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4* xt = reinterpret_cast<const uint4*>(xrow + it * 256 + StoredTile(j) * 32);
          const uint4 xlo = xt[0], xhi = xt[1];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            uint32_t w[3];
            row.Load(reinterpret_cast<const uint32_t*>(st + j * kTileBytes + i * 2 * (NW * 4)), w[2], w[1], w[0]);
            RowDot<KB>(w, xlo, xhi, h[i]);
          }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
          acc[i] += (__low2float(h[i][0]) + __high2float(h[i][0])) + (__low2float(h[i][1]) + __high2float(h[i][1]));
        next_block();
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) mine[i * 32 + lane] = ok ? acc[i] : __int_as_float(0x7FC00000);      // (a copy that never landed shows as NaN)
    } else {
      const int g = lane >> 2, c = lane & 3;
      TrellisRow<KB> ra, rb;                                 // (the lane's k-tile is (c >> 1) * 4 + kq * 2 + (c & 1))
      ra.Init(g);
      rb.Init(g + 8);
      float acc[4][4];
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
      // columns past the last row of x repeat it: a column of the product depends on its own column of x only
      const unsigned char* xrow = xs + static_cast<size_t>(min(g, T - 1)) * xstride + (kq * 4 + c) * 32;
      for (int it = team; it < my_blocks && ok; it += kTeams) {
        const uint4 xlo = *reinterpret_cast<const uint4*>(xrow + it * 256), xhi = *reinterpret_cast<const uint4*>(xrow + it * 256 + 16);
        const uint32_t bx[8] = {xlo.x, xlo.y, xlo.z, xlo.w, xhi.x, xhi.y, xhi.z, xhi.w};
        ok = ptx::MbarWaitAt(full_at + b * 8, phase, abort_flag, 2);
        if (!ok) break;
        const unsigned char* st = wst + s * kStageSlot + (c >> 1) * kHalfSlot + (kq * 2 + (c & 1)) * kTileBytes + nt0 * (NW * 4);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const uint32_t* tw = reinterpret_cast<const uint32_t*>(st + n * (NW * 4));
          uint32_t wa[3], wb[3];
          ra.Load(tw, wa[2], wa[1], wa[0]);
          rb.Load(tw, wb[2], wb[1], wb[0]);
#define R4DXB_STEP(I)                                                                                                  \
    {                                                                                                                   \
      const uint32_t a0 = Code2<KB, 4 * I>(wa), a1 = Code2<KB, 4 * I>(wb);                                               \
      const uint32_t a2 = Code2<KB, 4 * I + 2>(wa), a3 = Code2<KB, 4 * I + 2>(wb);                                       \
      MmaF16(acc[n], a0, a1, a2, a3, bx[2 * I], bx[2 * I + 1]);                                                          \
    }
          R4DXB_STEP(0) R4DXB_STEP(1) R4DXB_STEP(2) R4DXB_STEP(3)
#undef R4DXB_STEP
        }
        next_block();
      }
      // the sums of a row (k-tile half, team) meet in shared memory
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = 2 * c + (i & 1);
          if (t < T) mine[t * 128 + n * 16 + g + 8 * (i >> 1)] = ok ? acc[n][i] : __int_as_float(0x7FC00000);      // (a copy that never landed shows as NaN)
        }
    }
    if (!ok && lane == 0 && a.status != nullptr) atomicCAS(a.status, 0, 700 + *abort_flag);
    ConsumerSync();
    if (ksplit > 1) {
      // hand this CTA's rows to cluster rank 0: distributed-shared-memory stores + one remote mbarrier arrival per
      // warp; only rank 0 waits, the other CTAs are done
      asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
      float* dst = cluster.map_shared_rank(part, 0) + krank * TMAX * 128;
      for (int i = threadIdx.x; i < T * 128; i += kConsumerWarps * 32) {
        float v = 0.f;
#pragma unroll
        for (int r = 0; r < kSums; ++r) v += loc[r * TMAX * 128 + i];
        dst[i] = v;
      }
      __syncwarp();
      if (lane == 0) {
        uint32_t remote_bar;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote_bar) : "r"(ptx::SmemAddr(red_bar)), "r"(0));
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
      }
    }
  }
  if (warp == kConsumerWarps) {
    // lane 0 may still be feeding the ring while the other lanes are already here: reconverge first,
    // and use the per-thread (non-.aligned) form of the barrier
    __syncwarp();
    if (ksplit > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  }

    // ---------------- epilogue (cluster rank 0): warp t finishes row t ----------------
  if (krank == 0 && warp < T) {
    bool landed = ksplit == 1;
    if (ksplit > 1) {
      // wait (bounded) until every consumer warp of every CTA of the cluster has delivered its partial rows
      for (int i = 0; i < ptx::kSpinLimit && !landed; ++i) {
        uint32_t okw;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(okw) : "r"(ptx::SmemAddr(red_bar)), "r"(0) : "memory");
        landed = okw != 0;
      }
    }
    const float inv_sqrt = 0.08838834764831845f;
    const int t = warp, n = nb * 128 + lane * 4;
    const float* from = ksplit > 1 ? part : loc;
    const int parts = ksplit > 1 ? ksplit : kSums;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    for (int r = 0; r < parts; ++r) {          // fixed order: the result does not depend on timing
      const float4 p = *reinterpret_cast<const float4*>(from + (r * TMAX + t) * 128 + lane * 4);
      v[0] += p.x; v[1] += p.y; v[2] += p.z; v[3] += p.w;
    }
    if (!landed) {
      v[0] = __int_as_float(0x7FC00000);                 // a hand-off that never completes shows as NaN in the whole block
      if (lane == 0 && a.status != nullptr) atomicCAS(a.status, 0, 390);
    }
    WarpFwht128(v);
    const uint2 sv = *reinterpret_cast<const uint2*>(svh + n);
    const __half2 s01 = *reinterpret_cast<const __half2*>(&sv.x), s23 = *reinterpret_cast<const __half2*>(&sv.y);
    float o[4] = {v[0] * inv_sqrt * __low2float(s01), v[1] * inv_sqrt * __high2float(s01),
                  v[2] * inv_sqrt * __low2float(s23), v[3] * inv_sqrt * __high2float(s23)};
    if (a.residual != nullptr) {
      const uint2 rv = *reinterpret_cast<const uint2*>(a.residual + static_cast<size_t>(t) * N + n);
      o[0] += BfLo(rv.x); o[1] += BfHi(rv.x); o[2] += BfLo(rv.y); o[3] += BfHi(rv.y);
    }
    uint2 ov;
    ov.x = PackBf16(o[0], o[1]);
    ov.y = PackBf16(o[2], o[3]);
    const size_t out_row = kGrouped ? __ldg(a.g_perm + start + t) : t;
    *reinterpret_cast<uint2*>(a.w[sidx].y + out_row * N + n) = ov;
  }
}

template <int KB, int TMAX>
size_t SmemBytes(int kslice, int stages, int ksplit) {
  return sizeof(Ctl) + static_cast<size_t>(kSums + (ksplit > 1 ? ksplit : 0)) * TMAX * 128 * 4 +
         static_cast<size_t>(TMAX) * XStride(kslice) + static_cast<size_t>(stages) * (2 * (4 * 8 * 8 * KB * 4 + 64));
}

size_t SmemOf(int kb, int T, int K, int ksplit) {
  const int blocks = (K / 128 + ksplit - 1) / ksplit, stages = blocks < kMaxStages ? blocks : kMaxStages;
  if (T == 1) return kb == 3 ? SmemBytes<3, 1>(blocks * 128, stages, ksplit) : (kb == 4 ? SmemBytes<4, 1>(blocks * 128, stages, ksplit) : SmemBytes<5, 1>(blocks * 128, stages, ksplit));
  if (kb == 3) return T <= 4 ? SmemBytes<3, 4>(blocks * 128, stages, ksplit) : SmemBytes<3, 8>(blocks * 128, stages, ksplit);
  if (kb == 4) return T <= 4 ? SmemBytes<4, 4>(blocks * 128, stages, ksplit) : SmemBytes<4, 8>(blocks * 128, stages, ksplit);
  return T <= 4 ? SmemBytes<5, 4>(blocks * 128, stages, ksplit) : SmemBytes<5, 8>(blocks * 128, stages, ksplit);
}

template <int KB, int TMAX>
int LaunchRows(RowsArgs a, int ksplit, cudaStream_t stream) {
  a.kblocks_per_cta = (a.K / 128 + ksplit - 1) / ksplit;       // the longest slice
  // ring depth: everything in flight for short slices, otherwise up to 6 stages (48-60 KiB)
  a.stages = a.kblocks_per_cta < kMaxStages ? a.kblocks_per_cta : kMaxStages;
  size_t smem = SmemBytes<KB, TMAX>(a.kblocks_per_cta * 128, a.stages, ksplit);
  // a grid that fits one CTA per SM asks for more than half of the shared memory: a CTA keeps an SM busy by itself, and two of
  // a cluster on one SM leave another idle (5120 x 17408 at two rows inside a captured step: 48 against 25 us)
  if (ksplit * a.w[a.count - 1].nb_end <= 148 && smem < 116 * 1024) smem = 116 * 1024;
  auto kern = TrellisRowsKernel<KB, TMAX>;
  const cudaError_t ea = AllowAllSharedMemory(kern);
  if (ea != cudaSuccess) return static_cast<int>(ea);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ksplit, a.w[a.count - 1].nb_end, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ksplit;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  // programmatic dependent launch: the CTAs fill their rings while the rows are still being written
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_use_pdl ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
  ++g_launch_count;
  return static_cast<int>(e);
}

template <int KB, int TMAX>
int LaunchGroupedRows(RowsArgs a, int max_tiles, cudaStream_t stream) {
  a.kblocks_per_cta = a.K / 128;
  a.stages = a.kblocks_per_cta < kMaxStages ? a.kblocks_per_cta : kMaxStages;
  // a short slice: a shallower ring where that lets two CTAs share an SM
  while (a.stages > 4 && SmemBytes<KB, TMAX>(a.K, a.stages, 1) > 113 * 1024) --a.stages;
  const size_t smem = SmemBytes<KB, TMAX>(a.K, a.stages, 1);
  if (smem > 227 * 1024) return R4DXB_TOO_LARGE;
  auto kern = TrellisRowsKernel<KB, TMAX, true>;
  const cudaError_t e = AllowAllSharedMemory(kern);
  if (e != cudaSuccess) return static_cast<int>(e);
  kern<<<dim3(1, a.w[0].N / 128, max_tiles), kThreads, smem, stream>>>(a);
  return FinishLaunch();
}

template <int PRO>
int LaunchInput(const RowsArgs& a, cudaStream_t stream) {
  return LaunchPdl(TrellisRowsInputKernel<PRO, false>, dim3(a.T, InputParts(a.K), a.count), dim3(kInWarps * 32), 0, stream, a,
                   const_cast<__half*>(a.xh));
}

template <int KB>
int LaunchKb(const RowsArgs& a, int ksplit, cudaStream_t stream) {
  if (a.T == 1) return LaunchRows<KB, 1>(a, ksplit, stream);
  if (a.T <= 4) return LaunchRows<KB, 4>(a, ksplit, stream);
  return LaunchRows<KB, 8>(a, ksplit, stream);
}

}  // namespace
}  // namespace r4dxb

using namespace r4dxb;

extern "C" {

/* One to three trellis products over the same 1..8 rows (see the header).  The split of K widens beyond `ksplit` where a
 * slice would not fit into shared memory. */
int r4dxb_trellis_gemv_rows(int count, const void* const* words, const void* const* suh, const void* const* svh, void* const* y,
                            const int* n, const void* x, const void* residual, const void* norm_w, float eps, int prologue, int T,
                            int K, int kb, int ksplit, void* ws, int* status, void* stream) {
  if (count < 1 || count > kMaxSiblings || T < 1 || T > 8 || K < 128 || K % 128 || ksplit < 1 || ksplit > 8 || K / 128 < ksplit ||
      prologue < 0 || prologue > 3 || (prologue == 1 && norm_w == nullptr) || (residual != nullptr && count > 1) || ws == nullptr ||
      (reinterpret_cast<uintptr_t>(ws) & 15) || kb < 3 || kb > 5)
    return R4DXB_BAD_ARG;
  RowsArgs a = {};
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.residual = static_cast<const __nv_bfloat16*>(residual);
  a.norm_w = static_cast<const __nv_bfloat16*>(norm_w);
  a.eps = eps;
  a.T = T;
  a.K = K;
  a.act = prologue == 3 ? 1 : 0;           // GeGLU: the SwiGLU prologue with a tanh-GELU gate
  a.count = count;
  a.status = status;
  int end = 0;
  for (int i = 0; i < count; ++i) {
    if (n[i] < 128 || n[i] % 128) return R4DXB_BAD_ARG;
    end += n[i] / 128;
    a.w[i].words = static_cast<const uint32_t*>(words[i]);
    a.w[i].suh = static_cast<const __half*>(suh[i]);
    a.w[i].svh = static_cast<const __half*>(svh[i]);
    a.w[i].y = static_cast<__nv_bfloat16*>(y[i]);
    a.w[i].N = n[i];
    a.w[i].nb_end = end;
  }
  while (SmemOf(kb, T, K, ksplit) > 227 * 1024) {
    if (ksplit == 8 || K / 128 <= ksplit) return R4DXB_TOO_LARGE;
    ++ksplit;
  }
  a.xh = static_cast<const __half*>(ws);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int rc = prologue == 0 ? LaunchInput<0>(a, s) : (prologue == 1 ? LaunchInput<1>(a, s) : LaunchInput<2>(a, s));
  if (rc) return rc;
  switch (kb) {
    case 3: return LaunchKb<3>(a, ksplit, s);
    case 4: return LaunchKb<4>(a, ksplit, s);
    default: return LaunchKb<5>(a, ksplit, s);
  }
}

/* Expert products with a few rows per expert: y[perm[p]] = svh[e] * H128(Q_e . H128(suh[e] * act(x[perm[p] / xdiv]))) for the
 * planned pairs p (see the header). */
int r4dxb_trellis_rows_grouped(const void* words, const void* suh, const void* svh, const void* x, void* y, const int* offsets,
                               const int* perm, const int* tiles, const int* ntiles, int max_tiles, int tile_rows, int xdiv, int mode, int P,
                               int E, int N, int K, int kb, void* xh, int* status, void* stream) {
  if (P < 1 || E < 1 || N < 128 || N % 128 || K < 128 || K % 128 || max_tiles < 1 || max_tiles > 65535 || tile_rows < 1 || tile_rows > 8 || xdiv < 1 || mode < 0 || mode > 2 ||
      xh == nullptr || (reinterpret_cast<uintptr_t>(xh) & 15))
    return R4DXB_BAD_ARG;
  RowsArgs a = {};
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.T = P;
  a.K = K;
  a.act = mode == 2 ? 1 : 0;
  a.count = 1;
  a.status = status;
  a.w[0].words = static_cast<const uint32_t*>(words);
  a.w[0].suh = static_cast<const __half*>(suh);
  a.w[0].svh = static_cast<const __half*>(svh);
  a.w[0].y = static_cast<__nv_bfloat16*>(y);
  a.w[0].N = N;
  a.w[0].nb_end = N / 128;
  a.g_offsets = offsets;
  a.g_perm = perm;
  a.g_tiles = tiles;
  a.g_ntiles = ntiles;
  a.g_experts = E;
  a.g_xdiv = xdiv;
  a.g_tile_rows = tile_rows;
  a.g_words = static_cast<long long>(N / 16) * (K / 16) * 8 * kb;
  a.xh = static_cast<const __half*>(xh);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  auto input_kernel = mode == 0 ? TrellisRowsInputKernel<0, true> : TrellisRowsInputKernel<2, true>;
  const int warps = min(kInWarps, K / 128), parts = (K / 128 + warps * kInBlocks - 1) / (warps * kInBlocks);
  input_kernel<<<dim3(P, parts), 32 * warps, 0, s>>>(a, static_cast<__half*>(xh));
  if (int rc = FinishLaunch()) return rc;
  if (kb == 3) return LaunchGroupedRows<3, 8>(a, max_tiles, s);
  if (kb == 4) return LaunchGroupedRows<4, 8>(a, max_tiles, s);
  if (kb == 5) return LaunchGroupedRows<5, 8>(a, max_tiles, s);
  return R4DXB_BAD_ARG;
}

}  // extern "C"
