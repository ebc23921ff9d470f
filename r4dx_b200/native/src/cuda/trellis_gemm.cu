// Plain linears (dense 16-bit, w4a16, w8a16) and the 8-bit trellis product on the 5th-generation tensor cores (tcgen05 + TMEM), the
// input transforms of the trellis products, and the tile list of the grouped ones.  The 16-bit trellis product is in trellis_product.cu.
//
// "Swap-AB": the weight block is the UMMA A operand (M = 128 weight rows = the span of one output Hadamard), the activations are the B
// operand (N = TN tokens), so the fp32 accumulator sits in TMEM as [lane = weight row][column = token].  Weights are widened or
// decoded exactly once per CTA and reused by all TN tokens of the tile.
//
// Warp roles (DW + 3 warps, DW = 8 or 16 decode warps):
//   warps 0..DW-1  decode: packed words or 4- / 8-bit weights -> A tile in the canonical
//              K-major 128-byte-swizzled UMMA layout; later the epilogue (TMEM -> registers ->
//              shared transpose -> (trellis: FWHT128 over the weight rows -> svh) -> residual -> rows).
//   warp DW    producer: TMA tile of the activations [TN x 64] (128B swizzle)
//   warp DW+1  MMA issuer: one elected thread issues 4 x tcgen05.mma (K = 16) per 64-wide K slab
//              and commits to the stage's "empty" barrier; it also owns the TMEM allocation.
//   warp DW+2  producer: packed words, or the tiles of a dense A
// A Hadamard mode with a dense A (MODE 0) takes A from a plain fp16 [N, K] matrix: the bisecting aid for the tensor-core plumbing.
// K may be split over the CTAs of a cluster (plain modes): a router or an a / b projection has so few outputs that its row blocks
// alone occupy a few SMs.
#include <cuda_fp8.h>

#include "sm100_ptx.cuh"
#include "trellis_decode.cuh"

namespace r4dxb {
namespace {

constexpr int kSlabK = 64;                 // K per pipeline stage = one 128-byte swizzle row of fp16
constexpr int kATileBytes = 128 * kSlabK * 2;   // 16 KiB

// Three rings, sized independently so that cheap data is prefetched deep and the big tile is not:
//   words (<= 5 KiB per slab, WST deep)  producer W -> decode warps
//   A     (16 KiB per slab, AST deep)    decode warps -> MMA
//   X     (TN x 128 B per slab, XST deep) producer X -> MMA
template <int KB, int TN, int F8 = 0>
struct GemmSmem {
  // a slab is one 128-byte swizzle row of K per operand row: 64 fp16 values (4 k-tiles of 16) or 128 e4m3 values (8 k-tiles)
  static constexpr int kKTiles = F8 ? 8 : 4;
  static constexpr int kWordsBytes = (KB == 0) ? 0 : kKTiles * 8 * 8 * KB * 4;   // k-tiles x 8 n-tiles x 8KB words
  static constexpr int kWordsSlot = ((kWordsBytes + 1023) / 1024) * 1024;
  static constexpr int kXTileBytes = TN * kSlabK * 2;
  static constexpr int WST = F8 ? 4 : 6;      // (8-bit slabs carry twice the words: four of them are as much K in flight as six 16-bit ones)
  static constexpr int AST = KB == 0 ? 4 : 3;
  static constexpr int XST = TN >= 512 ? 2 : (TN >= 256 ? 3 : 4);
  static constexpr int kABytes = AST * kATileBytes;
  static constexpr int kXBytes = XST * kXTileBytes;
  static constexpr int kEpiStride = 132;                                     // floats per staged token row
  static constexpr int kEpiBytes = 32 * kEpiStride * 4;                      // per group of four epilogue warps
  static constexpr bool kSplits = KB == 0 && TN <= 256;                      // whether the CTAs of a cluster may split K
  // the epilogue staging reuses the (by then drained) rings: it must hold one buffer per warp group, or all sums where K is split
  static constexpr int kRingsRaw = kABytes + kXBytes + WST * kWordsSlot;
  static constexpr int kSums = kSplits ? TN * kEpiStride * 4 : 0;
  static constexpr int kEpiAll = kSums > 4 * kEpiBytes ? kSums : 4 * kEpiBytes;
  static constexpr int kRing = kRingsRaw > kEpiAll ? kRingsRaw : kEpiAll;
  static constexpr int kBars = 2 * WST + 2 * AST + 2 * XST + 1;
  static constexpr int kTotal = kRing + 1024 /*alignment slack*/ + 512 /*barriers*/;
};

// Plain linear modes of the same kernel (MODE 1: dense 16-bit A matrix, MODE 2: w4a16 group-quantised A): y = x W^T
// (+ bias) (+ residual) with no Hadamard epilogue; activations and a dense A may be bf16 instead of fp16, the result
// may be written as fp32 (vocabulary logits).  These are the tensor-core paths of the heads and of the dense towers for
// more than 8 rows (reference: third_party/libr4d/r4d_gemm_w4a16_nt_m64.hip:173 is the WMMA counterpart for w4a16).
__device__ __forceinline__ float GeluTanh(float v) {
  return 0.5f * v * (1.0f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
}
__device__ __forceinline__ float GeluErf(float v) { return 0.5f * v * (1.0f + erff(v * 0.7071067811865476f)); }

struct PlainArgs {
  const uint32_t* wsz;         // MODE 2: [N][K / group] (fp16 scale | fp16 -(1024 + zero) << 16)
  const __nv_bfloat16* bias;   // [N] or null
  int group;                   // MODE 2: quantisation group (32, 64 or 128)
  int bf16;                    // the 16-bit operands are bf16 (MODE 1 only)
  int out_f32;                 // y is fp32 [T, N] instead of bf16
  int act;                     // after the bias: 0 none, 1 tanh-GELU, 2 erf-GELU
  // MODE 4, 8-bit operands: the decode warps emit e4m3 code values, the activations are e4m3 rows with one fp32 scale per
  // row (xh = scale * e4m3); K per slab is 128 and the products run at the 8-bit rate with half the activation bytes
  const float* x_scale;        // [T]
};

// The rows of a tile whose wait ran out: NaN instead of what they held before.
__device__ __noinline__ void FillNan(void* y, bool f32, int t0, int t_end, int N, int n0, int n_end) {
  const int n = n0 + (threadIdx.x & 31) * 4;
  if (n >= n_end) return;
  for (int t = t0 + (threadIdx.x >> 5); t < t_end; t += blockDim.x >> 5) {
    const float nan = __int_as_float(0x7FC00000);
    if (f32) *reinterpret_cast<float4*>(static_cast<float*>(y) + static_cast<size_t>(t) * N + n) = make_float4(nan, nan, nan, nan);
    else *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(y) + static_cast<size_t>(t) * N + n) = make_uint2(0x7FC07FC0u, 0x7FC07FC0u);
  }
}

template <int KB, int TN, int DW, int MODE = 0>
__global__ void __launch_bounds__((DW + 3) * 32, 1)
TrellisGemmKernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_a,
                  const void* __restrict__ wsrc,
                  const __half* __restrict__ svh, __nv_bfloat16* __restrict__ y,
                  const __nv_bfloat16* __restrict__ residual, int T, int N, int K, int* __restrict__ status, PlainArgs pl) {
  using S = GemmSmem<KB, TN, MODE == 4>;
  constexpr int kSlabElems = MODE == 4 ? 2 * kSlabK : kSlabK;      // K values per slab (one 128-byte row per operand row)
  constexpr int kKTiles = S::kKTiles;
  constexpr int WST = S::WST, AST = S::AST, XST = S::XST;
  extern __shared__ unsigned char smem_dyn[];
  // 1024-byte alignment: required by the swizzled UMMA / TMA tiles
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  unsigned char* a_ring = smem;
  unsigned char* x_ring = smem + S::kABytes;
  unsigned char* w_ring = smem + S::kABytes + S::kXBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kRing);
  uint64_t* wfull = bars;                   // [WST] producer W -> decode
  uint64_t* wempty = wfull + WST;           // [WST] decode -> producer W
  uint64_t* afull = wempty + WST;           // [AST] decode -> MMA
  uint64_t* aempty = afull + AST;           // [AST] MMA -> decode
  uint64_t* xfull = aempty + AST;           // [XST] producer X -> MMA
  uint64_t* xempty = xfull + XST;           // [XST] MMA -> producer X
  uint64_t* accum = xempty + XST;           // [1]   MMA -> epilogue
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = blockIdx.x;                 // 128-row weight block
  const int t0 = blockIdx.y * TN;            // first token of the tile
  // this CTA's K slabs: all, or an even share where the CTAs of a cluster split K (a ragged last slab only in the dense plain
  // mode: TMA zero-fills X)
  const int ksplit = gridDim.z, krank = blockIdx.z;
  const int slabs_all = (K + kSlabElems - 1) / kSlabElems;
  const int slab0 = krank * slabs_all / ksplit, slabs = (krank + 1) * slabs_all / ksplit - slab0;
  constexpr uint32_t kTmemCols = TN < 32 ? 32 : TN;
  constexpr int kHalves = TN > 256 ? TN / 256 : 1;     // one MMA covers at most 256 token columns
  constexpr int kMmaN = TN > 256 ? 256 : TN;

  if (threadIdx.x == 0) {
    for (int s = 0; s < WST; ++s) {
      ptx::MbarInit(&wfull[s], 1);
      ptx::MbarInit(&wempty[s], DW);
    }
    for (int s = 0; s < AST; ++s) {
      ptx::MbarInit(&afull[s], MODE == 1 ? 1 : DW);
      ptx::MbarInit(&aempty[s], 1);
    }
    for (int s = 0; s < XST; ++s) {
      ptx::MbarInit(&xfull[s], 1);
      ptx::MbarInit(&xempty[s], 1);
    }
    ptx::MbarInit(accum, 1);
    *abort_flag = 0;
    ptx::MbarFenceInit();
  }
  if (warp == DW + 1) {
    ptx::TmemAlloc(tmem_slot, kTmemCols);
    ptx::TmemRelinquish();
  }
  if (warp == DW && lane == 0) ptx::PrefetchTensorMap(&tmap_x);
  ptx::TcFenceBefore();
  __syncthreads();
  ptx::TcFenceAfter();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == DW) {
    // ---------------- producer X: TMA tiles of the transformed activations ----------------
    if (lane == 0) {
      for (int it = 0; it < slabs; ++it) {
        const int s = it % XST, round = it / XST;
        if (!ptx::MbarWait(&xempty[s], (round & 1) ^ 1, abort_flag, 1)) break;
        ptx::MbarArriveExpectTx(&xfull[s], S::kXTileBytes);
#pragma unroll
        for (int h = 0; h < kHalves; ++h)
          ptx::TmaLoad2D(x_ring + s * S::kXTileBytes + h * (kMmaN * kSlabK * 2), &tmap_x, &xfull[s], (slab0 + it) * kSlabElems, t0 + h * kMmaN);
      }
    }
  } else if (warp == DW + 2) {
    // ---------------- producer W: packed words, prefetched WST slabs deep ----------------
    if (MODE == 1 && lane == 0) {
      // dense plain mode: the weight tile comes by TMA as well (rows and columns past the matrix read as zero)
      ptx::PrefetchTensorMap(&tmap_a);
      for (int it = 0; it < slabs; ++it) {
        const int s = it % AST, round = it / AST;
        if (!ptx::MbarWait(&aempty[s], (round & 1) ^ 1, abort_flag, 5)) break;
        ptx::MbarArriveExpectTx(&afull[s], kATileBytes);
        ptx::TmaLoad2D(a_ring + s * kATileBytes, &tmap_a, &afull[s], (slab0 + it) * kSlabK, nb * 128);
      }
    }
    if (KB != 0 && lane == 0) {
      const size_t slab_words = kKTiles * 8 * 8 * (KB == 0 ? 1 : KB);
      const uint32_t* wbase = static_cast<const uint32_t*>(wsrc) + static_cast<size_t>(nb) * (K / 16) * 8 * 8 * (KB == 0 ? 1 : KB);
      for (int it = 0; it < slabs; ++it) {
        const int s = it % WST, round = it / WST;
        if (!ptx::MbarWait(&wempty[s], (round & 1) ^ 1, abort_flag, 7)) break;
        ptx::MbarArriveExpectTx(&wfull[s], S::kWordsBytes);
        ptx::BulkLoad(w_ring + s * S::kWordsSlot, wbase + static_cast<size_t>(it) * slab_words, S::kWordsBytes, &wfull[s]);
      }
    }
  } else if (warp == DW + 1) {
    // ---------------- MMA issuer ----------------
    // (one thread's instruction latencies add up: addresses and ring positions are counted up, not derived at each use)
    if (ptx::ElectOne()) {
      const uint32_t idesc = MODE == 4 ? ptx::UmmaInstrDescE4m3(128, kMmaN) : ptx::UmmaInstrDescF16(128, kMmaN, MODE == 1 && pl.bf16 != 0);
      const uint32_t xfull_at = ptx::SmemAddr(xfull), xempty_at = ptx::SmemAddr(xempty), afull_at = ptx::SmemAddr(afull), aempty_at = ptx::SmemAddr(aempty);
      const uint64_t da0 = ptx::UmmaDescSw128(ptx::SmemAddr(a_ring)), db0 = ptx::UmmaDescSw128(ptx::SmemAddr(x_ring));      // (the address is the low field, in units of 16 bytes)
      int sa = 0, sx = 0;
      uint32_t pa = 0, px = 0, accumulate = 0;
      bool ok = true;
      for (int it = 0; it < slabs; ++it) {
        ok = ptx::MbarWaitAt(xfull_at + sx * 8, px, abort_flag, 2) && ptx::MbarWaitAt(afull_at + sa * 8, pa, abort_flag, 3);
        if (!ok) break;
        ptx::TcFenceAfter();
        const uint64_t da = da0 + sa * (kATileBytes >> 4), db = db0 + sx * (S::kXTileBytes >> 4);
#pragma unroll
        for (int h = 0; h < kHalves; ++h) {
#pragma unroll
          for (int k = 0; k < kSlabK / 16; ++k) {
            const uint64_t dbk = db + h * (kMmaN * kSlabK * 2 >> 4) + k * 2;
            if constexpr (MODE == 4) ptx::UmmaF8(tmem_base + h * kMmaN, da + k * 2, dbk, idesc, k > 0 ? 1u : accumulate);
            else ptx::UmmaF16(tmem_base + h * kMmaN, da + k * 2, dbk, idesc, k > 0 ? 1u : accumulate);
          }
        }
        accumulate = 1;
        ptx::UmmaCommitAt(aempty_at + sa * 8);         // frees the A tile and the X tile once these MMAs have read them
        ptx::UmmaCommitAt(xempty_at + sx * 8);
        if (++sa == AST) { sa = 0; pa ^= 1u; }
        if (++sx == XST) { sx = 0; px ^= 1u; }
      }
      if (ok) ptx::UmmaCommit(accum);         // accumulator complete
    }
  } else {
    // ---------------- decode warps ----------------
    // a slab is 32 tiles (8 n-tiles x 4 k-tiles); warp w takes tiles w, w + DW, ...
    // lane slot: row (lane % 16) of the 16-row n-tile, K half (lane / 16) -> conflict-free 16-byte stores
    const int row_in_tile = lane & 15, khalf = lane >> 4;
    TrellisLane<(KB == 0 ? 4 : KB)> tl;
    tl.Init(2 * row_in_tile + khalf);
    bool ok = true;
    for (int it = 0; MODE != 1 && it < slabs && ok; ++it) {
      const int sa = it % AST, ra = it / AST, sw = it % WST, rw = it / WST;
      if (KB != 0) ok = ptx::MbarWait(&wfull[sw], rw & 1, abort_flag, 4);
      ok = ok && ptx::MbarWait(&aempty[sa], (ra & 1) ^ 1, abort_flag, 5);
      if (!ok) break;
      unsigned char* at = a_ring + sa * kATileBytes;
      if constexpr (MODE == 5) {
        // w8a16: a lane widens 32 consecutive k of one row (32 offset-binary bytes): a byte b becomes the fp16 1024 + b by
        // pairing it with 0x64; subtracting 1152 gives b - 128 exactly, the group scale is the only rounding
        for (int idx = warp; idx < 8; idx += DW) {
          const int r = idx * 16 + (lane >> 1), half = lane & 1;
          const size_t n = static_cast<size_t>(nb) * 128 + r;
          const int kbase = (slab0 + it) * kSlabK + half * 32;
          const uint4* src = reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(wsrc) + n * K + kbase);
          const uint4 q0 = __ldg(src), q1 = __ldg(src + 1);
          const __half sc = __ldg(reinterpret_cast<const __half*>(pl.wsz) + n * (K / pl.group) + kbase / pl.group);
          const __half2 sc2 = __half2half2(sc), off2 = __half2half2(__float2half(1152.0f));      // 1024 + 128
          const uint32_t qw[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t hb[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t w32 = qw[2 * c + (i >> 1)];
              const uint32_t b = __byte_perm(w32, 0x00000064u, (i & 1) ? 0x4342 : 0x4140);      // (1024 + b_lo, 1024 + b_hi)
              const __half2 v = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&b), off2), sc2);   // (b - 128) exactly, one rounding
              hb[i] = *reinterpret_cast<const uint32_t*>(&v);
            }
            const int chunk = half * 4 + c;
            *reinterpret_cast<uint4*>(at + (r >> 3) * 1024 + (r & 7) * 128 + ((chunk ^ (r & 7)) << 4)) = make_uint4(hb[0], hb[1], hb[2], hb[3]);
          }
        }
      } else if constexpr (MODE == 2) {
        // w4a16: a lane widens 32 consecutive k of one row (16 bytes of nibbles): nibble -> fp16 1024 + n by or-ing
        // 0x6400, the stored -(1024 + zero) makes n - zero exact, one fp16 multiply by the group scale
        for (int idx = warp; idx < 8; idx += DW) {
          const int r = idx * 16 + (lane >> 1), half = lane & 1;
          const size_t n = static_cast<size_t>(nb) * 128 + r;
          const int kbase = (slab0 + it) * kSlabK + half * 32;
          const uint4 q = __ldg(reinterpret_cast<const uint4*>(static_cast<const uint32_t*>(wsrc) + n * (K / 8) + kbase / 8));
          const uint32_t sz = __ldg(pl.wsz + n * (K / pl.group) + kbase / pl.group);
          const uint32_t scb = (sz & 0xFFFFu) | (sz << 16), nzb = (sz >> 16) | (sz & 0xFFFF0000u);
          const __half2 sc2 = *reinterpret_cast<const __half2*>(&scb), nz2 = *reinterpret_cast<const __half2*>(&nzb);
          const uint32_t qw[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int wi = 0; wi < 4; ++wi) {
            uint32_t hb[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t b = ((qw[wi] >> (4 * i)) & 0x000F000Fu) | 0x64006400u;       // (k + i, k + i + 4)
              const __half2 v = __hmul2(__hadd2(*reinterpret_cast<const __half2*>(&b), nz2), sc2);
              hb[i] = *reinterpret_cast<const uint32_t*>(&v);
            }
            uint4 packed;
            packed.x = __byte_perm(hb[0], hb[1], 0x5410); packed.y = __byte_perm(hb[2], hb[3], 0x5410);
            packed.z = __byte_perm(hb[0], hb[1], 0x7632); packed.w = __byte_perm(hb[2], hb[3], 0x7632);
            const int chunk = half * 4 + wi;
            *reinterpret_cast<uint4*>(at + (r >> 3) * 1024 + (r & 7) * 128 + ((chunk ^ (r & 7)) << 4)) = packed;
          }
        }
      } else if constexpr (MODE == 4) {
        // 8-bit operands: a slab is 8 k-tiles; a lane's 8 code values become 8 e4m3 bytes, the two K halves of a row share
        // one 16-byte swizzle chunk (chunk index = k-tile)
#pragma unroll 4
        for (int idx = warp; idx < 64; idx += DW) {
          const int j = idx & 7, kt = idx >> 3;
          const int r = j * 16 + row_in_tile;
          constexpr int NW = 8 * (KB == 0 ? 4 : KB);
          const uint32_t* tw = reinterpret_cast<const uint32_t*>(w_ring + sw * S::kWordsSlot) + (kt * 8 + j) * NW;
          uint32_t hi, lo;
          tl.Window(tw[tl.i0], tw[tl.i1], (KB == 4) ? 0u : tw[tl.i2], hi, lo);
          __half2 w[4];
          TrellisDecode8<(KB == 0 ? 4 : KB)>(hi, lo, w);
          uint2 packed;
          packed.x = static_cast<uint32_t>(__nv_cvt_halfraw2_to_fp8x2(*reinterpret_cast<__half2_raw*>(&w[0]), __NV_SATFINITE, __NV_E4M3)) |
                     (static_cast<uint32_t>(__nv_cvt_halfraw2_to_fp8x2(*reinterpret_cast<__half2_raw*>(&w[1]), __NV_SATFINITE, __NV_E4M3)) << 16);
          packed.y = static_cast<uint32_t>(__nv_cvt_halfraw2_to_fp8x2(*reinterpret_cast<__half2_raw*>(&w[2]), __NV_SATFINITE, __NV_E4M3)) |
                     (static_cast<uint32_t>(__nv_cvt_halfraw2_to_fp8x2(*reinterpret_cast<__half2_raw*>(&w[3]), __NV_SATFINITE, __NV_E4M3)) << 16);
          *reinterpret_cast<uint2*>(at + (r >> 3) * 1024 + (r & 7) * 128 + ((kt ^ (r & 7)) << 4) + khalf * 8) = packed;
        }
      } else {
#pragma unroll
      for (int idx = warp; idx < 32; idx += DW) {
        const int j = idx & 7;                             // n-tile inside the 128-row block
        const int kt = idx >> 3;
        const int r = j * 16 + row_in_tile;                // row inside the block
        uint4 packed;
        if (KB != 0) {
          constexpr int NW = 8 * (KB == 0 ? 4 : KB);
          const uint32_t* tw = reinterpret_cast<const uint32_t*>(w_ring + sw * S::kWordsSlot) + (kt * 8 + j) * NW;
          uint32_t hi, lo;
          tl.Window(tw[tl.i0], tw[tl.i1], (KB == 4) ? 0u : tw[tl.i2], hi, lo);
          __half2 w[4];
          TrellisDecode8<(KB == 0 ? 4 : KB)>(hi, lo, w);
          packed.x = *reinterpret_cast<uint32_t*>(&w[0]);
          packed.y = *reinterpret_cast<uint32_t*>(&w[1]);
          packed.z = *reinterpret_cast<uint32_t*>(&w[2]);
          packed.w = *reinterpret_cast<uint32_t*>(&w[3]);
        } else {
          const __half* dense = static_cast<const __half*>(wsrc);
          const int n = nb * 128 + r, k = (slab0 + it) * kSlabK + kt * 16 + khalf * 8;
          if (MODE == 0 || (n < N && k < K))
            packed = __ldg(reinterpret_cast<const uint4*>(dense + static_cast<size_t>(n) * K + k));
          else
            packed = make_uint4(0u, 0u, 0u, 0u);
        }
        const int chunk = kt * 2 + khalf;                  // 16-byte chunk inside the 128-byte row
        *reinterpret_cast<uint4*>(at + (r >> 3) * 1024 + (r & 7) * 128 + ((chunk ^ (r & 7)) << 4)) = packed;
      }
      }
      ptx::FenceProxyAsyncShared();          // generic-proxy stores -> visible to the tensor core (async proxy)
      __syncwarp();
      if (lane == 0) {
        ptx::MbarArrive(&afull[sa]);
        if (KB != 0) ptx::MbarArrive(&wempty[sw]);
      }
    }

    // ---------------- epilogue (the decode warps: warp w reads TMEM lanes 32 (w % 4) .. +31) ----------------
    // groups of four warps take 32-column chunks round-robin; each group stages its chunk through its
    // own transpose buffer, which lives in the rings (every slot has drained by now)
    if (ok) ok = ptx::MbarWait(accum, 0, abort_flag, 6);
    ptx::TcFenceAfter();
    const float inv_sqrt = 0.08838834764831845f;
    constexpr int kGroups = DW / 4;
    const int q = warp & 3, grp = warp >> 2;
    float* epi = reinterpret_cast<float*>(smem + grp * S::kEpiBytes);
    constexpr int CW = TN < 32 ? 16 : 32;   // columns per TMEM load
    auto load_columns = [&](int c0, uint32_t (&v)[CW]) {
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + c0;
      if constexpr (CW == 32) ptx::TmemLoad32x32(taddr, v);
      else ptx::TmemLoad32x16(taddr, v);
      ptx::TmemLoadWait();
    };
    // four outputs of token t out of their sums
    auto finish = [&](int t, float (&f)[4]) {
      const int n = nb * 128 + lane * 4;
      if (MODE == 1 && n >= N) return;
      float o0, o1, o2, o3;
      if constexpr (MODE == 0 || MODE == 4) {
        if constexpr (MODE == 4) {
          const float xs = __ldg(pl.x_scale + t);               // the row's activation scale
          f[0] *= xs; f[1] *= xs; f[2] *= xs; f[3] *= xs;
        }
        WarpFwht128(f);
        const uint2 sv = *reinterpret_cast<const uint2*>(svh + n);
        const __half2 s01 = *reinterpret_cast<const __half2*>(&sv.x), s23 = *reinterpret_cast<const __half2*>(&sv.y);
        o0 = f[0] * inv_sqrt * __low2float(s01); o1 = f[1] * inv_sqrt * __high2float(s01);
        o2 = f[2] * inv_sqrt * __low2float(s23); o3 = f[3] * inv_sqrt * __high2float(s23);
      } else {
        o0 = f[0]; o1 = f[1]; o2 = f[2]; o3 = f[3];
        if (pl.bias != nullptr) {
          const uint2 bv = *reinterpret_cast<const uint2*>(pl.bias + n);
          o0 += BfLo(bv.x); o1 += BfHi(bv.x); o2 += BfLo(bv.y); o3 += BfHi(bv.y);
        }
        if (pl.act == 1) {
          o0 = GeluTanh(o0); o1 = GeluTanh(o1); o2 = GeluTanh(o2); o3 = GeluTanh(o3);
        } else if (pl.act == 2) {
          o0 = GeluErf(o0); o1 = GeluErf(o1); o2 = GeluErf(o2); o3 = GeluErf(o3);
        }
      }
      if (residual != nullptr) {
        const uint2 rv = *reinterpret_cast<const uint2*>(residual + static_cast<size_t>(t) * N + n);
        o0 += BfLo(rv.x); o1 += BfHi(rv.x); o2 += BfLo(rv.y); o3 += BfHi(rv.y);
      }
      if ((MODE == 1 || MODE == 2 || MODE == 5) && pl.out_f32)
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(y) + static_cast<size_t>(t) * N + n) = make_float4(o0, o1, o2, o3);
      else
        *reinterpret_cast<uint2*>(y + static_cast<size_t>(t) * N + n) = make_uint2(PackBf16(o0, o1), PackBf16(o2, o3));
    };
    if (S::kSplits && ksplit > 1) {
      // K was split: the CTAs of the cluster lay their sums side by side in shared memory, and each finishes its share of the
      // tokens, adding up over distributed shared memory in rank order
      const int tile_end = min(TN, T - t0);
      float* sums = reinterpret_cast<float*>(smem);
      const uint32_t sums_at = ptx::SmemAddr(sums);
      for (int c0 = grp * CW; c0 < tile_end; c0 += kGroups * CW) {
        uint32_t v[CW];
        if (ok) load_columns(c0, v);
#pragma unroll
        for (int c = 0; c < CW; ++c)         // (a wait that ran out shows as NaN)
          sums[(c0 + c) * S::kEpiStride + q * 32 + lane] = ok ? __uint_as_float(v[c]) : __int_as_float(0x7FC00000);
      }
      ptx::ClusterSync();
      for (int c = warp * ksplit + krank; c < tile_end; c += DW * ksplit) {
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        for (int r = 0; r < ksplit; ++r) {
          const float4 p = ptx::LoadRemote4(sums_at + (c * S::kEpiStride + lane * 4) * 4, r);
          f[0] += p.x; f[1] += p.y; f[2] += p.z; f[3] += p.w;
        }
        finish(t0 + c, f);
      }
      ptx::ClusterSync();
    } else if (MODE == 1 && ok) {
      // (a loop of its own for dense weights: with a trip count that the compiler sees and no question in it, 4304 outputs of 4096 rows
      // take 34.6 us at 64 columns of K in tiles of 256 and 30.2 in tiles of 512, and 37.9 and 33.5 in the general form below)
      for (int c0 = grp * 32; c0 < TN; c0 += kGroups * 32) {
        {
          uint32_t v[CW];
          load_columns(c0, v);
#pragma unroll
          for (int c = 0; c < CW; ++c) epi[c * S::kEpiStride + q * 32 + lane] = __uint_as_float(v[c]);
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
#pragma unroll
        for (int i = 0; i < CW / 4; ++i) {
          const int c = q + 4 * i, t = t0 + c0 + c;
          if (t < T) {
            const float4 p = *reinterpret_cast<const float4*>(epi + c * S::kEpiStride + lane * 4);
            float f[4] = {p.x, p.y, p.z, p.w};
            finish(t, f);
          }
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
      }
    } else {
      for (int c0 = grp * 32; c0 < TN; c0 += kGroups * 32) {
        if (ok) {
          uint32_t v[CW];
          load_columns(c0, v);
#pragma unroll
          for (int c = 0; c < CW; ++c) epi[c * S::kEpiStride + q * 32 + lane] = __uint_as_float(v[c]);
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
        if (ok) {
          for (int c = q; c < CW; c += 4) {
            const int t = t0 + c0 + c;
            if (t < T) {
              const float4 p = *reinterpret_cast<const float4*>(epi + c * S::kEpiStride + lane * 4);
              float f[4] = {p.x, p.y, p.z, p.w};
              finish(t, f);
            }
          }
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
      }
    }
  }
  if (S::kSplits && warp >= DW && ksplit > 1) {
    __syncwarp();
    ptx::ClusterSync();                      // the other warps take part in the cluster's barriers
    ptx::ClusterSync();
  }

  // ---------------- teardown ----------------
  ptx::TcFenceBefore();
  __syncthreads();
  if (*abort_flag != 0) {
    FillNan(y, (MODE == 1 || MODE == 2 || MODE == 5) && pl.out_f32, t0, min(t0 + TN, T), N, nb * 128, min(nb * 128 + 128, N));
    // give copies that may still be in flight time to land before the shared memory goes away
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    if (threadIdx.x == 0) atomicExch(status, *abort_flag);
  }
  if (warp == DW + 1) ptx::TmemDealloc(tmem_base, kTmemCols);
}

// ---- input transform: Xh = fp16(H128(suh * x)) -------------------------------------------------------
// Sixteen lanes per 128-column block, eight columns each (16-byte loads and stores); producer variants fold the preceding
// elementwise op into the transform (reference: src/kernels/src/trellis_transform.hip:84-486 fuses the same producers).
//   mode 0: x = in[t, k]                      (in: [T, K])
//   mode 1: x = silu(in[t, k]) * in[t, K + k] (in: [T, 2K] fused gate|up rows); mode 2: the same with a tanh-GELU gate
// Bound by memory; what costs is latency and instructions, so a half-warp takes R rows of one block (their loads are in flight
// together, the signs are read once) and half of the Hadamard stages stay inside a lane: 115 -> 76 us on average over the
// products of 8192 rows.
__device__ __forceinline__ void Fwht128Half(float (&v)[8]) {
  const int lane = threadIdx.x & 15;
#pragma unroll
  for (int m = 1; m < 8; m <<= 1)
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (!(i & m)) {
        const float a = v[i], b = v[i | m];
        v[i] = a + b;
        v[i | m] = a - b;
      }
#pragma unroll
  for (int m = 1; m < 16; m <<= 1) {
    const float sign = (lane & m) ? -1.f : 1.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = fmaf(v[i], sign, __shfl_xor_sync(0xffffffffu, v[i], m));
  }
}

// 16 bytes at p, as two halves where a base is only 8-byte aligned
__device__ __forceinline__ uint4 Load16(const void* p, bool a16) {
  if (a16) return *static_cast<const uint4*>(p);
  const uint2 lo = static_cast<const uint2*>(p)[0], hi = static_cast<const uint2*>(p)[1];
  return make_uint4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ void Store16(void* p, const uint4& v, bool a16) {
  if (a16) {
    *static_cast<uint4*>(p) = v;
  } else {
    static_cast<uint2*>(p)[0] = make_uint2(v.x, v.y);
    static_cast<uint2*>(p)[1] = make_uint2(v.z, v.w);
  }
}

__device__ __forceinline__ void Unpack8(const uint4& p, float (&v)[8]) {
  v[0] = BfLo(p.x); v[1] = BfHi(p.x); v[2] = BfLo(p.y); v[3] = BfHi(p.y);
  v[4] = BfLo(p.z); v[5] = BfHi(p.z); v[6] = BfLo(p.w); v[7] = BfHi(p.w);
}

// eight columns: act, signs, Hadamard, fp16
__device__ __forceinline__ uint4 TransformBlock(const uint4& x, const uint4& u, const uint4& sv, int mode) {
  float v[8];
  Unpack8(x, v);
  if (mode != 0) {
    // the product is rounded to bf16 exactly like the unfused silu_mul kernel rounds it
    const int act = mode == 2 ? 1 : 0;
    float w[8];
    Unpack8(u, w);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const uint32_t p = PackBf16(GateAct(v[i], act) * w[i], GateAct(v[i + 1], act) * w[i + 1]);
      v[i] = BfLo(p);
      v[i + 1] = BfHi(p);
    }
  }
  const uint32_t s[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2 h = *reinterpret_cast<const __half2*>(&s[i]);
    v[2 * i] *= __low2float(h);
    v[2 * i + 1] *= __high2float(h);
  }
  Fwht128Half(v);
  const float inv_sqrt = 0.08838834764831845f;
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2 h = __floats2half2_rn(v[2 * i] * inv_sqrt, v[2 * i + 1] * inv_sqrt);
    o[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

template <int R>
__global__ void __launch_bounds__(256) TrellisInputKernel(const __nv_bfloat16* __restrict__ in, const __half* __restrict__ suh,
                                                          __half* __restrict__ out, int T, int K, int mode, bool a16) {
  const int blocks_per_row = K / 128;
  const long long items = static_cast<long long>((T + R - 1) / R) * blocks_per_row;
  long long item = (static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) >> 4;
  const bool live = item < items;                       // (both halves of a warp take part in its shuffles)
  if (!live) item = items - 1;
  const int t0 = static_cast<int>(item / blocks_per_row) * R;
  const int k = static_cast<int>(item % blocks_per_row) * 128 + (threadIdx.x & 15) * 8;
  const size_t stride = mode == 0 ? K : 2 * static_cast<size_t>(K);
  const uint4 sv = Load16(suh + k, a16);
  uint4 x[R], u[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int t = min(t0 + r, T - 1);
    x[r] = Load16(in + t * stride + k, a16);
    u[r] = mode == 0 ? make_uint4(0u, 0u, 0u, 0u) : Load16(in + t * stride + K + k, a16);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint4 o = TransformBlock(x[r], u[r], sv, mode);
    if (live && t0 + r < T) Store16(out + static_cast<size_t>(t0 + r) * K + k, o, a16);
  }
}

// ---- grouped experts: tile list and per-expert input transform ---------------------------------------
// One block.  Expert e with n_e planned rows gets ceil(n_e / tn) tiles; tiles are written in expert order.
__global__ void MoeTilesKernel(const int* __restrict__ offsets, int E, int tn, int* __restrict__ tiles,
                               int* __restrict__ ntiles, int max_tiles) {
  __shared__ int scan[1024];
  const int e = threadIdx.x;
  const int n = e < E ? offsets[e + 1] - offsets[e] : 0;
  const int c = (n + tn - 1) / tn;
  scan[e] = c;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const int v = e >= d ? scan[e - d] : 0;
    __syncthreads();
    scan[e] += v;
    __syncthreads();
  }
  const int base = scan[e] - c;
  if (e < E) {
    const int o = offsets[e];
    for (int j = 0; j < c && base + j < max_tiles; ++j) {
      tiles[2 * (base + j)] = e;
      tiles[2 * (base + j) + 1] = o + j * tn;
    }
  }
  if (e == 1023) *ntiles = min(scan[1023], max_tiles);
}

// xh[p] = fp16(H128(suh[e(p)] * act(in[perm[p] / xdiv]))) for every planned pair p (sorted by expert); a warp takes
// 2 * kPasses blocks of one pair (grid.y covers the rest of a row), so that the expert of the pair and its row are looked up once and
// the loads of all its blocks are in flight together; with a gate, half as many blocks, so that four CTAs share an SM either way
// (40960 pairs, 2048 columns / gated 512: 81 / 71 -> 72 / 43 us; the first is bound by 500 MB through the L2).
template <bool kGated, int kPasses>
__global__ void __launch_bounds__(256, 4) TrellisInputGroupedKernel(const __nv_bfloat16* __restrict__ in, const __half* __restrict__ suh,
                                                                 __half* __restrict__ out, const int* __restrict__ offsets,
                                                                 const int* __restrict__ perm, int E, int P, int K, int xdiv, int mode, bool a16) {
  const int p = blockIdx.x * 8 + (threadIdx.x >> 5), half = (threadIdx.x >> 4) & 1;
  if (p >= P || p >= __ldg(offsets + E)) return;
  const int lo = LastAtOrBelow(offsets, E, p);
  const int t = __ldg(perm + p) / xdiv;
  const __nv_bfloat16* row = in + static_cast<size_t>(t) * (kGated ? 2 * static_cast<size_t>(K) : K);
  const __half* sg = suh + static_cast<size_t>(lo) * K;
  const int b0 = blockIdx.y * 2 * kPasses + half, blocks = K / 128;
  uint4 x[kPasses], u[kGated ? kPasses : 1], sv[kPasses];
  u[0] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int i = 0; i < kPasses; ++i) {
    const int k = min(b0 + 2 * i, blocks - 1) * 128 + (threadIdx.x & 15) * 8;
    x[i] = Load16(row + k, a16);
    if constexpr (kGated) u[i] = Load16(row + K + k, a16);
    sv[i] = Load16(sg + k, a16);
  }
#pragma unroll
  for (int i = 0; i < kPasses; ++i) {
    if (blockIdx.y * 2 * kPasses + 2 * i >= blocks) break;          // (uniform over the warp)
    const uint4 o = TransformBlock(x[i], u[kGated ? i : 0], sv[i], kGated ? mode : 0);
    if (b0 + 2 * i < blocks) Store16(out + static_cast<size_t>(p) * K + (b0 + 2 * i) * 128 + (threadIdx.x & 15) * 8, o, a16);
  }
}

// ---- 8-bit activations: xq = e4m3(xh / scale), scale = rowmax |xh| / 448, one CTA per row ---------------------------
__global__ void __launch_bounds__(256) QuantizeRowsE4m3Kernel(const __half* __restrict__ xh, uint8_t* __restrict__ xq,
                                                              float* __restrict__ scale, int K) {
  __shared__ float red[32];
  const __half* row = xh + static_cast<size_t>(blockIdx.x) * K;
  float amax = 0.f;
  for (int k = threadIdx.x * 8; k < K; k += 256 * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(row + k);
    const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) amax = fmaxf(amax, fmaxf(fabsf(__low2float(h[i])), fabsf(__high2float(h[i]))));
  }
  amax = WarpMax(amax);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) amax = fmaxf(amax, red[w]);
  const float sc = amax > 0.f ? amax * (1.0f / 448.0f) : 1.0f;
  const float inv = 1.0f / sc;
  if (threadIdx.x == 0) scale[blockIdx.x] = sc;
  uint8_t* out = xq + static_cast<size_t>(blockIdx.x) * K;
  for (int k = threadIdx.x * 8; k < K; k += 256 * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(row + k);
    const __half2* h = reinterpret_cast<const __half2*>(&v);
    uint32_t o[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 a = __half22float2(h[2 * i]), b = __half22float2(h[2 * i + 1]);
      const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a.x * inv, a.y * inv), __NV_SATFINITE, __NV_E4M3);
      const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(b.x * inv, b.y * inv), __NV_SATFINITE, __NV_E4M3);
      o[i] = lo | (hi << 16);
    }
    *reinterpret_cast<uint2*>(out + k) = make_uint2(o[0], o[1]);
  }
}

bool Aligned16(const void* a, const void* b, const void* c) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}

int g_decode_warps = 16;

template <int KB, int TN, int DW, int MODE = 0>
int LaunchGemm(const void* wsrc, const void* svh, const void* xh, void* y, const void* residual, int T, int N, int K,
               int* status, cudaStream_t stream, const PlainArgs& pl, int ksplit = 1) {
  using S = GemmSmem<KB, TN, MODE == 4>;
  static_assert(S::kTotal <= 227 * 1024, "shared memory budget");
  static_assert(S::kBars * 8 + 16 <= 512, "barrier block");
  CUtensorMap tmap;
  const int rc = MODE == 4 ? MakeTensorMap2D8(&tmap, xh, static_cast<uint64_t>(T), static_cast<uint64_t>(K), TN > 256 ? 256 : TN, 128)
                           : MakeTensorMap2D16(&tmap, xh, static_cast<uint64_t>(T), static_cast<uint64_t>(K), TN > 256 ? 256 : TN, kSlabK,
                                               MODE == 1 && pl.bf16 != 0);
  if (rc) return rc;
  CUtensorMap tmap_a = tmap;
  if (MODE == 1) {
    const int ra = MakeTensorMap2D16(&tmap_a, wsrc, static_cast<uint64_t>(N), static_cast<uint64_t>(K), 128, kSlabK, pl.bf16 != 0);
    if (ra) return ra;
  }
  auto kern = TrellisGemmKernel<KB, TN, DW, MODE>;
  if (ksplit > 1 && !S::kSplits) return R4DXB_BAD_ARG;
  // (clusters that wait with tensor memory in hand: see kClusterShared; two CTAs of a split then meet on an SM, with 64 columns each)
  constexpr int kSplitSmem = S::kTotal > static_cast<int>(ptx::kClusterShared) ? S::kTotal : static_cast<int>(ptx::kClusterShared);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSmem);
  if (e != cudaSuccess) return static_cast<int>(e);
  static_assert(!S::kSplits || TN <= 64 || 2 * (S::kTotal + 1024) > 228 * 1024, "two CTAs' columns fit into tensor memory");
  const int smem = ksplit > 1 ? kSplitSmem : S::kTotal;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((N + 127) / 128, (T + TN - 1) / TN, ksplit);
  cfg.blockDim = dim3((DW + 3) * 32, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = ksplit;
  cfg.attrs = attr;
  cfg.numAttrs = ksplit > 1 ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, kern, tmap, tmap_a, wsrc, static_cast<const __half*>(svh), static_cast<__nv_bfloat16*>(y),
                         static_cast<const __nv_bfloat16*>(residual), T, N, K, status, pl);
  ++g_launch_count;
  return static_cast<int>(e);
}

template <int MODE>
int LaunchPlain(const void* w, const void* xh, void* y, const void* residual, int T, int N, int K, int tn, int ksplit, int* status,
                cudaStream_t s, const PlainArgs& pl) {
  switch (tn) {
    case 16: return LaunchGemm<0, 16, 8, MODE>(w, nullptr, xh, y, residual, T, N, K, status, s, pl, ksplit);
    case 32: return LaunchGemm<0, 32, 8, MODE>(w, nullptr, xh, y, residual, T, N, K, status, s, pl, ksplit);
    case 64: return LaunchGemm<0, 64, 8, MODE>(w, nullptr, xh, y, residual, T, N, K, status, s, pl, ksplit);
    case 128: return LaunchGemm<0, 128, 8, MODE>(w, nullptr, xh, y, residual, T, N, K, status, s, pl, ksplit);
    case 256: return LaunchGemm<0, 256, 8, MODE>(w, nullptr, xh, y, residual, T, N, K, status, s, pl, ksplit);
    case 512: return LaunchGemm<0, 512, 8, MODE>(w, nullptr, xh, y, residual, T, N, K, status, s, pl, ksplit);
    default: return R4DXB_BAD_ARG;
  }
}

template <int DW>
int LaunchDense(const void* w, const void* svh, const void* xh, void* y, const void* residual, int T, int N, int K, int tn,
                int* status, cudaStream_t s) {
  const PlainArgs pl = {};
  switch (tn) {
    case 16: return LaunchGemm<0, 16, DW>(w, svh, xh, y, residual, T, N, K, status, s, pl);
    case 32: return LaunchGemm<0, 32, DW>(w, svh, xh, y, residual, T, N, K, status, s, pl);
    case 64: return LaunchGemm<0, 64, DW>(w, svh, xh, y, residual, T, N, K, status, s, pl);
    case 128: return LaunchGemm<0, 128, DW>(w, svh, xh, y, residual, T, N, K, status, s, pl);
    case 256: return LaunchGemm<0, 256, DW>(w, svh, xh, y, residual, T, N, K, status, s, pl);
    case 512: return LaunchGemm<0, 512, DW>(w, svh, xh, y, residual, T, N, K, status, s, pl);
    default: return R4DXB_BAD_ARG;
  }
}

}  // namespace

int TrellisProduct(const void* w, const void* svh, const void* xh, void* y, const void* residual, int T, int N, int K, int kb, int tn,
                   int ksplit, int* status, cudaStream_t s);         // trellis_product.cu
extern int g_grouped_decode_warps;

}  // namespace r4dxb

using namespace r4dxb;

extern "C" {

int r4dxb_trellis_input(const void* in, const void* suh, void* out, int T, int K, int mode, void* stream) {
  if (T < 1 || K % 128 || mode < 0 || mode > 2) return R4DXB_BAD_ARG;
  // Four rows per half-warp once they still fill the machine that way; with a gate, twice the loads of a row are in flight as it
  // is, and it takes more.  us with one / four: plain 512 x 5120 4.7 / 4.9, 512 x 6144 5.1 / 4.9, 1024 x 17408 19.3 / 16.0; gated
  // 512 x 2048 4.3 / 6.1, 2048 x 5120 19.1 / 19.5, 1024 x 17408 33.5 / 32.2, 8192 x 5120 74 / 68.
  const int r = static_cast<long long>(T) * K >= (mode == 0 ? 3LL << 20 : 1LL << 24) ? 4 : 1;
  const long long items = static_cast<long long>((T + r - 1) / r) * (K / 128);
  (r == 4 ? TrellisInputKernel<4> : TrellisInputKernel<1>)<<<static_cast<unsigned>((items + 15) / 16), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(in), static_cast<const __half*>(suh), static_cast<__half*>(out), T, K, mode, Aligned16(in, suh, out));
  return FinishLaunch();
}

/* y[T, N] (bf16) from xh[T, K] (fp16, already input-transformed).  kb = 0: `w` is a dense fp16 [N, K]
 * matrix (svh still applies; pass ones and set hadamard-free weights accordingly); kb in {3,4,5}: packed
 * trellis words.  tn = token tile (16/32/64/128/256/512).  status: device int, set non-zero if a bounded wait
 * inside the kernel ran out. */
/* decode warps per CTA of the dense Hadamard mode (4, 8 or 16) and of the grouped trellis product (8 or 16, 4: by tile size): a
 * tuning and A/B-measurement switch */
void r4dxb_set_gemm_decode_warps(int n) {
  g_decode_warps = (n == 4 || n == 8) ? n : 16;
  g_grouped_decode_warps = n == 8 ? 8 : (n == 16 ? 16 : 0);
}

int r4dxb_trellis_gemm(const void* w, const void* svh, const void* xh, void* y, const void* residual, int T, int N, int K,
                       int kb, int tn, int* status, void* stream) {
  return r4dxb_trellis_gemm_split(w, svh, xh, y, residual, T, N, K, kb, tn, 1, status, stream);
}

/* The same with K split over the `ksplit` (1..8, trellis weights only) CTAs of a cluster, which add up in rank order; 192 and 384
 * are token tiles of a trellis product as well. */
int r4dxb_trellis_gemm_split(const void* w, const void* svh, const void* xh, void* y, const void* residual, int T, int N, int K,
                             int kb, int tn, int ksplit, int* status, void* stream) {
  if (T < 1 || N % 128 || K % 128 || ksplit < 1 || ksplit > 8 || K / 128 < ksplit) return R4DXB_BAD_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (kb != 0) return TrellisProduct(w, svh, xh, y, residual, T, N, K, kb, tn, ksplit, status, s);
  if (ksplit > 1) return R4DXB_BAD_ARG;
  switch (g_decode_warps) {
    case 4: return LaunchDense<4>(w, svh, xh, y, residual, T, N, K, tn, status, s);
    case 8: return LaunchDense<8>(w, svh, xh, y, residual, T, N, K, tn, status, s);
    default: return LaunchDense<16>(w, svh, xh, y, residual, T, N, K, tn, status, s);
  }
}

/* Plain linear on the tensor cores, any number of rows: y[T, N] = x[T, K] W^T (+ bias) (+ residual).
 * kind 0: W is a dense 16-bit [N, K] matrix (bf16 != 0: W and x are bf16, else fp16), N a multiple of 4 and K of 8;
 * kind 1: W is w4a16 (wq nibbles [N][K/8] + wsz [N][K/group]), x is fp16, N and K multiples of 128;
 * kind 2: W is w8a16 (offset-binary bytes [N][K] + fp16 scales [N][K/group] passed as wsz), x is fp16, N and K multiples of 128.
 * out_f32: y is fp32 instead of bf16.  act (low byte of out_f32 >> 8): 0 none, 1 tanh-GELU, 2 erf-GELU after the bias. */
int r4dxb_linear_tc(const void* w, const void* wsz, int kind, int group, int bf16, const void* x, void* y, int out_f32,
                    const void* bias, const void* residual, int T, int N, int K, int tn, int* status, void* stream) {
  return r4dxb_linear_tc_split(w, wsz, kind, group, bf16, x, y, out_f32, bias, residual, T, N, K, tn, 1, status, stream);
}

/* The same with K split over the `ksplit` (1..8, tiles up to 256) CTAs of a cluster, which add up in rank order. */
int r4dxb_linear_tc_split(const void* w, const void* wsz, int kind, int group, int bf16, const void* x, void* y, int out_f32,
                          const void* bias, const void* residual, int T, int N, int K, int tn, int ksplit, int* status, void* stream) {
  if (T < 1 || N < 4 || K < 8 || kind < 0 || kind > 2 || ksplit < 1 || ksplit > 8 || (K + 63) / 64 < ksplit) return R4DXB_BAD_ARG;
  if (kind == 0 && (N % 4 || K % 8)) return R4DXB_BAD_ARG;
  if (kind >= 1 && (N % 128 || K % 128 || wsz == nullptr || (group != 32 && group != 64 && group != 128) || bf16))
    return R4DXB_BAD_ARG;
  PlainArgs pl = {};
  pl.wsz = static_cast<const uint32_t*>(wsz);
  pl.bias = static_cast<const __nv_bfloat16*>(bias);
  pl.group = group;
  pl.bf16 = bf16;
  pl.out_f32 = out_f32 & 1;
  pl.act = (out_f32 >> 8) & 0xFF;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (kind == 2) return LaunchPlain<5>(w, x, y, residual, T, N, K, tn, ksplit, status, s, pl);
  return kind == 0 ? LaunchPlain<1>(w, x, y, residual, T, N, K, tn, ksplit, status, s, pl)
                   : LaunchPlain<2>(w, x, y, residual, T, N, K, tn, ksplit, status, s, pl);
}

/* 8-bit prefill product: rows of fp16 transformed activations -> e4m3 rows + one fp32 scale per row, then the trellis GEMM
 * with e4m3 code values and e4m3 activations on tcgen05.mma kind::f8f6f4 (fp32 accumulate, the row scale applied in the
 * epilogue).  K a multiple of 128; token tiles 128 / 256 / 512. */
int r4dxb_quantize_rows_e4m3(const void* xh, void* xq, float* scale, int T, int K, void* stream) {
  if (T < 1 || K < 8 || K % 8) return R4DXB_BAD_ARG;
  QuantizeRowsE4m3Kernel<<<T, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const __half*>(xh), static_cast<uint8_t*>(xq), scale, K);
  return FinishLaunch();
}

int r4dxb_trellis_gemm_f8(const void* w, const void* svh, const void* xq, const float* x_scale, void* y, const void* residual,
                          int T, int N, int K, int kb, int tn, int* status, void* stream) {
  if (T < 1 || N % 128 || K % 128 || x_scale == nullptr) return R4DXB_BAD_ARG;
  PlainArgs pl = {};
  pl.x_scale = x_scale;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
#define R4DXB_F8(KBV, TNV) if (kb == KBV && tn == TNV) return LaunchGemm<KBV, TNV, 16, 4>(w, svh, xq, y, residual, T, N, K, status, s, pl);
  R4DXB_F8(3, 128) R4DXB_F8(3, 256) R4DXB_F8(3, 512) R4DXB_F8(4, 128) R4DXB_F8(4, 256) R4DXB_F8(4, 512)
  R4DXB_F8(5, 128) R4DXB_F8(5, 256) R4DXB_F8(5, 512)
#undef R4DXB_F8
  return R4DXB_BAD_ARG;
}

/* Grouped experts on the tensor cores (prefill and wide batches of the mixture-of-experts block).
 * r4dxb_moe_tiles: tile list of the routing plan for token tiles of tn rows (E <= 1024 local experts).
 * r4dxb_trellis_input_grouped: xh[p] = fp16(H128(suh[e(p)] * act(in[perm[p] / xdiv]))) for the planned pairs in expert order.
 * (the product itself: trellis_product.cu). */
int r4dxb_moe_tiles(const int* offsets, int E, int tn, int* tiles, int* ntiles, int max_tiles, void* stream) {
  if (E < 1 || E > 1024 || tn < 1 || max_tiles < 1) return R4DXB_BAD_ARG;
  MoeTilesKernel<<<1, 1024, 0, static_cast<cudaStream_t>(stream)>>>(offsets, E, tn, tiles, ntiles, max_tiles);
  return FinishLaunch();
}

int r4dxb_trellis_input_grouped(const void* in, const void* suh, void* out, const int* offsets, const int* perm, int E, int P,
                                int K, int xdiv, int mode, void* stream) {
  if (P < 1 || K % 128 || xdiv < 1 || mode < 0 || mode > 2) return R4DXB_BAD_ARG;
  const int per_warp = mode == 0 ? 8 : 4;            // 128-column blocks
  const dim3 grid((P + 7) / 8, (K / 128 + per_warp - 1) / per_warp);
  (mode == 0 ? TrellisInputGroupedKernel<false, 4> : TrellisInputGroupedKernel<true, 2>)<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(in), static_cast<const __half*>(suh), static_cast<__half*>(out), offsets, perm, E, P, K, xdiv, mode,
      Aligned16(in, suh, out));
  return FinishLaunch();
}

}  // extern "C"
