// Causal GQA attention for a prefill chunk on the 5th-generation tensor cores: tcgen05.mma with the score
// tile S, the probability tile P and the output accumulator O all in tensor memory.
//
// A pair of CTAs (cta_group::2) = 2 x 128 query rows over the same keys: the same rows of two query heads of a kv head, or, where a kv
// head has an odd number of them, two row tiles of a head.  It walks the visible keys in tiles of 128:
//     S = Q K^T   tcgen05.mma kind::f16, A = Q (shared memory, resident), B = K tile, 64 keys from each CTA; M 256, N 128, K = D in
//                 steps of 16; fp32 S in tensor memory (two buffers)
//     softmax     eight warps, thread = query row = TMEM lane, two warps share a row (64 keys each): tcgen05.ld S, running maximum
//                 in the log2 domain, P = 2^(S - m) rounded to fp16 and written over the scores with tcgen05.st
//     O += P V    tcgen05.mma with the A operand read from TENSOR MEMORY (the P tile) and B = V^T tile, half of the dimensions from
//                 each CTA; M 256, N D, K = 128 keys in steps of 16; fp32 O in tensor memory
// The cache holds fp8 e4m3 rows in 16-token pages.  Eight conversion warps widen this CTA's half of each K tile to fp16 in the
// canonical K-major 128-byte-swizzled layout, and write its half of the V tile TRANSPOSED ([dimension][token]) so that V is a plain
// K-major B operand as well; the raw bytes of the next tile wait in registers.  Q is pre-multiplied by softmax scale x log2(e) x the
// K descale while it is converted, so scores need no further scaling.  The issuer keeps one S tile ahead of the softmax (S_j+1 is
// issued before P_j V_j), V's conversion runs up to two tiles ahead and K's three.
//
// Why pairs and 128 keys: one CTA with 64 keys a tile spent 92 clocks on the issue of each of its 20 products a tile (its scores
// read 6 KB of shared memory for 32 clocks of work) and all of its conversion warps' time on K and V that the neighbour converted
// too: 3440 clocks for 64 keys, where the products take 1024.  In pairs each product is twice as long, reads half of B and meets half
// of the conversions.  What bounds it now is the chain scores -> softmax -> products over two score buffers (the accumulator takes the
// other half of tensor memory): 3300 clocks from announced probabilities to the scores after next, about as many in the softmax,
// whose 128 x 128 exponentials alone take 1024.  Output gates wait in K's buffers and output rows leave as one copy per row
// half: read and written directly by the lanes that own the rows, they took 25k clocks a CTA.
// 8192 rows, 24 heads over 4, D = 256: 1623 -> 953 us (865 TFLOP/s); 1024 rows after 29000 1499 -> 916; 333 rows 50 -> 29;
// 32 heads over 8, D = 128, 8192 rows 1304 -> 913.
//
// Rescaling of O when a row maximum grows is lazy: P is computed against the maximum in use, and only when some
// row's true maximum has moved more than 8 (a factor 256, harmless in fp16 / fp32) does the warp wait for the
// outstanding P V products, rescale its 32 rows of O in tensor memory and adopt the new maximum.
// Every wait is bounded; a wait that runs out sets the status word and the CTA unwinds (frees tensor memory).
//
// The reference's counterpart is a query-tiled WMMA kernel (reference:
// third_party/libr4d/r4d_attn_prefill_h256_gqa6.hip:112); nothing is shared with it.
#include "common.cuh"
#include "sm100_ptx.cuh"

namespace r4dxb {
namespace {

constexpr int kQRows = 128;               // of a CTA
constexpr int kKvTile = 128;              // keys of a step; each CTA of the pair prepares half of K's rows and half of V's columns
constexpr int kHalfTile = kKvTile / 2;
constexpr int kPage = 16;
constexpr int kSoftmaxWarps = 8;          // warp w: rows 32 (w % 4) .., keys 64 (w / 4) ..
constexpr int kMmaWarp = kSoftmaxWarps;
constexpr int kConvWarps = 8;
constexpr int kConvThreads = kConvWarps * 32;
constexpr int kThreads = (kSoftmaxWarps + 1 + kConvWarps) * 32;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kSCol = 256;           // S buffers: 256 + 128 b; P overwrites the scores that its own warp has read
constexpr float kRescaleStep = 8.f;

struct TcArgs {
  const __nv_bfloat16* q;      // [T, Hq, D] normed + roped
  const __nv_bfloat16* qg;     // [T, Hq, 2D] (gate in the upper half), may be null when !gated
  const uint8_t* cache;        // [page][Hkv][2][16][D] fp8
  const int* block_table;
  const float* k_descale;
  const float* v_descale;
  __nv_bfloat16* out;          // [T, Hq, D]
  int T, Hq, Hkv, pos0, gated, window;
  int by_head;                 // a pair is two query heads of a kv head over the same rows, else two row tiles of a head
  int* status;
};

struct Control {
  uint64_t q_full, k_full[2], v_full[2], p_full[2];      // those of the first CTA count both
  uint64_t s_full[2], pv_done[2], o_final;               // commits, to both CTAs
  uint64_t gates;                                        // the output gates lie in K's buffers (this CTA only)
  uint32_t tmem_base;
  int abort_flag;
  float row[2][2][kQRows];                               // [tile parity][half of the keys]: what the two warps of a row exchange
};

__device__ __forceinline__ uint32_t Fp8x2Bits(uint32_t v16) {
  __half2_raw r = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(v16 & 0xFFFFu), __NV_E4M3);
  return *reinterpret_cast<uint32_t*>(&r);
}
// four e4m3 bytes of one word -> two half2 words (bytes 0-1, bytes 2-3), without shifts or masks
__device__ __forceinline__ void Fp8x4ToHalf(uint32_t w, uint32_t& lo, uint32_t& hi) {
  asm("{ .reg .b16 l, h; mov.b32 {l, h}, %2; cvt.rn.f16x2.e4m3x2 %0, l; cvt.rn.f16x2.e4m3x2 %1, h; }"
      : "=r"(lo), "=r"(hi) : "r"(w));
}
__device__ __forceinline__ float Exp2Approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// offset of 16-byte chunk c of row r inside a [rows][128 B] tile in the K-major 128-byte-swizzled UMMA layout
__device__ __forceinline__ int Sw128(int r, int c) { return (r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4); }

// offset of gates 8 c .. 8 c + 7 of row r: rows of 2 D bytes whose 16-byte chunks are permuted, so that 32 lanes reading the same
// columns of 32 rows reach all banks
template <int D>
__device__ __forceinline__ int GateChunk(int r, int c) { return r * 2 * D + ((c ^ (r & 7)) << 4); }

template <int D>
__global__ void __launch_bounds__(kThreads, 1) AttnPrefillTcKernel(TcArgs a) {
  constexpr int NS = D / 64;                          // 64-dimension slabs (one 128-byte swizzle row of fp16 each)
  constexpr int kQBytes = NS * kQRows * 128;
  constexpr int kKBytes = NS * kHalfTile * 128;       // [slab][64 keys][128 B]
  constexpr int kVSlab = D / 2 * 128;                 // V^T: [64-key slab][half of the dimensions][128 B]
  constexpr int kVBytes = 2 * kVSlab;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  unsigned char* Qs = smem;
  unsigned char* Ks = Qs + kQBytes;                   // [2][kKBytes]
  unsigned char* Vs = Ks + 2 * kKBytes;               // [2][kVBytes]
  Control* ctl = reinterpret_cast<Control*>(Vs + 2 * kVBytes);
  volatile int* abort_flag = &ctl->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x & 1;
  const int hq = a.by_head ? blockIdx.x : blockIdx.x >> 1;
  const int hkv = hq / (a.Hq / a.Hkv);
  const int step = static_cast<int>(gridDim.y - 1 - blockIdx.y);            // the rows with the most keys start first, in all heads
  const int first_row = step * (a.by_head ? kQRows : 2 * kQRows);           // of the pair
  const int q0 = a.by_head ? first_row : first_row + rank * kQRows;
  const int rows = max(0, min(kQRows, a.T - q0));
  const int kv_limit = a.pos0 + a.T;                  // tokens present in the cache
  const int kv_end = a.pos0 + min(a.T, first_row + (a.by_head ? kQRows : 2 * kQRows));      // first key no row of the pair may see
  const int kv_first = a.window > 0 ? max(0, a.pos0 + first_row - a.window + 1) : 0;
  const int tile0 = kv_first / kKvTile;
  const int ntiles = (kv_end + kKvTile - 1) / kKvTile - tile0;              // at least 1

  if (threadIdx.x == 0) {
    ptx::MbarInit(&ctl->q_full, 2 * kConvWarps);
    for (int b = 0; b < 2; ++b) {
      ptx::MbarInit(&ctl->k_full[b], 2 * kConvWarps);
      ptx::MbarInit(&ctl->v_full[b], 2 * kConvWarps);
      ptx::MbarInit(&ctl->p_full[b], 2 * kSoftmaxWarps);
      ptx::MbarInit(&ctl->s_full[b], 1);
      ptx::MbarInit(&ctl->pv_done[b], 1);
    }
    ptx::MbarInit(&ctl->o_final, 1);
    ptx::MbarInit(&ctl->gates, kConvWarps);
    ctl->abort_flag = 0;
    ptx::MbarFenceInit();
  }
  if (warp == kMmaWarp) {
    ptx::TmemAllocPair(&ctl->tmem_base, kTmemCols);
    ptx::TmemRelinquishPair();
  }
  ptx::TcFenceBefore();
  __syncthreads();
  ptx::ClusterSync();                                 // the partner's barriers exist before anything arrives at them
  ptx::TcFenceAfter();
  const uint32_t tbase = ctl->tmem_base;

  if (warp > kMmaWarp) {
    // ---------------- conversion warps: Q once, then this CTA's half of K and of V^T of every key tile ----------------
    const int tid = threadIdx.x - (kMmaWarp + 1) * 32, cw = warp - (kMmaWarp + 1);
    const uint32_t q_full = ptx::MapToRank(ptx::SmemAddr(&ctl->q_full), 0);
    const uint32_t k_full = ptx::MapToRank(ptx::SmemAddr(&ctl->k_full[0]), 0), v_full = ptx::MapToRank(ptx::SmemAddr(&ctl->v_full[0]), 0);
    // K: a thread owns 16 dimensions of KI consecutive keys (16 lanes read a row); which of two neighbouring keys it stores first
    // depends on its slab, so that the 32 stores of an instruction spread over all banks.
    constexpr int CH = D / 16, KI = D / 64;
    const int ch = tid % CH, key0 = tid / CH * KI, flip = (ch >> 2) & 1;
    // V: a thread owns VD dimensions of 8 consecutive keys and turns them into VD rows of 16 bytes; the byte it starts with depends on
    // its lane, and the two halves of a warp are 4 key groups apart, for the same reason.
    constexpr int VD = D / 32, VW = VD / 4;
    const int dq = lane & 15, tg = (cw & 3) + ((lane >> 4) << 2) + ((cw >> 2) << 3);
    const size_t page_bytes = static_cast<size_t>(a.Hkv) * 2 * kPage * D;
    const uint8_t* cache_k = a.cache + static_cast<size_t>(hkv) * 2 * kPage * D + ch * 16;
    const uint8_t* cache_v = a.cache + static_cast<size_t>(hkv) * 2 * kPage * D + kPage * D + rank * (D / 2) + dq * VD;
    uint4 kraw[KI];
    uint32_t vraw[8][VW];
    // raw bytes of a tile into registers, zeros past the last token
    auto load_k = [&](int j) {
      const int kp0 = (tile0 + j) * kKvTile + rank * kHalfTile + key0;
#pragma unroll
      for (int i = 0; i < KI; ++i) kraw[i] = make_uint4(0u, 0u, 0u, 0u);
      if (j < ntiles && kp0 < kv_limit) {
        const uint8_t* base = cache_k + a.block_table[kp0 >> 4] * page_bytes;
#pragma unroll
        for (int i = 0; i < KI; ++i) {
          const int kp = kp0 + (i ^ flip);
          if (kp < kv_limit) kraw[i] = __ldg(reinterpret_cast<const uint4*>(base + (kp & 15) * D));
        }
      }
    };
    auto load_v = [&](int j) {
      const int kp0 = (tile0 + j) * kKvTile + tg * 8;
#pragma unroll
      for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int w = 0; w < VW; ++w) vraw[t][w] = 0u;
      if (j < ntiles && kp0 < kv_limit) {
        const uint8_t* base = cache_v + a.block_table[kp0 >> 4] * page_bytes + (kp0 & 15) * D;
#pragma unroll
        for (int t = 0; t < 8; ++t)
          if (kp0 + t < kv_limit) {
            if constexpr (VW == 2) {
              const uint2 v = __ldg(reinterpret_cast<const uint2*>(base + t * D));
              vraw[t][0] = v.x;
              vraw[t][1] = v.y;
            } else {
              vraw[t][0] = __ldg(reinterpret_cast<const uint32_t*>(base + t * D));
            }
          }
      }
    };
    unsigned char* k_dst = Ks + (ch >> 2) * (kHalfTile * 128);
    auto store_k = [&](int j) {
      unsigned char* at = k_dst + (j & 1) * kKBytes;
#pragma unroll
      for (int i = 0; i < KI; ++i) {
        const int off = Sw128(key0 + (i ^ flip), (ch & 3) * 2);              // the second chunk sits at off ^ 16
        uint4 lo, hi;
        Fp8x4ToHalf(kraw[i].x, lo.x, lo.y);
        Fp8x4ToHalf(kraw[i].y, lo.z, lo.w);
        Fp8x4ToHalf(kraw[i].z, hi.x, hi.y);
        Fp8x4ToHalf(kraw[i].w, hi.z, hi.w);
        *reinterpret_cast<uint4*>(at + off) = lo;
        *reinterpret_cast<uint4*>(at + (off ^ 16)) = hi;
      }
      ptx::FenceProxyAsyncShared();
      __syncwarp();
      if (lane == 0) ptx::MbarArriveRemote(k_full + (j & 1) * 8);
    };
    unsigned char* v_dst = Vs + (tg >> 3) * kVSlab;
    auto store_v = [&](int j) {
      unsigned char* at = v_dst + (j & 1) * kVBytes;
#pragma unroll
      for (int s = 0; s < VD; ++s) {
        const int byte = (s + dq) & 3;
        const uint32_t sel = byte * 0x11 + 0x40;                             // that byte of both words
        uint32_t h[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) h[t] = Fp8x2Bits(__byte_perm(vraw[2 * t][s >> 2], vraw[2 * t + 1][s >> 2], sel));
        *reinterpret_cast<uint4*>(at + Sw128(dq * VD + (s & 4) + byte, tg & 7)) = make_uint4(h[0], h[1], h[2], h[3]);
      }
      ptx::FenceProxyAsyncShared();
      __syncwarp();
      if (lane == 0) ptx::MbarArriveRemote(v_full + (j & 1) * 8);
    };

    load_k(0);
    {
      const float scale = rsqrtf(static_cast<float>(D)) * 1.4426950408889634f * a.k_descale[hkv];
#pragma unroll 4
      for (int i = tid; i < kQRows * (D / 8); i += kConvThreads) {
        const int r = i / (D / 8), c = i % (D / 8);
        uint4 o = make_uint4(0u, 0u, 0u, 0u);
        if (r < rows) {
          const uint4 v = *reinterpret_cast<const uint4*>(a.q + (static_cast<size_t>(q0 + r) * a.Hq + hq) * D + c * 8);
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
          uint32_t h[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const __half2 p = __floats2half2_rn(BfLo(w[j]) * scale, BfHi(w[j]) * scale);
            h[j] = *reinterpret_cast<const uint32_t*>(&p);
          }
          o = make_uint4(h[0], h[1], h[2], h[3]);
        }
        *reinterpret_cast<uint4*>(Qs + (c >> 3) * (kQRows * 128) + Sw128(r, c & 7)) = o;
      }
      ptx::FenceProxyAsyncShared();
      __syncwarp();
      if (lane == 0) ptx::MbarArriveRemote(q_full);
    }
    // K runs two tiles ahead of V: K's buffer is free when the scores are done, one product earlier than V's
    store_k(0);
    load_k(1);
    load_v(0);
    if (ntiles > 1) {
      store_k(1);
      load_k(2);
    }
    bool ok = true;
    for (int j = 0; j < ntiles && ok; ++j) {
      const uint32_t ph = static_cast<uint32_t>(j >> 1) & 1u;
      if (j >= 2) ok = ptx::WarpMbarWait(&ctl->pv_done[j & 1], ph ^ 1u, abort_flag, 12);    // P_(j-2) V_(j-2) has consumed the buffer
      if (!ok) break;
      store_v(j);
      load_v(j + 1);
      if (j + 2 < ntiles) {
        ok = ptx::WarpMbarWait(&ctl->s_full[j & 1], ph, abort_flag, 11);                    // S_j has consumed the buffer
        if (!ok) break;
        store_k(j + 2);
        load_k(j + 3);
      }
    }
    // the output gates of this CTA's rows, into K's buffers once the last scores have read them
    if (ok && a.gated) ok = ptx::WarpMbarWait(&ctl->s_full[(ntiles - 1) & 1], static_cast<uint32_t>((ntiles - 1) >> 1) & 1u, abort_flag, 13);
    if (ok && a.gated) {
#pragma unroll 4
      for (int i = tid; i < rows * (D / 8); i += kConvThreads) {
        const int r = i / (D / 8), c = i % (D / 8);
        const __nv_bfloat16* src = a.qg + ((static_cast<size_t>(q0 + r) * a.Hq + hq) * 2 + 1) * D + c * 8;
        uint4 g;
        if (reinterpret_cast<uintptr_t>(a.qg) % 16 == 0) {
          g = *reinterpret_cast<const uint4*>(src);
        } else {                              // (their base may lie at any 4 bytes)
          const uint32_t* w = reinterpret_cast<const uint32_t*>(src);
          g = make_uint4(w[0], w[1], w[2], w[3]);
        }
        *reinterpret_cast<uint4*>(Ks + GateChunk<D>(r, c)) = g;
      }
      __syncwarp();
      if (lane == 0) ptx::MbarArrive(&ctl->gates);
    }
  } else if (warp == kMmaWarp) {
    // ---------------- MMA issuer (one thread of the first CTA) ----------------
    if (rank == 0 && lane == 0) {
      constexpr uint32_t idesc_s = ptx::UmmaInstrDescF16(2 * kQRows, kKvTile, false);
      constexpr uint32_t idesc_o = ptx::UmmaInstrDescF16(2 * kQRows, D, false);
      const uint64_t qd = ptx::UmmaDescSw128(ptx::SmemAddr(Qs)), kd = ptx::UmmaDescSw128(ptx::SmemAddr(Ks));
      const uint64_t vd = ptx::UmmaDescSw128(ptx::SmemAddr(Vs));       // (the address is the low field, in units of 16 bytes)
      const uint32_t s_full = ptx::SmemAddr(&ctl->s_full[0]), pv_done = ptx::SmemAddr(&ctl->pv_done[0]);
      auto scores = [&](int b) {
        ptx::TcFenceAfter();
        const uint64_t kb = kd + b * (kKBytes / 16);
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            ptx::UmmaF16Pair(tbase + kSCol + b * kKvTile, qd + (s * (kQRows * 128) + k * 32) / 16, kb + (s * (kHalfTile * 128) + k * 32) / 16,
                             idesc_s, (s > 0 || k > 0) ? 1u : 0u);
        ptx::UmmaCommitPairAt(s_full + b * 8, 3);
      };
      bool ok = ptx::MbarWait(&ctl->q_full, 0, abort_flag, 1) && ptx::MbarWait(&ctl->k_full[0], 0, abort_flag, 2);
      if (ok) scores(0);
      for (int j = 0; j < ntiles && ok; ++j) {
        const int b = j & 1;
        const uint32_t ph = static_cast<uint32_t>(j >> 1) & 1u;
        if (j + 1 < ntiles) {
          // Its buffer's scores were read before P_(j-1) was announced, and P_(j-1) V_(j-1), which reads the probabilities that took
          // their place, was issued before it: products run in the order of their issue.
          ok = ptx::MbarWait(&ctl->k_full[b ^ 1], static_cast<uint32_t>((j + 1) >> 1) & 1u, abort_flag, 2);
          if (!ok) break;
          scores(b ^ 1);
        }
        ok = ptx::MbarWait(&ctl->v_full[b], ph, abort_flag, 4) && ptx::MbarWait(&ctl->p_full[b], ph, abort_flag, 3);
        if (!ok) break;
        ptx::TcFenceAfter();
        const uint64_t vb = vd + b * (kVBytes / 16);
        const uint32_t pt = tbase + kSCol + b * kKvTile;
#pragma unroll
        for (int k = 0; k < kKvTile / 16; ++k)
          ptx::UmmaF16PairFromTmem(tbase, pt + (k >> 2) * 64 + (k & 3) * 8, vb + ((k >> 2) * kVSlab + (k & 3) * 32) / 16, idesc_o,
                                   (j > 0 || k > 0) ? 1u : 0u);
        ptx::UmmaCommitPairAt(pv_done + b * 8, 3);
      }
      if (ok) ptx::UmmaCommitPairAt(ptx::SmemAddr(&ctl->o_final), 3);
    }
    __syncwarp();
  } else {
    // ---------------- softmax warps: thread = query row = TMEM lane, two warps share a row ----------------
    const int half = warp >> 2, r = (warp & 3) * 32 + lane;
    const int qp = a.pos0 + q0 + r;                               // position of this row's query
    const uint32_t t_lane = tbase + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const uint32_t p_full = ptx::MapToRank(ptx::SmemAddr(&ctl->p_full[0]), 0);
    float m_used = -INFINITY, l_run = 0.f;
    bool ok = true;
    // (both warps of a row reach every one of these, also after a wait that ran out)
    auto exchange = [&](int parity, float mine) -> float {
      ctl->row[parity][half][r] = mine;
      asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory");
      return ctl->row[parity][half ^ 1][r];
    };
    for (int j = 0; j < ntiles; ++j) {
      const int b = j & 1;
      const uint32_t ph = static_cast<uint32_t>(j >> 1) & 1u;
      const uint32_t scol = t_lane + kSCol + b * kKvTile + half * 64;
      if (ok) ok = ptx::WarpMbarWait(&ctl->s_full[b], ph, abort_flag, 6);
      uint32_t s0[32], s1[32];
      float mx = -INFINITY;
      if (ok) {
        ptx::TcFenceAfter();
        ptx::TmemLoad32x32(scol, s0);
        ptx::TmemLoad32x32(scol + 32, s1);
        ptx::TmemLoadWait();
        const int kv0 = (tile0 + j) * kKvTile, k_lo = kv0 + half * 64;
        // tiles that reach past the row's own position (or start before its window) need the mask
        if ((kv0 + kKvTile - 1 > a.pos0 + q0) || (a.window > 0 && kv0 < a.pos0 + q0 + kQRows - a.window)) {
          const int lo = a.window > 0 ? qp - a.window : -1;         // visible: lo < kp <= qp
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            const int k0 = k_lo + c, k1 = k_lo + 32 + c;
            if (!(k0 <= qp && k0 > lo)) s0[c] = 0xff800000u;        // -inf
            if (!(k1 <= qp && k1 > lo)) s1[c] = 0xff800000u;
          }
        }
        float mx2 = -INFINITY;
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          mx = fmaxf(mx, fmaxf(__uint_as_float(s0[c]), __uint_as_float(s1[c])));
          mx2 = fmaxf(mx2, fmaxf(__uint_as_float(s0[c + 1]), __uint_as_float(s1[c + 1])));
        }
        mx = fmaxf(mx, mx2);
      }
      mx = fmaxf(mx, exchange(b, mx));
      if (!ok) continue;
      // lazy rescale: adopt a new maximum only when some row of the warp has drifted by more than the step
      if (__any_sync(0xffffffffu, mx > m_used + kRescaleStep)) {
        const float m_new = fmaxf(m_used, mx);
        if (j > 0) {
          // every P V issued so far must have landed before O is touched; each warp takes half of the columns
          ok = ptx::WarpMbarWait(&ctl->pv_done[b ^ 1], static_cast<uint32_t>((j - 1) >> 1) & 1u, abort_flag, 7);
          if (!ok) continue;
          ptx::TcFenceAfter();
          const float f = (m_used == -INFINITY) ? 0.f : exp2f(m_used - m_new);
          l_run *= f;
#pragma unroll 1
          for (int c0 = half * (D / 2); c0 < (half + 1) * (D / 2); c0 += 16) {
            uint32_t o[16];
            ptx::TmemLoad32x16(t_lane + c0, o);
            ptx::TmemLoadWait();
#pragma unroll
            for (int c = 0; c < 16; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * f);
            ptx::TmemStore32x16(t_lane + c0, o);
          }
          ptx::TmemStoreWait();
        }
        m_used = m_new;
      }
      // P = 2^(S - m), fp16 pairs (k, k+1) per column
      float sum = 0.f, sum2 = 0.f;
      const float mref = (m_used == -INFINITY) ? 0.f : m_used;
      auto probabilities = [&](const uint32_t (&sv)[32], uint32_t col) {
        uint32_t p[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const float e0 = Exp2Approx(__uint_as_float(sv[2 * c]) - mref), e1 = Exp2Approx(__uint_as_float(sv[2 * c + 1]) - mref);
          sum += e0;
          sum2 += e1;
          const __half2 h = __floats2half2_rn(e0, e1);
          p[c] = *reinterpret_cast<const uint32_t*>(&h);
        }
        ptx::TmemStore32x16(col, p);
      };
      probabilities(s0, scol);
      probabilities(s1, scol + 16);
      l_run += sum + sum2;
      ptx::TmemStoreWait();
      ptx::TcFenceBefore();
      __syncwarp();
      if (lane == 0) ptx::MbarArriveRemote(p_full + b * 8);
    }
    // ---------------- epilogue: O / l, output gate, bf16 rows; each warp half of the columns ----------------
    const float l = l_run + exchange(ntiles & 1, l_run);
    if (ok && a.gated) ok = ptx::WarpMbarWait(&ctl->gates, 0, abort_flag, 10);
    if (ok) ok = ptx::WarpMbarWait(&ctl->o_final, 0, abort_flag, 9);
    if (ok) {
      ptx::TcFenceAfter();
      const float inv = (l > 0.f ? 1.f / l : 0.f) * a.v_descale[hkv];
      // a lane's half row, staged where Q (first half) or V (second) was and sent off as one copy
      constexpr int kHalfRow = D / 2 * 2, kStageRow = kHalfRow + 16;
      static_assert(kQRows * kStageRow <= kQBytes && kQRows * kStageRow <= 2 * kVBytes, "the output tile fits");
      unsigned char* stage = (half == 0 ? Qs : Vs) + r * kStageRow;
#pragma unroll 1
      for (int c0 = 0; c0 < D / 2; c0 += 32) {
        uint32_t o[32];
        ptx::TmemLoad32x32(t_lane + half * (D / 2) + c0, o);
        ptx::TmemLoadWait();
        if (r < rows) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            float x[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) x[c] = __uint_as_float(o[8 * v + c]) * inv;
            if (a.gated) {
              const uint4 g = *reinterpret_cast<const uint4*>(Ks + GateChunk<D>(r, (half * (D / 2) + c0) / 8 + v));
              const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                x[2 * c] *= Sigmoid(BfLo(gw[c]));
                x[2 * c + 1] *= Sigmoid(BfHi(gw[c]));
              }
            }
            *reinterpret_cast<uint4*>(stage + (c0 + 8 * v) * 2) =
                make_uint4(PackBf16(x[0], x[1]), PackBf16(x[2], x[3]), PackBf16(x[4], x[5]), PackBf16(x[6], x[7]));
          }
        }
      }
      ptx::FenceProxyAsyncShared();
      if (r < rows) {
        ptx::BulkStore(a.out + (static_cast<size_t>(q0 + r) * a.Hq + hq) * D + half * (D / 2), ptx::SmemAddr(stage), kHalfRow);
        ptx::BulkStoreCommit();
        ptx::BulkStoreWait();
      }
    }
  }

  // ---------------- teardown ----------------
  ptx::TcFenceBefore();
  __syncthreads();
  if (*abort_flag != 0) {
    if (threadIdx.x == 0 && a.status != nullptr) atomicCAS(a.status, 0, 600 + *abort_flag);
  }
  ptx::ClusterSync();                                 // neither CTA leaves or frees tensor memory while the other still uses it
  if (warp == kMmaWarp) {
    ptx::TcFenceAfter();
    ptx::TmemDeallocPair(tbase, kTmemCols);
  }
}

template <int D>
int LaunchTc(const TcArgs& a, cudaStream_t s) {
  constexpr int NS = D / 64;
  // kClusterAlone: so much of an SM's shared memory that no other CTA shares the SM whose cluster may wait with tensor memory in its
  // hands (sm100_ptx.cuh).  More would cost L1: 8192 rows of 32 heads of 128 columns take 808 us with 131 KB, 821 with 156, 878 with 227.
  constexpr size_t kSmem = NS * kQRows * 128 + 2 * NS * kHalfTile * 128 + 2 * D * 128 + sizeof(Control) + 1024;
  constexpr size_t smem = kSmem > ptx::kClusterAlone ? kSmem : ptx::kClusterAlone;
  auto kern = AttnPrefillTcKernel<D>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return static_cast<int>(e);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = a.by_head ? dim3(a.Hq, (a.T + kQRows - 1) / kQRows) : dim3(2 * a.Hq, (a.T + 2 * kQRows - 1) / (2 * kQRows));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, kern, a);
  if (e != cudaSuccess) return static_cast<int>(e);
  return FinishLaunch();
}

}  // namespace
}  // namespace r4dxb

using namespace r4dxb;

/* Same contract as r4dxb_attn_prefill (flags bit 0: sigmoid output gate, bits 1..: sliding-window length), for head
   dimensions 128 and 256.  status: device word that receives 600 + role code if a bounded wait ran out. */
extern "C" int r4dxb_attn_prefill_tc(const void* q, const void* qg, const void* cache, const int* block_table,
                                     const float* k_descale, const float* v_descale, void* out, int T, int Hq, int Hkv, int D,
                                     int pos0, int flags, int* status, void* stream) {
  if (T < 1 || Hq % Hkv || (D != 256 && D != 128)) return R4DXB_BAD_ARG;
  TcArgs a;
  a.q = static_cast<const __nv_bfloat16*>(q);
  a.qg = static_cast<const __nv_bfloat16*>(qg);
  a.cache = static_cast<const uint8_t*>(cache);
  a.block_table = block_table;
  a.k_descale = k_descale;
  a.v_descale = v_descale;
  a.out = static_cast<__nv_bfloat16*>(out);
  a.T = T; a.Hq = Hq; a.Hkv = Hkv; a.pos0 = pos0; a.gated = flags & 1; a.window = flags >> 1;
  a.by_head = Hq / Hkv % 2 == 0;
  a.status = status;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return D == 256 ? LaunchTc<256>(a, s) : LaunchTc<128>(a, s);
}
