// Weight-streaming w4a16 product for T <= 16 rows on mma.sync (the vocabulary head of decode steps, speculative windows and
// small batches).
//
//   y[t, n] = sum_groups scale[n, g] * sum_{k in g} (q[n, k] - zero[n, g]) * fp16(x[t, k])
//
// What bounds it: the packed weights are read once, 0.56 bytes per weight; at the measured copy rate that is 46 weights per
// clock and SM, so a kernel may spend fewer than three instructions per weight.  The CUDA-core kernel (w4a16_gemv.cu) spends
// one fp16 multiply-add chain per row of x: 218 / 1194 / 2414 us at 1 / 4 / 8 rows of a 248320 x 5120 head whose bytes take
// 109 us.  Here m16n8k16 takes 16 weight rows times 8 rows of x per instruction, so the cost hardly depends on T:
// (n - zero) is exact in fp16, products and sums are fp32, and the group's scale multiplies the group sum in fp32.
//
// Layout: a warp owns 16 weight rows at a time and keeps the next chunks' words of them (four groups each) in flight in registers,
// loaded straight from global memory: lane c of a quad takes words c * G / 32 .. of each group, so a quad's loads are whole
// sectors and all columns of an MMA share one group.  A ring slot is refilled group by group as its words are widened, through
// pointers that move along: with the words copied out first, and zeros put in place of absent rows of x, the kernel issued 49
// instructions per 512 weights and scheduler, 71 % of its slots, for 166 us at 1 row and 234 at 16; now 153 and 208.  What is left
// is the L1 (89 %): a load of 32-byte sectors from eight rows looks up eight lines.  Nothing synchronises across warps after the
// rows of x are staged.  (A ring of bulk copies into shared memory per warp, 16 copies of 256 bytes a stage, took 262 us at
// 248320 x 5120: the copy engine, not the math, set the pace.)  x is staged in the nibble order 0,4,1,5,2,6,3,7, so the 16 bytes of
// x behind one word of weights are one shared-memory load.
#include "common.cuh"

namespace r4dxb {
namespace {

constexpr int kWarps = 16;
constexpr int kW4Threads = kWarps * 32;
constexpr int kChunk = 4;                          // groups in flight per warp: one scale word per lane of a quad and row

__device__ __forceinline__ void MmaF16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// eight nibbles of a word -> four fp16 pairs (k, k + 4), each nibble minus the zero point, exact
__device__ __forceinline__ void Widen(uint32_t w, __half2 nz, __half2 nz16, uint32_t (&o)[4]) {
  const __half2 sixteenth = __float2half2_rn(0.0625f);
  const uint32_t v = w >> 8;
  uint32_t b[4] = {(w & 0x000F000Fu) | 0x64006400u, (w & 0x00F000F0u) | 0x64006400u,
                   (v & 0x000F000Fu) | 0x64006400u, (v & 0x00F000F0u) | 0x64006400u};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2 h = *reinterpret_cast<const __half2*>(&b[i]);
    // odd pairs hold 1024 + 16 n: a sixteenth of it is 64 + n
    const __half2 r = (i & 1) ? __hfma2(h, sixteenth, nz16) : __hadd2(h, nz);
    o[i] = *reinterpret_cast<const uint32_t*>(&r);
  }
}

template <int V>
__device__ __forceinline__ void LoadStream(const uint32_t* p, uint32_t (&o)[V]) {
  if constexpr (V == 1) {
    asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(o[0]) : "l"(p));
  } else if constexpr (V == 2) {
    asm volatile("ld.global.nc.L1::no_allocate.v2.b32 {%0, %1}, [%2];" : "=r"(o[0]), "=r"(o[1]) : "l"(p));
  } else {
    asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(o[0]), "=r"(o[1]), "=r"(o[2]), "=r"(o[3]) : "l"(p));
  }
}

// chunks in flight per warp: what 128 registers allow
template <int NT, int G, bool kRagged>
constexpr int Chunks() { return G == 32 ? 4 : (G == 64 ? (kRagged ? 2 : 3) : (NT == 1 ? 2 : 1)); }

// kRagged: zeros in place of the absent rows of the second eight, not loaded.  The rows of x then come out of the L1, which bounds the
// kernel, as often as there are rows: us of a 248320 x 5120 head, groups of 128, at 9 / 12 / 14 rows 187 / 189 / 204, without it 216 /
// 214 / 211 (groups of 32: 303 / 331 / 367 and 326 / 345 / 357; of 64, where it leaves two chunks in flight: 128256 x 4096 90 / 92 / 95
// and 94 / 94 / 95); the test costs more than it saves from there on.
template <int NT, int G, bool kRagged>
__global__ void __launch_bounds__(kW4Threads, 1)
W4MmaKernel(const uint32_t* __restrict__ wq, const uint32_t* __restrict__ wsz, const __nv_bfloat16* __restrict__ x,
            void* __restrict__ y, int T, int N, int K, int out_f32, int slices) {
  constexpr int V = G / 32;                        // words a lane takes of a row's group
  constexpr int D = Chunks<NT, G, kRagged>();               // chunks in flight per warp
  extern __shared__ __align__(128) unsigned char xs[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const int xstride = K * 2 + 16;                  // bytes: the eight rows of a fragment start 16 bytes apart modulo the banks
  const int tiles = N / 16, chunks = K / (kChunk * G), groups = K / G;
  // `slices` warps share a tile (each a run of its chunks); with more than one, every warp has one tile at most
  const int slice = warp % slices, c_lo = slice * chunks / slices, c_hi = (slice + 1) * chunks / slices;
  const int step = gridDim.x * (kWarps / slices);
  int tile = blockIdx.x + gridDim.x * (warp / slices), chunk = c_lo;
  uint32_t w0[D][kChunk][V], w1[D][kChunk][V], sz[D][2];
  // the next chunk to load; a ring slot is refilled group by group as its words are widened
  int load_tile = tile, load_chunk = c_lo;
  const size_t row8 = static_cast<size_t>(8) * (K / 8);
  const uint32_t* lp = wq + (static_cast<size_t>(tile) * 16 + g) * (K / 8) + c_lo * (kChunk * G / 8) + c * V;
  const uint32_t* ls = wsz + (static_cast<size_t>(tile) * 16 + g) * groups + c_lo * kChunk + c;
  auto load_group = [&](int i, uint32_t (&o0)[V], uint32_t (&o1)[V]) {
    if (load_tile >= tiles) return;
    LoadStream<V>(lp + i * (G / 8), o0);
    LoadStream<V>(lp + row8 + i * (G / 8), o1);
  };
  auto load_scales = [&](uint32_t (&o)[2]) {       // and on to the next chunk
    if (load_tile >= tiles) return;
    o[0] = __ldg(ls);
    o[1] = __ldg(ls + static_cast<size_t>(8) * groups);
    lp += kChunk * G / 8;
    ls += kChunk;
    if (++load_chunk == c_hi) {
      load_chunk = c_lo;
      load_tile += step;
      lp = wq + (static_cast<size_t>(load_tile) * 16 + g) * (K / 8) + c_lo * (kChunk * G / 8) + c * V;
      ls = wsz + (static_cast<size_t>(load_tile) * 16 + g) * groups + c_lo * kChunk + c;
    }
  };
#pragma unroll
  for (int d = 0; d < D; ++d) {
#pragma unroll
    for (int i = 0; i < kChunk; ++i) load_group(i, w0[d][i], w1[d][i]);
    load_scales(sz[d]);
  }

  // rows of x, fp16, in nibble order, while the first words are on their way
  for (int i = threadIdx.x; i < T * (K / 8); i += kW4Threads) {
    const int t = i / (K / 8), k8 = i % (K / 8);
    const uint4 v = *reinterpret_cast<const uint4*>(x + static_cast<size_t>(t) * K + k8 * 8);
    const __half2 p0 = __floats2half2_rn(BfLo(v.x), BfLo(v.z)), p1 = __floats2half2_rn(BfHi(v.x), BfHi(v.z));
    const __half2 p2 = __floats2half2_rn(BfLo(v.y), BfLo(v.w)), p3 = __floats2half2_rn(BfHi(v.y), BfHi(v.w));
    uint4 o;
    o.x = *reinterpret_cast<const uint32_t*>(&p0);
    o.y = *reinterpret_cast<const uint32_t*>(&p1);
    o.z = *reinterpret_cast<const uint32_t*>(&p2);
    o.w = *reinterpret_cast<const uint32_t*>(&p3);
    *reinterpret_cast<uint4*>(xs + static_cast<size_t>(t) * xstride + k8 * 16) = o;
  }
  __syncthreads();

  float tot[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int j = 0; j < 4; ++j) tot[nt][j] = 0.f;
  auto store = [&](int tl, const float (&v)[NT][4]) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = nt * 8 + 2 * c + (j & 1), n = tl * 16 + g + 8 * (j >> 1);
        if (t < T) {
          if (out_f32) static_cast<float*>(y)[static_cast<size_t>(t) * N + n] = v[nt][j];
          else static_cast<__nv_bfloat16*>(y)[static_cast<size_t>(t) * N + n] = __float2bfloat16(v[nt][j]);
        }
      }
  };
  // rows past T take the last one's x (kRagged: zeros): their columns of the product are never stored
  const unsigned char* xrow[NT];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) xrow[nt] = xs + static_cast<size_t>(min(nt * 8 + g, T - 1)) * xstride + c * (V * 16);
  const bool present = !kRagged || (NT - 1) * 8 + g < T;
  bool live = tile < tiles;
  while (live) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (!live) break;
      const unsigned char* xp[NT];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) xp[nt] = xrow[nt] + chunk * (kChunk * G * 2);
#pragma unroll
      for (int gi = 0; gi < kChunk; ++gi) {
        float acc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[nt][j] = 0.f;
        const uint32_t s0 = __shfl_sync(0xffffffffu, sz[d][0], (lane & ~3) | gi), s1 = __shfl_sync(0xffffffffu, sz[d][1], (lane & ~3) | gi);
        const uint32_t z0 = __byte_perm(s0, 0u, 0x3232), z1 = __byte_perm(s1, 0u, 0x3232);
        const __half2 k960 = __float2half2_rn(960.f);
        const __half2 nz0 = *reinterpret_cast<const __half2*>(&z0), nz1 = *reinterpret_cast<const __half2*>(&z1);
        const __half2 nzs0 = __hadd2(nz0, k960), nzs1 = __hadd2(nz1, k960);       // -(64 + zero)
#pragma unroll
        for (int v = 0; v < V; ++v) {
          uint32_t a[4], b[4];
          Widen(w0[d][gi][v], nz0, nzs0, a);
          Widen(w1[d][gi][v], nz1, nzs1, b);
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            uint4 xv = make_uint4(0u, 0u, 0u, 0u);
            if (!kRagged || nt < NT - 1 || present) xv = *reinterpret_cast<const uint4*>(xp[nt] + gi * (G * 2) + v * 16);
            MmaF16(acc[nt], a[0], b[0], a[1], b[1], xv.x, xv.y);
            MmaF16(acc[nt], a[2], b[2], a[3], b[3], xv.z, xv.w);
          }
        }
        load_group(gi, w0[d][gi], w1[d][gi]);
        const float f0 = __half2float(__ushort_as_half(static_cast<unsigned short>(s0 & 0xFFFFu)));
        const float f1 = __half2float(__ushort_as_half(static_cast<unsigned short>(s1 & 0xFFFFu)));
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          tot[nt][0] = fmaf(acc[nt][0], f0, tot[nt][0]);
          tot[nt][1] = fmaf(acc[nt][1], f0, tot[nt][1]);
          tot[nt][2] = fmaf(acc[nt][2], f1, tot[nt][2]);
          tot[nt][3] = fmaf(acc[nt][3], f1, tot[nt][3]);
        }
      }
      load_scales(sz[d]);
      if (++chunk == c_hi) {
        if (slices > 1) {
          live = false;
          break;
        }
        store(tile, tot);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int j = 0; j < 4; ++j) tot[nt][j] = 0.f;
        chunk = c_lo;
        tile += step;
        live = tile < tiles;
      }
    }
  }
  if (slices > 1) {
    // the slices' sums meet in shared memory and are added in slice order
    float* red = reinterpret_cast<float*>(xs + ((static_cast<size_t>(T) * xstride + 15) & ~static_cast<size_t>(15)));
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) red[(warp * NT * 4 + nt * 4 + j) * 32 + lane] = tot[nt][j];
    __syncthreads();
    if (slice == 0 && tile < tiles) {
      for (int s = 1; s < slices; ++s)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int j = 0; j < 4; ++j) tot[nt][j] += red[((warp + s) * NT * 4 + nt * 4 + j) * 32 + lane];
      store(tile, tot);
    }
  }
}

template <int NT, int G, bool kRagged = false>
int LaunchW4Mma(const void* wq, const void* wsz, const void* x, void* y, int T, int N, int K, int out_f32, cudaStream_t stream) {
  const size_t xbytes = (static_cast<size_t>(T) * (K * 2 + 16) + 15) & ~static_cast<size_t>(15), red = static_cast<size_t>(kWarps) * NT * 512;
  const int tiles = N / 16, grid = min(148, tiles);                 // one CTA per SM, a warp walks its 16-row tiles
  // a short matrix gives its tiles to several warps each, so that every SM still has its warps' loads in flight (a walk along K
  // by one warp is a chain of memory latencies: 8192 x 1024 takes 12 us unsplit)
  int slices = 1;
  while (slices * 2 <= K / (kChunk * G) && slices * 2 <= kWarps && static_cast<long long>(tiles) * slices * 2 <= static_cast<long long>(grid) * kWarps &&
         xbytes + red <= 227 * 1024)
    slices *= 2;
  const size_t smem = xbytes + (slices > 1 ? red : 0);
  auto kern = W4MmaKernel<NT, G, kRagged>;
  const cudaError_t e = AllowAllSharedMemory(kern);
  if (e != cudaSuccess) return static_cast<int>(e);
  kern<<<grid, kW4Threads, smem, stream>>>(static_cast<const uint32_t*>(wq), static_cast<const uint32_t*>(wsz),
                                           static_cast<const __nv_bfloat16*>(x), y, T, N, K, out_f32, slices);
  return FinishLaunch();
}

template <int G>
int LaunchW4MmaT(const void* wq, const void* wsz, const void* x, void* y, int T, int N, int K, int out_f32, cudaStream_t s) {
  if (T <= 8) return LaunchW4Mma<1, G>(wq, wsz, x, y, T, N, K, out_f32, s);
  if (T <= (G == 128 ? 14 : 12)) return LaunchW4Mma<2, G, true>(wq, wsz, x, y, T, N, K, out_f32, s);
  return LaunchW4Mma<2, G>(wq, wsz, x, y, T, N, K, out_f32, s);
}

}  // namespace

// Whether the kernel takes this call: whole 16-row tiles and whole chunks, aligned bases (vector loads of words and of x),
// and the staged rows of x fit into shared memory.
bool W4MmaCovers(const void* wq, const void* x, int T, int N, int K, int group) {
  return T >= 1 && T <= 16 && N % 16 == 0 && K % (kChunk * group) == 0 && (reinterpret_cast<uintptr_t>(wq) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(x) & 15) == 0 && static_cast<size_t>(T) * (K * 2 + 16) <= 227 * 1024;
}

int W4Mma(const void* wq, const void* wsz, const void* x, void* y, int T, int N, int K, int group, int out_f32, cudaStream_t s) {
  if (group == 32) return LaunchW4MmaT<32>(wq, wsz, x, y, T, N, K, out_f32, s);
  if (group == 64) return LaunchW4MmaT<64>(wq, wsz, x, y, T, N, K, out_f32, s);
  return LaunchW4MmaT<128>(wq, wsz, x, y, T, N, K, out_f32, s);
}

}  // namespace r4dxb
