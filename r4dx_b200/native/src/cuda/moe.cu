// Mixture-of-experts routing and combine kernels (softmax top-k router, device-side plan, weighted
// combine with the shared expert).  The grouped expert GEMV itself lives in trellis_gemv.cu.
//
// Semantics (reference: src/model/qwen4exp/include/r4dx/model/qwen4exp/moe_kernels.h:18-56):
//   * router: fp32 softmax over the expert logits, top-k (k <= 16, experts <= 1024), optional
//     renormalisation, weights rounded through bf16; ties go to the larger logit, then the lower id;
//   * plan: (token, slot) pairs sorted by expert id (stable), with per-expert offsets, built on
//     the device so that no routing decision is read back by the host;
//   * combine: out[t] = residual[t] + sum_j w[t,j] * y[pair(t,j)] in ascending expert id (a fixed
//     order: no atomics) + sigmoid(shared_gate[t]) * shared[t], one bf16 rounding.
#include <type_traits>

#include "common.cuh"

namespace r4dxb {
namespace {

constexpr int kMaxK = 16;

// one warp per token row
//
// mode 1 is the sigmoid router of the short-conv MoE family (reference:
// src/kernels/include/r4dx/kernels/lfm2_kernels.h:38-50): s[e] = sigmoid(logit[e]); the SELECTION ranks s[e] + bias[e]
// (ties to the lower id), the weights are the unbiased s of the selected experts, divided by (their sum + 1e-6) when
// renorm is set, then multiplied by `scale`.
// One warp routes one row.  The row's selection values live in registers (E <= 1024: 32 per lane) and a lane remembers its taken
// entries in a bit mask.  Every lane keeps its best entry; a round is two reductions over the lanes, and only the lane that loses
// its entry looks for the next one.  (With a search of all lanes and ten shuffles a round, 4096 rows of 512 experts took 30 us, now 18.)
// A NaN (what a wait that ran out leaves in a row) ranks last, so that every row gets k experts that exist; the softmax weights of
// such a row are NaN, and so is the sigmoid weight of a NaN that is picked.
__device__ __forceinline__ void RouteRow(const float* __restrict__ row, const float* __restrict__ bias, int E, int k, int renorm,
                                         int mode, float scale, int lane, int* __restrict__ ids, float* __restrict__ weights) {
  float v[32];
  float mx = -INFINITY, z = 0.f;
#pragma unroll
  for (int s = 0; s < 32; ++s) v[s] = -INFINITY;
#pragma unroll
  for (int s0 = 0; s0 < 32; s0 += 8) {       // (in groups of 256 experts: what the row does not have costs nothing)
    if (32 * s0 >= E) break;
#pragma unroll
    for (int s = s0; s < s0 + 8; ++s) {
      const int e = lane + 32 * s;
      if (e < E) v[s] = mode == 0 ? row[e] : 1.0f / (1.0f + expf(-row[e])) + (bias ? bias[e] : 0.f);
      mx = fmaxf(mx, v[s]);
    }
  }
  if (mode == 0) {
    mx = WarpMax(mx);
#pragma unroll
    for (int s0 = 0; s0 < 32; s0 += 8) {
      if (32 * s0 >= E) break;
#pragma unroll
      for (int s = s0; s < s0 + 8; ++s) z += (lane + 32 * s < E) ? __expf(v[s] - mx) : 0.f;
    }
    z = WarpSum(z);
  }
  float wsum = 0.f;
  uint32_t taken = 0;              // bit s: this lane's entry lane + 32 s is already picked
  float my_p = 0.f;                // lane j keeps the j-th pick (k <= 16 <= 32)
  int my_i = 0;
  float lv;                        // this lane's best entry that is not taken: value and expert (the larger value, then the lower id)
  int li;
  auto look = [&] {
    lv = -INFINITY;
    li = 0x7fffffff;
#pragma unroll
    for (int s0 = 0; s0 < 32; s0 += 8) {
      if (32 * s0 >= E) break;
#pragma unroll
      for (int s = s0; s < s0 + 8; ++s) {
        const int e = lane + 32 * s;
        if (e < E && !((taken >> s) & 1u) && (v[s] > lv || (v[s] == lv && e < li))) { lv = v[s]; li = e; }
      }
    }
  };
  look();
  for (int j = 0; j < k; ++j) {
    // (values as integers of the same order; adding zero makes the two zeros one)
    const uint32_t bits = __float_as_uint(lv + 0.0f), key = bits ^ ((bits >> 31) ? 0xFFFFFFFFu : 0x80000000u);
    const uint32_t top = __reduce_max_sync(0xffffffffu, key);
    int bi = static_cast<int>(__reduce_min_sync(0xffffffffu, key == top ? static_cast<uint32_t>(li) : 0x7fffffffu));
    float bv = __shfl_sync(0xffffffffu, lv, bi & 31);
    if (bi >= E) {                 // (no lane has a number left: the lowest id that is not taken)
      int next = 0x7fffffff;
      for (int s = 31; s >= 0; --s)
        if (lane + 32 * s < E && !((taken >> s) & 1u)) next = lane + 32 * s;
      bi = static_cast<int>(__reduce_min_sync(0xffffffffu, static_cast<uint32_t>(next)));
      bv = __int_as_float(0x7FC00000);
    }
    if ((bi & 31) == lane) {
      taken |= 1u << (bi >> 5);
      look();
    }
    __syncwarp();
    const float p = mode == 0 ? __expf(bv - mx) / z : 1.0f / (1.0f + expf(-row[bi]));
    if (lane == j) { my_p = p; my_i = bi; }
    wsum += p;
  }
  if (lane < k) {
    const float w = mode == 0 ? (renorm ? my_p / wsum : my_p) : (renorm ? my_p / (wsum + 1e-6f) : my_p) * scale;
    ids[lane] = my_i;
    weights[lane] = __bfloat162float(__float2bfloat16(w));
  }
}

__global__ void MoeRouterKernel(const float* __restrict__ logits, const float* __restrict__ bias, int T, int E, int k,
                                int renorm, int mode, float scale, int* __restrict__ ids, float* __restrict__ weights) {
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= T) return;
  RouteRow(logits + static_cast<size_t>(t) * E, bias, E, k, renorm, mode, scale, threadIdx.x & 31, ids + static_cast<size_t>(t) * k,
           weights + static_cast<size_t>(t) * k);
}

// The lanes that hold the same expert e (-1: none) of `bits`-bit expert ids: a ballot per bit.  (__match_any_sync goes through the
// distinct values one by one: thirty of them here.)
__device__ __forceinline__ unsigned SameExpert(int e, int bits) {
  unsigned same = __ballot_sync(0xffffffffu, e >= 0);
  if (e < 0) same = ~same;
  for (int b = 0; b < bits; ++b) {
    const unsigned set = __ballot_sync(0xffffffffu, (e >> b) & 1);
    same &= ((e >> b) & 1) ? set : ~set;
  }
  return same;
}

// v[0 .. n) becomes its running sums; every thread of the CTA takes part (blockDim a multiple of 32).
__device__ __forceinline__ void BlockInclusiveScan(int* v, int n, int* warp_sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int per = (n + blockDim.x - 1) / blockDim.x, lo = threadIdx.x * per, hi = min(n, lo + per);
  int sum = 0;
  for (int i = lo; i < hi; ++i) sum += v[i];
  int incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += u;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  int run = incl - sum;
  for (int w = 0; w < warps; ++w)
    if (w < warp) run += warp_sums[w];
  for (int i = lo; i < hi; ++i) {
    run += v[i];
    v[i] = run;
  }
  __syncthreads();
}

// Up to 8 rows (a decode step or a verify window): one CTA routes every row (a warp each) and then builds the plan of the
// T * k pairs itself, so routing is one launch instead of two.  Same results as MoeRouterKernel + MoePlanKernel.  (One row of 512
// experts, top 10: 15.5 -> 8.3 us; one thread's running sum over the experts was half of it.)
__global__ void __launch_bounds__(256)
MoeRoutePlanKernel(const float* __restrict__ logits, const float* __restrict__ bias, int T, int E, int k, int renorm, int mode,
                   float scale, int* __restrict__ ids, float* __restrict__ weights, int e_begin, int e_count,
                   int* __restrict__ offsets, int* __restrict__ perm) {
  extern __shared__ int cnt[];     // [e_count + 1]
  __shared__ int s_ids[8 * kMaxK], warp_sums[32];
  const int warp = threadIdx.x >> 5;
  for (int e = threadIdx.x; e <= e_count; e += blockDim.x) cnt[e] = 0;
  if (warp < T)
    RouteRow(logits + static_cast<size_t>(warp) * E, bias, E, k, renorm, mode, scale, threadIdx.x & 31, ids + warp * k, weights + warp * k);
  __syncthreads();                 // the ids written above are visible to the whole CTA
  const int npairs = T * k;
  if (threadIdx.x < npairs) {
    const int e = ids[threadIdx.x] - e_begin;
    s_ids[threadIdx.x] = e;
    if (e >= 0 && e < e_count) atomicAdd(&cnt[e + 1], 1);
  }
  __syncthreads();
  BlockInclusiveScan(cnt, e_count + 1, warp_sums);
  for (int e = threadIdx.x; e <= e_count; e += blockDim.x) offsets[e] = cnt[e];
  if (threadIdx.x < npairs) {      // stable placement: behind the expert's pairs of a lower index (at most 128 pairs)
    const int e = s_ids[threadIdx.x];
    if (e >= 0 && e < e_count) {
      int at = cnt[e];
      for (int p = 0; p < threadIdx.x; ++p) at += s_ids[p] == e ? 1 : 0;
      perm[at] = threadIdx.x;
    }
  }
}

// Single CTA: counting sort of the T*k pairs by expert (stable in pair order), a pair per thread; the warps place theirs one after
// the other.  (640 pairs of 512 experts: 28.8 -> 5.8 us; one thread did it.)  Few pairs and experts take a smaller CTA.
constexpr int kPlanThreads = 1024;
__global__ void __launch_bounds__(kPlanThreads) MoePlanKernel(const int* __restrict__ ids, int npairs, int E, int e_begin, int e_count,
                              int* __restrict__ offsets, int* __restrict__ perm) {
  extern __shared__ int cnt[];     // [e_count + 1]
  __shared__ int warp_sums[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto expert_of = [&](int p) {
    const int e = p < npairs ? ids[p] - e_begin : -1;
    return e < 0 || e >= e_count ? -1 : e;
  };
  for (int e = threadIdx.x; e <= e_count; e += blockDim.x) cnt[e] = 0;
  __syncthreads();
  for (int p = threadIdx.x; p < npairs; p += blockDim.x) {
    const int e = expert_of(p);
    if (e >= 0) atomicAdd(&cnt[e + 1], 1);
  }
  __syncthreads();
  BlockInclusiveScan(cnt, e_count + 1, warp_sums);
  for (int e = threadIdx.x; e <= e_count; e += blockDim.x) offsets[e] = cnt[e];
  __syncthreads();
  for (int base = 0; base < npairs; base += blockDim.x) {
    const int p = base + threadIdx.x, e = expert_of(p);
    const unsigned same = SameExpert(e, 32 - __clz(e_count - 1));
    for (int w = 0; w < (min(npairs - base, static_cast<int>(blockDim.x)) + 31) / 32; ++w) {
      if (warp == w && e >= 0) perm[cnt[e] + __popc(same & ((1u << lane) - 1u))] = p;
      __syncwarp();
      if (warp == w && e >= 0 && lane == __ffs(same) - 1) cnt[e] += __popc(same);
      __syncthreads();
    }
  }
}

// The same plan for many pairs (prefill chunks, wide batches): one CTA of 32 warps, warp w owns a contiguous run of the
// pairs.  Pass 1 counts per (warp, expert), a prefix over experts and warps turns the counts into each warp's first slot
// per expert, pass 2 places the pairs; inside a 32-pair step the lanes of one expert are ranked among themselves, so the
// order inside an expert is the pair order.  Eight steps' ids are requested together (40960 pairs of 512 experts: 96 -> 37 us).
constexpr int kPlanWarps = 32;
constexpr int kPlanAhead = 8;
__global__ void __launch_bounds__(kPlanWarps * 32)
MoePlanParallelKernel(const int* __restrict__ ids, int npairs, int e_begin, int e_count, int* __restrict__ offsets,
                      int* __restrict__ perm) {
  __shared__ int warp_sums[32];
  extern __shared__ int sm[];                  // [kPlanWarps][e_count] counts / cursors, then [e_count + 1] offsets
  int* hist = sm;
  int* offs = sm + kPlanWarps * e_count;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < kPlanWarps * e_count; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  const int per = ((npairs + kPlanWarps - 1) / kPlanWarps + 31) & ~31;       // pairs per warp, a multiple of 32
  const int p0 = warp * per, p1 = min(npairs, p0 + per);
  int* mine = hist + warp * e_count;
  int next[kPlanAhead];
  auto request = [&](int base) {
#pragma unroll
    for (int i = 0; i < kPlanAhead; ++i) {
      const int p = base + 32 * i + lane;
      const int e = p < p1 ? ids[p] - e_begin : -1;
      next[i] = e < 0 || e >= e_count ? -1 : e;
    }
  };
  for (int base = p0; base < p1; base += 32 * kPlanAhead) {
    request(base);
#pragma unroll
    for (int i = 0; i < kPlanAhead; ++i)
      if (base + 32 * i < p1 && next[i] >= 0) atomicAdd(&mine[next[i]], 1);
  }
  __syncthreads();
  // per expert: total, then each warp's first slot
  for (int e = threadIdx.x; e < e_count; e += blockDim.x) {
    int tot = 0;
    for (int w = 0; w < kPlanWarps; ++w) tot += hist[w * e_count + e];
    offs[e + 1] = tot;
  }
  if (threadIdx.x == 0) offs[0] = 0;
  __syncthreads();
  BlockInclusiveScan(offs, e_count + 1, warp_sums);
  for (int e = threadIdx.x; e <= e_count; e += blockDim.x) offsets[e] = offs[e];
  for (int e = threadIdx.x; e < e_count; e += blockDim.x) {
    int at = offs[e];
    for (int w = 0; w < kPlanWarps; ++w) {
      const int c = hist[w * e_count + e];
      hist[w * e_count + e] = at;              // becomes the warp's cursor
      at += c;
    }
  }
  __syncthreads();
  for (int base = p0; base < p1; base += 32 * kPlanAhead) {
    request(base);
#pragma unroll
    for (int i = 0; i < kPlanAhead; ++i) {
      if (base + 32 * i >= p1) break;
      const int e = next[i];
      const unsigned same = SameExpert(e, 32 - __clz(e_count - 1));
      if (e >= 0) perm[mine[e] + __popc(same & ((1u << lane) - 1u))] = base + 32 * i + lane;
      __syncwarp();
      if (e >= 0 && lane == __ffs(same) - 1) mine[e] += __popc(same);
      __syncwarp();
    }
  }
}

// grid (T, ceil(H / 512)): out[t] = residual + sum_j w_j y[pair] (ascending expert id) + sigmoid(sg) * shared; C columns a thread
// (eight by 16-byte loads, four experts' in flight, where the rows allow it: 4096 rows of 2048 columns, top 10, 74 -> 41 us).
constexpr int kCombineCols = 512;
template <int C>
__global__ void __launch_bounds__(kCombineCols / C)
MoeCombineKernel(const __nv_bfloat16* __restrict__ y_pairs, const int* __restrict__ ids,
                 const float* __restrict__ weights, const __nv_bfloat16* __restrict__ shared,
                 const float* __restrict__ shared_gate, const __nv_bfloat16* __restrict__ residual,
                 __nv_bfloat16* __restrict__ out, int H, int k) {
  const int t = blockIdx.x;
  __shared__ int order[kMaxK], sid[kMaxK];
  __shared__ float w[kMaxK], sw[kMaxK];
  if (threadIdx.x < k) {                     // one parallel read of the row's ids and weights; the sort runs on shared memory
    sid[threadIdx.x] = ids[t * k + threadIdx.x];
    sw[threadIdx.x] = weights[t * k + threadIdx.x];
  }
  __syncthreads();
  if (threadIdx.x < k) {                     // rank of slot j among the row's expert ids (ids of a row are distinct; ties by slot)
    const int mine = sid[threadIdx.x];
    int rank = 0;
    for (int j = 0; j < k; ++j) rank += (sid[j] < mine || (sid[j] == mine && j < static_cast<int>(threadIdx.x))) ? 1 : 0;
    order[rank] = threadIdx.x;
    w[rank] = sw[threadIdx.x];
  }
  __syncthreads();
  // grid.y splits the columns: a single row (decode) still spreads over several SMs
  const int c = blockIdx.y * kCombineCols + threadIdx.x * C;
  if (c >= H) return;
  using Vec = typename std::conditional<C == 8, uint4, uint32_t>::type;
  auto add = [&](const __nv_bfloat16* row, float f, float (&acc)[C]) {
    const Vec v = *reinterpret_cast<const Vec*>(row + c);
    const uint32_t* p = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
    for (int i = 0; i < C / 2; ++i) {
      acc[2 * i] = fmaf(f, BfLo(p[i]), acc[2 * i]);
      acc[2 * i + 1] = fmaf(f, BfHi(p[i]), acc[2 * i + 1]);
    }
  };
  float acc[C];
#pragma unroll
  for (int i = 0; i < C; ++i) acc[i] = 0.f;
  const __nv_bfloat16* y = y_pairs + static_cast<size_t>(t) * k * H;
#pragma unroll 4
  for (int j = 0; j < k; ++j) add(y + static_cast<size_t>(order[j]) * H, w[j], acc);
  if (shared) add(shared + static_cast<size_t>(t) * H, shared_gate ? Sigmoid(shared_gate[t]) : 0.f, acc);
  if (residual) add(residual + static_cast<size_t>(t) * H, 1.0f, acc);
  uint32_t o[C / 2];
#pragma unroll
  for (int i = 0; i < C / 2; ++i) o[i] = PackBf16(acc[2 * i], acc[2 * i + 1]);
  *reinterpret_cast<Vec*>(out + static_cast<size_t>(t) * H + c) = *reinterpret_cast<const Vec*>(o);
}

}  // namespace
}  // namespace r4dxb

using namespace r4dxb;

extern "C" {

int r4dxb_moe_router(const float* logits, int T, int E, int k, int renorm, int* ids, float* weights, void* stream) {
  if (T < 1 || k < 1 || k > kMaxK || E > 1024 || E < k) return R4DXB_BAD_ARG;
  MoeRouterKernel<<<(T + 3) / 4, 128, 0, static_cast<cudaStream_t>(stream)>>>(logits, nullptr, T, E, k, renorm, 0, 1.0f, ids,
                                                                              weights);
  return FinishLaunch();
}

/* Sigmoid router: selection by sigmoid(logit) + bias (bias may be null), weights = unbiased sigmoids / (sum + 1e-6) * scale */
int r4dxb_moe_router_sigmoid(const float* logits, const float* bias, int T, int E, int k, int renorm, float scale, int* ids,
                             float* weights, void* stream) {
  if (T < 1 || k < 1 || k > kMaxK || E > 1024 || E < k) return R4DXB_BAD_ARG;
  MoeRouterKernel<<<(T + 3) / 4, 128, 0, static_cast<cudaStream_t>(stream)>>>(logits, bias, T, E, k, renorm, 1, scale, ids,
                                                                              weights);
  return FinishLaunch();
}

/* Router (mode 0 softmax, 1 sigmoid + bias) and routing plan of up to 8 rows in one launch */
int r4dxb_moe_route_plan(const float* logits, const float* bias, int T, int E, int k, int renorm, int mode, float scale, int* ids,
                         float* weights, int e_begin, int e_count, int* offsets, int* perm, void* stream) {
  if (T < 1 || T > 8 || k < 1 || k > kMaxK || E > 1024 || E < k || e_count < 1 || e_count > 8192 || (mode != 0 && mode != 1))
    return R4DXB_BAD_ARG;
  MoeRoutePlanKernel<<<1, 256, (e_count + 1) * sizeof(int), static_cast<cudaStream_t>(stream)>>>(
      logits, bias, T, E, k, renorm, mode, scale, ids, weights, e_begin, e_count, offsets, perm);
  return FinishLaunch();
}

/* offsets: [e_count + 1], perm: [npairs] pair indices sorted by expert (only experts in [e_begin, e_begin+e_count)) */
int r4dxb_moe_plan(const int* ids, int npairs, int E, int e_begin, int e_count, int* offsets, int* perm, void* stream) {
  if (npairs < 1 || e_count < 1 || e_count > 8192) return R4DXB_BAD_ARG;
  const size_t big = (static_cast<size_t>(kPlanWarps) * e_count + e_count + 1) * sizeof(int);
  if (npairs > 1024 && big <= 200 * 1024) {
    // many pairs: the serial placement of the small kernel would take milliseconds (2 ms for 40960 pairs)
    if (big > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(MoePlanParallelKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(big));
      if (e != cudaSuccess) return static_cast<int>(e);
    }
    MoePlanParallelKernel<<<1, kPlanWarps * 32, big, static_cast<cudaStream_t>(stream)>>>(ids, npairs, e_begin, e_count, offsets, perm);
    return FinishLaunch();
  }
  const int threads = npairs <= 128 && e_count <= 128 ? 128 : kPlanThreads;
  MoePlanKernel<<<1, threads, (e_count + 1) * sizeof(int), static_cast<cudaStream_t>(stream)>>>(ids, npairs, E, e_begin, e_count,
                                                                                             offsets, perm);
  return FinishLaunch();
}

int r4dxb_moe_combine(const void* y_pairs, const int* ids, const float* weights, const void* shared, const float* shared_gate,
                      const void* residual, void* out, int T, int H, int k, void* stream) {
  if (T < 1 || k < 1 || k > kMaxK || H % 2) return R4DXB_BAD_ARG;
  const uintptr_t bases = reinterpret_cast<uintptr_t>(y_pairs) | reinterpret_cast<uintptr_t>(shared) | reinterpret_cast<uintptr_t>(residual) |
                          reinterpret_cast<uintptr_t>(out);
  // (one and 64 rows of 2048 columns: 4.1 and 5.5 us with two columns a thread, 4.5 and 6.5 with eight)
  const bool wide = H % 8 == 0 && (bases & 15) == 0 && static_cast<long long>(T) * H >= 1 << 20;
  (wide ? MoeCombineKernel<8> : MoeCombineKernel<2>)<<<dim3(T, (H + kCombineCols - 1) / kCombineCols), kCombineCols / (wide ? 8 : 2), 0,
                                                        static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(y_pairs), ids, weights, static_cast<const __nv_bfloat16*>(shared), shared_gate,
      static_cast<const __nv_bfloat16*>(residual), static_cast<__nv_bfloat16*>(out), H, k);
  return FinishLaunch();
}

}  // extern "C"
