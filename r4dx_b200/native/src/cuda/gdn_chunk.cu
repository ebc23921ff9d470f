// Chunked (WY-form) gated delta rule for long prefill chunks, D = 128, 64 tokens per chunk.
//
// With gamma_i the running product of the decay inside a chunk and S0 the state before it, the 64
// rank-one updates of the chunk collapse to
//   (I + A) U = beta V - (beta gamma K) S0^T,   A_ij = beta_i (gamma_i / gamma_j) (k_i . k_j), j < i
//   O   = diag(gamma) Q S0^T + P U,             P_ij = (gamma_i / gamma_j) (q_i . k_j),       j <= i
//   S64 = gamma_64 S0 + U^T diag(gamma_64 / gamma) K
// so the work splits in two kernels:
//   phase A (grid chunks x heads, no dependence on the state): A and P in fp32, then the triangular
//           solve for U~ = (I + A)^-1 beta V and W = (I + A)^-1 beta gamma K by forward substitution,
//           one right-hand-side column per thread with the 64 unknowns in registers.  The solve is right-looking (a
//           solved unknown is subtracted from all later ones at once): the sums are independent, where adding up
//           unknown i's terms when its turn comes is a chain of i multiply-adds behind a global load.  What bounds it is the
//           fp32 multiply-adds of the two products and the solve (packed in pairs: 27k of a CTA's 41k clocks, two CTAs to an SM)
//           and the waits for the rows between them: 601 -> 468 us for 8192 tokens of 48 heads with pairs and with the rows
//           of q and k copied asynchronously (three CTAs to an SM, in 80 registers with spills: 628);
//   phase B (grid heads x 2 or 4 row blocks of the state, sequential over chunks): U = U~ - W S0^T,
//           O, and the state update as TF32 tensor-core products (mma.sync m16n8k8, fp32
//           accumulate) out of shared memory; W, Q, P and K have a cp.async slot each that is refilled for the
//           next chunk as soon as its product is done, three products ahead of its use (two shared slots fetched one
//           product ahead left every one of the four products of a chunk waiting for its operand: 14k clocks a
//           chunk where the products take about five).  The fp32 state block lives in registers for
//           the whole sequence.
// The per-token recurrence (gdn_prefill.cu) stays as the reference path and for D = 64
// (reference: third_party/libr4d/r4d_gdn_chunk_scan_k128_v128_c64_bf16.hip:1-60 runs the same
// algebra in bf16 on its matrix cores).
#include <cuda_pipeline.h>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace r4dxb {
namespace {

constexpr int kC = 64;            // tokens per chunk
constexpr int kD = 128;           // key and value head width
constexpr int kLdK = kD + 4;      // phase A: row stride of k / q (conflict-free 16-byte row reads)
constexpr int kLdA = kC + 4;

struct PhaseASmem {
  float ks[kC][kLdK];
  float qs[kC][kLdK];
  float At[kC][kLdA];     // -A transposed: row j holds the factors of unknown j
  float G[kC];
  float B[kC];
  float BG[kC];           // beta gamma
};

__device__ __forceinline__ uint32_t Tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

// two products and two sums an instruction, the even and the odd columns apart
__device__ __forceinline__ float2 Dot4(const float4& a, const float4& b, float2 acc) {
  acc = ptx::Fma2(make_float2(a.x, a.y), make_float2(b.x, b.y), acc);
  return ptx::Fma2(make_float2(a.z, a.w), make_float2(b.z, b.w), acc);
}

// grid (chunks, H), 256 threads
__global__ void __launch_bounds__(256) GdnChunkPrepKernel(const float* __restrict__ q, const float* __restrict__ k,
                                                          const float* __restrict__ v, const float* __restrict__ eg,
                                                          const float* __restrict__ beta, float* __restrict__ ws_ut,
                                                          float* __restrict__ ws_w, float* __restrict__ ws_p,
                                                          float* __restrict__ ws_g, int T, int H, int Hk) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PhaseASmem& sm = *reinterpret_cast<PhaseASmem*>(smem_raw);
  const int c = blockIdx.x, h = blockIdx.y, hk = h / (H / Hk);
  const int t0 = c * kC, tid = threadIdx.x;
  const size_t ch = static_cast<size_t>(c) * H + h;

  // all rows in flight at once, zeros past the last token (through registers, two loads a step, this was 10k clocks of 41k a CTA)
#pragma unroll
  for (int i = tid; i < kC * kD / 4; i += 256) {
    const int row = i / (kD / 4), off = (i % (kD / 4)) * 4;
    const size_t at = (static_cast<size_t>(min(t0 + row, T - 1)) * Hk + hk) * kD + off;
    const size_t zeros = t0 + row < T ? 0 : 16;
    __pipeline_memcpy_async(&sm.ks[row][off], k + at, 16, zeros);
    __pipeline_memcpy_async(&sm.qs[row][off], q + at, 16, zeros);
  }
  __pipeline_commit();
  // the right-hand sides are read after the products: a line of v per thread on its way to L2 until then
  if (t0 + tid / 4 < T)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(v + (static_cast<size_t>(t0 + tid / 4) * H + h) * kD + tid % 4 * 32));
  if (tid < kC) {
    const int t = t0 + tid;
    // rows past the end are identity steps: decay 1, beta 0
    sm.B[tid] = t < T ? beta[static_cast<size_t>(t) * H + h] : 0.f;
    sm.G[tid] = t < T ? fmaxf(logf(eg[static_cast<size_t>(t) * H + h]), -80.f) : 0.f;
  }
  __syncthreads();
  // Running sum of the 64 log decays, each thread its own in token order: neighbouring sums then share all earlier roundings, so
  // they never rise and exp(G_i - G_j) stays below 1 (a tree of partial sums doubled the error of a pair's decay).
  float sum = 0.f;
  if (tid < kC) {
#pragma unroll
    for (int j = 0; j < kC; j += 4) {
      const float4 g4 = *reinterpret_cast<const float4*>(&sm.G[j]);
      if (j <= tid) sum += g4.x;
      if (j + 1 <= tid) sum += g4.y;
      if (j + 2 <= tid) sum += g4.z;
      if (j + 3 <= tid) sum += g4.w;
    }
  }
  __syncthreads();
  if (tid < kC) {
    sm.G[tid] = sum;
    sm.BG[tid] = sm.B[tid] * expf(sum);
  }
  __pipeline_wait_prior(0);
  __syncthreads();
  if (tid < kC) ws_g[ch * kC + tid] = sm.G[tid];

  // ---- k.k and q.k for the lower triangle: thread (ty, tx) owns rows ty + 16 rr, columns tx + 16 cc ----
  {
    const int ty = tid >> 4, tx = tid & 15;
    float2 kk[4][4], qk[4][4];
#pragma unroll
    for (int rr = 0; rr < 4; ++rr)
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) kk[rr][cc] = qk[rr][cc] = make_float2(0.f, 0.f);
    for (int kq = 0; kq < kD; kq += 4) {
      float4 kr[4], qr[4], kc[4];
#pragma unroll
      for (int rr = 0; rr < 4; ++rr) {
        kr[rr] = *reinterpret_cast<const float4*>(&sm.ks[ty + 16 * rr][kq]);
        qr[rr] = *reinterpret_cast<const float4*>(&sm.qs[ty + 16 * rr][kq]);
        kc[rr] = *reinterpret_cast<const float4*>(&sm.ks[tx + 16 * rr][kq]);
      }
#pragma unroll
      for (int rr = 0; rr < 4; ++rr)
#pragma unroll
        for (int cc = 0; cc < 4; ++cc)
          if (cc <= rr) {      // 16-wide column blocks right of the row block are entirely above the diagonal
            kk[rr][cc] = Dot4(kr[rr], kc[cc], kk[rr][cc]);
            qk[rr][cc] = Dot4(qr[rr], kc[cc], qk[rr][cc]);
          }
    }
#pragma unroll
    for (int rr = 0; rr < 4; ++rr)
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) {
        const int i = ty + 16 * rr, j = tx + 16 * cc;
        const float decay = j <= i ? expf(sm.G[i] - sm.G[j]) : 0.f;
        if (j < i) sm.At[j][i] = -(sm.B[i] * decay * (kk[rr][cc].x + kk[rr][cc].y));
        ws_p[(ch * kC + i) * kC + j] = __uint_as_float(Tf32(decay * (qk[rr][cc].x + qk[rr][cc].y)));     // (as phase B's product takes it)
      }
  }
  __syncthreads();

  // ---- forward substitution: thread = one right-hand-side column (128 of beta V, 128 of beta gamma K) ----
  {
    const bool is_u = tid < kD;
    const int col = is_u ? tid : tid - kD;
    float* dst = (is_u ? ws_ut : ws_w) + ch * kC * kD + col;
    float2 x[kC / 2];                        // unknowns 2 p and 2 p + 1
    auto at = [&](int i) -> float& { return i & 1 ? x[i >> 1].y : x[i >> 1].x; };
    if (is_u) {
      const float* src = v + (static_cast<size_t>(t0) * H + h) * kD + col;
#pragma unroll
      for (int i = 0; i < kC; ++i) at(i) = t0 + i < T ? src[static_cast<size_t>(i) * H * kD] : 0.f;
#pragma unroll
      for (int i = 0; i < kC; ++i) at(i) *= sm.B[i];
    } else {
#pragma unroll
      for (int i = 0; i < kC; ++i) at(i) = sm.BG[i] * sm.ks[i][col];
    }
#pragma unroll
    for (int j = 0; j < kC; ++j) {
      const float xj = at(j);
      const float2 xj2 = make_float2(xj, xj);
#pragma unroll
      for (int i4 = ((j + 1) / 4) * 4; i4 < kC; i4 += 4) {
        const float4 a = *reinterpret_cast<const float4*>(&sm.At[j][i4]);
        if (i4 > j) x[i4 / 2] = ptx::Fma2(make_float2(a.x, a.y), xj2, x[i4 / 2]);
        else if (i4 + 1 > j) x[i4 / 2].y = fmaf(a.y, xj, x[i4 / 2].y);
        if (i4 + 2 > j) x[i4 / 2 + 1] = ptx::Fma2(make_float2(a.z, a.w), xj2, x[i4 / 2 + 1]);
        else if (i4 + 3 > j) x[i4 / 2 + 1].y = fmaf(a.w, xj, x[i4 / 2 + 1].y);
      }
      // W is an operand of phase B's tensor-core products only: rounded here instead of at every read
      dst[static_cast<size_t>(j) * kD] = is_u ? xj : __uint_as_float(Tf32(xj));
    }
  }
}

// ---------------------------------------- phase B ----------------------------------------
constexpr int kLd = kD + 8;       // W / Q / K / state rows: conflict-free 8-byte fragment reads and strided scalar reads
constexpr int kLdP = kC + 4;      // P rows: conflict-free scalar fragment reads
static_assert(kC == 64, "the warps of a CTA tile 64 tokens by kRows columns");

// kRows: state rows (value columns) of a CTA, 32 or 64; kRows * 8 threads.
template <int kRows>
struct PhaseBSmem {
  static constexpr int kLdU = kRows + 8;   // U rows
  float W[kC * kLd];
  float Q[kC * kLd];
  float K[kC * kLd];
  float P[kC * kLdP];
  float S[kRows][kLd];
  float U[2][kC][kLdU];
  float G[2][kC];
  float eG[kC];
  float fG[kC];
};

// The same rounding (half away from zero) in two integer instructions: conversions run at a quarter of their rate, and the scan
// needs thousands of them per chunk.  It would carry the NaN that arithmetic produces into the sign bit and leave a zero, so
// the values it is applied to (q, k and U in shared memory) were written through PlainNan; RoundTf32Any takes any NaN.  (A
// compare and a select at every rounding: 1674 against 1582 us for 8192 tokens of 48 heads.)
__device__ __forceinline__ uint32_t RoundTf32(float x) { return (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u; }
__device__ __forceinline__ uint32_t RoundTf32Any(float x) { return RoundTf32(PlainNan(x)); }

__device__ __forceinline__ void MmaTf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// acc[nt] += A[m0 .. m0+16, 0 .. 128) * S[n0 + 8 nt .. +8, 0 .. 128)^T, both row-major along the contraction.
// Inside every block of 8 contraction columns the hardware index t maps to column 2t and t + 4 to 2t + 1, so
// that one 8-byte load feeds two fragment registers; A and B use the same map, so the product is unchanged.
// kRounded: A already holds TF32 values (S always does).
template <int NT, bool kRounded>
__device__ __forceinline__ void MmaRowRow(float (&acc)[NT][4], const float* __restrict__ A, int m0, const float* __restrict__ S,
                                          int n0, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const float* a_lo = A + (m0 + g) * kLd + 2 * t;
  const float* a_hi = a_lo + 8 * kLd;
  const float* b_base = S + (n0 + g) * kLd + 2 * t;
#pragma unroll 4
  for (int kb = 0; kb < kD / 8; ++kb) {
    const float2 lo = *reinterpret_cast<const float2*>(a_lo + kb * 8);
    const float2 hi = *reinterpret_cast<const float2*>(a_hi + kb * 8);
    const uint32_t a0 = kRounded ? __float_as_uint(lo.x) : RoundTf32(lo.x), a2 = kRounded ? __float_as_uint(lo.y) : RoundTf32(lo.y);
    const uint32_t a1 = kRounded ? __float_as_uint(hi.x) : RoundTf32(hi.x), a3 = kRounded ? __float_as_uint(hi.y) : RoundTf32(hi.y);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const float2 b = *reinterpret_cast<const float2*>(b_base + nt * 8 * kLd + kb * 8);
      MmaTf32(acc[nt], a0, a1, a2, a3, __float_as_uint(b.x), __float_as_uint(b.y));
    }
  }
}

template <int kThreads>
__device__ __forceinline__ void CopyRows(float* dst, int ld_dst, const float* src, size_t src_stride, int rows, int row_floats,
                                         int tid) {
  const int per_row = row_floats / 4;
  for (int i = tid; i < rows * per_row; i += kThreads) {
    const int r = i / per_row, o = (i % per_row) * 4;
    __pipeline_memcpy_async(dst + r * ld_dst + o, src + static_cast<size_t>(r) * src_stride + o, 16);
  }
}

// grid (H, 128 / kRows): CTA (h, vb) owns state rows [kRows vb, kRows vb + kRows) of head h
template <int kRows>
__global__ void __launch_bounds__(kRows * 8, 1) GdnChunkScanKernel(const float* __restrict__ q, const float* __restrict__ k,
                                                             const float* __restrict__ ws_ut, const float* __restrict__ ws_w,
                                                             const float* __restrict__ ws_p, const float* __restrict__ ws_g,
                                                             float* __restrict__ state, float* __restrict__ o, int T, int H,
                                                             int Hk) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PhaseBSmem<kRows>& sm = *reinterpret_cast<PhaseBSmem<kRows>*>(smem_raw);
  constexpr int kScanThreads = kRows * 8, kLdU = PhaseBSmem<kRows>::kLdU;
  const int h = blockIdx.x, vb = blockIdx.y, hk = h / (H / Hk);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int chunks = (T + kC - 1) / kC;
  const float scale = rsqrtf(static_cast<float>(kD));

  // every call commits one copy group, an empty one past the last chunk, so that "all but the two newest" always names
  // the operand of the next product
  auto issue_wug = [&](int c) {               // W, U~ (this CTA's columns) and G
    if (c < chunks) {
      const size_t ch = static_cast<size_t>(c) * H + h;
      CopyRows<kScanThreads>(sm.W, kLd, ws_w + ch * kC * kD, kD, kC, kD, tid);
      CopyRows<kScanThreads>(&sm.U[c & 1][0][0], kLdU, ws_ut + ch * kC * kD + vb * kRows, kD, kC, kRows, tid);
      if (tid < kC / 4) __pipeline_memcpy_async(&sm.G[c & 1][tid * 4], ws_g + ch * kC + tid * 4, 16);
    }
    __pipeline_commit();
  };
  auto issue_rows = [&](float* dst, const float* src, int c) {     // token rows of q or k (clamped past the end)
    if (c < chunks) {
      for (int i = tid; i < kC * (kD / 4); i += kScanThreads) {
        const int r = i / (kD / 4), off = (i % (kD / 4)) * 4;
        const int t = min(c * kC + r, T - 1);
        __pipeline_memcpy_async(dst + r * kLd + off, src + (static_cast<size_t>(t) * Hk + hk) * kD + off, 16);
      }
    }
    __pipeline_commit();
  };
  auto issue_p = [&](int c) {
    if (c < chunks) CopyRows<kScanThreads>(sm.P, kLdP, ws_p + (static_cast<size_t>(c) * H + h) * kC * kC, kC, kC, kC, tid);
    __pipeline_commit();
  };

  issue_wug(0);
  issue_rows(sm.Q, q, 0);
  issue_p(0);
  // The fp32 state stays in registers in the accumulator layout of product 3 (a warp: 16 rows x 32 columns); shared memory
  // holds its TF32 rounding, which is what products 1 and 2a read.
  const int sm0 = (warp % (kRows / 16)) * 16, sn0 = (warp / (kRows / 16)) * 32;
  float* s_lo = state + (static_cast<size_t>(h) * kD + vb * kRows + sm0 + g) * kD + sn0 + 2 * t4;
  float* s_hi = s_lo + 8 * kD;
  float st[4][4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const float2 lo = *reinterpret_cast<const float2*>(s_lo + nt * 8), hi = *reinterpret_cast<const float2*>(s_hi + nt * 8);
    st[nt][0] = lo.x; st[nt][1] = lo.y; st[nt][2] = hi.x; st[nt][3] = hi.y;
  }
  auto publish = [&] {
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      *reinterpret_cast<uint2*>(&sm.S[sm0 + g][sn0 + nt * 8 + 2 * t4]) = make_uint2(RoundTf32Any(st[nt][0]), RoundTf32Any(st[nt][1]));
      *reinterpret_cast<uint2*>(&sm.S[sm0 + g + 8][sn0 + nt * 8 + 2 * t4]) = make_uint2(RoundTf32Any(st[nt][2]), RoundTf32Any(st[nt][3]));
    }
  };
  publish();

  for (int c = 0; c < chunks; ++c) {
    const int buf = c & 1;
    __pipeline_wait_prior(2);
    __syncthreads();                       // W, U~, G of this chunk have landed; the state block is complete, K no longer read
    issue_rows(sm.K, k, c);
    if (tid < kC) {
      sm.eG[tid] = expf(sm.G[buf][tid]);
      sm.fG[tid] = expf(sm.G[buf][kC - 1] - sm.G[buf][tid]);
    }
    // ---- 1: U = U~ - W S^T   (64 x kRows; warp: 16 rows x 16 columns) ----
    const int m0 = (warp & 3) * 16, nh = (warp >> 2) * 16;
    {
      float acc[2][4] = {};
      MmaRowRow<2, true>(acc, sm.W, m0, &sm.S[0][0], nh, lane);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        float2* lo = reinterpret_cast<float2*>(&sm.U[buf][m0 + g][nh + nt * 8 + 2 * t4]);
        float2* hi = reinterpret_cast<float2*>(&sm.U[buf][m0 + g + 8][nh + nt * 8 + 2 * t4]);
        const float2 a = *lo, b = *hi;
        *lo = make_float2(PlainNan(a.x - acc[nt][0]), PlainNan(a.y - acc[nt][1]));
        *hi = make_float2(PlainNan(b.x - acc[nt][2]), PlainNan(b.y - acc[nt][3]));
      }
    }
    __pipeline_wait_prior(2);
    __syncthreads();                       // U complete, Q landed, W no longer read
    issue_wug(c + 1);
    // ---- 2a: O = diag(gamma) Q S^T ----
    float oacc[2][4] = {};
    MmaRowRow<2, false>(oacc, sm.Q, m0, &sm.S[0][0], nh, lane);
    {
      const float e_lo = sm.eG[m0 + g], e_hi = sm.eG[m0 + g + 8];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        oacc[nt][0] *= e_lo; oacc[nt][1] *= e_lo; oacc[nt][2] *= e_hi; oacc[nt][3] *= e_hi;
      }
    }
    __pipeline_wait_prior(2);
    __syncthreads();                       // P landed, Q no longer read
    issue_rows(sm.Q, q, c + 1);
    // ---- 2b: O += P U   (P was written rounded) ----
    {
#pragma unroll 4
      for (int kb = 0; kb < kC / 8; ++kb) {
        const uint32_t a0 = __float_as_uint(sm.P[(m0 + g) * kLdP + kb * 8 + t4]), a1 = __float_as_uint(sm.P[(m0 + g + 8) * kLdP + kb * 8 + t4]);
        const uint32_t a2 = __float_as_uint(sm.P[(m0 + g) * kLdP + kb * 8 + t4 + 4]), a3 = __float_as_uint(sm.P[(m0 + g + 8) * kLdP + kb * 8 + t4 + 4]);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const uint32_t b0 = RoundTf32(sm.U[buf][kb * 8 + t4][nh + nt * 8 + g]);
          const uint32_t b1 = RoundTf32(sm.U[buf][kb * 8 + t4 + 4][nh + nt * 8 + g]);
          MmaTf32(oacc[nt], a0, a1, a2, a3, b0, b1);
        }
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const int col = vb * kRows + nh + nt * 8 + 2 * t4;
        const int t_lo = c * kC + m0 + g, t_hi = t_lo + 8;
        if (t_lo < T)
          *reinterpret_cast<float2*>(o + (static_cast<size_t>(t_lo) * H + h) * kD + col) =
              make_float2(oacc[nt][0] * scale, oacc[nt][1] * scale);
        if (t_hi < T)
          *reinterpret_cast<float2*>(o + (static_cast<size_t>(t_hi) * H + h) * kD + col) =
              make_float2(oacc[nt][2] * scale, oacc[nt][3] * scale);
      }
    }
    __pipeline_wait_prior(2);
    __syncthreads();                       // K landed, P no longer read
    issue_p(c + 1);
    // ---- 3: S = gamma_C S + U^T diag(gamma_C / gamma) K   (kRows x 128; warp: 16 rows x 32 columns) ----
    {
      const float e_c = sm.eG[kC - 1];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) st[nt][i] *= e_c;
#pragma unroll 2
      for (int kb = 0; kb < kC / 8; ++kb) {
        const int j0 = kb * 8 + t4, j1 = j0 + 4;
        const float f0 = sm.fG[j0], f1 = sm.fG[j1];
        const uint32_t a0 = RoundTf32Any(sm.U[buf][j0][sm0 + g] * f0), a1 = RoundTf32Any(sm.U[buf][j0][sm0 + g + 8] * f0);
        const uint32_t a2 = RoundTf32Any(sm.U[buf][j1][sm0 + g] * f1), a3 = RoundTf32Any(sm.U[buf][j1][sm0 + g + 8] * f1);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const uint32_t b0 = RoundTf32(sm.K[j0 * kLd + sn0 + nt * 8 + g]), b1 = RoundTf32(sm.K[j1 * kLd + sn0 + nt * 8 + g]);
          MmaTf32(st[nt], a0, a1, a2, a3, b0, b1);
        }
      }
      publish();
    }
  }
  __pipeline_wait_prior(0);
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    *reinterpret_cast<float2*>(s_lo + nt * 8) = make_float2(st[nt][0], st[nt][1]);
    *reinterpret_cast<float2*>(s_hi + nt * 8) = make_float2(st[nt][2], st[nt][3]);
  }
}

}  // namespace

// Runs both phases on `stream`; ws must hold r4dxb_gdn_chunk_ws_floats(T, H) floats.
int LaunchGdnChunked(const float* q, const float* k, const float* v, const float* eg, const float* beta, float* state, float* o,
                     float* ws, int T, int H, int Hk, cudaStream_t s) {
  const int chunks = (T + kC - 1) / kC;
  const size_t per = static_cast<size_t>(chunks) * H * kC;
  float* ws_ut = ws;
  float* ws_w = ws_ut + per * kD;
  float* ws_p = ws_w + per * kD;
  float* ws_g = ws_p + per * kC;
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(GdnChunkPrepKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(PhaseASmem)));
    cudaFuncSetAttribute(GdnChunkScanKernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(PhaseBSmem<32>)));
    cudaFuncSetAttribute(GdnChunkScanKernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(PhaseBSmem<64>)));
    configured = true;
  }
  GdnChunkPrepKernel<<<dim3(chunks, H), 256, sizeof(PhaseASmem), s>>>(q, k, v, eg, beta, ws_ut, ws_w, ws_p, ws_g, T, H, Hk);
  int e = FinishLaunch();
  if (e) return e;
  // A CTA has an SM to itself.  32 state rows halve its four products and double the copies, so they pay while all CTAs of a
  // launch run at once (4 H <= 148); with more heads the second half of them would wait for the first.
  if (4 * H <= 148)
    GdnChunkScanKernel<32><<<dim3(H, kD / 32), 32 * 8, sizeof(PhaseBSmem<32>), s>>>(q, k, ws_ut, ws_w, ws_p, ws_g, state, o, T, H, Hk);
  else
    GdnChunkScanKernel<64><<<dim3(H, kD / 64), 64 * 8, sizeof(PhaseBSmem<64>), s>>>(q, k, ws_ut, ws_w, ws_p, ws_g, state, o, T, H, Hk);
  return FinishLaunch();
}

}  // namespace r4dxb

extern "C" {

/* fp32 workspace of the chunked GDN prefill for T tokens and H value heads (D = 128) */
long long r4dxb_gdn_chunk_ws_floats(int T, int H) {
  const long long chunks = (T + r4dxb::kC - 1) / r4dxb::kC;
  return chunks * H * r4dxb::kC * (2LL * r4dxb::kD + r4dxb::kC + 1);
}

}  // extern "C"
