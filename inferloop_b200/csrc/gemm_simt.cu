// out[M,N] (+)= A[M,K] * W[N,K]^T (+ bias[N]) on the ordinary 32-bit pipes.
//
// This is the exact path: every product and sum is an IEEE 32-bit operation, no tensor-core
// mode is involved.  Each output element is summed the same way whatever the tile shape, so a
// row of A gives bit-identical results whatever other rows share the launch: blocks of 16
// consecutive k are each one chain of fused multiply-adds from zero, and the block sums are
// added in increasing order with the rounding error of every addition carried along in a
// second 32-bit word (Knuth's two-sum) and added at the end.  A plain chain over K = 12288
// terms loses about sqrt(K) units in the last place; this one stays near sqrt(16).
// With bfloat16 inputs it doubles as the any-shape fallback of the bfloat16 path.
//
// Reference formula: y = W x, weights stored [out, in]
// (crates/testing/cpu/reference-ops/src/kernels.rs:168-183).
#include <type_traits>
#include "common.cuh"

using namespace ilb;

template <typename TA, typename TO, int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_simt_kernel(const TA* __restrict__ A, const TA* __restrict__ W,
                 const float* __restrict__ bias, TO* __restrict__ out, int M, int N, int K,
                 int lda, int ldw, int ldo, int accumulate, const int* __restrict__ block_group, long long group_stride) {
  ilb::pdl_launch_dependents();
  ilb::pdl_wait();
  if (block_group != nullptr) {                      // this block of rows multiplies its own group's matrix
    const int g = block_group[blockIdx.y];
    if (g < 0) return;
    W += (size_t)g * group_stride;
  }
  constexpr int BK = 16;
  constexpr int THREADS = (BM / TM) * (BN / TN);
  __shared__ float As[BK][BM + 1];
  __shared__ float Ws[BK][BN + 1];
  const int tid = threadIdx.x;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN], lost[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) { acc[i][j] = 0.f; lost[i][j] = 0.f; }

  for (int k0 = 0; k0 < K; k0 += BK) {
    for (int idx = tid; idx < BM * BK; idx += THREADS) {
      const int m = idx / BK, k = idx % BK;
      const int gm = m0 + m, gk = k0 + k;
      As[k][m] = (gm < M && gk < K) ? to_float(A[(size_t)gm * lda + gk]) : 0.f;
    }
    for (int idx = tid; idx < BN * BK; idx += THREADS) {
      const int n = idx / BK, k = idx % BK;
      const int gn = n0 + n, gk = k0 + k;
      Ws[k][n] = (gn < N && gk < K) ? to_float(W[(size_t)gn * ldw + gk]) : 0.f;
    }
    __syncthreads();
    const int kmax = (K - k0) < BK ? (K - k0) : BK;
    float part[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) part[i][j] = 0.f;
    for (int kk = 0; kk < kmax; ++kk) {
      float a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = Ws[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) part[i][j] = fmaf(a[i], w[j], part[i][j]);
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float s = __fadd_rn(acc[i][j], part[i][j]);
        const float bp = __fsub_rn(s, acc[i][j]);
        lost[i][j] = __fadd_rn(lost[i][j], __fadd_rn(__fsub_rn(acc[i][j], __fsub_rn(s, bp)), __fsub_rn(part[i][j], bp)));
        acc[i][j] = s;
      }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty * TM + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx * TN + j;
      if (gn >= N) continue;
      float v = __fadd_rn(acc[i][j], lost[i][j]);
      if (bias != nullptr) v += bias[gn];
      TO* o = out + (size_t)gm * ldo + gn;
      if (accumulate) v = to_float(*o) + v;
      *o = from_float<TO>(v);
    }
  }
}

// The same sums, faster: operands come in 16-byte pieces (four consecutive k of a row), the
// next PF K blocks are already in registers (or on their way) while one is multiplied, and
// shared memory is double-buffered (one barrier per block of 16).  Two shapes: 16 x 64 for up to 16 rows of
// bfloat16 and rows dealt to groups (the order of the sums forbids cutting K among CTAs, so the bytes in
// flight are all the parallelism there is: eight blocks ahead), and 128 x 128 where `big_tiles`
// says so.  A thread's rows and columns are strided
// (row ty + i * BM/TM, column tx + j * BN/TN), so a warp reads consecutive words.  Every output is
// still the same chains of 16 and the same compensated sum in k order as in the kernel above:
// bit for bit the same result (a zero-padded tail adds +0 to a chain).  Needs K and the leading
// dimensions multiples of 4 and 16-byte (bfloat16: 8-byte) aligned bases; rows of A beyond M
// are not multiplied by warps that hold none (a warp is one ty when BN / TN = 32).
// The loads are ordinary ones that stay where they are written: a kernel here is resident while the launch before still writes A
// (and a W that is not settled), so these are no read-only data in the sense of __ldg, and the compiler, which may move a read of
// such data across the dependency wait, did so once in the 64 x 64 kernel.
template <typename T> struct Vec4;
template <> struct Vec4<float> {
  float4 v;
  __device__ __forceinline__ void load(const float* p) {
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  }
  __device__ __forceinline__ void zero() { v = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ void get(float (&f)[4]) const { f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w; }
};
template <> struct Vec4<__nv_bfloat16> {
  uint2 v;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) {
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  }
  __device__ __forceinline__ void zero() { v = make_uint2(0u, 0u); }
  __device__ __forceinline__ void get(float (&f)[4]) const {
    f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xFFFF0000u);
    f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xFFFF0000u);
  }
};

template <typename TA, typename TO, int BM, int BN, int TM, int TN, int PF>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_simt_fast_kernel(const TA* __restrict__ A, const TA* __restrict__ W,
                      const float* __restrict__ bias, TO* __restrict__ out, int M, int N, int K,
                      int lda, int ldw, int ldo, int accumulate, const int* __restrict__ block_group, long long group_stride) {
  ilb::pdl_launch_dependents();
  ilb::pdl_wait();
  if (block_group != nullptr) {                      // this block of rows multiplies its own group's matrix
    const int g = block_group[blockIdx.y];
    if (g < 0) return;
    W += (size_t)g * group_stride;
  }
  constexpr int BK = 16;                             // K block; PF blocks are held in registers ahead of the one in shared memory
  static_assert(PF % 2 == 0, "the shared-memory buffer of a block follows from its register slot");
  constexpr int THREADS = (BM / TM) * (BN / TN);
  constexpr int XS = BN / TN, YS = BM / TM;          // strides of a thread's columns and rows
  constexpr int VA = (BM * 4 + THREADS - 1) / THREADS, VW = (BN * 4 + THREADS - 1) / THREADS;   // 4-element pieces per thread and block
  __shared__ float As[2][BK][BM + 1];
  __shared__ float Ws[2][BK][BN + 1];
  const int tid = threadIdx.x;
  const int tx = tid % XS, ty = tid / XS;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const bool has_rows = m0 + ty < M;                 // (rows ty + i * YS: if the first is outside, all are)
  float acc[TM][TN], lost[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) { acc[i][j] = 0.f; lost[i][j] = 0.f; }

  Vec4<TA> ras[PF][VA], rws[PF][VW];                 // (slots are only ever indexed by constants: see the unrolled loop below)
  auto fetch_into = [&](Vec4<TA> (&ra)[VA], Vec4<TA> (&rw)[VW], int k0) {
#pragma unroll
    for (int i = 0; i < VA; ++i) {
      const int v = tid + i * THREADS, row = v >> 2, k = k0 + (v & 3) * 4;
      if (v < BM * 4 && m0 + row < M && k < K) ra[i].load(A + (size_t)(m0 + row) * lda + k); else ra[i].zero();
    }
#pragma unroll
    for (int i = 0; i < VW; ++i) {
      const int v = tid + i * THREADS, row = v >> 2, k = k0 + (v & 3) * 4;
      if (v < BN * 4 && n0 + row < N && k < K) rw[i].load(W + (size_t)(n0 + row) * ldw + k); else rw[i].zero();
    }
  };
  auto stash_from = [&](const Vec4<TA> (&ra)[VA], const Vec4<TA> (&rw)[VW], int buf) {   // into shared memory, transposed
#pragma unroll
    for (int i = 0; i < VA; ++i) {
      const int v = tid + i * THREADS, row = v >> 2, k = (v & 3) * 4;
      if (v < BM * 4) {
        float f[4];
        ra[i].get(f);
#pragma unroll
        for (int j = 0; j < 4; ++j) As[buf][k + j][row] = f[j];
      }
    }
#pragma unroll
    for (int i = 0; i < VW; ++i) {
      const int v = tid + i * THREADS, row = v >> 2, k = (v & 3) * 4;
      if (v < BN * 4) {
        float f[4];
        rw[i].get(f);
#pragma unroll
        for (int j = 0; j < 4; ++j) Ws[buf][k + j][row] = f[j];
      }
    }
  };
  const int blocks = (K + BK - 1) / BK;
#pragma unroll
  for (int s = 0; s < PF; ++s)
    if (s < blocks) fetch_into(ras[s], rws[s], s * BK);
  stash_from(ras[0], rws[0], 0);
  __syncthreads();
  for (int b0 = 0; b0 < blocks; b0 += PF) {
#pragma unroll
   for (int s = 0; s < PF; ++s) {
    const int b = b0 + s;
    if (b >= blocks) break;
    const int buf = s & 1;                                         // = b & 1: b0 is a multiple of the even PF
    // block b is in shared memory and its slot s is free: block b + PF is requested into it
    if (b + PF < blocks) fetch_into(ras[s], rws[s], (b + PF) * BK);
    if (has_rows) {
      float part[TM][TN];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) part[i][j] = 0.f;
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) {
        float a[TM], w[TN];
#pragma unroll
        for (int i = 0; i < TM; ++i) a[i] = As[buf][kk][ty + i * YS];
#pragma unroll
        for (int j = 0; j < TN; ++j) w[j] = Ws[buf][kk][tx + j * XS];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) part[i][j] = fmaf(a[i], w[j], part[i][j]);
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const float s = __fadd_rn(acc[i][j], part[i][j]);
          const float bp = __fsub_rn(s, acc[i][j]);
          lost[i][j] = __fadd_rn(lost[i][j], __fadd_rn(__fsub_rn(acc[i][j], __fsub_rn(s, bp)), __fsub_rn(part[i][j], bp)));
          acc[i][j] = s;
        }
    }
    if (b + 1 < blocks) stash_from(ras[(s + 1) % PF], rws[(s + 1) % PF], buf ^ 1);   // block b + 1 into the other buffer (nobody reads it now)
    __syncthreads();
   }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty + i * YS;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx + j * XS;
      if (gn >= N) continue;
      float v = __fadd_rn(acc[i][j], lost[i][j]);
      if (bias != nullptr) v += bias[gn];
      TO* o = out + (size_t)gm * ldo + gn;
      if (accumulate) v = to_float(*o) + v;
      *o = from_float<TO>(v);
    }
  }
}

// The same sums again for a handful of tokens of 32-bit operands (in groups of 8), as a stream of weights.  Bound: HBM (a weight is
// read once and multiplied M times; 2 M + 7 M / 16 operations for 4 bytes).  The kernels above give a thread whole outputs, so
// K is a serial chain of barriers for one 64-column CTA; here the blocks of 16 k of one row go to the 32 lanes of a warp
// (lane l chains block l of 512 consecutive k), and the block sums then pass through shared memory to one lane per output,
// which adds them in k order with the same compensated sum: bit for bit the results above.  A warp has R rows of W, so a
// piece of A read from shared memory serves R products.  Operands come by cp.async, whole lines at a time, 512 k a stage, one
// stage ahead of the one that is multiplied (two buffers); blocks of 16 floats lie 20 floats apart, so eight lanes' 16-byte reads
// (one block each) touch all 32 banks once.
// Measured (4 layers of the 8B sizes with the output matrix, 4 tokens, one decode step): 7.3 -> 1.9 ms, of which the weights
// alone take 0.85 ms at the measured copy rate.
constexpr int kFewK = 512;                           // k of a stage: a block of 16 for every lane
constexpr int kFewPitch = 20;                        // floats from one block of 16 to the next in shared memory
constexpr int kFewRow = (kFewK / 16) * kFewPitch;    // floats of a staged row
constexpr int kFewWarps = 4;

constexpr size_t few_smem(int T, int R) {
  return sizeof(float) * ((size_t)2 * (T + kFewWarps * R) * kFewRow + (size_t)kFewWarps * 32 * (R * T + 1));
}

template <typename TO, int T, int R, bool kSettled>
__global__ void __launch_bounds__(kFewWarps * 32)
gemm_simt_few_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                     TO* __restrict__ out, int M, int N, int K, int lda, int ldw, int ldo, int accumulate) {
  static_assert(T * R <= 32, "one lane adds up one output");
  extern __shared__ __align__(16) float few[];
  float* As = few;                                   // [2][T][kFewRow]
  float* Ws = As + 2 * T * kFewRow;                  // [2][kFewWarps * R][kFewRow]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* parts = Ws + 2 * kFewWarps * R * kFewRow + warp * 32 * (R * T + 1);     // [block][output], one more float between blocks
  // groups of T tokens of the same weight rows are neighbours in the grid: the rows come from memory once
  const int groups = (M + T - 1) / T, g0 = (int)(blockIdx.x % (unsigned)groups) * T;
  A += (size_t)g0 * lda; out += (size_t)g0 * ldo; M -= g0;
  const int n0 = (int)(blockIdx.x / (unsigned)groups) * (kFewWarps * R);
  // one row of 512 k: 128 pieces of 16 bytes, a warp takes 32 neighbours at a time; what lies outside is filled with zeros
  auto copy_row = [&](const float* src, bool there, float* dst, int k0, int piece) {
    const int k = k0 + piece * 4;
    const bool on = there && k < K;
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst + (piece >> 2) * kFewPitch + (piece & 3) * 4);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(on ? src + k : src), "r"(on ? 16 : 0) : "memory");
  };
  auto fetch_w = [&](int it) {                       // a warp brings its own rows
    const int buf = it & 1, k0 = it * kFewK;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int n = n0 + warp * R + r;
      const bool there = n < N;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        copy_row(W + (size_t)(there ? n : 0) * ldw, there, Ws + (size_t)(buf * kFewWarps * R + warp * R + r) * kFewRow, k0, q * 32 + lane);
    }
  };
  auto fetch_a = [&](int it) {                       // the block shares A
    const int buf = it & 1, k0 = it * kFewK;
    for (int i = tid; i < T * 128; i += kFewWarps * 32) {
      const int t = i >> 7;
      copy_row(A + (size_t)(t < M ? t : 0) * lda, t < M, As + (size_t)(buf * T + t) * kFewRow, k0, i & 127);
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
  const int rounds = (K + kFewK - 1) / kFewK, blocks = (K + 15) / 16;
  ilb::pdl_launch_dependents();
  if constexpr (!kSettled) ilb::pdl_wait();
  fetch_w(0);
  if constexpr (kSettled) ilb::pdl_wait();
  fetch_a(0);
  commit();
  float acc = 0.f, lost = 0.f;                       // of output `lane` = r * T + t
  for (int it = 0; it < rounds; ++it) {
    if (it + 1 < rounds) { fetch_w(it + 1); fetch_a(it + 1); commit(); }
    if (it + 1 < rounds) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int buf = it & 1;
    float part[R][T];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int t = 0; t < T; ++t) part[r][t] = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float4 w[R];
#pragma unroll
      for (int r = 0; r < R; ++r)
        w[r] = *reinterpret_cast<const float4*>(Ws + (size_t)(buf * kFewWarps * R + warp * R + r) * kFewRow + lane * kFewPitch + q * 4);
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const float4 a = *reinterpret_cast<const float4*>(As + (size_t)(buf * T + t) * kFewRow + lane * kFewPitch + q * 4);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          part[r][t] = fmaf(a.x, w[r].x, part[r][t]);
          part[r][t] = fmaf(a.y, w[r].y, part[r][t]);
          part[r][t] = fmaf(a.z, w[r].z, part[r][t]);
          part[r][t] = fmaf(a.w, w[r].w, part[r][t]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int t = 0; t < T; ++t) parts[lane * (R * T + 1) + r * T + t] = part[r][t];
    __syncwarp();
    if (lane < R * T) {
      auto add = [&](float v) {
        const float s = __fadd_rn(acc, v);
        const float bp = __fsub_rn(s, acc);
        lost = __fadd_rn(lost, __fadd_rn(__fsub_rn(acc, __fsub_rn(s, bp)), __fsub_rn(v, bp)));
        acc = s;
      };
      const int here = min(32, blocks - it * 32);
      if (here == 32) {
#pragma unroll
        for (int b = 0; b < 32; ++b) add(parts[b * (R * T + 1) + lane]);
      } else {
        for (int b = 0; b < here; ++b) add(parts[b * (R * T + 1) + lane]);
      }
    }
    __syncthreads();                                 // the stage is free for the round after next, the parts for the next
  }
  const int t = lane % T, n = n0 + warp * R + lane / T;
  if (lane < R * T && t < M && n < N) {
    float v = __fadd_rn(acc, lost);
    if (bias != nullptr) v += bias[n];
    TO* o = out + (size_t)t * ldo + n;
    if (accumulate) v = to_float(*o) + v;
    *o = from_float<TO>(v);
  }
}

template <typename TO, int T, int R, bool kSettled>
static int launch_few_tiles(const float* A, const float* W, const float* bias, void* out, int M, int N, int K, int lda, int ldw,
                      int ldo, int accumulate, cudaStream_t stream) {
  static ilb::OncePerDevice once;
  constexpr size_t smem = few_smem(T, R);
  if (once.run([] { return cudaFuncSetAttribute(gemm_simt_few_kernel<TO, T, R, kSettled>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); }) != cudaSuccess)
    return fail("gemm_simt: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(cudaGetLastError()));
  ilb::launch(gemm_simt_few_kernel<TO, T, R, kSettled>, dim3((unsigned)((N + kFewWarps * R - 1) / (kFewWarps * R) * ((M + T - 1) / T))), dim3(kFewWarps * 32), smem, stream,
              A, W, bias, (TO*)out, M, N, K, lda, ldw, ldo, accumulate);
  return check_launch("gemm_simt");
}

template <typename TO, int T, int R>
static int launch_few(const float* A, const float* W, const float* bias, void* out, int M, int N, int K, int lda, int ldw,
                      int ldo, int accumulate, int settled, cudaStream_t stream) {
  return settled ? launch_few_tiles<TO, T, R, true>(A, W, bias, out, M, N, K, lda, ldw, ldo, accumulate, stream)
                 : launch_few_tiles<TO, T, R, false>(A, W, bias, out, M, N, K, lda, ldw, ldo, accumulate, stream);
}

// The same sums for many tokens.  Bound: the 32-bit pipes (per output and block of 16 k: 16 multiply-adds and 7 operations of the
// compensated sum).  A warp has a 32 x 32 tile and a lane 8 x 4 of it, rows in fours: three 16-byte reads of shared memory for 32
// products.  Two rows go through one packed instruction (fma.rn.f32x2: each half rounds as fmaf does; a - b is fma(b, -1, a), one
// rounding like __fsub_rn), at the same rate of the pipes and half the instructions to issue.  Operands come in pieces of four k
// (16 bytes, of bfloat16 8), 32 k ahead in registers, 16 rows x 2 pieces a warp and request (whole sectors of 32-bit operands, half
// ones of bfloat16; rows of k lie 4 floats beyond a multiple of 32, so the transposed stores take different banks).  Row tiles of
// the same columns are neighbours in the grid: a weight tile comes from memory once.  One layer's products of the 8B sizes in 32
// bits, against 128 x 128 tiles of 8 x 8 (256 threads, the chains as separate instructions; for 4,096 columns 32 CTAs up to 128
// tokens, 64 at 200, 128 at 512, 256 at 1,024): 64 tokens 5.03 -> 1.64 ms, 128: 5.15 -> 2.72, 200: 5.86 -> 3.98, 512: 8.74 -> 8.00,
// 1,024: 15.9 -> 15.1; bfloat16, 4,096 x 4,096: 64 tokens 0.696 -> 0.313 ms, 200: 0.721 -> 0.386, 1,024: 1.43 -> 1.33 (where the
// large tiles stay ahead: `big_tiles`).  Measured and dropped: separate instructions here (200 tokens 4.77), three blocks an SM at
// 168 registers (4.58: the reads are no longer a step ahead), 8 x 8 a lane with 4-byte cp.async (4.59; 512 tokens 6.87).
__device__ __forceinline__ uint64_t pack2(float a, float b) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }

constexpr int kWideM = 64, kWideN = 64, kWideK = 32;

template <typename TA, typename TO, bool kSettled>
__global__ void __launch_bounds__(kWideM * kWideN / 32, 2)
gemm_simt_wide_kernel(const TA* __restrict__ A, const TA* __restrict__ W, const float* __restrict__ bias, TO* __restrict__ out,
                      int M, int N, int K, int lda, int ldw, int ldo, int accumulate) {
  constexpr int BM = kWideM, BN = kWideN, BK = kWideK;
  constexpr int WARPS = (BM / 32) * (BN / 32);
  constexpr int HALVES = BK / 8;                                   // pairs of pieces of a row
  constexpr int CA = BM / 16 * HALVES / WARPS, CW = BN / 16 * HALVES / WARPS;   // requests of 16 rows x 2 pieces a warp makes per stage
  static_assert(CA * WARPS * 16 == BM * HALVES && CW * WARPS * 16 == BN * HALVES, "requests divide evenly");
  __shared__ __align__(16) float As[2][BK][BM + 4];
  __shared__ __align__(16) float Ws[2][BK][BN + 4];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m_tiles = (M + BM - 1) / BM;
  const int m0 = (int)(blockIdx.x % (unsigned)m_tiles) * BM, n0 = (int)(blockIdx.x / (unsigned)m_tiles) * BN;
  const int r0 = (warp / (BN / 32)) * 32 + (lane >> 3) * 4;        // rows r0 .. + 3 and r0 + 16 .. + 19
  const int c0 = (warp % (BN / 32)) * 32 + (lane & 7) * 4;         // columns c0 .. + 3
  const bool has_rows = m0 + (warp / (BN / 32)) * 32 < M;
  const int frow = lane & 15, fpiece = lane >> 4;
  Vec4<TA> ra[CA], rw[CW];
  auto fetch = [&](int k0, bool with_w, bool with_a) {
#pragma unroll
    for (int i = 0; i < CW; ++i) {
      const int c = warp + i * WARPS, n = n0 + (c / HALVES) * 16 + frow, k = k0 + ((c % HALVES) * 2 + fpiece) * 4;
      if (with_w) { if (n < N && k < K) rw[i].load(W + (size_t)n * ldw + k); else rw[i].zero(); }
    }
#pragma unroll
    for (int i = 0; i < CA; ++i) {
      const int c = warp + i * WARPS, m = m0 + (c / HALVES) * 16 + frow, k = k0 + ((c % HALVES) * 2 + fpiece) * 4;
      if (with_a) { if (m < M && k < K) ra[i].load(A + (size_t)m * lda + k); else ra[i].zero(); }
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int i = 0; i < CW; ++i) {
      const int c = warp + i * WARPS, row = (c / HALVES) * 16 + frow, k = ((c % HALVES) * 2 + fpiece) * 4;
      float f[4];
      rw[i].get(f);
#pragma unroll
      for (int j = 0; j < 4; ++j) Ws[buf][k + j][row] = f[j];
    }
#pragma unroll
    for (int i = 0; i < CA; ++i) {
      const int c = warp + i * WARPS, row = (c / HALVES) * 16 + frow, k = ((c % HALVES) * 2 + fpiece) * 4;
      float f[4];
      ra[i].get(f);
#pragma unroll
      for (int j = 0; j < 4; ++j) As[buf][k + j][row] = f[j];
    }
  };
  uint64_t acc[4][4], lost[4][4];                                  // [pair of rows][column]
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = lost[i][j] = 0;
  const uint64_t minus = pack2(-1.f, -1.f);
  ilb::pdl_launch_dependents();
  if constexpr (!kSettled) ilb::pdl_wait();
  fetch(0, true, false);
  if constexpr (kSettled) ilb::pdl_wait();
  fetch(0, false, true);
  stash(0);
  __syncthreads();
  const int blocks = (K + BK - 1) / BK;
  for (int b = 0; b < blocks; ++b) {
    const int buf = b & 1;
    if (b + 1 < blocks) fetch((b + 1) * BK, true, true);
    if (has_rows) {
#pragma unroll
      for (int h = 0; h < BK; h += 16) {
        uint64_t part[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) part[i][j] = 0;
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
          const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(&As[buf][h + kk][r0]);
          const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(&As[buf][h + kk][r0 + 16]);
          const float4 w4 = *reinterpret_cast<const float4*>(&Ws[buf][h + kk][c0]);
          const uint64_t a[4] = {a0.x, a0.y, a1.x, a1.y};
          const uint64_t w[4] = {pack2(w4.x, w4.x), pack2(w4.y, w4.y), pack2(w4.z, w4.z), pack2(w4.w, w4.w)};
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) part[i][j] = fma2(a[i], w[j], part[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint64_t s = add2(acc[i][j], part[i][j]);
            const uint64_t bp = fma2(acc[i][j], minus, s);           // s - acc
            const uint64_t ea = fma2(fma2(bp, minus, s), minus, acc[i][j]);
            const uint64_t eb = fma2(bp, minus, part[i][j]);
            lost[i][j] = add2(lost[i][j], add2(ea, eb));
            acc[i][j] = s;
          }
      }
    }
    if (b + 1 < blocks) stash(buf ^ 1);                            // (read last before the barrier at the end of block b - 1)
    __syncthreads();
  }
  if (!has_rows) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float v[2][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t t = add2(acc[i][j], lost[i][j]);
      unpack2(t, v[0][j], v[1][j]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int m = m0 + r0 + (i >> 1) * 16 + (i & 1) * 2 + h;
      if (m >= M) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + c0 + j;
        if (n >= N) continue;
        float r = v[h][j];
        if (bias != nullptr) r += bias[n];
        TO* o = out + (size_t)m * ldo + n;
        if (accumulate) r = to_float(*o) + r;
        *o = from_float<TO>(r);
      }
    }
  }
}

template <typename TA, typename TO>
static int launch_wide(const TA* A, const TA* W, const float* bias, void* out, int M, int N, int K, int lda, int ldw, int ldo,
                       int accumulate, int settled, cudaStream_t stream) {
  const long long tiles = (long long)((M + kWideM - 1) / kWideM) * ((N + kWideN - 1) / kWideN);
  ILB_REQUIRE(tiles <= 2147483647LL, "gemm_simt: grid too large for M=%d N=%d", M, N);
  ilb::launch(settled ? gemm_simt_wide_kernel<TA, TO, true> : gemm_simt_wide_kernel<TA, TO, false>, dim3((unsigned)tiles), dim3(kWideM * kWideN / 32), 0, stream,
              A, W, bias, (TO*)out, M, N, K, lda, ldw, ldo, accumulate);
  return check_launch("gemm_simt");
}

// Whether many tokens take 128 x 128 tiles (the kernel of 8 x 8 outputs a thread, a CTA to an SM) and not the 64 x 64 ones above
// (two to an SM).  Both are bound by the 32-bit pipes, so the time is the rounds a launch takes: counted in rounds of the small
// tiles (372 us at K = 4,096), a round of big ones takes 1.957 with 32-bit operands and 1.9 with bfloat16, 0.06 more once for
// its fill, and a last round with one small tile to an SM at most takes 0.6.  Measured, big / small tiles, us: bfloat16 512 x
// 4,096 x 4,096 735 / 762, 1,024 x 4,096 1,425 / 1,334, 1,024 x 24,576 7,614 / 7,818, 2,048 x 24,576 14,872 / 15,574, 200 x 6,144
// 729 / 582; 32 bits 512 x 4,096 759 / 760, 1,024 x 4,096 1,473 / 1,333, 2,048 x 6,144 4,314 / 3,958, 2,048 x 24,576 15,297 / 15,643.
constexpr int kSms = 148;
static bool big_tiles(int M, int N, bool wide_operands) {
  const long long small = (long long)((M + kWideM - 1) / kWideM) * ((N + kWideN - 1) / kWideN);
  const long long big = (long long)((M + 127) / 128) * ((N + 127) / 128);
  const long long rest = small % (2 * kSms);
  const long long t_small = small / (2 * kSms) * 1000 + (rest == 0 ? 0 : rest <= kSms ? 600 : 1000);
  const long long t_big = (big + kSms - 1) / kSms * (wide_operands ? 1957 : 1900) + 60;
  return t_big < t_small;
}

template <typename TA, typename TO>
static int launch(const void* A, const void* W, const float* bias, void* out, int M, int N, int K,
                  int lda, int ldw, int ldo, int accumulate, int settled, cudaStream_t stream,
                  const int* block_group = nullptr, long long group_stride = 0) {
  const bool pieces = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
                      (uintptr_t)A % (4 * sizeof(TA)) == 0 && (uintptr_t)W % (4 * sizeof(TA)) == 0;
  const bool grouped = block_group != nullptr;       // groups are dealt in blocks of kGroupRows rows: the 16-row tiles
  if constexpr (std::is_same<TA, float>::value) {
    // 16-byte pieces for cp.async; a lane adds up one output, so rows a warp x tokens <= 32.  The arithmetic grows with every
    // group of 8 tokens: one layer of the 8B sizes, this kernel against the tiles below: 24 tokens 0.86 / 1.31 ms, 40 tokens
    // 1.42 / 1.56, 64 tokens 2.27 / 1.64.  That is the line at layers of that width; the wider an output, the earlier the tiles
    // win (40 tokens here / 41 there, us: 24,576 x 4,096 663 / 522, 6,144 x 4,096 169 / 313, 1,024 x 4,096 39 / 199, 8 x 4,096 11 / 174).
    if (pieces && !grouped && M <= 40) {
      const float* a = (const float*)A;
      const float* w = (const float*)W;
      if (M == 1) return launch_few<TO, 1, 4>(a, w, bias, out, M, N, K, lda, ldw, ldo, accumulate, settled, stream);
      if (M == 2) return launch_few<TO, 2, 4>(a, w, bias, out, M, N, K, lda, ldw, ldo, accumulate, settled, stream);
      if (M <= 4) return launch_few<TO, 4, 4>(a, w, bias, out, M, N, K, lda, ldw, ldo, accumulate, settled, stream);
      return launch_few<TO, 8, 4>(a, w, bias, out, M, N, K, lda, ldw, ldo, accumulate, settled, stream);
    }
  }
  if (pieces && (M <= 16 || grouped)) {
    constexpr int BM = 16, BN = 64, TM = 4, TN = 2;            // 4 warps, one per group of rows ty, ty + 4, ty + 8, ty + 12
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    ilb::launch(gemm_simt_fast_kernel<TA, TO, BM, BN, TM, TN, 8>, dim3(grid), dim3((BM / TM) * (BN / TN)), 0, stream,
        (const TA*)A, (const TA*)W, bias, (TO*)out, M, N, K, lda, ldw, ldo, accumulate, block_group, group_stride);
  } else if (pieces && big_tiles(M, N, sizeof(TA) == 4)) {
    constexpr int BM = 128, BN = 128, TM = 8, TN = 8;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    ilb::launch(gemm_simt_fast_kernel<TA, TO, BM, BN, TM, TN, 2>, dim3(grid), dim3((BM / TM) * (BN / TN)), 0, stream,
        (const TA*)A, (const TA*)W, bias, (TO*)out, M, N, K, lda, ldw, ldo, accumulate, block_group, group_stride);
  } else if (pieces) {
    return launch_wide<TA, TO>((const TA*)A, (const TA*)W, bias, out, M, N, K, lda, ldw, ldo, accumulate, settled, stream);
  } else if (M <= 16 || grouped) {
    constexpr int BM = 16, BN = 32, TM = 2, TN = 2;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    ilb::launch(gemm_simt_kernel<TA, TO, BM, BN, TM, TN>, dim3(grid), dim3((BM / TM) * (BN / TN)), 0, stream, 
        (const TA*)A, (const TA*)W, bias, (TO*)out, M, N, K, lda, ldw, ldo, accumulate, block_group, group_stride);
  } else {
    constexpr int BM = 64, BN = 64, TM = 4, TN = 4;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    ilb::launch(gemm_simt_kernel<TA, TO, BM, BN, TM, TN>, dim3(grid), dim3((BM / TM) * (BN / TN)), 0, stream, 
        (const TA*)A, (const TA*)W, bias, (TO*)out, M, N, K, lda, ldw, ldo, accumulate, block_group, group_stride);
  }
  return check_launch("gemm_simt");
}

// in_dtype: element type of A and W; out_dtype: element type of out.
// accumulate != 0 adds the product (and bias) to what `out` already holds.
// `settled`: no launch that this one may overlap writes W: the kernels for 32-bit operands of few tokens and for many tokens ask
// for its first rows ahead of the dependency wait (small products: 1.3 against 1.6 us launch after launch).
ILB_EXPORT int ilb_gemm_simt(const void* A, const void* W, const float* bias, void* out,
                             int in_dtype, int out_dtype, int M, int N, int K, int lda, int ldw,
                             int ldo, int accumulate, int settled, cudaStream_t stream) {
  ILB_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_simt: bad sizes M=%d N=%d K=%d", M, N, K);
  ILB_REQUIRE(lda >= K && ldw >= K && ldo >= N, "gemm_simt: leading dimensions too small");
  ILB_REQUIRE((long long)((N + 31) / 32) <= 2147483647LL && (M + 15) / 16 <= 65535,
              "gemm_simt: grid too large for M=%d", M);
  if (M == 0) return 0;
  if (in_dtype == kF32 && out_dtype == kF32)
    return launch<float, float>(A, W, bias, out, M, N, K, lda, ldw, ldo, accumulate, settled, stream);
  if (in_dtype == kBF16 && out_dtype == kF32)
    return launch<__nv_bfloat16, float>(A, W, bias, out, M, N, K, lda, ldw, ldo, accumulate, settled, stream);
  if (in_dtype == kBF16 && out_dtype == kBF16)
    return launch<__nv_bfloat16, __nv_bfloat16>(A, W, bias, out, M, N, K, lda, ldw, ldo, accumulate, settled, stream);
  return fail("gemm_simt: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
}

// Rows and columns of a tile of the kernel that a product of many tokens on 16-byte (bfloat16: 8-byte) boundaries takes, 64 or 128 (for tests and notes).
ILB_EXPORT int ilb_gemm_simt_tile(int M, int N, int in_dtype) { return big_tiles(M, N, in_dtype == kF32) ? 128 : kWideM; }

// The same product for rows that are dealt to groups in blocks of 16 (ilb_gemm_simt_group_rows):
// block b of A (rows 16 b .. 16 b + 15) is multiplied by the matrix W + block_group[b] *
// group_stride elements, and left alone when block_group[b] < 0.  M is the number of rows that
// the blocks cover.  This is how a routed feed-forward runs its experts over rows sorted by expert.
ILB_EXPORT int ilb_gemm_simt_group_rows() { return 16; }

ILB_EXPORT int ilb_gemm_simt_grouped(const void* A, const void* W, void* out, int in_dtype, int out_dtype, int M, int N,
                                     int K, int lda, int ldw, int ldo, const int* block_group, long long group_stride,
                                     cudaStream_t stream) {
  ILB_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_simt_grouped: bad sizes M=%d N=%d K=%d", M, N, K);
  ILB_REQUIRE(lda >= K && ldw >= K && ldo >= N, "gemm_simt_grouped: leading dimensions too small");
  ILB_REQUIRE(block_group != nullptr && group_stride >= 0, "gemm_simt_grouped: needs the group of every block of rows");
  ILB_REQUIRE(M % 16 == 0 && M / 16 <= 65535, "gemm_simt_grouped: rows must come in blocks of 16 (at most 65535 blocks), found M=%d", M);
  if (M == 0) return 0;
  if (in_dtype == kF32 && out_dtype == kF32)
    return launch<float, float>(A, W, nullptr, out, M, N, K, lda, ldw, ldo, 0, 0, stream, block_group, group_stride);
  if (in_dtype == kBF16 && out_dtype == kF32)
    return launch<__nv_bfloat16, float>(A, W, nullptr, out, M, N, K, lda, ldw, ldo, 0, 0, stream, block_group, group_stride);
  if (in_dtype == kBF16 && out_dtype == kBF16)
    return launch<__nv_bfloat16, __nv_bfloat16>(A, W, nullptr, out, M, N, K, lda, ldw, ldo, 0, 0, stream, block_group, group_stride);
  return fail("gemm_simt_grouped: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
}

ILB_DEFINE_LAST_ERROR()
