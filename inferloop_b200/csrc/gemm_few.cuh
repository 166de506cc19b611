// bfloat16 products of up to 128 tokens, included by gemm_tcgen05.cu (whose helpers it uses):
//     out[T, N] (+)= A[T, K] * W[N, K]^T (+ bias), or the gated unit over interleaved gate and up rows.
//
// What bounds it: the weight is read once, so the floor is its bytes at the copy rate.  Three things kept the
// former deal (128 weight rows on the MMA's rows, one or two tiles to an SM) away from it: tiles of one height
// leave a quarter to a half of the SMs with half the work of the others (24,576 rows are 192 tiles of 128 for
// 148 SMs), the tokens' operand is fetched again for every tile, and many tokens leave a shallow ring.  Here the
// tokens are the MMA's rows (64 of them, or 128; a tile's operand A block holds the real tokens only, the MMA
// reads on into the weight block behind it and the rows that come of it are nobody's) and the weight rows its
// columns, so that a tile may be any multiple of 16 rows up to 256.  `few_plan` picks the height for which the CTAs, two to an
// SM, come out even; into how many K ranges a sum is cut belongs to the weight (`few_ranges`), unless the ranges meet in
// memory.  Launch after launch on rotating weights (us; former deal -> this one; in brackets the weight's bytes at 6.54 TB/s,
// the rate of a copy, which reads and writes: reads alone have reached 7.1): 24,576 x 4,096 gated, 8 tokens 34.8 -> 32.4
// (30.8), 64 tokens 43.8 -> 34.6, 128 tokens 54.1 -> 39.6; 51,200 x 5,120 gated, 1 token 83.6 -> 76.4 (80.2), 96 tokens
// 129.6 -> 83.4; 5,120 x 17,408 adding, 8 tokens 30.0 -> 28.6 (27.3), 24 tokens 33.7 -> 31.0, 64 tokens 39.5 -> 33.6;
// 6,144 x 4,096, 8 tokens 11.9 -> 11.6 (7.7), 96 tokens 22.1 -> 15.2; 10,240 x 5,120, 64 tokens 27.8 -> 22.6 (16.0).
// Over 29 weights at 19 token counts 0.81 of the time; 20 of the 551 take 1 to 4 % longer.
//
// Per CTA (320 threads):
//   warp 0     requests the weight blocks by TMA (128-byte swizzle; one box a block, or for gated weights boxes of up to 128 rows in
//              which eight gate rows and their eight up rows alternate, so that a tile need not be whole blocks of 64; boxes of 16
//              rows cost small weights: 6,144 x 1,024 at 24 tokens 7.05 -> 6.35 us) into a ring of `stages` buffers, the first ring before the kernel waits for its
//              predecessor; one lane requests the token blocks behind the wait;
//   warp 1     tensor memory; one lane issues tcgen05.mma, four to a K block of 64;
//   warps 2-9  the write-out.  With one K range, or ranges that meet in memory (red.add), the tile goes through the
//              idle ring so that a thread holds four neighbouring outputs; the ranges of a tile that must be added
//              in K order are the CTAs of a cluster, chunk j of 16 columns belonging to CTA j % split.  They send each
//              other their shares (st.async on the owner's mbarrier); where the area for these would leave too little
//              ring (LATE), each parks its share in its idle ring and the owners fetch, between two cluster barriers.
// (Tried and taken back: the RMS norm in front of a product of up to 16 tokens inside it, warps 2-9 reading the 32-bit rows, laying
// them out ahead of the stream and leaving the root mean square to the result.  Launch after launch it took 0.3 to 0.8 us where the
// norm's launch takes 1.7; in a step, where that launch hides behind its neighbours, 8B sizes lost 3 % at one token.)
// All mbarrier waits are bounded, as in the other kernels.  One that runs out raises the error flag and nothing else: every thread goes on to
// the end as if it had not (what it writes is flagged as invalid), so that no other one waits at a barrier that it left out and
// every share that a peer counts is sent; warp 0 then stays until what it has requested from memory has landed.

constexpr int kFewTokens = 128;
constexpr int kFewWarps = 8, kFewEpi = 32 * kFewWarps, kFewThreads = 64 + kFewEpi;
constexpr int kFewStages = 12;
// Two CTAs to an SM: 228 KB less 1 KB each that the system keeps, halved.
constexpr int kFewSmem = 112 * 1024;
// ... and never a third, however short the ring: a CTA holds up to 256 of an SM's 512 columns of tensor memory while it waits for the
// others of its cluster, and tcgen05.alloc waits without a limit, so two clusters could each hold what the other one needs.
// (Their registers, 76 to 94 of 320 threads, leave no room for a third either; that is the compiler's choice.)
constexpr int kFewLeast = 77 * 1024;
static_assert(3 * (kFewLeast + 1024) > 228 * 1024 && 2 * (kFewSmem + 1024) <= 228 * 1024, "two CTAs to an SM");

struct FewParams {
  void* out;
  const float* bias;
  int* error_flag;
  int T, N, K, ldo;
  int rows, tp, k_blocks, split, cluster, stages, tmem_cols, red, groups;
  int stage_bytes, ring_bytes, recv_bytes;
  int epilogue, out_f32, relu2, gate_relu;
  float act_limit, act_sharp, act_offset;
};

// MM: rows of the MMA, 64 or 128.  LATE: the shares of a cluster are parked and fetched, not sent.
template <int MM, bool LATE>
__global__ void __launch_bounds__(kFewThreads, 2)
gemm_few_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_y, const FewParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - smem_u32(smem_raw));
  float* recv = reinterpret_cast<float*>(smem + (LATE ? 0 : p.ring_bytes));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + p.ring_bytes + p.recv_bytes);
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * kFewStages, tfull = empty0 + 8 * kFewStages, rbar = tfull + 8;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * kFewStages + 2);
  volatile int* failed = reinterpret_cast<volatile int*>(bars + 2 * kFewStages + 3);

  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / p.split, part = blockIdx.x - tile * p.split;
  const int kb0 = (int)((long long)p.k_blocks * part / p.split), cnt = (int)((long long)p.k_blocks * (part + 1) / p.split) - kb0;
  const bool gated = p.epilogue == kSwiGLU;
  const int row0 = tile * p.rows;
  const int n_early = cnt < p.stages ? cnt : p.stages;
  const uint32_t w_off = (uint32_t)p.tp * 128u;
  const uint32_t tx = (uint32_t)(p.rows + p.tp) * 128u;
  const int boxes = gated ? p.rows / (16 * p.groups) : 1;
  auto load_w = [&](uint32_t dst, uint32_t bar, int kcol) {
    if (gated) {
      if (lane < boxes) {
        const int g = row0 / 16 + lane * p.groups;
        tma_load_5d(dst + w_off + (uint32_t)(lane * p.groups) * 2048u, &map_w, bar, kcol, 0, 0, g & 7, g >> 3);
      }
    } else if (lane == 0) {
      tma_load_2d(dst + w_off, &map_w, bar, kcol, row0);
    }
  };

  if (warp == 0) {
    if (lane == 0) {
      for (int s = 0; s < p.stages; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
      mbar_init(tfull, 1);
      if (p.cluster > 1 && !LATE) mbar_init(rbar, 1);
      *failed = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      if (p.cluster > 1 && !LATE) {
        const int nch = p.rows / 16, me = part;
        const int nloc = (nch - me + p.split - 1) / p.split;
        mbar_expect_tx(rbar, (uint32_t)(p.split * nloc * p.T * 64));
      }
      for (int it = 0; it < n_early; ++it) mbar_expect_tx(full0 + 8 * it, tx);
    }
    __syncwarp();
    for (int it = 0; it < n_early; ++it) load_w(base + it * p.stage_bytes, full0 + 8 * it, (kb0 + it) * kBlockK);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(p.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  if (p.cluster > 1) cluster_sync_all(); else __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = *tmem_slot;

  int armed = 0;                           // warp 0: blocks requested
  if (warp == 0) {
    bool ok = true;
    pdl_wait();
    if (lane == 0)
      for (int it = 0; it < n_early; ++it) tma_load_2d(base + it * p.stage_bytes, &map_y, full0 + 8 * it, (kb0 + it) * kBlockK, 0);
    int s = n_early == p.stages ? 0 : n_early;
    uint32_t ph = 0;
    armed = n_early;
    for (int it = n_early; it < cnt; ++it) {
      ok = mbar_wait(empty0 + 8 * s, ph);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      const uint32_t dst = base + s * p.stage_bytes;
      if (lane == 0) {
        mbar_expect_tx(full0 + 8 * s, tx);
        tma_load_2d(dst, &map_y, full0 + 8 * s, (kb0 + it) * kBlockK, 0);
      }
      __syncwarp();
      load_w(dst, full0 + 8 * s, (kb0 + it) * kBlockK);
      armed = it + 1;
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
    if (!ok && lane == 0) { *failed = 1; if (p.error_flag) *p.error_flag = 1; }
    __syncwarp();
    if (LATE) { cluster_sync_all(); cluster_sync_all(); }       // with the warps of the write-out
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.rows >> 3) << 17) | ((uint32_t)(MM >> 4) << 24);
      bool ok = true;
      int s = 0;
      uint32_t ph = 0;
      for (int it = 0; it < cnt; ++it) {
        ok = mbar_wait(full0 + 8 * s, ph);
        if (!ok) break;
        tcgen05_fence_after();
        const uint32_t a = base + s * p.stage_bytes;
        const uint64_t da = smem_desc(a), db = smem_desc(a + w_off);
#pragma unroll
        for (int k = 0; k < kBlockK / 16; ++k) mma_bf16(tmem, da + 2 * k, db + 2 * k, idesc, (it > 0 || k > 0) ? 1u : 0u);
        tcgen05_commit(empty0 + 8 * s);
        if (++s == p.stages) { s = 0; ph ^= 1; }
      }
      if (!ok) { *failed = 1; if (p.error_flag) *p.error_flag = 1; }
      tcgen05_commit(tfull);
    }
    __syncwarp();
    if (LATE) { cluster_sync_all(); cluster_sync_all(); }       // with the warps of the write-out
  } else {
    const int et = threadIdx.x - 64, ew = warp - 2;
    pdl_wait();
    const int quad = warp & 3, hf = ew >> 2;
    const int t = MM == 128 ? quad * 32 + lane : quad * 16 + lane;
    const bool warp_on = (MM == 128 ? quad * 32 : quad * 16) < p.T;
    const bool mine = t < p.T && (MM == 128 || lane < 16);
    const int nch = p.rows / 16;
    if (!mbar_wait(tfull, 0)) { *failed = 1; if (p.error_flag) *p.error_flag = 1; }
    __syncwarp();
    tcgen05_fence_after();
    const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16);
    if (LATE || p.cluster > 1) {
      // ---- the K ranges of a tile are the CTAs of a cluster: chunk j of 16 columns belongs to CTA j % split
      // A chunk is [four columns][token][4], tokens swizzled by the column: a warp's stores are whole lines of 128 bytes, and a quarter
      // warp that reads four columns of two tokens meets no bank twice.
      const uint32_t recv_addr = smem_u32(recv), plane = (uint32_t)p.tp * 16u;
      if (warp_on) {
        for (int j = hf; j < nch; j += 2) {
          float v[32];
          tmem_load_16(taddr + j * 16, v);
          if (mine) {
            const uint32_t owner = (uint32_t)(j % p.split);
            const uint32_t nl = (uint32_t)((nch - (int)owner + p.split - 1) / p.split);
            const uint32_t dst = LATE ? 0u : peer_addr(recv_addr + ((uint32_t)part * nl + (uint32_t)(j / p.split)) * 4u * plane, owner);
            const uint32_t bar = LATE ? 0u : peer_addr(rbar, owner);
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) {
              const uint32_t off = (uint32_t)c4 * plane + (uint32_t)(t ^ (c4 << 1)) * 16u;
              if (LATE) *reinterpret_cast<float4*>(smem + (uint32_t)j * 4u * plane + off) = make_float4(v[4 * c4], v[4 * c4 + 1], v[4 * c4 + 2], v[4 * c4 + 3]);
              else st_peer_v4(dst + off, bar, v[4 * c4], v[4 * c4 + 1], v[4 * c4 + 2], v[4 * c4 + 3]);
            }
          }
        }
      }
      __syncwarp();
      if (LATE) cluster_sync_all();
      const int nl = (nch - part + p.split - 1) / p.split;
      const bool vec = p.ldo % 4 == 0 && (uintptr_t)p.out % 16 == 0;
      bool arrived = LATE;
      const int per_shift = gated ? 1 : 2, n_end = gated ? p.N / 2 : p.N;       // units of four outputs: two or four a chunk
      for (int u0 = et; u0 < (nl * p.T) << per_shift; u0 += 2 * kFewEpi) {
        float old[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int u = u0 + i * kFewEpi;
          const int c4 = u & ((1 << per_shift) - 1), q = u >> per_shift, jl = q / p.T, tt = q - jl * p.T;
          const int n = row0 + (jl * p.split + part) * 16 + c4 * 4;
#pragma unroll
          for (int e = 0; e < 4; ++e) old[i][e] = 0.f;
          if (p.epilogue == kAccumulate && jl < nl) {
            const float* src = (const float*)p.out + (size_t)tt * p.ldo + n;
            if (vec && n + 4 <= p.N) {
              const float4 o = __ldcg(reinterpret_cast<const float4*>(src));
              old[i][0] = o.x; old[i][1] = o.y; old[i][2] = o.z; old[i][3] = o.w;
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e) if (n + e < p.N) old[i][e] = __ldcg(src + e);
            }
          }
        }
        if (!arrived) {
          if (!mbar_wait(rbar, 0)) { *failed = 1; if (p.error_flag) *p.error_flag = 1; break; }
          arrived = true;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int u = u0 + i * kFewEpi;
          const int c4 = u & ((1 << per_shift) - 1), q = u >> per_shift, jl = q / p.T, tt = q - jl * p.T;
          if (jl >= nl) continue;
          const int chunk = jl * p.split + part;
          const int n = gated ? row0 / 2 + chunk * 8 + c4 * 4 : row0 + chunk * 16 + c4 * 4;
          float a[4] = {0.f, 0.f, 0.f, 0.f}, up[4] = {0.f, 0.f, 0.f, 0.f};
          const uint32_t at = (uint32_t)c4 * plane + (uint32_t)(tt ^ (c4 << 1)) * 16u;
          const uint32_t at_up = (uint32_t)(c4 + 2) * plane + (uint32_t)(tt ^ ((c4 + 2) << 1)) * 16u;
          if (LATE) {                            // four peers' loads in flight
            for (int z0 = 0; z0 < p.split; z0 += 4) {
              float4 s4[4], u4[4];
#pragma unroll
              for (int z = 0; z < 4; ++z) {
                if (z0 + z >= p.split) break;
                const uint32_t src = peer_addr(recv_addr + (uint32_t)chunk * 4u * plane, (uint32_t)(z0 + z));
                s4[z] = ld_peer_v4(src + at);
                if (gated) u4[z] = ld_peer_v4(src + at_up);
              }
#pragma unroll
              for (int z = 0; z < 4; ++z) {
                if (z0 + z >= p.split) break;
                a[0] += s4[z].x; a[1] += s4[z].y; a[2] += s4[z].z; a[3] += s4[z].w;
                if (gated) { up[0] += u4[z].x; up[1] += u4[z].y; up[2] += u4[z].z; up[3] += u4[z].w; }
              }
            }
          } else {
            for (int z = 0; z < p.split; ++z) {
              const uint8_t* src = reinterpret_cast<const uint8_t*>(recv) + (uint32_t)(z * nl + jl) * 4u * plane;
              const float4 s4 = *reinterpret_cast<const float4*>(src + at);
              a[0] += s4.x; a[1] += s4.y; a[2] += s4.z; a[3] += s4.w;
              if (gated) {
                const float4 u4 = *reinterpret_cast<const float4*>(src + at_up);
                up[0] += u4.x; up[1] += u4.y; up[2] += u4.z; up[3] += u4.w;
              }
            }
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float b = (p.bias && n + e < n_end) ? p.bias[n + e] : 0.f;
            a[e] = gated ? gate_mul(p, a[e], up[e]) : relu2_if(p.relu2, a[e] + b + old[i][e]);
          }
          const size_t o = (size_t)tt * p.ldo + n;
          if (vec && n + 4 <= n_end) {
            if (p.out_f32) *reinterpret_cast<float4*>((float*)p.out + o) = make_float4(a[0], a[1], a[2], a[3]);
            else *reinterpret_cast<uint2*>((__nv_bfloat16*)p.out + o) = make_uint2(pack_bf16(a[0], a[1]), pack_bf16(a[2], a[3]));
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (n + e < n_end) { if (p.out_f32) ((float*)p.out)[o + e] = a[e]; else ((__nv_bfloat16*)p.out)[o + e] = __float2bfloat16_rn(a[e]); }
          }
        }
      }
      __syncwarp();
      if (LATE) cluster_sync_all();           // nobody leaves while a peer may still read its share
      else if (!arrived && !mbar_wait(rbar, 0)) { *failed = 1; if (p.error_flag) *p.error_flag = 1; }
    } else {
      // ---- the tile (or its K range) through shared memory: the ring is idle, everything in it has been consumed
      float* st = reinterpret_cast<float*>(smem);
      const int pitch = p.rows + 4;
      if (warp_on) {
        for (int j = hf; j < nch; j += 2) {
          float v[32];
          tmem_load_16(taddr + j * 16, v);
          if (mine) {
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4)
              *reinterpret_cast<float4*>(st + (size_t)t * pitch + j * 16 + c4 * 4) = make_float4(v[4 * c4], v[4 * c4 + 1], v[4 * c4 + 2], v[4 * c4 + 3]);
          }
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(kFewEpi) : "memory");
      const bool vec = p.ldo % 4 == 0 && (uintptr_t)p.out % 16 == 0;
      const int per = gated ? p.rows / 8 : p.rows / 4;       // units of four outputs a token
      const int n_end = gated ? p.N / 2 : p.N;
      for (int u = et; u < per * p.T; u += kFewEpi) {
        const int tt = u / per, f = u - tt * per;
        float a[4];
        int n;
        if (gated) {
          const float* src = st + (size_t)tt * pitch + (f >> 1) * 16 + (f & 1) * 4;
          const float4 g = *reinterpret_cast<const float4*>(src), up = *reinterpret_cast<const float4*>(src + 8);
          a[0] = gate_mul(p, g.x, up.x); a[1] = gate_mul(p, g.y, up.y);
          a[2] = gate_mul(p, g.z, up.z); a[3] = gate_mul(p, g.w, up.w);
          n = row0 / 2 + f * 4;
        } else {
          const float4 g = *reinterpret_cast<const float4*>(st + (size_t)tt * pitch + f * 4);
          a[0] = g.x; a[1] = g.y; a[2] = g.z; a[3] = g.w;
          n = row0 + f * 4;
        }
        const size_t o = (size_t)tt * p.ldo + n;
        if (p.epilogue == kAccumulate && !p.red) {
#pragma unroll
          for (int e = 0; e < 4; ++e) if (n + e < n_end) a[e] += __ldcg((const float*)p.out + o + e);
        }
        if (!gated && p.bias && (!p.red || part == 0)) {
#pragma unroll
          for (int e = 0; e < 4; ++e) a[e] += n + e < n_end ? p.bias[n + e] : 0.f;
        }
        if (p.red) {
          float* dst = (float*)p.out + o;
          if (vec && n + 4 <= n_end) {
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(a[0]), "f"(a[1]), "f"(a[2]), "f"(a[3]) : "memory");
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) if (n + e < n_end) atomicAdd(dst + e, a[e]);
          }
          continue;
        }
        if (p.relu2) {
#pragma unroll
          for (int e = 0; e < 4; ++e) a[e] = relu2_if(1, a[e]);
        }
        if (vec && n + 4 <= n_end) {
          if (p.out_f32) *reinterpret_cast<float4*>((float*)p.out + o) = make_float4(a[0], a[1], a[2], a[3]);
          else *reinterpret_cast<uint2*>((__nv_bfloat16*)p.out + o) = make_uint2(pack_bf16(a[0], a[1]), pack_bf16(a[2], a[3]));
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (n + e < n_end) { if (p.out_f32) ((float*)p.out)[o + e] = a[e]; else ((__nv_bfloat16*)p.out)[o + e] = __float2bfloat16_rn(a[e]); }
        }
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *failed)
    for (int it = armed > p.stages ? armed - p.stages : 0; it < armed; ++it) mbar_wait(full0 + 8 * (it % p.stages), (it / p.stages) & 1);
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
  }
}

// ------------------------------------------------------------------ host side
constexpr int kFewTail = (2 * kFewStages + 4) * 8;     // barriers, flags

// Groups of 16 gated rows in a box: as many as divide a tile, so that no box crosses a block of 128 rows.
int few_groups(int rows) {
  int n = 8;
  while (rows % (16 * n) != 0) n /= 2;
  return n;
}

// The interleaved weight [rows, cols]: boxes of `groups` times eight gate rows and their eight up rows, 64 deep, inside a block of 128 rows.
int make_gated_map(CUtensorMap* out, const void* ptr, int rows, int cols, int ld, int groups) {
  static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  static std::mutex mu;
  const MapKey key{ptr, rows, cols, ld, groups};
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(key);
  if (it != cache.end()) { *out = it->second; return 0; }
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail("gemm_tc: cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t ldb = (cuuint64_t)ld * 2;
  const cuuint64_t dims[5] = {(cuuint64_t)cols, 8, 2, 8, (cuuint64_t)(rows / 128)}, strides[4] = {ldb, 64 * ldb, 8 * ldb, 128 * ldb};
  const cuuint32_t box[5] = {(cuuint32_t)kBlockK, 8, 2, (cuuint32_t)groups, 1}, estr[5] = {1, 1, 1, 1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail("gemm_tc: cuTensorMapEncodeTiled failed with code %d (gated rows %d cols %d ld %d)", (int)r, rows, cols, ld);
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, *out);
  return 0;
}

template <int MM, bool LATE>
cudaError_t configure_few() {
  static OncePerDevice once;
  return once.run([] {
    const cudaError_t e = cudaFuncSetAttribute(gemm_few_kernel<MM, LATE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * kFewSmem);
    if (e == cudaSuccess)      // two CTAs share an SM only with the largest shared-memory carve-out
      cudaFuncSetAttribute(gemm_few_kernel<MM, LATE>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    return e;
  });
}

// What the deal depends on beside the sizes: SMs, and the clusters of 1 to 8 CTAs that the device holds at once with one CTA to an SM
// and with two.
struct FewDevice { int sms, one[9], two[9]; };

// An empty kernel of the same shape is asked about: the occupancy query counts one CTA to an SM for any kernel that allocates tensor
// memory.  A B200 answers 74, 33 and 15 clusters of 2, 4 and 8 with one CTA to an SM; 148, 71 and 33 with two (72 clusters of
// four did take a second round, 18 -> 26 us; 64 and 66 did not).
__global__ void __launch_bounds__(kFewThreads, 2) few_shape_kernel() {}

int few_clusters(int cluster, int smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster * 256);
  cfg.blockDim = dim3(kFewThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  int n = 0;
  cudaError_t e = cudaFuncSetAttribute(few_shape_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(few_shape_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, few_shape_kernel, &cfg);
  if (e != cudaSuccess) { cudaGetLastError(); n = 0; }
  return n;
}

FewDevice few_device() {
  constexpr int kMax = 64;
  static std::mutex mu;
  static FewDevice known[kMax] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMax) dev = 0;
  std::lock_guard<std::mutex> g(mu);
  if (known[dev].sms == 0) {
    FewDevice d{};
    if (cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || d.sms <= 0) d.sms = 148;
    for (int c = 1; c <= 8; c *= 2) { d.one[c] = few_clusters(c, 2 * kFewSmem); d.two[c] = few_clusters(c, kFewSmem); }
    known[dev] = d;
  }
  return known[dev];
}

// How a product of few tokens is dealt out.  late: the shares of a cluster are parked in the rings and fetched.
// deep: one CTA to an SM with the shared memory of two.
struct FewPlan { int rows, split, stages, cluster, late, deep, red, tiles, grid, ring, recv, smem; };    // recv: 0 when late

// Into how many K ranges a tile's sum is cut where their order is kept.  It belongs to the weight alone, so that a row's bits are the
// same whatever it is computed beside: what tiles of 128 rows allow, in ranges of equal length, of CTAs that the device
// holds at once.  0: more tiles than two CTAs to an SM, which are shared out block by block (`make_plan`).
int few_ranges(int N, int K, const FewDevice& d) {
  const long long tiles = (N + 127) / 128, kb = (K + kBlockK - 1) / kBlockK;
  if (tiles > 2ll * d.sms) return 0;
  int split = 1;
  while (split < 8 && tiles * split * 2 <= 2ll * d.sms && split * 2 <= kb) split *= 2;
  while (split > 1 && d.one[split / 2] < tiles) split /= 2;
  return split;
}

// Into how many ranges at most a product that adds into a 32-bit output cuts a tile's sum when the ranges may meet there (separate CTAs,
// red.add; the order is then not fixed); 1: it keeps the order.
int few_ranges_in_memory(int T, int N, int K, const FewDevice& d) {
  if (!g_sums_in_memory) return 1;
  if (T <= g_red_few_tokens) return N >= 2048 && K >= 2048 && few_ranges(N, K, d) > 1 ? g_red_few_split : 1;
  if (T <= 64 || N < 3072) return 1;
  const long long tiles = (N + 255) / 256, rest = tiles % d.sms;
  return rest != 0 && tiles * 12 >= d.sms && add_split(rest, (K + kBlockK - 1) / kBlockK) >= 2 ? 8 : 1;
}

// The shared memory of a plan, with as many stages as the CTAs of an SM leave room for; false when they do not fit.
bool few_memory(int T, int k_range, FewPlan& f) {
  const int most = f.deep ? 2 * kFewSmem : kFewSmem;
  const int tp = (T + 7) / 8 * 8, stage = (tp + f.rows) * 128, mm = T <= 64 ? 64 : 128;
  f.recv = f.cluster > 1 && !f.late ? f.split * ((f.rows / 16 + f.split - 1) / f.split) * tp * 64 : 0;
  const int room = most - 1024 - kFewTail - f.recv;
  f.stages = room / stage;
  if (f.stages > kFewStages) f.stages = kFewStages;
  if (f.stages > k_range) f.stages = k_range;
  if (f.stages < (k_range < 2 ? k_range : 2)) return false;
  f.ring = f.stages * stage;
  const int reach = (f.stages - 1) * stage + mm * 128;             // the MMA reads mm rows from the last stage's first
  if (reach > f.ring) f.ring = reach;
  const int staged = f.cluster == 1 ? (T * (f.rows + 4) * 4 + 15) / 16 * 16 : f.late ? f.rows * tp * 4 : 0;       // the tile on its way out
  if (staged > f.ring) f.ring = staged;
  f.smem = 1024 + f.ring + f.recv + kFewTail;                      // what the kernel lays out, in this order
  if (f.smem < kFewLeast) f.smem = kFewLeast;
  return f.smem <= most;
}

// What ranks the plans of a product (it is no time): a fit to 12,000 timed plans of 29 weights (256 to 51,200 rows, 256 to 25,600
// deep) at 18 token counts from 1 to 128.  The plan it picks is on average 1.5 % slower than the fastest that
// was timed, 22 % at worst (1,280 x 256 at 112 tokens, 5.2 against 4.3 us).  What decides is not an SM's share of the bytes
// but how long a CTA's stream is against its ring (a round trip for `stages` blocks of 64), how many MMAs are issued (four a block,
// each as long as 118 columns at least) and how many boxes a gated block is fetched in; a second CTA on some SMs leaves less
// room to the next kernel's first blocks; and the write-out costs by the value, in a cluster by what its busiest CTA adds up.
// Shares that are parked and fetched cost some us more than shares that are sent: they pay where the area for the latter would
// leave a ring of one to three stages (6,144 x 4,096 at 96 tokens 16.9 -> 15.2 us, 12,288 x 2,048 at 128 18.8 -> 15.6).
double few_cost(int T, int N, int K, bool gated, const FewPlan& f, const FewDevice& d) {
  const int kb = (K + kBlockK - 1) / kBlockK, range = (kb + f.split - 1) / f.split, sms = d.sms;
  const int per_sm = f.grid <= sms ? 1 : 2, chunks = f.rows / 16;
  const double bytes = (double)N * K * 2 / 7.0e6, ring = 2.868 * range / f.stages, tile = 1e-3 * T * f.rows;
  double t = (bytes > ring ? bytes : ring) + 0.118 * range + 0.14 * per_sm * range * (f.rows > 118 ? f.rows / 128.0 : 0.92);
  if (per_sm == 2) t += 0.551 + 2.02 * (f.grid - sms) / sms;
  if (gated) t += 0.006 * per_sm * range * (chunks / few_groups(f.rows));
  if (f.red) t += 0.952 * f.split * 4e-6 * T * N;
  else if (f.cluster > 1) {
    const double own = 1e-3 * T * 16 * f.split * ((chunks + f.split - 1) / f.split);
    t += (0.35 + 0.045 * per_sm) * tile + (0.137 + 0.125 * per_sm) * own + 0.187 * f.split + (f.late ? 5.149 + 0.081 * per_sm * tile : 0.0);
  } else t += 0.31 * tile;
  return t;
}

// `can_add`: the product adds into a 32-bit output whose rows are 16-byte multiples.  False where the kernel does not serve: more
// tokens, or a weight of more tiles than two CTAs to an SM.
bool few_plan(int T, int N, int K, bool can_add, bool gated, const FewDevice& d, FewPlan& best) {
  if (T > kFewTokens || (N + 255) / 256 > 2 * d.sms) return false;
  const int meet = can_add ? few_ranges_in_memory(T, N, K, d) : 1;
  int ranges = few_ranges(N, K, d);
  // A weight of more 128-row tiles than two CTAs to an SM: whole tiles here, but only where the adding products of its width let their
  // ranges meet in memory, so that the rows it reads differ from run to run as it is (51,200 x 5,120 gated, 8 tokens 76.7 us
  // here and 84.6 in `make_plan`'s form, 96 tokens 83.4 and 129.6).  Elsewhere it keeps that form, and so its bits, although 24
  // tokens take 91.2 us where whole tiles took 77.5.
  if (ranges == 0 && meet == 1) {
    if (few_ranges_in_memory(T, K, K, d) == 1) return false;
    ranges = 1;
  }
  struct Key { long long a, b, c; bool operator==(const Key& o) const { return a == o.a && b == o.b && c == o.c; } };
  struct Hash { size_t operator()(const Key& k) const { return std::hash<long long>()((k.a * 1000003ll ^ k.b) * 1000003ll ^ k.c); } };
  static std::unordered_map<Key, FewPlan, Hash> cache;
  static std::mutex mu;
  const Key key{((long long)T << 32) | (unsigned)N, ((long long)K << 16) | (gated ? 1 << 12 : 0) | (meet << 8) | ranges,
                ((((long long)d.sms << 10 | d.two[2]) << 10 | d.two[4]) << 10 | d.two[8])};        // all that a plan asks of the device
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(key);
  if (it != cache.end()) { best = it->second; return best.rows > 0; }
  const int kb = (K + kBlockK - 1) / kBlockK;
  // Clusters are not placed in the last slots while the kernel before still holds some: 280 and 292 CTAs lost 5 to 6 % to 256.
  // More than 64 tokens that add in memory: one CTA to an SM, as a product of many tokens has had them, with the shared memory of
  // two; with half of it a ring of three blocks of 144 rows was all there was room for (5,120 x 17,408 at 128 tokens 40.9 -> 34.2 us,
  // 5,120 x 25,600 at 96 55.7 -> 46.7, 4,096 x 12,288 at 96 25.0 -> 21.4).
  const int most = meet == 1 ? 2 * d.sms * 15 / 16 : T > 64 ? d.sms : 2 * d.sms;
  double least = 1e30;
  best = FewPlan{};
  auto consider = [&](int split, bool at_once) {
    for (int rows = 16; rows <= 256; rows += 16)
      for (int late = 0; late <= (meet == 1 && split > 1 ? 1 : 0); ++late) {
        FewPlan f{};
        f.rows = rows; f.split = split; f.red = meet > 1 && split > 1 ? 1 : 0; f.cluster = f.red ? 1 : split; f.late = late;
        f.tiles = (N + rows - 1) / rows; f.grid = f.tiles * split;
        f.deep = meet > 1 && T > 64 && f.grid <= d.sms ? 1 : 0;
        if (f.grid > (split > 1 ? most : 2 * d.sms) && at_once) continue;
        if (f.cluster > 1 && f.tiles > d.two[f.cluster] && at_once) continue;       // or the last ones cost a second round
        if (!few_memory(T, kb / split, f)) continue;
        const double t = few_cost(T, N, K, gated, f, d);
        if (t < least) { least = t; best = f; }
      }
  };
  if (meet > 1)
    for (int split = 2; split <= meet && split <= kb; ++split) consider(split, true);
  else
    consider(ranges, true);
  if (best.rows == 0 && meet > 1) consider(1, true);
  if (best.rows == 0 && meet == 1 && ranges > 1) consider(ranges, false);
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, best);
  return best.rows > 0;
}

template <int MM, bool LATE>
int launch_few(const CUtensorMap& mw, const CUtensorMap& my, const FewParams& p, const FewPlan& f, cudaStream_t stream) {
  const cudaError_t e = configure_few<MM, LATE>();
  if (e != cudaSuccess) return fail("gemm_tc: cannot reserve %d bytes of shared memory: %s", 2 * kFewSmem, cudaGetErrorString(e));
  ilb::launch_cluster(gemm_few_kernel<MM, LATE>, dim3(f.grid), dim3(kFewThreads), (size_t)f.smem, stream, p.cluster, mw, my, p);
  return check_launch("gemm_tc");
}

// Fills in the deal and launches; `p` holds everything else.
int run_few(FewParams& p, const FewPlan& f, const void* A, int lda, const void* W, int ldw, cudaStream_t stream) {
  p.rows = f.rows; p.groups = few_groups(f.rows); p.tp = (p.T + 7) / 8 * 8; p.k_blocks = (p.K + kBlockK - 1) / kBlockK; p.split = f.split; p.cluster = f.cluster;
  p.stages = f.stages; p.red = f.red; p.stage_bytes = (p.tp + p.rows) * 128; p.ring_bytes = f.ring; p.recv_bytes = f.recv;
  p.tmem_cols = p.rows <= 32 ? 32 : p.rows <= 64 ? 64 : p.rows <= 128 ? 128 : 256;
  CUtensorMap mw, my;
  if (p.epilogue == kSwiGLU ? make_gated_map(&mw, W, p.N, p.K, ldw, p.groups) : make_map(&mw, W, p.N, p.K, ldw, p.rows)) return -1;
  if (make_map(&my, A, p.T, p.K, lda, p.tp)) return -1;
  if (f.late) return p.T <= 64 ? launch_few<64, true>(mw, my, p, f, stream) : launch_few<128, true>(mw, my, p, f, stream);
  return p.T <= 64 ? launch_few<64, false>(mw, my, p, f, stream) : launch_few<128, false>(mw, my, p, f, stream);
}
