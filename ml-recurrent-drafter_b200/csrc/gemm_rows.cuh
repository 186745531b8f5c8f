// The projections of few tokens (one user's decode steps, small batches, one row's draft): included by gemm_tc.cu, whose
// epilogues, descriptors and waits it uses.
//
// Such a call is bound by the bytes of its weights, which one wave of these CTAs reads at 5.7 to 6.3 TB/s of a copy's 6.5 (the times
// below).  gemm_tc_pair_kernel reads them through few SMs (one pair per 256 features: 96 of 148 SMs for 12288 features, 32 for 4096)
// and only once the kernel before has finished.  With many tokens it wins all the same (rows_first).  Here
//   * every CTA owns `rows` weight rows (32 .. 256, the fewest that let one wave cover the matrix), all of K and all tokens: one
//     tile per CTA, and the sums of a row in the order of gemm_tc_pair_kernel.  Projections whose norm adds shares of K (kEpiResShares) have
//     slabs of 128 rows instead and a share a CTA (cut_shape has the rule and the figures);
//   * a load is a box of `rows` weight rows x KB k-blocks of 64 (a three-dimensional map: feature within a k-block, row, k-block), and
//     a step of the MMA loop is such a load: with few columns the thread that issues the products, not the tensor core, sets the
//     pace (a wait, a commit and the loop's own instructions cost it some 150 cycles a step, a product 23 to 39);
//   * launches of plans with early weights (rd_gemm_plan_early) begin before the kernels ahead of them have finished.  They request the
//     first ring of weights, and then every warp runs its own code once with nothing to do: no live rows, products, loads and
//     commits switched off.  Instructions that an SM has not run since the last kernel come from L2 or memory, about a microsecond at
//     each new stretch of code: after the dependency wait that was 1.5 us to the first load of tokens, 0.9 to the first product
//     and 2 to 4 for an epilogue that needs 0.6.
// Back to back in a stream, bf16, one B200, us (the pair kernel's, o and down with the norm that adds their shares, beside): 22016 x
// 4096, 1 token 30.7 (36.8), 110 tokens 36.5 (42.6); 12288 x 4096, 1 token 17.7 (27), 110 tokens 22.6 (31); 6144 x 4096, 24 tokens
// 11.8 (17.8); whole, 4096 x 4096 11.6 (12.4); 4096 x 11008 21.6 (22.1); 32000 x 4096, 1 token 41.5 (47).  In a decode step of 32 such layers
// 122 -> 94 us a layer, attention and norms included.
// Slabs of more than 128 rows take two MMAs per 16 features of K: rows [0, 128) and rows [rows - 128, rows), whose overlap is
// computed twice and stored once.  Slabs of 32 rows read past their end in shared memory: those accumulator rows are not stored.
// QKV projections with rotary embedding (heads of 128 rows) in slabs of 64 or 32 rows: the CTAs of a head are a cluster and hand
// their accumulators to one of them, block of 32 tokens by block, through distributed shared memory.
__host__ __device__ constexpr int row_map_index(int cols) { return cols <= 16 ? 0 : (cols + 31) / 32; }
__host__ __device__ constexpr int row_map_rows(int index) { return index == 0 ? 16 : 32 * index; }

constexpr int kRowsThreads = 224;  // as gemm_tc_kernel, and warp 6 loads the tokens
constexpr int kRowsMaxStages = 16;
constexpr int kRowsScratch = 32 * kScrLd * 4;               // of the run without work
constexpr int kRowsEpiBytes = kRopeMetaBytes + 1024;        // rope_meta_stage, reduction buffer of normed heads
constexpr int kRowsSmem = 227 * 1024;                       // one CTA on an SM: two with half the ring each were 10 to 20 % slower
constexpr int kRowsRing = kRowsSmem - 1024 /*alignment slack*/ - kRowsScratch - kRowsEpiBytes - 512 /*barriers*/;
static_assert((2 * kRowsMaxStages + 2) * 8 + 16 <= 512 && kRowsScratch % 16 == 0 && kRowsEpiBytes % 16 == 0 && kRowsRing % 16 == 0, "layout");
__host__ __device__ constexpr int rows_stages(int rows, int a_rows, int kb) {
  return kRowsRing / ((rows + a_rows) * kb * 128) < kRowsMaxStages ? kRowsRing / ((rows + a_rows) * kb * 128) : kRowsMaxStages;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
      "@p cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}" ::"r"(smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(on)
      : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_if(uint64_t* bar, uint32_t bytes, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t"
      "@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
      "r"(bytes), "r"(on)
      : "memory");
}
__device__ __forceinline__ void umma_f16_if(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t acc, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(acc), "r"(on)
      : "memory");
}
__device__ __forceinline__ void umma_commit_if(uint64_t* bar, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)),
      "r"(on)
      : "memory");
}

// All products of a CTA, issued by one thread; `on` = 0 runs one step without products and commits (`full` then never completes, and a
// wait for the phase before its first passes at once).
// MM: rows of a product.  Reading its weights takes the tensor core 32 cycles for 128 rows however few the tokens, so slabs of 32
// and 64 rows take products of 64.  TWO: slabs of more than 128 rows.  KB: k-blocks of a step; the last step's, past K, are zeros.  CUT: a
// share of K, which may end inside a load of two k-blocks, the second of them the next share's: half a step after the loop (asking in
// the loop cost every projection, 60.1 -> 60.8 us a layer of width 2048 at 24 tokens).
template <int MM, bool TWO, int KB, bool CUT>
__device__ __forceinline__ bool rows_mma(int rows, int cols, int steps, bool half, int stages, uint32_t tmem_base, uint32_t upper_cols, uint32_t s_w,
                                         uint32_t s_a, int a_block, uint64_t* full, uint64_t* empty, uint64_t* acc_full, volatile int* abort_flag, uint32_t on) {
  const uint32_t idesc = (umma_instr_desc(cols) & 0x00ffffffu) | ((uint32_t)(MM >> 4) << 24);
  const uint64_t dw0 = umma_smem_desc(s_w), da0 = umma_smem_desc(s_a);
  const uint32_t w_block = rows * 128 / 16, upper = (rows - BM) * 128 / 16;  // descriptors count 16-byte units
  a_block /= 16;
  uint64_t dw = dw0, da = da0;
  int stage = 0;
  uint32_t phase = on ^ 1, acc = 0;
  if (CUT && KB == 2 && half) --steps;
#pragma unroll 1
  for (int i = 0; i < steps; ++i) {
    if (!mbar_wait(&full[stage], phase, abort_flag)) return false;
    tc_fence_after();
#pragma unroll
    for (int b = 0; b < KB; ++b) {
#pragma unroll
      for (int k = 0; k < BK / UMMA_K; ++k) umma_f16_if(tmem_base, dw + b * w_block + 2 * k, da + b * a_block + 2 * k, idesc, acc | b | k, on);
      if (TWO) {
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_f16_if(tmem_base + upper_cols, dw + b * w_block + upper + 2 * k, da + b * a_block + 2 * k, idesc, acc | b | k, on);
      }
    }
    acc = 1;
    umma_commit_if(&empty[stage], on);
    dw += KB * w_block;
    da += KB * a_block;
    if (++stage == stages) {
      stage = 0;
      phase ^= 1;
      dw = dw0;
      da = da0;
    }
  }
  if (CUT && KB == 2 && half) {
    static_assert(!CUT || !TWO, "slabs of shares have 128 rows");
    if (!mbar_wait(&full[stage], phase, abort_flag)) return false;
    tc_fence_after();
#pragma unroll
    for (int k = 0; k < BK / UMMA_K; ++k) umma_f16_if(tmem_base, dw + 2 * k, da + 2 * k, idesc, acc | k, on);
  }
  umma_commit_if(acc_full, on);
  return true;
}

template <int V>
struct Int {
  static constexpr int value = V;
};

// The four epilogue warps' part; on = 0: without live tokens, on a barrier that never completes.
template <int EPI, bool OUT_F32>
__device__ __forceinline__ bool rows_epilogue(const EpiArgs& epi, const RowsShape& sh, int quarter, int lane, int row0, int M, int cols, int N,
                                              uint32_t tmem_base, float* ring, uint32_t on, int* s_pos, int* s_dst, float* ss_red,
                                              uint64_t* acc_full, volatile int* abort_flag) {
  constexpr int kOut = kGlu<EPI> ? 16 : 32;
  constexpr bool kRes = (EPI == RD_EPI_BIAS_SILU_RES || EPI == RD_EPI_RES);
  constexpr bool kBias = (EPI == RD_EPI_BIAS || EPI == RD_EPI_BIAS_SILU || EPI == RD_EPI_BIAS_SILU_RES);
  const int esz = OUT_F32 ? 4 : 2;
  const bool aligned = (((uintptr_t)epi.C | (uintptr_t)(kRes ? epi.R : epi.C)) % 16 == 0) && ((epi.ldc * esz) % 16 == 0) &&
                       (!kRes || (epi.ldr * esz) % 16 == 0);
  const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16);
  if constexpr (EPI == kEpiQkvRope) {
    const int head = row0 / BM;
    const int gate0 = row0 - (epi.nh + 2 * epi.nkv) * BM;  // of a slab of gates: its first one
    const bool is_v = head >= epi.nh + epi.nkv, gate = gate0 >= 0;
    rope_meta_stage(epi, s_pos, s_dst, 0, M, quarter * 32 + lane, head < epi.nh, is_v);
    asm volatile("bar.sync 1, 128;" ::: "memory");  // the staged entries are visible
    RopeRows cs;
    if (sh.rows == BM) cs.request(epi, s_pos, quarter, lane, 0, M, is_v);  // on its way while the products run
    if (!mbar_wait(acc_full, on ^ 1, abort_flag)) return false;
    tc_fence_after();
    if (sh.rows < BM) return true;  // the rest is the cluster's
#pragma unroll 1
    for (int c = 0; c < cols; c += 32) {
      uint32_t r[32];
      tmem_ld32(t_lane + c, r);
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
      if (gate) {
        epilogue_gate_block(v, epi, lane, gate0 + quarter * 32, c, M);
      } else {
        if (c > 0) cs.request(epi, s_pos, quarter, lane, c, M, is_v);
        epilogue_rope_block<true>(v, epi, ring, quarter, lane, head, c, M, s_dst + c, cs, nullptr, ss_red + ((c >> 5) & 1) * 128,
                                  on ? 32 * kScrLd : 0);
      }
    }
    return true;
  } else {
    const int groups = sh.rows / 32;
    float* scr = ring;  // the ring is free once the accumulators are complete; the run without work has room for one block
    auto finish = [&](float* v, int n_warp0, int c, bool vec_ok, float bias, const ResidualRegs<OUT_F32, kOut>& res) {
      if (EPI == kEpiArgmax) {
        epilogue_argmax_block(v, epi, scr, lane, n_warp0, c, M, N);
      } else if (EPI == kEpiResShares) {
        EpiArgs part = epi;
        part.C = epi.parts + (int64_t)blockIdx.y * epi.part_rows * N;
        part.ldc = N;
        epilogue_block<RD_EPI_NONE, true>(v, part, scr, lane, n_warp0, c, M, N, N % 4 == 0 && n_warp0 + 32 <= N, ResidualRegs<true, 32>(), nullptr,
                                          make_uint4(0u, 0u, 0u, 0u), ss_red);
      } else if (EPI == kEpiSplit && n_warp0 >= epi.n_split) {
        epilogue_hi_block(v, epi, lane, n_warp0, c, M, N);
      } else {
        epilogue_math<EPI>(v, epi, n_warp0 + lane, N, !vec_ok, bias);
        epilogue_block<EPI, OUT_F32>(v, epi, scr, lane, n_warp0, c, M, N, vec_ok, res, nullptr, make_uint4(0u, 0u, 0u, 0u), ss_red);
      }
    };
    if (sh.rows < BM) {
      // rows 16 q .. 16 q + 15 lie in the first lanes of quarter q: through shared memory to warps of 32 features, a unit (32 features,
      // 32 tokens) each
      const int units = groups * ((cols + 31) / 32);
      float* all = ring;
      const int block = on ? 32 * kScrLd : 0;
      scr = all + (units + quarter) * block;
      ResidualRegs<OUT_F32, kOut> res;
      auto prepare = [&](int u) {
        const int n_warp0 = row0 + 32 * (u % groups);
        if (kRes && u < units && aligned && n_warp0 + 32 <= N) res.load(epi, u / groups * 32, kGlu<EPI> ? (n_warp0 >> 1) : n_warp0, M, lane);
      };
      prepare(quarter);
      if (!mbar_wait(acc_full, on ^ 1, abort_flag)) return false;
      tc_fence_after();
      if (quarter * 16 < sh.rows) {
        const int f = quarter * 16 + lane;
#pragma unroll 1
        for (int i = 0; i < units / groups; ++i) {
          uint32_t r[32];
          tmem_ld32(t_lane + i * 32, r);
          if (lane < 16) {
            float* to = all + (i * groups + f / 32) * block + f % 32;
#pragma unroll
            for (int j = 0; j < 32; ++j) to[j * kScrLd] = __uint_as_float(r[j]);
          }
          __syncwarp();
        }
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll 1
      for (int u = quarter; u < units; u += 4) {
        const int n_warp0 = row0 + 32 * (u % groups);
        if (n_warp0 >= N) continue;
        const bool vec_ok = aligned && (n_warp0 + 32 <= N);
        const float bias = (kBias && on && n_warp0 + lane < N) ? __bfloat162float(epi.bias[n_warp0 + lane]) : 0.f;
        if (u != quarter) prepare(u);
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = all[u * block + j * kScrLd + lane];
        finish(v, n_warp0, u / groups * 32, vec_ok, bias, res);
      }
      return true;
    }
    scr = ring + (on ? quarter * 32 * kScrLd : 0);
    bool waited = false;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      // this warp's 32 lanes of the first accumulator, then of the second, where they hold rows that the first does not
      const int g = half == 0 ? quarter : quarter + groups - 4;
      if (half == 1 && g < 4) continue;
      const int n_warp0 = row0 + 32 * g;
      if (n_warp0 >= N) continue;
      const bool vec_ok = aligned && (n_warp0 + 32 <= N);
      const int out0 = kGlu<EPI> ? (n_warp0 >> 1) : n_warp0;
      const float bias = (kBias && on && n_warp0 + lane < N) ? __bfloat162float(epi.bias[n_warp0 + lane]) : 0.f;
      ResidualRegs<OUT_F32, kOut> res;
      if (kRes && vec_ok) res.load(epi, 0, out0, M, lane);
      if (!waited && !mbar_wait(acc_full, on ^ 1, abort_flag)) return false;
      waited = true;
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < cols; c += 32) {
        if (kRes && vec_ok && c > 0) res.load(epi, c, out0, M, lane);
        uint32_t r[32];
        tmem_ld32(t_lane + half * (sh.tmem_cols / 2) + c, r);
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
        finish(v, n_warp0, c, vec_ok, bias, res);
      }
    }
    return true;
  }
}

template <int EPI, bool OUT_F32>
__global__ void __launch_bounds__(kRowsThreads, 1)
    gemm_rows_kernel(const __grid_constant__ RowMaps maps_a, const __grid_constant__ CUtensorMap map_w, EpiArgs epi,
                     const RowsShape sh, int m_max, const int32_t* m_dev, int N, int K, int32_t* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int w_bytes = sh.rows * sh.kb * 128;  // of a stage
  float* ring = reinterpret_cast<float*>(smem);
  float* scratch = reinterpret_cast<float*>(smem + kRowsRing);
  int* s_pos = reinterpret_cast<int*>(smem + kRowsRing + kRowsScratch);
  int* s_dst = s_pos + kMaxChunk;
  float* ss_red = reinterpret_cast<float*>(s_dst + kMaxChunk);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kRowsRing + kRowsScratch + kRowsEpiBytes);  // weights and tokens have landed
  uint64_t* empty = full + kRowsMaxStages;
  uint64_t* acc_full = empty + kRowsMaxStages;
  uint64_t* idle = acc_full + 1;  // never completes: what the run without work waits on, whatever the other warps have come to
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(idle + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int block0 = 0, blocks = K / BK;  // k-blocks
  if (EPI == kEpiResShares) {
    // of this CTA's share: cut where gemm_tc_pair_kernel cuts, however many k-blocks a load has, so that a row's sums are the same at
    // every capacity
    const int all = blocks;
    block0 = (int)blockIdx.y * all / (int)gridDim.y;
    blocks = ((int)blockIdx.y + 1) * all / (int)gridDim.y - block0;
  }
  const int steps = (blocks + sh.kb - 1) / sh.kb;
  const int row0 = blockIdx.x * sh.rows;
  rd::pdl_launch_dependents();
  // weight loads before the dependency wait: as many stages as there are with the most tokens
  const int ahead = sh.early ? min(rows_stages(sh.rows, sh.a_rows, sh.kb), steps) : 0;
  if (warp == 0) {
    if (rd::elect_one()) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
      for (int s = 0; s < kRowsMaxStages; ++s) {
        mbar_init(&full[s], 2);
        mbar_init(&empty[s], 1);
      }
      mbar_init(acc_full, 1);
      mbar_init(idle, 1);
      *abort_flag = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      for (int i = 0; i < ahead; ++i) {
        mbar_expect_tx_if(&full[i], w_bytes, 1);
        tma_load_3d(smem + i * w_bytes, &map_w, &full[i], 0, row0, block0 + i * sh.kb, 1);
      }
    }
    __syncwarp();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(sh.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  bool ok = true;
  int M = 0, cols = 16;  // MMA N; without live rows nothing is stored
#pragma unroll 1
  for (uint32_t on = sh.early ? 0 : 1; on < 2; ++on) {
    if (on) {
      rd::pdl_wait();
      M = rd::live_rows(m_dev, m_max);
      cols = max(16, (M + 15) / 16 * 16);
    }
    const int a_map = row_map_index(cols);
    const int a_rows = row_map_rows(a_map), a_block = a_rows * 128, a_bytes = a_block * sh.kb;
    const int stages = rows_stages(sh.rows, a_rows, sh.kb);
    uint8_t* sA = smem + stages * w_bytes;
    if (warp == 0) {
      // ---------------- weights ----------------
      if (rd::elect_one()) {
        int stage = ahead == stages ? 0 : ahead;
        uint32_t phase = ahead == stages ? 1 : 0;
        for (int i = ahead; on && i < steps; ++i) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) {
            ok = false;
            break;
          }
          mbar_expect_tx_if(&full[stage], w_bytes, 1);
          tma_load_3d(smem + stage * w_bytes, &map_w, &full[stage], 0, row0, block0 + i * sh.kb, 1);
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) {
          if (atomicCAS((int*)abort_flag, 0, 1) == 0 && status) atomicExch(status, 31);
          for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        }
      }
    } else if (warp == 6) {
      // ---------------- tokens ----------------
      if (rd::elect_one()) {
        int stage = 0;
        uint32_t phase = 0;
        for (int i = 0; i < (on ? steps : 1); ++i) {
          if (!mbar_wait(on ? &empty[stage] : idle, phase ^ 1, abort_flag)) {
            ok = false;
            break;
          }
          mbar_expect_tx_if(&full[stage], a_bytes, on);
          tma_load_3d(sA + stage * a_bytes, &maps_a.m[a_map], &full[stage], 0, 0, block0 + i * sh.kb, on);
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) {
          if (atomicCAS((int*)abort_flag, 0, 1) == 0 && status) atomicExch(status, 32);
          for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        }
      }
    } else if (warp == 1) {
      // ---------------- MMA issuer ----------------
      if (rd::elect_one()) {
        const int n = on ? steps : 1;
        const uint32_t w = smem_u32(smem), a = smem_u32(sA);
        constexpr bool kCut = EPI == kEpiResShares;
        auto run = [&](auto mm, auto two, auto kb) {
          return rows_mma<mm.value, two.value, kb.value, kCut>(sh.rows, cols, n, kCut && on && blocks % 2 != 0, stages, tmem_base, sh.tmem_cols / 2, w, a,
                                                               a_block, on ? full : idle, empty, acc_full, abort_flag, on);
        };
        if constexpr (kCut) {  // slabs of 128 rows
          ok = sh.kb == 2 ? run(Int<128>(), Int<0>(), Int<2>()) : run(Int<128>(), Int<0>(), Int<1>());
        } else {
          if (sh.rows < BM)
            ok = sh.kb == 4 ? run(Int<64>(), Int<0>(), Int<4>()) : run(Int<64>(), Int<0>(), Int<2>());
          else if (sh.rows == BM)
            ok = sh.kb == 2 ? run(Int<128>(), Int<0>(), Int<2>()) : run(Int<128>(), Int<0>(), Int<1>());
          else
            ok = sh.kb == 2 ? run(Int<128>(), Int<1>(), Int<2>()) : run(Int<128>(), Int<1>(), Int<1>());
        }
        if (!ok && atomicCAS((int*)abort_flag, 0, 1) == 0 && status) atomicExch(status, 33);
      }
    } else {
      // ---------------- epilogue warps ----------------
      ok = rows_epilogue<EPI, OUT_F32>(epi, sh, warp & 3, lane, row0, M, cols, N, tmem_base, on ? ring : scratch, on, s_pos, s_dst,
                                       ss_red, on ? acc_full : idle, abort_flag);
      if (!ok && lane == 0 && atomicCAS((int*)abort_flag, 0, 1) == 0 && status) atomicExch(status, 34);
    }
    __syncwarp();
  }

  if constexpr (EPI == kEpiQkvRope) {
    if (sh.rows < BM) {
      // the CTAs of a head, `parts` of them: token block i goes to CTA i % parts, which finishes it
      const int parts = BM / sh.rows, rank = (int)cluster_ctarank();
      const int quarter = warp & 3, head = row0 / BM, blocks = (cols + 31) / 32;
      const bool epilogue = warp >= 2 && warp <= 5, is_v = head >= epi.nh + epi.nkv, gate = head >= epi.nh + 2 * epi.nkv;
      RopeRows cs;
      if (epilogue && !gate && rank < blocks) cs.request(epi, s_pos, quarter, lane, rank * 32, M, is_v);
      tc_fence_before();
      cluster_sync_all();  // every CTA's rings are free
      tc_fence_after();
      if (epilogue && quarter * 16 < sh.rows) {
        const int f = rank * sh.rows + quarter * 16 + lane;  // this lane's feature of the head; lanes 16 .. 31 have none
#pragma unroll 1
        for (int i = 0; i < blocks; ++i) {
          __syncwarp();
          uint32_t r[32];
          tmem_ld32(tmem_base + ((uint32_t)(quarter * 32) << 16) + i * 32, r);
          if (lane >= 16) continue;
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
          if (gate) {
            epilogue_gate_block(v, epi, lane, (head - epi.nh - 2 * epi.nkv) * BM + f - lane, i * 32, M);
            continue;
          }
          const uint32_t to = mapa_u32(smem_u32(ring + ((i / parts) * 4 + f / 32) * 32 * kScrLd + f % 32), i % parts);
          rope_round(v, epi, nullptr);
#pragma unroll
          for (int j = 0; j < 32; ++j)
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to + j * kScrLd * 4), "f"(v[j]) : "memory");
        }
        __syncwarp();
      }
      cluster_sync_all();
      if (epilogue && !gate) {
#pragma unroll 1
        for (int i = rank; i < blocks; i += parts) {
          if (i > rank) cs.request(epi, s_pos, quarter, lane, i * 32, M, is_v);
          epilogue_rope_block<false>(nullptr, epi, ring + (i / parts) * 4 * 32 * kScrLd, quarter, lane, head, i * 32, M, s_dst + i * 32, cs,
                                     nullptr, ss_red + (i & 1) * 128);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(sh.tmem_cols) : "memory");
  }
}
