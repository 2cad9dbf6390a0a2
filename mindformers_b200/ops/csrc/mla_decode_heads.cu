// Multi-latent attention decode over a paged latent cache, heads on the rows (sm_100a, tcgen05 + TMA).
//
//     s[h, t] = scale * <q[h, 0:576], c[t, 0:576]>   t < len          o[h, :] = sum_t softmax(s[h])[t] * c[t, 0:512]
//
// mla_decode.cu puts the tokens on the 128 rows of the tensor core and 16 heads on the columns: with 128 heads on one GPU every tile of the
// cache goes through shared memory sixteen times (eight chunks of heads, twice each). Here up to 128 heads are the rows:
//     S [128 heads x 128 tokens] = Q (A, K-major, resident) . C_tile^T (B, K-major)        -> tensor memory, two buffers
//     O [128 heads x 256]       += P (A, bf16, tensor memory) . C_tile (B, MN-major)
// and the products cost the same for 16 heads as for 128. O over all 512 columns would fill tensor memory alone, so a CTA takes one half of
// them and the scores are computed by both halves' CTAs. Q leaves no room for a whole tile beside it (147 of 227 KB at 128 heads),
// so a tile is streamed through a ring of 16 KB slots: nine units of 128 tokens x 64 columns for the scores, then, one tile later, the
// half again from L2 for the values as four units of 32 tokens x 256 columns: 208 KB per tile and CTA instead of 576 KB per tile and 32
// heads. The scores of tile j + 1 run under the softmax of tile j. A ring slot is free again when its products are done, nothing else
// holds the stream up.
//
// Bound by the stream: 32 sequences of 1152 - 2304 tokens, 128 heads: 146 us with 16 heads per CTA, 62 us here with one producer warp, 56 us
// with three; 8 sequences of 2000 - 4000 tokens in pages of 16 rows: 87, 46 and 36 us (with the merge, cold L2).
//
// Rows past the chunk's heads hold whatever shared memory held: rows of a product do not touch each other, and those are not stored.
//
// Roles (256 threads): warps 0, 6, 7 TMA producers (block-table lookups; the units in turn: announcing and issuing a unit takes a warp
// longer than its products take the tensor core), warp 1 MMA issuer + TMEM owner, warps 2..5 softmax / epilogue, one head per thread. Every
// wait is bounded (common.cuh). Partial results are merged by mla_combine_kernel (mla_decode.cu).
#include "common.cuh"

namespace mfb {
namespace mlah {

constexpr int kThreads = 256, kProducers = 3;
constexpr int kTile = 128;                 // tokens per tile
constexpr int kRank = 512, kDim = 576, kSubs = kDim / 64;
constexpr int kHalf = 256, kVSubs = kHalf / 64;
constexpr int kVRows = 32, kVSub = kVRows * 128;       // values: units of 32 tokens, [32 tokens][64 columns] swizzled sub-tiles
constexpr int kSub = kTile * 128;          // [128 tokens][64 columns] swizzled sub-tile, 16 KB
constexpr float kRescale = 8.0f;

// per number of query rows in shared memory: the fewer, the deeper the ring
template <int ROWS>
struct Shape {
  static constexpr int kQSub = ROWS * 128, kQBytes = kSubs * kQSub;
  static constexpr int kFixed = kQBytes + 64 * 8 + 16 + 1024;
  static constexpr int kFit = (232448 - kFixed) / kSub;
  static constexpr int kSlots = kFit < 12 ? kFit : 12;
  static constexpr int kSmem = kFixed + kSlots * kSub;
};

struct Args {
  const int* block_tables;   // [B, max_blocks]
  const int* context_lens;   // [B]
  int max_blocks, block_size, num_heads, splits;
  float scale_log2;
  float* part_o;             // [B, splits, num_heads, 512] unnormalised
  float* part_ml;            // [B, splits, num_heads, 2]: running max (log2 units), sum
  int* status;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16,"
      " %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

template <int ROWS>
__global__ void __launch_bounds__(kThreads, 1)
mla_decode_heads_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmC,
                        const __grid_constant__ CUtensorMap tmV, const Args args) {
  using Sh = Shape<ROWS>;
  constexpr int kSlots = Sh::kSlots, kQSub = Sh::kQSub;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sRing = sQ + Sh::kQBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sRing + kSlots * kSub);
  uint64_t* q_full = bars;                  // 1
  uint64_t* s_full = bars + 1;              // 2
  uint64_t* p_ready = bars + 3;             // 2: P of an even / odd tile written (128 arrivals)
  uint64_t* pv_done = bars + 5;             // 1
  uint64_t* full = bars + 8;                // kSlots
  uint64_t* empty = full + kSlots;          // kSlots
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(empty + kSlots);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = blockIdx.x & 1, split = blockIdx.x >> 1, b = blockIdx.z;
  const int len = args.context_lens[b];
  const int n_tiles_all = (len + kTile - 1) / kTile;
  const int per = (n_tiles_all + args.splits - 1) / args.splits;
  const int t0 = split * per;
  const int t1 = (t0 + per < n_tiles_all) ? t0 + per : n_tiles_all;
  const int n_tiles = t1 > t0 ? t1 - t0 : 0;
  const int head0 = blockIdx.y * ROWS;
  const int heads = args.num_heads - head0 < ROWS ? args.num_heads - head0 : ROWS;
  const size_t first_row = (static_cast<size_t>(b) * args.splits + split) * args.num_heads + head0;
  if (n_tiles == 0) {                       // the merge skips a split whose sum is zero
    if (half == 0)
      for (int h = threadIdx.x; h < heads; h += kThreads) {
        args.part_ml[(first_row + h) * 2] = -INFINITY;
        args.part_ml[(first_row + h) * 2 + 1] = 0.f;
      }
    return;
  }

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(smem_u32(q_full), 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&s_full[s]), 1);
      mbar_init(smem_u32(&p_ready[s]), 128);
    }
    mbar_init(smem_u32(pv_done), 1);
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(smem_u32(&full[s]), 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    fence_barrier_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmC);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_holder), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tmem_O = tmem_base, tmem_S = tmem_base + kHalf;       // two score buffers of 128 columns; P in the first 64 of each

  if (warp == 0 || warp >= 6) {
    // ------------------------------------ producers (the whole warp, one lane issues) ------------------------------------
    const bool leader = elect_one();
    const uint32_t mine = warp == 0 ? 0 : warp - 5;
    if (mine == 0) {
      if (leader) {
        mbar_expect_tx(smem_u32(q_full), Sh::kQBytes);
        for (int c = 0; c < kSubs; ++c) tma_load_2d(smem_u32(sQ) + c * kQSub, &tmQ, smem_u32(q_full), c * 64, b * args.num_heads + head0);
      }
      __syncwarp();
    }
    const int bs = args.block_size;
    const int* table = args.block_tables + static_cast<size_t>(b) * args.max_blocks;
    uint32_t unit = 0;
    bool ok = true;
    const int vrows = bs < kVRows ? bs : kVRows;              // rows of a value box
    // The slot of the next unit, or -1: another producer's. A free slot is announced to take 16 KB (the lanes agree on the outcome). A
    // producer's last unit was at most kProducers back, so that the parity of its wait names the right phase (kSlots > kProducers).
    auto claim = [&]() {
      const uint32_t u = unit++;
      if (u % kProducers != mine) return -1;
      const int slot = u % kSlots;
      ok = mbar_wait(smem_u32(&empty[slot]), ((u / kSlots) & 1) ^ 1, abort_flag, args.status, kStatusWaitTimeoutProducer);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return -1;
      if (leader) mbar_expect_tx(smem_u32(&full[slot]), kSub);
      __syncwarp();
      return slot;
    };
    int page = tile_page(table, bs, t0 * kTile, len), before = page;
    for (int j = 0; j <= n_tiles && ok; ++j) {
      const int next = j + 1 < n_tiles ? tile_page(table, bs, (t0 + j + 1) * kTile, len) : 0;
      if (j < n_tiles)
        for (int c = 0; c < kSubs && ok; ++c) {
          const int slot = claim();
          if (slot >= 0) tma_load_pages(leader, smem_u32(sRing + slot * kSub), kSub, &tmC, smem_u32(&full[slot]), page, bs, c * 64, 1);
        }
      if (j > 0)
        for (int t = 0; t < kTile && ok; t += kVRows) {
          const int slot = claim();
          if (slot < 0) continue;
          for (int r = 0; r < kVRows; r += vrows) {
            const int at = __reduce_add_sync(0xffffffffu, lane == (t + r) / bs ? before : 0) * bs + (t + r) % bs;
            for (int c = 0; c < kVSubs; ++c)
              tma_load_2d_warp(leader, smem_u32(sRing + slot * kSub + c * kVSub + r * 128), &tmV, smem_u32(&full[slot]),
                               half * kHalf + c * 64, at);
          }
        }
      before = page;
      page = next;
    }
  } else if (warp == 1) {
    // ------------------------------------ MMA issuer (the whole warp, one lane issues) ------------------------------------
    constexpr uint32_t IDESC_S = umma_idesc_bf16(kTile, kTile, 0, 0);    // A = Q K-major, B = cache K-major
    constexpr uint32_t IDESC_PV = umma_idesc_bf16(kTile, kHalf, 0, 1);   // A = P (tensor memory), B = cache MN-major
    const bool leader = elect_one();
    const uint64_t ring_k = umma_desc_kmajor_sw128(smem_u32(sRing)), ring_v = umma_desc_mnmajor_sw128(smem_u32(sRing), kVSub);
    const uint64_t q_desc = umma_desc_kmajor_sw128(smem_u32(sQ));
    uint32_t unit = 0;
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      ok = mbar_wait(smem_u32(bar), parity, abort_flag, args.status, kStatusWaitTimeoutMma);
      ok = __all_sync(0xffffffffu, ok);
    };
    wait(q_full, 0);
    for (int j = 0; j <= n_tiles && ok; ++j) {
      if (j < n_tiles) {
        // ---- S(j) = Q . C(j)^T: P(j - 2), which lay there, has been read by the product issued before this one ----
        const uint32_t d = tmem_S + (j & 1) * kTile;
        for (int c = 0; c < kSubs; ++c) {
          const int slot = unit % kSlots;
          wait(&full[slot], (unit / kSlots) & 1);
          if (!ok) break;
          tc_fence_after();
          const uint64_t ca = ring_k + slot * (kSub >> 4), qa = q_desc + c * (kQSub >> 4);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_f16_ss_warp(leader, d, qa + k * 2, ca + k * 2, IDESC_S, (c > 0 || k > 0) ? 1u : 0u);
          umma_commit_warp(leader, smem_u32(&empty[slot]));
          ++unit;
        }
        if (!ok) break;
        umma_commit_warp(leader, smem_u32(&s_full[j & 1]));
      }
      if (j > 0) {
        // ---- O += P(j - 1) . C(j - 1) ----
        const int i = j - 1;
        wait(&p_ready[i & 1], (i >> 1) & 1);
        for (int c = 0; c < kTile / kVRows && ok; ++c) {
          const int slot = unit % kSlots;
          wait(&full[slot], (unit / kSlots) & 1);
          if (!ok) break;
          tc_fence_after();
          const uint64_t ca = ring_v + slot * (kSub >> 4);
#pragma unroll
          for (int k = 0; k < kVRows / 16; ++k)          // bf16 pairs: 8 columns of P per 16 tokens
            umma_f16_ts_warp(leader, tmem_O, tmem_S + (i & 1) * kTile + (c * (kVRows / 16) + k) * 8, ca + ((k * 16 * 128) >> 4), IDESC_PV,
                             (i > 0 || c > 0 || k > 0) ? 1u : 0u);
          umma_commit_warp(leader, smem_u32(&empty[slot]));
          ++unit;
        }
        if (!ok) break;
        umma_commit_warp(leader, smem_u32(pv_done));
      }
    }
  } else {
    // ------------------------------------ softmax / epilogue ------------------------------------
    const int ew = warp & 3;                        // tensor-memory lane quarter of this warp
    const int row = ew * 32 + lane;                 // head of this thread
    const bool idle = ew * 32 >= heads;             // no head in this warp: it only keeps the barriers going
    const uint32_t lane_base = static_cast<uint32_t>(ew * 32) << 16;
    const uint64_t scale2 = pack2(args.scale_log2, args.scale_log2);
    float m_used = -INFINITY, l_sum = 0.f;
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      ok = mbar_wait(smem_u32(&s_full[j & 1]), (j >> 1) & 1, abort_flag, args.status, kStatusWaitTimeoutEpilogue);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (!idle) {
        tc_fence_after();
        const uint32_t s_tmem = tmem_S + (j & 1) * kTile + lane_base;
        const int left = len - (t0 + j) * kTile;    // tokens of this tile
        uint32_t sr[kTile];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(s_tmem + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&sr[c * 32]));
        tmem_ld_wait();
        float* s = reinterpret_cast<float*>(sr);
        if (left < kTile) {
#pragma unroll
          for (int i = 0; i < kTile; ++i)
            if (i >= left) s[i] = -INFINITY;
        }
        float mxs[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          float m = s[a * 32];
#pragma unroll
          for (int i = 1; i + 1 < 32; i += 2) m = fmax3(m, s[a * 32 + i], s[a * 32 + i + 1]);
          mxs[a] = fmaxf(m, s[a * 32 + 31]);
        }
        const float mx = fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3])) * args.scale_log2;
        float alpha = 1.f;
        if (m_used == -INFINITY) {
          m_used = mx;
        } else if (mx > m_used + kRescale) {
          alpha = ex2(m_used - mx);
          m_used = mx;
        }
        if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
          // O is touched between the products of tile j - 1 and those of tile j, which wait for p_ready below. (The scores of
          // tile j were issued behind the products of tile j - 2, so the parity means tile j - 1.)
          ok = mbar_wait(smem_u32(pv_done), (j - 1) & 1, abort_flag, args.status, kStatusWaitTimeoutEpilogue);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < kHalf / 16; ++c) {
            uint32_t r[16];
            tmem_ld_32x32b_x16(tmem_O + lane_base + c * 16, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            tmem_st_32x32b_x16(tmem_O + lane_base + c * 16, r);
          }
        }
        const float neg_m = m_used == -INFINITY ? 0.f : -m_used;
        const uint64_t negm2 = pack2(neg_m, neg_m);
        uint64_t rs2[4] = {0, 0, 0, 0};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t pk[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            float a0, a1;
            unpack2(fma2(pack2(s[h * 64 + 2 * i], s[h * 64 + 2 * i + 1]), scale2, negm2), a0, a1);
            const float e0 = ex2(a0), e1 = ex2(a1);
            rs2[i & 3] = add2(rs2[i & 3], pack2(e0, e1));
            pk[i] = pack_bf16x2(e0, e1);
          }
          tmem_st_32x32b_x32(s_tmem + h * 32, pk);
        }
        float r0, r1, r2, r3;
        unpack2(add2(rs2[0], rs2[1]), r0, r1);
        unpack2(add2(rs2[2], rs2[3]), r2, r3);
        l_sum = l_sum * alpha + ((r0 + r1) + (r2 + r3));
        tmem_st_wait();
        tc_fence_before();
      }
      mbar_arrive(smem_u32(&p_ready[j & 1]));
    }
    // a parity names one of two phases: the last but one first, the last scores only vouch for the products before it
    if (ok && n_tiles > 1) ok = mbar_wait(smem_u32(pv_done), n_tiles & 1, abort_flag, args.status, kStatusWaitTimeoutEpilogue);
    if (ok) ok = mbar_wait(smem_u32(pv_done), (n_tiles - 1) & 1, abort_flag, args.status, kStatusWaitTimeoutEpilogue);
    // one decision for the whole warpgroup: the stage below is the ring, which is free once every product is done
    ok = named_bar_and(2, 128, ok);
    if (!idle) {
      if (half == 0 && row < heads) {
        float* ml = args.part_ml + (first_row + row) * 2;
        ml[0] = ok ? m_used : -INFINITY;
        ml[1] = ok ? l_sum : 0.f;
      }
      if (ok) {
        tc_fence_after();
        // 32 columns at a time through 4 KB per warp, so that a row's 128 bytes are stored by eight neighbouring lanes
        uint8_t* stage = sRing + ew * 4096;
        float* obase = args.part_o + (first_row + ew * 32) * kRank + half * kHalf;
#pragma unroll 1
        for (int c = 0; c < kHalf / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(tmem_O + lane_base + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 8; ++q)
            *reinterpret_cast<uint4*>(stage + lane * 128 + ((q ^ (lane & 7)) << 4)) = make_uint4(r[q * 4], r[q * 4 + 1], r[q * 4 + 2], r[q * 4 + 3]);
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rr = i * 4 + (lane >> 3), q = lane & 7;
            if (ew * 32 + rr < heads)
              *reinterpret_cast<uint4*>(obase + static_cast<size_t>(rr) * kRank + c * 32 + q * 4) =
                  *reinterpret_cast<const uint4*>(stage + rr * 128 + ((q ^ (rr & 7)) << 4));
          }
          __syncwarp();
        }
        tc_fence_before();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int ROWS>
int launch(const CUtensorMap& tQ, const CUtensorMap& tC, const CUtensorMap& tV, const Args& a, int B, cudaStream_t stream) {
  static_assert(Shape<ROWS>::kSlots >= 5 && Shape<ROWS>::kSmem <= 232448, "shared memory budget exceeded");
  static_assert(Shape<ROWS>::kQBytes - Shape<ROWS>::kQSub + 128 * 128 <= Shape<ROWS>::kSmem - 1024, "a product's 128 rows lie in shared memory");
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(mla_decode_heads_kernel<ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<ROWS>::kSmem) != cudaSuccess) {
      mfb_host::set_error("mla_decode_heads: cannot raise the shared memory limit");
      return 10;
    }
    attr_set = true;
  }
  const dim3 grid(a.splits * 2, (a.num_heads + ROWS - 1) / ROWS, B);
  mla_decode_heads_kernel<ROWS><<<grid, kThreads, Shape<ROWS>::kSmem, stream>>>(tQ, tC, tV, a);
  if (cudaGetLastError() != cudaSuccess) { mfb_host::set_error("mla_decode_heads: launch failed"); return 11; }
  return 0;
}

int rows_per_cta(int num_heads) { return num_heads <= 32 ? 32 : num_heads <= 64 ? 64 : 128; }

}  // namespace mlah
}  // namespace mfb

extern "C" {
using namespace mfb;

// Number of sequence splits that fills the GPU for a batch of B sequences of up to max_len tokens: waves of CTAs over the 148 SMs x (tiles
// per CTA + about three tiles' time for the query, the first tile's way through and the result).
int mfb_mla_decode_heads_splits(int B, int num_heads, int max_len) {
  const int per = mlah::rows_per_cta(num_heads), chunks = (num_heads + per - 1) / per;
  const int tiles = (max_len + mlah::kTile - 1) / mlah::kTile;
  int best = 1;
  long long best_cost = -1;
  for (int s = 1; s <= tiles && s <= 32; ++s) {
    const long long ctas = static_cast<long long>(B) * chunks * s * 2;
    const long long cost = (ctas + 147) / 148 * ((tiles + s - 1) / s + 3);
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = s; }
  }
  return best;
}

// Arguments as in mfb_mla_decode_attention (mla_decode.cu), which launches this and the merge; part_o [B, splits, num_heads, 512], part_ml
// [B, splits, num_heads, 2].
int mfb_mla_decode_heads_launch(const void* q, const void* cache, const int* block_tables, const int* context_lens, float* part_o,
                                float* part_ml, int splits, int B, int num_heads, int num_blocks, int block_size, int max_blocks,
                                float scale, int* status, cudaStream_t stream) {
  CUtensorMap tQ, tC, tV;
  int rc;
  const CUtensorMapDataType BF = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const int rows = mlah::rows_per_cta(num_heads);
  const uint64_t slots = (uint64_t)num_blocks * block_size;
  if ((rc = mfb_host::make_tmap_2d(&tQ, q, 2, BF, (uint64_t)B * num_heads, mlah::kDim, mlah::kDim, rows, 64))) return 20 + rc;
  if ((rc = mfb_host::make_tmap_2d(&tC, cache, 2, BF, slots, mlah::kDim, mlah::kDim, block_size, 64))) return 30 + rc;
  if ((rc = mfb_host::make_tmap_2d(&tV, cache, 2, BF, slots, mlah::kDim, mlah::kDim,
                                   block_size < mlah::kVRows ? block_size : mlah::kVRows, 64))) return 40 + rc;
  mlah::Args a;
  a.block_tables = block_tables; a.context_lens = context_lens; a.max_blocks = max_blocks; a.block_size = block_size;
  a.num_heads = num_heads; a.splits = splits; a.scale_log2 = scale * 1.4426950408889634f;
  a.part_o = part_o; a.part_ml = part_ml; a.status = status;
  if (rows == 32) return mlah::launch<32>(tQ, tC, tV, a, B, stream);
  return rows == 64 ? mlah::launch<64>(tQ, tC, tV, a, B, stream) : mlah::launch<128>(tQ, tC, tV, a, B, stream);
}

}  // extern "C"
