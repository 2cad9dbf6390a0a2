// Decode attention over a paged int8 KV cache on warp-level tensor-core products (mma.sync m16n8k16, sm_100a): head dim 64 or 128, up to
// 16 query heads per KV head, one fp32 scale per cached token and KV head.
//
// Bound by memory: 2 (D + 4) bytes per cached token and KV head, read once for all query heads of the group. What competes with it is the
// conversion of the codes, so the products are chosen for the layout of their operands and not for their rate: a warp takes 16 tokens in
// the order in which mma.sync wants them (the reduction index of a product may be permuted at will, so 16 consecutive bytes of a
// row are a thread's share of it). Every thread copies its own bytes (cp.async, conflict-free, no barrier) and reads them back itself.
// tcgen05 would want the converted operands in shared memory, 2 bytes written and read again per code.
//
//   S = Q K^T   rows: heads, columns: tokens. Codes become fp16 exactly, two in a byte permutation and a subtraction (below); bf16
//               would take four instructions. q, 8 significant bits, is exact in fp16 too once a power of two has brought the
//               head's largest number to 2^13 (numbers below 2^-27 of it lose bits). The sums are fp32, scale_k is applied to them.
//   O = P V     P scale_v as the sum of two fp16 numbers (22 bits), brought into their range by a power of two that follows the
//               largest scale_v seen; the sums are fp32. Up to 8 heads leave half of the product's rows free for the second part.
//
// Work: grid (splits, KV heads, sequences), every sequence cut into `splits` equal ranges by its own length; 4 warps take the range's
// 16-token groups in turn, each with three groups (12 KB) in flight, 16 warps per SM, merge in shared memory and leave a partial
// result for paged_combine_kernel. Block sizes are multiples of 16, so that a group lies in one page.
//
// 48 sequences of 3000 - 6000 tokens, 28 / 4 heads of 128: 587 us on the CUDA cores (fp32 products and a five-step shuffle
// reduction per key and head); 90 us with bf16 operands (830 instructions per group) and one group ahead in registers; 76 us now, 3.0 TB/s:
// 590 instructions per group fill 44 % of the issue slots, for the rest the 15 warps of an SM wait for their copies; the 1344 CTAs are 2.3 waves,
// so that an SM is busy 80 % of the time.
#include <cuda_fp16.h>

#include "mma_sync.cuh"

namespace mfb {
namespace pd8 {

constexpr int kWarps = 4;
constexpr int kGroup = 16;        // tokens per step of a warp

struct Args {
  const __nv_bfloat16* q;         // rows ld_q, heads ld_head elements apart
  long long ld_q, ld_head;
  const int8_t *k, *v;            // [slots, Hkv, HD]
  const float *ks, *vs;           // [slots, Hkv]
  const int *tables, *lens;
  float *part_acc, *part_ml;      // [B, Hq, splits, HD], [B, Hq, splits, 2]
  int Hq, Hkv, block_size, max_blocks;
  float scale_log2;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Codes as offset bytes (code + 128) a pair at a time: 0x6400 | byte is 1024 + byte in fp16, and the difference is exact. PICK: which two
// bytes of x.
template <int PICK>
__device__ __forceinline__ uint32_t codes_to_f16(uint32_t x) {
  const uint32_t u = __byte_perm(x, 0x64646464u, PICK == 0 ? 0x4140 : 0x4342), off = 0x64806480u;
  const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&u), *reinterpret_cast<const __half2*>(&off));
  return *reinterpret_cast<const uint32_t*>(&d);
}
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// two fp32 numbers as a pair of fp16 numbers; they become what is left
__device__ __forceinline__ uint32_t take_f16(float& x, float& y) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  x -= f.x;
  y -= f.y;
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void cp4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 lds16(uint32_t addr) {
  uint4 r;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(addr) : "memory");
  return r;
}
__device__ __forceinline__ float2 lds8f(uint32_t addr) {
  float2 r;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(r.x), "=f"(r.y) : "r"(addr) : "memory");
  return r;
}

constexpr int kStages = 3;
constexpr float kLazy = 7.f;            // a new maximum counts when it is this much (log2) above the one in use: P <= 2^7
constexpr float kBase = 256.f;          // times this and vs / c <= 1: at most 2^15

// one group: K and V rows, then 16 scales of each
template <int HD>
constexpr int kStageBytes = 2 * kGroup * HD + 2 * kGroup * 4;
template <int HD, bool WIDE>
constexpr int kMergeBytes = kWarps * (WIDE ? 16 : 8) * (HD + 4) * 4;
template <int HD, bool WIDE>
constexpr int kSmem = kWarps * kStages * kStageBytes<HD> > kMergeBytes<HD, WIDE> ? kWarps * kStages * kStageBytes<HD> : kMergeBytes<HD, WIDE>;

// WIDE: more than eight query heads per KV head (rows 8 .. 15 of the products)
template <int HD, bool WIDE>
__global__ void __launch_bounds__(kWarps * 32, 4)
paged_decode_int8_kernel(const Args a) {
  constexpr int KL = HD / 64;     // 16-byte pieces of a key row per thread
  constexpr int NT = HD / 8;      // 8-column tiles of the result
  constexpr int VB = HD / 8;      // bytes of a value row per thread
  constexpr int HR = WIDE ? 16 : 8, R = WIDE ? 2 : 1;
  constexpr int kStage = kStageBytes<HD>;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float sh_m[kWarps][HR], sh_l[kWarps][HR];
  const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z, splits = gridDim.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int group = a.Hq / a.Hkv;
  const int* table = a.tables + static_cast<size_t>(b) * a.max_blocks;
  // an idle row of a captured step has a length but no blocks: no keys
  const int ctx = table[0] < 0 ? 0 : min(a.lens[b], a.max_blocks * a.block_size);
  // whole rounds of the four warps per split; the later splits of a short sequence stay empty
  const int rounds = (ctx + kWarps * kGroup - 1) / (kWarps * kGroup);
  const int per = (rounds + splits - 1) / splits * kWarps;                // groups per split
  const int groups_all = (ctx + kGroup - 1) / kGroup;
  const int g0 = split * per, g1 = min(g0 + per, groups_all);
  const size_t head0 = static_cast<size_t>(b) * a.Hq + static_cast<size_t>(kvh) * group;
  if (g0 >= g1) {                 // nothing here: the merge skips a split whose maximum is -inf
    for (int h = threadIdx.x; h < group; h += kWarps * 32) {
      float* ml = a.part_ml + ((head0 + h) * splits + split) * 2;
      ml[0] = -INFINITY;
      ml[1] = 0.f;
    }
    return;
  }

  // copies of a group: this thread's key bytes (rows gid, gid + 8), its value bytes (tokens 2 tig, 2 tig + 1 and 8 more of each) and one scale
  const long long row = static_cast<long long>(a.Hkv) * HD;
  const int8_t* k_mine = a.k + static_cast<long long>(kvh) * HD + gid * row + tig * 16;
  const int8_t* v_mine = a.v + static_cast<long long>(kvh) * HD + 2 * tig * row + gid * VB;
  const float* s_mine = (lane < 16 ? a.ks : a.vs) + static_cast<long long>(lane & 15) * a.Hkv + kvh;
  const uint32_t ring = smem_u32(smem) + warp * kStages * kStage;
  const int shift = (a.block_size & (a.block_size - 1)) == 0 ? __ffs(a.block_size) - 1 : -1;
  auto fetch = [&](int g, uint32_t dst) {
    const int tok0 = g * kGroup;
    const int at = shift >= 0 ? tok0 >> shift : tok0 / a.block_size;
    const int page = max(__ldg(table + at), 0);                   // a block that is missing belongs to a row nobody reads
    const long long slot = static_cast<long long>(page) * a.block_size + (tok0 - at * a.block_size);
    const int8_t *kp = k_mine + slot * row, *vp = v_mine + slot * row;
    dst += lane * 16;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int l = 0; l < KL; ++l) cp16(dst + (n * KL + l) * 512, kp + n * 8 * row + l * 64, 16);
    dst += 2 * KL * 512;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int8_t* p = vp + ((i & 1) + (i >> 1) * 8) * row;
      if constexpr (HD == 128) cp16(dst + i * 512, p, 16);
      else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst - lane * 8 + i * 256), "l"(p) : "memory");
    }
    dst += kGroup * HD - lane * 16;
    cp4(dst + lane * 4, s_mine + slot * a.Hkv);
  };

  int g = g0 + warp;
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) {
    if (g + i * kWarps < g1) fetch(g + i * kWarps, ring + i * kStage);
    cp_commit();
  }

  // Q as the A operand: step (l, w) of the scores reduces over the four columns l 64 + tig 16 + w 4 .. of every thread of a quad
  uint32_t qf[KL * 4][2 * R];
  float unscale[R];               // of the scores: the inverse of the power of two below, times the softmax scale
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int h = gid + 8 * r;
    uint2 u[KL * 4];
    float mx = 0.f;
#pragma unroll
    for (int l = 0; l < KL; ++l)
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        uint2& x = u[l * 4 + w];
        x = make_uint2(0u, 0u);
        if (h < group)
          x = *reinterpret_cast<const uint2*>(a.q + b * a.ld_q + (static_cast<long long>(kvh) * group + h) * a.ld_head + l * 64 +
                                              tig * 16 + w * 4);
        mx = fmaxf(mx, fmaxf(fmaxf(fabsf(__uint_as_float(x.x << 16)), fabsf(__uint_as_float(x.x & 0xffff0000u))),
                             fmaxf(fabsf(__uint_as_float(x.y << 16)), fabsf(__uint_as_float(x.y & 0xffff0000u)))));
      }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    // 2^13 over the power of two below the largest number; infinities stay what they are
    const int e = static_cast<int>(__float_as_uint(mx) >> 23);
    const float f = e == 0 || e == 255 ? 1.f : __uint_as_float(static_cast<uint32_t>(min(267 - e, 253)) << 23);
    unscale[r] = a.scale_log2 / f;
#pragma unroll
    for (int i = 0; i < KL * 4; ++i) {
      const __half2 x = __floats2half2_rn(__uint_as_float(u[i].x << 16) * f, __uint_as_float(u[i].x & 0xffff0000u) * f);
      const __half2 y = __floats2half2_rn(__uint_as_float(u[i].y << 16) * f, __uint_as_float(u[i].y & 0xffff0000u) * f);
      qf[i][r] = *reinterpret_cast<const uint32_t*>(&x);
      qf[i][R + r] = *reinterpret_cast<const uint32_t*>(&y);
    }
  }

  float o[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[j][i] = 0.f;
  float m[R], sum[R], c = __uint_as_float(0x0d800000u);       // c: power of two (2^-100 to 2^127), at least every value scale so far
#pragma unroll
  for (int r = 0; r < R; ++r) { m[r] = -INFINITY; sum[r] = 0.f; }

  int stage = 0;
  for (; g < g1; g += kWarps) {
    const uint32_t src = ring + stage * kStage;
    {
      const int ahead = stage == 0 ? kStages - 1 : stage - 1;             // the stage that was read last
      if (g + (kStages - 1) * kWarps < g1) fetch(g + (kStages - 1) * kWarps, ring + ahead * kStage);
      cp_commit();
      cp_wait<kStages - 1>();
      __syncwarp();               // the scales come from other lanes
      stage = stage == kStages - 1 ? 0 : stage + 1;
    }
    float s[2][4] = {};
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int l = 0; l < KL; ++l) {
        const uint4 u = lds16(src + lane * 16 + (n * KL + l) * 512);
        const uint32_t words[4] = {u.x ^ 0x80808080u, u.y ^ 0x80808080u, u.z ^ 0x80808080u, u.w ^ 0x80808080u};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const uint32_t (&q)[2 * R] = qf[l * 4 + w];
          mma_f16(s[n], q[0], WIDE ? q[R - 1] : 0u, q[R], WIDE ? q[2 * R - 1] : 0u, codes_to_f16<0>(words[w]), codes_to_f16<1>(words[w]));
        }
      }
    const int left = ctx - g * kGroup - 2 * tig;              // tokens of this group from this thread's first on
    const uint32_t sc = src + 2 * kGroup * HD + tig * 8;
    const float2 ka = lds8f(sc), kb = lds8f(sc + 32), va = lds8f(sc + 64), vb = lds8f(sc + 96);
    const float ks[4] = {ka.x, ka.y, kb.x, kb.y};
    // scales past the end may be anything
    const float vs[4] = {left > 0 ? va.x : 0.f, left > 1 ? va.y : 0.f, left > 8 ? vb.x : 0.f, left > 9 ? vb.y : 0.f};
    float vmax = fmaxf(fmaxf(vs[0], vs[1]), fmaxf(vs[2], vs[3]));
    float e[R][4], top[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      e[r][0] = left > 0 ? s[0][r * 2] * (ks[0] * unscale[r]) : -INFINITY;
      e[r][1] = left > 1 ? s[0][r * 2 + 1] * (ks[1] * unscale[r]) : -INFINITY;
      e[r][2] = left > 8 ? s[1][r * 2] * (ks[2] * unscale[r]) : -INFINITY;
      e[r][3] = left > 9 ? s[1][r * 2 + 1] * (ks[3] * unscale[r]) : -INFINITY;
      top[r] = fmaxf(fmaxf(e[r][0], e[r][1]), fmaxf(e[r][2], e[r][3]));
      top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 1));
      top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 2));
    }
    vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, 1));
    vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, 2));
    bool grows = vmax > c;
#pragma unroll
    for (int r = 0; r < R; ++r) grows = grows || top[r] > m[r] + kLazy;
    if (__any_sync(0xffffffffu, grows)) {
      const float c_new = vmax > c ? __uint_as_float(min((__float_as_uint(vmax) + 0x007fffffu) & 0xff800000u, 0x7f000000u)) : c;
      const float beta = c / c_new;
      c = c_new;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float alpha = 1.f;
        if (top[r] > m[r] + kLazy) {
          alpha = ex2(m[r] - top[r]);                         // 0 when nothing was accumulated yet
          m[r] = top[r];
        }
        sum[r] *= alpha;
        alpha *= beta;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          o[j][r * 2] *= alpha;
          o[j][r * 2 + 1] *= alpha;
          if constexpr (!WIDE) { o[j][2] *= alpha; o[j][3] *= alpha; }
        }
      }
    }
    uint32_t hi[4], lo[4];
    const float back = kBase / c;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float neg = m[r] == -INFINITY ? 0.f : -m[r];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        e[r][i] = ex2(e[r][i] + neg);
        sum[r] += e[r][i];
        e[r][i] *= vs[i] * back;
      }
      hi[r] = take_f16(e[r][0], e[r][1]);
      hi[2 + r] = take_f16(e[r][2], e[r][3]);
      lo[r] = take_f16(e[r][0], e[r][1]);
      lo[2 + r] = take_f16(e[r][2], e[r][3]);
    }
    if constexpr (!WIDE) { hi[1] = lo[0]; hi[3] = lo[2]; }      // rows 8 .. 15 are free: both parts in one product
    const uint32_t vsrc = src + kGroup * HD + lane * VB;
    auto product = [&](int j, uint32_t b0, uint32_t b1) {
      mma_f16(o[j], hi[0], hi[1], hi[2], hi[3], b0, b1);
      if constexpr (WIDE) mma_f16(o[j], lo[0], lo[1], lo[2], lo[3], b0, b1);
    };
    auto four = [&](int j, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
      const uint32_t x01 = __byte_perm(w0, w1, 0x5140) ^ 0x80808080u, x23 = __byte_perm(w0, w1, 0x7362) ^ 0x80808080u;
      const uint32_t y01 = __byte_perm(w2, w3, 0x5140) ^ 0x80808080u, y23 = __byte_perm(w2, w3, 0x7362) ^ 0x80808080u;
      product(j, codes_to_f16<0>(x01), codes_to_f16<0>(y01));
      product(j + 1, codes_to_f16<1>(x01), codes_to_f16<1>(y01));
      product(j + 2, codes_to_f16<0>(x23), codes_to_f16<0>(y23));
      product(j + 3, codes_to_f16<1>(x23), codes_to_f16<1>(y23));
    };
    if constexpr (HD == 128) {
      const uint4 w0 = lds16(vsrc), w1 = lds16(vsrc + 512), w2 = lds16(vsrc + 1024), w3 = lds16(vsrc + 1536);
      four(0, w0.x, w1.x, w2.x, w3.x);
      four(4, w0.y, w1.y, w2.y, w3.y);
      four(8, w0.z, w1.z, w2.z, w3.z);
      four(12, w0.w, w1.w, w2.w, w3.w);
    } else {
      const float2 w0 = lds8f(vsrc), w1 = lds8f(vsrc + 256), w2 = lds8f(vsrc + 512), w3 = lds8f(vsrc + 768);
      four(0, __float_as_uint(w0.x), __float_as_uint(w1.x), __float_as_uint(w2.x), __float_as_uint(w3.x));
      four(4, __float_as_uint(w0.y), __float_as_uint(w1.y), __float_as_uint(w2.y), __float_as_uint(w3.y));
    }
    __syncwarp();                 // the scales of this stage are read
  }
  cp_wait<0>();
  if constexpr (!WIDE) {
#pragma unroll
    for (int j = 0; j < NT; ++j) { o[j][0] += o[j][2]; o[j][1] += o[j][3]; }
  }

  // the four warps' results, through shared memory (the ring is free)
  __syncthreads();
  float* sh_o = reinterpret_cast<float*>(smem);           // [warp][head][HD + 4]
  const float unbase = c / kBase;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
    sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
    const int h = gid + 8 * r;
    if (tig == 0) { sh_m[warp][h] = m[r]; sh_l[warp][h] = sum[r]; }
    float* dst = sh_o + (warp * HR + h) * (HD + 4) + 2 * tig * VB;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      dst[j] = o[j][r * 2] * unbase;
      dst[VB + j] = o[j][r * 2 + 1] * unbase;
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < group * HD; idx += kWarps * 32) {
    const int h = idx / HD, d = idx % HD;
    float mx = sh_m[0][h];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) mx = fmaxf(mx, sh_m[w][h]);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = sh_m[w][h] == -INFINITY ? 0.f : ex2(sh_m[w][h] - mx);
      num += f * sh_o[(w * HR + h) * (HD + 4) + d];
      den += f * sh_l[w][h];
    }
    const size_t at = (head0 + h) * splits + split;
    a.part_acc[at * HD + d] = num;
    if (d == 0) { a.part_ml[at * 2] = mx; a.part_ml[at * 2 + 1] = den; }
  }
}

template <int HD, bool WIDE>
int launch(const Args& a, dim3 grid, cudaStream_t stream) {
  constexpr int SMEM = kSmem<HD, WIDE>;
  static_assert(4 * (SMEM + 2048) <= 232448, "four CTAs share an SM");
  auto kern = paged_decode_int8_kernel<HD, WIDE>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) {
      mfb_host::set_error("paged_decode_int8: cannot raise the shared memory limit");
      return 10;
    }
    attr_set = true;
  }
  kern<<<grid, kWarps * 32, SMEM, stream>>>(a);
  if (cudaGetLastError() != cudaSuccess) { mfb_host::set_error("paged_decode_int8: launch failed"); return 11; }
  return 0;
}

}  // namespace pd8
}  // namespace mfb

extern "C" {
using namespace mfb;

int mfb_paged_combine_ex(const float* part_acc, const float* part_ml, void* out, int splits, int rows, int hd, int Hq,
                         const int* cu_q, const float* sink, long long ld_out, float out_scale,
                         cudaStream_t stream);      // paged_attention.cu

// 1 when the kernel serves these shapes. Other block sizes and groups run on the CUDA-core kernel of paged_attention.cu.
int mfb_paged_decode_int8_supported(int Hq, int Hkv, int hd, int block_size) {
  return (hd == 64 || hd == 128) && Hkv >= 1 && Hq >= 1 && Hq % Hkv == 0 && Hq / Hkv <= 16 && block_size >= 16 && block_size % 16 == 0;
}

// Ranges per sequence. The lengths are on the device, so the number follows from what the tables could hold: two waves of the 4 x 148
// resident CTAs even out sequences of different lengths (64 x 2048 - 4096 tokens, 8 KV heads: 157 us with one range per sequence, 142 to 148 us
// with two to eight), and no range is shorter than 512 tokens if the tables are full (100 x 150 - 300 tokens, 4 KV heads, tables of 8192: 28, 32
// and 36 us with 1, 3 and 5). A sequence shorter than that uses 64-token ranges and leaves the rest empty.
int mfb_paged_decode_int8_splits(int B, int Hkv, int max_len) {
  const long long pairs = (long long)B * Hkv;
  long long s = (2 * 4 * 148 + pairs - 1) / pairs;
  const long long most = ((long long)max_len + 511) / 512;
  if (s > most) s = most;
  if (s > 64) s = 64;
  return s < 1 ? 1 : (int)s;
}

// q [B, Hq, hd] bf16 (rows ld_q, heads ld_head elements apart), caches [num_blocks, block_size, Hkv, hd] int8 with scales [num_blocks,
// block_size, Hkv], out [B, Hq, hd] bf16; scratch of mfb_paged_decode_scratch_bytes(B, Hq, hd, splits).
int mfb_paged_decode_attention_int8(const void* q, long long ld_q, long long ld_head, const void* key_cache, const void* value_cache,
                                    const float* key_scale, const float* value_scale, const int* block_tables, const int* context_lens,
                                    void* out, void* scratch, int splits, int B, int Hq, int Hkv, int hd, int block_size, int max_blocks,
                                    float scale, cudaStream_t stream) {
  if (!mfb_paged_decode_int8_supported(Hq, Hkv, hd, block_size) || splits < 1 || ld_q % 4 || ld_head % 4 ||
      (reinterpret_cast<uintptr_t>(q) & 7) || ((reinterpret_cast<uintptr_t>(key_cache) | reinterpret_cast<uintptr_t>(value_cache)) & 15)) {
    mfb_host::set_error("paged_decode_int8: unsupported Hq=%d Hkv=%d hd=%d block_size=%d splits=%d", Hq, Hkv, hd, block_size, splits);
    return 1;
  }
  if (B <= 0) return 0;
  pd8::Args a;
  a.q = (const __nv_bfloat16*)q; a.ld_q = ld_q; a.ld_head = ld_head;
  a.k = (const int8_t*)key_cache; a.v = (const int8_t*)value_cache; a.ks = key_scale; a.vs = value_scale;
  a.tables = block_tables; a.lens = context_lens;
  a.part_acc = (float*)scratch; a.part_ml = a.part_acc + (size_t)B * Hq * splits * hd;
  a.Hq = Hq; a.Hkv = Hkv; a.block_size = block_size; a.max_blocks = max_blocks; a.scale_log2 = scale * 1.4426950408889634f;
  const dim3 grid(splits, Hkv, B);
  const bool wide = Hq / Hkv > 8;
  const int rc = hd == 128 ? (wide ? pd8::launch<128, true>(a, grid, stream) : pd8::launch<128, false>(a, grid, stream))
                           : (wide ? pd8::launch<64, true>(a, grid, stream) : pd8::launch<64, false>(a, grid, stream));
  if (rc) return rc;
  return mfb_paged_combine_ex(a.part_acc, a.part_ml, out, splits, B * Hq, hd, Hq, nullptr, nullptr, (long long)Hq * hd, 1.f, stream);
}

}  // extern "C"
