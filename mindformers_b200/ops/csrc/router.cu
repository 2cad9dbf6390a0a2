// Top-k MoE router (sm_100a): score function, optional expert bias, group-limited selection, top-k,
// renormalisation, scaling and per-expert token counts in one pass; one warp per token.
//
//   logits (+ a bias of their own, forward only)
//   scores = softmax(logits) | sigmoid(logits)                                   [T, E] fp32
//   sel    = scores (+ bias); with G groups only the best `group_topk` groups stay eligible, a group being
//            ranked by its best score (no bias) or by the sum of its two best biased scores (bias given)
//   ids    = top-k of sel (ties: lower expert index first);  probs = scores[ids]
//   probs  = probs / (sum(probs) + 1e-20) when `norm`;  probs *= scale;  counts[e] += 1 per selected copy
//
// The backward kernel recomputes the scores from the logits and maps d(probs) (and an optional dense
// d(scores), used by the load-balancing loss) to d(logits). E <= 512 and k <= 32.
#include "common.cuh"

namespace mfb {

constexpr int kRouterMaxPerLane = 16;  // E / 32
constexpr int kRouterMaxK = 32;
constexpr int kRouterWarps = 4;

struct RouterArgs {
  int T, E, k, sigmoid, norm, groups, group_topk;
  float scale;
};

// (value, index) arg-max over the warp; ties go to the lower index
__device__ __forceinline__ void warp_argmax(float& v, int& i) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, i, o);
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
  }
}

template <int PER>
__device__ __forceinline__ void router_scores(const float* __restrict__ row, const float* __restrict__ logit_bias, int E, int lane,
                                              bool sigmoid, float (&s)[PER]) {
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int e = lane + 32 * j;
    s[j] = e < E ? (logit_bias ? row[e] + logit_bias[e] : row[e]) : -INFINITY;
    mx = fmaxf(mx, s[j]);
  }
  if (sigmoid) {
#pragma unroll
    for (int j = 0; j < PER; ++j) s[j] = (lane + 32 * j) < E ? 1.f / (1.f + expf(-s[j])) : 0.f;
    return;
  }
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    s[j] = (lane + 32 * j) < E ? expf(s[j] - mx) : 0.f;
    sum += s[j];
  }
  sum = warp_sum(sum);
  const float inv = 1.f / sum;
#pragma unroll
  for (int j = 0; j < PER; ++j) s[j] *= inv;
}

template <int PER>
__global__ void __launch_bounds__(kRouterWarps * 32)
router_fwd_kernel(const float* __restrict__ logits, const float* __restrict__ logit_bias, const float* __restrict__ bias,
                  float* __restrict__ probs,
                  long long* __restrict__ ids, float* __restrict__ scores_out, float* __restrict__ counts,
                  RouterArgs a) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * kRouterWarps + (threadIdx.x >> 5);
  if (t >= a.T) return;
  float s[PER], sel[PER];
  router_scores<PER>(logits + (long long)t * a.E, logit_bias, a.E, lane, a.sigmoid != 0, s);
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int e = lane + 32 * j;
    sel[j] = e < a.E ? (bias ? s[j] + bias[e] : s[j]) : -INFINITY;
    if (scores_out && e < a.E) scores_out[(long long)t * a.E + e] = s[j];
  }
  if (a.groups > 1 && a.group_topk > 0 && a.group_topk < a.groups) {
    // group score for every group (computed by the whole warp, group by group), then keep the best ones
    const int gsz = a.E / a.groups;
    float gscore = -INFINITY;  // lane g holds the score of group g (groups <= 32)
    for (int g = 0; g < a.groups; ++g) {
      float b1 = -INFINITY, b2 = -INFINITY;
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int e = lane + 32 * j;
        if (e < a.E && e / gsz == g) {
          if (sel[j] > b1) { b2 = b1; b1 = sel[j]; } else if (sel[j] > b2) { b2 = sel[j]; }
        }
      }
      // merge (best, second best) pairs over the warp
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float o1 = __shfl_xor_sync(0xffffffffu, b1, o), o2 = __shfl_xor_sync(0xffffffffu, b2, o);
        const float n1 = fmaxf(b1, o1);
        const float n2 = fmaxf(fminf(b1, o1), fmaxf(b2, o2));
        b1 = n1; b2 = n2;
      }
      const float sc = bias ? (b1 + (gsz > 1 ? b2 : 0.f)) : b1;
      if (lane == g) gscore = sc;
    }
    unsigned keep = 0;
    for (int r = 0; r < a.group_topk; ++r) {
      float v = gscore; int i = lane;
      warp_argmax(v, i);
      keep |= 1u << i;
      if (lane == i) gscore = -INFINITY;
    }
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int e = lane + 32 * j;
      if (e < a.E && !((keep >> (e / gsz)) & 1u)) sel[j] = -INFINITY;
    }
  }
  float psum = 0.f;
  float my_p = 0.f;  // lane r keeps the r-th selected probability
  int my_id = 0;
  for (int r = 0; r < a.k; ++r) {
    float bv = -INFINITY; int bi = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int e = lane + 32 * j;
      if (sel[j] > bv || (sel[j] == bv && e < bi)) { bv = sel[j]; bi = e; }
    }
    warp_argmax(bv, bi);
    // owner lane supplies the unbiased score and retires the expert
    float sv = 0.f;
#pragma unroll
    for (int j = 0; j < PER; ++j)
      if (lane + 32 * j == bi) { sv = s[j]; sel[j] = -INFINITY; }
    sv = __shfl_sync(0xffffffffu, sv, bi & 31);
    psum += sv;
    if (lane == r) { my_p = sv; my_id = bi; }
  }
  if (lane < a.k) {
    float p = my_p;
    if (a.norm) p = p / (psum + 1e-20f);
    probs[(long long)t * a.k + lane] = p * a.scale;
    ids[(long long)t * a.k + lane] = my_id;
    if (counts) atomicAdd(counts + my_id, 1.f);
  }
}

template <int PER>
__global__ void __launch_bounds__(kRouterWarps * 32)
router_bwd_kernel(const float* __restrict__ logits, const long long* __restrict__ ids,
                  const float* __restrict__ dprobs, const float* __restrict__ dscores,
                  float* __restrict__ dlogits, RouterArgs a) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * kRouterWarps + (threadIdx.x >> 5);
  if (t >= a.T) return;
  float s[PER], ds[PER];
  router_scores<PER>(logits + (long long)t * a.E, nullptr, a.E, lane, a.sigmoid != 0, s);
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int e = lane + 32 * j;
    ds[j] = (dscores && e < a.E) ? dscores[(long long)t * a.E + e] : 0.f;
  }
  // selected set: D = sum s_sel, A = sum dout_j * s_j
  const int my_id = lane < a.k ? (int)ids[(long long)t * a.k + lane] : -1;
  const float my_do = lane < a.k ? dprobs[(long long)t * a.k + lane] * a.scale : 0.f;
  float my_s = 0.f;
  for (int r = 0; r < a.k; ++r) {
    const int id = __shfl_sync(0xffffffffu, my_id, r);
    float sv = 0.f;
#pragma unroll
    for (int j = 0; j < PER; ++j)
      if (lane + 32 * j == id) sv = s[j];
    sv = __shfl_sync(0xffffffffu, sv, id & 31);
    if (lane == r) my_s = sv;
  }
  float D = warp_sum(my_s);
  float A = warp_sum(my_do * my_s);
  float my_ds = my_do;
  if (a.norm) {
    D += 1e-20f;
    my_ds = my_do / D - A / (D * D);
  }
  for (int r = 0; r < a.k; ++r) {
    const int id = __shfl_sync(0xffffffffu, my_id, r);
    const float g = __shfl_sync(0xffffffffu, my_ds, r);
#pragma unroll
    for (int j = 0; j < PER; ++j)
      if (lane + 32 * j == id) ds[j] += g;
  }
  if (a.sigmoid) {
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int e = lane + 32 * j;
      if (e < a.E) dlogits[(long long)t * a.E + e] = ds[j] * s[j] * (1.f - s[j]);
    }
  } else {
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < PER; ++j) dot += ds[j] * s[j];
    dot = warp_sum(dot);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int e = lane + 32 * j;
      if (e < a.E) dlogits[(long long)t * a.E + e] = s[j] * (ds[j] - dot);
    }
  }
}

// ---- the gate: logits [T, E] fp32 of bf16 rows and fp32 weights -------------------------------------------------------------------
// A few rows (a decode step): fp32 products on the CUDA cores. Bound by latency, so that the loads of a weight row are spread over four
// warps, four of them in flight per lane: a CTA has two experts and eight rows, a weight is read once for eight rows. 24 rows, 128 experts,
// 2048 columns: a conversion of the rows, a library product and its split reduction took 25 us; with a warp per expert 16 us.
constexpr int kGateRows = 8, kGateParts = 4, kGateExperts = 2;
__global__ void __launch_bounds__(kGateParts * kGateExperts * 32)
gate_rows_kernel(const __nv_bfloat16* __restrict__ x, long long ld, const float* __restrict__ w, float* __restrict__ logits, int T, int E,
                 int H) {
  __shared__ float part[kGateExperts][kGateParts][kGateRows];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = warp % kGateParts, le = warp / kGateParts;
  const int e = blockIdx.x * kGateExperts + le, t0 = blockIdx.y * kGateRows;
  const int n = T - t0 < kGateRows ? T - t0 : kGateRows;
  const float4* wr = reinterpret_cast<const float4*>(w + (long long)(e < E ? e : 0) * H);
  float acc[kGateRows] = {};
#pragma unroll 4
  for (int v = q * 32 + lane; v < H / 4; v += kGateParts * 32) {
    const float4 f = __ldg(wr + v);
#pragma unroll
    for (int i = 0; i < kGateRows; ++i) {
      const uint2 u = __ldg(reinterpret_cast<const uint2*>(x + (long long)(t0 + (i < n ? i : 0)) * ld) + v);
      acc[i] = fmaf(f.x, __uint_as_float(u.x << 16), acc[i]);
      acc[i] = fmaf(f.y, __uint_as_float(u.x & 0xffff0000u), acc[i]);
      acc[i] = fmaf(f.z, __uint_as_float(u.y << 16), acc[i]);
      acc[i] = fmaf(f.w, __uint_as_float(u.y & 0xffff0000u), acc[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < kGateRows; ++i) {
    const float s = warp_sum(acc[i]);
    if (lane == i) part[le][q][i] = s;
  }
  __syncthreads();
  if (threadIdx.x < kGateExperts * kGateRows) {
    const int k = threadIdx.x / kGateRows, i = threadIdx.x % kGateRows, f = blockIdx.x * kGateExperts + k;
    if (f < E && i < n) logits[(long long)(t0 + i) * E + f] = (part[k][0][i] + part[k][1][i]) + (part[k][2][i] + part[k][3][i]);
  }
}

// Many rows, backward: the products run on the tensor cores with an fp32 operand as the sum of three bf16 numbers, 24 bits, which is all of
// it. Their accumulators drop what does not fit instead of rounding it, so that a sum over thousands of products is 2e-6 to 4e-6 off where fp32
// library products are 0.5e-6 off; the weight's gradient is therefore summed over 256 rows at a time (0.24e-6) and the blocks are added
// here. (The rows' gradient has 6 E products and is rounded to bf16. The logits stay with fp32 products: an error of 2e-6 decides
// ten times as many ties between experts.) x [R, C] becomes six copies side by side (`across`: [R, 6 C]) or one below the other ([6 R, C]),
// each a part 0, 1 or 2 as `parts` says.
struct SplitArgs { int part[6]; };
__global__ void __launch_bounds__(256)
split3_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ out, long long R, int C, int across, SplitArgs a) {
  const int vecs = C / 8;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < R * vecs; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vecs;
    const int c = (int)(i - r * vecs);
    float f[8];
    *reinterpret_cast<float4*>(f) = reinterpret_cast<const float4*>(x)[2 * i];
    *reinterpret_cast<float4*>(f + 4) = reinterpret_cast<const float4*>(x)[2 * i + 1];
    uint4 p[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      uint32_t h[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        h[j] = pack_bf16x2(f[2 * j], f[2 * j + 1]);
        f[2 * j] -= __uint_as_float(h[j] << 16);
        f[2 * j + 1] -= __uint_as_float(h[j] & 0xffff0000u);
      }
      p[k] = make_uint4(h[0], h[1], h[2], h[3]);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const long long at = across ? (r * 6 + k) * vecs + c : (k * R + r) * vecs + c;
      reinterpret_cast<uint4*>(out)[at] = a.part[k] == 0 ? p[0] : a.part[k] == 1 ? p[1] : p[2];
    }
  }
}
// out [R, C] = the sum of `groups` times three blocks of x, `group_apart` and `apart` numbers apart, rows ld numbers apart; the third
// blocks, which hold the smallest numbers, first
__global__ void __launch_bounds__(256)
sum3_kernel(const float* __restrict__ x, float* __restrict__ out, long long R, int C, long long ld, long long apart, int groups,
            long long group_apart) {
  const int vecs = C / 4;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < R * vecs; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vecs;
    const float* p = x + r * ld + (i - r * vecs) * 4;
    float4 s[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) s[k] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int g = 0; g < groups; ++g)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float4 a = *reinterpret_cast<const float4*>(p + g * group_apart + k * apart);
        s[k].x += a.x; s[k].y += a.y; s[k].z += a.z; s[k].w += a.w;
      }
    reinterpret_cast<float4*>(out)[i] = make_float4((s[2].x + s[1].x) + s[0].x, (s[2].y + s[1].y) + s[0].y, (s[2].z + s[1].z) + s[0].z,
                                                    (s[2].w + s[1].w) + s[0].w);
  }
}

}  // namespace mfb

extern "C" {
using namespace mfb;

static int router_check(int T, int E, int k, int groups, int group_topk) {
  if (E < 1 || E > 32 * kRouterMaxPerLane || k < 1 || k > kRouterMaxK || k > E) {
    mfb_host::set_error("router: E=%d (max %d) / k=%d (max %d) out of range", E, 32 * kRouterMaxPerLane, k, kRouterMaxK);
    return 1;
  }
  if (groups > 1 && (groups > 32 || E % groups != 0 || group_topk > groups)) {
    mfb_host::set_error("router: %d groups (max 32, must divide E=%d), group_topk=%d", groups, E, group_topk);
    return 1;
  }
  return 0;
}

#define MFB_ROUTER_DISPATCH(KERNEL, ...)                                               \
  do {                                                                                 \
    const int per = (E + 31) / 32;                                                     \
    const unsigned grid = (unsigned)((T + kRouterWarps - 1) / kRouterWarps);           \
    if (per <= 4) KERNEL<4><<<grid, kRouterWarps * 32, 0, stream>>>(__VA_ARGS__);      \
    else if (per <= 8) KERNEL<8><<<grid, kRouterWarps * 32, 0, stream>>>(__VA_ARGS__); \
    else KERNEL<16><<<grid, kRouterWarps * 32, 0, stream>>>(__VA_ARGS__);              \
  } while (0)

// logits [T, E] fp32 (contiguous); logit_bias [E] or null: added to the logits; bias [E] or null; probs [T, k] fp32; ids [T, k] int64;
// scores_out [T, E] fp32 or null; counts [E] fp32 or null (incremented, not cleared).
int mfb_router_fwd(const float* logits, const float* logit_bias, const float* bias, float* probs, long long* ids, float* scores_out,
                   float* counts, int T, int E, int k, int sigmoid, int norm, int groups, int group_topk,
                   float scale, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (router_check(T, E, k, groups, group_topk)) return 1;
  RouterArgs a{T, E, k, sigmoid, norm, groups, group_topk, scale};
  MFB_ROUTER_DISPATCH(router_fwd_kernel, logits, logit_bias, bias, probs, ids, scores_out, counts, a);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

// dlogits [T, E] = d(probs) and optional dense d(scores) pulled back through the router.
int mfb_router_bwd(const float* logits, const long long* ids, const float* dprobs, const float* dscores,
                   float* dlogits, int T, int E, int k, int sigmoid, int norm, float scale, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (router_check(T, E, k, 0, 0)) return 1;
  RouterArgs a{T, E, k, sigmoid, norm, 0, 0, scale};
  MFB_ROUTER_DISPATCH(router_bwd_kernel, logits, ids, dprobs, dscores, dlogits, a);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

// logits [T, E] = x [T, H] (bf16, rows ld apart) times w [E, H] (fp32) transposed. H and ld multiples of 4; x on 8, w on 16 bytes.
int mfb_gate_rows(const void* x, long long ld, const float* w, float* logits, int T, int E, int H, cudaStream_t stream) {
  if (H % 4 || ld % 4 || E < 1 || (reinterpret_cast<uintptr_t>(x) & 7) || (reinterpret_cast<uintptr_t>(w) & 15)) {
    mfb_host::set_error("gate_rows: E=%d H=%d", E, H);
    return 1;
  }
  if (T <= 0) return 0;
  gate_rows_kernel<<<dim3((E + kGateExperts - 1) / kGateExperts, (T + kGateRows - 1) / kGateRows), kGateParts * kGateExperts * 32, 0, stream>>>(
      (const __nv_bfloat16*)x, ld, w, logits, T, E, H);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

// parts: six digits 0 .. 2, the first one highest. C a multiple of 8.
int mfb_split3(const float* x, void* out, long long R, int C, int across, int parts, cudaStream_t stream) {
  if (C % 8 || R < 0) { mfb_host::set_error("split3: %lld x %d", R, C); return 1; }
  if (R == 0 || C == 0) return 0;
  SplitArgs a;
  for (int k = 5; k >= 0; --k, parts /= 10) a.part[k] = parts % 10;
  long long blocks = (R * (C / 8) + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  split3_kernel<<<(unsigned)blocks, 256, 0, stream>>>(x, (__nv_bfloat16*)out, R, C, across, a);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int mfb_sum3(const float* x, float* out, long long R, int C, long long ld, long long apart, int groups, long long group_apart,
             cudaStream_t stream) {
  if (C % 4 || ld % 4 || apart % 4 || group_apart % 4 || R < 0) { mfb_host::set_error("sum3: %lld x %d", R, C); return 1; }
  if (R == 0 || C == 0) return 0;
  long long blocks = (R * (C / 4) + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  sum3_kernel<<<(unsigned)blocks, 256, 0, stream>>>(x, out, R, C, ld, apart, groups, group_apart);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // extern "C"
