// Causal softmax attention over the fp32 KV cache, head dim 64 (every GPT-2 size,
// apps/gpt2/gpt2.lisp:38-41).  Cache layout [B, H, T, 64]: one head's history is one contiguous
// stream of 256-byte rows.
//
// Reference semantics (external/llm/layers.lisp:3-5,19-51): cache[:, n:n+s] = k, v;
// S = (q.K^T) * 0.125 + mask; P = softmax(S) with exp(x) = exp2(x * 1/ln2); O = P.V.
#include "common.cuh"

namespace cb {

constexpr float kInvLn2 = 1.0f / 0.6931472f;  // (/ (log 2)) in single float, api/function.lisp:437-440

// ---------------------------------------------------------------------------------------------
// Decode (s = 1): one CTA per (head, sequence).  HBM-bound: K and V rows of this head are each
// read once, 16 lanes x 16 bytes per row, 4 rows in flight per half-warp.  The CTA first stores
// this step's k and v rows at position n, so no separate append kernel runs in decode.
// Scores are kept in shared memory (t <= T floats) and the softmax is the reference's two-pass
// form (max, then exp and sum), not an online rescaling.
// ---------------------------------------------------------------------------------------------
#ifndef ATT_U
#define ATT_U 4  // rows in flight per half-warp
#endif

__global__ void __launch_bounds__(256, 6) attn_decode_kernel(const float *__restrict__ qkv, float *__restrict__ kc,
                                                          float *__restrict__ vc, float *__restrict__ out, int H,
                                                          int T, int n, const int *__restrict__ d_n,
                                                          __nv_bfloat16 *__restrict__ ohi, __nv_bfloat16 *__restrict__ olo,
                                                          const PartIn pin, long long prefetch_bytes) {
  const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  float *kb = kc + ((int64_t)b * H + h) * T * 64;
  float *vb = vc + ((int64_t)b * H + h) * T * 64;
  // Under programmatic dependent launch the first CTAs of this grid become resident while the kernels before it
  // (LayerNorm, the qkv linear) still run, and would idle in the wait below.  The history of this head, rows [0, n)
  // of K and V, was written by earlier steps and depends on nothing in flight, so those CTAs ask for it to be
  // brought into L2 meanwhile (HBM is nearly idle during the linears): one bulk L2 prefetch of up to 32 KB per
  // participating thread.  Only a hint: L2 is coherent, nothing reads through it, and a stale position only changes
  // how much is asked for.  Limited to the streams that together fit `prefetch_bytes` of the 126 MB L2 (measured:
  // 2-5 % of a step; asking for more than ~100 MB, or asking a layer ahead from the LayerNorm kernels, which
  // delays the linears' own weight loads behind the prefetch, made steps slower).
  {
    constexpr long long PIECE = 32 << 10;
    int np = d_n ? *d_n : n;
    np = np < 0 ? 0 : (np > T - 1 ? T - 1 : np);
    const long long stream_bytes = 256ll * np;
    const int pieces = (int)((stream_bytes + PIECE - 1) / PIECE);
    if (tid < 2 * pieces && ((long long)b * H + h + 1) * 2 * 256ll * np <= prefetch_bytes) {
      const int which = tid >= pieces ? 1 : 0, i = tid - which * pieces;
      const char *src = reinterpret_cast<const char *>(which ? vb : kb) + (long long)i * PIECE;
      const long long left = stream_bytes - (long long)i * PIECE;
      const unsigned bytes = (unsigned)(left < PIECE ? left : PIECE);
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
    }
  }
  pdl_enter();
  if (d_n) n = *d_n;  // position kept on the device (decode replayed from a CUDA graph)
  extern __shared__ float smem[];
  float *q = smem;            // 64
  float *part = smem + 64;    // 16 x 64
  float *red = part + 1024;   // 32
  float *sc = red + 32;       // t
  const int d = H * 64, t = n + 1;
  const float *row = qkv + (int64_t)b * 3 * d;
  if (pin.splits > 0) {
    // the qkv linear left split-K partial tiles: sum this head's q, k, v entries here
    if (tid < 192) {
      const int which = tid >> 6, e = tid & 63;
      const float val = partin_load1(pin, b, which * d + h * 64 + e);
      if (which == 0) q[e] = val;
      else (which == 1 ? kb : vb)[(int64_t)n * 64 + e] = val;
    }
  } else if (tid < 64) {
    q[tid] = row[h * 64 + tid];
    kb[(int64_t)n * 64 + tid] = row[d + h * 64 + tid];
    vb[(int64_t)n * 64 + tid] = row[2 * d + h * 64 + tid];
  }
  __syncthreads();
  const int hw = tid >> 4, l16 = tid & 15;
  const float4 q4 = reinterpret_cast<const float4 *>(q)[l16];
  for (int j0 = 0; j0 < t; j0 += 16 * ATT_U) {
    float4 k4[ATT_U];
#pragma unroll
    for (int u = 0; u < ATT_U; ++u) {
      const int j = j0 + u * 16 + hw;
      k4[u] = j < t ? __ldcs(reinterpret_cast<const float4 *>(kb + (int64_t)j * 64) + l16) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < ATT_U; ++u) {
      float p = fmaf(q4.x, k4[u].x, fmaf(q4.y, k4[u].y, fmaf(q4.z, k4[u].z, q4.w * k4[u].w)));
      p += __shfl_xor_sync(0xffffffffu, p, 8);
      p += __shfl_xor_sync(0xffffffffu, p, 4);
      p += __shfl_xor_sync(0xffffffffu, p, 2);
      p += __shfl_xor_sync(0xffffffffu, p, 1);
      const int j = j0 + u * 16 + hw;
      if (l16 == 0 && j < t) sc[j] = p * 0.125f;
    }
  }
  __syncthreads();
  // row max
  float m = -INFINITY;
  for (int j = tid; j < t; j += 256) m = fmaxf(m, sc[j]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((tid & 31) == 0) red[tid >> 5] = m;
  __syncthreads();
  m = red[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) m = fmaxf(m, red[w]);
  __syncthreads();
  float ss = 0.0f;
  for (int j = tid; j < t; j += 256) {
    const float e = exp2f((sc[j] - m) * kInvLn2);
    sc[j] = e;
    ss += e;
  }
  ss = warp_sum(ss);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  ss = red[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) ss += red[w];
  const float inv = 1.0f / ss;
  // O = P.V
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j0 = 0; j0 < t; j0 += 16 * ATT_U) {
    float4 v4[ATT_U];
    float p[ATT_U];
#pragma unroll
    for (int u = 0; u < ATT_U; ++u) {
      const int j = j0 + u * 16 + hw;
      const bool ok = j < t;
      v4[u] = ok ? __ldcs(reinterpret_cast<const float4 *>(vb + (int64_t)j * 64) + l16) : make_float4(0.f, 0.f, 0.f, 0.f);
      p[u] = ok ? sc[j] * inv : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < ATT_U; ++u) {
      acc.x = fmaf(p[u], v4[u].x, acc.x);
      acc.y = fmaf(p[u], v4[u].y, acc.y);
      acc.z = fmaf(p[u], v4[u].z, acc.z);
      acc.w = fmaf(p[u], v4[u].w, acc.w);
    }
  }
  reinterpret_cast<float4 *>(part + hw * 64)[l16] = acc;
  __syncthreads();
  float o = 0.0f;
  if (tid < 64) {
#pragma unroll
    for (int w = 0; w < 16; ++w) o += part[w * 64 + tid];
  }
  if (tid < 64) {
    const int64_t at = (int64_t)b * d + h * 64 + tid;
    if (ohi) {  // split bf16 operand of the projection GEMM
      const __nv_bfloat16 hh = __float2bfloat16_rn(o);
      ohi[at] = hh;
      if (olo) olo[at] = __float2bfloat16_rn(o - __bfloat162float(hh));
    } else {
      out[at] = o;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Decode with few heads and sequences (two CTAs per SM at most): a launch is a few microseconds of dependent latencies, so
// the first FEW_U rows of K and V of every half-warp, which are history and depend on nothing in flight, are in registers before
// the wait for q (early: inside a model's step, where a kernel that waited for everything before the step is already over);
// a half-warp keeps a softmax of its own rows, running where they are more than it loads at once, and the halves meet
// behind one barrier.  A cluster of CTAs may share a history (contiguous parts of the positions); the first CTA joins the
// parts through distributed shared memory.  Below 96 positions one CTA does it, also where the launch, which for a device-side
// position is made for the longest context, has clusters: the cut depends on the position alone, and every entry gives the same
// bits (GPT-2 medium Q4_0, one sequence, us a step at 10 positions: all eight 473, one 436; at 130: 476, two 494).
// us a step with the kernel above (which had clusters too) / this one: XL Q4_0, one sequence at 640 positions 1197 / 1099; medium Q8_0, three
// at 300 896 / 818; medium Q4_0, 18 at 800 1513 / 1210; small fp32, one at 66 265 / 250.
// ---------------------------------------------------------------------------------------------
constexpr int ATT_PARTS = 8;
constexpr int FEW_U = 6;
__host__ __device__ inline int att_parts(int64_t t, int most) { return t >= 96 ? most : 1; }
// where part `rank` of `parts`, a power of two, begins
__device__ __forceinline__ int att_cut(int t, int rank, int parts) { return (int)(((long long)t * rank) >> (__ffs(parts) - 1)); }

template <bool SPLIT>
__global__ void __launch_bounds__(256, 3) attn_decode_few_kernel(const float *__restrict__ qkv, float *__restrict__ kc, float *__restrict__ vc,
                                                                 float *__restrict__ out, int H, int T, int n, const int *__restrict__ d_n,
                                                                 __nv_bfloat16 *__restrict__ ohi, __nv_bfloat16 *__restrict__ olo, const PartIn pin,
                                                                 const int cluster, const bool early) {
  const int h = SPLIT ? blockIdx.x / cluster : blockIdx.x, rank = SPLIT ? blockIdx.x % cluster : 0, b = blockIdx.y, tid = threadIdx.x;
  if (SPLIT) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // "my shared memory may be written to"
  __shared__ __align__(16) float fresh[192];            // q, k, v of this step where they come as partial tiles
  __shared__ __align__(16) float part[8][64];           // each warp's outputs
  __shared__ float2 stat[8];                            // its maximum and sum
  __shared__ float join[SPLIT ? ATT_PARTS * 66 : 1];    // of the first CTA: each part's maximum, sum and 64 outputs
  float *kb = kc + ((int64_t)b * H + h) * T * 64;
  float *vb = vc + ((int64_t)b * H + h) * T * 64;
  const int hw = tid >> 4, l16 = tid & 15, d = H * 64;
  float4 k4[FEW_U], v4[FEW_U];
  int t, parts, j_first, j_end;
  auto place = [&]() {
    t = n + 1;
    parts = SPLIT ? att_parts(t, cluster) : 1;
    j_first = SPLIT ? att_cut(t, rank, parts) : 0;
    j_end = SPLIT ? rank < parts ? att_cut(t, rank + 1, parts) : j_first : t;
  };
  auto load = [&](int j0) {   // rows of the history among the half-warp's next FEW_U
#pragma unroll
    for (int u = 0; u < FEW_U; ++u) {
      const int j = j0 + u * 16 + hw;
      const bool ok = j < j_end && j < n;
      k4[u] = ok ? __ldcs(reinterpret_cast<const float4 *>(kb + (int64_t)j * 64) + l16) : make_float4(0.f, 0.f, 0.f, 0.f);
      v4[u] = ok ? __ldcs(reinterpret_cast<const float4 *>(vb + (int64_t)j * 64) + l16) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  if (early) {
    if (d_n) n = min(max(*d_n, 0), T - 1);  // position kept on the device (decode replayed from a CUDA graph)
    place();
    load(j_first);
    pdl_enter();
  } else {
    pdl_enter();
    if (d_n) n = *d_n;
    place();
    load(j_first);
  }
  if (SPLIT && rank >= parts) return;   // (whole CTAs) one part at this length, whose CTA waits for no other
  const bool newest = !SPLIT || rank == parts - 1;   // position n is in the last part, which is never empty
  const float4 *qp, *kp, *vp;
  if (pin.splits > 0) {
    // the qkv linear left split-K partial tiles: sum this head's q, k, v entries here
    if (tid < (newest ? 192 : 64)) fresh[tid] = partin_load1(pin, b, (tid >> 6) * d + h * 64 + (tid & 63));
    __syncthreads();
    qp = reinterpret_cast<const float4 *>(fresh);
    kp = qp + 16;
    vp = qp + 32;
  } else {
    qp = reinterpret_cast<const float4 *>(qkv + (int64_t)b * 3 * d + h * 64);
    kp = qp + d / 4;
    vp = kp + d / 4;
  }
  const float4 q4 = qp[l16];
  float4 kn = make_float4(0.f, 0.f, 0.f, 0.f), vn = kn;
  if (newest) {
    kn = kp[l16];
    vn = vp[l16];
    if (hw == 0) {
      reinterpret_cast<float4 *>(kb + (int64_t)n * 64)[l16] = kn;
      reinterpret_cast<float4 *>(vb + (int64_t)n * 64)[l16] = vn;
    }
  }
  float m = -INFINITY, ss = 0.0f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j0 = j_first; j0 < j_end; j0 += 16 * FEW_U) {
    if (j0 > j_first) load(j0);
    float p[FEW_U], top = m;
#pragma unroll
    for (int u = 0; u < FEW_U; ++u) {
      const int j = j0 + u * 16 + hw;
      if (j == n) { k4[u] = kn; v4[u] = vn; }
      p[u] = fmaf(q4.x, k4[u].x, fmaf(q4.y, k4[u].y, fmaf(q4.z, k4[u].z, q4.w * k4[u].w)));
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
      for (int u = 0; u < FEW_U; ++u) p[u] += __shfl_xor_sync(0xffffffffu, p[u], o);
#pragma unroll
    for (int u = 0; u < FEW_U; ++u) {
      p[u] = j0 + u * 16 + hw < j_end ? p[u] * 0.125f : -INFINITY;
      top = fmaxf(top, p[u]);
    }
    if (top == -INFINITY) {   // no row yet, or none that counts: but a NaN, which the maximum passes over, does
#pragma unroll
      for (int u = 0; u < FEW_U; ++u) {
        ss += p[u] == p[u] ? 0.0f : p[u];
        acc.x = fmaf(0.0f, v4[u].x, acc.x);
        acc.y = fmaf(0.0f, v4[u].y, acc.y);
        acc.z = fmaf(0.0f, v4[u].z, acc.z);
        acc.w = fmaf(0.0f, v4[u].w, acc.w);
      }
      continue;
    }
    const float keep = exp2f((m - top) * kInvLn2);
    m = top;
    ss *= keep;
    acc.x *= keep; acc.y *= keep; acc.z *= keep; acc.w *= keep;
#pragma unroll
    for (int u = 0; u < FEW_U; ++u) {
      const float e = exp2f((p[u] - top) * kInvLn2);
      ss += e;
      acc.x = fmaf(e, v4[u].x, acc.x);
      acc.y = fmaf(e, v4[u].y, acc.y);
      acc.z = fmaf(e, v4[u].z, acc.z);
      acc.w = fmaf(e, v4[u].w, acc.w);
    }
  }
  {   // the two halves of the warp
    const float mo = __shfl_xor_sync(0xffffffffu, m, 16), top = fmaxf(m, mo), f = m == -INFINITY ? 0.0f : exp2f((m - top) * kInvLn2);
    m = top;
    ss *= f;
    acc.x *= f; acc.y *= f; acc.z *= f; acc.w *= f;
    ss += __shfl_xor_sync(0xffffffffu, ss, 16);
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, 16);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, 16);
    acc.z += __shfl_xor_sync(0xffffffffu, acc.z, 16);
    acc.w += __shfl_xor_sync(0xffffffffu, acc.w, 16);
  }
  if (!(hw & 1)) reinterpret_cast<float4 *>(part[tid >> 5])[l16] = acc;
  if ((tid & 31) == 0) stat[tid >> 5] = make_float2(m, ss);
  __syncthreads();
  float o = 0.0f, sum = 0.0f;
  m = -INFINITY;
  if (tid < 96) {   // (whole warps; 64 of them have an output)
#pragma unroll
    for (int w = 0; w < 8; ++w) m = fmaxf(m, stat[w].x);
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const float2 st = stat[w];
      const float f = st.x == -INFINITY ? 0.0f : exp2f((st.x - m) * kInvLn2);
      sum = fmaf(st.y, f, sum);
      o = fmaf(part[w][tid & 63], f, o);
    }
  }
  if (parts > 1) {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (tid < 66) {
      uint32_t at;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(&join[rank * 66 + tid])), "r"(0));
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(tid < 64 ? o : tid == 64 ? m : sum) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (rank != 0 || tid >= 64) return;
    float top = -INFINITY;   // an empty part has the maximum -inf, the sum 0 and outputs of 0
#pragma unroll
    for (int r = 0; r < ATT_PARTS; ++r) top = fmaxf(top, r < parts ? join[r * 66 + 64] : -INFINITY);
    o = sum = 0.0f;
#pragma unroll
    for (int r = 0; r < ATT_PARTS; ++r) {
      if (r >= parts) break;
      const float mr = join[r * 66 + 64], f = mr == -INFINITY ? 0.0f : exp2f((mr - top) * kInvLn2);
      sum = fmaf(join[r * 66 + 65], f, sum);
      o = fmaf(join[r * 66 + tid], f, o);
    }
  }
  if (tid < 64) {
    o = o / sum;
    const int64_t at = (int64_t)b * d + h * 64 + tid;
    if (ohi) {  // split bf16 operand of the projection GEMM
      const __nv_bfloat16 hh = __float2bfloat16_rn(o);
      ohi[at] = hh;
      if (olo) olo[at] = __float2bfloat16_rn(o - __bfloat162float(hh));
    } else {
      out[at] = o;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Prefill (s > 1): append kernel + tiled causal attention with running max / sum.
// ---------------------------------------------------------------------------------------------
__global__ void kv_append_kernel(const float *__restrict__ qkv, float *__restrict__ kc, float *__restrict__ vc,
                                 int s, int n, int H, int T) {
  pdl_enter();
  const int64_t r = blockIdx.x;  // row of qkv = b*s + i
  const int64_t b = r / s;
  const int i = (int)(r % s);
  const int d4 = H * 16;
  const float4 *row = reinterpret_cast<const float4 *>(qkv) + r * 3 * d4;
  for (int c = threadIdx.x; c < d4; c += blockDim.x) {
    const int h = c >> 4, l = c & 15;
    const int64_t dst = (((b * H + h) * T) + n + i) * 16 + l;
    reinterpret_cast<float4 *>(kc)[dst] = row[d4 + c];
    reinterpret_cast<float4 *>(vc)[dst] = row[2 * d4 + c];
  }
}

constexpr int PF_LD = 68;  // padded leading dimension of the 64x64 tiles (floats)

// One CTA = 64 queries of one (sequence, head); 256 threads as a 16x16 grid, each owning a 4x4
// block of the 64x64 score tile and of the 64x64 output tile.  Q and K tiles are stored
// transposed ([c][row]) so the inner products read float4s without bank conflicts.
__global__ void __launch_bounds__(256) attn_prefill_kernel(const float *__restrict__ qkv, const float *__restrict__ kc,
                                                           const float *__restrict__ vc, float *__restrict__ out,
                                                           int s, int n, int H, int T, __nv_bfloat16 *__restrict__ ohi,
                                                           __nv_bfloat16 *__restrict__ olo) {
  extern __shared__ float smem[];
  pdl_enter();
  float *Qt = smem;                 // [64 c][PF_LD i]
  float *Kt = Qt + 64 * PF_LD;      // [64 c][PF_LD j]
  float *Vs = Kt + 64 * PF_LD;      // [64 j][PF_LD c]
  float *Pt = Vs + 64 * PF_LD;      // [64 j][PF_LD i]
  const int q0 = blockIdx.x * 64, h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x;
  const int d = H * 64, t = n + s;
  const int tx = tid & 15, ty = tid >> 4;
  const int lane = tid & 31, warp = tid >> 5;
  const float *kb = kc + ((int64_t)b * H + h) * T * 64;
  const float *vb = vc + ((int64_t)b * H + h) * T * 64;
  // Q tile, transposed; lane <-> query row, so the shared-memory stores are conflict-free
  for (int it = 0; it < 2; ++it) {
    const int i = lane + 32 * it;
    const bool ok = q0 + i < s;
    const float4 *src = reinterpret_cast<const float4 *>(qkv + ((int64_t)b * s + q0 + i) * 3 * d + h * 64);
    for (int c4 = warp; c4 < 16; c4 += 8) {
      const float4 v = ok ? src[c4] : make_float4(0.f, 0.f, 0.f, 0.f);
      Qt[(4 * c4 + 0) * PF_LD + i] = v.x;
      Qt[(4 * c4 + 1) * PF_LD + i] = v.y;
      Qt[(4 * c4 + 2) * PF_LD + i] = v.z;
      Qt[(4 * c4 + 3) * PF_LD + i] = v.w;
    }
  }
  float m_run[4], l_run[4], o[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    m_run[a] = -INFINITY;
    l_run[a] = 0.0f;
#pragma unroll
    for (int c = 0; c < 4; ++c) o[a][c] = 0.0f;
  }
  const int kend = min(t, n + q0 + 64);  // keys beyond the last query of this tile are masked
  for (int j0 = 0; j0 < kend; j0 += 64) {
    __syncthreads();  // previous tile fully consumed (also orders the Q stores before first use)
    for (int it = 0; it < 2; ++it) {
      const int j = lane + 32 * it;
      const bool ok = j0 + j < t;
      const float4 *src = reinterpret_cast<const float4 *>(kb + (int64_t)(j0 + j) * 64);
      for (int c4 = warp; c4 < 16; c4 += 8) {
        const float4 v = ok ? src[c4] : make_float4(0.f, 0.f, 0.f, 0.f);
        Kt[(4 * c4 + 0) * PF_LD + j] = v.x;
        Kt[(4 * c4 + 1) * PF_LD + j] = v.y;
        Kt[(4 * c4 + 2) * PF_LD + j] = v.z;
        Kt[(4 * c4 + 3) * PF_LD + j] = v.w;
      }
    }
    for (int e = tid; e < 64 * 16; e += 256) {
      const int j = e >> 4, c4 = e & 15;
      const float4 v = j0 + j < t ? reinterpret_cast<const float4 *>(vb + (int64_t)(j0 + j) * 64)[c4]
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4 *>(Vs + j * PF_LD + 4 * c4) = v;
    }
    __syncthreads();
    float sacc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) sacc[a][c] = 0.0f;
#pragma unroll 8
    for (int c = 0; c < 64; ++c) {
      const float4 qv = *reinterpret_cast<const float4 *>(Qt + c * PF_LD + 4 * ty);
      const float4 kv = *reinterpret_cast<const float4 *>(Kt + c * PF_LD + 4 * tx);
      const float qa[4] = {qv.x, qv.y, qv.z, qv.w}, ka[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int e = 0; e < 4; ++e) sacc[a][e] = fmaf(qa[a], ka[e], sacc[a][e]);
    }
    // scale, mask, running softmax (rows = 4*ty + a, shared by the 16 lanes with equal ty)
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int qi = q0 + 4 * ty + a;  // query index within this step
      float mx = -INFINITY;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = j0 + 4 * tx + e;
        float v = sacc[a][e] * 0.125f;
        if (j >= qi + n + 1 || j >= t) v = -INFINITY;
        sacc[a][e] = v;
        mx = fmaxf(mx, v);
      }
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      const float m_new = fmaxf(m_run[a], mx);
      // a row past the end of the sequence, or one whose keys in this tile are all masked while
      // nothing has been seen yet, keeps m_new = -inf: guard the subtraction
      const float m_use = m_new == -INFINITY ? 0.0f : m_new;
      const float corr = exp2f((m_run[a] - m_use) * kInvLn2);
      float rs = 0.0f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float p = exp2f((sacc[a][e] - m_use) * kInvLn2);
        sacc[a][e] = p;
        rs += p;
      }
      rs += __shfl_xor_sync(0xffffffffu, rs, 8);
      rs += __shfl_xor_sync(0xffffffffu, rs, 4);
      rs += __shfl_xor_sync(0xffffffffu, rs, 2);
      rs += __shfl_xor_sync(0xffffffffu, rs, 1);
      l_run[a] = l_run[a] * corr + rs;
      m_run[a] = m_new;
#pragma unroll
      for (int c = 0; c < 4; ++c) o[a][c] *= corr;
    }
    // P tile, transposed: Pt[j][i]
#pragma unroll
    for (int e = 0; e < 4; ++e)
      *reinterpret_cast<float4 *>(Pt + (4 * tx + e) * PF_LD + 4 * ty) =
          make_float4(sacc[0][e], sacc[1][e], sacc[2][e], sacc[3][e]);
    __syncthreads();
#pragma unroll 8
    for (int j = 0; j < 64; ++j) {
      const float4 pv = *reinterpret_cast<const float4 *>(Pt + j * PF_LD + 4 * ty);
      const float4 vv = *reinterpret_cast<const float4 *>(Vs + j * PF_LD + 4 * tx);
      const float pa[4] = {pv.x, pv.y, pv.z, pv.w}, va[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < 4; ++c) o[a][c] = fmaf(pa[a], va[c], o[a][c]);
    }
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int qi = q0 + 4 * ty + a;
    if (qi < s) {
      const float inv = 1.0f / l_run[a];
      float4 r = make_float4(o[a][0] * inv, o[a][1] * inv, o[a][2] * inv, o[a][3] * inv);
      const int64_t at = ((int64_t)b * s + qi) * d + h * 64 + 4 * tx;
      if (ohi) {
        *reinterpret_cast<uint2 *>(ohi + at) = make_uint2(pack_bf16(r.x, r.y), pack_bf16(r.z, r.w));
        if (olo)
          *reinterpret_cast<uint2 *>(olo + at) = make_uint2(pack_bf16(bf16_lo(r.x), bf16_lo(r.y)), pack_bf16(bf16_lo(r.z), bf16_lo(r.w)));
      } else {
        *reinterpret_cast<float4 *>(out + at) = r;
      }
    }
  }
}

int launch_attention(caten_b200_ctx *ctx, const float *qkv, float *kc, float *vc, float *out, int64_t B, int64_t s,
                     int64_t n, int64_t H, int64_t T, const int *d_n, BfOut bf, const PartIn *pending_qkv, int tensor_cores) {
  if (B <= 0 || s <= 0) return 0;
  if (pending_qkv && pending_qkv->splits > 0 && s != 1) return fail(ctx, CATEN_B200_EINVAL, "attention: a pending qkv is only supported for single-token steps");
  if (n < 0 || n + s > T) return fail(ctx, CATEN_B200_EINVAL, "attention: positions [%lld,%lld) outside the cache (T=%lld)", (long long)n, (long long)(n + s), (long long)T);
  if (H > 65535 || B > 65535) return fail(ctx, CATEN_B200_EUNSUPPORTED, "attention: B or H > 65535");
  // (every kernel moves 16 bytes of these at a time; a single token's qkv and output may start at any float)
  if (((uintptr_t)kc | (uintptr_t)vc | (s > 1 ? (uintptr_t)qkv | (uintptr_t)out : 0)) & 15)
    return fail(ctx, CATEN_B200_EINVAL, "attention: the caches, and qkv and out of several tokens, must be 16-byte aligned");
  if (s == 1) {
    // with a device-side position the launch is sized for the longest context the cache allows
    const size_t smem = (64 + 1024 + 32 + (size_t)(d_n ? T : n + 1)) * sizeof(float);
    // one limit, that of the general kernel's scores, whatever kernel runs: a context that one sequence may have is not refused to many
    if (smem > 200 * 1024) return fail(ctx, CATEN_B200_EUNSUPPORTED, "attention: context too long for the decode kernel");
    // CTAs per history: as many as are resident twice per SM at most.  Two are not worth a cluster, whose CTAs start later beside the
    // linear before (us a step, one / two, at 10, 300, 640 and 1000 positions: medium Q4_0, 8 sequences 755 / 811, 895 / 952, 1076 /
    // 1119, 1258 / 1223; XL, 5 sequences 1982 / 2071, 2238 / 2301, 2581 / 2627, 2942 / 2930; small Q8_0, 8 sequences 424 / 423, 467 / 461, 557 / 525, 643 / 579);
    // and behind the fp32 GEMM more waiting CTAs cost that GEMM more than they save (small, 5 sequences, 300 positions: 5684 / 5900 with four).
    int most = 1;
    while (most < ATT_PARTS && B * H * most * 2 <= 2 * ctx->sm_count) most *= 2;
    if (most == 2 || (B > 4 && !tensor_cores)) most = 1;
    const int parts = att_parts(d_n ? T : n + 1, most);
    // (more CTAs are limited by bytes, and the kernel with more of them on an SM is the better one: us a step, few / other: medium Q4_0, 64
    // sequences, 200 positions 1358 / 1316; small Q8_0, 64 at 300 724 / 679; XL Q4_0, 16 at 100 2182 / 2118, but 16 at 800 3093 / 3343)
    // A caller's qkv may start at any float; the few-heads kernel reads it 16 bytes at a time.
    if (B * H > 2 * ctx->sm_count || ((uintptr_t)qkv & 15)) {
      if (smem > 44 * 1024) CB_CUDA(ctx, cudaFuncSetAttribute(attn_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
      launch_k(ctx, attn_decode_kernel, dim3((unsigned)H, (unsigned)B), dim3(256), smem, qkv, kc, vc, out, (int)H, (int)T, (int)n, d_n, bf.hi, bf.lo,
               pending_qkv ? *pending_qkv : PartIn(), ctx->attn_prefetch_bytes);
      CB_LAUNCH_CHECK(ctx, "attn_decode_kernel");
      return 0;
    }
    auto kernel = parts > 1 ? attn_decode_few_kernel<true> : attn_decode_few_kernel<false>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(H * parts), (unsigned)B);
    cfg.blockDim = dim3(256);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[2];
    int na = 0;
    if (parts > 1) {
      at[na].id = cudaLaunchAttributeClusterDimension;
      at[na].val.clusterDim.x = (unsigned)parts;
      at[na].val.clusterDim.y = at[na].val.clusterDim.z = 1;
      ++na;
    }
    if (take_pdl(ctx)) {
      at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[na].val.programmaticStreamSerializationAllowed = 1;
      ++na;
    }
    cfg.attrs = at;
    cfg.numAttrs = na;
    CB_CUDA(ctx, cudaLaunchKernelEx(&cfg, kernel, qkv, (float *)kc, (float *)vc, out, (int)H, (int)T, (int)n, d_n, bf.hi, bf.lo, pending_qkv ? *pending_qkv : PartIn(),
                                    parts, pending_qkv != nullptr));
    CB_LAUNCH_CHECK(ctx, "attn_decode_few_kernel");
    return 0;
  }
  if (d_n) return fail(ctx, CATEN_B200_EINVAL, "attention: a device-side position is only supported for single-token steps");
  if (tensor_cores) {
    const int rc = launch_attention_tc(ctx, qkv, kc, vc, out, B, s, n, H, T, bf);
    if (rc != AT_NO_ROOM) return rc;
  }
  launch_k(ctx, kv_append_kernel, dim3((unsigned)(B * s)), dim3(128), 0, qkv, kc, vc, (int)s, (int)n, (int)H, (int)T);
  CB_LAUNCH_CHECK(ctx, "kv_append_kernel");
  const size_t smem = 4 * 64 * PF_LD * sizeof(float);
  CB_CUDA(ctx, cudaFuncSetAttribute(attn_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch_k(ctx, attn_prefill_kernel, dim3((unsigned)((s + 63) / 64), (unsigned)H, (unsigned)B), dim3(256), smem, 
      qkv, kc, vc, out, (int)s, (int)n, (int)H, (int)T, bf.hi, bf.lo);
  CB_LAUNCH_CHECK(ctx, "attn_prefill_kernel");
  return 0;
}

}  // namespace cb
