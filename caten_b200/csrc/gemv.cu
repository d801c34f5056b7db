// Dequant-GEMV for decode with one to four sequences: y[m, o] = act(sum_k x[m, k] * W[o,k] + bias[o]) + res[m, o]
// (source/nn/linear.lisp:12-17 with few rows).  The packed weights are streamed once with 128-bit loads and
// unpacked in registers; x comes through shared memory, from where a thread keeps its block of it in registers
// (quantised types) or reads it as it goes (fp32 / fp16 / bf16 weights).  fp32 accumulation throughout.
#include "common.cuh"
#include "blocks32.cuh"
#include "gemv_blocks.cuh"

namespace cb {

// The rows of x, M x K4 float4 one after the other, on their way to shared memory: put(f, v, ok) takes float4 f (ok: it exists;
// the whole warp calls it).  All of a thread's loads are under way before it uses the first.
// With a norm every CTA normalises the rows for itself, which costs a linear less than a kernel of its own would (one more
// hand-off).  A row is in the threads' registers meanwhile, SLOTS float4 of each; gamma and beta are there before the wait for x
// (GemvGain).  Each warp has the mean and the squared deviations of its own part, and the parts are joined behind one barrier.
// What counts are latencies (by one warp a row, from shared memory, GPT-2 XL's row took 1.3 to 1.8 us of a linear's 6, with the parts
// joined in a loop over the warps 1.6, so 0.9: a step with 640 positions
// 1370, 1258 and 1198 us).
constexpr int GEMV_NORM_K = 2400;   // the longest row that is normalised: three float4 of each of at least 200 threads (launch_blocked's CTAs have 224)
struct GemvGain {
  float4 g[2], b[2];   // (a third float4 of very long rows is read when it is needed)
  __device__ __forceinline__ void load(const GemvNorm &n, int K4) {
    if (!n.g) return;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = u * blockDim.x + threadIdx.x;
      if (i < K4) {
        g[u] = reinterpret_cast<const float4 *>(n.g)[i];
        b[u] = reinterpret_cast<const float4 *>(n.b)[i];
      }
    }
  }
};

__device__ __forceinline__ void gemv_copy_async(float *to, const float4 *x4, int f) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to + 4 * f)), "l"(x4 + f) : "memory");
}
__device__ __forceinline__ void gemv_copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int SLOTS, int MOST, bool ASYNC, class Put>
__device__ __forceinline__ void gemv_norm_rows(const GemvNorm &n, const GemvGain &gain, const float4 *x4, int M, int K4, Put put, float *to) {
  __shared__ float4 stat[2][16];   // of a warp's part: sum, squared deviations from its mean, mean, elements
  const int tid = threadIdx.x, T = blockDim.x, warp = tid >> 5, lane = tid & 31;
  const float invd = 1.0f / (float)(K4 * 4);
  int have = 0;
#pragma unroll
  for (int u = 0; u < SLOTS; ++u) {
    const int left = K4 - (warp * 32 + u * T);
    have += left <= 0 ? 0 : left < 32 ? left : 32;
  }
  const float cnt = (float)(4 * have), inv = have ? 1.0f / cnt : 0.0f;
  // Several long rows wait where they will lie, a thread's own float4 brought there by itself: the next row in registers is more than
  // there are, and the compiler then stores weights that are still on their way (gemv_dense_kernel).
  constexpr bool STAGED = ASYNC && MOST > 1 && SLOTS > 1;
  const float4 *from = x4;
  if (STAGED) {
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int u = 0; u < SLOTS; ++u)
        if (u * T + tid < K4) gemv_copy_async(to, x4, m * K4 + u * T + tid);
    gemv_copies_wait();
    from = reinterpret_cast<const float4 *>(to);
  }
  float4 v[SLOTS], nx[STAGED ? 1 : SLOTS];
  auto load = [&](int m, float4 *d) {
#pragma unroll
    for (int u = 0; u < SLOTS; ++u) d[u] = m < M && u * T + tid < K4 ? from[m * K4 + u * T + tid] : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  load(0, v);
  for (int m = 0; m < M; ++m) {
    if (MOST > 1 && !STAGED) load(m + 1, nx);
    float sum = 0.0f, sq = 0.0f;
#pragma unroll
    for (int u = 0; u < SLOTS; ++u) sum += (v[u].x + v[u].y) + (v[u].z + v[u].w);
    sum = warp_sum(sum);
    const float mw = sum * inv;
#pragma unroll
    for (int u = 0; u < SLOTS; ++u) {
      const float a = v[u].x - mw, b = v[u].y - mw, c = v[u].z - mw, d = v[u].w - mw;
      sq += u * T + tid < K4 ? (a * a + b * b) + (c * c + d * d) : 0.0f;
    }
    sq = warp_sum(sq);
    if (lane == 0) stat[m & 1][warp] = make_float4(sum, sq, mw, cnt);
    __syncthreads();
    const float4 s = lane < (T >> 5) ? stat[m & 1][lane] : make_float4(0.f, 0.f, 0.f, 0.f);   // at most 16 warps
    float all = s.x;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
    const float u = __shfl_sync(0xffffffffu, all, 0) * invd;
    float dev = s.y + s.w * ((s.z - u) * (s.z - u));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) dev += __shfl_xor_sync(0xffffffffu, dev, o);
    const float rs = 1.0f / sqrtf(__shfl_sync(0xffffffffu, dev, 0) * invd + n.eps);
#pragma unroll
    for (int q = 0; q < SLOTS; ++q) {
      const int i = q * T + tid;
      float4 gg, bb;
      if (q < 2) {
        gg = gain.g[q];
        bb = gain.b[q];
      } else if (i < K4) {
        gg = reinterpret_cast<const float4 *>(n.g)[i];
        bb = reinterpret_cast<const float4 *>(n.b)[i];
      }
      const float4 y = v[q];
      put(m * K4 + i, make_float4(((y.x - u) * rs) * gg.x + bb.x, ((y.y - u) * rs) * gg.y + bb.y, ((y.z - u) * rs) * gg.z + bb.z, ((y.w - u) * rs) * gg.w + bb.w), i < K4);
    }
    if (MOST == 1) break;
    if (STAGED) {
      load(m + 1, v);
      continue;
    }
#pragma unroll
    for (int q = 0; q < SLOTS; ++q) v[q] = nx[q];
  }
}

// MOST: M is at most that.  ASYNC: put is the plain copy to `to`, rows without a norm go there without passing through registers.
// NORM: with the code for rows that have one.
template <int MOST, bool ASYNC, bool NORM, class Put>
__device__ __forceinline__ void gemv_rows_to_shared(const GemvNorm &n, const GemvGain &gain, const float *x, int M, int K4, Put put, float *to = nullptr) {
  const float4 *x4 = reinterpret_cast<const float4 *>(x);
  const int tid = threadIdx.x, T = blockDim.x;
  if (NORM && n.g) {
    if (K4 <= T) gemv_norm_rows<1, MOST, ASYNC>(n, gain, x4, M, K4, put, to);
    else if (K4 <= 2 * T) gemv_norm_rows<2, MOST, ASYNC>(n, gain, x4, M, K4, put, to);
    else gemv_norm_rows<3, MOST, ASYNC>(n, gain, x4, M, K4, put, to);
    return;
  }
  const int total = M * K4;
  if (ASYNC) {
    for (int f = tid; f < total; f += T) gemv_copy_async(to, x4, f);
    gemv_copies_wait();
    return;
  }
  for (int f0 = 0; f0 < total; f0 += 8 * T) {
    float4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int f = f0 + u * T + tid;
      v[u] = f < total ? x4[f] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (f0 + u * T >= total) break;   // (the same for the whole CTA)
      put(f0 + u * T + tid, v[u], f0 + u * T + tid < total);
    }
  }
}

struct GemvArgs {
  const void *qs;
  const __half *d, *m;   // scales; minima (Q4_1, Q5_1)
  const uint32_t *qh;    // fifth code bits (Q5_0, Q5_1)
  const float *x, *bias, *res;
  float *y;
  int act, N, nkb, G, M;
  GemvNorm norm;
};

constexpr int GEMV_MAX_THREADS = 512;
constexpr int GEMV_XPAD = 36;   // floats between the 32-wide blocks of x in shared memory (eight threads' 16-byte reads cover all banks); [32]: the block's sum

__device__ __forceinline__ uint4 ld_stream(const uint4 *p) { return __ldcs(p); }

// Thread t < G*nkb owns column block kb = t / G and row offset ro = t % G (the G threads of a block are neighbours and read
// their x from shared memory together: an eighth to a half of the reads that G passes over all blocks would be); a CTA covers G*RI consecutive rows (RI
// independent 16/32-byte loads in flight per thread), once, or (LOOP) again and again with the next rows' loads ahead.  The
// per-(row, block) partial sums go through shared memory and are added in a fixed order (lane
// strided, then a butterfly), so results do not depend on scheduling.
// A launch is a few microseconds of dependent latencies, so: the packed weights, which depend on no other kernel, are in
// registers before the wait for x; x comes through shared memory (thread by thread from global memory, 128 bytes apart, it
// took 256 L1 wavefronts a warp); small CTAs, three to an SM, leave the next launch room to load its own weights.
// GPT-2 XL Q4_0, one sequence, us a linear inside a step: 6.3 to 7.6 -> 3.0 to 5.0.
template <class BLK, int RI, bool LOOP, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS > 256 ? 1 : LOOP || RI * BLK::WORDS > 16 ? 2 : 3) gemv_blocked_kernel(const GemvArgs a) {
  extern __shared__ float gemv_smem[];
  pdl_launch_dependents();
  constexpr int W = BLK::WORDS;
  const int tid = threadIdx.x, nkb = a.nkb, G = a.G;
  float *xs = gemv_smem;                              // [M][nkb][GEMV_XPAD]
  float *red = gemv_smem + a.M * nkb * GEMV_XPAD;     // two buffers of [G * RI][nkb]
  const bool active = tid < G * nkb;
  const int kb = active ? tid / G : 0, ro = active ? tid - kb * G : 0;
  const uint4 *qs = reinterpret_cast<const uint4 *>(a.qs);
  const int rows_per_iter = G * RI;
  const int64_t stride = (int64_t)gridDim.x * rows_per_iter;

  uint32_t qn[RI][W];
  float scn[RI], mnn[RI];
  uint32_t qhn[RI];
  auto load = [&](int64_t base) {
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const int64_t row = base + i * G + ro;
      const bool ok = active && row < a.N;
      const int64_t bidx = row * nkb + kb;
#pragma unroll
      for (int j = 0; j < W / 4; ++j) {
        const uint4 v = ok ? ld_stream(qs + bidx * (W / 4) + j) : make_uint4(0, 0, 0, 0);
        qn[i][4 * j] = v.x; qn[i][4 * j + 1] = v.y; qn[i][4 * j + 2] = v.z; qn[i][4 * j + 3] = v.w;
      }
      scn[i] = ok ? __half2float(a.d[bidx]) : 0.0f;
      if (BLK::HAS_M) mnn[i] = ok ? __half2float(a.m[bidx]) : 0.0f;
      if (BLK::HAS_QH) qhn[i] = ok ? a.qh[bidx] : 0u;
    }
  };
  int64_t base = (int64_t)blockIdx.x * rows_per_iter;
  load(base);
  GemvGain gain;
  gain.load(a.norm, nkb * 8);
  pdl_wait();
  // lpr lanes (a power of two) add up one row; the first of them finishes it, having asked for bias and residual beforehand
  int lpr = 32;
  while (lpr * rows_per_iter > (int)blockDim.x) lpr >>= 1;
  const int rr = tid / lpr, rl = tid - rr * lpr;
  auto addends = [&](int m, float *b, float *r) {
    const bool has = rl == 0 && rr < rows_per_iter && base + rr < a.N;
    *b = has && a.bias ? a.bias[base + rr] : 0.0f;
    *r = has && a.res ? a.res[(int64_t)m * a.N + base + rr] : 0.0f;
  };
  float bz, rz;
  addends(0, &bz, &rz);
  gemv_rows_to_shared<4, false, true>(a.norm, gain, a.x, a.M, nkb * 8, [&](int f, float4 v, bool ok) {
    float *to = xs + (f >> 3) * GEMV_XPAD;
    if (BLK::SUMS) {
      float s = (v.x + v.y) + (v.z + v.w);
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (ok && (f & 7) == 0) to[32] = s;
    }
    if (ok) *reinterpret_cast<float4 *>(to + (f & 7) * 4) = BLK::stage(v, f & 7);
  });
  __syncthreads();
  BLK blk;
  int buf = 0;
  for (bool again = false; base < a.N; base += stride, again = true) {
    uint32_t q[RI][W], qhc[RI];
    float sc[RI], mn[RI];
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      sc[i] = scn[i];
      mn[i] = BLK::HAS_M ? mnn[i] : 0.0f;
      qhc[i] = BLK::HAS_QH ? qhn[i] : 0u;
#pragma unroll
      for (int j = 0; j < W; ++j) q[i][j] = qn[i][j];
    }
    if (LOOP && base + stride < a.N) load(base + stride);
    for (int m = 0; m < a.M; ++m) {   // rows of x share the packed blocks
#pragma unroll
      for (int i = 0; i < RI; ++i) {
        if (BLK::HAS_QH) asm volatile("" : "+r"(qhc[i]));
#pragma unroll
        for (int j = 0; j < W; ++j) asm volatile("" : "+r"(q[i][j]));   // unpacked again for every m: the codes would not fit unpacked
      }
      if (again || m > 0) addends(m, &bz, &rz);
      if (!again || a.M > 1) {
        float xv[32];
        const float4 *xp = reinterpret_cast<const float4 *>(xs + (m * nkb + kb) * GEMV_XPAD);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 v = xp[i];
          xv[4 * i] = v.x; xv[4 * i + 1] = v.y; xv[4 * i + 2] = v.z; xv[4 * i + 3] = v.w;
        }
        blk.prep(xv, BLK::SUMS ? xs[(m * nkb + kb) * GEMV_XPAD + 32] : 0.0f);
      }
      float *rb = red + buf * rows_per_iter * nkb;
      if (active) {
#pragma unroll
        for (int i = 0; i < RI; ++i) {
          float r;
          if constexpr (BLK::HAS_M || BLK::HAS_QH) r = blk.dotx(q[i], sc[i], mn[i], qhc[i]);
          else r = blk.dot(q[i], sc[i]);
          rb[(i * G + ro) * nkb + kb] = r;
        }
      }
      __syncthreads();
      float s = 0.0f;
      if (rr < rows_per_iter) {
        const float *rp = rb + rr * nkb;
#pragma unroll 4
        for (int k = rl; k < nkb; k += lpr) s += rp[k];
      }
      for (int o = lpr >> 1; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (rl == 0 && rr < rows_per_iter && base + rr < a.N) {
        s = apply_act(a.bias ? s + bz : s, a.act);
        a.y[(int64_t)m * a.N + base + rr] = a.res ? rz + s : s;
      }
      buf ^= 1;
    }
    if (!LOOP) break;
  }
}

// Many rows for one x: the block of x that a thread multiplies is in its registers from the start, and a CTA of 512 threads, one
// to an SM, walks down the rows with the next rows' loads ahead.  Where the rows do not fit the CTAs that are resident at once, this
// is the faster form (us, 20000 x 4128 Q5_1 44 / 55 with the kernel above and as many threads, 16384 x 5632 Q4_0 25 / 28, 4096 x 11008 12.9 / 38; 32000 x 2048 Q5_1 34 / 39).
template <class BLK, int RI>
__global__ void __launch_bounds__(GEMV_MAX_THREADS) gemv_stream_kernel(const GemvArgs a) {
  extern __shared__ float red[];   // two buffers of [G * RI][nkb]
  pdl_launch_dependents();
  constexpr int W = BLK::WORDS;
  const int tid = threadIdx.x, nkb = a.nkb, G = a.G;
  const bool active = tid < G * nkb;
  const int kb = active ? tid % nkb : 0, ro = active ? tid / nkb : 0;
  const uint4 *qs = reinterpret_cast<const uint4 *>(a.qs);
  const int rows_per_iter = G * RI;
  int lpr = 32;   // lanes that add up one row
  while (lpr * rows_per_iter > (int)blockDim.x) lpr >>= 1;
  const int rr = tid / lpr, rl = tid - rr * lpr;
  const int64_t stride = (int64_t)gridDim.x * rows_per_iter;
  uint32_t qn[RI][W], qhn[RI];
  float scn[RI], mnn[RI];
  auto load = [&](int64_t base) {
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const int64_t row = base + i * G + ro, bidx = row * nkb + kb;
      const bool ok = active && row < a.N;
#pragma unroll
      for (int j = 0; j < W / 4; ++j) {
        const uint4 v = ok ? ld_stream(qs + bidx * (W / 4) + j) : make_uint4(0, 0, 0, 0);
        qn[i][4 * j] = v.x; qn[i][4 * j + 1] = v.y; qn[i][4 * j + 2] = v.z; qn[i][4 * j + 3] = v.w;
      }
      scn[i] = ok ? __half2float(a.d[bidx]) : 0.0f;
      if (BLK::HAS_M) mnn[i] = ok ? __half2float(a.m[bidx]) : 0.0f;
      if (BLK::HAS_QH) qhn[i] = ok ? a.qh[bidx] : 0u;
    }
  };
  int64_t base = (int64_t)blockIdx.x * rows_per_iter;
  load(base);
  pdl_wait();
  BLK blk;
  {
    float xv[32], sum = 0.0f;
    const float4 *xp = reinterpret_cast<const float4 *>(a.x + (int64_t)kb * 32);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 v = xp[i], w = BLK::stage(v, i);
      sum += (v.x + v.y) + (v.z + v.w);
      xv[4 * i] = w.x; xv[4 * i + 1] = w.y; xv[4 * i + 2] = w.z; xv[4 * i + 3] = w.w;
    }
    blk.prep(xv, sum);
  }
  for (int buf = 0; base < a.N; base += stride, buf ^= 1) {
    uint32_t q[RI][W], qhc[RI];
    float sc[RI], mn[RI];
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      sc[i] = scn[i];
      mn[i] = BLK::HAS_M ? mnn[i] : 0.0f;
      qhc[i] = BLK::HAS_QH ? qhn[i] : 0u;
#pragma unroll
      for (int j = 0; j < W; ++j) q[i][j] = qn[i][j];
    }
    if (base + stride < a.N) load(base + stride);
    float *rb = red + buf * rows_per_iter * nkb;
    if (active) {
#pragma unroll
      for (int i = 0; i < RI; ++i) {
        float r;
        if constexpr (BLK::HAS_M || BLK::HAS_QH) r = blk.dotx(q[i], sc[i], mn[i], qhc[i]);
        else r = blk.dot(q[i], sc[i]);
        rb[(i * G + ro) * nkb + kb] = r;
      }
    }
    __syncthreads();
    float s = 0.0f;
    if (rr < rows_per_iter) {
      const float *rp = rb + rr * nkb;
#pragma unroll 4
      for (int k = rl; k < nkb; k += lpr) s += rp[k];
    }
    for (int o = lpr >> 1; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (rl == 0 && rr < rows_per_iter && base + rr < a.N) {
      const int64_t row = base + rr;
      s = apply_act(a.bias ? s + a.bias[row] : s, a.act);
      a.y[row] = a.res ? a.res[row] + s : s;
    }
  }
}

// fp32 / fp16 / bf16 weights.  16 bytes of a row as they are stored, and their fp32 values.
template <typename T> struct DenseLoad;
template <> struct DenseLoad<float> {
  static constexpr int VEC = 4;
  __device__ static __forceinline__ void expand(const uint4 &v, float *o) {
    o[0] = __uint_as_float(v.x); o[1] = __uint_as_float(v.y); o[2] = __uint_as_float(v.z); o[3] = __uint_as_float(v.w);
  }
};
template <> struct DenseLoad<__half> {
  static constexpr int VEC = 8;
  __device__ static __forceinline__ void expand(const uint4 &v, float *o) {
    const __half2 *h = reinterpret_cast<const __half2 *>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __half22float2(h[i]);
      o[2 * i] = f.x; o[2 * i + 1] = f.y;
    }
  }
};
template <> struct DenseLoad<__nv_bfloat16> {
  static constexpr int VEC = 8;
  __device__ static __forceinline__ void expand(const uint4 &v, float *o) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[2 * i] = __uint_as_float(w[i] << 16);
      o[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
  }
};

// A launch of these lasts a few microseconds whatever the matrix, so what counts is the chain after the wait for x.  RI rows
// are shared by `ks` warps (vectors of 16 bytes dealt out in turns), as many as let a lane hold its whole part of them:
// GEMV_PRE loads, all asked for before the wait, and the next rows' before the sums of these are reduced.  Up to NR
// rows of x are multiplied with a weight row read once.  Bias and residual are asked for beside x.  GPT-2 small fp32, one
// sequence, us a linear inside a step: one load per lane before the wait and one launch per row of x 6.2, this 3.4.
// blockIdx.y = group of `group_rows` output rows with an input plane of its own (one group: N rows).  EXPERTS: blockIdx.y
// is a (token, expert) pair; expert[pair] says which group of rows it uses, its input is row pair / xplane, its products
// are scaled by weight[pair].
constexpr int GEMV_PRE = 8;

struct GemvDense {
  const void *W;
  const float *x, *bias, *res;
  float *y;
  int act, N, K, M, ks, group_rows;
  int64_t xplane, ygroup, ldy;   // ldy: between the outputs of two rows of x
  const int *expert;
  const float *weight;
  GemvNorm norm;
};

template <typename T, int RI, int NR, bool EXPERTS, bool NORM>
__global__ void __launch_bounds__(256, RI == 2 ? 2 : 3) gemv_dense_kernel(const GemvDense a) {
  constexpr int PRE = GEMV_PRE;
  extern __shared__ float xs[];   // [NR][K]
  __shared__ float part[8][RI * NR];
  const T *W = reinterpret_cast<const T *>(a.W);
  const float *x = a.x, *bias = a.bias, *res = a.res;
  float *y = a.y;
  const int K = a.K;
  int N = a.group_rows;
  float wt = 1.0f;
  if (EXPERTS) {
    pdl_enter();   // which rows to read comes from the kernel before
    W += (int64_t)a.expert[blockIdx.y] * a.group_rows * K;
    x += (int64_t)(blockIdx.y / a.xplane) * K;
    y += (int64_t)blockIdx.y * a.ygroup;
    if (a.weight) wt = a.weight[blockIdx.y];
  } else {
    const int64_t r0 = (int64_t)blockIdx.y * a.group_rows;
    W += r0 * K;
    x += (int64_t)blockIdx.y * a.xplane * K;
    y += (int64_t)blockIdx.y * a.ygroup;
    if (bias) bias += r0;
    if (res) res += r0;
    if (a.N - r0 < N) N = (int)(a.N - r0);
    pdl_launch_dependents();
  }
  constexpr int VEC = DenseLoad<T>::VEC;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ks = a.ks;
  const int slot = warp / ks, share = warp - slot * ks, slots = 8 / ks;
  const int nvec = K / VEC, step = 32 * ks, c0 = share * 32 + lane;
  uint4 w[RI][PRE];
  auto load = [&](int64_t row, int c) {
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
      for (int u = 0; u < PRE; ++u)
        w[i][u] = row + i < N && c + u * step < nvec ? __ldcs(reinterpret_cast<const uint4 *>(W + (row + i) * K) + c + u * step) : make_uint4(0, 0, 0, 0);
  };
  int64_t base = ((int64_t)blockIdx.x * slots + slot) * RI;
  const int64_t stride = (int64_t)gridDim.x * slots * RI;
  load(base, c0);
  GemvGain gain;
  if (!EXPERTS) {
    if (NORM) gain.load(a.norm, K / 4);
    pdl_wait();
  }
  // the lane that finishes output (row base + i, row m of x) is lane i * NR + m of the slot's first warp
  const int fi = lane / NR, fm = lane % NR;
  const bool glu_rows = RI == 2 && act_is_glu(a.act);
  const bool fin = share == 0 && lane < RI * NR && fm < a.M;
  auto addends = [&](int64_t row, float *b, float *r) {
    *b = fin && bias && row + fi < N ? bias[row + fi] : 0.0f;
    *r = fin && res && row + fi < N ? res[fm * a.ldy + row + fi] : 0.0f;
  };
  float bz, rz;
  addends(base, &bz, &rz);
  for (int i = a.M * K / 4 + threadIdx.x; i < NR * K / 4; i += 256) reinterpret_cast<float4 *>(xs)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  gemv_rows_to_shared<NR, true, NORM>(a.norm, gain, x, a.M, K / 4, [&](int f, float4 v, bool ok) { if (ok) reinterpret_cast<float4 *>(xs)[f] = v; }, xs);
  __syncthreads();
  const int64_t rounds = ((int64_t)N + stride - 1) / stride;   // the same for every warp: the slots' warps meet at barriers
  for (int64_t it = 0; it < rounds; ++it) {
    float acc[RI][NR];
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
      for (int m = 0; m < NR; ++m) acc[i][m] = 0.0f;
    for (int c = c0; c - c0 < nvec; c += PRE * step) {
      if (c != c0) load(base, c);
#pragma unroll
      for (int u = 0; u < PRE; ++u) {
        if (c + u * step >= nvec) break;
        float wv[RI][VEC];
#pragma unroll
        for (int i = 0; i < RI; ++i) DenseLoad<T>::expand(w[i][u], wv[i]);
#pragma unroll
        for (int m = 0; m < NR; ++m)
#pragma unroll
          for (int q = 0; q < VEC / 4; ++q) {
            const float4 xv = reinterpret_cast<const float4 *>(xs + (size_t)m * K)[(c + u * step) * (VEC / 4) + q];
#pragma unroll
            for (int i = 0; i < RI; ++i) {   // four products by themselves: a lane that has a row's whole share adds up a long chain
              const float *we = wv[i] + 4 * q;
              acc[i][m] += fmaf(xv.w, we[3], fmaf(xv.z, we[2], fmaf(xv.y, we[1], xv.x * we[0])));
            }
          }
      }
    }
    const int64_t row = base + fi;
    const float b = bz, r = rz;
    base += stride;
    if (it + 1 < rounds) {
      load(base, c0);
      addends(base, &bz, &rz);
    }
    float mine = 0.0f;
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
      for (int m = 0; m < NR; ++m) {
        const float s = warp_sum(acc[i][m]);
        if (lane == i * NR + m) mine = s;
      }
    if (ks > 1) {
      if (lane < RI * NR) part[warp][lane] = mine;
      __syncthreads();
      if (share == 0 && lane < RI * NR)
        for (int q = 1; q < ks; ++q) mine += part[warp + q][lane];
    }
    if (share == 0) {   // (whole warps)
      float s = bias ? mine + b : mine;
      if (EXPERTS) s = s * wt;
      if (glu_rows) {  // rows (base, base + 1) are a (gate, up) pair: base is even
        const float up = __shfl_sync(0xffffffffu, s, (lane + NR) & 31);
        if (lane < NR && fin && row < N) y[fm * a.ldy + (row >> 1)] = glu(a.act, s, up);
      } else if (fin && row < N) {
        s = apply_act(s, a.act);
        if (res) s = r + s;
        y[fm * a.ldy + row] = s;
      }
    }
    if (ks > 1) __syncthreads();   // before the partial sums are written again
  }
}

template <class BLK, int RI, bool LOOP, int THREADS>
static int launch_blocked_t(caten_b200_ctx *ctx, GemvArgs a) {
  a.G = THREADS / a.nkb;
  const int threads = (a.G * a.nkb + 31) / 32 * 32;
  const size_t smem = ((size_t)a.M * a.nkb * GEMV_XPAD + 2 * (size_t)a.G * RI * a.nkb) * sizeof(float);
  auto kernel = gemv_blocked_kernel<BLK, RI, LOOP, THREADS>;
  if (smem > 48 * 1024) CB_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int64_t grid = ((int64_t)a.N + a.G * RI - 1) / (a.G * RI);
  if (LOOP) {
    const int occ = THREADS > 256 || smem > 100 * 1024 ? 1 : 2;
    if (grid > (int64_t)ctx->sm_count * occ) grid = (int64_t)ctx->sm_count * occ;
  }
  launch_k(ctx, kernel, dim3((unsigned)grid), dim3(threads), smem, a);
  CB_LAUNCH_CHECK(ctx, "gemv_blocked_kernel");
  return 0;
}

template <class BLK, int RI>
static int launch_stream_t(caten_b200_ctx *ctx, GemvArgs a) {
  a.G = GEMV_MAX_THREADS / a.nkb;
  const int threads = (a.G * a.nkb + 31) / 32 * 32;
  const size_t smem = 2 * (size_t)a.G * RI * a.nkb * sizeof(float);
  int occ = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, gemv_stream_kernel<BLK, RI>, threads, smem);
  int64_t grid = ((int64_t)a.N + a.G * RI - 1) / (a.G * RI);
  if (grid > (int64_t)ctx->sm_count * (occ < 1 ? 1 : occ)) grid = (int64_t)ctx->sm_count * (occ < 1 ? 1 : occ);
  launch_k(ctx, gemv_stream_kernel<BLK, RI>, dim3((unsigned)grid), dim3(threads), smem, a);
  CB_LAUNCH_CHECK(ctx, "gemv_stream_kernel");
  return 0;
}

template <class BLK>
static int launch_blocked(caten_b200_ctx *ctx, const GemvArgs &a) {
  // a handful of blocks per row: more threads leave fewer rows to each warp's sums (64 x 64: 3.4 us, 4.4 with 256)
  if (a.nkb < 8) return launch_blocked_t<BLK, 1, true, 512>(ctx, a);
  const bool alone = a.M == 1 && !a.norm.g;
  if (a.nkb > 256) {
    const bool deep = (int64_t)a.N >= (int64_t)4 * ctx->sm_count;   // few rows: keep every SM busy with single rows
    if (alone) return deep ? launch_stream_t<BLK, 4>(ctx, a) : launch_stream_t<BLK, 1>(ctx, a);
    return deep ? launch_blocked_t<BLK, 4, true, 512>(ctx, a) : launch_blocked_t<BLK, 1, true, 512>(ctx, a);
  }
  // one pass while the rows fit the resident CTAs (three to an SM where the blocks in flight leave the registers for it) with
  // up to eight loads per thread; more rows: CTAs that go on
  const int64_t slab = (int64_t)(256 / a.nkb) * ctx->sm_count;
  const bool small = (size_t)a.M * a.nkb * GEMV_XPAD * sizeof(float) < 60 * 1024;
  const int deep = 16 / BLK::WORDS;   // loads per thread with three CTAs
  if (a.N <= (small ? 3 : 1) * slab) return launch_blocked_t<BLK, 1, false, 256>(ctx, a);
  if (a.N <= (small ? 3 : 1) * 2 * slab) return launch_blocked_t<BLK, 2, false, 256>(ctx, a);
  if (a.N <= (small ? deep >= 4 ? 3 : 2 : 1) * 3 * slab) return launch_blocked_t<BLK, 3, false, 256>(ctx, a);
  if (a.N <= (small ? deep >= 4 ? 3 : 2 : 1) * 4 * slab) return launch_blocked_t<BLK, 4, false, 256>(ctx, a);
  // (Q8_0: 32000 x 2048 30 us there, 26 here, 20000 x 4128 40 and 38)
  // (Q4: 4096 x 4096 6.5 and 5.9, 11264 x 2048 9.4 and 9.1, 32000 x 2048 18.8 and 19.7, 50257 x 1600 25 and 27)
  if (alone && BLK::WORDS == 4 && (BLK::HAS_QH || a.nkb > 128 || a.N > 24 * slab)) return launch_stream_t<BLK, 4>(ctx, a);
  // over 128 blocks a CTA of 256 threads holds one row at a time (16384 x 5632 Q4_0, 4 rows of x: 143 us, 87 with 512 threads)
  return a.nkb > 128 ? launch_blocked_t<BLK, 4, true, 512>(ctx, a) : launch_blocked_t<BLK, 4, true, 256>(ctx, a);
}

template <typename T, int RI, int NR, bool EXPERTS>
static int launch_dense_t(caten_b200_ctx *ctx, GemvDense g, int groups) {
  const int nvec = g.K / DenseLoad<T>::VEC;
  // warps per RI rows: so many that a lane's share of a row is loaded at once, and more while the CTAs do not fill the
  // GPU twice, every lane still has two vectors and all CTAs stay resident at once (2304 x 768 fp32: with two warps a row 576
  // CTAs on 444 places, 5.2 us; with one 4.4).  Error of a row against 64 bits (2-norm) there 9.3e-8 by two warps, 1.1e-7 by one whose
  // lanes add product by product, 8.9e-8 by one that adds fours; 1024 x 4096 fp16 1.27e-7, 1.59e-7, 1.09e-7.
  int ks = 1;
  const auto ctas_of = [&](int k) { return ((int64_t)g.group_rows * k + 8 * RI - 1) / (8 * RI) * groups; };
  while (ks < 8 && (nvec > 32 * GEMV_PRE * ks ||
                    (nvec > 64 * ks && ctas_of(ks) < 2 * ctx->sm_count && ctas_of(2 * ks) <= (RI == 2 ? 2 : 3) * ctx->sm_count))) ks *= 2;
  g.ks = ks;
  const int64_t ctas = ((int64_t)g.group_rows * ks + 8 * RI - 1) / (8 * RI);
  const size_t smem = (size_t)NR * g.K * sizeof(float);
  // Several rows without a norm run a kernel without its code, whose registers (gamma, beta, a row) made the compiler store weights that
  // are still on their way, i.e. wait for them before the wait for x.  Two short rows keep the common kernel, which the launch before
  // left in the instruction cache (us a step, common / without / by this rule: small f32, two sequences 293 / 297 / 281, medium bf16, two
  // 729 / 740 / 711; XL bf16, two 1924 / 1837 / 1838; large f32, three 1700 / 1556 / 1570, f16, four 1978 / 1900 / 1911, medium
  // f32, four 1010 / 855 / 879; the middle figure with rows of all lengths staged).  One row: small f32 234 / 238.
  const bool bare = NR > 1 && !g.norm.g && (NR == 4 || g.K > 1024);
  auto kernel = bare ? gemv_dense_kernel<T, RI, NR, EXPERTS, NR == 1 && !EXPERTS> : gemv_dense_kernel<T, RI, NR, EXPERTS, !EXPERTS>;
  if (smem > 47 * 1024) CB_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int64_t grid = ((int64_t)ctx->sm_count * (smem > 72 * 1024 || RI == 2 ? 2 : 3) + groups - 1) / groups;   // resident at once
  if (grid > ctas) grid = ctas;
  launch_k(ctx, kernel, dim3((unsigned)grid, (unsigned)groups), dim3(256), smem, g);
  CB_LAUNCH_CHECK(ctx, "gemv_dense_kernel");
  return 0;
}

template <typename T, bool EXPERTS>
static int launch_dense(caten_b200_ctx *ctx, const GemvDense &g, int groups) {
  if (g.K % DenseLoad<T>::VEC) return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemv: cols %d not a multiple of %d", g.K, DenseLoad<T>::VEC);
  // two rows per warp when they are a pair or one row per warp would need more CTAs than are resident
  const bool two = act_is_glu(g.act) || ((int64_t)g.group_rows + 7) / 8 * groups > 4 * ctx->sm_count;
  if constexpr (EXPERTS) return two ? launch_dense_t<T, 2, 1, true>(ctx, g, groups) : launch_dense_t<T, 1, 1, true>(ctx, g, groups);
  else {
    if (g.M == 1) return two ? launch_dense_t<T, 2, 1, false>(ctx, g, groups) : launch_dense_t<T, 1, 1, false>(ctx, g, groups);
    if (g.M == 2) return two ? launch_dense_t<T, 2, 2, false>(ctx, g, groups) : launch_dense_t<T, 1, 2, false>(ctx, g, groups);
    return two ? launch_dense_t<T, 2, 4, false>(ctx, g, groups) : launch_dense_t<T, 1, 4, false>(ctx, g, groups);
  }
}

// M rows of x, 1 to 4
int launch_gemv(caten_b200_ctx *ctx, const caten_b200_weight *w, const float *x, const float *bias,
                const float *res, int act, float *y, int64_t M, LinGroups grp, GemvNorm norm) {
  if (w->rows > 0x7fffffff || w->cols > 0x7fffffff) return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemv: dimension too large");
  const int N = (int)w->rows, K = (int)w->cols;
  if (norm.g && (K % 4 || K > GEMV_NORM_K)) return fail(ctx, CATEN_B200_EUNSUPPORTED, "layernorm: d=%d (need d%%4==0, d<=%d)", K, GEMV_NORM_K);
  if (!type_is_packed(w->type) && (size_t)K * sizeof(float) > 160 * 1024) return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemv: cols=%d too wide", K);
  if (M > 1 && (M > 4 || (size_t)K * 4 * sizeof(float) > 160 * 1024)) {   // rows of x that do not fit shared memory together: one by one
    const int64_t ny = grp.ldy ? grp.ldy : act_is_glu(act) ? N / 2 : N;
    for (int64_t m = 0; m < M; ++m)
      if (int rc = launch_gemv(ctx, w, x + m * K, bias, res ? res + m * ny : nullptr, act, y + m * ny, 1, grp, norm)) return rc;
    return 0;
  }
  if (type_is_packed(w->type)) {
    if (grp.group_rows || act_is_glu(act)) return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemv: input groups and the gated activation take dense weights");
    GemvArgs a;
    a.qs = w->qs; a.d = w->d; a.m = w->m; a.qh = w->qh; a.x = x; a.bias = bias; a.res = res; a.y = y; a.act = act; a.N = N;
    a.nkb = (int)w->nkb; a.M = (int)M; a.norm = norm;
    if (a.nkb > GEMV_MAX_THREADS) return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemv: cols=%d too wide (max %d)", K, GEMV_MAX_THREADS * 32);
    switch (w->type) {
      case CATEN_B200_Q4_0: return launch_blocked<BlkQ4>(ctx, a);
      case CATEN_B200_Q4_1: return launch_blocked<BlkQ41>(ctx, a);
      case CATEN_B200_Q5_0: return launch_blocked<BlkQ5<false>>(ctx, a);
      case CATEN_B200_Q5_1: return launch_blocked<BlkQ5<true>>(ctx, a);
      default: return launch_blocked<BlkQ8>(ctx, a);
    }
  }
  GemvDense g;
  g.W = w->qs; g.x = x; g.bias = bias; g.res = res; g.y = y; g.act = act; g.N = N; g.K = K; g.M = (int)M;
  g.group_rows = grp.group_rows > 0 ? (int)grp.group_rows : N;
  g.xplane = grp.xplane; g.ygroup = grp.ygroup ? grp.ygroup : act_is_glu(act) ? g.group_rows / 2 : g.group_rows;
  g.ldy = grp.ldy ? grp.ldy : act_is_glu(act) ? N / 2 : N;
  g.expert = nullptr; g.weight = nullptr; g.norm = norm;
  const int ng = grp.group_rows > 0 ? (int)((N + grp.group_rows - 1) / grp.group_rows) : 1;
  switch (w->type) {
    case CATEN_B200_F32: return launch_dense<float, false>(ctx, g, ng);
    case CATEN_B200_F16: return launch_dense<__half, false>(ctx, g, ng);
    case CATEN_B200_BF16: return launch_dense<__nv_bfloat16, false>(ctx, g, ng);
    default: return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemv: weight type %d", w->type);
  }
}

int launch_gemv_experts(caten_b200_ctx *ctx, const caten_b200_weight *w, int64_t rows, const float *x, const int *expert, const float *weight,
                        int64_t pairs, int xdiv, int act, float *y) {
  if (pairs <= 0) return 0;
  const int64_t K = w->cols;
  if (w->type != CATEN_B200_BF16 || K % 8 || rows % 2) return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemv: experts take BF16 weights");
  if (K > 40 * 1024 || pairs > 65535) return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemv: cols=%lld or %lld pairs", (long long)K, (long long)pairs);
  GemvDense g;
  g.W = w->qs; g.x = x; g.bias = g.res = nullptr; g.y = y; g.act = act; g.N = g.group_rows = (int)rows; g.K = (int)K; g.M = 1;
  g.xplane = xdiv; g.ygroup = g.ldy = act_is_glu(act) ? rows / 2 : rows; g.expert = expert; g.weight = weight;
  return launch_dense<__nv_bfloat16, true>(ctx, g, (int)pairs);
}

}  // namespace cb
