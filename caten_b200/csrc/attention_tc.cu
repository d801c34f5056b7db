// Prefill attention (s > 1) on the 5th-generation tensor cores over an fp32 KV cache, for head sizes up
// to 128 (NQ / NE = 64-wide blocks of the query/key / value head), grouped query heads, an optional
// sliding window and a ring-buffered cache (attn_window.cuh).  GPT-2 (head dim 64, a cache
// [B, H, T, 64] that never wraps, no window) is the PLAIN case of NQ = NE = 1.  Same semantics as the SIMT kernels in attention.cu
// (external/llm/layers.lisp:3-5,19-51: S = (q.K^T) * 0.125 + causal mask; P = softmax(S) with
// exp(x) = exp2(x * 1/ln2), two passes: row maximum first, then exp and sum; O = P.V), with both
// contractions as bf16 hi/lo split products accumulated in fp32 (every operand x = x_hi + x_lo;
// q.K^T keeps all four products, P.V drops only lo*lo), so the result stays within about 2^-16
// of the fp32 one.
//
// Two kernels.  attn_tiles_kernel splits the visible keys and values into bf16 hi/lo once per call and leaves them as the
// operand tiles of the second kernel, 64 keys each, byte for byte as they lie in shared memory (128-byte swizzle), so that a
// tile is one contiguous bulk copy; for GPT-2 it also appends the step's keys and values to the cache.  (Every query tile of
// every query head used to convert the same rows again: 32 times for grouped heads at 1024 tokens.)
// attn_prefill_tc_kernel: one CTA = 128 queries of one (sequence, head) = the 128 lanes of tensor memory; keys go in steps
// of 64 (with a window: from the step that holds the first key any of the tile's queries sees).  By warp:
//   warp 8       one lane asks for the K and V tiles of the steps ahead (two stages each)
//   warp 9       issues the scores (Q_hi + Q_lo) . (K_hi + K_lo)^T, into one of two blocks of tensor memory and a step ahead
//                of the softmax, and O[128 x 64 NE] += P_hi.V_hi + P_lo.V_hi + P_hi.V_lo, all dims in one MMA
//   warps 0..7   read their query's scores (warps w and w + 4 share lanes and take 32 keys each), mask, take
//                p = exp2((s - max)/ln2), accumulate the row sum, split p into bf16 hi/lo and write it back to tensor
//                memory as the A operand of the second product
// so that the scores of step i + 1 and the output of step i - 1 are computed while the softmax of step i runs.  The softmax is
// what a step waits for (about 2.5 k cycles against 1.8 k of MMAs); with the phases one after the other, conversion included,
// a step took 11 k.  8 x 1024 tokens, 16 heads of 128 over 4: 378 -> 142 us and 14 us for the tiles; 16 x 512 tokens, 25 heads of 64: 193 us and
// 40 us for the append -> 92 us and 63 us for append and tiles.
// The softmax is single-pass with a lazily moved reference maximum: each step exchanges the
// maximum of its visible scores between the row's two threads; the reference only moves (and O and
// the row sum are rescaled, O by a TMEM load / multiply / store) when a step exceeds it by more
// than AT_TAU, which in causal attention happens in the first steps and then rarely.  Softmax is
// invariant to the reference, so this equals the reference's two-pass form up to rounding.
//
// The mbarrier waits are bounded; when one runs out the CTA records it in the context's status
// word, skips the remaining work and its output, frees its tensor memory and returns.
#include "attn_window.cuh"
#include "tcgen05.cuh"

namespace cb {

namespace {

constexpr float kAtInvLn2 = 1.0f / 0.6931472f;  // (/ (log 2)) in single float, api/function.lisp:437-440
constexpr int AT_Q = 128;                        // queries per CTA (MMA M)
constexpr int AT_K = 64;                         // keys per step
constexpr float AT_TAU = 8.0f;                   // slack of the running maximum, in units of the score
constexpr int AT_SOFTMAX_WARPS = 8, AT_THREADS = (AT_SOFTMAX_WARPS + 2) * 32;
template <int NQ, int NE> struct AtLayout {
  static constexpr int CTAS = NQ == 1 && NE == 1 ? 2 : 1;  // per SM
  // Where one CTA has the SM and its tensor memory to itself the rows of K_hi and K_lo are one operand of 128 rows: two MMAs of
  // 128 columns per 16 dims (an MMA of 64 columns takes hardly less time), whose two halves the softmax adds (16 heads of 128,
  // 8 x 1024 tokens: 183 -> 166 us).  Two CTAs share an SM otherwise, and a block of 128 columns each would leave them one
  // block instead of two (25 heads of 64, 16 x 512 tokens: 136 us with two of 64 columns, 161 us with one of 128).
  static constexpr bool STACK = CTAS == 1;
  // TMEM columns: two blocks of scores, P (hi 32, lo 32), O (64 NE); allocated: a power of two
  static constexpr uint32_t COLS = STACK ? 512 : 256, S_COLS = STACK ? 128 : 64, COL_P = 2 * S_COLS, COL_O = COL_P + 64;
  // Q: per block 128 rows hi, 128 rows lo (16 KB each); K, V: per block 64 rows hi, 64 rows lo (8 KB each), two stages
  static constexpr uint32_t K_BYTES = NQ * 16384, V_BYTES = NE * 16384, TILE = K_BYTES + V_BYTES;
  static constexpr uint32_t OFF_Q = 0, OFF_K = NQ * 32768, OFF_V = OFF_K + 2 * K_BYTES, OFF_MISC = OFF_V + 2 * V_BYTES;
  // tiles + exchange of the rows' maxima (2 steps) + barriers, TMEM slot, abort flag + alignment slack
  static constexpr size_t SMEM = OFF_MISC + 2048 + 160 + 1024;
};
static_assert(2 * (AtLayout<1, 1>::SMEM + 1024) <= 227 * 1024, "two CTAs per SM");
static_assert(AtLayout<2, 2>::SMEM <= 227 * 1024, "one CTA per SM");

// byte offset of 16-byte chunk `chunk` (0..7) of row `row` in a K-major tile with 128-byte rows
// and the 128-byte swizzle (8-row groups of 1024 bytes)
__device__ __forceinline__ uint32_t sw128(int row, int chunk) {
  return (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((chunk ^ (row & 7)) << 4));
}

__device__ __forceinline__ uint4 pack8(const float4 a, const float4 b) {
  return make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
}
__device__ __forceinline__ uint4 pack8_lo(const float4 a, const float4 b, const uint4 hi) {
  return make_uint4(pack_bf16_lo(a.x, a.y, hi.x), pack_bf16_lo(a.z, a.w, hi.y), pack_bf16_lo(b.x, b.y, hi.z), pack_bf16_lo(b.z, b.w, hi.w));
}
// 8 consecutive fp32 of one row -> one chunk of the hi row and one of the lo row
__device__ __forceinline__ void st_split8(unsigned char *tile, int row_hi, int row_lo, int chunk, const float4 a, const float4 b) {
  const uint4 hi = pack8(a, b);
  *reinterpret_cast<uint4 *>(tile + sw128(row_hi, chunk)) = hi;
  *reinterpret_cast<uint4 *>(tile + sw128(row_lo, chunk)) = pack8_lo(a, b, hi);
}

// 2^x by one PTX ex2.approx instruction; results below 2^-126 flush to zero (such probabilities do not
// register in a row sum >= 1/e^8)
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float4 scale4(float4 v, float c) { return make_float4(v.x * c, v.y * c, v.z * c, v.w * c); }

// first 64-key tile that a query of the step sees
__host__ __device__ inline int at_first_tile(const AttnArgs &p) {
  const int first = p.window > 0 ? p.n - p.window + 1 : 0;
  return first > 0 ? first / AT_K : 0;
}

}  // namespace

// One CTA = one tile of one key/value head: 64 rows of K and V -> hi and lo operand tiles; columns past the head are zero, and
// so are rows past the context up to a multiple of 16.  Rows above that are not written: their scores are masked, and the
// second product does not take them (prompts of a dozen tokens would write four times what they hold).  PLAIN (GPT-2): rows of this step come from the projections and go to the cache as well.
template <int NQ, int NE, bool PLAIN>
__global__ void __launch_bounds__(256) attn_tiles_kernel(const AttnArgs p, int b0, uint8_t *__restrict__ tiles) {
  using Lay = AtLayout<NQ, NE>;
  pdl_enter();
  const int g = p.g0 + blockIdx.y, b = b0 + blockIdx.z, t = p.n + p.s, j0 = (at_first_tile(p) + blockIdx.x) * AT_K;
  uint8_t *dst = tiles + (((int64_t)blockIdx.z * p.gn + blockIdx.y) * gridDim.x + blockIdx.x) * Lay::TILE;
  const int64_t head = (int64_t)b * p.G + g;
  const float *kx = !PLAIN && p.kx ? p.kx + b * p.cap * p.kx_ld - p.kx_from : nullptr;   // column c of the key, c >= kx_from
  constexpr int KP = AT_K * NQ * 8, PIECES = KP + AT_K * NE * 8;   // pieces of eight floats
  constexpr int IT = PIECES / 256;
  const int rows = min(AT_K, (t - j0 + 15) / 16 * 16);
  float4 v[IT][2];   // all of this thread's loads are in flight together: the stores below may alias them
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int i = it * 256 + threadIdx.x;
    const bool key = i < KP;
    const int nb = key ? NQ : NE, at = key ? i : i - KP;
    const int row = at / (8 * nb), c8 = at % (8 * nb), j = j0 + row;
    if (row >= rows) continue;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int c = 8 * c8 + 4 * u;
      const float *src = nullptr;
      if (PLAIN) {
        if (j < t) src = j >= p.n ? p.qkv + ((int64_t)b * p.s + j - p.n) * p.ld + (key ? p.k_off : p.v_off) + g * 64 + c : (key ? p.kc : p.vc) + (head * p.cap + j) * 64 + c;
      } else if (j < t && c < (key ? p.Dp : p.Ep)) {
        const int64_t slot = j % p.cap;
        if (key && c >= p.kx_from) src = kx + slot * p.kx_ld + c;
        else src = key ? p.kc + b * p.k_seq + g * p.k_head + slot * p.k_ld + c : p.vc + b * p.v_seq + g * p.v_head + slot * p.v_ld + c;
      }
      v[it][u] = src ? *reinterpret_cast<const float4 *>(src) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int i = it * 256 + threadIdx.x;
    const bool key = i < KP;
    const int nb = key ? NQ : NE, at = key ? i : i - KP;
    const int row = at / (8 * nb), c8 = at % (8 * nb), j = j0 + row;
    if (row >= rows) continue;
    if (PLAIN && j >= p.n && j < t) {
      float4 *keep = reinterpret_cast<float4 *>((key ? p.kc : p.vc) + (head * p.cap + j) * 64 + 8 * c8);
      keep[0] = v[it][0];
      keep[1] = v[it][1];
    }
    st_split8(dst + (key ? 0 : Lay::K_BYTES) + (c8 >> 3) * 16384, row, AT_K + row, c8 & 7, v[it][0], v[it][1]);
  }
}

// PLAIN: heads of exactly 64, no window, a cache that never wraps (GPT-2): the masks' lower ends and
// the zero-filled head columns compile away.
template <int NQ, int NE, bool PLAIN>
__global__ void __launch_bounds__(AT_THREADS, AtLayout<NQ, NE>::CTAS)
attn_prefill_tc_kernel(const AttnArgs p, float qscale, int *status, uint32_t idesc, int b0, const uint8_t *__restrict__ tiles, int ntiles) {
  using Lay = AtLayout<NQ, NE>;
  extern __shared__ unsigned char at_raw[];
  unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(at_raw) + 1023) & ~(uintptr_t)1023);
  float *red = reinterpret_cast<float *>(sm + Lay::OFF_MISC);   // [step & 1][half][row]
  const uint32_t bars = smem_u32(sm + Lay::OFF_MISC + 2048);
  auto k_full = [&](int i) { return bars + 8u * i; };
  auto k_empty = [&](int i) { return bars + 16u + 8u * i; };
  auto v_full = [&](int i) { return bars + 32u + 8u * i; };
  auto v_empty = [&](int i) { return bars + 48u + 8u * i; };
  auto s_full = [&](int i) { return bars + 64u + 8u * i; };
  auto s_empty = [&](int i) { return bars + 80u + 8u * i; };
  const uint32_t p_full = bars + 96u, pv_done = bars + 104u;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + Lay::OFF_MISC + 2048 + 112);
  // [0] some role gave up a wait; [1] never set (for waits that must run their full limit)
  volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + Lay::OFF_MISC + 2048 + 120);
  const int tid = threadIdx.x, lane = tid & 31, warp = warp_index();
  const int quad = warp & 3;  // 32-lane quadrant of tensor memory this warp may access
  const int hf = warp >> 2;   // which half (of a step's keys / of a block's head dims) this thread takes
  const int r = quad * 32 + lane;  // query row within the tile = TMEM lane
  const int q0 = (int)(gridDim.z - 1 - blockIdx.z) * AT_Q;  // of all heads, the tiles with the longest history first
  const int rep = PLAIN ? 1 : p.H / p.G;   // query heads per key/value head
  const int h = p.g0 * rep + blockIdx.x, b = b0 + blockIdx.y;
  const int s = p.s, n = p.n, t = n + s;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(k_full(i), 1);
      mbar_init(k_empty(i), 1);
      mbar_init(v_full(i), 1);
      mbar_init(v_empty(i), 1);
      mbar_init(s_full(i), 1);
      mbar_init(s_empty(i), AT_SOFTMAX_WARPS);
    }
    mbar_init(p_full, AT_SOFTMAX_WARPS);
    mbar_init(pv_done, 1);
    abort_flag[0] = 0;
    abort_flag[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(Lay::COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();   // the barriers are initialised
  pdl_wait();

  const int Dp = PLAIN ? 64 : p.Dp, Ep = PLAIN ? 64 : p.Ep;
  const int W = !PLAIN && p.window > 0 ? p.window : 0x3fffffff;
  const int kend = min(t, n + q0 + AT_Q);  // keys beyond the last query of this tile are masked
  const int kfirst = PLAIN ? 0 : n + q0 - W + 1;       // first key the tile's first query sees
  const int tile0 = kfirst > 0 ? kfirst / AT_K : 0, kbeg = tile0 * AT_K;
  const int nblk = (kend - kbeg + AT_K - 1) / AT_K;    // at least 1
  auto give_up = [&](int code) {
    if (!*abort_flag) { *abort_flag = 1; atomicCAS(status, 0, DEV_WAIT_TIMEOUT); status[1] = code; }
  };

  // the copies of step i; those of the first two steps, whose stages are free, start while Q is converted
  const uint8_t *src0 = tiles + (((int64_t)blockIdx.y * p.gn + blockIdx.x / rep) * ntiles + tile0 - at_first_tile(p)) * Lay::TILE;   // of the key/value head this query head reads
  auto copy_k = [&](int i) {
    const int st = i & 1;
    const uint32_t el = elect_one();
    mbar_expect_tx(k_full(st), Lay::K_BYTES, el);
    bulk_load(smem_u32(sm + Lay::OFF_K) + st * Lay::K_BYTES, src0 + (int64_t)i * Lay::TILE, Lay::K_BYTES, k_full(st), el);
  };
  auto copy_v = [&](int i) {
    const int st = i & 1;
    const uint32_t el = elect_one();
    mbar_expect_tx(v_full(st), Lay::V_BYTES, el);
    bulk_load(smem_u32(sm + Lay::OFF_V) + st * Lay::V_BYTES, src0 + (int64_t)i * Lay::TILE + Lay::K_BYTES, Lay::V_BYTES, v_full(st), el);
  };
  if (warp == 8)
    for (int i = 0; i < min(nblk, 2); ++i) {
      copy_k(i);
      copy_v(i);
    }
  // Q tiles: rows [0,128) hi, [128,256) lo per block; GPT-2's 1/8 score scale is folded in (a power of two: exact)
  if (warp < AT_SOFTMAX_WARPS) {
    // eight lanes a row (a thread's own row, piece by piece, takes 4.9 k cycles)
    const int rq = warp * 16 + (lane >> 3), c8 = lane & 7;
#pragma unroll
    for (int kb_ = 0; kb_ < NQ; ++kb_) {
      float4 v[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = rq + 4 * i, c = 64 * kb_ + 8 * c8;
        const bool okq = q0 + row < s;
        const float4 *src = reinterpret_cast<const float4 *>(p.qkv + ((int64_t)b * s + (okq ? q0 + row : 0)) * p.ld + p.q_off + (int64_t)h * Dp + c);
#pragma unroll
        for (int u = 0; u < 2; ++u) v[i][u] = okq && (PLAIN || c + 4 * u < Dp) ? src[u] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) st_split8(sm + Lay::OFF_Q + kb_ * 32768, rq + 4 * i, 128 + rq + 4 * i, c8, scale4(v[i][0], qscale), scale4(v[i][1], qscale));
    }
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();   // not before this CTA has its tensor memory: the next kernel's CTAs ask for theirs and then wait for this grid

  float m = -INFINITY;  // the row's reference maximum: the same value in both threads of a row
  float lsum = 0.0f;    // this thread's part of the row sum, relative to m
  bool ok = true;
  if (warp == 8) {
    // ---------------- tiles (uniform control flow, one elected lane issues) ----------------
    {
      int ki = min(nblk, 2), vi = ki;   // copies asked for
      for (int i = 2; i < nblk; ++i) {
        const uint32_t ph = ((uint32_t)(i >> 1) & 1u) ^ 1u;
        if (!mbar_wait(k_empty(i & 1), ph, abort_flag)) break;
        copy_k(i);
        ++ki;
        if (!mbar_wait(v_empty(i & 1), ph, abort_flag)) break;
        copy_v(i);
        ++vi;
      }
      if (vi < nblk && lane == 0) give_up(16);
      __syncwarp();
      // the copies this thread started land before the CTA's shared memory is released, whoever gives up
      for (int k = ki > 2 ? ki - 2 : 0; k < ki; ++k) mbar_wait_thread(k_full(k & 1), (uint32_t)(k >> 1) & 1u, abort_flag + 1);
      for (int k = vi > 2 ? vi - 2 : 0; k < vi; ++k) mbar_wait_thread(v_full(k & 1), (uint32_t)(k >> 1) & 1u, abort_flag + 1);
    }
  } else if (warp == 9) {
    // ---------------- MMAs (uniform control flow, one elected lane issues) ----------------
    const uint64_t dq = umma_desc(smem_u32(sm + Lay::OFF_Q)), dk0 = umma_desc(smem_u32(sm + Lay::OFF_K)), dv0 = umma_desc(smem_u32(sm + Lay::OFF_V)) - (1ull << 16) + ((uint64_t)(16384 >> 4) << 16);
    const uint32_t idesc_s = idesc | ((Lay::S_COLS >> 3) << 17);
    // B operand MN-major: V rows (keys) with the dims contiguous; blocks of 64 dims are 16 KB apart (the leading offset)
    const uint32_t idesc_pv = idesc | (1u << 16) | ((uint32_t)(64 * NE >> 3) << 17);
    const int ksteps = Dp / 16;
    auto scores = [&](int i) {   // S of step i
      const int st = i & 1;
      const uint32_t ph = (uint32_t)(i >> 1) & 1u;
      if (!mbar_wait(k_full(st), ph, abort_flag) || !mbar_wait(s_empty(st), ph ^ 1u, abort_flag)) return false;
      tc_fence_after();
      {
        const uint32_t el = elect_one();
        const uint64_t dk = dk0 + (uint64_t)(st * (Lay::K_BYTES >> 4));
        const uint32_t acc = tmem_base + Lay::S_COLS * st;
#pragma unroll
        for (int k = 0; k < 4 * NQ; ++k) {
          if (NQ == 1 || k < ksteps) {
            // 16 bf16 = 32 bytes = 2 descriptor units; a Q block is 32 KB = 2048 units, a K block 16 KB = 1024
            const uint64_t aq = dq + (uint64_t)((k >> 2) * 2048 + 2 * (k & 3)), ak = dk + (uint64_t)((k >> 2) * 1024 + 2 * (k & 3));
            umma_bf16(acc, aq, ak, idesc_s, k > 0 ? 1u : 0u, el);
            umma_bf16(acc, aq + 1024, ak, idesc_s, 1u, el);
            if (!Lay::STACK) {
              umma_bf16(acc, aq, ak + 512, idesc_s, 1u, el);
              umma_bf16(acc, aq + 1024, ak + 512, idesc_s, 1u, el);
            }
          }
        }
        umma_commit(k_empty(st), el);
        umma_commit(s_full(st), el);
      }
      return true;
    };
    ok = scores(0);
    for (int i = 0; i < nblk && ok; ++i) {
      if (i + 1 < nblk && !(ok = scores(i + 1))) break;
      const int st = i & 1;
      ok = mbar_wait(v_full(st), (uint32_t)(i >> 1) & 1u, abort_flag) && mbar_wait(p_full, (uint32_t)i & 1u, abort_flag);
      if (!ok) break;
      tc_fence_after();
      const int groups = (kend - kbeg - i * AT_K + 15) / 16;   // of 16 keys that some query of the tile sees
      {
        const uint32_t el = elect_one();
        const uint32_t acc = tmem_base + Lay::COL_O;
        const uint64_t dv_hi = dv0 + (uint64_t)(st * (Lay::V_BYTES >> 4)), dv_lo = dv_hi + 512;
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
          if (k4 >= groups) break;
          const uint64_t adv = (uint64_t)(64 * 2 * k4);  // 16 keys = 16 rows of 128 bytes = 128 descriptor units
          const uint32_t p_hi = tmem_base + Lay::COL_P + 8 * k4, p_lo = p_hi + 32;
          umma_bf16_ts(acc, p_hi, dv_hi + adv, idesc_pv, (i > 0 || k4 > 0) ? 1u : 0u, el);
          umma_bf16_ts(acc, p_lo, dv_hi + adv, idesc_pv, 1u, el);
          umma_bf16_ts(acc, p_hi, dv_lo + adv, idesc_pv, 1u, el);
        }
        umma_commit(v_empty(st), el);
        umma_commit(pv_done, el);
      }
    }
    if (!ok && lane == 0) give_up(17);
    // the last products are awaited here too: tensor memory is freed below
    if (ok && !mbar_wait(pv_done, (uint32_t)(nblk - 1) & 1u, abort_flag) && lane == 0) give_up(18);
    __syncwarp();
  } else {
    // ---------------- softmax ----------------
    const uint32_t tlane = tmem_base + ((uint32_t)(quad * 32) << 16);
    const int qi = min(q0 + r, s - 1);  // rows past the end of the step mask like the last row (their output is dropped)
    const int jmax = n + qi;            // last visible key of this query (< t)
    const int jmin = jmax - W + 1;      // first visible key (may be negative)
    // the warp's view of a wait; a warp whose wait ran out goes on through the pair barriers and touches nothing else
    auto wait = [&](uint32_t bar, uint32_t ph) {
      if (!ok) return;
      ok = mbar_wait(bar, ph, abort_flag);
      if (!ok && lane == 0) give_up(10);
    };
    auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + quad) : "memory"); };   // warps quad and quad + 4
    for (int i = 0; i < nblk; ++i) {
      const int st = i & 1, j0 = kbeg + i * AT_K;
      uint32_t a[32];
      wait(s_full(st), (uint32_t)(i >> 1) & 1u);
      float mloc = -INFINITY;
      // key e of this thread is visible iff low <= e <= lim
      const int lim = jmax - j0 - 32 * hf, low = jmin - j0 - 32 * hf;
      const bool whole = lim >= 31 && (PLAIN || low <= 0);
      if (ok) {
        tc_fence_after();
        const uint32_t block = tlane + Lay::S_COLS * st + 32 * hf;
        if constexpr (Lay::STACK) {
#pragma unroll
          for (int c = 0; c < 32; c += 16) {
            uint32_t lo[16];
            tmem_ld16(block + c, a + c);
            tmem_ld16(block + 64 + c, lo);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) a[c + e] = __float_as_uint(__uint_as_float(a[c + e]) + __uint_as_float(lo[e]));
          }
        } else {
          tmem_ld16(block, a);
          tmem_ld16(block + 16, a + 16);
          tmem_ld_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_empty(st));
        if (!__all_sync(0xffffffffu, whole)) {   // (only the tiles at the ends of what is visible)
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (e > lim || (!PLAIN && e < low)) a[e] = __float_as_uint(-INFINITY);
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) mloc = fmaxf(mloc, __uint_as_float(a[e]));
      }
      float *rd = red + st * 256;
      rd[hf * 128 + r] = mloc;
      pair_sync();
      if (!ok) continue;
      const float mstep = fmaxf(rd[r], rd[128 + r]);
      // The reference maximum only moves when the step's maximum exceeds it by more than AT_TAU
      // (probabilities then stay below e^AT_TAU, harmless in fp32 / split bf16); when it moves, O and
      // the row sum accumulated so far are rescaled.  Softmax is invariant to the shift, so this is
      // the two-pass result up to rounding.  Without a window step 0 always sees key 0; with one, m stays
      // -inf (and every probability zero) until the row's first visible key.
      const bool move = mstep > m + AT_TAU;  // also true at the first visible key (m = -inf)
      const float m_new = move ? mstep : m;
      const float scale = move ? exp2f((m - m_new) * kAtInvLn2) : 1.0f;
      lsum *= scale;
      m = m_new;
      const float m_ref = m == -INFINITY ? 0.0f : m;   // (nothing visible yet: every score is -inf)
      uint32_t phi[16], plo[16];
      float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float p0 = ex2_approx((__uint_as_float(a[2 * e]) - m_ref) * kAtInvLn2), p1 = ex2_approx((__uint_as_float(a[2 * e + 1]) - m_ref) * kAtInvLn2);
        s0 += p0;
        s1 += p1;
        phi[e] = pack_bf16(p0, p1);
        plo[e] = pack_bf16_lo(p0, p1, phi[e]);
      }
      lsum += s0 + s1;
      if (i > 0) {   // the step before has read P and added to O
        wait(pv_done, (uint32_t)(i - 1) & 1u);
        if (!ok) continue;
        tc_fence_after();
        if (__any_sync(0xffffffffu, move)) {
#pragma unroll
          for (int w = 0; w < NE; ++w) {
            uint32_t o[32];
            tmem_ld16(tlane + Lay::COL_O + 64 * w + 32 * hf, o);
            tmem_ld16(tlane + Lay::COL_O + 64 * w + 32 * hf + 16, o + 16);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * scale);
            tmem_st16(tlane + Lay::COL_O + 64 * w + 32 * hf, o);
            tmem_st16(tlane + Lay::COL_O + 64 * w + 32 * hf + 16, o + 16);
          }
        }
      }
      // key k of the step sits in column k / 2
      tmem_st16(tlane + Lay::COL_P + 16 * hf, phi);
      tmem_st16(tlane + Lay::COL_P + 32 + 16 * hf, plo);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    wait(pv_done, (uint32_t)(nblk - 1) & 1u);
    tc_fence_after();
    float *rd = red + (nblk & 1) * 256;
    rd[hf * 128 + r] = lsum;
    pair_sync();
    // The rows go out through shared memory (every tile has been read), 128 bytes at a time: a thread's own row in pieces of 16
    // bytes took 5.1 k cycles.  16 x 512 tokens, 25 heads of 64, with both: 141 -> 92 us.
    float inv = 1.0f / (rd[r] + rd[128 + r]);
    if (!PLAIN && p.gate_off >= 0 && q0 + r < s) inv *= 1.0f / (1.0f + expf(-p.qkv[((int64_t)b * s + q0 + r) * p.ld + p.gate_off + h]));
    if (ok) {
#pragma unroll
      for (int w = 0; w < NE; ++w) {
        uint32_t a[32];
        tmem_ld16(tlane + Lay::COL_O + 64 * w + 32 * hf, a);
        tmem_ld16(tlane + Lay::COL_O + 64 * w + 32 * hf + 16, a + 16);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float4 v[2];
#pragma unroll
          for (int u = 0; u < 2; ++u)
            v[u] = make_float4(__uint_as_float(a[8 * i + 4 * u]) * inv, __uint_as_float(a[8 * i + 4 * u + 1]) * inv, __uint_as_float(a[8 * i + 4 * u + 2]) * inv, __uint_as_float(a[8 * i + 4 * u + 3]) * inv);
          unsigned char *rows = sm + w * 32768;   // bf16: high parts of 64 dims, 16 KB on the low ones; fp32: dims 0 .. 31, 32 .. 63
          if (p.bf.hi) {
            const uint4 hi = pack8(v[0], v[1]);
            *reinterpret_cast<uint4 *>(rows + sw128(r, 4 * hf + i)) = hi;
            if (p.bf.lo) *reinterpret_cast<uint4 *>(rows + 16384 + sw128(r, 4 * hf + i)) = pack8_lo(v[0], v[1], hi);
          } else {
            *reinterpret_cast<float4 *>(rows + 16384 * hf + sw128(r, 2 * i)) = v[0];
            *reinterpret_cast<float4 *>(rows + 16384 * hf + sw128(r, 2 * i + 1)) = v[1];
          }
        }
      }
    }
    asm volatile("bar.sync 5, 256;" ::: "memory");
    if (!*abort_flag) {
      const int c8 = lane & 7;
#pragma unroll
      for (int w = 0; w < 2 * NE; ++w) {
        const bool bf = p.bf.hi != nullptr;
        if (bf && (w & 1) && !p.bf.lo) continue;
        const int c = bf ? 64 * (w >> 1) + 8 * c8 : 32 * w + 4 * c8;   // first dim of the lane's 16 bytes
        if (!PLAIN && c >= Ep) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = warp * 16 + 4 * i + (lane >> 3);
          if (q0 + row >= s) continue;
          const uint4 v = *reinterpret_cast<const uint4 *>(sm + w * 16384 + sw128(row, c8));
          const int64_t at = ((int64_t)b * s + q0 + row) * p.out_ld + (int64_t)h * Ep + c;
          if (!bf) *reinterpret_cast<uint4 *>(p.out + at) = v;
          else *reinterpret_cast<uint4 *>(((w & 1) ? p.bf.lo : p.bf.hi) + at) = v;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Lay::COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// GPT-2, steps of few tokens: where one or two tiles are all the queries of a head, tiles of keys made by a kernel of their own
// would be read once or twice; here the CTA splits the rows itself.  The step's rows come straight from the projections, and the
// last tile's CTA, which sees all of them, brings them to the cache; older ones come from the cache.  All eight warps do the
// same, step after step of 64 keys:
//   copy the NEXT step's K and V rows into a staging buffer in shared memory (cp.async, in flight during this step's products
//   and softmax); split the current step's into operand tiles as above; one lane issues S = (Q_hi + Q_lo) . (K_hi + K_lo)^T;
//   softmax as above; one lane issues O += P_hi.V_hi + P_lo.V_hi + P_hi.V_lo
// with block-wide barriers between (two CTAs share an SM and one's products run under the other's softmax).
// TMEM columns: [0, 64) scores, [128, 192) P (hi 32, lo 32), [192, 256) O.
// ---------------------------------------------------------------------------------------------
namespace {
constexpr uint32_t A1_COL_S = 0, A1_COL_P = 128, A1_COL_O = 192, A1_COLS = 256;
// Q: 128 rows hi, 128 rows lo; K, V: 64 rows hi, 64 rows lo; staging: raw fp32 rows of 256 bytes, padded by 16, so that threads
// reading one row each spread over all banks
constexpr uint32_t A1_OFF_Q = 0, A1_OFF_K = 32768, A1_OFF_V = A1_OFF_K + 16384, A1_LD = 256 + 16, A1_OFF_SK = A1_OFF_V + 16384, A1_OFF_SV = A1_OFF_SK + AT_K * A1_LD, A1_OFF_MISC = A1_OFF_SV + AT_K * A1_LD;
constexpr size_t A1_SMEM = A1_OFF_MISC + 1024 + 64 + 1024;   // + exchange of the rows' maxima, barrier, TMEM slot, abort flag, alignment slack
static_assert(2 * (A1_SMEM + 1024) <= 227 * 1024, "two CTAs per SM");

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t src_bytes) {  // src_bytes 0: zero fill
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
}  // namespace

__global__ void __launch_bounds__(256, 2) attn_direct_tc_kernel(const AttnArgs p, float qscale, int *status, uint32_t idesc) {
  extern __shared__ unsigned char at_raw[];
  unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(at_raw) + 1023) & ~(uintptr_t)1023);
  float *red = reinterpret_cast<float *>(sm + A1_OFF_MISC);
  const uint32_t bar = smem_u32(sm + A1_OFF_MISC + 1024);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + A1_OFF_MISC + 1024 + 8);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + A1_OFF_MISC + 1024 + 12);
  const int tid = threadIdx.x, lane = tid & 31, warp = warp_index();
  const int quad = warp & 3, hf = warp >> 2, r = quad * 32 + lane;   // quadrant of tensor memory; half of a step's keys or dims; query
  const int ck = tid & 63, cq = tid >> 6;                            // conversion: key row of the step, and which 16 dims
  const int h = blockIdx.x, b = blockIdx.y, q0 = (int)(gridDim.z - 1 - blockIdx.z) * AT_Q, s = p.s, n = p.n, t = n + s;

  if (tid == 0) {
    mbar_init(bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(A1_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot, tlane = tmem_base + ((uint32_t)(quad * 32) << 16);
  pdl_enter();

  const int64_t head = ((int64_t)b * p.G + h) * p.cap * 64;
  float *kb = p.kc + head, *vb = p.vc + head;
  const float *xb = p.qkv + ((int64_t)b * s - n) * p.ld + h * 64;   // row j >= n of the step at xb + j * ld
  const int nblk = (min(t, n + q0 + AT_Q) + AT_K - 1) / AT_K;
  const int jmax = n + min(q0 + r, s - 1);   // last key this query sees (rows past the step's end mask like its last: their output is dropped)

  const uint64_t dq = umma_desc(smem_u32(sm + A1_OFF_Q)), dk = umma_desc(smem_u32(sm + A1_OFF_K)), dv = umma_desc(smem_u32(sm + A1_OFF_V));
  const uint32_t idesc_s = idesc | ((64u >> 3) << 17), idesc_pv = idesc_s | (1u << 16);  // second product: B MN-major, V rows (keys) with the dims contiguous
  uint32_t ph = 0;
  int ok = 1;

  // the 64 rows [j0, j0 + 64) of K and V, zeros past the end of the context; a thread's pieces are 16 rows apart
  const int frow = tid >> 4, fcol = (tid & 15) * 4;
  auto fetch = [&](int j0) {
    const uint32_t dst = smem_u32(sm + A1_OFF_SK + frow * A1_LD + fcol * 4);
    if (j0 + AT_K <= n) {
      const float *k = kb + (int64_t)(j0 + frow) * 64 + fcol, *v = vb + (int64_t)(j0 + frow) * 64 + fcol;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        cp_async16(dst + i * 16 * A1_LD, k + i * 16 * 64, 16u);
        cp_async16(dst + (A1_OFF_SV - A1_OFF_SK) + i * 16 * A1_LD, v + i * 16 * 64, 16u);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int j = j0 + frow + 16 * i;
        const float *k = kb, *v = vb;
        if (j < n) { k += (int64_t)j * 64 + fcol; v += (int64_t)j * 64 + fcol; }
        else if (j < t) { k = xb + (int64_t)j * p.ld + p.k_off + fcol; v = xb + (int64_t)j * p.ld + p.v_off + fcol; }
        cp_async16(dst + i * 16 * A1_LD, k, j < t ? 16u : 0u);
        cp_async16(dst + (A1_OFF_SV - A1_OFF_SK) + i * 16 * A1_LD, v, j < t ? 16u : 0u);
      }
    }
    cp_async_commit();
  };
  auto staged_row = [&](uint32_t off, float4 *v) {  // this thread's 16 dims of its key row
    const float4 *src = reinterpret_cast<const float4 *>(sm + off + ck * A1_LD + 64 * cq);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = src[i];
  };
  // one warp polls the mbarrier; the others park at the block barrier instead of spinning
  auto wait_mma = [&]() {
    if (warp == 0 && !mbar_wait(bar, ph, abort_flag)) {
      ok = 0;
      *abort_flag = 1;
    }
    ph ^= 1u;
    ok = __syncthreads_and(ok);
  };

  fetch(0);
  {   // Q tiles: rows [0,128) hi, [128,256) lo; the score scale 1/8 is folded in (a power of two: exact)
    const float4 *src = reinterpret_cast<const float4 *>(p.qkv + ((int64_t)b * s + (q0 + r < s ? q0 + r : 0)) * p.ld + p.q_off + (int64_t)h * 64);
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = q0 + r < s ? scale4(src[8 * hf + i], qscale) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < 4; ++c) st_split8(sm + A1_OFF_Q, r, 128 + r, 4 * hf + c, v[2 * c], v[2 * c + 1]);
  }
  cp_async_wait_all();
  __syncthreads();  // step 0 of K and V is staged (and the Q tile is written)

  float m = -INFINITY;  // the row's reference maximum: the same value in both threads of a row
  float lsum = 0.0f;    // this thread's part of the row sum, relative to m
  for (int blk = 0; blk < nblk && ok; ++blk) {
    const int j0 = blk * AT_K;
    {
      // split this thread's part of the staged rows in registers, then (once the previous step's P.V has read the V tile and
      // P) store it into the tiles
      float4 kv[4], vv[4];
      staged_row(A1_OFF_SK, kv);
      staged_row(A1_OFF_SV, vv);
      if (q0 + AT_Q >= s && j0 + AT_K > n) {   // rows of this step: to the cache
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = frow + 16 * i, j = j0 + row;
          if (j < n || j >= t) continue;
          const unsigned char *src = sm + A1_OFF_SK + row * A1_LD + fcol * 4;
          *reinterpret_cast<float4 *>(kb + (int64_t)j * 64 + fcol) = *reinterpret_cast<const float4 *>(src);
          *reinterpret_cast<float4 *>(vb + (int64_t)j * 64 + fcol) = *reinterpret_cast<const float4 *>(src + (A1_OFF_SV - A1_OFF_SK));
        }
      }
      uint4 khi[2], klo[2], vhi[2], vlo[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        khi[c] = pack8(kv[2 * c], kv[2 * c + 1]);
        klo[c] = pack8_lo(kv[2 * c], kv[2 * c + 1], khi[c]);
        vhi[c] = pack8(vv[2 * c], vv[2 * c + 1]);
        vlo[c] = pack8_lo(vv[2 * c], vv[2 * c + 1], vhi[c]);
      }
      if (blk > 0) wait_mma();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        *reinterpret_cast<uint4 *>(sm + A1_OFF_K + sw128(ck, 2 * cq + c)) = khi[c];
        *reinterpret_cast<uint4 *>(sm + A1_OFF_K + sw128(64 + ck, 2 * cq + c)) = klo[c];
        *reinterpret_cast<uint4 *>(sm + A1_OFF_V + sw128(ck, 2 * cq + c)) = vhi[c];
        *reinterpret_cast<uint4 *>(sm + A1_OFF_V + 8192 + sw128(ck, 2 * cq + c)) = vlo[c];
      }
    }
    fence_proxy_async();
    tc_fence_before();
    ok = __syncthreads_and(ok);  // tiles complete, staging buffers free
    if (!ok) break;
    if (warp == 0) {  // converged warp, one elected lane: the descriptors stay in uniform registers
      tc_fence_after();
      {
        const uint32_t el = elect_one();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t aq = dq + (uint64_t)(2 * k), ak = dk + (uint64_t)(2 * k);   // 16 bf16 = 32 bytes = 2 descriptor units
          umma_bf16(tmem_base + A1_COL_S, aq, ak, idesc_s, k > 0 ? 1u : 0u, el);
          umma_bf16(tmem_base + A1_COL_S, aq + 1024, ak, idesc_s, 1u, el);
          umma_bf16(tmem_base + A1_COL_S, aq, ak + 512, idesc_s, 1u, el);
          umma_bf16(tmem_base + A1_COL_S, aq + 1024, ak + 512, idesc_s, 1u, el);
        }
        umma_commit(bar, el);
      }
    }
    if (blk + 1 < nblk) fetch(j0 + AT_K);   // (after the MMAs: they are the critical path)
    wait_mma();
    tc_fence_after();
    {
      uint32_t a[32];
      tmem_ld16(tlane + A1_COL_S + 32 * hf, a);
      tmem_ld16(tlane + A1_COL_S + 32 * hf + 16, a + 16);
      tmem_ld_wait();
      const int lim = jmax - j0 - 32 * hf;  // key e of this thread is visible iff e <= lim
      float mloc = -INFINITY;
#pragma unroll
      for (int e = 0; e < 32; ++e)
        if (e <= lim) mloc = fmaxf(mloc, __uint_as_float(a[e]));
      red[hf * 128 + r] = mloc;
      __syncthreads();
      const float mstep = fmaxf(red[r], red[128 + r]);
      const bool move = mstep > m + AT_TAU;  // also true at the first step (m = -inf), which sees key 0
      const float m_new = move ? mstep : m;
      if (blk > 0 && __any_sync(0xffffffffu, move)) {
        const float scale = move ? exp2f((m - m_new) * kAtInvLn2) : 1.0f;
        lsum *= scale;
        uint32_t o[32];
        tmem_ld16(tlane + A1_COL_O + 32 * hf, o);
        tmem_ld16(tlane + A1_COL_O + 32 * hf + 16, o + 16);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * scale);
        tmem_st16(tlane + A1_COL_O + 32 * hf, o);
        tmem_st16(tlane + A1_COL_O + 32 * hf + 16, o + 16);
      }
      m = m_new;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t phi[8], plo[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int e0 = 16 * c + 2 * e;
          const float p0 = e0 <= lim ? ex2_approx((__uint_as_float(a[e0]) - m) * kAtInvLn2) : 0.0f;
          const float p1 = e0 + 1 <= lim ? ex2_approx((__uint_as_float(a[e0 + 1]) - m) * kAtInvLn2) : 0.0f;
          lsum += p0;
          lsum += p1;
          phi[e] = pack_bf16(p0, p1);
          plo[e] = pack_bf16_lo(p0, p1, phi[e]);
        }
        tmem_st8(tlane + A1_COL_P + 16 * hf + 8 * c, phi);   // key k of the step sits in column k / 2
        tmem_st8(tlane + A1_COL_P + 32 + 16 * hf + 8 * c, plo);
      }
    }
    tmem_st_wait();
    tc_fence_before();
    cp_async_wait_all();
    ok = __syncthreads_and(ok);  // P is written; the next step's rows are staged
    if (!ok) break;
    if (warp == 0) {
      tc_fence_after();
      {
        const uint32_t el = elect_one();
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
          const uint64_t adv = (uint64_t)(64 * 2 * k4);  // 16 keys = 16 rows of 128 bytes = 128 descriptor units
          const uint32_t p_hi = tmem_base + A1_COL_P + 8 * k4, p_lo = p_hi + 32;
          umma_bf16_ts(tmem_base + A1_COL_O, p_hi, dv + adv, idesc_pv, (blk > 0 || k4 > 0) ? 1u : 0u, el);
          umma_bf16_ts(tmem_base + A1_COL_O, p_lo, dv + adv, idesc_pv, 1u, el);
          umma_bf16_ts(tmem_base + A1_COL_O, p_hi, dv + 512 + adv, idesc_pv, 1u, el);
        }
        umma_commit(bar, el);
      }
    }
  }
  if (ok) wait_mma();
  cp_async_wait_all();   // (left early: the copies land before the shared memory is released)
  tc_fence_after();
  red[hf * 128 + r] = lsum;
  ok = __syncthreads_and(ok);
  if (ok) {
    const float inv = 1.0f / (red[r] + red[128 + r]);
    uint32_t a[32];
    tmem_ld16(tlane + A1_COL_O + 32 * hf, a);
    tmem_ld16(tlane + A1_COL_O + 32 * hf + 16, a + 16);
    tmem_ld_wait();
    if (q0 + r < s) {
      const int64_t at = ((int64_t)b * s + q0 + r) * p.out_ld + (int64_t)h * 64 + 32 * hf;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(a[8 * i + e]) * inv;
        const float4 v0 = make_float4(v[0], v[1], v[2], v[3]), v1 = make_float4(v[4], v[5], v[6], v[7]);
        if (p.bf.hi) {
          const uint4 hi = pack8(v0, v1);
          *reinterpret_cast<uint4 *>(p.bf.hi + at + 8 * i) = hi;
          if (p.bf.lo) *reinterpret_cast<uint4 *>(p.bf.lo + at + 8 * i) = pack8_lo(v0, v1, hi);
        } else {
          *reinterpret_cast<float4 *>(p.out + at + 8 * i) = v0;
          *reinterpret_cast<float4 *>(p.out + at + 8 * i + 4) = v1;
        }
      }
    }
  } else if (tid == 0) {
    atomicCAS(status, 0, DEV_WAIT_TIMEOUT);
    status[1] = 10;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(A1_COLS) : "memory");
  }
}

template <int NQ, int NE, bool PLAIN = false>
static int launch_at(caten_b200_ctx *ctx, AttnArgs a, float qscale) {
  using Lay = AtLayout<NQ, NE>;
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(AT_Q >> 4) << 24);  // fp32 accumulate, bf16 x bf16, M = 128
  constexpr size_t smem = Lay::SMEM;
  CB_CUDA(ctx, cudaFuncSetAttribute(attn_prefill_tc_kernel<NQ, NE, PLAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int ntiles = (a.n + a.s + AT_K - 1) / AT_K - at_first_tile(a);
  const unsigned qtiles = (unsigned)((a.s + AT_Q - 1) / AT_Q);
  if (qtiles > 65535) return fail(ctx, CATEN_B200_EUNSUPPORTED, "attention: %d tokens in one step", a.s);
  // The tiles are as large as the visible keys and values in fp32 (a prompt of 8192 tokens of GPT-2 XL, the largest portion by
  // default, needs 105 MB).  As many whole sequences are taken at a time as attn_tiles_most or the memory that is free
  // allows, otherwise as many key/value heads of one.
  const size_t per_head = (size_t)ntiles * Lay::TILE, per_seq = per_head * a.G, most = ctx->attn_tiles_most;
  const size_t want = per_seq <= most ? per_seq * (most / per_seq < (size_t)a.B ? most / per_seq : (size_t)a.B) : per_head * (most > per_head ? most / per_head : 1);
  const size_t room = most ? tiles_reserve(ctx, per_head, want) : 0;
  if (room < per_head) return AT_NO_ROOM;
  uint8_t *tiles = (uint8_t *)ctx->attn_tiles.ptr;
  const int group = room >= per_seq ? (int)(room / per_seq < (size_t)a.B ? room / per_seq : (size_t)a.B) : 1;
  const int heads = room >= per_seq ? a.G : (int)(room / per_head);
  for (int b0 = 0; b0 < a.B; b0 += group) {
    const int nb = a.B - b0 < group ? a.B - b0 : group;
    for (a.g0 = 0; a.g0 < a.G; a.g0 += heads) {
      a.gn = a.G - a.g0 < heads ? a.G - a.g0 : heads;
      launch_k(ctx, attn_tiles_kernel<NQ, NE, PLAIN>, dim3((unsigned)ntiles, (unsigned)a.gn, (unsigned)nb), dim3(256), 0, a, b0, tiles);
      CB_LAUNCH_CHECK(ctx, "attn_tiles_kernel");
      launch_k(ctx, attn_prefill_tc_kernel<NQ, NE, PLAIN>, dim3((unsigned)(a.H / a.G * a.gn), (unsigned)nb, qtiles), dim3(AT_THREADS), smem, a, qscale, ctx->d_status, idesc,
               b0, (const uint8_t *)tiles, ntiles);
      CB_LAUNCH_CHECK(ctx, "attn_prefill_tc_kernel");
    }
  }
  return 0;
}

int launch_attention_tc_ex(caten_b200_ctx *ctx, const AttnArgs &args, float qscale) {
  AttnArgs a = args;
  a.fill_strides();
  if (a.Dp > 128 || a.Ep > 128) return fail(ctx, CATEN_B200_EUNSUPPORTED, "attention_tc: head size above 128");
  const bool wq = a.Dp > 64, we = a.Ep > 64;
  if (wq && we) return launch_at<2, 2>(ctx, a, qscale);
  if (wq) return launch_at<2, 1>(ctx, a, qscale);
  if (we) return launch_at<1, 2>(ctx, a, qscale);
  return launch_at<1, 1>(ctx, a, qscale);
}

// Which of GPT-2's steps go without the pass that makes tiles: those of one or two query tiles where the CTAs, one per tile and
// head, fill the GPU, or where the few blocks of keys that each walks through take less than a kernel and its hand-off.  us,
// tiles / direct: 25 heads, 64 sequences, 900 positions before 16 tokens 459 / 307 (append and a kernel like this one: 326), 16 sequences, none before 64 tokens 23 / 16, 1
// sequence, 480 before 64 tokens 21 / 29, 4 sequences, 900 before 64, keys from HBM, 7 less in a step of GPT-2 XL; two tiles: 64 sequences, 480 before 256 627 / 517, 8 sequences 85 / 92, none before 45 / 35.
static bool at_direct(int sm, int64_t heads, int64_t s, int64_t n) {
  const int64_t blocks = (n + s + AT_K - 1) / AT_K;
  const bool some = 16 * heads >= 5 * sm;   // 47 heads on 148 SMs
  if (s <= AT_Q) return heads >= sm || blocks <= (some ? 4 : 2);
  return s <= 2 * AT_Q && (2 * heads >= 5 * sm || blocks <= (some ? 8 : 3));
}

// the step's keys and values are appended to the cache here
int launch_attention_tc(caten_b200_ctx *ctx, const float *qkv, float *kc, float *vc, float *out, int64_t B, int64_t s,
                        int64_t n, int64_t H, int64_t T, BfOut bf) {
  AttnArgs a;
  a.qkv = const_cast<float *>(qkv);
  a.ld = 3 * H * 64;
  a.k_off = H * 64;
  a.v_off = 2 * H * 64;
  a.kc = kc;
  a.vc = vc;
  a.cap = T;
  a.out = out; a.bf = bf; a.out_ld = H * 64;
  a.B = (int)B; a.s = (int)s; a.n = (int)n; a.H = a.G = (int)H;
  a.D = a.Dp = a.E = a.Ep = 64;
  if (at_direct(ctx->sm_count, B * H, s, n)) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(AT_Q >> 4) << 24);   // fp32 accumulate, bf16 x bf16, M = 128
    CB_CUDA(ctx, cudaFuncSetAttribute(attn_direct_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)A1_SMEM));
    launch_k(ctx, attn_direct_tc_kernel, dim3((unsigned)H, (unsigned)B, (unsigned)((s + AT_Q - 1) / AT_Q)), dim3(256), A1_SMEM, a, 0.125f, ctx->d_status, idesc);
    CB_LAUNCH_CHECK(ctx, "attn_direct_tc_kernel");
    return 0;
  }
  return launch_at<1, 1, true>(ctx, a, 0.125f);
}

}  // namespace cb
