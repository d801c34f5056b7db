// Tensor-core GEMM for many activation rows (prefill, relu(matmul)):
//   y[m, o] = act(sum_k x[m,k] * W[o,k] + bias[o]) + res[m, o]          (source/nn/linear.lisp:12-17)
// With thousands of rows a weight tile is reused by many activation tiles, so the weights are
// expanded ONCE per call into a bf16 (hi[, lo]) copy in device memory and both operands of the MMA
// then come from shared memory through TMA; nothing is converted inside the GEMM loop.  The kernel
// is persistent (one CTA per SM walks over output tiles) and specialised by warp:
//   warp 0      one lane issues the TMA loads of the W and x tiles into a ring of stages
//   warp 1      issues tcgen05.mma (A = W tile, B = x tile, both K-major with 128-byte swizzle)
//               into one of TWO accumulators in tensor memory (2 x 256 columns)
//   warps 2..17 epilogue: read the other accumulator with tcgen05.ld, add bias, apply the
//               activation and the residual, store — while the next tile's MMAs run
// Tile = 128 output features (TMEM lanes) x 256 rows (TMEM columns); a stage holds 64 k (bf16) or 32 k (split bf16).
// Split-bf16 (NSPLIT = 3) issues W_hi.x_hi + W_lo.x_hi + W_hi.x_lo per k-step, as the decode GEMM.
// PAIR: two CTAs of a cluster work on 256 features x bn rows (cta_group::2): each loads its 128 features and half of the rows
// of x, the even one issues the MMAs for both, and each has the accumulators of its features in its own tensor memory.  Both
// CTAs' loads complete on the leader's barriers, commits arrive in both CTAs, and the epilogues of both free the accumulators.
// EXPERTS (mixture of experts): the rows of x are sorted by expert; expert e's rows [offsets[e], offsets[e + 1]), read on
// the device, are multiplied with its own rows of W.  The tile list is formed from the offsets in every CTA; a row tile
// may reach into the next expert's rows, whose products are not stored.  The row tile is as narrow as the experts' rows
// are few (bn), so that a decode step reads each weight once beside little else.  Products are scaled by the row's weight
// before the activation.
// Every mbarrier wait is bounded: when one runs out the role records it in the status word,
// every role leaves its loop, copies in flight are awaited, tensor memory is freed.
#include "blocks32.cuh"
#include "common.cuh"
#include "tcgen05.cuh"

namespace cb {

constexpr int GD_BM = 128;   // output features per tile (MMA M, TMEM lanes)
constexpr int GD_BN = 256;   // activation rows per tile (MMA N, TMEM columns)
constexpr int GD_BK = 64;    // k granularity of the operands (K % 64 == 0)
// k per stage: 64 (128-byte rows, 128-byte swizzle) in bf16; 32 (64-byte rows, 64-byte swizzle) in split bf16, where a
// 64-k stage of hi and lo tiles is 96 KB and only two would fit: four 48 KB stages keep three loads in flight
template <int NSPLIT> struct GdStage { static constexpr int BK = NSPLIT == 3 ? 32 : 64; };
constexpr int GD_EPI_WARPS = 16;
constexpr int GD_THREADS = (2 + GD_EPI_WARPS) * 32;
constexpr int GD_REGS = 72;  // a thread: what the epilogue would like beyond these is room that the next launch starts in

struct GdArgs {
  const float *bias, *res;
  float *y;
  __nv_bfloat16 *yhi, *ylo;   // when yhi is set the result is written as split bf16 instead of y
  int *status;
  int act, M, N, K;
  int tiles_f, tiles;         // feature tiles per row tile; all tiles
  int stages;
  // output rows [g * group_rows, ..) read input plane g, `xplane` rows after the one before it, and go to columns
  // [g * ygroup, ..) of rows of ldy; a group has tiles_per_group feature tiles, the last one possibly partial
  int group_rows, xplane, ygroup, ldy, tiles_per_group;
  uint32_t idesc;
  int bn;                     // activation rows per tile, 16 or a multiple of 32
  int splits, cps;            // split-K: `splits` work items per tile, each of cps k-stages; their sums go to part
  float *part;                // [split][tile][row of x][feature]; summed by the consumer or splitk_reduce_kernel
  int static_w;               // W depends on no kernel in flight: its first stages are loaded before the wait for x
  uint32_t tmem_cols;         // allocated: the accumulators, rounded up to a power of two
  ExpertRows er;
};

constexpr int GD_MAX_EXPERTS = 1024;
constexpr int GD_EXPAND_ROWS = 1536;   // expanded weights: rows from which every shape runs here
constexpr size_t GD_STAGE_BYTES = 227 * 1024 - 2048 - GD_EPI_WARPS * 2048;
constexpr int GD_SPLIT_ROWS = 512;     // rows up to which k is shared among CTAs

// One output tile: features [f0, f_end), activation rows [m0, m_end), first row of its x tile
struct GdTile {
  int f0, f_end, m0, m_end, x0, shift;
};
// (rank: of a CTA in its pair, which takes 128 features and half of the x rows to load each)
template <bool EXPERTS, bool PAIR>
__device__ __forceinline__ GdTile gd_tile(const GdArgs &a, int tile, const int *first, int rank) {
  GdTile t;
  if (EXPERTS) {   // first[e] = index of expert e's first tile
    int lo = 0, hi = a.er.experts;   // the last e with first[e] <= tile (an expert without rows has no tiles)
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (first[mid] <= tile) lo = mid; else hi = mid;
    }
    const int i = tile - first[lo];
    t.f0 = lo * a.group_rows + (i % a.tiles_f) * GD_BM;
    t.f_end = (lo + 1) * a.group_rows;
    t.m0 = t.x0 = a.er.offsets[lo] + (i / a.tiles_f) * a.bn;
    t.m_end = a.er.offsets[lo + 1];
    t.shift = lo * a.group_rows;
  } else {
    const int f = tile % a.tiles_f, g = f / a.tiles_per_group;
    t.f0 = PAIR ? (2 * f + rank) * GD_BM : g * a.group_rows + (f % a.tiles_per_group) * GD_BM;
    t.f_end = PAIR ? a.N : min(a.N, (g + 1) * a.group_rows);
    t.m0 = (tile / a.tiles_f) * a.bn;
    t.m_end = a.M;
    t.x0 = PAIR ? t.m0 + rank * (a.bn / 2) : t.m0 + g * a.xplane;
    t.shift = PAIR ? 0 : g * (a.group_rows - a.ygroup);
  }
  return t;
}

// ---- pre-pass: operands -> bf16 hi (and lo), K-major --------------------------------------------

__device__ __forceinline__ void store_split8(const float *w, __nv_bfloat16 *hi, __nv_bfloat16 *lo, int64_t at) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    h[e] = pack_bf16(w[2 * e], w[2 * e + 1]);
    l[e] = pack_bf16_lo(w[2 * e], w[2 * e + 1], h[e]);
  }
  *reinterpret_cast<uint4 *>(hi + at) = make_uint4(h[0], h[1], h[2], h[3]);
  if (lo) *reinterpret_cast<uint4 *>(lo + at) = make_uint4(l[0], l[1], l[2], l[3]);
}

// one thread = 8 consecutive weights of a row (a quarter of a 32-wide block)
template <int WT>
__global__ void __launch_bounds__(256) wsplit_kernel(const void *__restrict__ qs, const __half *__restrict__ d,
                                                     const __half *__restrict__ mins, const uint32_t *__restrict__ qh5, int64_t N,
                                                     int64_t K, __nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo) {
  pdl_enter();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t per_row = K / 8;
  if (idx >= N * per_row) return;
  const int64_t row = idx / per_row;
  const int o8 = (int)(idx - row * per_row);
  float w[8];
  load_w8<WT>(qs, d, mins, qh5, row, N, K, K / 32, o8 >> 2, o8 & 3, w);
  store_split8(w, hi, lo, row * K + (int64_t)o8 * 8);
}

// 8 consecutive fp32 of x -> bf16 hi (and lo)
__device__ __forceinline__ void xsplit8(const float *__restrict__ x, int64_t i, __nv_bfloat16 *hi, __nv_bfloat16 *lo) {
  const float4 a = reinterpret_cast<const float4 *>(x)[2 * i], c = reinterpret_cast<const float4 *>(x)[2 * i + 1];
  const float w[8] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
  store_split8(w, hi, lo, i * 8);
}

// x fp32 [M, K] -> bf16 hi (and lo)
__global__ void __launch_bounds__(256) xsplit_kernel(const float *__restrict__ x, int64_t n8, __nv_bfloat16 *__restrict__ hi,
                                                     __nv_bfloat16 *__restrict__ lo) {
  pdl_enter();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n8) xsplit8(x, i, hi, lo);
}

// Both operands of relu(a . b) in one launch: the first `tiles` CTAs bring 64 x 64 tiles of b[K, N] fp32 to [N, K] bf16 hi (and lo)
// through shared memory, the others do as above with a.  4096 x 768 x 3072, split bf16: a launch for each, with two
// bytes a store for b, 10.9 us of 54; so 8.8 of 52.
__global__ void __launch_bounds__(256) operands_split_kernel(const float *__restrict__ b, int K, int N, int tiles_n, int tiles, __nv_bfloat16 *__restrict__ bhi,
                                                             __nv_bfloat16 *__restrict__ blo, const float *__restrict__ x, int64_t n8,
                                                             __nv_bfloat16 *__restrict__ xhi, __nv_bfloat16 *__restrict__ xlo) {
  __shared__ float tile[64][65];
  pdl_enter();
  if ((int)blockIdx.x >= tiles) {
    const int64_t i = (int64_t)(blockIdx.x - tiles) * 256 + threadIdx.x;
    if (i < n8) xsplit8(x, i, xhi, xlo);
    return;
  }
  const int k0 = (int)(blockIdx.x / tiles_n) * 64, n0 = (int)(blockIdx.x % tiles_n) * 64;   // K is a multiple of 64
  const int tn = threadIdx.x & 63, tk = threadIdx.x >> 6;
  float v[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = n0 + tn < N ? b[(int64_t)(k0 + tk + 4 * i) * N + n0 + tn] : 0.0f;
#pragma unroll
  for (int i = 0; i < 16; ++i) tile[tk + 4 * i][tn] = v[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int n = (threadIdx.x >> 3) + 32 * i, k = (threadIdx.x & 7) * 8;
    float w[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) w[e] = tile[k + e][n];
    if (n0 + n < N) store_split8(w, bhi, blo, (int64_t)(n0 + n) * K + k0 + k);
  }
}

// ---- the GEMM -----------------------------------------------------------------------------------

// Epilogue of one 16-row x 32-feature block of a warp.  A thread reads its feature's 16 accumulators (one per
// row) from tensor memory; stored directly that would be 4-byte stores 128 bytes apart per warp instruction,
// which the store path sustains at a fraction of what the MMAs produce.  So the block goes through a 2 KB
// shared-memory tile of the warp and comes back transposed: a lane then owns four consecutive features of
// four rows and moves 16 bytes per instruction (bias, activation, residual and the optional split-bf16
// output are applied on that side).
// The residual of the block, rr, is asked for beforehand (gd_load_res): loads placed between the stores would each wait for
// the one before, since y may be the residual's own memory.  1665 rows, 1024 x 1024, plain bf16: 14.1 us, 10.6 with them ahead.
__device__ __forceinline__ void gd_load_res(const GdArgs &a, float4 *rr, int lane, int64_t o0, bool o_ok, int m_first, int m_end) {
  if (!a.res) return;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int64_t m = (int64_t)m_first + 4 * j + (lane >> 3);
    if (o_ok && m < m_end) rr[j] = *reinterpret_cast<const float4 *>(a.res + m * a.ldy + o0);
  }
}
template <int ACT, bool EXPERTS>
__device__ __forceinline__ void gd_store_block(const GdArgs &a, const float *stg, const float4 *rr, int lane, float4 bias4, int64_t o0, bool o_ok, int m_first, int m_end) {
  const int fg = lane & 7, tr = lane >> 3;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int t = 4 * j + tr;
    const int64_t m = (int64_t)m_first + t;
    if (!o_ok || m >= m_end) continue;
    const float4 acc = *reinterpret_cast<const float4 *>(stg + t * 32 + 4 * fg);
    float v[4] = {acc.x + bias4.x, acc.y + bias4.y, acc.z + bias4.z, acc.w + bias4.w};
    if (EXPERTS && a.er.weight) {
      const float wt = a.er.weight[m];
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = v[e] * wt;
    }
    if (act_is_glu(ACT)) {  // two (gate, up) pairs -> two outputs
      const float g0 = glu(ACT, v[0], v[1]), g1 = glu(ACT, v[2], v[3]);
      const int64_t at2 = m * a.ldy + o0 / 2;
      if (a.yhi) {
        const uint32_t h = pack_bf16(g0, g1);
        *reinterpret_cast<uint32_t *>(a.yhi + at2) = h;
        if (a.ylo) *reinterpret_cast<uint32_t *>(a.ylo + at2) = pack_bf16_lo(g0, g1, h);
      } else {
        *reinterpret_cast<float2 *>(a.y + at2) = make_float2(g0, g1);
      }
      continue;
    }
    const int64_t at = m * a.ldy + o0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (ACT == CATEN_B200_ACT_GELU) v[e] = gelu(v[e]);
      if (ACT == CATEN_B200_ACT_RELU) v[e] = v[e] > 0.0f ? v[e] : 0.0f;
    }
    if (a.res) {
      const float4 r = rr[j];
      v[0] = r.x + v[0]; v[1] = r.y + v[1]; v[2] = r.z + v[2]; v[3] = r.w + v[3];
    }
    if (a.yhi) {
      uint32_t h[2], l[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        h[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
        l[e] = pack_bf16_lo(v[2 * e], v[2 * e + 1], h[e]);
      }
      *reinterpret_cast<uint2 *>(a.yhi + at) = make_uint2(h[0], h[1]);
      if (a.ylo) *reinterpret_cast<uint2 *>(a.ylo + at) = make_uint2(l[0], l[1]);
    } else {
      *reinterpret_cast<float4 *>(a.y + at) = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
}

// K-major operand tile whose rows are BK bf16 wide: 128-byte rows with the 128-byte swizzle (8-row groups 1024 bytes
// apart) or 64-byte rows with the 64-byte swizzle (8-row groups 512 bytes apart)
template <int BK>
__device__ __forceinline__ uint64_t gd_desc(uint32_t saddr) {
  if (BK == 64) return umma_desc(saddr);
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;  // SWIZZLE_64B
  return d;
}

template <int NSPLIT, bool EXPERTS, bool WLO, bool PAIR>
__global__ void __maxnreg__(GD_REGS)
gemm_dense_kernel(const __grid_constant__ CUtensorMap tw_hi, const __grid_constant__ CUtensorMap tw_lo,
                  const __grid_constant__ CUtensorMap tx_hi, const __grid_constant__ CUtensorMap tx_lo, const GdArgs a) {
  constexpr int BK = GdStage<NSPLIT>::BK;
  constexpr uint32_t ROW_BYTES = BK * 2u;
  const int BN = a.bn;
  constexpr uint32_t W_BYTES = GD_BM * ROW_BYTES;
  const uint32_t X_BYTES = (uint32_t)(PAIR ? BN / 2 : BN) * ROW_BYTES;
  const uint32_t STAGE_BYTES = W_BYTES * (WLO ? 2u : 1u) + X_BYTES * (NSPLIT == 3 ? 2u : 1u);
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int S = a.stages;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
  smem += 1024;
  const uint32_t bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (S + s); };
  auto acc_full = [&](int b) { return bar0 + 8u * (2 * S + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (2 * S + 2 + b); };
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * S + 4);
  // [0] some role gave up a wait; [1] never set (for waits that must run their full limit)
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  // stage layout: W_hi, [W_lo,] x_hi[, x_lo]
  const uint32_t stage0 = smem_u32(smem);
  auto st_whi = [&](int s) { return stage0 + (uint32_t)s * STAGE_BYTES; };
  auto st_wlo = [&](int s) { return stage0 + (uint32_t)s * STAGE_BYTES + W_BYTES; };
  auto st_xhi = [&](int s) { return stage0 + (uint32_t)s * STAGE_BYTES + (WLO ? 2u : 1u) * W_BYTES; };
  auto st_xlo = [&](int s) { return st_xhi(s) + X_BYTES; };

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int num_k = a.K / BK;
  const int rank = PAIR ? (int)(blockIdx.x & 1) : 0, worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, workers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  // work item i: tile i % tiles, k-stages [i / tiles * cps, ..) of it
  auto k_of = [&](int z, int *k0) {
    *k0 = z * a.cps;
    return min(num_k - *k0, a.cps);
  };

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full(b), 1);
      mbar_init(acc_empty(b), PAIR ? 2 * GD_EPI_WARPS : GD_EPI_WARPS);
    }
    abort_flag[0] = 0;
    abort_flag[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(a.tmem_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(a.tmem_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();   // both CTAs' barriers are initialised
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();
  if (warp == 0 && lane == 0) {
    tma_prefetch_map(&tw_hi);
    tma_prefetch_map(&tx_hi);
    if (NSPLIT == 3) {
      if (WLO) tma_prefetch_map(&tw_lo);
      tma_prefetch_map(&tx_lo);
    }
  }
  // a stage's bytes, those of both CTAs of a pair, complete on the leader's barrier
  auto expect = [&](int s, uint32_t el) {
    if (rank == 0) mbar_expect_tx(full(s), PAIR ? 2 * STAGE_BYTES : STAGE_BYTES, el);
  };
  auto load = [&](uint32_t dst, const CUtensorMap *map, uint32_t bar, int x, int y, uint32_t el) {
    if (PAIR) tma_load_2d_pair(dst, map, bar, x, y, el);
    else tma_load_2d(dst, map, bar, x, y, el);
  };
  // Weights that no kernel writes are on their way before the wait below: in a decode step that is most of what this CTA
  // reads, and it arrives while the kernel that produces x still runs.
  int ahead = 0;   // stages whose W tiles have been asked for
  if (!EXPERTS && a.static_w && warp == 0) {
    const GdTile t = gd_tile<EXPERTS, PAIR>(a, worker % a.tiles, nullptr, rank);
    int k0;
    const int nk = k_of(worker / a.tiles, &k0);
    for (; ahead < nk && ahead < S; ++ahead) {
      const uint32_t el = elect_one();
      expect(ahead, el);
      load(st_whi(ahead), &tw_hi, full(ahead), (k0 + ahead) * BK, t.f0, el);
    }
  }
  // the activations, the residual and (otherwise) the weights were written by preceding kernels
  pdl_wait();
  int tiles = a.tiles;
  int *first = reinterpret_cast<int *>(smem + (size_t)S * STAGE_BYTES + GD_EPI_WARPS * 2048);   // EXPERTS: [experts + 1]
  if (EXPERTS) {
    if (warp == 0) {
      int sum = 0;
      for (int e0 = 0; e0 < a.er.experts; e0 += 32) {
        const int e = e0 + lane;
        const int mine = e < a.er.experts ? (a.er.offsets[e + 1] - a.er.offsets[e] + BN - 1) / BN * a.tiles_f : 0;
        int inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int up = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += up;
        }
        if (e < a.er.experts) first[e] = sum + inc - mine;
        sum += __shfl_sync(0xffffffffu, inc, 31);
      }
      if (lane == 0) first[a.er.experts] = sum;
    }
    __syncthreads();
    tiles = first[a.er.experts];
  }
  const int items = tiles * a.splits;

  if (warp == 0) {
    // ---------------- TMA producer (uniform control flow, one elected lane issues) ----------------
    int issued = 0, s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int item = worker; item < items && ok; item += workers) {
      const int tile = item % tiles;
      const GdTile t = gd_tile<EXPERTS, PAIR>(a, tile, first, rank);
      int k0;
      const int nk = k_of(item / tiles, &k0);
      for (int kc = k0; kc < k0 + nk; ++kc) {
        if (!mbar_wait(empty(s), ph ^ 1u, abort_flag)) {
          if (lane == 0 && !*abort_flag) { *abort_flag = 1; atomicCAS(a.status, 0, DEV_WAIT_TIMEOUT); a.status[1] = 11; a.status[2] = tile; }
          ok = false;
          break;
        }
        const uint32_t el = elect_one();
        if (issued >= ahead) {
          expect(s, el);
          load(st_whi(s), &tw_hi, full(s), kc * BK, t.f0, el);
        }
        if (WLO) load(st_wlo(s), &tw_lo, full(s), kc * BK, t.f0, el);
        load(st_xhi(s), &tx_hi, full(s), kc * BK, t.x0, el);
        if (NSPLIT == 3) load(st_xlo(s), &tx_lo, full(s), kc * BK, t.x0, el);
        ++issued;
        if (++s == S) { s = 0; ph ^= 1u; }
      }
    }
    __syncwarp();
    if (*abort_flag) {
      // let the copies this warp started land before the CTA's shared memory is released (those of a pair's second CTA
      // complete on the other's barrier: they are given a millisecond, a thousand times what a load takes)
      if (PAIR)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
      else
        for (int i = issued > S ? issued - S : 0; i < issued; ++i) mbar_wait_thread(full(i % S), (uint32_t)(i / S) & 1u, abort_flag + 1);
    }
  } else if (warp == 1) {
    if (rank == 0) {
    // ---------------- MMA issuer (uniform control flow, one elected lane issues) ----------------
    auto mma = [&](uint32_t acc, uint64_t da, uint64_t db, uint32_t accumulate, uint32_t el) {
      if (PAIR) umma_bf16_pair(acc, da, db, a.idesc, accumulate, el);
      else umma_bf16(acc, da, db, a.idesc, accumulate, el);
    };
    auto commit = [&](uint32_t bar, uint32_t el) {
      if (PAIR) umma_commit_pair(bar, el);
      else umma_commit(bar, el);
    };
    int s = 0, it = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int item = worker; item < items && ok; item += workers, ++it) {
      const int b = it & 1, tile = item % tiles;
      int k0;
      const int nk = k_of(item / tiles, &k0);
      // the epilogue has drained this accumulator (first use of each passes at once)
      if (!mbar_wait(acc_empty(b), (((uint32_t)it >> 1) & 1u) ^ 1u, abort_flag)) {
        if (lane == 0 && !*abort_flag) { *abort_flag = 1; atomicCAS(a.status, 0, DEV_WAIT_TIMEOUT); a.status[1] = 12; a.status[2] = tile; }
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t acc = tmem_base + (uint32_t)(b * BN);
      for (int kc = 0; kc < nk; ++kc) {
        if (!mbar_wait(full(s), ph, abort_flag)) {
          if (lane == 0 && !*abort_flag) { *abort_flag = 1; atomicCAS(a.status, 0, DEV_WAIT_TIMEOUT); a.status[1] = 13; a.status[2] = tile; }
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t dwh = gd_desc<BK>(st_whi(s)), dwl = gd_desc<BK>(st_wlo(s));
        const uint64_t dxh = gd_desc<BK>(st_xhi(s)), dxl = gd_desc<BK>(st_xlo(s));
        const uint32_t el = elect_one();
#pragma unroll
        for (int k4 = 0; k4 < BK / 16; ++k4) {
          const uint64_t adv = (uint64_t)(k4 * 2);  // 16 bf16 = 32 bytes = 2 descriptor units
          mma(acc, dwh + adv, dxh + adv, (kc > 0 || k4 > 0) ? 1u : 0u, el);
          if (NSPLIT == 3) {
            if (WLO) mma(acc, dwl + adv, dxh + adv, 1u, el);
            mma(acc, dwh + adv, dxl + adv, 1u, el);
          }
        }
        commit(empty(s), el);  // frees the stage when these MMAs have read it
        if (++s == S) { s = 0; ph ^= 1u; }
      }
      if (ok) commit(acc_full(b), elect_one());
    }
    }
  } else {
    // ---------------- epilogue ----------------
    // a warp reaches the TMEM lanes of quadrant (warp % 4); the four warps of a quadrant take blocks of 16 columns in turns
    // (with two warps per quadrant the epilogue was the longest part of a launch of one or two tiles per CTA: the linears of
    // 1665 rows of width 1024 took 25.8 us each, with four 21.4 us)
    const int quad = warp & 3, turn = (warp - 2) >> 2;
    float *stg = reinterpret_cast<float *>(smem + (size_t)S * STAGE_BYTES) + (warp - 2) * 512;  // 16 rows x 32 features
    int it = 0;
    bool ok = true;
    for (int item = worker; item < items && ok; item += workers, ++it) {
      const int b = it & 1, tile = item % tiles;
      const GdTile t = gd_tile<EXPERTS, PAIR>(a, tile, first, rank);
      // after the transpose a lane owns features o0 .. o0 + 3 (N % 4 == 0: all inside or all outside)
      const int64_t o0 = (int64_t)t.f0 + quad * 32 + 4 * (lane & 7);
      const bool o_ok = o0 < t.f_end;
      const int64_t oc = o0 - t.shift;   // output column
      float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f);
      if (a.bias && o_ok) bias4 = *reinterpret_cast<const float4 *>(a.bias + o0);
      float4 rr[4];
      if (16 * turn < BN) gd_load_res(a, rr, lane, oc, o_ok, t.m0 + 16 * turn, t.m_end);
      // (by all lanes: sixteen warps whose first lane alone polls slow the issuing warp down)
      if (!mbar_wait(acc_full(b), ((uint32_t)it >> 1) & 1u, abort_flag)) {
        if (lane == 0 && !*abort_flag) { *abort_flag = 1; atomicCAS(a.status, 0, DEV_WAIT_TIMEOUT); a.status[1] = 14; a.status[2] = tile; }
        ok = false;
        break;
      }
      __syncwarp();
      tc_fence_after();
      const uint32_t trow = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(b * BN);
      for (int c = 16 * turn; c < BN; c += 4 * GD_EPI_WARPS) {
        if (t.m0 + c >= t.m_end) break;
        if (!EXPERTS && a.part) {   // sums of this share of k: a warp stores 32 features of one row of x at a time
          uint32_t r[16];
          tmem_ld16(trow + (uint32_t)c, r);
          tmem_ld_wait();
          float *dst = a.part + ((int64_t)item * BN + c) * GD_BM + quad * 32 + lane;
#pragma unroll
          for (int i = 0; i < 16; ++i) dst[i * GD_BM] = __uint_as_float(r[i]);
          continue;
        }
        uint32_t r[16];
        tmem_ld16(trow + (uint32_t)c, r);
        tmem_ld_wait();
        __syncwarp();  // the previous block has been read out of the staging tile
#pragma unroll
        for (int i = 0; i < 16; ++i) stg[i * 32 + lane] = __uint_as_float(r[i]);
        __syncwarp();
        const int m_first = t.m0 + c;
        if (a.act == CATEN_B200_ACT_SILU_GLU) gd_store_block<CATEN_B200_ACT_SILU_GLU, EXPERTS>(a, stg, rr, lane, bias4, oc, o_ok, m_first, t.m_end);
        else if (a.act == CATEN_B200_ACT_RELU_GLU) gd_store_block<CATEN_B200_ACT_RELU_GLU, EXPERTS>(a, stg, rr, lane, bias4, oc, o_ok, m_first, t.m_end);
        else if (!EXPERTS && a.act == CATEN_B200_ACT_GELU) gd_store_block<CATEN_B200_ACT_GELU, EXPERTS>(a, stg, rr, lane, bias4, oc, o_ok, m_first, t.m_end);
        else if (!EXPERTS && a.act == CATEN_B200_ACT_RELU) gd_store_block<CATEN_B200_ACT_RELU, EXPERTS>(a, stg, rr, lane, bias4, oc, o_ok, m_first, t.m_end);
        else gd_store_block<CATEN_B200_ACT_NONE, EXPERTS>(a, stg, rr, lane, bias4, oc, o_ok, m_first, t.m_end);
        if (c + 4 * GD_EPI_WARPS < BN) gd_load_res(a, rr, lane, oc, o_ok, m_first + 4 * GD_EPI_WARPS, t.m_end);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_leader(acc_empty(b));
        else mbar_arrive(acc_empty(b));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();   // the other CTA signals into this one's shared memory, and reads it
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(a.tmem_cols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(a.tmem_cols) : "memory");
  }
}

// ---- host ---------------------------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// rows x K bf16, K contiguous; a box is `box_rows` rows of `bk` k (128 bytes with the 128-byte swizzle, or 64 with
// the 64-byte one), zero fill outside
static int make_map(caten_b200_ctx *ctx, CUtensorMap *map, const void *base, int64_t rows, int64_t K, int box_rows, int bk) {
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {(cuuint32_t)bk, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = ((EncodeTiledFn)ctx->encode_tiled)(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box,
                                                       estr, CU_TENSOR_MAP_INTERLEAVE_NONE, bk == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                                                       CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(ctx, CATEN_B200_ECUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return 0;
}

template <int WT>
static int launch_wsplit(caten_b200_ctx *ctx, const WSrc &ws, int64_t N, int64_t K, __nv_bfloat16 *hi, __nv_bfloat16 *lo) {
  const int64_t n8 = N * (K / 8);
  launch_k(ctx, wsplit_kernel<WT>, dim3((unsigned)((n8 + 255) / 256)), dim3(256), 0, ws.qs, ws.d, ws.m, ws.qh, N, K, hi, lo);
  CB_LAUNCH_CHECK(ctx, "wsplit_kernel");
  return 0;
}

// How a launch is cut: rows of x per tile and shares of k.
struct GdPlan {
  int bn, splits, cps;
  bool pair;
};

// Bytes of staging of the epilogue warps that have columns to store, and stages of a launch.  A CTA with one item leaves room on its
// SM for one of the next linear, which starts to load its weights meanwhile; a CTA that walks over items takes what there is: 1 KB
// slack + 1 KB barriers + stages + 32 KB of staging fit 227 KB.
static size_t gd_staging(int bn) { return 2048 * 4 * (size_t)(bn < 64 ? bn / 16 : 4); }
static int gd_stages(int sm, int64_t M, int64_t items, int bn, int cps, size_t stage) {
  int stages = (int)((items <= sm && M <= GD_SPLIT_ROWS ? 108 * 1024 - gd_staging(bn) : GD_STAGE_BYTES) / stage);
  if (stages > 8) stages = 8;
  if (stages > cps) stages = cps;
  return stages < 2 ? 2 : stages;
}

// The cut with the shortest expected time, in cycles.  A CTA's stage takes as long as its MMAs (bn / 2 cycles each, 32 at least, and
// 110 to 200 a stage that the tensor cores wait between stages), as its operands need from L2 (52 bytes a cycle for each of
// the SMs, shared by the CTAs that are at work), or as the stages in flight allow, which are back after about 1400 cycles.
// Wide tiles read least, narrow ones leave no SM without work and the last wave short; shares of k pay for a pass over their
// partial sums.  A pair of CTAs on 256 features loads half of x per CTA and starts later (both CTAs meet twice).  The constants
// are those with which this function comes closest to the fastest cut over 740 launches of 62 shapes (5 to 8192 rows, 768 to 11264 features,
// k of 704 to 6400, both precisions), except for what shares of k cost, which is taken from whole decode steps: on average 0.5 % from it, where the one before, which had pairs 256 rows wide only, was 4.8 %
// (us, before -> now: 2331 rows, plain bf16, 2048 x 5632 62.6 -> 46.6 by pairs 160 wide, 2048 x 4096 46.9 -> 36.4; 5000 rows, 1280 x 5120 61.4 -> 51.6; 64 rows,
// 1024 x 2048 9.8 -> 7.3 in four shares of 16 rows; 200 rows, 4096 x 1024 11.3 -> 9.0; split bf16, 5000 rows, 2304 x 768 45.4 -> 41.5).
static GdPlan gd_plan(int sm, int64_t M, int64_t N, int tiles_f, int64_t K, int nsplit, bool wlo, int bk, bool can_split, bool consumer_sums, bool can_pair, bool must_pair) {
  GdPlan best = {256, 1, (int)(K / bk), false};
  double least = 1e30;
  const int nk = (int)(K / bk), products = nsplit == 1 ? 1 : wlo ? 3 : 2, parts = nsplit == 1 ? 1 : 2;
  for (int pair = must_pair && can_pair ? 1 : 0; pair <= (can_pair ? 1 : 0); ++pair) {
    const int workers = pair ? sm / 2 : sm;
    for (int bn = pair ? 96 : 16; bn <= GD_BN; bn = bn < 32 ? 32 : bn + 32) {
      if (bn == 16 && M > 64) continue;
      const int64_t tiles = (M + bn - 1) / bn * (pair ? (N + 2 * GD_BM - 1) / (2 * GD_BM) : tiles_f);
      const double mma = (double)(bk / 16) * products * (bn > 64 ? bn / 2 : 32) + (nsplit == 1 ? 200.0 : 110.0);
      const double bytes = (double)bk * 2 * (GD_BM * (wlo ? 2 : 1) + (double)(pair ? bn / 2 : bn) * parts);
      const double epilogue = 1360 + 20.0 * bn;
      for (int splits = 1; splits <= 32; ++splits) {
        const int cps = (nk + splits - 1) / splits, s = (nk + cps - 1) / cps;
        if (splits > 1 && (pair || !can_split || tiles * s > sm || cps * bk < 256)) break;
        if (s != splits) continue;
        const int64_t items = tiles * s, waves = (items + workers - 1) / workers;
        const double busy = (items < workers ? (double)items : (double)workers) * (pair ? 2 : 1);
        const double in_flight = gd_stages(sm, M, items, bn, cps, (size_t)bytes);
        double stage = mma > bytes * busy / (52.0 * sm) ? mma : bytes * busy / (52.0 * sm);
        if (stage < 1400.0 / in_flight) stage = 1400.0 / in_flight;
        const double body = cps * stage;
        // (a single wave of the widest pairs lost where the model had them ahead: us alone / pairs, plain bf16, 1525 rows, 3072 x 1600
        // 18.0 / 19.5, 909 rows, 4096 x 2816 23.0 / 24.7)
        double t = (pair ? bn == GD_BN && waves == 1 ? 11900 : 8900 : 5900) + body + epilogue + (double)(waves - 1) * (body > 0.54 * epilogue ? body : 0.54 * epilogue);
        if (s > 1) t += (consumer_sums ? 500.0 + 60.0 * s : 6000.0) + (double)M * N * 4 * s / (sm * 17.0);
        t *= 1.0 + 0.0001 * (GD_BN - bn);   // traffic costs power too, which is what limits long launches
        if (t < least) { least = t; best = {bn, s, cps, pair != 0}; }
      }
      if (bn >= M) break;
    }
  }
  return best;
}

// Which linears run here.  In plain bf16, bf16 weights are the operand as they are: every one whose shape fits (us a call, other kernel ->
// this, plain bf16, 11264 x 2048: 16 rows 29 -> 13, 256 rows 42 -> 27, 777 rows 108 -> 39; 1024 x 4096: 1665 rows 45 -> 28).
// In split bf16 they follow the rule below: with few rows the other kernel, whose one MMA takes both parts of x and whose shares
// of k are shorter, is faster (27 rows of GPT-2 XL: a prompt 3.38 ms there, 3.77 here) and rounds less.
// Other formats are expanded once per call, which pays when the converting producers of the other kernel (one per output
// tile) repeat it often: with full waves of the widest tiles from 1024 rows on, otherwise from 1536 (split bf16, Q4_0,
// 1600 x 6400: 777 rows 65 here 87, 1024 rows 69 here 90, 1665 rows 113 here 106; 1600 x 1600: 1665 rows 38 here 32).
bool gemm_dense_applies(const caten_b200_ctx *ctx, int wt, int64_t M, int64_t N, int64_t K, int nsplit) {
  if (!ctx->dense_gemm || N % 4 || K % GD_BK || K < GD_BK) return false;
  if (wt == CATEN_B200_BF16 && nsplit == 1) return true;
  if (M >= GD_EXPAND_ROWS) {
    // .. except, in split bf16, long rows of packed or fp16 weights where equal shares of k of the other kernel's tiles of 128 x 256
    // about fill its one wave (us there / here, Q4_0: 768 x 3072 2048 rows 37 / 45, 1024 x 4096 1665 rows 51 / 58, 2048 rows 54 / 61, 1280 x 5120
    // 1665 rows 62 / 75, but 2048 rows, which half fill it, 92 / 78; fp32 weights cost it more: 1024 x 4096 2048 rows 70 / 63)
    const int64_t tiles = (M + GD_BN - 1) / GD_BN * ((N + GD_BM - 1) / GD_BM), sm = ctx->sm_count;
    return nsplit != 3 || wt == CATEN_B200_BF16 || wt == CATEN_B200_F32 || wt == WT_F32_T || K <= 2 * N || 2 * tiles > sm || 4 * (sm / tiles * tiles) < 3 * sm;
  }
  return M >= 1024 && (M + GD_BN - 1) / GD_BN * ((N + GD_BM - 1) / GD_BM) >= ctx->sm_count;
}

// wt: a ggml type or WT_F32_T (then ws.qs is b[K, N] fp32).  x: fp32 [M, K], or its split bf16 copy when xhi is given.
int launch_gemm_dense(caten_b200_ctx *ctx, int wt, const WSrc &ws, const float *x, const __nv_bfloat16 *xhi, const __nv_bfloat16 *xlo,
                      const float *bias, const float *res, int act, float *y, BfOut ybf, int64_t M, int64_t N, int64_t K, int nsplit,
                      LinGroups grp, PartIn *defer) {
  if (!ctx->encode_tiled) return fail(ctx, CATEN_B200_ECUDA, "gemm_dense: cuTensorMapEncodeTiled is not available");
  if (K % GD_BK || M > 0x7fffffff || N > 0x7fffffff || K > 0x7fffffff) return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemm_dense: shape %lldx%lldx%lld", (long long)M, (long long)N, (long long)K);
  if (nsplit != 1 && nsplit != 3) return fail(ctx, CATEN_B200_EINVAL, "gemm_dense: nsplit must be 1 or 3");
  const int parts = nsplit == 3 ? 2 : 1;
  // bf16 copy of the weights
  const bool as_is = wt == CATEN_B200_BF16;  // the weight is the operand: no copy, and no low part
  const size_t wb = ((size_t)N * K * 2 + 1023) & ~(size_t)1023;
  if (!as_is)
    if (int rc = scratch_reserve(ctx, &ctx->wbf, wb * parts)) return rc;
  __nv_bfloat16 *whi = (__nv_bfloat16 *)ctx->wbf.ptr, *wlo = parts == 2 && !as_is ? (__nv_bfloat16 *)((uint8_t *)ctx->wbf.ptr + wb) : nullptr;
  int rc = 0;
  if (as_is) whi = (__nv_bfloat16 *)ws.qs;
  else switch (wt) {
    case CATEN_B200_F32: rc = launch_wsplit<CATEN_B200_F32>(ctx, ws, N, K, whi, wlo); break;
    case CATEN_B200_F16: rc = launch_wsplit<CATEN_B200_F16>(ctx, ws, N, K, whi, wlo); break;
    case CATEN_B200_Q4_0: rc = launch_wsplit<CATEN_B200_Q4_0>(ctx, ws, N, K, whi, wlo); break;
    case CATEN_B200_Q4_1: rc = launch_wsplit<CATEN_B200_Q4_1>(ctx, ws, N, K, whi, wlo); break;
    case CATEN_B200_Q5_0: rc = launch_wsplit<CATEN_B200_Q5_0>(ctx, ws, N, K, whi, wlo); break;
    case CATEN_B200_Q5_1: rc = launch_wsplit<CATEN_B200_Q5_1>(ctx, ws, N, K, whi, wlo); break;
    case CATEN_B200_Q8_0: rc = launch_wsplit<CATEN_B200_Q8_0>(ctx, ws, N, K, whi, wlo); break;
    case WT_F32_T: break;   // together with x, below
    default: return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemm_dense: weight type %d", wt);
  }
  if (rc) return rc;
  // bf16 copy of the activations, unless their producer already wrote one
  if (!xhi) {
    const size_t xb = ((size_t)M * K * 2 + 1023) & ~(size_t)1023;
    if (int rc2 = scratch_reserve(ctx, &ctx->xbf, xb * parts)) return rc2;
    __nv_bfloat16 *h = (__nv_bfloat16 *)ctx->xbf.ptr, *l = parts == 2 ? (__nv_bfloat16 *)((uint8_t *)ctx->xbf.ptr + xb) : nullptr;
    const int64_t n8 = M * K / 8, xb_ctas = (n8 + 255) / 256;
    if (wt == WT_F32_T) {
      const int64_t tiles_n = (N + 63) / 64, tiles = tiles_n * (K / 64);
      if (tiles + xb_ctas > 0x7fffffff) return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemm_dense: shape %lldx%lldx%lld", (long long)M, (long long)N, (long long)K);
      launch_k(ctx, operands_split_kernel, dim3((unsigned)(tiles + xb_ctas)), dim3(256), 0, (const float *)ws.qs, (int)K, (int)N, (int)tiles_n, (int)tiles, whi, wlo, x, n8, h, l);
    } else {
      launch_k(ctx, xsplit_kernel, dim3((unsigned)xb_ctas), dim3(256), 0, x, n8, h, l);
    }
    CB_LAUNCH_CHECK(ctx, "xsplit_kernel");
    xhi = h;
    xlo = l;
  } else if (wt == WT_F32_T || (nsplit == 3 && !xlo)) {
    return fail(ctx, CATEN_B200_EINVAL, "gemm_dense: split-bf16 needs the lo part of x, relu(matmul) an fp32 x");
  }
  if (((uintptr_t)xhi | (uintptr_t)xlo) & 15) return fail(ctx, CATEN_B200_EINVAL, "gemm_dense: bf16 operand must be 16-byte aligned");

  CUtensorMap twh, twl, txh, txl;
  const int bk = nsplit == 3 ? GdStage<3>::BK : GdStage<1>::BK;
  if ((rc = make_map(ctx, &twh, whi, N, K, GD_BM, bk))) return rc;
  twl = twh;
  if (wlo && (rc = make_map(ctx, &twl, wlo, N, K, GD_BM, bk))) return rc;
  const int64_t xrows = grp.group_rows ? (N - 1) / grp.group_rows * grp.xplane + M : M;  // all planes of x

  GdArgs a;
  a.bias = bias; a.res = res; a.y = y; a.yhi = ybf.hi; a.ylo = ybf.lo; a.status = ctx->d_status;
  a.act = act; a.M = (int)M; a.N = (int)N; a.K = (int)K;
  a.group_rows = grp.group_rows ? (int)grp.group_rows : (int)((N + GD_BM - 1) / GD_BM * GD_BM); a.xplane = (int)grp.xplane;
  a.tiles_per_group = (a.group_rows + GD_BM - 1) / GD_BM;
  a.tiles_f = (int)((N + a.group_rows - 1) / a.group_rows) * a.tiles_per_group;
  a.ygroup = grp.ygroup ? (int)grp.ygroup : a.group_rows;
  a.ldy = grp.ldy ? (int)grp.ldy : (int)(act_is_glu(act) ? N / 2 : N);
  if (res && !grp.plain_output()) return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemm_dense: a residual needs the plain output layout");
  const bool can_defer = defer && act == CATEN_B200_ACT_NONE && !ybf.hi && grp.plain_output() && grp.group_rows % GD_BM == 0;
  const bool can_pair = ctx->dense_pair && M > GD_SPLIT_ROWS && !grp.group_rows && ctx->sm_count % 2 == 0;
  const GdPlan p = gd_plan(ctx->sm_count, M, N, a.tiles_f, K, nsplit, wlo != nullptr, bk, M <= GD_SPLIT_ROWS, can_defer, can_pair, ctx->dense_pair == 2);
  if (p.pair) a.tiles_f = a.tiles_per_group = (int)((N + 2 * GD_BM - 1) / (2 * GD_BM));
  a.bn = p.bn; a.splits = p.splits; a.cps = p.cps; a.part = nullptr;
  a.static_w = as_is && !ctx->weights_pending;
  if ((rc = make_map(ctx, &txh, xhi, xrows, K, p.pair ? p.bn / 2 : p.bn, bk))) return rc;
  txl = txh;
  if (nsplit == 3 && (rc = make_map(ctx, &txl, xlo, xrows, K, p.pair ? p.bn / 2 : p.bn, bk))) return rc;
  const int64_t tiles = (int64_t)a.tiles_f * ((M + p.bn - 1) / p.bn), items = tiles * p.splits;
  if (items > 0x7fffffff) return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemm_dense: too many tiles");
  a.tiles = (int)tiles;
  if (p.splits > 1) {
    if ((rc = scratch_reserve(ctx, &ctx->wtmp, (size_t)items * p.bn * GD_BM * sizeof(float)))) return rc;
    a.part = (float *)ctx->wtmp.ptr;
  }
  const size_t stage = (size_t)(GD_BM * (wlo ? 2 : 1) + (p.pair ? p.bn / 2 : p.bn) * parts) * (size_t)bk * 2;
  const int workers = p.pair ? ctx->sm_count / 2 : ctx->sm_count, busy = items < workers ? (int)items : workers, grid = p.pair ? 2 * busy : busy;
  const size_t staging = gd_staging(p.bn);
  const int stages = a.stages = gd_stages(ctx->sm_count, M, items, p.bn, p.cps, stage);
  a.idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.bn >> 3) << 17) | ((uint32_t)((p.pair ? 2 * GD_BM : GD_BM) >> 4) << 24);
  a.tmem_cols = p.pair ? 512 : 32;   // (a pair: all, so that its accumulators have the same columns in both CTAs)
  while (a.tmem_cols < (uint32_t)(p.bn * (items > busy ? 2 : 1))) a.tmem_cols *= 2;
  const size_t smem = 2048 + stage * stages + staging;

  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(GD_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[2];
  int na = 0;
  if (take_pdl(ctx)) {
    at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (p.pair) {
    at[na].id = cudaLaunchAttributeClusterDimension;
    at[na].val.clusterDim.x = 2;
    at[na].val.clusterDim.y = at[na].val.clusterDim.z = 1;
    ++na;
  }
  cfg.attrs = at;
  cfg.numAttrs = na;
  auto kernel = p.pair ? (nsplit == 1 ? gemm_dense_kernel<1, false, false, true> : wlo ? gemm_dense_kernel<3, false, true, true> : gemm_dense_kernel<3, false, false, true>)
                       : (nsplit == 1 ? gemm_dense_kernel<1, false, false, false> : wlo ? gemm_dense_kernel<3, false, true, false> : gemm_dense_kernel<3, false, false, false>);
  CB_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  CB_CUDA(ctx, cudaLaunchKernelEx(&cfg, kernel, twh, twl, txh, txl, a));
  CB_LAUNCH_CHECK(ctx, "gemm_dense_kernel");
  if (p.splits == 1) return 0;
  if (can_defer) {   // the consumer of this linear sums the shares itself (and adds bias and residual)
    defer->part = a.part; defer->bias = bias; defer->splits = p.splits; defer->tiles_x = a.tiles_f; defer->bnx = p.bn;
    defer->zstride = (long long)tiles * p.bn * GD_BM;
    return 0;
  }
  return launch_splitk_reduce(ctx, a.part, p.splits, a.tiles_f, a.tiles, p.bn, bias, res, y, ybf, act, a.M, a.N, a.group_rows, a.tiles_per_group, a.ygroup, a.ldy);
}

int launch_gemm_experts(caten_b200_ctx *ctx, const caten_b200_weight *w, const ExpertRows &er, BfOut x, int act, float *y, BfOut ybf, int nsplit) {
  if (er.pairs <= 0) return 0;
  if (!ctx->encode_tiled) return fail(ctx, CATEN_B200_ECUDA, "gemm_experts: cuTensorMapEncodeTiled is not available");
  const int64_t N = w->rows, K = w->cols;
  if (w->type != CATEN_B200_BF16 || K % GD_BK || er.experts < 1 || er.experts > GD_MAX_EXPERTS || N % er.experts || N / er.experts % 4 || N > 0x7fffffff || er.pairs > 0x7fffffff ||
      act == CATEN_B200_ACT_GELU || act == CATEN_B200_ACT_RELU || !x.hi || (nsplit == 3 && !x.lo))
    return fail(ctx, CATEN_B200_EUNSUPPORTED, "gemm_experts: %d experts, weight %lldx%lld", er.experts, (long long)N, (long long)K);
  GdArgs a;
  a.bias = a.res = nullptr; a.y = y; a.yhi = ybf.hi; a.ylo = ybf.lo; a.status = ctx->d_status;
  a.act = act; a.M = (int)er.pairs; a.N = (int)N; a.K = (int)K;
  a.group_rows = (int)(N / er.experts); a.xplane = 0; a.ygroup = a.group_rows;
  a.tiles_f = a.tiles_per_group = (a.group_rows + GD_BM - 1) / GD_BM;
  a.ldy = act_is_glu(act) ? a.group_rows / 2 : a.group_rows;
  a.tiles = 0;
  // twice the rows an expert has on average, so that most experts need one row tile
  int bn = 16;
  while (bn < GD_BN && (int64_t)bn * er.experts < 2 * er.pairs) bn *= 2;
  a.bn = bn; a.splits = 1; a.part = nullptr; a.static_w = 0;
  a.tmem_cols = 512;
  a.er = er;
  const int bk = nsplit == 3 ? GdStage<3>::BK : GdStage<1>::BK;
  a.cps = (int)(K / bk);
  CUtensorMap tw, txh, txl;
  if (int rc = make_map(ctx, &tw, w->qs, N, K, GD_BM, bk)) return rc;
  if (int rc = make_map(ctx, &txh, x.hi, er.pairs, K, bn, bk)) return rc;
  if (int rc = make_map(ctx, &txl, nsplit == 3 ? x.lo : x.hi, er.pairs, K, bn, bk)) return rc;
  const size_t stage = (size_t)bk * 2 * (GD_BM + (size_t)bn * (nsplit == 3 ? 2 : 1));
  int stages = (int)((GD_STAGE_BYTES - (GD_MAX_EXPERTS + 1) * sizeof(int)) / stage);
  if (stages > 10) stages = 10;
  a.stages = stages;
  a.idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(GD_BM >> 4) << 24);
  const size_t smem = 2048 + stage * stages + (size_t)GD_EPI_WARPS * 2048 + (GD_MAX_EXPERTS + 1) * sizeof(int);
  const int64_t most = (er.pairs / bn + (er.pairs < er.experts ? er.pairs : er.experts)) * a.tiles_f;
  const int grid = most < ctx->sm_count ? (int)most : ctx->sm_count;
  if (nsplit == 3) {
    CB_CUDA(ctx, cudaFuncSetAttribute(gemm_dense_kernel<3, true, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    launch_k(ctx, gemm_dense_kernel<3, true, false, false>, dim3((unsigned)grid), dim3(GD_THREADS), smem, tw, tw, txh, txl, a);
  } else {
    CB_CUDA(ctx, cudaFuncSetAttribute(gemm_dense_kernel<1, true, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    launch_k(ctx, gemm_dense_kernel<1, true, false, false>, dim3((unsigned)grid), dim3(GD_THREADS), smem, tw, tw, txh, txl, a);
  }
  CB_LAUNCH_CHECK(ctx, "gemm_dense_kernel");
  return 0;
}

}  // namespace cb
