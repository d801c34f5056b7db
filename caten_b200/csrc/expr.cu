// Generic schedule item: one kernel that interprets a fused element-wise (optionally reducing)
// expression per element.  It stands where the reference renders one C function per
// Schedule-Item (source/byoc/clang.lisp:163-205, op by op as in source/codegen/renderer.lisp:331-410)
// and compiles it with gcc at run time; here nothing is compiled on the host.
//
// One thread owns up to eight output elements of the innermost kept loop (32 apart, so that a warp's
// accesses are coalesced).  It decodes its multi-index once, then walks the reduced loops (if
// any) in loop order, exactly like the rendered loop nest, so a float sum is added in the
// reference's order.  The program is postfix over a small value stack whose slots hold the
// elements side by side, so decoding a program word is paid once for all of them; the top of
// the stack is in registers, the rest in shared memory, the program and the views in the
// kernel's constant parameter space.  Contiguous row reductions use a second kernel with the
// lanes along the reduced loop and an in-order accumulation of tiles in shared memory.
#include "common.cuh"

namespace cb {

__device__ __forceinline__ uint32_t expr_load(const void *p, int dtype, int64_t at) {
  switch (dtype) {
    case CATEN_B200_DT_F32: return __float_as_uint(reinterpret_cast<const float *>(p)[at]);
    case CATEN_B200_DT_I32: return (uint32_t) reinterpret_cast<const int32_t *>(p)[at];
    case CATEN_B200_DT_I64: return (uint32_t)(int32_t) reinterpret_cast<const int64_t *>(p)[at];
    default: return reinterpret_cast<const uint8_t *>(p)[at] ? 1u : 0u;
  }
}

// value of class `cls` -> the output buffer's element type (C conversion rules)
__device__ __forceinline__ void expr_store(void *p, int dtype, int64_t at, uint32_t v, int cls) {
  const bool is_f = cls == CATEN_B200_CLS_F32;
  switch (dtype) {
    case CATEN_B200_DT_F32: reinterpret_cast<float *>(p)[at] = is_f ? __uint_as_float(v) : (float)(int32_t)v; break;
    case CATEN_B200_DT_I32: reinterpret_cast<int32_t *>(p)[at] = is_f ? (int32_t)__uint_as_float(v) : (int32_t)v; break;
    case CATEN_B200_DT_I64: reinterpret_cast<int64_t *>(p)[at] = is_f ? (int64_t)__uint_as_float(v) : (int64_t)(int32_t)v; break;
    default: reinterpret_cast<uint8_t *>(p)[at] = is_f ? (__uint_as_float(v) != 0.0f) : (v != 0u); break;
  }
}

// A strip's values, as above with one switch for all of them (a switch per element, and spilled registers: int add over 12800 x 511 28.0 us, so 17.3).
template <int EV>
__device__ __forceinline__ void expr_store_ev(void *out, const int dtype, const int64_t at, const int64_t step, const int lanes, const uint32_t *v, const int cls) {
  const bool is_f = cls == CATEN_B200_CLS_F32;
  auto strip = [&](auto *p, auto value) {
    if (step == 32) {   // contiguous
#pragma unroll
      for (int j = 0; j < EV; ++j)
        if (j < lanes) p[32 * j] = value(v[j]);
    } else {
#pragma unroll
      for (int j = 0; j < EV; ++j)
        if (j < lanes) p[j * step] = value(v[j]);
    }
  };
  switch (dtype) {
    case CATEN_B200_DT_F32:
      if (is_f) strip(reinterpret_cast<float *>(out) + at, [](uint32_t x) { return __uint_as_float(x); });
      else strip(reinterpret_cast<float *>(out) + at, [](uint32_t x) { return (float)(int32_t)x; });
      break;
    case CATEN_B200_DT_I32:
      if (is_f) strip(reinterpret_cast<int32_t *>(out) + at, [](uint32_t x) { return (int32_t)__uint_as_float(x); });
      else strip(reinterpret_cast<int32_t *>(out) + at, [](uint32_t x) { return (int32_t)x; });
      break;
    case CATEN_B200_DT_I64:
      if (is_f) strip(reinterpret_cast<int64_t *>(out) + at, [](uint32_t x) { return (int64_t)__uint_as_float(x); });
      else strip(reinterpret_cast<int64_t *>(out) + at, [](uint32_t x) { return (int64_t)(int32_t)x; });
      break;
    default:
      if (is_f) strip(reinterpret_cast<uint8_t *>(out) + at, [](uint32_t x) { return (uint8_t)(__uint_as_float(x) != 0.0f); });
      else strip(reinterpret_cast<uint8_t *>(out) + at, [](uint32_t x) { return (uint8_t)(x != 0u); });
      break;
  }
}

__device__ __forceinline__ uint32_t expr_cast(uint32_t v, int from, int to) {
  if (from == to) return v;
  if (to == CATEN_B200_CLS_F32) return __float_as_uint((float)(int32_t)v);          // I32 / BOOL -> float
  if (from == CATEN_B200_CLS_F32) {
    const float f = __uint_as_float(v);
    return to == CATEN_B200_CLS_BOOL ? (f != 0.0f ? 1u : 0u) : (uint32_t)(int32_t)f;  // C truncation
  }
  return to == CATEN_B200_CLS_BOOL ? (v != 0u ? 1u : 0u) : v;                          // I32 <-> BOOL
}

// 2^x rounded once from double: x = n + f with n the nearest integer (the difference is exact), 2^f by 1 + f q(f), q the
// polynomial of degree 11 through (2^f - 1) / f at the Chebyshev nodes of [-1/2, 1/2] (relative error 2^-55, below double's own
// rounding; none at whole numbers), n added to the exponent; past +-160 the conversion gives 0 or inf either way.  Twelve fused
// steps and no branch: an exp2 item over 12800 x 511 takes 15.7 us (nine steps, 2^-44: 15.3; exp2(double) took
// 31.8 where nine steps took 18.2).
__device__ __forceinline__ float expr_exp2(float x) {
  x = x > 160.0f ? 160.0f : x;
  x = x < -160.0f ? -160.0f : x;
  const float big = 12582912.0f;           // 1.5 * 2^23: adding it rounds to an integer
  const float t = x + big;
  const double f = (double)(x - (t - big));
  double p = 2.5729324177362305e-11;
  p = fma(p, f, 4.4558179083360645e-10);
  p = fma(p, f, 7.0548973041554995e-09);
  p = fma(p, f, 1.0178057087733941e-07);
  p = fma(p, f, 1.3215486808705563e-06);
  p = fma(p, f, 1.5252733841556773e-05);
  p = fma(p, f, 0.00015403530393370734);
  p = fma(p, f, 0.001333355814640647);
  p = fma(p, f, 0.00961812910762848);
  p = fma(p, f, 0.055504108664821625);
  p = fma(p, f, 0.24022650695910072);
  p = fma(p, f, 0.6931471805599453);
  p = fma(p, f, 1.0);
  const float y = (float)__hiloint2double(__double2hiint(p) + ((__float_as_int(t) - 0x4b400000) << 20), __double2loint(p));
  return x != x ? x : y;
}

constexpr int EXPR_THREADS = 256;
constexpr int MAXD = CATEN_B200_EXPR_MAX_DIMS;

// Words as the kernels see them (expr_fuse writes them from the caller's program): bits 24..26 say where a binary word's right
// operand comes from, so that `LOAD b; ADD` or `CONST c; MUL` is one word that touches no stack slot; bit 27 / 28: the right
// operand is negated / replaced by its reciprocal first (`LOAD b; NEG; ADD` and `LOAD b; RECIP; MUL`, floats); bit 29: a binary
// word.  An op that floats and whole numbers share has a code of its own for the latter, so that a word computes one of the two.
enum ExprMode : uint32_t { EXPR_POP = 0, EXPR_WITH_CONST = 1u << 24, EXPR_WITH_LOAD = 2u << 24, EXPR_MODES = 7u << 24, EXPR_NEG_B = 1u << 27, EXPR_RECIP_B = 1u << 28, EXPR_BINARY = 1u << 29 };
constexpr int EXPR_WHOLE = 64;   // added to the code of NEG, RECIP, NOT, ADD, MUL, MAX, NE and LT on whole numbers, and to LOAD of them

// Per-thread state is kept out of local memory (some 30 bytes are spilled; in reducing items with eight elements a thread 300 to 500,
// around the reduced loop): with 2048 threads per SM a few hundred bytes of
// local arrays each overflow L1 and turn every stack access into L2 traffic.  The loop indices
// are ND registers (all loops over them are fully unrolled; the strides of loops that are not there are 0), operand
// offsets are recomputed from them at each LOAD (strides come from the kernel's parameter space), the top of the value
// stack is EV registers and the values under it live in shared memory, [slot][element][thread].
template <int ND> struct ExprIx {
  int v[ND];
};

// EV values of operand `arg`: element j is 32 j further along loop `va`; for j >= lanes the last element is re-read, so
// nothing outside the views is touched.
template <int ND, int EV>
__device__ __forceinline__ void expr_load_ev(const caten_b200_expr &e, const int arg, const ExprIx<ND> &ix, const int va, const int lanes, const bool whole, uint32_t *out) {
  int64_t o = e.operand_offset[arg];
#pragma unroll
  for (int d = 0; d < ND; ++d) o += (int64_t)ix.v[d] * e.operand_stride[arg][d];
  const int64_t step = va >= 0 ? 32 * e.operand_stride[arg][va] : 0;
  const int last = lanes > 0 ? lanes - 1 : 0;
  if (!whole) {
    const float *p = reinterpret_cast<const float *>(e.operand[arg]) + o;
    if (step == 32 && lanes == EV) {   // the strip is contiguous and full
#pragma unroll
      for (int j = 0; j < EV; ++j) out[j] = __float_as_uint(p[32 * j]);
    } else if (step == 0) {
      const uint32_t v = __float_as_uint(*p);
#pragma unroll
      for (int j = 0; j < EV; ++j) out[j] = v;
    } else {
#pragma unroll
      for (int j = 0; j < EV; ++j) out[j] = __float_as_uint(p[(j < last ? j : last) * step]);
    }
    return;
  }
  // (one switch for all of them)
  auto strip = [&](auto *p, auto value) {
    if (step == 0) {
      const uint32_t v = value(*p);
#pragma unroll
      for (int j = 0; j < EV; ++j) out[j] = v;
    } else if (step == 32 && lanes == EV) {
#pragma unroll
      for (int j = 0; j < EV; ++j) out[j] = value(p[32 * j]);
    } else {
#pragma unroll
      for (int j = 0; j < EV; ++j) out[j] = value(p[(j < last ? j : last) * step]);
    }
  };
  switch (e.operand_dtype[arg]) {
    case CATEN_B200_DT_I32: strip(reinterpret_cast<const int32_t *>(e.operand[arg]) + o, [](int32_t v) { return (uint32_t)v; }); break;
    case CATEN_B200_DT_I64: strip(reinterpret_cast<const int64_t *>(e.operand[arg]) + o, [](int64_t v) { return (uint32_t)(int32_t)v; }); break;
    default: strip(reinterpret_cast<const uint8_t *>(e.operand[arg]) + o, [](uint8_t v) { return v ? 1u : 0u; }); break;
  }
}

// Runs the program for EV elements at once: the decode of a word is shared.  Element j of the
// thread is 32 j further along loop `va` (va < 0: a single element).  HEAVY: with the words whose code takes twice the
// registers (sines and logarithms in double, integer division); programs without them run in the lean form, of which twice
// as many warps are resident (exp2 and division items over 12800 x 511: 36 us without the split, 27 us with it, 25 and 19 now).
template <int ND, int EV, int THREADS, bool HEAVY>
__device__ __forceinline__ void expr_run(const caten_b200_expr &e, const ExprIx<ND> &ix, const int va, const int lanes, uint32_t *tos, uint32_t *sm) {
  int sp = 0;  // values on the stack, the top one (registers) included
  auto slot = [&](int s, int j) -> uint32_t & { return sm[(s * EV + j) * THREADS]; };
  auto push = [&]() {
    if (sp > 0) {
#pragma unroll
      for (int j = 0; j < EV; ++j) slot(sp - 1, j) = tos[j];
    }
    ++sp;
  };
#define EXPR_UN(VALUE)                                                             \
  {                                                                                \
    _Pragma("unroll") for (int j = 0; j < EV; ++j) {                               \
      const uint32_t a = tos[j];                                                   \
      const float fa = __uint_as_float(a);                                         \
      const int32_t ia = (int32_t)a;                                               \
      (void)fa; (void)ia;                                                          \
      tos[j] = VALUE;                                                              \
    }                                                                              \
    break;                                                                         \
  }
#define EXPR_BIN(VALUE)                                                            \
  {                                                                                \
    _Pragma("unroll") for (int j = 0; j < EV; ++j) {                               \
      const uint32_t a = tos[j], b = r[j];                                         \
      const float fa = __uint_as_float(a), fb = __uint_as_float(b);                \
      const int32_t ia = (int32_t)a, ib = (int32_t)b;                              \
      (void)fa; (void)fb; (void)ia; (void)ib;                                      \
      tos[j] = VALUE;                                                              \
    }                                                                              \
    break;                                                                         \
  }
  for (int pc = 0; pc < e.n_code; ++pc) {
    const uint32_t w = e.code[pc];
    const int op = w & 255, arg = (w >> 8) & 255;
    uint32_t r[EV];   // right operand of a binary word; tos becomes the left one
    if (w & EXPR_BINARY) {
      const uint32_t mode = w & EXPR_MODES;
      if (mode == EXPR_POP) {
        --sp;
#pragma unroll
        for (int j = 0; j < EV; ++j) { r[j] = tos[j]; tos[j] = slot(sp - 1, j); }
      } else {
        const bool one = mode == EXPR_WITH_CONST || va < 0 || e.operand_stride[arg][va] == 0;   // one value for all of them
        if (mode == EXPR_WITH_LOAD) {
          expr_load_ev<ND, EV>(e, arg, ix, va, lanes, op >= EXPR_WHOLE || (op >= CATEN_B200_OP_MOD && op <= CATEN_B200_OP_XOR), r);
        } else {
          r[0] = e.consts[arg];
        }
        if (w & EXPR_NEG_B) {
#pragma unroll
          for (int j = 0; j < EV; ++j) r[j] = __float_as_uint(-__uint_as_float(r[j]));
        }
        if (one) {
          if (w & EXPR_RECIP_B) r[0] = __float_as_uint(1.0f / __uint_as_float(r[0]));
#pragma unroll
          for (int j = 1; j < EV; ++j) r[j] = r[0];
        } else if (w & EXPR_RECIP_B) {
#pragma unroll
          for (int j = 0; j < EV; ++j) r[j] = __float_as_uint(1.0f / __uint_as_float(r[j]));
        }
      }
    }
    switch (op) {
      case CATEN_B200_OP_LOAD:
      case CATEN_B200_OP_LOAD + EXPR_WHOLE:
        push();
        expr_load_ev<ND, EV>(e, arg, ix, va, lanes, op >= EXPR_WHOLE, tos);
        break;
      case CATEN_B200_OP_CONST:
        push();
#pragma unroll
        for (int j = 0; j < EV; ++j) tos[j] = e.consts[arg];
        break;
      case CATEN_B200_OP_INDEX: {
        push();
        int base = 0;
#pragma unroll
        for (int d = 0; d < ND; ++d)
          if (d == arg) base = ix.v[d];
#pragma unroll
        for (int j = 0; j < EV; ++j) tos[j] = (uint32_t)(base + (arg == va ? 32 * j : 0));
        break;
      }
      case CATEN_B200_OP_NEG: EXPR_UN(__float_as_uint(-fa))
      case CATEN_B200_OP_NEG + EXPR_WHOLE: EXPR_UN((uint32_t)(-ia))
      case CATEN_B200_OP_RECIP: EXPR_UN(__float_as_uint(1.0f / fa))
      case CATEN_B200_OP_RECIP + EXPR_WHOLE: EXPR_UN((ia == 1 || ia == -1 ? (uint32_t)ia : 0u))
      case CATEN_B200_OP_SIN: EXPR_UN(HEAVY ? __float_as_uint((float)sin((double)fa)) : a)
      case CATEN_B200_OP_EXP2: EXPR_UN(__float_as_uint(expr_exp2(fa)))
      case CATEN_B200_OP_LOG2: EXPR_UN(HEAVY ? __float_as_uint((float)log2((double)fa)) : a)
      case CATEN_B200_OP_SQRT: EXPR_UN(HEAVY ? __float_as_uint((float)sqrt((double)fa)) : a)
      case CATEN_B200_OP_NOT: EXPR_UN((fa == 0.0f ? 1u : 0u))
      case CATEN_B200_OP_NOT + EXPR_WHOLE: EXPR_UN((a == 0u ? 1u : 0u))
      case CATEN_B200_OP_CAST: {
        const int cls = (w >> 16) & 255;
#pragma unroll
        for (int j = 0; j < EV; ++j) tos[j] = expr_cast(tos[j], arg, cls);
        break;
      }
      case CATEN_B200_OP_ADD: EXPR_BIN(__float_as_uint(fa + fb))
      case CATEN_B200_OP_ADD + EXPR_WHOLE: EXPR_BIN((uint32_t)(ia + ib))
      case CATEN_B200_OP_MUL: EXPR_BIN(__float_as_uint(fa * fb))
      case CATEN_B200_OP_MUL + EXPR_WHOLE: EXPR_BIN((uint32_t)(ia * ib))
      case CATEN_B200_OP_MOD: EXPR_BIN((!HEAVY || ib == 0 ? 0u : (uint32_t)(ia % ib)))
      case CATEN_B200_OP_IDIV: EXPR_BIN((!HEAVY || ib == 0 ? 0u : (uint32_t)(ia / ib)))
      case CATEN_B200_OP_AND: EXPR_BIN(a & b)
      case CATEN_B200_OP_OR: EXPR_BIN(a | b)
      case CATEN_B200_OP_XOR: EXPR_BIN(a ^ b)
      case CATEN_B200_OP_MAX: EXPR_BIN((fa > fb ? a : b))
      case CATEN_B200_OP_MAX + EXPR_WHOLE: EXPR_BIN((ia > ib ? a : b))
      case CATEN_B200_OP_NE: EXPR_BIN((fa != fb ? 1u : 0u))
      case CATEN_B200_OP_NE + EXPR_WHOLE: EXPR_BIN((a != b ? 1u : 0u))
      case CATEN_B200_OP_LT: EXPR_BIN((fa < fb ? 1u : 0u))
      case CATEN_B200_OP_LT + EXPR_WHOLE: EXPR_BIN((ia < ib ? 1u : 0u))
      default: {  // WHERE: (cond a b) with b on top
        sp -= 2;
#pragma unroll
        for (int j = 0; j < EV; ++j) tos[j] = slot(sp - 1, j) != 0u ? slot(sp, j) : tos[j];
        break;
      }
    }
  }
#undef EXPR_UN
#undef EXPR_BIN
}

// loop indices of flat position `pos` over loops [first, last) -> ix (innermost fastest).  The outermost one is what is left;
// the others divide in 32 bits where the position has no more (a 64-bit division is some 80 instructions, paid per strip).
template <int ND>
__device__ __forceinline__ void expr_decode(const caten_b200_expr &e, int64_t pos, const int first, const int last, ExprIx<ND> &ix) {
#pragma unroll
  for (int d = ND - 1; d >= 0; --d) {
    if (d > first && d < last) {
      const uint32_t n = (uint32_t)e.shape[d];   // (an extent is at most 2^31 - 1)
      if ((uint64_t)pos >> 32) {
        ix.v[d] = (int)(pos % n);
        pos /= n;
      } else {
        const uint32_t q = (uint32_t)pos / n;
        ix.v[d] = (int)((uint32_t)pos - q * n);
        pos = q;
      }
    } else if (d == first && d < last) {
      ix.v[d] = (int)pos;
    }
  }
}

template <int ND>
__device__ __forceinline__ int64_t expr_out_at(const caten_b200_expr &e, const ExprIx<ND> &ix, const int nd_out) {
  int64_t at = e.out_offset;
#pragma unroll
  for (int d = 0; d < ND; ++d)
    if (d < nd_out) at += (int64_t)ix.v[d] * e.out_stride[d];
  return at;
}

struct ExprAcc {  // reduction state of one output element
  float f;
  int32_t i;
};

__device__ __forceinline__ ExprAcc expr_acc_init(const caten_b200_expr &e, const bool is_f, const int64_t out_at, const bool valid) {
  ExprAcc a;
  a.f = e.reduce_op == CATEN_B200_RED_MAX ? -INFINITY : 0.0f;
  a.i = e.reduce_op == CATEN_B200_RED_MAX ? INT32_MIN : 0;
  if (e.accumulate && valid) {  // the buffer's element type decides how its old value reads
    const uint32_t old = expr_load(e.out, e.out_dtype, out_at);
    if (is_f) a.f = e.out_dtype == CATEN_B200_DT_F32 ? __uint_as_float(old) : (float)(int32_t)old;
    else a.i = e.out_dtype == CATEN_B200_DT_F32 ? (int32_t)__uint_as_float(old) : (int32_t)old;
  }
  return a;
}

// acc <- acc (op) x (the least value that a MAX starts from gives way to any x)
__device__ __forceinline__ void expr_acc_add(ExprAcc &a, const uint32_t x, const bool is_f, const bool is_sum) {
  if (is_f) {
    const float xf = __uint_as_float(x);
    a.f = is_sum ? a.f + xf : (a.f > xf ? a.f : xf);
  } else {
    const int32_t xi = (int32_t)x;
    a.i = is_sum ? a.i + xi : (a.i > xi ? a.i : xi);
  }
}

// A warp owns strips of 32 * EV consecutive elements of the innermost kept loop; lane l takes
// elements l, l + 32, ... of a strip, so every load and store of the warp is coalesced.  Each
// warp takes `spw` consecutive strips of one row, so the index decoding is paid once per warp.
// Reduced loops (if any) are walked by each thread in loop order, exactly like the rendered loop
// nest, so a float sum is added in the reference's order.  What bounds an item is its words: some
// 2 us each over 12800 x 511 (a copy 10.2 us out of L2, gelu's 14 words 47; 12.8 and 65 with
// 64-bit divisions per warp, both classes computed by each word and a clamp per element).  Four
// elements a thread in place of eight: gelu 89 us, three CTAs per SM 57, where eight and four
// took 53.  Reducing programs are an instance of their own: with both in one, 430 bytes of a
// thread's registers lay in local memory (gelu 51 us, column sums 6.9 ms, 5.0 so).
template <int ND, int EV, bool HEAVY, bool REDUCES>
__global__ void __launch_bounds__(EXPR_THREADS, 4) expr_kernel(const __grid_constant__ caten_b200_expr e, const int64_t n_groups, const int groups_per_row, const int spw,
                                                            const int64_t n_red, const int result_cls) {
  extern __shared__ uint32_t expr_smem[];
  pdl_enter();
  const int64_t group = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (group >= n_groups) return;
  uint32_t *sm = expr_smem + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const int nd_out = e.ndim - e.n_reduce;
  const int va = nd_out - 1;  // the loop the strips run along (-1: a single output element)
  const int64_t vlen = va >= 0 ? e.shape[va] : 1;
  ExprIx<ND> ix;
#pragma unroll
  for (int d = 0; d < ND; ++d) ix.v[d] = 0;
  const int64_t row = (uint64_t)group >> 32 ? group / groups_per_row : (int64_t)((uint32_t)group / (uint32_t)groups_per_row);
  expr_decode(e, row, 0, va, ix);
  int64_t j0 = (group - row * groups_per_row) * spw * (32 * EV) + lane;  // this thread's first element; the others follow 32 apart
  const bool is_f = result_cls == CATEN_B200_CLS_F32, is_sum = e.reduce_op == CATEN_B200_RED_SUM;
  const int64_t ovs = va >= 0 ? 32 * e.out_stride[va] : 0;
  for (int s = 0; s < spw && j0 < vlen; ++s, j0 += 32 * EV) {
    const int lanes = (int)((vlen - j0 + 31) / 32 < EV ? (vlen - j0 + 31) / 32 : EV);  // elements of this thread in this strip
#pragma unroll
    for (int d = 0; d < ND; ++d)
      if (d == va) ix.v[d] = (int)j0;
    const int64_t out_at = expr_out_at(e, ix, nd_out);
    uint32_t val[EV];
    if (!REDUCES) {
      expr_run<ND, EV, EXPR_THREADS, HEAVY>(e, ix, va, lanes, val, sm);
      expr_store_ev<EV>(e.out, e.out_dtype, out_at, ovs, lanes, val, result_cls);
      continue;
    }
    ExprAcc acc[EV];
#pragma unroll
    for (int j = 0; j < EV; ++j) acc[j] = expr_acc_init(e, is_f, out_at + j * ovs, j < lanes);
    for (int64_t r = 0; r < n_red; ++r) {
      expr_decode(e, r, nd_out, e.ndim, ix);
      expr_run<ND, EV, EXPR_THREADS, HEAVY>(e, ix, va, lanes, val, sm);
#pragma unroll
      for (int j = 0; j < EV; ++j) expr_acc_add(acc[j], val[j], is_f, is_sum);
    }
#pragma unroll
    for (int j = 0; j < EV; ++j) val[j] = is_f ? __float_as_uint(acc[j].f) : (uint32_t)acc[j].i;
    expr_store_ev<EV>(e.out, e.out_dtype, out_at, ovs, lanes, val, result_cls);
  }
}

// Reduction whose single reduced loop is the contiguous one (row sums, softmax statistics).  Loads want lanes along the
// reduced loop, the reference's order of additions wants one adder per output element, and walking the lanes of a warp with
// shuffles spends a warp's instructions on a single sum.  So a CTA takes R output elements: eight warps evaluate tiles of
// R x C values with lanes along the reduced loop and leave them in shared memory (rows C + 1 apart, no bank conflicts), and a
// ninth warp, one lane per output element, adds the tile before in loop order meanwhile.  12800 rows of 511: 50 us with
// the shuffles (issue-bound: 8 instructions per value and row), 17 us with the tiles; 16 rows of 2048: 26 -> 14 us.  What is left
// of it is the chain of additions (4 cycles a value) and, on a cold input, the first tile's way from memory.
constexpr int RR_EV = 8, RR_WARPS = 8, RR_THREADS = (RR_WARPS + 1) * 32;
// columns of a tile: one strip, more where there are too few rows to give every warp one
__host__ __device__ constexpr int rr_cols(int R) { return R >= RR_WARPS ? 32 * RR_EV : 32 * RR_EV * RR_WARPS / R; }

// The ninth warp's part: adds the n values of each of a tile's rows to the row's accumulator (lane = row, or lanes row + R p).
__device__ __forceinline__ void rr_add_tile(const uint32_t *tile, const int pitch, const int n, const int R, const int rows, const int lane,
                                            const bool is_f, const bool is_sum, ExprAcc &acc) {
  if (is_f && is_sum) {
    if (lane < rows) {
      const uint32_t *src = tile + lane * pitch;
      int i = 0;
      if (n >= 16) {   // sixteen values on their way while sixteen are added
        uint32_t x[16], y[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) x[j] = src[j];
        for (; i + 32 <= n; i += 16) {
#pragma unroll
          for (int j = 0; j < 16; ++j) y[j] = src[i + 16 + j];
#pragma unroll
          for (int j = 0; j < 16; ++j) acc.f = acc.f + __uint_as_float(x[j]);
#pragma unroll
          for (int j = 0; j < 16; ++j) x[j] = y[j];
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) acc.f = acc.f + __uint_as_float(x[j]);
        i += 16;
      }
      for (; i < n; ++i) acc.f = acc.f + __uint_as_float(src[i]);
    }
    return;
  }
  // A maximum and an integer sum may be formed in parts, which are joined in order: up to 32 / R lanes take consecutive pieces of a
  // row (of odd length, for the banks), and a lane four consecutive parts of its piece side by side, so that its comparisons are
  // four chains.  A NaN forgets the values before it, as `acc > x ? acc : x` does.
  const int row = lane & (R - 1);
  int pieces = 32 / R;
  while (pieces > 1 && n < 32 * pieces) pieces >>= 1;
  const int len = ((n + pieces - 1) / pieces) | 1, i0 = min(n, lane / R * len), i1 = min(n, i0 + len);
  const uint32_t *src = tile + row * pitch;
  ExprAcc a = {-INFINITY, is_sum ? 0 : INT32_MIN};
  bool forgets = false;
  if (row < rows && i0 < i1) {
    if (is_f) {
      const int part = (i1 - i0) / 4;
      float m[4];
      bool nan[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) { m[q] = -INFINITY; nan[q] = false; }
#pragma unroll 4
      for (int i = 0; i < part; ++i) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float x = __uint_as_float(src[i0 + q * part + i]);
          m[q] = m[q] > x ? m[q] : x;
          nan[q] = nan[q] || x != x;
        }
      }
      if (part > 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          a.f = nan[q] || !(a.f > m[q]) ? m[q] : a.f;
          forgets = forgets || nan[q];
        }
      }
      for (int i = i0 + 4 * part; i < i1; ++i) {
        const float x = __uint_as_float(src[i]);
        a.f = a.f > x ? a.f : x;
        forgets = forgets || x != x;
      }
    } else {
#pragma unroll 8
      for (int i = i0; i < i1; ++i) expr_acc_add(a, src[i], false, is_sum);
    }
  }
  for (int p = 0; p < pieces; ++p) {
    const int from = row + p * R;
    const float f = __shfl_sync(0xffffffffu, a.f, from);
    const int i = __shfl_sync(0xffffffffu, a.i, from), any = __shfl_sync(0xffffffffu, (int)(i1 > i0), from), nan = __shfl_sync(0xffffffffu, (int)forgets, from);
    if (!any) continue;
    if (!is_f) expr_acc_add(acc, (uint32_t)i, false, is_sum);
    else acc.f = nan || !(acc.f > f) ? f : acc.f;
  }
}

// PLAIN: the program is one LOAD of floats, whose values go from memory to the tile by asynchronous copies, a whole tile ahead of
// the additions: through registers a warp had eight loads in flight, one strip after the other (12800 rows of 511, not in L2:
// sum 16.7 -> 13 us, maximum 17.5 -> 15).  Copies of four bytes: rows start anywhere.
template <int ND, bool HEAVY, bool PLAIN>
__global__ void __launch_bounds__(RR_THREADS, 3) expr_rowreduce_kernel(const __grid_constant__ caten_b200_expr e, const int64_t n_out, const int R,
                                                                    const int result_cls) {
  extern __shared__ uint32_t expr_smem[];
  pdl_enter();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int C = rr_cols(R), strips = C / (32 * RR_EV);   // per row of a tile
  uint32_t *tile = expr_smem;                              // 2 x R x (C + 1)
  uint32_t *sm = expr_smem + 2 * R * (C + 1) + tid;
  const int nd_out = e.ndim - 1, ra = e.ndim - 1;
  const int n_red = (int)e.shape[ra];
  const int64_t o0 = (int64_t)blockIdx.x * R;
  const int rows = n_out - o0 < R ? (int)(n_out - o0) : R;
  const bool is_f = result_cls == CATEN_B200_CLS_F32, is_sum = e.reduce_op == CATEN_B200_RED_SUM;
  ExprAcc acc = {0.0f, 0};
  int64_t out_at = 0;
  ExprIx<ND> ix;
#pragma unroll
  for (int d = 0; d < ND; ++d) ix.v[d] = 0;
  const int shift = 31 - __clz(strips);   // (a power of two)
  auto fill = [&](const int t) {
    uint32_t *dst = tile + (t & 1) * R * (C + 1);
    for (int s = warp; s < rows << shift; s += RR_WARPS) {
      const int row = s >> shift, col = (s & (strips - 1)) * (32 * RR_EV) + lane;   // this thread's first element of the strip, in the tile
      const uint32_t first = (uint32_t)t * C + col;                                 // and in the row
      if (first - lane >= (uint32_t)n_red) continue;
      const int n = first >= (uint32_t)n_red ? 0 : min(RR_EV, (int)(((uint32_t)n_red - first + 31) >> 5));   // its elements
      expr_decode(e, o0 + row, 0, nd_out, ix);
#pragma unroll
      for (int d = 0; d < ND; ++d)
        if (d == ra) ix.v[d] = n > 0 ? (int)first : 0;   // a lane past the end reads element 0 of the row
      uint32_t *to = dst + row * (C + 1) + col;
      if (PLAIN) {
        const int arg = (e.code[0] >> 8) & 255;
        int64_t o = e.operand_offset[arg];
#pragma unroll
        for (int d = 0; d < ND; ++d) o += (int64_t)ix.v[d] * e.operand_stride[arg][d];
        const float *p = reinterpret_cast<const float *>(e.operand[arg]) + o;
        const int64_t step = 32 * e.operand_stride[arg][ra];
        const uint32_t at = (uint32_t)__cvta_generic_to_shared(to);
        if (n == RR_EV && step == 32) {
#pragma unroll
          for (int j = 0; j < RR_EV; ++j) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(at + 128 * j), "l"(p + 32 * j) : "memory");
          continue;
        }
#pragma unroll
        for (int j = 0; j < RR_EV; ++j)
          if (j < n) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(at + 128 * j), "l"(p + j * step) : "memory");
        continue;
      }
      uint32_t val[RR_EV];
      expr_run<ND, RR_EV, RR_THREADS, HEAVY>(e, ix, ra, n, val, sm);
#pragma unroll
      for (int j = 0; j < RR_EV; ++j)
        if (j < n) to[32 * j] = val[j];
    }
  };
  if (PLAIN && warp < RR_WARPS) {
    for (int t = 0; t < 2; ++t) {
      fill(t);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
  }
  if (warp == RR_WARPS && lane < rows) {
    expr_decode(e, o0 + lane, 0, nd_out, ix);
    out_at = expr_out_at(e, ix, nd_out);
    acc = expr_acc_init(e, is_f, out_at, true);
  }
  const int tiles = n_red / C + (n_red % C != 0);
  auto add = [&](const int t) {
    const int64_t left = n_red - (int64_t)t * C;
    rr_add_tile(tile + (t & 1) * R * (C + 1), C + 1, left < C ? (int)left : C, R, rows, lane, is_f, is_sum, acc);
  };
  if (PLAIN) {
    for (int t = 0; t < tiles; ++t) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();   // tile t is there
      if (warp == RR_WARPS) add(t);
      if (t + 2 < tiles) {
        __syncthreads();   // its buffer is free
        if (warp < RR_WARPS) fill(t + 2);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");   // (empty at the end: the wait above counts groups)
    }
  } else {
    for (int t = 0; t <= tiles; ++t) {
      if (warp < RR_WARPS) {
        if (t < tiles) fill(t);
      } else if (t > 0) {
        add(t - 1);
      }
      __syncthreads();
    }
  }
  if (warp == RR_WARPS && lane < rows) expr_store(e.out, e.out_dtype, out_at, is_f ? __float_as_uint(acc.f) : (uint32_t)acc.i, result_cls);
}

// The same for short rows, which would leave most of a tile's strips empty: one warp per output element, lanes along the reduced
// loop; a warp evaluates 128 elements at a time and adds them in loop order by walking the lanes with shuffles.
constexpr int RW_EV = 4;
template <int ND, bool HEAVY>
__global__ void __launch_bounds__(EXPR_THREADS, 4) expr_rowwarp_kernel(const __grid_constant__ caten_b200_expr e, const int64_t n_out, const int result_cls) {
  extern __shared__ uint32_t expr_smem[];
  pdl_enter();
  const int64_t o_idx = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (o_idx >= n_out) return;  // whole warps leave together
  uint32_t *sm = expr_smem + threadIdx.x;
  const int lane = threadIdx.x & 31, nd_out = e.ndim - 1, ra = e.ndim - 1;
  const int64_t n_red = e.shape[ra];
  ExprIx<ND> ix;
#pragma unroll
  for (int d = 0; d < ND; ++d) ix.v[d] = 0;
  expr_decode(e, o_idx, 0, nd_out, ix);
  const int64_t out_at = expr_out_at(e, ix, nd_out);
  const bool is_f = result_cls == CATEN_B200_CLS_F32, is_sum = e.reduce_op == CATEN_B200_RED_SUM;
  ExprAcc acc = expr_acc_init(e, is_f, out_at, true);
  uint32_t val[RW_EV];
  for (int64_t r0 = 0; r0 < n_red; r0 += 32 * RW_EV) {
    const int64_t mine = r0 + lane;  // this lane's elements: mine, mine + 32, ...
    const int n = mine >= n_red ? 0 : (int)((n_red - mine + 31) / 32 < RW_EV ? (n_red - mine + 31) / 32 : RW_EV);
#pragma unroll
    for (int d = 0; d < ND; ++d)
      if (d == ra) ix.v[d] = n > 0 ? (int)mine : 0;   // a lane past the end reads element 0 of the row
    expr_run<ND, RW_EV, EXPR_THREADS, HEAVY>(e, ix, ra, n, val, sm);
#pragma unroll
    for (int j = 0; j < RW_EV; ++j) {
      const int64_t first = r0 + 32 * j;  // element of lane 0
      if (first >= n_red) break;
      const int n_here = (int)(n_red - first < 32 ? n_red - first : 32);
      auto walk = [&](auto add) {          // loop order: lane 0, 1, ..., 31
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          const uint32_t x = __shfl_sync(0xffffffffu, val[j], k);
          if (k < n_here) add(x);
        }
      };
      if (is_f && !is_sum) walk([&](uint32_t x) { expr_acc_add(acc, x, true, false); });
      else walk([&](uint32_t x) { expr_acc_add(acc, x, is_f, is_sum); });
    }
  }
  if (lane == 0) expr_store(e.out, e.out_dtype, out_at, is_f ? __float_as_uint(acc.f) : (uint32_t)acc.i, result_cls);
}

// Checks the program on the host (operand indices, stack discipline, classes) and returns the
// class of the value it leaves.
static int expr_validate(caten_b200_ctx *ctx, const caten_b200_expr *e, int *result_cls) {
  if (e->ndim < 1 || e->ndim > CATEN_B200_EXPR_MAX_DIMS) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: ndim %d outside 1..%d", e->ndim, CATEN_B200_EXPR_MAX_DIMS);
  if (e->n_reduce < 0 || e->n_reduce > e->ndim) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: n_reduce %d", e->n_reduce);
  if ((e->n_reduce > 0) != (e->reduce_op != CATEN_B200_RED_NONE) || e->reduce_op < 0 || e->reduce_op > CATEN_B200_RED_MAX)
    return fail(ctx, CATEN_B200_EINVAL, "eval_expr: reduce_op %d with %d reduced loops", e->reduce_op, e->n_reduce);
  if (e->n_operands < 0 || e->n_operands > CATEN_B200_EXPR_MAX_OPERANDS) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: %d operands", e->n_operands);
  if (e->n_code < 1 || e->n_code > CATEN_B200_EXPR_MAX_CODE) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: program of %d words", e->n_code);
  if (!e->out || e->out_dtype < 0 || e->out_dtype > CATEN_B200_DT_U8) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: output");
  for (int d = 0; d < e->ndim; ++d)
    if (e->shape[d] < 0 || e->shape[d] > 0x7fffffff) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: extent %lld of loop %d", (long long)e->shape[d], d);
  for (int i = 0; i < e->n_operands; ++i)
    if (!e->operand[i] || e->operand_dtype[i] < 0 || e->operand_dtype[i] > CATEN_B200_DT_U8)
      return fail(ctx, CATEN_B200_EINVAL, "eval_expr: operand %d", i);
  int cls_stack[16], sp = 0;
  for (int pc = 0; pc < e->n_code; ++pc) {
    const uint32_t w = e->code[pc];
    const int op = w & 255, arg = (w >> 8) & 255, cls = (w >> 16) & 255;
    if (cls > CATEN_B200_CLS_BOOL) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: class %d", pc, cls);
    if (op == CATEN_B200_OP_LOAD || op == CATEN_B200_OP_CONST || op == CATEN_B200_OP_INDEX) {
      if (op == CATEN_B200_OP_LOAD && arg >= e->n_operands) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d loads operand %d", pc, arg);
      if (op == CATEN_B200_OP_CONST && arg >= CATEN_B200_EXPR_MAX_CONSTS) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: constant %d", pc, arg);
      if (op == CATEN_B200_OP_INDEX && (arg >= e->ndim || cls != CATEN_B200_CLS_I32)) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: index of axis %d", pc, arg);
      if (op == CATEN_B200_OP_LOAD) {
        const int dt = e->operand_dtype[arg];
        const int want = dt == CATEN_B200_DT_F32 ? CATEN_B200_CLS_F32 : dt == CATEN_B200_DT_U8 ? CATEN_B200_CLS_BOOL : CATEN_B200_CLS_I32;
        if (cls != want) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: class %d for an operand of type %d", pc, cls, dt);
      }
      if (sp >= 16) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: stack deeper than 16");
      cls_stack[sp++] = cls;
    } else if (op >= CATEN_B200_OP_NEG && op <= CATEN_B200_OP_CAST) {
      if (sp < 1) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: empty stack", pc);
      const int have = cls_stack[sp - 1];
      if (op == CATEN_B200_OP_CAST) {
        if (arg != have) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: CAST from class %d, stack holds %d", pc, arg, have);
      } else {
        if (cls != have) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: class %d, stack holds %d", pc, cls, have);
        if (op >= CATEN_B200_OP_SIN && op <= CATEN_B200_OP_SQRT && cls != CATEN_B200_CLS_F32)
          return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: float-only op on class %d", pc, cls);
      }
      cls_stack[sp - 1] = op == CATEN_B200_OP_NOT ? CATEN_B200_CLS_BOOL : cls;
    } else if (op >= CATEN_B200_OP_ADD && op <= CATEN_B200_OP_LT) {
      if (sp < 2) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: needs two values", pc);
      if (cls_stack[sp - 1] != cls || cls_stack[sp - 2] != cls) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: operand classes differ from %d", pc, cls);
      if (op >= CATEN_B200_OP_MOD && op <= CATEN_B200_OP_XOR && cls == CATEN_B200_CLS_F32)
        return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: integer op on floats", pc);
      --sp;
      cls_stack[sp - 1] = (op == CATEN_B200_OP_NE || op == CATEN_B200_OP_LT) ? CATEN_B200_CLS_BOOL : cls;
    } else if (op == CATEN_B200_OP_WHERE) {
      if (sp < 3) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: needs three values", pc);
      if (cls_stack[sp - 1] != cls || cls_stack[sp - 2] != cls) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: branch classes differ from %d", pc, cls);
      sp -= 2;
      cls_stack[sp - 1] = cls;
    } else {
      return fail(ctx, CATEN_B200_EINVAL, "eval_expr: word %d: unknown opcode %d", pc, op);
    }
  }
  if (sp != 1) return fail(ctx, CATEN_B200_EINVAL, "eval_expr: the program leaves %d values", sp);
  *result_cls = cls_stack[0];
  return 0;
}

// Merges neighbouring loops that every view walks as one contiguous run (stride[d] ==
// stride[d+1] * extent[d+1], which also holds for two broadcast axes) and drops loops of extent
// 1, so that the strip a warp works on is as long as the data allows.  Kept and reduced loops
// are only merged among themselves; the visiting order of the elements does not change.
static void expr_collapse(caten_b200_expr *c) {
  for (int pc = 0; pc < c->n_code; ++pc)
    if ((c->code[pc] & 255) == CATEN_B200_OP_INDEX) return;  // loop indices are observable: keep the nest
  auto remove_loop = [&](int d) {
    for (int k = d; k + 1 < c->ndim; ++k) {
      c->shape[k] = c->shape[k + 1];
      c->out_stride[k] = c->out_stride[k + 1];
      for (int i = 0; i < c->n_operands; ++i) c->operand_stride[i][k] = c->operand_stride[i][k + 1];
    }
    --c->ndim;
  };
  int d = 0;
  while (d + 1 < c->ndim) {
    const int nd_out = c->ndim - c->n_reduce;
    const bool kept = d + 1 < nd_out, reduced = d >= nd_out;
    bool ok = kept || reduced;
    if (ok && c->shape[d + 1] != 1 && c->shape[d] != 1) {
      for (int i = 0; i < c->n_operands && ok; ++i) ok = c->operand_stride[i][d] == c->operand_stride[i][d + 1] * c->shape[d + 1];
      if (ok && kept) ok = c->out_stride[d] == c->out_stride[d + 1] * c->shape[d + 1];
    }
    // the kernels index a loop with an int: never build a fused loop longer than that
    if (ok && c->shape[d] > 1 && c->shape[d + 1] > 1 && c->shape[d] > (int64_t)INT32_MAX / c->shape[d + 1]) ok = false;
    if (!ok) { ++d; continue; }
    if (c->shape[d] == 1) {          // drop loop d
      remove_loop(d);
    } else if (c->shape[d + 1] == 1) {  // drop loop d + 1
      remove_loop(d + 1);
    } else {                         // fuse d + 1 into d: the fused loop steps with the inner stride
      c->shape[d] *= c->shape[d + 1];
      c->out_stride[d] = c->out_stride[d + 1];
      for (int i = 0; i < c->n_operands; ++i) c->operand_stride[i][d] = c->operand_stride[i][d + 1];
      remove_loop(d + 1);
    }
    if (reduced) --c->n_reduce;
  }
}

// Joins `LOAD b` / `CONST c` (and a NEG or RECIP of a float after it) with the binary word that uses it, and returns the
// depth of the stack that is left.  Values and the order of operations are those of the program given.
static int expr_fuse(caten_b200_expr *c) {
  int n = 0;
  for (int pc = 0; pc < c->n_code; ++pc) {
    uint32_t w = c->code[pc] & 0xffffffu;   // the bits above are the kernels' own
    const int op = w & 255, cls = (w >> 16) & 255;
    if (op >= CATEN_B200_OP_ADD && op <= CATEN_B200_OP_LT && n > 0) {
      uint32_t extra = 0;
      int from = n - 1, prev = c->code[from] & 255;
      if (cls == CATEN_B200_CLS_F32 && from > 0 && (prev == CATEN_B200_OP_NEG || prev == CATEN_B200_OP_RECIP)) {
        extra = prev == CATEN_B200_OP_NEG ? EXPR_NEG_B : EXPR_RECIP_B;
        prev = c->code[--from] & 255;
      }
      if (prev == CATEN_B200_OP_LOAD || prev == CATEN_B200_OP_CONST) {
        w = (w & 0xff00ffu) | (c->code[from] & 0xff00u) | (prev == CATEN_B200_OP_LOAD ? EXPR_WITH_LOAD : EXPR_WITH_CONST) | extra;
        n = from;
      }
    }
    c->code[n++] = w;
  }
  c->n_code = n;
  int sp = 0, depth = 1;
  for (int pc = 0; pc < n; ++pc) {
    const int op = c->code[pc] & 255;
    if (op == CATEN_B200_OP_LOAD || op == CATEN_B200_OP_CONST || op == CATEN_B200_OP_INDEX) ++sp;
    else if (op >= CATEN_B200_OP_ADD && op <= CATEN_B200_OP_LT) sp -= (c->code[pc] & EXPR_MODES) == EXPR_POP ? 1 : 0;
    else if (op == CATEN_B200_OP_WHERE) sp -= 2;
    if (sp > depth) depth = sp;
  }
  for (int pc = 0; pc < n; ++pc) {
    uint32_t &w = c->code[pc];
    const int op = w & 255;
    if (op >= CATEN_B200_OP_ADD && op <= CATEN_B200_OP_LT) w |= EXPR_BINARY;
    const bool shared = op == CATEN_B200_OP_LOAD || op == CATEN_B200_OP_NEG || op == CATEN_B200_OP_RECIP || op == CATEN_B200_OP_NOT || op == CATEN_B200_OP_ADD ||
                        op == CATEN_B200_OP_MUL || op == CATEN_B200_OP_MAX || op == CATEN_B200_OP_NE || op == CATEN_B200_OP_LT;
    if (shared && ((w >> 16) & 255) != CATEN_B200_CLS_F32) w += EXPR_WHOLE;
  }
  return depth;
}

template <int ND, int EV, bool HEAVY>
static int launch_expr_elements(caten_b200_ctx *ctx, const caten_b200_expr &e, int depth, int64_t rows, int64_t vlen, int64_t n_red, int result_cls) {
  // values under the top of the stack: [slot][element][thread] in shared memory
  const size_t smem = (size_t)(depth > 1 ? depth - 1 : 1) * EV * EXPR_THREADS * sizeof(uint32_t);
  auto kernel = e.n_reduce > 0 ? expr_kernel<ND, EV, HEAVY, true> : expr_kernel<ND, EV, HEAVY, false>;
  if (smem > 48 * 1024) CB_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t strips_per_row = (vlen + 32 * EV - 1) / (32 * EV);
  // strips per warp: as many as still leave every SM a full complement of warps, at most 16
  int64_t spw = (rows * strips_per_row) / ((int64_t)ctx->sm_count * 64);
  spw = spw < 1 ? 1 : spw > 16 ? 16 : spw;
  if (spw > strips_per_row) spw = strips_per_row;
  const int64_t groups_per_row = (strips_per_row + spw - 1) / spw;   // (a loop's extent has 31 bits)
  const int64_t n_groups = rows * groups_per_row;                    // one warp each
  const int64_t blocks = (n_groups + 7) / 8;
  if (blocks > 0x7fffffff) return fail(ctx, CATEN_B200_EUNSUPPORTED, "eval_expr: %lld output elements", (long long)(rows * vlen));
  launch_k(ctx, kernel, dim3((unsigned)blocks), dim3(EXPR_THREADS), smem, e, n_groups, (int)groups_per_row, (int)spw, n_red, result_cls);
  CB_LAUNCH_CHECK(ctx, "expr_kernel");
  return 0;
}

template <int ND, bool HEAVY>
static int launch_expr_rows(caten_b200_ctx *ctx, const caten_b200_expr &e, int depth, int64_t n_out, int result_cls) {
  // Short rows by a warp each (us, a warp each / tiles): 1000 rows of 64 sum 2.4 / 3.1, maximum 2.6 / 3.5, of 130 3.4 / 3.5, 3.9 /
  // 3.6; 12800 rows of 64 7.9 / 6.6.  With the heavy words, whose tiles have fewer warps: 12800 rows of 64 11 / 17, of 130 21 / 17.
  const int64_t n_red = e.shape[e.ndim - 1];
  if (n_red <= (HEAVY ? 128 : 96) && (HEAVY || n_out <= 8192)) {
    const int64_t blocks = (n_out + EXPR_THREADS / 32 - 1) / (EXPR_THREADS / 32);
    if (blocks > 0x7fffffff) return fail(ctx, CATEN_B200_EUNSUPPORTED, "eval_expr: %lld output elements", (long long)n_out);
    const size_t smem = (size_t)(depth > 1 ? depth - 1 : 1) * RW_EV * EXPR_THREADS * sizeof(uint32_t);
    if (smem > 48 * 1024) CB_CUDA(ctx, cudaFuncSetAttribute(expr_rowwarp_kernel<ND, HEAVY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    launch_k(ctx, expr_rowwarp_kernel<ND, HEAVY>, dim3((unsigned)blocks), dim3(EXPR_THREADS), smem, e, n_out, result_cls);
    CB_LAUNCH_CHECK(ctx, "expr_rowwarp_kernel");
    return 0;
  }
  // output elements per CTA: 32 keep the adding warp full; fewer while the CTAs are resident all at once (1000 rows of 768: two
  // per CTA are 500 CTAs and a second, short wave: 9.9 -> 11.5 us)
  int R = 32;
  while (R > 1 && (n_out + R / 2 - 1) / (R / 2) <= 3 * ctx->sm_count) R >>= 1;
  const int64_t blocks = (n_out + R - 1) / R;
  if (blocks > 0x7fffffff) return fail(ctx, CATEN_B200_EUNSUPPORTED, "eval_expr: %lld output elements", (long long)n_out);
  const bool plain = !HEAVY && e.n_code == 1 && (e.code[0] & 255) == CATEN_B200_OP_LOAD;   // (LOAD alone: of floats)
  const size_t tiles = 2 * (size_t)R * (rr_cols(R) + 1) * sizeof(uint32_t);
  const size_t smem = tiles + (plain ? 0 : (size_t)(depth > 1 ? depth - 1 : 1) * RR_EV * RR_THREADS * sizeof(uint32_t));
  auto kernel = plain ? expr_rowreduce_kernel<ND, false, true> : expr_rowreduce_kernel<ND, HEAVY, false>;
  if (smem > 48 * 1024) CB_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch_k(ctx, kernel, dim3((unsigned)blocks), dim3(RR_THREADS), smem, e, n_out, R, result_cls);
  CB_LAUNCH_CHECK(ctx, "expr_rowreduce_kernel");
  return 0;
}

int launch_expr(caten_b200_ctx *ctx, const caten_b200_expr *given) {
  int result_cls = 0;
  if (int rc = expr_validate(ctx, given, &result_cls)) return rc;
  caten_b200_expr collapsed = *given;
  expr_collapse(&collapsed);
  const int depth = expr_fuse(&collapsed);
  const caten_b200_expr *e = &collapsed;
  for (int d = e->ndim; d < MAXD; ++d) {   // loops that are not there do not move
    collapsed.out_stride[d] = 0;
    for (int i = 0; i < e->n_operands; ++i) collapsed.operand_stride[i][d] = 0;
  }
  bool heavy = false;
  for (int pc = 0; pc < e->n_code; ++pc) {
    const int op = e->code[pc] & 255;
    heavy = heavy || op == CATEN_B200_OP_SIN || op == CATEN_B200_OP_LOG2 || op == CATEN_B200_OP_SQRT || op == CATEN_B200_OP_MOD || op == CATEN_B200_OP_IDIV;
  }
  const int nd_out = e->ndim - e->n_reduce;
  int64_t n_out = 1, n_red = 1;
  for (int d = 0; d < nd_out; ++d) n_out *= e->shape[d];
  for (int d = nd_out; d < e->ndim; ++d) n_red *= e->shape[d];
  if (n_out == 0) return 0;
  if (e->n_reduce > 0 && n_red == 0 && !e->accumulate && e->reduce_op == CATEN_B200_RED_MAX)
    return fail(ctx, CATEN_B200_EINVAL, "eval_expr: max over an empty range");
  if (e->n_reduce == 1 && n_red >= 64) {
    // lanes along the reduced loop when that is where the operands are contiguous (or nothing else is left)
    bool unit_red = false, unit_kept = false;
    for (int i = 0; i < e->n_operands; ++i) {
      if (e->operand_stride[i][e->ndim - 1] == 1) unit_red = true;
      if (nd_out > 0 && e->operand_stride[i][nd_out - 1] == 1) unit_kept = true;
    }
    if (nd_out == 0 || (unit_red && !unit_kept)) {
      if (heavy) return e->ndim <= 2 ? launch_expr_rows<2, true>(ctx, *e, depth, n_out, result_cls) : launch_expr_rows<MAXD, true>(ctx, *e, depth, n_out, result_cls);
      return e->ndim <= 2 ? launch_expr_rows<2, false>(ctx, *e, depth, n_out, result_cls) : launch_expr_rows<MAXD, false>(ctx, *e, depth, n_out, result_cls);
    }
  }
  const int64_t vlen = nd_out > 0 ? e->shape[nd_out - 1] : 1, rows = n_out / vlen;
  if (heavy) return e->ndim <= 2 ? launch_expr_elements<2, 4, true>(ctx, *e, depth, rows, vlen, n_red, result_cls) : launch_expr_elements<MAXD, 4, true>(ctx, *e, depth, rows, vlen, n_red, result_cls);
  // Elements per thread: decoding a word costs about as much as applying it to four values, so eight, where that pads the
  // rows no further than four would and still gives every SM 16 warps; one where a row fits the lanes of a warp.
  const bool wide = (vlen + 255) / 256 * 256 == (vlen + 127) / 128 * 128 && rows * (vlen / 256) >= (int64_t)ctx->sm_count * 16;
  const int ev = vlen <= 32 ? 1 : wide ? 8 : 4;
#define EXPR_ELEMENTS(ND)                                                                              \
  ev == 1   ? launch_expr_elements<ND, 1, false>(ctx, *e, depth, rows, vlen, n_red, result_cls)        \
  : ev == 4 ? launch_expr_elements<ND, 4, false>(ctx, *e, depth, rows, vlen, n_red, result_cls)        \
            : launch_expr_elements<ND, 8, false>(ctx, *e, depth, rows, vlen, n_red, result_cls)
  return e->ndim <= 2 ? (EXPR_ELEMENTS(2)) : (EXPR_ELEMENTS(MAXD));
#undef EXPR_ELEMENTS
}

}  // namespace cb
