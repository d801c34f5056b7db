// Device-resident decoding shared by the models: input ids, position and produced ids live on the
// device, and the launch sequence of a single-token step is captured into a CUDA graph and replayed.
#pragma once
#include "common.cuh"

namespace cb {

struct StepLoop {
  int64_t *ids_io = nullptr;    // [B] input ids of the next step
  int64_t *out_ids = nullptr;   // [B] ids the last step produced
  int64_t *hist = nullptr;      // [T, B] row n = ids produced by the step that started at position n
  int *d_pos = nullptr;         // position of the next step
  cudaGraphExec_t graph = nullptr;
  cudaGraphExec_t host_graph = nullptr;   // a step between the loading of the host's ids and the publishing of the new ones
  int64_t host_launches = 0;
  int *h_pos = nullptr;         // pinned: position that the host's next step is at
  void *graph_xbf = nullptr, *graph_wtmp = nullptr, *graph_wbf = nullptr, *graph_side = nullptr;  // scratch pointers baked into the graph
  int64_t launches_per_step = 0;
};

inline int step_loop_alloc(caten_b200_ctx *ctx, StepLoop *l, int64_t B, int64_t T) {
  int rc = caten_b200_malloc(ctx, (size_t)B * sizeof(int64_t), (void **)&l->out_ids);
  if (!rc) rc = caten_b200_malloc(ctx, (size_t)B * sizeof(int64_t), (void **)&l->ids_io);
  if (!rc) rc = caten_b200_malloc(ctx, (size_t)B * T * sizeof(int64_t), (void **)&l->hist);
  if (!rc) rc = caten_b200_malloc(ctx, sizeof(int), (void **)&l->d_pos);
  if (!rc && cudaMallocHost(&l->h_pos, sizeof(int)) != cudaSuccess) rc = fail(ctx, CATEN_B200_ECUDA, "cudaMallocHost(pos)");
  return rc;
}

inline void step_loop_free(StepLoop *l) {
  if (l->graph) cudaGraphExecDestroy(l->graph);
  if (l->host_graph) cudaGraphExecDestroy(l->host_graph);
  if (l->h_pos) cudaFreeHost(l->h_pos);
  for (void *p : {(void *)l->ids_io, (void *)l->out_ids, (void *)l->hist, (void *)l->d_pos})
    if (p) cudaFree(p);
  *l = StepLoop();
}

// Captures one step's launches.  They are captured on the context's own stream, wherever the steps run: a caller's stream may
// be the legacy default stream, which cannot be captured, or one that synchronises with it.  Without a graph (*graph stays
// NULL) the steps are launched one by one.
template <class Step>
void step_loop_capture(caten_b200_ctx *ctx, StepLoop *l, cudaGraphExec_t *graph, int64_t *per_step, Step step, int64_t pos) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // of this thread: a capture of the caller's elsewhere forbids nothing here
  if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) { (void)cudaGetLastError(); return; }
  const cudaStream_t caller = ctx->stream;
  const int64_t before = ctx->launches;
  cudaGraph_t g = nullptr;
  ctx->stream = ctx->own_stream;
  if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
    const int rc = step(pos);
    if (cudaStreamEndCapture(ctx->stream, &g) != cudaSuccess || rc) *graph = nullptr;
    else if (cudaGraphInstantiate(graph, g, 0) != cudaSuccess) *graph = nullptr;
  }
  if (g) cudaGraphDestroy(g);
  if (!*graph) (void)cudaGetLastError();
  ctx->stream = caller;
  *per_step = ctx->launches - before;
  ctx->launches = before;  // captured, not launched
  cudaThreadExchangeStreamCaptureMode(&mode);
  l->graph_xbf = ctx->xbf.ptr;
  l->graph_wtmp = ctx->wtmp.ptr;
  l->graph_wbf = ctx->wbf.ptr;
  l->graph_side = ctx->wtmp_side.ptr;
}

// Scratch was re-allocated since a capture: its pointers are stale.
inline void step_loop_drop_stale(caten_b200_ctx *ctx, StepLoop *l) {
  if (l->graph_xbf == ctx->xbf.ptr && l->graph_wtmp == ctx->wtmp.ptr && l->graph_wbf == ctx->wbf.ptr && l->graph_side == ctx->wtmp_side.ptr) return;
  for (cudaGraphExec_t *g : {&l->graph, &l->host_graph}) {
    if (*g) cudaGraphExecDestroy(*g);
    *g = nullptr;
  }
}

// One single-token step between host buffers: begin(n) loads ids and position from pinned host memory (the position from l->h_pos),
// step(n) is as below, publish() brings the result to pinned host memory.  All three are one graph: a launch before it and copies
// behind it cost a decode step 8 to 20 us (what a step from the host takes longer than one of a device-side loop: GPT-2 small, one
// sequence 24 -> 14 us, XL 30 -> 18; Binusun 1024, 16 sequences 38 -> 27; Goselix 1024, 64 sequences 37 -> 17).
template <class Begin, class Step, class Publish>
int step_loop_host_step(caten_b200_ctx *ctx, StepLoop *l, int64_t n, int64_t T, bool use_graph, Begin begin, Step step, Publish publish) {
  *l->h_pos = (int)n;
  auto all = [&](int64_t pos) {
    if (int rc = begin(pos)) return rc;
    ctx->weights_pending = true;   // the step's kernels take it that the position is there before the first of them starts
    if (int rc = step(pos)) return rc;
    return publish();
  };
  use_graph = use_graph && !stream_is_capturing(ctx->stream) && !stream_is_capturing(ctx->own_stream);
  if (use_graph) step_loop_drop_stale(ctx, l);
  if (use_graph && l->host_graph) {
    CB_CUDA(ctx, cudaGraphLaunch(l->host_graph, ctx->stream));
    ctx->launches += l->host_launches;
    return 0;
  }
  if (int rc = all(n)) return rc;   // sizes the scratch buffers and sets kernel attributes, which must not happen during capture
  if (use_graph) step_loop_drop_stale(ctx, l);   // (that step may have grown the scratch that the other graph uses)
  if (use_graph) step_loop_capture(ctx, l, &l->host_graph, &l->host_launches, all, n + 1 < T ? n + 1 : T - 1);
  return 0;
}

// Runs `steps` single-token steps from the device-side state (ids_io and d_pos already loaded).  `step(n)` queues one
// step's kernels, which read ids and position from device memory; the host-side n only feeds argument checks.  With
// use_graph its launch sequence is captured the first time and replayed; into a stream that the caller is capturing the
// steps are launched one by one.
template <class Step>
int step_loop_run(caten_b200_ctx *ctx, StepLoop *l, int64_t n, int64_t steps, int64_t T, bool use_graph, Step step) {
  int64_t done = 0;
  use_graph = use_graph && !stream_is_capturing(ctx->stream) && !stream_is_capturing(ctx->own_stream);
  if (use_graph) step_loop_drop_stale(ctx, l);
  if (use_graph && !l->graph) {
    // the first step runs eagerly: it sizes the scratch buffers and sets kernel attributes, which
    // must not happen during capture
    if (int rc = step(n)) return rc;
    done = 1;
    step_loop_drop_stale(ctx, l);
    step_loop_capture(ctx, l, &l->graph, &l->launches_per_step, step, n + 1 < T ? n + 1 : T - 1);
  }
  for (; done < steps; ++done) {
    if (use_graph && l->graph) {
      CB_CUDA(ctx, cudaGraphLaunch(l->graph, ctx->stream));
      ctx->launches += l->launches_per_step;
    } else if (int rc = step(n + done)) {
      return rc;
    }
  }
  return 0;
}

}  // namespace cb
