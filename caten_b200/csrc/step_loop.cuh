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
  void *graph_xbf = nullptr, *graph_wtmp = nullptr, *graph_wbf = nullptr, *graph_side = nullptr;  // scratch pointers baked into the graph
  int64_t launches_per_step = 0;
};

inline int step_loop_alloc(caten_b200_ctx *ctx, StepLoop *l, int64_t B, int64_t T) {
  int rc = caten_b200_malloc(ctx, (size_t)B * sizeof(int64_t), (void **)&l->out_ids);
  if (!rc) rc = caten_b200_malloc(ctx, (size_t)B * sizeof(int64_t), (void **)&l->ids_io);
  if (!rc) rc = caten_b200_malloc(ctx, (size_t)B * T * sizeof(int64_t), (void **)&l->hist);
  if (!rc) rc = caten_b200_malloc(ctx, sizeof(int), (void **)&l->d_pos);
  return rc;
}

inline void step_loop_free(StepLoop *l) {
  if (l->graph) cudaGraphExecDestroy(l->graph);
  for (void *p : {(void *)l->ids_io, (void *)l->out_ids, (void *)l->hist, (void *)l->d_pos})
    if (p) cudaFree(p);
  *l = StepLoop();
}

// Captures one step's launches.  They are captured on the context's own stream, wherever the steps run: a caller's stream may
// be the legacy default stream, which cannot be captured, or one that synchronises with it.  Without a graph (l->graph stays
// NULL) the steps are launched one by one.
template <class Step>
void step_loop_capture(caten_b200_ctx *ctx, StepLoop *l, Step step, int64_t pos) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // of this thread: a capture of the caller's elsewhere forbids nothing here
  if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) { (void)cudaGetLastError(); return; }
  const cudaStream_t caller = ctx->stream;
  const int64_t before = ctx->launches;
  cudaGraph_t g = nullptr;
  ctx->stream = ctx->own_stream;
  if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
    const int rc = step(pos);
    if (cudaStreamEndCapture(ctx->stream, &g) != cudaSuccess || rc) l->graph = nullptr;
    else if (cudaGraphInstantiate(&l->graph, g, 0) != cudaSuccess) l->graph = nullptr;
  }
  if (g) cudaGraphDestroy(g);
  if (!l->graph) (void)cudaGetLastError();
  ctx->stream = caller;
  l->launches_per_step = ctx->launches - before;
  ctx->launches = before;  // captured, not launched
  cudaThreadExchangeStreamCaptureMode(&mode);
  l->graph_xbf = ctx->xbf.ptr;
  l->graph_wtmp = ctx->wtmp.ptr;
  l->graph_wbf = ctx->wbf.ptr;
  l->graph_side = ctx->wtmp_side.ptr;
}

// Runs `steps` single-token steps from the device-side state (ids_io and d_pos already loaded).  `step(n)` queues one
// step's kernels, which read ids and position from device memory; the host-side n only feeds argument checks.  With
// use_graph its launch sequence is captured the first time and replayed; into a stream that the caller is capturing the
// steps are launched one by one.
template <class Step>
int step_loop_run(caten_b200_ctx *ctx, StepLoop *l, int64_t n, int64_t steps, int64_t T, bool use_graph, Step step) {
  int64_t done = 0;
  use_graph = use_graph && !stream_is_capturing(ctx->stream) && !stream_is_capturing(ctx->own_stream);
  if (use_graph && l->graph && (l->graph_xbf != ctx->xbf.ptr || l->graph_wtmp != ctx->wtmp.ptr || l->graph_wbf != ctx->wbf.ptr || l->graph_side != ctx->wtmp_side.ptr)) {
    cudaGraphExecDestroy(l->graph);  // scratch was re-allocated since the capture: its pointers are stale
    l->graph = nullptr;
  }
  if (use_graph && !l->graph) {
    // the first step runs eagerly: it sizes the scratch buffers and sets kernel attributes, which
    // must not happen during capture
    if (int rc = step(n)) return rc;
    done = 1;
    step_loop_capture(ctx, l, step, n + 1 < T ? n + 1 : T - 1);
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
