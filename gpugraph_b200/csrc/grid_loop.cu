#include "grid_loop.cuh"

#include "host_util.h"

namespace mg {

std::mutex &loop_mutex(int device) {
  static std::mutex m[16];
  return m[device & 15];
}

cudaError_t loop_launch(mg_graph *g, const void *kernel, void **args, bool timed, cudaStream_t s) {
  cudaError_t e = timed ? cudaEventRecord(g->ev0, s) : cudaSuccess;
  if (e == cudaSuccess) e = cudaLaunchCooperativeKernel(kernel, dim3(g->num_sms), dim3(kLoopNT), args, 0, s);
  if (e == cudaSuccess && timed) e = cudaEventRecord(g->ev1, s);
  count_launch();
  return e;
}

GridLoop loop_begin(mg_graph *g, const mg_options *o) {
  GridLoop l;
  l.c = g->loop_ctl;
  l.base = g->loop_base;
  l.spin_limit = (unsigned long long)o->spin_limit;
  l.out = g->loop_out;
  g->loop_out->error = MG_ERR_TIMEOUT;  // what it stays at when no CTA lives to write it
  return l;
}

int loop_end(mg_graph *g, cudaStream_t s, const char *what) {
  const int err = g->loop_out->error;
  if (err == MG_OK) {
    g->loop_base += g->loop_out->barriers * (uint32_t)g->num_sms;
    return MG_OK;
  }
  // the arrivals of a run that broke off are not known: start afresh
  g->loop_base = 0;
  cudaError_t e = cudaMemsetAsync(g->loop_ctl, 0, sizeof(LoopCtl), s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_status(e, what);
  return set_error(err, std::string(what) + ": device reported " + mg_status_string(err));
}

}  // namespace mg
