#include "grid_loop.cuh"

#include "host_util.h"

namespace mg {

namespace {

std::mutex &loop_mutex(int device) {
  static std::mutex m[16];
  return m[device & 15];
}

// What mg_selftest_loops asks of this thread's runs.
struct LoopTest {
  int32_t mode = MG_LOOP_TEST_OFF;
};
thread_local LoopTest loop_test;

}  // namespace

// Waits for the work in a caller's stream. (An error of that work comes back from the
// launch.)
static void drain(mg_graph *g, cudaStream_t s) {
  unsigned flags = 0;
  if (cudaStreamGetFlags(s, &flags) == cudaSuccess && (flags & cudaStreamNonBlocking)) {
    if (cudaStreamQuery(s) != cudaSuccess) {
      cudaGetLastError();  // not ready
      cudaStreamSynchronize(s);
    }
  } else if (cudaEventRecord(g->ev0, s) == cudaSuccess) {
    cudaEventSynchronize(g->ev0);  // with the default stream's work, which a launch would wait for
  }
}

LoopRun::LoopRun(mg_graph *g, cudaStream_t s) : g_(g), s_(s), turn_(loop_mutex(g->device), std::defer_lock) {
  if (s != g->stream) drain(g, s);  // the graph's own stream holds nothing that waits for anyone
  turn_.lock();
}

LoopRun::~LoopRun() { settle(nullptr); }

GridLoop LoopRun::args(const mg_options *o) {
  GridLoop l;
  l.c = g_->loop_ctl;
  l.base = g_->loop_base;
  l.spin_limit = (unsigned long long)o->spin_limit;
  l.out = g_->loop_out;
  if (loop_test.mode == MG_LOOP_TEST_WAITS) l.spin_limit = 1;
  g_->loop_out->error = MG_ERR_TIMEOUT;  // what it stays at when no CTA lives to write it
  g_->loop_out->timed_out = 0;
  return l;
}

int LoopRun::launch(const void *kernel, void **args, bool timed, const char *what) {
  cudaError_t e = timed ? cudaEventRecord(g_->ev0, s_) : cudaSuccess;
  if (e != cudaSuccess) return cuda_status(e, what);
  e = loop_test.mode == MG_LOOP_TEST_REFUSE
          ? cudaErrorCooperativeLaunchTooLarge
          : cudaLaunchCooperativeKernel(kernel, dim3(g_->num_sms), dim3(kLoopNT), args, 0, s_);
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
    cudaGetLastError();
    turn_.unlock();
    return kLoopRefused;
  }
  if (e != cudaSuccess) return cuda_status(e, what);
  launched_ = true;
  count_launch();
  if (timed) e = cudaEventRecord(g_->ev1, s_);
  return cuda_status(loop_test.mode == MG_LOOP_TEST_FAIL ? cudaErrorUnknown : e, what);
}

cudaError_t LoopRun::settle(int *error) {
  if (error) *error = MG_OK;
  if (!launched_) return cudaSuccess;
  launched_ = false;
  cudaError_t e = cudaStreamSynchronize(s_);
  const int err = e != cudaSuccess ? (int)MG_ERR_CUDA : g_->loop_out->timed_out ? (int)MG_ERR_TIMEOUT : g_->loop_out->error;
  if (err == MG_OK) {
    g_->loop_base += g_->loop_out->barriers * (uint32_t)g_->num_sms;
  } else {
    // the arrivals of a run that broke off are not known: start afresh
    g_->loop_base = 0;
    if (e == cudaSuccess) e = cudaMemsetAsync(g_->loop_ctl, 0, sizeof(LoopCtl), s_);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s_);
  }
  turn_.unlock();
  if (error) *error = err;
  return e;
}

int LoopRun::finish(cudaError_t e, const char *what) {
  int err;
  const cudaError_t es = settle(&err);
  if (e != cudaSuccess) return cuda_status(e, what);
  if (es != cudaSuccess) return cuda_status(es, what);
  if (err != MG_OK) return set_error(err, std::string(what) + ": device reported " + mg_status_string(err));
  return MG_OK;
}

}  // namespace mg

extern "C" int mg_selftest_loops(int32_t mode) {
  mg::clear_error();
  if (mode < MG_LOOP_TEST_OFF || mode > MG_LOOP_TEST_REFUSE) return mg::set_error(MG_ERR_ARG, "unknown loop test");
  mg::loop_test.mode = mode;
  return MG_OK;
}
