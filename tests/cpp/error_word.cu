// Leaves an error word in a handle's device counters, as a call that ended
// with that error does.  Test infrastructure: built and loaded by
// tests/test_gpu_error_words.py.
#include "polymer_b200_engine.cuh"

extern "C" __attribute__((visibility("default"))) int leave_error_word(pm_graph *g, int slot, unsigned word) {
  if (cudaSetDevice(g->device) != cudaSuccess) return 1;
  return cudaMemcpy(&g->E.d_cnt[slot].err, &word, sizeof word, cudaMemcpyHostToDevice) != cudaSuccess;
}

// 0, or the status of the failure that reading the counters raises.
extern "C" __attribute__((visibility("default"))) int read_error_words(pm_graph *g) {
  try {
    g->E.read_counters();
    return 0;
  } catch (const pm::Failure &f) {
    return (int)f.status;
  }
}
