// A vertex-centric functor over a value of VALUE_WORDS four-byte words, of ints
// and floats in turn: every expand of the engine has to build for it.
#include "engine/executor.cuh"
using namespace gsw;
using G = device_graph_t<CSR, Empty>;

struct value_t {
  int a[(VALUE_WORDS + 1) / 2];
#if VALUE_WORDS > 1
  float b[VALUE_WORDS / 2];
#endif
};

struct Gather : Functor<VC, value_t, int, Empty> {
  __device__ Status filter(int v, G) { return *ra_of(v) ? Active : Inactive; }
  __device__ value_t emit(int v, Empty *, G) { return *wa_of(v); }
  __device__ bool cond(int, value_t, G) { return true; }
  __device__ bool comp(value_t *v, value_t m, G) {
    v->a[0] += m.a[0];
    return true;
  }
  __device__ bool compAtomic(value_t *v, value_t m, G) {
    atomicAdd(&v->a[0], m.a[0]);
    return true;
  }
};

void expand(executor_t &ex, active_set_t &as, G &g, Gather &f, stat_t &st, feature_t &fets, config_t &conf) {
  ex.expand(as, g, f, st, fets, conf);
}
